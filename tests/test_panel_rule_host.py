"""The rule that lets a panel of the integrand be interpolated (gfk_panel.cuh),
compiled for the host: a node that overflowed or is not a number is never
accepted, whatever its other part is. Such a node reaches every coefficient: none of the
table's rows has a zero."""
import pathlib
import shutil
import subprocess

import pytest

CSRC = next(pathlib.Path(__file__).resolve().parents[1].glob("*_b200")) / "csrc"
MAIN = """
#include "gfk_panel.cuh"
#include <cstdio>
#include <cstdlib>
int main(int argc, char** argv) {
    for (int i = 1; i + 1 < argc; i += 2) printf("%d", (int)gfk::panel_passes(atof(argv[i]), atof(argv[i + 1])));
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("panel")
    (d / "main.cpp").write_text(MAIN)
    cuda = pathlib.Path(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc").resolve().parents[1] / "include"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(CSRC), "-isystem", str(cuda), "-o", str(d / "rule"),
                    str(d / "main.cpp")], check=True)
    return lambda *v: subprocess.run([str(d / "rule"), *map(str, v)], check=True, capture_output=True, text=True).stdout


@pytest.mark.parametrize("tail,scale,passes", [
    (0.0, 1.0, "1"), (0.9e-15, 1.0, "1"), (1.1e-15, 1.0, "0"), (0.9e285, 1e300, "1"), (1.0, 1e300, "1"),
    ("inf", 1e300, "0"), ("inf", "inf", "0"), (0.0, "nan", "0"), ("nan", "nan", "0"),
    ("inf", "nan", "0"),
])
def test_overflowed_nodes_are_refused(rule, tail, scale, passes):
    assert rule(tail, scale) == passes


def test_every_node_reaches_every_last_coefficient(tmp_path):
    (tmp_path / "main.cpp").write_text("""
#include <cmath>
#include "gfk_panel.cuh"
#include <cstdio>
int main() {
    const auto t = gfk::panel_table();
    double least = 1;
    for (int c = 0; c < 3; c++) {
        for (int j = 0; j < gfk::kPanelE; j++) least = fmin(least, fabs(t[gfk::kPtRowsE + (j >> 2) * 32 + 4 * c + (j & 3)]));
        for (int j = 0; j < gfk::kPanelN; j++) least = fmin(least, fabs(t[gfk::kPtRowsN + (j >> 2) * 32 + 4 * c + (j & 3)]));
    }
    printf("%g", least);
}
""")
    cuda = pathlib.Path(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc").resolve().parents[1] / "include"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(CSRC), "-isystem", str(cuda), "-o", str(tmp_path / "t"),
                    str(tmp_path / "main.cpp")], check=True)
    assert float(subprocess.run([str(tmp_path / "t")], check=True, capture_output=True, text=True).stdout) > 0
