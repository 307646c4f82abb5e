"""The tile width of the prefill GEMMs (csrc/qkm_units.h): a shard that was sent the rows which chose one of its experts takes the
width that the same experts take when every row is at hand."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "qkm_units.h"
#include <cstdio>
#include <cstdlib>
int main(int, char** v) {
    const double m = qkm::mean_pairs(atoi(v[1]), atoi(v[2]), atoi(v[3]), atoi(v[4]), atoi(v[5]) != 0);
    std::printf("%.6f %u\n", m, qkm::wgemm_rows_per_unit(m));
    return 0;
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("units")
    (d / "units.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I" + os.path.join(ROOT, "qwen-kernel_b200", "csrc"), str(d / "units.cpp"), "-o", str(d / "units")], check=True)

    def call(*args):
        mean, rows = subprocess.run([str(d / "units"), *[str(int(a)) for a in args]], check=True, capture_output=True, text=True).stdout.split()
        return float(mean), int(rows)
    return call


def test_all_rows(rule):
    for tokens, want in ((77, 128), (3679, 128), (3712, 160), (4096, 160), (5280, 160), (5281, 128)):
        assert rule(tokens, 8, 256, 256, 0) == (pytest.approx(tokens * 8 / 256), want)


@pytest.mark.parametrize("ranks", [2, 4, 8])
def test_rows_sent_to_a_shard(rule, ranks):
    rng = np.random.default_rng(1)
    tokens, resident = 4096, 256 // ranks
    ids = np.argsort(rng.random((tokens, 256)), axis=1)[:, :8]
    here = ids < resident
    sent = int(here.any(axis=1).sum())
    mean, rows = rule(sent, 8, 256, resident, 1)
    assert mean == pytest.approx(here.sum() / resident, rel=0.03)   # (the experts of a row are drawn without replacement)
    assert rows == rule(tokens, 8, 256, 256, 0)[1] == 160
