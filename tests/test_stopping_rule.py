"""The resident solve's stopping bound (csrc/cg_limit.h) against the rule it stands
for, over every kind of ||b|| and eps a configuration can hold.  The header is
compiled for the host; a search that does not end fails by its time limit."""
import math
import os
import struct
import subprocess

import numpy as np
import pytest

from tests.conftest import REPO

SOURCE = """
#include <cstdio>
#include "cg_limit.h"
int main() {
  double v[2];
  while (fread(v, sizeof(double), 2, stdin) == 2) {
    const double t = frehd::res_limit(v[0], v[1]);
    fwrite(&t, sizeof t, 1, stdout);
  }
}
"""
BNORMS = [0.0, 5e-324, 1e-300, 1e-170, 1e-160, 1e-12, 1.0, 3.7, 1e12, 1e155, 1e300, math.inf, math.nan]
EPSES = [1e-12, 1e-6, 0.5, 1.0, 3.0, 1e-200, 1e-320, 1e200, 0.0, -1e-12, -1.0, math.inf, -math.inf, math.nan]


@pytest.fixture(scope="module")
def limits(tmp_path_factory):
    d = tmp_path_factory.mktemp("limit")
    (d / "limit.cpp").write_text(SOURCE)
    exe = str(d / "limit")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(REPO, "frehdc_b200", "csrc"),
                    str(d / "limit.cpp"), "-o", exe], check=True)

    def run(pairs):
        out = subprocess.run([exe], input=b"".join(struct.pack("dd", *p) for p in pairs), check=True,
                             stdout=subprocess.PIPE, timeout=20).stdout
        return struct.unpack("%dd" % len(pairs), out)
    return run


def _holds(rr, bnorm, eps):
    with np.errstate(all="ignore"):
        rn, c = np.sqrt(np.float64(rr)), np.float64(eps) * np.float64(bnorm)
        return bool(rn < c or (bnorm == 0.0 and 1.0 + rn == 1.0))


@pytest.mark.parametrize("bnorm", BNORMS)
def test_limit_is_the_rule(limits, bnorm):
    pairs = [(bnorm, e) for e in EPSES]
    for (b, e), t in zip(pairs, limits(pairs)):
        if t < 0:  # no residual meets the rule
            assert not any(_holds(r, b, e) for r in (0.0, 5e-324, 1e-300, 1e-30, 1.0, 1e300)), (b, e)
        else:
            assert _holds(t, b, e), (b, e, t)
            with np.errstate(over="ignore"):
                above = np.nextafter(t, np.inf)
            assert not _holds(above, b, e), (b, e, t)
