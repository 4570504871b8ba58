"""Where the host looks at a GMRES cycle: at the step where the residual's rate says
it ends, and not inside the cycle where it does not end there: a rate that reaches
past the restart, no fall, or a threshold of zero (a run to a fixed budget)."""
import ctypes as C
import math
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cfdrs_b200", "csrc")


@pytest.fixture(scope="module")
def next_look(tmp_path_factory):
    d = tmp_path_factory.mktemp("look")
    (d / "shim.cpp").write_text('#include "gmres_look.h"\nextern "C" int next_look(int done, int m, double rn, double thr, '
                                'double rate) { return cfd::gmres_next_look(done, m, rn, thr, rate); }\n')
    so = str(d / "shim.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", so, str(d / "shim.cpp")], check=True)
    f = C.CDLL(so).next_look
    f.argtypes = [C.c_int, C.c_int, C.c_double, C.c_double, C.c_double]
    return f


@pytest.mark.parametrize("done,m,rn,threshold,rate,look", [
    # four decades at one a step: the quotient of the logarithms rounds to 4 or just above
    (8, 32, 1e-4, 1e-8, 0.1, (12, 13)), (0, 32, 1e-4, 1e-8, 0.1, (4, 5)),
    (8, 32, 1e-4, 1e-8, 0.9, 32),                                # 88 steps: past the restart
    (8, 32, 1e-4, 0.0, 0.1, 32), (0, 32, 1e-4, 0.0, 0.1, 32),    # no threshold to pass
    (8, 32, 1e-4, 1e-8, 1.0, 32), (8, 32, 1e-4, 1e-8, 1.5, 32), (8, 32, 1e-4, 1e-8, 0.0, 32),
    (8, 32, 1e-4, 1e-8, math.nan, 32),
    (8, 32, 1e-9, 1e-8, 0.5, 9), (31, 32, 1e-4, 1e-8, 0.1, 32),  # already there; the cycle's end
    (8, 256, 1e-4, 1e-8, 1.0 - 1e-16, 256),
])
def test_next_look(next_look, done, m, rn, threshold, rate, look):
    assert next_look(done, m, rn, threshold, rate) in (look if isinstance(look, tuple) else (look,))
