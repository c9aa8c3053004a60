"""The caller's vectors after a solve that ends in an error: the host eigensolver
is replaced by one that fails from its third call on, in a process of its own
(the library loads its LAPACK once)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

SCRIPT = """
import ctypes, sys
import numpy as np, torch
import doublyexcited_b200 as de
from doublyexcited_b200._lib import de_complex, de_gmres, de_stats

precision, n, nev, sign = sys.argv[1], int(sys.argv[2]), int(sys.argv[3]), float(sys.argv[4])
with de.Problem(n=n, delta=2.0, theta=0.3, precision=precision) as h:
    h.set_stream(torch.cuda.current_stream().cuda_stream)
    gen = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(nev, h.m, h.m, dtype=torch.complex128, device="cuda", generator=gen)
    x = (x + sign * x.transpose(1, 2)).contiguous()
    e, gm, st = np.empty(nev, np.complex128), de_gmres(3, 1, 1e-3, 0), de_stats()
    status = de.lib().de_gplmr_eig_d(h.handle, x.data_ptr(), e.ctypes.data, h.m, h.m, de_complex(-0.78, 0.0), nev, 1, 9,
                                     1e-14, ctypes.byref(gm), 0, ctypes.byref(st))
    torch.cuda.synchronize()
    assert status == de._lib.DE_E_GEVP, status
    assert b"zggev info=3" in de.lib().de_last_error()
    norms = torch.linalg.vector_norm(x, dim=(1, 2))
    assert (norms - 1).abs().max().item() < 1e-12, norms
    assert torch.equal(x, sign * x.transpose(1, 2))
print("ok")
"""


@pytest.fixture(scope="module")
def failing_lapack(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("lapack") / "libfailing.so")
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", os.path.join(HERE, "failing_lapack.c"), "-o", out, "-ldl"],
                   check=True)
    return out


@pytest.mark.parametrize("precision,n,nev,sign", [("mixed", 5, 1, 1.0), ("mixed", 5, 2, -1.0), ("fp64", 5, 2, 1.0),
                                                  ("fp64", 3, 2, 1.0)])
def test_vectors_after_an_error_are_the_last_iterate(failing_lapack, precision, n, nev, sign):
    sys.path.insert(0, ROOT)
    from __graft_entry__ import _lapack_default

    env = dict(os.environ, DE_LAPACK_LIB=failing_lapack, REAL_LAPACK=_lapack_default() or "liblapack.so.3", FAIL_AT="3",
               PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", SCRIPT, precision, str(n), str(nev), str(sign)], env=env, cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stderr[-2000:]
