"""The mixed form's inner products on exchange-symmetric vectors (one cube
kernel and a transposed add): one preconditioned step from singlet and
triplet starts against the FP64 solve's, on grids whose 32 x 32 tiles end
ragged, for one column and a block; and starts whose symmetry is broken
above and below what switches the products over."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# After one step the Ritz values of the two forms differ by the complex64
# rounding of the search directions: 6e-8 times the spread of H's spectrum
# (about 10 at this spacing) times the handful of inner products chained.
TOL = 1e-5


def _one_step(de, n, x0, precision, nev):
    with de.Problem(n=n, delta=2.0, theta=0.3, precision=precision) as h:
        return h.gplmr_eig(x0, -0.78, ns=2, maxit=1, tol=1e-14, max_inner_iter=3)


@pytest.mark.parametrize("spin", ["singlet", "triplet"])
@pytest.mark.parametrize("n,nev", [(1, 1), (2, 1), (3, 1), (3, 3), (4, 1), (5, 2)])
def test_symmetric_products_match_fp64(de, oracle, n, nev, spin):
    x0 = oracle.seeded_start(oracle.Params(n=n, delta=2.0, theta=0.3), nev, 11 + n, spin)
    r64, r32 = (_one_step(de, n, x0, prec, nev) for prec in ("fp64", "mixed"))
    assert np.abs(r64.e - r32.e).max() < TOL
    m = (2 * n + 1) ** 3
    s = 1.0 if spin == "singlet" else -1.0
    for j in range(nev):  # the Ritz vectors stay in the start's sector
        x = r32.x[:, j].reshape(m, m)
        assert np.linalg.norm(x - s * x.T) < 1e-12 * np.linalg.norm(x)


@pytest.mark.parametrize("eps", [1e-10, 1e-6, 1e-2])
def test_nearly_symmetric_starts(de, oracle, eps):
    n = 3
    p = oracle.Params(n=n, delta=2.0, theta=0.3)
    x0 = oracle.seeded_start(p, 1, 3, "singlet") + eps * oracle.seeded_start(p, 1, 4, "triplet")
    r64, r32 = (_one_step(de, n, x0, prec, 1) for prec in ("fp64", "mixed"))
    # a part of size eps outside the sector enters the Ritz value squared, but
    # the mixed form drops it from the new directions where it keeps the sector
    assert np.abs(r64.e - r32.e).max() < TOL + 10 * eps


@pytest.mark.parametrize("precision,n,nev", [("mixed", 3, 1), ("mixed", 5, 1), ("mixed", 4, 2), ("fp64", 3, 4),
                                             ("fp64", 5, 2), ("fp64", 5, 5)])
@pytest.mark.parametrize("spin", ["singlet", "triplet"])
def test_iteration_keeps_the_sector_bit_for_bit(de, oracle, precision, n, nev, spin):
    """Nothing in the iteration may leave X^T = +-X by a single bit: sums and
    updates take the upper half of the vectors for granted (N >= 5), and no
    projection follows the preconditioner."""
    p = oracle.Params(n=n, delta=2.0, theta=0.3)
    x0 = oracle.seeded_start(p, nev, 21, spin)
    with de.Problem(n=n, delta=2.0, theta=0.3, precision=precision) as h:
        r = h.gplmr_eig(x0, -0.78, ns=2, maxit=3, tol=1e-14, max_inner_iter=3)
    s = 1.0 if spin == "singlet" else -1.0
    for j in range(nev):
        x = r.x[:, j].reshape(p.m, p.m)
        assert np.array_equal(x, s * x.T)
