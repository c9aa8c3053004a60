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


# nev 2, 5 and 9: the two widths of the upper-half update and, above 8 columns,
# the general one.  Both sides are FP64; their rounding (1e-15) is amplified by
# the conditioning of the k x k Grams, which the self-check holds below 1e5.
@pytest.mark.parametrize("nev,order", [(2, 6), (5, 3), (9, 2)])
def test_block_solve_on_upper_halves(de, oracle, nev, order):
    p = oracle.Params(n=5, delta=2.0, theta=0.3)
    x0 = oracle.seeded_start(p, nev, 31, "singlet")
    e = []
    for family in ("fma", "stream"):  # the latter's products keep no sector: whole vectors
        with de.Problem(n=5, delta=2.0, theta=0.3) as h:
            for pass_ in (0, 1):
                h.set_matvec_launch("c128", pass_, family, 0)
            e.append(h.gplmr_eig(x0, -0.78, ns=1, maxit=1, tol=1e-14, max_inner_iter=order).e)
    assert np.abs(e[0] - e[1]).max() < 1e-9


# The outer iteration's upper-half vectors, for one column with few and with
# more than nine basis vectors and for blocks; two iterations, so that all of X,
# AX, P and AP enter the second.  FP64 rounding as above; complex64 as TOL.
@pytest.mark.parametrize("precision,nev,ns", [("mixed", 1, 2), ("mixed", 1, 9), ("fp64", 3, 2), ("fp64", 9, 1)])
def test_outer_iteration_on_upper_halves(de, oracle, precision, nev, ns):
    x0 = oracle.seeded_start(oracle.Params(n=5, delta=2.0, theta=0.3), nev, 51, "triplet")
    e, res = [], []
    for family in ("fma", "stream"):
        with de.Problem(n=5, delta=2.0, theta=0.3, precision=precision) as h:
            for pass_ in (0, 1):
                h.set_matvec_launch("c128", pass_, family, 0)
            r = h.gplmr_eig(x0, -0.78, ns=ns, maxit=2, tol=1e-14, max_inner_iter=3)
            e.append(r.e)
            res.append(r.max_residual)
    tol = 1e-9 if precision == "fp64" else TOL
    assert np.abs(e[0] - e[1]).max() < tol
    assert abs(res[0] - res[1]) < tol


def test_block_solve_of_an_exhausted_space(de):
    """On 27 points a spherical singlet start reaches 24 states (the
    orbits of point pairs under the cube's symmetries and exchange), so Krylov
    blocks of two columns run out of them by the 12th: what Gram-Schmidt leaves of
    the next is rounding, and more blocks do not change the solution."""
    c = np.arange(3) - 1.0
    r2 = (c[:, None, None] ** 2 + c[None, :, None] ** 2 + c[None, None, :] ** 2).ravel()
    x0 = np.stack([np.outer(np.exp(-a * r2), np.exp(-b * r2)).ravel() + np.outer(np.exp(-b * r2), np.exp(-a * r2)).ravel()
                   for a, b in ((0.3, 0.3), (0.8, 0.1))], 1).astype(complex)
    e = []
    for order in (20, 30):
        with de.Problem(n=1, delta=2.0, theta=0.3) as h:
            e.append(h.gplmr_eig(x0, -0.78, ns=1, maxit=2, tol=1e-9, max_inner_iter=order).e)
    # the solves are exact but for the rounding the last blocks add
    assert np.abs(e[0] - e[1]).max() < 1e-9
