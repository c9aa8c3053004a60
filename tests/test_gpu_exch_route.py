"""Which starts a solve puts into their exchange sector, and the products of
those that it does: with maxit = 0 the solver normalises the start, detects its
symmetry, forms one product and returns the Ritz values and residual norms."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve_d(de, h, x, maxit, ns=0, order=2, sigma=-0.78):
    """de_gplmr_eig_d on a torch block, in place: (values, largest residual)."""
    from doublyexcited_b200._lib import de_complex, de_gmres, de_stats

    e = np.empty(x.shape[0], np.complex128)
    gm, st = de_gmres(order, 1, 1e-3, 0), de_stats()
    assert de.lib().de_gplmr_eig_d(h.handle, x.data_ptr(), e.ctypes.data, h.m, h.m, de_complex(sigma, 0.0), x.shape[0],
                                   ns, maxit, 1e-14, ctypes.byref(gm), 0, ctypes.byref(st)) == de.DE_OK
    return e, st.max_residual


def _sector(torch, n, nev, sign, seed):
    m = (2 * n + 1) ** 3
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(nev, m, m, dtype=torch.complex128, device="cuda", generator=gen)
    x = x + sign * x.transpose(1, 2)
    return x / torch.linalg.vector_norm(x, dim=(1, 2), keepdim=True)


@pytest.mark.parametrize("precision,n,nev", [("mixed", 2, 1), ("mixed", 3, 2), ("fp64", 3, 2), ("fp64", 5, 2),
                                             ("mixed", 5, 1)])
@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("eps", [5e-8, 1e-10, 1e-12])
def test_a_part_above_rounding_stays_in_the_start(de, precision, n, nev, sign, eps):
    import torch

    x = _sector(torch, n, nev, sign, 7 + n) + eps * _sector(torch, n, nev, -sign, 8 + n)
    with de.Problem(n=n, delta=2.0, theta=0.3, precision=precision) as h:
        h.set_stream(torch.cuda.current_stream().cuda_stream)
        _solve_d(de, h, x, 0)
    out = torch.linalg.vector_norm(x - sign * x.transpose(1, 2), dim=(1, 2)) / 2
    # the difference of two values of 1e-16 relative rounding leaves eps to 1e-16 / eps
    assert (out / eps - 1).abs().max().item() < 1e-3


@pytest.mark.parametrize("precision,n,nev", [("mixed", 3, 1), ("fp64", 5, 2)])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_rounding_leaves_the_sector(de, precision, n, nev, sign):
    """A start symmetric to a few units in the last place is made exactly so."""
    import torch

    x = _sector(torch, n, nev, sign, 9)
    gen = torch.Generator(device="cuda").manual_seed(1)
    ulps = torch.randint(-2, 3, x.shape, device="cuda", generator=gen).double()
    x = x * (1 + 2.0 ** -52 * ulps)
    assert not torch.equal(x, sign * x.transpose(1, 2))
    with de.Problem(n=n, delta=2.0, theta=0.3, precision=precision) as h:
        h.set_stream(torch.cuda.current_stream().cuda_stream)
        _solve_d(de, h, x, 0)
    assert torch.equal(x, sign * x.transpose(1, 2))


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("n", [1, 4, 5, 6, 7, 8, 9, 10, 11])
def test_one_symmetric_product_matches_the_general_one(de, n, sign):
    """Ritz value and residual norm of one product on an exactly symmetric start
    (the two-kernel product) against those of de_matblock_d's."""
    import torch

    x = _sector(torch, n, 2, sign, 10 + n)
    with de.Problem(n=n, delta=2.0, theta=0.3) as h:
        h.set_stream(torch.cuda.current_stream().cuda_stream)
        y = torch.empty_like(x)
        h.matblock_d(x.data_ptr(), y.data_ptr(), 2)
        e = (x.conj() * y).sum(dim=(1, 2))
        y -= e[:, None, None] * x
        want = torch.linalg.vector_norm(y, dim=(1, 2)).max().item()
        e = e.cpu().numpy()
        got, res = _solve_d(de, h, x, 0)
    # FP64 rounding of 6 NN products an output and of sums over the vector
    assert np.abs(got - e).max() < 1e-12 * np.abs(e).max()
    assert abs(res - want) < 1e-12 * want


@pytest.mark.parametrize("n", [6, 7, 8, 9])
def test_complex64_symmetric_products_match_the_general_ones(de, n):
    """One mixed iteration on a triplet start against the same one with the
    streaming kernels' complex64 products, which keep no sector."""
    import torch

    e = []
    for family in ("fma", "stream"):
        x = _sector(torch, n, 1, -1.0, 20 + n)
        with de.Problem(n=n, delta=2.0, theta=0.3, precision="mixed") as h:
            h.set_stream(torch.cuda.current_stream().cuda_stream)
            for pass_ in (0, 1):
                h.set_matvec_launch("c64", pass_, family, 0)
            e.append(_solve_d(de, h, x, 1, ns=1)[0])
            if family == "fma":
                assert torch.equal(x, -x.transpose(1, 2))
    # complex64 rounding of the search directions, 6e-8 times H's spread of
    # about 10, times a handful of chained products
    assert np.abs(e[0] - e[1]).max() < 1e-5


@pytest.mark.parametrize("precision,nev", [("mixed", 1), ("fp64", 3)])
@pytest.mark.parametrize("spin", [1.0, -1.0])
def test_reflection_symmetric_starts_keep_the_sector_bit_for_bit(de, precision, nev, spin):
    """Gaussian starts reach one reflection sector only, so every preconditioned
    block is also projected by reflections, on a grid whose sums and updates
    take the upper half for granted."""
    import torch

    n = 5
    c = torch.arange(-n, n + 1, dtype=torch.float64, device="cuda")
    r2 = (c[:, None, None] ** 2 + c[None, :, None] ** 2 + c[None, None, :] ** 2).reshape(-1)
    g = [torch.exp(-a * r2) for a in (0.9, 0.31, 0.12, 0.05)]
    x = torch.stack([torch.outer(g[j], g[j + 1]) * (1 + 0.3j) for j in range(nev)])
    x = (x + spin * x.transpose(1, 2)).contiguous()
    with de.Problem(n=n, delta=2.0, theta=0.3, precision=precision) as h:
        h.set_stream(torch.cuda.current_stream().cuda_stream)
        _solve_d(de, h, x, 3, ns=2, order=3)
    assert torch.equal(x, spin * x.transpose(1, 2))
    v = x.view(nev, *([2 * n + 1] * 6))  # (k2, j2, i2, k1, j1, i1)
    for axis in (1, 2, 3):
        assert torch.linalg.vector_norm(v - v.flip(axis, axis + 3)).item() < 1e-12
