"""Gram matrices on shared-memory output tiles (de_dots_d): widths at the
edges of the 4 x 4 tiles and of a launch's 8 tiles, row counts at the edges
of a stage, the shortest vector, and columns shared by both sides, against
torch in complex128."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [1, 63, 64, 65, 257, 16384, 262144, 300007, 1048577])
@pytest.mark.parametrize("nbra,nket,herm", [(4, 4, 1), (5, 4, 0), (1, 3, 1), (3, 2, 0), (8, 17, 1), (33, 4, 0),
                                            (13, 29, 1), (2, 32, 0), (32, 16, 1), (64, 1, 0), (40, 17, 1),
                                            (24, 24, 1), (1, 2, 0), (2, 2, 1), (12, 1, 1), (32, 1, 0)])
def test_dots_tiles(de, size, nbra, nket, herm):
    import torch

    gen = torch.Generator(device="cuda").manual_seed(size + 100 * nbra + nket)
    both = torch.randn(nbra + nket, size, dtype=torch.complex128, device="cuda", generator=gen)
    bras, kets = both[:nbra], both[nbra:]
    L = de.lib()
    with de.Problem(n=1, delta=2.0, theta=0.3) as g:
        g.set_stream(torch.cuda.current_stream().cuda_stream)

        def dots(b, k, nb, nk):
            out = np.full((nk, nb), np.nan, np.complex128)
            assert L.de_dots_d(g.handle, ctypes.c_void_p(b.data_ptr()), ctypes.c_void_p(k.data_ptr()), size, nb, nk,
                               ctypes.c_void_p(out.ctypes.data), herm) == de.DE_OK
            return out

        got = dots(bras, kets, nbra, nket)
        want = (kets @ (bras.conj() if herm else bras).T).cpu().numpy()
        # both sum `size` products of unit variance: rounding is below
        # size * 1.1e-16 of their absolute sum, itself about size
        tol = 1e-15 * (size + 100)
        assert np.abs(got - want).max() < tol
        assert np.array_equal(got, dots(bras, kets, nbra, nket))  # fixed order
        m = min(nbra, 5)  # the same columns on both sides
        same = dots(bras, bras, m, m)
        want = (bras[:m] @ (bras[:m].conj() if herm else bras[:m]).T).cpu().numpy()
        assert np.abs(same - want).max() < tol


@pytest.mark.parametrize("size", [1, 255, 257, 513, 300007])
@pytest.mark.parametrize("nbra", [2, 3, 5, 8, 9, 10])
def test_dots_one_ket(de, size, nbra):
    """One ket against 2..9 bras (their own kernel, the ket being the last bra
    or not) and 10 (the general one)."""
    import torch

    gen = torch.Generator(device="cuda").manual_seed(size + nbra)
    both = torch.randn(nbra + 1, size, dtype=torch.complex128, device="cuda", generator=gen)
    L = de.lib()
    with de.Problem(n=1, delta=2.0, theta=0.3) as g:
        g.set_stream(torch.cuda.current_stream().cuda_stream)
        for herm in (0, 1):
            for ket in (both[nbra], both[nbra - 1]):
                out = np.full(nbra, np.nan, np.complex128)
                assert L.de_dots_d(g.handle, ctypes.c_void_p(both.data_ptr()), ctypes.c_void_p(ket.data_ptr()), size,
                                   nbra, 1, ctypes.c_void_p(out.ctypes.data), herm) == de.DE_OK
                want = ((both[:nbra].conj() if herm else both[:nbra]) @ ket).cpu().numpy()
                assert np.abs(out - want).max() < 1e-15 * (size + 100)
