"""The default matvec kernels (whole lines in registers) at the sizes where
their tiles go wrong: the smallest and largest grids, runs and planes that
end ragged, odd block widths, more vectors than a grid dimension holds, and
an output block that holds NaN beforehand (the first kernel must not read
it)."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

# FP64: a product sums 3 NN terms per electron; 1e-13 is several hundred
# roundings of 1.1e-16.  FP32: the same count of 6e-8 within 1e-6.
TOL64, TOL32 = 1e-13, 1e-6


def _products(de, torch, n, nvec, seed):
    """H X in both storages into NaN-filled blocks: (x, y64, y32)."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    with de.Problem(n=n, delta=1.7, theta=0.3) as g64, \
            de.Problem(n=n, delta=1.7, theta=0.3, precision="mixed") as g32:
        st = torch.cuda.current_stream()
        g64.set_stream(st.cuda_stream)
        g32.set_stream(st.cuda_stream)
        x = torch.randn(nvec, g64.dim, dtype=torch.complex128, device="cuda", generator=gen)
        y = torch.full_like(x, complex(np.nan, np.nan))
        g64.matblock_d(x.data_ptr(), y.data_ptr(), nvec)
        x32 = x.to(torch.complex64)
        y32 = torch.full_like(x32, complex(np.nan, np.nan))
        g32.matblock32_d(x32.data_ptr(), y32.data_ptr(), nvec)
        torch.cuda.synchronize()
    return x, y, y32


@pytest.mark.parametrize("n,nvec", [(1, 1), (1, 7), (2, 3), (3, 5), (4, 2), (5, 1)])
def test_line_kernels_match_oracle(de, oracle, n, nvec):
    import torch

    h = oracle.init_hamiltonian(oracle.Params(n=n, delta=1.7, theta=0.3), nelec=2)
    x, y, y32 = _products(de, torch, n, nvec, 300 + n)
    for j in range(nvec):
        xj = x[j].cpu().numpy()
        assert rel_err(y[j].cpu().numpy(), h.matvec(xj)) < TOL64
        ref32 = h.matvec(xj.astype(np.complex64).astype(np.complex128))
        assert rel_err(y32[j].cpu().numpy().astype(np.complex128), ref32) < TOL32


@pytest.mark.parametrize("n", [6, 7, 8, 9, 10, 11])
def test_line_kernels_match_cube_kernels(de, n):
    """The larger grids against the streaming / cube kernels."""
    import torch

    x, y, y32 = _products(de, torch, n, 1, 400 + n)
    with de.Problem(n=n, delta=1.7, theta=0.3) as g:
        g.set_stream(torch.cuda.current_stream().cuda_stream)
        g.set_matvec_kernel("stream")
        ref = torch.empty_like(x)
        g.matblock_d(x.data_ptr(), ref.data_ptr(), 1)
        torch.cuda.synchronize()
    norm = torch.linalg.vector_norm(ref)
    assert (torch.linalg.vector_norm(y - ref) / norm).item() < TOL64
    assert (torch.linalg.vector_norm(y32 - ref) / norm).item() < TOL32


def test_line_kernels_loop_over_many_vectors(de):
    """65,538 vectors at N=1: the vector index wraps the grid's y extent."""
    import torch

    nvec = 65538
    x, y, y32 = _products(de, torch, 1, nvec, 5)
    with de.Problem(n=1, delta=1.7, theta=0.3) as g:
        g.set_stream(torch.cuda.current_stream().cuda_stream)
        for j in (0, 1, 2, 65534, 65535, 65536, 65537):
            one = torch.empty_like(x[j])
            g.matblock_d(x[j].data_ptr(), one.data_ptr(), 1)
            torch.cuda.synchronize()
            assert torch.equal(one, y[j])
            assert (torch.linalg.vector_norm(y32[j] - one) / torch.linalg.vector_norm(one)).item() < TOL32
