"""complex64 products of vectors whose values lie near and below the smallest
normal FP32 number: nothing may be flushed to zero on the way to the sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# Below the normal range each rounding is absolute, at most 2^-150 (half the
# smallest subnormal).  An output sums 3 NN products per electron, in halves
# (u, w), of complex values, then V x: at most 12 NN + 24 roundings, each
# scaled by |T|, |1/SCALE^2| and |V| below 4.
TINY = 2.0 ** -150


def _products(de, torch, n, x):
    with de.Problem(n=n, delta=2.0, theta=0.3, precision="mixed") as h:
        h.set_stream(torch.cuda.current_stream().cuda_stream)
        y = torch.empty_like(x)
        h.matblock32_d(x.data_ptr(), y.data_ptr(), x.shape[0])
        x64 = x.to(torch.complex128)
        want = torch.empty_like(x64)
        h.matblock_d(x64.data_ptr(), want.data_ptr(), x.shape[0])
        torch.cuda.synchronize()
    return y.to(torch.complex128), want


@pytest.mark.parametrize("scale", [1e-30, 1e-36, 1e-38, 1e-40])
@pytest.mark.parametrize("n,nvec", [(1, 3), (2, 1), (3, 1), (4, 2), (5, 1), (6, 1), (8, 1), (9, 1)])
def test_tiny_vectors(de, n, nvec, scale):
    import torch

    nn = 2 * n + 1
    gen = torch.Generator(device="cuda").manual_seed(n)
    x = (torch.randn(nvec, nn ** 6, dtype=torch.complex128, device="cuda", generator=gen) * scale).to(torch.complex64)
    y, want = _products(de, torch, n, x)
    # FP32 rounding relative to the norm (1e-6, as the other products), and the absolute one
    bound = 1e-6 * torch.linalg.vector_norm(want).item() + np.sqrt(nvec * nn ** 6) * 4 * (12 * nn + 24) * TINY
    assert torch.linalg.vector_norm(y - want).item() < bound


@pytest.mark.parametrize("n", [1, 3, 6])
def test_sparse_vector_keeps_tiny_values(de, n):
    """One entry of 1 and one of 1e-38: the lines through the first add zeros or
    ordinary values, those through the second subnormals, each into values that
    the earlier kernels left."""
    import torch

    nn = 2 * n + 1
    x = torch.zeros(1, nn ** 6, dtype=torch.complex64, device="cuda")
    x[0, 0] = 1.0
    x[0, -1] = 1e-38 * (1 + 2j)
    y, want = _products(de, torch, n, x)
    # no line holds both entries; an output is rounded like the largest product
    # of its line (the halves of a line cancel), relatively or absolutely
    big = want.abs() > 1e-20
    err = (y - want).abs()
    assert err[big].max() < 4e-6
    assert err[~big].max() < 1e-6 * 1e-37 + 4 * (12 * nn + 24) * TINY
