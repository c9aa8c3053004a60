"""The roofline figures of bench.py: the flops that a product executes, and
which solves count as exchange-symmetric."""
import math

import numpy as np
import pytest

import bench


@pytest.mark.parametrize("nn", [3, 5, 13])
def test_flops_are_those_of_the_even_odd_lines(nn):
    """Counted line by line: N+1 outputs from the N+1 sums u (the even half),
    N outputs from the N differences w, a real coefficient times a complex value
    each, two multiply-adds of two flops."""
    n = nn // 2
    line = sum(4 for a in range(n + 1) for b in range(n + 1)) + sum(4 for a in range(n) for b in range(n))
    lines = nn ** 5
    assert bench.alg_flops(nn) == 6 * lines * line + 8 * nn ** 6
    assert bench.alg_flops(nn, exch=True) == 3 * lines * line + 8 * nn ** 6
    assert bench.alg_flops(nn, exch=True) < bench.alg_flops(nn) < bench.dense_flops(nn)


def test_product_roofline_reports_bytes_and_executed_flops():
    r = bench.product_roofline(13, True, True, 45e-6, 64.0, "x")
    assert r["bound"] == "hbm" and r["unit"] == "GB/s"
    assert math.isclose(r["achieved"], r["traffic"] / 45e-6 / 1e9) and math.isclose(r["frac"], r["achieved"] / r["peak"])
    assert math.isclose(r["flops"]["achieved"], bench.alg_flops(13, True) / 45e-6 / 1e12)
    r = bench.product_roofline(7, False, False, 1e-5, 35.0, "x")  # no capture
    assert r["traffic"] is None and math.isclose(r["achieved"], 32 * 7 ** 6 / 1e-5 / 1e9)


class FakeProblem:
    m = 4

    def __init__(self, **families):
        self.families = families

    def get_matvec_launch(self, storage, pass_):
        return self.families.get(storage, "fma"), 0


def test_exchange_symmetric_follows_the_start_and_the_kernels():
    rng = np.random.default_rng(1)
    z = rng.standard_normal((2, 4, 4)) + 1j * rng.standard_normal((2, 4, 4))
    sym, anti = z + z.transpose(0, 2, 1), z - z.transpose(0, 2, 1)
    cols = lambda a: a.reshape(len(a), -1).T  # noqa: E731
    p = FakeProblem()
    assert bench.exchange_symmetric(p, cols(sym), "mixed") and bench.exchange_symmetric(p, cols(anti[:1]), "mixed")
    assert bench.exchange_symmetric(p, cols(sym), "fp64") and not bench.exchange_symmetric(p, cols(sym[:1]), "fp64")
    assert not bench.exchange_symmetric(p, cols(z), "mixed")
    assert not bench.exchange_symmetric(p, cols(np.stack([sym[0], anti[1]])), "mixed")
    assert not bench.exchange_symmetric(FakeProblem(c64="stream"), cols(sym), "mixed")
    assert bench.exchange_symmetric(FakeProblem(c64="stream"), cols(sym), "fp64")
