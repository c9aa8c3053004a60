"""Which candidate the matvec autotuner keeps."""
import pytest

from doublyexcited_b200 import tune


@pytest.mark.parametrize("storage,nn", [("c128", 13), ("c128", 15), ("c128", 19), ("c64", 17), ("c64", 19), ("c64", 23)])
def test_built_in_kernels_are_kept_within_the_margin(storage, nn):
    """The line kernels are built in on every grid: another family replaces them
    only when it is faster by more than the margin, wherever it stands in the
    list."""
    others = [c for c in tune.candidates(storage, nn) if c != tune.BUILT_IN]
    assert others and tune.BUILT_IN == ("ev", 0)
    for order in (others + [tune.BUILT_IN], [tune.BUILT_IN] + others):
        for ms, keep in ((1.01, tune.BUILT_IN), (0.99, tune.BUILT_IN), (0.97, others[0])):
            res = [(1.0 if c == tune.BUILT_IN else ms if c == others[0] else 2.0, *c) for c in order]
            assert tune.pick(res)[1:] == keep


def test_the_fastest_is_kept_without_the_built_in_kernels():
    assert tune.pick([(1.0, "stream", 0), (0.99, "dmma", 0)]) == (0.99, "dmma", 0)
