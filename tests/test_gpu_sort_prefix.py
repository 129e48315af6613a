"""The key sort beyond one cluster's keys, whose passes cover a prefix of them:
no, short and long runs of equal prefixes (the last start over on all bits),
ascending keys, ties in input order, every particle once."""
import numpy as np
import pytest

from test_gpu_sort_sizes import _sorted

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("spread", ["uniform", "pairs", "runs24", "runs25", "clump"])
@pytest.mark.parametrize("n", [(1 << 19) - 1, 1 << 19, (1 << 19) + 1, 700001, 1 << 20])
def test_sort(n, spread, dim):
    rng = np.random.Generator(np.random.PCG64(n + dim))
    x = rng.random((dim, n))
    if spread == "clump":
        x[:, 1:] = 0.5 + 1e-6 * (x[:, 1:] - 0.5)
        x[:, 0] = 40.0
    elif spread != "uniform":
        # the first `run` particles of each 1000 in one cell of the prefix:
        # their places differ in the last bits, and some not at all
        run = {"pairs": 2, "runs24": 24, "runs25": 25}[spread]
        for k in range(1, run):
            src = x[:, 0::1000][:, :n // 1000]
            x[:, k::1000][:, :n // 1000] = src + 1e-15 * rng.integers(0, 3, src.shape[1])
    keys, perm = _sorted(x, np.full(n, 1e-3), dim)
    assert np.array_equal(np.sort(perm), np.arange(n))
    before = np.empty(n, np.uint64)
    before[perm] = keys
    assert np.array_equal(np.argsort(before, kind="stable"), perm)
    assert np.array_equal(np.sort(before), keys)
