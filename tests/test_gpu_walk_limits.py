"""Tree build and walk on both sides of their limits: blocks of 128 leaves where
the nodes carry FP64 data, and the size from which a launch of its own finds the
walks' start nodes."""
import numpy as np
import pytest

from flecsph_gb300.abi import (KERNEL_WENDLAND_C6, PRECISION_FP64, PRECISION_MIXED, Params,
                               new_state)
from test_gpu_tree_sizes import _lists

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [127, 128, 129, 383, 384, 385])
def test_blocks_of_128(n, dim):
    for varying in (False, True):
        a, x, h = _lists(dim, n, varying, PRECISION_FP64, 0)
        b, _, _ = _lists(dim, n, varying, PRECISION_MIXED, 0)
        for i in range(n):
            assert np.array_equal(a[i], b[i]), (varying, i)
            if not varying:
                d2 = ((x[i] - x) ** 2).sum(1)
                assert np.array_equal(a[i], np.nonzero(d2 <= h[0] ** 2)[0]), i


def _walk(dim, n, varying, mode):
    from flecsph_gb300.sph import BodySystem
    rng = np.random.Generator(np.random.PCG64(n + dim))
    s = new_state(n)
    for d in "xyz"[:dim]:
        s[d][:] = rng.random(n)
    s["m"][:] = s["u"][:] = s["rho"][:] = s["P"][:] = 1.0
    s["h"][:] = 1.5 * n ** (-1.0 / dim)
    if varying:
        s["h"] *= np.exp(0.2 * rng.standard_normal(n))
    p = Params.defaults(dimension=dim, sph_kernel=KERNEL_WENDLAND_C6, precision_mode=mode,
                        max_neighbors=256)
    with BodySystem(p, n) as bs:
        bs.read_bodies(s)
        bs.update_iteration()
        off, idx = bs.neighbors()
        pos = bs.download(["x", "y", "z", "h"])
    row = np.repeat(np.arange(n), np.diff(off))
    return off, idx[np.lexsort((idx, row))], np.stack([pos[d] for d in "xyz"[:dim]], 1), pos["h"]


@pytest.mark.parametrize("varying", [False, True])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [(1 << 18) - 1, 1 << 18, (1 << 18) + 1])
def test_start_node_launch(n, dim, varying):
    off, idx, x, h = _walk(dim, n, varying, PRECISION_MIXED)
    off64, idx64, _, _ = _walk(dim, n, varying, PRECISION_FP64)
    assert np.array_equal(off, off64) and np.array_equal(idx, idx64)
    if not varying:
        for i in np.random.Generator(np.random.PCG64(1)).integers(0, n, 50):
            d2 = ((x[i] - x) ** 2).sum(1)
            assert np.array_equal(idx[off[i]:off[i + 1]], np.nonzero(d2 <= h[0] ** 2)[0]), i
