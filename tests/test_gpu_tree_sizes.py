"""Tree build and neighbour lists around the sizes at which the build's blocks
(256 leaves) and the walk groups change: the lists of both precisions against
every pair of particles, for equal h, and against each other for varying h."""
import numpy as np
import pytest

from flecsph_gb300.abi import (KERNEL_WENDLAND_C6, PRECISION_FP64, PRECISION_MIXED, Params,
                               new_state)

pytestmark = pytest.mark.gpu


def _lists(dim, n, varying, mode, group):
    from flecsph_gb300.sph import BodySystem
    rng = np.random.Generator(np.random.PCG64(10 * n + dim))
    s = new_state(n)
    for d in "xyz"[:dim]:
        # two clumps of different density: deep and shallow subtrees
        s[d][:] = np.where(np.arange(n) % 3 == 0, 1.0, 0.05) * rng.random(n)
    s["m"][:] = 1.0
    s["h"][:] = 0.6 * n ** (-1.0 / dim)
    if varying:
        s["h"] *= np.exp(0.3 * rng.standard_normal(n))
    s["u"][:] = s["rho"][:] = s["P"][:] = 1.0
    p = Params.defaults(dimension=dim, sph_kernel=KERNEL_WENDLAND_C6, precision_mode=mode,
                        max_neighbors=2048, group_size=group)
    with BodySystem(p, n) as bs:
        bs.read_bodies(s)
        bs.update_iteration()
        off, idx = bs.neighbors()
        pos = bs.download(["x", "y", "z", "h"])
    sets = [np.sort(idx[off[i]:off[i + 1]]) for i in range(n)]
    return sets, np.stack([pos[d] for d in "xyz"[:dim]], 1), pos["h"]


@pytest.mark.parametrize("group", [0, 5])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [2, 3, 31, 33, 255, 256, 257, 511, 513, 1300])
def test_lists(n, dim, group):
    for varying in (False, True):
        a, x, h = _lists(dim, n, varying, PRECISION_FP64, group)
        b, _, _ = _lists(dim, n, varying, PRECISION_MIXED, group)
        for i in range(n):
            assert np.array_equal(a[i], b[i]), (varying, i)
            if not varying:
                d2 = ((x[i] - x) ** 2).sum(1)
                assert np.array_equal(a[i], np.nonzero(d2 <= h[0] ** 2)[0]), i
