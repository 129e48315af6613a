"""The key sort remembers that its keys were crowded (long runs of one prefix)
and then starts with the passes over all bits: crowded and spread sets in every
order of succession, through the same scratch, must come out sorted, ties in
input order, every particle once."""
import numpy as np
import pytest

from test_gpu_sort_sizes import _sorted

pytestmark = pytest.mark.gpu


def _set(kind, n, dim, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    x = rng.random((dim, n))
    if kind == "c":  # all but one particle in a corner of the range
        x[:, 1:] = 0.5 + 1e-6 * (x[:, 1:] - 0.5)
        x[:, 0] = 40.0
    return x


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [700, 2250, 30000, 139264, 139265, 300001])
def test_successions(n, dim):
    # every pair of kinds follows the other; the last set of one size is the
    # first one's predecessor in the next
    for step, kind in enumerate("cc" "uu" "cu" "cuu"):
        x = _set(kind, n, dim, 100 * step + dim)
        keys, perm = _sorted(x, np.full(n, 1e-3), dim)
        assert np.array_equal(np.sort(perm), np.arange(n)), (step, kind)
        before = np.empty(n, np.uint64)
        before[perm] = keys
        assert np.array_equal(np.argsort(before, kind="stable"), perm), (step, kind)
        assert np.array_equal(np.sort(before), keys), (step, kind)


@pytest.mark.parametrize("side", [13, 52])
def test_context_lattice(side):
    """The same in a context's builds (below and above one cluster's keys): a
    lattice alone and beside one particle 39 times its size away, whose full
    keys differ; the particles come out in key order."""
    from flecsph_gb300.abi import KERNEL_WENDLAND_C6, PRECISION_MIXED, Params, new_state
    from flecsph_gb300.sph import BodySystem
    n = side ** 3
    g = (np.arange(side) + 0.5) / side
    lattice = np.stack(np.meshgrid(g, g, g, indexing="ij"), 0).reshape(3, -1)
    p = Params.defaults(dimension=3, sph_kernel=KERNEL_WENDLAND_C6,
                        precision_mode=PRECISION_MIXED, max_neighbors=64)
    with BodySystem(p, n) as bs:
        for step, far in enumerate((1, 1, 0, 0, 1)):
            s = new_state(n)
            x = lattice[:, np.random.Generator(np.random.PCG64(step)).permutation(n)]
            if far:
                x[:, 0] = 40.0
            for d, v in zip("xyz", x):
                s[d][:] = v
            s["m"][:] = 1.0
            s["h"][:] = 0.5 / side
            s["id"][:] = np.arange(n)
            bs.read_bodies(s)
            for _ in range(3):
                bs.update_iteration()
            out = bs.download(["x", "id", "key"])
            key = out["key"].astype(np.uint64)
            assert (key[1:] > key[:-1]).all(), (step, far)
            assert np.array_equal(np.sort(out["id"]), np.arange(n))
            assert np.array_equal(out["x"], x[0][out["id"]])
