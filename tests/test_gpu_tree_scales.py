"""Neighbour lists of varying h at scales where the FP32 estimate of the mixed
walk overflows: a power of two times every length changes no FP64 comparison,
so the lists are those of the unscaled set, in both precisions."""
import numpy as np
import pytest

from flecsph_gb300.abi import (KERNEL_WENDLAND_C6, PRECISION_FP64, PRECISION_MIXED, Params,
                               new_state)

pytestmark = pytest.mark.gpu


def _lists(dim, n, scale, mode):
    from flecsph_gb300.sph import BodySystem
    rng = np.random.Generator(np.random.PCG64(n + dim))
    s = new_state(n)
    for d in "xyz"[:dim]:
        s[d][:] = scale * rng.random(n)
    s["m"][:] = 1.0
    s["h"][:] = scale * 0.6 * n ** (-1.0 / dim) * np.exp(0.3 * rng.standard_normal(n))
    s["u"][:] = s["rho"][:] = s["P"][:] = 1.0
    p = Params.defaults(dimension=dim, sph_kernel=KERNEL_WENDLAND_C6, precision_mode=mode,
                        max_neighbors=1024)
    with BodySystem(p, n) as bs:
        bs.read_bodies(s)
        bs.update_iteration()
        off, idx = bs.neighbors()
    return [np.sort(idx[off[i]:off[i + 1]]) for i in range(n)]


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [33, 700])
def test_scaled(n, dim):
    want = _lists(dim, n, 1.0, PRECISION_FP64)
    assert max(len(v) for v in want) > 1
    for exponent in (-20, 56, 62, 64, 66, 70):  # h^2 overflows FP32 from 2^64 on
        for mode in (PRECISION_FP64, PRECISION_MIXED):
            got = _lists(dim, n, 2.0 ** exponent, mode)
            assert all(np.array_equal(a, b) for a, b in zip(want, got)), (exponent, mode)
