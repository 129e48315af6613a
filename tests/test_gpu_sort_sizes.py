"""The key sort at the sizes where its split over blocks and launches changes,
and on sets whose keys share long prefixes (a tight clump in a wide range),
where the short-prefix passes start over: keys ascending, ties in input
order, every particle once."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [2, 3, 31, 33, 1024, 1025, 2047, 2050, 4097, 8193, 16384, 16385, 30000, 147455,
         147456, 147457, 200001]


def _sorted(x, h, dim):
    import torch
    from flecsph_gb300.sph import library
    lib = library()
    n = len(h)
    d = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (*x, h)]
    keys = torch.zeros(n, dtype=torch.int64, device="cuda")
    perm = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    p = [C.c_void_p(t.data_ptr()) for t in d]
    st = lib.fsph_sort_keys_noalloc(p[0], p[1], p[2] if dim == 3 else None, p[-1],
                                    C.c_int64(n), C.c_int32(dim),
                                    C.c_void_p(keys.data_ptr()),
                                    C.c_void_p(perm.data_ptr()), None)
    assert st == 0
    torch.cuda.synchronize()
    return keys.cpu().numpy().view(np.uint64), perm.cpu().numpy()


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("spread", ["uniform", "clump", "pairs"])
@pytest.mark.parametrize("n", SIZES)
def test_sort(n, spread, dim):
    rng = np.random.Generator(np.random.PCG64(n * 7 + dim))
    x = rng.random((dim, n))
    if spread == "clump" and n > 8:
        # all but one particle within 1e-6 of the range: one long run of
        # equal prefixes, duplicate keys among them
        x[:, 1:] = 0.5 + 1e-6 * (x[:, 1:] - 0.5)
        x[:, 0] = 40.0
    elif spread == "pairs":
        # short runs of equal prefixes, some with equal full keys
        half = n // 2
        x[:, half:2 * half] = x[:, :half] * (1.0 + 1e-9 * rng.integers(0, 3, half))
    keys, perm = _sorted(x, np.full(n, 1e-3), dim)
    assert np.array_equal(np.sort(perm), np.arange(n))
    before = np.empty(n, np.uint64)
    before[perm] = keys
    assert np.array_equal(np.argsort(before, kind="stable"), perm)
    assert np.array_equal(np.sort(before), keys)
