"""The key sort on keys laid out bit by bit: runs of equal prefixes whose low
bits descend in input order, as long as the run passes take them and one longer,
at the sizes where the sort's route and its split over blocks change."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_sort_sizes import _sorted

pytestmark = pytest.mark.gpu

CLUSTER_MAX = 16 * 512 * 17      # keys of the one-cluster sort
RUN_CLUSTER, RUN_LARGE = 12, 24  # longest runs that are ordered in place
H = 2.0 ** -40


def _prefix_bits(n):
    lg = int(n - 1).bit_length()
    return (lg + 12) // 8 * 8 if n <= CLUSTER_MAX else (lg + 20) // 16 * 16


def _coordinates(key, dim):
    """Centres of the cells with these data bits, in the range [0, 1]."""
    md = 63 // dim
    x = np.zeros((dim, len(key)))
    for j in range(dim):
        c = np.zeros(len(key), np.uint64)
        for i in range(md):
            c |= ((key >> np.uint64(dim * i + j)) & np.uint64(1)) << np.uint64(i)
        x[j] = (c.astype(np.float64) + 0.5) / 2.0 ** md
    return x


def _keys(n, dim, run, rng):
    """n data keys: every prefix once, but `n // 1000 + 1` runs of `run` keys
    scattered over the input, their low bits descending."""
    bits, pb = 63 // dim * dim, _prefix_bits(n)
    low = bits - pb
    nruns = n // 1000 + 1 if run > 1 else 0
    # prefixes, without that of the corners, each once
    p = np.unique(rng.integers(1, (1 << pb) - 1, 2 * n + 64))
    p = rng.permutation(p)[:n - nruns * (run - 1)]
    place = rng.permutation(n)
    prefix = np.empty(n, np.uint64)
    tail = rng.integers(0, 1 << low, n).astype(np.uint64)
    prefix[place[:len(p)]] = p
    used = len(p)
    for k in range(nruns):
        at = np.sort(np.append(place[used:used + run - 1], place[k]))
        prefix[at] = p[k]
        t = np.unique(rng.integers(0, 1 << low, 4 * run))
        tail[at] = np.sort(rng.permutation(t)[:run])[::-1]
        used += run - 1
    return (prefix << np.uint64(low)) | tail, low


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n,run", [
    (512, 1), (513, 1), (1024, 2), (1025, 12), (4096, 13),
    (65537, 2), (132651, 12), (132651, 13), (CLUSTER_MAX - 4, 12), (CLUSTER_MAX - 3, 13),
    (CLUSTER_MAX - 1, 2), (CLUSTER_MAX, 1), (CLUSTER_MAX, 12), (CLUSTER_MAX, 13),
    (CLUSTER_MAX + 1, 1), (CLUSTER_MAX + 1, 24), (CLUSTER_MAX + 1, 25),
    (600001, 2), (600001, 24), (600001, 25), (1 << 20, 24), (1 << 20, 25)])
def test_runs(n, run, dim):
    rng = np.random.Generator(np.random.PCG64(n + 31 * run + dim))
    key, low = _keys(n, dim, run, rng)
    # two particles that make the range [0, 1] exactly, in the first and last cell
    key[0], key[-1] = 0, (1 << (63 // dim * dim)) - 1
    x = _coordinates(key, dim)
    x[:, 0], x[:, -1] = H, 1.0 - H
    _, counts = np.unique(key >> np.uint64(low), return_counts=True)
    assert counts.max() in (run, max(run - 1, 1))  # an end may have been one of a run
    got, perm = _sorted(x, np.full(n, H), dim)
    marker = np.uint64(1 << (63 // dim * dim))
    want = np.argsort(key, kind="stable")
    assert np.array_equal(perm, want)
    assert np.array_equal(got, key[want] | marker)
