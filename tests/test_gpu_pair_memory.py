"""Device memory of plain-FP64 contexts: what they hold beside the fields and
lists (the pair terms of the acceleration pass) stays within 1/32 of the
device's memory for all contexts together, and is given back."""
import gc

import pytest

from flecsph_gb300.abi import PRECISION_FP64, Params

pytestmark = pytest.mark.gpu

SLOT = 16  # bytes of pair terms per list slot


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()


def _taken(p, n):
    """A context and the device memory that its creation took."""
    from flecsph_gb300.sph import BodySystem
    before = _free()[0]
    bs = BodySystem(p, n)
    return bs, before - _free()[0]


def test_bounded_over_contexts_and_given_back():
    gc.collect()  # contexts that other tests left
    total = _free()[1]
    limit = total // 32
    p = Params.defaults(dimension=3, precision_mode=PRECISION_FP64, max_neighbors=1024)
    small = 32 * 64
    n = int(0.6 * limit) // (SLOT * 1024) // 32 * 32
    terms = SLOT * 1024 * n
    lists = 4 * 1024 * n
    keep, first = _taken(p, n)
    assert first >= lists + terms         # within the bound: kept
    other, second = _taken(p, n)
    assert second < lists + terms // 2    # both would exceed it: evaluated
    third, _ = _taken(p, small)           # what still fits is kept
    keep.close()
    other.close()
    again, fourth = _taken(p, n)          # given back by the first
    assert fourth >= lists + terms
    again.close()
    third.close()
    big, fifth = _taken(p, 2 * n)         # more than the bound by itself
    assert fifth < 2 * lists + terms
    big.close()
