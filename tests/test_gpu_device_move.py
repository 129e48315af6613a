"""Device-side upload and download in one launch: against the host copies, at
the sizes and alignments where the copy kernel's blocks and vectors end."""
import ctypes as C

import numpy as np
import pytest

from flecsph_gb300.abi import (DOUBLE_FIELDS, PRECISION_MIXED, Params, make_view_tensors,
                               new_state)

pytestmark = pytest.mark.gpu


def _params(dim):
    return Params.defaults(dimension=dim, precision_mode=PRECISION_MIXED)


def _state(n, dim, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    s = new_state(n)
    for f in DOUBLE_FIELDS:
        if dim == 2 and f in ("z", "vz", "vhz", "az", "gaz"):
            continue
        s[f][:] = rng.random(n) + 0.5
    s["id"][:] = rng.permutation(n)
    return s


def _shifted(a, shift):
    """A device copy of `a` that starts `shift` words into its allocation."""
    import torch
    buf = torch.full((len(a) + 3,), -7, dtype=torch.from_numpy(a).dtype, device="cuda")
    buf[shift:shift + len(a)] = torch.from_numpy(a).to("cuda")
    return buf, buf[shift:shift + len(a)]


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("n", [2, 3, 511, 2047, 2048, 2049, 6145])
def test_round_trip(n, shift, dim):
    import torch
    from flecsph_gb300.sph import BodySystem
    s = _state(n, dim, n)
    left_out = ("rho", "divv")  # cleared by an upload
    with BodySystem(_params(dim), n + 5) as bs:
        held = {f: _shifted(s[f], shift) for f in DOUBLE_FIELDS + ["id"] if f not in left_out}
        bs.read_bodies_device({f: v for f, (_, v) in held.items()})
        host = bs.download()
        outs = {f: _shifted(np.full(n, -3.0), shift) for f in DOUBLE_FIELDS}
        outs["id"] = _shifted(np.full(n, -3), shift)
        torch.cuda.synchronize()
        view = make_view_tensors({f: v for f, (_, v) in outs.items()}, n)
        bs._check(bs.lib.fsph_download_device(bs.ctx, C.byref(view)), "download_device")
        for f, (buf, v) in outs.items():
            flat = dim == 2 and f in ("z", "vz", "vhz", "az", "gaz")
            want = np.zeros(n) if f in left_out else s[f]
            if flat:  # not written in two dimensions
                want = np.full(n, -3.0)
            else:
                assert np.array_equal(host[f], want), f
            got = buf.cpu().numpy()
            assert np.array_equal(got[shift:shift + n], want), f
            # nothing beside the array
            assert (got[:shift] == -7).all() and (got[shift + n:] == -7).all(), f


def test_error_leaves_outputs():
    """A pending device-side error is raised before anything is written."""
    import torch
    from flecsph_gb300.abi import FsphError
    from flecsph_gb300.sph import BodySystem
    s = _state(64, 3, 6)
    s["u"][11] = np.nan
    with BodySystem(_params(3), 64) as bs:
        bs.read_bodies(s)
        bs.check_nans()
        out = torch.full((64,), -3.0, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        view = make_view_tensors({"m": out}, 64)
        with pytest.raises(FsphError):
            bs._check(bs.lib.fsph_download_device(bs.ctx, C.byref(view)), "download_device")
        assert (out == -3.0).all()
        # read once: the next download succeeds
        assert np.array_equal(bs.download_device(["m"], device="cuda")["m"].cpu(), s["m"])
