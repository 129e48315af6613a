"""FP64 passes: the energy passes from the acceleration pass's pair terms
against the same passes evaluating them, and the signal speed fused into the
acceleration against its own pass.  Both pairs do the same operations on the
same values, so they agree to the last bits; 2^-48 of the field's largest
value leaves room for the order in which a compiler contracts nothing."""
import numpy as np
import pytest

from flecsph_gb300 import setups
from flecsph_gb300.abi import (KERNEL_CUBIC_SPLINE, KERNEL_GAUSSIAN, KERNEL_WENDLAND_C2,
                               KERNEL_WENDLAND_C6, VISC_CULLEN, make_view)

pytestmark = pytest.mark.gpu
TOL = 2.0 ** -48


def _problem(dim, n, kernel, varying):
    rng = np.random.Generator(np.random.PCG64(n + dim))
    s, p, m = setups.sedov3d(12) if dim == 3 else setups.noh2d(44)
    s = {k: np.ascontiguousarray(v[:n]) for k, v in s.items()}
    s["id"] = np.arange(n, dtype=np.int64)
    for d in "xyz"[:dim]:
        s["v" + d] += 0.1 * rng.standard_normal(n)
    s["u"][:] = 1.0 + rng.random(n)
    if varying:
        s["h"] *= np.exp(0.2 * rng.standard_normal(n))
    p.sph_kernel = kernel
    p.max_neighbors = 2048  # no list may overflow: n at most
    return s, p


def _close(a, b, what):
    scale = np.abs(b).max()
    assert np.abs(a - b).max() <= TOL * scale, what


@pytest.mark.parametrize("varying", [False, True])
@pytest.mark.parametrize("dim,n,kernel", [
    (3, 1728, KERNEL_WENDLAND_C6), (3, 1001, KERNEL_CUBIC_SPLINE), (3, 65, KERNEL_WENDLAND_C2),
    (2, 1519, KERNEL_WENDLAND_C6), (2, 63, KERNEL_GAUSSIAN), (2, 2, KERNEL_WENDLAND_C6)])
def test_kept_pair_terms(dim, n, kernel, varying):
    from flecsph_gb300.sph import BodySystem
    s, p = _problem(dim, n, kernel, varying)
    with BodySystem(p, n) as bs:
        bs.read_bodies(s)
        bs.update_iteration()
        bs.eos_init()
        bs.set_total_energy()
        bs.density_pressure_soundspeed()
        bs.save_velocityhalf()
        bs.acceleration()
        bs.dedt()
        bs.dudt()
        kept = bs.download(["dedt", "dudt"])
        # writing a field makes the pair terms stale: the passes evaluate them
        now = bs.download()
        bs.upload_fields(make_view(now, fields={"rho"}))
        bs.dedt()
        bs.dudt()
        again = bs.download(["dedt", "dudt"])
    assert np.abs(again["dedt"]).max() > 0 or n == 2
    for f in ("dedt", "dudt"):
        _close(kept[f], again[f], f)


@pytest.mark.parametrize("cullen", [False, True])
@pytest.mark.parametrize("dim,n", [(3, 1727), (2, 1519), (2, 33)])
def test_fused_signal_speed(dim, n, cullen):
    from flecsph_gb300.sph import BodySystem
    s, p = _problem(dim, n, KERNEL_WENDLAND_C6, False)
    if cullen:
        p.sph_viscosity = VISC_CULLEN
    with BodySystem(p, n) as bs:
        bs.read_bodies(s)
        bs.step()
        fused = bs.download(["vsig", "id"])
    with BodySystem(p, n) as bs:
        bs.read_bodies(s)
        bs.update_iteration()
        bs.eos_init()
        bs.set_total_energy()
        bs.initialize_alpha()
        bs.density_pressure_soundspeed()
        own = bs.download(["vsig", "id"])
    assert np.array_equal(fused["id"], own["id"])
    _close(fused["vsig"], own["vsig"], "vsig")
