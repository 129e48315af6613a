"""NaN and infinities in the FP64 pair passes: viscosity::mu multiplies by
(dotp < 0) and the viscosity function is formed for every pair
(viscosity.h:81-158), so a v_half or a sound speed that is not finite reaches
the acceleration and the energy rates of its own particle and of every particle
that lists it, approaching or not.  The signal speed drops the pairs whose
approach speed is a NaN (default_physics.h:254-262)."""
import numpy as np
import pytest

from flecsph_gb300 import setups
from flecsph_gb300.abi import (EOS_NO_EOS, FsphError, KERNEL_CUBIC_SPLINE, KERNEL_WENDLAND_C6,
                               VISC_CULLEN, make_view)

pytestmark = pytest.mark.gpu


def _problem(dim, kernel, cullen):
    s, p, m = setups.sedov3d(9) if dim == 3 else setups.noh2d(24)
    n = len(s["x"])
    rng = np.random.Generator(np.random.PCG64(dim))
    # an expanding set: hardly a pair approaches
    for d in "xyz"[:dim]:
        s["v" + d][:] = 5.0 * s[d] + 1e-3 * rng.standard_normal(n)
    s["u"][:] = 1.0 + rng.random(n)
    s["P"][:] = 0.5 + rng.random(n)
    s["cs"][:] = 1.0 + rng.random(n)
    p.eos_type = EOS_NO_EOS  # the sound speed is the caller's
    p.thermokinetic_formulation = 0
    p.sph_kernel = kernel
    p.max_neighbors = 2048
    if cullen:
        p.sph_viscosity = VISC_CULLEN
    return s, p, n


@pytest.mark.parametrize("cullen", [False, True])
@pytest.mark.parametrize("dim,kernel", [(2, KERNEL_WENDLAND_C6), (3, KERNEL_WENDLAND_C6),
                                        (3, KERNEL_CUBIC_SPLINE)])
@pytest.mark.parametrize("field,value", [("cs", np.nan), ("cs", np.inf), ("vhx", np.nan),
                                         ("vhy", np.inf), ("alpha", np.nan),
                                         ("alpha", np.inf), ("rho", np.nan)])
def test_reaches_every_listing_particle(field, value, dim, kernel, cullen):
    from flecsph_gb300.sph import BodySystem
    if field == "alpha" and not cullen:
        pytest.skip("constant viscosity reads no alpha")
    s, p, n = _problem(dim, kernel, cullen)
    with BodySystem(p, n) as bs:
        bs.read_bodies(s)
        bs.update_iteration()
        bs.initialize_alpha()
        bs.density_pressure_soundspeed()
        bs.save_velocityhalf()
        off, idx = bs.neighbors()
        now = bs.download()
        assert np.isfinite(now[field]).all()
        for k in (0, n // 2, n - 1):
            now[field][k] = value
        bs.upload_fields(make_view(now, fields={field}))
        bs.acceleration()
        bs.dedt()   # from the acceleration's pair terms
        bs.dudt()
        kept = bs.download(["ax", "ay", "dedt", "dudt"])
        bs.upload_fields(make_view(now, fields={"rho"}))
        bs.dedt()   # evaluated
        bs.dudt()
        again = bs.download(["dedt", "dudt"])
    bad = set((0, n // 2, n - 1))
    want = np.array([bool(bad & set(idx[off[i]:off[i + 1]])) for i in range(n)])
    assert 3 <= want.sum() < n
    for out in (kept, again):
        for f, v in out.items():
            assert np.array_equal(~np.isfinite(v), want), f


@pytest.mark.parametrize("dim", [2, 3])
def test_fused_signal_speed(dim):
    """The signal speed of a driver iteration (in the acceleration pass) with a
    NaN velocity, against the pass of its own."""
    from flecsph_gb300.sph import BodySystem
    s, p, n = _problem(dim, KERNEL_WENDLAND_C6, False)
    s["vx"][n // 3] = np.nan
    with BodySystem(p, n) as bs:
        bs.read_bodies(s)
        bs.step()
        with pytest.raises(FsphError):  # check_nans
            bs.sync()
        fused = bs.download(["vsig", "id"])
    with BodySystem(p, n) as bs:
        bs.read_bodies(s)
        bs.update_iteration()
        bs.density_pressure_soundspeed()
        own = bs.download(["vsig", "id"])
    assert np.array_equal(fused["id"], own["id"])
    assert own["vsig"].min() == 0.0  # of the particle itself every pair drops out
    assert np.abs(fused["vsig"] - own["vsig"]).max() <= 2.0 ** -48 * own["vsig"].max()
