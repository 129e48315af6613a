"""A member's own pass before a step of the ensemble's graphs leaves records
(P / rho^2, pair terms, the pressure-only acceleration) of the state before the
step; the passes called after the step must not take them for the new state's."""
import numpy as np
import pytest

from flecsph_gb300 import setups
from flecsph_gb300.abi import PRECISION_FP64, PRECISION_MIXED

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("thermo", [0, 1])
@pytest.mark.parametrize("mode", [PRECISION_FP64, PRECISION_MIXED])
def test_own_pass_before_a_graph_step(mode, thermo):
    from flecsph_gb300.sph import BodySystem, Ensemble
    s, p, m = setups.noh2d(40)
    p.precision_mode = mode
    p.thermokinetic_formulation = thermo
    n = len(s["x"])
    fields = ["dedt", "dudt", "P", "cs"]

    def passes(bs, step):
        bs.acceleration()
        step()
        bs.dedt()
        bs.dudt()
        return bs.download(fields)

    ens = Ensemble()
    mb = ens.add(p, n)
    mb.read_bodies(s)
    ens.step(5)
    got = passes(mb, lambda: ens.step(1))
    ens.close()
    with BodySystem(p, n) as bs:
        bs.read_bodies(s)
        for _ in range(5):
            bs.step()
        want = passes(bs, bs.step)
    for f in fields:
        assert np.array_equal(got[f], want[f]), f
