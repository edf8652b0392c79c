"""Library options of the reference-layout walks: the x-chunk (key 1) reaches the drop-in step."""
import numpy as np
import pytest

from oracle import skyrme_oracle as O
from tests import _golden as G
from tests._gpu import host
from tests._profile import trace, traced
from tests.test_march import _set_option, options  # noqa: F401  (fixture)
from tests.test_walks import _simulation

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["nuclear", "omega", "coulomb"])
def test_the_chunk_option_reaches_the_step(options, name):  # noqa: F811
    """One (16-row at most, 32-column) tile column of 24 planes: a chunk of 24 gives one block per
    stage, of 4 six.  The results do not depend on it (bitwise), and match the oracle."""
    dims = (24, 12, 32)
    runs = {}
    for xc in (0, 24, 4):
        _set_option(1, xc)
        th, sim, F, V = _simulation(name, dims)
        prev = O.total_energy(O.THEORIES[name], F, sim.p_i_h, sim.p_f_h)
        out = sim.step(prev)
        runs[xc] = (out, host(sim.Field), host(sim.Velocity), host(sim.EnergyGradient))
        if xc:
            grids = [int(np.prod(e["args"]["grid"])) for e in traced(lambda: trace(lambda: sim.step(prev)))
                     if "k_plain_stage" in e["name"] and "grid" in e.get("args", {})]
            assert grids == [24 // xc] * 4
    for xc in (24, 4):
        assert runs[xc][0] == runs[0][0]
        assert all(np.array_equal(a, b) for a, b in zip(runs[xc][1:], runs[0][1:]))
    Fo, Vo, Eo, erro, _ = O.arrested_newton_step(O.THEORIES[name], F, V, sim.p_i_h, sim.p_f_h, prev)
    assert abs(runs[0][0][0] - Eo) <= 1e-10 * abs(Eo)
    assert G.rel_err(runs[0][1].reshape(F.shape), Fo) <= 1e-10
