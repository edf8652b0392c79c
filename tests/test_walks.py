"""The drop-in step's fused stages (gradient, slope, next stage field and update in one walk)
against the separate kernels and the oracle, on lattices at the edges of the 12- and 16-row,
32-column tiles: exactly one tile, one site more and one less in each direction, odd Z (8-byte
copies) and even Z (16-byte copies), and a lattice with less than one tile's rows.

Tolerances: the fused and separate kernels round identically (every RK4 operation is spelled
out), so they are compared bitwise; against the oracle 1e-10 relative, the step bound of the
parity tests.
"""
import numpy as np
import pytest

from oracle import skyrme_oracle as O
from tests import _golden as G
from tests._gpu import dev, host
from tests.test_march import inputs, params_for

pytestmark = pytest.mark.gpu

DIMS = [(6, 16, 32), (5, 17, 33), (9, 11, 31), (7, 13, 62), (8, 33, 34)]


def _simulation(name, dims):
    from skyrmion_solver_b200.core.simulation import Simulation
    th, p_i, p_f = params_for(name, dims)
    X, Y, Z = dims
    F, V = inputs(int(p_i[5]), dims, seed=3)
    prm = th.params.default_params(xlen=X, ylen=Y, zlen=Z, lsx=float(p_f[3]), lsy=float(p_f[4]), lsz=float(p_f[5]),
                                   time_step=float(p_f[7]))
    sim = Simulation(prm, th)
    sim.Field.copy_(dev(F))
    sim.Velocity.copy_(dev(V))
    return th, sim, F, V


class _Opaque:
    """A launchable the integrator does not recognise: it then runs the separate kernels."""

    def __init__(self, k):
        self.k = k

    def __getitem__(self, cfg):
        return self.k[cfg]

    def __call__(self, *a, **kw):
        return self.k(*a, **kw)


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("name", ["nuclear", "omega", "coulomb", "berger", "lightly_bound"])
def test_fused_stages_equal_separate_kernels(name, dims):
    from skyrmion_solver_b200.core.integrator import do_arrested_newton_flow
    th, a, F, V = _simulation(name, dims)
    _, b, _, _ = _simulation(name, dims)
    thd = O.THEORIES[name]
    prev = O.total_energy(thd, F, a.p_i_h, a.p_f_h)
    Fo, Vo, Eo, erro, _ = O.arrested_newton_step(thd, F, V, a.p_i_h, a.p_f_h, prev)
    ea, erra = a.step(prev)
    eb, errb = do_arrested_newton_flow(
        b.Velocity, b.Field, None, None, b.EnergyGradient, b.k1, b.k2, b.k3, b.k4, b.l1, b.l2, b.l3, b.l4, b.Temp,
        b.en, b.entmp, b.gridsum_partial, b.max_partial, b.p_i_d, b.p_f_d, b.p_i_h, b.p_f_h, prev,
        _Opaque(th.observables.compute_energy), _Opaque(th.kernels.do_gradient_step_kernel),
        _Opaque(th.kernels.do_rk4_kernel))
    assert ea == eb and erra == errb
    for buf in ("Field", "Velocity", "EnergyGradient", "k1", "k2", "k3", "k4", "l1", "l2", "l3", "l4", "Temp"):
        assert bool((getattr(a, buf) == getattr(b, buf)).all()), buf
    assert abs(ea - Eo) <= 1e-10 * abs(Eo) and abs(erra - erro) <= 1e-10 * max(1.0, abs(erro))
    assert G.rel_err(host(a.Field, F.shape), Fo) <= 1e-10
