"""The drop-in step's fused stages (gradient, slope, next stage field and update in one walk)
against the separate kernels and the oracle, on lattices at the edges of the 12- and 16-row,
32-column tiles: exactly one tile, one site more and one less in each direction, odd Z (8-byte
copies) and even Z (16-byte copies), and a lattice with less than one tile's rows.

Then the resident engine's walks on the same lattices, and rho's two FP32 kernel sets (all
components in one walk up to 56^3 sites, separate walks over the rho and the pion components
beyond).

Tolerances: the fused and separate kernels round identically (every RK4 operation is spelled
out), so they are compared bitwise; against the oracle 1e-10 relative, the step bound of the
parity tests, in FP64, and 2e-5 in FP32, the bound of the engine's FP32 marching tests.
"""
import numpy as np
import pytest

from oracle import skyrme_oracle as O
from tests import _golden as G
from tests._gpu import dev, host
from tests.test_march import _plain_gradient, inputs, params_for

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


def _engine_steps(name, dims, precision, steps=2):
    from skyrmion_solver_b200.engine import Engine
    th, p_i, p_f = params_for(name, dims)
    F, V = inputs(int(p_i[5]), dims, seed=5)
    thd = O.THEORIES[name]
    tol = 1e-10 if precision == "fp64" else 2e-5
    Fr, Vr, E = F, V, O.total_energy(thd, F, p_i, p_f)
    with Engine(0) as eng:
        iid = eng.add(name, (p_i, p_f), F, V, precision=precision)
        assert abs(eng.stats(iid).energy - E) <= tol * abs(E)
        for _ in range(steps):
            Fr, Vr, E, err, _ = O.arrested_newton_step(thd, Fr, Vr, p_i, p_f, E)
            eng.step(1)
            assert abs(eng.stats(iid).energy - E) <= tol * abs(E)
        f, v = eng.read(iid)
    assert G.rel_err(f, Fr) <= tol
    if np.any(Vr) and precision == "fp64":
        assert G.rel_err(v, Vr) <= tol


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("precision", ["fp64", "fp32", "fp32d"])
@pytest.mark.parametrize("name", ["nuclear", "omega", "coulomb", "rho"])
def test_engine_walks_at_tile_edges(name, precision, dims):
    _engine_steps(name, dims, precision)


@pytest.mark.parametrize("dims", [(56, 56, 56), (57, 57, 57), (49, 61, 60)])
@pytest.mark.parametrize("precision", ["fp32", "fp32d"])
def test_rho_fp32_kernel_sets(precision, dims):
    """The largest lattice of the one and the smallest of the other kernel set; odd Z (cp.async)
    and Z a multiple of four (TMA)."""
    _engine_steps("rho", dims, precision, steps=1)


@pytest.mark.parametrize("dims", DIMS)
def test_rho_gradient_at_tile_edges(dims):
    """The drop-in gradient (a walk over the rho components, then one over the pions') against the
    oracle, 1e-10 relative."""
    _, p_i, p_f = params_for("rho", dims)
    F, _ = inputs(13, dims, seed=4)
    want_eg, want_l = O.gradient(O.THEORIES["rho"], F, p_i, p_f)
    eg, l = _plain_gradient("rho", F, p_i, p_f)
    assert G.rel_err(eg, want_eg) <= 1e-10
    assert G.rel_err(l, want_l) <= 1e-10
