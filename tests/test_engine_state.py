"""Everything a resident instance reports after some steps -- field, velocity, energy, signed and
absolute gradient maxima, kinetic energy -- against the oracle, for every row length modulo four
(the engine pads its rows to whole 16-byte chunks; nothing of the padding may reach a result).

The flow is not arrested (killkinen = 0), so that the velocity is compared in every case.
Tolerances: FP64 1e-10 relative (to the maximum), the step bound of the parity tests; FP32 2e-5,
the bound of the engine's FP32 marching tests, for the velocity as well: it is dt times a sum of
gradients whose relative error to the largest one is that of the field's stencils.
"""
import numpy as np
import pytest

from oracle import skyrme_oracle as O
from tests import _golden as G
from tests.test_march import inputs, params_for

pytestmark = pytest.mark.gpu


def run_against_oracle(name, dims, precision, steps=2, period=None, seed=5):
    from skyrmion_solver_b200.engine import Engine
    th, p_i, p_f = params_for(name, dims)
    p_i = p_i.copy()
    p_i[8] = 0
    F, V = inputs(int(p_i[5]), dims, seed=seed)
    thd = O.THEORIES[name]
    tol = 1e-10 if precision == "fp64" else 2e-5
    vol = float(p_f[6])
    E = O.total_energy(thd, F, p_i, p_f)
    with Engine(0) as eng:
        i = eng.add(name, (p_i, p_f), F, V, precision=precision)
        if period is not None:
            eng.set_defect_period(i, period)
        for _ in range(steps):
            Fo, Vo, Eo, err, eg = O.arrested_newton_step(thd, F, V, p_i, p_f, E)
            F, V, E = Fo, Vo, Eo
            eng.step(1)
            st = eng.stats(i)
            big = float(np.max(np.abs(eg)))
            assert abs(st.energy - E) <= tol * abs(E)
            assert abs(st.err - err) <= tol * big and abs(st.gabs - big) <= tol * big
            kin = 0.5 * vol * float(np.sum(V * V))
            assert abs(st.kinetic - kin) <= tol * kin
        f, v = eng.read(i)
    assert G.rel_err(f, F) <= tol and G.rel_err(v, V) <= tol


@pytest.mark.parametrize("z", [32, 33, 34, 35])
@pytest.mark.parametrize("precision", ["fp64", "fp32", "fp32c", "fp32d"])
@pytest.mark.parametrize("name", ["nuclear", "omega", "rho"])
def test_state_for_every_row_length(name, precision, z):
    run_against_oracle(name, (7, 13, z), precision)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("z", [33, 34, 36])
def test_rows_are_padded_to_sixteen_byte_chunks(precision, z):
    """The arrays of an instance hold rows of a multiple of four values, so that rows of every
    length are copied in whole chunks; the choice of staging stays that of aligned rows."""
    from skyrmion_solver_b200._lib import SkyInvalidArgument
    from skyrmion_solver_b200.engine import Engine
    size = 8 if precision == "fp64" else 4
    with Engine(0) as eng:
        _, p_i, p_f = params_for("omega", (40, 24, 36))
        eng.add("omega", (p_i, p_f), inputs(5, (40, 24, 36))[0], None, precision=precision)
        whole = eng.bytes
        _, p_i, p_f = params_for("omega", (40, 24, z))
        F, _ = inputs(5, (40, 24, z))
        i = eng.add("omega", (p_i, p_f), F, None, precision=precision)
        assert eng.bytes == 2 * whole
        aligned = z * size % 16 == 0
        assert eng.staging(i)[0] == aligned
        if not aligned:
            eng.set_staging(i, False)
            with pytest.raises(SkyInvalidArgument):
                eng.set_staging(i, True)
        f, v = eng.read(i)
        assert np.max(np.abs(f - F)) <= (0.0 if precision == "fp64" else 2.0 ** -24 * np.max(np.abs(F)))
        assert not np.any(v)


@pytest.mark.parametrize("dims", [(56, 56, 56), (57, 57, 57), (49, 61, 60), (13, 25, 37)])
@pytest.mark.parametrize("precision", ["fp32", "fp32d"])
def test_rho_state_with_a_refresh_in_every_step(precision, dims):
    """The largest lattice of the fused FP32 rho kernels and the smallest of the separate walks (odd
    rows and whole chunks) over three steps; defect-corrected, the correction is refreshed in each of
    them, so that the refresh kernels, the stage 1 that follows them and stages with a correction
    that is not zero all run."""
    run_against_oracle("rho", dims, precision, steps=3, period=1 if precision == "fp32d" else None)


@pytest.mark.parametrize("dims", [(6, 16, 32), (5, 17, 33), (9, 11, 31), (7, 13, 62), (8, 33, 34)])
@pytest.mark.parametrize("name", ["nuclear", "omega", "coulomb", "berger", "lightly_bound"])
def test_state_with_refreshes_at_tile_edges(name, dims):
    """Defect-corrected FP32 with a refresh in every second step, at the edges of the 12- and 16-row,
    32-column tiles."""
    run_against_oracle(name, dims, "fp32d", steps=3, period=2)


@pytest.mark.parametrize("precision", ["fp32", "fp32c"])
@pytest.mark.parametrize("name,dims", [("nuclear", (9, 17, 36)), ("omega", (9, 13, 33)), ("coulomb", (9, 13, 34)),
                                       ("rho", (9, 13, 36)), ("rho", (57, 57, 57))])
def test_velocity_is_rounded_once(name, precision, dims):
    """V' = V + (l1 + 2 l2 + 2 l3 + l4)/6 with an FP32 velocity near one and increments far below it:
    the increment is summed first, so V' is the exact sum rounded once, at most half a unit in the
    last place of values in [0.5, 1] (2^-25) away.  To that comes the increment's own FP32 error, at
    most the 2e-5 of its maximum that the engine's FP32 gradients are held to, and the units in which
    an increment is summed (four roundings of 2^-24 of it).  No projection (unit_length = 0)."""
    from skyrmion_solver_b200.engine import Engine
    _, p_i, p_f = params_for(name, dims)
    p_i, p_f = p_i.copy(), p_f.copy()
    p_i[8] = p_i[10] = 0
    p_f[7] = 1e-8
    F, V = inputs(int(p_i[5]), dims, seed=6)
    V = np.random.default_rng(8).uniform(0.5, 1.0 - 1e-3, size=F.shape).astype(np.float32).astype(np.float64)
    _, Vo, _, _, _ = O.arrested_newton_step(O.THEORIES[name], F, V, p_i, p_f, 0.0)
    inc = float(np.max(np.abs(Vo - V)))
    assert 2.0 ** -24 < inc < 1e-3
    with Engine(0) as eng:
        i = eng.add(name, (p_i, p_f), F, V, precision=precision)
        eng.step(1)
        _, v = eng.read(i)
    assert float(np.max(np.abs(v - Vo))) <= 2.0 ** -25 + (2e-5 + 2.0 ** -22) * inc


@pytest.mark.parametrize("name,precision", [("nuclear", "fp32d"), ("omega", "fp32"), ("coulomb", "fp64"), ("rho", "fp32d"),
                                            ("rho", "fp64")])
@pytest.mark.parametrize("z", [33, 38])
def test_padded_rows_in_both_stagings(name, precision, z):
    """Rows that are no whole chunks in the caller's arrays: TMA boxes and cp.async chunks of the padded
    ones give bitwise the same records and state (a box ends at the last site, a chunk is cut there)."""
    from skyrmion_solver_b200 import _lib
    from skyrmion_solver_b200.engine import Engine
    dims = (11, 19, z)
    _, p_i, p_f = params_for(name, dims)
    F, V = inputs(int(p_i[5]), dims, seed=12)
    old = int(_lib.load().sky_get_option(2))
    out = []
    try:
        for tma in (1, 0):
            _lib.call("sky_set_option", 2, tma)
            with Engine(0) as eng:
                i = eng.add(name, (p_i, p_f), F, V, precision=precision)
                if precision == "fp32d":
                    eng.set_defect_period(i, 3)
                eng.step(7)
                s = eng.stats(i)
                out.append(((s.energy, s.baryon, s.err, s.gabs, s.kinetic),) + eng.read(i))
    finally:
        _lib.call("sky_set_option", 2, old)
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][2], out[1][2])
