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
