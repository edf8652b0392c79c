"""A field that is constant has no derivatives: its second differences vanish exactly, in FP32 too."""
import numpy as np
import pytest

from tests.test_march import params_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(14, 13, 36), (9, 18, 33)])
@pytest.mark.parametrize("precision", ["fp64", "fp32", "fp32c", "fp32d"])
def test_a_constant_field_stays_at_rest(precision, dims):
    """A constant isospin vector without pion mass: the gradient is zero at every site and so is the
    velocity after steps from rest, to the last bit."""
    from skyrmion_solver_b200.engine import Engine
    _, p_i, p_f = params_for("nuclear", dims)
    p_f = p_f.copy()
    p_f[8] = 0.0
    v = np.random.default_rng(2).normal(size=4)
    v = (v / np.sqrt((v * v).sum())).astype(np.float32).astype(np.float64)
    F = np.broadcast_to(v.reshape(4, 1, 1, 1), (4,) + dims).copy()
    with Engine(0) as eng:
        i = eng.add("nuclear", (p_i, p_f), F, None, precision=precision)
        eng.step(3)
        st = eng.stats(i)
        _, got = eng.read(i)
    assert st.gabs == 0.0 and st.kinetic == 0.0
    assert not np.any(got)
