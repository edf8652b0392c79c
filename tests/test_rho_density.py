"""Rho's energy density (thirteen components in one walk) and its sum for odd rows, which are copied
value by value a column at a time, and for even ones, at the edges of the 8-row, 32-column tiles."""
import numpy as np
import pytest

from oracle import skyrme_oracle as O
from tests import _golden as G
from tests._gpu import dev, host
from tests.test_march import inputs, params_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(3, 8, 31), (6, 7, 33), (5, 9, 65), (9, 17, 32), (4, 6, 1), (37, 11, 34)])
def test_energy_density_of_rho(dims):
    """1e-12 relative to the largest density, the density bound of the parity tests."""
    from skyrmion_solver_b200 import _lib
    from skyrmion_solver_b200._lib import THEORY_IDS, f64p, i32p
    _, p_i, p_f = params_for("rho", dims)
    F, _ = inputs(13, dims, seed=17)
    field = dev(F)
    en = dev(np.zeros(dims))
    scratch = dev(np.zeros(int(_lib.load().sky_reduce_scratch_size(1))))
    args = (THEORY_IDS["rho"], i32p(p_i), len(p_i), f64p(p_f), len(p_f))
    _lib.call("sky_energy_density", *args, _lib.dptr(en), _lib.dptr(field), _lib.stream_ptr())
    total = np.zeros(1)
    _lib.call("sky_total_energy", *args, _lib.dptr(field), _lib.dptr(scratch), scratch.numel(), f64p(total),
              _lib.stream_ptr())
    want = O.energy_density(O.THEORIES["rho"], F, p_i, p_f)
    assert G.rel_err(host(en, dims), want) <= 1e-12
    assert abs(total[0] - np.sum(want)) <= 1e-12 * np.sum(np.abs(want))
