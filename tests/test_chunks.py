"""The x-chunk that the engine chooses for an instance (how many tiles a stage launch has)."""
import pytest

from tests.test_march import inputs, params_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,side,most", [("nuclear", 40, 148), ("nuclear", 48, 148), ("omega", 56, 148),
                                            ("coulomb", 48, 148), ("nuclear", 64, 296), ("omega", 64, 296)])
def test_small_fp32_lattices_do_not_share_sms_for_shorter_tiles(name, side, most):
    """Two tiles on one SM take longer than one: where one tile per SM (148) with a chunk that is a
    plane or two longer covers the lattice, the engine takes that, and never more than one wave of
    two per SM here.  (Rows of a stage tile: 16 nuclear, 12 omega and Coulomb; columns: 32.)"""
    from skyrmion_solver_b200.engine import Engine
    th, p_i, p_f = params_for(name, (side,) * 3)
    F, _ = inputs(int(p_i[5]), (side,) * 3)
    rows = 16 if name == "nuclear" else 12
    with Engine(0) as eng:
        i = eng.add(name, (p_i, p_f), F, None, precision="fp32")
        xc = eng.xc(i)
        tiles = -(-side // 32) * -(-side // rows) * -(-side // xc)
        assert tiles <= most
        assert tiles >= 64
