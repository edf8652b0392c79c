"""The x-chunk that the engine chooses for an instance (how many tiles a stage launch has)."""
import pytest

from tests.test_march import inputs, params_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,side,rows,blocks,per_sm", [("nuclear", 40, 16, 2, 1), ("nuclear", 48, 16, 2, 1),
                                                          ("coulomb", 48, 12, 2, 1), ("nuclear", 64, 16, 2, 1),
                                                          ("omega", 48, 8, 3, 2), ("omega", 64, 8, 3, 2)])
def test_small_fp32_lattices_do_not_share_sms_for_shorter_tiles(name, side, rows, blocks, per_sm):
    """Tiles that share an SM slow each other down: where a chunk that is a plane or two longer covers
    the lattice with fewer tiles per SM than the kernels have room for (`blocks`), the engine takes
    that.  rows: of a stage tile, which has 32 columns."""
    from skyrmion_solver_b200.engine import Engine
    th, p_i, p_f = params_for(name, (side,) * 3)
    F, _ = inputs(int(p_i[5]), (side,) * 3)
    with Engine(0) as eng:
        i = eng.add(name, (p_i, p_f), F, None, precision="fp32")
        tiles = -(-side // 32) * -(-side // rows) * -(-side // eng.xc(i))
    assert 64 <= tiles <= 148 * per_sm and per_sm < blocks
