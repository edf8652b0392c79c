"""The ray march over texels that show nothing but whose colour is not a number."""
import numpy as np
import pytest

from oracle import render_oracle as R
from skyrmion_solver_b200.visualization import HeadlessRenderer
from skyrmion_solver_b200.visualization.headless import inv_view_rows
from tests.test_render import _image_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("component", [1, 3])
def test_a_colour_that_is_no_number_below_the_level_set(bad, component):
    """A bright bump, and in front of it texels of no density whose pion vector has a component that
    is no number: zero times it is none either, so rays through those texels end without a colour
    (black) where the lightness is concerned (component 3), and with the bump's where only the
    direction is (1).  The oracle samples every step; its colours that are no numbers are black."""
    import torch
    dims = (24, 24, 24)
    x, y, z = np.meshgrid(*[(np.arange(n) + 0.5) * 2.0 / n - 1.0 for n in dims], indexing="ij")
    dens = np.exp(-10.0 * (x ** 2 + y ** 2 + z ** 2))
    vol = np.zeros(dims[::-1] + (4,), np.float32)
    vol[..., 0] = dens.transpose(2, 1, 0)
    vol[..., 3] = 0.6
    vol[..., 1] = 0.8
    vol[20:22, 9:13, 9:13, component] = bad     # towards the viewer, density far below the level set

    class _Sim:
        p_i_h = np.array(dims, np.int32)
        p_f_h = np.array(dims, np.float64)
    r = HeadlessRenderer(48, 36)
    r.bind_sim(_Sim())
    r.set_display_mode(2)
    r.set_render_params(opacity_scale=0.05, levelset=0.2, transfer_scale=4.0)
    r.volume.copy_(torch.from_numpy(vol))
    got = r.draw().cpu().numpy()
    with np.errstate(invalid="ignore"):
        want = R.render(vol, inv_view_rows(), box=r.box_scale, width=48, height=36, opacity_scale=0.05, color_mode=1)
    hidden = np.isnan(want).any(axis=-1)
    assert hidden.any() == (component == 3)
    assert _image_close(got, np.nan_to_num(want, nan=0.0))
