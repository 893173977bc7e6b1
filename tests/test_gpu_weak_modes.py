"""Weak fluctuations on a strong mean flow in the FP64 step: the products of the
mean flow alone are constant over a plane, exactly so, and must not leave
rounding in the modes (FP64 transforms of a constant leave none)."""
import numpy as np
import pytest

from conftest import box_params, copy_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", ({"vbulk": 0.2}, {"chi": 0.4}, {"vbulk": 0.2, "chi": -1.0},
                                {"vbulk": 0.2, "temperature": 1, "fkappa": 0.01, "gbeta": 0.3}))
@pytest.mark.parametrize("grid,weak", [((64, 32, 48), 1e-25), ((96, 33, 64), 1e-60),
                                       ((192, 48, 32), 1e-160), ((128, 32, 96), 1e-60)])
def test_weak_fluctuations_stay_weak(grid, weak, kw):
    """One step changes the modes by a fraction of themselves; a unit's noise of
    the mean products would be 1e-20 and more.  (The (0,0) entry of tb is none of
    the state: tb00 stands for it.)"""
    import shear_nnf_gb300 as sb
    p = sb.make_params(**box_params(*grid, rez=2000.0, fixed_dt=0.004, keep_laminar=1, **kw))
    st = sb.seed_state(p, 5)
    y = np.arange(p.my) * (2 * np.pi / p.my)
    keys = ("vor", "phi") + (("tb",) if p.temperature else ())
    for k in keys:
        st[k] = st[k] * weak
    st["u00"], st["w00"] = 0.7 * np.cos(y), 0.3 * np.sin(2 * y)
    if p.temperature:
        st["tb00"] = 0.5 * np.sin(y)
    g = copy_state(st)
    sb.ShearBox(p).cross(g, 1)
    size = max(np.abs(st[k]).max() for k in keys)
    if p.temperature:
        g["tb"][0, 0] = 0.0
    for k in keys:
        assert np.abs(g[k]).max() < 3 * size, (k, np.abs(g[k]).max(), size)
