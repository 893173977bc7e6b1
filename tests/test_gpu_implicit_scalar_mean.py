"""The semi-implicit step with the scalar on banded solves where its y-line
kernel has more blocks than run at once: the block of the mean profiles reads
-vT of the (0,0) line, which no other block may have overwritten by then."""
import numpy as np
import pytest

from conftest import copy_state, rel_l2
from test_gpu_step import ONE_STEP
from test_gpu_temperature import KEYS, _temp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,xoffb", [((160, 48, 80), -0.4), ((192, 48, 96), -0.4),
                                        ((160, 50, 80), -0.7), ((160, 48, 80), -0.7)])
def test_mean_scalar_of_many_lines(grid, xoffb):
    """Unequal offsets, a line length without waves, and waves."""
    import oracle
    import shear_nnf_gb300 as sb
    pp = dict(_temp(grid, 1500.0), implicit_visc=1, fixed_dt=0.003, vbulk=0.2)
    p = sb.make_params(**pp)
    st = sb.seed_state(p, 86)
    st["tb00"] = st["tb00"] + 0.1 * np.cos(np.arange(p.my) * (2 * np.pi / p.my))
    st["xofft"], st["xoffb"] = 0.7, xoffb
    g, o = copy_state(st), copy_state(st)
    sb.ShearBox(p).cross(g, 1)
    oracle.Oracle(**pp).cross(o, 1)
    for k in KEYS:
        assert rel_l2(g[k], o[k]) < ONE_STEP, (k, rel_l2(g[k], o[k]))
