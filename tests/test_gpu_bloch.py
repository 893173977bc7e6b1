"""The Bloch-wave form of the y-line stage (k_lineQ) at every line length it
covers, against the oracle and the banded split form: sheared states (nonzero
image offsets), ragged kx counts, mean profiles, LES; boxes whose image offsets
are not opposite, which keep the banded solves."""
import numpy as np
import pytest

from conftest import box_params, copy_state, rel_l2
from test_gpu_step import ONE_STEP

pytestmark = pytest.mark.gpu
LENGTHS = (32, 48, 64, 80, 96, 128, 160, 192, 256, 320, 384)


def _state(p, seed, xofft, xoffb=None):
    import shear_nnf_gb300 as sb
    st = sb.seed_state(p, seed)
    y = np.arange(p.my) * (2 * np.pi / p.my)
    st["u00"] = 0.1 * np.sin(y) + 0.02 * np.cos(3 * y)
    st["w00"] = 1e-6 * np.cos(2 * y)
    st["xofft"], st["xoffb"] = xofft, -xofft if xoffb is None else xoffb
    return st


def _parity(pp, st, nstep=1, tol=ONE_STEP, box=None):
    import oracle
    import shear_nnf_gb300 as sb
    box = box or sb.ShearBox(sb.make_params(**pp))
    g, o = copy_state(st), copy_state(st)
    box.cross(g, nstep)
    oracle.Oracle(**pp).cross(o, nstep)
    for k in ("vor", "phi", "u00", "w00"):
        assert rel_l2(g[k], o[k]) < tol, (k, rel_l2(g[k], o[k]))
    return box, g


@pytest.mark.parametrize("my", LENGTHS)
def test_one_step_at_every_length(my):
    """nkx = 16 (two full column blocks) and 21 (a ragged third)."""
    import shear_nnf_gb300 as sb
    for x in (48, 64):
        pp = box_params(x, my, 32, rez=2000.0, fixed_dt=0.3 * 2 * np.pi / my / 4)
        st = _state(sb.make_params(**pp), my + x, 1.7)
        box, _ = _parity(pp, st)
        assert box.tuning()["line_form"] == "fused"


@pytest.mark.parametrize("my", (32, 96, 160))
@pytest.mark.parametrize("kw", ({"les": 1, "cs": 0.1}, {"damping": 1, "damp_up": 0.5, "damp_aa": 0.2,
                                                        "force": -1, "xforce": 0.03}))
def test_options(my, kw):
    import shear_nnf_gb300 as sb
    pp = box_params(48, my, 32, rez=2000.0, fixed_dt=0.002, **kw)
    _parity(pp, _state(sb.make_params(**pp), my, -0.8), nstep=2, tol=4 * ONE_STEP)


@pytest.mark.parametrize("my", LENGTHS)
def test_mixed_close_to_the_banded_form(my):
    """Two steps in the FP32-mixed form: the two forms differ by FP32 rounding."""
    import shear_nnf_gb300 as sb
    p = sb.make_params(**box_params(64, my, 32, rez=2000.0, fixed_dt=0.002))
    st = _state(p, my, 2.9)
    out = {}
    for form in ("split", "fused"):
        box = sb.ShearBox(p, precision=sb.SB_MIXED)
        box.set_line_form(form)
        s = copy_state(st)
        box.cross(s, 2)
        out[form] = s
    for k in ("vor", "phi", "u00"):
        assert rel_l2(out["fused"][k], out["split"][k]) < 1e-6, k


@pytest.mark.parametrize("my", LENGTHS)
def test_semi_implicit_at_every_length(my):
    """implicit_visc = 1: two steps against the oracle, and in the FP32-mixed
    form against the banded solves (set_line_form("split"))."""
    import shear_nnf_gb300 as sb
    pp = box_params(48, my, 32, rez=1500.0, implicit_visc=1,
                    fixed_dt=0.3 * 2 * np.pi / my / 4)
    p = sb.make_params(**pp)
    st = _state(p, my, 1.3)
    box, _ = _parity(pp, st, nstep=2, tol=4 * ONE_STEP)
    assert box.tuning()["line_form"] == "implicit"
    out = {}
    for form in ("split", "waves"):
        box = sb.ShearBox(p, precision=sb.SB_MIXED)
        if form == "split":
            box.set_line_form(form)
        s = copy_state(st)
        box.cross(s, 2)
        out[form] = s
    for k in ("vor", "phi", "u00"):
        assert rel_l2(out["waves"][k], out["split"][k]) < 1e-6, k


def test_semi_implicit_options():
    """Damping and forcing of the mean, and unequal offsets (banded)."""
    import shear_nnf_gb300 as sb
    pp = box_params(48, 96, 32, rez=1500.0, implicit_visc=1, fixed_dt=0.003, damping=1,
                    damp_up=0.5, damp_aa=0.2, force=-1, xforce=0.03)
    p = sb.make_params(**pp)
    box, _ = _parity(pp, _state(p, 2, -0.8), nstep=2, tol=4 * ONE_STEP)
    _parity(pp, _state(p, 2, 1.1, xoffb=-0.9), nstep=2, tol=4 * ONE_STEP, box=box)
    _parity(pp, _state(p, 3, 0.7), nstep=2, tol=4 * ONE_STEP, box=box)


@pytest.mark.parametrize("my", LENGTHS)
def test_les_at_every_length(my):
    """The LES y-operators (k_lineLQ): one step against the oracle, and in the
    FP32-mixed form against the banded solves."""
    import shear_nnf_gb300 as sb
    pp = box_params(64, my, 32, rez=2000.0, les=1, cs=0.1, fixed_dt=0.3 * 2 * np.pi / my / 4)
    p = sb.make_params(**pp)
    st = _state(p, my, 1.7)
    _parity(pp, st)
    out = {}
    for form in ("split", "fused"):
        box = sb.ShearBox(p, precision=sb.SB_MIXED)
        box.set_line_form(form)
        s = copy_state(st)
        box.cross(s, 2)
        out[form] = s
    for k in ("vor", "phi", "u00"):
        assert rel_l2(out["fused"][k], out["split"][k]) < 1e-6, k


def test_unequal_offsets_keep_the_banded_solves():
    """xoffb != -xofft: one handle steps such a state (banded), then opposite
    offsets again, with the bits of a fresh handle."""
    import shear_nnf_gb300 as sb
    pp = box_params(64, 48, 32, rez=2000.0, fixed_dt=0.004)
    p = sb.make_params(**pp)
    even, odd = _state(p, 5, 1.1), _state(p, 5, 1.1, xoffb=-0.9)
    box, a = _parity(pp, even)
    _parity(pp, odd, box=box)
    _, b = _parity(pp, even, box=box)
    for k in ("vor", "phi", "u00", "w00"):
        assert np.array_equal(a[k], b[k]), k


def test_scales_of_a_batch_are_independent():
    """Boxes of amplitudes 1 and 1e-9 and a NaN box in one batch: each is the
    box it would be alone, bit for bit."""
    import shear_nnf_gb300 as sb
    p = sb.make_params(**box_params(64, 48, 32, rez=2000.0, fixed_dt=0.004, keep_laminar=1))
    st = [_state(p, 3, 0.4) for _ in range(3)]
    for k in ("vor", "phi", "u00", "w00"):
        st[1][k] = st[1][k] * 1e-9
    st[2]["phi"][3, 4, 5] = np.nan
    box = sb.ShearBox(p, batch=3)
    for m in range(3):
        box.set_state(st[m], m)
    box.step(2)
    for m in range(2):
        one = sb.ShearBox(p)
        one.set_state(st[m])
        one.step(2)
        a, b = one.get_state(), box.get_state(m)
        for k in ("vor", "phi", "u00", "w00"):
            assert np.array_equal(a[k], b[k]), (m, k)
    assert np.isnan(box.get_state(2)["vor"]).any() and box.status(2).flags & 2


# the semi-implicit block with the scalar takes lines up to 256
@pytest.mark.parametrize("my,implicit", [(n, i) for n in LENGTHS for i in (0, 1)
                                         if not (i and n > 256)])
def test_temperature_at_every_length(my, implicit):
    """The scalar's lines (tb and tb00, buoyancy in phi): two steps against the
    oracle, and in the FP32-mixed form against the banded solves."""
    import oracle
    import shear_nnf_gb300 as sb
    from test_gpu_temperature import _temp
    pp = dict(_temp((48, my, 32), 1500.0), fixed_dt=0.3 * 2 * np.pi / my / 4, implicit_visc=implicit)
    p = sb.make_params(**pp)
    st = _state(p, my, 1.3)
    st["tb00"] = st["tb00"] + 0.2 * np.cos(np.arange(my) * (2 * np.pi / my))
    keys = ("vor", "phi", "u00", "w00", "tb", "tb00")
    box, g, o = sb.ShearBox(p), copy_state(st), copy_state(st)
    box.cross(g, 2)
    oracle.Oracle(**pp).cross(o, 2)
    for k in keys:
        assert rel_l2(g[k], o[k]) < 4 * ONE_STEP, (k, rel_l2(g[k], o[k]))
    out = {}
    for form in ("split", "waves"):
        box = sb.ShearBox(p, precision=sb.SB_MIXED)
        if form == "split":
            box.set_line_form(form)
        s = copy_state(st)
        box.cross(s, 2)
        out[form] = s
    for k in ("vor", "phi", "u00", "tb", "tb00"):
        assert rel_l2(out["waves"][k], out["split"][k]) < 1e-6, k
