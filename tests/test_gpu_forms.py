"""Which y-line form a handle runs and what may change it: "split" on handles
that have no choice of form, the autotuner on boxes with unequal image offsets,
boxes without shear, changes of form between calls, single stages, memory that
does not hold the waves."""
import time

import numpy as np
import pytest

from conftest import box_params, copy_state, rel_l2
from test_gpu_bloch import LENGTHS, _state
from test_gpu_temperature import _temp

pytestmark = pytest.mark.gpu
KINDS = ("plain", "implicit", "temperature", "implicit_temperature")


def _params(kind, my=48, **kw):
    import shear_nnf_gb300 as sb
    base = dict(fixed_dt=0.004, **({"implicit_visc": 1} if "implicit" in kind else {}))
    base.update(kw)
    if "temperature" in kind:
        return sb.make_params(**_temp((64, my, 32), 1500.0, **base))
    return sb.make_params(**box_params(64, my, 32, rez=1500.0, **base))


def _cross(box, st, n=2):
    s = copy_state(st)
    box.cross(s, n)
    return s


def _keys(kind):
    return ("vor", "phi", "u00", "w00") + (("tb", "tb00") if "temperature" in kind else ())


def _same(kind, a, b):
    for k in _keys(kind):
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("kind", ("implicit", "temperature", "implicit_temperature"))
def test_split_changes_nothing_where_there_is_no_choice(kind):
    """These handles refuse "fused", so "split" must not take them off the
    step that they run."""
    import shear_nnf_gb300 as sb
    p = _params(kind)
    st = _state(p, 3, 1.3)
    ref = _cross(sb.ShearBox(p), st)
    box = sb.ShearBox(p)
    form = box.tuning()["line_form"]
    box.set_line_form("split")
    assert box.tuning()["line_form"] == form
    _same(kind, _cross(box, st), ref)
    with pytest.raises(sb.ShearBoxError):
        box.set_line_form("fused")
    _same(kind, _cross(box, st), ref)


def test_split_and_back():
    import shear_nnf_gb300 as sb
    p = _params("plain")
    st = _state(p, 3, 1.3)
    box = sb.ShearBox(p)
    ref = _cross(box, st)
    box.set_line_form("split")
    assert box.tuning()["line_form"] == "split"
    a = _cross(box, st)
    assert not np.array_equal(a["phi"], ref["phi"]) and rel_l2(a["phi"], ref["phi"]) < 1e-13
    box.set_line_form("fused")
    assert box.tuning()["line_form"] == "fused"
    _same("plain", _cross(box, st), ref)


@pytest.mark.parametrize("kind", KINDS)
def test_tuning_on_unequal_offsets_keeps_the_waves(kind):
    """The autotuner on a box with xoffb != -xofft picks among the banded
    kernels; opposite offsets afterwards run as on a fresh handle."""
    import shear_nnf_gb300 as sb
    p = _params(kind)
    st = _state(p, 4, 1.1)
    ref = _cross(sb.ShearBox(p), st)
    box = sb.ShearBox(p)
    box.set_state(_state(p, 4, 1.1, xoffb=-0.9))
    box.autotune()
    _same(kind, _cross(box, st), ref)


@pytest.mark.parametrize("kind", ("implicit", "temperature", "implicit_temperature"))
@pytest.mark.parametrize("my,precision", [(48, 0)] + [(n, 1) for n in LENGTHS])
def test_waves_close_to_the_banded_solves(kind, my, precision):
    """A box beside one with unequal offsets (banded solves for both) against
    the same box alone (waves): FP64 rounding, FP32 rounding in the mixed form.
    (The semi-implicit block with the scalar takes lines up to 256.)"""
    import shear_nnf_gb300 as sb
    if kind == "implicit_temperature" and my > 256:
        return
    p = _params(kind, my, fixed_dt=0.002)
    st = _state(p, 5, 1.3)
    one, two = sb.ShearBox(p, precision=precision), sb.ShearBox(p, batch=2, precision=precision)
    one.set_state(st)
    two.set_state(st, 0)
    two.set_state(_state(p, 6, 1.3, xoffb=-0.9), 1)
    one.step(2)
    two.step(2)
    a, b = one.get_state(), two.get_state(0)
    for k in set(_keys(kind)) - {"w00"}:
        assert rel_l2(a[k], b[k]) < (1e-6 if precision else 4e-12), k
    assert not np.array_equal(a["phi"], b["phi"])


def test_offsets_do_not_matter_without_shear():
    """s = 0: the image phases are one whatever the offsets."""
    import shear_nnf_gb300 as sb
    p = _params("plain", s=0.0)
    a = _cross(sb.ShearBox(p), _state(p, 7, 1.1))
    _same("plain", _cross(sb.ShearBox(p), _state(p, 7, 1.1, xoffb=-0.9)), a)


def test_changes_of_form_cost_one_capture():
    """Equal and unequal offsets in turn: the bits of fresh handles, and after
    the first pair no step call waits or captures again."""
    import shear_nnf_gb300 as sb
    p = _params("plain")
    st = [_state(p, 8, 1.1), _state(p, 8, 1.1, xoffb=-0.9)]
    ref = [_cross(sb.ShearBox(p), s) for s in st]
    box = sb.ShearBox(p)
    for q in (0, 1, 0, 1):
        _same("plain", _cross(box, st[q]), ref[q])

    def enqueue(order):
        best = []
        for q in order:
            box.set_state(st[q])
            t = time.perf_counter()
            box.step(1)
            best.append(time.perf_counter() - t)
            box.sync()
        return min(best)

    same = max(enqueue([0] * 10), enqueue([1] * 10))
    # a call takes 12 us, a capture of the step graph 120 more
    assert enqueue([0, 1] * 10) < 3 * same + 2e-5


@pytest.mark.parametrize("kind", ("plain", "implicit"))
def test_banded_stages_on_a_handle_on_waves(kind):
    """Substep 2 of a step by single stages, the banded y-line kernels on a
    handle that steps on waves, against a handle that runs them (beside a box
    with unequal offsets): stages 1-4, then 5 and 6, or 13 and 14."""
    import shear_nnf_gb300 as sb
    p = _params(kind)
    st = _state(p, 9, 1.3)
    one, two = sb.ShearBox(p), sb.ShearBox(p, batch=2)
    two.set_state(_state(p, 6, 1.3, xoffb=-0.9), 1)
    out = []
    for box in (one, two):
        box.set_state(st, 0)
        box.step(1)
        for stage in (1, 2, 3, 4) + ((13, 14) if kind == "implicit" else (5, 6)):
            box.launch_stage(stage, 2)
        box.sync()
        out.append(box.get_state(0))
    for k in ("vor", "phi", "u00"):
        assert np.isfinite(out[0][k]).all() and rel_l2(out[0][k], out[1][k]) < 4e-12, k
    # and the next step is the handle's own again
    _same(kind, _cross(one, st), _cross(sb.ShearBox(p), st))


def test_memory_for_the_banded_form_alone():
    """Where memory does not hold the waves the handle steps without them, as
    it would have before there were any."""
    torch = pytest.importorskip("torch")
    import shear_nnf_gb300 as sb
    p = _params("plain")
    batch = 512
    st = _state(p, 10, 1.3)

    def run(box):
        for m in (0, 1, batch - 1):
            box.set_state(st, m)
        box.step(2)
        return box.get_state(batch - 1)

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    for _ in range(2):  # the first loads the kernels
        before = free()
        box = sb.ShearBox(p, batch=batch)
        used = before - free()
        a = run(box)
        box.close()
    waves = 8 * batch * 2 * 2 * st["vor"].size  # 16 bytes for each number of vor and phi
    fill = torch.empty(free() - used + waves // 2, dtype=torch.uint8, device="cuda")
    try:
        box = sb.ShearBox(p, batch=batch)
        left = free()
        b = run(box)
        box.close()
    finally:
        del fill
        torch.cuda.empty_cache()
    assert left > waves // 4  # not for want of anything else
    for k in ("vor", "phi", "u00"):
        assert rel_l2(b[k], a[k]) < 4e-12, k
    assert not np.array_equal(a["phi"], b["phi"])


def test_side_work_does_not_slow_the_banded_semi_implicit_step():
    """The side branch of the step graph may not cost what it hides: its time
    against the same work in order (medians of nine; the branches differ by a
    few percent)."""
    torch = pytest.importorskip("torch")
    import shear_nnf_gb300 as sb
    p = sb.make_params(**box_params(128, 72, 128, rez=1500.0, fixed_dt=0.001, implicit_visc=1))
    box = sb.ShearBox(p)
    st = sb.seed_state(p, 1)
    stream = torch.cuda.ExternalStream(box.stream)
    took = {}
    for mask in (0, 1, 2, 3):
        box.set_side_branch(mask)
        box.set_state(st)
        box.step(2)
        times = []
        for _ in range(9):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record(stream)
            box.step(2)
            b.record(stream)
            b.synchronize()
            times.append(a.elapsed_time(b))
        took[mask] = sorted(times)[4]
    assert max(took.values()) < 1.15 * min(took.values()), took
