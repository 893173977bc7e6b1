"""The third moments of hist 'p' (stats columns 17-19 of a plane: the sums of
v u^2, v w^2 and v^3 over its points) in the FP64 step: to FP64 rounding of the
sum of |terms|.  The terms are good to a few 2^-53 at random (errors of the
transforms), and the oracle adds a plane's points one after the other, an error
of about sqrt(points) 2^-53 of the sum at most: 2^-47 for up to 2^12 rounding
errors of one sign, 2^-49 here, with the errors of either sign."""
import numpy as np
import pytest

from conftest import box_params, copy_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,kw", [((32, 32, 32), {}), ((96, 48, 64), {}), ((192, 32, 48), {}),
                                     ((64, 32, 32), {"temperature": 1, "fkappa": 0.01, "bym": 0.3})])
def test_third_moments_to_rounding(grid, kw):
    import oracle
    import shear_nnf_gb300 as sb
    pp = box_params(*grid, rez=2000.0, fixed_dt=0.004, **kw)
    p = sb.make_params(**pp)
    st = sb.seed_state(p, 2)
    box, orc = sb.ShearBox(p), oracle.Oracle(**pp)
    box.set_state(st)
    f = {k: v.reshape(p.my, -1) for k, v in box.physical(fields=("u", "v", "w")).items()}
    # the moments are those of the velocity without the mean shear
    y = np.arange(p.my) * (p.Ly / p.my) - p.Ly / 2
    u, v, w = f["u"] - y[:, None], f["v"], f["w"]
    size = np.stack([np.abs(v * u * u).sum(1), np.abs(v * w * w).sum(1), np.abs(v ** 3).sum(1)], 1)
    box.cross(copy_state(st), 1)
    orc.cross(copy_state(st), 1)
    a, b = box.statistics()["stats"][:, 16:19], orc.statistics()["stats"][:, 16:19]
    assert (np.abs(b) <= 1.0001 * size).all() and np.abs(b).max() > 1e-3 * size.max()
    err = np.abs(a - b) / size
    assert err.max() < 2.0 ** -49, (err.max(0), err.mean(0))


@pytest.mark.parametrize("key,value", [("vor", np.nan), ("phi", np.nan), ("vor", np.inf)])
def test_maxima_of_the_fields_that_are_finite(key, value):
    """The time step of a state with a number that is not finite in every plane
    of omega_y: that of max |v|, which does not depend on it; of phi: no
    maximum at all.  As the oracle's, record by record."""
    import oracle
    import shear_nnf_gb300 as sb
    pp = box_params(64, 32, 32, rez=2000.0, cfl=0.5, etime=50.0)
    p = sb.make_params(**pp)
    st = sb.seed_state(p, 4)
    st[key][3, 5, :] = value
    box, g = sb.ShearBox(p), copy_state(st)
    tr, status = box.cross(g, 1)
    ref, _ = oracle.Oracle(**pp).cross(copy_state(st), 1)
    ref = np.asarray(ref)
    assert tr.shape == ref.shape == (1, 24)
    # time, Delta t; the maxima u + shear, v, w and u
    for q in (0, 1, 14, 15, 16, 19):
        np.testing.assert_allclose(tr[:, q], ref[:, q], rtol=1e-12)
    assert status.time == pytest.approx(tr[0, 1], rel=1e-15)


def _moments(pp, st):
    import oracle
    import shear_nnf_gb300 as sb
    box, orc = sb.ShearBox(sb.make_params(**pp)), oracle.Oracle(**pp)
    box.cross(copy_state(st), 1)
    orc.cross(copy_state(st), 1)
    return [np.asarray(x.statistics()["stats"])[:, 16:19] for x in (box, orc)]


def test_moments_of_the_fields_that_are_finite():
    """A NaN in one plane of omega_y: u and w are lost in that plane alone, v
    nowhere, and with them the moments."""
    import shear_nnf_gb300 as sb
    pp = box_params(64, 32, 48, rez=2000.0, fixed_dt=0.004)
    st = sb.seed_state(sb.make_params(**pp), 6)
    st["vor"][2, 3, 11] = np.nan
    a, b = _moments(pp, st)
    assert np.array_equal(np.isfinite(a), np.isfinite(b))
    assert np.isfinite(a[:, 2]).all() and np.isfinite(a[:, :2]).sum() == 2 * 31
    ok = np.isfinite(a)
    np.testing.assert_allclose(a[ok], b[ok], rtol=1e-11, atol=1e-11 * np.abs(b[ok]).max())


@pytest.mark.parametrize("scale,finite", [(1e90, True), (1e120, False)])
def test_moments_past_the_range(scale, finite):
    """Velocities whose third powers pass the range of FP64 give no number."""
    import shear_nnf_gb300 as sb
    pp = box_params(64, 32, 48, rez=2000.0, fixed_dt=0.004)
    st = sb.seed_state(sb.make_params(**pp), 6)
    for k in ("vor", "phi", "u00", "w00"):
        st[k] = st[k] * scale
    a, b = _moments(pp, st)
    assert np.isfinite(a).all() == np.isfinite(b).all() == finite
    if finite:
        assert np.abs(a / scale ** 3 - b / scale ** 3).max() < 1e-11 * np.abs(b / scale ** 3).max()
    else:
        assert not np.isfinite(a).any()
