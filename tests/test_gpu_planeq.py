"""The fixed-point plane stages of the FP64 step (k_z1, k_x2, k_z3) against the
oracle: every transform length in x and z, fields of very different sizes (each
sequence and product has its own scale), the rotation term, the temperature's
fields, the statistics of the products."""
import numpy as np
import pytest

from conftest import box_params, copy_state, rel_l2
from test_gpu_step import ONE_STEP

pytestmark = pytest.mark.gpu
LENGTHS = (32, 48, 64, 80, 96, 128, 160, 192, 256, 320, 384)


def _parity(pp, st, tol=ONE_STEP):
    import oracle
    import shear_nnf_gb300 as sb
    g, o = copy_state(st), copy_state(st)
    tr, _ = sb.ShearBox(sb.make_params(**pp)).cross(g, 1)
    ref = oracle.Oracle(**pp).cross(o, 1)
    for k in ("vor", "phi", "u00", "w00", "tb", "tb00"):
        if k in st:
            assert rel_l2(g[k], o[k]) < tol, (k, rel_l2(g[k], o[k]))
    return tr, ref


@pytest.mark.parametrize("n", LENGTHS)
def test_every_length(n):
    """Rotation, vbulk and a mean flow; n points in x, and in z where it is a
    z length; with the temperature where z allows it."""
    import shear_nnf_gb300 as sb
    for x, z, temp in ((n, 32, 0), (32, n, 0), (n, 48, 1), (48, n, 1)):
        if z == 320 or (temp and z > 256):
            continue
        kw = dict(temperature=1, fkappa=0.01, bym=0.4, gbeta=0.3) if temp else {}
        pp = box_params(x, 32, z, rez=2000.0, fixed_dt=0.002, chi=0.7, vbulk=0.05, **kw)
        st = sb.seed_state(sb.make_params(**pp), n + z)
        st["u00"] = 0.2 * np.cos(np.arange(32) * np.pi / 16)
        _parity(pp, st)


@pytest.mark.parametrize("small", (1e-6, 1e-13))
def test_fields_of_different_sizes(small):
    """Products of fields whose scales differ by many powers of two: a weak
    mean flow, weak omega_y fluctuations.  (With all fluctuations weak the
    products of the mean flow cancel to rounding in any arithmetic.)"""
    import shear_nnf_gb300 as sb
    for weak in (("u00", "w00"), ("vor",)):
        pp = box_params(64, 32, 48, rez=2000.0, fixed_dt=0.004, chi=0.1, keep_laminar=1)
        st = sb.seed_state(sb.make_params(**pp), 9)
        y = np.arange(32) * np.pi / 16
        st["u00"], st["w00"] = 0.7 * np.cos(y), 0.3 * np.sin(2 * y)
        for k in weak:
            st[k] = st[k] * small
        _parity(pp, st)


def test_statistics_of_the_products():
    """|u| maxima with the mean shear and the third moments (hist 'p')."""
    import oracle
    import shear_nnf_gb300 as sb
    pp = box_params(96, 48, 64, rez=2000.0, cfl=0.5)
    p = sb.make_params(**pp)
    st = sb.seed_state(p, 2)
    g, o = copy_state(st), copy_state(st)
    box, orc = sb.ShearBox(p), oracle.Oracle(**pp)
    tr, _ = box.cross(g, 2)
    ref = orc.cross(o, 2)[0]
    np.testing.assert_allclose(tr, np.asarray(ref)[: len(tr)], rtol=1e-11, atol=1e-13)
    a, b = box.statistics()["stats"][:, 16:19], orc.statistics()["stats"][:, 16:19]
    assert np.abs(a - b).max() < 1e-11 * np.abs(b).max()
