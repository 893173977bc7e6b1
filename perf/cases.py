"""Performance cases of the shearing-box time stepper: what they are, their
inputs, one pass of each through the public entry points, and what a pass
returns as plain torch gives it in 64 bits.

Kinds of case:
  cross     the drop-in call on host arrays: state in, `steps` RK3 steps, state
            out (ShearBox.cross; crosst with the temperature)
  box       steps of resident boxes from packed device states to packed device
            states, as the period map of a search or a loop with GPU
            post-processing does (set_state_packed, step, get_state_packed)
  jv        a block of finite-difference products of the period map
            (ShearBox.jv_batch)
  krylov    one block Gram-Schmidt sweep on device-resident vectors (KSpace)
"""
from __future__ import annotations

import math

import numpy as np
import torch

import shear_nnf_gb300 as sb
from shear_nnf_gb300.krylov import KSpace

LZ = 2 * math.pi
GAMMA = (8.0 / 15.0, 5.0 / 12.0, 3.0 / 4.0)
ZETA = (-17.0 / 60.0, -5.0 / 12.0, 0.0)
CK = (8.0 / 15.0, 2.0 / 3.0, 1.0)
ALPHA = (29.0 / 96.0, -3.0 / 40.0, 1.0 / 6.0)
IBETA = (160.0 / 37.0, 24.0 / 5.0, 6.0)


def _grid(x, y, z, **kw):
    c = {"x": x, "y": y, "z": z, "batch": 1, "mixed": False, "les": False, "temperature": False,
         "implicit": False, "tune": False, "rez": 1000.0, "fixed_dt": 0.0}
    c.update(kw)
    return c


def listed():
    return [
        # the smallest run: one step of the 64x32x32 box per call of the
        # drop-in, latency bound
        dict(_grid(64, 32, 32, fixed_dt=0.005), kind="cross", steps=1, name="cross_64x32x32"),
        # the drop-in at the benchmark box: host copies and one step per call
        dict(_grid(192, 96, 96, rez=4000.0), kind="cross", steps=1, name="cross_192x96x96"),
        # a long FP64 run of the benchmark box, tiles tuned as such a run does
        dict(_grid(192, 96, 96, rez=4000.0, tune=True), kind="box", steps=10, name="box_192x96x96"),
        # the same in the FP32-mixed form
        dict(_grid(192, 96, 96, rez=4000.0, tune=True, mixed=True), kind="box", steps=10,
             name="box_192x96x96_mixed"),
        # the largest FP64 box
        dict(_grid(384, 192, 192, rez=20000.0), kind="box", steps=2, name="box_384x192x192"),
        # large-eddy simulation, FP32-mixed
        dict(_grid(384, 192, 192, rez=20000.0, mixed=True, les=True), kind="box", steps=2,
             name="les_384x192x192_mixed"),
        # ensemble: 64 small boxes of different Reynolds numbers in one batch
        dict(_grid(64, 32, 32, batch=64, mixed=True, tune=True), kind="box", steps=10,
             name="ensemble_64x32x32x64_mixed"),
        # a few boxes of an odd grid (5-smooth x and z, my = 75), default tiles
        dict(_grid(160, 75, 80, batch=3), kind="box", steps=4, name="boxes_160x75x80x3"),
        # Boussinesq scalar through the drop-in crosst
        dict(_grid(192, 96, 96, rez=4000.0, temperature=True), kind="cross", steps=4,
             name="crosst_192x96x96"),
        # semi-implicit viscous terms
        dict(_grid(96, 48, 48, rez=1200.0, implicit=True), kind="box", steps=6,
             name="implicit_96x48x48"),
        # a block of 8 FP64 products of the period map for Newton-Krylov
        dict(_grid(96, 48, 48, rez=1200.0, batch=9), kind="jv", ndir=8, period=0.5,
             name="jv_96x48x48x8"),
        # orthogonalisation of a block of 16 vectors against 48 (96x48x48 unknowns)
        {"kind": "krylov", "n": 187488, "basis": 48, "block": 16, "name": "krylov_187488x48x16"},
    ]


XLEN = (32, 48, 64, 80, 96, 128, 160, 192, 256, 320, 384)
ZLEN = (32, 48, 64, 80, 96, 128, 160, 192, 256, 384)


def _points(c):
    return c["x"] * c["y"] * c["z"] * c["batch"]


def draw(rng):
    kind = rng.choice(["cross", "cross", "box", "box", "box", "box", "box", "jv", "krylov"])
    if kind == "krylov":
        return {"kind": kind, "n": int(math.exp(rng.uniform(math.log(2e4), math.log(6e5)))),
                "basis": rng.randint(4, 64), "block": rng.randint(1, 32)}
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))  # noqa: E731
    top = 384 * 192 * 192 * (0.1 if kind == "cross" else 0.02 if kind == "jv" else 1.0)
    while True:
        c = _grid(rng.choice(XLEN), log(16, 224), rng.choice(ZLEN))
        if rng.random() < 0.5:  # the usual lengths in y
            c["y"] = rng.choice((32, 48, 64, 80, 96, 128, 160, 192))
        if kind == "jv":
            c["batch"] = rng.randint(3, 12)
        elif kind == "box" and rng.random() < 0.4:
            c["batch"] = log(2, 64)
        if 20000 <= _points(c) <= top:
            break
    c["kind"] = kind
    c["rez"] = float(log(500, 20000))
    if rng.random() < 0.2:
        c["fixed_dt"] = 0.004
    if kind == "jv":
        c["ndir"], c["period"] = c["batch"] - 1, rng.uniform(0.15, 0.4)
        return c
    c["steps"] = rng.randint(1, 3) if kind == "cross" else rng.randint(1, 4)
    opt = rng.choice(["plain", "plain", "plain", "les", "temperature", "implicit"])
    if opt == "les" and c["x"] <= 256 and c["z"] <= 192:
        c["les"] = True
    elif opt == "implicit":
        c["implicit"] = True
    elif opt == "temperature" and kind == "cross" and c["z"] <= 256:
        c["temperature"] = True
    if kind == "box":
        c["mixed"] = rng.random() < 0.4
        c["tune"] = rng.random() < 0.2
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _params(c):
    return dict(mgalx=c["x"], my=c["y"], mgalz=c["z"], Re=c["rez"] / LZ ** 2, alp=0.5, Ly=LZ,
                gam=1.0, s=1.0, CFL=0.5, fixed_dt=c["fixed_dt"], les=int(c["les"]), cs=0.1,
                temperature=int(c["temperature"]), implicit_visc=int(c["implicit"]),
                fkappa=LZ ** 2 / c["rez"] / 0.7 if c["temperature"] else 0.0,
                bym=0.3 if c["temperature"] else 0.0, gbeta=0.2 if c["temperature"] else 0.0)


def _wavenumbers(c, dev="cpu"):
    """kx (nkx), kz (mz) of the kept modes."""
    nkx, nz = c["x"] // 3, (2 * (c["z"] // 3) - 2) // 2
    kx = 0.5 * torch.arange(nkx, dtype=torch.float64, device=dev)
    kz = torch.cat([torch.arange(nz + 1), torch.arange(-nz, 0)]).to(torch.float64).to(dev)
    return kx, kz


def _conj_sym(f):
    """The kx = 0 entries of negative kz as conjugates of those of positive kz."""
    nz = (f.shape[-3] - 1) // 2
    f[..., nz + 1:, 0, :] = f[..., 1:nz + 1, 0, :].flip(-2).conj()
    return f


def _initial(c, seed):
    """Seeded turbulent-like states: vor, phi [B, mz, nkx, my], u00, w00 [B, my],
    the image offset xofft [B] (and tb, tb00 with the temperature), made on the
    GPU."""
    dev = "cuda"
    g = torch.Generator(device=dev).manual_seed(int(seed) * 1000003 + 17)
    kx, kz = _wavenumbers(c, dev)
    B, my, k0 = c["batch"], c["y"], 6.0 if c["les"] else 4.0
    ky = torch.fft.fftfreq(my, 1.0 / my, dtype=torch.float64, device=dev)
    kh2 = kx[None, :, None] ** 2 + kz[:, None, None] ** 2
    k2 = kh2 + ky ** 2
    # velocity modes of E(k) ~ k^4 exp(-2 (k/k0)^2), nothing at the y cut-off
    amp = torch.sqrt(k2) * torch.exp(-k2 / k0 ** 2) * (ky.abs() < my // 3)
    urms = 0.1 * LZ

    def modes(a):
        z = torch.randn((B,) + a.shape + (2,), generator=g, dtype=torch.float64, device=dev)
        f = _conj_sym(torch.fft.ifft(torch.view_as_complex(z) * a, dim=-1) * my)
        f[:, 0, 0] = 0
        return f

    norm = urms / math.sqrt(2.0 * float((amp ** 2).sum()))
    st = {"phi": modes(-amp * k2 * norm), "vor": modes(amp * torch.sqrt(kh2) * norm)}
    y = torch.arange(my, dtype=torch.float64, device=dev) * (2 * math.pi / my)

    def profile():
        a = torch.randn((B, 3, 2), generator=g, dtype=torch.float64, device=dev) * 0.05
        return sum(a[:, q, :1] * torch.cos((q + 1) * y) + a[:, q, 1:] * torch.sin((q + 1) * y)
                   for q in range(3))

    st["u00"], st["w00"] = profile(), profile()
    if c["temperature"]:
        st["tb"], st["tb00"] = modes(amp * norm), profile()
    st["xofft"] = LZ * torch.rand(B, generator=g, dtype=torch.float64, device=dev)
    return st


def _members_re(c):
    """Reynolds numbers of a batch, log-uniform around the case's."""
    return [c["rez"] / LZ ** 2 * 2.0 ** ((m + 0.5) / c["batch"] * 2 - 1) if c["batch"] > 1
            else c["rez"] / LZ ** 2 for m in range(c["batch"])]


def _pack(vor, phi, u00, w00):
    """The packed unknown vector of one state [mz, nkx, my]: the profiles, then
    per plane and mode (without (0,0) and the kx = 0 entries of negative kz)
    vor.re, phi.re, vor.im, phi.im."""
    x = torch.stack([vor.real, phi.real, vor.imag, phi.imag], -1).permute(2, 0, 1, 3)
    return torch.cat([u00, w00, x[:, _kept(vor.shape[0], vor.shape[1], vor.device)].reshape(-1)])


def _kept(mz, nkx, dev):
    keep = torch.ones((mz, nkx), dtype=torch.bool, device=dev)
    keep[0, 0] = False
    keep[(mz - 1) // 2 + 1:, 0] = False
    return keep


def prepare(case, seed):
    c = case
    if c["kind"] == "krylov":
        g = torch.Generator(device="cuda").manual_seed(int(seed) * 7 + 1)
        n, m, p = c["n"], c["basis"], c["block"]
        v = torch.randn((n, m + p), generator=g, dtype=torch.float64, device="cuda")
        q = torch.linalg.qr(v[:, :m])[0].T.contiguous()
        ks = KSpace(n, m + p)
        for i in range(m):
            ks_col(ks, i, n).copy_(q[i])
        w = v[:, m:].T.contiguous()
        return {"case": c, "ks": ks, "w": w, "q": q, "out": torch.empty_like(w)}
    st = _initial(c, seed)
    p = sb.make_params(**_params(c))
    box = sb.ShearBox(p, batch=c["batch"], precision=sb.SB_MIXED if c["mixed"] else sb.SB_FP64)
    if c["kind"] == "cross":
        host = {k: np.ascontiguousarray(st[k][0].cpu().numpy())
                for k in ("vor", "phi", "u00", "w00", "tb", "tb00") if k in st}
        xt = float(st["xofft"][0])
        host.update(time=0.0, xoffb=-xt, xofft=xt)
        return {"case": c, "box": box, "state": host}
    if c["kind"] == "jv":
        vec = [torch.cat([torch.view_as_real(st["vor"][b]).reshape(-1),
                          torch.view_as_real(st["phi"][b]).reshape(-1), st["u00"][b],
                          st["w00"][b]]).cpu().numpy() for b in range(c["ndir"] + 1)]
        return {"case": c, "box": box, "x0": vec[0], "dirs": np.stack(vec[1:]),
                "xofft": float(st["xofft"][0])}
    for m, re in enumerate(_members_re(c)):
        if c["batch"] > 1:
            box.set_re(m, re)
    x = [_pack(st["vor"][b], st["phi"][b], st["u00"][b], st["w00"][b]) for b in range(c["batch"])]
    s = {"case": c, "box": box, "x": torch.stack(x), "xofft": st["xofft"].tolist(),
         "stream": torch.cuda.ExternalStream(box.stream)}
    s["out"] = torch.empty_like(s["x"])
    if c["mixed"]:
        s["out32"] = torch.empty_like(s["x"], dtype=torch.float32)
    if c["tune"]:
        torch.cuda.synchronize()
        _set(s)
        box.autotune()
    return s


def ks_col(ks, col, n):
    """A column of the Krylov space as a torch tensor on its device memory."""
    class _Mem:
        __cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ks.col(col), False),
                                    "version": 2, "strides": None}
    return torch.as_tensor(_Mem(), device="cuda")


def _set(s):
    row = s["x"].stride(0) * 8
    for b, xt in enumerate(s["xofft"]):
        s["box"].set_state_packed(b, s["x"].data_ptr() + b * row, (1.0, 1.0, 1.0), 0.0, -xt, xt)


def run(state):
    s = state
    c = s["case"]
    if c["kind"] == "krylov":
        # classical Gram-Schmidt, twice: new vectors in, the part outside the
        # basis and the coefficients out
        ks, n, m, p = s["ks"], c["n"], c["basis"], c["block"]
        with torch.cuda.stream(torch.cuda.ExternalStream(int(sb.lib().sb_kspace_stream(ks.h)))):
            for i in range(p):
                ks_col(ks, m + i, n).copy_(s["w"][i], non_blocking=True)
            h = ks.gram(0, m, m, p)
            ks.update(0, m, m, p, h, -1.0)
            h2 = ks.gram(0, m, m, p)
            ks.update(0, m, m, p, h2, -1.0)
            for i in range(p):
                s["out"][i].copy_(ks_col(ks, m + i, n), non_blocking=True)
        return {"h": h + h2, "w": s["out"]}
    box = s["box"]
    if c["kind"] == "cross":
        st = s["state"]
        box.cross(st, c["steps"])
        return {k: st[k] for k in ("vor", "phi", "u00", "w00", "tb", "tb00", "time", "xofft")
                if k in st}
    if c["kind"] == "jv":
        return box.jv_batch(s["x0"], s["dirs"], c["period"], eps_jacobi=1e-4, xoffb=-s["xofft"],
                            xofft=s["xofft"])
    _set(s)
    box.step(c["steps"])
    row = s["out"].stride(0) * 8
    for b in range(c["batch"]):
        box.get_state_packed(b, s["out"].data_ptr() + b * row, (1.0, 1.0, 1.0))
    if not c["mixed"]:
        return {"x": s["out"]}
    with torch.cuda.stream(s["stream"]):  # an FP32-mixed state holds 32-bit numbers
        s["out32"].copy_(s["out"])
    return {"x": s["out32"]}


def work(case):
    """Bytes: each input read once and each output written once, and the state
    (vor, phi) read and written once per RK3 substep; flops: the 2-D
    transforms of nine fields per substep at 5 N log2 N per complex transform
    of length N, the products, and 60 per mode for the banded y-operators."""
    c = case
    if c["kind"] == "krylov":
        n, m, p = c["n"], c["basis"], c["block"]
        return {"bytes": 8.0 * n * (m + 3 * p), "flops": 8.0 * n * m * p}
    nkx, mz = c["x"] // 3, 2 * (c["z"] // 3) - 1
    modes = float(nkx * mz * c["y"] * c["batch"])
    nf = 9 + (4 if c["temperature"] else 0) + (14 if c["les"] else 0)
    z = nf * nkx * 5.0 * c["z"] * math.log2(c["z"])
    x = nf * c["z"] / 2 * 5.0 * c["x"] * math.log2(c["x"])
    sub = (z + x + 12.0 * c["x"] * c["z"]) * c["y"] * c["batch"] + 6 * 2 * 60.0 * modes
    word = 8 if c["mixed"] else 16
    steps = c["steps"] if "steps" in c else max(2, round(c["period"] * max(c["x"], c["z"]) / 3))
    nst = 3 if c["temperature"] else 2
    return {"bytes": 2 * 16 * nst * modes + 2 * nst * word * modes * 3 * steps,
            "flops": 3.0 * steps * sub}


# ---------------------------------------------------------------------------
# the same in 64 bits, plain torch: y-operators applied to the Bloch waves of a
# line, u_j ~ exp(i t_m j), t_m = (2 pi m - kx xofft)/my, which diagonalise the
# shear-periodic compact schemes
# ---------------------------------------------------------------------------
def _compact():
    """pr1, rh1*dy, pr2, rh2*dy^2 of the seven-point compact schemes (entries
    d = 0..3; rh1 antisymmetric): order conditions and three wavenumbers where
    the modified wavenumber is exact."""
    j = np.arange(1, 4)
    kap = np.array([0.5, 0.9, 0.7]) * math.pi
    m, v = np.zeros((6, 6)), np.zeros(6)
    for r, k in enumerate((1, 3, 5)):
        m[r, :3], m[r, 3:] = k * j.astype(float) ** (k - 1), -j.astype(float) ** k
    v[0] = -0.5
    for r, k in enumerate(kap):
        m[3 + r, :3], m[3 + r, 3:], v[3 + r] = k * np.cos(k * j), -np.sin(k * j), -0.5 * k
    a = np.linalg.solve(m, v)
    pr1, rh1 = np.r_[1.0, a[:3]], np.r_[0.0, a[3:]]
    kap = np.array([0.9, 0.5, 0.7]) * math.pi
    m, v = np.zeros((7, 7)), np.zeros(7)
    m[0, 3], m[0, 4:] = 0.5, 1.0
    for r, k in enumerate((2, 4, 6)):
        m[1 + r, :3], m[1 + r, 4:] = k * (k - 1) * j.astype(float) ** (k - 2), -j.astype(float) ** k
    v[1] = -1.0
    for r, k in enumerate(kap):
        m[4 + r, :3], m[4 + r, 3], m[4 + r, 4:] = k * k * np.cos(k * j), 0.5, np.cos(k * j)
        v[4 + r] = -0.5 * k * k
    a = np.linalg.solve(m, v)
    return pr1, rh1, np.r_[1.0, a[:3]], a[3:]


class _Lines:
    """y-operators on [B, mz, nkx, my] lines at the image offsets xt [B]."""

    def __init__(self, c, kx, xt):
        my = c["y"]
        j = torch.arange(my, dtype=torch.float64, device=kx.device)
        t0 = -(kx[None, :] * xt[:, None]) / my
        self.tw = torch.polar(torch.ones_like(t0)[..., None] * torch.ones_like(j),
                              -t0[..., None] * j)[:, None]
        t = (t0[..., None] + 2 * math.pi * j / my)[:, None]
        pr1, rh1, pr2, rh2 = _compact()
        dy = LZ / my
        s1 = sum(2 * rh1[d] * torch.sin(d * t) for d in (1, 2, 3)) / dy
        p1 = 1 + sum(2 * pr1[d] * torch.cos(d * t) for d in (1, 2, 3))
        s2 = (rh2[0] + sum(2 * rh2[d] * torch.cos(d * t) for d in (1, 2, 3))) / dy ** 2
        p2 = 1 + sum(2 * pr2[d] * torch.cos(d * t) for d in (1, 2, 3))
        self.l1, self.l2 = 1j * s1 / p1, s2 / p2

    def _apply(self, f, lam):
        return torch.fft.ifft(torch.fft.fft(f * self.tw, dim=-1) * lam, dim=-1) * self.tw.conj()

    def d1(self, f):
        return self._apply(f, self.l1)

    def d2(self, f):
        return self._apply(f, self.l2)

    def helm(self, f, k2):
        """The solution of (d2/dy2 - k2) p = f; zero where k2 = 0."""
        z = torch.as_tensor(k2 == 0)
        den = self.l2 - k2
        return self._apply(f, torch.where(z, torch.zeros_like(den), 1.0 / den))


def _to_phys(c, f):
    """[B, mz, nkx, my] spectra to [B, my, Z, X] values."""
    B, mz, nkx, my = f.shape
    nz = (mz - 1) // 2
    g = torch.zeros((B, my, c["z"], c["x"] // 2 + 1), dtype=f.dtype, device=f.device)
    f = f.permute(0, 3, 1, 2)
    g[:, :, :nz + 1, :nkx] = f[:, :, :nz + 1]
    g[:, :, c["z"] - nz:, :nkx] = f[:, :, nz + 1:]
    g = torch.fft.ifft(g, dim=2, norm="forward")
    g[..., 0].imag.zero_()
    return torch.fft.irfft(g, n=c["x"], dim=3, norm="forward")


def _to_modes(c, r):
    nkx, nz = c["x"] // 3, (2 * (c["z"] // 3) - 2) // 2
    g = torch.fft.fft(torch.fft.rfft(r, dim=3, norm="forward")[..., :nkx], dim=2, norm="forward")
    return torch.cat([g[:, :, :nz + 1], g[:, :, c["z"] - nz:]], 2).permute(0, 2, 3, 1).contiguous()


def _step_exact(c, st, re, steps=None, etime=None):
    """RK3 steps of a batch of states in place (dict of _initial, with time
    [B]); re [B].  With etime, steps until every member has reached it."""
    dev = st["vor"].device
    kx, kz = _wavenumbers(c, dev)
    my = c["y"]
    nkx, mz = len(kx), len(kz)
    B = st["vor"].shape[0]
    kh2 = (kz[:, None] ** 2 + kx ** 2)[None, :, :, None]
    a, g = kx[None, None, :, None], kz[None, :, None, None]
    ik = torch.where(kh2 > 0, 1.0 / kh2.clamp(min=1e-30), torch.zeros_like(kh2))
    zero = torch.zeros(B, dtype=torch.float64, device=dev)
    y = torch.arange(my, dtype=torch.float64, device=dev) * (LZ / my) - LZ / 2
    dx, dy, dz = 4 * math.pi / (2 * nkx), LZ / my, LZ / mz
    vv = max((math.pi / dx) ** 2, 6.25 / dy ** 2, (math.pi / dz) ** 2)
    nu = (1.0 / re)[:, None, None, None]
    par = _params(c)
    kap, bym, gb = par["fkappa"], par["bym"], par["gbeta"]
    les, impl, temp = c["les"], c["implicit"], c["temperature"]
    flat = _Lines(c, kx[:1], zero)  # kx = 0: the periodic operators of the mean profiles
    prof = lambda f, op: getattr(flat, op)(f.to(torch.complex128)[:, None, None, :])[:, 0, 0].real  # noqa: E731
    c00 = lambda f: f.to(torch.complex128)  # noqa: E731
    keys = ["vor", "phi"] + (["tb"] if temp else [])
    means = ["u00", "w00"] + (["tb00"] if temp else [])
    for k in keys:
        _conj_sym(st[k])
    st.setdefault("time", zero.clone())
    live = torch.ones(B, dtype=torch.bool, device=dev)
    nutmax = zero.clone()
    it = 0
    while it < steps if etime is None else bool(live.any()) and it < 1000:
        it += 1
        old = {k: v.clone() for k, v in st.items()} if etime is not None else None
        xt0 = st["xofft"].clone()
        wk = {}
        xt = xt0
        for rk in range(3):
            L = _Lines(c, kx, xt)
            v = L.helm(st["phi"], kh2)
            dv, dw = L.d1(v), L.d1(st["vor"])
            sym = {k: _conj_sym(st[k].clone()) for k in ("vor", "phi")}
            u1 = 1j * ik * (a * dv - g * sym["vor"])
            u3 = 1j * ik * (g * dv + a * sym["vor"])
            o1 = 1j * ik * (a * dw + g * sym["phi"])
            o3 = 1j * ik * (g * dw - a * sym["phi"])
            du, dwm = prof(st["u00"], "d1"), prof(st["w00"], "d1")
            u1[:, 0, 0], u3[:, 0, 0] = c00(st["u00"]), c00(st["w00"])
            o1[:, 0, 0], o3[:, 0, 0] = c00(dwm), c00(-du)
            v[:, 0, 0] = 0
            U, V, W = _to_phys(c, u1), _to_phys(c, v), _to_phys(c, u3)
            les_rhs = None
            if les:
                S = [1j * a * u1, dv, 1j * g * u3, 2j * g * v + o1, 2j * a * v - o3,
                     1j * g * u1 + 1j * a * u3]
                ux, vy, wz, vz, uy, uz = [_to_phys(c, f) for f in S]
                uy = uy + 1.0
                S2 = 2 * (ux * ux + vy * vy + wz * wz) + uy * uy + uz * uz + vz * vz
                S2 = _to_phys(c, _to_modes(c, S2))
                nut = (0.1 * (dx * dy * dz) ** (1 / 3)) ** 2 * torch.sqrt(S2.abs())
                if rk == 0:
                    nutmax = torch.maximum(nutmax, nut.abs().amax((1, 2, 3)))
                t11, t22, t33, t12, t13, t23 = [_to_modes(c, nut * f) for f in
                                                (2 * ux, 2 * vy, 2 * wz, uy, uz, vz)]
                les_rhs = (a * a * t11 + 2 * a * g * t13 + g * g * t33 - kh2 * t22,
                           1j * a * t12 + 1j * g * t23,
                           -a * g * (t11 - t33) + (a * a - g * g) * t13,
                           1j * g * t12 - 1j * a * t23, t12[:, 0, 0].real, t23[:, 0, 0].real)
                del S, ux, vy, wz, vz, uy, uz, S2, nut
            if rk == 0:
                um = [f.abs().amax((1, 2, 3)) for f in (U, V, W)]
                if c["fixed_dt"] > 0:
                    dt = torch.full_like(zero, c["fixed_dt"])
                else:
                    m = torch.maximum(torch.maximum(um[0] * math.pi / dx, um[1] * 2.5 / dy),
                                      um[2] * math.pi / dz) / 0.5
                    dt = 1.0 / m
                    vis = torch.maximum(1.0 / re, nutmax) * vv / 0.5
                    cv = 0.5 * vis * dt
                    if temp:
                        ck = kap * vv * dt
                        lim = torch.where(ck > cv, torch.full_like(dt, 0.5 / (kap * vv)), 1.0 / vis)
                        dt = (torch.where(cv > 2.0, lim / 0.5 * 6.0, dt) if impl else
                              torch.where(cv > 0.5, lim, dt))
                    elif not impl:
                        dt = torch.where(cv > 0.5, 1.0 / vis, dt)
                if etime is not None:
                    over = st["time"] + dt > etime
                    dt = torch.where(over, (etime - st["time"]).abs(), dt)
            O1, O2, O3 = _to_phys(c, o1), _to_phys(c, sym["vor"]), _to_phys(c, o3)
            rhs, rmean = {}, {}
            if temp:
                tc = st["tb"].clone()
                tc[:, 0, 0] = c00(st["tb00"])
                T = _to_phys(c, tc)
                uT, wT, vT = [_to_modes(c, f * T) for f in (U, W, V)]
                rhs["tb"] = -1j * a * uT - 1j * g * wT - bym * L.helm(st["phi"], kh2) - L.d1(vT)
                rmean["tb00"] = -prof(vT[:, 0, 0].real, "d1")
            H1, H2, H3 = [_to_modes(c, f) for f in (V * O3 - W * O2, W * O1 - U * O3,
                                                    U * O2 - V * O1)]
            del U, V, W, O1, O2, O3
            rmean["u00"], rmean["w00"] = H1[:, 0, 0].real, H3[:, 0, 0].real
            vin = L.helm(st["phi"], kh2)
            dd = 1j * a * H1 + 1j * g * H3
            hg = 1j * g * (H1 - vin) - 1j * a * H3
            hv = -kh2 * H2
            if les:
                dd = dd - les_rhs[0]
                hg = hg + les_rhs[2] + L.d1(les_rhs[3])
                f = les_rhs[1]
                hv = hv - (L.d2(f) + kh2 * f) * (kh2 > 0)
                rmean["u00"] = rmean["u00"] + prof(les_rhs[4], "d1")
                rmean["w00"] = rmean["w00"] + prof(les_rhs[5], "d1")
            hv = hv - L.d1(dd)
            on = kh2 > 0
            lap = {k: (L.d2(st[k]) - kh2 * st[k]) * on for k in keys}
            lmean = {k: prof(st[k], "d2") for k in means}
            if temp:
                hv = hv + gb * lap["tb"]
            rhs["vor"], rhs["phi"] = hg, hv
            dif = {"vor": nu, "phi": nu, "tb": kap}
            dmean = {"u00": 1.0 / re[:, None], "w00": 1.0 / re[:, None], "tb00": kap}
            D4, D2 = dt[:, None, None, None], dt[:, None]
            xn = xt0 + CK[rk] * dt * LZ
            N = _Lines(c, kx, xn)
            df = CK[rk] - (CK[rk - 1] if rk else 0.0)
            ph = torch.polar(torch.ones_like(D4) * torch.ones_like(a * y), -(a * y) * (df * D4))
            f1 = GAMMA[0] if rk == 0 else GAMMA[1] + ZETA[0]
            pz = torch.polar(torch.ones_like(D4) * torch.ones_like(a * y), -(a * y) * (f1 * D4))
            for k in keys:
                f = st[k]
                h = rhs[k] if impl else rhs[k] + dif[k] * lap[k]
                w = GAMMA[rk] * h + (wk[k] if rk else 0)
                if impl:
                    d = dif[k]
                    fac = -IBETA[rk] / d * (w + ALPHA[rk] * d * lap[k] + f / D4)
                    new = N.helm(fac * ph, kh2 + IBETA[rk] / d / D4)
                    st[k] = torch.where(on, new, f)  # the (0,0) lines keep their state
                else:
                    st[k] = (f + D4 * w) * ph
                if rk < 2:
                    wk[k] = ZETA[rk] * h * pz
            for k in means:
                f = st[k]
                h = rmean[k] if impl else rmean[k] + dmean[k] * lmean[k]
                w = GAMMA[rk] * h + (wk[k] if rk else 0)
                if impl:
                    d = dmean[k]
                    fac = -IBETA[rk] / d * (w + ALPHA[rk] * d * lmean[k] + f / D2)
                    k2 = (IBETA[rk] / d / D2)[:, None, None, :]
                    st[k] = flat.helm(c00(fac)[:, None, None, :], k2)[:, 0, 0].real
                else:
                    st[k] = f + D2 * w
                if rk < 2:
                    wk[k] = ZETA[rk] * h
            xt = xn
        st["xofft"] = xt
        st["time"] = st["time"] + dt
        if etime is not None:
            for k in st:
                m = live.reshape((B,) + (1,) * (st[k].dim() - 1))
                st[k] = torch.where(m, st[k], old[k])
            live = live & ~(over & torch.tensor(it >= 2, device=dev))
    return st


def exact(case, seed):
    c = case
    if c["kind"] == "krylov":
        s = prepare(c, seed)
        q, w = s["q"].cpu().numpy(), s["w"].cpu().numpy()
        h = q @ w.T
        r = w - h.T @ q
        h2 = q @ r.T
        return {"h": h + h2, "w": r - h2.T @ q}
    if _points(c) * (c["steps"] if "steps" in c else 30) * (3 if c["les"] else 1) > 8e7:
        return None
    st = _initial(c, seed)
    dev = st["vor"].device
    if c["kind"] == "jv":
        re = torch.full((c["batch"],), c["rez"] / LZ ** 2, dtype=torch.float64, device=dev)
        flat = lambda b: torch.cat([torch.view_as_real(st["vor"][b]).reshape(-1),  # noqa: E731
                                    torch.view_as_real(st["phi"][b]).reshape(-1), st["u00"][b],
                                    st["w00"][b]])
        x = torch.stack([flat(b) for b in range(c["batch"])])
        x0 = x[0].clone()
        eps = 1e-4 * x0.norm() / x[1:].norm(dim=1)
        x[1:] = x0 + ((x0 + eps[:, None] * x[1:]) - x0)
        x[0] = x0
        B, shape = c["batch"], st["vor"].shape
        n = 2 * st["vor"][0].numel()
        cur = {"vor": torch.view_as_complex(x[:, :n].reshape(shape + (2,)).contiguous()).clone(),
               "phi": torch.view_as_complex(x[:, n:2 * n].reshape(shape + (2,)).contiguous()).clone(),
               "u00": x[:, 2 * n:2 * n + c["y"]].clone(), "w00": x[:, 2 * n + c["y"]:].clone(),
               "xofft": st["xofft"][:1].repeat(B)}
        cur = _step_exact(c, cur, re, etime=c["period"])
        out = torch.cat([torch.view_as_real(cur["vor"]).reshape(B, -1),
                         torch.view_as_real(cur["phi"]).reshape(B, -1), cur["u00"], cur["w00"]], 1)
        return ((out[1:] - out[:1]) / eps[:, None]).cpu().numpy()
    re = torch.tensor(_members_re(c), dtype=torch.float64, device=dev)
    st = _step_exact(c, st, re, steps=c["steps"])
    if c["kind"] == "cross":
        out = {k: st[k][0].cpu().numpy() for k in ("vor", "phi", "u00", "w00", "tb", "tb00")
               if k in st}
        out.update(time=float(st["time"][0]), xofft=float(st["xofft"][0]))
        return out
    return {"x": torch.stack([_pack(st["vor"][b], st["phi"][b], st["u00"][b], st["w00"][b])
                              for b in range(c["batch"])])}
