"""Performance cases of the 4D-Var inner loop: what a user's program calls
through the package's public entry points, over the range of sizes, types and
options it is used with.

Families (``kind``):

- ``qg``      the QG 1.5-layer model call of one assimilation sub-window:
              ``QG1LPlan.step`` (forward), ``step_tgl`` (tangent), ``step_adj``
              (adjoint, which recomputes its trajectory) and ``rev``, the
              reverse sweep of a stored trajectory (``advance_adj``, what the
              window engines run between two observation times);
- ``window``  one whole cost + gradient evaluation of a batch of windows whose
              control is the initial SSH (``QGWindows4DVar.cost_and_grad``,
              captured as users run it), float64;
- ``sw``      steps of the multilayer shallow-water model (``SWPlan.step``)
              and their adjoint;
- ``mgd``     the PV inversion of the masked multilayer QG model, one system
              per vertical mode (``MaskedDirichletMG.solve``);
- ``mg``      the masked multigrid Helmholtz solve (``MG_Helmholtz.solve``);
- ``basis``   the Gaussian reduced basis at one basis time: G X and G^T phi
              (``BasisPlan.project`` / ``project_T``).

``exact`` restates each of them in float64 with plain torch operations.

The upwind scheme's derivative jumps where a velocity changes sign, so the
pointwise float32 gradient with respect to an SSH field moves by some 1e-5
when a rounding anywhere upstream changes. The float32 reverse sweep is
therefore taken on a given trajectory, and the whole evaluation is float64.
"""
import math

import numpy as np
import torch

G, F0, C0, DT_QG = 9.81, 1.0e-4, 2.7, 900.0
BETA, KDIFF = 2.0e-11, 20.0
SW_H, SW_GP, SW_DX = (350.0, 750.0, 2900.0), (9.81, 0.025, 0.0125), 5.0e3
DEV = "cuda"
DTYPES = {"f32": torch.float32, "f64": torch.float64}


# --------------------------------------------------------------------------
# The cases
# --------------------------------------------------------------------------
def listed():
    return [
        # one small float64 window of 128^2: a test of a set-up, or one tile of
        # a regional run; launches and latency decide
        dict(name="qg_fwd_f64_128", kind="qg", op="step", ny=128, nx=128, batch=1, dtype="f64", scheme="rk2",
             nstep=6, coast=False),
        # the batched windows of the 512^2 benchmark between two observation
        # times, forward and adjoint
        dict(name="qg_fwd_512x16", kind="qg", op="step", ny=512, nx=512, batch=16, dtype="f32", scheme="rk2",
             nstep=4, coast=False),
        dict(name="qg_rev_512x16", kind="qg", op="rev", ny=512, nx=512, batch=16, dtype="f32", scheme="rk2",
             nstep=4, coast=False),
        # small windows of a mixed-size set, reverse sweep
        dict(name="qg_rev_192x12", kind="qg", op="rev", ny=192, nx=192, batch=12, dtype="f32", scheme="rk2",
             nstep=4, coast=False),
        # one large window (the reduced-basis configuration's grid)
        dict(name="qg_fwd_1024", kind="qg", op="step", ny=1024, nx=1024, batch=1, dtype="f32", scheme="rk2",
             nstep=6, coast=False),
        # a regional domain with a coast, beta plane, diffusion and boundary
        # SSH, of no round size; the tangent of an incremental scheme
        dict(name="qg_tgl_coast_287x410", kind="qg", op="tgl", ny=287, nx=410, batch=3, dtype="f32", scheme="rk3",
             nstep=3, coast=True),
        # one gradient of a small batch of mid-sized windows, in float64 as
        # the reference's own USE_FLOAT64 runs
        dict(name="window_f64_256x4", kind="window", ny=256, nx=256, batch=4, dtype="f64", nstep=8, nobs=2000),
        # three-layer shallow water with land, forward and adjoint
        dict(name="sw_fwd_3l_1024x768", kind="sw", op="step", nx=1024, ny=768, nl=3, dtype="f32", nstep=2),
        dict(name="sw_adj_3l_1024x768", kind="sw", op="adj", nx=1024, ny=768, nl=3, dtype="f32", nstep=2),
        # PV inversion of the masked three-layer QG model, one mode per system
        dict(name="mgd_3m_1023x767", kind="mgd", n0=1023, n1=767, modes=3),
        # masked multigrid Helmholtz solve (20 V-cycles)
        dict(name="mg_1024x768", kind="mg", nx=1024, ny=768),
        # reduced basis of nine components on the 1024^2 window
        dict(name="basis_9c_1024", kind="basis", n=1024, batch=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["qg", "qg", "qg", "qg", "window", "sw", "sw", "mgd", "mg", "basis"])
    if kind == "qg":
        dtype = rng.choice(["f32", "f32", "f64"])
        ny, nx = _log(rng, 64, 1024), _log(rng, 64, 1024)
        op = rng.choice(["step", "rev", "tgl"] + (["adj"] if dtype == "f64" else []))
        cells = 16 * 512 * 512 if dtype == "f32" else 4 * 256 * 256
        batch = _log(rng, 1, max(1, min(16, cells // (ny * nx))))
        return dict(kind="qg", op=op, ny=ny, nx=nx, batch=batch, dtype=dtype,
                    scheme=rng.choice(["rk2", "rk2", "rk3", "Euler"]), nstep=rng.randint(1, 3),
                    coast=rng.random() < 0.4)
    if kind == "window":
        ny, nx = _log(rng, 96, 384), _log(rng, 96, 384)
        return dict(kind="window", ny=ny, nx=nx, batch=_log(rng, 1, max(1, min(8, 4 * 256 * 256 // (ny * nx)))),
                    dtype="f64", nstep=rng.randint(3, 8), nobs=_log(rng, 200, 4000))
    if kind == "sw":
        return dict(kind="sw", op=rng.choice(["step", "adj"]), nx=_log(rng, 80, 1024), ny=_log(rng, 80, 768),
                    nl=rng.choice([1, 2, 3]), dtype="f32", nstep=rng.randint(1, 2))
    if kind == "mgd":
        a, b = rng.choice([8, 12, 16, 24, 32]), rng.choice([8, 10, 12, 16, 24])
        return dict(kind="mgd", n0=32 * a - 1, n1=32 * b - 1, modes=rng.choice([1, 2, 3]))
    if kind == "mg":
        return dict(kind="mg", nx=16 * rng.choice([8, 12, 16, 24, 32, 48, 64]),
                    ny=16 * rng.choice([8, 10, 14, 16, 24, 32, 48]))
    return dict(kind="basis", n=_log(rng, 192, 1024), batch=rng.choice([1, 1, 2]))


# --------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _ssh(batch, ny, nx, gen, dx=5.0e3, rms=0.1, cutoff=50.0e3):
    """Mesoscale SSH [m], float64 [batch, ny, nx]: k^-3 power, no power below
    the cutoff wavelength."""
    k1 = torch.fft.fftfreq(nx, d=dx, dtype=torch.float64, device=DEV)
    k0 = torch.fft.fftfreq(ny, d=dx, dtype=torch.float64, device=DEV)
    k = torch.sqrt(k1[None, :] ** 2 + k0[:, None] ** 2)
    amp = torch.where((k > 0) & (k <= 1.0 / cutoff), k.clamp_min(1e-30) ** -1.5, torch.zeros_like(k))
    s = torch.randn(2, batch, ny, nx, generator=gen, dtype=torch.float64, device=DEV)
    h = torch.fft.ifft2(amp * torch.complex(s[0], s[1])).real
    h = h - h.mean(dim=(1, 2), keepdim=True)
    return h * (rms / h.std(dim=(1, 2), keepdim=True).clamp_min(1e-12))


def _disks(n0, n1):
    """Two smooth islands, True on land."""
    i = np.arange(n0)[:, None] / n0
    j = np.arange(n1)[None, :] / n1
    return ((i - 0.42) ** 2 + (j - 0.38) ** 2 < 0.006) | ((i - 0.7) ** 2 + ((j - 0.68) * 1.5) ** 2 < 0.003)


def _blobs(n0, n1, frac=0.2):
    """Ocean mask with ``frac`` of land in smooth blobs (~50 km at 5 km)."""
    r = np.random.default_rng(5000)
    k0, k1 = np.fft.fftfreq(n0)[:, None], np.fft.rfftfreq(n1)[None, :]
    w = np.fft.irfft2(np.fft.rfft2(r.standard_normal((n0, n1))) * np.exp(-200 * np.pi ** 2 * (k0 ** 2 + k1 ** 2)),
                      s=(n0, n1))
    return (w <= np.quantile(w, 1 - frac)).astype(np.float64)


def _qg_inputs(case, seed):
    g = _gen(seed)
    ny, nx, b = case["ny"], case["nx"], case["batch"]
    h = _ssh(b, ny, nx, g)
    hb = _ssh(b, ny, nx, g, rms=0.02, cutoff=200.0e3) if case["coast"] else torch.zeros_like(h)
    w = _ssh(b, ny, nx, g, rms=1.0) if case["op"] == "adj" else _ssh(b, ny, nx, g, rms=0.01)
    if case["coast"]:
        sea = torch.as_tensor(~_disks(ny, nx), dtype=torch.float64, device=DEV)
        h, hb, w = h * sea, hb * sea, w * sea
    d = DTYPES[case["dtype"]]
    return h.to(d), hb.to(d), w.to(d)


def _beta(ny, nx):
    return np.full((ny, nx), BETA)


def _tracks(case, seed):
    """Observations on straight tracks: per window (idx [n, 4], weights [n, 4],
    step, noise-free target field's seed is the caller's), bilinear."""
    ny, nx = case["ny"], case["nx"]
    out = []
    for b in range(case["batch"]):
        r = np.random.default_rng(10007 * int(seed) + 31 * b + 5)
        x, y, st, n = [], [], [], 0
        while n < case["nobs"]:
            a, cx, cy = r.uniform(0, np.pi), r.uniform(0.25, 0.75) * nx, r.uniform(0.25, 0.75) * ny
            s = np.arange(-(nx + ny), nx + ny, 1.4)
            px, py = cx + s * np.cos(a), cy + s * np.sin(a)
            ok = (px > 3) & (px < nx - 5) & (py > 3) & (py < ny - 5)
            px, py = px[ok][:case["nobs"] - n], py[ok][:case["nobs"] - n]
            x.append(px)
            y.append(py)
            st.append(np.full(px.size, r.integers(1, case["nstep"] + 1)))
            n += px.size
        x, y, st = np.concatenate(x), np.concatenate(y), np.concatenate(st)
        i, j = np.floor(x).astype(np.int64), np.floor(y).astype(np.int64)
        fx, fy = x - i, y - j
        idx = np.stack([j * nx + i, j * nx + i + 1, (j + 1) * nx + i, (j + 1) * nx + i + 1], 1)
        w = np.stack([(1 - fx) * (1 - fy), fx * (1 - fy), (1 - fx) * fy, fx * fy], 1)
        out.append((idx, w, st, 0.03 * r.standard_normal(x.size)))
    return out


def _qg_traj(case, seed):
    """A stage trajectory [nstep*S + 1, 2, batch, ny, nx] of slowly turning
    eddies with their PV, and the adjoint (adh, adq) behind its end."""
    g = _gen(seed)
    ny, nx, b, d = case["ny"], case["nx"], case["batch"], DTYPES[case["dtype"]]
    slots = {"Euler": 1, "rk2": 2, "rk3": 3}[case["scheme"]] * case["nstep"] + 1
    m = _QG(ny, nx, case["scheme"], case["coast"])
    sea = (m.mask != 0).double()
    a, c = _ssh(b, ny, nx, g) * sea, _ssh(b, ny, nx, g) * sea
    t = torch.empty(slots, 2, b, ny, nx, dtype=d, device=DEV)
    for k in range(slots):
        h = math.cos(0.02 * k) * a + math.sin(0.02 * k) * c
        t[k, 0] = h
        t[k, 1] = m.h2pv(h, torch.zeros_like(h))
    adh = _ssh(b, ny, nx, g, rms=1.0) * sea
    adq = _ssh(b, ny, nx, g, rms=4.0e4) * (m.mask == 3).double()
    return t, adh.to(d), adq.to(d)


def _window_inputs(case, seed):
    g = _gen(seed)
    h0 = _ssh(case["batch"], case["ny"], case["nx"], g).to(DTYPES[case["dtype"]])
    truth = _ssh(case["batch"], case["ny"], case["nx"], g).cpu().numpy()
    tr = _tracks(case, seed)
    return h0, [(i, w, st, (truth[b].ravel()[i] * w).sum(1) + e) for b, (i, w, st, e) in enumerate(tr)]


def _sw_param(case):
    nx, ny, nl = case["nx"], case["ny"], case["nl"]
    H, gp = np.array(SW_H[:nl]), np.array(SW_GP[:nl])
    yw = np.arange(ny + 1)[None, :] * SW_DX + np.zeros((nx + 1, 1))
    f = 1.0e-4 + 1.6e-11 * (yw - yw.mean())
    cmax = math.sqrt(gp[0] * H.sum())
    dt = float(max(d for d in range(1, 3601) if 3600 % d == 0 and d <= 0.5 * SW_DX / cmax))
    return H, gp, f, dt, _blobs(nx, ny)


SW_OPT = dict(slip_coef=1.0, bottom_drag_coef=1e-7, visc_coef=50.0, diff_coef=20.0)


def _sw_inputs(case, seed):
    """Geostrophic eddies of every layer on the ocean faces, and the cotangent
    of the adjoint."""
    g = _gen(seed)
    nx, ny, nl = case["nx"], case["ny"], case["nl"]
    mask = torch.as_tensor(_blobs(nx, ny), device=DEV)
    psi = _ssh(nl, nx + 2, ny + 2, g, dx=SW_DX, rms=1.0, cutoff=60.0e3)
    amp = torch.tensor([0.08, 0.04, 0.02][:nl], dtype=torch.float64, device=DEV).view(nl, 1, 1) * (G / F0 / SW_DX)
    u = -(amp * (psi[:, :nx + 1, 1:ny + 1] - psi[:, :nx + 1, :ny]))
    v = amp * (psi[:, 1:nx + 1, :ny + 1] - psi[:, :nx, :ny + 1])
    h = psi[:, :nx, :ny] * torch.tensor([0.1, 8.0, 8.0][:nl], dtype=torch.float64, device=DEV).view(nl, 1, 1)
    mu = torch.zeros(nx + 1, ny, dtype=torch.float64, device=DEV)
    mv = torch.zeros(nx, ny + 1, dtype=torch.float64, device=DEV)
    mu[1:-1] = mask[1:] * mask[:-1]
    mv[:, 1:-1] = mask[:, 1:] * mask[:, :-1]
    x = [a[None].to(DTYPES[case["dtype"]]) for a in (u * mu, v * mv, h * mask)]
    w = [torch.randn(a.shape, generator=g, dtype=torch.float64, device=DEV).to(a.dtype) for a in x]
    return x, w


def _mgd_param(case):
    return np.array([0.0, 1.1e-9, 6.2e-9])[:case["modes"]], _blobs(case["n0"], case["n1"])


def _mgd_rhs(case, seed):
    b = _ssh(case["modes"], case["n0"], case["n1"], _gen(seed), rms=1.0e-9, cutoff=30.0e3)
    return b[:, None].contiguous()


def _mg_param(case):
    m = _blobs(case["nx"], case["ny"])
    mu, mv = np.zeros((case["nx"] + 1, case["ny"])), np.zeros((case["nx"], case["ny"] + 1))
    mu[1:-1], mv[:, 1:-1] = m[1:] * m[:-1], m[:, 1:] * m[:, :-1]
    return m, 4000.0 * mu, 4000.0 * mv, np.array([1.0 / (9.81 * 12.0 * 24.0)])


def _mg_rhs(case, seed):
    m = torch.as_tensor(_blobs(case["nx"], case["ny"]), device=DEV)
    return _ssh(1, case["nx"], case["ny"], _gen(seed), rms=1.0) * m


BASIS_COMPS = [(sd, st) for sd in (100.0, 200.0, 300.0) for st in (5.0, 10.0, 20.0)]
BASIS_FACNS, BASIS_DX = 0.85, 4.0
BASIS_TIME = np.arange(0.0, 30.25, 0.25)
BASIS_K = 40


def _basis_inputs(case, seed, nbasis):
    g = _gen(seed)
    X = torch.randn(case["batch"], nbasis, generator=g, dtype=torch.float64, device=DEV).float()
    phi = _ssh(case["batch"], case["n"], case["n"], g, dx=4.0e3).float()
    return X, phi


# --------------------------------------------------------------------------
# prepare / run
# --------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "qg":
        from vardyn_gb300.qg1l import QG1LPlan, build_mask
        ny, nx = case["ny"], case["nx"]
        kw = {}
        if case["coast"]:
            land = np.where(_disks(ny, nx), np.nan, 0.0)
            kw = dict(mask=build_mask(ny, nx, land), beta=_beta(ny, nx), Kdiffus=KDIFF)
        plan = QG1LPlan(ny, nx, 5.0e3, 5.0e3, DT_QG, F0, C0, time_scheme=case["scheme"],
                        dtype=DTYPES[case["dtype"]], **kw)
        if case["op"] == "rev":
            traj, adh, adq = _qg_traj(case, seed)
            return dict(case=case, plan=plan, traj=traj, start=(adh, adq), adh=adh.clone(), adq=adq.clone())
        h, hb, w = _qg_inputs(case, seed)
        return dict(case=case, plan=plan, h=h, hb=hb, w=w)
    if kind == "window":
        from vardyn_gb300.fourdvar import QGWindows4DVar
        from vardyn_gb300.obsop import AlongTrackObs
        from vardyn_gb300.qg1l import QG1LPlan
        ny, nx, d = case["ny"], case["nx"], DTYPES[case["dtype"]]
        h0, obs = _window_inputs(case, seed)
        plan = QG1LPlan(ny, nx, 5.0e3, 5.0e3, DT_QG, F0, C0, dtype=d)
        wins = [dict(step=st, yobs=y, err=np.full(y.size, 0.03)) for _, _, st, y in obs]
        ob = AlongTrackObs(wins, ny, nx, 5.0e3, 5.0e3, dtype=d, operator=[(i, w) for i, w, _, _ in obs])
        hb = torch.zeros(case["batch"], ny, nx, dtype=d, device=DEV)
        eng = QGWindows4DVar(plan, hb, case["nstep"], ob)
        eng.capture()
        return dict(case=case, eng=eng, h0=h0)
    if kind == "sw":
        from vardyn_gb300.sw import SWPlan
        H, gp, f, dt, mask = _sw_param(case)
        plan = SWPlan(case["nx"], case["ny"], case["nl"], SW_DX, SW_DX, f, H, gp, dt, mask=mask,
                      dtype=DTYPES[case["dtype"]], **SW_OPT)
        x, w = _sw_inputs(case, seed)
        return dict(case=case, plan=plan, x=x, w=w)
    if kind == "mgd":
        from vardyn_gb300.helmholtz_mg import MaskedDirichletMG
        lam, mask = _mgd_param(case)
        mg = MaskedDirichletMG(case["n0"], case["n1"], SW_DX, SW_DX, lam, mask=mask)
        return dict(case=case, mg=mg, b=_mgd_rhs(case, seed))
    if kind == "mg":
        from vardyn_gb300.helmholtz_mg import MG_Helmholtz
        m, cu, cv, lam = _mg_param(case)
        mg = MG_Helmholtz(SW_DX, SW_DX, case["nx"], case["ny"], cu, cv, lambd=lam, mask=m, niter_bottom=20)
        return dict(case=case, mg=mg, b=_mg_rhs(case, seed))
    from vardyn_gb300.basis import BasisPlan, Gauss3dParams
    xk = np.arange(case["n"]) * BASIS_DX
    comps = [Gauss3dParams(sd, st, facns=BASIS_FACNS, facnlt=st / 2.0, sigma_Q=0.01) for sd, st in BASIS_COMPS]
    plan = BasisPlan(xk, xk, BASIS_TIME, comps, dtype=torch.float32)
    X, phi = _basis_inputs(case, seed, plan.nbasis)
    return dict(case=case, plan=plan, X=X, phi=phi, adX=torch.zeros_like(X))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "qg":
        p, n = state["plan"], case["nstep"]
        if case["op"] == "step":
            return p.step(state["h"], state["hb"], nstep=n)
        if case["op"] == "tgl":
            return p.step_tgl(state["w"], state["h"], state["hb"], nstep=n)
        if case["op"] == "rev":
            adh, adq = state["adh"].copy_(state["start"][0]), state["adq"].copy_(state["start"][1])
            p.advance_adj(case["batch"], state["traj"], n, 0, n, adh, adq)
            return [adh, adq]
        return p.step_adj(state["w"], state["h"], state["hb"], nstep=n)
    if kind == "window":
        J, grad = state["eng"].cost_and_grad(state["h0"])
        return dict(J=J, grad=grad)
    if kind == "sw":
        if case["op"] == "step":
            return state["plan"].step(*state["x"], nstep=case["nstep"])
        r = state["plan"].step_adj(*state["x"], *state["w"], nstep=case["nstep"])
        return [r["u0"], r["v0"], r["h0"]]
    if kind in ("mgd", "mg"):
        return state["mg"].solve(state["b"])
    state["adX"].zero_()
    return [state["plan"].project(BASIS_K, state["X"]),
            state["plan"].project_T(BASIS_K, state["phi"], state["adX"])]


# --------------------------------------------------------------------------
# work: every input read once, every output written once, and the arithmetic
# of the path with O(n log n) transforms / optimal multigrid
# --------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("qg", "window"):
        es = 4 if case["dtype"] == "f32" else 8
        pts = case["batch"] * case["ny"] * case["nx"]
        stages = {"Euler": 1, "rk2": 2, "rk3": 3}[case.get("scheme", "rk2")]
        per = 60 + 2 * 2.5 * math.log2(2 * case["nx"]) * 2 + 8
        if kind != "qg":
            n = case["batch"] * case["nobs"]
            # a stored trajectory is written by the forward and read by the
            # reverse sweep: two fields a stage
            return dict(bytes=es * (2 * pts * (1 + 2 * stages * case["nstep"]) + 10.0 * n),
                        flops=3.0 * per * pts * stages * case["nstep"])
        f = {"step": 1, "tgl": 2, "adj": 3, "rev": 2}[case["op"]]
        io = {"step": 3, "tgl": 4, "adj": 4, "rev": 4}[case["op"]]
        traj = {"adj": 4, "rev": 2}.get(case["op"], 0) * stages * case["nstep"]
        return dict(bytes=float(es * pts * (io + traj)), flops=f * per * pts * stages * case["nstep"])
    if kind == "sw":
        es = 4 if case["dtype"] == "f32" else 8
        pts = 3 * case["nl"] * case["nx"] * case["ny"]
        f, io = (1, 2) if case["op"] == "step" else (4, 3)
        return dict(bytes=float(es * pts * io), flops=f * 180.0 * pts * 3 * case["nstep"])
    if kind == "mgd":
        pts = case["modes"] * case["n0"] * case["n1"]
        return dict(bytes=16.0 * pts, flops=12 * 90.0 * pts)
    if kind == "mg":
        pts = case["nx"] * case["ny"]
        return dict(bytes=16.0 * pts + 24.0 * pts, flops=21 * 160.0 * pts)
    n = case["n"]
    rows = sum((n * BASIS_DX * BASIS_FACNS / sd + 4) for sd, _ in BASIS_COMPS)
    act = sum((n * BASIS_DX * BASIS_FACNS / sd + 4) ** 2 * st for sd, st in BASIS_COMPS)
    b = case["batch"]
    return dict(bytes=4.0 * b * (2 * n * n + 2 * act), flops=b * (2 * 9 * 2 * 3.4 * n * n + 4 * rows * n * 8))


# --------------------------------------------------------------------------
# exact: the same in float64 with plain torch
# --------------------------------------------------------------------------
def _t(a):
    return torch.as_tensor(np.asarray(a), dtype=torch.float64, device=DEV)


def _qg_mask(ny, nx, coast):
    m = np.full((ny, nx), 3)
    m[0] = m[-1] = 1
    m[:, 0] = m[:, -1] = 1
    m[1, 1:-1] = m[-2, 1:-1] = m[-3, 1:-1] = 2
    m[1:-1, 1] = m[1:-1, -2] = m[1:-1, -3] = 2
    if coast:
        land = _disks(ny, nx)

        def grow(r):
            p = np.pad(land, r)
            return np.any([p[a:a + ny, c:c + nx] for a in range(2 * r + 1) for c in range(2 * r + 1)], axis=0)
        new = m.copy()
        new[grow(2) & (m == 3)] = 2
        new[grow(1) & (m >= 2)] = 1
        new[land] = 0
        m = new
    return torch.as_tensor(m, device=DEV)


class _QG:
    """The QG 1.5-layer model on [batch, ny, nx] float64 tensors."""

    def __init__(self, ny, nx, scheme, coast):
        self.scheme, self.coast, self.dx = scheme, coast, 5.0e3
        self.mask = _qg_mask(ny, nx, coast)
        n, m = nx - 2, ny - 2

        def sines(n):
            k = torch.arange(1, n + 1, dtype=torch.int64, device=DEV)
            a = (k[:, None] * k[None, :]) % (2 * (n + 1))
            return math.sqrt(2.0 / (n + 1)) * torch.sin(math.pi * a.double() / (n + 1))
        self.Sx, self.Sy = sines(n), sines(m)
        kx, ky = _t(np.arange(1, n + 1)), _t(np.arange(1, m + 1))
        lap = 2 * (torch.cos(math.pi / (n + 1) * kx) - 1)[None, :] / self.dx ** 2 + \
            2 * (torch.cos(math.pi / (m + 1) * ky) - 1)[:, None] / self.dx ** 2
        self.eig = G / F0 * lap - G * F0 / C0 ** 2

    def h2pv(self, h, hb):
        d2 = self.dx ** 2
        c = h[:, 1:-1, 1:-1]
        inner = G / F0 * ((h[:, 2:, 1:-1] + h[:, :-2, 1:-1] - 2 * c) / d2 +
                          (h[:, 1:-1, 2:] + h[:, 1:-1, :-2] - 2 * c) / d2) - G * F0 / C0 ** 2 * c
        q = torch.nn.functional.pad(inner, (1, 1, 1, 1))
        edge = (self.mask == 1) | (self.mask == 2)
        q = torch.where(edge, -G * F0 / C0 ** 2 * hb, q)
        return torch.where(self.mask == 0, torch.zeros_like(q), q)

    def pv2h(self, q, hb, qb):
        r = (q - qb)[:, 1:-1, 1:-1]
        r = self.Sy @ ((self.Sy @ r @ self.Sx) / self.eig) @ self.Sx
        return torch.nn.functional.pad(r, (1, 1, 1, 1)) + hb

    def tend(self, h, q):
        dx = self.dx
        pad = torch.nn.functional.pad
        u = pad(-G / F0 * (h[:, 2:, :-1] + h[:, 2:, 1:] - h[:, :-2, 1:] - h[:, :-2, :-1]) / (4 * dx), (1, 0, 1, 1))
        v = pad(G / F0 * (h[:, 1:, 2:] + h[:, :-1, 2:] - h[:, :-1, :-2] - h[:, 1:, :-2]) / (4 * dx), (1, 1, 1, 0))
        uT = 0.5 * (u[:, 2:-2, 2:-2] + u[:, 2:-2, 3:-1])
        vT = 0.5 * (v[:, 2:-2, 2:-2] + v[:, 3:-1, 2:-2])
        z = torch.zeros_like(uT)
        up, um = torch.where(uT < 0, z, uT), torch.where(uT > 0, z, uT)
        vp, vm = torch.where(vT < 0, z, vT), torch.where(vT > 0, z, vT)
        c = q[:, 2:-2, 2:-2]
        e = 1.0 / (6 * dx)
        r = (-up * e * (2 * q[:, 2:-2, 3:-1] + 3 * c - 6 * q[:, 2:-2, 1:-3] + q[:, 2:-2, :-4])
             + um * e * (q[:, 2:-2, 4:] - 6 * q[:, 2:-2, 3:-1] + 3 * c + 2 * q[:, 2:-2, 1:-3])
             - vp * e * (2 * q[:, 3:-1, 2:-2] + 3 * c - 6 * q[:, 1:-3, 2:-2] + q[:, :-4, 2:-2])
             + vm * e * (q[:, 4:, 2:-2] - 6 * q[:, 3:-1, 2:-2] + 3 * c + 2 * q[:, 1:-3, 2:-2]))
        if self.coast:
            r = r - BETA * (v[:, 2:-2, 2:-2] + v[:, 3:-1, 2:-2]) / 2 + KDIFF / dx ** 2 * (
                q[:, 2:-2, 3:-1] + q[:, 2:-2, 1:-3] + q[:, 3:-1, 2:-2] + q[:, 1:-3, 2:-2] - 4 * c)
        return torch.where(self.mask == 3, pad(r, (2, 2, 2, 2)), torch.zeros_like(q))

    def one_step(self, h, q, hb, qb):
        dt = DT_QG
        k1 = self.tend(h, q)
        if self.scheme == "Euler":
            q1 = q + dt * k1
        elif self.scheme == "rk2":
            qa = q + 0.5 * dt * k1
            q1 = q + dt * self.tend(self.pv2h(qa, hb, qb), qa)
        else:
            qa = q + 0.5 * dt * k1
            k2 = self.tend(self.pv2h(qa, hb, qb), qa)
            qc = q - dt * k1 + 2 * dt * k2
            k3 = self.tend(self.pv2h(qc, hb, qb), qc)
            q1 = q + dt / 6 * (k1 + 4 * k2 + k3)
        return self.pv2h(q1, hb, qb), q1

    def step(self, h, hb, nstep):
        q, qb = self.h2pv(h, hb), self.h2pv(hb, hb)
        for _ in range(nstep):
            h, q = self.one_step(h, q, hb, qb)
        return h


def _exact_rev(case, seed):
    """The reverse sweep over the trajectory's stages, each stage's tendency
    transposed at the given (h, q); PV moves on the tendency points only."""
    traj, adh, adq = (a.double() for a in _qg_traj(case, seed))
    m = _QG(case["ny"], case["nx"], case["scheme"], case["coast"])
    dt, on, z = DT_QG, (m.mask == 3).double(), torch.zeros_like(adh)
    A, b = {"Euler": ([[]], [dt]), "rk2": ([[], [0.5 * dt]], [0.0, dt]),
            "rk3": ([[], [0.5 * dt], [-dt, 2 * dt]], [dt / 6, 4 * dt / 6, dt / 6])}[case["scheme"]]
    S = len(b)
    for n in reversed(range(case["nstep"])):
        Gs = [on * (m.pv2h(adh, z, z) + adq)] + [None] * (S - 1)
        for s in reversed(range(S)):
            h, q = (x.clone().requires_grad_(True) for x in traj[n * S + s])
            g = b[s] * Gs[0] + sum(A[t][s] * Gs[t] for t in range(s + 1, S))
            ah, aq = torch.autograd.grad((m.tend(h, q) * g).sum(), (h, q))
            if s:
                Gs[s] = on * (m.pv2h(ah, z, z) + aq)
        adh, adq = ah, on * (aq + sum(Gs))
    return [adh, adq]


def _exact_qg(case, seed):
    if case["op"] == "rev":
        return _exact_rev(case, seed)
    h, hb, w = (a.double() for a in _qg_inputs(case, seed))
    m = _QG(case["ny"], case["nx"], case["scheme"], case["coast"])
    sea = m.mask != 0
    if case["op"] == "step":
        out = m.step(h, hb, case["nstep"])
        return torch.where(sea, out, torch.full_like(out, float("nan")))
    f = lambda x: torch.where(sea, m.step(x, hb, case["nstep"]), torch.zeros_like(x))  # noqa: E731
    if case["op"] == "tgl":
        return torch.func.jvp(f, (h,), (w,))[1]
    h.requires_grad_(True)
    return torch.autograd.grad((f(h) * w).sum(), h)[0]


def _exact_window(case, seed):
    h0, obs = _window_inputs(case, seed)
    h0 = h0.double().requires_grad_(True)
    m = _QG(case["ny"], case["nx"], "rk2", False)
    hb = torch.zeros_like(h0)
    J = [0.0] * case["batch"]
    at = [[(torch.as_tensor(i[st == s], device=DEV), _t(w[st == s]), _t(y[st == s])) for i, w, st, y in obs]
          for s in range(case["nstep"] + 1)]
    h, q = h0, m.h2pv(h0, hb)
    qb = torch.zeros_like(q)
    for s in range(1, case["nstep"] + 1):
        h, q = m.one_step(h, q, hb, qb)
        for b, (i, w, y) in enumerate(at[s]):
            if y.numel():
                r = ((h[b].reshape(-1)[i] * w).sum(1) - y) / 0.03
                J[b] = J[b] + 0.5 * (r * r).sum()
    J = torch.stack([torch.as_tensor(j, dtype=torch.float64, device=DEV) for j in J])
    grad = torch.autograd.grad(J.sum(), h0)[0]
    return dict(J=J.detach(), grad=grad)


def _gauss(case_x, comps, facns, facnlt, times, k):
    """(offset, W_x, W_y, time weights) of every component at times[k];
    case_x = (x, y) coordinates in km."""
    win = lambda s: np.cos(0.5 * np.pi * s) ** 2  # noqa: E731
    parts, nb = [], 0
    for sd, st in comps:
        W, nl = [], facnlt(st)
        for x in case_x:
            d = sd / facns
            c = np.arange(x[0] - x[0] % d - sd * (1 - 1 / facns), x[-1] + 1.5 * d, d)
            e = x[:, None] - c[None, :]
            W.append(_t(np.where(np.abs(e) <= sd, win(e / sd), 0.0)))
        tc = np.arange(-st * (1 - 1 / nl), times[-1] - times[0] + 1.5 * st / nl, st / nl)
        tt = np.linspace(-st, st)
        norm = np.cumsum(win(tt[:-1] / st) * np.diff(tt)).max()
        wt = np.where(np.abs(times[k] - tc) < st, win((times[k] - tc) / st), 0.0) / norm
        parts.append((nb, W[0], W[1], _t(wt)))
        nb += tc.size * W[0].shape[1] * W[1].shape[1]
    return parts, nb


def _gauss_G(parts, X):
    """[batch, ny, nx] projection of X [batch, nbasis]."""
    out = 0.0
    for o, Wx, Wy, wt in parts:
        n = wt.numel() * Wy.shape[1] * Wx.shape[1]
        out = out + Wy @ torch.einsum("t,btyx->byx", wt, X[:, o:o + n].reshape(
            X.shape[0], wt.numel(), Wy.shape[1], Wx.shape[1])) @ Wx.T
    return out


def _pool(x, k0, k1, p0, p1):
    x = np.pad(x, ((p0, p0), (p1, p1)))
    n0, n1 = x.shape[0] - k0 + 1, x.shape[1] - k1 + 1
    return sum(x[a:a + n0, b:b + n1] for a in range(k0) for b in range(k1))


class _SW:
    """The shallow-water model of the ``sw`` cases on [nl, ...] tensors."""

    def __init__(self, case):
        H, gp, f, self.dt, h = _sw_param(case)
        self.nl, self.gp = case["nl"], _t(gp).view(-1, 1, 1)
        u, v = _pool(h, 2, 1, 1, 0) == 2, _pool(h, 1, 2, 0, 1) == 2
        w4 = _pool(h, 2, 2, 1, 1)
        w = (w4 >= 1).astype(float)
        nv, nu = _pool(v.astype(float), 2, 1, 1, 0) == 1, _pool(u.astype(float), 1, 2, 0, 1) == 1
        self.valid = _t((w > 0) & ~nv & ~nu)          # slip 1: the coastal classes carry no vorticity

        def sten(e2, e4, e6, on, full=False):
            """2-, 4- and 6-point selectors of window sums e2, e4, e6."""
            eq2 = (e2 == 2) & (e4 < 4) & on
            gt4 = ~eq2 & on
            eq4 = (e6 < 6) & gt4
            return [_t(a) for a in (eq2, eq4, gt4 if full else ~eq4 & gt4)]
        self.u_hx = sten(_pool(h, 2, 1, 1, 0), _pool(h, 4, 1, 2, 0), _pool(h, 6, 1, 3, 0), u)
        self.v_hy = sten(_pool(h, 1, 2, 0, 1), _pool(h, 1, 4, 0, 2), _pool(h, 1, 6, 0, 3), v)
        self.u_wy = sten(_pool(w, 1, 2, 0, 0), _pool(w, 1, 4, 0, 1), _pool(w, 1, 6, 0, 2), u, full=True)
        self.v_wx = sten(_pool(w, 2, 1, 0, 0), _pool(w, 4, 1, 1, 0), _pool(w, 6, 1, 2, 0), v)
        self.h, self.u, self.v = _t(h), _t(u), _t(v)
        self.dx, self.area = SW_DX, SW_DX ** 2
        f = _t(f)
        self.fu, self.fv = 0.5 * (f[:, 1:] + f[:, :-1]) * self.area, 0.5 * (f[1:] + f[:-1]) * self.area
        self.href = _t(H).view(-1, 1, 1) * self.area

    @staticmethod
    def _w4(a, b, c, d):
        e = 1e-4
        b1, b2 = (b - a) ** 2, (c - b) ** 2
        t = torch.sqrt((b2 - b1) ** 2 + e * e)
        w1, w2 = (1 / 3) * (1 + t / (b1 + e)), (2 / 3) * (1 + t / (b2 + e))
        return (w1 * (1.5 * b - 0.5 * a) + w2 * 0.5 * (b + c)) / (w1 + w2)

    @staticmethod
    def _w6(a, b, c, d, g, _):
        e = 1e-4
        b1 = 13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2
        b2 = 13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2
        b3 = 13 / 12 * (c - 2 * d + g) ** 2 + 0.25 * (3 * c - 4 * d + g) ** 2
        t = torch.sqrt((b1 - b3) ** 2 + e * e)
        w1, w2, w3 = 0.1 * (1 + t / (b1 + e)), 0.6 * (1 + t / (b2 + e)), 0.3 * (1 + t / (b3 + e))
        return (w1 * (a / 3 - 7 / 6 * b + 11 / 6 * c) + w2 * (-b / 6 + 5 / 6 * c + d / 3) +
                w3 * (c / 3 + 5 / 6 * d - g / 6)) / (w1 + w2 + w3)

    def flux(self, q, vel, axis, sel):
        if axis == 0:
            return self.flux(q.transpose(-1, -2), vel.transpose(-1, -2), 1,
                             [s.transpose(-1, -2) for s in sel]).transpose(-1, -2)
        n, pad = q.shape[-1], torch.nn.functional.pad
        m2, m4, m6 = sel
        p2 = 0.5 * (q[..., :-1] + q[..., 1:])
        t = [q[..., k:n - 3 + k] for k in range(4)]
        s = [q[..., k:n - 5 + k] for k in range(6)]
        p4, n4 = pad(self._w4(*t), (1, 1)), pad(self._w4(*t[::-1]), (1, 1))
        p6, n6 = pad(self._w6(*s), (2, 2)), pad(self._w6(*s[::-1]), (2, 2))
        up = torch.maximum(vel, torch.zeros_like(vel))
        return up * (m2 * p2 + m4 * p4 + m6 * p6) + (vel - up) * (m2 * p2 + m4 * n4 + m6 * n6)

    def rhs(self, u, v, h):
        pad, dx, a = torch.nn.functional.pad, self.dx, self.area
        curl = torch.diff(pad(v, (0, 0, 1, 1)), dim=-2) - torch.diff(pad(u, (1, 1)), dim=-1)
        om = self.valid * curl
        eta = torch.flip(torch.cumsum(torch.flip(h / a, (0,)), 0), (0,))
        p = torch.cumsum(self.gp * eta, 0)
        U, V = u / a, v / a
        ip = lambda x: 0.25 * (x[:, 1:, 1:] + x[:, 1:, :-1] + x[:, :-1, 1:] + x[:, :-1, :-1])  # noqa: E731
        Um, Vm = ip(U), ip(V)
        us, vs = u * U, v * V
        ke = 0.25 * (us[:, 1:] + us[:, :-1] + vs[..., 1:] + vs[..., :-1]) * self.h
        hm = 0.1 * a
        ht = hm + torch.logaddexp((self.href + h - hm) * 10.0, torch.zeros_like(h)) / 10.0
        fy = self.flux(ht, V[..., 1:-1], 1, [s[:, 1:-1] for s in self.v_hy])
        fx = self.flux(ht, U[:, 1:-1], 0, [s[1:-1] for s in self.u_hx])
        dh = -(pad(torch.diff(fx, dim=-2), (0, 0, 1, 1)) + pad(torch.diff(fy, dim=-1), (1, 1))) * self.h

        def rep(x, p):
            return torch.nn.functional.pad(x[None], p, mode="replicate")[0]

        def lap(x):
            return (x[:, 2:, 1:-1] + x[:, :-2, 1:-1] + x[:, 1:-1, 2:] + x[:, 1:-1, :-2] - 4 * x[:, 1:-1, 1:-1]) / a
        dh = dh + SW_OPT["diff_coef"] * lap(rep(h / a, (1, 1, 1, 1))) * a * self.h
        du = self.flux(om[:, 1:-1], Vm, 1, [s[1:-1] for s in self.u_wy]) + self.fu[1:-1] * Vm
        dv = -(self.flux(om[..., 1:-1], Um, 0, [s[:, 1:-1] for s in self.v_wx]) + self.fv[:, 1:-1] * Um)
        kp = ke + p
        du, dv = du - torch.diff(kp, dim=-2), dv - torch.diff(kp, dim=-1)
        low = torch.zeros(self.nl, 1, 1, dtype=torch.float64, device=DEV)
        low[-1] = SW_OPT["bottom_drag_coef"]
        du, dv = du - low * u[:, 1:-1], dv - low * v[..., 1:-1]
        du = du + SW_OPT["visc_coef"] * lap(rep(u, (1, 1, 0, 0)) / dx) * dx
        dv = dv + SW_OPT["visc_coef"] * lap(rep(v, (0, 0, 1, 1)) / dx) * dx
        return pad(du, (0, 0, 1, 1)) * self.u, pad(dv, (1, 1)) * self.v, dh

    def step(self, u, v, h, nstep):
        x = (u * self.u * self.dx, v * self.v * self.dx, h * self.h * self.area)
        dt = self.dt
        for _ in range(nstep):
            k0 = self.rhs(*x)
            x = [a + dt * k for a, k in zip(x, k0)]
            k1 = self.rhs(*x)
            x = [a + dt / 4 * (p - 3 * k) for a, p, k in zip(x, k1, k0)]
            k2 = self.rhs(*x)
            x = [a + dt / 12 * (8 * r - p - k) for a, r, p, k in zip(x, k2, k1, k0)]
        return x[0] / self.dx, x[1] / self.dx, x[2] / self.area


def _exact_sw(case, seed):
    x, w = _sw_inputs(case, seed)
    x = [a[0].double() for a in x]
    m = _SW(case)
    if case["op"] == "step":
        return [a[None] for a in m.step(*x, case["nstep"])]
    for a in x:
        a.requires_grad_(True)
    y = m.step(*x, case["nstep"])
    return [a[None] for a in torch.autograd.grad(sum((a * b[0].double()).sum() for a, b in zip(y, w)), x)]


def _cg(A, b, diag, tol=1e-14, most=30000):
    """Diagonally preconditioned conjugate gradients of the SPD operator A."""
    x, r = torch.zeros_like(b), b.clone()
    z = r / diag
    p, rho, b2 = z.clone(), (r * z).sum(), float((b * b).sum())
    for it in range(most):
        q = A(p)
        al = rho / (p * q).sum()
        x += al * p
        r -= al * q
        if it % 100 == 99 and float((r * r).sum()) <= tol * tol * b2:
            break
        z = r / diag
        new = (r * z).sum()
        p = z + (new / rho) * p
        rho = new
    return x


def _exact_mgd(case, seed):
    lam, mask = _mgd_param(case)
    m, c = _t(mask), 1.0 / SW_DX ** 2
    b = _mgd_rhs(case, seed)
    out = []
    for k, lm in enumerate(lam):
        def A(x, lm=float(lm)):
            p = torch.nn.functional.pad(x, (1, 1, 1, 1))
            return m * ((4 * c + lm) * x - c * (p[2:, 1:-1] + p[:-2, 1:-1] + p[1:-1, 2:] + p[1:-1, :-2]))
        out.append(-_cg(A, b[k, 0] * m, 4 * c + float(lm)))
    return torch.stack(out)[:, None]


def _exact_mg(case, seed):
    mask, cu, cv, lam = (_t(a) for a in _mg_param(case))
    c = 1.0 / SW_DX ** 2
    diag = lam[0] + c * (cu[1:] + cu[:-1] + cv[:, 1:] + cv[:, :-1])

    def A(x):
        p = torch.nn.functional.pad(x, (1, 1, 1, 1))
        return mask * (diag * x - c * (cu[1:] * p[2:, 1:-1] + cu[:-1] * p[:-2, 1:-1] +
                                       cv[:, 1:] * p[1:-1, 2:] + cv[:, :-1] * p[1:-1, :-2]))
    return -_cg(A, _mg_rhs(case, seed)[0], diag)[None]


def _exact_basis(case, seed):
    x = np.arange(case["n"]) * BASIS_DX
    parts, nb = _gauss((x, x), BASIS_COMPS, BASIS_FACNS, lambda st: st / 2.0, BASIS_TIME, BASIS_K)
    X, phi = (a.double() for a in _basis_inputs(case, seed, nb))
    ad = torch.zeros_like(X)
    for o, Wx, Wy, wt in parts:
        g = torch.einsum("t,byx->btyx", wt, Wy.T @ phi @ Wx).reshape(X.shape[0], -1)
        ad[:, o:o + g.shape[1]] = g
    return [_gauss_G(parts, X), ad]


def exact(case, seed):
    return {"qg": _exact_qg, "window": _exact_window, "sw": _exact_sw, "mgd": _exact_mgd,
            "mg": _exact_mg, "basis": _exact_basis}[case["kind"]](case, seed)
