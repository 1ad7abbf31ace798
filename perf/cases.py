"""The work that users of this framework have it do, as cases that can be timed and checked.

A case names a kind of call and its sizes.  prepare() makes what a program has in hand before the
call (bands, fields, a propagator handle, states on the GPU), run() makes the call through the public
classes, and exact() computes the same outputs in plain float64 torch from the same inputs: dense
matrices in a basis orthonormal in the spline overlap, none of the package's code.

Kinds: "step" one propagate call; "run" the driver loop; "dipole" the loop with the per-step dipole;
"mask" the loop with the absorbing mask after every step; "arnoldi" the Krylov propagator; "vgwr" the
elliptical velocity gauge; "pcs" momentum amplitudes of final states; "mlp_grad" and "mlp_predict"
the surrogate network.
"""
import importlib
import math

import numpy as np
import torch

q = importlib.import_module("qpc-tdse-cpc_gb300")

DT = 0.05
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def listed():
    return [
        # one step of one small wavefunction between two host-side decisions: launches and latency
        {"name": "step_small", "kind": "step", "n_r": 96, "p": 5, "n_l": 9, "n_inst": 1, "steps": 1},
        # a single pulse on the small hydrogen grid (400 splines, l <= 20), a window of its loop
        {"name": "run_single", "kind": "run", "n_r": 400, "p": 6, "n_l": 21, "n_inst": 1, "steps": 120},
        # the harmonic spectrum of one pulse on the scan's grid: the per-step dipole is recorded
        {"name": "dipole_single", "kind": "dipole", "n_r": 800, "p": 6, "n_l": 41, "n_inst": 1, "steps": 60},
        # a few pulses of different lengths with field-free tails, other degree and odd sizes
        {"name": "run_uneven", "kind": "run", "n_r": 517, "p": 5, "n_l": 30, "n_inst": 24, "steps": 30},
        # the batched laser scan: 256 pulses on 800 splines, l <= 40
        {"name": "run_scan", "kind": "run", "n_r": 800, "p": 6, "n_l": 41, "n_inst": 256, "steps": 12},
        # spectra labels for the surrogate: a batch with the dipole recorded in the loop
        {"name": "dipole_batch", "kind": "dipole", "n_r": 800, "p": 6, "n_l": 41, "n_inst": 48, "steps": 20},
        # a pulse train with an absorber at the end of the box, the mask applied after every step
        {"name": "mask_batch", "kind": "mask", "n_r": 640, "p": 7, "n_l": 25, "n_inst": 8, "steps": 20},
        # model atoms: one screened potential per wavefunction on one grid
        {"name": "run_potentials", "kind": "run", "n_r": 400, "p": 6, "n_l": 21, "n_inst": 4, "steps": 40, "potentials": True},
        # the Krylov propagator at its usual dimension, one screened potential per wavefunction
        {"name": "arnoldi_batch", "kind": "arnoldi", "n_r": 400, "p": 6, "n_l": 21, "n_inst": 8, "steps": 2, "kmax": 12},
        # an elliptical pulse in the velocity gauge (l <= 12 for |m| <= 12)
        {"name": "vgwr_elliptical", "kind": "vgwr", "n_r": 400, "p": 6, "n_l": 13, "n_m": 25, "n_inst": 2, "steps": 4},
        # momentum amplitudes of a batch of final states on a (|k|, theta) grid
        {"name": "pcs_batch", "kind": "pcs", "n_r": 800, "p": 6, "n_l": 41, "n_inst": 64, "nkr": 250, "nkt": 91},
        # one gradient of the surrogate ensemble on a minibatch
        {"name": "mlp_grad", "kind": "mlp_grad", "rows": 256, "hidden": 256, "layers": 4, "members": 5},
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["step", "run", "run", "run", "dipole", "dipole", "mask", "potentials", "arnoldi", "vgwr", "pcs", "mlp_grad", "mlp_predict"])
    if kind in ("mlp_grad", "mlp_predict"):
        return {"kind": kind, "rows": log(32, 2048), "hidden": 16 * rng.randint(6, 20), "layers": rng.randint(2, 5), "members": rng.randint(1, 6)}
    c = {"kind": "run" if kind == "potentials" else kind, "n_r": log(90, 800), "p": rng.randint(4, 7), "n_l": rng.randint(5, 41)}
    if kind == "vgwr":
        m = rng.randint(2, 9)
        return dict(c, n_r=log(90, 500), n_l=rng.randint(3, 11), n_m=2 * m + 1, n_inst=rng.randint(1, 3), steps=rng.randint(1, 4))
    if kind == "arnoldi":
        return dict(c, n_r=log(90, 400), n_l=rng.randint(5, 24), n_inst=log(1, 8), steps=rng.randint(1, 2), kmax=rng.randint(6, 12))
    if kind == "pcs":
        return dict(c, n_inst=log(1, 64), nkr=log(40, 250), nkt=rng.randint(1, 91))
    if kind == "step":
        return dict(c, n_inst=log(1, 64), steps=1)
    if kind == "mask":
        return dict(c, n_r=log(90, 640), n_inst=log(1, 12), steps=rng.randint(4, 20))
    if kind == "potentials":
        return dict(c, n_r=log(90, 400), n_l=rng.randint(5, 21), n_inst=rng.randint(1, 4), steps=rng.randint(10, 40), potentials=True)
    n_inst = log(1, 256) if kind == "run" else log(1, 48)
    return dict(c, n_inst=n_inst, steps=max(4, min(120, 1200 // (n_inst + 8))))


# ------------------------------------------------------------------ inputs

def knots(case):
    """uniform breakpoints 0.5 a.u. apart, the end points repeated"""
    n, p = case["n_r"], case["p"]
    rmax = 0.5 * n
    return np.concatenate([np.zeros(p), np.linspace(0.0, rmax, n - p + 3), np.full(p, rmax)])


def bands(case, zs=0.0, sigma=1.0, mask=None):
    """Upper bands [n_r][p+1] of <B|B>, <B|r|B>, <B|1/r|B>, <B|d/dr|B>, <B|1/r^2|B>, of the kinetic plus
    potential energy for V = -(1 + zs e^(-sigma r))/r, and of <B|mask(r)|B>: Gauss-Legendre on every interval
    over the splines that vanish at both ends."""
    n, p, t = case["n_r"], case["p"], knots(case)
    x, w = np.polynomial.legendre.leggauss(2 * p + 2)
    a, b = t[p:-p - 1], t[p + 1:-p]
    r = (0.5 * (a + b)[:, None] + 0.5 * (b - a)[:, None] * x).reshape(-1)
    wt = (0.5 * (b - a)[:, None] * w).reshape(-1)
    iv = np.repeat(np.arange(a.size) + p, x.size)
    B = np.zeros((r.size, p + 1))
    B[:, 0] = 1.0
    dB = None
    for k in range(1, p + 1):       # Cox-de Boor: B[:, j] is spline iv - k + j of degree k
        if k == p:
            low = B.copy()
        C = np.zeros_like(B)
        for j in range(k):
            tl, tr = t[iv - k + 1 + j], t[iv + 1 + j]
            f = B[:, j] / (tr - tl)
            C[:, j] += f * (tr - r)
            C[:, j + 1] += f * (r - tl)
        B = C
    dB = np.zeros_like(B)
    for j in range(p):
        f = p * low[:, j] / (t[iv + 1 + j] - t[iv - p + 1 + j])
        dB[:, j] -= f
        dB[:, j + 1] += f
    first = iv - p - 1              # the first active spline of a point's interval (spline 0 is left out)

    def form(f, left, right):
        out = np.zeros((n, p + 1))
        for j in range(p + 1):
            for k in range(j, p + 1):
                i = first + j
                ok = (i >= 0) & (first + k < n)
                np.add.at(out, (i[ok], np.full(ok.sum(), k - j)), (wt * f * left[:, j] * right[:, k])[ok])
        return out

    one = np.ones_like(r)
    out = {"S": form(one, B, B), "R": form(r, B, B), "I": form(1 / r, B, B), "D": form(one, B, dB), "C": form(1 / r ** 2, B, B),
           "H": form(-(1.0 + zs * np.exp(-sigma * r)) / r, B, B) + 0.5 * form(one, dB, dB)}
    if mask is not None:
        m = np.where(r < mask, 1.0, np.abs(np.cos(0.5 * np.pi * (r - mask) / (t[-1] - mask))) ** (1.0 / 6.0))
        out["M"] = form(m, B, B)
    return out


def hamiltonian(b, lmax):
    ll = np.arange(lmax + 1.0)
    return b["H"] + 0.5 * (ll * (ll + 1))[:, None, None] * b["C"]


def packets(case, seed, n_m=1):
    """c[inst][m][l][r]: every channel a few wave packets of smooth radial shape whose weight falls with l, as
    a pulse leaves a state: most of it near the nucleus, some of it on its way out."""
    g = torch.Generator(device=DEV).manual_seed(1000 + seed)
    B, L, N = case["n_inst"], case["n_l"], case["n_r"]
    r = torch.arange(1, N + 1, device=DEV, dtype=torch.float64) * 0.5

    def u(a, b):
        return a + (b - a) * torch.rand((B, n_m, L, 1), generator=g, device=DEV, dtype=torch.float64)

    c = torch.zeros((B, n_m, L, N), device=DEV, dtype=torch.complex128)
    l = torch.arange(L, device=DEV, dtype=torch.float64)[:, None]
    for weight, lo, hi in ((1.0, 0.0, 0.05), (0.2, 0.05, 0.3), (0.05, 0.2, 0.7)):
        env = weight * torch.exp(-((r - u(lo, hi) * r[-1]) / u(2.0, 12.0)) ** 2) * torch.exp(-0.15 * l)
        ph = u(-1.2, 1.2) * r + u(0.0, 6.28)
        c += torch.complex(env * torch.cos(ph), env * torch.sin(ph))
    c *= (r / (1.0 + r)) ** torch.clamp(l + 1, max=8.0)
    return c / torch.sqrt((c.abs() ** 2).sum(dim=(1, 2, 3), keepdim=True))


def pulses(case, seed, steps):
    """fields of the laser scan: 5e13-5e14 W/cm^2, 400-2000 nm, 2-10 cycles, any phase, a window inside the pulse"""
    rng = np.random.default_rng(2025 + seed)
    B = case["n_inst"]
    e0 = np.sqrt(10 ** rng.uniform(np.log10(5e13), np.log10(5e14), B) / 3.50944758e16)
    w = 45.5633525 / rng.uniform(400.0, 2000.0, B)
    tau = rng.integers(2, 11, B) * 2 * np.pi / w
    t = (rng.uniform(0.2, 0.6, B) * tau)[:, None] + DT * np.arange(steps + 1)
    return e0[:, None] * np.sin(np.pi * t / tau[:, None]) ** 2 * np.sin(w[:, None] * t + rng.uniform(0, 2 * np.pi, B)[:, None])


def step_counts(case, seed):
    """(steps in the pulse, all steps) of every wavefunction; batches that are not the scan are uneven"""
    B, n = case["n_inst"], case["steps"]
    if case["kind"] != "run" or B < 2 or B > 64:
        return np.full(B, n), np.full(B, n)
    rng = np.random.default_rng(7 + seed)
    f = rng.integers(max(1, n // 2), n + 1, B)
    f[rng.integers(B)] = n
    return f, np.minimum(f + rng.integers(0, max(2, n // 4), B), n + n // 4)


def inputs(case, seed):
    d = {"case": case}
    rng = np.random.default_rng(99 + seed)
    kind, L, B = case["kind"], case["n_l"], case["n_inst"]
    n_m = case.get("n_m", 1)
    lmax = L - 1 + n_m // 2
    if case.get("potentials") or kind == "arnoldi":
        bs = [bands(case, rng.uniform(0.0, 17.0), rng.uniform(1.0, 3.0)) for _ in range(B)]
        d["H"], b = np.stack([hamiltonian(x, lmax) for x in bs]), bs[0]
    else:
        b = bands(case, mask=0.35 * case["n_r"] if kind == "mask" else None)
        d["H"] = hamiltonian(b, lmax)
    d["b"] = b
    d["c0"] = packets(case, seed, n_m)
    if kind == "pcs":
        # radial integrals of outgoing waves sin(k r - l pi/2 + phase)/k, as the far field of the Coulomb waves
        k = np.linspace(0.02, 2.5, case["nkr"])
        ll = np.arange(L)
        r = 0.5 * np.arange(1, case["n_r"] + 1)
        th = np.linspace(0.0, np.pi, case["nkt"])
        sig = rng.uniform(-1.0, 1.0, (k.size, L))
        arg = k[:, None, None] * r - ll[:, None] * np.pi / 2 + np.log(2 * k[:, None, None] * r) / k[:, None, None] + sig[:, :, None]
        plm = np.stack([np.polynomial.legendre.legval(np.cos(th), np.eye(L)[i]) * np.sqrt((2 * i + 1) / (4 * np.pi)) for i in ll], 1)
        d["tables"] = {"kr": k, "kt": th, "kp": np.zeros(1), "ijl": np.sin(arg) * (0.5 / k)[:, None, None], "plm": plm[:, None, :],
                       "exm": np.ones((1, 1), complex), "cps": np.exp(1j * (sig - ll * np.pi / 2))}
    elif kind == "vgwr":
        a = pulses(case, seed, case["steps"]) / 0.057
        d["A"] = np.stack([a, 0.5 * np.roll(a, 1, axis=1)], 2)
    else:
        d["f"] = pulses(case, seed, case["steps"])
        d["nf"], d["nt"] = step_counts(case, seed)
    return d


def mlp_inputs(case, seed):
    rng = np.random.default_rng(3 + seed)
    x = rng.standard_normal((case["rows"], 10)).astype(np.float32)
    y = np.cumsum(rng.standard_normal((case["rows"], 384)), 1).astype(np.float32) / 12
    h = case["hidden"]
    sizes = [(h, 16)] + [(h, h)] * (case["layers"] - 1) + [(384, h)]
    params = []
    for _ in range(case["members"]):
        flat = []
        for n, k in sizes:
            w = rng.standard_normal((n, k)) * math.sqrt(2.0 / min(k, 10 if k == 16 else k))
            if k == 16:
                w[:, 10:] = 0.0
            flat += [w.reshape(-1), 0.1 * rng.standard_normal(n)]
        params.append(np.concatenate(flat).astype(np.float32))
    return x, y, params, sizes


# ------------------------------------------------------------------ the calls

def prepare(case, seed):
    kind = case["kind"]
    if kind.startswith("mlp"):
        x, y, params, _ = mlp_inputs(case, seed)
        net = q.mlp_ensemble(10, 384, case["hidden"], case["layers"], case["members"], seed=seed)
        for i, p in enumerate(params):
            net.set_params(i, p)
        return {"kind": kind, "net": net, "x": x, "y": y}
    d = inputs(case, seed)
    b, n_r, p, L, B = d["b"], case["n_r"], case["p"], case["n_l"], case["n_inst"]
    s = {"kind": kind, "c0": d["c0"], "d": d}
    if kind == "pcs":
        s["spec"] = q.spectrum_c_pcs(case["nkr"], case["nkt"], 1).initialize(n_r, p, L, knots(case), 0.02, 2.5, 0.0, np.pi, 0.0, 0.0, 1.0,
                                                                          tables=d["tables"])
        s["prop"] = q.propagator_cn_hc_lgwz().initialize(n_r, p, L, b["S"], b["R"], d["H"], DT, n_inst=B)
        s["prop"].put_device(d["c0"].data_ptr())
    elif kind == "arnoldi":
        s["prop"] = q.propagator_hc_lgwz(case["kmax"], 1e-14, 1e-8).initialize(n_r, p, L, b["S"], b["R"], d["H"], q.y10_coupling(L), DT, n_inst=B)
    elif kind == "vgwr":
        s["prop"] = q.propagator_cn_hc_vgwr().initialize(n_r, p, L, case["n_m"], -(case["n_m"] // 2), b["S"], b["I"], b["D"], d["H"], DT, n_inst=B)
        s["host"] = d["c0"].cpu().numpy()
    else:
        s["prop"] = q.propagator_cn_hc_lgwz().initialize(n_r, p, L, b["S"], b["R"], d["H"], DT, n_inst=B)
    s["out"] = torch.empty_like(d["c0"])
    torch.cuda.synchronize()
    return s


def run(s):
    kind = s["kind"]
    if kind == "mlp_grad":
        loss, grad = s["net"].loss_grad(s["x"], s["y"])
        return {"loss": loss, "grad": grad}
    if kind == "mlp_predict":
        return s["net"].predict(s["x"])
    prop, d = s["prop"], s["d"]
    if kind == "pcs":
        return s["spec"].measure_prj(prop)
    if kind == "vgwr":
        prop.put(s["host"])
        n = d["case"]["steps"]
        prop.run(d["A"], np.full(d["case"]["n_inst"], n))
        return prop.get()
    prop.put_device(s["c0"].data_ptr())
    res = {"state": s["out"]}
    if kind == "step":
        prop.propagate(d["f"][:, 0], d["f"][:, 1])
    elif kind == "run":
        prop.run(d["f"], d["nf"], d["nt"])
    elif kind == "dipole":
        res["z"] = prop.run_dipole(d["f"], d["nf"], d["nt"], d["b"]["R"])
    elif kind == "mask":
        prop.run_ex(d["f"], d["nf"], d["nt"], mask=d["b"]["M"])
    elif kind == "arnoldi":
        res["crit"] = prop.run(d["f"][:, :-1])
    prop.get_device(s["out"].data_ptr())
    return res


def work(case):
    """Bytes: the state in and out once, the bands and tables once.  Operations: of the banded solves and the
    l transforms (or the products) that one pass cannot do without."""
    if case["kind"].startswith("mlp"):
        h, n = case["hidden"], case["members"]
        w = 16 * h + (case["layers"] - 1) * h * h + 384 * h
        back = 3 if case["kind"] == "mlp_grad" else 1
        out = n * (w * 4 if back == 3 else case["rows"] * 384 * 4)
        return {"bytes": n * w * 4 + case["rows"] * 394 * 4 + out, "flops": 2.0 * back * n * w * case["rows"]}
    N, p, L, B = case["n_r"], case["p"], case["n_l"], case["n_inst"]
    ch = L * case.get("n_m", 1)
    state = 16.0 * B * ch * N
    if case["kind"] == "pcs":
        k, t = case["nkr"], case["nkt"]
        return {"bytes": state + 8.0 * k * L * N + 16.0 * B * k * t, "flops": 4.0 * B * k * L * (N + t)}
    if case["kind"] == "arnoldi":
        k = case["kmax"]
        return {"bytes": 2 * state + 8.0 * B * L * N * (p + 1), "flops": case["steps"] * B * L * N * k * (12.0 * (2 * p + 1) + 8.0 * p + 14.0 * k)}
    solve = 2.0 * (8 * p + 4 * p + 8)
    if case["kind"] == "vgwr":
        return {"bytes": 2 * state + 8.0 * ch * N, "flops": case["steps"] * B * N * (9.0 * ch * solve + 2.5 * ch * ch)}
    bytes_ = 2 * state + 8.0 * (B if case.get("potentials") else 1) * L * N * (p + 1) + 8.0 * B * case["steps"]
    extra = {"mask": 16.0 * p, "dipole": 4.0}.get(case["kind"], 0.0)
    return {"bytes": bytes_, "flops": case["steps"] * B * L * N * (2 * solve + 4.0 * L + extra)}


# ------------------------------------------------------------------ the same outputs in 64 bits

def T(x):
    return torch.as_tensor(np.asarray(x), device=DEV)


def dense(b, sign=1.0):
    n, ne = b.shape
    a = torch.diag(T(b[:, 0]))
    for k in range(1, ne):
        v = T(b[:n - k, k])
        a += torch.diag(v, k) + sign * torch.diag(v, -k)
    return a


def cayley(h, g):
    """2 (1 + i g h)^-1 - 1 of real symmetric h"""
    one = torch.eye(h.shape[-1], device=DEV, dtype=torch.complex128)
    return 2 * torch.linalg.inv(one + 1j * g * h) - one


class Basis:
    """radial functions orthonormal in S that diagonalise <B|r|B>; y = c S V, c = y V^T"""

    def __init__(self, d):
        b = d["b"]
        S = dense(b["S"])
        Linv = torch.linalg.inv(torch.linalg.cholesky(S))
        self.r, Q = torch.linalg.eigh(Linv @ dense(b["R"]) @ Linv.T)
        self.V = Linv.T @ Q
        self.into = (S @ self.V).to(torch.complex128)
        self.back = self.V.T.contiguous().to(torch.complex128)

    def rep(self, band, sign=1.0):
        a = self.V.T @ dense(band, sign) @ self.V
        return 0.5 * (a + sign * a.T)


def exact(case, seed):
    if case["kind"].startswith("mlp"):
        return exact_mlp(case, seed)
    d = inputs(case, seed)
    if case["kind"] == "pcs":
        t = d["tables"]
        amp = torch.einsum("klr,ilr->ikl", T(t["ijl"]).to(torch.complex128), d["c0"][:, 0]) * T(t["cps"])
        return (math.sqrt(2 / math.pi) * torch.einsum("ikl,tl->ikt", amp, T(t["plm"][:, 0]).to(torch.complex128)))[..., None].cpu().numpy()
    bas = Basis(d)
    y = d["c0"] @ bas.into
    L, B = case["n_l"], case["n_inst"]
    if case["kind"] == "vgwr":
        return (exact_vgwr(case, d, bas, y) @ bas.back).cpu().numpy()
    ll = np.arange(1.0, L)
    y10 = T(np.sqrt(ll * ll / ((2 * ll - 1) * (2 * ll + 1))))
    Y = torch.diag(y10, 1) + torch.diag(y10, -1)
    per = d["H"].ndim == 4
    H = torch.stack([torch.stack([bas.rep(h) for h in one]) for one in (d["H"] if per else d["H"][None])])
    y = y[:, 0]
    f, n = T(d["f"]), case["steps"]
    if case["kind"] == "arnoldi":
        return exact_arnoldi(case, bas, y, H, Y, f)
    lam, P = torch.linalg.eigh(Y)
    P = P.to(torch.complex128)
    F = torch.stack([cayley(h, DT / 2) for h in H])          # [1 or inst][l][r][r]
    M = bas.rep(d["b"]["M"]).to(torch.complex128) if case["kind"] == "mask" else None
    nf, nt = T(d["nf"]), T(d["nt"])
    z = torch.zeros((B, int(nt.max())), device=DEV, dtype=torch.float64)

    def couple(v, s, on):
        g = torch.where(on, f[:, s], torch.zeros_like(f[:, s]))[:, None, None] * lam[:, None] * bas.r * (DT / 4)
        return torch.einsum("lk,ikr->ilr", P, (1 - 1j * g) / (1 + 1j * g) * torch.einsum("lk,ilr->ikr", P, v))

    for s in range(int(nt.max())):
        live = s < nt
        if case["kind"] == "dipole":
            z[:, s] = 2 * (y10[:, None] * (y[:, :-1].conj() * y[:, 1:]).real * bas.r).sum((1, 2))
        v = couple(y, s, s < nf) if s < n else y
        v = torch.einsum("ilrk,ilk->ilr", F, v) if per else torch.einsum("lrk,ilk->ilr", F[0], v)
        v = couple(v, s + 1, s < nf) if s < n else v
        y = torch.where(live[:, None, None], v, y)
        if M is not None:
            y = torch.where(live[:, None, None], y @ M, y)
    res = {"state": (y @ bas.back)[:, None]}
    if case["kind"] == "dipole":
        res["z"] = z.cpu().numpy()
    return res


def exact_arnoldi(case, bas, w, H, Y, f):
    """w <- exp(-i dt H) w in a Krylov space of kmax vectors, H = H_l + f r Y in the orthonormal basis"""
    out, crit = [], np.zeros((case["n_inst"], case["steps"]), np.int8)
    Hc, Yc = H.to(torch.complex128), Y.to(torch.complex128)
    for i in range(case["n_inst"]):
        v = w[i]
        for s in range(case["steps"]):
            norm = torch.linalg.vector_norm(v)
            u, a, b = [v / norm], [], []
            while len(a) < case["kmax"]:
                t = torch.einsum("lrk,lk->lr", Hc[i], u[-1]) + f[i, s] * (Yc @ (u[-1] * bas.r))
                x = [(e.conj() * t).sum() for e in u]
                for j, e in enumerate(u):
                    if j == len(u) - 1 or abs(x[j]) ** 2 > 4e-27:
                        t = t - x[j] * e
                a.append(float(x[-1].real))
                nu = float(torch.linalg.vector_norm(t)) ** 2
                if nu < 1e-13:
                    break
                b.append(math.sqrt(nu))
                u.append(t / b[-1])
            m = len(a)
            e, z = np.linalg.eigh(np.diag(a) + np.diag(b[:m - 1], 1) + np.diag(b[:m - 1], -1))
            x = (z * (np.exp(-1j * DT * e) * z[0])).sum(1) * float(norm)
            v = sum(complex(x[j]) * u[j] for j in range(m))
            eps = abs(x[-1]) ** 2 if m > 1 else 0.0
            crit[i, s] = 0 if eps > 1e-8 else 1 if eps > 1e-14 else 2
        out.append(v)
    return {"state": (torch.stack(out) @ bas.back)[:, None], "crit": crit}


def exact_vgwr(case, d, bas, y):
    """Cayley factors of the four couplings (m -> m + 1, l -> l +- 1) x (d/dr or 1/r), x first, around the
    field-free step; Z Hermitian over (m, l), the radial operator diagonalised too."""
    n_m, L, B, N = case["n_m"], case["n_l"], case["n_inst"], case["n_r"]
    m0, ch = -(n_m // 2), case["n_l"] * case["n_m"]
    radial = []
    o, v = torch.linalg.eigh(1j * bas.rep(d["b"]["D"], -1.0))
    radial.append((-1j * o, v))
    o, v = torch.linalg.eigh(bas.rep(d["b"]["I"]))
    radial.append((o.to(torch.complex128), v.to(torch.complex128)))
    comps = []
    for q11, turned in ((False, False), (True, True), (False, True), (True, False)):
        Z = np.zeros((ch, ch), complex)
        for im in range(n_m - 1):
            for il in range(L):
                m = m0 + im
                l = il + abs(m)
                for up in (1, -1):
                    jl = l + up - abs(m + 1)
                    if l + up < 0 or jl < 0 or jl >= L:
                        continue
                    if up > 0:
                        e = -math.sqrt((l + m + 1) * (l + m + 2) / ((2 * l + 1) * (2 * l + 3))) * ((l + 1) if q11 else 1)
                    else:
                        e = math.sqrt((l - m) * (l - m - 1) / ((2 * l + 1) * (2 * l - 1))) * (-l if q11 else 1)
                    i, j = im * L + il, (im + 1) * L + jl
                    Z[j, i] = (-1.0 if q11 else 1.0) * e * (-1j if turned else 1.0)
                    Z[i, j] = np.conj(Z[j, i])
        lam, P = torch.linalg.eigh(T(Z))
        comps.append((lam, P, radial[1 if q11 else 0], q11))
    l_of = [il + abs(m0 + im) for im in range(n_m) for il in range(L)]
    F = torch.stack([cayley(bas.rep(h), DT / 2) for h in d["H"]])
    y = y.reshape(B, ch, N)

    def couple(c, a):
        lam, P, (o, v), q11 = comps[c]
        g = (a * (DT / 4))[:, None, None] * lam[:, None] * o
        g = 1j * g if q11 else -g
        t = torch.einsum("ck,icr->ikr", P.conj(), y) @ v.conj()
        return torch.einsum("ck,ikr->icr", P, (1 - g) / (1 + g) * t) @ v.T

    A = T(d["A"]) / 2
    for s in range(case["steps"]):
        for c, a in ((0, -A[:, s, 0]), (1, A[:, s, 0]), (2, -A[:, s, 1]), (3, -A[:, s, 1])):
            y = couple(c, a)
        z = torch.empty_like(y)
        for j, l in enumerate(l_of):
            z[:, j] = y[:, j] @ F[l].T
        y = z
        for c, a in ((3, -A[:, s + 1, 1]), (2, -A[:, s + 1, 1]), (1, A[:, s + 1, 0]), (0, -A[:, s + 1, 0])):
            y = couple(c, a)
    return y.reshape(B, n_m, L, N)


def exact_mlp(case, seed):
    x, y, params, sizes = mlp_inputs(case, seed)
    x, y = T(x).double(), T(y).double()
    x = torch.cat([x, torch.zeros((x.shape[0], 6), device=DEV, dtype=torch.float64)], 1)
    losses, grads, outs = [], [], []
    for flat in params:
        leaf = T(flat).double().requires_grad_(True)
        a, o = x, 0
        for j, (n, k) in enumerate(sizes):
            w, o = leaf[o:o + n * k].reshape(n, k), o + n * k
            b, o = leaf[o:o + n], o + n
            a = a @ w.T + b
            if j < len(sizes) - 1:
                a = torch.nn.functional.gelu(a)
        outs.append(a.detach().cpu().numpy())
        if case["kind"] == "mlp_grad":
            loss = ((a - y) ** 2).mean()
            loss.backward()
            losses.append(loss.item())
            grads.append(leaf.grad.cpu().numpy())
    return {"loss": np.array(losses), "grad": np.stack(grads)} if losses else np.stack(outs)
