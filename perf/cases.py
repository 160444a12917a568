"""The workloads on which this package's speed is measured.

``listed`` names them and ``draw`` gives others of the same ranges; ``prepare``
makes what a program holds before the call (line lists on the device, a plan,
output buffers), ``run`` is one pass through the package's public entry points,
``work`` what a pass cannot do without, and ``exact`` the same results in FP64
torch on the same inputs, written from the method alone.

Line lists are synthetic, made on the GPU from the seed, with the distributions
of ``radis_gb300/synthetic.py``; ``moderate`` ones keep the lower-state energies
below 5000 cm-1, and their path lengths put the mean absorbance of a window
near one, so that emissivity and transmittance are neither 0 nor 1.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from radis_gb300 import _lib as L
from radis_gb300 import autodiff
from radis_gb300.gpu import gpuApp
from radis_gb300.slit import convolve_device

# constants of the method (SI; the Doppler width's k in CGS)
C2 = 6.62607015e-34 * 2.99792458e8 / 1.3806490e-23 * 100.0
NA, KB, KB_CGS, C_CGS = 6.02214076e23, 1.3806490e-23, 1.380648813e-16, 2.99792458e10
TREF, ATM = 296.0, 1.01325
LN2 = math.log(2.0)
# default node spacings in log width
DXL = math.log((0.01 / 0.20) ** 0.5 + 1)
DXG = math.log((0.01 / 0.46) ** 0.5 + 1)
Q_POWER = 1.5      # Q(T) ~ T^1.5 where a case uses partition functions
MODERATE = (1e-31, 1e-25, 1500.0, 5000.0)   # intensities, mean and largest lower-state energy
DEV = "cuda:0"

BASE = dict(kind="spectrum", lines="uniform", n_lines=10_000, lo=1900.0, hi=2300.0, mass=28.0, n_iso=1, shift=False,
            moderate=False, vmin=1900.0, dv=0.002, n_v=200_001, n_G=0, n_L=0, T=700.0, p=1.01325, x=0.1, path=1.0)


def listed():
    def case(name, **kw):
        return dict(BASE, name=name, **kw)

    return [
        # the smallest spectrum: a 10 cm-1 survey window at low pressure on a
        # coarse step, where folded lineshape terms are active
        case("narrow_low_pressure", n_lines=2000, lo=2000.0, hi=2010.0, vmin=2000.0, dv=0.02, n_v=501, T=1500.0,
             p=0.02, x=0.3),
        # an everyday small-molecule spectrum: 10k CO-like lines, 200k points, default node spacing
        case("co_10k"),
        # the headline spectrum: 5M CO2-like lines, 400k points, 8 x 16 nodes
        case("co2_5M", n_lines=5_000_000, lo=2000.0, hi=2400.0, mass=44.0, vmin=2000.0, dv=0.001, n_v=400_001,
             n_G=8, n_L=16, T=1500.0, p=1.0),
        # the largest: a 100M-line H2O-like hot list over 7500 cm-1, 12 x 24 nodes
        case("h2o_100M", lines="h2o", n_lines=100_000_000, lo=500.0, hi=8000.0, mass=18.0, vmin=500.0, dv=0.005,
             n_v=1_500_001, n_G=12, n_L=24, T=2000.0, p=1.0, x=0.2),
        # the core of a hot band on a coarse step: thousands of lines per grid column
        case("dense_band", n_lines=12_000_000, lo=1600.0, hi=1650.0, mass=18.0, vmin=1600.0, dv=0.01, n_v=5001,
             T=2000.0, p=1.0, x=0.2),
        # isotopologues, pressure shifts and partition functions, with absorbance,
        # emissivity, transmittance and radiance computed on the device
        case("isotopes_quantities", kind="quantities", n_lines=600_000, lo=2150.0, hi=2400.0, mass=44.0, n_iso=3,
             shift=True, moderate=True, vmin=2160.0, dv=0.002, n_v=112_347, T=900.0, p=3.0, x=0.04, path=0.11),
        # the drop-in application object: one iterate into host memory, as the
        # recalculation behind an interactive slider does
        case("app_iterate", kind="iterate", n_lines=300_000, moderate=True, T=1000.0, n_v=150_000, lo=1980.0,
             vmin=1990.0, x=0.05, path=0.34),
        # gradients of an absorbance with respect to (T, p, x), as in a fit
        case("adjoint_co", kind="adjoint", dv=0.001, n_v=400_001),
        # derivative spectra dA/d(T, p, x) of the same configuration
        case("jacobian_co", kind="jacobian", dv=0.001, n_v=400_001),
        # a 0.5 cm-1 instrument slit on a 400k-point spectrum already on the device
        dict(name="slit_1001", kind="slit", n_v=400_001, dv=0.001, taps=1001, valid=True),
        # a stream of mixed requests over resident lists
        dict(name="served_stream", kind="served", requests=24, stream=1, n_co=10_000, n_co2=2_000_000,
             n_h2o=10_000_000, slots=8),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _unit_path(n_lines, lo, hi, T, p, x):
    """Path (cm) of mean absorbance 1 through a ``moderate`` list: 1 / (lines
    per cm-1 x mean intensity at T x number density)."""
    s_lo, s_hi, mean, cap = MODERATE
    a = C2 * (1 / TREF - 1 / T) - 1 / mean
    boltz = (math.expm1(a * cap) / (a * mean) if abs(a * cap) > 1e-9 else cap / mean) + math.exp(a * cap)
    s = (s_hi - s_lo) / math.log(s_hi / s_lo) * boltz
    return 1.0 / (n_lines / (hi - lo) * s * p * 1e5 / (KB * T) * 1e-6 * x)


def draw(rng: random.Random):
    kind = rng.choice(["spectrum", "spectrum", "spectrum", "quantities", "iterate", "adjoint", "jacobian", "slit",
                       "served"])
    if kind == "slit":
        return dict(kind=kind, n_v=int(_log(rng, 2_000, 1_500_000)), dv=rng.choice([0.001, 0.002, 0.005, 0.01]),
                    taps=int(_log(rng, 3, 4000)), valid=rng.random() < 0.5)
    if kind == "served":
        return dict(kind=kind, requests=rng.randint(4, 32), stream=rng.randrange(1 << 30),
                    n_co=int(_log(rng, 1_000, 50_000)), n_co2=int(_log(rng, 50_000, 3_000_000)),
                    n_h2o=int(_log(rng, 500_000, 15_000_000)), slots=rng.choice([2, 4, 8]))
    small = kind in ("adjoint", "jacobian", "iterate")
    dv = rng.choice([0.001, 0.002, 0.005, 0.01])
    n_v = int(_log(rng, 501, 500_000 if small else 1_500_000))
    vmin = rng.uniform(500.0, 2500.0)
    width = (n_v - 1) * dv
    extra = rng.choice([0.0, 0.05, 0.5]) * width
    n_lines = int(_log(rng, 1_000, min(400_000 if small else 10_000_000, 2500 * n_v)))
    lo, hi = vmin - min(extra, 0.5 * vmin), vmin + width + extra
    T, p, x = (round(_log(rng, 300.0, 1200.0 if small else 3000.0), 2), round(_log(rng, 0.1, 10.0), 4),
               round(_log(rng, 0.01, 1.0), 4))
    n_iso = rng.choice([1, 1, 3])
    fixed = rng.random() < 0.4 and kind != "iterate"   # the application object takes spacings
    return dict(BASE, kind=kind, n_lines=n_lines, lo=lo, hi=hi, mass=rng.choice([18.0, 28.0, 44.0]), n_iso=n_iso,
                shift=rng.random() < 0.5, moderate=kind != "spectrum", vmin=vmin, dv=dv, n_v=n_v,
                n_G=rng.randint(4, 12) if fixed else 0, n_L=rng.randint(6, 24) if fixed else 0, T=T, p=p, x=x,
                path=float("%.3g" % _unit_path(n_lines, lo, hi, T, p, x)) if kind != "spectrum" else 1.0)


# --- inputs ---------------------------------------------------------------------
def _gen(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1_000_003 + salt) % (1 << 62))
    return g


def _make_lines(c, seed, salt=0):
    """Line columns on the GPU, ascending v0."""
    g, n = _gen(seed, salt), int(c["n_lines"])

    def u(lo, hi, dtype=torch.float64):
        return torch.rand(n, generator=g, device=DEV, dtype=dtype) * (hi - lo) + lo

    if c["lines"] == "h2o":   # bands near 1600 and 3700 cm-1 over a log-uniform background
        which = u(0.0, 1.0, torch.float32)
        v0 = torch.exp(u(math.log(c["lo"]), math.log(c["hi"])))
        for lo, hi, centre, sig in ((0.0, 0.45, 1600.0, 0.06), (0.45, 0.8, 3700.0, 0.04)):
            z = torch.randn(n, generator=g, device=DEV, dtype=torch.float64)
            v0 = torch.where((which >= lo) & (which < hi), torch.exp(z * sig + math.log(centre)), v0)
            del z
        v0 = v0.clamp_(c["lo"], c["hi"] - 1e-6)
        s_lo, s_hi, mean, cap = 1e-30, 1e-18, 5000.0, 40000.0
    else:
        v0 = u(c["lo"], c["hi"])
        s_lo, s_hi, mean, cap = 1e-26, 1e-19, 3000.0, 20000.0
    if c["moderate"]:
        s_lo, s_hi, mean, cap = MODERATE
    d = dict(v0=torch.sort(v0).values)
    d["S_ref"] = torch.exp(u(math.log(s_lo), math.log(s_hi)))
    d["El"] = (-torch.log1p(-u(0.0, 1.0)) * mean).clamp_(max=cap).float()
    d["g_air"] = u(0.03, 0.08, torch.float32)
    d["g_self"] = u(0.05, 0.1, torch.float32)
    d["n_air"] = u(0.5, 0.8, torch.float32)
    if c["shift"]:
        d["delta"] = u(-0.01, 0.01, torch.float32)
    if c["n_iso"] > 1:
        d["iso"] = torch.randint(0, c["n_iso"], (n,), generator=g, device=DEV, dtype=torch.uint8)
    return d


def _masses(c):
    return np.array([c["mass"] + i for i in range(c["n_iso"])])


def _q(c):
    """Q(Tref)/Q(T) per isotopologue, where the case has several (else 1)."""
    return None if c["n_iso"] == 1 else np.array([(TREF / c["T"]) ** (Q_POWER + 0.1 * i) for i in range(c["n_iso"])])


def _q_calls(c):
    return [lambda T, k=Q_POWER + 0.1 * i: (T / TREF) ** k for i in range(c["n_iso"])]


def _nodes(c):
    return dict(n_G=c["n_G"], n_L=c["n_L"]) if c["n_G"] else dict(dxG=DXG, dxL=DXL)


_CTX = []


def _context():
    if not _CTX:
        _CTX.append(L.Context(0))
    return _CTX[0]


def _upload(c, seed, salt=0):
    d = {k: v.cpu().numpy() for k, v in _make_lines(c, seed, salt).items()}
    return L.Lines(_context(), d, _masses(c))


def _slit(c):
    m = int(c["taps"])
    s = 1.0 - np.abs(np.arange(m) - (m - 1) / 2) / (m / 2)
    return (s / (s.sum() * c["dv"])).astype(np.float32)


def _spectrum_in(c, seed):
    return torch.rand(int(c["n_v"]), generator=_gen(seed), device=DEV, dtype=torch.float32) ** 8


def _weights(c, seed):   # upstream gradient of a band integral: a positive detector response
    return torch.rand(int(c["n_v"]), generator=_gen(seed, 7), device=DEV, dtype=torch.float32) + 0.5


def _served_lists(c):
    return {"co": dict(BASE, n_lines=c["n_co"]),
            "co2": dict(BASE, n_lines=c["n_co2"], lo=2000.0, hi=2400.0, mass=44.0),
            "h2o": dict(BASE, lines="h2o", n_lines=c["n_h2o"], lo=500.0, hi=8000.0, mass=18.0)}


def _served_requests(c):
    """Window, step and conditions of each request, from the case alone."""
    rng = random.Random(int(c["stream"]))
    out = []
    for _ in range(int(c["requests"])):
        name = rng.choice(["co", "co2", "h2o"])
        lo, hi = {"co": (1900.0, 2300.0), "co2": (2000.0, 2400.0), "h2o": (500.0, 8000.0)}[name]
        width = min(_log(rng, 50.0, 2000.0), hi - lo)
        dv = rng.choice([0.001, 0.002, 0.005, 0.01])
        vmin = lo + rng.uniform(0.0, hi - lo - width)
        n_v = min(int(width / dv) + 1, 1_000_000)
        out.append(dict(list=name, vmin=vmin, dv=dv, n_v=n_v, T=_log(rng, 300.0, 3000.0), p=_log(rng, 0.1, 10.0),
                        x=_log(rng, 0.01, 1.0)))
    return out


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "slit":
        s = dict(kind=kind, c=c, I=_spectrum_in(c, seed), slit=torch.from_numpy(_slit(c)).to(DEV))
        s["out"] = torch.empty_like(s["I"])
        return s
    if kind == "served":
        lists = {k: _upload(d, seed, i) for i, (k, d) in enumerate(_served_lists(c).items())}
        req = _served_requests(c)
        for r in req:
            r["out"] = torch.empty(r["n_v"], dtype=torch.float32, pin_memory=True).numpy()
        return dict(kind=kind, c=c, lists=lists, req=req, server=L.Server(_context(), slots=c["slots"]))
    if kind == "iterate":
        d = {k: v.cpu().numpy() for k, v in _make_lines(c, seed).items()}
        n = len(d["v0"])
        iso = d["iso"] if "iso" in d else np.zeros(n, np.int64)
        app = gpuApp(c["vmin"], c["n_v"], c["dv"], DXG, DXL, d["v0"], d.get("delta", np.zeros(n, np.float32)), d["n_air"],
                     None, d["El"], np.array([d["g_self"], d["g_air"]]), iso, _masses(c), _q_calls(c), S_ref=d["S_ref"])
        return dict(kind=kind, c=c, app=app)
    ln = _upload(c, seed)
    s = dict(kind=kind, c=c, lines=ln, q=_q(c),
             plan=L.Plan(ln, c["vmin"], c["dv"], c["n_v"], **_nodes(c)))
    if kind == "adjoint":
        s["w"] = _weights(c, seed)
        s["cond"] = [torch.tensor(c[k], dtype=torch.float32, requires_grad=True) for k in ("T", "p", "x")]
    elif kind != "jacobian":
        rows = 5 if kind == "quantities" else 1
        s["out"] = torch.empty((rows, c["n_v"]), dtype=torch.float32, device=DEV)
    return s


def run(state):
    c, kind = state["c"], state["kind"]
    stream = torch.cuda.current_stream().cuda_stream or 1
    if kind == "spectrum":
        info = state["plan"].synthesize_device(c["T"], c["p"], c["x"], state["out"].data_ptr(), stream,
                                               q_ratio=state["q"])
        return {"abscoeff": state["out"][0], "log_scale": info.log_scale}
    if kind == "quantities":
        info = state["plan"].synthesize_quantities(c["T"], c["p"], c["x"], c["path"], state["out"].data_ptr(), stream,
                                                   q_ratio=state["q"])
        return {"rows": list(state["out"]), "log_scale": info.log_scale}
    if kind == "iterate":
        rows, _times = state["app"].iterate_quantities(c["p"], c["T"], c["x"], c["path"])
        return rows
    if kind == "adjoint":
        A = autodiff.absorbance(state["plan"], *state["cond"], path_length=c["path"], Q=_q_calls(c))
        return {"absorbance": A.detach(), "grad": torch.autograd.grad(A, state["cond"], state["w"])}
    if kind == "jacobian":
        return autodiff.jacobian(state["plan"], c["T"], c["p"], c["x"], Q=_q_calls(c))
    if kind == "slit":
        return convolve_device(state["I"], state["slit"], c["dv"], mode="valid" if c["valid"] else "same",
                               out=state["out"], stream=stream)
    srv = state["server"]
    tickets = [srv.submit(state["lists"][r["list"]], r["vmin"], r["dv"], r["n_v"], r["T"], r["p"], r["x"], dxG=DXG,
                          dxL=DXL, out=r["out"], axes_window=True) for r in state["req"]]
    done = [srv.wait(t) for t in tickets]
    return {"spectra": [o for o, _, _ in done], "log_scale": [i.log_scale for _, i, _ in done]}


# --- necessary work ---------------------------------------------------------------
def _ft_length(n_v):
    """Shortest supported transform of at least 2 n_v points: n1 n2 with n1 in
    {512, 64, 8} and n2 = 32 x a 5-smooth number, at most 8192; n1 = 8 only
    when it is a quarter shorter than the others or nothing else fits."""
    best = 0
    for n1 in (512, 64, 8):
        m = max(1, -(-(-(-2 * n_v // n1)) // 32))
        while True:
            r = m
            for f in (2, 3, 5):
                while r % f == 0:
                    r //= f
            if r == 1:
                break
            m += 1
        n = n1 * 32 * m
        if 32 * m > 8192 or n < 2 * n_v or (n1 == 8 and best and 4 * n > 3 * best):
            continue
        if not best or n < best:
            best = n
    return best


def _spectrum_work(c, per_line=100.0):
    """Line records read once, a real transform of the accumulated rows and one
    back (at least one row each); ~100 operations a line for its intensity,
    widths and weights."""
    frac = min(1.0, (c["n_v"] - 1) * c["dv"] / (c["hi"] - c["lo"]))
    n = c["n_lines"] * frac
    nf = _ft_length(c["n_v"])
    return {"bytes": n * (28 + (4 if c["shift"] else 0) + (1 if c["n_iso"] > 1 else 0)) + 4.0 * c["n_v"],
            "flops": n * per_line + 2 * 2.5 * nf * math.log2(nf)}


def work(case):
    c, kind = case, case["kind"]
    if kind == "slit":
        return {"bytes": 8.0 * c["n_v"] + 4.0 * c["taps"], "flops": 2.0 * c["n_v"] * c["taps"]}
    if kind == "served":
        lists = _served_lists(c)
        tot = {"bytes": 0.0, "flops": 0.0}
        for r in _served_requests(c):
            w = _spectrum_work(dict(lists[r["list"]], **{k: r[k] for k in ("vmin", "dv", "n_v")}))
            tot = {k: tot[k] + w[k] for k in tot}
        return tot
    w = _spectrum_work(c)
    if kind in ("quantities", "iterate"):
        w["bytes"] += 16.0 * c["n_v"]
    elif kind == "adjoint":       # forward, then the transposed pass over the same lines
        w = {"bytes": 2 * w["bytes"], "flops": 2.5 * w["flops"]}
    elif kind == "jacobian":      # forward and three tangents; one read of the lines
        w = {"bytes": w["bytes"] + 12.0 * c["n_v"], "flops": 4 * w["flops"]}
    return w


# --- FP64 results -----------------------------------------------------------------
def _axes(c, d, T, p, x, masses, window=False):
    """(log_wG_min, dxG, n_G, log_wL_min, dxL, n_L): log-width bounds of the
    list (or, for ``window``, of the v0 the window can reach), the top raised by 1e-4."""
    p_atm = p / ATM
    lc = [math.log(2.0 / C_CGS * math.sqrt(2.0 * NA * KB_CGS * LN2 / m)) for m in masses]
    lo, hi = math.inf, -math.inf
    for i in range(len(masses)):
        v = d["v0"] if "iso" not in d else d["v0"][d["iso"] == i]
        if not v.numel():
            continue
        a, b = math.log(float(v.min())), math.log(float(v.max()))
        if window:
            sh = c["dv"] + (float(d["delta"].abs().max()) * p_atm if "delta" in d else 0.0)
            a, b = max(a, math.log(c["vmin"] - sh)), min(b, math.log(c["vmin"] + (c["n_v"] - 1) * c["dv"] + sh))
        lo, hi = min(lo, a + lc[i]), max(hi, b + lc[i])
    lo, hi = lo + 0.5 * math.log(T), hi + 0.5 * math.log(T) + 1e-4
    t, l2p = math.log(TREF / T), math.log(2.0 * p_atm)
    ga, gs, na = (d[k].double() for k in ("g_air", "g_self", "n_air"))
    ll = float((torch.log(torch.minimum(ga, gs)) + na * t).min()) + l2p
    lh = float((torch.log(torch.maximum(ga, gs)) + na * t).max()) + l2p + 1e-4
    out = []
    for a, b, dx, n in ((lo, hi, DXG, c["n_G"]), (ll, lh, DXL, c["n_L"])):
        n, dx = (n, (b - a) / (n - 1)) if n else (max(2, math.ceil((b - a) / dx) + 1), dx)
        out += [a, dx, n]
    return out


def _exact_ldm(c, d, T, p, x, axes, masses, q, ls, theta=None, dlnq=None):
    """LDM [node, n_v] in units of exp(ls), or its derivative along theta (0: T, 1: p, 2: x)."""
    lg0, dxG, NG, ll0, dxL, NL = axes
    n_v, p_atm = c["n_v"], p / ATM
    dens = p * 1e5 / (KB * T) * 1e-6 * x
    ldm = torch.zeros(NG * NL * n_v, dtype=torch.float64, device=DEV)
    lc = torch.tensor([math.log(2.0 / C_CGS * math.sqrt(2.0 * NA * KB_CGS * LN2 / m)) for m in masses],
                      dtype=torch.float64, device=DEV)
    lq = torch.tensor(np.log(q), dtype=torch.float64, device=DEV)
    dq = torch.tensor(np.zeros(len(masses)) if dlnq is None else dlnq, dtype=torch.float64, device=DEV)
    step = 4_000_000
    for a in range(0, d["v0"].numel(), step):
        e = {k: v[a:a + step] for k, v in d.items()}
        shift = e["delta"].double() if "delta" in e else 0.0
        pos = ((e["v0"] - c["vmin"]) + shift * p_atm) / c["dv"]
        k0 = torch.floor(pos)
        keep = (k0 >= 0) & (k0 + 1 < n_v)
        e = {k: v[keep] for k, v in e.items()}
        tv, k0 = (pos - k0)[keep], k0[keep].long()
        v0, El, ga, gs, na = (e[k].double() for k in ("v0", "El", "g_air", "g_self", "n_air"))
        iso = e["iso"].long() if "iso" in e else torch.zeros_like(k0)
        gam = ga + x * (gs - ga)
        pl = (torch.log(v0) + lc[iso] + 0.5 * math.log(T) - lg0) / dxG
        pm = (torch.log(gam) + na * math.log(TREF / T) + math.log(2.0 * p_atm) - ll0) / dxL
        l0 = torch.floor(pl).clamp(0, NG - 2)
        m0 = torch.floor(pm).clamp(0, NL - 2)
        tG, tL, l0, m0 = pl - l0, pm - m0, l0.long(), m0.long()
        I = torch.exp(torch.log(e["S_ref"]) - torch.log(-torch.expm1(-C2 * v0 / TREF)) - C2 * El * (1 / T - 1 / TREF)
                      + torch.log(-torch.expm1(-C2 * v0 / T)) + lq[iso] + math.log(dens) - ls)
        zero = torch.zeros_like(I)
        if theta == 0:
            rate = C2 * El / T ** 2 - C2 * v0 / T ** 2 / torch.expm1(C2 * v0 / T) + dq[iso] - 1.0 / T
            dv_, dG, dL = zero, zero + 0.5 / (T * dxG), -na / (T * dxL)
        elif theta == 1:
            rate, dG, dL = zero + 1.0 / p, zero, zero + 1.0 / (p * dxL)
            dv_ = e["delta"].double() / (ATM * c["dv"]) if "delta" in e else zero
        elif theta == 2:
            rate, dv_, dG, dL = zero + 1.0 / x, zero, zero, (gs - ga) / gam / dxL
        for ck in (0, 1):
            wk, sk = (tv, 1.0) if ck else (1 - tv, -1.0)
            for cl in (0, 1):
                wl, sl = (tG, 1.0) if cl else (1 - tG, -1.0)
                for cm in (0, 1):
                    wm, sm = (tL, 1.0) if cm else (1 - tL, -1.0)
                    w = wk * wl * wm
                    if theta is not None:
                        w = rate * w + sk * dv_ * wl * wm + wk * sl * dG * wm + wk * wl * sm * dL
                    ldm.index_add_(0, ((l0 + cl) * NL + m0 + cm) * n_v + k0 + ck, I * w)
    return ldm.view(NG * NL, n_v)


def _exact_convolve(c, ldm, axes, n_ft):
    """Sum over the nodes of rfft(row) x folded Voigt transform, one irfft, / dv."""
    lg0, dxG, NG, ll0, dxL, NL = axes
    f = torch.arange(n_ft // 2 + 1, dtype=torch.float64, device=DEV) / (n_ft * c["dv"])
    h = 0.5 / c["dv"]
    acc = torch.zeros(n_ft // 2 + 1, dtype=torch.complex128, device=DEV)
    for node in range(NG * NL):
        wG, wL = math.exp(lg0 + node // NL * dxG), math.exp(ll0 + node % NL * dxL)

        def V(g):
            if torch.is_tensor(g):
                return torch.exp(-(math.pi * wG * g) ** 2 / (4 * LN2) - math.pi * wL * g)
            return math.exp(-(math.pi * wG * g) ** 2 / (4 * LN2) - math.pi * wL * g)

        prof, k = V(f), 1
        while V(k * h) >= 1e-6:
            prof = prof + V(k * h + (f.flip(0) if k & 1 else f))
            k += 1
        acc += torch.fft.rfft(ldm[node], n=n_ft) * (prof / prof[0])
    return torch.fft.irfft(acc, n=n_ft)[:c["n_v"]] / c["dv"]


def _exact_setup(c, d, T, p, x, q, masses, window=False):
    axes = _axes(c, d, T, p, x, masses, window)
    dens = p * 1e5 / (KB * T) * 1e-6 * x
    lnS = torch.log(d["S_ref"]) - torch.log(-torch.expm1(-C2 * d["v0"] / TREF)) - C2 * d["El"].double() * (1 / T - 1 / TREF)
    ls = float(lnS.max()) + math.log(dens) + max(math.log(v) for v in q)
    head = ls + math.log(d["v0"].numel() / c["dv"])
    return axes, ls, 0.0 if head < 85.0 and ls > -60.0 else ls


def _exact_spectrum(c, d, T, p, x, q, masses, window=False):
    """(abscoeff exp(-log_scale), log_scale)."""
    axes, ls, ls_out = _exact_setup(c, d, T, p, x, q, masses, window)
    ldm = _exact_ldm(c, d, T, p, x, axes, masses, q, ls)
    return _exact_convolve(c, ldm, axes, _ft_length(c["n_v"])) * math.exp(ls - ls_out), ls_out


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "slit":
        I, s = _spectrum_in(c, seed).double(), torch.from_numpy(_slit(c)).to(DEV).double()
        n, m = c["n_v"], int(c["taps"])
        full = torch.fft.irfft(torch.fft.rfft(I, n=n + m) * torch.fft.rfft(s, n=n + m), n=n + m) * c["dv"]
        out = full[(m - 1) // 2:(m - 1) // 2 + n].clone()
        if c["valid"]:
            la = min(n, m)
            out[:(la - 1) // 2] = math.nan
            out[n - la // 2:] = math.nan
        return out
    if kind == "served":
        lists = _served_lists(c)
        cols = {k: _make_lines(e, seed, i) for i, (k, e) in enumerate(lists.items())}
        spectra, scale = [], []
        for r in _served_requests(c):
            e = dict(lists[r["list"]], **{k: r[k] for k in ("vmin", "dv", "n_v")})
            A, ls = _exact_spectrum(e, cols[r["list"]], r["T"], r["p"], r["x"], [1.0], _masses(e), window=True)
            spectra.append(A)
            scale.append(ls)
        return {"spectra": spectra, "log_scale": scale}
    d = _make_lines(c, seed)
    T, p, x = c["T"], c["p"], c["x"]
    if kind == "adjoint":   # the conditions as the FP32 tensors hold them
        T, p, x = (float(np.float32(v)) for v in (T, p, x))
    masses = _masses(c)
    with_q = c["n_iso"] > 1 or kind in ("adjoint", "jacobian", "iterate")
    power = [Q_POWER + 0.1 * i for i in range(c["n_iso"])]
    q = [(TREF / T) ** k if with_q else 1.0 for k in power]
    if kind in ("spectrum", "quantities", "iterate"):
        A, ls = _exact_spectrum(c, d, T, p, x, q, masses)
        if kind == "spectrum":
            return {"abscoeff": A, "log_scale": ls}
        tau = A * math.exp(ls) * c["path"]
        eps = -torch.expm1(-tau)
        nu = c["vmin"] + c["dv"] * torch.arange(c["n_v"], dtype=torch.float64, device=DEV)
        lam = 0.01 / nu
        h, cl = 6.62607015e-34, 2.99792458e8
        planck = 2 * h * cl ** 2 / lam ** 5 / torch.expm1(C2 / T * nu) * 1e-10
        rows = [A, A * c["path"], eps, 1.0 - eps, eps * planck]
        if kind == "quantities":
            return {"rows": rows, "log_scale": ls}
        rows[:2] = [r * math.exp(ls) for r in rows[:2]]
        return dict(zip(gpuApp.QUANTITIES, (r.cpu().numpy() for r in rows)))
    dlnq = np.array([-k / T for k in power])
    axes, ls, _ = _exact_setup(c, d, T, p, x, q, masses)
    n_ft = _ft_length(c["n_v"])
    cols = []
    for th in (None, 0, 1, 2):
        ldm = _exact_ldm(c, d, T, p, x, axes, masses, q, ls, th, dlnq)
        cols.append(_exact_convolve(c, ldm, axes, n_ft) * math.exp(ls))
    if kind == "jacobian":
        return tuple(cols)
    w = _weights(c, seed).double()
    return {"absorbance": cols[0] * c["path"], "grad": tuple(torch.dot(w, v) * c["path"] for v in cols[1:])}
