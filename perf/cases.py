"""The work this package is measured on: whole advances through the public entry points.

Every case advances seeded relativistic-MHD boxes.  Three forms of use are covered:

* "box"      -- an application that keeps its states on the GPU: the primitives go in with
               Solver.upload_device, a few steps are enqueued with advance_async, the outcome
               (failed zones, MaxLambda) and the primitives are read back on the device;
* "ensemble" -- a parameter study: uneven 2D boxes advanced together by one Ensemble;
* "host"     -- the reference's driver loop, Mara.advance(buf, dt) on a host buffer.

A single-precision ("fp32") box hands its snapshots on in 32 bits, the precision its
primitives are kept in.
"""
import ctypes
import math

import numpy as np
import torch

from ctf_b200.ensemble import Ensemble
from ctf_b200.mara import MaraModule, Scheme, Solver

NG = 3
GAMMA = 4.0 / 3.0
THETA = 2.0
CFL = 0.3        # of the cell width: the signal speed never exceeds 1


def _box(n, extrap, riemann, advance, precision, layout="standard", learned=False, godunov="plm-split", steps=1, name=None):
    c = {"kind": "box", "n0": n[0], "n1": n[1], "n2": n[2] if len(n) > 2 else 0, "extrap": extrap, "riemann": riemann,
         "advance": advance, "precision": precision, "layout": layout, "learned": learned, "godunov": godunov,
         "steps": steps}
    if name:
        c["name"] = name
    return c


def listed():
    def named(c, name):
        return dict(c, name=name)
    return [
        # the smallest box of the tests and the smoke check: every launch counts
        _box((16, 16, 16), "plm", "hlld", "rk2", "fp64", steps=2, name="box16_fp64"),
        # a 2D parameter run at odd sizes in the parity precision
        _box((97, 130), "weno5", "hlld", "rk3", "fp64", steps=2, name="box97x130_fp64"),
        # a ragged small 3D box in the lean FP32 layout
        _box((47, 61, 53), "weno5", "hlld", "rk3", "fp32", layout="lean", steps=2, name="box47x61x53_lean_fp32"),
        # the 64^3 turbulence box the reference's parity is stated on
        _box((64, 64, 64), "plm", "hlld", "rk2", "fp64", steps=2, name="turb64_fp64"),
        # the driven-turbulence driver's operator (CTU-Hancock, single step)
        _box((72, 64, 80), "plm", "hlld", "single", "fp64", godunov="plm-muscl", name="ctu72x64x80_fp64"),
        # FP32 bulk with stored fluxes (the layout that diffuses and keeps a failure mask)
        _box((96, 101, 90), "plm", "hlld", "rk2", "fp32", name="box96x101x90_std_fp32"),
        # plain FP64 at a production resolution
        _box((128, 128, 128), "weno5", "hlld", "rk3", "fp64", name="turb128_fp64"),
        # 256^3 turbulence with the learned c2p guess (the headline configuration at 256^3)
        _box((256, 256, 256), "weno5", "hlld", "rk3", "fp32", layout="lean", learned=True, name="turb256_lean_learned"),
        # the headline size: 512^3 PLM + HLLD + RK3, FP32 bulk
        _box((512, 512, 512), "plm", "hlld", "rk3", "fp32", layout="lean", name="turb512_lean_fp32"),
        # a parameter study of 2D Kelvin-Helmholtz layers, sides log-uniform in 64..512
        named({"kind": "ensemble", "boxes": 40, "lo": 64, "hi": 512, "extrap": "plm", "riemann": "hllc", "advance": "rk3",
               "precision": "fp32", "steps": 2}, "kh_ensemble40_fp32"),
        # the reference's driver loop with its default scheme: Mara.advance on a pageable buffer
        named({"kind": "host", "n0": 64, "n1": 64, "n2": 64, "extrap": "plm", "riemann": "hlld", "advance": "rk2",
               "precision": "fp64", "layout": "standard", "pinned": False}, "host64_fp64"),
        # the same loop on a pinned buffer of a larger lean box, where the copies are pipelined
        named({"kind": "host", "n0": 160, "n1": 144, "n2": 152, "extrap": "plm", "riemann": "hlld", "advance": "rk3",
               "precision": "fp32", "layout": "lean", "pinned": True}, "host160x144x152_lean_fp32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lean", "lean", "lean", "std32", "fp64", "fp64", "flat", "ctu", "ensemble", "host"])
    extrap, rk = rng.choice(["plm", "weno5"]), rng.choice(["rk2", "rk3"])

    def sides(lo, hi, nd=3):
        n = _log(rng, lo, hi)
        return tuple(max(12, int(round(n * rng.uniform(0.8, 1.2)))) for _ in range(nd))
    if kind == "lean":
        return _box(sides(24, 320), extrap, "hlld", rk, "fp32", layout="lean", learned=rng.random() < 0.25,
                    steps=rng.choice([1, 2]))
    if kind == "std32":
        return _box(sides(24, 200), extrap, "hlld", rng.choice(["rk2", "rk3", "rk4"]), "fp32", steps=rng.choice([1, 2]))
    if kind == "fp64":
        return _box(sides(14, 150), extrap, "hlld", rk, "fp64", layout=rng.choice(["standard", "standard", "lean"]),
                    steps=rng.choice([1, 2]))
    if kind == "flat":
        return _box(sides(48, 700, 2), extrap, rng.choice(["hlld", "hlld", "hll"]), rk, rng.choice(["fp64", "fp32"]),
                    steps=rng.choice([1, 2, 4]))
    if kind == "ctu":
        return _box(sides(20, 110), "plm", "hlld", "single", "fp64", godunov="plm-muscl", steps=rng.choice([1, 2]))
    if kind == "ensemble":
        return {"kind": "ensemble", "boxes": rng.randint(4, 60), "lo": rng.choice([32, 64]), "hi": rng.choice([256, 512]),
                "extrap": extrap, "riemann": "hllc", "advance": rk, "precision": "fp32", "steps": rng.choice([1, 2, 4])}
    lean = rng.random() < 0.5
    n = sides(48, 200) if lean else sides(16, 100)
    return {"kind": "host", "n0": n[0], "n1": n[1], "n2": n[2], "extrap": extrap, "riemann": "hlld", "advance": rk,
            "precision": "fp32" if lean else "fp64", "layout": "lean" if lean else "standard",
            "pinned": lean and rng.random() < 0.5}


# ---- inputs ---------------------------------------------------------------------------------------
def _sizes(case):
    return tuple(case[k] for k in ("n0", "n1", "n2") if case.get(k))


def _ensemble_sizes(case):
    """Square boxes with sides log-uniform in lo..hi, the same for every seed of a case."""
    rng = np.random.default_rng(12345)
    sides = np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), case["boxes"]))
    return [(int(s), int(s) + 8 * int(k)) for s, k in zip(sides, rng.integers(0, 3, case["boxes"]))]


def _modes(rng, nd, kmax=4):
    """Complex amplitudes of the wave vectors 0 < |k| <= kmax, power ~ |k|^-2 per mode."""
    k = np.arange(-kmax, kmax + 1)
    K = np.meshgrid(*([k] * nd), indexing="ij")
    kk = np.sqrt(sum(x.astype(float) ** 2 for x in K))
    amp = np.where((kk >= 1) & (kk <= kmax), 1.0 / np.maximum(kk, 1), 0.0)
    return (rng.standard_normal(kk.shape) + 1j * rng.standard_normal(kk.shape)) * amp, K


def _field(coef, n, device):
    """The real field of those modes on the n-grid (a Fourier sum, one axis at a time)."""
    k = torch.arange(-4, 5, dtype=torch.float64, device=device)
    out = torch.from_numpy(coef).to(device)
    for m in n:
        x = torch.arange(m, dtype=torch.float64, device=device) / m
        out = torch.tensordot(out, torch.exp(2j * math.pi * k[:, None] * x[None, :]), dims=([0], [0]))
    return out.real


def _rms(*f):
    return torch.sqrt(sum((x * x).mean() for x in f))


def _guarded(P, n):
    """(8, n...) interior primitives -> the reference's AoS array with periodic guard zones."""
    for d in range(len(n)):
        i = torch.arange(-NG, n[d] + NG, device=P.device) % n[d]
        P = P.index_select(d + 1, i)
    P = P.reshape((8,) + tuple(P.shape[1:]) + (1,) * (3 - len(n)))
    return P.permute(1, 2, 3, 0).contiguous()


def _turbulence(n, seed, device):
    """Decaying-turbulence state: velocity rms 0.3 below 0.9, a unit mean field plus a solenoidal
    perturbation of rms 0.1 (free of the corner divergence flux-CT keeps), and density and
    pressure fluctuations as the flow develops them."""
    rng, nd = np.random.default_rng(seed), len(n)
    P = torch.zeros((8,) + n, dtype=torch.float64, device=device)
    for q in (0, 1):
        f = _field(_modes(rng, nd)[0], n, device)
        P[q] = torch.exp(0.15 * (f - f.mean()) / _rms(f))
    for q in range(3):
        P[2 + q] = _field(_modes(rng, nd)[0], n, device)
    P[2:5] *= 0.3 / _rms(*P[2:5])
    speed = torch.sqrt((P[2:5] ** 2).sum(0))
    P[2:5] *= torch.where(speed > 0.9, 0.9 / speed, torch.ones_like(speed))
    C, K = [], None
    for _ in range(nd):
        c, K = _modes(rng, nd)
        C.append(c)
    sn = [np.sin(math.pi * K[d] / n[d]) for d in range(nd)]
    cs = [np.cos(math.pi * K[d] / n[d]) for d in range(nd)]
    # the unit box's cells may not be cubes: weight each direction by its resolution
    D = [sn[d] * n[d] * np.prod([cs[e] for e in range(nd) if e != d], axis=0) for d in range(nd)]
    dot, norm = sum(D[d] * C[d] for d in range(nd)), sum(x * x for x in D)
    for d in range(nd):
        P[5 + d] = _field(C[d] - np.where(norm > 0, D[d] * dot / np.where(norm > 0, norm, 1.0), 0.0), n, device)
    P[5:5 + nd] *= 0.1 / _rms(*P[5:5 + nd])
    P[7 if nd == 3 else 5] += 1.0
    return _guarded(P, n)


def _kelvin_helmholtz(n, seed, device):
    """Two shear layers (density 1 and 2, v = 0.25, thin interfaces) with seeded perturbations."""
    rng = np.random.default_rng(seed)
    x = ((torch.arange(n[0], dtype=torch.float64, device=device) + 0.5) / n[0])[:, None]
    y = ((torch.arange(n[1], dtype=torch.float64, device=device) + 0.5) / n[1])[None, :]
    prof = torch.tanh((y - 0.25) / 0.03) - torch.tanh((y - 0.75) / 0.03) - 1.0 + 0 * x
    phase, kick = rng.uniform(0, 2 * math.pi, 4), rng.uniform(0.5, 1.5)
    wave = sum(torch.sin(2 * math.pi * (m + 1) * x + phase[m]) for m in range(4)) / 4
    P = torch.zeros((8,) + n, dtype=torch.float64, device=device)
    P[0] = 1.0 + 0.5 * (1.0 - prof)
    P[1] = 1.0
    P[2] = 0.25 * prof
    P[3] = 0.01 * kick * wave * (torch.exp(-((y - 0.25) / 0.05) ** 2) + torch.exp(-((y - 0.75) / 0.05) ** 2))
    P[5] = 0.01
    return _guarded(P, n)


def _dt(n):
    return CFL / max(n)


def _scheme(case):
    return Scheme(gamma=GAMMA, theta=THETA, extrap=case["extrap"], riemann=case["riemann"], advance=case["advance"],
                  precision=case["precision"], layout=case.get("layout", "standard"),
                  learned_c2p=bool(case.get("learned")), godunov=case.get("godunov", "plm-split"))


def prepare(case, seed):
    if case["kind"] == "host":
        n = _sizes(case)
        P = _turbulence(n, seed, "cuda").cpu()
        P = (P.pin_memory() if case["pinned"] else P).numpy()
        if case["layout"] == "lean":
            return {"kind": "host", "prim": P, "dt": _dt(n), "mara": None, "solver": Solver(_scheme(case), n)}
        m = MaraModule()
        m.start()
        m.set_fluid("rmhd")
        m.set_eos("gamma-law", GAMMA)
        m.set_boundary("periodic")
        m.set_riemann(case["riemann"])
        m.set_godunov("plm-split")
        m.set_advance(case["advance"])
        m.config_solver({"extrap": case["extrap"], "theta": THETA, "precision": case["precision"]}, quiet=True)
        m.set_domain((0.0,) * 3, (1.0,) * 3, n)
        m.set_primitive(P)
        return {"kind": "host", "prim": P, "dt": _dt(n), "mara": m, "solver": None}
    stream = torch.cuda.Stream()
    if case["kind"] == "ensemble":
        sizes = _ensemble_sizes(case)
        E = Ensemble(_scheme(case), sizes)
        E.set_stream(stream.cuda_stream)
        prim = [_kelvin_helmholtz(n, 1000 * seed + b, "cuda") for b, n in enumerate(sizes)]
        return {"kind": "ensemble", "ensemble": E, "stream": stream, "prim": prim, "steps": case["steps"],
                "out": [torch.empty_like(p) for p in prim],
                "snap": [torch.empty_like(p, dtype=torch.float32) for p in prim], "dt": [_dt(n) for n in sizes]}
    n = _sizes(case)
    s = Solver(_scheme(case), n, stream=stream.cuda_stream)
    if case["learned"]:
        from ctf_b200.train_c2p import load
        s.set_c2p_network(load())
    P = _turbulence(n, seed, "cuda")
    return {"kind": "box", "solver": s, "stream": stream, "prim": P, "out": torch.empty_like(P), "steps": case["steps"],
            "snap": torch.empty_like(P, dtype=torch.float32) if case["precision"] == "fp32" else None, "dt": _dt(n)}


def run(state):
    if state["kind"] == "host":
        who = state["mara"]
        _, errors = who.advance(state["prim"], state["dt"]) if who else state["solver"].advance_host(state["prim"], state["dt"])
        return {"prim": state["prim"], "errors": errors}
    if state["kind"] == "ensemble":
        E, lib = state["ensemble"], state["ensemble"].lib
        for b, p in enumerate(state["prim"]):
            E._check(lib.mgpu_ensemble_upload_prim_device(E.h, b, ctypes.c_void_p(p.data_ptr())))
        E.advance(dt=state["dt"], nsteps=state["steps"])
        for b, p in enumerate(state["out"]):
            E._check(lib.mgpu_ensemble_download_prim_device(E.h, b, ctypes.c_void_p(p.data_ptr())))
        with torch.cuda.stream(state["stream"]):
            for p, q in zip(state["out"], state["snap"]):
                q.copy_(p)
        return {"prim": state["snap"], "errors": E.errors()}
    s = state["solver"]
    s.upload_device(state["prim"].data_ptr())
    s.advance_async(state["steps"], dt=state["dt"])
    s.download_device(state["out"].data_ptr())
    out = state["out"]
    if state["snap"] is not None:
        with torch.cuda.stream(state["stream"]):
            out = state["snap"].copy_(out)
    st = s.stats()
    if state["snap"] is not None:   # FP32 wave speeds carry the quartic's rounding (up to 6% of the
        return {"prim": out, "errors": st["errors"]}   # largest one): nothing to hold to a bound
    return {"prim": out, "errors": st["errors"], "max_lambda": st["max_lambda"]}


STAGES = {"single": 1, "rk2": 2, "rk3": 3, "rk4": 4}


def work(case):
    """Each primitive array in and out once; floating-point operations of one zone's share of a
    stage: reconstruction and Riemann solve per face (two passes of faces and a predictor
    inversion per direction under CTU-Hancock), one inversion, the update."""
    boxes = _ensemble_sizes(case) if case["kind"] == "ensemble" else [_sizes(case)]
    nd = len(boxes[0])
    face = {"plm": 160, "weno5": 900}[case["extrap"]] + {"hll": 350, "hllc": 450, "hlld": 1100}[case["riemann"]]
    ctu = case.get("godunov") == "plm-muscl"
    zone = (2 if ctu else 1) * nd * face + (nd + 1 if ctu else 1) * 400 + 150
    size = 4 if case["precision"] == "fp32" and case["kind"] != "host" else 8
    guarded = sum(math.prod(m + 2 * NG for m in n) for n in boxes)
    zones = sum(math.prod(n) for n in boxes)
    return {"bytes": guarded * 8 * (8 + size), "flops": zones * zone * STAGES[case["advance"]] * case.get("steps", 1)}


# ---- the same advances in plain 64-bit torch ---------------------------------------------------------
# Component lists of flattened guarded arrays: rho p vx vy vz Bx By Bz, or D tau Sx Sy Sz Bx By Bz.
def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _to_cons(P):
    r, p, v, B = P[0], P[1], P[2:5], P[5:8]
    W2 = 1 / (1 - _dot(v, v))
    vB, B2 = _dot(v, B), _dot(B, B)
    w = (r + GAMMA / (GAMMA - 1) * p) * W2 + B2                # total enthalpy times W^2, lab frame
    D = r * torch.sqrt(W2)
    tau = w - p - 0.5 * (B2 / W2 + vB * vB) - D
    return [D, tau] + [w * v[i] - vB * B[i] for i in range(3)] + list(B)


def _to_prim(U):
    """Primitives by Newton's method in (Z, W); None of the measured states needs a second try."""
    D, tau, S, B = U[0], U[1], U[2:5], U[5:8]
    S2, B2, SB = _dot(S, S), _dot(B, B), _dot(S, B)
    g = (GAMMA - 1) / GAMMA
    Z = torch.sqrt(S2 + D * D)
    W = Z / D
    for _ in range(60):
        T2 = SB * SB / (Z * Z)
        f = (Z + B2) ** 2 * (1 - 1 / (W * W)) - (2 * Z + B2) * T2 - S2
        h = Z + B2 - g * (Z / (W * W) - D / W) - 0.5 * B2 / (W * W) - 0.5 * T2 - D - tau
        fZ = 2 * (Z + B2) * (1 - 1 / (W * W)) - 2 * T2 + 2 * (2 * Z + B2) * T2 / Z
        fW = 2 * (Z + B2) ** 2 / W ** 3
        hZ = 1 - g / (W * W) + T2 / Z
        hW = -g * (D / (W * W) - 2 * Z / W ** 3) + B2 / W ** 3
        det = fZ * hW - fW * hZ
        dZ, dW = -(hW * f - fW * h) / det, -(fZ * h - hZ * f) / det
        Z, W = torch.abs(Z + dZ), torch.clamp(W + dW, min=1.0)
        if not bool(((dZ / Z).abs() + (dW / W).abs() > 1e-14).any()):
            break
    vB = SB / Z
    return [D / W, g * (Z / (W * W) - D / W)] + [(S[i] + vB * B[i]) / (Z + B2) for i in range(3)] + list(B)


def _flux_x(P, U):
    r, p, v, B = P[0], P[1], P[2:5], P[5:8]
    W2 = 1 / (1 - _dot(v, v))
    vB = _dot(v, B)
    pt = p + 0.5 * (_dot(B, B) / W2 + vB * vB)
    b = [B[i] / W2 + vB * v[i] for i in range(3)]              # b^i / W
    F = [U[0] * v[0], U[1] * v[0] - vB * B[0] + pt * v[0]]
    F += [U[2 + i] * v[0] - b[i] * B[0] for i in range(3)]
    F[2] = F[2] + pt
    return F + [torch.zeros_like(r), v[0] * B[1] - v[1] * B[0], v[0] * B[2] - v[2] * B[0]]


def _speeds_x(P):
    """Fast magnetosonic speeds: Newton's method down to the extreme roots of the quartic."""
    r, p, v, B = P[0], P[1], P[2:5], P[5:8]
    W2 = 1 / (1 - _dot(v, v))
    W = torch.sqrt(W2)
    vB, B2 = _dot(v, B), _dot(B, B)
    b0, b2 = W * vB, B2 / W2 + vB * vB
    bx = B[0] / W + b0 * v[0]
    rh = r + GAMMA / (GAMMA - 1) * p
    cs2 = GAMMA * p / rh
    K, L, x = rh * (1 / cs2 - 1) * W2 * W2, -(rh + b2 / cs2) * W2, v[0]
    a = [K - L - b0 * b0, -4 * K * x + 2 * L * x + 2 * b0 * bx, 6 * K * x * x + L * (1 - x * x) + b0 * b0 - bx * bx,
         -4 * K * x ** 3 - 2 * L * x - 2 * b0 * bx, K * x ** 4 + L * x * x + bx * bx]
    out = []
    for start in (1.0, -1.0):
        t = torch.full_like(r, start)
        for _ in range(60):
            f = (((a[0] * t + a[1]) * t + a[2]) * t + a[3]) * t + a[4]
            d = ((4 * a[0] * t + 3 * a[1]) * t + 2 * a[2]) * t + a[3]
            s = f / d
            t = t - s
            if not bool((s.abs() > 1e-15).any()):
                break
        out.append(t)
    return out


def _hll(L, R, UL, UR, FL, FR, ap, am):
    U = [(ap * UR[i] - am * UL[i] + FL[i] - FR[i]) / (ap - am) for i in range(8)]
    F = [(ap * FL[i] - am * FR[i] + ap * am * (UR[i] - UL[i])) / (ap - am) for i in range(8)]
    return U, F


def _pick(ap, am, mid, FL, FR):
    return [torch.where(am >= 0, FL[i], torch.where(ap < 0, FR[i], mid[i])) for i in range(8)]


def _hllc(L, R, UL, UR, FL, FR, ap, am):
    """Mignone & Bodo (2006); total energies."""
    U, F = _hll(L, R, UL, UR, FL, FR, ap, am)
    full = U[5].abs() > 1e-12
    bf = torch.where(full, U[6] * F[6] + U[7] * F[7], torch.zeros_like(ap))
    sq = torch.where(full, U[6] ** 2 + U[7] ** 2 + F[6] ** 2 + F[7] ** 2, torch.zeros_like(ap))
    a, b, c = F[1] - bf, -F[2] - U[1] + sq, U[2] - bf
    lin = a.abs() < 1e-10
    vs = torch.where(lin, -c / b, (-b - torch.sqrt(torch.clamp(b * b - 4 * a * c, min=0))) / (2 * torch.where(lin, torch.ones_like(a), a)))
    bx = torch.where(full, U[5], torch.ones_like(ap))
    v = [vs] + [torch.where(full, (U[k] * vs - F[k]) / bx, torch.zeros_like(ap)) for k in (6, 7)]
    B = [U[5], U[6], U[7]]
    vB, v2 = _dot(v, B), _dot(v, v)
    vB = torch.where(full, vB, torch.zeros_like(vB))
    b1 = torch.where(full, B[0], torch.zeros_like(vB))
    ps = F[2] + b1 * b1 * (1 - v2) - (F[1] - b1 * vB) * vs
    star = []
    for P, V, G, s in ((L, UL, FL, am), (R, UR, FR, ap)):
        k = 1 / (s - vs)
        D = (s - P[2]) * k * V[0]
        E = (s * V[1] - V[2] + ps * vs - vB * b1) * k
        Q = [D, E, (E + ps) * vs - vB * b1]
        for m in (1, 2):
            Q.append(torch.where(full, (-b1 * (B[m] * (1 - v2) + vB * v[m]) + s * V[2 + m] - G[2 + m]) * k, (s - P[2]) * k * V[2 + m]))
        Q.append(B[0])
        Q += [torch.where(full, B[m], (s - P[2]) * k * V[5 + m]) for m in (1, 2)]
        star.append([G[i] + s * (Q[i] - V[i]) for i in range(8)])
    return _pick(ap, am, [torch.where(vs >= 0, star[0][i], star[1][i]) for i in range(8)], FL, FR)


def _hlld_inner(q, p):
    """Mignone, Ugliano & Bodo (2009), eqs 23-45 at total pressure p: both sides' states."""
    out = []
    for J, lam, sign in ((q["JL"], q["am"], -1.0), (q["JR"], q["ap"], 1.0)):
        D, E, m, B, bx = J[0], J[1], J[2:5], J[5:8], q["bx"]
        A = m[0] - lam * E + p * (1 - lam * lam)
        G, C = B[1] ** 2 + B[2] ** 2, B[1] * m[1] + B[2] * m[2]
        Q = -A - G + bx * bx * (1 - lam * lam)
        X = bx * (A * lam * bx + C) - (A + G) * (lam * p + E)
        X = torch.where(X.abs() < 1e-8, torch.full_like(X, 1e-8), X)
        t = C + bx * (lam * m[0] - E)
        v = [(bx * (A * bx + lam * C) - (A + G) * (p + m[0])) / X, (Q * m[1] + B[1] * t) / X, (Q * m[2] + B[2] * t) / X]
        b = [(B[k] - bx * v[k]) / (lam - v[0]) for k in range(3)]
        w = p + (E - _dot(v, m)) / (lam - v[0])
        eta = sign * torch.sign(bx) * torch.sqrt(w.abs())
        den = lam * p + E + bx * eta
        Kv = [(m[0] + p + B[0] * eta) / den, (m[1] + B[1] * eta) / den, (m[2] + B[2] * eta) / den]
        out.append((v, b, w.abs(), eta, Kv))
    (vl, bl, wl, el, Kl), (vr, br, wr, er, Kr) = out
    dK = Kr[0] - Kl[0]
    flat = dK.abs() < 1e-10
    safe = torch.where(flat, torch.ones_like(dK), dK)
    Bc = [torch.where(flat, torch.zeros_like(dK), ((br[k] * (Kr[0] - vr[0]) + br[0] * vr[k]) - (bl[k] * (Kl[0] - vl[0]) + bl[0] * vl[k])) / safe)
          for k in range(3)]
    return out, Bc, dK, flat


def _hlld_residual(q, p):
    ((_, _, _, el, Kl), (_, _, _, er, Kr)), Bc, dK, flat = _hlld_inner(q, p)
    Y = [(1 - _dot(K, K)) / (e * dK - dK * _dot(K, Bc)) for K, e in ((Kl, el), (Kr, er))]
    y = torch.where(Bc[0].abs() < 1e-10, dK, dK * (1 - Bc[0] * (Y[1] - Y[0])))
    return torch.where(flat, torch.zeros_like(y), y)


def _hlld_flux(q, p):
    """The flux at x/t = 0 and whether the solution passes the solver's checks."""
    ((vl, bl, wl, el, Kl), (vr, br, wr, er, Kr)), Bc, dK, _ = _hlld_inner(q, p)
    c = []
    for K, e, v in ((Kl, el, vl), (Kr, er, vr)):
        den = e - _dot(K, Bc)
        small = den.abs() < 1e-10
        s = (1 - _dot(K, K)) / torch.where(small, torch.ones_like(den), den)
        c.append([torch.where(small, v[k], K[k] - Bc[k] * s) for k in range(3)])
    lc = c[1][0]
    am, ap = q["am"], q["ap"]
    ok = (p >= 0) & (Kl[0] >= -1) & (Kr[0] <= 1) & (lc.abs() <= 1) & (wl > p) & (wr > p)
    ok &= (vl[0] > am - 1e-14) & (c[0][0] > Kl[0] - 1e-14) & (vr[0] < ap + 1e-14) & (c[1][0] < Kr[0] + 1e-14)
    ok &= (c[1][0] - c[0][0]).abs() <= 1e-8
    left = lc >= 0

    def side(a, b):
        return torch.where(left, a, b)
    J = [side(x, y) for x, y in zip(q["JL"], q["JR"])]
    lam, K0 = side(am, ap), side(Kl[0], Kr[0])
    v, b, cv = [[side(x, y) for x, y in zip(a, e)] for a, e in ((vl, vr), (bl, br), (c[0], c[1]))]
    vb = _dot(v, b)
    den = lam - v[0]
    E = (J[1] + p * v[0] - vb * b[0]) / den
    a = [J[0] / den, E] + [(E + p) * v[k] - vb * b[k] for k in range(3)] + b
    vB = _dot(cv, Bc)
    den = K0 - lc
    near = den.abs() < 1e-8
    den = torch.where(near, torch.ones_like(den), den)
    E = (K0 * a[1] - a[2] + p * lc - vB * Bc[0]) / den
    u = [a[0] * (K0 - v[0]) / den, E] + [(E + p) * cv[k] - vB * Bc[k] for k in range(3)] + Bc
    u = [torch.where(near, a[i], u[i]) for i in range(8)]
    outer = [lam * side(q["UL"][i], q["UR"][i]) - J[i] for i in range(8)]
    Fa = [lam * a[i] - J[i] for i in range(8)]
    inner = torch.where(left, Kl[0] >= 0, Kr[0] < 0)
    F = [torch.where(inner, Fa[i], Fa[i] + K0 * (u[i] - a[i])) for i in range(8)]
    out = side(am >= 0, ap < 0)
    return [torch.where(out, outer[i], F[i]) for i in range(8)], ok


def _hlld(L, R, UL, UR, FL, FR, ap, am):
    U, F = _hll(L, R, UL, UR, FL, FR, ap, am)
    prim = _to_prim([U[0], U[1] - U[0]] + U[2:])
    vB = _dot(prim[2:5], prim[5:8])
    p0 = prim[1] + 0.5 * (_dot(prim[5:8], prim[5:8]) * (1 - _dot(prim[2:5], prim[2:5])) + vB * vB)
    b, c = U[1] - F[2], F[1] * U[2] - U[1] * F[2]
    root = torch.sqrt(torch.clamp(b * b - 4 * c, min=0))
    p1 = torch.minimum(((-b + root) / 2).abs(), ((-b - root) / 2).abs())
    q = {"am": am, "ap": ap, "bx": L[5], "UL": UL, "UR": UR, "JL": [am * UL[i] - FL[i] for i in range(8)],
         "JR": [ap * UR[i] - FR[i] for i in range(8)]}
    direct = L[5].abs() < 1e-8
    flux, done = None, torch.zeros_like(direct)
    for guess in (p0, p1, torch.zeros_like(p0)):
        p = torch.where(direct, p1, guess)
        go = ~(direct | done)
        for _ in range(16):
            y = _hlld_residual(q, p)
            jac = (_hlld_residual(q, p + 0.5e-8) - _hlld_residual(q, p - 0.5e-8)) / 1e-8
            p = torch.where(go, p - y / jac, p)
            go = go & (y.abs() > 1e-12)
            if not bool(go.any()):
                break
        f, ok = _hlld_flux(q, p)
        ok = ok & ~go & torch.isfinite(p)
        flux = f if flux is None else [torch.where(done, flux[i], f[i]) for i in range(8)]
        done = done | ok
        if bool(done.all()):
            break
    if not bool(done.all()):
        rest = _hllc(L, R, UL, UR, FL, FR, ap, am)
        flux = [torch.where(done, flux[i], rest[i]) for i in range(8)]
    return flux


def _plm(a, b, c):
    x, y, z = THETA * (b - a), 0.5 * (c - a), THETA * (c - b)
    lo = torch.minimum(torch.minimum(x.abs(), y.abs()), z.abs())
    s = (torch.sign(x) + torch.sign(y)).abs() * (torch.sign(x) + torch.sign(z)) * 0.25
    return s * lo


def _weno(a, b, c, d, e):
    """Fifth-order WENO (Jiang & Shu) to the face between c and d, point-value tables."""
    t = [3 / 8 * c + 3 / 4 * d - 1 / 8 * e, -1 / 8 * b + 3 / 4 * c + 3 / 8 * d, 3 / 8 * a - 5 / 4 * b + 15 / 8 * c]
    i = [13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2,
         13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2,
         13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2]
    w = [g / (1e-6 + s) ** 2 for g, s in zip((5 / 16, 5 / 8, 1 / 16), i)]
    return sum(x * y for x, y in zip(w, t)) / sum(w)


PIECE = 4 << 20   # faces solved at a time


def _sweep(A, S, dim, case, keep):
    """Fluxes (8, nz) of one direction over the flattened guarded array, and the largest speed."""
    nz = A.shape[1]
    m = [0, 1] + [2 + (dim + k) % 3 for k in range(3)] + [5 + (dim + k) % 3 for k in range(3)]
    F, top = torch.zeros_like(A), 0.0
    for f0 in range(2 * S, nz - 3 * S, PIECE):
        f1 = min(f0 + PIECE, nz - 3 * S)

        def at(k, q):
            return A[q, f0 + k * S:f1 + k * S]
        if case["extrap"] == "plm":
            L = [at(0, q) + 0.5 * _plm(at(-1, q), at(0, q), at(1, q)) for q in m]
            R = [at(1, q) - 0.5 * _plm(at(0, q), at(1, q), at(2, q)) for q in m]
        else:
            L = [_weno(*(at(k, q) for k in (-2, -1, 0, 1, 2))) for q in m]
            R = [_weno(*(at(k, q) for k in (3, 2, 1, 0, -1))) for q in m]
        if case["riemann"] != "hll":
            L[5] = R[5] = 0.5 * (L[5] + R[5])
        UL, UR = _to_cons(L), _to_cons(R)
        FL, FR = _flux_x(L, UL), _flux_x(R, UR)
        (pl, ml), (pr, mr) = _speeds_x(L), _speeds_x(R)
        ap, am = torch.maximum(pl, pr), torch.minimum(ml, mr)
        lam = torch.maximum(ap.abs(), am.abs())
        top = max(top, float((lam if keep is None else torch.where(keep[dim][f0:f1], lam, torch.zeros_like(lam))).max()))
        if case["riemann"] == "hll":
            out = _pick(ap, am, _hll(L, R, UL, UR, FL, FR, ap, am)[1], FL, FR)
        else:
            for a in (UL, UR, FL, FR):
                a[1] = a[1] + a[0]
            out = (_hllc if case["riemann"] == "hllc" else _hlld)(L, R, UL, UR, FL, FR, ap, am)
            out[1] = out[1] - out[0]
        for k, q in enumerate(m):
            F[q, f0:f1] = out[k]
    return F, top


def _emf(F, G, sa, sb):
    """Eight-point average of the transverse field fluxes (flux-CT): F along sa, G along sb."""
    def r(x, k):
        return torch.roll(x, -k)
    return (2 * F + r(F, sb) + r(F, -sb) - G - r(G, sa) - r(G, -sb) - r(G, sa - sb)) / 8


def _advance(P, case, n, dt):
    """One advance of the flattened guarded primitives P (8, nz); (P, MaxLambda)."""
    nd = len(n)
    G = [m + 2 * NG for m in n]
    strides = [math.prod(G[d + 1:]) for d in range(nd)]
    inner = (slice(None),) + (slice(NG, -NG),) * nd

    def fill(U):
        for d in range(nd):
            U = U.index_select(d + 1, torch.arange(-NG, n[d] + NG, device=U.device) % n[d])
        return U.reshape(8, -1)

    def prims(U):
        flat = U.reshape(8, -1)
        parts = [torch.stack(_to_prim(list(flat[:, i:i + PIECE]))) for i in range(0, flat.shape[1], PIECE)]
        return fill(torch.cat(parts, 1).reshape(U.shape))

    keep = None
    if case.get("layout") == "lean":   # that layout's faces: interior rows and one row of halo
        keep = []
        for d in range(nd):
            k = torch.ones([1] * nd, dtype=torch.bool, device=P.device)
            for e in range(nd):
                x = torch.arange(G[e], device=P.device)
                k = k & ((x >= NG - 1) & (x < NG + n[e] + (e != d))).reshape([-1 if i == e else 1 for i in range(nd)])
            keep.append(k.reshape(-1))
    top = 0.0

    def rate(U):
        nonlocal top
        A = prims(U)
        F = []
        for d in range(nd):
            f, t = _sweep(A, strides[d], d, case, keep)
            F.append(f)
            top = max(top, t)
        if nd > 1:
            E = {(d, e): _emf(F[d][5 + e], F[e][5 + d], strides[d], strides[e]) for d in range(nd) for e in range(nd) if d != e}
            for (d, e), x in E.items():
                F[d][5 + e] = x
            for d in range(nd):
                F[d][5 + d] = 0
        L = 0
        for d in range(nd):
            L = L - (F[d] - torch.roll(F[d], strides[d], 1)) * n[d]
        return L.reshape([8] + G)[inner]

    U = torch.stack(_to_cons(list(P))).reshape([8] + G)[inner]
    how = case["advance"]
    if how == "rk2":
        V = U + dt * rate(U)
        U = 0.5 * (U + V + dt * rate(V))
    elif how == "rk3":
        V = U + dt * rate(U)
        V = 0.75 * U + 0.25 * (V + dt * rate(V))
        U = (U + 2 * (V + dt * rate(V))) / 3
    elif how == "rk4":
        a = dt * rate(U)
        b = dt * rate(U + 0.5 * a)
        c = dt * rate(U + 0.5 * b)
        U = U + (a + 2 * b + 2 * c + dt * rate(U + c)) / 6
    else:
        U = U + dt * rate(U)
    return prims(U), top


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    steps = case.get("steps", 1)
    if case.get("godunov", "plm-split") != "plm-split":
        return None   # the predictor-corrector operator has no plain restatement here
    boxes = _ensemble_sizes(case) if case["kind"] == "ensemble" else [_sizes(case)]
    if sum(math.prod(n) for n in boxes) * steps > 2e7:
        return None   # too long, or too large for the temporaries
    out, top = [], 0.0
    for b, n in enumerate(boxes):
        P = _kelvin_helmholtz(n, 1000 * seed + b, dev) if case["kind"] == "ensemble" else _turbulence(n, seed, dev)
        shape = P.shape
        P = P.reshape(-1, 8).t().contiguous()
        for _ in range(steps):
            P, top = _advance(P, case, n, _dt(n))
        out.append(P.t().reshape(shape).contiguous())
    if case["kind"] == "ensemble":
        return {"prim": out, "errors": None}
    known = case["kind"] == "box" and case["precision"] == "fp64"
    return {"prim": out[0], "errors": None} | ({"max_lambda": top} if known else {})
