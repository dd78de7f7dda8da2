"""Timing cases of the operator-split step: what a run of this framework spends its time on.

Each case is one call (or one short sequence of calls) of the public entry points on seeded
inputs of ``verb4d_b200.workload``: whole steps, single phases, the assimilation updates and
the per-slice operators.  ``exact`` gives the same results from plain torch in 64 bits,
written from the equations, without this package's kernels.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

# the package lives one folder below the repository's root, the working folder
_PKG = os.path.join(os.getcwd(), "verb-4d_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from verb4d_b200 import Context, _lib, ops  # noqa: E402
from verb4d_b200 import workload as W  # noqa: E402

FIELDS = ("psd", "Pg", "Rg", "Vg", "Kg", "Lg", "DLL", "DVV", "DKK", "DVK", "VP", "VR", "G_local",
          "G_radial", "G_conv", "S", "loss_local", "loss_radial", "loss_conv")
# assimilation: model and observation error of the radial and the (MLT, L) filter
KF_RADIAL = (1e-4, 1e-3)
KF_CONV = (1e-3, 1e-2)


def listed():
    return [
        # one local (E, alpha) system and one (MLT, L) slice on host arrays: what a program
        # linked against the per-slice operators calls, where latency and launches count
        dict(name="slice_local_31x31", op="slice_local", P=1, R=1, V=31, K=31, kp=3.0),
        dict(name="slice_conv_24x25", op="slice_conv", P=24, R=25, V=1, K=1, kp=3.0),
        # a time step of the workstation-size run (24 MLT x 25 L x 31 E x 31 alpha), default
        # arithmetic, with the negative count that the driver's log prints
        dict(name="step_24x25x31x31", op="step", P=24, R=25, V=31, K=31, kp=3.0, arith="exact"),
        # a time step at the production resolution in MLT, L and E (8 pitch angles, so that the
        # local factors of several runs fit one GPU), default arithmetic
        dict(name="step_48x101x101x8", op="step", P=48, R=101, V=101, K=8, kp=4.0, arith="exact"),
        # the convection phase in the arithmetic long runs use, workstation and production slices
        dict(name="conv_24x25x31x31", op="conv", P=24, R=25, V=31, K=31, kp=3.0, arith="stream"),
        dict(name="conv_48x101x101x16", op="conv", P=48, R=101, V=101, K=16, kp=4.0,
             arith="stream"),
        # the local phase with cached factors: every step between two coefficient updates
        dict(name="local_48x101x101x12", op="local", P=48, R=101, V=101, K=12, kp=3.0,
             prec="fp64"),
        # the local phase after an update of its coefficients (an hourly wave-model table):
        # upload, factorise, solve; FP64 factors at the production band, and the mixed form
        # (FP32 factors, two refinement steps) at the workstation size
        dict(name="newcoef_24x51x101x21", op="newcoef", P=24, R=51, V=101, K=21, kp=3.0,
             prec="fp64"),
        dict(name="newcoef_mixed_24x25x31x31", op="newcoef", P=24, R=25, V=31, K=31, kp=3.0,
             prec="mixed"),
        # the radial phase of a step at which Kp changed: new D_LL scale, factors and solve
        dict(name="radial_48x101x101x16", op="radial", P=48, R=101, V=101, K=16, kp=3.0),
        # hourly assimilation: the radial filter at one MLT, the (MLT, L) filter on every slice
        dict(name="kf_radial_48x101x31x31", op="kf_radial", P=48, R=101, V=31, K=31, kp=3.0),
        dict(name="kf_conv_24x25x11x11", op="kf_conv", P=24, R=25, V=11, K=11, kp=3.0),
    ]


# the ranges the listed cases stand for: grid sizes and the largest work of one drawn case
_RANGES = {
    "slice_local": dict(P=(1, 1), R=(1, 1), V=(9, 101), K=(9, 31)),
    "slice_conv": dict(P=(12, 48), R=(13, 101), V=(1, 1), K=(1, 1)),
    "step": dict(P=(12, 48), R=(13, 101), V=(11, 101), K=(8, 45)),
    "conv": dict(P=(12, 48), R=(13, 101), V=(11, 101), K=(8, 91)),
    "local": dict(P=(12, 48), R=(13, 101), V=(11, 101), K=(8, 91)),
    "newcoef": dict(P=(12, 24), R=(13, 51), V=(15, 101), K=(9, 45)),
    "radial": dict(P=(12, 48), R=(13, 101), V=(11, 101), K=(8, 91)),
    "kf_radial": dict(P=(12, 48), R=(25, 101), V=(11, 31), K=(11, 31)),
    "kf_conv": dict(P=(11, 24), R=(11, 25), V=(4, 11), K=(4, 11)),
}
_MOST_POINTS = {"step": 3.9e6, "conv": 7.8e6, "local": 5.8e6, "newcoef": 2.6e6, "radial": 7.8e6}


def draw(rng):
    """A case of the same ranges, sizes spread over their logarithm."""
    op = rng.choice(list(_RANGES))
    while True:
        c = dict(op=op)
        for ax, (lo, hi) in _RANGES[op].items():
            c[ax] = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        if c["P"] * c["R"] * c["V"] * c["K"] <= _MOST_POINTS.get(op, 1e9):
            break
    c["kp"] = round(rng.uniform(1.0, 5.0), 2)
    if op in ("step", "conv"):
        c["arith"] = "exact" if op == "step" else rng.choice(["exact", "stream"])
    if op in ("local", "newcoef"):
        c["prec"] = rng.choice(["fp64", "fp64", "mixed"])
    return c


def _workload(case, seed):
    spec = W.GridSpec(case["P"], case["R"], case["V"], case["K"])
    wl = W.make_workload(spec, seed=seed, kp=case["kp"], sources=True)
    if case["op"] in ("kf_radial", "kf_conv"):
        return wl
    # a state that some steps have roughened, as independent coefficients at every point do
    rng = np.random.default_rng(seed + 104729)
    wl.fields["psd"] = wl.fields["psd"] * np.exp(0.05 * rng.standard_normal(spec.shape))
    if case["P"] > 1:
        wl.fields["psd"][-1] = wl.fields["psd"][0]  # the MLT endpoint is the first point again
    return wl


def _observations(case, wl, seed):
    """Two percent of the points observed with 5 % scatter, at least one in every unit."""
    rng = np.random.default_rng(seed + 15485863)
    psd = wl.fields["psd"]
    obs = np.full(psd.shape, np.nan)
    # only MLT 0 is assimilated by the radial filter; its edges in L are boundaries
    part = obs[:1] if case["op"] == "kf_radial" else obs
    src = psd[:part.shape[0]]
    mask = rng.uniform(size=part.shape) < (0.1 if case["op"] == "kf_radial" else 0.02)
    mask[:, part.shape[1] // 2] |= case["op"] == "kf_radial"
    mask[part.shape[0] // 2, part.shape[1] // 2] = True
    mask[:, 0] = mask[:, -1] = False
    part[mask] = src[mask] * np.exp(0.05 * rng.standard_normal(int(mask.sum())))
    return obs


class _DeviceField:
    """A context's field as a tensor without a copy; keeps the context alive."""

    def __init__(self, ctx, name):
        ptr = _lib._dp()
        _lib.check(ctx.lib.verb_field_device_ptr(ctx.h, _lib.FIELD_IDS[name], ctypes.byref(ptr)),
                   "field_device_ptr")
        self.ctx = ctx
        self.__cuda_array_interface__ = dict(
            shape=ctx.shape, typestr="<f8", version=3,
            data=(ctypes.cast(ptr, ctypes.c_void_p).value, False))


def _put(ctx, name, dev):
    """A field from device memory (the caller's CUDA code holds its state there)."""
    _lib.check(ctx.lib.verb_upload_field_device(ctx.h, _lib.FIELD_IDS[name],
                                                ctypes.c_void_p(dev.data_ptr())), name)


def prepare(case, seed):
    op = case["op"]
    wl = _workload(case, seed)
    f = wl.fields
    s = dict(op=op, dt=wl.dt, sub=wl.sub_dt, turn=0)
    if op in ("slice_local", "slice_conv"):
        s["args"] = _slice_args(case, wl)
        return s
    ctx = Context(*wl.spec.shape)
    s["ctx"] = ctx
    ctx.set_bc_types(wl.bc_types)
    fl = wl.flags
    ctx.set_options(fl["radial_sources"], fl["local_sources"], fl["include_boundary"],
                    fl["positive_psd"])
    for name in FIELDS:
        ctx.upload(name, f[name])
    for name in _lib.BC_FIELDS:
        ctx.upload(name, f[name])
    if "arith" in case:
        ctx.set_convection_arith(case["arith"])
    if "prec" in case:
        ctx.set_local_precision(case["prec"], 2 if case["prec"] == "mixed" else 0)
    if op == "step":
        ctx.set_step_graph(True)
    if op in ("conv", "kf_radial"):
        s["psd0"] = torch.from_numpy(f["psd"]).cuda()
    if op == "newcoef":
        s["coef"] = [[torch.from_numpy(a).cuda() for a in h] for h in _coefficients(wl)]
    if op in ("kf_radial", "kf_conv"):
        s["obs"] = _observations(case, wl, seed)
    if op == "local":  # the factors of the first step are there
        ctx.local(wl.dt, wl.sub_dt)
        _put(ctx, "psd", torch.from_numpy(f["psd"]).cuda())
    if op == "kf_conv":  # so are the model matrices of the hour
        ctx.assimilate_convection(s["obs"], wl.dt, *KF_CONV, has_vx_updated=True)
        _put(ctx, "psd", torch.from_numpy(f["psd"]).cuda())
    ctx.sync()
    s["psd"] = torch.as_tensor(_DeviceField(ctx, "psd"), device="cuda")
    torch.cuda.synchronize()
    return s


def _slice_args(case, wl):
    f = wl.fields
    P, R, V, K = wl.spec.shape
    t = wl.bc_types
    if case["op"] == "slice_local":
        q = lambda n: np.ascontiguousarray(f[n][0, 0])  # noqa: E731
        return (q("psd"), q("Vg"), q("Kg"), V, K, f["Vl"][0, 0], f["Vu"][0, 0], f["Kl"][0, 0],
                f["Ku"][0, 0], t["Vl"], t["Vu"], t["Kl"], t["Ku"], q("DVV"), q("DKK"), q("DVK"),
                q("DVK"), q("G_local"), q("S"), q("loss_local"), wl.dt, wl.sub_dt)
    q = lambda n: np.ascontiguousarray(f[n][:, :, 0, 0])  # noqa: E731
    return (q("psd"), q("Pg"), q("Rg"), P, R, np.ascontiguousarray(f["Pl"][:, 0, 0]),
            np.ascontiguousarray(f["Pu"][:, 0, 0]), np.ascontiguousarray(f["Rl"][:, 0, 0]),
            np.ascontiguousarray(f["Ru"][:, 0, 0]), t["Pl"], t["Pu"], t["Rl"], t["Ru"], q("VP"),
            q("VR"), q("S"), q("loss_conv"), q("G_conv"), wl.dt)


def _coefficients(wl):
    """(D_VV, D_KK, D_VK) of two hours: the second table is the first one of the next MLT."""
    a = [wl.fields[n] for n in ("DVV", "DKK", "DVK")]
    return a, [np.ascontiguousarray(np.roll(x, 1, axis=0)) for x in a]


def run(s):
    op = s["op"]
    if op == "slice_local":
        return ops.Diffusion_2D(*s["args"])
    if op == "slice_conv":
        return ops.Convection_2D(*s["args"])
    ctx, dt = s["ctx"], s["dt"]
    turn = s["turn"]
    s["turn"] = turn + 1
    if op == "step":
        neg = ctx.step(dt, s["sub"], count_negatives=True)
        return dict(psd=s["psd"], negatives=neg)
    if op == "conv":
        _put(ctx, "psd", s["psd0"])
        ctx.convection(dt)
    elif op == "local":
        ctx.local(dt, s["sub"])
    elif op == "newcoef":
        for name, d in zip(("DVV", "DKK", "DVK"), s["coef"][turn & 1]):
            _put(ctx, name, d)
        ctx.local(dt, s["sub"])
    elif op == "radial":
        ctx.set_scale("DLL", _dll_scale(turn))
        ctx.radial(dt)
    elif op == "kf_radial":
        _put(ctx, "psd", s["psd0"])
        ctx.assimilate_radial(s["obs"], dt, *KF_RADIAL, p_index=0)
    elif op == "kf_conv":
        ctx.assimilate_convection(s["obs"], dt, *KF_CONV)
    return s["psd"]


def _dll_scale(turn):
    return 10.0 ** (0.506 * (0.5 if turn & 1 else -0.7))  # Kp up, then down again


def work(case):
    P, R, V, K = (case[a] for a in "PRVK")
    n = P * R * V * K
    op = case["op"]

    def conv():
        _, nsub = _substeps(case)
        faces = float(nsub.sum()) * ((R - 1) * P + P * R)
        return dict(bytes=8.0 * 7 * n, flops=179.0 * faces)

    def local(sub_solves=1):
        kl, item = V + 1, 4 if case.get("prec") == "mixed" else 8
        return dict(bytes=sub_solves * (n * (3 * kl + 1) * item + 20.0 * n),
                    flops=sub_solves * 2.0 * n * 3 * kl)

    def factor():
        kl = V + 1
        item = 4 if case.get("prec") == "mixed" else 8
        return dict(bytes=n * (3 * kl + 1) * item + 8.0 * 7 * n, flops=2.0 * n * kl * 2 * kl)

    def both(*w):
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}

    radial = dict(bytes=8.0 * 5 * n, flops=10.0 * n)
    if op == "slice_local":
        return both(factor(), local())
    if op in ("slice_conv", "conv"):
        return conv()
    if op == "step":
        return both(conv(), radial, local(), dict(bytes=8.0 * n, flops=n))
    if op == "local":
        return local(3 if case["prec"] == "mixed" else 1)
    if op == "newcoef":
        return both(factor(), local(3 if case["prec"] == "mixed" else 1))
    if op == "radial":
        return dict(bytes=8.0 * 8 * n, flops=40.0 * n)
    if op == "kf_radial":
        return dict(bytes=8.0 * V * K * (2 * R * R + 4 * R), flops=V * K * 4.0 * R ** 3)
    N = P * R
    # M^36 by squarings (6 products), Q, M Pa M^T (two products), the update
    return dict(bytes=8.0 * V * K * 3 * N * N, flops=V * K * 2.0 * N ** 3 * 9)


def _substeps(case):
    spec = W.GridSpec(case["P"], case["R"], case["V"], case["K"])
    mlt, L, _, _ = W.axes(spec)
    VP, VR = W.drift_velocities(spec, case["kp"])
    a = W.DT_5MIN * np.abs(VP).max(axis=(0, 1)) / (mlt[1] - mlt[0]) / 0.25
    b = W.DT_5MIN * np.abs(VR).max(axis=(0, 1)) / (L[1] - L[0]) / 0.25
    nsub = np.maximum(np.where(a <= 1, 1, np.ceil(a)), np.where(b <= 1, 1, np.ceil(b)))
    return spec, nsub.astype(np.int64)


# ---------------------------------------------------------------- 64-bit results in plain torch

def exact(case, seed):
    wl = _workload(case, seed)
    op = case["op"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f = {k: torch.from_numpy(np.ascontiguousarray(v)).to(dev) for k, v in wl.fields.items()}
    psd = f["psd"]
    if op == "slice_local":
        return _local(psd, f, wl)[0, 0].cpu().numpy()
    if op == "slice_conv":
        return _convection(psd, f, wl)[:, :, 0, 0].cpu().numpy()
    if op == "conv":
        return _convection(psd, f, wl)
    if op == "local":
        return _local(psd, f, wl)
    if op == "newcoef":
        return _local(psd, f, wl)
    if op == "radial":
        return _radial(psd, f, wl, _dll_scale(0))
    if op == "step":
        x = _radial(_convection(psd, f, wl), f, wl, 1.0)
        return dict(psd=_local(x, f, wl), negatives=None)
    if op == "kf_radial":
        obs = torch.from_numpy(_observations(case, wl, seed)).to(dev)
        return _kf_radial(psd.clone(), f, wl, obs)
    # a pass of the (MLT, L) filter starts from an earlier update's covariances and its gain is
    # ill-conditioned where the PSD is far below the model error
    return None


def _radial_rows(f, wl, scale, psd_like):
    """Tridiagonal rows [P,R,V,K] of the Crank-Nicolson radial operator and 1/dt."""
    L, D, G = f["Lg"], f["DLL"] * scale, f["G_radial"]
    lo, d, up = (torch.zeros_like(psd_like) for _ in range(3))
    x0, xm, xp = L[:, 1:-1], L[:, :-2], L[:, 2:]
    d[:, 1:-1] = 1.0 / wl.dt - f["loss_radial"][:, 1:-1]
    Dm, D0, Dp = D[:, :-2], D[:, 1:-1], D[:, 2:]
    Gm, G0, Gp = G[:, :-2], G[:, 1:-1], G[:, 2:]
    for xa, xb, Da, Ga, near, far in ((xm, xp, Dm, Gm, lo, up), (xp, xm, Dp, Gp, up, lo)):
        cp = -0.5 / G0 / (x0 - xa)
        c1, c2 = cp / (x0 - xb) * D0 * G0, cp / (xa - x0) * Da * Ga
        d[:, 1:-1] += c1 + c2
        far[:, 1:-1] -= c1
        near[:, 1:-1] -= c2
    d[:, 0] = d[:, -1] = 1.0  # constant value at both ends
    return lo, d, up


def _radial(psd, f, wl, scale):
    lo, d, up = _radial_rows(f, wl, scale, psd)
    n = psd.shape[1]
    rhs = psd / wl.dt
    rhs[:, 0], rhs[:, -1] = f["Ll"], f["Lu"]
    gam, u = torch.zeros_like(psd), torch.zeros_like(psd)
    bet = d[:, 0]
    u[:, 0] = rhs[:, 0] / bet
    for r in range(1, n):
        gam[:, r] = up[:, r - 1] / bet
        bet = d[:, r] - lo[:, r] * gam[:, r]
        u[:, r] = (rhs[:, r] - lo[:, r] * u[:, r - 1]) / bet
    for r in range(n - 1, 0, -1):
        u[:, r - 1] -= gam[:, r] * u[:, r]
    return u


def _local(psd, f, wl):
    """The (V, K) systems by block elimination over K, blocks of V unknowns."""
    P, R, V, K = psd.shape
    out = torch.empty_like(psd)
    step = max(1, int(2e9 / (8.0 * V * V * K)))
    flat = lambda a: a.reshape(P * R, V, K)  # noqa: E731
    q = {k: flat(f[k]) for k in ("Vg", "Kg", "DVV", "DKK", "DVK", "G_local", "S", "loss_local")}
    for s0 in range(0, P * R, step):
        sl = slice(s0, min(P * R, s0 + step))
        out.view(P * R, V, K)[sl] = _local_chunk(flat(psd)[sl], {k: a[sl] for k, a in q.items()},
                                                 f, wl, sl)
    return out


def _local_chunk(psd, q, f, wl, sl):
    N, V, K = psd.shape
    x, G = q["Vg"] + q["Kg"], q["G_local"]
    at = lambda a, i, j: a[:, 1 + i:V - 1 + i, 1 + j:K - 1 + j]  # noqa: E731
    A = {(i, j): torch.zeros_like(psd) for i in (-1, 0, 1) for j in (-1, 0, 1)}
    A[0, 0][:, 1:-1, 1:-1] = 1.0 / wl.sub_dt - at(q["loss_local"], 0, 0)
    xl, xr, yl, yr = (-1, 0), (1, 0), (0, -1), (0, 1)
    pairs = [(xl, xr, "DVV", -0.5), (xr, xl, "DVV", -0.5), (yl, yr, "DKK", -0.5),
             (yr, yl, "DKK", -0.5)]
    pairs += [(a, b, "DVK", -0.25) for a in (yl, yr) for b in (xl, xr)]
    pairs += [(b, a, "DVK", -0.25) for a in (yl, yr) for b in (xl, xr)]
    for a, b, name, mult in pairs:
        D, ab = q[name], (a[0] + b[0], a[1] + b[1])
        cp = mult / at(G, 0, 0) / (at(x, 0, 0) - at(x, *a))
        c1 = cp / (at(x, 0, 0) - at(x, *b)) * at(D, 0, 0) * at(G, 0, 0)
        c2 = cp / (at(x, *a) - at(x, *ab)) * at(D, *a) * at(G, *a)
        A[0, 0][:, 1:-1, 1:-1] += c1
        A[b][:, 1:-1, 1:-1] -= c1
        A[a][:, 1:-1, 1:-1] -= c2
        A[ab][:, 1:-1, 1:-1] += c2
    rhs = psd / wl.sub_dt + q["S"]
    P, R = wl.spec.shape[:2]
    # zero gradient at both pitch-angle edges, constant value at both energy edges
    for j, k in ((0, 1), (K - 1, -1)):
        h = 1.0 / (q["Kg"][:, :, j + k] - q["Kg"][:, :, j]).abs()
        A[0, 0][:, :, j], A[0, k][:, :, j] = h, -h
    rhs[:, :, 0], rhs[:, :, -1] = (f[b].reshape(P * R, V)[sl] for b in ("Kl", "Ku"))
    for i in (0, V - 1):
        A[0, 0][:, i] = 1.0
        for o in ((0, 1), (0, -1)):
            A[o][:, i] = 0.0
    rhs[:, 0], rhs[:, -1] = (f[b].reshape(P * R, K)[sl] for b in ("Vl", "Vu"))
    block = lambda j, k: (torch.diag_embed(A[0, j][:, :, k])  # noqa: E731
                          + torch.diag_embed(A[-1, j][:, 1:, k], -1)
                          + torch.diag_embed(A[1, j][:, :-1, k], 1))
    C, y = [], []
    for k in range(K):
        B, r = block(0, k), rhs[:, :, k:k + 1].clone()
        if k:
            lower = block(-1, k)
            B = B - lower @ C[-1]
            r = r - lower @ y[-1]
        sol = torch.linalg.solve(B, torch.cat([block(1, k), r], 2))
        C.append(sol[:, :, :V])
        y.append(sol[:, :, V:])
    out = torch.empty_like(psd)
    z = y[-1]
    out[:, :, -1] = z[..., 0]
    for k in range(K - 2, -1, -1):
        z = y[k] - C[k] @ z
        out[:, :, k] = z[..., 0]
    return out


def _kf_radial(psd, f, wl, obs):
    """The radial filter at MLT 0 from the first-use covariance, dense, one batch."""
    me, oe = KF_RADIAL
    P, R, V, K = psd.shape
    cols = lambda a: a[0].reshape(R, V * K).T  # noqa: E731
    lo, d, up = (cols(a) for a in _radial_rows(f, wl, 1.0, psd))
    lo = lo.clone()
    lo[:, -1] = 0.0  # the reference's dense matrix drops it
    A = torch.diag_embed(d) + torch.diag_embed(lo[:, 1:], -1) + torch.diag_embed(up[:, :-1], 1)
    b = torch.full_like(d, 1.0 / wl.dt)
    b[:, 0] = b[:, -1] = 0.0
    F = torch.linalg.solve(A, torch.diag_embed(b), left=False)
    eye = torch.eye(R, dtype=psd.dtype, device=psd.device)
    Pf = 5 * me * F @ F.mT + me * eye
    x, o = cols(psd), cols(obs)
    seen = torch.isfinite(o)
    h = seen.to(psd.dtype)
    # unobserved points: a unit row in the innovation covariance and no gain
    S = Pf * h[:, :, None] * h[:, None, :] + torch.diag_embed(oe * h + (1 - h))
    gain = torch.linalg.solve(S, Pf * h[:, None, :], left=False)
    x = x + (gain @ (torch.where(seen, o - x, torch.zeros_like(x)))[..., None])[..., 0]
    psd[0] = x.T.reshape(R, V, K)
    return psd


def _convection(psd, f, wl):
    """Convection_2D on every (V, K) slice: MLT lines, then L lines, sub-step by sub-step."""
    P, R, V, K = psd.shape
    sl = lambda a: a.reshape(P, R, V * K).permute(2, 0, 1)  # noqa: E731
    x = sl(psd).clone()
    VP, VR, G, S, loss = (sl(f[k]) for k in ("VP", "VR", "G_conv", "S", "loss_conv"))
    dP, dR = sl(f["Pg"])[0, 1, 0] - sl(f["Pg"])[0, 0, 0], sl(f["Rg"])[0, 0, 1] - sl(f["Rg"])[0, 0, 0]
    need = torch.maximum(wl.dt * VP.abs().amax((1, 2)) / dP, wl.dt * VR.abs().amax((1, 2)) / dR)
    nsub = torch.ceil(need / 0.25).clamp(min=1).to(torch.int64)
    order = torch.argsort(nsub, descending=True)
    x, VP, VR, G, S, loss, nsub = (a[order] for a in (x, VP, VR, G, S, loss, nsub))
    rl, ru = (f[k].reshape(P, V * K).T[order] for k in ("Rl", "Ru"))
    dt = (wl.dt / nsub.to(torch.float64))[:, None, None]
    cp, cr = (VP / dP * dt).mT.contiguous(), VR / dR * dt
    grow, add = torch.exp(loss * dt), S * dt
    add[:, :, 0] = add[:, :, -1] = 0.0
    rl, ru = (rl * G[:, :, 0])[..., None], (ru * G[:, :, -1])[..., None]
    counts = nsub.cpu().numpy()
    for it in range(int(counts[0])):
        m = int((counts > it).sum())
        y = x[:m].clone()
        y[:, :, :-1] = _line(x[:m].mT[:, :-1], cp[:m, :-1], None, None).mT
        y = _line(y * G[:m], cr[:m], rl[:m], ru[:m])
        x[:m] = y / G[:m] * grow[:m] + add[:m]
    back = torch.empty_like(x)
    back[order] = x
    return back.permute(1, 2, 0).reshape(P, R, V, K).contiguous()


def _line(t, cour, lbc, ubc):
    """One ULTIMATE-QUICKEST step (9th order) along the last axis; lbc None: periodic lines,
    whose last point is the first again, else constant values at both ends."""
    n = t.shape[-1]

    def ghosts(a, low):
        if lbc is None:
            return torch.cat([low[..., n - 6:n - 1], a, a[..., 1:6]], -1)
        e = a.shape[:-1] + (5,)
        return torch.cat([lbc.expand(e), a, ubc.expand(e)], -1)

    c = torch.zeros_like(cour)
    c[..., 1:] = (cour[..., :-1] + cour[..., 1:]) / 2
    if lbc is None:
        c[..., 0] = (cour[..., n - 2] + cour[..., 0]) / 2
    pos = c >= 0
    ca, cs = c.abs(), c * c

    def stencil(g):
        # value at upwind-oriented offset o of face i: o = 0 centre, negative upwind
        def pick(o):
            return torch.where(pos, g[..., 4 + o:4 + o + n], g[..., 5 - o:5 - o + n])
        return pick

    g = ghosts(t, t)
    w = stencil(g)
    U = [None] + [w(-i) for i in range(1, 5)]
    D = [None] + [w(i) for i in range(1, 6)]
    C = w(0)
    face = 0.5 * (C + D[1]) + 0.5 * ca * (C - D[1])
    face += (cs - 1) / 6 * ((U[1] - C - D[1] + D[2]) / 2
                            + ca / 4 * (U[1] - 3 * C + 3 * D[1] - D[2]))
    face += (cs - 1) * (cs - 4) / 120 * (
        (U[2] - 3 * U[1] + 2 * C + 2 * D[1] - 3 * D[2] + D[3]) / 2
        + ca / 6 * (U[2] - 5 * U[1] + 10 * C - 10 * D[1] + 5 * D[2] - D[3]))
    face += (cs - 1) * (cs - 4) * (cs - 9) / 5040 * (
        (U[3] - 5 * U[2] + 9 * U[1] - 5 * C - 5 * D[1] + 9 * D[2] - 5 * D[3] + D[4]) / 2
        + ca / 8 * (U[3] - 7 * U[2] + 21 * U[1] - 35 * C + 35 * D[1] - 21 * D[2] + 7 * D[3]
                    - D[4]))
    face += (cs - 1) * (cs - 4) * (cs - 9) * (cs - 16) / 362880 * (
        (U[4] - 7 * U[3] + 20 * U[2] - 28 * U[1] + 14 * C + 14 * D[1] - 28 * D[2] + 20 * D[3]
         - 7 * D[4] + D[5]) / 2
        + (U[4] - 9 * U[3] + 36 * U[2] - 84 * U[1] + 126 * C - 126 * D[1] + 84 * D[2]
           - 36 * D[3] + 9 * D[4] - D[5]) / 2)

    def cells(fc):
        out = t.clone()
        flux = c * fc
        if lbc is None:
            out[..., :-1] -= flux[..., 1:] - flux[..., :-1]
            out[..., -1] = out[..., 0]
        else:
            out[..., 1:-1] -= flux[..., 2:] - flux[..., 1:-1]
            out[..., :1], out[..., -1:] = lbc, ubc
        return out

    u = cells(face)
    w = stencil(ghosts(u, t))
    UU = [None] + [w(-i) for i in range(1, 4)]
    UD = [None] + [w(i) for i in range(1, 4)]
    UC = w(0)
    w = stencil(g)
    ou, oc, od = w(-1), w(0), w(1)
    DEL, CURV = od - ou, od - 2 * oc + ou
    d1, d2, d3 = UD[2] - UD[3], UD[1] - UD[2], UC - UD[1]
    d4, d5, d6 = UU[1] - UC, UU[2] - UU[1], UU[3] - UU[2]

    def peak(a, b, p, q):
        return (a > 0) & (b > 0) & (p < 0) & (q < 0) & (b < a) & (p > q)

    peaks = peak(d1, d2, d3, d4) | peak(d2, d3, d4, d5) | peak(d3, d4, d5, d6)
    moving = ca > 1e-31
    ref = ou + (oc - ou) / torch.where(moving, ca, torch.ones_like(ca))
    rise = torch.minimum(torch.maximum(face, oc), torch.minimum(ref, od))
    fall = torch.maximum(torch.minimum(face, oc), torch.maximum(ref, od))
    lim = torch.where(DEL > 0, rise, torch.where(DEL < 0, fall, face))
    lim = torch.where(moving, lim, face)
    lim = torch.where(CURV.abs() >= DEL.abs(), oc, lim)
    return cells(torch.where(peaks, face, lim))
