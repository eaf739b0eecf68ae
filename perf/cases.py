"""The work a user of this framework has it do, as cases that can be timed.

Every case goes through the public classes (tricubic, quadcubic,
TricubicField, BatchedTricubic, genfromtxt) with their defaults except the
options a case names.  Fields are the seeded generators of
arbinterp_gb300.synth (the reference ships no data); queries are uniform over
the interpolation volume with 1 % of the rows just outside it (which must
come back NaN), or a Gaussian cloud around the middle of the volume, as trapped
particles are.

op     point  one point through Query on a kept interpolant
       job    construct from the field rows, then Query (a program's first use)
       query  Query on a kept interpolant (every later use)
       table  allCoeffs and a Query from the table, on a kept interpolant
       grad   TricubicField forward and backward (values and queries)
       traj   RK4 trajectories on a kept interpolant
       batch  one launch over many fields
       csv    a field file's text to a table on the device
"""
import math

import numpy as np
import torch

from arbinterp_gb300 import genfromtxt, quadcubic, synth, tricubic
from arbinterp_gb300.autograd import TricubicField
from arbinterp_gb300.batched import BatchedTricubic

DEV = "cuda"


def _case(op, n, mode, precision, rows, **more):
    c = {"op": op, "nx": n[0], "ny": n[1], "nz": n[2], "nt": n[3] if len(n) == 4 else 0, "mode": mode,
         "precision": precision, "rows": rows, "spread": "uniform", "order": "ij", "host": False, "f32": False}
    c.update(more)
    return c


def listed():
    return [
        # the smallest call: one point of the 41^3 scalar example, NumPy in and out
        dict(_case("point", (41, 41, 41), "scalar", "fp64", 1, host=True), name="point"),
        # the 41^3 scalar example: construct, then 1e5 points plus 1 % outside
        dict(_case("job", (41, 41, 41), "scalar", "fp64", 101_000), name="example41_fp64"),
        # the headline workload in the default precision and in mixed precision
        dict(_case("job", (256, 256, 256), "both", "fp64", 10_100_000), name="both256_fp64"),
        dict(_case("job", (256, 256, 256), "both", "mixed", 10_100_000), name="both256_mixed"),
        # a particle cloud through a field file's rows (x fastest), NumPy in and out, |B| and its gradient
        dict(_case("job", (101, 87, 93), "norm", "fp64", 1_000_003, spread="cloud", order="xfast", host=True),
             name="cloud_norm_numpy"),
        # time-dependent fields: every later query of a kept quadcubic
        dict(_case("query", (64, 64, 64, 32), "scalar", "mixed", 10_000_000), name="quad_scalar_mixed"),
        dict(_case("query", (33, 41, 29, 17), "scalar", "fp64", 1_500_007), name="quad_scalar_fp64"),
        # the coefficient table the reference builds, and a query from it
        dict(_case("table", (112, 96, 101), "both", "mixed", 1_000_000), name="table_both_mixed"),
        # fit of a scalar field to measurements: forward and backward, float32 values
        dict(_case("grad", (128, 128, 128), "scalar", "mixed", 1_000_000, f32=True), name="fit128_mixed"),
        # particles in a magnetic trap
        dict(_case("traj", (128, 128, 128), "both", "mixed", 200_003, spread="cloud", steps=25),
             name="trajectories_mixed"),
        # many fields of uneven sizes in one launch
        dict(_case("batch", (24, 24, 24), "scalar", "mixed", 3_000_000, fields=48, nx1=96), name="batch48_mixed"),
        # reading the field file
        dict(_case("csv", (96, 96, 96), "both", "fp64", 96 ** 3, host=True), name="fieldfile96"),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    op = rng.choice(["point", "job", "job", "job", "query", "query", "query", "table", "grad", "traj", "batch", "csv"])
    prec = rng.choice(["fp64", "mixed"])
    mode = rng.choice(["scalar", "vector", "norm", "both"])
    four = op in ("point", "job", "query") and rng.random() < 0.3
    if four:
        n = tuple(_log(rng, 8, 40) for _ in range(3)) + (_log(rng, 6, 24),)
    else:
        top = {"table": 110, "grad": 140, "csv": 90}.get(op, 256)
        n = tuple(_log(rng, 12, top) for _ in range(3))
    cells = math.prod(v - 3 for v in n)
    most = {"point": 1, "traj": 200_000, "grad": 1_000_000}.get(op, 10_000_000)
    if four and prec == "fp64":
        most = 500_000 if mode in ("vector", "both") else 1_500_000
    rows = 1 if op == "point" else min(_log(rng, 1000, most) | 1, max(1001, 4 * cells))
    c = _case(op, n, mode, prec, rows, spread=rng.choice(["uniform", "uniform", "cloud"]),
              order=rng.choice(["ij", "ij", "xfast", "shuffled"]))
    if op in ("job", "query"):
        c["f32"] = rng.random() < 0.2
        c["host"] = rows <= 1_000_000 and rng.random() < 0.3
    if op == "point":
        c["host"] = True
    if op == "grad":
        c.update(mode="scalar", f32=prec == "mixed")
    if op == "traj":
        c.update(mode=rng.choice(["scalar", "norm", "both"]), steps=rng.randint(4, 25) if prec == "mixed" else 4,
                 spread="cloud")
    if op == "batch":
        a = rng.randint(14, 32)
        c.update(nx=a, ny=a, nz=a, nx1=_log(rng, a, 96), mode="scalar", fields=rng.randint(6, 48),
                 rows=_log(rng, 1e4, 3e6) if prec == "mixed" else _log(rng, 1e4, 1e6))
    if op == "csv":
        c.update(rows=math.prod(n), precision="fp64", host=True, mode=rng.choice(["scalar", "both"]))
    return c


# ---------------------------------------------------------------------------- inputs
def _n(case):
    n = (case["nx"], case["ny"], case["nz"])
    return n + (case["nt"],) if case["nt"] else n


def _field_rows(n, mode, seed, f32=False, order="ij"):
    """Field rows on the device, and their axes (float64, x first)."""
    d = len(n)
    if mode == "scalar":
        f = (synth.gaussian_field3(n, seed=seed, device=DEV) if d == 3
             else synth.moving_gaussian_field4(n, seed=seed, device=DEV))
    elif d == 3:
        f = synth.dipole_field3(n, seed=seed, device=DEV)
    else:  # three moving-Gaussian components
        parts = [synth.moving_gaussian_field4(n, seed=seed + 7919 * k, device=DEV) for k in range(3)]
        f = torch.cat([parts[0], parts[1][:, 4:], parts[2][:, 4:]], 1)
    if f32:
        f = f.to(torch.float32)
    grid = f.view(*n, -1)
    axes = [grid[tuple(slice(None) if b == a else 0 for b in range(d)) + (a,)].to(torch.float64) for a in range(d)]
    if order == "xfast":
        f = grid.permute(*reversed(range(d)), d).reshape(-1, grid.shape[-1])
    elif order == "shuffled":
        g = torch.Generator(device=DEV).manual_seed(seed + 5)
        f = f[torch.randperm(len(f), generator=g, device=DEV)]
    return f.contiguous(), axes


def _queries(axes, rows, seed, spread, f32=False, outside=True):
    g = torch.Generator(device=DEV).manual_seed(seed + 17)
    lo = torch.stack([a[1] for a in axes])
    hi = torch.stack([a[-2] for a in axes])
    h = torch.stack([a[1] - a[0] for a in axes])
    if f32:      # float32 axes are not evenly spaced to the last bit: stay off the upper faces
        hi = hi - 0.5 * h
    d = len(axes)
    if spread == "cloud":
        q = 0.5 * (lo + hi) + 0.125 * (hi - lo) * torch.randn(rows, d, generator=g, device=DEV, dtype=torch.float64)
        if not outside or f32:
            q = torch.minimum(torch.maximum(q, lo + 0.01 * h), hi - 0.01 * h)
    else:
        q = lo + (hi - lo) * torch.rand(rows, d, generator=g, device=DEV, dtype=torch.float64)
    if outside and spread != "cloud":
        k = rows // 101
        if k:
            at = torch.randperm(rows, generator=g, device=DEV)[:k]
            ax = torch.randint(0, d, (k,), generator=g, device=DEV)
            depth = (1e-3 + 2.0 * torch.rand(k, generator=g, device=DEV, dtype=torch.float64)) * h[ax]
            q[at, ax] = lo[ax] - depth
    return q


def _build(case, field):
    cls = quadcubic if case["nt"] else tricubic
    kw = {} if case["mode"] == "scalar" else {"mode": case["mode"]}
    if case["op"] == "table":
        kw["strategy"] = "table"
    return cls(field, "quiet", precision=case["precision"], **kw)


def _batch_specs(case, seed):
    """(edge, rows, field seed, spacings) of every field: the sizes are the case's, the rest the seed's."""
    rng, own = np.random.default_rng(case["fields"] * 1000 + case["nx1"]), np.random.default_rng(seed)
    specs = []
    for i in range(case["fields"]):
        e = int(round(math.exp(rng.uniform(math.log(case["nx"]), math.log(max(case["nx1"], case["nx"]))))))
        m = int(rng.uniform(0.2, 1.8) * case["rows"] / case["fields"])
        specs.append((e, max(1, min(m, 4 * (e - 3) ** 3)), int(own.integers(1 << 30)),
                      tuple(own.uniform(0.05, 0.2, 3))))
    return specs


def prepare(case, seed):
    op = case["op"]
    if op == "csv":
        text = synth.field_csv_text(_n(case), 1 if case["mode"] == "scalar" else 3, seed=seed, device=DEV)
        return {"case": case, "text": text.cpu().numpy().tobytes()}
    if op == "batch":
        specs = _batch_specs(case, seed)
        fields, qs = [], []
        for e, m, s, h in specs:
            f = synth.gaussian_field3((e, e, e), h=h, seed=s, device=DEV)
            g = f.view(e, e, e, 4)
            fields.append(f)
            qs.append(_queries([g[:, 0, 0, 0], g[0, :, 0, 1], g[0, 0, :, 2]], m, s, case["spread"], outside=False))
        return {"case": case, "obj": BatchedTricubic(fields, precision=case["precision"]), "q": torch.cat(qs),
                "counts": [m for _, m, _, _ in specs]}
    f, axes = _field_rows(_n(case), case["mode"], seed, case["f32"], case["order"])
    q = _queries(axes, case["rows"], seed, case["spread"], case["f32"], outside=op not in ("point", "grad", "traj"))
    s = {"case": case}
    if op == "grad":
        n = case["rows"]
        g = torch.Generator(device=DEV).manual_seed(seed + 29)
        field = TricubicField(f, precision=case["precision"])
        v = field.initial_values().to(torch.float32 if case["f32"] else torch.float64)
        s.update(obj=field, values=v.requires_grad_(True), q=q.requires_grad_(True),
                 up=(torch.randn(n, generator=g, device=DEV, dtype=v.dtype),
                     0.1 * torch.randn(n, 3, generator=g, device=DEV, dtype=v.dtype)))
        return s
    if op == "traj":
        g = torch.Generator(device=DEV).manual_seed(seed + 31)
        span = torch.stack([a[-2] - a[1] for a in axes])
        v = 0.05 * span * torch.randn(case["rows"], 3, generator=g, device=DEV, dtype=torch.float64)
        mid = torch.stack([0.5 * (a[-2] + a[1]) for a in axes])
        s.update(obj=_build(case, f), x=mid + 0.5 * (q - mid), v=v)
        return s
    if op == "point":
        s.update(obj=_build(case, f), q=q[0].cpu().numpy())
        return s
    if case["host"]:
        f, q = f.cpu().numpy(), q.cpu().numpy()
    s["q"] = q
    if op == "job":
        s["field"] = f
    else:
        s["obj"] = _build(case, f)
    return s


TRAJ_DT, TRAJ_COEF = 0.01, -1e-3


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "csv":
        return genfromtxt(s["text"], delimiter=",")
    if op == "batch":
        return s["obj"].query(s["q"], s["counts"])
    if op == "grad":
        value, grad = s["obj"](s["values"], s["q"])
        gv, gq = torch.autograd.grad((value, grad), (s["values"], s["q"]), s["up"])
        return value, grad, gv, gq
    if op == "traj":
        return s["obj"].trajectories(s["x"], s["v"], TRAJ_DT, case["steps"], coef=TRAJ_COEF)
    if op == "point":
        return s["obj"].Query(s["q"])
    obj = _build(case, s["field"]) if op == "job" else s["obj"]
    if op == "table":
        obj.allCoeffs()
    out = obj.Query(s["q"])
    # the query array comes back with its outside rows set to NaN
    return (out if isinstance(out, tuple) else (out,)) + (s["q"],)


def work(case):
    """Each input read once, each output written once; multiply-adds of the separable contraction (x, y, z[, t]:
    4^d + ... + 4 per field, and those of the gradient) counted as two."""
    n = _n(case)
    d = len(n)
    pts, rows = math.prod(n), case["rows"]
    op, mode = case["op"], case["mode"]
    ncol = d + (1 if mode == "scalar" else 3)
    F = {"scalar": 1, "vector": 3, "norm": 1, "both": 4}[mode]
    nout = {"scalar": 1 + d, "vector": 3, "norm": 1 + d, "both": 4 + d}[mode]
    madds = (F * 84 + (0 if mode == "vector" else 90)) * (4 if d == 4 else 1)
    item = 4 if case["f32"] else 8
    if op == "csv":
        return {"bytes": pts * ncol * (25 + 8), "flops": 0}
    if op == "batch":
        specs = _batch_specs(case, 1)
        pts = sum(e ** 3 for e, _, _, _ in specs)
        rows = sum(m for _, m, _, _ in specs)
        return {"bytes": pts * 8 + rows * (24 + 32), "flops": 2 * 174 * rows}
    if op == "traj":
        return {"bytes": pts * 8 + rows * 96, "flops": 2.0 * 174 * rows * 4 * case["steps"]}
    if op == "grad":
        # forward, scatter of 64 weights, query gradient with the Hessian
        return {"bytes": pts * 2 * item + rows * (24 + 32 + 32 + 24), "flops": 2 * rows * (174 + 256 + 270)}
    q = rows * 8 * (d + nout)
    if op == "job":
        return {"bytes": pts * ncol * item + q, "flops": 2 * madds * rows}
    if op == "table":
        table = math.prod(v - 3 for v in n) * F * 4 ** d * (4 if case["precision"] == "mixed" else 8)
        return {"bytes": pts * 8 * F + table + q, "flops": 2 * (480 * table / 256 + madds * rows)}
    touched = min(pts, rows * 4 ** d)
    return {"bytes": touched * F * 8 + q, "flops": 2 * madds * rows}


# ---------------------------------------------------------------------------- plain 64-bit values
def _weights(t):
    w = torch.stack([t * (-0.5 + t * (1 - 0.5 * t)), 1 + t * t * (-2.5 + 1.5 * t), t * (0.5 + t * (2 - 1.5 * t)),
                     t * t * (-0.5 + 0.5 * t)], -1)
    dw = torch.stack([-0.5 + t * (2 - 1.5 * t), t * (-5 + 4.5 * t), 0.5 + t * (4 - 4.5 * t), t * (-1 + 1.5 * t)], -1)
    return w, dw


def _contract(blk, ws):
    """blk [N, (4,) 4, 4, 4, F] with x the last 4; ws per axis, x first."""
    for w in ws:
        k = blk.dim() - 2
        blk = (blk * w.view(w.shape[0], *([1] * (k - 1)), 4, 1)).sum(k)
    return blk


def _geometry(axes, f32):
    h = [(a[0].float() - a[1].float()).abs().double() if f32 else (a[0] - a[1]).abs() for a in axes]
    return h, [a[1] for a in axes], [a[-2] for a in axes]


def _interp(axes, V, q, f32=False, want_grad=True):
    """Values [N, F] and the last field's gradient [N, d] of the grid V [(t,) z, y, x, F] at q, in float64;
    rows outside the volume NaN."""
    d = len(axes)
    h, lo, hi = _geometry(axes, f32)
    n = [len(a) for a in axes]
    inside = torch.ones(len(q), dtype=torch.bool, device=q.device)
    base = torch.zeros(len(q), dtype=torch.int64, device=q.device)
    stride, ws, dws, fr = 1, [], [], []
    offs = torch.zeros(1, dtype=torch.int64, device=q.device)
    for a in range(d):
        x = q[:, a]
        inside &= (x >= lo[a]) & (x <= hi[a])
        iu = torch.where((x >= lo[a]) & (x <= hi[a]), x - lo[a], torch.zeros_like(x)) / h[a]
        k = torch.floor(iu).detach().clamp(0, n[a] - 4)
        t = iu - k
        fr.append(t)
        w, dw = _weights(t)
        ws.append(w)
        dws.append(dw / h[a])
        base = base + k.to(torch.int64) * stride
        offs = (torch.arange(4, device=q.device)[:, None] * stride + offs[None, :]).reshape(-1)
        stride *= n[a]
    F = V.shape[-1]
    blk = V.reshape(-1, F)[base[:, None] + offs[None, :]].view(-1, *([4] * d), F)
    vals = _contract(blk, ws)
    last = blk[..., F - 1:]
    grads = [_contract(last, [dws[b] if b == a else ws[b] for b in range(d)])[:, 0] for a in range(d)] \
        if want_grad else []
    if d == 4:
        # the reference's quadcubic matrix lacks one of its rows and shifts the 15 after it by one: the mixed
        # fourth differences S_c enter with the next corner's slope basis less their own
        S = blk
        for a in range(4):
            k = S.dim() - 2 - a
            S = 0.5 * (S.narrow(k, 2, 2) - S.narrow(k, 0, 2))
        S = S.reshape(len(q), 16, F)                       # corner index x fastest
        T = torch.cat([-S[:, :1], S[:, :-1] - S[:, 1:]], 1).view(-1, 2, 2, 2, 2, F)
        hb = [torch.stack([t * (1 - t) ** 2, t * t * (t - 1)], -1) for t in fr]
        dhb = [torch.stack([1 - 4 * t + 3 * t * t, 3 * t * t - 2 * t], -1) / h[a] for a, t in enumerate(fr)]

        def con(B, w):
            for u in w:
                k = B.dim() - 2
                B = (B * u.view(u.shape[0], *([1] * (k - 1)), 2, 1)).sum(k)
            return B
        vals = vals + con(T, hb)
        if want_grad:
            grads = [g + con(T[..., F - 1:], [dhb[b] if b == a else hb[b] for b in range(4)])[:, 0]
                     for a, g in enumerate(grads)]
    nan = torch.full((), float("nan"), dtype=torch.float64, device=q.device)
    vals = torch.where(inside[:, None], vals, nan)
    g = torch.where(inside[:, None], torch.stack(grads, 1), nan) if want_grad else None
    return vals, g


def _grid(n, f, mode):
    """[(t,) z, y, x, F] interpolated fields of 'ij' rows f."""
    d = len(n)
    v = f[:, d:]
    if mode in ("norm", "both"):
        b = ((v[:, 0] * v[:, 0] + v[:, 1] * v[:, 1]) + v[:, 2] * v[:, 2]).sqrt()[:, None]
        v = b if mode == "norm" else torch.cat([v, b], 1)
    return v.double().view(*n, -1).permute(*reversed(range(d)), d).contiguous()


def exact(case, seed):
    op, mode, n = case["op"], case["mode"], _n(case)
    if op == "csv":
        return None
    if op == "batch":
        vs, gs = [], []
        for e, m, s, h in _batch_specs(case, seed):
            f = synth.gaussian_field3((e, e, e), h=h, seed=s, device=DEV)
            g = f.view(e, e, e, 4)
            axes = [g[:, 0, 0, 0], g[0, :, 0, 1], g[0, 0, :, 2]]
            v, dv = _interp(axes, _grid((e, e, e), f, "scalar"),
                            _queries(axes, m, s, case["spread"], outside=False))
            vs.append(v)
            gs.append(dv)
        return torch.cat(vs), torch.cat(gs)
    f, axes = _field_rows(n, mode, seed, case["f32"])
    V = _grid(n, f, mode)
    q = _queries(axes, case["rows"], seed, case["spread"], case["f32"], outside=op not in ("point", "grad", "traj"))
    if op == "traj":
        V = V[..., -1:].contiguous()
        g = torch.Generator(device=DEV).manual_seed(seed + 31)
        span = torch.stack([a[-2] - a[1] for a in axes])
        v = 0.05 * span * torch.randn(case["rows"], 3, generator=g, device=DEV, dtype=torch.float64)
        mid = torch.stack([0.5 * (a[-2] + a[1]) for a in axes])
        x, dt = mid + 0.5 * (q - mid), TRAJ_DT
        acc = lambda p: TRAJ_COEF * _interp(axes, V, p)[1]  # noqa: E731
        for _ in range(case["steps"]):
            k1 = acc(x)
            k2 = acc(x + 0.5 * dt * v)
            k3 = acc(x + 0.5 * dt * (v + 0.5 * dt * k1))
            k4 = acc(x + dt * (v + 0.5 * dt * k2))
            x = x + dt / 6 * (v + 2 * (v + 0.5 * dt * k1) + 2 * (v + 0.5 * dt * k2) + (v + dt * k3))
            v = v + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
        return x, v
    if op == "grad":
        m = case["rows"]
        g = torch.Generator(device=DEV).manual_seed(seed + 29)
        dt = torch.float32 if case["f32"] else torch.float64
        up = (torch.randn(m, generator=g, device=DEV, dtype=dt).double(),
              0.1 * torch.randn(m, 3, generator=g, device=DEV, dtype=dt).double())
        V.requires_grad_(True)
        gv = torch.zeros_like(V)
        vs, gs, gqs = [], [], []
        for a in range(0, m, 100_000):
            qa = q[a:a + 100_000].clone().requires_grad_(True)
            v, dv = _interp(axes, V, qa, case["f32"])
            x, y = torch.autograd.grad((v[:, 0], dv), (V, qa), (up[0][a:a + 100_000], up[1][a:a + 100_000]))
            gv += x
            gqs.append(y)
            vs.append(v[:, 0].detach())
            gs.append(dv.detach())
        return torch.cat(vs), torch.cat(gs), gv.reshape(-1), torch.cat(gqs)
    step = 500_000 if len(n) == 3 else 50_000
    parts = [_interp(axes, V, q[a:a + step], case["f32"], mode != "vector") for a in range(0, len(q), step)]
    v = torch.cat([p[0] for p in parts])
    g = None if mode == "vector" else torch.cat([p[1] for p in parts])
    del parts
    if op == "point":
        v, g = v[0].cpu().numpy(), None if g is None else g[0].cpu().numpy()
        return {"scalar": (v[0], g), "norm": (v[0], g), "vector": v[:3],
                "both": (v[:3], v[-1], g)}[mode]
    return {"scalar": (v, g, None), "norm": (v, g, None), "vector": (v[:, :3], None),
            "both": (v[:, :3], v[:, 3:], g, None)}[mode]
