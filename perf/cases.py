"""The work that is timed on the GPU: calls of this package's public entry
points as a FlOF program makes them, over the sizes it uses.

A case is a dict of plain values; `op` names the call and the other keys give
its sizes and options.  `listed()` gives the fixed cases and `draw(rng)` one
more of the same ranges.  `prepare` makes the inputs from a seed (falling drops
over a pool, the generator of ofblend_gb300/synth.py restated on the GPU),
`run` is one pass, `work` the bytes and operations a pass cannot do without and
`exact` the same outputs in 64 bits by plain torch.
"""
import math
import random

import torch

import ofblend_gb300 as F
from ofblend_gb300 import scene as S

DEV = "cuda:0"
LS_FACTOR = -0.1 / 20.0
# scenes/flof.py's solve (mode 1); the final projection is a call of its own below
SOLVE = dict(wSmooth=0.001, wEnergy=0.0001, cgAccuracy=1e-4, postVelBlur=4, cfl=999, multiStep=3,
             minGridSize=20, resetBndWidth=0.1, doFinalProject=False)


def listed():
    return [
        # mode 1, the headline size: one direction of a two-way pair
        dict(name="solve_64", op="solve", X=64, Y=64, Z=64, T=64, solver="pcg"),
        # mode 1, the smallest pair of the batched workload: launches and host decisions count
        dict(name="solve_24x16", op="solve", X=24, Y=24, Z=24, T=16, solver="pcg"),
        # mode 1 with the multigrid preconditioner and the separable stencils
        dict(name="solve_mg_64", op="solve", X=64, Y=64, Z=64, T=64, solver="mg"),
        # many small deformations at once (one call, worker streams)
        dict(name="batch_24_40", op="batch", smin=24, smax=40, tmin=16, tmax=32, pairs=8),
        # one linear solve of a level with uneven extents
        dict(name="flow_ragged", op="flow", X=45, Y=38, Z=41, T=30),
        # the final projection of a computed deformation
        dict(name="project_64", op="project", X=64, Y=64, Z=64, T=64),
        # mode 2: the two-way apply on the low-res 4D grid
        dict(name="deform_64", op="deform", X=64, Y=64, Z=64, T=64, alpha=0.5),
        # mode 3: output frames of the hi-res series, two-way
        dict(name="frames_128", op="frames", R=64, H=128, T=64, frames=8, alpha=0.25),
        # a deformation taken to a finer grid of odd extents
        dict(name="prolong_odd", op="resample", X=31, Y=33, Z=29, T=32, num=2, den=1, vec=True),
        # the error metric of a small pair: one short call, its answer read by the host
        dict(name="error_24x16", op="error", X=24, Y=24, Z=24, T=16),
        # input conditioning of a loaded data set (flof.py postProcessPhiData)
        dict(name="condition_48", op="condition", res=48),
        # the warm-start network: forward and backward of one training sample
        dict(name="net_grad_16", op="net", R=16, grad=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["solve", "solve", "solve", "batch", "flow", "flow", "project", "project", "deform",
                     "frames", "resample", "error", "condition", "net"])
    if op == "solve":
        s = _log(rng, 21, 60)
        return dict(op=op, X=s, Y=max(20, s - rng.randint(0, 6)), Z=max(20, s - rng.randint(0, 6)),
                    T=_log(rng, 16, 56), solver=rng.choice(["pcg", "pcg", "mg"]))
    if op == "batch":
        a = rng.randint(20, 28)
        return dict(op=op, smin=a, smax=a + rng.randint(2, 14), tmin=16, tmax=rng.randint(18, 32),
                    pairs=rng.randint(3, 10))
    if op in ("flow", "project"):
        s = _log(rng, 16, 58)
        return dict(op=op, X=s, Y=max(12, s + rng.randint(-8, 4)), Z=max(12, s + rng.randint(-8, 4)),
                    T=_log(rng, 12, 56))
    if op == "deform":
        s = _log(rng, 12, 63)
        return dict(op=op, X=s, Y=max(8, s + rng.randint(-6, 1)), Z=max(8, s + rng.randint(-6, 1)),
                    T=_log(rng, 8, 64), alpha=rng.choice([0.25, 0.5, 0.75, 1.0]))
    if op == "frames":
        return dict(op=op, R=rng.randint(24, 64), H=_log(rng, 40, 144), T=rng.randint(16, 64),
                    frames=rng.randint(2, 10), alpha=rng.choice([0.25, 0.5, 0.75]))
    if op == "resample":
        num, den = rng.choice([(2, 1), (1, 2), (3, 2)])
        s = _log(rng, 10, 34 if num > den else 62)
        return dict(op=op, X=s, Y=max(8, s + rng.randint(-4, 3)), Z=max(8, s + rng.randint(-4, 3)),
                    T=_log(rng, 8, 32 if num > den else 62), num=num, den=den, vec=rng.random() < 0.6)
    if op == "error":
        s = _log(rng, 12, 64)
        return dict(op=op, X=s, Y=max(8, s - rng.randint(0, 5)), Z=s, T=_log(rng, 8, 64))
    if op == "condition":
        return dict(op=op, res=_log(rng, 20, 56))
    return dict(op="net", R=rng.choice([8, 12, 16, 20]), grad=rng.random() < 0.6)


# --- inputs -----------------------------------------------------------------

def _scene(rng, ndrops):
    drops = []
    for _ in range(ndrops):
        ax = [rng.uniform(4.0, 8.0) for _ in range(3)] if rng.random() < 0.4 else [rng.uniform(4.0, 6.0)] * 3
        drops.append((rng.uniform(8.0, 24.0), rng.uniform(8.0, 24.0), ax))
    return 6.0 + rng.uniform(-1.0, 1.0), drops


def _axes(dims, dtype=torch.float32):
    X, Y, Z, T = dims
    ar = lambda n: torch.arange(n, device=DEV, dtype=dtype)  # noqa: E731
    return (ar(X).view(1, 1, 1, X), ar(Y).view(1, 1, Y, 1), ar(Z).view(1, Z, 1, 1), ar(T).view(T, 1, 1, 1))


def _sdf(sc, dims):
    """Signed distance in cells, clamped to [-4, 4], (T, Z, Y, X)."""
    X, Y, Z, T = dims
    x, y, z, t = _axes(dims)
    s = X / 32.0
    x, y, z, tau = (x + 0.5) / s, (y + 0.5) / s, (z + 0.5) / s, t * (32.0 / T)
    pool, drops = sc
    phi = (y - pool).expand(T, Z, Y, X).contiguous()
    for x0, z0, (a, b, c) in drops:
        cy = 24.0 - 0.025 * tau * tau
        k = torch.sqrt(((x - x0) / a) ** 2 + ((y - cy) / b) ** 2 + ((z - z0) / c) ** 2)
        phi = torch.minimum(phi, (k - 1.0) * min(a, b, c))
    return (phi * s).clamp_(-4.0, 4.0)


def _deformation(sc0, sc1, dims, rng):
    """A smooth field that moves the drops of sc0 onto those of sc1, with a
    slow wave on top; zero on the border ring, as a solve leaves it."""
    X, Y, Z, T = dims
    x, y, z, t = _axes(dims)
    s = X / 32.0
    xb, yb, zb, tau = (x + 0.5) / s, (y + 0.5) / s, (z + 0.5) / s, t * (32.0 / T)
    v = torch.zeros((T, Z, Y, X, 4), device=DEV)
    (xa, za, _), (x1, z1, ax) = sc0[1][0], sc1[1][0]
    cy = 24.0 - 0.025 * tau * tau
    w = torch.exp(-((xb - x1) ** 2 + (yb - cy) ** 2 + (zb - z1) ** 2) / (2.0 * max(ax)) ** 2)
    v[..., 0] += w * ((x1 - xa) * s * 0.8)
    v[..., 2] += w * ((z1 - za) * s * 0.8)
    v[..., 1] += torch.exp(-((yb - sc1[0]) / 6.0) ** 2) * ((sc1[0] - sc0[0]) * s)
    for c in range(4):
        f = [rng.uniform(0.05, 0.25) for _ in range(4)]
        ph = rng.uniform(0.0, 6.0)
        v[..., c] += 0.4 * torch.sin(f[0] * x + f[1] * y + f[2] * z + f[3] * t + ph)
    v[0], v[-1] = 0.0, 0.0
    v[:, 0], v[:, -1] = 0.0, 0.0
    v[:, :, 0], v[:, :, -1] = 0.0, 0.0
    v[:, :, :, 0], v[:, :, :, -1] = 0.0, 0.0
    return v


def _dims(c):
    return c["X"], c["Y"], c["Z"], c["T"]


def _real(a, dims):
    return F.Grid4Real(dims=dims, data_ptr=a.data_ptr())


def _vec(a, dims):
    return F.Grid4Vec4(dims=dims, data_ptr=a.data_ptr())


def _like(dims, nc):
    X, Y, Z, T = dims
    return torch.zeros((T, Z, Y, X, 4) if nc == 4 else (T, Z, Y, X), device=DEV)


def _pair(seed, dims, ndrops=1):
    rng = random.Random(seed)
    return _scene(rng, ndrops), _scene(rng, ndrops), rng


def _solve_kw(solver):
    return dict(SOLVE, solver=solver, blurType=2 if solver == "mg" else 1)


def _res_of(c):
    """Target extents of a resampling case."""
    return tuple(max(4, n * c["num"] // c["den"]) for n in _dims(c))


def _batch_dims(c, seed):
    """Uneven sizes of the batch: the same for every seed, so that passes compare."""
    rng = random.Random(c["smin"] * 1000 + c["smax"] * 10 + c["pairs"])
    out = []
    for _ in range(c["pairs"]):
        s = rng.randint(c["smin"], c["smax"])
        out.append((s, s, s, rng.randint(c["tmin"], c["tmax"])))
    return out


NET = [(2, 16, 3, 1), (16, 32, 3, 2), (32, 32, 3, 1), (32, 64, 3, 2), (64, 64, 3, 1), (96, 32, 3, 1),
       (48, 16, 3, 1), (16, 4, 1, 1)]  # (cin, cout, kernel, stride) of the warm-start network


def _net_inputs(c, seed):
    R = c["R"]
    gen = torch.Generator(device="cpu").manual_seed(seed)
    ps = []
    for cin, cout, k, _ in NET:
        n = k ** 4 * cin
        ps.append(torch.randn(n * cout, generator=gen) * math.sqrt(2.0 / n))
        ps.append(torch.randn(cout, generator=gen) * 0.01)
    p = torch.cat(ps).to(torch.bfloat16).to(torch.float32)
    dims = (R, R, R, R)
    s0, s1, rng = _pair(seed, dims)
    i0, i1 = _sdf(s0, dims) * LS_FACTOR, _sdf(s1, dims) * LS_FACTOR
    return p, i0.contiguous(), i1.contiguous(), _deformation(s0, s1, dims, rng), dims


def _inputs(c, seed):
    """The tensors of a case whose exact() needs them again."""
    op = c["op"]
    if op == "flow":
        dims = _dims(c)
        s0, s1, _ = _pair(seed, dims)
        return dims, (_sdf(s0, dims) * LS_FACTOR).contiguous(), (_sdf(s1, dims) * LS_FACTOR).contiguous()
    if op == "deform":
        dims = _dims(c)
        s0, s1, rng = _pair(seed, dims)
        return (dims, _sdf(s0, dims), _sdf(s1, dims), _deformation(s0, s1, dims, rng),
                _deformation(s1, s0, dims, rng))
    if op == "frames":
        d, h = (c["R"],) * 3 + (c["T"],), (c["H"],) * 3 + (c["T"],)
        s0, s1, rng = _pair(seed, d)
        return d, h, _sdf(s0, h), _sdf(s1, h), _deformation(s0, s1, d, rng), _deformation(s1, s0, d, rng)
    if op == "resample":
        dims = _dims(c)
        s0, s1, rng = _pair(seed, dims)
        return dims, (_deformation(s0, s1, dims, rng) if c["vec"] else _sdf(s0, dims))
    if op == "error":
        dims = _dims(c)
        s0, s1, _ = _pair(seed, dims)
        return dims, (_sdf(s0, dims) * LS_FACTOR).contiguous(), (_sdf(s1, dims) * LS_FACTOR).contiguous()
    raise ValueError(op)


def prepare(c, seed):
    op = c["op"]
    st = {"c": c, "op": op}
    if op in ("solve", "project"):
        dims = _dims(c)
        s0, s1, rng = _pair(seed, dims)
        a = [(_sdf(s0, dims) * LS_FACTOR).contiguous(), (_sdf(s1, dims) * LS_FACTOR).contiguous(), _like(dims, 4)]
        st.update(keep=a, i0=_real(a[0], dims), i1=_real(a[1], dims), vel=_vec(a[2], dims))
        if op == "solve":
            st["kw"] = _solve_kw(c["solver"])
        else:
            a += [_deformation(s0, s1, dims, rng), _like(dims, 4)]
            st.update(start=_vec(a[3], dims), dst=_vec(a[4], dims))
    elif op == "batch":
        i0, i1, v, keep = [], [], [], []
        for k, dims in enumerate(_batch_dims(c, seed)):
            s0, s1, _ = _pair(seed * 64 + k, dims)
            a = [(_sdf(s0, dims) * LS_FACTOR).contiguous(), (_sdf(s1, dims) * LS_FACTOR).contiguous(),
                 _like(dims, 4)]
            keep.append(a)
            i0.append(_real(a[0], dims))
            i1.append(_real(a[1], dims))
            v.append(_vec(a[2], dims))
        st.update(keep=keep, i0=i0, i1=i1, vel=v, kw=_solve_kw("pcg"))
    elif op == "flow":
        dims, i0, i1 = _inputs(c, seed)
        v = _like(dims, 4)
        st.update(keep=[i0, i1, v], i0=_real(i0, dims), i1=_real(i1, dims), vel=_vec(v, dims))
    elif op == "deform":
        dims, p0, p1, v, w = _inputs(c, seed)
        o = _like(dims, 1)
        st.update(keep=[p0, p1, v, w, o], i0=_real(p0, dims), i1=_real(p1, dims), vel=_vec(v, dims),
                  inv=_vec(w, dims), out=_real(o, dims))
    elif op == "frames":
        d, h, p0, p1, v, w = _inputs(c, seed)
        H = c["H"]
        o = [torch.zeros((H, H, H), device=DEV) for _ in range(c["frames"])]
        st.update(keep=[p0, p1, v, w, o], phi0=_real(p0, h), phi1=_real(p1, h), v0=_vec(v, d), v1=_vec(w, d),
                  dst=[F.RealGrid(dims=(H, H, H, 1), data_ptr=q.data_ptr()) for q in o])
    elif op == "resample":
        dims, a = _inputs(c, seed)
        td, nc = _res_of(c), 4 if c["vec"] else 1
        o = _like(td, nc)
        mk = _vec if c["vec"] else _real
        st.update(keep=[a, o], src=mk(a, dims), dst=mk(o, td))
    elif op == "error":
        dims, i0, i1 = _inputs(c, seed)
        st.update(keep=[i0, i1], i0=_real(i0, dims), i1=_real(i1, dims))
    elif op == "condition":
        r = c["res"]
        dims = (r, r, r, r * 3 // 2)
        s0, _, _ = _pair(seed, dims, ndrops=2)
        a = [_sdf(s0, dims).contiguous(), _like(dims, 1)]
        ofsd = S.flof_ofsd(r)
        off = S.vec4(0.0, 0.0, 0.0, dims[3] * ofsd["autoBorder"] + ofsd["repeatStartDist"])
        st.update(keep=a, src=_real(a[0], dims), phi=_real(a[1], dims), ofsd=ofsd, off=off)
    else:
        p, i0, i1, tgt, dims = _net_inputs(c, seed)
        m = F.Model(c["R"])
        m.set_params(p.numpy())
        o = _like(dims, 4)
        st.update(keep=[i0, i1, tgt, o], model=m, i0=_real(i0, dims), i1=_real(i1, dims), tgt=_vec(tgt, dims),
                  out=_vec(o, dims))
    return st


def run(st):
    op, c = st["op"], st["c"]
    if op == "solve":
        st["vel"].clear()
        err = F.opticalFlowMultiscale4d(st["vel"], st["i0"], st["i1"], **st["kw"])
        return st["keep"][2], err
    if op == "batch":
        for v in st["vel"]:
            v.clear()
        errs = F.opticalFlowMultiscale4d_batch(st["vel"], st["i0"], st["i1"], **st["kw"])
        return [a[2] for a in st["keep"]], errs
    if op == "flow":
        st["vel"].clear()
        F.opticalFlow4d(st["vel"], st["i0"], st["i1"], wSmooth=0.001, wEnergy=0.0001, cgAccuracy=1e-4)
        return st["keep"][2]
    if op == "project":
        st["vel"].copyFrom(st["start"])
        F.corrVelsOf4d(st["dst"], st["vel"], st["i0"], None, st["i1"], threshPhi=4.0, postVelBlur=4.0,
                       resetBndWidth=0.1, maxIter=40)
        return st["keep"][2], st["keep"][4]
    if op == "deform":
        F.deform4d(st["out"], st["i0"], st["i1"], st["vel"], st["inv"], alpha=c["alpha"], twoway=1)
        return st["keep"][4]
    if op == "frames":
        R, H, T, n = c["R"], c["H"], c["T"], c["frames"]
        F.loadAdvectTimeSlice_OptInit(1, st["v0"])
        F.loadAdvectTimeSlice_OptInit(2, st["v1"])
        for k in range(n):
            F.loadAdvectTimeSlice_OptRunTwoway(1, 2, st["dst"][k], st["phi0"], st["phi1"], _frame_time(c, k),
                                               c["alpha"], 1.0, (0, 0, 0, 0), (1, 1, 1, 1),
                                               (H / R, H / R, H / R, 1.0), overrideSize=(H, H, H, T),
                                               bordSkip=int(H * 0.1))
        F.loadAdvectTimeSlice_Finish(1)
        F.loadAdvectTimeSlice_Finish(2)
        return st["keep"][4]
    if op == "resample":
        (F.interpolateGrid4dVec if c["vec"] else F.interpolateGrid4d)(st["dst"], st["src"])
        return st["keep"][1]
    if op == "error":
        return F.calcLsDiff4d(st["i0"], st["i1"], correction=0.1 / 20.0, bnd=2)
    if op == "condition":
        st["phi"].copyFrom(st["src"])
        S.postProcessPhiData(st["phi"], loadOffset=st["off"], ofsd=st["ofsd"])
        return st["keep"][1]
    if c["grad"]:
        loss, g = st["model"].loss_grad(st["i0"], st["i1"], st["tgt"])
        return loss, g
    st["model"].predict(st["i0"], st["i1"], st["out"])
    return st["keep"][3]


def _frame_time(c, k):
    return k * (c["T"] - 1) // max(1, c["frames"] - 1) + 0.5


# --- what a pass cannot do without -----------------------------------------

def _solve_work(dims, solver):
    """Inputs once, the deformation once; the operations of the conjugate
    gradients (about 1.8 X iterations per solve and two solves a level with
    Jacobi, 9 with the multigrid; about 170 operations per cell and iteration)
    and of the blurs (two passes of 625 taps, or 40 separable ones)."""
    X, Y, Z, T = dims
    cells = X * Y * Z * T
    it = 2 * (1.8 * X if solver == "pcg" else 9 * 2.5)
    blur = 2 * 2 * (625 * 8 if solver == "pcg" else 40 * 4)
    return dict(bytes=24.0 * cells, flops=cells * (it * 170.0 + blur))


def work(c):
    op = c["op"]
    if op == "solve":
        return _solve_work(_dims(c), c["solver"])
    if op == "batch":
        w = [_solve_work(d, "pcg") for d in _batch_dims(c, 0)]
        return dict(bytes=sum(a["bytes"] for a in w), flops=sum(a["flops"] for a in w))
    if op == "frames":
        R, H, n = c["R"], c["H"], c["frames"]
        # per frame: two deformation slices and about one time slice of phi each way, the frame once
        return dict(bytes=n * (2 * 2 * 16.0 * R ** 3 + 3 * 4.0 * H ** 3), flops=n * H ** 3 * 2 * 120.0)
    if op == "condition":
        cells = c["res"] ** 4 * 3 // 2
        return dict(bytes=8.0 * cells, flops=cells * 2 * 40.0)
    if op == "net":
        R, f = c["R"], 0.0
        for (cin, cout, k, _), div in zip(NET, [1, 2, 2, 4, 4, 2, 1, 1]):
            f += 2.0 * k ** 4 * cin * cout * (R / div) ** 4
        n = sum(k ** 4 * a * b + b for a, b, k, _ in NET)
        g = c["grad"]
        return dict(bytes=R ** 4 * (8.0 + 16.0) + n * (2.0 + (4.0 if g else 0.0)), flops=f * (3.0 if g else 1.0))
    X, Y, Z, T = _dims(c)
    cells = X * Y * Z * T
    if op == "flow":
        return dict(bytes=24.0 * cells, flops=cells * 1.8 * X * 170.0)
    if op == "project":
        # three rounds: the projection, about X/2 sweeps of 324 adds, two blur passes
        return dict(bytes=(16 + 4 + 4 + 32.0) * cells, flops=cells * (3 * X / 2 * 324.0 + 2 * (5000 + 2 * 650)))
    if op == "deform":
        return dict(bytes=44.0 * cells, flops=cells * 2 * 80.0)
    if op == "resample":
        a, b, e, f = _res_of(c)
        nc = 4 if c["vec"] else 1
        return dict(bytes=4.0 * nc * (cells + a * b * e * f), flops=a * b * e * f * 46.0 * nc)
    return dict(bytes=8.0 * cells, flops=6.0 * cells)


# --- 64-bit values ------------------------------------------------------------

def _axis(p, n):
    px = p - 0.5
    b = torch.trunc(px)
    w = px - b
    w = torch.where(px < 0, torch.zeros_like(w), w)
    b = torch.where(px < 0, torch.zeros_like(b), b)
    hi = b >= n - 1
    w = torch.where(hi, torch.ones_like(w), w)
    b = torch.where(hi, torch.full_like(b, n - 2), b)
    return b.long(), w


def _sample(a, pos):
    """Multilinear sample of a (..., Z, Y, X) tensor, or (..., Z, Y, X, 4), at
    positions pos = [x, y, z(, t)] (cell centres at index + 0.5)."""
    n = len(pos)
    vec = a.dim() == n + 1
    shape = list(a.shape[:n])
    flat = a.reshape(-1, a.shape[-1]) if vec else a.reshape(-1)
    stride, base, ws = 1, 0, []
    strides = []
    for k in range(n):
        ext = shape[n - 1 - k]
        b, w = _axis(pos[k], ext)
        base = base + b * stride
        ws.append(w)
        strides.append(stride)
        stride *= ext
    out = 0.0
    for corner in range(1 << n):
        w, idx = 1.0, base
        for k in range(n):
            if corner >> k & 1:
                w, idx = w * ws[k], idx + strides[k]
            else:
                w = w * (1.0 - ws[k])
        val = flat[idx].double()
        out = out + (val * w.unsqueeze(-1) if vec else val * w)
    return out


def _exact_advect(phi, vel, dt, t):
    """Plane t of the semi-Lagrangian advection, zero on the border ring."""
    T, Z, Y, X = phi.shape
    x, y, z, _ = _axes((X, Y, Z, T), torch.float64)
    v = vel[t].double() * dt
    e = (Z, Y, X)
    pos = [(x[0] + 0.5).expand(e) - v[..., 0], (y[0] + 0.5).expand(e) - v[..., 1],
           (z[0] + 0.5).expand(e) - v[..., 2], (t + 0.5) - v[..., 3]]
    o = _sample(phi, pos)
    if t < 1 or t >= T - 1:
        return torch.zeros_like(o)
    m = torch.zeros_like(o)
    m[1:-1, 1:-1, 1:-1] = o[1:-1, 1:-1, 1:-1]
    return m


def _exact_flow(dims, i0, i1):
    """Conjugate gradients in 64 bits with the same preconditioner and stop rule."""
    X, Y, Z, T = dims
    wS, wE, acc = 0.001, 0.0001, 1e-4
    a, b = i0.double(), i1.double()
    inner = (slice(1, -1),) * 4
    g = torch.zeros(b.shape + (4,), device=DEV, dtype=torch.float64)
    for c, ax in enumerate((3, 2, 1, 0)):
        d = (torch.roll(b, -1, ax) - torch.roll(b, 1, ax)) * (X / 2.0)
        g[inner + (c,)] = d[inner]
    r = torch.zeros_like(g)
    r[inner] = (-g * (b - a).unsqueeze(-1))[inner]
    diag = 8 * wS + wE
    pre = torch.zeros_like(g)
    pre[inner] = (1.0 / (g * g + diag))[inner]

    def mul(p):
        q = torch.zeros_like(p)
        s = sum(torch.roll(p, k, ax) for ax in range(4) for k in (-1, 1))
        q[inner] = (g * (g * p).sum(-1, keepdim=True) + diag * p - wS * s)[inner]
        return q

    x = torch.zeros_like(r)
    res0 = max(float(r.max()), 0.0)
    p = pre * r
    sigma = (p * r).sum()
    for _ in range(1000):
        q = mul(p)
        alpha = sigma / (p * q).sum()
        x += alpha * p
        r -= alpha * q
        if max(float(r.max()), 0.0) <= acc * res0:
            break
        z = pre * r
        new = (z * r).sum()
        p = z + (new / sigma) * p
        sigma = new
    return x * X


def _exact_net(c, seed):
    p, i0, i1, tgt, dims = _net_inputs(c, seed)
    p = p.to(DEV).double().requires_grad_(c["grad"])
    R = c["R"]
    off, ws = 0, []
    for cin, cout, k, _ in NET:
        n = k ** 4 * cin * cout
        ws.append((p[off:off + n].view(k ** 4, cin, cout), p[off + n:off + n + cout]))
        off += n + cout

    def conv(a, l):
        cin, cout, k, s = NET[l]
        w, b = ws[l]
        if k == 1:
            return a @ w[0] + b
        r = a.shape[0] // s
        ap = torch.nn.functional.pad(a, (0, 0) + (1, 1) * 4)
        o = 0.0
        for tap in range(81):
            ox, oy, oz, ot = tap % 3, tap // 3 % 3, tap // 9 % 3, tap // 27
            o = o + ap[ot:ot + s * r:s, oz:oz + s * r:s, oy:oy + s * r:s, ox:ox + s * r:s] @ w[tap]
        return torch.relu(o + b)

    def up(a, skip):
        for ax in range(4):
            a = a.repeat_interleave(2, ax)
        return torch.cat([a, skip], -1)

    a0 = conv(torch.stack([i0, i1], -1).double() * -200.0, 0)
    a2 = conv(conv(a0, 1), 2)
    a4 = conv(conv(a2, 3), 4)
    out = conv(conv(up(conv(up(a4, a2), 5), a0), 6), 7)
    if not c["grad"]:
        return out
    loss = ((out - tgt.double()) ** 2).mean()
    loss.backward()
    return float(loss), p.grad.cpu().numpy()


def exact(c, seed):
    op = c["op"]
    if op == "deform":
        dims, p0, p1, v, w = _inputs(c, seed)
        al = c["alpha"]
        return torch.stack([_exact_advect(p0, v, al, t) * (1.0 - al) + al * _exact_advect(p1, w, 1.0 - al, t)
                            for t in range(dims[3])])
    if op == "frames":
        d, h, p0, p1, v, w = _inputs(c, seed)
        H, R, al = c["H"], c["R"], c["alpha"]
        lo = max(10, int(H * 0.1))
        x, y, z, _ = _axes(h, torch.float64)
        e = (H, H, H)
        x, y, z = x[0].expand(e), y[0].expand(e), z[0].expand(e)
        fac, outs = R / H, []
        for k in range(c["frames"]):
            tm = _frame_time(c, k)
            t0 = min(int(tm), d[3] - 1)
            t1 = min(int(tm) + 1, d[3] - 1)
            o = 0.0
            for phi, vel, dt, wt in ((p0, v, al, 1.0 - al), (p1, w, 1.0 - al, al)):
                sl = 0.5 * vel[t0].double() + 0.5 * vel[t1].double()
                q = _sample(sl, [(x + 0.5) * fac, (y + 0.5) * fac, (z + 0.5) * fac])
                q = q * torch.tensor([1 / fac, 1 / fac, 1 / fac, 1.0], device=DEV, dtype=torch.float64) * dt
                o = o + wt * _sample(phi, [x + 0.5 - q[..., 0], y + 0.5 - q[..., 1], z + 0.5 - q[..., 2],
                                           (tm + 0.5) - q[..., 3]])
            m = torch.zeros_like(o)
            if H > 2 * lo:
                s = slice(lo, H - lo)
                m[s, s, s] = o[s, s, s]
            outs.append(m)
        return outs
    if op == "resample":
        dims, a = _inputs(c, seed)
        td = _res_of(c)
        x, y, z, _ = _axes(td, torch.float64)
        f = [dims[k] / td[k] for k in range(4)]
        e = (td[2], td[1], td[0])
        return torch.stack([_sample(a, [(x[0] * f[0] + f[0] * 0.5).expand(e), (y[0] * f[1] + f[1] * 0.5).expand(e),
                                        (z[0] * f[2] + f[2] * 0.5).expand(e),
                                        torch.full(e, t * f[3] + f[3] * 0.5, device=DEV, dtype=torch.float64)])
                            for t in range(td[3])])
    if op == "error":
        dims, i0, i1 = _inputs(c, seed)
        s = (slice(2, -2),) * 4
        a, b = i0[s].double(), i1[s].double()
        same = ((a < 0) & (b < 0)) | ((a >= 0) & (b >= 0))
        d = torch.where(same, torch.zeros_like(a), ((a - b).abs() * (0.1 / 20.0)).clamp(max=1.0))
        return float(d.sum() * 1e6 / a.numel())
    if op == "flow":
        return _exact_flow(*_inputs(c, seed))
    if op == "net":
        return _exact_net(c, seed)
    return None
