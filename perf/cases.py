"""The measured cases: the calls of a time step and of the learned preconditioner's life, through the public
entry points, from the smallest grids to the largest.

Every case names its `kind`:

  projection   the pressure projection of a time step: right-hand side, the Poisson solve from zero, the
               three velocity corrections (plain FP64 CG, mixed-precision CG, the learned two-level FCG)
  momentum     the three implicit momentum predictors of a time step on a closed cavity or a channel
  scalar       the upwind concentration equation of a time step on a channel
  apply        one operator row evaluation y = A x - s with the dot (x, y), as a Krylov iteration calls it
  lines        the tridiagonal lines of the three ADI sweeps over a box
  markers      the immersed boundary of one time step: velocities at the markers, their forces, the spreading
  conv         one 3x3x3 convolution layer of the network on the tensor cores
  train        one training step (forward, backward, Adam) of the network on a (residual, error) pair

The solves run to the round-off of their FP64 refinement (1e-12), not to the default 1e-8, so that two correct
solvers agree to the precision of the velocities that they return.  A pressure is defined up to a constant per
closed region; what a projection gives its caller is the velocities.
"""
import ctypes as C
import math

import numpy as np
import torch

import xflow_gb300 as xf
from xflow_gb300 import capi, workloads
from xflow_gb300 import timeloop as tl

RTOL = 1e-12
SIZES = ("nx", "ny", "nz")


def listed():
    return [
        # the row evaluation of the smallest systems, where one launch and one scalar read back are all there is
        dict(name="apply_vardiv_ragged_33x29x27", kind="apply", op="vardiv", nx=33, ny=29, nz=27),
        # the same rows at the largest size, the constant-density operator
        dict(name="apply_laplace_256", kind="apply", op="laplace", nx=256, ny=256, nz=256),
        # the closed cavity of 64^3, all in FP64
        dict(name="projection_cavity_64_fp64", kind="projection", solver="fp64", nx=64, ny=64, nz=64, length=1.0,
             spheres=0, inflow=0.0),
        # the immersed-body channel with the spheres in the mask, mixed-precision CG
        dict(name="projection_channel_256x64x64_mixed", kind="projection", solver="mixed", nx=256, ny=64, nz=64,
             length=4.0, spheres=3, inflow=1.0),
        # a ragged box (odd rows: no fused path takes it)
        dict(name="projection_ragged_75x61x83_mixed", kind="projection", solver="mixed", nx=75, ny=61, nz=83,
             length=1.0, spheres=5, inflow=0.0),
        # the headline: 256^3 with 64 spheres, the learned two-level preconditioner
        dict(name="projection_spheres_256_learned", kind="projection", solver="learned", nx=256, ny=256, nz=256,
             length=1.0, spheres=64, inflow=0.0),
        # the momentum predictors of the small cavity and of the largest channel
        dict(name="momentum_cavity_64", kind="momentum", flow="cavity", nx=64, ny=64, nz=64),
        dict(name="momentum_channel_512x128x128", kind="momentum", flow="channel", nx=512, ny=128, nz=128),
        # the passive scalar of the middle channel
        dict(name="scalar_channel_256x64x64", kind="scalar", flow="channel", nx=256, ny=64, nz=64),
        # the ADI sweeps of a box of 128^3
        dict(name="lines_128", kind="lines", nx=128, ny=128, nz=128),
        # the sphere's 2,562 markers in the middle channel
        dict(name="markers_2562_channel_256x64x64", kind="markers", nx=256, ny=64, nz=64, subdiv=4),
        # training at the size the network is trained at
        dict(name="train_64", kind="train", nx=64, ny=64, nz=64),
    ]


def _log(rng, lo, hi, step=1, offset=0):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step + offset


def draw(rng):
    kind = rng.choice(["apply", "projection", "projection", "projection", "momentum", "scalar", "lines", "markers",
                       "conv", "train"])
    if kind == "apply":
        return dict(kind=kind, op=rng.choice(["laplace", "vardiv"]),
                    **{d: _log(rng, 16, 256) for d in SIZES})
    if kind == "projection":
        solver = rng.choice(["fp64", "mixed", "learned"])
        if solver == "learned":   # blocks of 4^3 whose coarse box halves twice: multiples of 16
            n = {d: _log(rng, 32, 192, 16) for d in SIZES}
        else:
            n = {d: _log(rng, 16, 128) for d in SIZES}
        inflow = rng.choice([0.0, 1.0])
        return dict(kind=kind, solver=solver, **n, length=n["nx"] / n["nz"], spheres=rng.choice([0, 2, 6]),
                    inflow=inflow)
    if kind in ("momentum", "scalar"):
        flow = "channel" if kind == "scalar" else rng.choice(["cavity", "channel"])
        return dict(kind=kind, flow=flow, **{d: _log(rng, 16, 160) for d in SIZES})
    if kind == "lines":
        return dict(kind=kind, **{d: _log(rng, 8, 200) for d in SIZES})
    if kind == "markers":
        return dict(kind=kind, nx=_log(rng, 64, 256), ny=_log(rng, 32, 96), nz=_log(rng, 32, 96),
                    subdiv=rng.choice([2, 3, 4, 5]))
    if kind == "conv":
        ci, co = rng.choice([(16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (96, 32), (48, 16)])
        return dict(kind=kind, ci=ci, co=co, relu=rng.choice([True, False]), **{d: _log(rng, 8, 80) for d in SIZES})
    return dict(kind=kind, **{d: _log(rng, 16, 64, 4) for d in SIZES})


# ---------------------------------------------------------------------------
# Inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


class _Raw:
    """The device box of a Vec as torch sees it: no copy, and the Vec (with its grid and context) lives as long as
    any tensor over it does."""

    def __init__(self, vec):
        self.vec = vec
        self.__cuda_array_interface__ = dict(data=(int(capi.lib().xf_vec_data(vec.h)), False), version=2, strides=None,
                                             shape=tuple(vec.grid.shape),
                                             typestr="<f8" if vec.dtype == xf.XF_F64 else "<f4")


def _view(v):
    return torch.as_tensor(_Raw(v), device="cuda")


def _put(grid, t, dtype=xf.XF_F64):
    """A Vec of `grid` holding the torch box t."""
    v = grid.vec(None, dtype)
    grid.ctx.synchronize()
    _view(v).copy_(t)
    torch.cuda.synchronize()
    return v


def _shape(case):
    return tuple(case[d] for d in SIZES)


def _solid(case, g, h):
    """Point codes of the pressure box: Actual interior, Fictive ghost layer and spheres (clear of the channel's
    ends), single cells without an open face Fictive too."""
    n = _shape(case)
    act = torch.zeros([m + 2 for m in n], dtype=torch.bool, device="cuda")
    act[1:-1, 1:-1, 1:-1] = True
    ext = [n[d] * h[d] for d in range(3)]
    if case["spheres"]:
        small = min(ext)
        c = torch.rand((case["spheres"], 3), generator=g, device="cuda", dtype=torch.float64).cpu().numpy()
        r = torch.rand(case["spheres"], generator=g, device="cuda", dtype=torch.float64).cpu().numpy()
        for q in range(case["spheres"]):
            rad = small * ((0.02 + 0.04 * r[q]) if case["spheres"] > 8 else (0.05 + 0.08 * r[q]))
            ctr = [rad + c[q, d] * (ext[d] - 2 * rad) for d in range(3)]
            if case["inflow"]:
                ctr[0] = ext[0] * (0.25 + 0.5 * c[q, 0])
            lo = [max(1, int((ctr[d] - rad) / h[d]) - 1) for d in range(3)]
            hi = [min(n[d] + 1, int((ctr[d] + rad) / h[d]) + 3) for d in range(3)]
            x = [(torch.arange(lo[d], hi[d], device="cuda", dtype=torch.float64) - 0.5) * h[d] - ctr[d] for d in range(3)]
            inside = x[0][:, None, None] ** 2 + x[1][None, :, None] ** 2 + x[2][None, None, :] ** 2 < rad * rad
            act[lo[0]:hi[0], lo[1]:hi[1], lo[2]:hi[2]] &= ~inside
    near = torch.zeros_like(act)
    for d in range(3):
        near |= torch.roll(act, 1, d) | torch.roll(act, -1, d)
    return act & near


def _faces(act, d):
    """Both cells of each face across axis d active; exactly one active, the face inside the box's walls or on them."""
    m = act.shape[d]
    a, b = act.narrow(d, 0, m - 1), act.narrow(d, 1, m - 1)
    return a & b, a ^ b


def _projection_inputs(case, seed):
    g = _gen(seed)
    n = _shape(case)
    h = [case["length"] / n[0], 1.0 / n[1], 1.0 / n[2]]
    if case["solver"] == "learned":
        h = [1.0 / n[2]] * 3   # the network's grid has cubic cells
    act = _solid(case, g, h)
    comps = []
    for d in range(3):
        both, one = _faces(act, d)
        t = torch.randn(both.shape, generator=g, device="cuda", dtype=torch.float64) * 0.1
        border = torch.zeros_like(t)
        if d == 0 and case["inflow"]:
            border[0][one[0]] = case["inflow"]
            border[-1][one[-1]] = case["inflow"]
            t += case["inflow"]
        t = torch.where(both, t, torch.where(one, border, torch.zeros_like(t)))
        codes = (both.int() + 3 * one.int()).to(torch.int32)
        comps.append((codes, t, border))
    return act, h, comps


def _multilevel_params():
    """Weights of the network as a linear three-level smoother (the signal in channel 0, its negative part in
    channel 1): coarse levels weigh 4 and 16 times the fine one's, the coarsest one is smoothed twice.  It
    stands for trained weights, which no file of the repository holds, and converges like them."""
    box = np.array([1.0, 2.0, 1.0])
    ker = (box[:, None, None] * box[None, :, None] * box[None, None, :] / 64.0).reshape(27)   # sum 1
    ident = np.zeros(27)
    ident[13] = 1.0
    spread = ident + 2.0 * ker

    def layer(ci, co, taps, out=False):
        w = np.zeros((27, co, ci))
        for src, ker27 in taps:
            for o, so in ((0, 1.0),) if out else ((0, 1.0), (1, -1.0)):
                w[:, o, src] += so * ker27
                if src or ci > 16 or not first:
                    w[:, o, src + 1] -= so * ker27
        return w

    parts = []
    for name, ci, co in xf.UNET_LAYERS:
        first = name == "enc0a"
        if name in ("enc0a", "enc0b", "enc1a", "enc1b"):
            taps = [(0, ident)]
        elif name in ("mid_a", "mid_b"):
            taps = [(0, spread)]
        elif name == "dec1a":
            taps = [(0, 4.0 * ker), (64, ident)]
        elif name == "dec0a":
            taps = [(0, 4.0 * ker), (32, ident)]
        else:
            taps = [(0, ker)] if name != "out" else [(0, ident)]
        parts += [layer(ci, co, taps, name == "out").ravel(), np.zeros(co)]
    return np.concatenate(parts).astype(np.float32)


def _prepare_projection(case, seed):
    act, h, comps = _projection_inputs(case, seed)
    ctx = xf.Context(0)
    sep = [np.full(act.shape[d] - 1, h[d]) for d in range(3)]
    codes = act.int().cpu().numpy()
    gp = xf.Grid(ctx, codes, *sep)
    s = dict(ctx=ctx, gp=gp, tau=1e-3, solver=case["solver"], A=xf.Operator(gp, xf.XF_OP_LAPLACE),
             p=gp.vec(None), rhs=gp.vec(None), prev=[], border=[], vel=[])
    for d, (cc, t, border) in enumerate(comps):
        hh = [sep[a][:-1] if a == d else sep[a] for a in range(3)]
        g = xf.Grid(ctx, cc.cpu().numpy(), *hh)
        s["prev"].append(_put(g, t))
        s["border"].append(_put(g, border))
        s["vel"].append(g.vec(None))
    if case["solver"] == "learned":
        cc, c1, c2, c3 = workloads.coarse_grid(codes, sep[0], 4)
        s["net"] = xf.UNet(xf.Grid(ctx, cc, c1, c2, c3), params=_multilevel_params())
    s["out"] = [_view(v) for v in s["vel"]]
    return s


def _run_projection(s):
    xf.pressure_rhs(s["gp"], *s["prev"], s["tau"], s["rhs"])
    s["p"].fill(0.0)
    if s["solver"] == "learned":
        st = xf.solve_fcg(s["A"], s["p"], s["rhs"], unet=s["net"], precond=xf.XF_PRECOND_UNET2, rtol=RTOL, window=1,
                          degree=4, ratio=6, precision=xf.XF_PREC_MIXED)
    else:
        st = xf.solve(s["A"], s["p"], s["rhs"], method=xf.XF_CG, rtol=RTOL,
                      precision=xf.XF_PREC_MIXED if s["solver"] == "mixed" else xf.XF_PREC_FP64)
    if st.status != capi.XF_OK:
        raise xf.XFError(st.status, "pressure")
    for d in range(3):
        xf.velocity_correct(d + 1, s["prev"][d], s["p"], s["tau"], s["vel"][d], border=s["border"][d])
    return s["out"]


def _exact_projection(case, seed):
    act, h, comps = _projection_inputs(case, seed)
    tau = 1e-3
    both = [(c == 1).double() for c, _, _ in comps]
    vel = [t for _, t, _ in comps]

    def div(f, out):
        out.zero_()
        for d in range(3):
            m = act.shape[d]
            out.narrow(d, 1, m - 2).add_(f[d].narrow(d, 1, m - 2) - f[d].narrow(d, 0, m - 2), alpha=1.0 / h[d])
        return out

    def grad(p, d):
        m = act.shape[d]
        return (p.narrow(d, 1, m - 1) - p.narrow(d, 0, m - 1)) * both[d] / h[d]

    a = act.double()
    diag = torch.zeros_like(a)
    for d in range(3):
        m = act.shape[d]
        diag.narrow(d, 0, m - 1).add_(both[d], alpha=1.0 / h[d] ** 2)
        diag.narrow(d, 1, m - 1).add_(both[d], alpha=1.0 / h[d] ** 2)
    diag = torch.where(diag > 0, diag, torch.ones_like(diag))
    buf = torch.zeros_like(a)
    b = -(div(vel, buf) * a) / tau
    p, r = torch.zeros_like(a), b.clone()
    z = r / diag
    q = z.clone()
    rz, bb = (r * z).sum(), float((b * b).sum())
    for it in range(20000):
        ap = -(div([grad(q, d) for d in range(3)], buf) * a)
        alpha = rz / (q * ap).sum()
        p.addcmul_(alpha, q)
        r.addcmul_(-alpha, ap)
        if it % 20 == 19 and float((r * r).sum()) <= 1e-28 * bb:
            break
        z = r / diag
        new = (r * z).sum()
        q.mul_(new / rz).add_(z)
        rz = new
    return [vel[d] - tau * grad(p, d) for d in range(3)]


# ---------------------------------------------------------------------------
def _smooth(shape, g, modes=4):
    """A smooth seeded field of unit scale: a few low modes of a box."""
    out = torch.zeros(shape, dtype=torch.float64, device="cuda")
    x = [torch.linspace(0, 1, m, dtype=torch.float64, device="cuda") for m in shape]
    k = torch.randint(1, 4, (modes, 3), generator=g, device="cuda").cpu().tolist()
    ph = (torch.rand((modes, 4), generator=g, device="cuda", dtype=torch.float64)).cpu().tolist()
    for q in range(modes):
        f = [torch.cos(2 * math.pi * (k[q][d] * x[d] + ph[q][d])) for d in range(3)]
        out += (ph[q][3] + 0.5) / modes * f[0][:, None, None] * f[1][None, :, None] * f[2][None, None, :]
    return out


def _flow(case, seed):
    """The statement of a cavity or channel with a developed flow: Defined and PreDefined points consistent with
    their border values."""
    g = _gen(seed)
    n = _shape(case)
    pshape = tuple(m + 2 for m in n)
    cavity = case["flow"] == "cavity"
    length = 1.0 if cavity else 4.0
    hs = [length / n[0], 1.0 / n[1], 1.0 / n[2]]
    sep = [np.full(pshape[d] - 1, hs[d]) for d in range(3)]
    faces = [{(2, 1): 1.0}, {}, {}] if cavity else [{(0, 0): 1.0, (0, 1): 1.0}, {}, {}]
    comps = []
    for d in range(3):
        codes, nrm, bc = tl.velocity_box(pshape, d, faces[d])
        bt = torch.from_numpy(bc).cuda()
        ct = torch.from_numpy(codes).cuda()
        v = 0.3 * _smooth(codes.shape, g) + 0.02 * torch.randn(codes.shape, generator=g, device="cuda",
                                                               dtype=torch.float64)
        if d == 0 and not cavity:
            v += 1.0
        v = torch.where(ct == 1, v, torch.where(ct == 3, bt, torch.zeros_like(v)))
        v = _ghosts(v, bt, d)
        comps.append(dict(codes=codes, nrm=nrm, bc=bt, v=v, sep=[sep[a][:-1] if a == d else sep[a] for a in range(3)]))
    return dict(pshape=pshape, sep=sep, hs=hs, comps=comps, vis=0.01 if cavity else 0.005,
                tau=1e-3 if cavity else 2e-3)


def _ghosts(v, bc, d):
    """The PreDefined face points of component d (the faces tangential to it) as 2 border - neighbour."""
    v = v.clone()
    for a in range(3):
        if a == d:
            continue
        m = v.shape[a]
        for side, inner in ((0, 1), (m - 1, m - 2)):
            sl = [slice(1, -1)] * 3
            sl[a] = side
            nb = list(sl)
            nb[a] = inner
            v[tuple(sl)] = 2 * bc[tuple(sl)] - v[tuple(nb)]
    return v


def _prepare_momentum(case, seed):
    f = _flow(case, seed)
    ctx = xf.Context(0)
    pc = np.zeros(f["pshape"], np.int32)
    pc[1:-1, 1:-1, 1:-1] = 1
    gp = xf.Grid(ctx, pc, *f["sep"])
    s = dict(ctx=ctx, gp=gp, tau=f["tau"], vis=_put(gp, torch.full(f["pshape"], f["vis"], dtype=torch.float64,
                                                                   device="cuda")), eq=[])
    for c in f["comps"]:
        g = xf.Grid(ctx, c["codes"], *c["sep"], c["nrm"])
        s["eq"].append(dict(g=g, v=_put(g, c["v"]), bc=_put(g, c["bc"]), mid=g.vec(None), rhs=g.vec(None),
                            tr=tuple(g.vec(None) for _ in range(5)), A=xf.Operator(g, xf.XF_OP_ADVDIFF)))
    s["out"] = [_view(e["mid"]) for e in s["eq"]] + [_view(e["rhs"]) for e in s["eq"]]
    return s


def _run_momentum(s):
    vel = [e["v"] for e in s["eq"]]
    for d, e in enumerate(s["eq"]):
        u, v, w, vis, rp = xf.momentum_rhs(d + 1, e["g"], *vel, vis=s["vis"], border=e["bc"], out=e["tr"])
        e["A"].set_advection(u, v, w, s["tau"], 0.0, capi.XF_ADV_CONVECTIVE | capi.XF_ADV_DIFFUSIVE)
        e["A"].set_diffusion_field(vis)
        xf.transfer_rhs(e["v"], rp, s["tau"], e["rhs"])
        e["mid"].assign(e["v"])
        st = xf.solve(e["A"], e["mid"], e["rhs"], method=xf.XF_BICGSTAB, precond=capi.XF_PRECOND_JACOBI,
                      atol=RTOL * e["rhs"].absmax()[0], maxit=20000)
        if st.status != capi.XF_OK:
            raise xf.XFError(st.status, "momentum")
        xf.border_recalc(e["mid"], e["bc"])
    return s["out"]


def _off(t, d, s):
    """The interior of t shifted by s along axis d."""
    sl = [slice(1, -1)] * 3
    m = t.shape[d]
    sl[d] = slice(1 + s, m - 1 + s)
    return t[tuple(sl)]


def _transport(f0, rhs, tr, D, hs, tau, upwind, ghosts):
    """The implicit transfer equation of the interior by Jacobi iteration (its rows are dominated by 1/tau)."""
    mid = (slice(1, -1),) * 3
    diag = 1.0 / tau
    off = []
    for d in range(3):
        h, v = hs[d], tr[d][mid]
        hhh = h * h * (2 * h) / 2
        if upwind:
            neg = (v < 0).double()
            diag = diag + 0.5 * v.abs() / h + 0.5 * D * 2 * h / hhh
            off.append((-(1 - neg) * 0.5 * v / h - 0.5 * D * h / hhh, neg * 0.5 * v / h - 0.5 * D * h / hhh))
        else:
            diag = diag + 0.5 * D * 2 * h / hhh
            off.append((-0.5 * v / (2 * h) - 0.5 * D * h / hhh, 0.5 * v / (2 * h) - 0.5 * D * h / hhh))
    f = f0.clone()
    for it in range(4000):
        f = ghosts(f)
        new = rhs[mid].clone()
        for d in range(3):
            new -= off[d][0] * _off(f, d, -1) + off[d][1] * _off(f, d, 1)
        new /= diag
        done = it % 10 == 9 and float((new - f[mid]).abs().max()) <= 1e-15 * float(new.abs().max())
        f[mid] = new
        if done:
            break
    return ghosts(f)


def _exact_momentum(case, seed):
    f = _flow(case, seed)
    mid = (slice(1, -1),) * 3
    v = [c["v"] for c in f["comps"]]
    outs, rhss = [], []
    for d in range(3):
        c = f["comps"][d]
        inner = [m - 2 for m in c["v"].shape]
        tr = []
        for a in range(3):
            full = torch.zeros_like(c["v"])
            if a == d:
                full[mid] = v[d][mid]
            else:   # the mean of the four neighbours of component a around the node
                acc = 0.0
                for sd in (0, 1):
                    for sa in (-1, 0):
                        sl = [slice(1, 1 + inner[x]) for x in range(3)]
                        sl[d] = slice(1 + sd, 1 + sd + inner[d])
                        sl[a] = slice(1 + sa, 1 + sa + inner[a])
                        acc = acc + v[a][tuple(sl)]
                full[mid] = acc / 4
            tr.append(full)
        vis = torch.zeros_like(c["v"])
        vis[mid] = f["vis"]
        rp = 0.0
        for a in range(3):
            dv = (_off(vis, a, 1) - _off(vis, a, -1)) / (2 * f["hs"][a])
            dvel = (_off(tr[d], a, 1) - _off(tr[d], a, -1)) / (2 * f["hs"][a])
            dmix = (_off(tr[a], d, 1) - _off(tr[a], d, -1)) / (2 * f["hs"][d])
            rp = rp + dv * (dvel + dmix)
        # border rows hold the border values; points off the active set the previous values
        codes = torch.from_numpy(c["codes"]).cuda()
        rhs = torch.where(codes == 4, c["bc"], v[d])
        rhs[mid] = v[d][mid] / f["tau"] + rp
        rhss.append(rhs)
        outs.append(_transport(v[d], rhs, tr, f["vis"], f["hs"], f["tau"], False, lambda x: _ghosts(x, c["bc"], d)))
    return outs + rhss


# ---------------------------------------------------------------------------
def _scalar_inputs(case, seed):
    f = _flow(case, seed)
    g = _gen(seed + 1000003)
    shape = f["pshape"]
    inlet_face = torch.from_numpy(tl.gaussian_inlet(shape, f["sep"], sigma=0.15)).cuda()
    codes, nrm = tl.scalar_box(shape, np.ones(shape[1:], bool))
    ct = torch.from_numpy(codes).cuda()
    inlet = torch.zeros(shape, dtype=torch.float64, device="cuda")
    inlet[0] = torch.where(ct[0] == 4, inlet_face, torch.zeros_like(inlet_face))
    c = torch.where(ct == 1, (0.5 + 0.4 * _smooth(shape, g)).clamp(0, 1), torch.zeros(shape, dtype=torch.float64, device="cuda"))
    return f, codes, nrm, inlet, c


def _prepare_scalar(case, seed):
    f, codes, nrm, inlet, c = _scalar_inputs(case, seed)
    ctx = xf.Context(0)
    gc = xf.Grid(ctx, codes, *f["sep"], nrm)
    s = dict(ctx=ctx, g=gc, tau=f["tau"], D=f["vis"], inlet=_put(gc, inlet), c=_put(gc, c), nxt=gc.vec(None),
             rhs=gc.vec(None), tr=tuple(gc.vec(None) for _ in range(4)), A=xf.Operator(gc, xf.XF_OP_ADVDIFF), vel=[])
    for q in f["comps"]:
        s["vel"].append(_put(xf.Grid(ctx, q["codes"], *q["sep"], q["nrm"]), q["v"]))
    s["out"] = [_view(s["nxt"]), _view(s["rhs"])]
    return s


def _run_scalar(s):
    u, v, w, rp = xf.conc_transfer(s["g"], *s["vel"], inlet=s["inlet"], out=s["tr"])
    s["A"].set_advection(u, v, w, s["tau"], s["D"],
                         capi.XF_ADV_CONVECTIVE | capi.XF_ADV_DIFFUSIVE | capi.XF_ADV_UPWIND)
    xf.transfer_rhs(s["c"], rp, s["tau"], s["rhs"])
    s["nxt"].assign(s["c"])
    st = xf.solve(s["A"], s["nxt"], s["rhs"], method=xf.XF_BICGSTAB, precond=capi.XF_PRECOND_JACOBI,
                  atol=RTOL * s["rhs"].absmax()[0], maxit=20000)
    if st.status != capi.XF_OK:
        raise xf.XFError(st.status, "scalar")
    return s["out"]


def _exact_scalar(case, seed):
    f, codes, nrm, inlet, c = _scalar_inputs(case, seed)
    mid = (slice(1, -1),) * 3
    tr = []
    for d in range(3):
        full = torch.zeros_like(c)
        full[mid] = (_off_box(f["comps"][d]["v"], d, 0, c.shape) + _off_box(f["comps"][d]["v"], d, -1, c.shape)) / 2
        tr.append(full)

    def ghosts(x):
        x = x.clone()
        for a in range(3):
            m = x.shape[a]
            for side, inner in ((0, 1), (m - 1, m - 2)):
                sl = [slice(1, -1)] * 3
                sl[a] = side
                nb = list(sl)
                nb[a] = inner
                x[tuple(sl)] = x[tuple(nb)]
        face = (0, slice(1, -1), slice(1, -1))
        x[face] = 2 * inlet[face] - x[(1,) + face[1:]]
        return x

    ct = torch.from_numpy(codes).cuda()
    rhs = torch.where(ct == 4, inlet, torch.zeros_like(c))
    rhs[mid] = c[mid] / f["tau"]
    return [_transport(c, rhs, tr, f["vis"], f["hs"], f["tau"], True, ghosts), rhs]


def _off_box(v, d, s, shape):
    """Component d's face values at offset s of the interior cells of a box of `shape`."""
    sl = [slice(1, m - 1) for m in shape]
    sl[d] = slice(1 + s, shape[d] - 1 + s)
    return v[tuple(sl)]


# ---------------------------------------------------------------------------
def _apply_inputs(case, seed):
    g = _gen(seed)
    shape = tuple(m + 2 for m in _shape(case))
    act = torch.zeros(shape, dtype=torch.bool, device="cuda")
    act[1:-1, 1:-1, 1:-1] = True
    act &= torch.rand(shape, generator=g, device="cuda") > 0.05
    near = torch.zeros_like(act)
    for d in range(3):
        near |= torch.roll(act, 1, d) | torch.roll(act, -1, d)
    act &= near
    sep = []
    for m in shape:
        q = 1.0 + 0.2 * torch.rand(m - 1, generator=g, device="cuda", dtype=torch.float64).cpu().numpy()
        sep.append(q / q.sum() if case["op"] == "vardiv" else np.full(m - 1, 1.0 / (m - 2)))
    x = torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)
    s = torch.randn(shape, generator=g, device="cuda", dtype=torch.float64) / float(min(map(min, sep))) ** 2
    rho = 0.5 + 1.5 * torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)
    return act, sep, x, s, rho


def _prepare_apply(case, seed):
    act, sep, x, b, rho = _apply_inputs(case, seed)
    ctx = xf.Context(0)
    g = xf.Grid(ctx, act.int().cpu().numpy(), *sep)
    A = xf.Operator(g, xf.XF_OP_VARDIV, density=rho.cpu().numpy()) if case["op"] == "vardiv" else xf.Operator(g)
    s = dict(ctx=ctx, A=A, x=_put(g, x), b=_put(g, b), y=g.vec(None))
    s["out"] = _view(s["y"])
    return s


def _run_apply(s):
    dot = s["A"].apply(s["x"], s["y"], s=s["b"], sign=-1, want_dot=True)
    return [s["out"], dot]


def _exact_apply(case, seed):
    act, sep, x, b, rho = _apply_inputs(case, seed)
    y = torch.zeros_like(x)
    mid = (slice(1, -1),) * 3
    lap, ddens = 0.0, 0.0
    for d in range(3):
        h = torch.from_numpy(sep[d]).cuda()
        form = [1, 1, 1]
        form[d] = -1
        lo, hi = h[:-1].reshape(form), h[1:].reshape(form)
        up, dn = _off(act, d, 1).double(), _off(act, d, -1).double()
        ru, rd = (_off(rho, d, 1), _off(rho, d, -1)) if case["op"] == "vardiv" else (1.0, 1.0)
        lap = lap + (ru * up * (_off(x, d, 1) - x[mid]) / hi - rd * dn * (x[mid] - _off(x, d, -1)) / lo) / ((lo + hi) / 2)
        ddens = ddens + up * (_off(rho, d, 1) - rho[mid]) / lo
    row = -(rho[mid] * lap - ddens * x[mid]) if case["op"] == "vardiv" else -lap
    y[mid] = torch.where(act[mid], row - b[mid], torch.zeros_like(row))
    return [y, float((x * y).sum())]


# ---------------------------------------------------------------------------
def _lines_inputs(case, seed):
    g = _gen(seed)
    shape = tuple(m + 2 for m in _shape(case))
    rnd = lambda: torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    a, c = -(0.5 + rnd()), -(0.5 + rnd())
    b = 1.0 + rnd() - a - c
    f = 2 * rnd() - 1
    u = [2 * rnd() - 1 for _ in range(3)]
    return shape, a, b, c, f, u


def _prepare_lines(case, seed):
    shape, a, b, c, f, u = _lines_inputs(case, seed)
    ctx = xf.Context(0)
    codes, _ = workloads.neumann_box(*shape)
    grid = xf.Grid(ctx, codes, *[np.full(m - 1, 1.0 / (m - 2)) for m in shape])
    s = dict(ctx=ctx, shape=shape, abcf=[_put(grid, t) for t in (a, b, c, f)], u=[_put(grid, t) for t in u])
    s["out"] = [_view(v) for v in s["u"]]
    return s


def _run_lines(s):
    for axis in (1, 2, 3):
        M, nl1, nl2, ls1, ls2, ms = xf.box_lines(s["shape"], axis)
        xf.thomas_lines(s["ctx"], M, s["u"][axis - 1], *s["abcf"], nl1, nl2, ls1, ls2, ms)
    return s["out"]


def _exact_lines(case, seed):
    shape, a, b, c, f, u = _lines_inputs(case, seed)
    for d in range(3):
        M = shape[d] - 1
        at = lambda t, m: t.select(d, m)  # noqa: E731
        al, be = [torch.zeros_like(at(a, 0))], [at(u[d], 0).clone()]
        for m in range(1, M):
            den = at(a, m) * al[-1] + at(b, m)
            al.append(-at(c, m) / den)
            be.append((at(f, m) - at(a, m) * be[-1]) / den)
        for m in range(M - 1, 0, -1):
            at(u[d], m).copy_(al[m] * at(u[d], m + 1) + be[m])
    return u


# ---------------------------------------------------------------------------
def _marker_inputs(case, seed):
    g = _gen(seed)
    n = _shape(case)
    hs = [4.0 / n[0], 1.0 / n[1], 1.0 / n[2]]
    m = tl.sphere_markers((1.0, 0.5, 0.5), 0.15, subdiv=case["subdiv"])
    nn = len(m["pos"])
    m["pos"] = m["ref"] + 0.01 * torch.randn((nn, 3), generator=g, device="cuda", dtype=torch.float64).cpu().numpy()
    vel = []
    for d in range(3):
        shape = [q + 2 for q in n]
        shape[d] -= 1
        vel.append(0.3 * _smooth(shape, g) + (1.0 if d == 0 else 0.0))
    return hs, m, vel


def _prepare_markers(case, seed):
    hs, m, vel = _marker_inputs(case, seed)
    ctx = xf.Context(0)
    s = dict(ctx=ctx, h0=np.array(hs), vel=[], force=[], out=[])
    for v in vel:
        codes, _ = workloads.neumann_box(*v.shape)
        g = xf.Grid(ctx, codes, *[np.full(q - 1, h) for q, h in zip(v.shape, hs)])
        s["vel"].append(_put(g, v))
        s["force"].append(g.vec(None))
    s["m"] = xf.Markers(ctx, m["pos"], m["ref"], m["kind"], m["nxt"], m["prv"], m["dist0"], m["curv0"], m["stiff"],
                        m["params"])
    s["out"] = [_view(v) for v in s["force"]]
    return s


def _run_markers(s):
    for d in range(3):
        s["m"].interpolate(s["vel"][d], s["h0"], d + 1)
        s["m"].compute_forces(d + 1)
        s["m"].spread(s["force"][d], s["h0"], d + 1)
    return s["out"] + [s["m"].get(xf.XF_IB_VEL), s["m"].get(xf.XF_IB_FORCE)]


def _exact_markers(case, seed):
    hs, m, vel = _marker_inputs(case, seed)
    pos = torch.from_numpy(m["pos"]).cuda()
    ref = torch.from_numpy(m["ref"]).cuda()
    nn = len(pos)
    boxes, nvel, nforce = [], [], []
    for d in range(3):
        shape = vel[d].shape
        idx, wts = [], []
        for a in range(3):
            half = 0.5 * hs[a] if a != d else 0.0
            q = torch.floor((pos[:, a] + half) / hs[a]).long()
            q = q.clamp(max=shape[a] - 2 - 3).clamp(min=3)
            cells = q[:, None] + torch.arange(-3, 4, device="cuda")
            dist = (pos[:, a, None] - (cells * hs[a] - half)).abs()
            wts.append(torch.where(dist < 2 * hs[a], (1 + torch.cos(math.pi * dist / (2 * hs[a]))) / (4 * hs[a]),
                                   torch.zeros_like(dist)))
            idx.append(cells)
        w = wts[0][:, :, None, None] * wts[1][:, None, :, None] * wts[2][:, None, None, :]
        flat = ((idx[0][:, :, None, None] * shape[1] + idx[1][:, None, :, None]) * shape[2] + idx[2][:, None, None, :])
        nvel.append((vel[d].reshape(-1)[flat] * w).sum((1, 2, 3)) * hs[d] ** 3)
        force = -m["params"][0] * (pos[:, d] - ref[:, d]) * m["params"][3]
        nforce.append(force)
        box = torch.zeros(shape, dtype=torch.float64, device="cuda").reshape(-1)
        box.index_add_(0, flat.reshape(-1), (force[:, None, None, None] * w).reshape(-1))
        boxes.append(box.reshape(shape))
    return boxes + [torch.stack(nvel).cpu().numpy().reshape(3, nn), torch.stack(nforce).cpu().numpy().reshape(3, nn)]


# ---------------------------------------------------------------------------
def _conv_inputs(case, seed):
    g = _gen(seed)
    shape = tuple(m + 2 for m in _shape(case))
    mask = torch.zeros(shape, device="cuda")
    mask[1:-1, 1:-1, 1:-1] = 1
    mask *= torch.rand(shape, generator=g, device="cuda") > 0.05
    x = torch.randn(shape + (case["ci"],), generator=g, device="cuda").clamp(min=0).bfloat16() * mask[..., None].bfloat16()
    W = (torch.randn((27, case["co"], case["ci"]), generator=g, device="cuda") * math.sqrt(2.0 / (27 * case["ci"]))).bfloat16()
    bias = 0.1 * torch.randn(case["co"], generator=g, device="cuda")
    return shape, mask, x, W, bias


def _prepare_conv(case, seed):
    shape, mask, x, W, bias = _conv_inputs(case, seed)
    n = shape[0] * shape[1] * shape[2]
    margin = shape[1] * shape[2] + shape[2] + 1 + 128
    rows = n + 2 * margin
    xb = torch.zeros((case["ci"] // 8, rows, 8), dtype=torch.bfloat16, device="cuda")
    xb[:, margin:margin + n] = x.reshape(n, case["ci"] // 8, 8).permute(1, 0, 2)
    out = torch.zeros((n, case["co"]), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    return dict(ctx=xf.Context(0), shape=shape, xb=xb, first=xb.data_ptr() + margin * 16, ps=rows * 8, ci=case["ci"],
                co=case["co"], W=W.contiguous(), bias=bias, mask=mask.to(torch.uint8).contiguous(), out=out,
                relu=case["relu"])


def _run_conv(s):
    p = C.c_void_p
    st = capi.lib().xf_conv3d_bf16(s["ctx"].h, *s["shape"], p(s["first"]), s["ps"], s["ci"], p(s["W"].data_ptr()),
                                   p(s["bias"].data_ptr()), s["co"], p(s["mask"].data_ptr()), p(s["out"].data_ptr()),
                                   s["co"], s["co"], 1, int(s["relu"]))
    if st != capi.XF_OK:
        raise xf.XFError(st, "convolution")
    return s["out"]


def _conv64(x, W, b):
    """x [ci, ...box], W [27, co, ci] in 64 bits, zero outside the box."""
    k = W.permute(1, 2, 0).reshape(W.shape[1], W.shape[2], 3, 3, 3)
    return torch.nn.functional.conv3d(x[None], k, b, padding=1)[0]


def _exact_conv(case, seed):
    shape, mask, x, W, bias = _conv_inputs(case, seed)
    y = _conv64(x.double().permute(3, 0, 1, 2), W.double(), bias.double())
    if case["relu"]:
        y = y.clamp(min=0)
    return (y * mask.double()).permute(1, 2, 3, 0).reshape(-1, case["co"]).contiguous()


# ---------------------------------------------------------------------------
def _train_inputs(case, seed):
    """A (residual, error) pair as a partly converged solve leaves it: the error smooth, the residual its image."""
    g = _gen(seed)
    n = _shape(case)
    shape = tuple(m + 2 for m in n)
    act = torch.zeros(shape, dtype=torch.bool, device="cuda")
    act[1:-1, 1:-1, 1:-1] = True
    ctr = [0.5 * m for m in shape]
    x = [torch.arange(m, device="cuda", dtype=torch.float64) - c for m, c in zip(shape, ctr)]
    act &= x[0][:, None, None] ** 2 + x[1][None, :, None] ** 2 + x[2][None, None, :] ** 2 >= (0.2 * min(n)) ** 2
    e = torch.where(act, _smooth(shape, g, 6), torch.zeros(shape, dtype=torch.float64, device="cuda"))
    h = 1.0 / n[2]
    r = torch.zeros_like(e)
    mid = (slice(1, -1),) * 3
    acc = 0.0
    for d in range(3):
        for s in (-1, 1):
            acc = acc + _off(act, d, s).double() * (e[mid] - _off(e, d, s)) / h ** 2
    r[mid] = torch.where(act[mid], acc, torch.zeros_like(acc))
    return act, h, r, e


def _prepare_train(case, seed):
    act, h, r, e = _train_inputs(case, seed)
    ctx = xf.Context(0)
    g = xf.Grid(ctx, act.int().cpu().numpy(), *[np.full(m - 1, h) for m in act.shape])
    return dict(ctx=ctx, net=xf.UNet(g, params=xf.unet_init_params(seed)), A=xf.Operator(g), r=_put(g, r),
                e=_put(g, e))


def _run_train(s):
    loss = s["net"].train_step(s["r"], s["e"], lr=1e-3, update=True, op=s["A"])
    return [loss, s["net"].grads()]


def _exact_train(case, seed):
    act, h, r, e = _train_inputs(case, seed)
    flat = torch.from_numpy(xf.unet_init_params(seed)).cuda().double()
    P, leaf, o = {}, [], 0
    for name, ci, co in xf.UNET_LAYERS:
        w = flat[o:o + 27 * co * ci].reshape(27, co, ci).clone().requires_grad_()
        b = flat[o + 27 * co * ci:o + 27 * co * ci + co].clone().requires_grad_()
        o += 27 * co * ci + co
        P[name] = (w, b)
        leaf += [w, b]
    pool = torch.nn.functional.avg_pool3d
    inner = lambda t: t[..., 1:-1, 1:-1, 1:-1]  # noqa: E731
    padded = lambda t: torch.nn.functional.pad(t, (1,) * 6)  # noqa: E731
    M = [act.double()]
    for _ in range(2):
        M.append(padded((pool(inner(M[-1])[None, None], 2)[0, 0] > 0).double()))

    def layer(name, x, lev, relu=True):
        y = _conv64(x, *P[name])
        return (y.clamp(min=0) if relu else y) * M[lev]

    down = lambda t, lev: padded(pool(inner(t)[None], 2)[0]) * M[lev]  # noqa: E731
    up = lambda t, lev: padded(inner(t).repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)) * M[lev]  # noqa: E731
    x0 = torch.zeros((16,) + tuple(act.shape), dtype=torch.float64, device="cuda")
    x0[0] = r / torch.sqrt((r[act] ** 2).mean())
    s0 = layer("enc0b", layer("enc0a", x0, 0), 0)
    s1 = layer("enc1b", layer("enc1a", down(s0, 1), 1), 1)
    m2 = layer("mid_b", layer("mid_a", down(s1, 2), 2), 2)
    d1 = layer("dec1b", layer("dec1a", torch.cat([up(m2, 1), s1]), 1), 1)
    d0 = layer("dec0b", layer("dec0a", torch.cat([up(d1, 0), s0]), 0), 0)
    z = layer("out", d0, 0, relu=False)[0]
    mid = (slice(1, -1),) * 3
    az = 0.0
    for d in range(3):
        for s in (-1, 1):
            az = az + _off(act, d, s).double() * (z[mid] - _off(z, d, s)) / h ** 2
    zaz = (z[mid] * az * act[mid].double()).sum()
    loss = 1 - (z * r).sum() / torch.sqrt(zaz * (e * r).sum())
    grads = torch.autograd.grad(loss, leaf)
    return [float(loss), torch.cat([t.reshape(-1) for t in grads]).cpu().numpy()]


# ---------------------------------------------------------------------------
_PREPARE = dict(projection=_prepare_projection, momentum=_prepare_momentum, scalar=_prepare_scalar,
                apply=_prepare_apply, lines=_prepare_lines, markers=_prepare_markers, conv=_prepare_conv,
                train=_prepare_train)
_RUN = dict(projection=_run_projection, momentum=_run_momentum, scalar=_run_scalar, apply=_run_apply,
            lines=_run_lines, markers=_run_markers, conv=_run_conv, train=_run_train)
_EXACT = dict(projection=_exact_projection, momentum=_exact_momentum, scalar=_exact_scalar, apply=_exact_apply,
              lines=_exact_lines, markers=_exact_markers, conv=_exact_conv, train=_exact_train)


def prepare(case, seed):
    s = _PREPARE[case["kind"]](case, seed)
    s["kind"] = case["kind"]
    s["ctx"].synchronize()
    torch.cuda.synchronize()
    return s


def run(state):
    return _RUN[state["kind"]](state)


def exact(case, seed):
    return _EXACT[case["kind"]](case, seed)


def work(case):
    """Compulsory bytes (inputs read once, outputs written once) and operations: for a solve, those of one
    residual evaluation, since how many it takes is the solver's matter."""
    n = 1
    for d in SIZES:
        n *= case[d] + 2
    kind = case["kind"]
    if kind == "projection":
        return dict(bytes=n * (3 * 8 + 3 * 8 + 1), flops=n * (8 + 14 + 9))
    if kind == "momentum":
        return dict(bytes=n * (4 * 8 + 6 * 8 + 3), flops=3 * n * (30 + 20))
    if kind == "scalar":
        return dict(bytes=n * (4 * 8 + 2 * 8 + 1), flops=n * (6 + 20))
    if kind == "apply":
        vd = case["op"] == "vardiv"
        return dict(bytes=n * (3 * 8 + 8 * vd + 1), flops=n * (40 if vd else 20))
    if kind == "lines":
        return dict(bytes=3 * n * 5 * 8, flops=3 * n * 9)
    if kind == "markers":
        nn = 10 * 4 ** case["subdiv"] + 2
        return dict(bytes=3 * n * 8 + nn * (3 * 343 * 8 + 12 * 8), flops=nn * 3 * 343 * 8)
    flops = 2 * 27 * n * case.get("ci", 0) * case.get("co", 0)
    if kind == "conv":
        return dict(bytes=n * (2 * case["ci"] + 4 * case["co"] + 1), flops=flops)
    per, scale = 0, {"enc1a": 8, "enc1b": 8, "mid_a": 64, "mid_b": 64, "dec1a": 8, "dec1b": 8}
    for name, ci, co in xf.UNET_LAYERS:
        per += 2 * 27 * ci * co / scale.get(name, 1)
    return dict(bytes=n * (2 * 8 + 1) + 4 * 4 * 350000, flops=3 * n * per)
