"""What is measured of this framework: the work its users have it do, through
its public entry points (samrai_b200.fac), as plain-value cases.

Kinds of case:

* ``solve``: one FAC solve of every problem of a context from host buffers
  (``FacContext.solve_host``: right-hand side up, solution down), as an
  application does once per time step on a hierarchy it keeps.
* ``operators``: FACPreconditioner's own loop written over the level operators
  (``FacContext.smooth``, ``comp_residual``, ``restrict``, ...), as a program
  that brings its own cycle does, with the solution downloaded at the end.
* ``vectors``: the composite dot product and norms a Krylov or Newton method
  takes of device-resident vectors.
* ``regrid``: tagging by the adaption estimate and Berger-Rigoutsos clustering
  of the finest level of every problem.
* ``cnn_forward`` / ``cnn_gradients``: the correction network's prediction, and
  its loss and weight gradients, on a batch of patches.

The hierarchies are those of samrai_b200.configs (2-D base grid with refined
boxes; 3-D base grid with seeded random boxes at ratio 2), the coefficients
and right-hand sides its random fields and Gaussian bumps, made here on the
GPU from the seed.  A case fixes its hierarchy; the seed fixes the data on it.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from samrai_b200 import configs, fac

S = fac.CNN_BOX


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

# The solver settings in use: the reference's FAC semantics (two sweeps either
# side, up to 500 red-black sweeps on the coarsest level), and the cycle of the
# multigrid-extended variant (no pre-smoothing, three post-smoothing sweeps, 40
# sweeps on the coarsest extension level).
PLAIN = dict(pre=2, post=2, coarse_it=500)
FAST = dict(pre=0, post=3, coarse_it=40)


def _case(name, kind, **kw):
    c = dict(name=name, kind=kind)
    c.update(kw)
    return c


def _solve(name, dim, nx, **kw):
    c = dict(dim=dim, nx=nx, ny=nx, nlev=2 if dim == 2 else 3, nprob=1, hier=1, max_patch=16,
             max_patch0=32, block=8, var_d=False, var_c=False, robin=False, mixed=False, krylov=0,
             ext=0, max_cycles=100)
    c.update(PLAIN)
    c.update(kw)
    return _case(name, "solve", **c)


def listed():
    return [
        # the norms and dot product of one Newton-Krylov step on the smallest
        # hierarchy in use (64^2 base, one refined box): launches and latency
        _case("vectors_2d", "vectors", dim=2, nx=64, ny=64, nlev=2, hier=1, max_patch=32,
              max_patch0=64, block=8),
        # the same on a 128^3 base with two refined levels in 8..32-cell patches
        _case("vectors_3d", "vectors", dim=3, nx=128, ny=128, nlev=3, hier=2, max_patch=32,
              max_patch0=32, block=8),
        # one small 2-D Poisson solve with the reference's semantics: a short
        # chain of tiny launches and the 500-sweep coarsest solve
        _solve("solve_2d", 2, 64, max_patch0=64),
        # ragged 2-D grid, variable D and C, Robin sides
        _solve("solve_2d_var", 2, 57, ny=76, max_patch0=128, var_d=True, var_c=True, robin=True),
        # small 3-D AMR solve in FP64, base level in several patches (the
        # coarsest solve runs over patches), variable D
        _solve("solve_3d", 3, 32, hier=7, max_patch0=16, block=4, var_d=True, coarse_it=100),
        # one large constant-coefficient 3-D problem in FP64 (128^3 base in 32^3
        # patches), stationary FAC over the multigrid coarse extension
        _solve("solve_3d_large", 3, 128, hier=2, max_patch=32, ext=4, coarse_it=20),
        # a few variable-coefficient problems in one context, mixed precision
        # under FGMRES(20): an ordinary batch
        _solve("batch_4", 3, 0, nprob=4, var_d=True, mixed=True, krylov=20, ext=3, **FAST),
        # the batch that fills the GPU (about 25 million cells)
        _solve("batch_16", 3, 0, nprob=16, hier=20, var_d=True, mixed=True, krylov=20, ext=3,
               **FAST),
        # a program's own V-cycles over the level operators, FP64
        _case("operators_3d", "operators", dim=3, nx=48, ny=48, nlev=3, hier=5, max_patch=16,
              max_patch0=16, block=8, ext=2, cycles=3, var_d=True),
        # regrid step of a batch: tags and boxes of the finest levels
        _case("regrid_8", "regrid", nprob=8, hier=40, nx=0),
        # network prediction on the patches of a level, and a training batch
        _case("cnn_forward", "cnn_forward", batch=100),
        _case("cnn_gradients", "cnn_gradients", batch=256),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["vectors", "solve2", "solve2", "solve3", "batch", "batch", "operators",
                       "regrid", "cnn_forward", "cnn_gradients"])
    hier = rng.randrange(1, 100)
    if kind == "vectors":
        dim = rng.choice([2, 3])
        if dim == 2:
            c = _case("", "vectors", dim=2, nx=rng.randrange(24, 160), ny=rng.randrange(24, 160),
                      nlev=2, hier=hier, max_patch=rng.choice([16, 32, 48]),
                      max_patch0=rng.choice([32, 64, 160]), block=8)
        else:
            n = 8 * rng.randrange(4, 17)
            c = _case("", "vectors", dim=3, nx=n, ny=n, nlev=rng.choice([2, 3]), hier=hier,
                      max_patch=rng.choice([8, 16, 32]), max_patch0=32, block=8)
    elif kind == "solve2":
        c = _solve("", 2, rng.randrange(24, 97), ny=rng.randrange(24, 97), hier=hier,
                   max_patch0=rng.choice([128, 40, 41]), var_d=rng.random() < 0.5,
                   var_c=rng.random() < 0.3, robin=rng.random() < 0.3,
                   coarse_it=rng.randrange(100, 501), max_cycles=rng.randrange(10, 41))
    elif kind == "solve3":
        if rng.random() < 0.5:
            c = _solve("", 3, 4 * rng.randrange(5, 11), hier=hier, max_patch0=16, block=4,
                       var_d=rng.random() < 0.5, coarse_it=rng.randrange(40, 121),
                       max_cycles=rng.randrange(10, 31))
        else:
            c = _solve("", 3, 16 * rng.randrange(3, 9), hier=hier,
                       max_patch=rng.choice([16, 32]), ext=rng.choice([2, 3]), coarse_it=20,
                       var_d=rng.random() < 0.3)
        c["ny"] = c["nx"]
    elif kind == "batch":
        c = _solve("", 3, 0, hier=hier, nprob=_log_int(rng, 1, 12), var_d=True,
                   mixed=rng.random() < 0.75, krylov=rng.choice([0, 20, 20]), ext=3, **FAST)
    elif kind == "operators":
        n = 8 * rng.randrange(4, 9)
        c = _case("", "operators", dim=3, nx=n, ny=n, nlev=rng.choice([2, 3]), hier=hier,
                  max_patch=rng.choice([8, 16]), max_patch0=rng.choice([16, 32]), block=8, ext=2,
                  cycles=rng.randrange(1, 4), var_d=rng.random() < 0.7)
    elif kind == "regrid":
        c = _case("", "regrid", nprob=_log_int(rng, 1, 12), hier=hier, nx=0)
    else:
        c = _case("", kind, batch=_log_int(rng, 1, 256))
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# hierarchies (fixed by the case) and data on them (fixed by the seed)
# ---------------------------------------------------------------------------

def _split(n, side):
    """[0, n) in runs of at most `side` cells."""
    return [(a, min(a + side, n) - 1) for a in range(0, n, side)]


@functools.lru_cache(maxsize=None)
def _levels(dim, nx, ny, nlev, hier, max_patch, max_patch0, block):
    """Levels of one problem: 3-D as configs.build_3d_hierarchy; 2-D the base
    grid and a refined box over its middle half, in patches of max_patch."""
    if dim == 3:
        return tuple(configs.build_3d_hierarchy(hier, nx, nbox=(3, 3), nlev=nlev, block=block,
                                                side=(8, 48) if block == 8 else (8, 24),
                                                max_patch=max_patch, max_patch0=max_patch0)[0])
    base = [[x0, y0, 0, x1, y1, 0] for y0, y1 in _split(ny, max_patch0)
            for x0, x1 in _split(nx, max_patch0)]
    levels = [configs.Level((1, 1, 1), np.array(base, dtype=np.int32))]
    ox, oy = 2 * (nx // 4), 2 * (ny // 4)
    fine = [[ox + x0, oy + y0, 0, ox + x1, oy + y1, 0] for y0, y1 in _split(2 * (ny // 2), max_patch)
            for x0, x1 in _split(2 * (nx // 2), max_patch)]
    levels.append(configs.Level((2, 2, 1), np.array(fine, dtype=np.int32)))
    return tuple(levels)


def _nprob(case):
    return case.get("nprob", 1)


def _problems(case):
    """Problems without data.  nx = 0: base grids of 64..128 cells a side
    (a multiple of 8), drawn per problem from the hierarchy's number, with the
    refined levels in patches of 8..16 cells."""
    out = []
    for i in range(_nprob(case)):
        hier = case["hier"] + i
        if case["nx"]:
            nx, ny = case["nx"], case["ny"]
            levels = _levels(case["dim"], nx, ny, case["nlev"], hier, case["max_patch"],
                             case["max_patch0"], case["block"])
            dim = case["dim"]
        else:
            dim = 3
            nx = ny = 8 * int(np.random.default_rng(10_000 + hier).integers(8, 17))
            levels = _levels(3, nx, nx, 3, hier, 16, 32, 8)
        n0 = (nx, ny, nx) if dim == 3 else (nx, ny, 1)
        out.append(configs.Problem(dim=dim, n0=n0, xlo=(0.0, 0.0, 0.0), xup=(1.0, 1.0, 1.0),
                                   levels=list(levels)))
    return out


def _points(prob, ln, ghost=0, axis=None):
    """Coordinates (x, y, z) of every element of a level's cell data (with
    ghost cells) or, with an axis, of its side data of all axes, in the
    framework's order, as FP64 tensors on the GPU; plus the axis selector of
    side data."""
    dim = prob.dim
    boxes = prob.levels[ln].boxes.astype(np.int64)
    lo, hi = boxes[:, :3].copy(), boxes[:, 3:].copy()
    shift = np.full(lo.shape, 0.5)
    if axis is None:
        lo[:, :dim] -= ghost
        hi[:, :dim] += ghost
    else:
        lo, hi = np.repeat(lo, dim, axis=0), np.repeat(hi, dim, axis=0)
        shift = np.full(lo.shape, 0.5)
        for a in range(dim):
            hi[a::dim, a] += 1
            shift[a::dim, a] = 0.0
    n = hi - lo + 1
    count = n.prod(axis=1)
    dev = "cuda"
    tot = int(count.sum())
    cnt = torch.from_numpy(count).to(dev)
    q = torch.arange(tot, device=dev) - torch.repeat_interleave(
        torch.from_numpy(np.cumsum(count) - count).to(dev), cnt, output_size=tot)

    def spread(v):
        return torch.repeat_interleave(torch.from_numpy(np.ascontiguousarray(v)).to(dev), cnt,
                                       output_size=tot)
    nx, ny = spread(n[:, 0]), spread(n[:, 1])
    ijk = (q % nx, (q // nx) % ny, q // (nx * ny))
    dx = prob.dx(ln)
    return [prob.xlo[t] + (ijk[t] + spread(lo[:, t]) + spread(shift[:, t])) * dx[t]
            if t < dim else torch.zeros((), device=dev, dtype=torch.float64) for t in range(3)]


def _bumps(pts, dim, seed, width):
    """Sum of seeded Gaussian bumps (configs.gaussian_bumps)."""
    centers, amps, _ = configs.gaussian_bumps(seed, dim)
    out = torch.zeros_like(pts[0])
    for c, a in zip(centers, amps):
        r2 = sum((pts[t] - float(c[t])) ** 2 for t in range(dim))
        out += float(a) * torch.exp(-r2 / (2.0 * width ** 2))
    return out


def _coefficient(pts, dim, seed):
    """exp(g), g a smooth Gaussian random field (configs.random_field): 1e3
    contrast, correlation length 0.1."""
    fld = configs.random_field(seed, dim)
    out = torch.zeros_like(pts[0])
    for m in range(len(fld.amp)):
        k = fld.k[m]
        out += float(fld.amp[m]) * torch.cos(sum(float(k[t]) * pts[t] for t in range(dim)) +
                                             float(fld.phase[m]))
    return torch.exp(out * float(fld.scale))


def _pinned(n):
    return torch.empty(int(n), dtype=torch.float64, pin_memory=True)


def _context(case, problems, **kw):
    prm = dict(max_cycles=case.get("max_cycles", 100), residual_tol=1e-300,
               relative_residual_tol=1e-10, pre_sweeps=case.get("pre", 2),
               post_sweeps=case.get("post", 2), coarse_tol=1e-300,
               coarse_max_it=case.get("coarse_it", 40), ewing=1)
    return fac.FacContext(problems, params=prm, precision="mixed" if case.get("mixed") else "fp64",
                          coarse_extension=case.get("ext", 0), **kw)


# Robin a u + b du/dn = g on the four sides of a 2-D domain
ROBIN = (np.array([1.0, 2.0, 1.0, 0.5, 0, 0]), np.array([0.5, 1.0, 0.25, 1.0, 0, 0]),
         np.array([0.1, -0.2, 0.05, 0.3, 0, 0]))


def _prepare_fac(case, seed):
    """Context with D and C resident, right-hand sides in pinned host memory
    (solve) or resident too (operators)."""
    problems = _problems(case)
    rhs = []
    for i, p in enumerate(problems):
        ds = 1000 * seed + i
        # _points of cell centres serves f and C
        f, c, d = [], [], []
        for ln in range(p.nlev):
            pts = _points(p, ln)
            f.append(_bumps(pts, p.dim, ds, 0.05 if p.dim == 3 and p.n0[0] > 48 else 0.1))
            if case.get("var_c"):
                c.append((-5.0 * (1.0 + pts[0] + pts[1])).cpu().numpy())
            if case.get("var_d"):
                d.append(_coefficient(_points(p, ln, axis=True), p.dim, ds).cpu().numpy())
        if case.get("var_c"):
            p.c_kind, p.c = 2, c
        if case.get("var_d"):
            p.d_variable, p.d = True, d
        rhs.append(f)
    ctx = _context(case, problems, bc=ROBIN if case.get("robin") else None)
    return problems, rhs, ctx


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        problems, rhs, ctx = _prepare_fac(case, seed)
        ctx.set_krylov(case["krylov"])
        f = _pinned(sum(t.numel() for fl in rhs for t in fl))
        u = _pinned(sum(configs.field_size(p, ln, 1) for p in problems for ln in range(p.nlev)))
        fs, us, of, ou = [], [], 0, 0
        for p, fl in zip(problems, rhs):
            for ln, t in enumerate(fl):
                f[of:of + t.numel()].copy_(t)
                fs.append(f[of:of + t.numel()].numpy())
                of += t.numel()
                n = configs.field_size(p, ln, 1)
                us.append(u[ou:ou + n].numpy())
                ou += n
        return dict(kind=kind, ctx=ctx, f=f, fs=fs, u=u, us=us)
    if kind == "operators":
        problems, rhs, ctx = _prepare_fac(case, seed)
        for ln, t in enumerate(rhs[0]):
            ctx.upload(fac.F, 0, ln + ctx.ext, t.cpu().numpy())
        return dict(kind=kind, ctx=ctx, cycles=case["cycles"])
    if kind == "vectors":
        (p,) = _problems(case)
        ctx = _context(case, [p])
        for ln in range(p.nlev):
            for fid, x in _vectors(p, ln, seed):
                ctx.upload(fid, 0, ln, x.cpu().numpy())
        return dict(kind=kind, ctx=ctx)
    if kind == "regrid":
        problems = _problems(case)
        ctx = _context(case, problems)
        bounds = []
        for i, p in enumerate(problems):
            ln = p.nlev - 1
            ctx.upload(fac.U, i, ln, _front(p, ln, case["hier"] + i, seed).cpu().numpy())
            b = p.levels[ln].boxes
            bounds.append([[int(v) for v in b[:, :3].min(axis=0)] +
                           [int(v) for v in b[:, 3:].max(axis=0)]])
        return dict(kind=kind, ctx=ctx, ln=problems[0].nlev - 1, bounds=bounds)
    # the network: inputs of unit scale on patches of 8..16 cells with their
    # one-cell halo, zero outside, targets and masks on the patch interiors
    x, t, m, ws = _cnn_inputs(case, seed)
    net = fac.CNN(max_batch=case["batch"], seed=1)
    net.set_weights(ws)
    return dict(kind=kind, net=net, x=x, t=t, m=m, n=case["batch"], y=torch.empty_like(x))


def _vectors(p, ln, seed):
    """The two vectors of a level: U (with ghost cells) and F."""
    pts = _points(p, ln, ghost=1)
    yield fac.U, _bumps(pts, p.dim, seed, 0.1) + 0.01 * torch.cos(40.0 * pts[0] + 31.0 * pts[1])
    pts = _points(p, ln)
    yield fac.F, _bumps(pts, p.dim, seed + 1, 0.1) + 0.02 * torch.sin(23.0 * pts[0] - 17.0 * pts[1])


def _front(p, ln, hier, seed):
    """A solution with a steep spherical front around each refined centre."""
    rng = np.random.default_rng(seed)
    centers, _, _ = configs.gaussian_bumps(hier, p.dim)
    h = p.dx(ln)[0]
    pts = _points(p, ln, ghost=1)
    out = torch.zeros_like(pts[0])
    for c in centers:
        r0, w = h * rng.uniform(6.0, 14.0), h * rng.uniform(1.5, 3.0)
        r = torch.sqrt(sum((pts[t] - float(c[t])) ** 2 for t in range(p.dim)))
        out += torch.tanh((r - r0) / w)
    return out


FRONT_THRESHOLD = 0.05
BOXES = 2048


def _cnn_inputs(case, seed):
    n = case["batch"]
    g = torch.Generator(device="cpu").manual_seed(seed)
    x = torch.randn((n, S, S, S), generator=g).cuda()
    t = 0.1 * torch.randn((n, S, S, S), generator=g).cuda()
    m = torch.zeros((n, S, S, S))
    sides = torch.randint(1, 3, (n, 3), generator=g) * 8  # patch sides of 8 or 16 cells
    for i, (a, b, c) in enumerate(sides.tolist()):
        m[i, 1:c + 1, 1:b + 1, 1:a + 1] = 1.0
    m = m.cuda()
    x = x * torch.nn.functional.max_pool3d(m[:, None], 3, 1, 1)[:, 0]  # patch and halo
    ws = []
    for shape in fac.CNN_SHAPES:
        fan = 27 * (shape[1] if len(shape) == 3 else (16 if len(ws) == 3 else 1))
        ws.append((torch.randn(shape, generator=g) * math.sqrt(2.0 / fan)).numpy())
    return x.contiguous(), (t * m).contiguous(), m.contiguous(), ws


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _v_cycle(ctx, ln):
    """FACPreconditioner's recursive cycle over the level operators."""
    if ln == 0:
        ctx.solve_coarsest()
        return
    ctx.smooth(fac.E, fac.R, ln, 2)
    ctx.comp_residual(fac.TR, fac.E, fac.R, ln, True)
    ctx.restrict(fac.TR, fac.R, ln - 1)
    _v_cycle(ctx, ln - 1)
    ctx.prolong_correct(fac.E, fac.E, ln)
    ctx.smooth(fac.E, fac.R, ln, 2)


def _operators(ctx, cycles):
    top = ctx.nlev - 1
    norms = []
    ctx.zero(fac.U)
    for _ in range(cycles):
        ctx.comp_residual(fac.R, fac.U, fac.F, top, False)
        for ln in range(top - 1, -1, -1):
            ctx.restrict_solution(fac.U, ln)
            ctx.comp_residual(fac.R, fac.U, fac.F, ln, False)
            ctx.restrict(fac.R, fac.R, ln)
        norms.append(float(ctx.rms_norm(fac.R)[0]))
        ctx.zero(fac.E)
        _v_cycle(ctx, top)
        ctx.vec_linear_sum(fac.U, 1.0, fac.U, 1.0, fac.E)
    return {"norms": norms, "u": [ctx.download(fac.U, 0, ln) for ln in range(ctx.nlev)]}


def run(state):
    kind = state["kind"]
    if kind == "solve":
        conv, _, _ = state["ctx"].solve_host(state["fs"], state["us"])
        return {"u": state["u"], "converged": conv.astype(np.int32)}
    if kind == "operators":
        return _operators(state["ctx"], state["cycles"])
    if kind == "vectors":
        ctx = state["ctx"]
        return {"dot": ctx.vec_dot(fac.U, fac.F), "l2": ctx.vec_l2_norm(fac.F),
                "max": ctx.vec_max_norm(fac.F), "rms": ctx.rms_norm(fac.U)}
    if kind == "regrid":
        ctx = state["ctx"]
        tags = ctx.tag_gradient(fac.U, state["ln"], FRONT_THRESHOLD)
        boxes = ctx.cluster_tags_all(state["ln"], state["bounds"], (4, 4, 4))
        # every problem's boxes in one table (room for BOXES a problem, -1 after the last)
        table = np.full((BOXES * len(boxes), 6), -1, dtype=np.int32)
        rows = np.concatenate(boxes)
        table[:len(rows)] = rows
        return {"tags": tags, "count": np.array([len(b) for b in boxes]), "boxes": table}
    net, x = state["net"], state["x"]
    if kind == "cnn_forward":
        net.forward(x.data_ptr(), state["n"], state["y"].data_ptr())
        return state["y"]
    loss, grads = net.gradients(x.data_ptr(), state["t"].data_ptr(), state["m"].data_ptr(),
                                state["n"])
    return {"loss": loss, "gradients": grads}


# ---------------------------------------------------------------------------
# the least a pass can do, and its exact value
# ---------------------------------------------------------------------------

def work(case):
    """Inputs read once and outputs written once.  Solves: f and D in and u
    out, and the operations of forming one composite residual (about 20 a
    cell); how many cycles a solve takes is the method's."""
    kind = case["kind"]
    if kind.startswith("cnn"):
        cells = case["batch"] * S ** 3
        fwd = 2 * 27 * (16 + 256 + 256 + 16)
        if kind == "cnn_forward":
            return {"bytes": 8 * cells, "flops": fwd * cells}
        return {"bytes": 12 * cells, "flops": (2 * fwd + 2 * 27 * (256 + 256 + 16)) * cells}
    problems = _problems(case)
    if kind == "regrid":
        n1 = sum(configs.field_size(p, p.nlev - 1, 1) for p in problems)
        n0 = sum(configs.field_size(p, p.nlev - 1, 0) for p in problems)
        return {"bytes": 8 * n1 + n0, "flops": 30 * n0}
    n0 = sum(p.num_cells() for p in problems)
    if kind == "vectors":
        return {"bytes": 24 * n0, "flops": 12 * n0}
    n1 = sum(configs.field_size(p, ln, 1) for p in problems for ln in range(p.nlev))
    ns = sum(configs.side_size(p, ln) for p in problems for ln in range(p.nlev))
    by = 8 * (n0 + n1 + (ns if case.get("var_d") else 0) + (n0 if case.get("var_c") else 0))
    return {"bytes": by, "flops": 20 * n0}


def _covered(p, ln):
    """Whether each cell of a level lies under the next finer level, by
    rasterising that level (coarsened) over the domain."""
    if ln == p.nlev - 1:
        return None
    _, hi = p.domain(ln)
    mask = torch.zeros((hi[2] + 1, hi[1] + 1, hi[0] + 1), dtype=torch.bool, device="cuda")
    r = p.levels[ln + 1].ratio
    for b in p.levels[ln + 1].boxes.tolist():
        mask[b[2] // r[2]:b[5] // r[2] + 1, b[1] // r[1]:b[4] // r[1] + 1,
             b[0] // r[0]:b[3] // r[0] + 1] = True
    return torch.cat([mask[b[2]:b[5] + 1, b[1]:b[4] + 1, b[0]:b[3] + 1].reshape(-1)
                      for b in p.levels[ln].boxes.tolist()])


def _interior(p, ln, x):
    """Interior cells of a ghost-1 level array."""
    out, off = [], 0
    for b in p.levels[ln].boxes.tolist():
        e = [b[3 + t] - b[t] + (3 if t < p.dim else 1) for t in range(3)]
        n = e[0] * e[1] * e[2]
        v = x[off:off + n].reshape(e[2], e[1], e[0])[:, 1:-1, 1:-1]
        out.append((v[1:-1] if p.dim == 3 else v).reshape(-1))
        off += n
    return torch.cat(out)


def _exact_vectors(case, seed):
    (p,) = _problems(case)
    sxy = syy = sxx = sw = 0.0
    big = 0.0
    for ln in range(p.nlev):
        (_, u), (_, f) = _vectors(p, ln, seed)
        u = _interior(p, ln, u)
        w = torch.full_like(f, float(np.prod(p.dx(ln)[:p.dim])))
        cov = _covered(p, ln)
        if cov is not None:
            w[cov] = 0.0
        sxy += float((w * u * f).sum())
        syy += float((w * f * f).sum())
        sxx += float((w * u * u).sum())
        sw += float(w.sum())
        big = max(big, float((f.abs() * (w > 0)).max()))
    return {"dot": np.array([sxy]), "l2": np.array([math.sqrt(syy)]), "max": np.array([big]),
            "rms": np.array([math.sqrt(sxx / sw)])}


def _conv_weight(w):
    """(27, in, out) weights, tap = (dz+1)*9 + (dy+1)*3 + (dx+1), as a conv3d
    weight (out, in, 3, 3, 3)."""
    return w.reshape(3, 3, 3, w.shape[1], w.shape[2]).permute(4, 3, 0, 1, 2).contiguous()


def _exact_cnn(case, seed):
    conv = torch.nn.functional.conv3d
    x, t, m, ws = _cnn_inputs(case, seed)
    shapes = [(27, 1, 16), (27, 16, 16), (27, 16, 16), (27, 16, 1)]
    ws = [torch.from_numpy(w).cuda().double().reshape(s).requires_grad_()
          for w, s in zip(ws, shapes)]
    train = case["kind"] == "cnn_gradients"
    total = m.double().sum()
    ys, loss = [], 0.0
    step = 16
    with torch.set_grad_enabled(train):
        for b in range(0, case["batch"], step):
            h = x[b:b + step, None].double()
            for i, w in enumerate(ws):
                h = conv(h, _conv_weight(w), padding=1)
                h = torch.relu(h) if i < 3 else h
            if train:
                part = (m[b:b + step].double() * (h[:, 0] - t[b:b + step].double()) ** 2).sum() / total
                part.backward()
                loss += float(part.detach())
            else:
                ys.append(h[:, 0])
    if not train:
        return torch.cat(ys)
    return {"loss": loss, "gradients": [w.grad.reshape(s) for w, s in zip(ws, fac.CNN_SHAPES)]}


def exact(case, seed):
    """Vectors and the network in 64 bits.  A composite solve has no such
    value here: a direct solution of its system takes longer than the limit,
    and the level operators' intermediate fields have no closed form."""
    kind = case["kind"]
    if kind == "vectors":
        return _exact_vectors(case, seed)
    if kind.startswith("cnn"):
        return _exact_cnn(case, seed)
    return None
