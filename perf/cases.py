"""Performance cases of the PPM-DE hydro path: the calls a user of this library makes.

A pass is what Enzo's cycle does around the hydro call: grid::SolvePPM_DE on device fields
with the time step of the next cycle folded into its last sweep, then the ghost-zone fill
(single grids and levels of patches), or the whole host-memory call with subgrid-flux
capture (the drop-in call of a rank whose fields live in host memory).  One context per
build serves every grid, as one context per rank does in Enzo.  The cases span rank 1 to 3,
both builds (exact and tolerance), 100 cells to 512^3, gravity, slope corrections, colour
fields, the HLLC solver, dual energy on and off, and levels of many patches.

`exact` restates the same step in plain torch (FP64), without this repository's code.
"""
import math
import sys

import numpy as np
import torch

sys.path.insert(0, "enzo-dev_b200")

from ppm_b200 import capi  # noqa: E402
from ppm_b200 import harness as H  # noqa: E402

NAMES = ("d", "te", "v1", "v2", "v3", "ge")
DEV = "cuda"
F64 = torch.float64
HLLC = 4


def _case(kind, nx, ny=1, nz=1, **kw):
    """kind: tube (rank 1), plane (rank 2), box (rank 3), level (patches), host (rank 3)."""
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "build": "fast", "dual": True,
         "gravity": False, "mach": 3.0, "bc": "periodic", "riemann": 5, "colours": 0,
         "flatten": 0, "steepen": 0, "patches": 0}
    c.update(kw)
    return c


def listed():
    def named(name, *a, **kw):
        return dict(_case(*a, **kw), name=name)

    return [
        # the answer-test shock tube (run/Hydro/Hydro-1D), the smallest call: latency alone
        named("tube_100", "tube", 100, build="exact", bc="outflow"),
        # a two-dimensional test problem, without the dual-energy formalism
        named("plane_256x192", "plane", 256, 192, build="exact", dual=False, mach=1.0),
        # one small AMR patch solved by itself (the grid loop of EvolveLevel.C)
        named("patch_16", "box", 16, 16, 16),
        # a ragged self-gravitating patch with the HLLC solver
        named("patch_37x24x53_hllc", "box", 37, 24, 53, build="exact", gravity=True,
              riemann=HLLC, bc="outflow"),
        # an ordinary uniform grid with the build a user gets by default
        named("box_128_exact", "box", 128, 128, 128, build="exact"),
        # the benchmark's headline grid
        named("box_256", "box", 256, 256, 256),
        # a ragged grid of odd sides with gravity
        named("box_189x131x157", "box", 189, 131, 157, gravity=True, bc="outflow"),
        # the largest grid of the benchmark (Mach-10 turbulence)
        named("box_512_mach10", "box", 512, 512, 512, mach=10.0),
        # a sparse level: a few small patches in one batch
        named("level_24", "level", 16, 32, patches=24, build="exact"),
        # an AMR level of mixed patches, half Sedov blasts, half turbulence
        named("level_200", "level", 16, 112, patches=200),
        # a chemistry run: nine species, flattening and steepening
        named("box_96_species", "box", 96, 96, 96, colours=9, flatten=3, steepen=1, mach=2.0),
        # the drop-in call on pageable host fields, fluxes of one subgrid captured
        named("host_64_subgrid", "host", 64, 64, 64, build="exact"),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    build = rng.choice(["exact", "fast"])
    kind = rng.choice(["tube", "plane", "box", "box", "box", "level", "host"])
    if kind == "tube":
        return _case("tube", size(64, 1000), build=build, bc="outflow")
    if kind == "plane":
        return _case("plane", size(32, 900), size(32, 900), build=build,
                     dual=rng.random() < 0.5, mach=rng.choice([0.5, 1.0]),
                     gravity=rng.random() < 0.3)
    if kind == "level":
        n = size(8, 200)
        return _case("level", 16, size(24, 96), patches=n, build=build)
    if kind == "host":
        return _case("host", size(16, 96), size(16, 96), size(16, 96), build=build)
    extra = rng.choice(["none", "none", "gravity", "hllc", "species", "corrections"])
    hi = 200 if extra != "none" else 280
    c = _case("box", size(12, hi), size(12, hi), size(12, hi), build=build,
              mach=rng.choice([2.0, 3.0]), bc=rng.choice(["periodic", "outflow"]))
    if extra == "gravity":
        c["gravity"] = True
    elif extra == "hllc":
        c["riemann"] = HLLC
    elif extra == "species":
        c.update(colours=rng.choice([1, 4, 9]), flatten=rng.choice([0, 3]), mach=2.0)
    elif extra == "corrections":
        c.update(flatten=3, steepen=1, mach=2.0)
    return c


# ------------------------------------------------------------------ inputs
def _rank(case):
    return {"tube": 1, "plane": 2}.get(case["kind"], 3)


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _spectrum(shape, slope, gen, ncomp):
    """ncomp Gaussian fields of one shape (z, y, x), P(k) ~ k^slope, solenoidal if several."""
    dims = [i for i in range(3) if shape[i] > 1]
    ks = []
    for i in range(3):
        n = shape[i]
        k = torch.fft.fftfreq(n, device=DEV, dtype=F64) * n if n > 1 else torch.zeros(
            1, device=DEV, dtype=F64)
        if dims and i == dims[-1]:
            k = torch.fft.rfftfreq(n, device=DEV, dtype=F64) * n
        ks.append(k.reshape([-1 if j == i else 1 for j in range(3)]))
    k2 = ks[0] ** 2 + ks[1] ** 2 + ks[2] ** 2
    amp = torch.where(k2 > 0, torch.clamp(k2, min=1.0) ** (slope / 4.0), torch.zeros_like(k2))
    noise = [torch.complex(torch.randn(k2.shape, generator=gen, device=DEV, dtype=F64),
                           torch.randn(k2.shape, generator=gen, device=DEV, dtype=F64)) * amp
             for _ in range(ncomp)]
    if ncomp == 3:
        div = noise[0] * ks[2] + noise[1] * ks[1] + noise[2] * ks[0]
        div = div / torch.clamp(k2, min=1.0)
        for i in range(3):
            noise[i] = noise[i] - ks[2 - i] * div
    size = [shape[i] for i in dims]
    return [torch.fft.irfftn(x, s=size, dim=dims) for x in noise]


def _turbulence(case, shape, seed):
    """Active cells: lognormal density, solenoidal velocity at rms Mach, uniform pressure."""
    gen = _gen(seed)
    g = _spectrum(shape, -2.0, gen, 1)[0]
    rho = torch.exp(0.5 * (g - g.mean()) / g.std())
    rho = rho / rho.mean()
    vel = _spectrum(shape, -4.0, gen, 3)
    rank = _rank(case)
    for i in range(rank, 3):
        vel[i] = torch.zeros_like(vel[i])
    scale = case["mach"] / torch.sqrt(sum((v * v).mean() for v in vel))
    vel = [v * scale for v in vel]
    eint = 1.0 / (5.0 / 3.0 * (5.0 / 3.0 - 1.0)) / rho
    out = {"d": rho, "te": eint + 0.5 * (vel[0] ** 2 + vel[1] ** 2 + vel[2] ** 2)}
    for i in range(rank):
        out["v%d" % (i + 1)] = vel[i]
    if case["dual"]:
        out["ge"] = eint
    return out


def _tube(case, seed):
    """Two constant states (Sod-like, jumps drawn from the seed)."""
    gen = _gen(seed)
    r = torch.rand(4, generator=gen, device=DEV, dtype=F64).tolist()
    n = case["nx"]
    left = torch.arange(n, device=DEV) < int(n * (0.35 + 0.3 * r[0]))
    left = left.reshape(1, 1, n)
    val = lambda a, b: torch.where(left, a, b).to(F64)  # noqa: E731
    rho = val(torch.tensor(1.0, device=DEV), torch.tensor(0.1 + 0.2 * r[1], device=DEV))
    p = val(torch.tensor(1.0, device=DEV), torch.tensor(0.05 + 0.1 * r[2], device=DEV))
    u = val(torch.tensor(0.3 * r[3], device=DEV), torch.tensor(0.0, device=DEV))
    eint = p / ((5.0 / 3.0 - 1.0) * rho)
    out = {"d": rho, "te": eint + 0.5 * u * u, "v1": u}
    if case["dual"]:
        out["ge"] = eint
    return out


def _wrap(n, bc):
    i = torch.arange(n + 6, device=DEV) - 3
    return i % n if bc == "periodic" else i.clamp(0, n - 1)


def _pad(a, rank, bc):
    """Three ghost zones on each side of the active axes."""
    for ax in range(3):
        if 2 - ax < rank:
            a = a.index_select(ax, _wrap(a.shape[ax], bc))
    return a.contiguous()


def _box_inputs(case, seed):
    rank = _rank(case)
    shape = (case["nz"], case["ny"], case["nx"])
    act = _tube(case, seed) if rank == 1 else _turbulence(case, shape, seed)
    if case["colours"]:
        g = _spectrum(shape, -3.0, _gen(seed + 7), 1)[0]
        g = g / g.std()
        for n in range(case["colours"]):
            frac = 0.5 ** (n + 1) * (1.0 + 0.3 * torch.tanh(g * (1.0 if n % 2 else -1.0)))
            act["col%d" % n] = act["d"] * frac
    f = {k: _pad(v, rank, case["bc"]) for k, v in act.items()}
    acc = None
    if case["gravity"]:
        acc = []
        for d in range(rank):
            n = shape[2 - d]
            ph = float(torch.rand(1, generator=_gen(seed + 11 + d), device=DEV, dtype=F64))
            x = (torch.arange(n + 6, device=DEV, dtype=F64) - 2.5) / n + ph
            a = 0.5 * torch.sin(2.0 * math.pi * x)
            a = a.reshape([-1 if ax == 2 - d else 1 for ax in range(3)])
            acc.append(a.expand(tuple(s + 6 if 2 - ax < rank else 1
                                      for ax, s in enumerate(shape))).contiguous())
    return f, acc


def _level_edges(case, seed):
    """Patch edges, log-uniform per axis in [nx, ny]; the first 8 the same for every seed."""
    rng = np.random.default_rng(1000 + case["patches"] * 131 + case["ny"])
    lo, hi = case["nx"], case["ny"]
    e = np.floor(np.exp(rng.uniform(math.log(lo), math.log(hi + 1), size=(case["patches"], 3))))
    return np.clip(e, lo, hi).astype(int)


def _level_inputs(case, seed):
    """Flat buffers (one per field), every patch a view: half blasts, half turbulence crops."""
    edges = _level_edges(case, seed)
    shapes = [tuple(int(e) + 6 for e in ed[::-1]) for ed in edges]
    offs, at = [], 0
    for s in shapes:
        offs.append(at)
        at += (s[0] * s[1] * s[2] + 31) // 32 * 32
    flat = {k: torch.zeros(at, device=DEV, dtype=F64) for k in NAMES}
    views = [{k: flat[k][o:o + s[0] * s[1] * s[2]].view(s) for k in NAMES}
             for o, s in zip(offs, shapes)]
    src_n = 96
    src = _turbulence(case, (src_n,) * 3, seed)
    rng = np.random.default_rng(seed)
    gm1 = 5.0 / 3.0 - 1.0
    for n, (v, s) in enumerate(zip(views, shapes)):
        if n % 2:
            idx = [(torch.arange(s[i], device=DEV) + int(rng.integers(src_n))) % src_n
                   for i in range(3)]
            for k in NAMES:
                a = src[k]
                for ax in range(3):
                    a = a.index_select(ax, idx[ax])
                v[k].copy_(a)
        else:
            v["d"].fill_(1.0 + 0.5 * float(rng.random()))
            e0 = 1e-2 / gm1
            v["te"].fill_(e0)
            v["ge"].fill_(e0)
            c = [x // 2 for x in s]
            blast = 100.0 * (1.0 + float(rng.random()))
            sl = tuple(slice(x - 1, x + 1) for x in c)
            v["te"][sl] += blast
            v["ge"][sl] += blast
    return edges, flat, views


def _uniform_grid(edges, width):
    return H.Grid.uniform(tuple(int(e) for e in edges), width=width)


def _hp(case):
    return H.HydroParams(gamma=5.0 / 3.0, cfl=0.4, dual=case["dual"], gravity=case["gravity"],
                         riemann=case["riemann"], flatten=case["flatten"],
                         steepen=case["steepen"])


_CTX = {}


def _context(build):
    if build not in _CTX:
        _CTX[build] = capi.Context(0, variant=build)
    return _CTX[build]


HOST_DT_SHARE = 0.01  # of the Courant step: the host call is repeated without a ghost fill


def prepare(case, seed):
    hp, ctx = _hp(case), _context(case["build"])
    s = {"case": case, "hp": hp, "ctx": ctx, "cycle": 0}
    dt = torch.zeros(1, device=DEV, dtype=F64)
    if case["kind"] == "level":
        edges, flat, views = _level_inputs(case, seed)
        s.update(grids=[_uniform_grid(e, tuple(float(x) / 128.0 for x in e)) for e in edges],
                 flat=flat, fields=views, dt=dt)
        torch.cuda.synchronize()
        ctx.compute_timestep_level(s["grids"], hp, views, dt_device=dt, want_host=False)
        return s
    f, acc = _box_inputs(case, seed)
    edges = (case["nx"], case["ny"], case["nz"])[:_rank(case)]
    grid = _uniform_grid(edges, tuple(float(e) / edges[0] for e in edges))
    s.update(grid=grid, fields=f, acc=acc, dt=dt)
    torch.cuda.synchronize()
    value = ctx.compute_timestep(grid, hp, f, memory=capi.MEM_DEVICE, dt_device=dt)
    if case["kind"] == "host":
        s["fields"] = {k: v.cpu().numpy() for k, v in f.items()}
        s["dt_host"] = HOST_DT_SHARE * value
        s["box"] = _subgrid_box(case)
    return s


def _subgrid_box(case):
    """One subgrid over the middle half of the grid; its flux arrays, zeroed."""
    n = (case["nx"], case["ny"], case["nz"])
    lo = [3 + e // 4 for e in n]
    hi = [3 + e // 4 + e // 2 - 1 for e in n]
    box = {k: [[0] * 3 for _ in range(3)] for k in
           ("left_start", "left_end", "right_start", "right_end")}
    box["left"] = [[None] * 3 for _ in range(6)]
    box["right"] = [[None] * 3 for _ in range(6)]
    for dim in range(3):
        for i in range(3):
            box["left_start"][dim][i] = lo[i]
            box["left_end"][dim][i] = lo[i] if i == dim else hi[i]
            box["right_start"][dim][i] = hi[i] if i == dim else lo[i]
            box["right_end"][dim][i] = hi[i]
        count = 1
        for i in range(3):
            if i != dim:
                count *= hi[i] - lo[i] + 1
        for side in ("left", "right"):
            for slot in range(6):
                box[side][slot][dim] = np.zeros(count)
    return box


def run(s):
    ctx, hp, case = s["ctx"], s["hp"], s["case"]
    cycle = s["cycle"]
    s["cycle"] = cycle + 1
    if case["kind"] == "host":
        ctx.set_cfl(None)
        ctx.solve_ppm_de(s["grid"], hp, s["dt_host"], 0, s["fields"], memory=capi.MEM_HOST,
                         subgrids=[s["box"]])
        out = dict(s["fields"])
        out["left"] = [list(r) for r in s["box"]["left"]]
        out["right"] = [list(r) for r in s["box"]["right"]]
        return out
    ctx.set_cfl(s["dt"], courant=hp.cfl)
    if case["kind"] == "level":
        ctx.solve_level(s["grids"], hp, 0.0, cycle, s["fields"], dt_device=s["dt"])
        ctx.set_boundary_level(s["grids"], s["fields"], True, ("outflow",) * 3)
        return dict(s["flat"], dt=s["dt"])
    ctx.solve_ppm_de(s["grid"], hp, 0.0, cycle, s["fields"], memory=capi.MEM_DEVICE,
                     accel=s["acc"], want_stats=False, dt_device=s["dt"])
    ctx.set_boundary(s["grid"], s["fields"], hp.dual, (case["bc"],) * 3)
    return dict(s["fields"], dt=s["dt"])


# ------------------------------------------------------------------ work and tolerance
def _cells(case):
    if case["kind"] == "level":
        return int(sum(int(np.prod(e + 6)) for e in _level_edges(case, 0)))
    n = 1
    for e in (case["nx"], case["ny"], case["nz"])[:_rank(case)]:
        n *= e + 6
    return n


def work(case):
    """Every field read once and written once; the point-wise arithmetic of the sweeps
    (reconstruction about 350, the Riemann problem about 250, the update about 60)."""
    rank, cells = _rank(case), _cells(case)
    nf = 2 + rank + (1 if case["dual"] else 0) + case["colours"]
    n = 2 * nf + (rank if case["gravity"] else 0)
    flops = rank * (660 + 80 * case["colours"]) * cells
    return {"bytes": 8.0 * n * cells, "flops": float(flops)}


def tolerance(case):
    """The exact build's arithmetic is fixed to the last bit.  The tolerance build differs
    from it by round-off (fused multiply-adds, another order of the same products): after
    two and three passes 1.3e-15 and 1.8e-15 of a field's norm, 2.2e-14 and 2.4e-14 of a
    single value at most (the thermal energy of cold supersonic gas), over the listed and
    the drawn cases; four times that."""
    if case["build"] == "exact":
        return "exact"
    return {"rel": 8e-15, "max": 1e-13}


# ------------------------------------------------------------------ 64-bit restatement
GAMMA, TINY, SMALL_RHO, PMIN = 5.0 / 3.0, 1e-20, 1e-30, 1e-20
ETA1, ETA2, CFL = 0.001, 0.1, 0.4
CHUNK = 1 << 23


class _Fallback(Exception):
    """A cell needs the per-cell HLL fallback, which this restatement leaves out."""


def _mx(a, b):
    return torch.maximum(a, b) if torch.is_tensor(b) else a.clamp(min=b)


def _mn(a, b):
    return torch.minimum(a, b) if torch.is_tensor(b) else a.clamp(max=b)


def _slopes(q):
    """Limited slopes of cells 1 .. n-2 (uniform spacing)."""
    qp, qm = q[:, 2:] - q[:, 1:-1], q[:, 1:-1] - q[:, :-2]
    qc = 0.5 * qp + 0.5 * qm
    qv = 2.0 * qp * qm / (qm + qp)
    t = _mn(_mn(_mn(qc.abs(), qv.abs()), 2.0 * qm.abs()), 2.0 * qp.abs())
    return torch.where(qp * qm > 0.0, t * torch.sign(qc), torch.zeros_like(t))


def _parabola(q, st=None, fl=None):
    """(ql, qr, q6, dq) of cells 2 .. n-3."""
    n = q.shape[1]
    dq = _slopes(q)  # entry c - 1
    a, b = q[:, 1:n - 2], q[:, 2:n - 1]
    edge = 0.5 * a + 0.5 * b + dq[:, :n - 3] / 6.0 - dq[:, 1:n - 2] / 6.0  # cells 2 .. n-2
    ql, qr = edge[:, :-1], edge[:, 1:]
    qm, q0, qp = q[:, 1:n - 3], q[:, 2:n - 2], q[:, 3:n - 1]
    if st is not None:
        ql = (1.0 - st) * ql + st * (qm + 0.5 * dq[:, 0:n - 4])
        qr = (1.0 - st) * qr + st * (qp - 0.5 * dq[:, 2:n - 2])
    t1, t2 = (qr - q0) * (q0 - ql), qr - ql
    t3 = 6.0 * (q0 - 0.5 * (qr + ql))
    ql, qr = torch.where(t1 <= 0.0, q0, ql), torch.where(t1 <= 0.0, q0, qr)
    t22, t23 = t2 * t2, t2 * t3
    ql = torch.where(t22 < t23, 3.0 * q0 - 2.0 * qr, ql)
    qr = torch.where(t22 < -t23, 3.0 * q0 - 2.0 * ql, qr)
    if fl is not None:
        ql, qr = q0 * fl + ql * (1.0 - fl), q0 * fl + qr * (1.0 - fl)
    ql = _mn(_mx(q0, qm), _mx(_mn(q0, qm), ql))
    qr = _mn(_mx(q0, qp), _mx(_mn(q0, qp), qr))
    return ql, qr, 6.0 * (q0 - 0.5 * (ql + qr)), qr - ql


FT = 4.0 / 3.0


def _from_left(p, x):
    return p[1] - x * (p[3] - (1.0 - FT * x) * p[2])


def _from_right(p, x):
    return p[0] - x * (p[3] + (1.0 + FT * x) * p[2])


def _from_right_char(p, x):
    return p[0] + x * (p[3] + (1.0 - FT * x) * p[2])


def _flattening(d, e, u, p):
    """PPMFlatteningParameter 3, cells 2 .. n-3 (index 0 = cell 2)."""
    n = d.shape[1]
    k = lambda a, o: a[:, 2 + o:n - 2 + o]  # noqa: E731
    qb = (k(p, 1) - k(p, -1)).abs() / _mn(k(p, 1), k(p, -1))
    w = ((qb > 0.33) & (k(u, -1) > k(u, 1))).to(F64)
    dp1, dp2 = k(p, 1) - k(p, -1), k(p, 2) - k(p, -2)
    de1, de2 = k(e, 1) - k(e, -1), k(e, 2) - k(e, -2)
    zero = torch.zeros_like(dp1)
    om_t = _mx(torch.where(dp2 != 0, dp1 / dp2, zero), torch.where(de2 != 0, de1 / de2, zero))
    neg = torch.signbit(dp1)
    pick = lambda a, b: torch.where(neg, a, b)  # noqa: E731
    d_post, u_post = pick(k(d, -2), k(d, 2)), pick(k(u, -2), k(u, 2))
    d_up, u_up, p_up = pick(k(d, 2), k(d, -2)), pick(k(u, 2), k(u, -2)), pick(k(p, 2), k(p, -2))
    s = -torch.sign(dp1)
    sig_t = w * dp2.abs() / _mn(k(p, 2), k(p, -2))
    sigma = _mx((sig_t - 0.5) / (sig_t + 1.0), 0.0)
    omega = _mx(10.0 * (om_t - 0.75), 0.0)
    z = torch.sqrt((_mx(k(p, 2), k(p, -2)) + 0.5 * (k(p, 2) + k(p, -2)) * (GAMMA - 1.0)) /
                   _mx(1.0 / k(d, 2), 1.0 / k(d, -2)))
    ze = s * z / d_post + u_post + TINY
    kap_t = ((ze - u_up + s * torch.sqrt(GAMMA * p_up / d_up)) / ze).abs()
    kappa = _mx((kap_t - 2.0) / (kap_t + 0.01), 0.0)
    f = _mn(_mn(kappa, w * omega), w * sigma)
    fm = torch.cat([f[:, :1], f[:, :-1]], 1)
    fp = torch.cat([f[:, 1:], f[:, -1:]], 1)
    return torch.where(dp1 < 0.0, _mx(f, fp), _mx(f, fm))


def _steepening(d, p, dx):
    n = d.shape[1]
    k = lambda a, o: a[:, 2 + o:n - 2 + o]  # noqa: E731
    d2 = lambda a, b, c: ((c - b) / (2 * dx) - (b - a) / (2 * dx)) / (3 * dx)  # noqa: E731
    d2m, d2p = d2(k(d, -2), k(d, -1), k(d, 0)), d2(k(d, 0), k(d, 1), k(d, 2))
    qc = (k(d, 1) - k(d, -1)).abs() - 0.01 * _mn(k(d, 1).abs(), k(d, -1).abs())
    s1 = (d2m - d2p) * (2 * dx ** 3) / (2 * dx * (k(d, 1) - k(d, -1) + TINY))
    s1 = torch.where((d2p * d2m > 0.0) | (qc <= 0.0), torch.zeros_like(s1), s1)
    s2 = (20.0 * (s1 - 0.05)).clamp(0.0, 1.0)
    qa = (k(d, 1) - k(d, -1)).abs() / _mn(k(d, 1), k(d, -1))
    qb = (k(p, 1) - k(p, -1)).abs() / _mn(k(p, 1), k(p, -1))
    return torch.where(GAMMA * 0.1 * qa >= qb, s2, torch.zeros_like(s2))


def _side(par, pr, left, dual, dt, g):
    """Corrected (d, p, u) of one side of every face, and the density before the override."""
    f = _from_left if left else _from_right
    fa = _from_left if left else _from_right_char
    cs, cm, c0, cp = pr
    da, d0 = fa(par[0], cs), f(par[0], c0)
    pa, p0, pm, pp = fa(par[1], cs), f(par[1], c0), f(par[1], cm), f(par[1], cp)
    ua, um, up = fa(par[2], cs), f(par[2], cm), f(par[2], cp)
    c = torch.sqrt(_mx(GAMMA * pa * da, 0.0))
    bp = (ua - up) + (pa - pp) / c
    bm = (ua - um) - (pa - pm) / c
    b0 = (pa - p0) / (c * c) + 1.0 / da - 1.0 / d0
    if g is not None:
        bp, bm = bp - 0.25 * dt * g, bm - 0.25 * dt * g
    bp, bm = -bp * 0.5 / c, bm * 0.5 / c
    off = (lambda x: x <= 0.0) if left else (lambda x: x >= 0.0)
    zero = torch.zeros_like(bp)
    bp, bm, b0 = (torch.where(off(x), zero, b) for x, b in ((cp, bp), (cm, bm), (c0, b0)))
    p, u, d = pa + (bp + bm) * (c * c), ua + (bp - bm) * c, 1.0 / (1.0 / da - (b0 + bp + bm))
    dc = d
    ov = torch.zeros_like(d, dtype=torch.bool)
    if dual:
        m = _mx(_mx(cm.abs(), c0.abs()), cp.abs())
        ov = (GAMMA * pa / da < ETA2 * ua * ua) | (m < 1e-3) | (d / da > 5.0)
        p, u, d = torch.where(ov, pa, p), torch.where(ov, ua, u), torch.where(ov, da, d)
    return {"d": _mx(d, TINY), "p": _mx(p, TINY), "u": u, "da": da, "d0": d0, "dc": dc, "ov": ov}


def _two_shock(L, R):
    qa, gp1 = (GAMMA + 1.0) / (2.0 * GAMMA), GAMMA + 1.0
    cl, cr = torch.sqrt(GAMMA * L["p"] * L["d"]), torch.sqrt(GAMMA * R["p"] * R["d"])
    ps = _mx((cr * L["p"] + cl * R["p"] + cr * cl * (L["u"] - R["u"])) / (cr + cl), PMIN)
    on = torch.ones_like(ps, dtype=torch.bool)
    keep = [torch.zeros_like(ps) for _ in range(4)]
    for _ in range(7):
        zl = cl * torch.sqrt(1.0 + qa * (ps / L["p"] - 1.0))
        zr = cr * torch.sqrt(1.0 + qa * (ps / R["p"] - 1.0))
        ul, ur = L["u"] - (ps - L["p"]) / zl, R["u"] + (ps - R["p"]) / zr
        al, ar = 4.0 * zl * zl / L["d"], 4.0 * zr * zr / R["d"]
        dl = -zl * al / (al - gp1 * (ps - L["p"]))
        dr = zr * ar / (ar - gp1 * (ps - R["p"]))
        new = _mx(ps + (ur - ul) * dr * dl / (dr - dl), PMIN)
        keep = [torch.where(on, a, b) for a, b in zip((ul, ur, dl, dr), keep)]
        new = torch.where(on, new, ps)
        on = on & ~(((new - ps) / new).abs() < 1e-14)
        ps = new
        if not bool(on.any()):
            break
    ul, ur, dl, dr = keep
    return ps, ul + (ur - ul) * dr / (dr - dl)


def _two_shock_flux(L, R, dual, qc):
    """Fluxes times dt/dx, the Godunov velocity and density."""
    pbar, ubar = _two_shock(L, R)
    qa, gm1 = (GAMMA + 1.0) / (2.0 * GAMMA), GAMMA - 1.0
    left = torch.signbit(-ubar)
    u0, p0, d0 = (torch.where(left, L[k], R[k]) for k in ("u", "p", "d"))
    sn = torch.where(left, -1.0, 1.0)
    c0 = torch.sqrt(_mx(GAMMA * p0 / d0, TINY))
    z0 = c0 * d0 * torch.sqrt(_mx(1.0 + qa * (pbar / p0 - 1.0), TINY))
    dbar = 1.0 / (1.0 / d0 - (pbar - p0) / _mx(z0 * z0, TINY))
    cbar = torch.sqrt(_mx(GAMMA * pbar / dbar, TINY))
    rare = pbar < p0
    l0 = torch.where(rare, u0 * sn + c0, u0 * sn + z0 / d0)
    lb = torch.where(rare, sn * ubar + cbar, l0)
    fr = (-lb / _mx(l0 - lb, TINY)).clamp(0.0, 1.0)
    mix = lambda a, b: torch.where(l0 < 0.0, a, torch.where(  # noqa: E731
        lb >= 0.0, b, a * fr + b * (1.0 - fr)))
    pb, db, ub = mix(p0, pbar), mix(d0, dbar), mix(u0, ubar)
    vb, wb, gb = (torch.where(ub > 0.0, L[k], R[k]) for k in ("v", "w", "ge"))
    eb = pb / (gm1 * db) + 0.5 * (ub * ub + vb * vb + wb * wb)
    m = qc * ub * db
    return {"d": m, "e": m * eb + qc * pb * ub, "u": m * ub + qc * pb, "v": m * vb, "w": m * wb,
            "ge": m * gb, "ub": ub, "db": db}


def _hllc_flux(L, R, dual, qc):
    gm1 = GAMMA - 1.0
    sl_, sr_ = torch.sqrt(L["d"]), torch.sqrt(R["d"])
    inv = 1.0 / (sl_ + sr_)
    roe = [(sl_ * L[k] + sr_ * R[k]) * inv for k in ("u", "v", "w")]
    v2 = roe[0] ** 2 + roe[1] ** 2 + roe[2] ** 2
    e = [s["p"] / gm1 + 0.5 * s["d"] * (s["u"] ** 2 + s["v"] ** 2 + s["w"] ** 2) for s in (L, R)]
    h = ((e[0] + L["p"]) / sl_ + (e[1] + R["p"]) / sr_) * inv
    cs = torch.sqrt(gm1 * _mx(h - 0.5 * v2, TINY))
    csl = _mn(L["u"] - torch.sqrt(GAMMA * L["p"] / L["d"]), roe[0] - cs)
    csr = _mx(R["u"] + torch.sqrt(GAMMA * R["p"] / R["d"]), roe[0] + cs)
    bm, bp = _mn(csl, 0.0), _mx(csr, 0.0)
    tl = L["p"] - (csl - L["u"]) * L["d"] * L["u"]
    tr = R["p"] - (csr - R["u"]) * R["d"] * R["u"]
    dl, dr = L["d"] * (csl - L["u"]), -(R["d"] * (csr - R["u"]))
    q = 1.0 / (dl + dr)
    cw, cp = (tr - tl) * q, _mx((dl * tr + dr * tl) * q, 0.0)
    right = cw >= 0.0
    zero = torch.zeros_like(cw)
    sl = torch.where(right, cw / (cw - bm), zero)
    sr = torch.where(right, zero, -cw / (bp - cw))
    sm = torch.where(right, -bm / (cw - bm), bp / (bp - cw))
    bl, br = L["u"] - bm, R["u"] - bp
    f = {"d": sl * L["d"] * bl + sr * R["d"] * br,
         "u": sl * (L["d"] * L["u"] * bl + L["p"]) + sr * (R["d"] * R["u"] * br + R["p"]) +
         sm * cp,
         "e": sl * (e[0] * bl + L["p"] * L["u"]) + sr * (e[1] * br + R["p"] * R["u"]) +
         sm * cp * cw}
    for k in ("v", "w", "ge"):
        f[k] = sl * L["d"] * L[k] * bl + sr * R["d"] * R[k] * br
    f = {k: qc * x for k, x in f.items()}
    f["div"] = sl * bl + sr * br
    f["w4"] = (sl, bl, sr, br)
    return f


def _sweep_pencils(F, p, acc, cols, dx, dt, case):
    """One sweep of pencils: F = d, e, u, v, w, ge as (pencils, n); colours changed too."""
    dual, n = case["dual"], p.shape[1]
    hllc = case["riemann"] == HLLC
    qc = dt / dx
    fl = _flattening(F["d"], F["e"], F["u"], p) if case["flatten"] else None
    st = _steepening(F["d"], p, dx) if case["steepen"] else None
    cells = slice(2, n - 2)
    cs = torch.sqrt(GAMMA * p[:, cells] / F["d"][:, cells])
    u = F["u"][:, cells]
    h = 0.5 * dt / dx
    cm, c0, cp = (u - cs) * h, u * h, (u + cs) * h
    par = [_parabola(F["d"], st, fl), _parabola(p, None, fl), _parabola(F["u"], None, fl)]
    lo, hi = slice(0, n - 5), slice(1, n - 4)  # cells left and right of faces 3 .. n-3
    cut = lambda q, s: tuple(a[:, s] for a in q)  # noqa: E731
    g = acc[:, 2:n - 3] + acc[:, 3:n - 2] if acc is not None else None
    ch = (_mx(cp, 0.0), _mx(-cm, 0.0))
    L = _side([cut(q, lo) for q in par], tuple(x[:, lo] for x in (ch[0], cm, c0, cp)), True,
              dual, dt, g)
    R = _side([cut(q, hi) for q in par], tuple(x[:, hi] for x in (ch[1], cm, c0, cp)), False,
              dual, dt, g)
    ul, ur = u[:, lo], u[:, hi]
    side = lambda q: (  # noqa: E731
        torch.where(ul <= 0.0, _from_left(cut(q, lo), ch[0][:, lo]),
                    _from_left(cut(q, lo), c0[:, lo])),
        torch.where(ur >= 0.0, _from_right_char(cut(q, hi), ch[1][:, hi]),
                    _from_right(cut(q, hi), c0[:, hi])))
    for k in ("v", "w", "ge"):
        L[k], R[k] = side(_parabola(F[k], None, fl)) if F[k] is not None else (
            torch.zeros_like(L["d"]), torch.zeros_like(L["d"]))
    fx = (_hllc_flux if hllc else _two_shock_flux)(L, R, dual, qc)
    act = slice(3, n - 3)
    d, e = F["d"][:, act], F["e"][:, act]
    df = {k: fx[k][:, :-1] - fx[k][:, 1:] for k in ("d", "e", "u", "v", "w", "ge")}
    bad = (d + df["d"] <= 0.0) if hllc else (d + df["d"] <= 0.0) | (e < 0.0)
    if bool(bad.any()):
        raise _Fallback()
    inv = 1.0 / _mx(d + df["d"], SMALL_RHO)
    out = {k: (x.clone() if x is not None else None) for k, x in F.items()}
    for k in ("u", "v", "w"):
        if F[k] is not None:
            out[k][:, act] = (F[k][:, act] * d + df[k]) * inv
    en = _mx((e * d + df["e"]) * inv, 0.1 * e)
    if dual:
        ge = F["ge"][:, act]
        pc = _mx((GAMMA - 1.0) * ge * d, TINY)
        ges = qc * pc * ((fx["div"][:, :-1] - fx["div"][:, 1:]) if hllc else
                         (fx["ub"][:, :-1] - fx["ub"][:, 1:]))
        out["ge"][:, act] = _mx((ge * d + df["ge"] + ges) * inv, 0.5 * ge)
    if acc is not None:
        ga = acc[:, act]
        uo = out["u"][:, act] + dt * ga * 0.5 * (d * inv + 1.0)
        out["u"][:, act] = uo
        en = _mx(en + dt * ga * 0.5 * (uo + F["u"][:, act] * d * inv), TINY)
    out["e"][:, act] = en
    out["d"][:, act] = _mx(d + df["d"], SMALL_RHO)
    if dual:
        ke = 0.5 * sum(out[k] ** 2 for k in ("u", "v", "w") if out[k] is not None)
        ge1 = out["e"] - ke
        de = out["d"] * out["e"]
        right = torch.cat([de[:, 1:], de[:, -1:]], 1)
        new = de
        for _ in range(n):  # the left neighbour's energy is the updated one
            left = torch.cat([de[:, :1], new[:, :-1]], 1)
            top = _mx(_mx(de, left), right)
            ge = torch.where(ge1 * out["d"] / top > ETA2, ge1, out["ge"])
            g2 = torch.where(ge1 / out["e"] > ETA1, ge1, ge)
            g2 = _mx(g2, PMIN / ((GAMMA - 1.0) * out["d"]))
            ee = out["e"] - ge1 + g2
            again = out["d"] * ee
            if torch.equal(again, new):
                break
            new = again
        out["ge"], out["e"] = ge, ee
    for i, c in enumerate(cols):
        q = _parabola(c, None, fl)
        a, b = _from_left(cut(q, lo), ch[0][:, lo]), _from_left(cut(q, lo), c0[:, lo])
        ls = torch.where(ul <= 0.0, a * L["dc"] / L["da"], b * L["dc"] / L["d0"])
        a, b = _from_right_char(cut(q, hi), ch[1][:, hi]), _from_right(cut(q, hi), c0[:, hi])
        rs = torch.where(ur >= 0.0, a * R["dc"] / R["da"], b * R["dc"] / R["d0"])
        ls = _mx(torch.where(L["ov"], ls * L["da"] / L["dc"], ls), 1e-35)
        rs = _mx(torch.where(R["ov"], rs * R["da"] / R["dc"], rs), 1e-35)
        if hllc:
            w = fx["w4"]
            cf = qc * (w[0] * w[1] * ls + w[2] * w[3] * rs)
        else:
            cf = qc * fx["ub"] * fx["db"] * torch.where(fx["ub"] > 0.0, ls / L["d"], rs / R["d"])
        c[:, act] = _mx(c[:, act] + (cf[:, :-1] - cf[:, 1:]), 1e-5 * TINY)
    return out, fx


def _sweep(f, p, acc, dim, dx, dt, case, want_flux=False):
    """One sweep of a grid (fields (z, y, x), changed in place); its fluxes if wanted."""
    ax, rank = 2 - dim, _rank(case)
    n = p.shape[ax]
    roles = {"d": "d", "e": "te", "u": "v%d" % (dim + 1), "v": "v%d" % ((dim + 1) % 3 + 1),
             "w": "v%d" % ((dim + 2) % 3 + 1), "ge": "ge"}
    flat = lambda a: a.movedim(ax, 2).reshape(-1, n)  # noqa: E731
    shape = p.movedim(ax, 2).shape
    src = {r: (flat(f[k]) if k in f else None) for r, k in roles.items()}
    cols = [flat(f["col%d" % i]).clone() for i in range(case["colours"])]
    pf = flat(p)
    gf = flat(acc[dim]) if acc is not None else None
    parts, flux = [], []
    step = max(1, CHUNK // n)
    for i in range(0, pf.shape[0], step):
        s = slice(i, i + step)
        cc = [c[s] for c in cols]
        o, fx = _sweep_pencils({r: (a[s] if a is not None else None) for r, a in src.items()},
                               pf[s], gf[s] if gf is not None else None, cc, dx, dt, case)
        parts.append(o)
        if want_flux:
            flux.append({k: fx[k] for k in ("d", "e", "u", "v", "w", "ge")})
    for r, k in roles.items():
        if k in f:
            f[k].copy_(torch.cat([o[r] for o in parts]).reshape(shape).movedim(2, ax))
    for i, c in enumerate(cols):
        f["col%d" % i].copy_(c.reshape(shape).movedim(2, ax))
    if want_flux:
        return {roles[k]: torch.cat([x[k] for x in flux]).reshape(shape[0], shape[1], n - 5)
                for k in flux[0] if roles[k] in f}
    return None


def _pressure(f, case):
    if case["dual"]:
        ge = f["ge"]
    else:
        ge = f["te"] - 0.5 * sum(f["v%d" % (i + 1)] ** 2 for i in range(_rank(case)))
    return _mx((GAMMA - 1.0) * f["d"] * ge, PMIN)


def _courant(f, case, dxs):
    rank = _rank(case)
    act = tuple(slice(3, -3) if 2 - ax < rank else slice(None) for ax in range(3))
    cs = torch.sqrt(GAMMA * _pressure(f, case) / f["d"])[act]
    s = sum((cs + f["v%d" % (i + 1)][act].abs()) / dxs[i] for i in range(rank))
    return 1.0 / s.max()


def _step(f, acc, case, dxs, dt, want_flux=False):
    p = _pressure(f, case)
    return [_sweep(f, p, acc, d, dxs[d], dt, case, want_flux) for d in range(_rank(case))]


def _ghosts(a, rank, bc):
    act = tuple(slice(3, -3) if 2 - ax < rank else slice(None) for ax in range(3))
    return _pad(a[act], rank, bc)


def exact(case, seed):
    try:
        return _exact(case, seed)
    except _Fallback:
        return None


def _exact(case, seed):
    if case["kind"] == "level":
        if _cells(case) > 4e7 or case["patches"] > 260:
            return None
        edges, flat, views = _level_inputs(case, seed)
        dx = 1.0 / 128.0
        dt = CFL * min(_courant(v, case, (dx,) * 3) for v in views)
        new = []
        for v in views:
            _step(v, None, case, (dx,) * 3, dt)
            new.append(_courant(v, case, (dx,) * 3))
            for k in NAMES:
                v[k].copy_(_ghosts(v[k], 3, "outflow"))
        return dict(flat, dt=(CFL * min(new)).reshape(1))
    rank = _rank(case)
    f, acc = _box_inputs(case, seed)
    dxs = (1.0 / case["nx"],) * 3
    dt = CFL * _courant(f, case, dxs)
    if case["kind"] == "host":
        dt = HOST_DT_SHARE * dt
    fx = _step(f, acc, case, dxs, dt, case["kind"] == "host")
    if case["kind"] == "host":
        out = {k: v.cpu().numpy() for k, v in f.items()}
        out["left"], out["right"] = _captured(case, fx)
        return out
    new = CFL * _courant(f, case, dxs)
    f = {k: _ghosts(v, rank, case["bc"]) for k, v in f.items()}
    return dict(f, dt=new.reshape(1))


def _captured(case, fx):
    """The subgrid's face fluxes, laid out like the capture arrays (first axis fastest)."""
    box = _subgrid_box(case)
    out = {"left": [[None] * 3 for _ in range(6)], "right": [[None] * 3 for _ in range(6)]}
    for dim in range(3):
        for side in ("left", "right"):
            lo, hi = box[side + "_start"][dim], box[side + "_end"][dim]
            face = lo[dim] - 3 + (1 if side == "right" else 0)
            for slot, k in enumerate(NAMES):
                a = fx[dim][k][:, :, face]  # (outer, inner) transverse axes, z y x order
                t = [i for i in (2, 1, 0) if i != dim]
                a = a[lo[t[0]]:hi[t[0]] + 1, lo[t[1]]:hi[t[1]] + 1]
                out[side][slot][dim] = a.reshape(-1).cpu().numpy()
    return out["left"], out["right"]
