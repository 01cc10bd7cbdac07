"""The work a user has this library do, as cases that can be timed and compared.

Each case is one call (or forward/backward pair) through the public Python
binding, on inputs made on the GPU from a seed: Zel'dovich-displaced lattices
or clustered sets with their periodic overload copies, sorted by grid cell as
the simulation's resort leaves them before a kick.  Where a call permutes or
moves the caller's arrays in place, a pass starts from the step's arrays by
copying them first, so that every pass does the same work.

`listed` gives the fixed cases, `draw` more of the same ranges, `prepare` a
case's inputs, `run` one pass, `work` the bytes and operations a pass cannot do
without and `exact` the 64-bit result in plain torch.
"""
import dataclasses
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "hacc-coral_gb300"))

import hsr  # noqa: E402
import synth  # noqa: E402
import treepm  # noqa: E402

DEV = "cuda"
FIELDS = synth.FIELDS
RMAX = float(synth.RMAX)
OVERLOAD = 4  # overload cells: 8 Mpc/h at 2 Mpc/h per cell
LIST_CELL = 4  # cells a side of a caller-held leaf


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # the smallest kick that is made in earnest: a rank of a test run, where
        # launches and host work are the time
        dict(name="kick_8", do="kick", kind="zeldovich", ng=8, z=50.0, nd=32, tdpts=1, angle=0.1,
             law=0),
        # the benchmark's kick: a rank's 128^3 cells at the start of a run
        dict(name="kick_128", do="kick", kind="zeldovich", ng=128, z=50.0, nd=128, tdpts=1,
             angle=0.1, law=0),
        # the largest: a late-time rank, 256^3 particles with halos
        dict(name="kick_clustered_256", do="kick", kind="clustered", ng=256, z=0.0, nd=256,
             tdpts=1, angle=0.1, law=0),
        # the drop-in constructor on the simulation's own host arrays, odd size
        dict(name="tree_host_45", do="tree", kind="zeldovich", ng=45, z=10.0, nd=64, tdpts=1,
             angle=0.1, law=0),
        # one PM step's five sub-cycles of a small single-rank run, host arrays
        dict(name="subcycle_32", do="subcycle", kind="zeldovich", ng=32, z=50.0, nd=128, tdpts=1,
             angle=0.1, law=0, nsub=5),
        # a whole TreePM step with the arrays resident: both PM kicks, 5 sub-cycles
        dict(name="treepm_96", do="treepm", kind="zeldovich", ng=96, z=50.0, nd=128, tdpts=1,
             angle=0.1, law=0, nsub=5, f64=True),
        # force and its gradient, as a differentiable program calls the pair
        dict(name="grad_64", do="grad", kind="zeldovich", ng=64, z=10.0, nd=128, tdpts=1,
             angle=0.1, law=0, nbox=1),
        # the same through 12-point pseudo-particles in a clustered box
        dict(name="grad_quad_clustered_48", do="grad", kind="clustered", ng=48, z=0.0, nd=32,
             tdpts=12, angle=0.5, law=0, nbox=1),
        # several independent boxes in one launch each way, as the multi-step
        # adjoint runs them
        dict(name="grad_boxes_8x96", do="grad", kind="zeldovich", ng=96, z=50.0, nd=128, tdpts=1,
             angle=0.1, law=0, nbox=8),
        # the long-range kick in the reference's precision
        dict(name="pm_128", do="pm", kind="zeldovich", ng=128, z=50.0, f64=True),
        # its adjoint, single precision, a size that is not a power of two
        dict(name="pm_vjp_100", do="pm_vjp", kind="zeldovich", ng=100, z=10.0, f64=False),
        # the kick over lists that the caller holds, the 5th-order law
        dict(name="lists_50", do="lists", kind="zeldovich", ng=50, z=10.0, law=1),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    do = rng.choice(["kick", "kick", "tree", "subcycle", "treepm", "grad", "grad", "pm", "pm_vjp",
                     "lists"])
    kind = rng.choice(["zeldovich", "zeldovich", "clustered"])
    c = dict(do=do, kind=kind, z=round(rng.uniform(5.0, 50.0), 1) if kind == "zeldovich" else 0.0)
    if do in ("pm", "pm_vjp"):
        return dict(c, ng=2 * size(6, 96), f64=rng.random() < 0.6)
    if do == "lists":
        return dict(c, kind="zeldovich", z=round(rng.uniform(5.0, 50.0), 1), ng=size(8, 90),
                    law=rng.choice([0, 1]))
    quad = do in ("kick", "grad") and rng.random() < 0.25
    c.update(nd=rng.choice([32, 64, 128, 256]), tdpts=12 if quad else 1,
             angle=round(rng.uniform(0.3, 0.8), 2) if quad else 0.1,
             law=rng.choice([0, 0, 0, 1]))
    if do == "kick":
        return dict(c, ng=size(8, 64 if quad else 160))
    if do == "tree":
        return dict(c, ng=size(8, 80))
    if do in ("subcycle", "treepm"):
        # early times only: later, a last bit of a velocity soon decides on which
        # side of a split a particle of the next sub-cycle's tree falls
        c.update(kind="zeldovich", z=round(rng.uniform(20.0, 50.0), 1), nsub=rng.choice([1, 3, 5]))
        if do == "subcycle":
            return dict(c, ng=size(8, 64))
        return dict(c, ng=2 * size(6, 40), f64=rng.random() < 0.6)
    nbox = rng.choice([1, 1, 2, 5])
    return dict(c, ng=size(8, 48 if quad else 64 if nbox > 1 else 112), nbox=nbox)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _wave_numbers(ng):
    k = torch.fft.fftfreq(ng, device=DEV, dtype=torch.float64) * (2 * math.pi)
    kz = torch.fft.rfftfreq(ng, device=DEV, dtype=torch.float64) * (2 * math.pi)
    return k[:, None, None], k[None, :, None], kz[None, None, :]


def _zeldovich(ng, z, gen):
    """Positions and velocities of a displaced ng^3 lattice, P(k) ~ k^-2, the
    rms displacement synth.SIGMA_Z50 at z = 50 grown linearly."""
    noise = torch.randn(ng, ng, ng, generator=gen, device=DEV, dtype=torch.float64)
    K = _wave_numbers(ng)
    k2 = K[0] ** 2 + K[1] ** 2 + K[2] ** 2
    k2[0, 0, 0] = 1.0
    dk = torch.fft.rfftn(noise) / k2.sqrt()
    dk[0, 0, 0] = 0.0
    psi = torch.stack([torch.fft.irfftn(1j * k / k2 * dk, s=(ng,) * 3) for k in K])
    psi *= synth.SIGMA_Z50 * 51.0 / (1.0 + z) / psi.std()
    q = torch.arange(ng, device=DEV, dtype=torch.float64) + 0.5
    lattice = torch.stack(torch.meshgrid(q, q, q, indexing="ij"))
    a = 1.0 / (1.0 + z)
    rate = a * dataclasses.replace(synth.stepper(), pp=a).adot
    return ((lattice + psi).reshape(3, -1).T % ng, psi.reshape(3, -1).T * rate)


def _clustered(ng, gen):
    """60 % uniform, 40 % in NFW halos: 4000 of them in 256^3 cells, masses over
    two decades (slope -1.9), concentrations 4..10, radii 0.5..4 cells."""
    def rand(*s):
        return torch.rand(*s, generator=gen, device=DEV, dtype=torch.float64)

    total, nhalo = ng ** 3, max(1, round(4000 * (ng / 256) ** 3))
    in_halos = int(0.4 * total)
    m = (1.0 + rand(nhalo) * (100.0 ** -0.9 - 1.0)) ** (-1.0 / 0.9)
    owner = torch.searchsorted((m / m.sum()).cumsum(0), rand(in_halos)).clamp(max=nhalo - 1)
    lo = 100.0 ** (-1.0 / 3.0)
    rvir = 0.5 + 3.5 * ((m / 100.0) ** (1.0 / 3.0) - lo) / (1.0 - lo)
    conc, centre = 4.0 + 6.0 * rand(nhalo), rand(nhalo, 3) * ng
    xs = torch.linspace(0.0, 10.0, 8193, device=DEV, dtype=torch.float64)
    mu = torch.log1p(xs) - xs / (1.0 + xs)
    c = conc[owner]
    want = rand(in_halos) * (torch.log1p(c) - c / (1.0 + c))
    at = torch.searchsorted(mu, want).clamp(1, 8192)
    x = xs[at - 1] + (want - mu[at - 1]) / (mu[at] - mu[at - 1]) * (xs[1] - xs[0])
    way = torch.randn(in_halos, 3, generator=gen, device=DEV, dtype=torch.float64)
    way /= way.norm(dim=1, keepdim=True)
    pos = torch.cat([rand(total - in_halos, 3) * ng,
                     centre[owner] + (x / c * rvir[owner])[:, None] * way])
    vel = 0.01 * torch.randn(pos.shape, generator=gen, device=DEV, dtype=torch.float64)
    return pos % ng, vel


def _particles(case, seed):
    """A rank's ten arrays on the GPU and its grid size: the box with its
    overload copies in [0, ng + 2 OVERLOAD + 1)^3, sorted by unit cell."""
    ng = case["ng"]
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    pos, vel = (_clustered(ng, gen) if case["kind"] == "clustered"
                else _zeldovich(ng, case["z"], gen))
    ngo, nglt = OVERLOAD, ng + 2 * OVERLOAD + 1
    pos = (pos + ngo).float()
    ids = torch.arange(len(pos), device=DEV)
    ghost = torch.zeros(len(pos), device=DEV, dtype=torch.int16)
    for d in range(3):
        up, down = pos[:, d] + ng < nglt, pos[:, d] - ng >= 0
        copies = [pos[up], pos[down]]
        copies[0][:, d] += ng
        copies[1][:, d] -= ng
        pos = torch.cat([pos] + copies)
        vel, ids = (torch.cat([a, a[up], a[down]]) for a in (vel, ids))
        ghost = torch.cat([ghost, torch.ones_like(ghost[up]), torch.ones_like(ghost[down])])
    # a rank's particle count is fixed here (inputs of another seed have the same
    # shapes): the overload copies nearest to the box, or some at random more
    want = int(0.97 * (nglt ** 3 - ng ** 3))
    out = torch.maximum(ngo - pos, pos - (ngo + ng)).amax(1)
    out = torch.where(ghost > 0, out, -1.0)
    keep = torch.sort(out, stable=True)[1][:ng ** 3 + want]
    pos, vel, ids, ghost = (a[keep] for a in (pos, vel, ids, ghost))
    more = ng ** 3 + want - len(pos)
    if more > 0:
        extra = torch.rand(more, 3, generator=gen, device=DEV) * nglt
        extra[:, 0] *= ngo / nglt
        pos, vel = torch.cat([pos, extra]), torch.cat([vel, torch.zeros_like(extra).double()])
        ids = torch.cat([ids, torch.zeros_like(ids[:1]).expand(more)])
        ghost = torch.cat([ghost, torch.ones_like(ghost[:1]).expand(more)])
    pos = pos.clamp(min=0.0, max=float(np.nextafter(np.float32(nglt), np.float32(0))))
    cell = pos.long()
    order = torch.sort((cell[:, 0] * nglt + cell[:, 1]) * nglt + cell[:, 2], stable=True)[1]
    pos, vel, ids, ghost = pos[order], vel[order].float(), ids[order], ghost[order]
    f = {k: pos[:, d].contiguous() for d, k in enumerate("xyz")}
    f.update({k: vel[:, d].contiguous() for d, k in enumerate(("vx", "vy", "vz"))})
    f.update(mass=torch.ones_like(f["x"]), phi=torch.zeros_like(f["x"]), id=ids, mask=ghost)
    return f, nglt


class _Arrays:
    """The ten arrays in one allocation (each on a 256-byte boundary), so that a
    pass starts from the step's arrays with one copy."""

    def __init__(self, fields, host=False):
        at, where = 0, {}
        for k in FIELDS:
            where[k] = at
            at += (fields[k].numel() * fields[k].element_size() + 255) & ~255
        self.n = fields["x"].numel()
        self.first = torch.zeros(at, dtype=torch.uint8, device=DEV)
        for k in FIELDS:
            self._view(self.first, where[k], fields[k]).copy_(fields[k])
        if host:
            self.first = self.first.cpu()
        self.now = torch.empty_like(self.first, pin_memory=host)
        self.views = {k: self._view(self.now, where[k], fields[k]) for k in FIELDS}
        for k in FIELDS:
            setattr(self, k, self.views[k].numpy() if host else self.views[k])
        if host:
            self.mask = self.mask.view(np.uint16)

    @staticmethod
    def _view(flat, at, like):
        return flat[at:at + like.numel() * like.element_size()].view(like.dtype)

    def restore(self):
        self.now.copy_(self.first)
        if self.now.is_cuda:
            torch.cuda.current_stream().synchronize()


def _box(nglt):
    """What synth.kick_params reads of a particle set."""
    class Box:
        pass

    b = Box()
    b.nglt = (nglt,) * 3
    return b


def _kick_params(case, nglt):
    kp = synth.kick_params(_box(nglt), nd=case["nd"], open_angle=case["angle"],
                           tdpts=case["tdpts"], nsub=case.get("nsub", 5))
    return dataclasses.replace(kp, law=case["law"])


def _caller_lists(f, nglt):
    """Leaves of LIST_CELL^3 cells with lists of their 27 neighbours' particles:
    the table in leaf order and the index lists, leaves of the interior only."""
    nc = -(-nglt // LIST_CELL)
    pos = torch.stack([f["x"], f["y"], f["z"]], 1)
    cell = (pos / LIST_CELL).long()
    key = (cell[:, 0] * nc + cell[:, 1]) * nc + cell[:, 2]
    key, order = torch.sort(key, stable=True)
    count = torch.bincount(key, minlength=nc ** 3)
    begin = count.cumsum(0) - count
    i = torch.arange(1, nc - 1, device=DEV)
    leaf = torch.stack(torch.meshgrid(i, i, i, indexing="ij"), -1).reshape(-1, 3)
    o = torch.arange(-1, 2, device=DEV)
    off = torch.stack(torch.meshgrid(o, o, o, indexing="ij"), -1).reshape(-1, 3)
    near = leaf[:, None, :] + off[None]
    near = (near[..., 0] * nc + near[..., 1]) * nc + near[..., 2]
    leaf = (leaf[:, 0] * nc + leaf[:, 1]) * nc + leaf[:, 2]
    runs = count[near.reshape(-1)]
    ends = runs.cumsum(0)
    index = torch.arange(int(ends[-1]), device=DEV)
    index = index + torch.repeat_interleave(begin[near.reshape(-1)] - (ends - runs), runs)
    length = count[near].sum(1)
    table = torch.cat([pos[order], f["mass"][order][:, None]], 1).contiguous()
    return dict(table=table, leaf_offset=begin[leaf].int(), leaf_count=count[leaf].int(),
                list_begin=length.cumsum(0) - length, list_len=length.int(),
                list_index=index.int())


def prepare(case, seed):
    do = case["do"]
    s = dict(do=do, ctx=hsr.default_context())
    nbox = case.get("nbox", 1)
    sets = [_particles(case, seed * 16 + b) for b in range(nbox)]
    f, nglt = sets[0]
    if do in ("kick", "tree", "subcycle", "treepm"):
        s["p"] = _Arrays(f, host=do in ("tree", "subcycle"))
        s["kp"] = _kick_params(case, nglt)
    if do in ("subcycle", "treepm"):
        s["step"] = treepm.plan(50.0, 20.0, 3)[0]
        s["nglt"], s["nsub"] = (nglt,) * 3, case["nsub"]
    if do == "treepm":
        s["step"] = treepm.step_params(
            s["step"], s["kp"], case["nsub"], case["ng"], OVERLOAD, s["nglt"],
            precision=hsr.PM_F64 if case["f64"] else hsr.PM_F32)
    if do == "grad":
        s["x"] = [[p[k] for k in "xyz"] for p, _ in sets]
        s["m"] = [p["mass"] for p, _ in sets]
        s["kp"] = [_kick_params(case, n) for _, n in sets]
    if do in ("grad", "pm_vjp"):
        gen = torch.Generator(device=DEV)
        gen.manual_seed(seed * 16 + 15)
        s["u"] = [[torch.randn(p["x"].shape, generator=gen, device=DEV) for _ in range(3)]
                  for p, _ in sets]
    if do in ("pm", "pm_vjp"):
        s["p"] = f
        s["v"] = [f[k].clone() for k in ("vx", "vy", "vz")]
        ts = synth.stepper()
        s["prm"] = treepm.pm_params(ts, 1.0, case["ng"], OVERLOAD,
                                    precision=hsr.PM_F64 if case["f64"] else hsr.PM_F32)
    if do == "lists":
        s["lists"] = _caller_lists(f, nglt)
        s["v"] = [torch.zeros_like(f["x"]) for _ in range(3)]
        s["law"] = case["law"]
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def run(s):
    return _RUN[s["do"]](s)


def _run_kick(s):
    p = s["p"]
    p.restore()
    s["ctx"].rcb_kick_device(p.views, p.n, s["kp"])
    return dict(p.views)


def _run_tree(s):
    p, kp = s["p"], s["kp"]
    p.restore()
    hsr.RCBForceTree(kp.min, kp.max, kp.min_force, kp.max_force, p.n, p.x, p.y, p.z, p.vx, p.vy,
                     p.vz, p.mass, p.phi, p.id, p.mask, kp.avg_mass, kp.fsrrmax, kp.rsm,
                     kp.open_angle, kp.nd, kp.ds, kp.tmin, hsr.ForceLawSR(kp.rsm, kp.law),
                     kp.fcoeff, kp.ppc, kp.tdpts, ctx=s["ctx"])
    return {k: s["p"].views[k] for k in FIELDS}


def _run_subcycle(s):
    p, ts = s["p"], s["step"].mid
    p.restore()
    s["ctx"].subcycle(p, s["kp"], s["nsub"], s["nglt"], ts.alpha, ts.pp,
                      float(synth.stream_tau(ts, s["nsub"])), ts.adot)
    return {k: s["p"].views[k] for k in FIELDS}


def _run_treepm(s):
    p = s["p"]
    p.restore()
    treepm.step_device(s["ctx"], p.views, p.n, s["step"])
    return dict(p.views)


def _run_grad(s):
    ctx = s["ctx"]
    dv, xb = ([[torch.empty_like(a) for a in box] for box in s["x"]] for _ in range(2))
    if len(s["x"]) == 1:
        ctx.force_fwd_device(*s["x"][0], s["m"][0], *dv[0], s["kp"][0])
        ctx.force_vjp_device(*s["u"][0], *xb[0])
    else:
        ctx.force_fwd_batch_device(s["x"], s["m"], dv, s["kp"])
        ctx.force_vjp_batch_device(s["u"], xb)
    return dict(dv=dv, xbar=xb)


def _run_pm(s):
    s["ctx"].pm_kick_device(*[s["p"][k] for k in "xyz"], *s["v"], s["prm"])
    return s["v"]


def _run_pm_vjp(s):
    xb = [torch.empty_like(a) for a in s["v"]]
    s["ctx"].pm_vjp_device(*[s["p"][k] for k in "xyz"], *s["u"][0], *xb, s["prm"])
    return xb


def _run_lists(s):
    a = s["lists"]
    hsr.kick_lists_noalloc(a["table"], len(a["table"]), a["leaf_offset"], a["leaf_count"],
                           a["list_begin"], a["list_len"], a["list_index"], *s["v"], 1e-3,
                           law=s["law"])
    return s["v"]


_RUN = dict(kick=_run_kick, tree=_run_tree, subcycle=_run_subcycle, treepm=_run_treepm,
            grad=_run_grad, pm=_run_pm, pm_vjp=_run_pm_vjp, lists=_run_lists)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def work(case):
    """The caller's arrays once each way, and 31 operations for every pair
    within the cutoff (about three times that for its derivative); a PM solve is
    four real transforms."""
    ng, do = case["ng"], case["do"]
    box, n = ng ** 3, (ng + 2 * OVERLOAD + 1) ** 3
    mean = 4.0 / 3.0 * math.pi * RMAX ** 3  # particles within the cutoff of one
    active = min(n, (ng + 2 * OVERLOAD + 1 - 2 * synth.EDGE + 2) ** 3)
    pairs = active * mean
    if case["kind"] == "clustered":
        # the uniform part, and halos whose particles mostly see one another
        nhalo = max(1, round(4000 * (ng / 256) ** 3))
        u = (np.arange(nhalo) + 0.5) / nhalo
        m = (1.0 + u * (100.0 ** -0.9 - 1.0)) ** (-1.0 / 0.9)
        halo = m / m.sum() * 0.4 * box
        pairs = active * mean * 0.84 + 0.7 * active / box * float((halo ** 2).sum())
    fft = 4 * 2.5 * box * math.log2(box) + 20 * box
    pm = dict(bytes=n * 36 + box * 16, flops=fft + n * 100)
    if do in ("kick", "tree"):
        return dict(bytes=84 * n, flops=31 * pairs)
    if do in ("subcycle", "treepm"):
        w = dict(bytes=84 * n, flops=case["nsub"] * (31 * pairs + 12 * n))
        return w if do == "subcycle" else {k: w[k] + 2 * pm[k] for k in w}
    if do == "grad":
        return dict(bytes=case["nbox"] * 52 * n, flops=case["nbox"] * 31 * 3.5 * pairs)
    if do == "pm":
        return pm
    if do == "pm_vjp":
        return dict(bytes=n * 36 + box * 32, flops=2 * fft + n * 250)
    nc = -(-(ng + 2 * OVERLOAD + 1) // LIST_CELL)
    entries = (nc - 2) ** 3 * 27 * LIST_CELL ** 3
    return dict(bytes=40 * n + 4 * entries, flops=31 * (nc - 2) ** 3 * LIST_CELL ** 3 * mean)


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

_POLY = {0: (0.271431, -0.0783394, 0.0133122, -0.00159485, 0.000132336, -0.00000663394,
             0.000000147305),
         1: (0.269327, -0.0750978, 0.0114808, -0.00109313, 0.0000605491, -0.00000147177)}


def _direct(pos, mass, active, law, rsm, u=None):
    """sum_j m_j g(r2) (x_j - x_i) over the particles within the cutoff, for
    the active i; with u (the cotangent of m_i times that), also its gradient
    for every position.  Cell lists, float64."""
    coeff = [float(np.float32(a)) for a in _POLY[law]]
    side = RMAX * (1 + 1e-6)
    cell = (pos / side).long() + 1
    nc = int(cell.max()) + 2
    key, order = torch.sort((cell[:, 0] * nc + cell[:, 1]) * nc + cell[:, 2])
    count = torch.bincount(key, minlength=nc ** 3)
    begin = count.cumsum(0) - count
    most = int(count.max())
    slot = torch.arange(len(pos), device=DEV) - begin[key]
    padded = torch.full((nc ** 3, most), -1, device=DEV, dtype=torch.int64)
    padded[key, slot] = order
    used = torch.nonzero(count).flatten()
    acc = torch.zeros(len(pos), 3, device=DEV, dtype=torch.float64)
    grad = torch.zeros_like(acc) if u is not None else None
    wi = active.double() * (mass if law == 0 else 1.0)
    chunk = max(1, 12_000_000 // (most * most))
    for c0 in range(0, len(used), chunk):
        here = used[c0:c0 + chunk]
        i = padded[here]
        for o in range(27):
            j = padded[here + (o // 9 - 1) * nc * nc + (o // 3 % 3 - 1) * nc + o % 3 - 1]
            d = pos[j.clamp(min=0)][:, None, :, :] - pos[i.clamp(min=0)][:, :, None, :]
            r2 = d.square().sum(-1)
            on = (r2 < RMAX * RMAX) & (i >= 0)[:, :, None] & (j >= 0)[:, None, :]
            on &= i[:, :, None] != j[:, None, :]
            s = r2 + rsm * rsm
            g = s ** -1.5
            p, dp = torch.zeros_like(r2), torch.zeros_like(r2)
            for k in range(len(coeff) - 1, -1, -1):
                if u is not None:
                    dp = dp * r2 + p
                p = p * r2 + coeff[k]
            g = torch.where(on, (g - p) * mass[j.clamp(min=0)][:, None, :], 0.0)
            a = (g[..., None] * d).sum(2)
            acc.index_add_(0, i.clamp(min=0).flatten(), a.reshape(-1, 3))
            if u is not None:
                mj, mi = mass[j.clamp(min=0)][:, None, :], mass[i.clamp(min=0)][:, :, None]
                g2 = torch.where(on, 2.0 * (-1.5 * s ** -2.5 - dp), 0.0)
                # particle i as a source of every active j, less its own force's share
                uj = (u * wi[:, None])[j.clamp(min=0)][:, None, :, :] * mi[..., None]
                ui = (u * wi[:, None])[i.clamp(min=0)][:, :, None, :] * mj[..., None]
                w = uj - ui
                g1 = torch.where(on, s ** -1.5 - p, 0.0)
                v = (g1[..., None] * w + (g2 * (w * d).sum(-1))[..., None] * d).sum(2)
                grad.index_add_(0, i.clamp(min=0).flatten(), v.reshape(-1, 3))
    acc *= wi[:, None]
    return (acc, grad) if u is not None else acc


def _rcb(pos, mass, kp):
    """The reference's tree order (input index by tree slot) and which particles
    lie in leaves that touch the force box, from float32 positions."""
    n = len(pos)
    order = torch.arange(n, device=DEV)
    active = torch.zeros(n, dtype=torch.bool, device=DEV)
    offset, count = (torch.tensor([v], device=DEV) for v in (0, n))
    while len(offset):
        nodes = len(offset)
        node = torch.repeat_interleave(torch.arange(nodes, device=DEV), count)
        rank = torch.arange(len(node), device=DEV) - (count.cumsum(0) - count)[node]
        slot = offset[node] + rank
        p, m = pos[order[slot]], mass[order[slot]]
        by = node[:, None].expand(-1, 3)
        lo = torch.zeros(nodes, 3, device=DEV).scatter_reduce(0, by, p, "amin", include_self=False)
        hi = torch.zeros(nodes, 3, device=DEV).scatter_reduce(0, by, p, "amax", include_self=False)
        total = torch.zeros(nodes, 4, device=DEV, dtype=torch.float64)
        total.index_add_(0, node, torch.cat([(p * m[:, None]), m[:, None]], 1).double())
        centre = (total[:, :3] / total[:, 3:]).float()
        size = hi - lo
        axis = torch.where((size[:, 0] > size[:, 1]) & (size[:, 0] > size[:, 2]), 0,
                           torch.where(size[:, 1] > size[:, 2], 1, 2))
        split = centre.gather(1, axis[:, None])[:, 0]
        left = p.gather(1, axis[node][:, None])[:, 0] < split[node]
        nleft = torch.zeros(nodes, device=DEV, dtype=torch.int64).index_add_(0, node, left.long())
        inner = (count > kp.nd) & (nleft > 0) & (nleft < count)
        touch = torch.ones(nodes, dtype=torch.bool, device=DEV)
        for d in range(3):
            a, b = kp.min_force[d], kp.max_force[d]
            touch &= (((hi[:, d] < b) & (hi[:, d] > a)) | ((lo[:, d] < b) & (lo[:, d] > a)))
        active[order[slot]] = (touch & ~inner)[node]
        # a node too small to split keeps its order; any other is partitioned
        part = (count > kp.nd)[node]
        lrank = left.long().cumsum(0) - left.long()
        lrank = lrank - lrank[(count.cumsum(0) - count)[node]]
        idx = torch.zeros(n, device=DEV, dtype=torch.int64)
        mine = left & part
        idx[offset[node[mine]] + lrank[mine]] = slot[mine]
        to = torch.where(mine, offset[node] + lrank, slot)
        end = (offset + nleft)[node]
        go = torch.nonzero(part & ~left & (to < end)).flatten()
        while len(go):  # the swap sequence carries a right element from slot to slot
            to[go] = idx[to[go]]
            go = go[to[go] < end[go]]
        moved = order[slot]
        order[to] = moved
        offset, count, nleft = offset[inner], count[inner], nleft[inner]
        offset = torch.stack([offset, offset + nleft], 1).flatten()
        count = torch.stack([nleft, count - nleft], 1).flatten()
    return order, active


def _quiet_spectra(ng):
    """The quiet solver's i g(k_a) Green's functions on the full spectrum."""
    step = 2.0 * math.pi / ng
    kk = torch.arange(ng, device=DEV, dtype=torch.float64)
    k = torch.where(kk < ng // 2, kk, kk - ng) * step
    kn = torch.where(k == 0, 1.0, k)
    filt = torch.where(k == 0, 1.0, torch.exp(-0.16 * k * k) * (torch.sin(0.5 * kn) / (0.5 * kn)) ** 3)
    grad = 4.0 / 3.0 * torch.sin(k) - 1.0 / 6.0 * torch.sin(2.0 * k)
    c = kk * step
    den = (-21.0 / 8.0 + 128.0 / 45.0 * torch.cos(c) - 2.0 / 9.0 * torch.cos(2 * c)
           + torch.cos(4 * c) / 360.0)
    f = filt[:, None, None] * filt[None, :, None] * filt[None, None, :]
    d = den[:, None, None] + den[None, :, None] + den[None, None, :]
    d[0, 0, 0] = 1.0
    green = f / d
    green[0, 0, 0] = 0.0
    return [-1j * grad.reshape([-1 if b == a else 1 for b in range(3)]) * green for a in range(3)]


def _corners(pos, ng):
    """Per CIC corner: the alive cell or -1, the image cell or -1, the weight and
    its gradient."""
    base = pos.floor()
    t = pos - base
    base = base.long()
    nglt = ng + 2 * OVERLOAD + 1
    for o in range(8):
        bit = torch.tensor([o >> 2 & 1, o >> 1 & 1, o & 1], device=DEV)
        w = torch.where(bit == 1, t, 1.0 - t)
        sign = torch.where(bit == 1, 1.0, -1.0).double()
        dw = torch.stack([sign[0] * w[:, 1] * w[:, 2], sign[1] * w[:, 0] * w[:, 2],
                          sign[2] * w[:, 0] * w[:, 1]], 1)
        cell = base + bit
        local, alive = cell - OVERLOAD, ((cell >= OVERLOAD) & (cell < OVERLOAD + ng)).all(1)
        inside = ((cell >= 0) & (cell < nglt)).all(1)
        image = local % ng
        at = (image[:, 0] * ng + image[:, 1]) * ng + image[:, 2]
        yield alive, inside, at, w.prod(1), dw


def _exact_pm(case, s, vjp):
    ng, prm = case["ng"], s["prm"]
    pos = torch.stack([s["p"][k] for k in "xyz"], 1).double()
    scale = prm.fscal * prm.tau
    S = _quiet_spectra(ng)
    rho = torch.zeros(ng ** 3, device=DEV, dtype=torch.float64)
    for alive, _, at, w, _ in _corners(pos, ng):
        rho.index_add_(0, at, torch.where(alive, w, 0.0))
    rk = torch.fft.fftn(rho.reshape(ng, ng, ng))
    field = torch.stack([torch.fft.ifftn(x * rk).real.flatten() for x in S], 1)
    if not vjp:
        f = torch.zeros_like(pos)
        for _, inside, at, w, _ in _corners(pos, ng):
            f += torch.where(inside, w, 0.0)[:, None] * field[at]
        return [s["p"][k].double() + scale * f[:, d] for d, k in enumerate(("vx", "vy", "vz"))]
    u = torch.stack(s["u"][0], 1).double()
    adj = torch.zeros(ng ** 3, 3, device=DEV, dtype=torch.float64)
    xb = torch.zeros_like(pos)
    for _, inside, at, w, dw in _corners(pos, ng):
        w = torch.where(inside, w, 0.0)
        adj.index_add_(0, at, w[:, None] * u)
        xb += dw * torch.where(inside, (field[at] * u).sum(1), 0.0)[:, None]
    spec = sum(S[a].conj() * torch.fft.fftn(adj[:, a].reshape(ng, ng, ng)) for a in range(3))
    phi = torch.fft.ifftn(spec).real.flatten()
    for alive, _, at, _, dw in _corners(pos, ng):
        xb += dw * torch.where(alive, phi[at], 0.0)[:, None]
    return [scale * xb[:, d] for d in range(3)]


def exact(case, seed):
    """None where pseudo-particles, or positions rounded at every sub-cycle,
    make the result the tree's own rather than the direct sum's."""
    do = case["do"]
    if do in ("subcycle", "treepm"):
        return None
    if do not in ("pm", "pm_vjp") and (case["kind"] == "clustered" or case.get("tdpts", 1) != 1):
        return None
    s = prepare(case, seed)
    if do in ("pm", "pm_vjp"):
        return _exact_pm(case, s, do == "pm_vjp")
    if do == "lists":
        a = s["lists"]
        t = a["table"].double()
        active = torch.zeros(len(t), dtype=torch.bool, device=DEV)
        first = torch.repeat_interleave(a["leaf_offset"].long(), a["leaf_count"].long())
        n = a["leaf_count"].long()
        active[first + torch.arange(len(first), device=DEV)
               - torch.repeat_interleave(n.cumsum(0) - n, n)] = True
        acc = _direct(t[:, :3].contiguous(), t[:, 3].contiguous(), active, case["law"], 0.1)
        return [1e-3 * acc[:, d] for d in range(3)]
    if do == "grad":
        out = dict(dv=[], xbar=[])
        for x, m, u, kp in zip(s["x"], s["m"], s["u"], s["kp"]):
            pos = torch.stack(x, 1)
            _, active = _rcb(pos, m, kp)
            dv, xb = _direct(pos.double(), m.double(), active, case["law"], kp.rsm,
                             torch.stack(u, 1).double())
            out["dv"].append([kp.fcoeff * dv[:, d] for d in range(3)])
            out["xbar"].append([kp.fcoeff * xb[:, d] for d in range(3)])
        return out
    kp, arrays = s["kp"], s["p"]
    arrays.restore()
    f = {k: v.to(DEV) for k, v in arrays.views.items()}
    pos = torch.stack([f[k] for k in "xyz"], 1)
    order, active = _rcb(pos, f["mass"], kp)
    acc = _direct(pos.double(), f["mass"].double(), active, case["law"], kp.rsm)
    for d, k in enumerate(("vx", "vy", "vz")):
        f[k] = f[k].double() + kp.fcoeff * acc[:, d]
    return {k: None if k in ("id", "mask") else f[k].double()[order] for k in FIELDS}
