"""The work that is timed when a change is judged: force passes, whole steps
from particles to forces, the PM force, the far field and served boxes, each
through the calls a program makes.

Kinds of case (the "kind" of the dict):

  resident  p2p.Session.run_device on lists that stay on the device, then the
            result back in the caller's order: repeated passes over one list
            (the batching workload), replayed as a graph
  host      p2p.Session.force_pass on host arrays: what PhotoNs' drop-in entry
            points do once per step
  step      the tree rebuilt in place, the lists walked on the device, the pass
            and the result back in the caller's order: a time step of a program
            that keeps its particles on the device
  pm        p2p.ParticleMesh.forces: the long-range part of the same step
  far       p2p.FarField.far: the multipole part within the cutoff, when lists
            are walked with an open angle above 0
  serve     serve.Server: a burst of one request per resident box

Particles are the repository's mixes: a lattice with Gaussian displacements
("lattice") and 60% uniform with 40% in NFW halos ("clustered"), n per side,
spacing 1/n, split radius 1.2 cells of an n^3 mesh, list cutoff 4.5 split
radii, Plummer softening of 1/40 spacing (the drop-in settings: 1.25 cells of a
(2n)^3 mesh, clamp softening, cutoff x = 2.8125, open angle 0.4).
"""
import itertools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "photons-on-mt3000_b200"))

from photons_p2p import abi, serve  # noqa: E402
from photons_p2p import lists as host_lists  # noqa: E402
from photons_p2p import workloads as W  # noqa: E402
from photons_p2p.p2p import DeviceTree, FarField, ParticleMesh, Session, params_for  # noqa: E402

DEVICE = 0
FORMS = {"plain": abi.FORM_PLAIN_FP64, "split": abi.FORM_SPLIT, "kahan": abi.FORM_KAHAN_FP32}


def listed():
    return [
        # the smallest pass anyone runs (the smoke test's size): latency and launches
        dict(name="resident_12_plain", kind="resident", n=12, shape="lattice", leaf=32, form="plain", soft="clamp"),
        # the plain configuration's size, still short of filling the GPU
        dict(name="resident_32_split", kind="resident", n=32, shape="lattice", leaf=32, form="split", soft="plummer"),
        # the FP64 form, which PhotoNs gets by default, over clustered particles; an odd size
        dict(name="resident_65_plain", kind="resident", n=65, shape="clustered", leaf=32, form="plain", soft="clamp"),
        # the clustered configuration at the size the profiles use
        dict(name="resident_128_split", kind="resident", n=128, shape="clustered", leaf=32, form="split", soft="plummer"),
        # PhotoNs' own force step with its production settings, from and to host memory
        dict(name="host_32_dropin", kind="host", n=32, shape="lattice", leaf=32, form="plain", soft="dropin"),
        # a small time step: many short kernels
        dict(name="step_33_split", kind="step", n=33, shape="lattice", leaf=32, form="split", soft="plummer"),
        # an ordinary time step with large leaves; an odd size
        dict(name="step_101_leaf64", kind="step", n=101, shape="clustered", leaf=64, form="split", soft="plummer"),
        # the headline configuration, from particles to forces
        dict(name="step_256_split", kind="step", n=256, shape="clustered", leaf=32, form="split", soft="plummer"),
        # the long-range part of the headline configuration, particles in cell order
        dict(name="pm_256_ordered", kind="pm", n=256, mesh=256, shape="clustered", ordered=True),
        # a mesh finer than the particles, particles as they come, a tenth of them not deposited
        dict(name="pm_91_scattered", kind="pm", n=91, mesh=128, shape="clustered", ordered=False),
        # the far field with the production open angle
        dict(name="far_128", kind="far", n=128, shape="clustered", leaf=32),
        # a burst of requests to an ensemble of boxes of different sizes
        dict(name="serve_6_boxes", kind="serve", boxes=6, n=32, n_max=64, form="split"),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["resident"] * 3 + ["step"] * 3 + ["host", "pm", "far", "serve"])
    shape = rng.choice(["lattice", "clustered"])
    if kind == "pm":
        return dict(kind=kind, n=_logint(rng, 16, 256), mesh=2 * _logint(rng, 16, 128), shape=shape,
                    ordered=rng.random() < 0.5)
    if kind == "far":
        return dict(kind=kind, n=_logint(rng, 24, 160), shape="clustered", leaf=rng.choice([16, 32, 32, 64]))
    if kind == "serve":
        lo = _logint(rng, 16, 40)
        return dict(kind=kind, boxes=rng.randint(2, 8), n=lo, n_max=lo + rng.randint(0, 30),
                    form=rng.choice(["split", "split", "plain"]))
    form = rng.choice(["split", "split", "split", "plain", "plain", "kahan"])
    soft = rng.choice(["plummer", "plummer", "clamp", "dropin"])
    leaf = rng.choice([8, 16, 32, 32, 32, 64])
    top = {"plain": 80, "split": 128, "kahan": 128}[form]
    if kind == "step" and form != "plain":
        top = 224
    if leaf == 8:
        top = min(top, 64)
    if kind == "host":
        top = min(top, 100)
    if shape == "lattice" or soft == "dropin":
        top = min(top, 160)
    return dict(kind=kind, n=_logint(rng, 12, top), shape=shape, leaf=leaf, form=form, soft=soft)


# ------------------------------------------------------------------ inputs ---

def _device():
    return torch.device("cuda", DEVICE)


def _config(case):
    n, leaf = case["n"], case.get("leaf", 32)
    soft = case.get("soft", "plummer")
    if soft == "dropin":
        return W.ref_dropin_config(n, 2 * n, leaf)
    mode = W.SOFT_CLAMP if soft == "clamp" else W.SOFT_PLUMMER
    return W.PassConfig(f"{case['kind']}_{n}", n, n, 1.2, 4.5, mode, 1.0 / (40 * n), 2.25, leaf,
                        0.4 if case["kind"] == "far" else 0.0)


def _rng(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(1_000_003 * (int(seed) + 1))
    return g


def _lattice(n, seed):
    g = _rng(seed)
    i = (torch.arange(n, dtype=torch.float64, device=_device()) + 0.5) / n
    pos = torch.stack([c.reshape(-1) for c in torch.meshgrid(i, i, i, indexing="ij")])
    return torch.remainder(pos + torch.randn(pos.shape, generator=g, dtype=torch.float64, device=_device()) * (0.2 / n), 1.0)


def _clustered(n, seed):
    """60% uniform, 40% in NFW halos (concentration 4 to 12, counts from
    dN/dM ~ M^-1.9, truncated at r200), as workloads.clustered draws on the host."""
    g, dev = _rng(seed), _device()
    total = n ** 3
    nhalo = max(1, int(round(2000 * (n / 256.0) ** 3)))
    in_halos = int(round(0.4 * total))
    counts = torch.from_numpy(W.halo_counts(nhalo, in_halos, np.random.default_rng(int(seed) + 17))).to(dev)
    in_halos = int(counts.sum())

    def rand(*shape):
        return torch.rand(*shape, generator=g, dtype=torch.float64, device=dev)

    centre, conc = rand(3, nhalo), 4.0 + 8.0 * rand(nhalo)
    r200 = (3.0 * counts.double() / total / (4.0 * math.pi * 200.0)) ** (1.0 / 3.0)
    h = torch.repeat_interleave(torch.arange(nhalo, device=dev), counts, output_size=in_halos)
    c = conc[h]
    want = rand(in_halos) * (torch.log1p(c) - c / (1.0 + c))  # ln(1 + s) - s / (1 + s) at s = r / r_scale
    lo, hi = torch.zeros_like(want), c.clone()
    for _ in range(48):
        s = 0.5 * (lo + hi)
        below = torch.log1p(s) - s / (1.0 + s) < want
        lo, hi = torch.where(below, s, lo), torch.where(below, hi, s)
    v = torch.randn(3, in_halos, generator=g, dtype=torch.float64, device=dev)
    halos = centre[:, h] + (hi * r200[h] / c / v.norm(dim=0)) * v
    return torch.remainder(torch.cat([rand(3, total - in_halos), halos], dim=1), 1.0)[:, :total].contiguous()


def _particles(shape, n, seed):
    return _lattice(n, seed) if shape == "lattice" else _clustered(n, seed)


def _ghosted(pos, width):
    """The particles and their periodic images within `width` of the unit box
    (the caller's boundary exchange), and 1 for local, 0 for an image."""
    parts = [pos]
    for s in itertools.product((-1.0, 0.0, 1.0), repeat=3):
        if any(s):
            q = pos + torch.tensor(s, dtype=torch.float64, device=pos.device)[:, None]
            parts.append(q[:, ((q > -width) & (q < 1.0 + width)).all(dim=0)])
    allpos = torch.cat(parts, dim=1).contiguous()
    tag = torch.zeros(allpos.shape[1], dtype=torch.int32, device=pos.device)
    tag[:pos.shape[1]] = 1
    return allpos, tag


def _host_lists(cfg, allpos, tag):
    return host_lists.build_tree_lists(allpos.cpu().numpy(), tag.cpu().numpy(), cfg.maxleaf, cfg.box,
                                       cfg.cutoff_radius, cfg.open_angle)


class _Serving:
    """A server and its boxes; closed with the state."""

    def __init__(self, case, seed):
        cfg = _config(case)
        self.server = serve.Server(serve.serving_shape(FORMS[case["form"]], cfg.eps / cfg.split_radius),
                                   device=DEVICE, hbm_bytes=3 << 30)
        for pos, c in _boxes(case, seed):
            tl = _host_lists(c, *_ghosted(pos, c.cutoff_radius))
            k = self.server.add_box(tl, 0.5 / c.split_radius, 1.0 / pos.shape[1])
            self.server.preload(k, release_host=False)
        self.server.reserve_outputs(1)

    def __del__(self):
        if hasattr(self, "server"):
            self.server.close()


def _boxes(case, seed):
    """The serving ensemble's boxes: n spread from n to n_max, a lattice and a
    clustered box in turn."""
    out = []
    for b in range(case["boxes"]):
        n = case["n"] + (case["n_max"] - case["n"]) * b // max(1, case["boxes"] - 1)
        pos = _particles("clustered" if b % 2 else "lattice", n, 64 * int(seed) + b)
        out.append((pos, _config(dict(kind="serve", n=n))))
    return out


def prepare(case, seed):
    dev, kind = _device(), case["kind"]
    if kind == "serve":
        return dict(kind=kind, serving=_Serving(case, seed))
    n = case["n"]
    pos = _particles(case["shape"], n, seed)
    nlocal = pos.shape[1]
    if kind == "pm":
        m = case["mesh"]
        if case["ordered"]:
            pos = _cell_order(pos, m)
        tag = _pm_tag(case, nlocal)
        s = Session(DEVICE)
        return dict(kind=kind, session=s, pm=ParticleMesh(s, m, 1.0, 1.2 / m), pos=pos, tag=tag, mass=1.0 / nlocal,
                    acc=torch.empty((3, nlocal), dtype=torch.float64, device=dev))
    cfg = _config(case)
    mass = 1.0 / nlocal
    allpos, tag = _ghosted(pos, cfg.cutoff_radius)
    if kind == "host":
        tl = _host_lists(cfg, allpos, tag)
        slot = np.empty(tl.npart, np.int64)
        slot[tl.perm] = np.arange(tl.npart)  # where the tree put each of the caller's particles
        return dict(kind=kind, session=Session(DEVICE, params_for(cfg, FORMS[case["form"]], mass)), lists=tl,
                    slot=slot[:nlocal])
    s = Session(DEVICE, params_for(cfg, FORMS[case.get("form", "plain")], mass))
    state = dict(kind=kind, session=s, cfg=cfg, mass=mass, nlocal=nlocal, allpos=allpos, tag=tag,
                 tree=DeviceTree(s, allpos, tag, cfg.maxleaf, cfg.box),
                 out=torch.empty(allpos.shape, dtype=torch.float64, device=dev))
    if kind == "resident":
        tl = _host_lists(cfg, allpos, tag)
        d = [torch.from_numpy(np.ascontiguousarray(a)).to(dev)
             for a in (tl.pos, tl.leaf_ipart, tl.leaf_npart, tl.task_t, tl.task_s)]
        state["arrays"] = d
        state["call"] = (tl.npart, d[0].data_ptr(), tl.nleaf, d[1].data_ptr(), d[2].data_ptr(), tl.ntask,
                         d[3].data_ptr(), d[4].data_ptr())
    elif kind == "far":
        state["far"] = FarField(s)
        state["acc"] = torch.empty(allpos.shape, dtype=torch.float64, device=dev)
    torch.cuda.synchronize()  # the inputs are written before the session's own stream reads them
    return state


def _cell_order(pos, mesh):
    """Particles sorted by mesh cell, as a program that keeps them sorted has them."""
    cell = (pos * mesh).long().clamp_(0, mesh - 1)
    return pos[:, torch.argsort((cell[0] * mesh + cell[1]) * mesh + cell[2], stable=True)].contiguous()


def _pm_tag(case, nlocal):
    if case["ordered"]:
        return None
    tag = torch.ones(nlocal, dtype=torch.int32, device=_device())
    tag[::10] = 0
    return tag


# -------------------------------------------------------------------- runs ---

def run(state):
    kind = state["kind"]
    if kind == "serve":
        server = state["serving"].server
        tickets = [server.submit(k) for k in range(len(server.boxes))]
        return [server.wait(t)[0] for t in tickets]
    s = state["session"]
    if kind == "pm":
        state["pm"].forces(state["pos"], state["tag"], state["mass"], state["acc"])
        return state["acc"]
    if kind == "host":
        tl = state["lists"]
        acc, _ = s.force_pass(tl.pos, tl.leaf_ipart, tl.leaf_npart, tl.task_t, tl.task_s)
        return acc[:, state["slot"]]
    tree, out = state["tree"], state["out"]
    if kind == "resident":
        s.run_device(*state["call"])
        s.end()
        tree.unpermute(s.result_device(), out.data_ptr())
    elif kind == "step":
        cfg = state["cfg"]
        tree.rebuild(state["allpos"], state["tag"], cfg.maxleaf, cfg.box)
        _begin_on_tree(s, tree)
        s.submit_walk(tree, cfg.cutoff_radius, cfg.open_angle)
        s.end()
        tree.unpermute(s.result_device(), out.data_ptr())
    else:
        cfg, acc = state["cfg"], state["acc"]
        d_pos, _, d_ip, d_np = tree.device_arrays()
        state["far"].far(tree.struct, d_pos, d_ip, d_np, tree.npart, state["mass"], cfg.split_radius,
                         cfg.cutoff_radius, cfg.open_angle, 1e-15, acc.data_ptr())
        tree.unpermute(acc.data_ptr(), out.data_ptr())
    return out[:, :state["nlocal"]]


def _begin_on_tree(s, tree):
    d_pos, _, d_ip, d_np = tree.device_arrays()
    if s.lib.p2p_pass_begin_device(s.h, tree.npart, d_pos, None, tree.nleaf, d_ip, d_np):
        raise RuntimeError(s.lib.p2p_last_error().decode())


# ------------------------------------------------ work, tolerance, 64 bits ---

# Pairs within the cutoff sphere per particle at the mean density (cutoff of
# 5.4 spacings).
_SPHERE = 4.0 / 3.0 * math.pi * 5.4 ** 3


def _neighbours(shape, n):
    """Particles within the cutoff, averaged over a set's particles. Clustered
    sets: a fit to counts of seeded ones (800 at 12^3, 2800 at 33^3, 9000 to
    12000 from 65^3 to 256^3, where the halos are resolved alike)."""
    return _SPHERE * (1.0 if shape == "lattice" else min(15.0, 1.25 * (n / 12.0) ** 1.4))


# Floating-point operations of one pair: separation, squared distance,
# inverse cube root and the cutoff function, three multiply-adds.
_PAIR_FLOPS = {"split": 39, "kahan": 39, "plain": 75}


def work(case):
    kind = case["kind"]
    if kind == "serve":
        w = [work(dict(kind="host", n=case["n"] + (case["n_max"] - case["n"]) * b // max(1, case["boxes"] - 1),
                       shape="clustered" if b % 2 else "lattice", leaf=32, form=case["form"]))
             for b in range(case["boxes"])]
        return {"bytes": sum(x["bytes"] for x in w), "flops": sum(x["flops"] for x in w)}
    n = case["n"] ** 3
    if kind == "pm":
        m = case["mesh"] ** 3
        # positions twice (deposit, interpolation), forces once, the mesh written and read once per step
        return {"bytes": 72.0 * n + 16.0 * 4 * m, "flops": 250.0 * n + 5.0 * m * math.log2(m)}
    if kind == "far":
        # about one accepted pair per particle, 20 x 20 / 2 multiply-adds each
        return {"bytes": 48.0 * n, "flops": 450.0 * n}
    ghosted = (1.0 + 2 * 5.4 / case["n"]) ** 3 * n
    pairs = _neighbours(case["shape"], case["n"]) * n
    return {"bytes": 24.0 * ghosted + 24.0 * n, "flops": _PAIR_FLOPS[case["form"]] * pairs}


def tolerance(case):
    """About four times what was seen against exact(), and, for the PM, between
    runs whose atomics add in another order."""
    if case["kind"] == "pm":
        return {"rel": 1e-13, "max": 1e-12}
    if case["kind"] == "far":
        return {"rel": 1e-12, "max": 1e-11}
    if case["form"] == "plain":
        return {"rel": 2e-13, "max": 1e-11}
    # FP32 pair terms, each off by a few 2^-24 of itself; the largest where a
    # particle's sum is small beside its closest pairs' terms
    return {"rel": 3e-6, "max": 2e-4}


def exact(case, seed):
    kind = case["kind"]
    if kind == "pm":
        return _pm_exact(case, seed)
    if kind == "serve":
        if case["boxes"] * case["n_max"] ** 3 > 2_500_000:
            return None
        return [_direct(pos, c, 1.0 / pos.shape[1]).cpu().numpy() for pos, c in _boxes(case, seed)]
    # The far field is defined by its tree's accepted pairs, the drop-in
    # settings' sums by their lists (pairs beyond the list cutoff in part).
    if kind == "far" or case["soft"] == "dropin" or case["n"] > 66:
        return None
    pos = _particles(case["shape"], case["n"], seed)
    acc = _direct(pos, _config(case), 1.0 / pos.shape[1])
    return acc.cpu().numpy() if kind == "host" else acc


def _direct(pos, cfg, mass):
    """Short-range accelerations summed directly over every particle and
    periodic image within the pair cutoff, in 64 bits: sinks a block of the
    x order at a time against the sources within the cutoff along x."""
    src, _ = _ghosted(pos, cfg.cutoff_radius)
    src = src[:, torch.argsort(src[0])].contiguous()
    order = torch.argsort(pos[0])
    sink = pos[:, order]
    out = torch.zeros_like(sink)
    reach = 2.0 * cfg.split_radius * cfg.x_cut * (1.0 + 1e-9)
    eps2 = cfg.eps ** 2
    block = 256
    first = torch.searchsorted(src[0], sink[0, ::block].contiguous() - reach).tolist()
    last = torch.searchsorted(src[0], sink[0, block - 1::block].contiguous() + reach).tolist() + [src.shape[1]]
    for b, i in enumerate(range(0, sink.shape[1], block)):
        t = sink[:, i:i + block]
        s = src[:, first[b]:last[b]]
        d = [s[a][None, :] - t[a][:, None] for a in range(3)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        at, js = torch.nonzero(r2 < reach * reach, as_tuple=True)
        r2 = r2[at, js]
        r2 = r2 + eps2 if cfg.soft_mode == W.SOFT_PLUMMER else r2.clamp_min(eps2)
        r = r2.sqrt()
        x = r * (0.5 / cfg.split_radius)
        f = (torch.erfc(x) + (2.0 / math.sqrt(math.pi)) * x * torch.exp(-x * x)) / (r2 * r)
        f = torch.where(x > cfg.x_cut, torch.zeros_like(f), f) * mass
        for a in range(3):
            out[a, i:i + block].index_add_(0, at, f * d[a][at, js])
    back = torch.empty_like(out)
    back[:, order] = out
    return back


def _pm_exact(case, seed):
    n, nlocal = case["mesh"], case["n"] ** 3
    pos = _particles(case["shape"], case["n"], seed)
    if case["ordered"]:
        pos = _cell_order(pos, n)
    tag = _pm_tag(case, nlocal)
    on = torch.ones(nlocal, dtype=torch.bool, device=pos.device) if tag is None else tag == 1
    p = pos[:, on]
    i = (p * n).long()
    w = (p - (i.double() + 0.5) / n) * n
    side = torch.where(w > 0, i + 1, i - 1)
    idx = [torch.remainder(i, n), torch.remainder(side, n)]
    wt = [1.0 - w.abs(), w.abs()]
    corners = []
    for q in itertools.product((0, 1), repeat=3):
        corners.append(((idx[q[0]][0] * n + idx[q[1]][1]) * n + idx[q[2]][2], wt[q[0]][0] * wt[q[1]][1] * wt[q[2]][2]))
    mesh = torch.zeros(n ** 3, dtype=torch.float64, device=pos.device)
    for at, v in corners:
        mesh.index_add_(0, at, v / nlocal)
    l = torch.arange(n, dtype=torch.float64, device=pos.device)
    l = torch.where(l > n // 2, l - n, l)
    lz = torch.arange(n // 2 + 1, dtype=torch.float64, device=pos.device)
    k2 = l[:, None, None] ** 2 + l[None, :, None] ** 2 + lz[None, None, :] ** 2
    ff = 1.0 / (torch.sinc(l / n)[:, None, None] * torch.sinc(l / n)[None, :, None] * torch.sinc(lz / n)[None, None, :])
    s2 = (2 * math.pi * 1.2 / n) ** 2
    green = torch.exp(-k2 * s2) / k2 * ff ** 4 / (math.pi * n ** 3) * float(n) ** 3
    green[0, 0, 0] = 0.0
    phi = torch.fft.irfftn(torch.fft.rfftn(mesh.reshape(n, n, n)) * green, s=(n, n, n), norm="forward")
    acc = torch.zeros_like(pos)
    for a in range(3):
        g = (4.0 / 3.0) * 0.5 * n * (phi.roll(-1, a) - phi.roll(1, a)) - (1.0 / 6.0) * 0.5 * n * (phi.roll(-2, a) - phi.roll(2, a))
        g = g.reshape(-1)
        acc[a, on] = sum(v * g[at] for at, v in corners)
    return acc
