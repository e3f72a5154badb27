"""What a program that uses this framework has it do, as cases to be timed.

Every case goes through the package's public entry points: a device-resident `Simulation` that steps
and hands its state back, `step_host` for a program that owns positions and momenta itself (the
drop-in for the reference's step), pure PM runs, the learned short-range force, the `Ensemble`, the
reference's single functions called on host arrays, and the net alone (inference and training).

Particles are a lattice displaced by a Gaussian field of a CDM-like spectrum (one unit of length per
mean spacing, the resolution of every configuration of this repository); late states also hold half
of their particles in haloes of a power-law mass function, with isothermal profiles and virial
velocities, which is what the step meets at z = 0. Passes advance the simulations in steps of 0.2 % in
the scale factor, so that the state a pass meets stays the one that was prepared.

`exact` restates the paths in 64 bits with plain torch: CIC, FFT Poisson solve, octree walk, KDK
step and the convolutional net with its gradient and Adam step.
"""
import importlib
import math
from pathlib import Path

import numpy as np
import torch

cpm = importlib.import_module("cosmological-particle-simulation_b200")

ROOT = Path(__file__).resolve().parents[1]
NET_WEIGHTS = ROOT / "cosmological-particle-simulation_b200" / "weights" / "short_range_net.npz"
OMEGA_M, OMEGA_L, H0 = 0.3, 0.7, 70.0
THETA, SOFTENING = 0.5, 1.0 / 30.0
A_EARLY, A_LATE, STEP = 0.05, 0.5, 1.002
MESHES = (32, 48, 64, 80, 96, 128, 160, 192, 256, 320, 384, 512)
NET_IN_SCALE, NET_LR = 1.0 / 16.0, 2e-3


def listed():
    return [
        # The reference's CPU-runnable box: interactive use, where launches and latency count.
        dict(name="box-32", kind="resident", n_side=32, mesh=64, late=False, flags=0, steps=4),
        # A particle count that fills no tile and a mesh that is no power of two, in a clustered state.
        dict(name="odd-45-late", kind="resident", n_side=45, mesh=80, late=True, flags=0, steps=4),
        # Precision mode: fixed-point positions and quadrupole moments.
        dict(name="precision-64", kind="resident", n_side=64, mesh=128, late=False, flags=0x1 | 0x10, steps=4),
        # A production box stepped by a program that owns the state, early and late in its run.
        dict(name="host-128", kind="host", n_side=128, mesh=256, late=False, tree=True, learned=False),
        dict(name="host-128-late", kind="host", n_side=128, mesh=256, late=True, tree=True, learned=False),
        # The headline box.
        dict(name="host-256", kind="host", n_side=256, mesh=512, late=False, tree=True, learned=False),
        # Pure PM (no short-range force).
        dict(name="pm-192", kind="host", n_side=192, mesh=384, late=False, tree=False, learned=False),
        # The learned short-range force for the underdense particles.
        dict(name="learned-128", kind="host", n_side=128, mesh=256, late=True, tree=True, learned=True),
        # Realisations of two sizes stepped together.
        dict(name="ensemble", kind="ensemble", n_side=64, mesh=128, boxes=4, n_side2=96, mesh2=192, boxes2=2, steps=4),
        # The reference's functions one by one on host arrays: density, PM force, tree force.
        dict(name="functions-50", kind="functions", n_side=50, mesh=96, late=True),
        # The net alone on a mesh: inference at the training resolution, and one training step.
        dict(name="net-forward-256", kind="net_forward", mesh=256),
        dict(name="net-train-128", kind="net_train", n_side=64, mesh=128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mesh_for(rng, n_side, tree=True):
    """A compiled mesh length: about two cells per mean spacing with the tree, one or two without."""
    fit = [m for m in MESHES if (1.6 if tree else 1.0) * n_side <= m <= 2.4 * n_side]
    return rng.choice(fit)


def draw(rng):
    kind = rng.choice(("resident", "resident", "host", "host", "ensemble", "functions", "net_forward", "net_train"))
    if kind == "resident":
        n = _log_int(rng, 16, 96)
        return dict(kind=kind, n_side=n, mesh=_mesh_for(rng, n), late=rng.random() < 0.5,
                    flags=rng.choice((0, 0, 0, 0x1, 0x2, 0x1 | 0x10)), steps=rng.randint(2, 6))
    if kind == "host":
        n = _log_int(rng, 24, 160)
        tree = rng.random() < 0.7
        mesh = _mesh_for(rng, n, tree)
        learned = tree and n >= 48 and mesh % 16 == 0 and rng.random() < 0.25
        return dict(kind=kind, n_side=n, mesh=mesh, late=rng.random() < 0.5, tree=tree, learned=learned)
    if kind == "ensemble":
        n, n2 = rng.choice((32, 48, 64, 80)), rng.choice((32, 64, 80, 96))
        return dict(kind=kind, n_side=n, mesh=_mesh_for(rng, n), boxes=rng.randint(1, 8), n_side2=n2,
                    mesh2=_mesh_for(rng, n2), boxes2=rng.randint(1, 3), steps=rng.randint(2, 5))
    if kind == "functions":
        n = _log_int(rng, 17, 64)
        return dict(kind=kind, n_side=n, mesh=_mesh_for(rng, n), late=rng.random() < 0.5)
    mesh = 16 * _log_int(rng, 2, 20 if kind == "net_forward" else 10)
    return dict(kind=kind, mesh=mesh) if kind == "net_forward" else dict(kind=kind, n_side=mesh // 2 + rng.randint(-5, 5), mesh=mesh)


# ------------------------------------------------------------------------------------------ inputs


def _cosmo():
    return cpm.Cosmology(0.0, OMEGA_M, OMEGA_L, H0)


def _hubble(a):
    return math.sqrt(OMEGA_M / a ** 3 + OMEGA_L)


def _field_k(n, gen):
    """White noise with a CDM-like spectrum, and the wavenumbers, on an n^3 lattice of unit spacing."""
    w = torch.fft.rfftn(torch.randn(n, n, n, generator=gen, device="cuda", dtype=torch.float64))
    kf = 2 * math.pi * torch.fft.fftfreq(n, device="cuda", dtype=torch.float64)
    kr = 2 * math.pi * torch.fft.rfftfreq(n, device="cuda", dtype=torch.float64)
    k = (kf[:, None, None], kf[None, :, None], kr[None, None, :])
    k2 = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    k2[0, 0, 0] = 1.0
    kk = k2.sqrt()
    w *= (kk ** 0.96 / (1.0 + 12.0 * kk + 20.0 * kk ** 1.5 + 30.0 * kk ** 2) ** 2).sqrt()
    w[0, 0, 0] = 0.0
    return w, k, k2


def _particles(n, late, seed):
    """Positions and momenta (float32, CUDA, (n^3, 3)) in a box of side n at A_EARLY or A_LATE."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 2 + 1)
    a = A_LATE if late else A_EARLY
    w, k, k2 = _field_k(n, gen)
    disp = torch.stack([torch.fft.irfftn(1j * kc * w / k2, s=(n, n, n)).reshape(-1) for kc in k], 1)
    disp *= 4.0 * a / disp.square().mean().sqrt()  # a few spacings at a = 1
    q = torch.arange(n, device="cuda", dtype=torch.float64)
    x = torch.stack(torch.meshgrid(q, q, q, indexing="ij"), -1).reshape(-1, 3) + 0.5 + disp
    u = disp.clone()  # peculiar velocity over a H, in units of length
    if late:
        total = n ** 3
        hi = float(min(3000, max(40, total // 100)))
        m = (torch.rand(total // 20, generator=gen, device="cuda", dtype=torch.float64)
             * (hi ** -0.9 - 20.0 ** -0.9) + 20.0 ** -0.9) ** (-1 / 0.9)  # dn/dm ~ m^-1.9
        m = m.floor().long()
        m = m[m.cumsum(0) <= total // 2]
        halo = torch.repeat_interleave(torch.arange(len(m), device="cuda"), m)
        member = torch.randperm(total, generator=gen, device="cuda")[:len(halo)]
        head = member[torch.cat([m.new_zeros(1), m.cumsum(0)[:-1]])[halo]]
        r200 = (3.0 * m.double() / (4 * math.pi * 200.0)) ** (1 / 3)
        d = torch.randn(len(halo), 3, generator=gen, device="cuda", dtype=torch.float64)
        d *= (r200[halo] * (0.002 + torch.rand(len(halo), generator=gen, device="cuda", dtype=torch.float64))
              / d.norm(dim=1))[:, None]
        x[member] = x[head] + d
        u[member] = u[head] + 4.0 * r200[halo][:, None] * torch.randn(len(halo), 3, generator=gen, device="cuda", dtype=torch.float64)
    x = torch.remainder(x, float(n)).float()
    x[x >= n] = 0.0
    p = (a * a * _hubble(a) * u).float()
    # the caller's order is no spatial order once a run has mixed its particles
    perm = torch.randperm(n ** 3, generator=gen, device="cuda") if late else slice(None)
    return x[perm].contiguous(), p[perm].contiguous(), a


def _split(case):
    return cpm.ForceSplit.with_(float(case["n_side"]), case["mesh"], case["n_side"], SOFTENING, THETA)


def _net_sample(case, seed):
    """delta on the mesh, positions, a short-range force to learn, weights, loss norm (CUDA, f32)."""
    n, mesh = case["n_side"], case["mesh"]
    x, _, _ = _particles(n, True, seed)
    delta = _density64(x.double(), mesh, float(n))
    k = _mesh_k(mesh, 1.0)
    k2 = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    high = torch.fft.rfftn(delta) * -torch.expm1(-k2 * 1.25 ** 2) / torch.where(k2 == 0, torch.ones_like(k2), k2)
    force = [torch.fft.irfftn(-1j * kc * high, s=(mesh,) * 3) for kc in k]
    target = torch.stack([_gather64(f, x.double(), float(n)) for f in force], 1).float()
    weight = (_gather64(delta, x.double(), float(n)) < 1.0).float()
    norm = float((target.double() ** 2 * weight[:, None].double()).sum())
    return delta.float().contiguous(), x, target.contiguous(), weight.contiguous(), 1.0 / max(norm, 1e-30)


def _train_weights(seed):
    rng = np.random.default_rng(seed)
    w = np.zeros((3, 27, 16, 16), np.float32)
    w[0, :, :, 0] = rng.standard_normal((27, 16)) * math.sqrt(2.0 / 27.0)
    w[1] = rng.standard_normal((27, 16, 16)) * math.sqrt(2.0 / (27.0 * 16.0))
    w[2, :, :3, :] = rng.standard_normal((27, 3, 16)) * 0.1 * math.sqrt(2.0 / (27.0 * 16.0))
    return w


def _net_delta(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 2 + 1)
    n = case["mesh"]
    w, _, _ = _field_k(n, gen)
    g = torch.fft.irfftn(w, s=(n, n, n))
    return (torch.exp(1.2 * g / g.std() - 0.72) - 1.0).float().reshape(-1).contiguous()  # lognormal, mean 0


def prepare(case, seed):
    kind = case["kind"]
    if kind == "resident":
        x, p, a = _particles(case["n_side"], case["late"], seed)
        sim = cpm.Simulation(_cosmo(), float(case["n_side"]), case["mesh"], x.cpu().numpy(), p.cpu().numpy(), a,
                             _split(case), flags=case["flags"])
        return dict(case=case, sim=sim, a=a)
    if kind == "host":
        x, p, a = _particles(case["n_side"], case["late"], seed)
        hx, hp = (torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t) for t in (x, p))
        del x, p
        torch.cuda.empty_cache()
        sim = cpm.Simulation(_cosmo(), float(case["n_side"]), case["mesh"], hx.numpy(), hp.numpy(), a,
                             _split(case) if case["tree"] else None)
        if case["learned"]:
            with np.load(NET_WEIGHTS) as f:
                net = cpm.ShortRangeNet(case["mesh"], f["weights"])
                sim.set_learned(net, float(f["threshold"]), float(f["in_scale"]))
        return dict(case=case, sim=sim, a=a, hx=hx, hp=hp, x=hx.numpy(), p=hp.numpy())
    if kind == "ensemble":
        box = 64.0
        classes = [(case["n_side" + q], case["mesh" + q], case["boxes" + q], (seed * 64 + 17 * len(q)) % (1 << 40),
                    cpm.ForceSplit.with_(box, case["mesh" + q], case["n_side" + q], SOFTENING, THETA)) for q in ("", "2")]
        return dict(case=case, a=A_EARLY, ens=cpm.Ensemble(_cosmo(), box, 0.96, 0.8, A_EARLY, classes))
    if kind == "functions":
        x, _, a = _particles(case["n_side"], case["late"], seed)
        return dict(case=case, x=x.cpu().numpy(), a=a, cosmo=_cosmo(), split=_split(case),
                    solver=cpm.PoissonSolver(case["mesh"], float(case["n_side"])))
    if kind == "net_forward":
        with np.load(NET_WEIGHTS) as f:
            net = cpm.ShortRangeNet(case["mesh"], f["weights"])
        return dict(case=case, net=net, delta=_net_delta(case, seed))
    delta, x, target, weight, inv_norm = _net_sample(case, seed)
    return dict(case=case, net=cpm.ShortRangeNet(case["mesh"], _train_weights(seed)), delta=delta, x=x, target=target,
                weight=weight, inv_norm=inv_norm)


# -------------------------------------------------------------------------------------------- passes


def _next_a(a):
    return float(np.float32(a * STEP))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("resident", "ensemble"):
        target = state["sim"] if kind == "resident" else state["ens"]
        for _ in range(case["steps"]):
            state["a"] = _next_a(state["a"])
            target.step_to(state["a"])
        if kind == "resident":
            return target.state()
        return [target.state(c, b) for c, boxes in enumerate((case["boxes"], case["boxes2"])) for b in range(boxes)]
    if kind == "host":
        state["a"] = _next_a(state["a"])
        state["sim"].step_host(state["a"], state["x"], state["p"])
        return [state["x"], state["p"]]
    if kind == "functions":
        x, box = state["x"], float(case["n_side"])
        delta = cpm.api.density_contrast(x, case["mesh"], box)
        g = state["solver"].acceleration(delta, state["cosmo"], state["a"], state["split"].r_split)
        pm = cpm.interpolate3(*g, x)
        sr = cpm.tree_accelerations(x, box, state["split"], _coupling(case, state["a"]))
        return dict(delta=delta.cells, gx=g[0].cells, gy=g[1].cells, gz=g[2].cells, pm=pm, short_range=sr)
    if kind == "net_forward":
        return state["net"].forward(state["delta"], in_scale=NET_IN_SCALE)
    net = state["net"]
    loss = net.train_step(state["delta"], state["x"], state["target"], state["weight"], float(case["n_side"]),
                          state["inv_norm"], NET_LR, in_scale=NET_IN_SCALE)
    return dict(loss=loss, weights=net.weights, grads=net.grads())


def work(case):
    """Bytes that have to enter and leave, and the arithmetic of the pairs, transforms and convolutions."""
    kind = case["kind"]

    def step(n, m, tree, late):
        # positions, momenta and accelerations in and out; four real transforms; pairs within r_cut
        pairs = (4.0 / 3.0 * math.pi * (5.625 * n / m) ** 3 + (250.0 if late else 0.0)) if tree else 0.0
        return 72.0 * n ** 3, 4 * 2.5 * m ** 3 * math.log2(m ** 3) + n ** 3 * (pairs * 40.0 + 100.0)

    def net(m, passes):
        return passes * 2.0 * 27.0 * (16 + 256 + 48) * m ** 3

    if kind in ("resident", "ensemble"):
        parts = [(case["n_side"], case["mesh"], case.get("boxes", 1))]
        if kind == "ensemble":
            parts.append((case["n_side2"], case["mesh2"], case["boxes2"]))
        b = f = 0.0
        for n, m, boxes in parts:
            bytes_, flops = step(n, m, True, case.get("late", False))
            b += boxes * (bytes_ * case["steps"] + 36.0 * n ** 3)
            f += boxes * flops * case["steps"]
        return dict(bytes=b, flops=f)
    if kind == "host":
        b, f = step(case["n_side"], case["mesh"], case["tree"], case["late"])
        return dict(bytes=b, flops=f + (net(case["mesh"], 1) if case["learned"] else 0.0))
    if kind == "functions":
        n, m = case["n_side"], case["mesh"]
        return dict(bytes=24.0 * n ** 3 + 12.0 * n ** 3 + 20.0 * m ** 3, flops=step(n, m, True, case["late"])[1])
    m = case["mesh"]
    if kind == "net_forward":
        return dict(bytes=20.0 * m ** 3, flops=net(m, 1))
    return dict(bytes=4.0 * m ** 3 + 28.0 * case["n_side"] ** 3, flops=net(m, 3))


# ------------------------------------------------------------------------------- the paths in 64 bits


def _mesh_k(n, box):
    kf = torch.fft.fftfreq(n, device="cuda", dtype=torch.float64) * n
    kr = torch.fft.rfftfreq(n, device="cuda", dtype=torch.float64) * n
    kf[n // 2] = 0.0  # the Nyquist index carries no gradient
    kr[n // 2] = 0.0
    w = 2 * math.pi / box
    return w * kf[:, None, None], w * kf[None, :, None], w * kr[None, None, :]


def _stencil64(x, n, box):
    s = x / (box / n) - 0.5
    base = s.floor()
    f = s - base
    base = base.long()
    for c in range(8):
        d = torch.tensor([c >> 2 & 1, c >> 1 & 1, c & 1], device=x.device)
        i = torch.remainder(base + d, n)
        yield (i[:, 0] * n + i[:, 1]) * n + i[:, 2], torch.where(d.bool(), f, 1.0 - f).prod(1)


def _density64(x, n, box):
    rho = torch.zeros(n ** 3, device="cuda", dtype=torch.float64)
    for i, w in _stencil64(x, n, box):
        rho.index_add_(0, i, w)
    return (rho * (n ** 3 / len(x)) - 1.0).view(n, n, n)


def _gather64(field, x, box):
    return sum(field.reshape(-1)[i] * w for i, w in _stencil64(x, field.shape[0], box))


def _poisson64(delta, box, a, r_split, deconvolve=False):
    n = delta.shape[0]
    k = _mesh_k(n, box)
    k2 = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    zero = k2 == 0
    k2 = torch.where(zero, torch.ones_like(k2), k2)
    phi = torch.fft.rfftn(delta) * (-1.5 * OMEGA_M / a) / k2 * torch.exp(-k2 * r_split ** 2)
    phi[zero] = 0.0
    if deconvolve:
        win = torch.sinc(torch.fft.fftfreq(n, device="cuda", dtype=torch.float64)) ** -4
        phi *= win[:, None, None] * win[None, :, None] * win[None, None, : n // 2 + 1]
    return [torch.fft.irfftn(-1j * kc * phi, s=(n, n, n)) for kc in k]


def _coupling(case, a):
    n = case["n_side"]
    return 1.5 * OMEGA_M * float(n) ** 3 / (4 * math.pi * a * n ** 3)


def _tree64(x, box, r_split, r_cut, eps, k):
    """The octree of at most 8 particles a leaf and its walk (prune, direct sum where octant 0 is empty,
    opening angle), all particles of a chunk level by level."""
    cell = (x * (2.0 ** 21 / box)).floor().long()
    key = torch.zeros(len(x), dtype=torch.long, device=x.device)
    for b in range(20, -1, -1):
        o = (cell >> b) & 1
        key = (key << 3) | o[:, 0] | (o[:, 1] << 1) | (o[:, 2] << 2)
    key, order = key.sort()
    xs = x[order]
    prefix = torch.cat([xs.new_zeros(1, 3), xs.cumsum(0)])
    levels = []
    start, end = torch.tensor([0], device=x.device), torch.tensor([len(x)], device=x.device)
    centre = torch.full((1, 3), box / 2, dtype=torch.float64, device=x.device)
    for depth in range(22):
        half = box / 2 / 2 ** depth
        split = (end - start > 8) & (depth < 21)
        child = torch.full((len(start), 8), -1, dtype=torch.long, device=x.device)
        com = (prefix[end] - prefix[start]) / (end - start)[:, None]
        nxt = None
        if split.any():
            sh = 3 * (20 - depth)
            pre = (key[start[split]] >> (sh + 3)) << 3
            edge = torch.searchsorted(key, (pre[:, None] + torch.arange(8, device=x.device)) << sh)
            edge = torch.cat([edge, end[split][:, None]], 1)
            lo, hi = edge[:, :8], edge[:, 1:]
            full = hi > lo
            idx = torch.full_like(lo, -1)
            idx[full] = torch.arange(int(full.sum()), device=x.device)
            child[split] = idx
            o = torch.arange(8, device=x.device)
            off = torch.stack([(o & 1), (o >> 1 & 1), (o >> 2 & 1)], 1) * half - half / 2
            nxt = (lo[full], hi[full], (centre[split][:, None, :] + off)[full])
        levels.append((start, end, centre, half, com, child))
        if nxt is None:
            break
        start, end, centre = nxt

    def image(d):
        return d - box * torch.round(d / box)

    def factor(r2, m):
        r = r2.sqrt()
        u = r / (2 * r_split)
        s = torch.special.erfc(u) + 2 / math.sqrt(math.pi) * u * torch.exp(-u * u)
        return -k * m * s / (r2 + eps * eps) ** 1.5

    acc = torch.zeros_like(xs)
    for c0 in range(0, len(xs), 16384):
        who = torch.arange(c0, min(c0 + 16384, len(xs)), device=x.device)
        node = torch.zeros_like(who)
        for start, end, centre, half, com, child in levels:
            d = image(centre[node] - xs[who])
            near = (d * d).sum(1) <= (r_cut + math.sqrt(3.0) * half) ** 2
            who, node = who[near], node[near]
            direct = child[node, 0] < 0
            w, nd = who[direct], node[direct]
            count = end[nd] - start[nd]
            w = torch.repeat_interleave(w, count)
            first = torch.repeat_interleave(start[nd] - (count.cumsum(0) - count), count)
            j = first + torch.arange(len(first), device=x.device)
            d = image(xs[w] - xs[j])
            r2 = (d * d).sum(1)
            keep = (r2 <= r_cut * r_cut) & (j != w)
            acc.index_add_(0, w[keep], d[keep] * factor(r2[keep], 1.0)[:, None])
            who, node = who[~direct], node[~direct]
            d = image(com[node] - xs[who])
            r2 = (d * d).sum(1)
            far = 2 * half < THETA * r2.sqrt()
            m = (end - start)[node[far]].double()
            acc.index_add_(0, who[far], -d[far] * factor(r2[far], m)[:, None])
            who, node = who[~far], child[node[~far]]
            who = who[:, None].expand(-1, 8)[node >= 0]
            node = node[node >= 0]
            if not len(who):
                break
    out = torch.empty_like(acc)
    out[order] = acc
    return out


def _accelerations64(x, case, a, tree, deconvolve):
    n, mesh = case["n_side"], case["mesh"]
    box = float(n)
    r_split = 1.25 * box / mesh
    g = _poisson64(_density64(x, mesh, box), box, a, r_split if tree else 0.0, deconvolve)
    acc = torch.stack([_gather64(f, x, box) for f in g], 1)
    if tree:
        acc += _tree64(x, box, r_split, 4.5 * r_split, SOFTENING, _coupling(case, a))
    return acc


def _simpson(lo, hi, f):
    t = np.linspace(lo, hi, 257)
    w = np.where(np.arange(257) % 2 == 1, 4.0, 2.0)
    w[0] = w[-1] = 1.0
    return float((w * f(t)).sum() * (hi - lo) / 256 / 3)


def _steps64(case, seed, steps, tree, deconvolve):
    x, p, a = _particles(case["n_side"], case["late"], seed)
    x, p, box = x.double(), p.double(), float(case["n_side"])
    hub = lambda t: np.sqrt(OMEGA_M / t ** 3 + OMEGA_L)  # noqa: E731
    kick = lambda lo, hi: _simpson(lo, hi, lambda t: 1.0 / (t * hub(t)))  # noqa: E731
    acc = _accelerations64(x, case, a, tree, deconvolve)
    for _ in range(steps):
        a1 = _next_a(a)
        half = kick(a, a1) / 2  # each half-kick takes half of the kick integral
        p += half * acc
        x = torch.remainder(x + p * _simpson(a, a1, lambda t: 1.0 / (t ** 3 * hub(t))), box)
        acc = _accelerations64(x, case, a1, tree, deconvolve)
        p += half * acc
        a = a1
    return x.cpu().numpy(), p.cpu().numpy(), acc.cpu().numpy(), a


def _net64(delta, w, mesh):
    """The three periodic convolutions in 64 bits; w is (3, 27, 16, 16), field (3, n, n, n)."""
    pad = torch.nn.functional.pad
    v = delta.double().view(1, 1, mesh, mesh, mesh)
    for layer, (cin, cout) in enumerate(((1, 16), (16, 16), (16, 3))):
        kern = w[layer, :, :cout, :cin].permute(1, 2, 0).reshape(cout, cin, 3, 3, 3)
        v = pad(v, (1,) * 6, mode="circular")
        v = sum(torch.einsum("oi,ixyz->oxyz", kern[:, :, i, j, l], v[0, :, i:i + mesh, j:j + mesh, l:l + mesh])
                for i in range(3) for j in range(3) for l in range(3))[None]
        if layer < 2:
            v = torch.nn.functional.leaky_relu(v, 0.125)
    return v[0]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("resident", "host"):
        tree = case.get("tree", True)
        flags = case.get("flags", 0)
        # quadrupoles and the learned force have no 64-bit form here; larger trees take too long
        if flags & 0x10 or case.get("learned") or case["n_side"] > (70 if tree else 200):
            return None
        steps = case.get("steps", 1)
        x, p, acc, a = _steps64(case, seed, steps, tree, bool(flags & 0x2))
        return dict(x=x, p=p, acc=acc, a=a) if kind == "resident" else [x, p]
    if kind == "ensemble":
        return None  # its initial conditions are the library's own random numbers
    if kind == "functions":
        x, _, a = _particles(case["n_side"], case["late"], seed)
        x, box, mesh = x.double(), float(case["n_side"]), case["mesh"]
        r_split = 1.25 * box / mesh
        delta = _density64(x, mesh, box)
        g = _poisson64(delta, box, a, r_split)
        pm = torch.stack([_gather64(f, x, box) for f in g], 1)
        sr = _tree64(x, box, r_split, 4.5 * r_split, SOFTENING, _coupling(case, a))
        flat = lambda t: t.reshape(-1).cpu().numpy()  # noqa: E731
        return dict(delta=flat(delta), gx=flat(g[0]), gy=flat(g[1]), gz=flat(g[2]), pm=pm.cpu().numpy(),
                    short_range=sr.cpu().numpy())
    if case["mesh"] > 128:
        return None
    mesh = case["mesh"]
    if kind == "net_forward":
        with np.load(NET_WEIGHTS) as f:
            w = torch.from_numpy(f["weights"]).double().cuda()
        with torch.no_grad():
            field = _net64(NET_IN_SCALE * _net_delta(case, seed), w, mesh)
        out = torch.zeros(mesh ** 3, 4, dtype=torch.float64, device="cuda")
        out[:, :3] = field.reshape(3, -1).T
        return out
    delta, x, target, weight, inv_norm = _net_sample(case, seed)
    w = torch.from_numpy(_train_weights(seed)).double().cuda().requires_grad_(True)
    field = _net64(NET_IN_SCALE * delta, w, mesh)
    at = torch.stack([_gather64(f, x.double(), float(case["n_side"])) for f in field], 1)
    loss = inv_norm * (weight.double()[:, None] * (at - target.double()) ** 2).sum()
    g, = torch.autograd.grad(loss, w)
    with torch.no_grad():
        new = w - NET_LR * g / (g.abs() + 1e-8)  # Adam's first step
    return dict(loss=float(loss.detach()), weights=new.cpu().numpy(), grads=g.cpu().numpy())
