"""The engine's work as its users have it done, through woo_gb300.abi.Handle: what is timed, on which inputs.

A case is one scene kind at one size.  A pass is a run of `steps` steps of Leapfrog, collider and ContactLoop
through wdem_step, followed by reading the kinematic state back to pinned host memory (what a script between two
of its own actions does); the kinds differ in the scene and in what else a pass does:

* bed      a settled dense bed of spheres in a walled box, the long end of every pouring job
* cloud    a cloud falling at speed; the caller owns the state and writes it in before each run, as the plug-in
           inside Woo's loop and any restart from a stored state do
* peri     a dense packing in a periodic cell under simple shear (homoDeform gradV2)
* batch    many independent oedometric scenes in one handle, each with its own material and dt
* ell      a bed of ellipsoids (Perram-Wertheim geometry, Brent or Newton with the previous step's maximiser)
* hopper   a bed whose outlet takes spheres out and whose inlet puts them back in before each run
* net      gradient (training) or prediction of the warm-start network on a batch of solver records

Inputs come from the seed alone.  Packings are made by relaxing the overlaps of a jittered lattice, with ids in
the order of the radii (as wdem_make_cloud gives them), so that neighbours in space are not neighbours in memory.
"""
import ctypes
import math

import numpy as np
import torch

LOCAL = "cuda" if torch.cuda.is_available() else "cpu"
BLOCKED = 63            # all degrees of freedom of a wall
MOVABLE, BOUNDARY = 0b0101, 0b0011


def listed():
    return [
        # one step per call with the state in and out: a small scene driven step by step from a host program
        dict(name="plugin_300", kind="cloud", n=300, law="frict", arith="exact", steps=1, speed=1.0),
        # ten thousand equal spheres falling fast: a collider rebuild every few steps
        dict(name="cloud_15k", kind="cloud", n=15000, law="frict", arith="exact", steps=40, speed=1.5),
        # a million polydisperse Hertz spheres falling: the first half of a large pouring job
        dict(name="cloud_1m", kind="cloud", n=1000000, law="hertz", arith="fma", steps=40, speed=1.0),
        # the reference's arithmetic, bit for bit, on a bed of ten thousand spheres
        dict(name="bed_10k", kind="bed", n=10000, law="frict", arith="exact", steps=50, energy=0),
        # the same with the energy balance tracked, as runs that check it do
        dict(name="bed_30k_energy", kind="bed", n=30011, law="frict", arith="fma", steps=10, energy=1),
        # the settled end of the million-sphere job in double-word arithmetic, and a tenth of it in FP64
        dict(name="bed_100k", kind="bed", n=100003, law="hertz", arith="fma", steps=20, energy=0),
        dict(name="bed_1m", kind="bed", n=1000000, law="hertz", arith="dw", steps=10, energy=0),
        # simple shear of a dense periodic packing
        dict(name="peri_400k", kind="peri", n=400000, law="frict", arith="fma", steps=10, rate=5.0),
        # a parametric study of oedometric tests, all scenes in one handle
        dict(name="batch_96", kind="batch", n=96, law="frict", arith="fma", steps=12),
        # ellipsoids, the fastest solver setting
        dict(name="ell_40k", kind="ell", n=40000, law="frict", arith="fma", steps=10, solver="newton"),
        # particles taken out and put back in between runs
        dict(name="hopper_120k", kind="hopper", n=120000, law="frict", arith="fma", steps=10, moved=500),
        # training of the warm-start network
        dict(name="net_grad_64k", kind="net", n=65536, what="grad"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cloud", "bed", "bed", "peri", "batch", "ell", "hopper", "net"])
    law, arith = rng.choice(["frict", "hertz"]), rng.choice(["exact", "fma", "dw"])
    if kind == "cloud":
        n = _log(rng, 100, 900000)
        return dict(kind=kind, n=n, law=law, arith=rng.choice(["exact", "fma"]), steps=rng.randint(1, 40),
                    speed=rng.choice([0.5, 1.0, 1.5]))
    if kind == "bed":
        n = _log(rng, 200, 700000)
        energy = 1 if n < 50000 and rng.random() < 0.3 else 0
        return dict(kind=kind, n=n, law=law, arith=arith, steps=rng.randint(5, 20 if n > 20000 else 60), energy=energy)
    if kind == "peri":
        return dict(kind=kind, n=_log(rng, 1500, 350000), law=law, arith=arith, steps=rng.randint(3, 12),
                    rate=rng.choice([1.0, 5.0, 10.0]))
    if kind == "batch":
        return dict(kind=kind, n=_log(rng, 2, 96), law="frict", arith=rng.choice(["exact", "fma"]), steps=rng.randint(4, 12))
    if kind == "ell":
        solver = rng.choice(["newton", "brent"])
        return dict(kind=kind, n=_log(rng, 300, 40000 if solver == "newton" else 15000), law="frict",
                    arith=rng.choice(["exact", "fma"]), steps=rng.randint(3, 12), solver=solver)
    if kind == "hopper":
        n = _log(rng, 2000, 200000)
        return dict(kind=kind, n=n, law=law, arith=rng.choice(["exact", "fma"]), steps=rng.randint(3, 15),
                    moved=max(1, n // rng.choice([20, 100, 500])))
    return dict(kind=kind, n=_log(rng, 200, 300000), what=rng.choice(["grad", "predict"]))


# ------------------------------------------------------------------------------------------------ packings
def _gen(seed):
    g = torch.Generator(device=LOCAL)
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _uniform(g, shape, lo, hi):
    return torch.rand(shape, generator=g, device=LOCAL, dtype=torch.float64) * (hi - lo) + lo


_HALF = [(dz, dy, dx) for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1) if (dz, dy, dx) > (0, 0, 0)]


def _packing(g, radii, phi, periodic, rounds):
    """Centres (k, 3), radii and box lengths of about the given radii at solid fraction phi: a jittered simple cubic
    lattice whose overlaps between lattice neighbours (and with the box) are pushed apart `rounds` times."""
    k = radii.numel()
    a = float(((radii ** 3).mean() * (4.0 / 3.0 * math.pi) / phi) ** (1.0 / 3.0))
    nx = max(1, int(round(k ** (1.0 / 3.0))))
    nz = -(-k // (nx * nx))
    shape = (nz, nx, nx)
    r = torch.zeros(nz * nx * nx, device=LOCAL, dtype=torch.float64)
    r[:k] = radii
    r = r.reshape(shape)
    here = r > 0
    zz, yy, xx = torch.meshgrid(*[torch.arange(v, device=LOCAL, dtype=torch.float64) for v in shape], indexing="ij")
    p = (torch.stack([xx, yy, zz], dim=-1) + 0.5 + _uniform(g, shape + (3,), -0.15, 0.15)) * a
    box = torch.tensor([nx * a, nx * a, nz * a], device=LOCAL, dtype=torch.float64)
    for _ in range(rounds):
        move = torch.zeros_like(p)
        for o in _HALF:
            sh = tuple(-v for v in o)
            d = torch.roll(p, sh, (0, 1, 2)) - p
            ok = here & torch.roll(here, sh, (0, 1, 2))
            if periodic:
                d = d - box * torch.round(d / box)
            else:
                for ax, v in enumerate(o):
                    if v:
                        edge = torch.arange(shape[ax], device=LOCAL) + v
                        inside = (edge >= 0) & (edge < shape[ax])
                        ok = ok & inside.reshape([-1 if q == ax else 1 for q in range(3)])
            dist = d.square().sum(-1).sqrt()
            over = (r + torch.roll(r, sh, (0, 1, 2)) - dist).clamp(min=0) * ok
            push = d * (0.22 * over / dist.clamp(min=1e-12)).unsqueeze(-1)
            move = move - push + torch.roll(push, o, (0, 1, 2))
        p = p + move
        if not periodic:
            rr = r.unsqueeze(-1)
            p = torch.maximum(torch.minimum(p, box - 0.9999 * rr), 0.9999 * rr)
    p = p.reshape(-1, 3)[:k]
    return p, _shrink(p, radii, box, periodic), box


def _shrink(x, r, box, periodic):
    """The radii with every overlap above 1.2 % of the mean radius taken off the two spheres in equal parts."""
    i, j, shift = _close_pairs(x, r, box if periodic else None)
    d = x[j] - x[i]
    if periodic:
        d = d + shift * box
    over = r[i] + r[j] - d.square().sum(1).sqrt()
    cut = 0.5 * (over - 0.006 * (r[i] + r[j])).clamp(min=0)
    return r - torch.zeros_like(r).scatter_reduce(0, torch.cat([i, j]), torch.cat([cut, cut]), "amax")


def _order(g, radii):
    """Ids by falling radius, ties in random order."""
    shuffled = torch.randperm(radii.numel(), generator=g, device=LOCAL)
    return shuffled[torch.argsort(radii[shuffled], descending=True, stable=True)]


def _box_walls(lo, hi, mat, scene=0):
    return [(ax, sense, end[ax], mat, scene, 0.0) for ax in range(3) for sense, end in ((1, lo), (-1, hi))]


FRICT = dict(density=3000.0, young=1e7, ktDivKn=0.2, tanPhi=0.5, surfEnergy=0.0)
HERTZ = [dict(density=1000.0, young=5e7, ktDivKn=0.2, tanPhi=t, surfEnergy=0.01) for t in (0.3, 0.6)]


def _axes():
    """Semi-axes of the ellipsoids over the largest one."""
    return torch.tensor([1.0, 0.7, 0.5], device=LOCAL, dtype=torch.float64)


def _scene(case, seed):
    """The scene in plain arrays: pos, vel, angVel, ori, r (bounding radius), semi, mass, inertia, mat, scene of the
    bodies, walls (axis, sense, position, material, scene, velocity along the axis), materials and the parameters."""
    g = _gen(seed)
    kind, n = case["kind"], int(case["n"])
    law = case["law"]
    S = dict(law=law, gravity=(0.0, 0.0, -9.81), damping=0.2, cell=None, semi=None, matDt=None)
    mats = [dict(FRICT)] if law == "frict" else [dict(m) for m in HERTZ]
    scene = None
    if kind == "batch":
        # oedometric boxes cut out of one dense packing: only whole spheres, the top wall just above them
        tile_r = _uniform(g, (48000,), 1e-3, 3e-3)
        c, tile_r, box = _packing(g, tile_r, 0.52, False, 100)
        # counts spread evenly over the logarithm of 500 .. 20000, in an order of their own
        size = [int(round(500 * 40 ** (((7 * k + 3) % n + 0.5) / n))) for k in range(n)]
        young = torch.exp(_uniform(g, (n,), math.log(1e6), math.log(1e8))).tolist()
        tanphi = _uniform(g, (n,), 0.1, 0.8).tolist()
        corner = _uniform(g, (n, 3), 0, 1)
        mats, walls, parts, mat_dt, step_x = [], [], [], [], 1.3 * float(box.max())
        for k in range(n):
            scale = (1.3 * size[k] / 48000.0) ** (1.0 / 3.0)
            while True:
                edge = min(scale, 1.0) * box
                lo = corner[k] * (box - edge)
                inside = ((c - tile_r[:, None] >= lo) & (c + tile_r[:, None] <= lo + edge)).all(1).nonzero()[:, 0]
                if len(inside) >= size[k]:
                    break
                scale *= 1.04
            inside = inside[torch.argsort(c[inside, 2], stable=True)[:size[k]]]
            ck, rk = c[inside] - lo, tile_r[inside]
            ck[:, 0] += k * step_x
            top = float((ck[:, 2] + rk).max()) + 1e-4
            e = edge.tolist()
            x0 = k * step_x
            walls += _box_walls((x0, 0.0, 0.0), (x0 + e[0], e[1], top), 2 * k + 1, k)
            walls[-1] = walls[-1][:5] + (-0.05,)
            mats += [dict(FRICT, density=2600.0, young=young[k], tanPhi=tanphi[k]), dict(FRICT, density=2600.0, young=young[k], tanPhi=0.0)]
            mat_dt += [0.9 * float(rk.min()) / math.sqrt(young[k] / 2600.0)] * 2
            o = _order(g, rk)
            parts.append((ck[o], rk[o], torch.full((len(o),), k, device=LOCAL)))
        pos, r, scene = (torch.cat([p[q] for p in parts]) for q in range(3))
        mat = 2 * scene
        S.update(gravity=(0.0, 0.0, -10.0), damping=0.4, matDt=mat_dt, verletDist=1e-4, dt=min(mat_dt))
    else:
        if kind == "peri":
            r = torch.exp(torch.randn(n, generator=g, device=LOCAL, dtype=torch.float64) * 0.25 + math.log(1e-3)).clamp(0.5e-3, 2e-3)
            phi, rounds = 0.52, 100
            mats = [dict(m, young=1e8, density=1000.0) for m in mats]
        elif kind == "ell":
            r = _uniform(g, (n,), 3e-3, 6e-3)
            phi, rounds = 0.52, 100
            mats = [dict(FRICT, density=1000.0, young=1e7, tanPhi=0.4)]
        else:
            r = torch.full((n,), 5e-3, device=LOCAL, dtype=torch.float64) if law == "frict" else _uniform(g, (n,), 2e-3, 6e-3)
            phi, rounds = (0.3, 40) if kind == "cloud" else (0.52, 100)
        pos, r, box = _packing(g, r, phi, kind == "peri", rounds)
        if kind == "ell":
            # parallel ellipsoids: the packing of spheres stretched along the axes
            pos, box = pos * _axes(), box * _axes()
        if kind == "cloud":
            pos[:, 2] += 0.5 * float(box[2])  # above the floor of a box half as high again
            box[2] *= 1.5
        o = _order(g, r)
        pos, r = pos[o], r[o]
        mat = torch.arange(n, device=LOCAL) % len(mats)
        E = torch.tensor([m["young"] for m in mats], device=LOCAL, dtype=torch.float64)[mat]
        rho = torch.tensor([m["density"] for m in mats], device=LOCAL, dtype=torch.float64)[mat]
        walls = [] if kind == "peri" else _box_walls((0.0, 0.0, 0.0), box.tolist(), 0)
        rmin = float(r.min()) * (0.5 if kind == "ell" else 1.0)
        S["dt"] = {"peri": 0.9, "ell": 0.9, "cloud": 0.4}.get(kind, 0.4 if law == "frict" else 0.3) * rmin / float((E / rho).max()) ** 0.5
        S["verletDist"] = -0.05 if law == "frict" else 0.1 * rmin
        if kind == "peri":
            grad = np.zeros((3, 3))
            grad[0, 2] = float(case["rate"])
            S.update(gravity=(0.0, 0.0, 0.0), damping=0.0, cell=dict(hSize=np.diag(box.cpu().numpy()), nextGradV=grad))
        if kind == "cloud" and law == "hertz":
            S["damping"] = 0.0
    k = len(r)
    rho = torch.tensor([m["density"] for m in mats], device=LOCAL, dtype=torch.float64)[mat]
    if kind == "ell":
        semi = r[:, None] * _axes()
        mass = (4.0 / 3.0 * math.pi) * semi.prod(1) * rho
        q = semi.square()
        inertia = mass[:, None] / 5.0 * (q.sum(1, keepdim=True) - q)
        S["semi"] = semi.cpu().numpy()
        tilt = torch.randn((k, 3), generator=g, device=LOCAL, dtype=torch.float64) * 0.01  # about a degree
        ori = _unit(torch.cat([torch.ones(k, 1, device=LOCAL, dtype=torch.float64), tilt], dim=1))
    else:
        mass = (4.0 / 3.0 * math.pi) * r ** 3 * rho
        inertia = (0.4 * mass * r * r)[:, None].expand(k, 3)
        ori = torch.zeros(k, 4, device=LOCAL, dtype=torch.float64)
        ori[:, 0] = 1.0
    sd = {"bed": 0.05, "hopper": 0.1, "peri": 0.2, "batch": 0.1, "ell": 0.1, "cloud": 0.05}[kind]
    vel = torch.randn((k, 3), generator=g, device=LOCAL, dtype=torch.float64) * sd
    ang = torch.randn((k, 3), generator=g, device=LOCAL, dtype=torch.float64) * (10 * sd)
    if kind == "cloud":
        vel[:, 2] -= float(case["speed"])
    if kind == "peri":
        vel[:, 0] += float(case["rate"]) * pos[:, 2]
    if kind == "hopper":
        # the outlet takes spheres of the lowest layers, the inlet brings them back where they were, at rest
        m = int(case["moved"])
        low = torch.argsort(pos[:, 2])[: max(m, k // 4)]
        S["moved"] = low[torch.randperm(len(low), generator=g, device=LOCAL)[:m]].sort().values.cpu().numpy()
    for name, v in (("pos", pos), ("vel", vel), ("angVel", ang), ("ori", ori), ("r", r), ("mass", mass), ("inertia", inertia)):
        S[name] = np.ascontiguousarray(v.cpu().numpy())
    S["mat"] = mat.cpu().numpy().astype(np.int32)
    S["scene"] = np.zeros(k, np.int32) if scene is None else scene.cpu().numpy().astype(np.int32)
    S["walls"], S["mats"] = walls, mats
    return S


# ------------------------------------------------------------------------------------------------ the engine
def _particles(abi, S, which=None, wall=True):
    walls = S["walls"] if wall else []
    nw, idx = len(walls), np.arange(len(S["r"])) if which is None else which
    pa = abi.ParticleArrays(nw + len(idx))
    for i, (ax, sense, at, mi, sc, v) in enumerate(walls):
        pa.shape[i], pa.wallAxis[i], pa.wallSense[i], pa.material[i], pa.scene[i] = abi.SHAPE_WALL, ax, sense, mi, sc
        pa.pos[i, ax], pa.vel[i, ax] = at, v
        pa.mask[i], pa.flags[i] = BOUNDARY, BLOCKED
    s = slice(nw, None)
    pa.shape[s] = abi.SHAPE_SPHERE if S["semi"] is None else abi.SHAPE_ELLIPSOID
    if S["semi"] is None:
        pa.radius[s] = S["r"][idx]
    else:
        pa.semiAxes[s] = S["semi"][idx]
    pa.mask[s] = MOVABLE
    for name in ("pos", "vel", "angVel", "ori", "mass", "inertia", "scene"):
        getattr(pa, name)[s] = S[name][idx]
    pa.material[s] = S["mat"][idx]
    pa.force[s] = pa.mass[s, None] * np.asarray(S["gravity"])
    return pa


def prepare(case, seed):
    from woo_gb300 import abi, scenes
    if case["kind"] == "net":
        w, rec = _net(case, seed)
        h = abi.Handle(1)
        h.warm_set_weights(w)
        return dict(case=case, h=h, rec=rec, x=np.ascontiguousarray(rec[:, :13]))
    S = _scene(case, seed)
    frict = S["law"] == "frict"
    mats = scenes.materials_array([dict(m, kind=abi.MAT_FRICT if frict else abi.MAT_HERTZ) for m in S["mats"]])
    extra = {} if frict else dict(cp2=abi.CP2_HERTZ, law=abi.LAW_HERTZ_DMT, en=0.8)
    if S["semi"] is not None:
        newton = case["solver"] == "newton"
        extra.update(ellSolver=abi.ELL_NEWTON if newton else abi.ELL_BRENT, warmStart=abi.WARM_HISTORY if newton else abi.WARM_COLD)
    par = scenes.default_params(mats, dt=S["dt"], gravity=S["gravity"], damping=S["damping"], verletDist=S["verletDist"],
                                trackEnergy=int(case.get("energy", 0)), **extra)
    par.arith = {"exact": abi.ARITH_EXACT, "fma": abi.ARITH_FMA, "dw": abi.ARITH_DW}[case["arith"]]
    keep = [mats]
    if S["matDt"] is not None:
        keep.append((ctypes.c_double * len(S["matDt"]))(*S["matDt"]))
        par.materialDt = keep[-1]
    pa = _particles(abi, S)
    h = abi.Handle(pa.n)
    h.set_params(par)
    h.upload_particles(pa)
    if S["cell"] is not None:
        h.set_cell(**S["cell"])
    state = dict(case=case, h=h, n=pa.n, steps=int(case["steps"]), keep=keep)
    host = lambda a: torch.from_numpy(np.ascontiguousarray(a)).pin_memory()  # noqa: E731
    state["out"] = {k: torch.empty((pa.n, 4 if k == "ori" else 3), dtype=torch.float64).pin_memory() for k in ("pos", "vel", "angVel", "ori")}
    if case["kind"] == "cloud":
        state["in"] = {k: host(getattr(pa, k)) for k in state["out"]}
    if case["kind"] == "hopper":
        state["ids"] = S["moved"] + len(S["walls"])
        state["put"] = _particles(abi, S, S["moved"], wall=False)
        state["park"] = np.ascontiguousarray(state["put"].pos)
    return state


def run(state):
    h, case = state["h"], state["case"]
    if case["kind"] == "net":
        if case["what"] == "predict":
            return {"y": h.warm_predict(state["x"])}
        grad, loss = h.warm_grad(state["rec"])
        return {"grad": grad, "loss": np.float32(loss)}
    if "in" in state:
        h.write_state(state["n"], *[state["in"][k].data_ptr() for k in ("pos", "vel", "angVel", "ori")])
    if "ids" in state:
        h.remove_particles(state["ids"], state["park"])
        h.add_particles(state["put"], state["ids"])
    h.step(state["steps"])
    out = state["out"]
    h.read_state(state["n"], *[out[k].data_ptr() for k in ("pos", "vel", "angVel", "ori")])
    if case.get("energy"):
        e = h.energy()
        return dict(out, energy=np.array([e[k] for k in ("kinetic", "grav", "nonviscDamp", "elast")]))
    return dict(out)


def work(case):
    n = int(case["n"])
    if case["kind"] == "net":
        mac = 13 * 64 + 2 * 64 * 64 + 64 * 4
        grad = case["what"] == "grad"
        return {"bytes": n * 4.0 * (17 if grad else 17) + 4.0 * 9476 * (2 if grad else 1), "flops": 2.0 * mac * n * (3 if grad else 1)}
    steps = int(case["steps"])
    bodies = n if case["kind"] != "batch" else 5286.0 * n  # the mean of 500 .. 20000 over the logarithm
    # per step and body: position, velocity, spin and orientation read and written; per contact: the two bodies'
    # gathered state is theirs already, its own history (frame, contact point, force, stiffnesses) read and written
    per_body = {"cloud": 0.02, "bed": 2.4, "peri": 2.8, "batch": 2.2, "ell": 2.0, "hopper": 2.4}[case["kind"]]
    flops = 1200.0 if case["kind"] == "ell" else 400.0
    return {"bytes": steps * bodies * (208.0 + 224.0 * per_body) + 104.0 * bodies * (2 if case["kind"] == "cloud" else 1),
            "flops": steps * bodies * (40.0 + flops * per_body)}


# ------------------------------------------------------------------------------------------------ in 64 bits
def _net(case, seed):
    """Weights (He-uniform) and training records: 13 features of a pair (relative centre, relative orientation,
    semi-axes, lengths over the sum of the largest semi-axes) and its maximiser and contact point."""
    rng = np.random.default_rng(seed)
    n = int(case["n"])
    layers = []
    for fi, fo in ((13, 64), (64, 64), (64, 64), (64, 4)):
        lim = math.sqrt(6.0 / fi)
        layers += [rng.uniform(-lim, lim, fi * fo), rng.uniform(-0.1, 0.1, fo)]
    a = rng.uniform(3, 6, (n, 2))
    s = a.sum(1)
    q = rng.normal(size=(n, 4))
    q /= np.linalg.norm(q, axis=1)[:, None]
    q[:, 0] = np.abs(q[:, 0])
    d = rng.normal(size=(n, 3))
    d *= (rng.uniform(0.55, 1.0, n) / np.linalg.norm(d, axis=1))[:, None]
    ratios = np.array([1.0, 0.7, 0.5])
    semi = np.concatenate([a[:, :1] * ratios, a[:, 1:] * ratios], axis=1) / s[:, None]
    lam = a[:, 0] / s
    rec = np.concatenate([d, q, semi, lam[:, None], d * lam[:, None]], axis=1)
    return np.concatenate(layers).astype(np.float32), np.ascontiguousarray(rec.astype(np.float32))


def _net_exact(case, seed):
    w, rec = _net(case, seed)
    at, layers, leaves = 0, [], []
    for fi, fo in ((13, 64), (64, 64), (64, 64), (64, 4)):
        W = torch.tensor(w[at:at + fi * fo].reshape(fi, fo), dtype=torch.float64, device=LOCAL, requires_grad=True)
        b = torch.tensor(w[at + fi * fo:at + fi * fo + fo], dtype=torch.float64, device=LOCAL, requires_grad=True)
        at += fi * fo + fo
        layers.append((W, b))
        leaves += [W, b]
    R = torch.tensor(rec, dtype=torch.float64, device=LOCAL)
    x = R[:, :13]
    for k, (W, b) in enumerate(layers):
        x = x @ W + b
        if k < 3:
            x = x.relu()
    if case["what"] == "predict":
        return {"y": x.detach().cpu().numpy()}
    lw = torch.tensor([1.0, 0.1, 0.1, 0.1], dtype=torch.float64, device=LOCAL)
    loss = ((x - R[:, 13:]).square() * lw).sum() / len(R)
    loss.backward()
    return {"grad": torch.cat([v.grad.reshape(-1) for v in leaves]).cpu().numpy(), "loss": np.float64(loss.item())}


def _dot(a, b):
    return (a * b).sum(-1)


def _cross(a, b):
    return torch.linalg.cross(a, b)


def _unit(a):
    return a / a.square().sum(-1, keepdim=True).sqrt()


def _qmul(a, b):
    aw, av, bw, bv = a[:, :1], a[:, 1:], b[:, :1], b[:, 1:]
    return torch.cat([aw * bw - (av * bv).sum(1, keepdim=True), aw * bv + bw * av + _cross(av, bv)], dim=1)


def _rotate(q, v):
    uv = 2 * _cross(q[:, 1:], v)
    return v + q[:, :1] * uv + _cross(q[:, 1:], uv)


def _conj(q):
    return torch.cat([q[:, :1], -q[:, 1:]], dim=1)


def _close_pairs(x, reach, box=None):
    """Pairs (i < j) whose centres are closer than the sum of their reaches, with the period shift of j."""
    n, dev = len(x), x.device
    width = 2 * float(reach.max())
    lo = torch.zeros(3, device=dev, dtype=x.dtype) if box is not None else x.min(0).values
    span = box if box is not None else x.max(0).values - lo + 1e-12
    nc = torch.clamp((span / width).floor(), 1, 400).long()
    shift0 = torch.floor((x - lo) / span) if box is not None else torch.zeros_like(x)
    y = x - shift0 * span if box is not None else x
    cell = torch.minimum(((y - lo) / span * nc).long().clamp(min=0), nc - 1)
    key = (cell[:, 2] * nc[1] + cell[:, 1]) * nc[0] + cell[:, 0]
    order = torch.argsort(key)
    start = torch.searchsorted(key[order].contiguous(), torch.arange(int(nc.prod()) + 1, device=dev))
    most = int((start[1:] - start[:-1]).max())
    got = []
    seen_axes = [sorted({d % int(nc[a]) if box is not None else d for d in (-1, 0, 1)}) for a in range(3)]
    ids = torch.arange(n, device=dev)
    for dz in seen_axes[2]:
        for dy in seen_axes[1]:
            for dx in seen_axes[0]:
                c = cell + torch.tensor([dx, dy, dz], device=dev)
                if box is not None:
                    c = c % nc
                    ok = torch.ones(n, dtype=torch.bool, device=dev)
                else:
                    ok = ((c >= 0) & (c < nc)).all(1)
                    c = torch.minimum(c.clamp(min=0), nc - 1)
                k2 = (c[:, 2] * nc[1] + c[:, 1]) * nc[0] + c[:, 0]
                beg, end = start[k2], start[k2 + 1]
                for q in range(most):
                    live = ok & (beg + q < end)
                    i = ids[live]
                    if not len(i):
                        break
                    j = order[(beg + q)[live]]
                    d = x[j] - x[i]
                    s = torch.round(d / span) if box is not None else torch.zeros_like(d)
                    d = d - s * span if box is not None else d
                    near = (i < j) & (d.square().sum(1) < (reach[i] + reach[j]).square())
                    got.append((i[near], j[near], -s[near]))
    return tuple(torch.cat([v[k] for v in got]) for k in range(3))



def _ell_matrix(q, semi):
    eye = torch.eye(3, dtype=q.dtype, device=q.device)
    A = torch.zeros(len(q), 3, 3, dtype=q.dtype, device=q.device)
    for k in range(3):
        u = _rotate(q, eye[k].expand(len(q), 3))
        A = A + u[:, :, None] * u[:, None, :] * semi[:, k].square()[:, None, None]
    return A


def _sym_solve(G, b):
    """x with G x = b for symmetric positive 3x3 matrices, by the adjugate."""
    c0, c1, c2 = G[:, :, 0], G[:, :, 1], G[:, :, 2]
    k0, k1, k2 = _cross(c1, c2), _cross(c2, c0), _cross(c0, c1)
    return torch.stack([_dot(k0, b), _dot(k1, b), _dot(k2, b)], 1) / _dot(c0, k0)[:, None]


def _simulate(case, seed):
    """`steps` steps of the scene in 64-bit torch: forces and torques of the step before, Leapfrog, contacts."""
    S = _scene(case, seed)
    T = lambda a: torch.as_tensor(np.array(a), device=LOCAL, dtype=torch.float64)  # noqa: E731
    steps, ell, hertz = int(case["steps"]), S["semi"] is not None, S["law"] == "hertz"
    x, v, w, q = (T(S[k]) for k in ("pos", "vel", "angVel", "ori"))
    r, m, inertia, g = T(S["r"]), T(S["mass"]), T(S["inertia"]), T(S["gravity"])
    mat = torch.as_tensor(S["mat"].astype(np.int64), device=LOCAL)
    semi = T(S["semi"]) if ell else None
    n = len(r)
    prop = {k: T([p[k] for p in S["mats"]]) for k in ("young", "tanPhi", "ktDivKn", "surfEnergy")}
    dt = (T(S["matDt"])[mat] if S["matDt"] is not None else torch.full((n,), S["dt"], device=LOCAL, dtype=torch.float64))
    damping, walls = S["damping"], S["walls"]
    scene = torch.as_tensor(S["scene"].astype(np.int64), device=LOCAL)
    # pairs that can meet in these steps
    fast = float(v.square().sum(1).max().sqrt()) + (15.0 if ell else 2.0)
    slack = 2 * fast * float(dt.max()) * (steps + 1) + 0.02 * float(r.max())
    hS = box = None
    if S["cell"] is not None:
        hS, grad_next = S["cell"]["hSize"].copy(), S["cell"]["nextGradV"]
        grad = np.zeros((3, 3))
        box = T(np.diag(hS))
    i, j, shift = _close_pairs(x, r + slack, box)
    if S["matDt"] is not None:
        same = scene[i] == scene[j]
        i, j, shift = i[same], j[same], shift[same]
    # walls: candidate contacts with the wall as the first body
    wa, wb = [], []
    for k, (ax, sense, at, mi, sc, vw) in enumerate(walls):
        near = ((x[:, ax] - at).abs() < r + slack) & (scene == sc)
        b = near.nonzero()[:, 0]
        wa.append(torch.full_like(b, k))
        wb.append(b)
    nw = len(walls)
    wa, wb = (torch.cat(t) if walls else torch.zeros(0, dtype=torch.long, device=LOCAL) for t in (wa, wb))
    A, B = torch.cat([wa, i + nw]), torch.cat([wb, j]) + nw  # body ids with the walls first
    isw = A < nw
    shift = torch.cat([torch.zeros(len(wa), 3, device=LOCAL, dtype=torch.float64), shift])
    wax = torch.tensor([t[0] for t in walls] + [0], device=LOCAL)
    wsense = torch.tensor([t[1] for t in walls] + [0], device=LOCAL)
    W0 = torch.zeros(nw, 3, device=LOCAL, dtype=torch.float64)
    Wv = W0.clone()
    for k, t in enumerate(walls):
        W0[k, t[0]], Wv[k, t[0]] = t[2], t[5]
    wdt = T(S["matDt"])[torch.tensor([t[3] for t in walls], device=LOCAL)] if S["matDt"] is not None else torch.full((nw,), S["dt"], device=LOCAL, dtype=torch.float64)
    matAll = torch.cat([torch.tensor([t[3] for t in walls], device=LOCAL, dtype=torch.long), mat])
    rAll = torch.cat([torch.zeros(nw, device=LOCAL, dtype=torch.float64), r])
    mAll = torch.cat([torch.zeros(nw, device=LOCAL, dtype=torch.float64), m])
    dtC = torch.cat([wdt, dt])[A][:, None]
    real = torch.zeros(len(A), dtype=torch.bool, device=LOCAL)
    z3 = torch.zeros(len(A), 3, device=LOCAL, dtype=torch.float64)
    ax0, ax1, cp, fl = z3.clone(), z3.clone(), z3.clone(), z3.clone()
    # Cp2: constants of a contact of bodies A and B (spheres: by their radii)
    mA, mB = matAll[A], matAll[B]
    tanphi = torch.minimum(prop["tanPhi"][mA], prop["tanPhi"][mB])
    F, Tq = m[:, None] * g, torch.zeros_like(x)
    E = dict(kinetic=0.0, grav=0.0, nonviscDamp=0.0, elast=0.0)
    am = None
    kn = torch.zeros(len(A), device=LOCAL, dtype=torch.float64)
    kt = kn.clone()
    axis1 = torch.nn.functional.one_hot(wax[torch.where(isw, A, torch.full_like(A, nw))], 3).to(torch.float64)
    wsideA = wsense[torch.where(isw, A, torch.full_like(A, nw))]
    nu = 0.2
    if hertz:
        K = (4 / 3.0) / ((1 - nu * nu) / prop["young"][mA] + (1 - nu * nu) / prop["young"][mB])
        len0, len1 = torch.where(isw, rAll[B], rAll[A]), rAll[B]
        R = 1 / (1 / len0 + 1 / len1)
        kn0 = K * R.sqrt()
        G = 0.5 * (prop["young"][mA] + prop["young"][mB]) / (2 * (1 + nu))
        kt0 = 2 * (4 * R).sqrt() * G / (2 - nu)
        adh = 4 * math.pi * R * torch.minimum(prop["surfEnergy"][mA], prop["surfEnergy"][mB])
        ln = math.log(0.8)
        alpha = -math.sqrt(5) * ln / math.sqrt(ln * ln + math.pi ** 2)
        mbar = torch.where(mAll[A] <= 0, mAll[B], mAll[A] * mAll[B] / (mAll[A] + mAll[B]).clamp(min=1e-300))
        visc = alpha * (mbar * kn0).sqrt()
    h1 = dt[:, None]
    for step in range(steps):
        # ---- cell and Leapfrog
        if hS is not None:
            half = grad * S["dt"] / 2
            prev = hS
            hS = np.linalg.inv(np.eye(3) - half) @ (np.eye(3) + half) @ hS
            mid = 0.5 * (prev + hS)
            LL = (grad_next + grad) * S["dt"] / 4
            Mi, Mp, ML = T(np.linalg.inv(np.eye(3) - LL)), T(np.eye(3) + LL), T(grad_next - grad)
            sp = [0.5 * (a - a.T) for a in (grad, grad_next)]
            lc = [np.array([s[1, 2] - s[2, 1], s[2, 0] - s[0, 2], s[0, 1] - s[1, 0]]) for s in sp]
            dspin, hST, shvT = T(-0.5 * lc[0] + 0.5 * lc[1]), T(hS), T(grad @ mid)
        acc = F / m[:, None]
        if case.get("energy"):
            E["nonviscDamp"] += float((_dot(v.abs(), F.abs()) * damping * dt + _dot(w.abs(), Tq.abs()) * damping * dt).sum())
            E["grav"] += float((-(v @ g) * m * dt).sum())
        if damping:
            acc = acc * (1 - damping * torch.sign(F * (v + 0.5 * h1 * acc)))
        ali = Tq / inertia
        if damping and not ell:
            ali = ali * (1 - damping * torch.sign(Tq * (w + 0.5 * h1 * ali)))
        if case.get("energy"):
            cv, cw = v + 0.5 * h1 * acc, w + 0.5 * h1 * ali
            E["kinetic"] = float((0.5 * m * cv.square().sum(1) + 0.5 * (inertia * cw.square()).sum(1)).sum())
        if hS is not None:
            v = (x @ ML.T + v @ Mp.T + acc * h1) @ Mi.T
        else:
            v = v + h1 * acc
        x = x + v * h1
        if ell:
            tq = Tq * (1 - damping * torch.sign(Tq * w))
            qc = _conj(q)
            if am is None:
                am = inertia * _rotate(qc, w)
            rate = lambda b, p: 0.5 * torch.cat([-(p[:, 1:] * b).sum(1, keepdim=True), p[:, :1] * b + _cross(p[:, 1:], b)], dim=1)  # noqa: E731
            wb_ = _rotate(qc, am + 0.5 * h1 * tq) / inertia
            qh = q + 0.5 * h1 * rate(wb_, q)
            am = am + h1 * tq
            wh = _rotate(qc, am) / inertia
            q = q + h1 * rate(wh, qh)
            w = _rotate(q, wh)
            q = _unit(q)
        else:
            w = w + h1 * ali
            if hS is not None:
                w = w - dspin
            wn = w.square().sum(1, keepdim=True).sqrt()
            ha = 0.5 * wn * h1
            q = _unit(_qmul(torch.cat([torch.cos(ha), torch.sin(ha) * w / wn.clamp(min=1e-300)], dim=1), q))
        W0 = W0 + Wv * wdt[:, None]
        # ---- contacts
        X, V, Om = torch.cat([W0, x]), torch.cat([Wv, v]), torch.cat([torch.zeros_like(W0), w])
        p1, p2, v1, v2, o1, o2 = X[A], X[B], V[A], V[B], Om[A], Om[B]
        vs = 0.0
        if hS is not None:
            p2 = p2 + shift @ hST.T
            vs = shift @ shvT.T
        d = p2 - p1
        if ell:
            nrm, pt, uN, r1, r2, touch = _ell_geometry(A, B, isw, nw, axis1, wsideA, p1, p2, q, semi)
            touch = touch | real
        else:
            dist = d.square().sum(1).sqrt()
            along = (d * axis1).sum(1)
            side = torch.where(wsideA == 0, torch.sign(along), wsideA.to(torch.float64))
            r1, r2 = torch.where(isw, -rAll[B], rAll[A]), rAll[B]
            touch = torch.where(isw, along.abs() <= rAll[B], dist <= rAll[A] + rAll[B]) | real
            uN = torch.where(isw, side * along - rAll[B], dist - rAll[A] - rAll[B])
            nrm = torch.where(isw[:, None], axis1 * side[:, None], d / dist[:, None])
            on_wall = p2 + axis1 * ((p1 - p2) * axis1).sum(1, keepdim=True)
            pt = torch.where(isw[:, None], on_wall, p1 + (rAll[A] + 0.5 * uN)[:, None] * nrm)
        new = touch & ~real
        # new contacts: local axes and the stiffnesses of the law
        e = torch.where((nrm[:, 1].abs() < nrm[:, 2].abs())[:, None], T([0, 1, 0]), T([0, 0, 1]))
        y0 = _cross(nrm, e)
        y0 = _unit(y0 - nrm * _dot(y0, nrm)[:, None])
        # kept contacts: the frame turned with the pair, relative velocity in the middle of the step
        mid0 = _unit(0.5 * (ax0 + nrm) + torch.where(real[:, None], 0.0, 1.0) * nrm)
        rt = _cross(ax0, nrm) + mid0 * (dtC * 0.5 * _dot(mid0, o1 + o2)[:, None])
        mid1 = ax1 - 0.5 * _cross(ax1, rt)
        mid2 = _cross(mid0, mid1)
        c1 = ax1 - _cross(mid1, rt)
        c0 = nrm
        if step % 100 == 0:
            c1 = c1 - c0 * _dot(c1, c0)[:, None]
            c1 = torch.where(real[:, None], _unit(c1), c1)
        pm = 0.5 * (cp + pt)
        l1, l2 = pm - (p1 - 0.5 * dtC * v1), pm - (p2 - 0.5 * dtC * (v2 + vs))
        rel = (v2 + vs + _cross(o2, l2)) - (v1 + _cross(o1, l1))
        gv = torch.stack([_dot(mid0, rel), _dot(mid1, rel), _dot(mid2, rel)], 1) * real[:, None]
        ax0, ax1 = torch.where(real[:, None], c0, nrm), torch.where(real[:, None], c1, y0)
        fl = fl * real[:, None]
        # law
        if hertz:
            sq = (-uN).clamp(min=0).sqrt()
            kt = kt0 * sq
            eta = visc * sq.sqrt()
            fel = -kn0 * sq ** 3
            fv = eta * gv[:, 0]
            fv = torch.where(fel + fv > 0, -fel, fv)
            fx = fel + adh + fv
            cap = (tanphi * fx.clamp(max=0)).abs()
        else:
            if ell:
                len0, len1 = r1.abs(), r2.abs()
            else:
                len0, len1 = torch.where(isw, rAll[B], rAll[A]), rAll[B]
            rr = torch.where(isw, len1, torch.minimum(len0, len1))
            area = math.pi * rr * rr
            kn_new = 1 / (1 / (prop["young"][mA] * area / len0) + 1 / (prop["young"][mB] * area / len1))
            kn = torch.where(new, kn_new, kn)
            kt = 0.5 * (prop["ktDivKn"][mA] + prop["ktDivKn"][mB]) * kn
            fx = kn * uN
            cap = fx.abs() * tanphi
        ft = fl[:, 1:] + dtC * kt[:, None] * gv[:, 1:]
        norm = ft.square().sum(1).sqrt()
        slip = norm > cap
        ratio = torch.where(slip, cap / norm.clamp(min=1e-300), torch.ones_like(norm))
        ft = ft * ratio[:, None]
        if hertz:
            ft = torch.where(slip[:, None], ft, ft + eta[:, None] * gv[:, 1:])
        keep = touch & ~(uN > 0)
        real = keep
        cp = pt
        fl = torch.cat([fx[:, None], ft], dim=1) * keep[:, None]
        if case.get("energy"):
            el = 0.5 * (fl[:, 0].square() / kn + fl[:, 1:].square().sum(1) / kt)
            E["elast"] = float(torch.where(keep, el, torch.zeros_like(el)).nan_to_num().sum())
        ax2 = _cross(ax0, ax1)
        tx = _frame_rotate(ax0, ax1, ax2, fl) * keep[:, None]
        tA, tB = _cross(pt - p1, tx), -_cross(pt - p2, tx)
        live = keep.nonzero()[:, 0]
        both = torch.cat([torch.zeros_like(W0), m[:, None] * g])
        tor = torch.zeros_like(X)
        both.index_add_(0, A[live], tx[live]).index_add_(0, B[live], -tx[live])
        tor.index_add_(0, A[live], tA[live]).index_add_(0, B[live], tB[live])
        F, Tq = both[nw:], tor[nw:]
        if hS is not None:
            grad = grad_next
    qw = torch.zeros(nw, 4, device=LOCAL, dtype=torch.float64)
    qw[:, 0] = 1
    out = dict(pos=torch.cat([W0, x]), vel=torch.cat([Wv, v]), angVel=torch.cat([torch.zeros_like(W0), w]), ori=torch.cat([qw, q]))
    out = {k: a.cpu().numpy() for k, a in out.items()}
    if case.get("energy"):
        out["energy"] = np.array([E[k] for k in ("kinetic", "grav", "nonviscDamp", "elast")])
    return out


def _frame_rotate(c0, c1, c2, f):
    """f rotated by the quaternion that Shoemake's method takes from the (nearly orthonormal) frame c0, c1, c2."""
    M = torch.stack([c0, c1, c2], dim=2)
    tr = M.diagonal(dim1=1, dim2=2).sum(1)
    dg = M.diagonal(dim1=1, dim2=2)
    out = torch.zeros(len(f), 4, device=f.device, dtype=f.dtype)
    t = (tr + 1).clamp(min=1e-300).sqrt()
    pos = torch.stack([0.5 * t, (M[:, 2, 1] - M[:, 1, 2]) * 0.5 / t, (M[:, 0, 2] - M[:, 2, 0]) * 0.5 / t, (M[:, 1, 0] - M[:, 0, 1]) * 0.5 / t], 1)
    top = torch.where(dg[:, 1] > dg[:, 0], 1, 0)
    top = torch.where(dg[:, 2] > dg.gather(1, top[:, None])[:, 0], 2, top)
    for a in range(3):
        b, c = (a + 1) % 3, (a + 2) % 3
        t = (M[:, a, a] - M[:, b, b] - M[:, c, c] + 1).clamp(min=1e-300).sqrt()
        o = torch.zeros_like(out)
        o[:, 1 + a] = 0.5 * t
        o[:, 0] = (M[:, c, b] - M[:, b, c]) * 0.5 / t
        o[:, 1 + b] = (M[:, b, a] + M[:, a, b]) * 0.5 / t
        o[:, 1 + c] = (M[:, c, a] + M[:, a, c]) * 0.5 / t
        out = torch.where((top == a)[:, None], o, out)
    return _rotate(torch.where((tr > 0)[:, None], pos, out), f)


def _ell_geometry(A, B, isw, nw, axis1, side, p1, p2, q, semi):
    """Normal, contact point, overlap, lever arms and touch flag of ellipsoid-ellipsoid and wall-ellipsoid pairs."""
    sA, sB = semi[(A - nw).clamp(min=0)], semi[B - nw]
    Ai, Bi = _ell_matrix(q[(A - nw).clamp(min=0)], sA), _ell_matrix(q[B - nw], sB)
    R = p2 - p1
    lo, hi = torch.zeros(len(A), device=q.device, dtype=q.dtype), torch.ones(len(A), device=q.device, dtype=q.dtype)
    D = Bi - Ai
    for _ in range(60):  # the sign of the derivative of l (1-l) R^T G^-1 R, which is concave
        l = 0.5 * (lo + hi)
        y = _sym_solve((1 - l)[:, None, None] * Ai + l[:, None, None] * Bi, R)
        slope = (1 - 2 * l) * _dot(R, y) - l * (1 - l) * _dot(y, torch.einsum("kij,kj->ki", D, y))
        lo, hi = torch.where(slope > 0, l, lo), torch.where(slope > 0, hi, l)
    l = 0.5 * (lo + hi)
    y = _sym_solve((1 - l)[:, None, None] * Ai + l[:, None, None] * Bi, R)
    fab = l * (1 - l) * _dot(R, y)
    pt = p1 + (1 - l)[:, None] * torch.einsum("kij,kj->ki", Ai, y)
    nrm, dist = _unit(y), R.square().sum(1).sqrt()
    uN = dist * (1 - 1 / fab.clamp(min=1e-300).sqrt()) * _dot(R / dist[:, None], nrm)
    r1, r2, touch = (pt - p1).square().sum(1).sqrt(), (pt - p2).square().sum(1).sqrt(), fab <= 1
    # walls: the extent of the ellipsoid along the wall's axis and the point that reaches it
    ext = torch.einsum("ki,kij,kj->k", axis1, Bi, axis1).sqrt()
    along = _dot(R, axis1)
    s = torch.where(side == 0, torch.where(along > 0, 1.0, -1.0).to(q.dtype), side.to(q.dtype))
    col = torch.einsum("kij,kj->ki", Bi, axis1) / ext[:, None]
    wp = p2 - s[:, None] * col
    wp = wp + axis1 * _dot(p1 - wp, axis1)[:, None]
    arm = (wp - p2).square().sum(1).sqrt()
    pick = lambda a, b: torch.where(isw if a.dim() == 1 else isw[:, None], a, b)  # noqa: E731
    return (pick(axis1 * s[:, None], nrm), pick(wp, pt), pick(s * along - ext, uN), pick(-arm, r1), pick(arm, r2),
            torch.where(isw, along.abs() <= ext, touch))


def exact(case, seed):
    if case["kind"] == "net":
        return _net_exact(case, seed)
    bodies = int(case["n"]) * (5286 if case["kind"] == "batch" else 1)
    if bodies * int(case["steps"]) > 6e7:  # the 64-bit run would take too long
        return None
    return _simulate(case, seed)
