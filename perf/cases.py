"""Performance cases: the calls a user of this framework makes, over the
sizes, models and options that the path serves.

A program sends one system's initial conditions in, steps it and reads the
final state back (Hertz-Mindlin, soft penalty or PSOR contact), does the same
with a batch of uneven systems, asks for the contacts or the contact forces
of given positions, or trains the warm-start network.  `listed()` holds one case of each at the sizes of the repository's
own workloads (rodgpu.scene.WORKLOADS and bench.py) and at odd ones,
`draw(rng)` gives others of the same ranges.

Packings: random sequential addition, drawn with a slightly smaller diameter
than the rods then have, so the system is not contact-free at the start but
has about as many touching pairs as one that has run for a while.  Aspect
ratio A means L = 1, d = 1 / A; the volume fraction stays below the isotropic
packing's limit near 1.6 / A.
"""
import math
import os
import sys

import numpy as np

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rod-dynamics-3d_b200"))

import rodgpu  # noqa: E402
from rodgpu import scene  # noqa: E402

# Time steps of the workloads: Hertz-Mindlin and soft contact 1e-4 (2e-5 for
# the stiff large system), PSOR 5e-4.
DT = {"hertz-mindlin": 1e-4, "harmonic": 1e-4, "nsc": 5e-4}


def listed():
    return [
        # the smallest call of the soft models: forces at given positions
        dict(name="forces_1k", kind="forces", model="hertz-mindlin", rods=1000, aspect=10, phi=0.10, mu=0.5,
             friction="smooth", squeeze=0.95),
        # contacts of positions that another program supplies
        dict(name="contacts_50k", kind="contacts", model="nsc", rods=50021, aspect=20, phi=0.09, mu=0.3,
             friction="smooth", squeeze=0.9),
        # the plain soft-contact workload: 1000 rods, 200 of its steps
        dict(name="hm_1k", kind="steps", model="hertz-mindlin", rods=1000, aspect=10, phi=0.10, mu=0.5,
             friction="smooth", squeeze=0.995, steps=200),
        # an ordinary Hertz-Mindlin run
        dict(name="hm_20k", kind="steps", model="hertz-mindlin", rods=20011, aspect=20, phi=0.08, mu=0.4,
             friction="smooth", squeeze=0.995, steps=100),
        # the large Hertz-Mindlin system
        dict(name="hm_1m", kind="steps", model="hertz-mindlin", rods=1000000, aspect=50, phi=0.045, mu=0.5,
             friction="smooth", squeeze=0.995, steps=400),
        # soft penalty contact with Cundall friction (tangential history)
        dict(name="soft_5k", kind="steps", model="harmonic", rods=5003, aspect=10, phi=0.12, mu=0.5,
             friction="cundall", squeeze=0.995, steps=100),
        # the smallest PSOR system: a tiny box whose lists hold every pair
        dict(name="nsc_500", kind="steps", model="nsc", rods=500, aspect=20, phi=0.08, mu=0.6, friction="smooth",
             squeeze=0.995, steps=100),
        # the dense PSOR workload
        dict(name="nsc_20k", kind="steps", model="nsc", rods=20000, aspect=20, phi=0.10, mu=0.3,
             friction="smooth", squeeze=0.995, steps=100),
        # the large PSOR workload (the learned warm start's system size)
        dict(name="nsc_50k", kind="steps", model="nsc", rods=50000, aspect=20, phi=0.10, mu=0.45,
             friction="smooth", squeeze=0.995, steps=50),
        # the uneven batch with the learned warm start (PSOR members only)
        dict(name="batch_nsc", kind="batch", members=32, rods_lo=500, rods_hi=20000, sweep=1, soft_half=False,
             learned=True, steps=20),
        # the uneven batch as described: half Hertz-Mindlin, half PSOR
        dict(name="batch_mixed", kind="batch", members=24, rods_lo=500, rods_hi=8000, sweep=2, soft_half=True,
             learned=False, steps=20),
        # training of the warm-start network on recorded contacts
        dict(name="train_64k", kind="train", records=65536, minibatch=4096, epochs=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "steps", "batch", "batch", "contacts", "forces", "train"])
    if kind == "train":
        return dict(kind=kind, records=_log_int(rng, 8192, 65536), minibatch=rng.choice([512, 1000, 2048, 4096]),
                    epochs=rng.randint(1, 4))
    if kind == "batch":
        soft = rng.random() < 0.5
        lo = _log_int(rng, 500, 2000)
        return dict(kind=kind, members=rng.randint(4, 32), rods_lo=lo, rods_hi=_log_int(rng, 2 * lo, 12000),
                    sweep=rng.randint(3, 1 << 30), soft_half=soft, learned=rng.random() < 0.5, steps=rng.randint(5, 20))
    aspect = rng.choice([5, 10, 20, 40])
    phi = round(min(rng.uniform(0.05, 0.25), scene.rsa_phi_max(aspect)), 4)
    model = rng.choice(["hertz-mindlin", "harmonic", "nsc"])
    c = dict(kind=kind, model=model, aspect=aspect, phi=phi, mu=round(rng.uniform(0.1, 0.9), 3),
             friction=rng.choice(["smooth", "cundall", "karnopp"]) if model == "harmonic" else "smooth")
    if kind == "steps":
        rods = _log_int(rng, 500, 50000 if model == "nsc" else 200000)
        c.update(rods=rods, squeeze=0.995, steps=_log_int(rng, 20, 100 if rods > 20000 else 200))
    elif kind == "contacts":
        c.update(model="nsc", friction="smooth", rods=_log_int(rng, 1000, 100000), squeeze=round(rng.uniform(0.85, 0.99), 3))
    else:
        c.update(model=rng.choice(["hertz-mindlin", "harmonic"]), friction="smooth", rods=_log_int(rng, 500, 50000),
                 squeeze=round(rng.uniform(0.9, 0.995), 3))
    return c


# ---------------------------------------------------------------------------
# Inputs.
# ---------------------------------------------------------------------------
def _packing(rods, aspect, phi, squeeze, seed):
    """Rods of diameter 1 / aspect at volume fraction phi, no two closer than
    squeeze x their diameter; boxes too narrow for the device generator come
    from the host one."""
    d = 1.0 / aspect
    side = scene.box_side(rods, 1.0, d, phi)
    make = scene.make_rods_device if side >= 3.0 * (1.0 + d) else scene.make_rods
    sc = make(rods, 1.0, squeeze * d, side=side, seed=seed, max_attempts=20000)
    m = sc["n"]
    sc["radius"] = np.full(m, 0.5 * d)
    # unit density; mass and inertia of the cylinder part, as the scene
    # generator has them
    r = 0.5 * d
    mass = math.pi * r * r
    sc["mass"] = np.full(m, mass)
    sc["inertia"] = np.tile([mass * (3.0 * r * r + 1.0) / 12.0, 0.5 * mass * r * r, mass * (3.0 * r * r + 1.0) / 12.0], (m, 1))
    return sc


def _config(model, mu, friction, sc, dt=None, warm="cache"):
    kw = dict(model=model, dt=dt or DT[model], gravity=(0.0, 0.0, 0.0), lin_damp=0.0, ang_damp=0.0)
    if model == "nsc":
        kw.update(nsc_mu=mu, nsc_omega=1.0, nsc_tol=1e-6, nsc_velocity_iters=500, nsc_warm_start=warm)
    elif model == "harmonic":
        kw.update(soft_mu=mu, soft_friction_mode=friction, soft_damping=0.05)
    else:
        kw.update(hm_youngs_modulus=1e5, hm_poisson_ratio=0.3, hm_restitution=0.5, hm_friction=mu)
    kw.update(scene.pbc_kwargs(sc))
    return kw


def _case_scene(case, seed):
    sc = _packing(case["rods"], case["aspect"], case["phi"], case["squeeze"], 1 + seed)
    big = case["model"] == "hertz-mindlin" and case["rods"] >= 500000
    kw = _config(case["model"], case["mu"], case["friction"], sc, dt=2e-5 if big else None)
    if big:
        kw.update(hm_youngs_modulus=1e6, hm_restitution=0.3)
    return kw, sc


def _members(case, seed):
    """(model, config, scene) of a batch's members: rod counts log-uniform,
    aspect ratios 5 / 10 / 20 / 40, friction U[0, 1] (drawn from the case's
    own number: another seed gives other packings of the same sizes)."""
    rng = np.random.default_rng(case["sweep"])
    out = []
    for k in range(case["members"]):
        n = int(round(math.exp(rng.uniform(math.log(case["rods_lo"]), math.log(case["rods_hi"])))))
        ar = int(rng.choice([5, 10, 20, 40]))
        phi = float(min(rng.uniform(0.05, 0.25), scene.rsa_phi_max(ar)))
        mu = float(rng.uniform(0.0, 1.0))
        model = "hertz-mindlin" if case["soft_half"] and k % 2 == 0 else "nsc"
        sc = _packing(n, ar, phi, 0.995, 64 * (1 + seed) + k)
        warm = "mlp" if case["learned"] and model == "nsc" else "cache"
        out.append((model, _config(model, mu, "smooth", sc, warm=warm), sc))
    return out


def _network(seed):
    """Parameters of a warm-start network as a program holds them: seeded
    weights whose predicted impulse changes are a few per mille of a rod's
    momentum."""
    rng = np.random.default_rng(7 + seed)
    w = [rng.uniform(-1, 1, (o, i)) * math.sqrt(6.0 / i) for o, i in ((128, 8), (128, 128), (128, 128), (3, 128))]
    p = []
    for k in range(4):
        p += [w[k].ravel() * (0.1 if k == 3 else 1.0), np.zeros(w[k].shape[0])]
    p += [np.zeros(8), np.array([1e3, 10, 10, 10, 1e5, 1e5, 1e5, 1.0]), np.full(3, 1e-7)]
    return np.concatenate(p).astype(np.float32)


def _records(case, seed):
    """Recorded contacts: features in the units the step writes them (gap,
    three relative velocities, previous impulses, degree) and converged
    impulses that follow from them with some noise."""
    rng = np.random.default_rng(11 + seed)
    n = case["records"]
    f = np.empty((n, 8))
    f[:, 0] = -np.abs(rng.normal(0, 2e-4, n))
    f[:, 1:4] = rng.normal(0, 0.08, (n, 3))
    f[:, 4] = np.where(rng.random(n) < 0.7, np.abs(rng.normal(0, 5e-5, n)), 0.0)
    f[:, 5:7] = f[:, 4:5] * rng.uniform(-0.4, 0.4, (n, 2))
    f[:, 7] = rng.integers(0, 5, n)
    ln = np.maximum(0.0, f[:, 4] - 4e-4 * f[:, 1] / (1 + f[:, 7]) + rng.normal(0, 5e-6, n))
    lt = np.clip(f[:, 5:7] - 2e-4 * f[:, 2:4], -0.3 * ln[:, None], 0.3 * ln[:, None])
    return f.astype(np.float32), np.concatenate([ln[:, None], lt], 1).astype(np.float32)


def prepare(case, seed):
    if case["kind"] == "train":
        f, t = _records(case, seed)
        s = rodgpu.System(rodgpu.default_config(n_bodies=16, model="nsc"))
        return {"case": case, "sys": s, "features": f, "targets": t, "seed": seed}
    if case["kind"] == "batch":
        mem = _members(case, seed)
        b = rodgpu.Batch([rodgpu.default_config(n_bodies=sc["n"], **kw) for _, kw, sc in mem])
        for k, (_, _, sc) in enumerate(mem):
            b.set_bodies(k, sc["radius"], sc["half_height"], sc["mass"], sc["inertia"], sc["restitution"])
            b.set_state(k, sc["x"], sc["q"], sc["v"], sc["w"])
        # the network is loaded for the tuning, whose trials step with it, and
        # again for the runs that follow
        net = _network(seed) if case["learned"] else None
        if net is not None:
            b.set_mlp(net)
        b.autotune(trial_steps=5)
        if net is not None:
            b.set_mlp(net)
        soft = np.concatenate([np.full(sc["n"], m != "nsc") for m, _, sc in mem])
        state = tuple(np.concatenate([sc[k] for _, _, sc in mem]) for k in ("x", "q", "v", "w"))
        return {"case": case, "batch": b, "soft": soft, "state": state}
    kw, sc = _case_scene(case, seed)
    s = rodgpu.System(rodgpu.default_config(n_bodies=sc["n"], **kw))
    s.set_bodies(sc["radius"], sc["half_height"], sc["mass"], sc["inertia"], sc["restitution"])
    s.set_state(sc["x"], sc["q"], sc["v"], sc["w"])
    state = {"case": case, "sys": s, "scene": sc}
    if case["kind"] == "contacts":
        # the program's own contact arrays, of a fixed capacity (zero beyond
        # the contacts found)
        cap = int(3 * _contacts_estimate(case)) + 256
        state["buffers"] = {"pairs": np.zeros((cap, 2), np.int32), "geom": np.zeros((cap, 12)), "shift": np.zeros((cap, 3))}
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "train":
        s = state["sys"]
        loss = s.mlp_train(state["features"], state["targets"], epochs=case["epochs"], batch=case["minibatch"],
                           lr=1e-3, seed=3 + state["seed"])
        return {"params": s.mlp_get_params(), "loss": loss}
    if case["kind"] == "batch":
        # every call starts from the same initial conditions (a sweep's
        # trial): states up, steps, states and statistics back
        b = state["batch"]
        b.set_state_all(*state["state"])
        st = b.step(case["steps"])
        x, q, v, w = b.get_state_all()
        soft = state["soft"]
        out = {"contacts": np.array([m["contacts"] for m in st])}
        for name, rows in (("soft", soft), ("nsc", ~soft)):
            if rows.all():
                out[name] = [x, q, v, w]
            elif rows.any():
                out[name] = [x[rows], q[rows], v[rows], w[rows]]
        return out
    s, sc = state["sys"], state["scene"]
    if case["kind"] == "forces":
        s.set_state(sc["x"], sc["q"], sc["v"], sc["w"])
        f, tau, pe = s.compute_forces()
        return {"f": f, "tau": tau, "potential": pe}
    if case["kind"] == "contacts":
        s.set_state(sc["x"], sc["q"], sc["v"], sc["w"])
        out = state["buffers"]
        for buf, found in zip(out.values(), s.detect(0.0)):
            buf[:len(found)] = found
        return out
    s.set_state(sc["x"], sc["q"], sc["v"], sc["w"])
    st = s.step(case["steps"])
    out = s.get_state()
    out.update(contacts=st["contacts"], kinetic=st["kinetic_energy"])
    if case["model"] == "nsc":
        del out["f"], out["tau"]  # cleared by every step
    else:
        out["potential"] = st["potential_energy"]
    return out


def _contacts_estimate(case):
    """Touching pairs of an isotropic packing: pairs whose surfaces lie
    within the shell that the smaller generation diameter leaves (at the
    mean density; packings hold up to twice as many)."""
    d = 1.0 / case["aspect"]
    n = case["phi"] / scene.capsule_volume(1.0, d)
    shell = (1.0 - case["squeeze"]) * d + (0.005 if case["model"] == "harmonic" else 0.0)
    return 0.25 * math.pi * case["rods"] * n * shell


def work(case):
    """FP64 structure-of-arrays bytes that a pass has to move: per rod-step
    one read of the state (104 B) and the body properties (88 B) and one
    write of what changes (104 B); per contact and evaluation the pair, its
    two records and its history or row; the state sent in and read back
    once (104 B a rod each).  Operations: the rod's integrators and the contacts."""
    if case["kind"] == "train":
        rows = case["records"] // case["minibatch"] * case["minibatch"] * case["epochs"]
        return {"bytes": rows * 44.0, "flops": rows * 6.0 * 34432}
    if case["kind"] == "batch":
        mean = (case["rods_hi"] - case["rods_lo"]) / math.log(case["rods_hi"] / case["rods_lo"])
        rods = case["members"] * mean
        return {"bytes": rods * (296.0 * case["steps"] + 208.0), "flops": rods * case["steps"] * 400.0}
    n, c = case["rods"], _contacts_estimate(case)
    if case["kind"] == "forces":
        return {"bytes": n * (104.0 + 88.0 + 48.0) + c * 200.0, "flops": n * 50.0 + c * 400.0}
    if case["kind"] == "contacts":
        return {"bytes": n * (104.0 + 16.0) + c * 128.0, "flops": n * 50.0 + c * 200.0}
    per = 2 * 200.0 if case["model"] != "nsc" else 616.0 + 3 * 568.0
    frame = n * (2 * 104.0 + 48.0)
    return {"bytes": case["steps"] * (n * 296.0 + c * per) + frame, "flops": case["steps"] * (n * 400.0 + c * 1000.0)}


# ---------------------------------------------------------------------------
# The same in plain numpy, 64 bits.
# ---------------------------------------------------------------------------
def _axis(q):
    w, x, y, z = q.T
    return np.stack([2 * (x * y - w * z), 1 - 2 * (x * x + z * z), 2 * (y * z + w * x)], 1)


def _dot(a, b):
    return np.einsum("ij,ij->i", a, b)


def _image(d, side):
    return d - np.floor(d / side + 0.5) * side


def _closest(xa, ua, xb, ub, h):
    """Closest points of the segments x +- h u, as distances s, t in [0, 1]
    along them from their lower ends (Lumelsky's method)."""
    e1, e2 = 2 * h * ua, 2 * h * ub
    e12 = (xb - h * ub) - (xa - h * ua)
    d1, d2, s1, s2, r = _dot(e1, e1), _dot(e2, e2), _dot(e1, e12), _dot(e2, e12), _dot(e1, e2)
    den = d1 * d2 - r * r
    s = np.where(den == 0.0, 0.0, np.clip((s1 * d2 - s2 * r) / np.where(den == 0.0, 1.0, den), 0.0, 1.0))
    t = (s * r - s2) / d2
    u = np.clip(t, 0.0, 1.0)
    s = np.where(u != t, np.clip((u * r + s1) / d1, 0.0, 1.0), s)
    return s, u


def _candidates(x, u, side, reach):
    """Pairs a < b, sorted, whose segments come within `reach`."""
    n = len(x)
    nc = max(1, int(side / (1.0 + reach)))
    if nc < 3:
        nc = 1
    cell = np.minimum((np.mod(x / side, 1.0) * nc).astype(np.int64), nc - 1)
    cid = (cell[:, 2] * nc + cell[:, 1]) * nc + cell[:, 0]
    order = np.argsort(cid, kind="stable")
    start = np.searchsorted(cid[order], np.arange(nc ** 3 + 1))
    offs = [(0, 0, 0)] if nc == 1 else [(i, j, k) for i in (-1, 0, 1) for j in (-1, 0, 1) for k in (-1, 0, 1)
                                        if (k, j, i) >= (0, 0, 0)]
    got = []
    for c in range(nc ** 3):
        home = order[start[c]:start[c + 1]]
        if not len(home):
            continue
        ci = np.array([c % nc, c // nc % nc, c // (nc * nc)])
        for o in offs:
            m = (ci + o) % nc
            k = (m[2] * nc + m[1]) * nc + m[0]
            other = order[start[k]:start[k + 1]]
            for lo in range(0, len(home), 512):
                a = home[lo:lo + 512]
                d = _image(x[other][None] - x[a][:, None], side)
                near = np.einsum("ijk,ijk->ij", d, d) < (1.0 + reach) ** 2
                if k == c:
                    near &= a[:, None] < other[None]
                i, j = np.nonzero(near)
                if len(i):
                    d = d[i, j]
                    a, b = a[i], other[j]
                    s, t = _closest(np.zeros_like(d), u[a], d, u[b], 0.5)
                    gap = d + (t - 0.5)[:, None] * u[b] - (s - 0.5)[:, None] * u[a]
                    keep = _dot(gap, gap) < reach * reach
                    got.append(np.stack([np.minimum(a, b), np.maximum(a, b)], 1)[keep])
    p = np.concatenate(got) if got else np.zeros((0, 2), np.int64)
    return p[np.lexsort((p[:, 1], p[:, 0]))] if n else p


def _touching(x, q, p, side, surf, delta):
    """Geometry of the listed pairs closer than surf + delta."""
    a, b = p[:, 0], p[:, 1]
    u = _axis(q)
    sh = -(np.floor((x[b] - x[a]) / side + 0.5) * side)
    a1, a2 = x[a] - u[a] * 0.5, x[a] + u[a] * 0.5
    b1, b2 = x[b] - u[b] * 0.5 + sh, x[b] + u[b] * 0.5 + sh
    s, t = _closest(x[a], u[a], x[b] + sh, u[b], 0.5)
    pa, pb = a1 + (a2 - a1) * s[:, None], b1 + (b2 - b1) * t[:, None]
    diff = pb - pa
    dist = np.sqrt(_dot(diff, diff))
    hit = dist < surf + delta
    a, b, s, t, pa, pb, sh, diff, dist = (v[hit] for v in (a, b, s, t, pa, pb, sh, diff, dist))
    return dict(a=a, b=b, s=s, t=t, pa=pa, pb=pb, sh=sh, n=diff / dist[:, None], dist=dist)


def _rot_apply(q, diag, v):
    w, x, y, z = q.T
    m = np.empty((len(q), 3, 3))
    m[:, :, 0] = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y + w * z), 2 * (x * z - w * y)], 1)
    m[:, :, 1] = np.stack([2 * (x * y - w * z), 1 - 2 * (x * x + z * z), 2 * (y * z + w * x)], 1)
    m[:, :, 2] = np.stack([2 * (x * z + w * y), 2 * (y * z - w * x), 1 - 2 * (x * x + y * y)], 1)
    return np.einsum("nij,nj->ni", m, np.einsum("nij,ni->nj", m, v) * diag)


class _Plain:
    """A soft or Hertz-Mindlin system in numpy (rods of length 1)."""

    def __init__(self, kw, sc, steps):
        self.c = rodgpu.abi.config_from(rodgpu.host(), n_bodies=sc["n"], **kw)
        self.hm = kw["model"] == "hertz-mindlin"
        self.n, self.side, self.surf = sc["n"], sc["side"], float(2 * sc["radius"][0])
        self.x, self.q, self.v, self.w = (sc[k].copy() for k in ("x", "q", "v", "w"))
        self.mass, self.inertia, self.r = sc["mass"][0], sc["inertia"], float(sc["radius"][0])
        self.key, self.val, self.frame, self.now = np.zeros(0, np.int64), np.zeros((0, 3)), np.zeros(0, np.int64), 0
        self.delta = 0.0 if self.hm else self.c.soft_delta
        # no rod end moves further than this in the run (speeds of the
        # thermal draw; checked at the end)
        self.slack = 0.02 + 3.0 * steps * self.c.dt
        self.pairs = _candidates(self.x, _axis(self.q), self.side, self.surf + self.delta + self.slack)
        self.x0, self.u0 = self.x.copy(), _axis(self.q)

    def moved_too_far(self):
        dx, du = _image(self.x - self.x0, self.side), _axis(self.q) - self.u0
        return 2 * np.max(np.linalg.norm(dx, axis=1) + 0.5 * np.linalg.norm(du, axis=1)) > self.slack

    def forces(self):
        c, dt = self.c, self.c.dt
        g = _touching(self.x, self.q, self.pairs, self.side, self.surf, self.delta)
        a, b, n, dist = g["a"], g["b"], g["n"], g["dist"]
        self.now += 1
        key = a.astype(np.int64) * self.n + b
        at = np.searchsorted(self.key, key)
        known = (at < len(self.key)) & (np.append(self.key, -1)[np.minimum(at, len(self.key))] == key)
        old = np.where(known[:, None], np.concatenate([self.val, np.zeros((1, 3))])[np.where(known, at, len(self.val))], 0.0)
        ra, rb = g["pa"] - self.x[a], g["pb"] - (self.x[b] + g["sh"])
        va, vb = self.v[a] + np.cross(self.w[a], ra), self.v[b] + np.cross(self.w[b], rb)
        touched = np.ones(len(a), bool)
        add_a = add_b = 0.0
        if self.hm:
            nu, E, res = c.hm_poisson_ratio, c.hm_youngs_modulus, c.hm_restitution
            es, gs = E / (2 * (1 - nu * nu)), E / (2 * (1 + nu))
            gam = -math.log(res) / math.sqrt(math.pi ** 2 + math.log(res) ** 2) if res < 1 else 0.0
            rs, ms, pen = 0.5 * self.r, 0.5 * self.mass, self.surf - dist
            sq = np.sqrt(np.maximum(pen, 0.0))
            kn = 4.0 / 3.0 * es * math.sqrt(rs) * sq
            vr = vb - va
            vn = _dot(vr, n)
            fn = np.maximum(0.0, kn * np.maximum(pen, 0.0) * sq - gam * 2 * np.sqrt(ms * kn) * vn)
            kt = 8 * gs * math.sqrt(rs) * sq
            vt = vr - n * vn[:, None]
            xi = old + vt * dt
            ft = -xi * kt[:, None] - vt * (gam * 2 * np.sqrt(ms * kt))[:, None]
            mu = np.full(len(a), c.hm_friction)
            if c.hm_friction_static > c.hm_friction and c.hm_friction_transition_vel > 0:
                mu = mu + (c.hm_friction_static - c.hm_friction) * np.exp(-np.linalg.norm(vt, axis=1) / c.hm_friction_transition_vel)
            m, most = np.linalg.norm(ft, axis=1), mu * fn
            slip = (m > most) & (m > 1e-10)
            ft = np.where(slip[:, None], ft * (most / np.where(m > 0, m, 1.0))[:, None], ft)
            new = np.where((slip & (kt > 1e-10))[:, None], ft / -np.where(kt > 0, kt, 1.0)[:, None], xi)
            wr = self.w[a] - self.w[b]
            wm = np.linalg.norm(wr, axis=1)
            if c.hm_enable_rolling:
                roll = np.where((wm >= 1e-10)[:, None], wr / np.where(wm > 0, wm, 1.0)[:, None], 0.0) * (-c.hm_rolling_friction * rs * fn)[:, None]
                add_a, add_b = 0.5 * roll, -0.5 * roll
            fb = n * fn[:, None] + ft
            fa = -fb
            self.pe = float(np.sum(8.0 / 15.0 * es * math.sqrt(rs) * np.maximum(pen, 0.0) ** 2.5))
        else:
            k1 = 15.0 / c.soft_delta
            e = np.exp(np.minimum(k1 * (self.surf - dist), 60.0))
            soft = dist > self.surf - c.soft_delta
            grad = np.where(soft, -2 / k1 ** 2 * np.log(1 + e) * e / (1 + e), -2 * (self.surf - dist))
            self.pe = float(np.sum(c.soft_k_scaler * np.where(soft, (np.log(1 + e) / k1) ** 2, (self.surf - dist) ** 2)))
            fa = n * (c.soft_k_scaler * grad)[:, None]
            fb = -fa
            vr = va - vb
            vn = _dot(vr, n)
            if c.soft_damping > 1e-9:
                fa, fb = fa - n * (c.soft_damping * vn)[:, None], fb + n * (c.soft_damping * vn)[:, None]
            fm, vt = np.linalg.norm(fa, axis=1), vr - n * vn[:, None]
            vm = np.linalg.norm(vt, axis=1)
            moving, safe = vm >= 1e-10, np.where(vm > 0, vm, 1.0)
            new = np.zeros((len(a), 3))
            touched = np.zeros(len(a), bool)
            if c.soft_friction_mode == rodgpu.FRICTION["cundall"]:
                ft = old - vt * (c.soft_kt * dt)
                ft = ft - n * _dot(ft, n)[:, None]
                m, lim = np.linalg.norm(ft, axis=1), c.soft_mu * fm
                fr = np.where((m > lim)[:, None], np.where((m > 1e-8)[:, None], ft * (lim / np.where(m > 0, m, 1.0))[:, None], 0.0), ft)
                new, touched = fr, moving
            elif c.soft_friction_mode == rodgpu.FRICTION["karnopp"]:
                stop = vt * (-(0.5 * self.mass) / dt)
                m, most = np.linalg.norm(stop, axis=1), c.soft_mu_static * fm
                held = np.where((m <= most)[:, None], stop, np.where((m > 1e-12)[:, None], stop * (most / np.where(m > 0, m, 1.0))[:, None], 0.0))
                fr = np.where((vm < c.soft_vel_deadband)[:, None], held, -vt / safe[:, None] * (c.soft_mu * fm)[:, None])
            else:
                gam = np.where(vm > c.soft_nu, 1.0, 2 / (1 + np.exp(-15.0 / c.soft_nu * vm)) - 1)
                mu = c.soft_mu + (max(c.soft_mu_static - c.soft_mu, 0.0)) * np.exp(-vm / c.soft_nu)
                fr = -vt / safe[:, None] * (mu * gam * fm)[:, None]
            fr = np.where(moving[:, None], fr, 0.0)
            fa, fb = fa + fr, fb - fr
        f, tau = np.zeros((self.n, 3)), np.zeros((self.n, 3))
        for idx, force, arm, more in ((a, fa, ra, add_a), (b, fb, rb, add_b)):
            np.add.at(f, idx, force)
            np.add.at(tau, idx, np.cross(arm, force) + more)
        keep = np.ones(len(self.key), bool) if not self.hm else ~((self.now - self.frame > 4) | (self.frame == 0))
        keep[at[known & touched]] = False
        k2 = np.concatenate([self.key[keep], key[touched]])
        o = np.argsort(k2)
        self.key = k2[o]
        self.val = np.concatenate([self.val[keep], new[touched]])[o]
        self.frame = np.concatenate([self.frame[keep], np.full(int(touched.sum()), self.now)])[o]
        self.contacts = len(a)
        return f, tau

    def accel(self, f, tau):
        gyro = np.cross(self.w, _rot_apply(self.q, self.inertia, self.w))
        return f / self.mass, _rot_apply(self.q, 1.0 / self.inertia, tau - gyro)

    def step(self):
        dt = self.c.dt
        lo = -0.5 * self.side
        al, aa = self.accel(*self.forces())
        self.v, self.w = self.v + 0.5 * dt * al, self.w + 0.5 * dt * aa
        x = self.x + self.v * dt
        self.x = np.where(x < lo, x + self.side, np.where(x >= lo + self.side, x - self.side, x))
        wl = np.linalg.norm(self.w, axis=1)
        turn = wl > 1e-8
        ax = self.w / np.where(turn, wl, 1.0)[:, None]
        half = 0.5 * wl * dt
        rw, rv = np.cos(half), ax * np.sin(half)[:, None]
        qw, qv = self.q[:, 0], self.q[:, 1:]
        p = np.concatenate([(rw * qw - _dot(rv, qv))[:, None], rw[:, None] * qv + qw[:, None] * rv + np.cross(rv, qv)], 1)
        self.q = np.where(turn[:, None], p / np.linalg.norm(p, axis=1)[:, None], self.q)
        self.f, self.tau = self.forces()
        al, aa = self.accel(self.f, self.tau)
        self.v, self.w = self.v + 0.5 * dt * al, self.w + 0.5 * dt * aa
        wl = np.linalg.norm(self.w, axis=1)
        self.w = np.where((wl > self.c.w_max)[:, None], self.w * (self.c.w_max / np.where(wl > 0, wl, 1.0))[:, None], self.w)


def exact(case, seed):
    """What run() returns in numpy, 64 bits.  PSOR has none: it stops at a
    residual, and what it then holds depends on its start and its order; nor
    has training, whose weights follow from roundings to bfloat16."""
    if case["kind"] == "train":
        return None
    if case["kind"] == "batch":
        if not case["soft_half"]:
            return None
        parts, contacts, spent = [], [], 0
        for model, kw, sc in _members(case, seed):
            spent += sc["n"] if model != "nsc" else 0
            if model == "nsc":
                contacts.append(0)
                continue
            if spent > 40000:
                return None
            p = _Plain(kw, sc, case["steps"])
            for _ in range(case["steps"]):
                p.step()
            if p.moved_too_far():
                return None
            parts.append((p.x, p.q, p.v, p.w))
            contacts.append(p.contacts)
        return {"contacts": None, "soft": [np.concatenate(v) for v in zip(*parts)], "nsc": [None] * 4}
    if case["kind"] == "contacts":
        if case["rods"] > 60000:
            return None
        _, sc = _case_scene(case, seed)
        surf = float(2 * sc["radius"][0])
        g = _touching(sc["x"], sc["q"], _candidates(sc["x"], _axis(sc["q"]), sc["side"], surf + 1e-6), sc["side"], surf, 0.0)
        s, t, eps = g["s"], g["t"], 1e-6
        end_s, end_t = (s < eps) | (s > 1 - eps), (t < eps) | (t > 1 - eps)
        kind = np.where(((s < eps) & (t < eps)) | ((s > 1 - eps) & (t > 1 - eps)), 0.0, np.where(end_s | end_t, 1.0, 2.0))
        m = len(s)
        geom = np.concatenate([g["pa"], g["pb"], g["n"], g["dist"][:, None], np.full((m, 1), surf), kind[:, None]], 1)
        cap = int(3 * _contacts_estimate(case)) + 256
        out = (np.stack([g["a"], g["b"]], 1).astype(np.int32), geom, g["sh"])
        return {k: np.concatenate([a, np.zeros((cap - m, a.shape[1]), a.dtype)]) for k, a in zip(("pairs", "geom", "shift"), out)}
    if case["model"] == "nsc":
        return None
    steps = case.get("steps", 0)
    if case["rods"] > 60000 or case["rods"] * steps > 2500000:
        return None
    kw, sc = _case_scene(case, seed)
    p = _Plain(kw, sc, steps)
    if case["kind"] == "forces":
        f, tau = p.forces()
        return {"f": f, "tau": tau, "potential": p.pe}
    for _ in range(steps):
        p.step()
    if p.moved_too_far():
        return None
    kin = 0.5 * p.mass * np.sum(p.v * p.v) + 0.5 * np.sum(p.w * _rot_apply(p.q, p.inertia, p.w))
    return {"x": p.x, "q": p.q, "v": p.v, "w": p.w, "f": p.f, "tau": p.tau, "contacts": p.contacts, "kinetic": float(kin),
            "potential": p.pe}
