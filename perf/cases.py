"""Performance cases of the GB300 hackcode1 library, through its Python entry points.

A case is one call that a user's program makes again and again: a force
evaluation of host positions (hackforce's contract), a leapfrog step, forces
at test points, an ensemble's step, the training of the opening network.
Sizes run from hackcode1's default of 128 bodies to the 2^24-body galaxy.

The walk's sums are 32-bit floats (stored in 64-bit arrays); the cases hand
accelerations, potentials and what follows from them on as 32-bit, the
precision that they carry.  exact() is an octree code in plain 64-bit torch.
"""
import math

import numpy as np
import torch

from nemo_gb300 import hackcode as hc

GUARD = 256          # bodies of the per-evaluation guard's sample


def listed():
    return [
        # hackcode1's defaults: nbody=128, tol=1, eps=0.05, no quadrupoles -- pure latency
        {"name": "host_128", "kind": "evaluate", "model": "plummer", "n": 128, "criterion": "body", "theta": 1.0,
         "eps": 0.05, "quad": False},
        # the CPU-size configuration: Plummer 4096, tol=0.7, eps=0.05, freq=32, snapshot each step
        {"name": "step_4096", "kind": "step", "model": "plummer", "n": 4096, "theta": 0.7, "eps": 0.05,
         "quad": False, "dt": 0.03125},
        # an odd size, quadrupoles, per-body interaction counts kept (the parity checks' way of calling)
        {"name": "counts_50021", "kind": "evaluate", "model": "plummer", "n": 50021, "criterion": "body",
         "theta": 0.6, "eps": 0.02, "quad": True, "counts": True},
        # hackforce test=: forces at points that are not in the tree
        {"name": "points_65537", "kind": "points", "model": "plummer", "n": 131072, "points": 65537, "theta": 0.6,
         "eps": 0.02, "quad": True},
        # treecode1's default radii in the group walk, a cuspy model, no quadrupoles
        {"name": "barnes_262143", "kind": "evaluate", "model": "hernquist", "n": 262143, "criterion": "barnes",
         "theta": 0.8, "eps": 0.01, "quad": False},
        # the benchmark's system with the reference's rule: Plummer 2^20, tol=0.5, eps=0.01, quadrupoles
        {"name": "body_1m", "kind": "evaluate", "model": "plummer", "n": 1048576, "criterion": "body", "theta": 0.5,
         "eps": 0.01, "quad": True},
        # the same system with the error rule and its guard, at the fixed rule's RMS error
        {"name": "error_1m", "kind": "evaluate", "model": "plummer", "n": 1048576, "criterion": "error",
         "theta": 0.053, "eps": 0.01, "quad": True, "guard": True},
        # the same system with the learned criterion: the headline
        {"name": "learned_1m", "kind": "evaluate", "model": "plummer", "n": 1048576, "criterion": "learned",
         "theta": 0.043, "eps": 0.01, "quad": True, "guard": True},
        # the Hernquist sphere of the large evaluation: 2^22 bodies, eps=0.005, error rule
        {"name": "hernquist_4m", "kind": "evaluate", "model": "hernquist", "n": 4194304, "criterion": "error",
         "theta": 0.3, "eps": 0.005, "quad": True, "guard": True},
        # the largest: disk galaxy of 2^24 bodies
        {"name": "galaxy_16m", "kind": "evaluate", "model": "galaxy", "n": 16777216, "criterion": "error",
         "theta": 0.3, "eps": 0.01, "quad": True, "guard": True},
        # independent Plummer spheres of uneven size, direct sums up to 1024 bodies
        {"name": "ensemble_96", "kind": "ensemble", "nsys": 96, "nmin": 64, "nmax": 16384, "theta": 0.6,
         "eps": 0.02, "quad": False, "dt": 0.00390625},
        # training of the opening network: one epoch of Adam over labelled samples
        {"name": "train_262144", "kind": "train", "samples": 262144, "batch": 4096, "lr": 0.002},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["evaluate"] * 6 + ["step", "points", "ensemble", "train"])
    if kind == "train":
        return {"kind": "train", "samples": size(5000, 400000), "batch": rng.choice([1024, 4096, 8192]),
                "lr": rng.choice([0.001, 0.002])}
    quad = rng.random() < 0.5
    eps = rng.choice([0.005, 0.01, 0.02, 0.05])
    if kind == "ensemble":
        return {"kind": "ensemble", "nsys": rng.randint(3, 160), "nmin": 64, "nmax": size(256, 16384),
                "theta": rng.choice([0.5, 0.6, 0.7]), "eps": eps, "quad": quad, "dt": 0.00390625}
    model = rng.choice(["plummer", "plummer", "hernquist", "galaxy"])
    if kind == "step":
        return {"kind": "step", "model": model, "n": size(100, 300000), "theta": rng.choice([0.6, 0.7, 0.8, 1.0]),
                "eps": eps, "quad": quad, "dt": 0.0078125}
    if kind == "points":
        return {"kind": "points", "model": model, "n": size(1000, 500000), "points": size(100, 100000),
                "theta": rng.choice([0.5, 0.6, 0.8]), "eps": eps, "quad": quad}
    criterion = rng.choice(["body", "body", "error", "error", "learned", "group", "barnes"])
    c = {"kind": "evaluate", "model": model, "n": size(100, 3000000), "criterion": criterion, "eps": eps,
         "quad": quad}
    if criterion in ("error", "learned"):
        c.update(theta=rng.choice([0.05, 0.1, 0.2]), guard=rng.random() < 0.7 and c["n"] > 4 * GUARD)
    else:
        c.update(theta=rng.choice([0.5, 0.6, 0.7, 0.8]))
        if criterion == "body" and c["n"] < 200000:
            c.update(counts=rng.random() < 0.5)
    return c


# ---------------------------------------------------------------- inputs

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rand(n, g):
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64)


def _isotropic(r, g):
    """Points at radius r in random directions."""
    z = 2.0 * _rand(len(r), g) - 1.0
    p = 2.0 * math.pi * _rand(len(r), g)
    s = torch.sqrt(torch.clamp(1.0 - z * z, min=0.0))
    return torch.stack([r * s * torch.cos(p), r * s * torch.sin(p), r * z], 1)


def _invert(x, cdf, u):
    """x at which the increasing table cdf (0..1) takes the value u."""
    i = torch.clamp(torch.searchsorted(cdf, u), 1, len(cdf) - 1)
    w = (u - cdf[i - 1]) / torch.clamp(cdf[i] - cdf[i - 1], min=1e-300)
    return x[i - 1] + torch.clamp(w, 0.0, 1.0) * (x[i] - x[i - 1])


def _nfw_mass(r, rs):
    return torch.log1p(r / rs) - (r / rs) / (1.0 + r / rs)


def _model(model, n, g):
    """(mass, position, velocity, acceleration of the smooth model), FP64 on the GPU."""
    if model == "plummer":                       # virial units, as mkplummer's
        a = 3.0 * math.pi / 16.0
        u = 0.999 * _rand(n, g) + 1e-12
        r = a / torch.sqrt(u ** (-2.0 / 3.0) - 1.0)
        pos = _isotropic(r, g)
        q = torch.linspace(0.0, 1.0, 4097, device="cuda", dtype=torch.float64)
        f = q * q * (1.0 - q * q) ** 3.5
        cdf = torch.cumsum(f, 0)
        v = _invert(q, cdf / cdf[-1], _rand(n, g)) * math.sqrt(2.0) * (r * r + a * a) ** -0.25
        return (torch.full((n,), 1.0 / n, device="cuda", dtype=torch.float64), pos, _isotropic(v, g),
                -pos * ((r * r + a * a) ** -1.5)[:, None])
    if model == "hernquist":                     # G = M = a = 1, truncated at 100
        s = torch.sqrt(_rand(n, g)) * (100.0 / 101.0)
        r = torch.clamp(s / (1.0 - s), min=1e-6)
        pos = _isotropic(r, g)
        mt = (100.0 / 101.0) ** 2
        return (torch.full((n,), mt / n, device="cuda", dtype=torch.float64), pos,
                _isotropic(0.3 * torch.ones_like(r), g), -pos / (r * (1.0 + r) ** 2)[:, None])
    # exponential disk (a quarter of the bodies), Hernquist bulge (1/16), NFW halo: the composite galaxy's masses
    nd, nb = max(1, n // 4), max(1, n // 16)
    nh = n - nd - nb
    R = -torch.log(torch.clamp(_rand(nd, g) * _rand(nd, g), min=1e-12))
    R = torch.clamp(R, max=15.0)
    p = 2.0 * math.pi * _rand(nd, g)
    disk = torch.stack([R * torch.cos(p), R * torch.sin(p),
                        0.1 * torch.atanh(torch.clamp(2.0 * _rand(nd, g) - 1.0, -0.999999, 0.999999))], 1)
    s = torch.sqrt(_rand(nb, g)) * 0.99
    bulge = _isotropic(torch.clamp(0.2 * s / (1.0 - s), min=1e-6), g)
    x = torch.logspace(-5, math.log10(30.0), 4097, device="cuda", dtype=torch.float64)
    cdf = _nfw_mass(x, 3.0) / _nfw_mass(x[-1], 3.0)
    halo = _isotropic(_invert(x, cdf, _rand(nh, g)), g)
    pos = torch.cat([disk, bulge, halo])
    mass = torch.cat([torch.full((k,), m / k, device="cuda", dtype=torch.float64)
                      for k, m in ((nd, 0.1), (nb, 0.033), (nh, 1.0))])
    r = torch.clamp(torch.linalg.vector_norm(pos, dim=1), min=1e-6)
    inside = 0.1 * (1.0 - (1.0 + r) * torch.exp(-r)) + 0.033 * (r / (r + 0.2)) ** 2 + \
        _nfw_mass(torch.clamp(r, max=30.0), 3.0) / _nfw_mass(torch.tensor(30.0, device="cuda"), 3.0)
    vel = torch.stack([-pos[:, 1], pos[:, 0], torch.zeros_like(r)], 1) * (torch.sqrt(inside / r) / r)[:, None]
    return mass, pos, vel, -pos * (inside / r ** 3)[:, None]


def _bodies(case, seed):
    g = _gen(seed)
    m, x, v, a = _model(case["model"], case["n"], g)
    return m, x, v, a, g


def _network():
    """Weights of an opening network, as a program loads them from a file: the logit falls with the cell's
    error proxy (feature 3), with small contributions of the other features."""
    r = np.random.default_rng(12)
    w1, w2, w3 = r.normal(0, 0.15, (64, 12)), r.normal(0, 0.06, (64, 64)), r.normal(0, 0.03, 64)
    w1[0], w1[1] = 0.0, 0.0
    w1[0, 3], w1[1, 3] = 2.0, -2.0               # silu(z) - silu(-z) = z
    w2[0, :2], w2[1, :2] = (1.0, -1.0), (-1.0, 1.0)
    w3[:2] = (-2.0, 2.0)
    b1, b2 = r.normal(0, 0.05, 64), r.normal(0, 0.05, 64)
    return np.concatenate([w1.ravel(), b1, w2.ravel(), b2, w3, [1.0]]).astype(np.float32)


def _pinned(t):
    return torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t)


def _samples(case, seed):
    """Feature rows and labels like the label walk's: a smooth rule with noise."""
    r = np.random.default_rng(seed)
    x = np.clip(r.normal(0.0, 1.2, (case["samples"], 12)), -8, 8).astype(np.float32)
    z = 2.0 - 3.0 * x[:, 3] + x[:, 1] * x[:, 6] - 0.5 * x[:, 11] + r.normal(0, 0.7, case["samples"])
    return x, (z > 0).astype(np.float32)


def _sizes(case):
    r = np.random.default_rng(case["nsys"])      # the case's own: every seed has the same systems
    return np.exp(r.uniform(math.log(case["nmin"]), math.log(case["nmax"] + 1), case["nsys"])).astype(np.int64)


def _spheres(case, seed):
    """Concatenated Plummer spheres: (counts, mass, position, velocity)."""
    counts, g = _sizes(case), _gen(seed)
    parts = [_model("plummer", int(k), g)[:3] for k in counts]
    return (counts,) + tuple(torch.cat([p[i] for p in parts]) for i in range(3))


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "k": 0}
    if kind == "train":
        x, y = _samples(case, seed)
        s["ctx"] = hc.Context(1024)
        s["ctx"].learn_load_samples(x, y)
        return s
    if kind == "ensemble":
        counts, m, x, v = _spheres(case, seed)
        e = hc.Ensemble(counts, tol=case["theta"], eps=case["eps"], usequad=case["quad"], direct_max=1024)
        e.upload(m.cpu().numpy(), torch.stack([x, v], 1).cpu().numpy())
        s["ens"] = e
        return s
    m, x, v, a, g = _bodies(case, seed)
    crit = case.get("criterion", "body")
    ctx = hc.Context(case["n"], tol=case["theta"] if crit == "body" else 0.5, eps=case["eps"],
                     usequad=case["quad"], count_per_body=bool(case.get("counts")))
    ctx.upload(m.cpu().numpy(), torch.stack([x, v], 1).cpu().numpy())
    s["ctx"] = ctx
    if kind == "points":
        y = _model(case["model"], case["points"], g)[1]
        s["points"] = y.cpu().numpy()
        ctx.build_tree()
        return s
    if kind == "step":
        return s
    if crit != "body":
        ctx.set_criterion(crit, case["theta"])
    if crit == "learned":
        ctx.learn_params(_network())
        ctx.learn_band(0.5, 16.0)
    if case.get("guard"):
        ctx.set_guard(GUARD, rms_max=0.02)
    s["pos"], s["prev"] = _pinned(x), _pinned(a)
    s["acc"], s["phi"] = torch.empty_like(s["pos"], pin_memory=True), torch.empty(case["n"], dtype=torch.float64,
                                                                                  pin_memory=True)
    return s


# ---------------------------------------------------------------- one pass

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "train":
        ctx = s["ctx"]
        ctx.learn_init(5)
        loss = ctx.learn_train(epochs=1, batch=case["batch"], lr=case["lr"], seed=3)
        return {"params": ctx.learn_params(), "loss": np.float32(loss)}
    if kind == "ensemble":
        s["ens"].step(case["dt"], s["k"])
        s["k"] += 1
        ph, a, p = s["ens"].download()
        return {"phase": ph.astype(np.float32), "acc": a.astype(np.float32), "phi": p.astype(np.float32)}
    ctx = s["ctx"]
    if kind == "points":
        a, p = ctx.forces_at(s["points"])
        return {"acc": a.astype(np.float32), "phi": p.astype(np.float32)}
    if kind == "step":
        d, ph, a, p = ctx.step(case["dt"], s["k"], snapshot=True)
        s["k"] += 1
        return {"phase": ph.astype(np.float32), "acc": a.astype(np.float32), "phi": p.astype(np.float32),
                "n2b": int(d.n2b), "nbc": int(d.nbc)}
    prev = s["prev"].data_ptr() if case["criterion"] in ("error", "learned") else None
    ctx.evaluate_host_ptr(s["pos"].data_ptr(), prev, s["acc"].data_ptr(), s["phi"].data_ptr())
    if case["n"] <= 65536:
        out = {"acc": s["acc"].numpy().astype(np.float32), "phi": s["phi"].numpy().astype(np.float32)}
    else:                                        # a torch program carries on with them on the GPU
        out = {"acc": s["acc"].cuda().float(), "phi": s["phi"].cuda().float()}
    if case.get("counts"):
        out["n2b"], out["nbc"] = ctx.body_counts()
    return out


def _terms(n, theta):
    """Interactions per body of an opening angle theta, about."""
    return min(float(n), 2270.0 * (0.5 / theta) ** 2.5 * max(1.0, math.log2(n) - 6.0) / 14.0)


def work(case):
    kind = case["kind"]
    if kind == "train":
        n = case["samples"]
        return {"bytes": 56.0 * n + 8.0 * 5057, "flops": 6.0 * 4928 * n}
    per = 59.0 if case["quad"] else 20.0
    if kind == "ensemble":
        flops = by = 0.0
        for k in _sizes(case):
            flops += k * (20.0 * k if k <= 1024 else per * _terms(k, case["theta"]))
            by += 88.0 * k + 80.0 * k
        return {"bytes": float(by), "flops": float(flops)}
    n = case["n"]
    if kind == "points":
        return {"bytes": 56.0 * case["points"] + 32.0 * n, "flops": case["points"] * per * _terms(n, case["theta"])}
    theta = case["theta"] if case.get("criterion", "body") not in ("error", "learned") else \
        0.5 * (case["theta"] / 0.05) ** 0.2
    return {"bytes": (64.0 if kind == "evaluate" else 144.0) * n, "flops": n * per * _terms(n, theta)}


# ---------------------------------------------------------------- 64-bit values

def _root_box(x):
    """expandbox over the bodies in order, from hackcode1's first box."""
    p = x.cpu().numpy()
    lo, size = np.full(3, -2.0), 4.0
    while True:
        t = (p - lo) / size
        out = np.flatnonzero(((t < 0.0) | (t >= 1.0)).any(1))
        if not len(out):
            return lo, size
        q = p[out[0]]
        while True:
            t = (q - lo) / size
            if ((t >= 0.0) & (t < 1.0)).all():
                break
            mid = lo + 0.5 * size
            lo, size = np.where(q < mid, lo - size, lo), 2.0 * size


class _Octree:
    """Cells of two or more bodies (no leaf buckets), breadth first; moments in 64 bits."""

    def __init__(self, m, x):
        lo, size = _root_box(x)
        self.size = size
        lo = torch.tensor(lo, device="cuda")
        ic = torch.floor((x - lo) / size * 2.0 ** 30).to(torch.int64)
        key = torch.zeros(len(x), dtype=torch.int64, device="cuda")
        for b in range(20, -1, -1):
            for d in range(3):
                key = (key << 1) | ((ic[:, d] >> (b + 9)) & 1)
        key, self.order = torch.sort(key)
        if len(key) > 1 and bool((key[1:] == key[:-1]).any()):
            raise ValueError("bodies closer than the key's 21 bits")
        self.m, self.x = m[self.order], x[self.order]
        n = len(x)
        dev = x.device
        idx = torch.arange(n, device=dev)
        levels = []                              # per level: first body, bodies, parent (node number)
        first, count = torch.zeros(1, dtype=torch.int64, device=dev), torch.tensor([n], device=dev)
        parent, base, level = torch.tensor([-1], device=dev), 0, 0
        while len(first):
            levels.append((first, count, parent))
            cell = torch.full((n,), -1, dtype=torch.int64, device=dev)
            big = torch.nonzero(count > 1).flatten()
            if not len(big):
                break
            span = torch.repeat_interleave(big, count[big])
            at = idx[:len(span)] - torch.repeat_interleave(torch.cumsum(count[big], 0) - count[big], count[big])
            cell[first[span] + at] = span + base
            level += 1
            if level > 21:
                raise ValueError("deeper than the key")
            pre = key >> (3 * (21 - level))
            new = torch.ones(n, dtype=torch.bool, device=dev)
            new[1:] = pre[1:] != pre[:-1]
            starts = torch.nonzero(new).flatten()
            counts = torch.diff(starts, append=torch.tensor([n], device=dev))
            keep = cell[starts] >= 0
            base += len(first)
            first, count, parent = starts[keep], counts[keep], cell[starts[keep]]
        self.first, self.count, self.parent = (torch.cat([v[i] for v in levels]) for i in range(3))
        self.depth = torch.cat([torch.full((len(v[0]),), i, dtype=torch.int64, device=dev)
                                for i, v in enumerate(levels)])
        k = len(self.first)
        self.body = self.count == 1
        self.child = torch.full((k,), k, dtype=torch.int64, device=dev)
        self.child.scatter_reduce_(0, self.parent[1:], torch.arange(1, k, device=dev), "amin")
        self.nchild = torch.bincount(self.parent[1:], minlength=k)
        self.m_ = torch.where(self.body, self.m[self.first], 0.0)
        self.c_ = torch.where(self.body[:, None], self.x[self.first], 0.0)
        self.q_ = torch.zeros(k, 3, 3, dtype=torch.float64, device=dev)
        self.b_ = torch.zeros(k, dtype=torch.float64, device=dev)
        eye = torch.eye(3, dtype=torch.float64, device=dev)
        ends = np.cumsum([len(v[0]) for v in levels])
        for i in range(len(levels) - 1, 0, -1):
            c = torch.arange(int(ends[i - 1]), int(ends[i]), device=dev)
            p = self.parent[c]
            self.m_.index_add_(0, p, self.m_[c])
            self.c_.index_add_(0, p, self.m_[c, None] * self.c_[c])
            up = torch.unique(p)
            self.c_[up] /= self.m_[up, None]
            d = self.c_[c] - self.c_[p]
            r2 = (d * d).sum(1)
            self.q_.index_add_(0, p, self.q_[c] + self.m_[c, None, None] *
                               (3.0 * d[:, :, None] * d[:, None, :] - r2[:, None, None] * eye))
            self.b_.scatter_reduce_(0, p, torch.sqrt(r2) + self.b_[c], "amax")
        self.s2 = (size * 0.5 ** self.depth.to(torch.float64)) ** 2
        sh = 30 - self.depth
        corner = (ic[self.order][self.first] >> sh[:, None]) << sh[:, None]
        self.centre = lo + corner.to(torch.float64) * (size * 2.0 ** -30) + 0.5 * torch.sqrt(self.s2)[:, None]

    def groups(self, gmax):
        """Walk groups: cells of at most gmax bodies whose parent has more, siblings packed: (first, count)."""
        first, count, parent, child, nchild = (v.cpu().numpy() for v in (self.first, self.count, self.parent,
                                                                         self.child, self.nchild))
        if count[0] <= gmax:
            return self.first[:1], self.count[:1]
        got = []
        for k in np.flatnonzero(count > gmax):
            cur = None
            for c in range(child[k], child[k] + nchild[k]):
                if cur is not None and (count[c] > gmax or cur[1] + count[c] > gmax):
                    got.append(cur)
                    cur = None
                if count[c] > gmax:
                    continue
                cur = (first[c], count[c]) if cur is None else (cur[0], cur[1] + count[c])
            if cur is not None:
                got.append(cur)
        a = torch.tensor(np.array(sorted(got)), device="cuda")
        return a[:, 0].contiguous(), a[:, 1].contiguous()


def _walk(t, x, lo, hi, first, count, accept, eps, quad, own):
    """Forces at the points x[first : first + count] of each target box [lo, hi]; own: the points are the bodies."""
    acc, phi = torch.zeros_like(x), torch.zeros(len(x), dtype=torch.float64, device="cuda")
    chunk = max(1, int(2.0e4 / max(1.0, float(count.double().mean()))))
    for t0 in range(0, len(lo), chunk):
        t1 = min(len(lo), t0 + chunk)
        tgt = torch.arange(t0, t1, device="cuda")
        node = torch.zeros_like(tgt)
        b0, b1 = int(first[t0]), int(first[t1 - 1] + count[t1 - 1])
        while len(tgt):
            c = t.c_[node]
            d = torch.clamp(torch.maximum(lo[tgt] - c, c - hi[tgt]), min=0.0)
            take = t.body[node] | accept(t, node, tgt, (d * d).sum(1))
            a_t, a_n = tgt[take], node[take]
            # one row per (point, node); rows of one point are brought together
            rep = count[a_t]
            row = torch.repeat_interleave(torch.arange(len(a_t), device="cuda"), rep)
            pt = first[a_t[row]] + torch.arange(len(row), device="cuda") - \
                torch.repeat_interleave(torch.cumsum(rep, 0) - rep, rep)
            nd = a_n[row]
            if own:
                keep = ~(t.body[nd] & (t.first[nd] == pt))
                pt, nd = pt[keep], nd[keep]
            pt, o = torch.sort(pt, stable=True)
            nd = nd[o]
            dr = t.c_[nd] - x[pt]
            r2 = (dr * dr).sum(1) + eps * eps
            ri = torch.rsqrt(r2)
            mr = t.m_[nd] * ri
            p, f = -mr, (mr / r2)[:, None] * dr
            if quad:
                qd = (t.q_[nd] @ dr[:, :, None])[:, :, 0]
                r5 = ri / (r2 * r2)
                dqd = (dr * qd).sum(1) * r5
                p = p - 0.5 * dqd
                f = f + (2.5 * dqd / r2)[:, None] * dr - r5[:, None] * qd
            n = torch.bincount(pt - b0, minlength=b1 - b0)
            sums = torch.segment_reduce(torch.cat([f, p[:, None]], 1), "sum", lengths=n, axis=0, unsafe=True)
            acc[b0:b1] += sums[:, :3]
            phi[b0:b1] += sums[:, 3]
            tgt, node = tgt[~take], node[~take]
            k = t.nchild[node]
            at = torch.arange(int(k.sum()), device="cuda") - torch.repeat_interleave(torch.cumsum(k, 0) - k, k)
            node = torch.repeat_interleave(t.child[node], k) + at
            tgt = torch.repeat_interleave(tgt, k)
    return acc, phi


def _forces(case, m, x, prev=None, points=None):
    """The case's force evaluation in 64 bits: (acc, phi), in the bodies' or points' order."""
    t = _Octree(m, x)
    crit, theta = case.get("criterion", "body"), case["theta"]
    if crit == "body":
        y = t.x if points is None else points
        one = torch.ones(len(y), dtype=torch.int64, device="cuda")
        a, p = _walk(t, y, y, y, torch.arange(len(y), device="cuda"), one,
                     lambda t, nd, tg, d2: theta * theta * d2 >= t.s2[nd], case["eps"], case["quad"], points is None)
    else:
        first, count = t.groups(64)
        g = torch.repeat_interleave(torch.arange(len(first), device="cuda"), count)
        lo = torch.full((len(first), 3), math.inf, dtype=torch.float64, device="cuda")
        hi = -lo
        gi = g[:, None].expand(-1, 3)
        lo.scatter_reduce_(0, gi, t.x, "amin")
        hi.scatter_reduce_(0, gi, t.x, "amax")
        if crit == "error":
            amin = torch.full((len(first),), math.inf, dtype=torch.float64, device="cuda")
            amin.scatter_reduce_(0, g, torch.linalg.vector_norm(prev[t.order], dim=1), "amin")
            pw = 3 if case["quad"] else 2

            def accept(t, nd, tg, d2):
                gap = torch.sqrt(d2) - t.b_[nd]
                err = t.m_[nd] * t.b_[nd] ** pw / torch.clamp(gap, min=1e-300) ** (pw + 2)
                return (gap > 0.0) & (d2 >= t.s2[nd] / 16.0) & (err <= theta * amin[tg])
        elif crit == "barnes":
            r2 = (torch.sqrt(t.s2) / theta + torch.linalg.vector_norm(t.c_ - t.centre, dim=1)) ** 2

            def accept(t, nd, tg, d2):
                return d2 > r2[nd]
        else:
            def accept(t, nd, tg, d2):
                return theta * theta * d2 >= t.s2[nd]
        a, p = _walk(t, t.x, lo, hi, first, count, accept, case["eps"], case["quad"], True)
    if points is not None:
        return a, p
    acc, phi = torch.empty_like(a), torch.empty_like(p)
    acc[t.order], phi[t.order] = a, p
    return acc, phi


def _direct(m, x, eps):
    d = x[None, :, :] - x[:, None, :]
    r2 = (d * d).sum(2) + eps * eps
    w = m[None, :] * torch.rsqrt(r2)
    w.fill_diagonal_(0.0)
    return ((w / r2)[:, :, None] * d).sum(1), -w.sum(1)


def _lcg(state):
    return (state * 6364136223846793005 + 1442695040888963407) & (2 ** 64 - 1)


def _trained(case, seed):
    """The training pass in 64 bits: learn_init's weights and learn_train's order of the samples, weights and
    activations rounded to bfloat16 where the network rounds them."""
    st, p = _lcg(5), []
    for rows, fan, zeros in ((64 * 12, 76, 64), (64 * 64, 128, 64), (64, 65, 1)):
        for _ in range(rows):
            st = _lcg(st)
            p.append(math.sqrt(6.0 / fan) * ((st >> 11) / 2.0 ** 53 * 2.0 - 1.0))
        p += [0.0] * zeros
    p = torch.tensor(p, dtype=torch.float32, device="cuda").double()
    x, y = _samples(case, seed)
    n, batch = len(x), min(case["batch"], 8192)
    perm, st = list(range(n)), (3 * 2862933555777941757 + 3037000493) & (2 ** 64 - 1)
    for i in range(n - 1, 0, -1):
        st = _lcg(st)
        j = (st >> 33) % (i + 1)
        perm[i], perm[j] = perm[j], perm[i]
    x, y = (torch.from_numpy(v[perm]).cuda().double() for v in (x, y))

    class Round(torch.autograd.Function):
        @staticmethod
        def forward(ctx, v):
            return v.float().bfloat16().double()

        @staticmethod
        def backward(ctx, g):
            return g

    r, silu = Round.apply, torch.nn.functional.silu
    mom, var = torch.zeros_like(p), torch.zeros_like(p)
    for step, o in enumerate(range(0, n - 63, batch), 1):
        q = p.clone().requires_grad_(True)
        w1, b1, w2, b2, w3, b3 = torch.split(q, [64 * 12, 64, 64 * 64, 64, 64, 1])
        h = r(silu(r(x[o:o + batch]) @ r(w1).reshape(64, 12).T + b1))
        h = r(silu(h @ r(w2).reshape(64, 64).T + b2))
        torch.nn.functional.binary_cross_entropy_with_logits(h @ r(w3) + b3, y[o:o + batch]).backward()
        g = q.grad
        mom, var = 0.9 * mom + 0.1 * g, 0.999 * var + 0.001 * g * g
        p = p - case["lr"] * (mom / (1 - 0.9 ** step)) / (torch.sqrt(var / (1 - 0.999 ** step)) + 1e-8)
    return p


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return {"params": _trained(case, seed), "loss": None}
    if kind == "ensemble":
        counts, m, x, v = _spheres(case, seed)
        accs, phis = [], []
        for k, mm, xx in zip(counts, torch.split(m, counts.tolist()), torch.split(x, counts.tolist())):
            if k <= 1024:
                a, p = _direct(mm, xx, case["eps"])
            else:
                a, p = _forces(case, mm, xx)
            accs.append(a)
            phis.append(p)
        a, p = torch.cat(accs), torch.cat(phis)
        h = v + 0.5 * case["dt"] * a             # the first pass: forces, then kick and drift
        return {"phase": torch.stack([x + case["dt"] * h, h + 0.5 * case["dt"] * a], 1), "acc": a, "phi": p}
    if case["n"] > 1100000 or case.get("criterion") == "learned":
        return None
    m, x, v, prev, g = _bodies(case, seed)
    try:
        if kind == "points":
            a, p = _forces(case, m, x, points=_model(case["model"], case["points"], g)[1])
            return {"acc": a, "phi": p}
        a, p = _forces(case, m, x, prev)
    except ValueError:                           # bodies closer than the 21 bits this octree resolves
        return None
    out = {"acc": a, "phi": p}
    if kind == "step":
        out.update(phase=torch.stack([x, v], 1), n2b=None, nbc=None)
    elif case.get("counts"):
        out.update(n2b=None, nbc=None)
    return out
