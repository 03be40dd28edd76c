"""The transfers that programs have this package do, as cases to be timed and compared.

A case is one call (or one training step) through the public entry points: the
RBF-PUM transfer from host arrays and from device tensors in both precisions, a
coupling loop's plan that keeps its factorisations, the differentiable transfer
with its backward pass, a batch of small uneven problems, and the two point
methods beside it (moving least squares, nearest source).  The clouds, fields,
bases and sizes are those of ``pacman_b200.workloads`` and of the tests, made
here on the device so that the inputs of a new seed are quick to make.
"""
import math
import random

import torch

import pacman_b200 as pacman
from pacman_b200.autograd import rbf_pum_transfer

BASES = {"C0": 0x10, "C2": 0x11, "C4": 0x12, "C6": 0x13, "C8": 0x14}
SUPPORT = 0.1
OVERLAP = 0.15
CUDA = pacman.execspaces.CUDA
F64 = torch.float64


def listed():
    return [
        # A small 2D surface mesh transfer from host arrays, called once per
        # coupling step by a script: launches and waits are all there is.
        dict(name="mesh_2d_host", kind="transfer", cloud="uniform", dim=2, n=3001, m=4099,
             fields=1, basis="C2", npc=50, precision="fp64", host=True),
        # The 20k volume transfer at the default precision, device tensors.
        dict(name="uniform_20k", kind="transfer", cloud="uniform", dim=3, n=20000, m=20000,
             fields=1, basis="C2", npc=30, precision="fp64", host=False),
        # The same call for a large volume mesh and several fields, both
        # precisions in use.
        dict(name="uniform_500k_f4_mixed", kind="transfer", cloud="uniform", dim=3, n=500000,
             m=500000, fields=4, basis="C4", npc=50, precision="mixed", host=False),
        dict(name="uniform_200k_fp64", kind="transfer", cloud="uniform", dim=3, n=200003,
             m=150001, fields=1, basis="C6", npc=50, precision="fp64", host=False),
        # Locally refined sources: most patches small, a few with thousands of
        # points.  The headline workload in the fast precision, and a quarter
        # of it in the reference's arithmetic.
        dict(name="blobs_1m_mixed", kind="transfer", cloud="blobs", dim=3, n=1000000,
             m=1000000, fields=1, basis="C4", npc=50, precision="mixed", host=False),
        dict(name="blobs_250k_fp64", kind="transfer", cloud="blobs", dim=3, n=250000, m=250000,
             fields=1, basis="C4", npc=50, precision="fp64", host=False),
        # Surface plus volume sources, eight fields at once.
        dict(name="shell_1m_f8_mixed", kind="transfer", cloud="shell", dim=3, n=1000000,
             m=500000, fields=8, basis="C2", npc=50, precision="mixed", host=False),
        # One step of a coupling loop over fixed meshes: new values, kept plan.
        dict(name="plan_blobs_400k", kind="plan", cloud="blobs", dim=3, n=400000, m=400000,
             fields=1, basis="C4", npc=50, precision="mixed", host=False),
        # One training step: forward and both gradients.
        dict(name="grad_uniform_150k_f4", kind="grad", cloud="uniform", dim=3, n=150000,
             m=150000, fields=4, basis="C4", npc=50, precision="fp64", host=False),
        # Many small independent problems in one call.
        dict(name="batch_48", kind="batch", cloud="uniform", dim=3, n=1000, m=30000, fields=4,
             basis="mix", npc=50, precision="mixed", host=False, count=48),
        # The point methods on the refined cloud.
        dict(name="mls_blobs_500k", kind="mls", cloud="blobs", dim=3, n=500000, m=500000,
             fields=1, basis="-", npc=0, precision="fp64", host=False),
        dict(name="nearest_blobs_1m", kind="nearest", cloud="blobs", dim=3, n=1000000,
             m=1000000, fields=1, basis="-", npc=0, precision="fp64", host=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed ranges: any dimension, size, basis and field count
    that they stand for, no dearer than the dearest of them."""
    kind = rng.choice(["uniform", "uniform", "blobs", "blobs", "shell", "plan", "grad", "batch",
                       "mls", "nearest"])
    c = dict(kind="transfer", cloud="uniform", dim=3, fields=1, npc=50, host=False,
             precision=rng.choice(["fp64", "mixed"]))
    if kind == "uniform":
        c["host"] = rng.random() < 0.4
        c["dim"] = rng.choice([2, 3, 3])
        c["n"] = _log_int(rng, 2500, 500000 if c["dim"] == 3 else 100000)
        c["m"] = max(1000, min(500000, int(c["n"] * rng.uniform(0.5, 2.0))))
        c["fields"] = rng.choice([1, 1, 2, 4])
        c["basis"] = rng.choice(["C0", "C2", "C4", "C6"])
        c["npc"] = rng.choice([30, 50, 50])
    elif kind == "blobs":
        c.update(cloud="blobs", basis=rng.choice(["C2", "C4"]), fields=rng.choice([1, 1, 3]))
        c["n"] = _log_int(rng, 60000, 900000 if c["precision"] == "mixed" else 220000)
        c["m"] = int(c["n"] * rng.uniform(0.6, 1.0))
    elif kind == "shell":
        c.update(cloud="shell", basis=rng.choice(["C0", "C2"]), fields=rng.choice([1, 2, 5, 8]),
                 precision="mixed")
        c["n"] = _log_int(rng, 60000, 900000)
        c["m"] = int(c["n"] * rng.uniform(0.3, 0.5))
    elif kind == "plan":
        c.update(kind="plan", cloud="blobs", basis=rng.choice(["C2", "C4"]), precision="mixed",
                 fields=rng.choice([1, 2, 4]))
        c["n"] = _log_int(rng, 40000, 400000)
        c["m"] = int(c["n"] * rng.uniform(0.6, 1.0))
    elif kind == "grad":
        c.update(kind="grad", basis=rng.choice(["C2", "C4"]), fields=rng.choice([1, 2, 4]))
        c["n"] = _log_int(rng, 5000, 150000)
        c["m"] = int(c["n"] * rng.uniform(0.6, 1.0))
    elif kind == "batch":
        c.update(kind="batch", basis="mix", fields=rng.choice([1, 2, 4]),
                 count=rng.randint(6, 48), n=1000, m=_log_int(rng, 6000, 30000))
    else:
        c.update(kind=kind, cloud=rng.choice(["uniform", "blobs"]), basis="-", npc=0,
                 precision="fp64")
        if c["cloud"] == "uniform":
            c["dim"] = rng.choice([1, 2, 3])
        c["n"] = _log_int(rng, 5000, 500000)
        c["m"] = int(c["n"] * rng.uniform(0.5, 1.0))
    return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _uniform(n, dim, g, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(n, dim, generator=g, device="cuda", dtype=F64)


def _blobs(n, g):
    """Half jittered grid points of spacing 0.01 in a sub-box of volume n / 1M,
    half Gaussian blobs of sigma 0.02 there: the patch sizes of the 1M cloud."""
    scale = n / 1.0e6
    side = max(2, int(round(100 * scale ** (1.0 / 3.0))))
    n_grid = min(n // 2, side ** 3)
    cell = torch.randperm(side ** 3, generator=g, device="cuda")[:n_grid]
    ijk = torch.stack([cell // (side * side), cell // side % side, cell % side], 1).to(F64)
    grid = (ijk + 0.5) / 100.0 + _uniform(n_grid, 3, g, -0.003, 0.003)
    nb = max(1, int(round(64 * scale)))
    centres = _uniform(nb, 3, g, 0.0, side / 100.0)
    n_blob = n - n_grid
    which = torch.arange(n_blob, device="cuda") % nb
    blobs = centres[which] + 0.02 * torch.randn(n_blob, 3, generator=g, device="cuda", dtype=F64)
    pts = torch.cat([grid, blobs])
    return pts[torch.randperm(n, generator=g, device="cuda")].contiguous()


def _shell(n, g):
    """60% on a perturbed unit sphere, 40% in the cube around it."""
    ns = int(round(0.6 * n))
    v = torch.randn(ns, 3, generator=g, device="cuda", dtype=F64)
    v = v / v.norm(dim=1, keepdim=True)
    theta, phi = torch.arccos(v[:, 2].clamp(-1, 1)), torch.atan2(v[:, 1], v[:, 0])
    v = v * (1.0 + 0.05 * torch.sin(5 * theta) * torch.cos(3 * phi))[:, None]
    pts = torch.cat([v, _uniform(n - ns, 3, g, -1.05, 1.05)])
    return pts[torch.randperm(n, generator=g, device="cuda")].contiguous()


def _clouds(cloud, n, m, dim, g):
    if cloud == "blobs":
        side = max(2, int(round(100 * (n / 1.0e6) ** (1.0 / 3.0)))) / 100.0
        return _blobs(n, g), _uniform(m, 3, g, 0.0, side)
    if cloud == "shell":
        return _shell(n, g), _shell(m, g)
    return _uniform(n, dim, g), _uniform(m, dim, g)


def _fields(p, fields, g):
    """Franke's function of the points, then random low Fourier modes."""
    x = 9.0 * p[:, 0]
    y = 9.0 * p[:, 1] if p.shape[1] > 1 else torch.zeros_like(x)
    z = 9.0 * p[:, 2] if p.shape[1] > 2 else torch.zeros_like(x)
    f = (0.75 * torch.exp(-((x - 2) ** 2 + (y - 2) ** 2 + (z - 2) ** 2) / 4)
         + 0.75 * torch.exp(-((x + 1) ** 2 / 49 + (y + 1) / 10 + (z + 1) / 10))
         + 0.5 * torch.exp(-((x - 7) ** 2 + (y - 3) ** 2 + (z - 5) ** 2) / 4)
         - 0.2 * torch.exp(-((x - 4) ** 2 + (y - 7) ** 2 + (z - 5) ** 2)))
    a = 0.1 * torch.randn(8, generator=g, device="cuda", dtype=F64)
    cols = []
    for k in range(fields):
        w = torch.randint(-4, 5, (p.shape[1], 8), generator=g, device="cuda").to(F64)
        wave = torch.cos(2 * math.pi * (p @ w) + k) @ a
        cols.append(f + wave if k == 0 else 4.0 * wave)
    return torch.stack(cols, 1).contiguous()


def _problems(case):
    """Sizes, bases and field counts of a batch: of the case, not of the seed."""
    r = random.Random("%d %d %d" % (case["count"], case["m"], case["fields"]))
    for _ in range(case["count"]):
        n = _log_int(r, case["n"], case["m"])
        yield n, max(64, int(n * r.uniform(0.8, 1.0))), r.uniform(0.5, 2.0), \
            r.choice(["C0", "C2", "C4", "C6"]), r.randint(1, case["fields"])


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _inputs(case, seed):
    g = _generator(seed)
    if case["kind"] == "batch":
        items = []
        for n, m, side, basis, nf in _problems(case):
            src, tgt = _uniform(n, 3, g, 0.0, side), _uniform(m, 3, g, 0.0, side)
            items.append((3, BASES[basis], src, _fields(src / side, nf, g), tgt))
        return items
    src, tgt = _clouds(case["cloud"], case["n"], case["m"], case["dim"], g)
    vals = _fields(src, case["fields"], g)
    if case["fields"] == 1:
        vals = vals[:, 0].contiguous()
    return src, vals, tgt


def prepare(case, seed):
    if case["kind"] == "batch":
        return dict(case=case, problems=_inputs(case, seed))
    src, vals, tgt = _inputs(case, seed)
    s = dict(case=case, src=src, vals=vals, tgt=tgt)
    if case["kind"] == "grad":
        g = _generator(seed + 7)
        s["up"] = torch.randn(vals.shape[:0] + (case["m"],) + vals.shape[1:], generator=g,
                              device="cuda", dtype=F64)
        s["vals"] = vals.requires_grad_()
        s["tgt"] = tgt.requires_grad_()
    elif case["kind"] == "plan":
        # The program's plan after its first step: geometry and factors kept.
        plan = pacman.rbf.Plan(case["dim"], src, tgt, nodes_per_cluster=case["npc"],
                               precision=case["precision"])
        plan.execute(BASES[case["basis"]], torch.ones_like(vals), keep_factors=True)
        s["plan"] = plan
    elif case["host"]:
        for k in ("src", "vals", "tgt"):
            s[k] = s[k].cpu().numpy()
    return s


def run(state):
    c = state["case"]
    if c["kind"] == "batch":
        return pacman.rbf.interpolate_batch(state["problems"], nodes_per_cluster=c["npc"],
                                            precision=c["precision"])
    src, vals, tgt = state["src"], state["vals"], state["tgt"]
    if c["kind"] == "mls":
        return pacman.mls.interpolate(c["dim"], CUDA, src, vals, tgt)
    if c["kind"] == "nearest":
        return pacman.fe.interpolate(c["dim"], CUDA, pacman.fe.methods.NEAREST_NEAREST, src, vals,
                                     None, None, None, tgt)
    if c["kind"] == "plan":
        return state["plan"].execute(BASES[c["basis"]], vals, keep_factors=True)
    if c["kind"] == "grad":
        out = rbf_pum_transfer(src, vals, tgt, BASES[c["basis"]], nodes_per_cluster=c["npc"],
                               precision=c["precision"])
        return (out.detach(),) + torch.autograd.grad(out, (vals, tgt), state["up"])
    return pacman.rbf.interpolate(c["dim"], CUDA, BASES[c["basis"]], src, vals, tgt,
                                  nodes_per_cluster=c["npc"], precision=c["precision"])


# ---------------------------------------------------------------------------
# Work
# ---------------------------------------------------------------------------

def _solve_flops(cloud, n, m, npc, fields):
    """FP64 work of the patch solves: n_k^3 / 3 for the factorisation, 2 n_k^2
    per field for the solves and, per pair of a target or source with a
    patch's source, about 12 for the distance and basis and 2 per field.  Each
    point is in about 4.7 patches (their spacing is 0.98 radii); on a uniform
    cloud the patches hold npc points, on the refined ones the sums are
    dominated by the dense patches: 2.3e6 per source of the blobs (measured
    2,237 GFLOP at 1M, the same at every size), and on the shell patches of
    about 0.8 n^(1/3) npc^(2/3) sources."""
    if cloud == "blobs":
        return 2.3e6 * n + 4.7 * m * 500.0 * (12 + 2 * fields)
    size = npc if cloud == "uniform" else 0.8 * n ** (1.0 / 3.0) * npc ** (2.0 / 3.0)
    k = 4.7 * n / size
    return k * (size ** 3 / 3 + size ** 2 * (6 + 2 * fields)) + 4.7 * m * size * (12 + 2 * fields)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        b = f = 0.0
        for n, m, _, _, nf in _problems(case):
            b += 8.0 * (n * (3 + nf) + m * (3 + nf))
            f += _solve_flops("uniform", n, m, case["npc"], nf)
        return {"bytes": b, "flops": f}
    n, m, nf, d = case["n"], case["m"], case["fields"], case["dim"]
    b = 8.0 * (n * (d + nf) + m * (d + nf))
    if kind == "mls":
        k = {1: 3, 2: 6, 3: 10}[d]
        # Distances to the neighbours, moment matrix, one K x K solve.
        return {"bytes": b, "flops": float(m) * (8 * k + k * k * (k + 1) + 2.0 * k ** 3 / 3)}
    if kind == "nearest":
        return {"bytes": b + 4.0 * m, "flops": 8.0 * m}
    f = _solve_flops(case["cloud"], n, m, case["npc"], nf)
    if kind == "plan":
        # Kept factors: two triangular solves (2 n_k^2 per field each way) and
        # the evaluation; the factors themselves are read, n_k^2 / 2 doubles:
        # 16 KB per source of the blobs.
        return {"bytes": b + 1.6e4 * n, "flops": 4.0e3 * n * nf + 4.7 * m * 500.0 * (12 + 2 * nf)}
    if kind == "grad":
        # The transpose solve uses the forward's factor; gradients of values
        # and target coordinates out, upstream in.
        b += 8.0 * (m * nf + n * nf + m * d)
        f += 4.7 * m * case["npc"] * (24 + 8 * nf) + 4.7 * n * case["npc"] * 2 * nf
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# The same values in plain 64-bit torch
# ---------------------------------------------------------------------------

def _d2(a, b):
    """Squared distances, (..., A, B), by differences."""
    s = None
    for d in range(a.shape[-1]):
        t = a[..., :, None, d] - b[..., None, :, d]
        s = t * t if s is None else s.addcmul_(t, t) if not s.requires_grad else s + t * t
    return s


def _phi(basis, d2, support):
    p = torch.sqrt(d2) / support
    q = (1 - p).clamp(min=0)
    if basis == 0x10:
        return q ** 2
    if basis == 0x11:
        return q ** 4 * (4 * p + 1)
    if basis == 0x12:
        return q ** 6 * (35 * p ** 2 + 18 * p + 3)
    if basis == 0x13:
        return q ** 8 * (32 * p ** 3 + 25 * p ** 2 + 8 * p + 1)
    return q ** 10 * (1287 * p ** 4 + 1350 * p ** 3 + 630 * p ** 2 + 150 * p + 15)


def _chunks(count, per):
    step = max(1, int(per))
    return [(i, min(i + step, count)) for i in range(0, count, step)]


def _nearest(q, pts, room=2.0e8):
    best, at = [], []
    for i, j in _chunks(len(q), room / len(pts)):
        v, k = _d2(q[i:j], pts).min(dim=1)
        best.append(v)
        at.append(k)
    return torch.cat(best), torch.cat(at)


def _lists(centres, pts, r, room=2.0e8):
    rows, cols = [], []
    for i, j in _chunks(len(centres), room / len(pts)):
        a, b = torch.nonzero(torch.sqrt(_d2(centres[i:j], pts)) <= r, as_tuple=True)
        rows.append(a + i)
        cols.append(b)
    return torch.cat(rows), torch.cat(cols)


def _cover(src, tgt, npc):
    """Patch radius and centres."""
    n, dim = src.shape
    lo, hi = src.min(0).values, src.max(0).values
    mid, quarter = (lo + hi) / 2, (hi - lo) / 4
    samples = [mid] + [mid + s * quarter * torch.eye(dim, device="cuda", dtype=F64)[a]
                       for s in (-1, 1) for a in range(dim)]
    at = _nearest(torch.stack(samples), src)[1]
    kth = _d2(src[at], src).kthvalue(min(npc, n), dim=1).values
    r = float(torch.sqrt(kth.sort().values[dim]))
    spacing = math.sqrt(4.0 / dim) * r * (1 - OVERLAP)
    shape = [math.ceil(max(1.0, float(e) / spacing)) for e in hi - lo]
    dist = [float(e) / s for e, s in zip(hi - lo, shape)]
    shape = [s + 1 for s in shape]
    axes = [lo[a] + dist[a] * torch.arange(shape[a], device="cuda", dtype=F64) for a in range(dim)]
    cand = torch.stack(torch.meshgrid(*axes, indexing="ij"), -1).reshape(-1, dim)
    d, at = _nearest(cand, src)
    alive = (d <= r * r) & (_nearest(cand, tgt)[0] <= r * r)
    pos = torch.where(alive[:, None], src[at], cand)
    # A candidate goes if a close neighbour after it was alive at the start, or
    # a close neighbour before it stayed.
    nb, thr = len(cand), (0.4 * min(dist)) ** 2
    steps = [1]
    for s in reversed(shape[1:]):
        steps.insert(0, steps[0] * s)
    offsets = {sum(o * s for o, s in zip(off, steps)) for off in
               _grid_offsets(dim)} - {0}
    idx = torch.arange(nb, device="cuda")
    before = []
    state = alive.clone()
    for o in sorted(offsets):
        j = idx + o
        ok = (j >= 0) & (j < nb)
        j = j.clamp(0, nb - 1)
        close = ok & alive & alive[j] & (((pos - pos[j]) ** 2).sum(1) < thr)
        if o > 0:
            state &= ~close
        else:
            before.append((o, close))
    open_ = torch.zeros_like(state)
    for _, close in before:
        open_ |= close
    open_ &= state
    keep = state & ~open_
    while bool(open_.any()):
        hit, wait = torch.zeros_like(keep), torch.zeros_like(keep)
        for o, close in before:
            j = (idx + o).clamp(0, nb - 1)
            hit |= close & keep[j]
            wait |= close & open_[j]
        stay = open_ & ~hit & ~wait
        keep |= stay
        open_ &= ~hit & ~stay
    pos = pos[keep]
    return r, pos[_nearest(pos, tgt)[0] <= r * r]


def _grid_offsets(dim):
    out = [()]
    for _ in range(dim):
        out = [o + (s,) for o in out for s in (-1, 0, 1)]
    return out


def _transfer(src, vals, tgt, basis, npc):
    """The whole partition-of-unity transfer; differentiable in vals and tgt."""
    dim = src.shape[1]
    with torch.no_grad():
        t0 = tgt.detach()
        r, centres = _cover(src, t0, npc)
        sr, sc = _lists(centres, src, r)
        tr, tc = _lists(centres, t0, r - 1e-14)
        K = len(centres)
        ns, nt = torch.bincount(sr, minlength=K), torch.bincount(tr, minlength=K)
        so, to = torch.cumsum(ns, 0) - ns, torch.cumsum(nt, 0) - nt
        order = torch.argsort(ns)
        order = order[nt[order] > 0]
        if float(ns.max()) > 4000 or float((ns.double() ** 3).sum()) > 3.0e12:
            return None  # more than this takes in seconds
    values = vals if vals.dim() == 2 else vals[:, None]
    num = torch.zeros(len(tgt), values.shape[1], device="cuda", dtype=F64)
    den = torch.zeros(len(tgt), device="cuda", dtype=F64)
    at = 0
    sizes, targets = ns[order].tolist(), nt[order].tolist()
    while at < len(order):
        end, wide = at, 0
        while end < len(order):
            wide = max(wide, targets[end])
            if end > at and (end + 1 - at) * sizes[end] * max(sizes[end], wide) > 4.0e7:
                break
            if end > at and sizes[end] > 1.3 * sizes[at] + 8:
                break
            end += 1
        ks = order[at:end]
        n, m = sizes[end - 1], int(nt[ks].max())
        at = end
        ar, am = torch.arange(n, device="cuda"), torch.arange(m, device="cuda")
        has, gets = ar < ns[ks][:, None], am < nt[ks][:, None]
        si = sc[(so[ks][:, None] + ar).clamp(max=len(sc) - 1)]
        ti = tc[(to[ks][:, None] + am).clamp(max=len(tc) - 1)]
        c = centres[ks][:, None, :]
        x = torch.where(has[..., None], src[si], c + 50.0)
        b = torch.where(has[..., None], values[si], torch.zeros((), device="cuda", dtype=F64))
        y = torch.where(gets[..., None], tgt[ti], c - 50.0)
        with torch.no_grad():
            A = _phi(basis, _d2(x, x), SUPPORT)
            pair = has[:, :, None] & has[:, None, :]
            A = torch.where(pair, A, torch.eye(n, device="cuda", dtype=F64))
            L = torch.linalg.cholesky(A)
            one = has[..., None].to(F64)
            Q = torch.cat([one, (x - c) * one], 2)
            # The axes that stay: the least-spread one goes while the monomials
            # [1, x] of the patch are worse conditioned than 1e5.
            act = torch.ones(len(ks), dim + 1, device="cuda", dtype=F64)
            full = torch.cat([one, x * one], 2)
            spread = (torch.where(has[..., None], x, -math.inf).amax(1)
                      - torch.where(has[..., None], x, math.inf).amin(1))
            for _ in range(dim):
                qa = full * act[:, None, :]
                e = torch.linalg.eigvalsh(qa.transpose(1, 2) @ qa)
                low = torch.gather(e, 1, (dim + 1 - act.sum(1).long())[:, None])[:, 0]
                bad = (~(e[:, -1] < 1.0e10 * low.clamp(min=1e-28))) & (act.sum(1) > 1)
                if not bool(bad.any()):
                    break
                sp = torch.where(act[:, 1:] > 0, spread, math.inf)
                act[bad, 1 + sp.argmin(1)[bad]] = 0.0
            Q = Q * act[:, None, :]
            gram = Q.transpose(1, 2) @ Q + torch.diag_embed(1.0 - act)
        beta = torch.linalg.solve(gram, Q.transpose(1, 2) @ b) * act[..., None]
        res = b - Q @ beta
        alpha = torch.linalg.solve_triangular(
            L.transpose(1, 2), torch.linalg.solve_triangular(L, res, upper=False), upper=True)
        V = torch.cat([torch.ones_like(y[..., :1]), y - c], 2)
        loc = _phi(basis, _d2(y, x), SUPPORT) @ alpha + V @ beta
        dist = torch.sqrt(((y - c) ** 2).sum(-1))
        q = (1 - dist / r).clamp(min=0)
        w = q ** 4 * (4 * dist / r + 1)
        w, loc, ti = w[gets], loc[gets], ti[gets]
        num = num.index_add(0, ti, w[:, None] * loc)
        den = den.index_add(0, ti, w)
    out = torch.where(den[:, None] > 0, num / torch.where(den > 0, den, 1.0)[:, None],
                      torch.zeros((), device="cuda", dtype=F64))
    return out if vals.dim() == 2 else out[:, 0]


def _mls(src, vals, tgt):
    dim = src.shape[1]
    k = {1: 3, 2: 6, 3: 10}[dim]
    out = []
    for i, j in _chunks(len(tgt), 1.0e8 / len(src)):
        d2, at = _d2(tgt[i:j], src).topk(k, dim=1, largest=False)
        d = torch.sqrt(d2)
        rad = 1.1 * d.amax(1, keepdim=True).clamp(min=10 * 2.0 ** -52)
        w = 1 - d / rad  # the square root of the weight
        x = (src[at] - tgt[i:j, None, :]) / rad[..., None]
        cols = [torch.ones_like(d)] + [x[..., a] for a in range(dim)]
        cols += [x[..., a] * x[..., e] for a in range(dim) for e in range(a, dim)]
        u, s, vh = torch.linalg.svd(torch.stack(cols, 2) * w[..., None])
        inv = torch.where(s * s > 1e-13 * s[:, :1] ** 2, 1 / s, torch.zeros_like(s))
        out.append((vh[:, :, 0] * inv * ((w * vals[at])[:, None, :] @ u)[:, 0]).sum(1))
    return torch.cat(out)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return [_transfer(s, v, t, b, case["npc"]) for _, b, s, v, t in _inputs(case, seed)]
    src, vals, tgt = _inputs(case, seed)
    if kind in ("mls", "nearest"):
        if len(src) * len(tgt) > (2.6e11 if kind == "mls" else 1.1e12):
            return None  # every pair is looked at
        if kind == "mls":
            return _mls(src, vals, tgt)
        return vals[_nearest(tgt, src)[1]], None
    if kind == "grad":
        g = _generator(seed + 7)
        up = torch.randn((case["m"],) + vals.shape[1:], generator=g, device="cuda", dtype=F64)
        vals.requires_grad_()
        tgt.requires_grad_()
        out = _transfer(src, vals, tgt, BASES[case["basis"]], case["npc"])
        return (out.detach(),) + torch.autograd.grad(out, (vals, tgt), up)
    with torch.no_grad():
        out = _transfer(src, vals, tgt, BASES[case["basis"]], case["npc"])
    return out.cpu().numpy() if out is not None and case["host"] else out
