"""Performance cases of the library's public entry points.

Each case is one thing that a program around the Potts segmentation does with a volume on the GPU:
the solve itself (small, ordinary and full-size cores; the exact and the fast arithmetic; two to four
labels; FP32 and 16-bit state; from host buffers and from device buffers; a batch of uneven volumes),
the gradient of the unrolled solve, TV-L2 denoising, the inputs of the label search and the ingest of a
16-bit scan.  Sizes are those of this repository's own configurations (a 128^3 core of radius 60, the
768 x 768 x 1024 core of radius 370, 64 .. 256 sides for batches, a 192^3 core for gradients) and odd
ones between them.

listed()            the cases
draw(rng)           another case of the same ranges
prepare(case, seed) inputs on the GPU (or pinned host buffers) and the handles that a program keeps
run(state)          one pass through the entry points; returns its outputs
work(case)          bytes and operations that a pass cannot do without
exact(case, seed)   the outputs in 64 bits, from plain torch
"""
from __future__ import annotations

import math

import numpy as np
import torch

from segmentctscans_b200 import potts
from segmentctscans_b200.layout import CylinderMapping

# the solver's and the denoiser's parameters as the reference's command-line tools set them
LAMBDA = 30.0
TV_LAMBDA, TV_TAU = 0.06, 0.99 / 6.0
LOSS_EPS = 1e-3
TAIL = 1e-4
# phase intensities of a scan (scCO2, brine, a fourth phase, glass) and its noise
PHASES = {2: (3.39e-2, 5.27e-2), 3: (3.39e-2, 4.09e-2, 5.27e-2), 4: (3.39e-2, 4.09e-2, 4.6e-2, 5.27e-2)}
# volume fraction below which each phase boundary lies
CUTS = {2: (0.2,), 3: (0.08, 0.2), 4: (0.08, 0.17, 0.2)}
NOISE = 7e-3


def _tau() -> float:
    return potts.reference_tau()


def listed() -> list[dict]:
    return [
        # a small core at the library's default options: few voxels, one launch per iteration
        # and the whole state back, which a program needs to go on from it
        dict(_solve("solve_small", 128, 128, 128, 60.0, 3, "exact", "f32", 100), dual=True),
        # a core of odd extents from host buffers and back (what a command-line tool does), default options
        dict(_solve("solve_host_odd", 203, 301, 287, 140.0, 3, "exact", "f32", 60), host=True),
        # the full-size core in the fast arithmetic, with the energies that a stopping rule reads
        dict(_solve("solve_core", 1024, 768, 768, 370.0, 3, "fast", "f32", 50), gap_every=50),
        # four labels
        _solve("solve_four_labels", 256, 512, 512, 246.0, 4, "fast", "f32", 40),
        # 16-bit state, for volumes whose FP32 state would need slabs
        _solve("solve_bf16", 512, 512, 512, 246.0, 3, "fast", "bf16", 40),
        # a sweep over many small volumes of uneven size, planned once and replayed
        {"name": "batch_sweep", "kind": "batch", "count": 24, "side_min": 64, "side_max": 256, "iters": 60,
         "arith": "fast"},
        # gradients of the segmentation loss through the unrolled solve: forward and backward
        {"name": "unrolled_grad", "kind": "unroll", "n": 192, "rows": 192, "cols": 192, "radius": 90.0, "k": 3,
         "iters": 40, "every": 20},
        # denoising of a large core, and of a small one of odd extents
        _tv("tv_core", 512, 512, 512, 246.0, 150),
        _tv("tv_small_odd", 99, 130, 127, 60.0, 150),
        # the inputs of the label search: range, gradient magnitude, 1-D and 2-D histogram
        _labels("labels_core", 1024, 768, 768, 370.0, 1024, 512),
        _labels("labels_odd", 317, 300, 300, 146.0, 1000, 300),
        # a 16-bit scan: its intensity range, then its conversion to [0, 1]
        _ingest("ingest_core", 1024, 768, 768, 370.0),
    ]


def _solve(name, n, rows, cols, radius, k, arith, storage, iters) -> dict:
    return {"name": name, "kind": "solve", "n": n, "rows": rows, "cols": cols, "radius": radius, "k": k,
            "arith": arith, "storage": storage, "iters": iters, "gap_every": 0, "host": False,
            "dual": False}


def _tv(name, n, rows, cols, radius, iters) -> dict:
    return {"name": name, "kind": "tv", "n": n, "rows": rows, "cols": cols, "radius": radius, "iters": iters}


def _labels(name, n, rows, cols, radius, bins, bins2) -> dict:
    return {"name": name, "kind": "labels", "n": n, "rows": rows, "cols": cols, "radius": radius, "bins": bins,
            "bins2": bins2}


def _ingest(name, n, rows, cols, radius) -> dict:
    return {"name": name, "kind": "ingest", "n": n, "rows": rows, "cols": cols, "radius": radius}


def draw(rng) -> dict:
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def extents(hi):
        rows = log_int(64, hi)
        cols = max(48, min(hi, int(rows * rng.uniform(0.85, 1.15))))
        return {"n": log_int(48, hi), "rows": rows, "cols": cols,
                "radius": round(min(rows, cols) * rng.uniform(0.40, 0.49), 2)}

    kind = rng.choice(["solve", "solve", "solve", "batch", "unroll", "tv", "labels", "ingest"])
    if kind == "solve":
        case = {"kind": kind, **extents(448), "k": rng.choice([2, 3, 3, 4]), "arith": rng.choice(["exact", "fast"]),
                "storage": rng.choice(["f32", "f32", "bf16", "f16"]), "iters": log_int(20, 100),
                "gap_every": rng.choice([0, 0, 20]), "host": rng.random() < 0.25, "dual": rng.random() < 0.3}
    elif kind == "batch":
        lo = rng.randint(48, 128)
        case = {"kind": kind, "count": rng.randint(2, 24), "side_min": lo, "side_max": rng.randint(lo + 32, 256),
                "iters": log_int(20, 60), "arith": rng.choice(["exact", "fast"])}
    elif kind == "unroll":
        case = {"kind": kind, **extents(192), "k": rng.choice([2, 3, 3, 4]), "iters": rng.randint(10, 40),
                "every": rng.randint(5, 20)}
    elif kind == "tv":
        case = {"kind": kind, **extents(512), "iters": log_int(30, 150)}
    elif kind == "labels":
        case = {"kind": kind, **extents(768), "bins": log_int(64, 4096), "bins2": log_int(64, 1024)}
    else:
        case = {"kind": kind, **extents(768)}
    return case


# ---- inputs ---------------------------------------------------------------------------------------
def _mapping(case) -> CylinderMapping:
    return CylinderMapping.cylinder(case["n"], case["rows"], case["cols"], case["radius"])


def _core(mapping, k: int, seed: int, noise: float = NOISE):
    """A noisy scan of a core: pore phases where a smooth random field (grains of about 16 voxels) is
    low, glass elsewhere, soft phase boundaries, Gaussian noise, normalised to [0, 1] by its in-mask
    range.  Returns (u, true label, labels in the units of u), u and truth in the mapping's span."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) * 1000003 + 7)
    shape = (mapping.cols, mapping.rows, mapping.n_images)
    coarse = [max(2, s // 16 + 2) for s in shape]
    low = torch.randn((1, 1, *coarse), generator=gen, device="cuda")
    t = torch.nn.functional.interpolate(low, size=shape, mode="trilinear", align_corners=True)[0, 0]
    rows, cols = mapping.lines()
    rows, cols = torch.from_numpy(rows).cuda(), torch.from_numpy(cols).cuda()
    t = t[cols, rows, :]  # in-mask lines
    sample = t.reshape(-1)[:: max(1, t.numel() // 1_000_000)].sort().values
    level = PHASES[k]
    x = torch.full_like(t, level[-1])
    truth = torch.full(t.shape, k - 1, dtype=torch.uint8, device="cuda")
    for i in range(k - 2, -1, -1):
        cut = float(sample[int(CUTS[k][i] * (sample.numel() - 1))])
        x += (level[i] - level[i + 1]) * torch.sigmoid((cut - t) * 20.0)
        truth[t < cut] = i
    del t
    x += noise * torch.randn(x.shape, generator=gen, device="cuda")
    lo, hi = float(x.min()), float(x.max())
    x.sub_(lo).div_(hi - lo).clamp_(0.0, 1.0)
    u = torch.zeros((mapping.n_lines, mapping.nstride), device="cuda")
    u[:, : mapping.n_images] = x
    tr = torch.zeros((mapping.n_lines, mapping.nstride), dtype=torch.uint8, device="cuda")
    tr[:, : mapping.n_images] = truth
    ci = [float((np.float32(v) - np.float32(lo)) / (np.float32(hi) - np.float32(lo))) for v in level]
    return u.reshape(-1), tr.reshape(-1), ci


def _batch_volumes(case, seed: int):
    """(mapping, u, labels, lambda) of every volume: sides uniform in the case's range, lambda
    log-uniform in [10, 100], noise uniform in [4e-3, 1.2e-2].  The sizes and lambda belong to the
    case (one sweep), the voxels to the seed."""
    sizes = np.random.default_rng(1234)
    vols = []
    for i in range(case["count"]):
        n, rows, cols = (int(v) for v in sizes.integers(case["side_min"], case["side_max"] + 1, size=3))
        lam = float(np.exp(sizes.uniform(np.log(10.0), np.log(100.0))))
        noise = float(sizes.uniform(4e-3, 1.2e-2))
        m = CylinderMapping.cylinder(n, rows, cols, 0.47 * min(rows, cols))
        u, _, ci = _core(m, 3, seed * 64 + i, noise)
        vols.append((m, u, ci, lam))
    return vols


def prepare(case, seed):
    kind = case["kind"]
    ctx = potts.make_context(0, stream=torch.cuda.current_stream().cuda_stream)
    st = {"case": case, "ctx": ctx}
    if kind == "batch":
        st["vols"] = _batch_volumes(case, seed)
        st["V"] = [torch.zeros((2, m.span), device="cuda") for m, _, _, _ in st["vols"]]
        st["labels"] = [torch.zeros(m.span, dtype=torch.uint8, device="cuda") for m, _, _, _ in st["vols"]]
        vols = [potts.BatchVolume(m, u.data_ptr(), ci, lam, labels_ptr=lab.data_ptr(), V_ptr=v.data_ptr())
                for (m, u, ci, lam), v, lab in zip(st["vols"], st["V"], st["labels"])]
        st["batch"] = potts.Batch(ctx, vols, _tau(), _tau(), case["iters"], arith=case["arith"])
        return st
    m = st["map"] = _mapping(case)
    u, truth, ci = _core(m, case.get("k", 3), seed)
    if kind == "solve":
        k, st["ci"] = case["k"], ci
        if case["host"]:
            for name, dt in (("u", torch.float32), ("res", torch.float32), ("labels", torch.uint8)):
                st[name] = torch.zeros(m.span, dtype=dt, pin_memory=True)
            st["u"].copy_(u)
        else:
            st["u"] = u
            st["res"] = torch.zeros(m.span, device="cuda")
            st["labels"] = torch.zeros(m.span, dtype=torch.uint8, device="cuda")
            st["V"] = torch.zeros((k - 1, m.span), device="cuda")
            if case["dual"]:
                st["Xi"] = torch.zeros((3 * (k - 1), m.span), device="cuda")
    elif kind == "unroll":
        st.update(u=u, truth=truth, ci=ci, grad=torch.zeros_like(u), V=torch.zeros((case["k"] - 1, m.span),
                                                                                  device="cuda"))
    elif kind == "tv":
        st.update(u=u, out=torch.zeros_like(u))
    elif kind == "labels":
        st.update(u=u, grad=torch.zeros_like(u))
    elif kind == "ingest":
        st.update(raw=(u * 30000.0 + 12000.0).to(torch.int32).to(torch.int16), out=torch.zeros_like(u))
    return st


# ---- one pass -------------------------------------------------------------------------------------
def run(st):
    case, ctx = st["case"], st["ctx"]
    kind = case["kind"]
    if kind == "batch":
        st["batch"].run(stats=False)
        return {"V": st["V"], "labels": st["labels"]}
    m = st["map"]
    if kind == "solve":
        opts = {"arith": case["arith"], "storage": case["storage"], "gap_every": case["gap_every"]}
        if case["host"]:
            stats = potts.solve_host(ctx, m, st["u"].numpy(), st["ci"], LAMBDA, _tau(), _tau(), case["iters"],
                                     res=st["res"].numpy(), labels=st["labels"].numpy(), stats=True, **opts)
            out = {"res": st["res"], "labels": st["labels"]}
        else:
            stats = potts.solve_device(ctx, m, st["u"].data_ptr(), st["ci"], LAMBDA, _tau(), _tau(), case["iters"],
                                       res_ptr=st["res"].data_ptr(), labels_ptr=st["labels"].data_ptr(),
                                       V_ptr=st["V"].data_ptr(),
                                       Xi_ptr=st["Xi"].data_ptr() if case["dual"] else 0, **opts)
            out = {"res": st["res"], "labels": st["labels"], "V": st["V"]}
            if case["dual"]:
                out["Xi"] = st["Xi"]
        out["dq"] = stats.dq_trace
        if case["gap_every"]:
            out["energy"] = stats.energy_trace
        return out
    if kind == "unroll":
        with potts.Tape(ctx, m, st["u"].data_ptr(), st["truth"].data_ptr(), st["ci"], LAMBDA, _tau(), _tau(),
                        case["iters"], case["every"], LOSS_EPS, V_ptr=st["V"].data_ptr()) as tape:
            grad_c, grad_lam = tape.backward(st["grad"].data_ptr())
            return {"loss": tape.loss, "V": st["V"], "grad_u": st["grad"], "grad_c": grad_c, "grad_lambda": grad_lam}
    if kind == "tv":
        st["out"].copy_(st["u"])  # the scan itself is kept: the denoiser works in place
        potts.tv_denoise(ctx, m, st["out"].data_ptr(), TV_LAMBDA, TV_TAU, case["iters"], stats=False)
        return st["out"]
    if kind == "labels":
        u, g = st["u"].data_ptr(), st["grad"].data_ptr()
        lo, hi = potts.min_max(ctx, m, u)
        potts.grad_magn(ctx, m, u, g)
        counts, density, _, _ = potts.calc_hist_auto(ctx, m, u, case["bins"])
        hist2, ranges = potts.uv_hist_auto(ctx, m, u, g, case["bins2"])
        return {"range": [lo, hi], "grad": st["grad"], "counts": counts, "density": density, "hist2": hist2,
                "ranges2": list(ranges)}
    lo, hi, hist = potts.find_intensity_range(ctx, m, st["raw"].data_ptr(), TAIL)
    potts.convert_to_fp(ctx, m, "u16", st["raw"].data_ptr(), float(lo), float(hi), st["out"].data_ptr())
    return {"lo": lo, "hi": hi, "hist": hist, "u": st["out"]}


# ---- what a pass cannot do without ------------------------------------------------------------------
def _voxels(case) -> int:
    if case["kind"] == "batch":
        sizes = np.random.default_rng(1234)
        total = 0
        for _ in range(case["count"]):
            n, rows, cols = (int(v) for v in sizes.integers(case["side_min"], case["side_max"] + 1, size=3))
            sizes.uniform(), sizes.uniform()
            total += CylinderMapping.cylinder(n, rows, cols, 0.47 * min(rows, cols)).data_size
        return total
    return _mapping(case).data_size


def work(case):
    """Iterations follow one another, so each has to read and write the state once: 4 (K - 1) values
    (the dual field's three components and the relaxed indicator of all labels but the last) and u.
    Operations: a divergence, a projection onto the simplex, a gradient and the pair distances."""
    kind, vox = case["kind"], _voxels(case)
    k = case.get("k", 3)
    step_flops = 33 * k + 8 * k * (k - 1) // 2
    if kind in ("solve", "batch"):
        es = 2 if case.get("storage", "f32") in ("bf16", "f16") else 4
        return {"bytes": vox * (case["iters"] * (8 * (k - 1) * es + 4) + 4 * (k - 1) + 1),
                "flops": vox * case["iters"] * step_flops}
    if kind == "unroll":
        # the forward pass; then per iteration the state of that iteration recomputed and read, and the
        # adjoints of the state read and written
        it = 2 * (8 * (k - 1) * 4 + 4) + (4 * (k - 1) + 8 * (k - 1)) * 4 + 12
        return {"bytes": vox * case["iters"] * it, "flops": vox * case["iters"] * 4 * step_flops}
    if kind == "tv":
        return {"bytes": vox * (case["iters"] * 28 + 8), "flops": vox * case["iters"] * 40}
    if kind == "labels":
        # u for the range, u in and its gradient out, u for the 1-D histogram's range and counts, both
        # fields for the 2-D histogram's ranges and counts
        return {"bytes": vox * (4 + 8 + 8 + 16), "flops": vox * 40}
    return {"bytes": vox * (2 + 2 + 4), "flops": vox * 3}


# ---- the same in 64 bits ----------------------------------------------------------------------------
class _Box:
    """Dense (col, row, n) boxes of a mapping in 64 bits; zero outside the mask."""

    def __init__(self, mapping):
        self.m = mapping
        rows, cols = mapping.lines()
        self.rows, self.cols = torch.from_numpy(rows).cuda(), torch.from_numpy(cols).cuda()
        mask = torch.zeros((mapping.cols, mapping.rows, 1), dtype=torch.float64, device="cuda")
        mask[self.cols, self.rows, 0] = 1.0
        self.mask = mask
        self.fwd_r, self.fwd_c = torch.zeros_like(mask), torch.zeros_like(mask)
        self.fwd_r[:, :-1] = mask[:, :-1] * mask[:, 1:]
        self.fwd_c[:-1] = mask[:-1] * mask[1:]

    def of(self, span):
        lines = span.view(self.m.n_lines, self.m.nstride)[:, : self.m.n_images].double()
        box = torch.zeros((self.m.cols, self.m.rows, self.m.n_images), dtype=torch.float64, device="cuda")
        box[self.cols, self.rows] = lines
        return box

    def span(self, box):
        out = torch.zeros((self.m.n_lines, self.m.nstride), dtype=box.dtype, device="cuda")
        out[:, : self.m.n_images] = box[self.cols, self.rows]
        return out.reshape(-1)

    def grad(self, v):
        pad = torch.nn.functional.pad
        return (pad(v[:, :, 1:] - v[:, :, :-1], (0, 1)) * self.mask,
                pad(v[:, 1:] - v[:, :-1], (0, 0, 0, 1)) * self.fwd_r,
                pad(v[1:] - v[:-1], (0, 0, 0, 0, 0, 1)) * self.fwd_c)

    def div(self, x):
        pad = torch.nn.functional.pad
        a = pad(x[0][:, :, :-1], (0, 1)) * self.mask  # nothing leaves through the last slice
        b, c = x[1] * self.fwd_r, x[2] * self.fwd_c
        return (a - pad(a[:, :, :-1], (1, 0)) + b - pad(b[:, :-1], (0, 0, 1, 0)) + c
                - pad(c[:-1], (0, 0, 0, 0, 1, 0)))


def _project_pairs(q):
    """Dykstra's projection of q[label][axis] onto |q_i - q_j| <= 1: at most 20 sweeps over the pairs,
    until every step of a sweep is shorter than 1e-6 (voxel by voxel)."""
    k = len(q)
    pairs = [(i, j) for i in range(k - 1) for j in range(i + 1, k)]
    with torch.no_grad():
        far = None
        for i, j in pairs:
            s = sum((q[j][a] - q[i][a]) ** 2 for a in range(3)) > 1.0
            far = s if far is None else far | s
        at = far.nonzero(as_tuple=True)
    if at[0].numel() == 0:
        return q
    z = [torch.stack([q[i][a][at] for a in range(3)]) for i in range(k)]
    p = [torch.zeros_like(z[0]) for _ in pairs]
    live = torch.ones(z[0].shape[1], dtype=torch.float64, device=z[0].device)
    for _ in range(20):
        longest = torch.zeros_like(live)
        for w, (i, j) in enumerate(pairs):
            h = z[j] - z[i] + p[w]
            new = h * (1.0 - 1.0 / (h * h).sum(0).clamp(min=1.0).sqrt())
            d = 0.5 * (new - p[w]) * live
            longest = torch.maximum(longest, (d.detach() ** 2).sum(0).sqrt())
            z[i], z[j] = z[i] + d, z[j] - d
            p[w] = p[w] + (new - p[w]) * live
        live = live * (longest >= 1e-6)
        if not bool(live.any()):
            break
    return [[q[i][a].index_put(at, z[i][a]) for a in range(3)] for i in range(k)]


def _project_simplex(q):
    k = len(q)
    u = list(q)
    for r in range(k):
        for i in range(r & 1, k - 1, 2):
            u[i], u[i + 1] = torch.maximum(u[i], u[i + 1]), torch.minimum(u[i], u[i + 1])
    total, theta = u[0], u[0] - 1.0
    for i in range(1, k):
        total = total + u[i]
        theta = torch.maximum(theta, (total - 1.0) / (i + 1))
    return [(x - theta).clamp(min=0.0) for x in q]


def _iterate(box, v, vb, xi, u, c, lam, tau):
    """One primal-dual iteration: v, vb lists of K - 1 boxes, xi of K - 1 triples."""
    k = len(v) + 1
    full = [*vb, 1.0 - sum(vb)]
    last = [-sum(x[a] for x in xi) for a in range(3)]
    xs = [*xi, last]
    q = []
    for i in range(k):
        g = box.grad(full[i])
        q.append([xs[i][a] + tau * g[a] for a in range(3)])
    q = _project_pairs(q)
    xi = q[:-1]
    xs = [*xi, [-sum(x[a] for x in xi) for a in range(3)]]
    vs = [*v, 1.0 - sum(v)]
    w = _project_simplex([vs[i] + tau * (box.div(xs[i]) - lam * (u - c[i]) ** 2) for i in range(k)])
    dq = sum((w[i] - vs[i]) ** 2 for i in range(k))
    return w[:-1], [2.0 * w[i] - vs[i] for i in range(k - 1)], xi, dq


def _start(box, u, c):
    k = len(c)
    near = torch.stack([(u - x).abs() for x in c]).argmin(0)
    v = [(near == i).double() for i in range(k - 1)]
    zero = torch.zeros_like(u)
    return v, list(v), [[zero, zero, zero] for _ in range(k - 1)]


def _f32(*values):
    return [float(np.float32(x)) for x in values]


def _solve64(mapping, u_span, ci, lam, iters, gap_every=0):
    box = _Box(mapping)
    u = box.of(u_span)
    c = _f32(*ci)
    lam, tau = _f32(lam, _tau())
    v, vb, xi = _start(box, u, c)
    trace, energy = [], []
    for it in range(iters):
        v, vb, xi, dq = _iterate(box, v, vb, xi, u, c, lam, tau)
        trace.append(float((dq * box.mask).max()))
        if gap_every and (it + 1) % gap_every == 0:
            xs = [*xi, [-sum(x[a] for x in xi) for a in range(3)]]
            e = torch.stack([lam * (u - c[i]) ** 2 - box.div(xs[i]) for i in range(len(c))])
            lag = float((e * torch.stack([*v, 1.0 - sum(v)]) * box.mask).sum())
            dual = float((e.min(0).values * box.mask).sum())
            energy.append([lag, dual, lag - dual])
    full = torch.stack([*v, 1.0 - sum(v)])
    label = full.argmax(0)
    res = torch.tensor(c, dtype=torch.float64, device="cuda")[label]
    # the energies' difference cancels: only the two sums have a value to compare
    return {"V": torch.stack([box.span(x) for x in v]), "labels": box.span(label.to(torch.uint8)),
            "Xi": torch.stack([box.span(a) for x in xi for a in x]), "res": box.span(res), "dq": np.array(trace),
            "energy": np.array(energy) if gap_every else None}


def _unroll64(case, u_span, truth_span, ci):
    from torch.utils.checkpoint import checkpoint

    m = _mapping(case)
    box = _Box(m)
    k = case["k"]
    (tau, eps) = _f32(_tau(), LOSS_EPS)
    u = box.of(u_span).requires_grad_(True)
    c = torch.tensor(_f32(*ci), dtype=torch.float64, device="cuda", requires_grad=True)
    lam = torch.tensor(_f32(LAMBDA)[0], dtype=torch.float64, device="cuda", requires_grad=True)
    with torch.no_grad():
        v, vb, xi = _start(box, u.detach(), c.detach())

    def step(u, c, lam, *flat):
        v, vb = list(flat[: k - 1]), list(flat[k - 1: 2 * k - 2])
        x = flat[2 * k - 2:]
        v, vb, xi, _ = _iterate(box, v, vb, [list(x[3 * i: 3 * i + 3]) for i in range(k - 1)], u, c, lam, tau)
        return (*v, *vb, *(a for t in xi for a in t))

    flat = (*v, *vb, *(a for t in xi for a in t))
    for _ in range(case["iters"]):
        flat = checkpoint(step, u, c, lam, *flat, use_reentrant=False)
    v = list(flat[: k - 1])
    t = box.of(truth_span).long()
    vt = torch.stack([*v, 1.0 - sum(v)]).gather(0, t[None])[0]
    loss = -(torch.log(vt + eps) * box.mask).sum() / m.data_size
    loss.backward()
    return {"loss": float(loss.detach()), "V": torch.stack([box.span(x.detach()) for x in v]),
            "grad_u": box.span(u.grad), "grad_c": c.grad.cpu().numpy(), "grad_lambda": float(lam.grad)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        got = [_solve64(m, u, ci, lam, case["iters"]) for m, u, ci, lam in _batch_volumes(case, seed)]
        return {"V": [g["V"] for g in got], "labels": [g["labels"] for g in got]}
    vox = _voxels(case)
    m = _mapping(case)
    if kind == "solve":
        if vox * case["iters"] * (case["k"] - 1) > 12e9:
            return None
        u, _, ci = _core(m, case["k"], seed)
        got = _solve64(m, u, ci, LAMBDA, case["iters"], case["gap_every"])
        if case["host"]:
            del got["V"]
        if case["host"] or not case["dual"]:
            del got["Xi"]
        if not case["gap_every"]:
            del got["energy"]
        return got
    if kind == "unroll":
        u, truth, ci = _core(m, case["k"], seed)
        return _unroll64(case, u, truth, ci)
    u, _, _ = _core(m, 3, seed)
    if kind == "tv":
        if vox * case["iters"] > 40e9:
            return None
        box = _Box(m)
        g = box.of(u)
        lam, tau = _f32(TV_LAMBDA, TV_TAU)
        gg = [x / lam for x in box.grad(g)]
        xi = [torch.zeros_like(g) for _ in range(3)]
        for _ in range(case["iters"]):
            d = [a - b for a, b in zip(box.grad(box.div(xi)), gg)]
            denom = 1.0 + tau * (d[0] ** 2 + d[1] ** 2 + d[2] ** 2).sqrt()
            xi = [(x + tau * y) / denom for x, y in zip(xi, d)]
        return box.span(g - lam * box.div(xi))
    if kind == "labels":
        box = _Box(m)
        g = box.of(u)
        inner = torch.zeros_like(g)
        inner[1:-1, 1:-1, 1:-1] = (box.mask[1:-1, 1:-1] * box.mask[1:-1, 2:] * box.mask[1:-1, :-2]
                                   * box.mask[2:, 1:-1] * box.mask[:-2, 1:-1])
        s = torch.zeros_like(g)
        s[:, :, 1:-1] += (g[:, :, 2:] - g[:, :, :-2]) ** 2
        s[:, 1:-1] += (g[:, 2:] - g[:, :-2]) ** 2
        s[1:-1] += (g[2:] - g[:-2]) ** 2
        v = box.span(torch.where(inner > 0, 0.5 * s.sqrt(), torch.full_like(s, -1.0)))
        values = u.view(m.n_lines, m.nstride)[:, : m.n_images]
        pos = v[v > 0]
        lo, hi = float(values.min()), float(values.max())
        # the counts are whole numbers of the FP32 positions
        return {"range": [lo, hi], "grad": v, "counts": None, "density": None, "hist2": None,
                "ranges2": [lo, hi, float(pos.min()), float(pos.max())]}
    raw = (u * 30000.0 + 12000.0).to(torch.int32)
    lines = raw.view(m.n_lines, m.nstride)[:, : m.n_images].reshape(-1)
    hist = torch.bincount(lines.long(), minlength=65536).cpu().numpy()
    cum, total = np.cumsum(hist).astype(np.float64), float(hist.sum())
    below = np.nonzero(TAIL * total >= cum)[0]
    lo = int(below[-1]) if below.size else 0
    hi = int(np.nonzero((1.0 - TAIL) * total <= cum)[0][0])
    out = torch.zeros((m.n_lines, m.nstride), dtype=torch.float64, device="cuda")
    x = raw.view(m.n_lines, m.nstride)[:, : m.n_images].double()
    out[:, : m.n_images] = ((x - lo) / float(hi - lo)).clamp(0.0, 1.0)
    return {"lo": lo, "hi": hi, "hist": None, "u": out.reshape(-1)}
