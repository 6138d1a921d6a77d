"""The differentiable solve for every list layout of its kernels (K = 2, 4 and 6: up to 512 or 256 loop
voxels per block) against the same iterations unrolled in FP64 by PyTorch's autograd on the CPU: the whole
gradient of u, those of the labels and lambda, and the loss.

Two volumes: one whose blocks empty their list between chunks (most voxels in the projection loop, two
chunks per line, the last block not full) and one with short ragged lines.  Bound: this unroll in FP32 is off
from the FP64 one by at most 9.1e-5 (relative L2, over the six cases and four outputs); ten times that."""
import numpy as np
import pytest
import torch

from segmentctscans_b200 import potts
from segmentctscans_b200.layout import CylinderMapping

pytestmark = pytest.mark.gpu

EPS = 1e-3
BOUND = 1e-3
# share: the least share of voxels in the projection loop in the last iteration
CASES = [
    {"name": "full_lists", "n": 509, "rows": 9, "cols": 9, "r": 3.9, "lam": 2.0, "tau1": 0.2, "tau2": 1.5, "iters": 4,
     "share": 0.6},
    {"name": "ragged_lines", "n": 37, "rows": 15, "cols": 14, "r": 6.7, "lam": 6.0, "tau1": 0.28, "tau2": 0.28,
     "iters": 6, "share": 0.0},
]


def inputs(case, K):
    """Every voxel its own label and some noise, so that neighbours differ."""
    rng = np.random.default_rng(10 * K + case["n"])
    m = CylinderMapping.cylinder(case["n"], case["rows"], case["cols"], case["r"])
    ci = [float(np.float32((i + 0.5) / K)) for i in range(K)]
    u = (np.asarray(ci, np.float32)[rng.integers(0, K, m.span)] + rng.uniform(-0.3, 0.3, m.span) / K).astype(np.float32)
    return m, u, rng.integers(0, K, m.span).astype(np.uint8), ci


class Box:
    """Dense (col, row, n) boxes of a mapping; zero outside the mask."""

    def __init__(self, m, dtype):
        rows, cols = m.lines()
        self.m, self.dtype = m, dtype
        self.rows, self.cols = torch.from_numpy(rows), torch.from_numpy(cols)
        mask = torch.zeros((m.cols, m.rows, 1), dtype=dtype)
        mask[self.cols, self.rows, 0] = 1
        self.fwd = [torch.ones((m.cols, m.rows, m.n_images), dtype=dtype) * mask, torch.zeros_like(mask),
                    torch.zeros_like(mask)]
        self.fwd[0][:, :, -1] = 0
        self.fwd[1][:, :-1] = mask[:, :-1] * mask[:, 1:]
        self.fwd[2][:-1] = mask[:-1] * mask[1:]
        self.mask = mask

    def of(self, span):
        lines = torch.from_numpy(span).view(self.m.n_lines, self.m.nstride)[:, : self.m.n_images]
        box = torch.zeros((self.m.cols, self.m.rows, self.m.n_images), dtype=lines.dtype)
        box[self.cols, self.rows] = lines
        return box

    @staticmethod
    def next(v, a):  # the next voxel along n, row, column (what lies past the end is masked)
        return torch.roll(v, -1, (2, 1, 0)[a])

    def grad(self, v):
        return [(self.next(v, a) - v) * self.fwd[a] for a in range(3)]

    def div(self, x):
        return sum(x[a] * self.fwd[a] - torch.roll(x[a] * self.fwd[a], 1, (2, 1, 0)[a]) for a in range(3))


def project_pairs(q):
    """q[label][axis] onto |q_i - q_j| <= 1 by Dykstra's algorithm; the share of voxels that need it."""
    K = len(q)
    pairs = [(i, j) for i in range(K - 1) for j in range(i + 1, K)]
    z = [torch.stack(x) for x in q]
    with torch.no_grad():
        far = torch.stack([((z[j] - z[i]) ** 2).sum(0) > 1 for i, j in pairs]).any(0)
    live = far.to(z[0].dtype)
    p = [torch.zeros_like(z[0]) for _ in pairs]
    for _ in range(20):
        longest = torch.zeros_like(live)
        for w, (i, j) in enumerate(pairs):
            h = z[j] - z[i] + p[w]
            step = (h * (1 - 1 / (h * h).sum(0).clamp(min=1).sqrt()) - p[w]) * live
            longest = torch.maximum(longest, (0.25 * step.detach() ** 2).sum(0))
            z[i], z[j], p[w] = z[i] + 0.5 * step, z[j] - 0.5 * step, p[w] + step
        live = live * (longest >= 1e-12)
        if not live.any():
            break
    return [list(x) for x in z], far


def project_simplex(q):
    s = torch.stack(q).sort(0, descending=True).values
    theta = ((s.cumsum(0) - 1) / torch.arange(1, len(q) + 1, dtype=s.dtype).view(-1, 1, 1, 1)).max(0).values
    return [(x - theta).clamp(min=0) for x in q]


def unroll(case, m, u, truth, ci, dtype):
    box = Box(m, dtype)
    K = len(ci)
    tau1, tau2 = (torch.tensor(np.float32(case[t]), dtype=dtype) for t in ("tau1", "tau2"))
    ub = box.of(u).to(dtype).requires_grad_(True)
    c = torch.tensor(ci, dtype=dtype, requires_grad=True)
    lam = torch.tensor(case["lam"], dtype=dtype, requires_grad=True)
    near = torch.stack([(ub.detach() - x).abs() for x in c.detach()]).argmin(0)
    v = [(near == i).to(dtype) for i in range(K)]
    vb, xi = list(v), [[torch.zeros_like(v[0])] * 3 for _ in range(K)]
    for _ in range(case["iters"]):
        q = []
        for i in range(K):
            g = box.grad(vb[i])
            q.append([xi[i][a] + tau2 * g[a] for a in range(3)])
        xi, far = project_pairs(q)
        w = project_simplex([v[i] + tau1 * (box.div(xi[i]) - lam * (ub - c[i]) ** 2) for i in range(K)])
        v, vb = w, [2 * w[i] - v[i] for i in range(K)]
    vt = torch.stack(v).gather(0, box.of(truth).long()[None])[0]
    loss = -(torch.log(vt + EPS) * box.mask).sum() / m.data_size
    loss.backward()
    return {"loss": float(loss.detach()), "grad_u": ub.grad[box.cols, box.rows].double().numpy(),
            "grad_c": c.grad.double().numpy(), "grad_lam": float(lam.grad),
            "share": float((far * box.mask).sum()) / m.data_size}


@pytest.mark.parametrize("K", [2, 4, 6])
@pytest.mark.parametrize("case", CASES, ids=[c["name"] for c in CASES])
def test_gradient_of_the_unrolled_solve(cuda_device, case, K):
    m, u, truth, ci = inputs(case, K)
    want = unroll(case, m, u, truth, ci, torch.float64)
    assert want["share"] > case["share"]
    du, dt = torch.from_numpy(u).cuda(), torch.from_numpy(truth).cuda()
    g = torch.zeros(m.span, device="cuda")
    torch.cuda.synchronize()
    with potts.make_context(0) as ctx:
        with potts.Tape(ctx, m, du.data_ptr(), dt.data_ptr(), ci, case["lam"], case["tau1"], case["tau2"],
                        case["iters"], 2) as t:
            gc, gl = t.backward(g.data_ptr())
            loss = t.loss
        ctx.synchronize()
    got = m.mask_values(g.cpu().numpy())
    assert abs(loss - want["loss"]) <= BOUND * abs(want["loss"])
    assert np.linalg.norm(got - want["grad_u"]) <= BOUND * np.linalg.norm(want["grad_u"])
    assert np.linalg.norm(gc - want["grad_c"]) <= BOUND * np.linalg.norm(want["grad_c"])
    assert abs(gl - want["grad_lam"]) <= BOUND * abs(want["grad_lam"])
