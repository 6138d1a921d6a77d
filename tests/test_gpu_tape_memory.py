"""The device buffers that are kept of a closed tape: bounded by what is free, given back to whoever in the
process asks through the library, safe with several threads, and not touched under stream capture."""
import queue
import threading

import numpy as np
import pytest

from segmentctscans_b200 import potts
from tests._cases import TAU, random_volume

pytestmark = pytest.mark.gpu

MB = 1 << 20


def volume(n, side, k, seed):
    m, u, ci = random_volume(n, side, side, 0.45 * side, k, seed=seed)
    rng = np.random.default_rng(seed)
    return m, u, ci, rng.integers(0, k, m.span).astype(np.uint8)


class Inputs:
    def __init__(self, vol):
        import torch

        self.m, u, self.ci, truth = vol
        self.u, self.truth = torch.from_numpy(u).cuda(), torch.from_numpy(truth).cuda()
        self.g = torch.zeros(self.m.span, device="cuda")
        torch.cuda.synchronize()

    def tape(self, ctx, every=9):
        return potts.Tape(ctx, self.m, self.u.data_ptr(), self.truth.data_ptr(), self.ci, 30.0, TAU, TAU, 9, every)


def free_bytes():
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def test_any_context_and_its_end_give_the_memory_back(cuda_device):
    a = Inputs(volume(160, 150, 3, 6))
    with potts.make_context(0) as ctx, potts.make_context(0) as other:
        before = free_bytes()
        a.tape(ctx).close()
        kept = before - free_bytes()
        assert 256 * MB < kept
        assert abs(other.device_memory()[0] - before) < 64 * MB
        other.trim()
        assert abs(free_bytes() - before) < 64 * MB
        a.tape(ctx).close()
        ctx.close()
        assert abs(free_bytes() - before) < 64 * MB
        # a tape closed after its context is not kept, though another context lives
        third = potts.make_context(0)
        t = a.tape(third)
        third.close()
        t.close()
        assert abs(free_bytes() - before) < 64 * MB


def test_scarce_memory(cuda_device):
    """A solve of another context that does not fit beside the kept buffers gets their memory; nothing is
    kept where it would be more than an eighth of what is free."""
    import torch

    a = Inputs(volume(160, 150, 3, 6))
    u = a.u.cpu().numpy()
    with potts.make_context(0) as ctx, potts.make_context(0) as other:
        a.tape(ctx).close()
        filler = torch.empty(free_bytes() - 600 * MB, dtype=torch.uint8, device="cuda")
        try:
            kept = free_bytes()
            st = potts.solve_host(other, a.m, u, a.ci, 30.0, TAU, TAU, 2, stats=True)
            assert st.n_slabs == 1
            other.close()
            assert free_bytes() > kept + 256 * MB
            before = free_bytes()
            a.tape(ctx).close()
            assert abs(free_bytes() - before) < 64 * MB
        finally:
            del filler
            torch.cuda.empty_cache()


def test_threads_close_each_other_s_tapes(cuda_device):
    """Two threads with a context each, tapes of several sizes; every tape is closed by the other thread."""
    vols = [volume(24, 22, 3, 1), volume(40, 30, 3, 3), volume(24, 22, 4, 4), volume(9, 12, 2, 5)]
    want = []
    for v in vols:
        a = Inputs(v)
        with potts.make_context(0) as ctx, a.tape(ctx, 4) as t:
            t.backward(a.g.data_ptr())
            want.append(a.g.cpu().numpy())
    before = free_bytes()
    boxes = [queue.Queue(), queue.Queue()]
    start, errors = threading.Barrier(2), []

    def work(me):
        try:
            with potts.make_context(0) as ctx:
                inputs = [Inputs(v) for v in vols]
                start.wait(30)
                for rep in range(24):
                    i = (rep * (me + 1) + me) % len(vols)
                    t = inputs[i].tape(ctx, 4)
                    t.backward(inputs[i].g.data_ptr())
                    ctx.synchronize()
                    if not np.array_equal(inputs[i].g.cpu().numpy(), want[i]):
                        errors.append((me, rep, i))
                    boxes[1 - me].put(t)
                    boxes[me].get(timeout=60).close()
        except Exception as e:  # reported below
            errors.append((me, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(180)
    assert not any(t.is_alive() for t in threads) and not errors, errors
    assert abs(free_bytes() - before) < 64 * MB


def test_a_captured_solve_leaves_the_kept_buffers(cuda_device):
    """Nothing can be freed while a stream is captured: a split solve on a planned mapping is captured and
    replayed with a closed tape's buffers in place."""
    import torch

    a = Inputs(volume(24, 22, 3, 1))
    lab = torch.zeros(a.m.span, dtype=torch.uint8, device="cuda")
    side = torch.cuda.Stream()

    def solve(ctx):
        potts.solve_device(ctx, a.m, a.u.data_ptr(), a.ci, 30.0, TAU, TAU, 6, labels_ptr=lab.data_ptr(), variant=1,
                           track_dq=0, stats=False)

    with potts.make_context(0, stream=side.cuda_stream) as ctx:
        solve(ctx)
        side.synchronize()
        want = lab.clone()
        a.tape(ctx).close()
        lab.zero_()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            solve(ctx)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(lab, want)
        del graph
