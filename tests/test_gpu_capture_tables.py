"""A call captured while the context's work list is another call's: the list's host memory ends with the call,
so its copy must not become a node of the graph, which would read it again at every replay.  Such a
capture is refused; planned, the call is captured and replayed."""
import pytest

from segmentctscans_b200 import _native, potts
from tests._cases import TAU, random_volume

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
def test_work_lists_under_capture(cuda_device, mode):
    import torch

    m, u, ci = random_volume(68, 66, 61, 29.2, 3, seed=2)
    du = torch.from_numpy(u).cuda()
    g = du.clone()
    lab = torch.zeros(m.span, dtype=torch.uint8, device="cuda")
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with potts.make_context(0, stream=side.cuda_stream) as ctx:
        def solve():
            potts.solve_device(ctx, m, du.data_ptr(), ci, 30.0, TAU, TAU, 5, labels_ptr=lab.data_ptr(), stats=False)
            side.synchronize()

        def denoise():
            potts.tv_denoise(ctx, m, g.data_ptr(), 0.06, 0.16, 6, stats=False)

        def reset():
            g.copy_(du)
            lab.zero_()
            torch.cuda.synchronize()

        denoise()
        side.synchronize()
        want = g.clone()
        solve()  # the list is now the solve's
        labels = lab.clone()
        refused = torch.cuda.CUDAGraph()
        with torch.cuda.graph(refused, stream=side, capture_error_mode=mode):
            with pytest.raises(_native.PottsError):
                denoise()
        reset()
        solve()  # its list is as it was
        denoise()
        side.synchronize()
        assert torch.equal(lab, labels) and torch.equal(g, want)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side, capture_error_mode=mode):
            denoise()
        for _ in range(2):
            reset()
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(g, want)
        del graph, refused
