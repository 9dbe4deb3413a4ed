"""Float64 TaylorF2 with time marginalisation captured into a CUDA graph: the same
kernel, and so the same bits, as an eager call, whatever was evaluated before."""
import numpy as np
import pytest

from oracle import data as OD
from tests.gpu_helpers import device_analysis, draw_points, params_block, small_workload

pytestmark = pytest.mark.gpu


# windows whose convolutions differ, and an FFT length (7 * 512) that no other test has
@pytest.mark.parametrize("before,after", [(0.2, 0.02), (0.6, 0.3)])
def test_captured_directly_after_the_window_changed(gpu, before, after):
    torch = pytest.importorskip("torch")
    w = small_workload("tf2_marg_8s", duration=7.0, sampling_frequency=1024.0)
    w = small_workload("tf2_marg_8s", **{**w.__dict__, "injection": dict(w.injection, geocent_time=w.start_time + 3.5)})
    an = device_analysis(OD.build_workload(w), w.model, w)
    mid = w.start_time + 3.5
    p = draw_points(w, 40, np.random.default_rng(2))
    p["geocent_time"] = np.full(40, w.start_time)
    block = torch.from_numpy(params_block(p)).cuda()
    out = torch.zeros(40, dtype=torch.float64, device="cuda")
    stream = torch.cuda.Stream()
    an.set_time_marginalization(True, True, mid - before, mid + before)
    with torch.cuda.stream(stream):
        an.log_likelihood_ratio_device(block.data_ptr(), 40, out.data_ptr(), "fp64", stream.cuda_stream)
        an.log_likelihood_ratio_device(block.data_ptr(), 40, out.data_ptr(), "mixed", stream.cuda_stream)
    torch.cuda.synchronize()
    an.set_time_marginalization(True, True, mid - after, mid + after)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        an.log_likelihood_ratio_device(block.data_ptr(), 40, out.data_ptr(), "fp64", stream.cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), an.log_likelihood_ratio_host(params_block(p), "fp64"))
    an.close()
