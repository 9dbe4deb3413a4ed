"""The float64 TaylorF2 likelihood with time marginalisation on the 32-bit pipes
(csrc/gwl_wide_tm.cu) against the oracle, where the convolution's plan changes.

Tolerance: the marginalised lnL moves by at most the largest error of a sample's
<d|h>(t_j), so the bound of tests/test_gpu_wide.py holds with the scale max(1,
max_j |<d|h>(t_j)|, <h|h> / 2)."""
import numpy as np
import pytest

from oracle import data as OD
from oracle import restate as R
from tests.gpu_helpers import device_analysis, draw_points, params_block, point, small_workload

pytestmark = pytest.mark.gpu


# samples of the prior window: two, 502 and 503 (the convolution's length goes from
# 1024 to 2048), 2038 and 2039 (4096 to 8192), 4086 and 4087 (the longest, then the
# whole transform); bands inside one block of the convolution (10-40 Msun), of many
# (0.7-2 Msun at 8 s) and empty (f_ISCO below 20 Hz); FFT lengths 2^p, 3 2^p
@pytest.mark.parametrize("detectors,duration,fs,masses,samples,phase", [
    (2, 6.0, 2048.0, (10.0, 40.0), 410, True), (1, 4.0, 2048.0, (1.0, 2.0), 2, False),
    (3, 8.0, 2048.0, (0.7, 2.0), 502, False), (3, 8.0, 2048.0, (0.7, 2.0), 503, True),
    (4, 4.0, 4096.0, (5.0, 40.0), 2038, True), (2, 4.0, 4096.0, (5.0, 40.0), 2039, False),
    (1, 8.0, 2048.0, (2.0, 60.0), 4086, False), (1, 8.0, 2048.0, (2.0, 60.0), 4087, True),
    (2, 3.0, 640.0, (100.0, 300.0), 100, False), (2, 3.0, 1024.0, (3.0, 9.0), 100, True)])
def test_against_the_oracle(gpu, detectors, duration, fs, masses, samples, phase):
    w = small_workload("tf2_marg_8s", detectors=("H1", "L1", "V1")[:min(detectors, 3)], duration=duration,
                       sampling_frequency=fs, mass_range=masses)
    w = small_workload("tf2_marg_8s", **{**w.__dict__, "injection": dict(
        w.injection, mass_1=masses[1], mass_2=masses[0], geocent_time=w.start_time + 0.6 * duration)})
    dets = OD.build_workload(w)
    dets = (dets + dets)[:detectors]
    an = device_analysis(dets, "taylorf2", w)
    mid, half = w.start_time + 0.6 * duration, samples / fs
    lo, hi = max(mid - half, w.start_time - 0.01), mid + half
    lo = hi - 2 * half if lo < mid - half else lo
    an.set_time_marginalization(True, True, lo, hi)
    an.set_phase_marginalization(phase)
    p = draw_points(w, 7, np.random.default_rng(3))
    for k in w.injection:
        p[k][0] = w.injection[k]
    p["geocent_time"] = np.full(7, w.start_time)
    if phase:
        p["phase"] = np.zeros(7)
    block = params_block(p)
    got = an.log_likelihood_ratio_host(block, "fp64")
    assert np.array_equal(np.concatenate([an.log_likelihood_ratio_host(block[:, i:i + 1], "fp64") for i in range(7)]), got)
    m = R.Marginalization(time=True, phase=phase)
    R.setup_time_marginalization(m, w.start_time, duration, fs, lo, hi)
    src = OD.source_for(w.model, w.minimum_frequency)
    for i in range(7):
        q = point(p, i)
        ref = R.log_likelihood_ratio(dets, src, q, m, lambda t: np.full(len(t), 1 / (hi - lo)))
        q["geocent_time"] += q["time_jitter"]
        parts = [R.snrs(d, src(d.frequency, **q), q, True) for d in dets]
        scale = max(1.0, np.max(np.abs(sum(x[2] for x in parts))), sum(x[1] for x in parts) / 2)
        mc = (q["mass_1"] * q["mass_2"]) ** 0.6 / (q["mass_1"] + q["mass_2"]) ** 0.2 * 4.925490947641267e-06
        psi = 3 / 128 * (np.pi * mc * 20.0) ** (-5 / 3)
        assert abs(got[i] - ref) <= max(1e-9, 8 * 2.0 ** -53 * psi) * scale, (i, got[i], ref)
    an.close()


# the sum of the samples' I0 below 500, their lnL above; a flat and a tabulated prior
@pytest.mark.parametrize("tabulated", [False, True])
@pytest.mark.parametrize("largest", [3.0, 499.0, 501.0, 5000.0])
def test_loudness(gpu, largest, tabulated):
    w = small_workload("tf2_marg_8s", duration=4.0, sampling_frequency=2048.0)
    w = small_workload("tf2_marg_8s", **{**w.__dict__, "injection": dict(w.injection, geocent_time=w.start_time + 2.0)})
    dets = OD.build_workload(w)
    an = device_analysis(dets, "taylorf2", w)
    lo, hi = w.start_time + 1.9, w.start_time + 2.1
    an.set_time_marginalization(True, True, lo, hi)
    an.set_phase_marginalization(True)
    density = lambda t: np.full(np.shape(t), 1 / (hi - lo))
    if tabulated:  # linear in time: exact in the four-node interpolation
        h, t0 = 2.0 ** -8, np.floor(lo * 2 ** 8 - 2) * 2.0 ** -8
        nodes = t0 + h * np.arange(int((hi - t0) / h) + 4)
        density = lambda t: 5.0 + 20.0 * (np.asarray(t) - (w.start_time + 2.0))
        an.set_time_prior(np.maximum(density(nodes), 0.0), t0, h)
    m = R.Marginalization(time=True, phase=True)
    R.setup_time_marginalization(m, w.start_time, w.duration, w.sampling_frequency, lo, hi)
    src = OD.source_for(w.model, w.minimum_frequency)
    q = dict(w.injection, phase=0.0, geocent_time=w.start_time, time_jitter=1e-4)
    late = dict(q, geocent_time=w.start_time + 1e-4)
    arr = sum(R.snrs(d, src(d.frequency, **late), late, True)[2] for d in dets)
    inside = (m.times + 1e-4 >= lo) & (m.times + 1e-4 <= hi)
    q["luminosity_distance"] *= np.max(np.abs(arr[inside])) / largest
    ref = R.log_likelihood_ratio(dets, src, q, m, density)
    hh = sum(R.snrs(d, src(d.frequency, **q), q)[1] for d in dets)
    got = an.log_likelihood_ratio_host(params_block(q), "fp64")[0]
    assert abs(got - ref) <= 1e-9 * max(1.0, largest, hh / 2), (got, ref)
    an.close()


# mixed precision at FFT length 16384: the last pass for the window's outputs alone up
# to 512 of them (two per group of 16), the whole pass above.  Tolerance: the mixed
# precision's 1e-3 against float64 (windows at the start, the middle and the wrap).
@pytest.mark.parametrize("samples", [1, 255, 256, 257, 502, 503, 504, 700])
@pytest.mark.parametrize("at", [0.02, 0.5, 0.999])
def test_mixed_windows(gpu, samples, at):
    w = small_workload("tf2_marg_8s")
    w = small_workload("tf2_marg_8s", **{**w.__dict__, "injection": dict(w.injection, geocent_time=w.start_time + 8 * at)})
    an = device_analysis(OD.build_workload(w), "taylorf2", w)
    mid, half = w.start_time + 8 * at, (samples - 0.5) * 8 / 16384 / 2
    an.set_time_marginalization(True, True, mid - half, mid + half)
    an.set_phase_marginalization(True)
    p = draw_points(w, 8, np.random.default_rng(6))
    for k, v in w.injection.items():
        p[k][:3] = v
    p["geocent_time"], p["phase"] = np.full(8, w.start_time), np.zeros(8)
    block = params_block(p)
    fp64, mixed = an.log_likelihood_ratio_host(block, "fp64"), an.log_likelihood_ratio_host(block, "mixed")
    same = np.isinf(fp64)
    assert np.array_equal(mixed[same], fp64[same])
    assert np.all(np.abs(mixed - fp64)[~same] <= 1e-3), np.abs(mixed - fp64).max()
    an.close()


@pytest.mark.parametrize("time", [False, True])
@pytest.mark.parametrize("workload", ["tf2_marg_8s", "sg_4s"])
def test_float64_captured_after_a_mixed_call(gpu, workload, time):
    """A mixed call leaves nothing for a float64 call of the same size to allocate."""
    torch = pytest.importorskip("torch")
    w = small_workload(workload, duration=4.0, sampling_frequency=2048.0)
    w = small_workload(workload, **{**w.__dict__, "injection": dict(w.injection, geocent_time=w.start_time + 2.0)})
    an = device_analysis(OD.build_workload(w), w.model, w)
    if time:
        an.set_time_marginalization(True, True, w.start_time + 1.92, w.start_time + 2.08)
    p = draw_points(w, 40, np.random.default_rng(2))
    block = torch.from_numpy(params_block(p)).cuda()
    out = torch.zeros(40, dtype=torch.float64, device="cuda")
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        an.log_likelihood_ratio_device(block.data_ptr(), 40, out.data_ptr(), "mixed", stream.cuda_stream)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        an.log_likelihood_ratio_device(block.data_ptr(), 40, out.data_ptr(), "fp64", stream.cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), an.log_likelihood_ratio_host(params_block(p), "fp64"))
    an.close()
