"""The float64 sine-Gaussian likelihood on the 32-bit pipes (csrc/gwl_wide_sg.cu):
every launch shape against the oracle, and bit for bit against each other.

Tolerance: the oracle's float64 terms carry the time shift's 2 pi f dt 2^-53
(1e4 rad: 1e-12) and a few roundings of the Gaussian's exponent (below 40 where
a term counts: 2e-14), so 1e-10 of the scale max(1, |<d|h>|, <h|h> / 2) leaves
two orders of magnitude."""
import numpy as np
import pytest

from oracle import data as OD
from oracle import restate as R
from tests.gpu_helpers import device_analysis, draw_points, params_block, point, small_workload

pytestmark = pytest.mark.gpu


# quality factors below one (both Gaussians cover the band and nearly cancel in
# h_x) to 200 (a Gaussian of a few bins); centres below, inside and above the
# band, on a bin and between bins; an odd grid and a long one
@pytest.mark.parametrize("detectors,duration,fs", [(1, 4.0, 2048.0), (2, 3.0, 1000.0), (3, 16.0, 512.0), (4, 2.0, 2048.0)])
def test_against_the_oracle_in_every_launch_shape(gpu, detectors, duration, fs):
    w = small_workload("sg_4s", detectors=("H1", "L1", "V1")[:min(detectors, 3)], duration=duration,
                       sampling_frequency=fs)
    w = small_workload("sg_4s", **{**w.__dict__, "injection": dict(w.injection, geocent_time=w.start_time + duration / 2)})
    dets = OD.build_workload(w)
    dets = (dets + dets)[:detectors]
    an = device_analysis(dets, "sinegaussian", w)
    n = 70
    rng = np.random.default_rng(6)
    p = draw_points(w, n, rng)
    p["Q"] = 10 ** rng.uniform(-0.5, 2.3, n)
    p["frequency"] = rng.uniform(10, 0.7 * fs, n)
    p["frequency"][:20] = np.round(p["frequency"][:20])
    block = params_block(p)
    full = an.log_likelihood_ratio_host(block, "fp64")
    # one CTA per point, then a lane per point, then ordered (the switches of
    # test_gpu_wide.py)
    chunks = -(-(int((fs / 2 - 20) * duration) + 17) // 256)
    edge = max(12, 3200 // chunks)
    for size in (1, 12, 13, 32, 33, edge, edge + 1, edge + 40, 32768 // chunks + 70):
        many = np.ascontiguousarray(np.tile(block, -(-size // n))[:, :size])
        got = an.log_likelihood_ratio_host(many, "fp64")
        assert np.array_equal(got, np.tile(full, -(-size // n))[:size]), size
    src = OD.source_for(w.model, w.minimum_frequency)
    terms = [R.plain_terms(dets, src, point(p, i)) for i in range(n)]
    scale = np.array([R.parity_scale(dh, hh) for dh, hh in terms])
    lnl = np.array([np.real(dh) - hh / 2 for dh, hh in terms])
    assert np.all(np.abs(full - lnl) <= 1e-10 * scale)
    dh, hh = an.inner_products_host(block, "fp64")
    assert np.all(np.abs(dh - np.array([t[0] for t in terms])) <= 1e-10 * scale)
    assert np.all(np.abs(hh - np.array([t[1] for t in terms])) <= 1e-10 * scale)
    few, hfew = an.inner_products_host(block[:, :3], "fp64")
    assert np.array_equal(few, dh[:3]) and np.array_equal(hfew, hh[:3])
    an.close()
