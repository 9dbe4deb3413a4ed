"""The float64 TaylorF2 likelihood on the 32-bit pipes (csrc/gwl_wide.cu): every
launch shape against the oracle, and bit for bit against each other.

Tolerance: the oracle's float64 phase psi carries a few roundings of psi
2^-53 (and the time shift's 2 pi f dt 2^-53), coherent over the bins, so its
lnL errs by up to about 8 * 2^-53 * max(psi, 2 pi f dt) of the scale
max(1, |<d|h>|, <h|h> / 2); the 1e-9 of the other parity tests covers it up to
1e6 rad, and heavier phases get the bound itself."""
import numpy as np
import pytest

from oracle import data as OD
from oracle import restate as R
from tests.gpu_helpers import device_analysis, draw_points, params_block, point, small_workload

pytestmark = pytest.mark.gpu


def _case(detectors, duration, fs, masses):
    w = small_workload("tf2_marg_8s", detectors=("H1", "L1", "V1")[:min(detectors, 3)], duration=duration,
                       sampling_frequency=fs, mass_range=masses, time_marginalization=False,
                       phase_marginalization=False, distance_marginalization=False)
    w = small_workload("tf2_marg_8s", **{**w.__dict__, "injection": dict(
        w.injection, mass_1=masses[1], mass_2=masses[0], geocent_time=w.start_time + 0.7 * duration)})
    dets = OD.build_workload(w)
    dets = (dets + dets)[:detectors]
    return w, dets, device_analysis(dets, "taylorf2", w)


# bins at the tiles' edges: 4 s at 2048 Hz (17 chunks of 256 from bin 80), 3 s at
# 1000 Hz (1501 bins, an odd grid), 16 s; masses whose band ends inside and
# beyond the grid, and a thousandth of a solar mass (10^9 cycles)
@pytest.mark.parametrize("detectors,duration,fs,masses", [
    (1, 4.0, 2048.0, (10.0, 40.0)), (2, 3.0, 1000.0, (2.0, 60.0)), (3, 16.0, 2048.0, (1.0, 2.0)),
    (4, 4.0, 2048.0, (0.5, 90.0)), (2, 4.0, 2048.0, (1e-3, 2e-3))])
def test_against_the_oracle_in_every_launch_shape(gpu, detectors, duration, fs, masses):
    w, dets, an = _case(detectors, duration, fs, masses)
    n = 70
    p = draw_points(w, n, np.random.default_rng(5))
    block = params_block(p)
    full = an.log_likelihood_ratio_host(block, "fp64")
    # one CTA per point, then a lane per point, then ordered: the switches lie at 12
    # points or 3200 points x chunks, and at 32768 points x chunks
    chunks = -(-(int((fs / 2 - 20) * duration) + 17) // 256)
    edge = max(12, 3200 // chunks)
    for size in (1, 12, 13, 32, 33, edge, edge + 1, edge + 40, 32768 // chunks + 70):
        many = np.ascontiguousarray(np.tile(block, -(-size // n))[:, :size])
        got = an.log_likelihood_ratio_host(many, "fp64")
        assert np.array_equal(got, np.tile(full, -(-size // n))[:size]), size
    src = OD.source_for(w.model, w.minimum_frequency)
    terms = [R.plain_terms(dets, src, point(p, i)) for i in range(n)]
    lnl = np.array([np.real(dh) - hh / 2 for dh, hh in terms])
    scale = np.array([R.parity_scale(dh, hh) for dh, hh in terms])
    mc = (p["mass_1"] * p["mass_2"]) ** 0.6 / (p["mass_1"] + p["mass_2"]) ** 0.2 * 4.925490947641267e-06
    psi = 3 / 128 * (np.pi * mc * 20.0) ** (-5 / 3)
    assert np.all(np.abs(full - lnl) <= np.maximum(1e-9, 8 * 2.0 ** -53 * psi) * scale)
    # the complex inner products (the sine as well as the cosine)
    dh, hh = an.inner_products_host(block, "fp64")
    err = np.abs(dh - np.array([t[0] for t in terms]))
    assert np.all(err <= np.maximum(1e-9, 8 * 2.0 ** -53 * psi) * scale)
    assert np.all(np.abs(hh - np.array([t[1] for t in terms])) <= 1e-9 * scale)
    few, _ = an.inner_products_host(block[:, :3], "fp64")
    assert np.array_equal(few, dh[:3])
    an.close()
