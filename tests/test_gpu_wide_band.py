"""The float64 TaylorF2 likelihood (csrc/gwl_wide.cu, gwl_wide_tm.cu) with a waveform
that starts below the detectors' data: the bins without data change nothing."""
import numpy as np
import pytest

from bilby_gb300.analysis import Analysis, DetectorData
from oracle import data as OD
from tests.gpu_helpers import draw_points, params_block, small_workload

pytestmark = pytest.mark.gpu


def _workload(duration):
    masses = (10.0, 40.0) if duration < 60 else (1.0, 2.0)
    w = small_workload("tf2_128s", duration=duration, sampling_frequency=1024.0, mass_range=masses)
    return small_workload("tf2_128s", **{**w.__dict__, "injection": dict(
        w.injection, mass_1=masses[1], mass_2=masses[0], geocent_time=w.start_time + 0.8 * duration)})


def _analysis(dets, w, fmin, open_mask=False):
    dd = []
    for d in dets:
        psd, mask = np.array(d.psd), np.array(d.mask)
        if open_mask:  # the data's band is in the PSD alone
            psd, mask = np.where(mask, psd, np.inf), np.ones_like(mask)
        dd.append(DetectorData(d.name, d.vertex, d.tensor, d.start_time, d.masked_strain, psd, mask))
    return Analysis("taylorf2", dets[0].frequency, dd, w.duration, w.sampling_frequency, fmin)


# one CTA per point and a lane per point; 8 s and 128 s (10^5 rad at 20 Hz, 10^10 at 1 / 128 Hz)
@pytest.mark.parametrize("duration,fmin", [(8.0, 0.0), (8.0, 0.3), (128.0, 0.0), (128.0, 0.3), (128.0, 5.0)])
@pytest.mark.parametrize("time", [False, True])
def test_same_bits_as_from_the_first_bin_with_data(gpu, duration, fmin, time):
    w = _workload(duration)
    dets = OD.build_workload(w)
    low, at = _analysis(dets, w, fmin), _analysis(dets, w, 20.0)
    p = draw_points(w, 40, np.random.default_rng(7))
    if time:
        for an in (low, at):
            an.set_time_marginalization(True, True, w.injection["geocent_time"] - 0.05, w.injection["geocent_time"] + 0.05)
        p["geocent_time"] = np.full(40, w.start_time)
    block = params_block(p)
    for n in (3, 40):
        part = np.ascontiguousarray(block[:, :n])
        assert np.array_equal(low.log_likelihood_ratio_host(part, "fp64"), at.log_likelihood_ratio_host(part, "fp64"))


def test_bins_of_infinite_psd(gpu):
    """The same with masks that are open down to zero frequency.  The chunks begin at
    another bin, so the sums round differently: 8 * 2^-53 psi of the scale max(1,
    |<d|h>|, <h|h> / 2) (tests/test_gpu_wide.py), once for each side."""
    w = _workload(128.0)
    dets = OD.build_workload(w)
    p = draw_points(w, 40, np.random.default_rng(7))
    block = params_block(p)
    low, hh = _analysis(dets, w, 0.0, True).inner_products_host(block, "fp64")
    at, _ = _analysis(dets, w, 20.0).inner_products_host(block, "fp64")
    mc = (p["mass_1"] * p["mass_2"]) ** 0.6 / (p["mass_1"] + p["mass_2"]) ** 0.2 * 4.925490947641267e-06
    psi = 3 / 128 * (np.pi * mc * 20.0) ** (-5 / 3)
    scale = np.maximum(np.maximum(1.0, np.abs(at)), hh / 2)
    assert np.all(np.abs(low - at) <= 16 * 2.0 ** -53 * psi * scale)
