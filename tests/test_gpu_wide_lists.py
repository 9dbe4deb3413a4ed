"""Float64 relative binning and multi-banding on the 32-bit pipes
(csrc/gwl_wide_relbin.cu; csrc/gwl_wide.cu over a list of rows) against the
oracle's evaluation of the same bins and bands, and bit for bit between batch
sizes.

Tolerance: as in tests/test_gpu_wide.py, 8 * 2^-53 * max(psi, 2 pi f dt) of the
scale max(1, |<d|h>|, <h|h> / 2), below 1e-9 for these phases."""
import numpy as np
import pytest

from bilby_gb300 import random as grandom
from bilby_gb300.detector import InterferometerList
from bilby_gb300.waveform_generator import WaveformGenerator
from bilby_gb300.workloads import draw_points, point
from oracle import data as OD
from oracle import multiband as OM
from oracle import relbin as OR
from oracle import restate as R
from tests.gpu_helpers import small_workload

pytestmark = pytest.mark.gpu


def _data(detectors, duration, fs, masses, model):
    w = small_workload("tf2_128s", detectors=("H1", "L1", "V1")[:detectors], duration=duration, sampling_frequency=fs,
                       mass_range=masses)
    w = small_workload("tf2_128s", **{**w.__dict__, "injection": dict(
        w.injection, mass_1=masses[1], mass_2=masses[0], geocent_time=w.start_time + duration - 1.5)})
    grandom.seed(w.seed)
    ifos = InterferometerList(list(w.detectors))
    ifos.set_strain_data_from_power_spectral_densities(fs, duration, w.start_time)
    wfg = WaveformGenerator(duration=duration, sampling_frequency=fs, start_time=w.start_time,
                            frequency_domain_source_model=model, waveform_arguments=dict(minimum_frequency=20.0))
    ifos.inject_signal(waveform_generator=wfg, parameters=dict(w.injection))
    return w, ifos, wfg, OD.build_workload(w)


def _check(like, terms, pts, n):
    params = {k: np.array([q[k] for q in pts]) for k in pts[0]}
    full = like.log_likelihood_ratio_batch(params)
    for size in (1, 12, 13, 32, 65, 300, 3500, 12000):
        part = like.log_likelihood_ratio_batch({k: np.resize(v, size) for k, v in params.items()})
        assert np.array_equal(part, np.resize(full, size)), size
    t = [terms(q) for q in pts]
    lnl = np.array([np.real(dh) - hh / 2 for dh, hh in t])
    scale = np.array([R.parity_scale(dh, hh) for dh, hh in t])
    assert np.all(np.abs(full - lnl) <= 1e-9 * scale), np.max(np.abs(full - lnl) / scale)
    from bilby_gb300.analysis import params_block
    dh, hh = like.analysis.inner_products_host(params_block(like._prepare(params)), "fp64")
    assert np.all(np.abs(dh - np.array([x[0] for x in t])) <= 1e-9 * scale)
    assert np.all(np.abs(hh - np.array([x[1] for x in t])) <= 1e-9 * scale)


# bins at the edges of the warp's passes of 31, templates whose band ends inside
# the bins, an odd grid
@pytest.mark.parametrize("detectors,duration,fs,masses,epsilon", [
    (1, 16.0, 2048.0, (5.0, 8.0), 2.0), (2, 16.0, 2048.0, (5.0, 12.0), 1.0), (3, 6.0, 2048.0, (10.0, 30.0), 0.5),
    (2, 8.0, 1000.0, (8.0, 20.0), 0.13)])
def test_relative_binning(gpu, detectors, duration, fs, masses, epsilon):
    from bilby_gb300.relative import RelativeBinningGravitationalWaveTransient
    from bilby_gb300.source import taylorf2_aligned_relative_binning
    w, ifos, wfg, dets = _data(detectors, duration, fs, masses, taylorf2_aligned_relative_binning)
    fiducial = dict(w.injection, mass_1=0.5 * sum(masses), mass_2=masses[0])
    like = RelativeBinningGravitationalWaveTransient(ifos, wfg, fiducial_parameters=fiducial, epsilon=epsilon)
    for d, ifo in zip(dets, ifos):  # the same injected data
        d.strain = np.asarray(ifo.strain_data.frequency_domain_strain)
    setup = OR.RelbinSetup(like.bin_inds, like.bin_freqs,
                           [np.asarray(like.per_detector_fiducial_waveforms[i.name]) for i in ifos],
                           [like.summary_data[i.name] for i in ifos], 0.0)
    n = 67
    p = draw_points(w, n, np.random.default_rng(9))
    _check(like, lambda q: OR.terms(dets, OD.source_for("taylorf2", 20.0), setup, q), [point(p, i) for i in range(n)], n)


@pytest.mark.parametrize("detectors,duration,fs,masses", [(1, 32.0, 2048.0, (2.5, 5.0)), (2, 24.0, 2048.0, (3.0, 6.0)),
                                                          (3, 32.0, 1024.0, (2.5, 20.0))])
def test_multi_banding(gpu, detectors, duration, fs, masses):
    from bilby_gb300.multiband import MBGravitationalWaveTransient
    from bilby_gb300.source import taylorf2_aligned_frequency_sequence
    w, ifos, wfg, dets = _data(detectors, duration, fs, masses, taylorf2_aligned_frequency_sequence)
    like = MBGravitationalWaveTransient(ifos, wfg, reference_chirp_mass=masses[0] * 2 ** -0.2 * 0.999, time_offset=1.7,
                                        delta_f_end=53.0)
    weights = dict(waveform_frequencies=wfg.waveform_arguments["frequencies"],
                   unique_to_original_frequencies=like.unique_to_original_frequencies,
                   banded_frequency_points=like.banded_frequency_points)
    for q, ifo in enumerate(ifos):
        weights[f"linear_coeffs_{q}"] = like.linear_coeffs[ifo.name]
        weights[f"quadratic_coeffs_{q}"] = like.quadratic_coeffs[ifo.name]
    n = 67
    p = draw_points(w, n, np.random.default_rng(10))
    _check(like, lambda q: OM.terms(dets, OD.source_for("taylorf2", 20.0), weights, q), [point(p, i) for i in range(n)], n)
