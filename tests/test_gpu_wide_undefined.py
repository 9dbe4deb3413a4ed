"""Points and data that are not defined, in the float64 kernels on the 32-bit pipes
(csrc/gwl_wide*.cu): what they leave untouched and what they make undefined."""
import numpy as np
import pytest

from bilby_gb300 import random as grandom
from bilby_gb300.analysis import Analysis, DetectorData
from bilby_gb300.detector import InterferometerList
from bilby_gb300.multiband import MBGravitationalWaveTransient
from bilby_gb300.relative import RelativeBinningGravitationalWaveTransient
from bilby_gb300.source import taylorf2_aligned_frequency_sequence, taylorf2_aligned_relative_binning
from bilby_gb300.waveform_generator import WaveformGenerator
from oracle import data as OD
from tests.gpu_helpers import device_analysis, draw_points, params_block, small_workload

pytestmark = pytest.mark.gpu

TF2_UNDEFINED = [dict(mass_1=-1.0), dict(mass_2=np.nan), dict(luminosity_distance=0.0), dict(phase=np.nan),
                 dict(ra=np.inf), dict(geocent_time=np.nan), dict(chi_1=np.inf)]
SG_UNDEFINED = [dict(Q=0.0), dict(Q=-5.0), dict(frequency=-100.0), dict(frequency=0.0), dict(hrss=np.nan), dict(ra=np.nan)]


def _workload(name):
    w = small_workload(name, duration=4.0, sampling_frequency=2048.0, mass_range=(10.0, 40.0))
    inj = dict(w.injection, geocent_time=w.start_time + 2.5)
    if w.model == "taylorf2":
        inj.update(mass_1=30.0, mass_2=25.0)
    return small_workload(name, **{**w.__dict__, "injection": inj})


def _list_analysis(kind, w):
    """The analysis of a multi-banded or relative-binning likelihood."""
    grandom.seed(w.seed)
    ifos = InterferometerList(list(w.detectors))
    ifos.set_strain_data_from_power_spectral_densities(w.sampling_frequency, w.duration, w.start_time)
    model = taylorf2_aligned_frequency_sequence if kind == "multiband" else taylorf2_aligned_relative_binning
    wfg = WaveformGenerator(duration=w.duration, sampling_frequency=w.sampling_frequency, start_time=w.start_time,
                            frequency_domain_source_model=model, waveform_arguments=dict(minimum_frequency=20.0))
    if kind == "multiband":
        return MBGravitationalWaveTransient(ifos, wfg, reference_chirp_mass=8.0)
    return RelativeBinningGravitationalWaveTransient(ifos, wfg, fiducial_parameters=dict(w.injection))


@pytest.mark.parametrize("many", [1, 700])  # one CTA per point, and a lane per point
@pytest.mark.parametrize("kind", ["burst", "full", "multiband", "relbin"])
def test_inner_products_of_an_undefined_point_are_zero(gpu, kind, many):
    """Nothing is summed for it: <d|h> is 0 and, where <h|h> is a sum too, so is that."""
    w = _workload("sg_4s" if kind == "burst" else "tf2_128s")
    keep = _list_analysis(kind, w) if kind in ("multiband", "relbin") else None
    an = keep.analysis if keep is not None else device_analysis(OD.build_workload(w), w.model, w)
    bad = SG_UNDEFINED if kind == "burst" else TF2_UNDEFINED
    n = (len(bad) + 1) * many
    p = draw_points(w, n, np.random.default_rng(4))
    for q, changes in enumerate(bad):
        for k, v in changes.items():
            p[k][q::len(bad) + 1] = v
    dh, hh = an.inner_products_host(params_block(p), "fp64")
    good = np.arange(n) % (len(bad) + 1) == len(bad)
    assert np.all(dh[~good] == 0.0), dh[:len(bad)]
    if kind != "full":
        assert np.all(hh[~good] == 0.0), hh[:len(bad)]
    assert np.all(np.isfinite(dh[good])) and np.all(hh[good] > 0.0)
    lnl = an.log_likelihood_ratio_host(params_block(p), "fp64")
    assert np.all(lnl[~good] == -1.7976931348623157e308) and np.all(np.isfinite(lnl[good]))


def _with_infinite_bin(dets, w, model, k):
    dd = []
    for q, d in enumerate(dets):
        strain = np.array(d.masked_strain)
        if q == 0 and k is not None:
            strain[k] = np.inf
        dd.append(DetectorData(d.name, d.vertex, d.tensor, d.start_time, strain, d.psd, d.mask))
    return Analysis(model, dets[0].frequency, dd, w.duration, w.sampling_frequency, w.minimum_frequency)


@pytest.mark.parametrize("n", [4, 60])  # one CTA per point, and a lane per point
@pytest.mark.parametrize("time", [False, True])
def test_an_infinite_bin_beyond_the_band_changes_nothing(gpu, n, time):
    """The templates that end below it keep their bits; the others are undefined."""
    w = _workload("tf2_128s")
    dets = OD.build_workload(w)
    cut = 4400.0 / 40.0  # f_ISCO of 40 solar masses, 110 Hz
    an = [_with_infinite_bin(dets, w, "taylorf2", k) for k in (None, int((cut + 8.0) * w.duration))]
    p = draw_points(w, n, np.random.default_rng(4))
    p["mass_1"], p["mass_2"] = np.where(np.arange(n) % 2, 25.0, 12.0), np.where(np.arange(n) % 2, 20.0, 11.0)
    if time:
        for a in an:
            a.set_time_marginalization(True, True, w.start_time + 2.45, w.start_time + 2.55)
        p["geocent_time"] = np.full(n, w.start_time)
    clean, dirty = (a.log_likelihood_ratio_host(params_block(p), "fp64") for a in an)
    heavy = np.arange(n) % 2 == 1
    assert np.array_equal(dirty[heavy], clean[heavy])
    assert np.all(np.isfinite(clean)) and not np.any(np.isfinite(dirty[~heavy]))


@pytest.mark.parametrize("kind", ["multiband", "relbin"])
def test_an_infinite_coefficient_beyond_the_band_changes_nothing(gpu, kind):
    w = _workload("tf2_128s")
    like = _list_analysis(kind, w)
    n = 60
    p = draw_points(w, n, np.random.default_rng(4))
    # f_ISCO 63 and 191 Hz
    p["mass_1"], p["mass_2"] = np.where(np.arange(n) % 2, 36.0, 12.0), np.where(np.arange(n) % 2, 34.0, 11.0)
    clean = like.log_likelihood_ratio_batch(p)
    name = like.interferometers[0].name
    if kind == "multiband":
        like.linear_coeffs[name][np.searchsorted(like.banded_frequency_points, 70.0)] = np.inf
    else:
        like.summary_data[name][0][np.searchsorted(like.bin_freqs, 70.0)] = np.inf
    like._upload()
    dirty = like.log_likelihood_ratio_batch(p)
    heavy = np.arange(n) % 2 == 1
    assert np.array_equal(dirty[heavy], clean[heavy])
    assert np.all(np.isfinite(clean)) and not np.any(np.isfinite(dirty[~heavy]))


@pytest.mark.parametrize("n", [2, 300])  # one CTA per point, and a lane per point
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_an_undefined_bin_of_the_data_is_noticed_by_every_burst(gpu, n, value):
    """Also by those whose Gaussian at that bin is below the sums' last digit; outside
    the mask it is not data."""
    w = _workload("sg_4s")
    dets = OD.build_workload(w)
    dd, k = [], int(900 * w.duration)
    p = draw_points(w, n, np.random.default_rng(4))
    p["frequency"], p["Q"] = np.linspace(50.0, 300.0, n), np.full(n, 20.0)
    lnl = []
    for inside in (True, False):
        for q, d in enumerate(dets):
            strain, mask = np.array(d.masked_strain), np.array(d.mask)
            strain[k] = value
            mask[k] = inside
            dd.append(DetectorData(d.name, d.vertex, d.tensor, d.start_time, strain, d.psd, mask))
        an = Analysis("sinegaussian", dets[0].frequency, dd[-len(dets):], w.duration, w.sampling_frequency, 20.0)
        lnl.append(an.log_likelihood_ratio_host(params_block(p), "fp64"))
    assert not np.any(np.isfinite(lnl[0])) and np.all(np.isfinite(lnl[1]))
