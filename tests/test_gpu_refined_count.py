"""The number of points that the last mixed evaluation recomputed
(``Analysis.last_refined``) stays what it was through float64 evaluations."""
import numpy as np
import pytest

from bilby_gb300 import random as grandom
from bilby_gb300.detector import InterferometerList
from bilby_gb300.multiband import MBGravitationalWaveTransient
from bilby_gb300.source import taylorf2_aligned_frequency_sequence
from bilby_gb300.waveform_generator import WaveformGenerator
from oracle import data as OD
from tests.gpu_helpers import device_analysis, draw_points, params_block, small_workload

pytestmark = pytest.mark.gpu


# a small mixed batch (counted beside no ordering), an ordered one, bursts, multi-banding;
# the float64 batch is one that is ordered (32768 points x chunks)
@pytest.mark.parametrize("kind,mixed", [("full", 40), ("full", 12000), ("burst", 300), ("multiband", 300)])
def test_float64_calls_leave_the_count(gpu, kind, mixed):
    w = small_workload("sg_4s" if kind == "burst" else "tf2_128s", duration=4.0, sampling_frequency=2048.0,
                       mass_range=(10.0, 40.0))
    inj = dict(w.injection, geocent_time=w.start_time + 2.5)
    if kind != "burst":
        inj.update(mass_1=30.0, mass_2=25.0)
    w = small_workload("tf2_128s", **{**w.__dict__, "injection": inj})
    if kind == "multiband":
        grandom.seed(w.seed)
        ifos = InterferometerList(list(w.detectors))
        ifos.set_strain_data_from_power_spectral_densities(w.sampling_frequency, w.duration, w.start_time)
        wfg = WaveformGenerator(duration=w.duration, sampling_frequency=w.sampling_frequency, start_time=w.start_time,
                                frequency_domain_source_model=taylorf2_aligned_frequency_sequence,
                                waveform_arguments=dict(minimum_frequency=20.0))
        keep = MBGravitationalWaveTransient(ifos, wfg, reference_chirp_mass=8.0)
        an = keep.analysis
    else:
        an = device_analysis(OD.build_workload(w), w.model, w)
    block = params_block(draw_points(w, 40000, np.random.default_rng(3)))
    part = np.ascontiguousarray(block[:, :mixed])
    an.log_likelihood_ratio_host(block, "fp64")  # the work space of the largest call
    an.refinement_tolerance = 1e-9
    an.log_likelihood_ratio_host(part, "mixed")
    count = an.last_refined()
    assert 0 < count <= mixed
    an.log_likelihood_ratio_host(block, "fp64")
    assert an.last_refined() == count
    an.inner_products_host(block, "fp64")
    assert an.last_refined() == count
