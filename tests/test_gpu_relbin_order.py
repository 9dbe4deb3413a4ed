"""Mixed relative binning with time marginalisation (csrc/gwl_marg_window.cu) at
the column lengths and counts where the order of its tables changes: fewer than
eight blocks per column, exactly eight, more, whole columns of 2048, and numbers of
columns that do not fill a group of four.

Tolerance: the mixed precision's |dlnL| <= 1e-3 against float64 (the loudest points
recomputed by the error bound, as in use); a bin read at the wrong place moves the lnL by a sizeable part of <d|h>, asserted above 3."""
import numpy as np
import pytest

from bilby_gb300.prior import Uniform
from bilby_gb300.workloads import draw_points
from tests.test_gpu_wide_lists import _data

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("detectors,duration,fs,masses", [
    (1, 2.0, 64.0, (20.0, 35.0)), (2, 2.0, 128.0, (15.0, 30.0)), (3, 3.0, 256.0, (15.0, 30.0)),
    (2, 3.0, 1024.0, (10.0, 30.0)), (2, 4.0, 2048.0, (10.0, 30.0)), (1, 10.0, 2048.0, (6.0, 12.0))])
def test_mixed_against_float64(gpu, detectors, duration, fs, masses):
    from bilby_gb300.relative import RelativeBinningGravitationalWaveTransient
    from bilby_gb300.source import taylorf2_aligned_relative_binning
    w, ifos, wfg, _ = _data(detectors, duration, fs, masses, taylorf2_aligned_relative_binning)
    tc = w.injection["geocent_time"]
    half = min(0.1, duration / 8)
    priors = {"geocent_time": Uniform(tc - half, tc + half)}
    like = RelativeBinningGravitationalWaveTransient(
        ifos, wfg, fiducial_parameters=dict(w.injection), epsilon=0.5, time_marginalization=True, precision="mixed",
        priors=priors)
    p = draw_points(w, 9, np.random.default_rng(4))
    for k, v in w.injection.items():
        if k in p:
            p[k][:4] = v
    p["luminosity_distance"][:] = np.linspace(100.0, 400.0, 9)
    p["geocent_time"] = np.full(9, float(priors["geocent_time"]))
    p["time_jitter"] = np.linspace(-1.0, 1.0, 9) / fs
    got = like.log_likelihood_ratio_batch(p)
    assert like.analysis.last_refined() < 9  # not all of them recomputed in float64
    ref = like.log_likelihood_ratio_batch(p, precision="fp64")
    assert np.max(np.abs(ref)) > 3
    assert np.all(np.abs(got - ref) <= 1e-3), np.abs(got - ref).max()
