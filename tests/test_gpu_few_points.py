"""Small mixed-precision TaylorF2 batches (csrc/gwl_kernels.cu, k_mixed_tf2_few) give
the bits of large ones: the band's edges inside a unit of 16 bins, chunks
evaluated directly (the first bins of a short segment), every split-K depth,
marked points, the real and the complex sums."""
import numpy as np
import pytest

from oracle import data as OD
from tests.gpu_helpers import device_analysis, draw_points, params_block, small_workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("detectors,duration,fs,masses,minimum", [
    (1, 4.0, 2048.0, (10.0, 40.0), 20.0), (2, 3.0, 1000.0, (2.0, 60.0), 21.3), (3, 16.0, 2048.0, (1.0, 2.0), 20.0),
    (4, 4.0, 2048.0, (0.5, 90.0), 33.0)])
def test_few_points_give_the_bits_of_many(gpu, detectors, duration, fs, masses, minimum):
    w = small_workload("tf2_128s", detectors=("H1", "L1", "V1")[:min(detectors, 3)], duration=duration,
                       sampling_frequency=fs, mass_range=masses, minimum_frequency=minimum)
    w = small_workload("tf2_128s", **{**w.__dict__, "injection": dict(
        w.injection, mass_1=masses[1], mass_2=masses[0], luminosity_distance=40.0,
        geocent_time=w.start_time + 0.7 * duration)})
    dets = OD.build_workload(w)
    an = device_analysis((dets + dets)[:detectors], "taylorf2", w)
    p = draw_points(w, 200, np.random.default_rng(4))
    p["luminosity_distance"][:40] = np.geomspace(1.0, 40.0, 40)  # over the error bound: the accurate kernel
    p["mass_1"][-1] = -1.0  # no waveform
    block = params_block(p)
    chunks = -(-(int((fs / 2 - 20) * duration) + 17) // 512)
    many = -(-(144 * 1024 // (chunks * detectors) + 1) // 200)  # repeats that leave the few-points kernel
    big = np.ascontiguousarray(np.tile(block, many))
    for depth in (1, 2, 4, 16):
        an.chunks_per_group = depth
        full = an.log_likelihood_ratio_host(big, "mixed")
        assert an.last_refined() % many == 0 and an.last_refined() > 0
        marked = an.last_refined() // many
        for size in (1, 7, 200):
            part = an.log_likelihood_ratio_host(block[:, :size], "mixed")
            assert np.array_equal(part, full[:size]), (depth, size)
        assert an.last_refined() == marked
        dh, hh = an.inner_products_host(big, "mixed")
        few, hfew = an.inner_products_host(block, "mixed")
        assert np.array_equal(few, dh[:200], equal_nan=True) and np.array_equal(hfew, hh[:200], equal_nan=True)
    an.close()
