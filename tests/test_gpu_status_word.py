"""An analysis's status word, which lies in pinned host memory: what a kernel records in
it after a bounded wait that ran out reaches the next host evaluation, once."""
import ctypes

import numpy as np
import pytest

from oracle import data as OD
from tests.gpu_helpers import device_analysis, draw_points, params_block, small_workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points", [1, 600])
def test_a_kernels_timeout_reaches_the_next_host_evaluation(gpu, points):
    from bilby_gb300 import _capi
    w = small_workload("sg_4s")
    an, other = (device_analysis(OD.build_workload(w), w.model, w) for _ in range(2))
    block = params_block(draw_points(w, points, np.random.default_rng(3)))
    good = an.log_likelihood_ratio_host(block, "fp64")
    arrived = ctypes.c_int(-1)
    _capi.check(_capi.load().gwl_selftest_analysis_wait(an._h, 2000, ctypes.byref(arrived)), "wait")
    assert arrived.value == 0
    assert np.array_equal(other.log_likelihood_ratio_host(block, "fp64"), good)  # a word per analysis
    with pytest.raises(TimeoutError):
        an.log_likelihood_ratio_host(block, "fp64")
    assert np.array_equal(an.log_likelihood_ratio_host(block, "fp64"), good)
    an.close()
    other.close()
