"""The parameters the kernels read, by the short conversion and packing: the same
numbers as the full conversion and numpy's broadcasting give."""
import numpy as np
import pytest
import torch

from bilby_gb300 import _capi
from bilby_gb300.analysis import params_block
from bilby_gb300.conversion import convert_to_kernel_parameters, convert_to_lal_binary_black_hole_parameters

BASE = dict(chi_1=0.1, chi_2=-0.2, luminosity_distance=300.0, psi=0.3, ra=1.0, dec=-0.4, geocent_time=1126259642.4)
MASSES = [dict(mass_1=3.0, mass_2=2.0), dict(chirp_mass=1.2, mass_ratio=0.8), dict(total_mass=5.0, mass_ratio=0.5),
          dict(total_mass=5.0, chirp_mass=2.0), dict(mass_1=3.0, mass_ratio=0.4),
          dict(chirp_mass=2.0, symmetric_mass_ratio=0.24)]
ANGLES = [dict(theta_jn=0.4, phase=1.0), dict(cos_theta_jn=-0.3, phase=1.0), dict(cos_theta_jn=0.6, delta_phase=2.0),
          dict(theta_jn=0.4, phase=1.0, a_1=0.3, cos_tilt_1=1.0, cos_tilt_2=-1.0)]
FORMS = [float, np.float64, lambda v: np.array([v, 1.01 * v]), lambda v: torch.tensor([v, 1.01 * v], dtype=torch.float64)]


@pytest.mark.parametrize("form", range(len(FORMS)))
@pytest.mark.parametrize("angles", ANGLES)
@pytest.mark.parametrize("masses", MASSES)
def test_short_conversion_and_packing(masses, angles, form):
    given = {k: FORMS[form](v) for k, v in {**BASE, **masses, **angles}.items()}
    before = dict(given)
    short = convert_to_kernel_parameters(given)
    assert given == before or form > 1
    full, _ = convert_to_lal_binary_black_hole_parameters(given)
    assert given.keys() == before.keys()
    for k in _capi.SLOT:
        assert (k in short) == (k in full)
        if k in full:
            assert np.array_equal(np.asarray(short[k]), np.asarray(full[k])), k
    if form < 3:
        n = 1 if form < 2 else 2
        want = np.zeros((_capi.NPARAM, n))
        for k, slot in _capi.SLOT.items():
            if k in full:
                want[slot] = np.broadcast_to(np.asarray(full[k], dtype=np.float64), (n,))
        assert np.array_equal(params_block(short), want)
