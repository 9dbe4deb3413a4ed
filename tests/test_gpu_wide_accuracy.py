"""The float64 likelihoods on the 32-bit pipes (csrc/gwl_wide.cu, gwl_wide_sg.cu) against
extended precision: the part of <d|h> and <h|h> that their float pairs and fixed
points could lose, which the parity tests' 1e-9 against a float64 oracle would hide.

Tolerance: the sum over bins and detectors of |term| times
  2 pi f (2^-52 |dt| + 2^-49 R / c)   the delay's and the hour angle's roundings,
  4 * 2^-53 psi                       those of the post-Newtonian coefficients,
  2^-42                               the cosine, 3e-14 rms from its table,
and for <h|h> 2^-47 of it (some sixty roundings of 2^-53: antenna patterns, amplitude, squares)."""
import numpy as np
import pytest

from oracle import data as OD
from oracle import restate as R
from tests.gpu_helpers import device_analysis, draw_points, params_block, small_workload

pytestmark = pytest.mark.gpu

LD = np.longdouble
PI = LD("3.14159265358979323846264338327950288419716939937510")
MTSUN, PC, C = LD(4.925490947641267e-06), LD(3.085677581491367e16), LD(299792458)


def _burst(p, f):
    q, f0 = p["Q"], p["frequency"]
    tau, temp = q / (np.sqrt(LD(2)) * PI * f0), q / (4 * np.sqrt(PI) * f0)
    down, up = (np.exp(-((f - s * f0) * PI * tau) ** 2) for s in (1, -1))
    amp = p["hrss"] * np.sqrt(PI) * tau / 2
    zero = 0 * down
    plus = amp * (down + up) / np.sqrt(temp * (1 + np.exp(-q * q)))
    return (plus, zero), (zero, -amp * (down - up) / np.sqrt(temp * (1 - np.exp(-q * q)))), zero


def _taylorf2(p, f):
    m1, m2 = p["mass_1"], p["mass_2"]
    m, eta = m1 + m2, m1 * m2 / (m1 + m2) ** 2
    delta, s, a = (m1 - m2) / m, (p["chi_1"] + p["chi_2"]) / 2, (p["chi_1"] - p["chi_2"]) / 2
    r = lambda n, d=1: LD(n) / LD(d)
    euler = LD("0.577215664901532860606512090082402431")
    c5 = (PI * (r(38645, 756) - r(65, 9) * eta) - (r(732985, 2268) - r(24260, 81) * eta - r(340, 9) * eta ** 2) * s
          - (r(732985, 2268) + r(140, 9) * eta) * delta * a)
    series = [
        1, 0, r(3715, 756) + r(55, 9) * eta,
        -16 * PI + r(113, 3) * delta * a + (r(113, 3) - r(76, 3) * eta) * s,
        r(15293365, 508032) + r(27145, 504) * eta + r(3085, 72) * eta ** 2 + (200 * eta - r(405, 8)) * a ** 2
        - r(405, 4) * delta * s * a + (r(5, 2) * eta - r(405, 8)) * s ** 2,
        c5,
        r(11583231236531, 4694215680) - 640 * PI ** 2 / 3 - r(6848, 21) * (euler + np.log(LD(4)))
        + eta * (r(2255, 12) * PI ** 2 - r(15737765635, 3048192)) + r(76055, 1728) * eta ** 2 - r(127825, 1296) * eta ** 3
        + PI * (r(2270, 3) * delta * a + (r(2270, 3) - 520 * eta) * s) + (r(75515, 144) - r(8225, 18) * eta) * delta * s * a
        + (r(75515, 288) - r(263245, 252) * eta - 480 * eta ** 2) * a ** 2
        + (r(75515, 288) - r(232415, 504) * eta + r(1255, 9) * eta ** 2) * s ** 2,
        PI * (r(77096675, 254016) + r(378515, 1512) * eta - r(74045, 756) * eta ** 2)
        + (r(-25150083775, 3048192) + r(10566655595, 762048) * eta - r(1042165, 3024) * eta ** 2
           + r(5345, 36) * eta ** 3) * s
        + delta * (r(-25150083775, 3048192) + r(26804935, 6048) * eta - r(1985, 48) * eta ** 2) * a]
    x = PI * m * MTSUN * f
    lnv = np.log(x) / 3
    v = np.exp(lnv)
    total = sum(c * v ** k for k, c in enumerate(series)) + lnv * (3 * c5 * v ** 5 - r(6848, 21) * v ** 6)
    phase = 3 / (128 * eta) * total / v ** 5
    psi = phase - 2 * p["phase"] - PI / 4
    mc = eta ** r(3, 5) * m * MTSUN
    amp = np.sqrt(r(5, 24)) * PI ** r(-2, 3) * mc ** r(5, 6) * C / (p["luminosity_distance"] * r(10 ** 6) * PC) * f ** r(-7, 6)
    amp = np.where(f < 1 / (6 * np.sqrt(LD(6)) * PI * m * MTSUN), amp, 0)
    psi = psi - 2 * PI * np.rint(psi / (2 * PI))
    re, im, ci = amp * np.cos(psi), -amp * np.sin(psi), np.cos(p["theta_jn"])
    return (re * (1 + ci ** 2) / 2, im * (1 + ci ** 2) / 2), (ci * im, -ci * re), np.abs(phase)


@pytest.mark.parametrize("workload,duration,fs,masses", [
    ("sg_4s", 2.0, 2048.0, None), ("sg_4s", 4.0, 2048.0, None), ("tf2_128s", 4.0, 2048.0, (10.0, 40.0)),
    ("tf2_128s", 16.0, 2048.0, (5.0, 10.0))])
def test_against_extended_precision(gpu, workload, duration, fs, masses):
    w = small_workload(workload, duration=duration, sampling_frequency=fs, detectors=("H1", "L1"),
                       **({} if masses is None else dict(mass_range=masses)))
    inj = dict(w.injection, geocent_time=w.start_time + 0.6 * duration)
    if masses:
        inj.update(mass_1=masses[1], mass_2=masses[0])
    w = small_workload(workload, **{**w.__dict__, "injection": inj})
    dets = OD.build_workload(w)
    an = device_analysis(dets, w.model, w)
    n = 12
    p = draw_points(w, n, np.random.default_rng(8))
    block = params_block(p)
    few = an.inner_products_host(np.ascontiguousarray(block[:, :3]), "fp64")
    dh, hh = an.inner_products_host(np.ascontiguousarray(np.tile(block, 60)), "fp64")  # a lane per point
    assert np.array_equal(few[0], dh[:3]) and np.array_equal(few[1], hh[:3])
    k0 = int(20 * duration)
    f = dets[0].frequency[k0:].astype(LD)
    for i in range(n):
        q = {k: LD(v[i]) for k, v in p.items()}
        plus, cross, psi = (_burst if masses is None else _taylorf2)(q, f)
        want, norm, tol = np.zeros(2, LD), LD(0), 0.0
        for d in dets:
            t = float(p["geocent_time"][i])
            ra, dec, pol = (float(p[k][i]) for k in ("ra", "dec", "psi"))
            fp, fx = (LD(R.antenna_response(d.tensor, ra, dec, t, pol, mode)) for mode in ("plus", "cross"))
            dt = LD(t - d.start_time) + LD(R.time_delay_from_geocenter(d.vertex, ra, dec, t))
            re, im = plus[0] * fp + cross[0] * fx, plus[1] * fp + cross[1] * fx
            turn = dt * f
            turn = 2 * PI * (turn - np.rint(turn))
            hr, hi = re * np.cos(turn) + im * np.sin(turn), im * np.cos(turn) - re * np.sin(turn)
            with np.errstate(divide="ignore"):
                weight = np.where(d.mask[k0:], 4 / LD(duration) / d.psd[k0:].astype(LD), 0)
            s = d.masked_strain[k0:]
            sr, si = s.real.astype(LD), s.imag.astype(LD)
            want += [((hr * sr + hi * si) * weight).sum(), ((hr * si - hi * sr) * weight).sum()]
            norm += ((hr * hr + hi * hi) * weight).sum()
            size = np.hypot(hr, hi) * np.hypot(sr, si) * weight
            each = 2 * PI * f * (2.0 ** -52 * abs(dt) + 2.0 ** -49 * 0.0213) + 4 * 2.0 ** -53 * psi + 2.0 ** -42
            tol += float((size * each).sum())
        err = max(abs(float(LD(dh[i].real) - want[0])), abs(float(LD(dh[i].imag) - want[1])))
        assert err <= tol, (i, err, tol)
        assert abs(float(LD(hh[i]) - norm)) <= 2.0 ** -47 * float(norm), (i, hh[i], norm)
    an.close()
