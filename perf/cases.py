"""The likelihood evaluations that a user of this package runs, sized as the
configurations in ``bilby_gb300/workloads.py`` and the benchmark have them.

A case is one call of a public entry point on a likelihood that the program
set up beforehand (seeded detector noise with one injected signal):

``point``      ``log_likelihood_ratio(dict)``, one point per call: what a
               sampler that knows nothing of batches does.
``batch``      ``log_likelihood_ratio_batch(dict of arrays)``: a population of
               live points, an ensemble of walkers or a set of prior draws.
``relbin``     the same on the relative-binning likelihood.
``multiband``  the same on the multi-banded likelihood.
``served``     one ``Batcher`` launch over several analyses of uneven length,
               as the serving loop runs it.

``precision`` is the likelihood's own option ("fp64", the default, or
"mixed"); ``marg`` names the marginalised parameters (t, p, d).  ``prepare``
makes everything from the seed: the noise, the likelihood and the points.
"""
from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch

from bilby_gb300 import random as package_random
from bilby_gb300.analysis import params_block
from bilby_gb300.batching import Batcher
from bilby_gb300.detector import InterferometerList
from bilby_gb300.likelihood import GravitationalWaveTransient
from bilby_gb300.multiband import MBGravitationalWaveTransient
from bilby_gb300.prior import PowerLaw, Uniform
from bilby_gb300.relative import RelativeBinningGravitationalWaveTransient
from bilby_gb300.source import sinegaussian, taylorf2_aligned
from bilby_gb300.waveform_generator import WaveformGenerator

START = 1126259640.0
FMIN = 20.0
DISTANCE = dict(alpha=2.0, minimum=100.0, maximum=5000.0)
# component-mass ranges whose inspirals from 20 Hz fit the segment
MASSES = {4.0: (10.0, 40.0), 6.0: (10.0, 40.0), 8.0: (10.0, 40.0), 16.0: (5.0, 10.0), 32.0: (2.5, 5.0),
          64.0: (1.5, 3.0), 128.0: (1.0, 2.0)}


def _case(name, kind, source, duration, rate, detectors, points, precision, marg=""):
    return dict(name=name, kind=kind, source=source, duration=float(duration), rate=float(rate),
                detectors=int(detectors), points=int(points), precision=precision, marg=marg)


def listed():
    return [
        # a sampler's single call on a 4 s burst segment: latency of the smallest analysis
        _case("burst_point", "point", "burst", 4, 2048, 2, 1, "fp64"),
        # a sampler's single call on a binary-neutron-star segment, the default precision
        _case("bns_point", "point", "tf2", 128, 4096, 3, 1, "fp64"),
        # the same call with the precision="mixed" option
        _case("bns_point_mixed", "point", "tf2", 128, 4096, 3, 1, "mixed"),
        # ten thousand prior draws of the burst search
        _case("burst_batch", "batch", "burst", 4, 2048, 2, 10000, "fp64"),
        # a nested sampler's live points on the neutron-star segment, default precision
        _case("bns_batch", "batch", "tf2", 128, 4096, 3, 512, "fp64"),
        # a large mixed-precision batch on the same segment
        _case("bns_batch_mixed", "batch", "tf2", 128, 4096, 3, 4096, "mixed"),
        # black-hole segment of 6 s (FFT length 3 x 2048), time and phase marginalised, a ragged batch
        _case("bbh_marg", "batch", "tf2", 6, 2048, 2, 2047, "fp64", "tp"),
        # black-hole segment of 8 s, time, phase and distance marginalised, mixed precision
        _case("bbh_marg_mixed", "batch", "tf2", 8, 4096, 2, 8192, "mixed", "tpd"),
        # relative binning: a proposal's worth of points
        _case("relbin", "relbin", "tf2", 128, 4096, 3, 16384, "fp64"),
        # relative binning with time marginalisation (the window of a 2^18-point transform)
        _case("relbin_time_mixed", "relbin", "tf2", 128, 4096, 3, 1024, "mixed", "t"),
        # multi-banding
        _case("multiband", "multiband", "tf2", 128, 4096, 3, 4001, "fp64"),
        # a serving step: eight analyses of 4 s to 32 s, a few hundred to a few thousand points each
        _case("served_mixed", "served", "tf2", 0, 0, 0, 8, "mixed"),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["point", "batch", "batch", "batch", "marg", "marg", "relbin", "multiband", "served"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "served":
        return _drawn("served", "tf2", 0, 0, 0, rng.randint(2, 8), "mixed", "", rng)
    if kind in ("relbin", "multiband"):
        duration, rate = rng.choice([(64, 2048), (64, 4096), (128, 2048), (128, 4096)])
        return _drawn(kind, "tf2", duration, rate, rng.choice([1, 2, 3]), _spread(rng, 64, 4096), precision,
                      rng.choice(["", "p"]), rng)
    if kind == "marg":
        duration, rate = rng.choice([(4, 2048), (4, 4096), (6, 2048), (8, 2048), (8, 4096)])
        return _drawn("batch", "tf2", duration, rate, rng.choice([1, 2, 3]), _spread(rng, 16, 4096), precision,
                      rng.choice(["t", "tp", "tpd", "pd"]), rng)
    source = rng.choice(["burst", "tf2", "tf2"])
    if source == "burst":
        duration, rate = rng.choice([(2, 2048), (4, 2048), (4, 4096), (8, 2048)])
        most = 10000
    else:
        duration, rate = rng.choice([(4, 2048), (8, 4096), (16, 2048), (32, 4096), (64, 2048), (128, 4096)])
        # as many point-bins as the largest listed batch of this precision at most
        most = int((4096 if precision == "mixed" else 512) * 128 * 4096 / (duration * rate))
        most = min(most, 10000)
    points = 1 if kind == "point" else _spread(rng, 2, most)
    return _drawn(kind, source, duration, rate, rng.choice([1, 2, 3]), points, precision,
                  rng.choice(["", "", "p"]), rng)


def _drawn(kind, source, duration, rate, detectors, points, precision, marg, rng):
    c = _case("", kind, source, duration, rate, detectors, points, precision, marg)
    del c["name"]
    c["mix"] = rng.randint(0, 1 << 20)
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _injection(source, duration, rng):
    sky = dict(ra=float(rng.uniform(0, 2 * np.pi)), dec=float(np.arcsin(rng.uniform(-1, 1))),
               psi=float(rng.uniform(0, np.pi)))
    if source == "burst":
        return dict(hrss=1e-22, Q=float(rng.uniform(5, 15)), frequency=float(rng.uniform(100, 300)),
                    geocent_time=START + duration / 2, **sky)
    lo, hi = MASSES[duration]
    m = np.sort(rng.uniform(lo, hi, 2))[::-1]
    return dict(mass_1=float(m[0]), mass_2=float(m[1]), chi_1=0.02, chi_2=-0.01,
                luminosity_distance=float(rng.uniform(80, 160) * (1 if duration >= 64 else 7.5)), theta_jn=0.4, phase=1.3,
                geocent_time=START + duration - min(4.0, duration / 4), **sky)


def _data(source, duration, rate, detectors, rng):
    package_random.seed(int(rng.integers(1 << 30)))
    ifos = InterferometerList(["H1", "L1", "V1"][:detectors])
    ifos.set_strain_data_from_power_spectral_densities(rate, duration, START)
    wfg = WaveformGenerator(duration=duration, sampling_frequency=rate, start_time=START,
                            frequency_domain_source_model=sinegaussian if source == "burst" else taylorf2_aligned,
                            waveform_arguments=None if source == "burst" else dict(minimum_frequency=FMIN))
    injection = _injection(source, duration, rng)
    ifos.inject_signal(waveform_generator=wfg, parameters=dict(injection))
    return ifos, wfg, injection


def _points(source, duration, rate, injection, n, marg, rng):
    p = {}
    if source == "burst":
        p["hrss"] = 10 ** rng.uniform(-23, -21, n)
        p["Q"] = rng.uniform(3, 30, n)
        p["frequency"] = rng.uniform(50, 500, n)
    else:
        lo, hi = MASSES[duration]
        m = np.sort(rng.uniform(lo, hi, (2, n)), axis=0)
        p["mass_1"], p["mass_2"] = m[1], m[0]
        p["chi_1"] = rng.uniform(-0.05, 0.05, n)
        p["chi_2"] = rng.uniform(-0.05, 0.05, n)
        p["luminosity_distance"] = rng.uniform(20, 200, n) * (1 if duration >= 64 else 5)
        p["theta_jn"] = np.arccos(rng.uniform(-1, 1, n))
        p["phase"] = rng.uniform(0, 2 * np.pi, n)
    p["ra"] = rng.uniform(0, 2 * np.pi, n)
    p["dec"] = np.arcsin(rng.uniform(-1, 1, n))
    p["psi"] = rng.uniform(0, np.pi, n)
    p["geocent_time"] = injection["geocent_time"] + rng.uniform(-0.1, 0.1, n)
    if "t" in marg:  # the marginalised likelihood's fixed time, and its jitter
        p["geocent_time"] = np.full(n, START)
        p["time_jitter"] = rng.uniform(-1 / rate, 1 / rate, n)
    if "p" in marg:
        p["phase"] = np.zeros(n)
    return p


def _likelihood(case, rng):
    duration, rate, marg = case["duration"], case["rate"], case["marg"]
    if case["source"] == "burst":
        marg = marg.replace("d", "")
    ifos, wfg, injection = _data(case["source"], duration, rate, case["detectors"], rng)
    tc = injection["geocent_time"]
    priors = {"geocent_time": Uniform(tc - 0.1, tc + 0.1), "phase": Uniform(0, 2 * np.pi, boundary="periodic"),
              "luminosity_distance": PowerLaw(**DISTANCE)} if marg else None
    options = dict(priors=priors, precision=case["precision"], time_marginalization="t" in marg,
                   phase_marginalization="p" in marg, distance_marginalization="d" in marg)
    if "d" in marg:  # the distance table is cached on disk, as in the reference
        options["distance_marginalization_lookup_table"] = os.path.join(
            tempfile.gettempdir(), f"perf_distance_{'p' in marg}_{os.getpid()}.npz")
    if case["kind"] == "relbin":
        like = RelativeBinningGravitationalWaveTransient(ifos, wfg, fiducial_parameters=dict(injection), **options)
    elif case["kind"] == "multiband":
        lo = MASSES[duration][0]
        like = MBGravitationalWaveTransient(ifos, wfg, reference_chirp_mass=lo * 2 ** -0.2 * 0.999,
                                            time_offset=2.12, delta_f_end=53.0, **options)
    else:
        like = GravitationalWaveTransient(ifos, wfg, **options)
    points = _points(case["source"], duration, rate, injection, case["points"], marg, rng)
    if "d" in marg:
        points["luminosity_distance"] = np.full(case["points"], priors["luminosity_distance"])  # set to the reference
    return like, points, ifos


def _served(case, seed):
    """[(case of one analysis, seed)] of a serving step."""
    rng = np.random.default_rng([int(case.get("mix", 5)), 64])
    out = []
    for q in range(case["points"]):
        c = _case("", "batch", "tf2", rng.choice([4, 8, 16, 32]), rng.choice([2048, 4096]), rng.choice([2, 3]),
                  round(math.exp(rng.uniform(math.log(256), math.log(4096)))), "mixed")
        out.append((c, [int(seed), q]))
    return out


def prepare(case, seed):
    if case["kind"] == "served":
        items, keep = [], []
        for c, s in _served(case, seed):
            like, points, _ = _likelihood(c, np.random.default_rng(s))
            block = torch.from_numpy(params_block(points)).cuda()
            out = torch.empty(c["points"], dtype=torch.float64, device="cuda")
            items.append((like.analysis, block.data_ptr(), c["points"], out.data_ptr()))
            keep.append((like, block, out))
        return dict(kind="served", batcher=Batcher(use_graphs=True), items=items, keep=keep)
    like, points, _ = _likelihood(case, np.random.default_rng(int(seed)))
    if case["kind"] == "point":
        points = {k: float(v[0]) for k, v in points.items()}
    return dict(kind=case["kind"], like=like, points=points)


def run(state):
    if state["kind"] == "served":
        state["batcher"].eval_device(state["items"], "mixed", torch.cuda.current_stream().cuda_stream)
        return [out for _, _, out in state["keep"]]
    if state["kind"] == "point":
        return state["like"].log_likelihood_ratio(state["points"])
    return state["like"].log_likelihood_ratio_batch(state["points"])


# ---------------------------------------------------------------------------
# work: each input read once, the arithmetic of the definition
# ---------------------------------------------------------------------------
def _band_bins(case):
    """Bins between 20 Hz and the last one a typical template reaches."""
    top = case["rate"] / 2
    if case["source"] != "burst":
        top = min(top, 4397.0 / (2 * MASSES[case["duration"]][0] * 1.5))  # f_ISCO of the middle of the mass range
    return max(1.0, (top - FMIN) * case["duration"])


def work(case):
    if case["kind"] == "served":
        parts = [work(c) for c, _ in _served(case, 0)]
        return {k: float(sum(p[k] for p in parts)) for k in ("bytes", "flops")}
    n, d, bins = case["points"], case["detectors"], _band_bins(case)
    per_bin = 60.0 + 24.0 * d  # phase, sine and cosine; per detector the shift and the product
    nbytes = 16.0 * 8 * n + 24.0 * d * bins
    if case["kind"] == "relbin" and "t" not in case["marg"]:
        edges = 64.0
        return dict(bytes=16.0 * 8 * n + 64.0 * d * edges, flops=n * edges * (per_bin + 40.0 * d))
    if case["kind"] == "relbin":
        return dict(bytes=nbytes, flops=n * (bins * 12.0 * d + 5 * _fft(case) * math.log2(_fft(case))))
    if case["kind"] == "multiband":
        bins /= 20.0
        return dict(bytes=16.0 * 8 * n + 24.0 * d * bins, flops=n * bins * per_bin)
    flops = n * bins * per_bin
    if "t" in case["marg"]:
        flops += n * 5 * _fft(case) * math.log2(_fft(case))
    return dict(bytes=nbytes, flops=flops)


def _fft(case):
    return case["duration"] * case["rate"] / 2


# ---------------------------------------------------------------------------
# the same numbers in float64 from numpy and torch
# ---------------------------------------------------------------------------
MTSUN, PC, C = 4.925490947641267e-06, 3.085677581491367e16, 299792458.0
LEAP = np.array([46828800, 78364801, 109900802, 173059203, 252028804, 315187205, 346723206, 393984007, 425520008,
                 457056009, 504489610, 551750411, 599184012, 820108813, 914803214, 1025136015, 1119744016,
                 1167264017], dtype=np.float64)


def _gmst(gps):
    second = np.floor(gps)
    # the day number is rounded in this order in the reference, and its last digit is 4e-5 s
    jd = 723231 + (second - np.sum(second[:, None] > LEAP, axis=1)) / 86400.0 + 1721013.5
    hi, lo = (jd - 2451545.0) / 36525.0, (gps % 1) / (36525.0 * 86400.0)
    t = hi + lo
    st = (-6.2e-6 * t + 0.093104) * t ** 2 + 67310.54841 + 8640184.812866 * lo + 3155760000.0 * lo \
        + 8640184.812866 * hi + 3155760000.0 * hi
    return (st * 2 * np.pi / 86400.0) % (2 * np.pi)


def _antenna(ifo, p):
    """F+, Fx and the time from the segment start to the signal's arrival."""
    time = p["geocent_time"] + p.get("time_jitter", 0.0)
    phi, theta, psi = p["ra"] - _gmst(time), np.pi / 2 - p["dec"], p["psi"]
    u = np.array([np.cos(phi) * np.cos(theta), np.cos(theta) * np.sin(phi), -np.sin(theta)])
    v = np.array([-np.sin(phi), np.cos(phi), np.zeros_like(phi)])
    m, n = -u * np.sin(psi) - v * np.cos(psi), -u * np.cos(psi) + v * np.sin(psi)
    tensor = np.asarray(ifo.geometry.detector_tensor)
    plus = np.einsum("ij,ip,jp->p", tensor, m, m) - np.einsum("ij,ip,jp->p", tensor, n, n)
    cross = np.einsum("ij,ip,jp->p", tensor, m, n) + np.einsum("ij,ip,jp->p", tensor, n, m)
    omega = np.array([np.sin(theta) * np.cos(phi), np.sin(theta) * np.sin(phi), np.cos(theta)])
    delay = -(np.asarray(ifo.geometry.vertex) @ omega) / C
    return plus, cross, (time - ifo.strain_data.start_time) + delay


def _polarizations(source, p, f):
    """Complex plus and cross of the points (rows) at the frequencies f."""
    col = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda()[:, None] for k, v in p.items()}
    if source == "burst":
        tau = col["Q"] / (2 ** 0.5 * np.pi * col["frequency"])
        temp = col["Q"] / (4 * np.pi ** 0.5 * col["frequency"])
        down = torch.exp(-((f - col["frequency"]) ** 2) * np.pi ** 2 * tau ** 2)
        up = torch.exp(-((f + col["frequency"]) ** 2) * np.pi ** 2 * tau ** 2)
        amp = col["hrss"] * np.pi ** 0.5 * tau / 2
        plus = amp * (down + up) / torch.sqrt(temp * (1 + torch.exp(-col["Q"] ** 2)))
        cross = -1j * amp * (down - up) / torch.sqrt(temp * (1 - torch.exp(-col["Q"] ** 2)))
        return plus.to(torch.complex128), cross
    m1, m2, c1, c2 = col["mass_1"], col["mass_2"], col["chi_1"], col["chi_2"]
    m, pi = m1 + m2, np.pi
    eta, delta, s, a = m1 * m2 / m ** 2, (m1 - m2) / m, (c1 + c2) / 2, (c1 - c2) / 2
    gamma = ((732985 / 2268 - 24260 * eta / 81 - 340 * eta ** 2 / 9) * s + (732985 / 2268 + 140 * eta / 9) * delta * a)
    c5 = pi * (38645 / 756 - 65 * eta / 9) - gamma
    pn = [torch.ones_like(eta), 0 * eta, 3715 / 756 + 55 * eta / 9,
          -16 * pi + 113 / 3 * delta * a + (113 / 3 - 76 * eta / 3) * s,
          15293365 / 508032 + 27145 * eta / 504 + 3085 * eta ** 2 / 72 + (-405 / 8 + 200 * eta) * a ** 2
          - 405 / 4 * delta * s * a + (-405 / 8 + 5 * eta / 2) * s ** 2,
          c5,
          11583231236531 / 4694215680 - 640 * pi ** 2 / 3 - 6848 * 0.5772156649015329 / 21
          - 6848 / 21 * math.log(4.0) + eta * (-15737765635 / 3048192 + 2255 * pi ** 2 / 12)
          + 76055 * eta ** 2 / 1728 - 127825 * eta ** 3 / 1296
          + pi * (2270 / 3 * delta * a + (2270 / 3 - 520 * eta) * s) + (75515 / 144 - 8225 * eta / 18) * delta * s * a
          + (75515 / 288 - 263245 * eta / 252 - 480 * eta ** 2) * a ** 2
          + (75515 / 288 - 232415 * eta / 504 + 1255 * eta ** 2 / 9) * s ** 2,
          pi * (77096675 / 254016 + 378515 * eta / 1512 - 74045 * eta ** 2 / 756)
          + (-25150083775 / 3048192 + 10566655595 * eta / 762048 - 1042165 * eta ** 2 / 3024 + 5345 * eta ** 3 / 36) * s
          + delta * (-25150083775 / 3048192 + 26804935 * eta / 6048 - 1985 * eta ** 2 / 48) * a]
    logs = {5: 3 * c5, 6: -6848 / 21 + 0 * eta}
    sec = m * MTSUN
    f = f.clamp(min=1e-3)  # zero frequency is out of band
    v = torch.exp(torch.log(pi * sec * f) / 3)
    v = v - (v * v * v - pi * sec * f) / (3 * v * v)  # a Newton step towards the cube root
    lnv = torch.log(v)
    total = torch.zeros_like(v)
    for k in reversed(range(8)):
        total = total * v + pn[k] + (logs[k] * lnv if k in logs else 0.0)
    psi = -2 * col["phase"] - pi / 4 + 3 / (128 * eta) * total / v ** 5
    mc = eta ** 0.6 * sec
    amp = (5 / 24) ** 0.5 * pi ** (-2 / 3) * mc ** (5 / 6) * C / (col["luminosity_distance"] * 1e6 * PC) * f ** (-7 / 6)
    on = (f >= FMIN) & (f < 1 / (6 * 6 ** 0.5 * pi * sec))
    wave = torch.where(on, amp, torch.zeros_like(amp)) * torch.exp(-1j * psi)
    ci = torch.cos(col["theta_jn"])
    return wave * (1 + ci ** 2) / 2, -1j * ci * wave


def _response(ifo, source, p, f, pols):
    plus, cross, dt = (torch.from_numpy(np.ascontiguousarray(x)).cuda()[:, None] for x in _antenna(ifo, p))
    return (pols[0] * plus + pols[1] * cross) * torch.exp(-2j * np.pi * f * dt)


def _ln_i0(x):
    return torch.log(torch.special.i0e(x)) + x


def _basis(t, x):
    """The interval and the four cubic B-splines of knots t at x (Cox, de Boor)."""
    left = (torch.searchsorted(t, x, right=True) - 1).clamp(3, len(t) - 5)
    h = [torch.ones_like(x)]
    for k in range(1, 4):
        new = [torch.zeros_like(x) for _ in range(k + 1)]
        for i in range(k):
            lo, hi = t[left + i + 1 - k], t[left + i + 1]
            new[i] = new[i] + h[i] * (hi - x) / (hi - lo)
            new[i + 1] = h[i] * (x - lo) / (hi - lo)
        h = new
    return left, h


def _spline(like, x, y):
    """The distance table's bicubic spline at x (matrix) and y (column)."""
    tx, ty, c = (torch.from_numpy(np.ascontiguousarray(q, dtype=np.float64)).cuda() for q in like._spline_tck)
    box = like._spline_bbox
    y = y.expand_as(x).contiguous()
    inside = (x >= box[0]) & (x <= box[1]) & (y >= box[2]) & (y <= box[3])
    (lx, hx), (ly, hy) = (_basis(t, q.clamp(b0, b1).contiguous())
                          for t, q, b0, b1 in ((tx, x, box[0], box[1]), (ty, y, box[2], box[3])))
    total = torch.zeros_like(x)
    for i in range(4):
        for j in range(4):
            total = total + c[(lx - 3 + i) * (len(ty) - 4) + ly - 3 + j] * hx[i] * hy[j]
    return torch.where(inside, total, torch.full_like(total, -math.inf))


def _marginalised(like, marg, dh, hh, p):
    """Phase and distance marginalisation of <d|h> (matrix) and <h|h> (column)."""
    scale = 1.0
    if "d" in marg:
        scale = torch.from_numpy(p["luminosity_distance"] / like._ref_dist).cuda()[:, None]
        x = (dh.abs() if "p" in marg else dh.real) * scale
        return _spline(like, x, hh * scale ** 2)
    return (_ln_i0(dh.abs()) if "p" in marg else dh.real) - hh / 2


def _time_sum(like, case, marg, z, hh, p):
    """Time marginalisation of the integrand's transform."""
    n = z.shape[1]
    series = torch.fft.fft(z)
    step = case["duration"] / n
    prior = (like.priors["geocent_time"].minimum, like.priors["geocent_time"].maximum)
    times = START + torch.arange(1, n + 1, dtype=torch.float64, device="cuda") * step \
        + torch.from_numpy(p["time_jitter"]).cuda()[:, None]
    lo = max(0, int((prior[0] - START) / step) - 4)
    hi = min(n, int((prior[1] - START) / step) + 4)
    times, series = times[:, lo:hi], series[:, lo:hi]
    lnl = _marginalised(like, marg, series, hh, p)
    lnl = torch.where((times >= prior[0]) & (times <= prior[1]), lnl, torch.full_like(lnl, -math.inf))
    return torch.logsumexp(lnl, dim=1) + math.log(2 / case["rate"] / (prior[1] - prior[0]))


def _exact(case, rng):
    like, points, ifos = _likelihood(case, rng)
    marg = case["marg"] if case["source"] != "burst" else case["marg"].replace("d", "")
    norm, n = 4 / case["duration"], case["points"]
    full = np.asarray(ifos[0].strain_data.frequency_array)
    if case["kind"] == "multiband":
        f = np.asarray(like.banded_frequency_points)
    elif case["kind"] == "relbin":
        f = np.asarray(like.bin_freqs)
    else:
        f = full[:-1] if "t" in marg else full  # (no black-hole template reaches the Nyquist bin)
    weights = []
    for ifo in ifos:
        mask, psd = np.asarray(ifo.strain_data.frequency_mask), np.asarray(ifo.power_spectral_density_array)
        weight = np.where(mask & np.isfinite(psd), 1 / psd, 0.0)
        weights.append((torch.from_numpy(np.asarray(ifo.strain_data.frequency_domain_strain)).cuda(),
                        torch.from_numpy(weight).cuda()))
    grid, ft = torch.from_numpy(full).cuda(), torch.from_numpy(f).cuda()
    cells = len(full) if "t" in marg else len(f)
    result, step = [], max(1, min(n, int(2e7 // cells)))
    for at in range(0, n, step):
        p = {k: v[at:at + step] for k, v in points.items()}
        pols = _polarizations(case["source"], p, ft)
        dh = torch.zeros((len(p["ra"]), 1), dtype=torch.complex128, device="cuda")
        hh = torch.zeros((len(p["ra"]), 1), dtype=torch.float64, device="cuda")
        z = torch.zeros((len(p["ra"]), len(full) - 1), dtype=torch.complex128, device="cuda") if "t" in marg else None
        for ifo, (strain, weight) in zip(ifos, weights):
            h = _response(ifo, case["source"], p, ft, pols)
            if case["kind"] == "multiband":
                lin = torch.from_numpy(np.asarray(like.linear_coeffs[ifo.name])).cuda()
                quad = torch.from_numpy(np.asarray(like.quadratic_coeffs[ifo.name])).cuda()
                dh += (h * lin).sum(1, keepdim=True).conj()
                hh += (h.abs() ** 2 * quad).sum(1, keepdim=True)
            elif case["kind"] == "relbin":
                ratio = h / torch.from_numpy(np.asarray(like.per_detector_fiducial_waveform_points[ifo.name])).cuda()
                width = ft[1:] - ft[:-1]
                r0, r1 = (ratio[:, 1:] + ratio[:, :-1]) / 2, (ratio[:, 1:] - ratio[:, :-1]) / width
                a0, a1, b0, b1 = (torch.from_numpy(np.asarray(s)).cuda() for s in like.summary_data[ifo.name])
                hh += (b0 * r0.abs() ** 2 + 2 * b1 * (r0 * r1.conj()).real).real.sum(1, keepdim=True)
                if "t" not in marg:
                    dh += (a0 * r0.conj() + a1 * r1.conj()).sum(1, keepdim=True)
                    continue
                k0, k1 = int(like.bin_inds[0]), int(like.bin_inds[-1])
                which = torch.repeat_interleave(torch.arange(len(width)), torch.as_tensor(like.bin_sizes)).cuda()
                offset = grid[k0:k1 + 1] - ((ft[1:] + ft[:-1]) / 2)[which]
                h0 = torch.from_numpy(np.asarray(like.per_detector_fiducial_waveforms[ifo.name])).cuda()
                g = norm * h0 * strain.conj() * weight
                z[:, k0:k1 + 1] += (g[k0:k1 + 1] * (r0[:, which] + r1[:, which] * offset))[:, :z.shape[1] - k0]
            else:
                s, w = strain[:len(f)], weight[:len(f)]
                hh += norm * (h.abs() ** 2 * w).sum(1, keepdim=True)
                if "t" in marg:
                    z += norm * h * (s.conj() * w)
                else:
                    dh += norm * (h.conj() * (s * w)).sum(1, keepdim=True)
        if "t" in marg:
            result.append(_time_sum(like, case, marg, z, hh, p))
        else:
            result.append(_marginalised(like, marg, dh, hh, p)[:, 0])
    return torch.cat(result).cpu().numpy()


def exact(case, seed):
    if case["kind"] == "served":
        return [torch.from_numpy(_exact(c, np.random.default_rng(s))) for c, s in _served(case, seed)]
    value = _exact(case, np.random.default_rng(int(seed)))
    return float(value[0]) if case["kind"] == "point" else value
