"""The work that users of this framework have it do, as cases to measure.

One case is one call of the Python API on an engine that holds a segment:

  search     Engine.search: sky points x spindowns -> trigger records (what the
             reference's search() loop does, one or many job_core() calls at once)
  spectrum   Engine.fstat: the F-statistic spectrum of one template
  segments   Engine.search_segments_device: several resident segments in one call

over segments of 1 to 6 sidereal days at dt = 2 .. 16 s (N = 5385 .. 258492
samples, FFTs of 2^13 .. 2^18 points), one to three detectors, the split and
the FP64 form, directed and all-sky spindown ranges, zero padding of the
spindown FFT by 1 or 2, with and without blocks_avg.  Inputs are seeded:
Gaussian noise with zeroed gaps and one weak CW signal, a circular orbit plus
Earth rotation, and a lower-triangular grid matrix.
"""
import ctypes as C
import math

import numpy as np
import torch

from tdfstat_b200 import _abi, host
from tdfstat_b200.engine import Engine

DETECTORS = ("H1", "L1", "V1")
BASE = {"call": "search", "form": "split", "dt": 2, "nod": 2, "nifo": 2, "points": 1, "spindowns": 1, "allsky": False,
        "fftpad": 1, "blocks_avg": False, "thr": 14.5, "segments": 1}


def _case(name=None, **kw):
    c = dict(BASE, **kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the spectrum around a candidate that someone looks at: the smallest call, all latency
        _case("spectrum H1L1 2d", call="spectrum"),
        # one job_core() call of a directed single-detector search
        _case("H1 2d 1x65", nifo=1, spindowns=65),
        # one job_core() call of a two-detector search: how the reference's own loop calls the drop-in
        _case("H1L1 2d 1x401", spindowns=401),
        # an all-sky search of a short segment: tens of spindowns at every sky point
        _case("H1L1 1d allsky 24", nod=1, points=24, allsky=True),
        # coarse sampling, short transforms: many sky points, little work at each
        _case("H1L1 dt16 2d 48x33", dt=16, points=48, spindowns=33),
        # an ordinary patch of the two-day configuration
        _case("H1L1 2d 32x401", points=32, spindowns=401, thr=20.0),
        # the precision configuration (six days, 2^18 points), the longest calls
        _case("H1L1 6d 64x401", nod=6, points=64, spindowns=401, thr=20.0),
        # three detectors (compensated network sums), four days
        _case("H1L1V1 4d 4x201", nod=4, nifo=3, points=4, spindowns=201, thr=16.0),
        # block normalisation of F and a padded spindown FFT, three days
        _case("H1L1 3d pad2 avg 4x101", nod=3, points=4, spindowns=101, fftpad=2, blocks_avg=True),
        # several segments resident on one GPU, searched by one call
        _case("4 segments 3d 8x101", call="segments", nod=3, segments=4, points=8, spindowns=101, thr=20.0),
        # the plain FP64 form: a follow-up of a few points, two and six days
        _case("fp64 H1L1 2d 1x65", form="fp64", spindowns=65),
        _case("fp64 H1L1 6d 4x201", form="fp64", nod=6, points=4, spindowns=201, thr=16.0),
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, evenly over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.999)))))))


def draw(rng):
    form = "fp64" if rng.random() < 0.25 else "split"
    call = rng.choice(["search"] * 8 + ["spectrum", "segments"])
    dt = rng.choice([2, 2, 2, 2, 4, 8, 16])
    nod = rng.choice([1, 2, 3, 4, 6])
    fftpad = 2 if rng.random() < 0.2 else 1
    nifo = rng.choice([1, 2, 2, 2, 2, 3])
    points, spindowns = _log(rng, 1, 64), _log(rng, 1, 401)
    c = _case(call=call, form=form, dt=dt, nod=nod, nifo=nifo, fftpad=fftpad)
    nfftf = _settings(c).nfftf
    if form == "fp64" and nfftf > 1 << 18:
        c["fftpad"], nfftf = 1, nfftf // 2
    if call == "spectrum":
        # any template of the segment; another size of segment each time
        return c
    c["segments"] = rng.choice([2, 3, 5]) if call == "segments" else 1
    # at most about 6000 templates of 2^18 points
    cap = max(1, 6000 * (1 << 18) // nfftf // (4 if form == "fp64" else 1) // c["segments"])
    c["allsky"] = rng.random() < 0.2
    c["spindowns"] = 1 if c["allsky"] else spindowns
    per = spindowns if not c["allsky"] else 33
    c["points"] = max(1, min(points, cap // per))
    c["blocks_avg"] = call == "search" and rng.random() < 0.15
    # the threshold that keeps a few hundred triggers at most
    bins = c["points"] * per * c["segments"] * nfftf / 2
    c["thr"] = next(t for t in (14.5, 16.0, 18.0, 20.0, 24.0) if t == 24.0 or bins * math.exp(-t) * (1 + t) < 300)
    return c


# ---------------------------------------------------------------- inputs

EPS = math.radians(84381.448 / 3600.0)          # obliquity
OMEGA_R = 7.2921151467064e-5                    # sidereal rate [rad/s]
YEAR = 365.25 * 86400.0
BAND_FPO = 100.0                                # reference frequency [Hz]
SOURCE = dict(ra=4.0, dec=0.9, iota=0.9, psi=0.4, phase=2.2, f=100.0, fdot=-3e-10)


def _settings(c):
    st = host.Settings(fpo=BAND_FPO, dt=float(c["dt"]), nod=c["nod"], fftpad=c["fftpad"], M=[0.0] * 16).compute()
    return st


def _grid(c, st, rng):
    """A lower-triangular grid matrix with the magnitudes of the reference's example."""
    j = lambda: 1.0 + 0.05 * rng.uniform(-1, 1)  # noqa: E731
    M = [0.0] * 16
    M[0] = 2.0 * math.pi / st.nfftf
    M[5] = math.pi * st.dt * st.dt * 1e-10
    M[4] = -3.63 * M[0] * j()
    M[8] = -517.0 * M[0] * j()
    M[12] = 200.0 * M[0] * j()
    M[9] = -0.78 * M[5] * j()
    M[13] = 1.44 * M[5] * j()
    M[10] = st.oms / 16.0 * j()
    M[14] = -0.516 * M[10] * j()
    M[15] = 0.759 * M[10] * j()
    return M


def _modvir(amod, cphir, sphir, cosm, sinm, ra, dec, x):
    """Amplitude modulations a(t), b(t) of a detector for a source at (ra, dec); 0 in the gaps."""
    ca, sa, cd, sd = math.cos(ra), math.sin(ra), math.cos(dec), math.sin(dec)
    calfr, salfr = ca * cphir + sa * sphir, sa * cphir - ca * sphir
    c, s = calfr * cosm + salfr * sinm, salfr * cosm - calfr * sinm
    c2d, c2sd = cd * cd, sd * cd
    c2s, cs = 2 * c * c, c * s
    a = amod[0] * (2 - c2d) * c2s + amod[1] * (2 - c2d) * 2 * cs + amod[2] * c2sd * c + amod[3] * c2sd * s \
        - amod[0] * (2 - c2d) + amod[4] * c2d
    b = amod[5] * sd * c2s + amod[6] * sd * 2 * cs + amod[7] * cd * c + amod[8] * cd * s - amod[5] * sd
    return a * (x != 0), b * (x != 0)


def _inputs(c, seed, k=0):
    """The arrays and scalars of segment k: what a program reads from its files."""
    rng = np.random.default_rng([seed, k])
    grng = np.random.default_rng([seed, 7919])   # the ephemeris and the signal are the same for all segments
    st = _settings(c)
    st.M = _grid(c, st, np.random.default_rng(7919))   # one grid, whatever the data
    N, dt = st.N, st.dt
    orbit, gmst = grng.uniform(0, 2 * math.pi), grng.uniform(0, 2 * math.pi)
    i = np.arange(N, dtype=np.float64)
    t = i * dt
    cosm, sinm = np.cos(st.omr * i), np.sin(st.omr * i)
    th = orbit + 2 * math.pi / YEAR * t
    AU, RE = 499.00478383615643, 6378.140 / 299792.458
    ex, ey, ez = AU * np.cos(th), AU * np.sin(th) * math.cos(EPS), AU * np.sin(th) * math.sin(EPS)
    dets, sigs = [], []
    f0, f1 = 2 * math.pi * SOURCE["f"] * dt, math.pi * SOURCE["fdot"] * dt * dt
    # the signal lies in the lower quarter of the band
    f0 += math.pi / 4 * (1 + 0.5 * grng.uniform(-1, 1))
    ci, psi, phi = math.cos(SOURCE["iota"]), SOURCE["psi"], SOURCE["phase"]
    cp = (1 + ci * ci) / 2
    amp = (math.cos(2 * psi) * cp * math.cos(phi) - math.sin(2 * psi) * ci * math.sin(phi),
           math.sin(2 * psi) * cp * math.cos(phi) + math.cos(2 * psi) * ci * math.sin(phi),
           -math.cos(2 * psi) * cp * math.sin(phi) - math.sin(2 * psi) * ci * math.cos(phi),
           -math.sin(2 * psi) * cp * math.sin(phi) + math.cos(2 * psi) * ci * math.cos(phi))
    for d in range(c["nifo"]):
        name = DETECTORS[d]
        ephi, elam = host.detector_geometry(name)[:2]
        phir = math.fmod(gmst + elam + 2 * math.pi, 2 * math.pi)
        ro = phir + OMEGA_R * t
        e = np.empty(3 * N)
        e[0::3] = (ex + RE * math.cos(ephi) * np.cos(ro)) / dt
        e[1::3] = (ey + RE * math.cos(ephi) * np.sin(ro)) / dt
        e[2::3] = (ez + RE * math.sin(ephi)) / dt
        x = rng.normal(0.0, (1.0, 1.3, 1.6)[d], N)
        gap = max(1, int(N * 0.05 / 3))
        for s in rng.integers(1, N - gap - 1, size=3):
            x[s:s + gap] = 0.0
        det = host.Detector(name=name, xdat=x.astype(np.float32), detssb=e, phir=phir, epsm=EPS).finish()
        a, b = _modvir(det.amod, det.cphir, det.sphir, cosm, sinm, SOURCE["ra"], SOURCE["dec"], x)
        cr, sr = math.cos(SOURCE["ra"]), math.sin(SOURCE["ra"])
        cd, sd = math.cos(SOURCE["dec"]), math.sin(SOURCE["dec"])
        sh = cr * cd * e[0::3] + sr * cd * e[1::3] + sd * e[2::3]
        ph = f0 * (i + sh) + f1 * (2 * sh * i + i * i + sh * sh) - 2 * math.pi * dt * st.fpo * i
        sn, cn = np.sin(ph), np.cos(ph)
        sigs.append((amp[0] * a + amp[1] * b) * cn + (amp[2] * a + amp[3] * b) * sn)
        dets.append((x, det))
    h0 = 10.0 / math.sqrt(sum(float(np.sum(s * s)) / d.sig2 for s, (_, d) in zip(sigs, dets)))   # network SNR 10
    out = []
    for s, (x, det) in zip(sigs, dets):
        out.append(host.Detector(name=det.name, xdat=(x + h0 * s).astype(np.float32), detssb=det.detssb, phir=det.phir,
                                 epsm=EPS).finish())
    # the patch: grid points around the source, in grid units (float, as the reference holds them)
    be0 = math.cos(EPS) * math.sin(SOURCE["ra"]) * math.cos(SOURCE["dec"]) + math.sin(EPS) * math.sin(SOURCE["dec"])
    be1 = math.cos(SOURCE["ra"]) * math.cos(SOURCE["dec"])
    M = st.M
    m0 = be1 * st.oms / M[15]
    n0 = (be0 * st.oms - m0 * M[14]) / M[10]
    s0 = round((f1 - n0 * M[9] - m0 * M[13]) / M[5])
    side = max(1, math.isqrt(c["points"] - 1) + 1)
    q = np.arange(c["points"])
    mm = (m0 + 0.1 * (q // side - side // 2)).astype(np.float32)
    nn = (n0 + 0.1 * (q % side - side // 2)).astype(np.float32)
    pm = np.full(c["points"], host.ast2lin(SOURCE["ra"], SOURCE["dec"], EPS)[0], dtype=np.int32)
    return dict(st=st, dets=out, cosm=cosm, sinm=sinm, pm=pm, mm=mm, nn=nn,
                smin=float(np.float32(s0 - c["spindowns"] // 2)), smax=float(np.float32(s0 - c["spindowns"] // 2 + c["spindowns"] - 1)))


def _capacity(records):
    """Floats of the pairs array a program provides for so many records."""
    return 4096 + 8 * records


def _ptr(a, t):
    return a.ctypes.data_as(C.POINTER(t))


def _segment(inp):
    """The tdf_segment of the inputs (its arrays stay alive with `inp`)."""
    st, s = inp["st"], _abi.TdfSegment()
    s.N, s.nfft, s.nfftf, s.Ninterp = st.N, st.nfft, st.nfftf, st.Ninterp
    s.interpftpad, s.nifo = st.interpftpad, len(inp["dets"])
    s.dt, s.oms, s.sepsm, s.cepsm, s.Smin, s.Smax = st.dt, st.oms, math.sin(EPS), math.cos(EPS), st.Smin, st.Smax
    for k in range(16):
        s.M[k] = st.M[k]
    s.cosmodf, s.sinmodf = _ptr(inp["cosm"], C.c_double), _ptr(inp["sinm"], C.c_double)
    for k, d in enumerate(inp["dets"]):
        s.det[k].xdat, s.det[k].detssb = _ptr(d.xdat, C.c_float), _ptr(d.detssb, C.c_double)
        s.det[k].sig2, s.det[k].sphir, s.det[k].cphir = d.sig2, d.sphir, d.cphir
        for j in range(9):
            s.det[k].amod[j] = d.amod[j]
    return s


def _opts(c, inp):
    st, o = inp["st"], _abi.TdfSearchOpts()
    o.thr = c["thr"]
    o.fr[0], o.fr[1] = st.nmin, st.nmax
    o.allsky, o.blocks_avg = int(c["allsky"]), int(c["blocks_avg"])
    o.spndr[0], o.spndr[1], o.sstep = inp["smin"], inp["smax"], 1.0
    o.bufsize = st.nfftf // 16 if c["allsky"] else st.nfftf
    o.numlines = 0
    inp["lines"] = np.zeros(2)
    o.lines = _ptr(inp["lines"], C.c_double)
    return o


# ---------------------------------------------------------------- prepare and run

def prepare(case, seed):
    inp = _inputs(case, seed)
    eng = Engine(_segment(inp), _opts(case, inp), form=case["form"])
    state = dict(call=case["call"], form=case["form"], eng=eng, inp=inp, pm=inp["pm"], mm=inp["mm"], nn=inp["nn"], ss=inp["smin"])
    if case["call"] == "segments":
        for k in range(1, case["segments"]):
            more = _inputs(case, seed, k)   # its arrays are read until the call returns
            eng.add_segment(_segment(more))
        n = case["segments"]
        state["slots"] = np.arange(n, dtype=np.int32)
        state["npts"] = np.full(n, case["points"], dtype=np.int32)
        state["pm"], state["mm"], state["nn"] = (np.tile(inp[v], n) for v in ("pm", "mm", "nn"))
    return state


def run(state):
    eng = state["eng"]
    if state["call"] == "spectrum":
        F = eng.fstat(int(state["pm"][0]), float(state["mm"][0]), float(state["nn"][0]), state["ss"])
        # the split form's F is single precision (the call widens it)
        return F if state["form"] == "fp64" else F.astype(np.float32)
    if state["call"] == "segments":
        nrec, ntrig = eng.search_segments_device(state["slots"], state["npts"], state["pm"], state["mm"], state["nn"])
        return {"records": nrec, "triggers": ntrig}
    r = eng.search(state["pm"], state["mm"], state["nn"])
    # the (f, F) pairs go into the program's own array, whose size does not depend on what is found
    pairs = np.zeros(_capacity(len(r)), dtype=np.float32)
    pairs[:len(r.pairs_flat)] = r.pairs_flat
    return {"headers": r.hdr, "lengths": r.lens, "offsets": r.offsets, "pairs": pairs, "per_point": r.per_point}


# ---------------------------------------------------------------- the same in 64 bits

def _sky(inp, p):
    """Sky geometry and grid offsets of point p: (sin, cos of alpha and delta, het0, ra, dec)."""
    st, M = inp["st"], inp["st"].M
    mm, nn = float(inp["mm"][p]), float(inp["nn"][p])
    be1, be2 = (nn * M[10] + mm * M[14]) / st.oms, (nn * M[11] + mm * M[15]) / st.oms
    sd = be1 * math.sin(EPS) - (2 * int(inp["pm"][p]) - 3) * math.sqrt(1 - be1 * be1 - be2 * be2) * math.cos(EPS)
    cd = math.sqrt(1 - sd * sd)
    sa, ca = (be1 - math.sin(EPS) * sd) / (math.cos(EPS) * cd), be2 / cd
    het0 = math.fmod(nn * M[8] + mm * M[12], M[0])
    return sa, ca, sd, cd, het0, math.fmod(math.atan2(sa, ca) + 2 * math.pi, 2 * math.pi), math.asin(sd)


def _spindowns(c, inp, p):
    st, M = inp["st"], inp["st"].M
    mm, nn = float(inp["mm"][p]), float(inp["nn"][p])
    lo, hi = inp["smin"], inp["smax"]
    if c["allsky"]:
        lo = float(np.float32(math.trunc((st.Smin - nn * M[9] - mm * M[13]) / M[5])))
        hi = float(np.float32(math.trunc(-(nn * M[9] + mm * M[13] + st.Smax) / M[5])))
        lo, hi = min(lo, hi), max(lo, hi)
    n = max(0, int(hi - lo + 1))
    return [lo + k for k in range(n)]


def _operands(inp, p, dev):
    """Per detector the resampled series over sig2, the spindown phase terms, and the network sums aa, bb."""
    st = inp["st"]
    N, n = st.N, st.interpftpad * st.N
    sa, ca, sd, cd, het0, _, _ = _sky(inp, p)
    i = torch.arange(N, dtype=torch.float64, device=dev)
    aa = bb = 0.0
    ops = []
    for d in inp["dets"]:
        x = torch.from_numpy(d.xdat).to(dev).double()
        e = torch.from_numpy(d.detssb).to(dev).reshape(N, 3)
        a, b = _modvir(d.amod, d.cphir, d.sphir, torch.from_numpy(inp["cosm"]).to(dev), torch.from_numpy(inp["sinm"]).to(dev),
                       math.atan2(sa, ca), math.asin(sd), x)
        sh = ca * cd * e[:, 0] + sa * cd * e[:, 1] + sd * e[:, 2]
        rot = torch.polar(torch.ones_like(i), -(het0 * i + st.oms * sh))
        aa += float((a * a).sum()) / d.sig2
        bb += float((b * b).sum()) / d.sig2
        at = st.interpftpad * (i - (sh - sh[0]))
        lo = at.floor().clamp(0, n - 2).long()
        B = at - lo
        A = 1 - B
        res = []
        for m in (a, b):
            X = torch.fft.fft(x * m * rot, n=st.nfft)
            half = st.nfft // 2 + 1
            Z = torch.zeros(st.Ninterp, dtype=torch.complex128, device=dev)
            Z[:half] = X[:half]
            Z[st.Ninterp - (st.nfft - half):] = X[half:]
            y = torch.fft.ifft(Z)[:n] * st.interpftpad
            # natural cubic spline: (1, 4, 1) y2 = 6 d with y2 = 0 at both ends, by the decaying
            # inverse of the infinite matrix on the right-hand side extended oddly at the ends
            r = torch.zeros(n, dtype=torch.complex128, device=dev)
            r[1:-1] = 6 * (y[2:] - 2 * y[1:-1] + y[:-2])
            K, z = 40, math.sqrt(3.0) - 2
            ext = torch.cat([-r[1:K + 1].flip(0), r, -r[n - 1 - K:n - 1].flip(0)])
            y2 = sum(z ** abs(k) * ext[K + k:K + k + n] for k in range(-K, K + 1)) / (2 * math.sqrt(3.0))
            v = A * y[lo] + B * y[lo + 1] + ((A ** 3 - A) * y2[lo] + (B ** 3 - B) * y2[lo + 1]) / 6
            res.append(torch.where((at >= 0) & (at <= n - 1), v, torch.zeros_like(v)) / d.sig2)
        ops.append((torch.stack(res), i * i + 2 * i * sh))
    return ops, aa, bb


def _fstat(inp, p, ss, ops, aa, bb, dev, blocks_avg):
    """F of the spindowns ss of point p: (spectra over [fr0, fr1], het0 + het1 of each)."""
    st, M = inp["st"], inp["st"].M
    mm, nn = float(inp["mm"][p]), float(inp["nn"][p])
    het0 = _sky(inp, p)[4]
    het1 = [math.fmod(s * M[4], M[0]) for s in ss]
    het1 = [h + M[0] if h < 0 else h for h in het1]
    spnd = [s * M[5] + nn * M[9] + mm * M[13] for s in ss]
    i = torch.arange(st.N, dtype=torch.float64, device=dev)
    h, w = (torch.tensor(v, dtype=torch.float64, device=dev)[:, None] for v in (het1, spnd))
    x = torch.zeros(len(ss), 2, st.N, dtype=torch.complex128, device=dev)
    for series, term in ops:
        ph = h * i + w * term
        x += torch.polar(torch.ones_like(ph), -ph)[:, None, :] * series
    X = torch.fft.fft(x, n=st.nfftf)[:, :, st.nmin:st.nmax + 1]
    F = X[:, 0].abs().square() / aa + X[:, 1].abs().square() / bb
    nb = (st.nmax - st.nmin) // 4096
    if blocks_avg and nb:
        f = F[:, :nb * 4096].reshape(len(ss), nb, 4096)
        F[:, :nb * 4096] = (f / (f.sum(-1, keepdim=True) / (2.0 * 4096))).reshape(len(ss), -1)
    return F, [het0 + v for v in het1], spnd


def exact(case, seed):
    if case["call"] == "segments":
        return None   # whole numbers only
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    inp = _inputs(case, seed)
    st = inp["st"]
    if case["call"] == "spectrum":
        ops, aa, bb = _operands(inp, 0, dev)
        return _fstat(inp, 0, [inp["smin"]], ops, aa, bb, dev, case["blocks_avg"])[0][0]
    hdr, lens, pairs, per = [], [], [], []
    for p in range(case["points"]):
        ss = _spindowns(case, inp, p)
        per.append(len(ss))
        if not ss:
            continue
        ops, aa, bb = _operands(inp, p, dev)
        ra, dec = _sky(inp, p)[5:]
        for k in range(0, len(ss), 32):
            part = ss[k:k + 32]
            F, het, spnd = _fstat(inp, p, part, ops, aa, bb, dev, case["blocks_avg"])
            mid = F[:, 1:-2]
            peak = (mid >= case["thr"]) & (F[:, :-3] <= mid) & (mid >= F[:, 2:-1])
            for j, (row, at) in enumerate(zip(F, peak)):
                bins = at.nonzero().flatten() + 1
                f = 2.0 * (bins + st.nmin) / st.nfftf * math.pi + het[j]
                pairs.append(torch.stack([f, row[bins]], 1).flatten().cpu().numpy())
                lens.append(2 * len(bins))
                hdr.append([float(inp["mm"][p]), float(inp["nn"][p]), part[j], ra, dec,
                            spnd[j] / (math.pi * st.dt * st.dt)])
    lens = np.array(lens, dtype=np.int64)
    flat = np.zeros(_capacity(len(lens)))
    found = np.concatenate(pairs + [np.zeros(0)])
    flat[:len(found)] = found
    return {"headers": np.array(hdr, dtype=np.float64).reshape(-1, 6), "lengths": lens,
            "offsets": np.concatenate([[0], np.cumsum(lens)])[:-1].astype(np.int64),
            "pairs": flat, "per_point": np.array(per, dtype=np.int32)}


# ---------------------------------------------------------------- work

def work(case):
    st = _settings(case)
    nifo, segs = case["nifo"], case["segments"]
    points = 1 if case["call"] == "spectrum" else case["points"]
    spindowns = 1 if case["call"] == "spectrum" else case["spindowns"]
    if case["allsky"]:
        spindowns = max(1, int((st.Smax + st.Smin) / (math.pi * st.dt * st.dt * 1e-10)) + 1)
    fft = lambda n: 5.0 * n * math.log2(n)  # noqa: E731
    nF = st.nmax - st.nmin + 1
    # a template: per sample and detector the phase, its sine and cosine and the
    # rotation of two complex values; two FFTs; F of the kept bins
    template = 30.0 * nifo * st.N + 2 * fft(st.nfftf) + 9.0 * nF
    # a sky point: modulation and phase, interpolation by FFT, spline
    point = nifo * (100.0 * st.N + 2 * fft(st.nfft) + 2 * fft(st.Ninterp) + 2 * 2 * st.N * 14.0 + 60.0 * st.N)
    inputs = nifo * st.N * (4 + 24) + 2 * 8 * st.N
    out = 4 * nF if case["call"] == "spectrum" else 40 * points * spindowns
    return {"bytes": float(segs * (inputs + out)), "flops": float(segs * points * (point + spindowns * template))}
