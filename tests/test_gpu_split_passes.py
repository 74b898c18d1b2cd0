"""The spindown passes of both forms (tdf_split.cuh) at the sizes where their
index arithmetic and their variants change: every transform length from 2^12
up to 2^17 (square and 2:1 four-step splits, line lengths 64 .. 512), one to
four detectors (compile-time counts and the run-time one), short data in a
long transform (operand columns that end early: fftpad 4), an F range past
nfftf/2, phases past 2^18 turns, and one against two templates per thread.

Spectra are compared with the FP64 oracle, normalised per bin by max(F, 1), at
the forms' tolerances (split 1e-4, FP64 1e-10); records of different launch
shapes must be equal bit for bit."""
import copy
import ctypes as C
import shutil
import tempfile

import numpy as np
import pytest

from tdfstat_b200 import host, synth
from tdfstat_b200.engine import Engine

pytestmark = pytest.mark.gpu

TOL = {"split": 1e-4, "fp64": 1e-10}


def _job(root, dt, nod, nifo, fftpad, thr=14.5, spindowns=1, float_build=False):
    dets = ("H1", "L1", "V1")[:min(nifo, 3)]
    c = synth.Case(dt=float(dt), nod=nod, band=int(180 * dt), dets=dets, sigma=(1.0, 1.3, 0.8), seed=77 + nifo, thr=thr,
                   fdot_step=1e-10, sky_cells=16.0, fftpad=fftpad, gtype="directed_range",
                   gcenter=(100.05, -1e-10, 1.2, 0.3), gsizes=(100, float(spindowns // 2), 0.0, 0.0),
                   gsteps=(1, 1.0, 1.0, 1.0))
    job = host.Job(synth.write_case(root, c), float_build=float_build)
    job.range.fr = [job.sett.nmin, job.sett.nmax]
    job.sett.bufsize = job.sett.nfftf
    for k in range(3, nifo):   # detectors beyond the three known ones: the first, with other noise
        d = copy.copy(job.dets[0])
        d.xdat = np.roll(job.dets[0].xdat, 1000 * k)
        job.dets.append(d)
    job.sett.nifo = len(job.dets)
    return job


@pytest.fixture
def root():
    r = tempfile.mkdtemp(prefix="tdf_split_")
    yield r
    shutil.rmtree(r, ignore_errors=True)


def _spectra(oracle, job, ss, form):
    pm, mm, nn = job.sky_points()
    seg, opts = job.segment(), job.search_opts()
    eng = Engine(seg, opts, form=form)
    F = eng.fstat(pm[0], mm[0], nn[0], ss)
    eng.close()
    Fo = np.zeros_like(F)
    assert oracle.orc_fstat_spectrum(C.byref(seg), C.byref(opts), pm[0], mm[0], nn[0], ss,
                                     Fo.ctypes.data_as(C.POINTER(C.c_double)), len(Fo)) == 0
    return F, Fo


# (dt, nod, fftpad) -> nfftf: 2^12, 2^13, 2^14, 2^15, 2^15 from 2^13, 2^16, 2^17
SIZES = [(32, 1, 1, 12), (16, 1, 1, 13), (8, 1, 1, 14), (4, 1, 1, 15), (16, 1, 4, 15), (2, 1, 1, 16), (2, 2, 1, 17)]


@pytest.mark.parametrize("nifo", [1, 2, 3, 4])
@pytest.mark.parametrize("dt,nod,fftpad,log2", SIZES)
@pytest.mark.parametrize("form", ["split", "fp64"])
def test_spectrum_matches_oracle(oracle, root, form, dt, nod, fftpad, log2, nifo):
    job = _job(root, dt, nod, nifo, fftpad)
    assert job.sett.nfftf == 1 << log2
    F, Fo = _spectra(oracle, job, float(job.range.spndr[0]), form)
    assert np.max(np.abs(F - Fo) / np.maximum(Fo, 1.0)) <= TOL[form]


@pytest.mark.parametrize("form", ["split", "fp64"])
def test_whole_rows(oracle, root, form):
    """An F range past nfftf/2: the row pass forms every output."""
    job = _job(root, 8, 1, 2, 1)
    job.range.fr = [5, job.sett.nfftf - 3]
    F, Fo = _spectra(oracle, job, float(job.range.spndr[0]), form)
    assert np.max(np.abs(F - Fo) / np.maximum(Fo, 1.0)) <= TOL[form]


@pytest.mark.parametrize("turns", [0.9, 1.1, 40.0])
def test_phases_past_2_to_18_turns(oracle, root, turns):
    """The fixed-point phase holds 2^18 turns; larger ones take another
    branch.  The detectors are put at the barycentre, so that the FP32
    per-detector term (whose size grows with the spindown) vanishes and the
    FP64 phase alone is compared."""
    job = _job(root, 8, 1, 2, 1)
    for d in job.dets:
        d.detssb = np.zeros_like(d.detssb)
    N = job.sett.N
    ss = float(np.float32(turns * 2.0 ** 18 * 2 * np.pi / N ** 2 / job.sett.M[5]))
    F, Fo = _spectra(oracle, job, ss, "split")
    assert np.max(np.abs(F - Fo) / np.maximum(Fo, 1.0)) <= TOL["split"]


@pytest.mark.parametrize("rad", [1e5, 1e9, 3e9])
def test_fp64_large_phases(oracle, root, rad):
    """The FP64 form's sine and cosine reduce phases up to 2^30 rad
    themselves.  The library and the oracle round the same phase (its last
    place grows to 5e-7 rad at 3e9), so the spectra still agree."""
    job = _job(root, 8, 1, 2, 1)
    N = job.sett.N
    ss = float(np.float32(rad / float(N) ** 2 / job.sett.M[5]))
    F, Fo = _spectra(oracle, job, ss, "fp64")
    assert np.max(np.abs(F - Fo) / np.maximum(Fo, 1.0)) <= TOL["fp64"]


def _records(eng, pts):
    r = eng.search(*pts)
    return r.hdr.copy(), r.lens.copy(), r.pairs_flat.copy()


@pytest.mark.parametrize("nifo,dt,nod", [(1, 2, 2), (2, 2, 2), (3, 2, 2), (2, 4, 1), (2, 32, 1)])
def test_templates_per_thread_give_the_same_records(root, nifo, dt, nod):
    """Large chunks take two templates per thread (pairs within one sky point,
    and, with 13 spindowns at each of 9 points, pairs of different points and
    a last template alone); single-template chunks take one.  Chunks of 96
    templates of 2^17 points also give the row pass's CTAs many blocks each."""
    job = _job(root, dt, nod, nifo, 1, thr=9.0, spindowns=13, float_build=True)
    pm, mm, nn = job.sky_points()
    k = np.arange(9)
    pts = (np.full(9, pm[0], np.int32), (mm[0] - 0.01 * (k % 3)).astype(np.float32),
           (nn[0] - 0.01 * (k // 3)).astype(np.float32))
    eng = Engine(job.segment(), job.search_opts(), form="split", max_sky_batch=9)
    ref = None
    for tc in (96, 95, 38, 2, 1):
        eng.templates_per_chunk = tc
        got = _records(eng, pts)
        assert len(got[0]) == 9 * 13 and len(got[2]) > 0
        if ref is None:
            ref = got
        for a, b in zip(got, ref):
            np.testing.assert_array_equal(a, b)
    eng.close()
