"""The interpolation of the sky stage (forward FFT, inverse FFT that delivers
spline coefficients, natural-spline evaluation) where its end conditions and
its variants matter: series of a few samples (both ends of the spline within
reach of each other), series that fill the transform (the periodic
coefficients wrap), resampling shifts that leave the data at either end, and
interpolation factors other than two (the passes that are fused for a factor
of two run apart).  The FP64 form's spectra are compared with the FP64 oracle
at that form's tolerance (1e-10, normalised per bin by max(F, 1))."""
import ctypes as C
import shutil
import tempfile

import numpy as np
import pytest

from tdfstat_b200 import host, synth
from tdfstat_b200.engine import Engine

pytestmark = pytest.mark.gpu

TOL = 1e-10


@pytest.fixture(scope="module")
def job():
    root = tempfile.mkdtemp(prefix="tdf_interp_")
    c = synth.Case(dt=8.0, nod=1, band=1440, dets=("H1", "L1"), sigma=(1.0, 1.3), seed=91, fdot_step=1e-10,
                   gtype="directed_range", gcenter=(100.02, -1e-10, 1.2, 0.3), gsizes=(100, 0.0, 0.0, 0.0),
                   gsteps=(1, 1.0, 1.0, 1.0))
    yield host.Job(synth.write_case(root, c), float_build=False)
    shutil.rmtree(root, ignore_errors=True)


# the job's series has N = 10771 samples; the transforms asked for are its own 2^14, or shorter with fewer samples
@pytest.mark.parametrize("N,nfft,pad,shift", [
    (10771, 1 << 14, 2, 0.0), (8192, 1 << 13, 2, 0.0), (4096, 1 << 12, 2, 300.0), (4095, 1 << 12, 2, -300.0),
    (3000, 1 << 12, 1, 50.0), (3000, 1 << 12, 4, 50.0), (4096, 1 << 12, 4, -50.0), (4096, 1 << 12, 1, 0.0),
    (150, 1 << 12, 2, 3.0), (40, 1 << 12, 2, -3.0), (11, 1 << 12, 2, 1.0), (3, 1 << 12, 2, 0.0)])
def test_spectrum_matches_oracle(oracle, job, N, nfft, pad, shift):
    seg, opts = job.segment(), job.search_opts()
    seg.N, seg.nfft, seg.nfftf, seg.interpftpad, seg.Ninterp = N, nfft, nfft, pad, pad * nfft
    opts.fr[0], opts.fr[1] = 1, nfft // 2 - 1
    keep = []
    for d in range(seg.nifo):
        # the start is the reference point of the resampling: a ramp over the series shifts its far end
        e = job.dets[d].detssb[:3 * N].copy().reshape(N, 3)
        ramp = np.linspace(0.0, 1.0, N)[:, None] * shift
        e = np.ascontiguousarray((e - e[0]) * (1.0 if N > 1000 else 0.0) + ramp * np.array([0.3, 0.9, 0.3]))
        keep.append(e)
        seg.det[d].detssb = e.ctypes.data_as(C.POINTER(C.c_double))
    pm, mm, nn = job.sky_points()
    ss = float(job.range.spndr[0])
    eng = Engine(seg, opts, form="fp64")
    F = eng.fstat(pm[0], mm[0], nn[0], ss)
    eng.close()
    Fo = np.zeros_like(F)
    assert oracle.orc_fstat_spectrum(C.byref(seg), C.byref(opts), pm[0], mm[0], nn[0], ss,
                                     Fo.ctypes.data_as(C.POINTER(C.c_double)), len(Fo)) == 0
    assert np.all(np.isfinite(Fo)) and np.max(Fo) > 0
    assert np.max(np.abs(F - Fo) / np.maximum(Fo, 1.0)) <= TOL
