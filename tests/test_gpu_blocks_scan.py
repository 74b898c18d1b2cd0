"""The scan of every bin that blocks_avg needs (k_block_means, k_threshold):
F ranges of no, one and several 4096-bin blocks with remainders on either side
of the 2048 bins a CTA looks at, and thresholds in the noise, at zero and
below it, where the test that passes bins over must not drop any.  The
triggers are those of MAX_ALG 3 run on the engine's own normalised spectrum
(which the parity tests hold against the oracle), value for value."""
import shutil
import tempfile

import numpy as np
import pytest

from tdfstat_b200 import host, synth
from tdfstat_b200.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def jobs():
    root = tempfile.mkdtemp(prefix="tdf_scan_")
    c = synth.Case(dt=4.0, nod=1, band=720, dets=("H1", "L1"), sigma=(1.0, 1.3), seed=411, fstat_norm="blocks_avg",
                   fdot_step=1e-10, gtype="directed_range", gcenter=(100.05, -1e-10, 1.2, 0.3),
                   gsizes=(100, 1.0, 0.0, 0.0), gsteps=(1, 1.0, 1.0, 1.0))
    ini = synth.write_case(root, c)
    yield {form: host.Job(ini, float_build=form == "split") for form in ("split", "fp64")}
    shutil.rmtree(root, ignore_errors=True)


def _local_maxima(F, thr):
    out, i = [], 1
    while i < len(F) - 2:   # bins fr0+1 .. fr1-2
        if F[i] >= thr and F[i - 1] <= F[i] and F[i] >= F[i + 1]:
            out.append(F[i])
            i += 1
        i += 1
    return np.array(out)


@pytest.mark.parametrize("nbins", [100, 2049, 4095, 4096, 4097, 6144, 8193, 10239, 12289])
@pytest.mark.parametrize("thr", [4.0, 1.0, 0.0, -1.0])
@pytest.mark.parametrize("form", ["split", "fp64"])
def test_triggers_are_the_spectrums_local_maxima(jobs, form, thr, nbins):
    job = jobs[form]
    seg, opts = job.segment(), job.search_opts()
    assert opts.blocks_avg == 1 and job.sett.nfftf >= 1 << 15
    opts.fr[0], opts.fr[1] = 321, 321 + nbins - 1
    opts.thr, opts.bufsize = thr, job.sett.nfftf
    pm, mm, nn = job.sky_points()
    eng = Engine(seg, opts, form=form)
    res = eng.search(pm[:1], mm[:1], nn[:1])
    assert len(res) == 3
    at = 0
    for r in range(len(res)):
        F = eng.fstat(int(pm[0]), *(float(v) for v in res.hdr[r, :3]))
        assert len(F) == nbins
        got = res.pairs_flat[at:at + res.lens[r]].reshape(-1, 2)[:, 1]
        at += int(res.lens[r])
        np.testing.assert_array_equal(got, _local_maxima(F, thr).astype(np.float32))
    eng.close()
