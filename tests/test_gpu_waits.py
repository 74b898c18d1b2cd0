"""Failure detection of the bounded waits, without a GPU fault: a warp waits
on a barrier whose copy never arrives (nothing is issued), then one thread on
a block count that nothing raises (the fused passes' row-block wait); each
wait gives up after a short limit, the kernel reports TDF_WAIT_TIMEOUT_BIT
and TDF_ORDER_TIMEOUT_BIT, the host reads them, and the device stays
usable."""
import ctypes as C
import time

import pytest

from tdfstat_b200 import _abi

pytestmark = pytest.mark.gpu

TDF_WAIT_TIMEOUT_BIT = 2
TDF_ORDER_TIMEOUT_BIT = 8


def test_wait_gives_up_and_reports(golden):
    from tdfstat_b200.engine import Engine, load_library
    lib = load_library()
    st = C.c_uint32(0)
    t0 = time.monotonic()
    assert lib.tdf_check_bounded_wait(0, 1000, C.byref(st)) == _abi.TDF_OK
    assert time.monotonic() - t0 < 5.0
    assert st.value & TDF_WAIT_TIMEOUT_BIT
    assert st.value & TDF_ORDER_TIMEOUT_BIT
    # the context is intact: a search right after gives its records
    g = golden("g2_h1l1_inj")
    eng = Engine.from_job(g.job32, form="split")
    res = eng.search(*g.job32.sky_points())
    assert len(res) > 0
    eng.close()


def _small():
    """Two sky points x 3 spindowns of 2^13 points, two detectors."""
    import shutil
    import tempfile

    import numpy as np

    from tdfstat_b200 import host, synth
    root = tempfile.mkdtemp(prefix="tdf_wait_")
    c = synth.Case(dt=16.0, nod=1, band=2880, dets=("H1", "L1"), seed=5, thr=7.0, fdot_step=1e-10, sky_cells=16.0,
                   gtype="directed_range", gcenter=(100.05, -1e-10, 1.2, 0.3), gsizes=(100, 1.0, 0.0, 0.0),
                   gsteps=(1, 1.0, 1.0, 1.0))
    job = host.Job(synth.write_case(root, c), float_build=True)
    shutil.rmtree(root, ignore_errors=True)
    job.range.fr = [job.sett.nmin, job.sett.nmax]
    job.sett.bufsize = job.sett.nfftf
    pm, mm, nn = job.sky_points()
    k = np.arange(2)
    return job, (np.full(2, pm[0], np.int32), (mm[0] - 0.01 * k).astype(np.float32), np.full(2, nn[0], np.float32))


def _calls(eng, job, pts):
    """The three kinds of call, as functions."""
    return {"search": lambda: eng.search(*pts),
            "segments": lambda: eng.search_segments_device([0], [2], *pts),
            "spectrum": lambda: eng.fstat(int(pts[0][0]), float(pts[1][0]), float(pts[2][0]), float(job.range.spndr[0]))}


def _gives_up(monkeypatch, name, form, kinds, env=()):
    import numpy as np

    from tdfstat_b200.engine import Engine, TdfError
    job, pts = _small()
    monkeypatch.setenv(name, "0")
    for k, v in env:
        monkeypatch.setenv(k, v)
    eng = Engine(job.segment(), job.search_opts(), form=form, max_sky_batch=1)
    for kind in kinds:
        for rep in range(3):   # plain launches, capture, replay
            with pytest.raises(TdfError) as ei:
                _calls(eng, job, pts)[kind]()
            assert ei.value.status == _abi.TDF_ERR_CUDA and "wait limit" in str(ei.value), (kind, rep)
    eng.close()
    # the copies were waited for and the context is intact
    monkeypatch.delenv(name)
    for k, _ in env:
        monkeypatch.delenv(k)
    got = []
    for _ in range(2):
        eng = Engine(job.segment(), job.search_opts(), form=form)
        got.append((eng.search(*pts), _calls(eng, job, pts)["segments"](), _calls(eng, job, pts)["spectrum"]()))
        eng.close()
    a, b = got
    assert len(a[0]) == 6 and a[0].ntrig > 0 and a[1] == b[1]
    np.testing.assert_array_equal(a[0].hdr, b[0].hdr)
    np.testing.assert_array_equal(a[0].pairs_flat, b[0].pairs_flat)
    np.testing.assert_array_equal(a[2], b[2])


@pytest.mark.parametrize("form", ["split", "fp64"])
@pytest.mark.parametrize("name,kinds", [("TDF_ROW_WAIT_PROBES", ("search", "segments", "spectrum")),
                                        ("TDF_SKY_WAIT_PROBES", ("segments",))])
def test_row_pass_that_gives_up_stops_copying_and_reports(monkeypatch, form, name, kinds):
    """With a limit of no probes at all the row passes' waits give up at once.
    The call reports it, the groups start no copy whose buffer is still being
    filled, and the copies in flight are waited for before the CTA leaves."""
    _gives_up(monkeypatch, name, form, kinds)


@pytest.mark.parametrize("overlap", ["1", "0"])
@pytest.mark.parametrize("form", ["split", "fp64"])
def test_sky_stage_that_gives_up_is_reported(monkeypatch, form, overlap):
    """The sky stage reports from its own stream into a word that each batch
    starts at zero: the clearing comes before the stage, for a spectrum, a
    call's first batches and the batches that follow in the same slot."""
    _gives_up(monkeypatch, "TDF_SKY_WAIT_PROBES", form, ("spectrum", "search"), (("TDF_SKY_OVERLAP", overlap),))
