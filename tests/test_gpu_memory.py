"""Device memory over an engine's life: a call whose buffers cannot grow is
refused and leaves the engine as it was."""
import shutil
import tempfile

import numpy as np
import pytest

from tdfstat_b200 import _abi, host, synth
from tdfstat_b200.engine import Engine, TdfError

pytestmark = pytest.mark.gpu


def _job(dt, nod, band, fdots, thr):
    root = tempfile.mkdtemp(prefix="tdf_mem_")
    c = synth.Case(dt=dt, nod=nod, band=band, dets=("H1",), seed=9, thr=thr, fdot_step=1e-10, sky_cells=16.0,
                   gtype="directed_range", gcenter=(100.05, -1e-10, 1.2, 0.3), gsizes=(100, fdots, 0.0, 0.0),
                   gsteps=(1, 1.0, 1.0, 1.0))
    job = host.Job(synth.write_case(root, c), float_build=True)
    shutil.rmtree(root, ignore_errors=True)
    job.range.fr = [job.sett.nmin, job.sett.nmax]
    job.sett.bufsize = job.sett.nfftf
    return job


def test_trigger_buffers_that_cannot_grow():
    """More than 2^21 triggers in a batch make the trigger buffers grow.  When
    the device has no room for that the call returns TDF_ERR_OUT_OF_MEMORY; the
    engine keeps the buffers it has, searches with fewer triggers still run,
    and the same call succeeds once there is room."""
    import torch
    job = _job(2.0, 1, 360, 200.0, 3.0)   # about 2900 triggers in each of 401 templates of 2^16 points
    pm, mm, nn = job.sky_points()
    k = np.arange(4)
    pts = (np.full(4, pm[0], np.int32), (mm[0] - 0.01 * k).astype(np.float32), np.full(4, nn[0], np.float32))
    eng = Engine(job.segment(), job.search_opts(), form="split")
    few = eng.search_device(*(v[:1] for v in pts))
    assert few[0] == 401 and few[1] < 2 ** 21
    torch.cuda.init()
    free = torch.cuda.mem_get_info()[0]
    hold = torch.empty(free - (48 << 20), dtype=torch.uint8, device="cuda")   # the growth takes 128 MB and more
    for _ in range(2):
        with pytest.raises(TdfError) as ei:
            eng.search_device(*pts)
        assert ei.value.status == _abi.TDF_ERR_OUT_OF_MEMORY
        assert eng.search_device(*(v[:1] for v in pts)) == few
    del hold
    torch.cuda.empty_cache()
    many = eng.search_device(*pts)
    assert many[0] == 4 * 401 and many[1] > 2 ** 21
    assert eng.search_device(*(v[:1] for v in pts)) == few
    eng.close()


def test_engines_give_back_their_memory():
    """Creating, using and closing engines takes no device memory for good: a
    buffer of the smallest kind (512 bytes) left behind per lane keeps about 20 KB
    of the device's memory from being given back, 6 MB after 300 engines."""
    import torch
    job = _job(16.0, 1, 2880, 1.0, 14.5)
    seg, opts = job.segment(), job.search_opts()
    pm, mm, nn = job.sky_points()

    def rounds(n):
        for k in range(n):
            eng = Engine(seg, opts, form=("split", "fp64")[k % 2], max_sky_batch=1)
            if k % 100 < 2:
                eng.search_device(pm, mm, nn)
            eng.close()

    torch.cuda.init()
    rounds(8)
    free = torch.cuda.mem_get_info()[0]
    rounds(300)
    assert torch.cuda.mem_get_info()[0] >= free
