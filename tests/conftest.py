import os
import sys
import pathlib

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (GB300) and the built libmfx.so")


@pytest.fixture(scope="session")
def mfxlib():
    from monofonic_gb300 import build, mfx
    build.build()
    return mfx


@pytest.fixture(scope="session")
def engine(mfxlib):
    import torch  # noqa: F401  (only to report a clear skip reason)
    eng = mfxlib.Engine(0)
    yield eng
    eng.close()


@pytest.fixture(scope="session")
def oracle():
    from oracle import lpt
    lpt.build_lib()
    return lpt


# Tests whose premise is a job that runs for longer than the waits measured
# beside it (ms, with room): name -> (that job's grid, the time).  The one below
# was written with a 192^3 3LPT job of the plain FP64 form, 96 ms then and 13 ms
# since its transforms left cuFFT, against waits of 30 ms.  It gets the smallest
# grid whose own run is long enough on the kernels as they are.
LONG_JOB = {"test_server_small_jobs_beside_the_slots": (192, 70.0)}


@pytest.fixture(autouse=True)
def _long_job(request, monkeypatch):
    name = request.node.name.split("[")[0]
    if name not in LONG_JOB:
        return
    import time
    grid, least = LONG_JOB[name]
    engine, given = request.getfixturevalue("engine"), request.module.spec

    def run_ms(mfx, sp):
        job, times = mfx.Job(engine, **sp), []
        for _ in range(2):
            t = time.perf_counter()
            job.run()
            job.wait()
            times.append(1e3 * (time.perf_counter() - t))
        job.close()
        return min(times)

    def spec(mfx, n, *args, **kw):
        if n != grid:
            return given(mfx, n, *args, **kw)
        for m in (grid, 256, 320, 384, 448, 512):
            sp = given(mfx, m, *args, **kw)
            if run_ms(mfx, sp) >= least:
                return sp
        raise AssertionError("no grid up to 512 runs for %g ms" % least)

    monkeypatch.setattr(request.module, "spec", spec)
