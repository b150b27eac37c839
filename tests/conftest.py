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


# Tests whose premise is a job that holds the GPU for tens of milliseconds: a
# 192^3 3LPT job in the plain FP64 form took 95 ms on the cuFFT route and 18 ms
# on the fixed-point one, less than the waits that these tests measure against
# it.  They run on the cuFFT route (MFX_FUSED=0).
SLOW_BLOCKER = {"test_server_small_jobs_beside_the_slots"}


@pytest.fixture(autouse=True)
def _slow_blocker_route(request, monkeypatch):
    if request.node.name.split("[")[0] in SLOW_BLOCKER:
        monkeypatch.setenv("MFX_FUSED", "0")
