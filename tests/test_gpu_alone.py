"""Launches overlap only while a job has the GPU to itself: work that is done, or
only captured, is no company, work that runs is.

A 32^3 2LPT pass takes 59 us with overlapping launches and 70 with plain ones; the
bar lies between, and each side's time is the least of several groups.
"""
import time

import pytest

from test_gpu_batch import spec

pytestmark = pytest.mark.gpu


def pass_us(job, groups=8, count=100):
    best = 1e9
    for _ in range(groups):
        t = time.perf_counter()
        for _ in range(count):
            job.run()
        best = min(best, 1e6 * (time.perf_counter() - t) / count)
    return best


@pytest.fixture()
def small(mfxlib, engine):
    sp = spec(mfxlib, 32, 100.0, 24.0, 2, 5, precision=mfxlib.FP32C)
    job = mfxlib.Job(engine, **sp)
    pass_us(job, groups=2)
    yield job, sp
    job.close()


def test_beside_work_that_is_done(mfxlib, engine, small):
    job, sp = small
    alone = pass_us(job)

    def same():
        assert pass_us(job) < 1.08 * alone

    batch = mfxlib.Batch(engine, [sp, sp])
    same()  # captured, never launched
    batch.run()
    batch.wait()
    same()
    batch.close()
    srv = mfxlib.Server(engine, 1)
    ticket = srv.submit(sp)
    srv.wait(ticket, 60000)
    same()  # its result not yet released
    srv.release(ticket)
    srv.close()
    other = mfxlib.Job(engine, **sp)
    other.capture()
    same()
    other.run(wait=False)
    other.particles()  # waits by itself
    same()
    other.close()
    same()


def test_beside_work_that_runs(mfxlib, engine, small):
    """A captured job's launches and a batch's count like any other's."""
    job, sp = small
    alone = pass_us(job)
    other = mfxlib.Job(engine, **sp)
    other.capture()
    other.run()
    other.run(wait=False)  # a graph's second launch: running until it is waited for
    assert pass_us(job) > 1.08 * alone
    other.wait()
    assert pass_us(job) < 1.08 * alone
    batch = mfxlib.Batch(engine, [sp, sp])
    batch.run()
    assert pass_us(job) > 1.08 * alone
    batch.wait()
    assert pass_us(job) < 1.08 * alone
    batch.close()
    other.close()
