"""Failure detection, exercised without faulting the GPU.

* A stalled pipeline: FLETCHER_InjectFault(FLETCHER_FAULT_STALL, n, wait_us)
  makes CTA 0 of the next propagate launch skip the loads of its n-th step.
  Its bounded waits for that stage run out after wait_us (the kernel's own
  limit is 2 s), it drains the loads it has in flight and returns; the host
  reads the error word and DRIVER_Propagate reports FLETCHER_ERR_TIMEOUT.
  Nothing waits forever and no address is touched out of bounds.  The
  process then re-initialises and runs a correct simulation.
* An allocation failure: FLETCHER_FAULT_ALLOC fails one device allocation of
  DRIVER_Initialize (host-side fake of cudaMalloc); the call reports
  FLETCHER_ERR_NOMEM, releases the rest, and the next set-up succeeds.
* Non-finite model values are rejected at set-up, naming array and cell.
"""
import time

import numpy as np
import pytest

from conftest import gpu_available
from fletcher_petrobras_gb300 import FletcherError, Problem, Propagator

pytestmark = pytest.mark.gpu

FAULT_NONE, FAULT_ALLOC, FAULT_STALL, FAULT_QUIT = 0, 1, 2, 3
ERR_TIMEOUT, ERR_NOMEM, ERR_ARGS = 3, 4, 1

PROB = Problem("faults", 36, 30, 28, absorb=5, dt=0.0006, steps=12, fcut=45.0, kind="layered", layers=3, seed=6)


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    if not gpu_available():
        pytest.fail("these tests need a CUDA GPU")


def rel_l2(a, b):
    a = np.asarray(a, np.float64)
    b = np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def clean_run(orc, prob=PROB):
    """A full run after a failure, checked against the oracle."""
    m = prob.model()
    prop = Propagator()
    prop.initialize(prob.sx, prob.sy, prob.sz, prob.bord, prob.dx, prob.dy, prob.dz, prob.dt, m)
    prop.run(prob.steps, prob.i_source, prob.sources())
    prop.synchronize()
    p, q = prop.field(0), prop.field(1)
    prop.finalize()
    op, oq, _, _ = orc.run_f32(prob, m)
    assert rel_l2(p, op) < 1e-5 and rel_l2(q, oq) < 1e-5


@pytest.mark.parametrize("stall_step", [0, 5])
def test_stalled_pipeline_reports_timeout_then_recovers(stall_step, orc):
    prop = Propagator()
    lib = prop.lib
    m = PROB.model()
    prop.initialize(PROB.sx, PROB.sy, PROB.sz, PROB.bord, PROB.dx, PROB.dy, PROB.dz, PROB.dt, m)
    prop.propagate(1)  # a normal step first
    assert lib.FLETCHER_InjectFault(FAULT_STALL, stall_step, 20000) == 0
    with pytest.raises(FletcherError, match=r"gave up waiting.*\(code 3\)"):
        prop.propagate(2)
    # The injection applied to that one launch only.
    lib.FLETCHER_ClearError()
    prop.finalize()
    clean_run(orc)


def failing_step(prob, kind, arg, wait_us, zchunks, **kw):
    """A step with a source in which the fault is injected, after a normal
    one; returns the seconds it took to report the give-up."""
    prop = Propagator(zchunks=zchunks, **kw)
    prop.initialize(prob.sx, prob.sy, prob.sz, prob.bord, prob.dx, prob.dy, prob.dz, prob.dt, prob.model())
    prop.insert_source(1, prob.i_source, 1.0)
    prop.propagate(1)
    prop.insert_source(2, prob.i_source, 1.0)
    assert prop.lib.FLETCHER_InjectFault(kind, arg, wait_us) == 0
    t = time.perf_counter()
    with pytest.raises(FletcherError, match=r"gave up waiting.*\(code 3\)"):
        prop.propagate(2)
    t = time.perf_counter() - t
    prop.lib.FLETCHER_ClearError()
    prop.finalize()
    Propagator()  # the default form, numerics and shape again
    return t


FORMS = [dict(), dict(form="fp16"), dict(form="fp16x"), dict(numerics="d1d1")]
# The source's plane is step 16 of CTA 0's column; in the second problem every
# CTA has several items, the source's plane in one of the later ones.
DEEP = PROB.with_(source=(20, 20, 16))
SHORT = Problem("short", 170, 130, 30, absorb=5, dt=0.0006, steps=9, fcut=45.0, kind="layered", layers=4, seed=12,
                source=(68, 52, 30))


@pytest.mark.parametrize("prob,zchunks,step", [(DEEP, -1, 0), (DEEP, -1, 16), (DEEP, -1, 20), (SHORT, -16, 1)])
@pytest.mark.parametrize("kw", FORMS, ids=lambda k: next(iter(k.values()), "fp32"))
def test_helper_warp_that_gives_up_leaves_no_other_waiting(kw, prob, zchunks, step, orc):
    """A helper warp whose wait runs out while its sisters' waits succeed: they
    meet at a barrier once a plane (16-bit forms) or on the source's plane, and
    every warp leaves."""
    failing_step(prob, FAULT_QUIT, step, 20000, zchunks, **kw)
    clean_run(orc)


@pytest.mark.parametrize("kw", FORMS, ids=lambda k: next(iter(k.values()), "fp32"))
def test_counted_waits_end_in_time(kw, orc):
    """Waits limited by a count of tries end within the limit they stand for:
    the stalled stage's readers after one, the producer, which waits for them,
    after another, then its drain of the missing loads (200 ms), and a second
    for the rest."""
    wait_s = 0.4
    t = failing_step(DEEP, FAULT_STALL, 3, int(wait_s * 1e6), -1, **kw)
    print(f"gave up after {t:.3f} s")
    assert t < 2 * wait_s + 0.2 + 1.0
    clean_run(orc)


def test_stall_argument_checks():
    lib = Propagator().lib
    lib.FLETCHER_ClearError()
    assert lib.FLETCHER_InjectFault(FAULT_STALL, 0, 10) == ERR_ARGS  # wait below 1 ms
    lib.FLETCHER_ClearError()
    assert lib.FLETCHER_InjectFault(FAULT_STALL, -1, 20000) == ERR_ARGS
    lib.FLETCHER_ClearError()
    assert lib.FLETCHER_InjectFault(7, 0, 0) == ERR_ARGS
    lib.FLETCHER_ClearError()
    assert lib.FLETCHER_InjectFault(FAULT_NONE, 0, 0) == 0


@pytest.mark.parametrize("which", [0, 2, 4])
def test_allocation_failure_reports_nomem_then_recovers(which, orc):
    prop = Propagator()
    lib = prop.lib
    assert lib.FLETCHER_InjectFault(FAULT_ALLOC, which, 0) == 0
    with pytest.raises(FletcherError, match=r"\(code 4\)"):
        prop.initialize(PROB.sx, PROB.sy, PROB.sz, PROB.bord, PROB.dx, PROB.dy, PROB.dz, PROB.dt, PROB.model())
    assert lib.FLETCHER_DeviceBytes() == 0  # nothing kept
    lib.FLETCHER_InjectFault(FAULT_NONE, 0, 0)
    clean_run(orc)


@pytest.mark.parametrize("array,value", [(2, np.nan), (0, np.inf), (5, -np.inf)])
def test_non_finite_model_values_rejected(array, value, orc):
    m = PROB.model()
    cell = PROB.n // 3 + 7
    m[array, cell] = value
    names = ["vpz", "vsv", "epsilon", "delta", "phi", "theta"]
    prop = Propagator()
    with pytest.raises(FletcherError, match=rf"{names[array]} holds a value that is not finite at cell {cell}"):
        prop.initialize(PROB.sx, PROB.sy, PROB.sz, PROB.bord, PROB.dx, PROB.dy, PROB.dz, PROB.dt, m)
    clean_run(orc)
