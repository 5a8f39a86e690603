"""Failure detection on the GPU without a fault: the bounded barrier wait.

The cooperative-grid form of the LU-SGS/GS sweeps separates hyperplanes with a
software grid barrier whose wait is bounded (ORION_SWEEP_SPIN_LIMIT polls,
read when a case is made).  With a limit of one poll the first CTA to arrive
gives up at once: the kernel records the error and every CTA returns, the host
reports ORION_E_TIMEOUT, and the context stays usable for the next case.
"""
import ctypes as C
import os

import numpy as np
import pytest

from orion_b200 import _lib, cases, output, shard, solver
from orion_b200._lib import OrionError

pytestmark = pytest.mark.gpu


def test_grid_barrier_timeout_is_reported_and_the_context_survives():
    case = cases.small_case("timeout", dims=(33, 25, 23), noise_seed=5)
    os.environ["ORION_SWEEP_SPIN_LIMIT"] = "1"
    try:
        fs = solver.FlowFieldSet(case, precision=_lib.PREC_FP64)
    finally:
        del os.environ["ORION_SWEEP_SPIN_LIMIT"]
    fs.set_schedule("grid", 0, 32)
    with pytest.raises(OrionError) as err:
        fs.step(1)
    assert "-6" in str(err.value) and "gave up waiting" in str(err.value)
    fs.close()
    # a new case on the same context runs and matches a fresh reference run
    a = solver.FlowFieldSet(case, precision=_lib.PREC_FP64)
    b = solver.FlowFieldSet(case, precision=_lib.PREC_FP64)
    a.set_schedule("grid", 0, 32)
    assert np.array_equal(a.step(3), b.step(3))
    a.close()
    b.close()


def test_tile_wavefront_wait_timeout_is_reported_and_the_context_survives():
    """The tile wavefront's waits on its upstream tiles are bounded too: with a
    limit of one poll a tile that finds its upstream tile behind gives up, the
    error word stops every other waiting tile, and the host reports
    ORION_E_TIMEOUT.  The case is made of blocks wide enough in j and k to hold
    several tiles each, so that tiles do wait on one another."""
    case = cases.small_case("timeout_tiles", dims=(33, 70, 25), split=(1, 1, 1), noise_seed=5)
    os.environ["ORION_SWEEP_SPIN_LIMIT"] = "1"
    try:
        fs = solver.FlowFieldSet(case, precision=_lib.PREC_FP64)
    finally:
        del os.environ["ORION_SWEEP_SPIN_LIMIT"]
    fs.set_schedule("tiles", 0, 32)
    with pytest.raises(OrionError) as err:
        fs.step(1)
    assert "-6" in str(err.value)
    fs.close()
    a = solver.FlowFieldSet(case, precision=_lib.PREC_FP64)
    b = solver.FlowFieldSet(case, precision=_lib.PREC_FP64)
    b.set_schedule("planes", 0, 32)
    assert np.array_equal(a.step(3), b.step(3))
    a.close()
    b.close()


def _limited(case, precision=_lib.PREC_FP64, make=solver.FlowFieldSet):
    """A case whose device waits give up after one poll."""
    os.environ["ORION_SWEEP_SPIN_LIMIT"] = "1"
    try:
        return make(case, precision=precision)
    finally:
        del os.environ["ORION_SWEEP_SPIN_LIMIT"]


def _restart(fs):
    _lib.check(_lib.load().orion_case_init_flow(fs.handle, fs.case.noise_seed, fs.case.noise_amp))


def _stages(fs):
    halo = solver.HaloExchanger()
    halo.exchange_bc(None, fs)
    solver.apply_physical_bc(None, fs)
    solver.StateUpdater.update_flow_states(fs)
    solver.TimeIntegrator.calculate_time_step(fs)
    solver.FluxComputer.compute_viscous_rhs(fs)
    halo.average_interface_residuals(None, fs)
    solver.InviscidFluxComputer.compute_inviscid_rhs(fs)
    halo.average_interface_residuals(None, fs)
    solver.StateUpdater.update_solution(fs)


def _phydtime(fs):
    v = C.c_double()
    _lib.check(_lib.load().orion_phydtime(fs.handle, C.byref(v)))


# what hands out a result: how the steps were enqueued, the call that waits
WAITS = {
    "stages-residual": (_stages, lambda fs: solver.ResidualMonitor.compute(fs)),
    "stages-download": (_stages, lambda fs: fs.download(0, "prim")),
    "async-sync": (lambda fs: fs.step_async(1), lambda fs: fs.sync()),
    "async-download": (lambda fs: fs.step_async(1), lambda fs: fs.download(0, "dq")),
    "async-pack": (lambda fs: fs.step_async(1), lambda fs: output.pack_block(fs, 0)),
    "async-last": (lambda fs: fs.step_async(1), lambda fs: fs.last_residual()),
    "async-phydtime": (lambda fs: fs.step_async(1), _phydtime),
}


@pytest.mark.parametrize("precision", [_lib.PREC_FP64, _lib.PREC_MIXED], ids=["plain", "mixed"])
@pytest.mark.parametrize("how", list(WAITS))
def test_every_call_that_hands_out_a_result_reports_the_timeout(how, precision):
    """Sweeps that gave up leave a state and a residual of no use: the first
    call that waits for them says so, whichever it is, and the case steps on
    from a new state."""
    send, wait = WAITS[how]
    case = cases.small_case("timeout_waits", dims=(33, 70, 25), noise_seed=5)
    fs = _limited(case, precision)
    send(fs)
    with pytest.raises(OrionError, match="-6"):
        wait(fs)
    wait(fs)  # reported once
    fs.set_schedule("planes", 0, 16)
    _restart(fs)
    ref = solver.FlowFieldSet(case, precision=precision)
    ref.set_schedule("planes", 0, 16)
    assert np.array_equal(fs.step(2), ref.step(2))
    fs.close()
    ref.close()


def test_a_shard_reports_the_timeout_with_its_residual():
    case = cases.small_case("timeout_shard", dims=(33, 141, 25), split=(1, 2, 1), noise_seed=5)
    shards = [_limited(case, make=lambda c, precision, r=r: shard.Shard(c, [0, 1], r, precision=precision))
              for r in range(2)]
    try:
        with pytest.raises(OrionError, match="-6"):
            shard.ShardGroup(shards, shard.LocalTransport()).run(1)
    finally:
        for s in shards:
            s.close()


GROUP = [dict(name="tg0", dims=(33, 70, 25), noise_seed=5), dict(name="tg1", dims=(25, 33, 61), noise_seed=6),
         dict(name="tg2", dims=(33, 75, 23), split=(2, 1, 1), noise_seed=7)]


def _group(limited=0):
    """A group whose member `limited` bounds its waits by one poll; so does the group."""
    members = [(_limited if m == limited else solver.FlowFieldSet)(cases.small_case(**sp)) for m, sp in enumerate(GROUP)]
    return members, solver.CaseGroup(members)


@pytest.mark.parametrize("limited", [0, 2])
def test_a_group_takes_its_members_wait_limit(limited):
    members, g = _group(limited)
    g.submit(1)
    with pytest.raises(OrionError, match="-6"):
        g.sync()
    g.close()
    for fs in members:
        fs.close()


def _poll(fs):
    while True:
        h = fs.poll()
        if h is not None:
            return h


def _steps_like_a_new_case(fs):
    """In the tile form: the edge records that the group's sweeps left are gone."""
    _restart(fs)
    ref = solver.FlowFieldSet(fs.case)
    assert np.array_equal(fs.step(2), ref.step(2))
    ref.close()


@pytest.mark.parametrize("ask", ["poll", "sync", "download", "destroyed"])
def test_every_member_of_a_group_reports_the_timeout(ask):
    members, g = _group(limited=1)
    g.submit(1)
    if ask == "sync":
        with pytest.raises(OrionError, match="-6"):
            g.sync()
        g.sync()  # reported once
    if ask == "destroyed":
        g.close()
    for fs in members:
        with pytest.raises(OrionError, match="-6"):
            _poll(fs) if ask == "poll" else fs.download(0, "prim")
    for fs in members:
        if ask == "poll":
            assert len(_poll(fs)) == 0  # nor is that history given out later
        fs.sync()
    g.close()
    for m, fs in enumerate(members):
        if m != 1:  # this one still gives up after one poll
            _steps_like_a_new_case(fs)
        fs.close()


def test_a_group_that_told_its_timeout_starts_anew():
    members, g = _group()
    for _ in range(2):  # the second round's reports are its own
        g.submit(1)
        with pytest.raises(OrionError, match="-6"):
            g.sync()
    for fs in members:
        with pytest.raises(OrionError, match="-6"):
            _poll(fs)
        assert len(_poll(fs)) == 0
    g.submit(0)
    g.sync()
    g.close()
    for fs in members:
        fs.close()
