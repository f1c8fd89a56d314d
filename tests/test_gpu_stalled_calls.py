"""The calls around a solve that stalls, that is, needs more pressure passes than the step's graph runs (Solver::settle):
each leaves the cavity where the same steps leave one that runs kernel by kernel (CAVITY_GRAPHS=0), whose refinement loop
the host drives anyway.  Two forms stall in their first step: the tensor-core transforms (two passes a solve) above 2^18
cells, where the projection starts in two launches, and the FP64 ones (one pass) in one launch."""
import time

import numpy as np
import pytest

from les_impulse3d_64_b200 import workloads
from les_impulse3d_64_b200.api import Batch, Cavity

pytestmark = pytest.mark.gpu
FIELDS = ('u', 'v', 'w', 'mx', 'my', 'mz', 'phi')
# precision, CAVITY_FDM, passes a solve that the graph runs, cells along x and y, along z, tolerance
FORMS = {'tc': ('mixed', 'tc', 2, 72, 64, 1e-14), 'fp64': ('fp64', '', 1, 64, 64, 3e-15)}


def make(form, monkeypatch, eager=False, seed=5, **changes):
    precision, fdm, _, n, nz, rtol = FORMS[form]
    monkeypatch.setenv('CAVITY_FDM', fdm)
    if eager:
        monkeypatch.setenv('CAVITY_GRAPHS', '0')
    s = workloads.settings(n, 400.0, nz=nz, beta=1.5, cfl=0.5, **{'fdm_rtol': rtol, **changes})
    cav = Cavity(s, precision=precision)
    monkeypatch.delenv('CAVITY_GRAPHS', raising=False)
    cav.initialize(*workloads.initial_noise(cav.shapes, 1e-2, seed))
    return cav


def stalling_step(cav, form):
    """One step of a kernel-by-kernel cavity; its solves take more passes than the graph of a step runs."""
    before = cav.pressure_passes()
    cav.step()
    assert cav.pressure_passes() - before > 3 * FORMS[form][2]


def assert_same(a, b):
    assert a.report() == b.report()
    for k in FIELDS:
        assert np.array_equal(a.field(k), b.field(k)), k


@pytest.mark.parametrize('form', FORMS)
def test_queued_outputs(form, monkeypatch):
    """Steps queued with their outputs, the first of which stalls, and a batch's: the same state, probes, statistics and
    passes as step by step (the batch's fields to 1e-6: its sums group their terms by other blocks)."""
    queued, member, eager = (make(form, monkeypatch, eager=e) for e in (False, False, True))
    batch = Batch([member])
    try:
        queued.step_outputs_async(4, statistics=True)
        report, values = queued.sync_outputs()
        batch.step_async(4)
        batched = batch.sync()[0]
        stalling_step(eager, form)
        eager.add_statistics(eager.report()['dt'])
        passes, probes = [eager.report()['phi_passes']], [eager.probes()]
        for _ in range(3):
            passes.append(eager.step()['phi_passes'])
            probes.append(eager.probes())
            eager.add_statistics(eager.report()['dt'])
        assert form != 'tc' or passes[0] > 2              # more than its graph runs
        assert report == eager.report() and batched['steps'] == 4
        assert queued.pressure_passes() == eager.pressure_passes()
        assert np.array_equal(values, np.array(probes))
        assert np.array_equal(queued.statistics(), eager.statistics())
        assert_same(queued, eager)
        for k in FIELDS:
            x, y = member.field(k), eager.field(k)
            assert np.abs(x - y).max() <= 1e-6 * np.abs(y).max(), k
    finally:
        batch.close()
        for cav in (queued, member, eager):
            cav.close()


@pytest.mark.parametrize('form', FORMS)
def test_time_steps(form, monkeypatch):
    """The first timed step stalls: the steps go on, and its time runs to the end of the host's part."""
    timed, eager = make(form, monkeypatch), make(form, monkeypatch, eager=True)
    try:
        ms, kms = timed.time_steps(0, 3, flush_l2=False)
        stalling_step(eager, form)
        for _ in range(5):
            eager.step()
        assert_same(timed, eager)
        assert ms[0] > 0.8 * ms[1:].min() > 0 and kms.min() > 0
        times = timed.kernel_times()
        assert all(times[k] > 0 for k in ('sweep', 'projection_start', 'finish', 'transforms'))
    finally:
        timed.close()
        eager.close()


@pytest.mark.parametrize('form', FORMS)
def test_autotune(form, monkeypatch):
    """Stalls under the tuner's candidates: none is thrown out or timed over an aborted step, the state comes back, and the
    tuned cavity steps on as an untuned one (the sweep kernel is fixed: the other choices are bit for bit the same)."""
    monkeypatch.setenv('CAVITY_SWEEP', 'tile')
    tuned, eager = make(form, monkeypatch), make(form, monkeypatch, eager=True)
    try:
        report = tuned.report()
        chunks, tile, fused, ms = tuned.autotune(steps=3)
        assert tuned.report() == report
        stalling_step(eager, form)
        assert tuned.step() == eager.report()
        for _ in range(3):
            assert tuned.step() == eager.step()
        assert_same(tuned, eager)
        assert chunks == 0 and ms > 0.8 * float(tuned.time_steps(2, 8, flush_l2=False)[0].min())
    finally:
        tuned.close()
        eager.close()


def test_part_times(monkeypatch):
    """A batch's parts: the first pass is one pass of the two that a tensor-core graph runs, also on stalling steps, and
    the steps are ordinary ones.  Its transforms and residual are those that a cavity alone times (within a half)."""
    member, alone = make('tc', monkeypatch), make('tc', monkeypatch)
    batch = Batch([member])
    try:
        first, second = batch.part_times(2), batch.part_times(2)
        alone.time_steps(0, 2, flush_l2=False)
        times = alone.kernel_times()
        one_pass = times['transforms'] + times['guess_residual']
        for parts in (first, second):
            assert 0.5 * one_pass < parts['first_pass'] < 1.5 * one_pass
        assert all(first[k] > 0.5 * second[k] for k in first)
        assert member.report()['steps'] == alone.report()['steps'] == 4
        for k in FIELDS:           # the sums of a batch group their terms by other blocks (1e-6 of the FP32 fields)
            x, y = member.field(k), alone.field(k)
            assert np.abs(x - y).max() <= 1e-6 * np.abs(y).max(), k
    finally:
        batch.close()
        member.close()
        alone.close()


def test_reading_a_member_before_the_batch_waits(monkeypatch):
    """A member's getters and its own wait finish its batch's queued steps first, also one that stalls."""
    a, b = make('tc', monkeypatch), make('tc', monkeypatch)
    batch = Batch([a, b])
    try:
        batch.step_async(3)
        early = a.field('u')
        assert b.sync()['steps'] == 3
        assert [r['steps'] for r in batch.sync()] == [3, 3]
        assert np.array_equal(early, a.field('u'))
        for k in FIELDS:
            assert np.array_equal(a.field(k), b.field(k)), k
        batch.step_async(2)
        assert [r['steps'] for r in batch.sync()] == [5, 5]
    finally:
        batch.close()
        a.close()
        b.close()


@pytest.mark.parametrize('form', FORMS)
def test_set_clock_while_steps_are_queued(form, monkeypatch):
    """The clock is set after the queued steps, the stalled one among them, and the wait reports it."""
    queued, eager = make(form, monkeypatch), make(form, monkeypatch, eager=True)
    try:
        queued.step_async(3)
        queued.set_clock(7.0, 100, 2e-3)
        report = queued.sync()
        assert (report['time'], report['steps'], report['dt']) == (7.0, 100, 2e-3)
        stalling_step(eager, form)
        for _ in range(2):
            eager.step()
        eager.set_clock(7.0, 100, 2e-3)
        assert_same(queued, eager)
        queued.step_async(2)
        queued.sync()
        for _ in range(2):
            eager.step()
        assert_same(queued, eager)
    finally:
        queued.close()
        eager.close()


@pytest.mark.parametrize('form', FORMS)
def test_initialize_while_steps_are_queued(form, monkeypatch):
    """The steps queued before belong to the old state: a stall among those queued after is not taken for one of them."""
    queued, eager = make(form, monkeypatch), make(form, monkeypatch, eager=True)
    try:
        queued.step_async(1)
        for cav in (queued, eager):
            cav.initialize(*workloads.initial_noise(cav.shapes, 2e-2, 9))
        queued.step_async(2)
        queued.sync()
        stalling_step(eager, form)
        eager.step()
        assert_same(queued, eager)
    finally:
        queued.close()
        eager.close()


def test_failing_step_queued_behind_a_stall(monkeypatch):
    """The first queued step stalls, the third does not converge: the wait says so as kernel-by-kernel steps do, and both
    cavities stand at the second step's state, probes and statistics included."""
    queued, eager = (make('fp64', monkeypatch, eager=e, fdm_rtol=1e-15) for e in (False, True))
    try:
        queued.step_outputs_async(4, statistics=True)
        with pytest.raises(RuntimeError, match='residual .* > FDM_RTOL after 8 passes') as error:
            queued.sync_outputs()
        for _ in range(2):
            eager.step_outputs_async(1, statistics=True)
            eager.sync_outputs()
        with pytest.raises(RuntimeError) as same:
            eager.step()
        assert str(error.value) == str(same.value)
        assert_same(queued, eager)
        assert np.array_equal(queued.probes(), eager.probes())
        assert np.array_equal(queued.statistics(), eager.statistics())
    finally:
        queued.close()
        eager.close()


def test_graphs_without_loops_return(monkeypatch):
    """A cavity of 32 x 32 x 8 cells that stalls in its first step only: 100 steps later its steps take as long as those of
    one that never does (measured, us: with the refinement loops 154, without 121)."""
    monkeypatch.setenv('CAVITY_FDM', '')
    fastest = {}
    for rtol in (3e-15, 1e-9):
        cav = Cavity(workloads.settings(32, 400.0, nz=8, beta=1.5, cfl=0.5, fdm_rtol=rtol))
        try:
            cav.initialize(*workloads.initial_noise(cav.shapes, 1e-2, 5))
            before = cav.pressure_passes()
            cav.step()
            assert (cav.pressure_passes() - before > 3) == (rtol < 1e-9)
            cav.step_async(100)
            cav.sync()
            fastest[rtol] = float(cav.time_steps(2, 40, flush_l2=False)[0].min())
        finally:
            cav.close()
    assert fastest[3e-15] < 1.12 * fastest[1e-9], fastest


def test_batch_follows_its_members(monkeypatch):
    """A batch runs graphs with refinement loops while it holds a cavity that stalled, and others once that one has left its
    slot: then its steps take as long as a batch's that never held it, and the other member's are the same throughout."""
    monkeypatch.setenv('CAVITY_FDM', '')

    def cavity(rtol, seed):
        cav = Cavity(workloads.settings(32, 400.0, nz=8, beta=1.5, cfl=0.5, fdm_rtol=rtol))
        cav.initialize(*workloads.initial_noise(cav.shapes, 1e-2, seed))
        return cav

    def seconds(batch):
        t = []
        for _ in range(6):
            t0 = time.perf_counter()
            batch.step_async(40)
            batch.sync()
            t.append(time.perf_counter() - t0)
        return min(t)

    stalls, member, alone = cavity(3e-15, 5), cavity(1e-9, 6), cavity(1e-9, 6)
    batch, calm = Batch([stalls, member]), Batch([alone], capacity=2)
    try:
        before = stalls.pressure_passes()
        for b in (batch, calm):
            for _ in range(2):
                b.step_async(1)
                b.sync()
        assert stalls.pressure_passes() - before > 2 * 3
        batch.set_member(0, None)
        after, never = seconds(batch), seconds(calm)
        batch.set_member(0, stalls)
        for b in (batch, calm):
            b.step_async(2)
            b.sync()
        assert_same(member, alone)
        assert stalls.report()['steps'] == 4
        assert after < 1.12 * never
    finally:
        batch.close()
        calm.close()
        for cav in (stalls, member, alone):
            cav.close()


def test_time_steps_behind_queued_steps(monkeypatch):
    """Steps that do not stall are queued, with their tail, when the timing begins: the wait reads the control block after
    the timed step, not the tail's earlier copy."""
    cav, eager = (make('fp64', monkeypatch, eager=e, fdm_rtol=1e-9) for e in (False, True))
    try:
        cav.step_async(2)
        ms = np.zeros(1, dtype=np.float32)
        cav._call('cavity_time_steps', cav.handle, 0, 1, 0, ms.ctypes.data, None)
        for _ in range(3):
            eager.step()
        assert_same(cav, eager)
    finally:
        cav.close()
        eager.close()


def test_set_field_while_steps_are_queued(monkeypatch):
    """A field set behind queued steps clears the potential's history for good: the wait, and a clock set after it, do not
    bring the steps' back."""
    queued, eager = (make('fp64', monkeypatch, eager=e, fdm_rtol=1e-9) for e in (False, True))
    try:
        queued.step_async(3)
        for _ in range(3):
            eager.step()
        u = 0.9 * eager.field('u')
        for cav in (queued, eager):
            cav.set_field('u', u)
        r = queued.sync()
        for cav in (queued, eager):
            cav.set_clock(r['time'], r['steps'], r['dt'])
            for _ in range(2):
                cav.step()
        assert_same(queued, eager)
    finally:
        queued.close()
        eager.close()
