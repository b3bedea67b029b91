"""Which form of a kernel a call takes, where only its time tells: the results of all forms are bitwise the same.

A form for few systems is several times faster than the one for full groups on a lone system, so a factor of 1.6
between two times of the same work separates them.
"""
import numpy as np
import pytest
import torch

import nbg
from conftest import has_gpu
from nbg import workloads as W

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA GPU")]


def lone(ctx, n, steps, grad=True):
    """The device times (total, orbit, transits, Jacobian) of one system of n bodies, the least of three calls."""
    els, hs, _ = W.batch_uneven(1, seed=40 + n, nmin=n, nmax=n)
    b = nbg.Batch([n], 0, hs, [hs[0] * steps], [steps], grad)
    best = None
    for _ in range(4):
        b.set_system(0, nbg.State(W.ic_of(els[0])), nbg.TransitTiming(hs[0] * steps, W.ic_of(els[0]), ntt=steps))
        b.run(ctx)
        t = np.array(ctx.last_timing())
        best = t if best is None else np.minimum(best, t)
    assert b.arrays["count"].sum() > 0
    return best


@pytest.mark.parametrize("n", [5, 8])
def test_few_searches_take_a_blocks_lanes_in_every_mode(n):
    """The searches of few systems are as fast with a one-lane or team producer as with the lanes one."""
    took = {}
    for mode in (0, 1, 2):
        ctx = nbg.Context(0)
        ctx.set_orbit_team(mode)
        ctx.set_profiling(1)
        took[mode] = lone(ctx, n, 120)[2]
        ctx.close()
    assert took[0] < 1.6 * took[2] and took[1] < 1.6 * took[2], took


def tuned(n, count, steps, trial_steps):
    """A context after autotuning on `count` systems of n bodies, and the report."""
    els, hs, _ = W.batch_uneven(count, seed=9, nmin=n, nmax=n)
    b = nbg.Batch([n] * count, 0, hs, [h * steps for h in hs], [steps // 10 + 4] * count, True)
    for q, (x, v, jac) in enumerate(nbg.init_nbody_batch([W.ic_of(el) for el in els])):
        b.view("x", q)[:], b.view("v", q)[:] = x.ravel(order="F"), v.ravel(order="F")
        b.view("m", q)[:] = els[q][:, 0]
        b.view("jac_init", q)[:] = jac.ravel(order="F")
        b.view("jac_step", q)[:: 7 * n + 1] = 1.0
    dev = {k: torch.from_numpy(a).cuda() for k, a in b.arrays.items()}
    ctx = nbg.Context(0)
    return ctx, b, dev, b.autotune_device(dev, ctx, trial_steps=trial_steps)


def test_a_lone_system_after_autotuning_takes_the_forms_for_few_systems():
    """Tuned on a full batch of four-body systems, where one lane a system is the fastest producer."""
    fresh = nbg.Context(0)
    before = lone(fresh, 8, 120)[0]
    fresh.close()
    ctx, _, _, report = tuned(4, 1500, 64, 16)
    assert report[0]["ms"] > 0
    after = lone(ctx, 8, 120)[0]
    ctx.close()
    assert after < 1.6 * before, (before, after, report[0])


def test_autotuner_tries_the_default_layout_and_producers_on_sms_of_their_own():
    ctx, b, dev, report = tuned(5, 64, 48, 8)
    tried = {(r["producer_warps"], r["producer_smem_kb"]) for r in report}
    ctx.close()
    assert tried == {(1, 0), (4, 200)}


def test_a_layout_for_full_groups_does_not_hold_up_the_forms_for_few_systems():
    """400 four-body systems: their blocks of the lanes form, each with an SM to itself, would run in three waves."""
    took = []
    for layout in ((1, 0, 0), (4, 200, 32)):
        ctx, b, dev, _ = tuned(4, 400, 64, 8)
        ctx.set_tuning(64)
        ctx.set_orbit_team(-1)
        ctx.set_producer_layout(*layout)
        best = []
        for _ in range(3):
            work = {k: t.clone() for k, t in dev.items()}
            torch.cuda.synchronize()  # the call runs on the library's own streams
            b.run_device(work, ctx)
            best.append(ctx.last_timing()[0])
        took.append(min(best))
        ctx.close()
    assert took[1] < 1.3 * took[0], took


def test_autotuner_trials_run_at_the_candidates_chunk():
    """The last trial, 128 steps at a chunk of 128, is one chunk: fewer launches than a call of 128 steps takes, which
    is cut into four chunks so that they overlap."""
    ctx, b, dev, report = tuned(3, 64, 128, 64)
    trial = ctx.last_launch_count()
    assert max(r["chunk_steps"] for r in report) == 128
    ctx.set_tuning(128)
    b.run_device(dev, ctx)
    call = ctx.last_launch_count()
    ctx.close()
    assert trial < call, (trial, call)


def test_a_short_call_without_overlap_is_one_chunk():
    """Chunks of a quarter of a short call's steps are for overlapping them: on one stream 64 steps stay one chunk."""
    count = {}
    for overlap in (0, 1):
        ctx = nbg.Context(0)
        ctx.set_tuning(64, overlap)
        lone(ctx, 3, 64)
        count[overlap] = ctx.last_launch_count()
        ctx.close()
    assert count[0] < count[1], count


@pytest.mark.parametrize("n, count, cut", [(3, 200, True), (4, 40, True), (4, 200, False), (6, 200, False)])
def test_short_calls_of_full_groups_keep_their_chunk(n, count, cut):
    """From four bodies on, where each search takes one lane and lasts as long whatever the chunk, 64 steps are one
    chunk, as without overlap; fewer bodies or few systems overlap in four."""
    els, hs, _ = W.batch_uneven(count, seed=3, nmin=n, nmax=n)
    b = nbg.Batch([n] * count, 0, hs, [h * 64 for h in hs], [10] * count, False)
    launches = {}
    for overlap in (0, 1):
        ctx = nbg.Context(0)
        ctx.set_tuning(64, overlap)
        for q, el in enumerate(els):
            b.set_system(q, nbg.State(W.ic_of(el)), nbg.TransitTiming(hs[q] * 64, W.ic_of(el), ntt=10))
        b.run(ctx)
        launches[overlap] = ctx.last_launch_count()
        ctx.close()
    assert (launches[0] < launches[1]) == cut, launches


def test_full_team_groups_on_sms_of_their_own():
    """A full team group's default layout, on SMs of its own, against one of two warps a block anywhere: the same bits,
    and not slower (1.15 for noise; without SMs of its own this takes half as long again)."""
    n, count, steps = 6, 1100, 256
    els, hs, _ = W.batch_uneven(count, seed=5, nmin=n, nmax=n)
    b = nbg.Batch([n] * count, 0, hs, [h * steps for h in hs], [steps // 10 + 4] * count, True)
    start = nbg.init_nbody_batch([W.ic_of(el) for el in els])
    got, took = [], []
    for layout in ((1, 0, 0), (2, 0, 0)):
        ctx = nbg.Context(0)
        ctx.set_producer_layout(*layout)
        times = []
        for _ in range(3):
            for k in b.arrays:
                b.arrays[k][...] = 0
            for q, (x, v, jac) in enumerate(start):
                b.view("x", q)[:], b.view("v", q)[:] = x.ravel(order="F"), v.ravel(order="F")
                b.view("m", q)[:] = els[q][:, 0]
                b.view("jac_init", q)[:] = jac.ravel(order="F")
                b.view("jac_step", q)[:: 7 * n + 1] = 1.0
            b.run(ctx)
            times.append(ctx.last_timing()[0])
        got.append({k: a.copy() for k, a in b.arrays.items()})
        took.append(min(times))
        ctx.close()
    for k in got[0]:
        np.testing.assert_array_equal(got[0][k], got[1][k], err_msg=k)
    assert took[0] < 1.15 * took[1], took
