"""The latency-bound and the throughput-bound forms of the kernels against each other and the oracle.

A batch's chunk runs in one of several forms by its size: the orbit producer and the transit searches with one
lane or a block's lanes a system, the Jacobian consumer with one or six lanes a column.  Every form does the same
operations in the same order, so their results are bitwise the same (no tolerance); mode 0 is one lane throughout,
2 the wide forms throughout, 1 the level-parallel team, -1 the automatic choice.
"""
import numpy as np
import pytest
import torch

import nbg
import oracle_lib as O
import parity as P
from conftest import has_gpu
from nbg import workloads as W

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA GPU")]

OUT = ("x", "v", "xerror", "verror", "tt", "count", "jac_step", "jac_error", "dqdt", "dtdq0", "dtdelements")


def systems(n, count, kick=None, massless=()):
    els, hs, _ = W.batch_uneven(count, seed=300 + n, nmin=n, nmax=n)
    states = []
    for el in els:
        s = nbg.State(W.ic_of(el))
        if kick is not None:
            s.pair[...] = kick
        for b in massless:
            s.m[b] = 0.0
        states.append(s)
    return states, hs


def run(states, hs, steps, mode, grad=True, ntt=8, layout=None):
    ctx = nbg.Context(0)
    ctx.set_orbit_team(mode)
    if layout:
        ctx.set_producer_layout(*layout)
    b = nbg.Batch([s.n for s in states], 0, list(hs), [h * steps for h in hs], [ntt] * len(states), grad)
    for q, s in enumerate(states):
        b.set_system(q, s)
    b.run(ctx)
    ctx.close()
    return b


def same(a, b):
    for k in OUT:
        assert np.array_equal(a.arrays[k], b.arrays[k], equal_nan=True), k
    assert np.array_equal(a.status, b.status)


def kicks(n, which):
    p = np.zeros((n, n), dtype=np.uint8, order="F")
    if which == "planets":
        p[1:, 1:] = 1
    elif which == "one":
        p[0, 1] = p[1, 0] = 1
    elif which == "all":
        p[...] = 1
    return p


# steps around a chunk's (a quarter of a short run's, 16) and a tile's ends; 3 and 5 systems: an odd one out
# where two share a warp
@pytest.mark.parametrize("n, count, steps", [(2, 1, 1), (2, 3, 65), (3, 5, 3), (3, 2, 64), (4, 3, 17), (5, 2, 63),
                                             (6, 1, 16), (7, 3, 4), (8, 2, 33), (9, 1, 5), (10, 2, 15)])
@pytest.mark.parametrize("which", ["none", "planets", "one", "all"])
def test_forms_agree_bitwise(n, count, steps, which):
    states, hs = systems(n, count, kicks(n, which))
    ref = run(states, hs, steps, 0)
    assert np.all(np.isfinite(ref.arrays["jac_step"]))
    for mode in (1, 2, 3, -1):
        same(ref, run(states, hs, steps, mode))
    plain = run(states, hs, steps, 0, grad=False)
    for mode in (2, -1):
        wide = run(states, hs, steps, mode, grad=False)
        for k in ("x", "v", "xerror", "verror", "tt", "count"):
            assert np.array_equal(plain.arrays[k], wide.arrays[k]), k
            assert np.array_equal(plain.arrays[k], ref.arrays[k]), k


@pytest.mark.parametrize("n, massless", [(3, (1, 2)), (3, (0, 1)), (5, (2, 4)), (5, (0, 1, 2, 3, 4))])
def test_forms_agree_on_pairs_without_mass(n, massless):
    states, hs = systems(n, 3, massless=massless)
    ref = run(states, hs, 20, 0)
    for mode in (1, 2, -1):
        b = run(states, hs, 20, mode)
        for k in OUT:
            assert np.array_equal(ref.arrays[k], b.arrays[k], equal_nan=True), k


@pytest.mark.parametrize("n, systems_per_sm", [(2, 96 / 14), (3, 96 / 21), (4, 96 / 28), (6, 64 / 42), (8, 64 / 56),
                                               (8, 64 / 13), (10, 64 / 17)])
@pytest.mark.parametrize("beside", [0, 1])
def test_sizes_where_the_form_changes(n, systems_per_sm, beside):
    """The last size of a wide form and the first beyond it; systems also as in a small call (staged copies)."""
    count = int(systems_per_sm * torch.cuda.get_device_properties(0).multi_processor_count) + beside
    few, hs = systems(n, 5)
    small = run(few, hs, 18, 0)
    full = run([few[q % 5] for q in range(count)], [hs[q % 5] for q in range(count)], 18, -1)
    for k in OUT:
        for q in (0, 1, 2, 3, 4, count - 1):
            assert np.array_equal(full.view(k, q), small.view(k, q % 5)), (k, q)


@pytest.mark.parametrize("count", [1023, 1024, 2051])
def test_full_group_of_one_lane_producers(count):
    """From 1024 systems on, with derivatives, the one-lane producer takes three warps a block."""
    few, hs = systems(3, 7)
    states, hh = [few[q % 7] for q in range(count)], [hs[q % 7] for q in range(count)]
    same(run(states, hh, 9, -1, ntt=2), run(states, hh, 9, 0, ntt=2, layout=(1, 0, 0)))


# h in inner periods: below, around and beyond the eighth of a period where the half-angle iteration takes over
@pytest.mark.parametrize("share", [0.05, 0.11, 0.13, 0.2, 0.3])
@pytest.mark.parametrize("n", [3, 5])
def test_long_steps_match_the_oracle(n, share):
    els, _, _ = W.batch_uneven(1, seed=400 + n, nmin=n, nmax=n)
    el = els[0]
    h = share * float(el[1, 1])
    s = nbg.State(W.ic_of(el))
    so = O.OState(s.x.copy(order="F"), s.v.copy(order="F"), s.m, jac_init=s.jac_init.copy(order="F"), t=0.0)
    O.integrate_nsteps(so, h, 12)
    outs = [run([s], [h], 12, mode) for mode in (0, 2)]
    same(*outs)
    got = type("S", (), {})()
    got.x = outs[0].view("x", 0).reshape((3, n), order="F")
    got.v = outs[0].view("v", 0).reshape((3, n), order="F")
    got.jac_step = outs[0].view("jac_step", 0).reshape((7 * n, 7 * n), order="F")
    got.dqdt = outs[0].view("dqdt", 0)
    P.check_state(got, so)


def test_initial_conditions_packed_and_alone():
    els = [W.batch_uneven(1, seed=500 + n, nmin=n, nmax=n)[0][0] for n in (2, 5, 3, 10, 3)]
    ics = [W.ic_of(el) for el in els]
    for got, ic in zip(nbg.init_nbody_batch(ics), ics):
        for a, b in zip(got, nbg.init_nbody_batch([ic])[0]):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("n", [2, 3, 5, 8])
@pytest.mark.parametrize("grad", [True, False])
def test_search_forms_agree_on_transit_parameters(n, grad):
    """The three adjoint rows of a search on one lane and on a block's lanes."""
    els, hs, _ = W.batch_uneven(1, seed=600 + n, nmin=n, nmax=n)
    h, tmax = hs[0], 70 * hs[0]
    ctx, out = nbg.default_context(), []
    try:
        for mode in (0, 2):
            ctx.set_orbit_team(mode)
            ic = W.ic_of(els[0])
            s, tp = nbg.State(ic), nbg.TransitParameters(tmax, ic)
            nbg.Integrator(nbg.ahl21, h, 0.0, tmax)(s, tp, grad=grad)
            out.append((s, tp))
    finally:
        ctx.set_orbit_team(-1)
    (s0, a), (s1, b) = out
    assert a.count.sum() > 0 and np.array_equal(a.count, b.count)
    assert np.array_equal(s0.x, s1.x) and np.array_equal(a.ttbv, b.ttbv)
    if grad:
        assert np.array_equal(a.dtbvdq0, b.dtbvdq0) and np.array_equal(a.dtbvdelements, b.dtbvdelements)
