"""The status words of batches, and the digits of x, v and the transit times that they hang on.

NBG_STATUS_NEWTON_ITMAX says that a transit search's iterates did not repeat within 20, and which searches those are
follows the last digit of the state they start from.  The words are whole numbers that a caller may keep beside his
results, so a change of the kernels leaves them as they are: transit_status.npz holds the inputs of nine batches
and, from the kernels that round x and v operation by operation as the reference's expressions do, each system's status
word and transit counts, and the bits of x, v and tt folded by exclusive or.  Every form of the kernels has to return
them, with derivatives and without: bitwise, no tolerance.

The batches: near-resonant three-body and compact eight-body systems (15 and 2 of which are flagged), mixed body counts
and lengths, kicks between planets, for one pair and for all, steps of a fifth of the shortest period (half angles over
pi/4, the closed forms of G3, H1, H2), two planets without mass, and eccentricities of 0.6 to 0.9.
"""
import os

import numpy as np
import pytest

import nbg
from conftest import has_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA GPU")]

GOLD = np.load(os.path.join(os.path.dirname(os.path.abspath(__file__)), "transit_status.npz"))
NAMES = sorted({k.split(".")[0] for k in GOLD.files})


def folded(a):
    return np.bitwise_xor.reduce(np.ascontiguousarray(a).view(np.uint64))


def run(name, grad, mode):
    get = lambda k: GOLD["%s.%s" % (name, k)]  # noqa: E731
    n, steps = [int(q) for q in get("n")], [int(q) for q in get("steps")]
    b = nbg.Batch(n, 0, list(get("h")), [float(h) * k for h, k in zip(get("h"), steps)], [k // 4 + 8 for k in steps], grad)
    for k in ("x", "v", "m", "pair"):
        b.arrays[k][...] = get(k)
    for q, bodies in enumerate(n):
        b.view("jac_init", q)[:: 7 * bodies + 1] = 1.0
        b.view("jac_step", q)[:: 7 * bodies + 1] = 1.0
    ctx = nbg.Context(0)
    ctx.set_orbit_team(mode)
    b.run(ctx)
    ctx.close()
    return b


@pytest.mark.parametrize("mode", [-1, 0, 1, 2])
@pytest.mark.parametrize("name", NAMES)
def test_status_and_digits(name, mode):
    for grad in (False, True):
        b = run(name, grad, mode)
        assert np.array_equal(b.status, GOLD[name + ".status"]), np.flatnonzero(b.status != GOLD[name + ".status"])
        assert np.array_equal(b.arrays["count"], GOLD[name + ".count"])
        for k, kept in (("x", "x_end"), ("v", "v_end"), ("tt", "tt")):
            got = np.array([folded(b.view(k, q)) for q in range(b.nsys)])
            assert np.array_equal(got, GOLD["%s.%s" % (name, kept)]), (grad, k)
