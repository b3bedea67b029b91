"""A batched call from host arrays refuses a null array, input or output, and leaves the others as they were."""
import numpy as np
import pytest

import nbg
from conftest import has_gpu
from nbg import _lib
from nbg import workloads as W

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a CUDA GPU")]

NAMES = ["t", "x", "v", "m", "xerror", "verror", "jac_step", "jac_error", "dqdt", "pair", "jac_init", "tt", "dtdq0",
         "dtdelements", "count"]


@pytest.mark.parametrize("null", NAMES)
def test_null_array_is_refused(null):
    els, h, _ = W.batch_3body(1, 7)
    ic = W.ic_of(els[0])
    b = nbg.Batch([3], 0, [h], [20 * h], [8], True)
    b.set_system(0, nbg.State(ic), nbg.TransitTiming(20 * h, ic, ntt=8))
    before = {k: a.copy() for k, a in b.arrays.items()}
    ctype = {"pair": _lib._U8, "count": _lib._I64}
    ptr = [None if k == null else _lib.ptr(b.arrays[k], ctype.get(k, _lib._D)) for k in NAMES]
    rc = _lib.load().nbg_batch_integrate_transits(nbg.default_context().handle, 1, b.descriptors(), *ptr, None)
    assert rc == _lib.NBG_EINVAL
    for k, a in before.items():
        np.testing.assert_array_equal(b.arrays[k], a)
