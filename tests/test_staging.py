"""The page-locked staging memory a context keeps (csrc/nbg_staging.hpp), host only: a C++ check with an allocator that
counts and can refuse.  The memory stays under its limit whatever a call asks for, and a refusal is no error: the call
then gathers its arrays in pageable memory."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import nbg
from conftest import has_gpu
from nbg import workloads as W

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "nbodygradient.jl_gb300", "csrc")


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_staging_block_is_bounded_and_survives_a_refusal(tmp_path):
    exe = str(tmp_path / "staging_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", CSRC, os.path.join(HERE, "native", "staging_check.cpp"),
                    "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout


@pytest.mark.gpu
@pytest.mark.skipif(not has_gpu(), reason="needs a CUDA GPU")
def test_a_plan_over_the_limit():
    """45 000 copies of a two-body system: over 4 MiB of offsets and scalars, gathered in pageable memory."""
    count, (els, hs, _) = 45000, W.batch_uneven(1, seed=3, nmin=2, nmax=2)
    ctx = nbg.Context(0)
    out = []
    for n in (1, count):
        b = nbg.Batch([2] * n, 0, hs * n, [3 * hs[0]] * n, [1] * n, False)
        s = nbg.State(W.ic_of(els[0]))
        for k in ("x", "v", "m"):
            b.arrays[k][...] = np.tile(getattr(s, k).ravel(order="F"), n)
        b.run(ctx)
        out.append(b)
    ctx.close()
    for k in ("t", "x", "v"):
        assert np.array_equal(out[1].arrays[k], np.tile(out[0].arrays[k], count)), k
    assert not out[1].status.any()
