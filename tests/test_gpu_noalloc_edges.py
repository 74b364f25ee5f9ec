"""The allocation-free call at the edges of its warps, tiles, chunks and of the
change to two rows per thread, from hardly any near pair to every pair near."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

from starsmasher_b200 import _lib, inputs

from conftest import err_report

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 33, 127, 129, 255, 257, 511, 513, 2049, 16383, 16384, 16385])
@pytest.mark.parametrize("width", [0.05, 1.0, 30.0])
def test_against_the_context_call(gpu_ctx, n, width):
    import torch
    s = inputs.single_polytrope(max(n, 66), 1.5, seed=n)
    a = [getattr(s, f)[:n].copy() for f in ("x", "y", "z", "m", "range2")]
    a[4] *= min(width, 30.0 if n <= 2049 else 3.0) ** 2
    if n > 4:
        a[4][2] = -a[4][2]  # a point mass; two coincident particles
        a[0][4], a[1][4], a[2][4] = a[0][3], a[1][3], a[2][3]
    nkernel = n % 3
    ref = gpu_ctx.forces(*a, nkernel, "fp64")
    X = [torch.from_numpy(v).cuda() for v in a]
    out = [torch.full((n,), float("nan"), dtype=torch.float64, device="cuda") for _ in range(4)]
    st = _lib.load().sphgrav_forces_fp64_noalloc(
        n, *(ctypes.c_void_p(t.data_ptr()) for t in X), nkernel,
        *(ctypes.c_void_p(t.data_ptr()) for t in out),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == _lib.OK
    got = [t.cpu().numpy() for t in out]
    if n == 1:
        assert got[0][0] == 0.0 and abs(got[3][0] - ref[3][0]) <= 1e-12 * abs(ref[3][0])
        return
    e = err_report(*got, *ref)
    assert e["acc_max"] <= 1e-12 and e["pot_max"] <= 1e-12, e
    if n > 4:
        assert np.isfinite(e["acc_max_ill"])


@pytest.mark.parametrize("n", [129, 300, 16400])
def test_separations_whose_square_overflows(n):
    """Two particles farther away than 1e154: no force and no potential, as 1/r underflows."""
    import torch
    s = inputs.single_polytrope(n, 1.5, seed=n)
    a = [getattr(s, f).copy() for f in ("x", "y", "z", "m", "range2")]
    a[4][-1] = -a[4][-1]  # no potential of its own

    def call(*a):
        k = len(a[0])
        X = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in a]
        out = [torch.zeros(k, dtype=torch.float64, device="cuda") for _ in range(4)]
        st = _lib.load().sphgrav_forces_fp64_noalloc(
            k, *(ctypes.c_void_p(t.data_ptr()) for t in X), 0,
            *(ctypes.c_void_p(t.data_ptr()) for t in out),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert st == _lib.OK
        return [t.cpu().numpy() for t in out]

    ref = call(*(v[1:-1] for v in a))
    a[0][-1], a[1][0] = 1e160, -1e200
    got = call(*a)
    e = err_report(*(v[1:-1] for v in got), *ref)
    assert e["acc_max"] <= 1e-12 and e["pot_max"] <= 1e-12, e
    assert all(v[-1] == 0.0 for v in got)


_CAPTURE = """
import ctypes, sys
import torch
from starsmasher_b200 import _lib, inputs
lib = _lib.load()
def call(n, X, out):
    assert lib.sphgrav_forces_fp64_noalloc(
        n, *(ctypes.c_void_p(t.data_ptr()) for t in X), 0, *(ctypes.c_void_p(t.data_ptr()) for t in out),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == _lib.OK
def model(n):
    s = inputs.single_polytrope(n, 1.5, seed=n)
    return ([torch.from_numpy(getattr(s, f)).cuda() for f in ("x", "y", "z", "m", "range2")],
            torch.zeros(4, n, dtype=torch.float64, device="cuda"))
first, then = (int(v) for v in sys.argv[1:])
X, out = model(first)
call(first, X, out)
torch.cuda.synchronize()
X, out = model(then)
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    call(then, X, out)
assert not out.any()
graph.replay()
torch.cuda.synchronize()
got = out.clone()
call(then, X, out)
torch.cuda.synchronize()
assert torch.equal(got, out) and bool((out[3] < 0).all())
"""


@pytest.mark.parametrize("first, then", [(100, 16384), (16384, 100), (16383, 40000)])
def test_capture_after_one_call_of_another_size(first, then):
    """In a process of its own: the first call of any size readies every size for a capture."""
    env = dict(os.environ, PYTHONPATH=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    r = subprocess.run([sys.executable, "-c", _CAPTURE, str(first), str(then)], env=env,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
