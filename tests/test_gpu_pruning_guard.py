"""The residual guard (correlation.cpp:521-528) and plane pruning.

A page without a report may leave out planes only where the FP32 error bound
says that no overlap count's residual can reach the guard of 0.25 anywhere.
Above that bound a residual has to be looked for on every legal plane, as a
page with a report does: both move the same bytes through pass A, and the
greedy's heads those of every plane."""

import ctypes
import math

import numpy as np
import pytest

from conftest import package

pytestmark = pytest.mark.gpu


def _pass_a_bytes(ctx, call):
    lib = package("compute").lib()
    lib.spk_context_set_profiling.argtypes = [ctypes.c_void_p, ctypes.c_int]
    lib.spk_context_pass_bytes.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint32]
    out = np.zeros(1, np.float64)
    lib.spk_context_set_profiling(ctx.handle, 1)
    result = call()
    lib.spk_context_pass_bytes(ctx.handle, out.ctypes.data, 1)
    lib.spk_context_set_profiling(ctx.handle, 0)
    return float(out[0]), result


def _bound(s):
    """2^-14 log2(N) rms sqrt(cells), with the largest plane's rms."""
    env = s.field("occupancy").astype(np.float64), s.field("proximity")
    depth = s.environment_shape[2]
    norm = max(sum(float((f ** 2).sum()) for f in plane) for plane in zip(*(e.reshape(depth, -1) for e in env)))
    rms = math.sqrt(norm / (s.fft_shape[0] * s.fft_shape[1]))
    cells = min(int(s.field("kernel", o).sum()) for o in range(len(s.catalog)))
    return 2.0 ** -14 * math.log2(math.prod(s.fft_shape)) * rms * math.sqrt(cells)


@pytest.mark.parametrize("radius,guarded", [((20.0, 23.0), False), ((5.0, 7.0), True)])
def test_planes_are_left_out_only_under_the_bound(gpu_ctx, radius, guarded):
    assets, geometry, session_mod, synthetic = (package(n) for n in ("assets", "geometry", "session", "synthetic"))
    item = assets.accept_stl(synthetic.blob_stl(3, level=3, radius_range=radius))
    s = session_mod.Session(item, (126.0, 126.0, 126.0), (0.0, 0.0, 0.0), 1.0, geometry.hopf_catalog(4, 4),
                            context=gpu_ctx)
    s.pages([0])  # the layout is up to date
    bound = _bound(s)
    assert (bound < 0.25) == guarded and bound < 1.0
    reports = []
    every, whole = _pass_a_bytes(gpu_ctx, lambda: s.pages(range(4), reports=reports))
    some, pruned = _pass_a_bytes(gpu_ctx, lambda: s.pages(range(4)))
    heads, _ = _pass_a_bytes(gpu_ctx, lambda: s.greedy(1))
    # One slab over the window: its planes once, and per orientation its kernel's
    # planes and its legal ones (whole pages may add threshold passes to that).
    depth, (lx, ly, _) = s.environment_shape[2], s.fft_shape
    all_planes = 8 * lx * ly * (depth + 4 * (depth + 1))
    s.close()
    assert max(r["max_integer_residual"] for r in reports) < 0.25
    assert pruned == whole
    if guarded:
        assert some < every and heads < all_planes
    else:
        assert some == every and heads == all_planes
