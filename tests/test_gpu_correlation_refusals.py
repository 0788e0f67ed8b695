"""A correlation that is refused after its work was queued (here by the
context's memory cap, at the mask's buffer) returns with nothing in flight: its
inputs are copied from the context's pinned buffer, which the next call
overwrites."""

import ctypes

import numpy as np
import pytest

from conftest import package

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["FP64", "FP32"])
def test_refused_call_leaves_nothing_in_flight(precision):
    torch = pytest.importorskip("torch")
    compute = package("compute")
    rng = np.random.default_rng(4)
    es, ks = (40, 36, 30), (7, 6, 5)
    env = (rng.random(int(np.prod(es))) < 0.02).astype(np.uint8)
    ker = np.ones(int(np.prod(ks)), np.uint8)
    spec, bits = compute.CorrelationSpec(es, ks), getattr(compute, precision)
    limits = compute.CorrelationLimits(max_working_bytes=4 << 30)
    legal = tuple(e - k + 1 for e, k in zip(es, ks))

    def mask(ctx, box):
        return compute.correlate_binary_mask(spec, env, ker, (0, 0, 0), box, compute.MASK_ZERO, limits=limits,
                                             precision=bits, context=ctx)

    lib = compute.lib()
    lib.spk_context_stream.restype = ctypes.c_void_p
    lib.spk_context_stream.argtypes = [ctypes.c_void_p]
    with compute.Context(0) as ctx:
        want = mask(ctx, legal).mask
    with compute.Context(0, 64 << 20) as ctx:
        stream = torch.cuda.ExternalStream(lib.spk_context_stream(ctx.handle))
        assert stream.query()
        for _ in range(3):
            refused = mask(ctx, (512, 512, 512))  # 134 MB of mask
            idle = stream.query()
            assert refused.code == "CORRELATION_MEMORY_LIMIT"
            assert idle
            assert np.array_equal(mask(ctx, legal).mask, want)
