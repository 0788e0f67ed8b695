"""A correlation that is refused after its work was queued (here by the
context's memory cap, at the mask's buffer) returns with nothing in flight: its
inputs are copied from the context's pinned buffer, which the next call
overwrites.  A cap that holds two transform grids, the inputs and the outputs
refuses nothing: the checks' bookkeeping lies outside it."""

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


@pytest.mark.parametrize("es,ks,grid", [((12, 10, 11), (4, 3, 5), (15, 12, 15)), ((20, 24, 22), (5, 6, 4), (24, 30, 25)),
                                        ((1, 1, 1), (1, 1, 1), (2, 2, 2))])
@pytest.mark.parametrize("precision", ["FP64", "FP32"])
def test_a_cap_of_two_grids_inputs_and_outputs_suffices(es, ks, grid, precision):
    compute = package("compute")
    rng = np.random.default_rng(5)
    env = (rng.random(int(np.prod(es))) < 0.2).astype(np.uint8)
    ker = np.ones(int(np.prod(ks)), np.uint8)
    cells = int(np.prod([e + k - 1 for e, k in zip(es, ks)]))
    cap = 2 * int(np.prod(grid)) * (16 if precision == "FP64" else 8) + env.size + ker.size + 8 * cells
    # Per-block sums of the outputs' checks: 24 bytes for each 256 of them.
    cap += 24 * -(-cells // 256) + 32
    with compute.Context(0, cap) as ctx:
        got = compute.correlate_binary(compute.CorrelationSpec(es, ks), env, ker, precision=getattr(compute, precision),
                                       context=ctx)
        assert not isinstance(got, compute.CorrelationFailure), got
