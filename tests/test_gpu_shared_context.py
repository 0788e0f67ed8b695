"""Calls that share a context with an open session leave its state alone: a
proximity field whose table is larger than the session's, and stateless pages
over larger and smaller windows, between the session's own calls."""

import numpy as np
import pytest

from conftest import package
from scenes import scene

pytestmark = pytest.mark.gpu


def _other_calls(ctx, seed, shape, kernel):
    compute, pl = package("compute"), package("pipeline")
    sc = scene(seed, shape=shape, kernel_shape=kernel, blobs=5)
    page = pl.spectral_page(
        pl.PageScene(sc["env_first"], sc["env_shape"], sc["lattice"][:3], sc["lattice"][3], sc["cmin_z"],
                     sc["height"]),
        sc["occ"], sc["kernel_first"], sc["kernel_shape"], sc["kernel"], sc["max_z"], context=ctx)
    return page, compute.build_proximity(sc["env_shape"], sc["occ"], context=ctx)


def _fill(ctx, between):
    """A session's pages and placements, with other calls between its own."""
    assets, geometry, session_mod, synthetic = (package(n) for n in ("assets", "geometry", "session", "synthetic"))
    item = assets.accept_stl(synthetic.blob_stl(5, level=3, radius_range=(4.0, 6.0)))
    s = session_mod.Session(item, (40.0, 36.0, 30.0), (0.0, 0.0, 0.0), 1.0, geometry.hopf_catalog(8, 5), context=ctx)
    out, others = [], []

    def step(call):
        out.append(call())
        if between:
            others.append((_other_calls(ctx, 1, (72, 60, 50), (9, 7, 8)), _other_calls(ctx, 2, (24, 20, 18), (5, 4, 6))))

    step(lambda: s.pages(range(8)))
    for _ in range(2):
        step(lambda: [(p.orientation_index, p.translation, p.score) for p in s.greedy(1)])
    step(lambda: s.place(3, (14, 15, 12)))
    step(lambda: s.pages(range(8)))
    step(s.remove_last)
    step(lambda: [(p.orientation_index, p.translation, p.score) for p in s.greedy(2)])
    s.close()
    return out, others


def test_other_calls_leave_an_open_session_alone():
    compute = package("compute")
    with compute.Context(0) as ctx:
        alone, _ = _fill(ctx, False)
    with compute.Context(0) as ctx:
        shared, others = _fill(ctx, True)
    assert shared == alone
    with compute.Context(0) as ctx:
        want = _other_calls(ctx, 1, (72, 60, 50), (9, 7, 8)), _other_calls(ctx, 2, (24, 20, 18), (5, 4, 6))
    for got in others:
        for (page, field), (want_page, want_field) in zip(got, want):
            assert page == want_page
            assert np.array_equal(np.asarray(field), np.asarray(want_field))
