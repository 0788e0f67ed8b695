"""Sessions under a device-memory cap.

Opening takes orientations in batches.  A batch is bounded by its cells, not
only by its mesh, and shrinks to one orientation at a time where the context may
not have more.  The caps leave a third to a half more than opening one
orientation at a time takes, and the same again for the fill."""

import pytest

from conftest import package

pytestmark = pytest.mark.gpu

# item, box, orientations, cap of the open and of the fill in MB
SCENES = [((40.0, 50.0, 44.0), 94.0, 64, 33, 66), ((9.0, 12.0, 15.0), 64.0, 24, 15, 28)]


@pytest.mark.parametrize("item,box,orientations,open_mb,fill_mb", SCENES)
def test_capped_sessions_open_and_fill_like_uncapped_ones(item, box, orientations, open_mb, fill_mb):
    assets, compute, geometry, session_mod, synthetic = (
        package(n) for n in ("assets", "compute", "geometry", "session", "synthetic"))
    mesh = assets.accept_stl(synthetic.cuboid_stl(item))
    catalog = geometry.hopf_catalog(orientations, 5)

    def opened(ctx):
        return session_mod.Session(mesh, (box, box, box), (0.0, 0.0, 0.0), 1.0, catalog, context=ctx)

    with compute.Context(0, open_mb * 1_000_000) as ctx:
        opened(ctx).close()
    fills = []
    for cap in (0, fill_mb * 1_000_000):
        with compute.Context(0, cap) as ctx:
            s = opened(ctx)
            fills.append([(p.orientation_index, p.translation, p.score) for p in s.greedy(2)])
            kernels = [s.field("kernel", o).tobytes() for o in range(0, orientations, 7)]
            fills[-1].append(kernels)
            s.close()
    assert len(fills[0]) == 3
    assert fills[0] == fills[1]
