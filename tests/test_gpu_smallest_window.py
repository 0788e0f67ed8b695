"""Pages over the smallest windows: the depths of a kernel's cells index the
proximity table like the window's distances, and in a window of one cell the
kernel is deeper than any distance there."""

import numpy as np
import pytest

from conftest import package
from oracle.bindings import oracle_page

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,kernel", [((1, 1, 1), (1, 1, 1)), ((1, 1, 3), (1, 1, 2)), ((2, 2, 2), (2, 2, 2)),
                                          ((3, 3, 3), (3, 3, 3)), ((1, 2, 2), (1, 1, 1))])
@pytest.mark.parametrize("blocked", [False, True])
def test_pages_of_the_smallest_windows(oracle_c, shape, kernel, blocked):
    compute, pl = package("compute"), package("pipeline")
    occ = np.zeros(int(np.prod(shape)), np.uint8)
    occ[-1] = blocked
    ker = np.ones(int(np.prod(kernel)), np.uint8)
    height, max_z = float(shape[2]), float(kernel[2]) / 2
    scene = pl.PageScene((0, 0, 0), shape, (0.0, 0.0, 0.0), 1.0, 0.0, height)
    with compute.Context(0) as ctx:
        page = pl.spectral_page(scene, occ, (0, 0, 0), kernel, ker, max_z, context=ctx)
    prox, _ = oracle_c.build_proximity(shape, occ)
    want = oracle_page(oracle_c, (0, 0, 0), shape, occ, prox, (0, 0, 0), kernel, ker, (0.0, 0.0, 0.0, 1.0), max_z,
                       0.0, height)
    assert [(p.translation, p.score) for p in page] == [(tuple(t), s) for t, s, _ in want]
