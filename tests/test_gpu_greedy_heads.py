"""The greedy's pruned heads: an orientation whose free planes lie above the
best head's bound comes back with an empty page whose planes above were not
visited.  Such a page says nothing about them: it must not count as "admits no
copy", and the orientation need not be paged again until its floor could win.

The scene is a narrow tower of plates: flat items fit into every gap from the
floor up, upright ones only above the top plate, far past the bound of the
best flat head.  The last test walks a fill through several pages of one
orientation."""

import numpy as np
import pytest

from conftest import package
from oracle import proposal_net

pytestmark = pytest.mark.gpu

HALF = 2 ** -0.5
# Flat twice (identity, half a turn about z), upright twice (a quarter about x and y).
CATALOG = np.array([[0, 0, 0, 1], [0, 0, 1, 0], [HALF, 0, 0, HALF], [0, HALF, 0, HALF]], np.float64)
FLAT, UPRIGHT = (0, 1), (2, 3)


def _tower(ctx, top, catalog=CATALOG):
    """A 16 x 16 x 180 box with plates every nine cells up to `top`."""
    assets, session_mod, synthetic = package("assets"), package("session"), package("synthetic")
    item = assets.accept_stl(synthetic.cuboid_stl((14.0, 14.0, 4.0)))
    s = session_mod.Session(item, (16.0, 16.0, 180.0), (0.0, 0.0, 0.0), 1.0, catalog, context=ctx)
    x, y, z = min((c.translation for c in s.pages([0])[0]), key=lambda t: t[2])
    for above in range(9, top, 9):
        s.place(0, (x, y, z + above))
    return s


def _net(ctx):
    net = package("proposal").Proposal(context=ctx)
    net.set_parameters(proposal_net.he_parameters(9).astype(np.float32))
    return net


@pytest.mark.parametrize("top,upright_fits", [(150, True), (176, False)])
def test_widening_counts_orientations_that_are_free_high_up(gpu_ctx, top, upright_fits):
    proposal = package("proposal")
    s = _tower(gpu_ctx, top)
    fits = [bool(page) for page in s.pages(range(4))]  # whole pages
    assert fits == [True, True, upright_fits, upright_fits]
    best = s.greedy(1)[0]
    s.remove_last()
    net = _net(gpu_ctx)
    # Any three of the four hold a flat and an upright one.
    placed, fallbacks, widenings = proposal.greedy_proposed_adaptive(s, net, 3, 3, 1)
    assert widenings == (0 if upright_fits else 1)
    assert fallbacks == 0
    assert placed[0].score == best.score
    net.close()
    s.close()


def _pages_of_a_step(s, rejections):
    """Orientations paged during one greedy step that rejects its first poses."""
    seen = []
    s.set_validator(lambda *pose: len(seen) >= rejections or seen.append(pose))
    s.pages([0])  # the layout is up to date
    before = s.stats()["pages"]
    placed = s.greedy(1)
    paged = s.stats()["pages"] - before
    s.set_validator(None)
    assert len(placed) == 1 and len(seen) == rejections
    return paged, seen + [placed[0].translation]


@pytest.mark.parametrize("rejections", [1, 12])
def test_rejected_poses_page_undecided_orientations_only_when_they_could_win(gpu_ctx, rejections):
    s = _tower(gpu_ctx, 150, CATALOG[:2])
    flat_alone, poses_alone = _pages_of_a_step(s, rejections)
    s.close()
    s = _tower(gpu_ctx, 150)
    paged, poses = _pages_of_a_step(s, rejections)
    s.close()
    assert poses == poses_alone
    if rejections == 1:
        # The other flat orientation's head has the rejected one's score, which
        # the floors of the upright ones exceed: they are not paged again.
        assert paged == flat_alone + len(UPRIGHT)
    else:
        # Their floors are reached at some rejection; a whole page settles them.
        assert paged <= flat_alone + 2 * len(UPRIGHT)


def test_rejections_walk_through_more_than_one_page(gpu_ctx):
    assets, session_mod, synthetic = package("assets"), package("session"), package("synthetic")
    item = assets.accept_stl(synthetic.cuboid_stl((9.0, 7.0, 5.0)))
    s = session_mod.Session(item, (24.0, 22.0, 20.0), (0.0, 0.0, 0.0), 1.0, CATALOG[:1], context=gpu_ctx)
    want, cursor = [], None
    while len(want) < 81:  # three pages of 32, each after the one before
        page = s.pages([0], cursors=[cursor])[0]
        assert len(page) == 32
        want += [c.translation for c in page]
        cursor = page[-1]
    seen = []

    def validate(_orientation, translation, _pose, _q):
        seen.append(translation)
        return len(seen) > 80

    s.set_validator(validate)
    placed = s.greedy(1)
    s.set_validator(None)
    s.close()
    assert seen == want[:81]
    assert [p.translation for p in placed] == want[80:81]
