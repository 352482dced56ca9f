"""What destroyed batches leave for the next ones: one set for contexts that take turns, no more than
256 MB idle on the device however many contexts made a batch, and nothing once the contexts are gone."""
import pytest

import fake_lib


@pytest.fixture
def fake(tmp_path):
    with fake_lib.bound(fake_lib.build(tmp_path)) as L:
        yield L


def _batch(N, ctx):
    return N.Batch([ctx], [(0, 0, 1, 0, ctx.n_outer)], N.make_tune(mask_filters=2, count_stages=0))


def test_idle_sets_are_bounded_and_given_back(fake):
    import es_gb300
    import es_native as N
    plan = es_gb300.Plan(60)
    start = fake.fake_live()
    ctxs = [N.Context(plan, N.make_tune(mask_filters=2, count_stages=0)) for _ in range(12)]
    mine = fake.fake_live()
    for c in ctxs:                       # one after another: one set serves them all
        _batch(N, c).close()
    assert fake.fake_live() <= mine + 3          # device, pinned, survivors
    together = [_batch(N, c) for c in ctxs]      # 12 sets of 42 MB
    for b in together:
        b.close()
    assert mine + 3 <= fake.fake_live() <= mine + 3 * 6
    ctxs[0].set_capacity(1 << 23)                # a set of 335 MB is not kept
    before = fake.fake_live()
    _batch(N, ctxs[0]).close()
    assert fake.fake_live() <= before
    for c in ctxs[1:]:
        c.close()
    last = _batch(N, ctxs[0])
    ctxs[0].close()                              # either may go first
    last.close()
    assert fake.fake_live() == start
