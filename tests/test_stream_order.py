"""The library's streams are non-blocking ones, so nothing orders them after the legacy default
stream: whatever a launch reads or counts with has to be written on the launch's own stream, or be
there before the call that wrote it returns."""
import numpy as np
import pytest

import fake_lib


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    with fake_lib.bound(fake_lib.build(tmp_path_factory.mktemp("fake"))) as L:
        yield L


@pytest.mark.parametrize("first", ["launch", "launch_list", "set_tune", "batch", "counts"])
def test_nothing_waits_on_another_stream_at_a_launch(fake, first):
    import es_gb300
    import es_native as N
    before, launches = fake.fake_faults(), fake.fake_launches()
    plan = es_gb300.Plan(60)
    ctx = N.Context(plan, N.make_tune(layout=N.LAYOUT_AUTO, mask_filters=4, count_stages=int(first == "counts")))
    ctx.set_block(3)
    batch = None
    if first == "batch":
        tune = N.make_tune(layout=N.LAYOUT_AUTO, mask_filters=2, count_stages=0)
        batch = N.Batch([ctx], [(0, 0, 1, 0, ctx.n_outer)], tune)
        batch.run(use_graph=False)
    elif first == "launch_list":
        ctx.launch_list(np.arange(min(5, ctx.n_outer), dtype=np.uint64))
    else:
        if first == "set_tune":
            ctx.set_tune(N.make_tune(layout=N.LAYOUT_AUTO, mask_filters=2, count_stages=0))
        ctx.launch(0, ctx.n_outer)
    ctx.sync()
    fake.fake_drain()   # late work of the default stream, if there is any
    ctx.launch(0, ctx.n_outer)
    ctx.sync()
    assert fake.fake_launches() > launches
    assert fake.fake_faults() == before
    if batch:
        batch.close()
    ctx.close()


def test_mitm_engine_is_there_when_its_creation_returns(fake):
    import es_mitm
    before, launches = fake.fake_faults(), fake.fake_launches()
    e = es_mitm.MitmEngine(es_mitm.MitmPlan(40, 1.0), capacity=16)
    e.scan(1000)
    assert fake.fake_launches() > launches
    assert fake.fake_faults() == before
    e.close()
