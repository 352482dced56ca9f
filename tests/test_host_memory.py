"""Host allocations that fail inside the calls that build things: an error code and nothing left behind,
never an exception across the C ABI.  (In a process of its own, which an exception would end.)"""
import subprocess
import sys

import pytest

import fake_lib

CHILD = """
import sys
sys.path[:0] = {paths!r}
import fake_lib, es_gb300, es_mitm, es_native as N
with fake_lib.bound({so!r}) as L:
    plan = es_gb300.Plan(60)
    tune = N.make_tune(layout=N.LAYOUT_AUTO, mask_filters=2, count_stages=0)
    ctx = N.Context(plan, N.make_tune(count_stages=0))
    makers = {{
        "context": lambda: N.Context(plan, N.make_tune(count_stages=1)),
        "batch": lambda: N.Batch([ctx], [(0, i, i, 0, ctx.n_outer) for i in range(40)], tune),
        "mitm": lambda: es_mitm.MitmEngine(HALVES, capacity=16),
    }}
    make = makers[{what!r}]
    HALVES = es_mitm.MitmPlan(40, 1.0)
    make().close()          # what is kept from then on is there already
    n, failed = 1, 0
    while True:
        live = L.fake_live()
        L.fake_fail_alloc(n)
        try:
            made = make()
        except N.EsError as e:
            assert e.code == -5, e   # ES_ERR_NOMEM
            assert L.fake_live() == live, (n, live, L.fake_live())
            failed += 1
        else:
            left = L.fake_fail_alloc(0)
            made.close()
            if left:   # fewer than n allocations
                break
        n += 1 if n < 60 else 1 + n // 12
    print("failed", failed)
"""


@pytest.mark.parametrize("what,at_least", [("context", 40), ("batch", 10), ("mitm", 40)])
def test_failed_allocations_come_back_as_codes(tmp_path, what, at_least):
    code = CHILD.format(paths=[p for p in sys.path if p], so=fake_lib.build(tmp_path), what=what)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    assert int(r.stdout.split()[-1]) >= at_least


def test_a_capacity_that_does_not_fit_leaves_no_buffer_to_write_to(tmp_path):
    """The old buffer is gone when the new one is refused: launches then count survivors and store none,
    and reading them says so."""
    import es_gb300
    import es_native as N
    with fake_lib.bound(fake_lib.build(tmp_path)) as L:
        ctx = N.Context(es_gb300.Plan(60), N.make_tune(mask_filters=2, count_stages=0))
        ctx.set_block(0)
        before = L.fake_faults()
        with pytest.raises(N.EsError):
            ctx.set_capacity(1 << 32)
        ctx.launch(0, ctx.n_outer)
        ctx.sync()
        assert L.fake_faults() == before
        ctx.set_capacity(1 << 10)
        ctx.launch(0, ctx.n_outer)
        ctx.sync()
        assert L.fake_faults() == before
        ctx.close()
