"""The production cascade (es_cascade_image): its tables against the definition.

CPU: for random ring-1 cycles of plans of every width, the kernel's own steps on the tables (keys,
bucket entry, unreduced table rows, wrap distance) in Python integers: every row lies inside its
table, the carry split and wrap are exact wherever the kernel does not take its exact path, and
the mask bits equal each entry's parts on n itself.  The parts are necessary conditions of the
plan's filters, and the entries together cover every filter in full.

GPU: production launches (range, ragged, list, batch, static) against the C oracle."""
import ctypes as C

import numpy as np
import pytest

from conftest import golden


def image(plan, tables, smem=180 * 1024):
    import es_native as N
    A = N.PlanArrays(plan)
    info = N.CascadeInfo()

    def call(small, tabs, parts):
        def ptr(a):
            return a.ctypes.data_as(C.c_void_p) if a is not None else None
        N.check(N.lib().es_cascade_image(
            C.byref(A.desc), tables, smem, C.byref(info), ptr(small), 0 if small is None else small.size,
            ptr(tabs), 0 if tabs is None else tabs.size, ptr(parts), 0 if parts is None else parts.size))
    call(None, None, None)
    small = np.zeros(info.small_bytes, dtype=np.uint8)
    tabs = np.zeros(max(info.tab_words, 1), dtype=np.uint32)
    parts = np.zeros(3 * info.n_parts + 3, dtype=np.uint32)
    call(small, tabs, parts)
    return info, small, tabs, parts[:3 * info.n_parts].reshape(-1, 3)


WHEELS = {(c["k"], c["role"]): c["wheel"] for c in golden("replay_blocks.json")["cases"]}


def _plan(spec):
    import es_gb300
    k, role = spec
    if role is None or isinstance(role, list):
        return es_gb300.Plan(k, None, role)
    return es_gb300.Plan(k, None, WHEELS[(k, role)])


# one to four words, wider rings, wheels below and above 32 bits, no wheel, few filters
PLANS = [(1, None), (3, None), (12, None), (40, None), (60, None), (80, None), (120, None), (200, None),
         (300, None), (390, "primary"), (384, "confirmation"), (379, "primary"), (378, "primary"),
         (300, [[13, 3], [2, 9], [5, 2]]), (250, [[199, 1], [17, 2], [3, 2]]), (30, [[2, 5], [29, 1], [3, 4]])]


@pytest.mark.parametrize("spec", PLANS, ids=lambda s: f"k{s[0]}")
def test_tables_match_definition(spec):
    P = _plan(spec)
    rng = np.random.default_rng(P.k)
    radix = (list(P.radix) + [1, 1, 1])[:max(3, len(P.radix))]
    terms = P.terms() + [[0]] * (3 - len(P.radix)) if len(P.radix) < 3 else P.terms()
    r0, r1 = radix[0], radix[1]
    filters = [(P.info[p][0], set(P.info[p][1])) for p in P.rest]
    for F in (1, 3, 4, 6):
        info, small, tabs, parts = image(P, F)
        u32 = small.view(np.uint32)
        sorted_terms = [int(small[info.o_sorted + 16 * i:info.o_sorted + 16 * i + 8].view("<u8")[0]) |
                        int(small[info.o_sorted + 16 * i + 8:info.o_sorted + 16 * i + 16].view("<u8")[0]) << 64
                        for i in range(r0)]
        assert sorted_terms == sorted(terms[0])
        digits = u32[info.o_digits // 4:info.o_digits // 4 + r0]
        assert [terms[0][d] for d in digits] == sorted_terms
        entry = {}
        for e, f, d in parts.tolist():
            entry.setdefault(e, []).append((f, d))
            assert filters[f][0] % d == 0
        # every filter is tested in full somewhere
        assert {f for ps in entry.values() for f, d in ps if d == filters[f][0]} == set(range(len(filters)))
        inner = [entry.get(e, []) for e in range(F)]
        q = [int(np.prod([d for _, d in ps])) if ps else 2 for ps in inner]
        proj = [[(d, {x % d for x in filters[f][1]}) for f, d in ps] for ps in inner]
        starts = [info.tab_base[i] + min(0, info.tab_wrap[i]) for i in range(F)] + [4 * info.tab_words]   # table after table
        W = -(-r0 // 32)
        RS = 4 if W == 3 else W
        assert info.row_bytes == (8 * RS if W <= 1 else 4 * RS)   # one word: both masks in a row
        sh, up, ssh = info.key_shift, info.key_up, info.bucket_log2
        bsh, band, flag, mask32 = 32 - ssh, 3 << ssh, (1 << ssh) - 1, 0xffffffff
        t_blk = int(rng.integers(0, 1 << 30))
        for _ in range(6):
            b2 = sum(terms[j][int(rng.integers(radix[j]))] for j in range(2, len(radix))) % P.M
            A = P.M - b2
            KA, KM = (A >> sh << up) & mask32, P.M >> sh << up
            for d1 in ([0, r1 - 1] + rng.integers(0, r1, size=6).tolist()):
                row = info.o_row1 // 4 + d1 * info.row1_bytes // 4
                k1 = int(u32[row])
                wrap1 = k1 > KA
                t = (KA - k1 + (KM if wrap1 else 0)) & mask32
                bucket = t >> bsh
                assert bucket < 2048
                e4 = int(u32[info.o_buckets // 4 + bucket])
                ts = (t << ssh) & mask32
                split = (e4 & flag) + (1 if e4 < ts else 0)
                rare = ((e4 - ts) & mask32) < band or (e4 & flag) == flag or k1 == KA
                exact1 = terms[1][d1] >= A
                b = (b2 + terms[1][d1]) % P.M
                exact_split = sum(1 for s in sorted_terms if b + s < P.M)
                if rare:
                    wrap1, split = exact1, exact_split
                assert wrap1 == exact1 and split == exact_split
                for i in range(F):
                    mul = info.tab_mul[i]
                    assert np.gcd(mul, q[i]) == 1
                    tc = t_blk * P.M % q[i]
                    corr = -P.M * mul % q[i]
                    B = (b2 + tc) * mul % q[i]
                    if wrap1:
                        B = (B + corr) % q[i]
                    a = info.tab_base[i] + info.row_bytes * B + int(u32[row + 1 + i])
                    for at in (a, a + info.tab_wrap[i]):
                        assert starts[i] <= at <= starts[i + 1] - 4 * RS
                    lo = tabs[a // 4:a // 4 + RS]
                    hi = tabs[(a + info.tab_wrap[i]) // 4:(a + info.tab_wrap[i]) // 4 + RS]
                    for s in range(RS * 32):
                        got = (int((hi if s >= split else lo)[s >> 5]) >> (s & 31)) & 1
                        if s >= r0:
                            assert got == 0
                            continue
                        n = t_blk * P.M + (b + sorted_terms[s]) % P.M
                        assert got == int(all(n % d in ok for d, ok in proj[i])), (F, i, s)
        assert W <= RS


def test_tables_fit_the_room_they_are_given():
    for spec in PLANS:
        for room in (24 * 1024, 64 * 1024, 180 * 1024):
            info, _, _, _ = image(_plan(spec), 4, room)
            # fill-in tables (at most four rows each) may exceed a room that holds nothing
            assert info.small_bytes + 4 * info.tab_words <= max(room, info.small_bytes) + 6 * 5 * info.row_bytes


def test_tables_never_exceed_their_room():
    """Whatever multipliers are chosen: not the room, and not what a block of its length may spend on
    tables.  (The wheels' wrap corrections lie anywhere below their tables' moduli.)"""
    for spec in PLANS + [(k, None) for k in (192, 212, 258, 294)] + [(382, "primary"), (392, "primary"),
                                                                     (400, "confirmation")]:
        P = _plan(spec)
        most = (12 if P.R < 1 << 22 else 48 if P.R < 1 << 28 else 144) * 1024
        for tables in range(1, 7):
            for room in (64 * 1024, 180 * 1024):
                info, _, _, _ = image(P, tables, room)
                fill_ins = tables * -(-4 * info.row_bytes // 16) * 16   # four rows each, whatever the room
                left = max(0, room - info.small_bytes)
                assert 4 * info.tab_words <= max(min(left, most), fill_ins), (spec, tables, room)


# plans whose candidates per digit with four tables lie on either side of the line of their ring's words
@pytest.mark.parametrize("spec,want", [
    ((316, None), 4), ((196, None), 4), ((340, None), 5), ((394, "primary"), 5), ((244, None), 4),
    ((390, "confirmation"), 4), ((395, "confirmation"), 5), ((384, "primary"), 5), ((380, "confirmation"), 4),
    ((379, "primary"), 4), ((400, "primary"), 5), ((378, "primary"), 5), ((391, "primary"), 5),
    ((250, [[199, 1], [7, 3], [137, 1], [89, 1], [17, 2], [131, 1], [37, 1], [43, 1], [2, 8], [127, 1], [11, 1], [23, 1],
            [3, 2]]), 4)], ids=str)
def test_one_more_table_where_it_pays(spec, want, tmp_path):
    import es_native as N
    import fake_lib
    with fake_lib.bound(fake_lib.build(tmp_path)) as L:
        ctx = N.Context(_plan(spec), N.make_tune(layout=N.LAYOUT_AUTO, mask_filters=4, count_stages=0))
        ctx.set_block(0)
        ctx.launch(0, 1)
        ctx.sync()
        ctx.close()
        assert L.fake_tables() == want


@pytest.mark.parametrize("r1,want", [(2000, (16, 4)), (3300, (16, 3))])
def test_one_more_table_only_where_it_fits(r1, want, tmp_path):
    """Three tables of weak filters, which ask for a fourth; its rows of a long ring 1 may not fit a CTA
    where the three tables' do (16: the production cascade, 1: the scalar layout)."""
    import es_native as N
    import fake_lib
    rng = np.random.default_rng(r1)
    M, radix, q = (1 << 89) - 1, [32, r1, 4, 5], [11, 13, 17, 19, 23, 29]
    terms = [int(x) * int(y) % M for x, y in zip(rng.integers(1, 1 << 62, size=sum(radix)), rng.integers(1, 1 << 62, size=sum(radix)))]
    arrays = N.PlanArrays.from_arrays(
        30, np.array(radix, dtype=np.uint32), np.array([t & (1 << 64) - 1 for t in terms], dtype=np.uint64),
        np.array([t >> 64 for t in terms], dtype=np.uint64), np.array(q, dtype=np.uint32),
        np.concatenate([N.bit_table(x, range(1, x)) for x in q]), M)
    with fake_lib.bound(fake_lib.build(tmp_path)) as L:
        ctx = N.Context.from_arrays(arrays, N.make_tune(layout=N.LAYOUT_AUTO, mask_filters=3, count_stages=0), len(q))
        ctx.set_block(0, np.zeros(len(q), dtype=np.uint32))
        ctx.launch(0, 1)
        ctx.sync()
        ctx.close()
        assert (L.fake_layout(), L.fake_tables()) == want


# ------------------------------------------------------------------ GPU
def _ranges(P):
    outer = P.R // P.radix[0]
    r1 = P.radix[1] if len(P.radix) > 1 else 1
    r2 = P.radix[2] if len(P.radix) > 2 else 1
    row = r1 * r2
    cand = [(0, min(outer, 40 * row + 7)), (5, 6), (r1 - 1, r1 + 1), (3 * r1 + 2, 7 * r1 + 5), (row - 1, row + 1),
            (5 * row + 3 * r1 + 1, 70 * row), (outer - 3, outer), (outer // 2, outer // 2 + 33 * row)]
    return sorted({(max(0, a), min(outer, b)) for a, b in cand if 0 <= a < b and a < outer})


@pytest.mark.gpu
@pytest.mark.parametrize("spec", PLANS, ids=lambda s: f"k{s[0]}")
def test_production_scan_matches_c_oracle(native, spec):
    """Ragged ranges, every table count, several strips and blocks; production survivors against
    the C oracle.  Filters are cut to the first few so that survivors are plenty."""
    import es_oracle as O
    N = native
    P = _plan(spec)
    keep = P.rest[:2 if isinstance(spec[1], list) else (5 if P.k > 100 else 3)]

    class Few:   # the plan with only its first filters
        pass
    few = Few()
    few.__dict__.update(P.__dict__, rest=keep)
    few.idx_to_n = P.idx_to_n
    outer = P.R // (P.radix[0] if P.radix else 1)
    ranges = _ranges(P) if P.radix else [(0, 1)]
    ranges = [(a, min(b, a + (1 << 17) // (P.radix[0] if P.radix else 1) + 1)) for a, b in ranges]
    for t in (0, 3):
        want = {r: O.scan_c(few, t, o_range=r)[0] for r in ranges}
        for F, strip, threads in ((1, 8, 512), (2, 1, 64), (3, 8, 512), (4, 3, 256), (5, 64, 512), (8, 8, 96)):
            ctx = N.Context(few, N.make_tune(layout=5, mask_filters=F, strip=strip, threads=threads, count_stages=0))
            ctx.set_block(t)
            for r in ranges:
                ctx.reset()
                ctx.launch(r[0], r[1] - r[0])
                assert sorted(int(x) for x in ctx.survivors()) == want[r], (F, strip, t, r)
            # the same indices as an explicit list, in reverse and with repeats
            a, b = ranges[0]
            lst = np.arange(a, min(b, a + 500), dtype=np.uint64)[::-1]
            lst = np.concatenate([lst, lst[:7]])
            ctx.reset()
            ctx.launch_list(lst)
            ws = O.scan_c(few, t, outer=lst)[0]
            assert sorted(int(x) for x in ctx.survivors()) == sorted(ws), (F, strip, t, "list")
            ctx.close()
    assert outer >= 1


@pytest.mark.gpu
@pytest.mark.parametrize("spec", [(300, None), (390, "primary"), (379, "primary")], ids=lambda s: f"k{s[0]}")
def test_production_windows_of_several_digits(native, spec):
    """Ranges long enough for the launch to give a lane several ring-2 digits per unit (few warps,
    so that the strip rule picks 4 to 8), whose queue outlives the steps: against the C oracle."""
    import es_oracle as O
    N = native
    P = _plan(spec)

    class Few:
        pass
    few = Few()
    few.__dict__.update(P.__dict__, rest=P.rest[:6])
    few.idx_to_n = P.idx_to_n
    o = 1234567
    n = (1 << 27) // P.radix[0]
    want = O.scan_c(few, 1, o_range=(o, o + n))[0]
    assert len(want) > 1000
    for F, threads in ((3, 64), (4, 64), (4, 512), (6, 128)):
        ctx = N.Context(few, N.make_tune(layout=5, mask_filters=F, strip=8, threads=threads, ctas_per_sm=1,
                                         count_stages=0))
        ctx.set_block(1)
        ctx.reset()
        ctx.launch(o, n)
        assert sorted(int(x) for x in ctx.survivors()) == want, (F, threads)
        ctx.close()


@pytest.mark.gpu
def test_production_batch_matches_c_oracle(native):
    """Plans of every width in one batch, with and without the graph: survivors per item and the
    least good one per group."""
    import es_oracle as O
    N = native
    plans = [_plan(s) for s in PLANS if s[0] >= 40]
    for layout, F in ((5, 4), (0, 3), (2, 2)):
        tune = N.make_tune(layout=layout, mask_filters=F, strip=4, count_stages=0)
        ctxs = [N.Context(p, tune) for p in plans]
        items = []
        for i, p in enumerate(plans):
            o = p.R // p.radix[0]
            a = min(12345 * i, o // 2)
            items.append((i, i, i % 3, a, min(o, a + (1 << 21) // p.radix[0])))
        want = [O.scan_c(p, it[2], o_range=(it[3], it[4]))[0] for p, it in zip(plans, items)]
        b = N.Batch(ctxs, items, tune)
        for graph in (False, True, True):
            b.run(use_graph=graph)
            b.sync()
            surv = b.survivors()
            for i, (p, it) in enumerate(zip(plans, items)):
                got = sorted(int(r["idx"]) for r in surv if r["item"] == i)
                assert got == want[i], (layout, i, p.k)
                good = sorted(n for n in (p.idx_to_n(x, it[2]) for x in got) if n > p.k + 1)
                m = b.group_min(i)
                assert (m is None) == (not good)
                if good:
                    assert m[0] * p.M + m[1] == good[0]
        b.close()
