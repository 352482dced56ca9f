"""Descriptors that no planner makes but es_mitm_create accepts: the engine against sums in Python
integers.

CPU: the launch the host prepares (fake_cuda.cpp).  GPU: survivors and candidates."""
import numpy as np
import pytest

import fake_lib


class Halves:
    """What MitmEngine reads of a plan: two halves of one or more rings of terms, and filters."""

    def __init__(self, M, half1, half2, filters):
        self.k, self.M, self.w1, self.w2 = 12, M, half1, half2
        self.rest = [q for q, _ in filters]
        self.info = {q: (q, sorted(ok)) for q, ok in filters}

    def terms(self, half):
        return [len(r) for r in half], [t for r in half for t in r]

    def brute(self, B):
        def sums(half):
            s = [0]
            for r in half:
                s = [(x + t) % self.M for x in s for t in r]
            return s
        tested = [n for a in sums(self.w1) for b in sums(self.w2) if (n := (a + b) % self.M) < B]
        return sorted(n for n in tested if all(n % q in set(ok) for q, ok in self.info.values())), len(tested)


def _random(M, radix1, radix2, filters, seed):
    rng = np.random.default_rng(seed)

    def half(radix):
        return [[int(x) % M for x in rng.integers(0, 1 << 62, size=r)] for r in radix]
    return Halves(M, half(radix1), half(radix2),
                  [(q, sorted({int(x) for x in rng.integers(0, q, size=max(1, q * 2 // 3))})) for q in filters])


# one filter that fills the merged tables' budget by itself, and two that share it
@pytest.fixture(params=[[1 << 18], [(1 << 18) - 5, 3], [130817, 131317]], ids=str)
def wide(request):
    return _random(1000003, [30], [25], request.param, 1)


def test_merged_tables_fit_the_launch(wide, tmp_path):
    import es_mitm
    with fake_lib.bound(fake_lib.build(tmp_path)) as L:
        before, launches = L.fake_faults(), L.fake_launches()
        e = es_mitm.MitmEngine(wide, capacity=16)
        e.scan(wide.M)
        e.close()
        assert L.fake_launches() > launches and L.fake_faults() == before


@pytest.mark.gpu
def test_gpu_filters_of_large_moduli(native, wide):
    import es_mitm
    e = es_mitm.MitmEngine(wide)
    for B in (wide.M, wide.M // 3):
        assert e.scan(B) == wide.brute(B)
    e.close()


@pytest.mark.gpu
@pytest.mark.parametrize("M", [2, 3, 7, 8, 29])
def test_gpu_modulus_below_the_slices(native, M):
    """Fewer residues than the value-ordered sweep of S1 would have slices: every s1 counts once."""
    import es_mitm
    h = _random(M, [700, 3], [5, 2], [5], M)
    e = es_mitm.MitmEngine(h)
    for B in range(1, M + 1):
        assert e.scan(B) == h.brute(B)
    assert e.scan(M, 11, 901)[1] == 890 * 10   # B = M: every pair
    e.close()


def test_creation_does_not_hang_on_the_size_of_a_small_s1(tmp_path):
    """An engine of 131,072 s1 is made in about the time of one of 1,024: what a scan of them takes
    (a tenth of a millisecond) is not worth sorting them."""
    import time
    import es_mitm
    with fake_lib.bound(fake_lib.build(tmp_path)):
        def best(radix1):
            h = _random((1 << 89) - 1, radix1, [40, 40], [101, 103], 3)
            times = []
            for _ in range(7):
                t = time.perf_counter()
                e = es_mitm.MitmEngine(h, capacity=16)
                times.append(time.perf_counter() - t)
                e.close()
            return min(times)
        small, large = best([32, 32]), best([64, 64, 32])
        assert large < 4 * small + 1e-3, (small, large)
