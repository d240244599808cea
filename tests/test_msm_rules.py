"""The rules that plan an MSM batch from its sizes (csrc/gb_msm_rules.h), over
their range: the affine rounds' scratch stays below its bound, and large
batches are divided into groups that stay below theirs and leave no item out."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG, REPO

SLOTS = 152 * 4  # blocks resident at once


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("rules") / "msm_rules.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(PKG, "csrc"), "-o", so,
                           os.path.join(REPO, "tests", "msm_rules_harness.cpp")])
    L = ctypes.CDLL(so)
    u64 = ctypes.c_uint64
    L.r_choose_window.argtypes = [ctypes.c_size_t, ctypes.c_int]
    L.r_rounds.argtypes = [u64, u64, u64, u64]
    L.r_scratch.argtypes = [u64, u64, ctypes.c_int, u64]
    L.r_scratch.restype = L.r_rounds_limit.restype = u64
    L.r_groups.argtypes = [ctypes.c_void_p, ctypes.c_size_t, ctypes.c_int, ctypes.c_int, ctypes.c_void_p]
    L.r_table_items.argtypes = [ctypes.c_size_t, ctypes.c_size_t]
    L.r_table_items.restype = ctypes.c_size_t
    L.r_sum_groups.argtypes = [u64, ctypes.c_uint32, ctypes.c_int]
    L.r_pairs_per_thread.argtypes = [u64, u64]
    L.r_groups.restype = ctypes.c_size_t
    L.r_typical.argtypes = [ctypes.c_void_p, ctypes.c_size_t, ctypes.c_int, ctypes.c_int]
    L.r_typical.restype = ctypes.c_double
    L.r_short_span.argtypes = [ctypes.c_double, ctypes.c_double, ctypes.c_uint32]
    return L


@pytest.mark.parametrize("buckets", [1 << 10, 1 << 15, 1 << 20, 1 << 25])
def test_rounds_scratch_is_bounded(rules, buckets):
    limit = rules.r_rounds_limit()
    assert limit <= 16 << 30  # a sixteenth of the device
    for lg in np.arange(10, 31, 0.25):
        digits = int(2 ** lg)
        r = rules.r_rounds(digits, buckets, SLOTS, limit)
        assert rules.r_scratch(digits, buckets, r, SLOTS) <= limit
        assert rules.r_rounds(digits, buckets, SLOTS, 0) == 0
        # less room, fewer rounds
        for most in (limit >> 2, limit >> 6):
            less = rules.r_rounds(digits, buckets, SLOTS, most)
            assert less <= r and rules.r_scratch(digits, buckets, less, SLOTS) <= most


def test_rounds_of_ordinary_batches(rules):
    """The bound does not touch what is measured in the rule's table, nor long
    lists, which go through the rounds in slices."""
    for digits, avg, want in ((1 << 20, 80, 0), (4_700_000, 72, 2), (16_800_000, 512, 4), (48_000_000, 23, 2),
                              (1 << 28, 8192, 4), (1 << 28, 8, 1), (1 << 30, 32768, 4)):
        assert rules.r_rounds(digits, digits // avg, SLOTS, rules.r_rounds_limit()) == want


def groups(rules, sizes, c, precomputed):
    sizes = np.asarray(sizes, dtype=np.uint64)
    out = np.zeros(len(sizes) + 2, dtype=np.uint64)
    n = rules.r_groups(sizes.ctypes.data, len(sizes), c, precomputed, out.ctypes.data)
    return [int(x) for x in out[:n]]


@pytest.mark.parametrize("c,precomputed", [(8, 0), (11, 1), (13, 0), (16, 1), (16, 0)])
@pytest.mark.parametrize("sizes", [[0], [5], [1 << 20] * 3, [1 << 20] * 100, [700] * 70000, [1 << 24] * 3 + [9] * 50,
                                   [1 << 26, 1, 1 << 26, 0, 1 << 26], [0] * 5000])
def test_groups(rules, sizes, c, precomputed):
    first = groups(rules, sizes, c, precomputed)
    assert first[0] == 0 and first[-1] == len(sizes) and all(a < b for a, b in zip(first, first[1:]))
    nwin = rules.r_windows(c)
    per_item = (1 << (c - 1)) * (1 if precomputed else nwin)
    parts = [(sum(sizes[a:b]) * nwin, (b - a) * per_item, b - a) for a, b in zip(first, first[1:])]
    for digits, buckets, items in parts:
        if items > 1:
            assert digits <= 1 << 28 and buckets <= 1 << 25
        assert buckets < 1 << 28  # the count scan's range
        r = rules.r_rounds(digits, buckets, SLOTS, rules.r_rounds_limit())
        assert rules.r_scratch(digits, buckets, r, SLOTS) <= rules.r_rounds_limit()
    # no more groups than needed: the next item does not fit
    for (digits, _, items), nxt in zip(parts, first[1:-1]):
        assert digits + sizes[nxt] * nwin > 1 << 28 or (items + 1) * per_item > 1 << 25


def test_ordinary_batches_are_one_group(rules):
    assert len(groups(rules, [1 << 18] * 20, 16, 1)) == 2
    assert len(groups(rules, [1 << 20] * 16, 16, 1)) == 2
    assert len(groups(rules, [2049] * 145, 9, 0)) == 2


def typical(rules, sizes, c, precomputed):
    sizes = np.asarray(sizes, dtype=np.uint64)
    return rules.r_typical(sizes.ctypes.data, len(sizes), c, precomputed)


@pytest.mark.parametrize("c,precomputed", [(9, 0), (15, 1), (16, 1)])
def test_typical_bucket(rules, c, precomputed):
    """Of equal MSMs the mean; of an uneven batch the large items' buckets, and
    these may then be added up without the block-wide fix-up."""
    rows = rules.r_windows(c) if precomputed else 1
    assert typical(rules, [3000] * 7, c, precomputed) == pytest.approx(3000 * rows / (1 << (c - 1)))
    assert typical(rules, [0, 0], c, precomputed) == 0
    for small in (32, 200):
        sizes = [1 << 16] * 2 + [256] * small
        large = (1 << 16) * rows / (1 << (c - 1))
        t = typical(rules, sizes, c, precomputed)
        assert 0.5 * large < t <= large
        mean = sum(sizes) / len(sizes) * rows / (1 << (c - 1))
        assert all(rules.r_short_span(mean, t, L) >= min(32, large / L) for L in range(3, 65))


@pytest.mark.parametrize("K,n,count,table", [  # both routes measured, the faster one
    (1 << 15, 512, 32, True), (1 << 15, 512, 48, False), (1 << 15, 512, 384, False), (1 << 15, 1024, 32, True),
    (1 << 15, 1024, 48, False), (1 << 15, 2048, 32, True), (1 << 15, 2048, 64, False), (1 << 15, 4095, 64, True),
    (1 << 15, 4095, 192, False), (1 << 14, 256, 128, True), (1 << 14, 256, 256, False), (1 << 14, 512, 128, True),
    (1 << 14, 1024, 192, True), (1 << 14, 1024, 384, False), (1 << 14, 2047, 256, True), (1 << 14, 2047, 384, False),
    (1 << 12, 64, 384, True), (1 << 12, 511, 384, True)])
def test_many_small_items_leave_the_table(rules, K, n, count, table):
    assert (count <= rules.r_table_items(K, n)) == table


@pytest.mark.parametrize("log_n", range(9))
def test_groups_a_sum(rules, log_n):
    """Few sums get all of a block's groups; many get no more than have two
    points each, so that none of a block's groups is idle."""
    n = 1 << log_n
    assert rules.r_sum_groups(8 * 152, n, 152) == 5
    for sums in (8 * 152 + 1, 1 << 20):
        groups = 1 << rules.r_sum_groups(sums, n, 152)
        assert groups == max(1, min(32, n // 2))


def test_tiles_of_fewer_pairs_than_planned(rules):
    """The rounds' kernel makes its tiles from the pairs that there are, with
    no more a thread than planned: each block then has a tile as long as there
    are pairs for one, and none is longer than the prefix buffer's."""
    for lg in np.arange(20, 30, 0.3):
        planned = int(2 ** lg)
        most = rules.r_pairs_per_thread(planned, SLOTS)
        assert 1 <= most <= 64
        for share in (1, 2, 3, 10, 1000, planned):
            pairs = planned // share
            per = min(most, rules.r_pairs_per_thread(pairs, SLOTS))
            assert 1 <= per <= most
            tiles = -(-pairs // (per * 128))
            assert tiles >= min(SLOTS, -(-pairs // 128)) // 2


def test_no_size_is_refused_for_its_window(rules):
    """Digits are numbered with 31 bits, and the widest windows have the fewest:
    whatever these can number, the chosen window can."""
    for n in [1, 255, 1 << 16, (1 << 24) + 1, 107_374_181, 107_374_182, 113_000_000, 120_000_000, 134_217_726]:
        assert n < 0x7FFFFFFF // rules.r_windows(16)
        for precomputed in (0, 1):
            assert n < 0x7FFFFFFF // rules.r_windows(rules.r_choose_window(n, precomputed)), n
    assert [rules.r_choose_window(1 << k, 0) for k in (11, 13, 15, 17, 19, 26)] == [8, 9, 10, 11, 12, 13]


@pytest.mark.parametrize("count", [1, 3, 4, 8, 40])
def test_server_estimate_follows_the_plan(rules, count):
    """serve.msm_scratch_bytes, the server's admission estimate, covers what the
    engine allocates for the entries of a batch, and not much more."""
    from gb_prover import serve
    for k in range(5, 24):
        for n in (1 << k, 3 << (k - 1)):
            c = rules.r_choose_window(n, 1)
            sizes = np.full(count, n, dtype=np.uint64)
            first = groups(rules, sizes, c, 1)
            items = max(b - a for a, b in zip(first, first[1:]))
            digits, buckets = items * n * rules.r_windows(c), items << (c - 1)
            r = rules.r_rounds(digits, buckets, SLOTS, rules.r_rounds_limit())
            lists = rules.r_scratch(digits, buckets, r, SLOTS)
            entries = digits + buckets * ((1 << r) - 1)
            known = 4 * (digits + entries) + lists + 192 * buckets
            got = serve.msm_scratch_bytes(n, count)
            assert known <= got + 1024 and got <= 1.35 * known + 48 * digits * (r == 0), (n, count, known, got)


def test_bench_counts_the_tables_windows(rules):
    """The roofline's digits are those of the table the context holds."""
    import sys
    sys.path.insert(0, REPO)
    import bench

    class Context:
        def __init__(self, n):
            self.bytes = 96 * n * rules.r_windows(rules.r_choose_window(n, 1))

        def device_bytes(self):
            return self.bytes

    for k in (8, 11, 12, 15, 16, 20):
        n = 1 << k
        assert bench.table_rows(Context(n), n) == rules.r_windows(rules.r_choose_window(n, 1))
