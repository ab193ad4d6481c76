"""The on-chip sorts of 33..4096 strings (squeezed 32-bit values): segment
sizes at the edges of its size classes, and key sets that reach each of its
branches (no ties, tied runs in order, short and long tied runs out of
order, all keys equal, runs that continue in the next round)."""
import numpy as np
import pytest

import cases
import pyoracle
import pyssort

pytestmark = pytest.mark.gpu

SIZES = (33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 2047,
         2048, 2049)


def _strings(kind, n, rng):
    if kind == "random":  # distinct within the squeezed bits, all byte values
        return [bytes(rng.integers(1, 256, size=rng.integers(1, 20)).tolist()) for _ in range(n)]
    if kind == "letters":
        return [bytes(rng.integers(97, 123, size=rng.integers(1, 24)).tolist()) for _ in range(n)]
    if kind == "pairs":  # short tied runs: 13 shared letters, then two differing tails
        return [b"abcdefgh" + bytes(rng.integers(97, 99, size=8).tolist()) + bytes([97 + i % 3])
                for i in range(n)]
    if kind == "few":  # long tied runs, distinguished in the last key byte, and equal keys
        return [b"xyzzyxyz"[:int(rng.integers(4, 9))] + b"q" * int(rng.integers(0, 8)) +
                bytes([int(rng.integers(97, 100))]) for _ in range(n)]
    if kind == "late":  # the first 27 differing bits agree for most strings
        return [(b"\x01\xff" * 7 if rng.random() < 0.9 else b"\xfe\x01" * 7) +
                bytes([int(rng.integers(1, 256)), int(rng.integers(1, 256))]) for _ in range(n)]
    if kind == "equal":
        return [b"the same sixteen bytes and more"] * n
    if kind == "runs":  # runs of equal 16-byte keys that go on differently
        return [b"0123456789abcde" + bytes([int(rng.integers(97, 101))]) +
                bytes(rng.integers(97, 100, size=rng.integers(0, 20)).tolist()) for _ in range(n)]
    raise ValueError(kind)


@pytest.mark.parametrize("kind", ["random", "letters", "pairs", "few", "late", "equal", "runs"])
def test_one_warp_sort_sizes(sorter, kind):
    rng = np.random.default_rng(sum(kind.encode()))
    for n in SIZES:
        arena, offs = cases.arena_of(_strings(kind, n, rng))
        p, l = sorter.sort_host(arena, offs)
        rp, rl = pyoracle.oracle_sort(arena, offs)
        assert np.array_equal(p, rp), n
        assert np.array_equal(l, rl), n


@pytest.mark.parametrize("kind", ["letters", "pairs", "few", "late", "runs"])
def test_one_warp_sort_of_partitioned_segments(sorter, kind):
    """The same key sets behind a sample partition: keys come from the key
    buffer (asynchronous copies) instead of the arena."""
    rng = np.random.default_rng(7 + sum(kind.encode()))
    arena, offs = cases.arena_of(_strings(kind, 60_000, rng))
    p, l = sorter.sort_host(arena, offs)
    rp, rl = pyoracle.oracle_sort(arena, offs)
    assert np.array_equal(p, rp) and np.array_equal(l, rl)


def test_large_leaf_buckets():
    """Sorts of at least 4 Mi strings sort range buckets of 2049..4096 strings
    on chip (with 12-bit positions, so that a difference in key byte 15 is found
    in the full keys): wide buckets, strings that differ in their last key byte
    only, and duplicates."""
    n = 4_300_000
    rng = np.random.default_rng(5)
    rows = np.full((n, 17), 97, dtype=np.uint8)
    rows[:, 0:3] = rng.integers(97, 123, size=(n, 3))
    rows[:, 13:16] = rng.integers(97, 123, size=(n, 3))
    rows[:, 16] = 0
    arena = np.concatenate([rows.ravel(), np.zeros(16, np.uint8)])
    offs = np.arange(n, dtype=np.uint64) * 17
    with pyssort.Sorter(0) as s:
        s.set_param(pyssort.SSORT_PARAM_TARGET_BUCKET, 2048)
        p, l = s.sort_host(arena, offs)
    bad, first = pyoracle.oracle_check(arena, offs, p, l)
    assert bad == 0, (bad, first)


@pytest.mark.parametrize("kind", ["tied_windows", "one_splitter", "outside_prefix", "bytes15"])
def test_partition_classification(sorter, kind):
    """Splitter classification at its branches: splitters that share their first
    64 differing bits, one distinct splitter, keys without the splitters'
    common prefix on either side, and splitters that differ in the last byte."""
    rng = np.random.default_rng(sum(kind.encode()))
    n = 30_000
    def tail(k):
        return bytes(rng.integers(97, 123, size=k).tolist())
    if kind == "tied_windows":
        strings = [bytes([97 + int(rng.integers(0, 2))]) + b"mmmmmmmmmm" + tail(5) for _ in range(n)]
    elif kind == "one_splitter":
        strings = [b"the same key all over"] * n + [b"the", b"thf"]
    elif kind == "outside_prefix":
        strings = [b"middle/" + tail(9) for _ in range(n)] + \
            [tail(3) for _ in range(40)] + [b"", b"\xff\xff", b"middle", b"middle/"]
    else:
        strings = [b"fifteen bytes15" + bytes([int(rng.integers(1, 256))]) + tail(2)
                   for _ in range(n)]
    arena, offs = cases.arena_of(strings)
    p, l = sorter.sort_host(arena, offs)
    rp, rl = pyoracle.oracle_sort(arena, offs)
    assert np.array_equal(p, rp) and np.array_equal(l, rl)


@pytest.mark.parametrize("n", [75_775, 75_776, 75_777, 606_208, 606_209])
def test_tile_size_limits(sorter, n):
    """Sorts on either side of the sizes at which partition tiles grow (1024,
    2048 and 4096 strings per tile)."""
    ss = pyssort.gen_uniform(n, 1, 12, ord("a"), 26, n)
    p, l = sorter.sort_host(ss.arena, ss.offs)
    rp, rl = pyoracle.oracle_sort(ss.arena, ss.offs)
    assert np.array_equal(p, rp) and np.array_equal(l, rl)
