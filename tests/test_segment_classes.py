"""The on-chip sorts where each launches: segments at the edges of the four
size classes in the launch that classes share and in launches of their own
(a plain sort of up to 2048 strings runs in one CTA and reaches neither),
tied runs at the lengths where their repair changes, and which sorts the
one-CTA form leaves to the general loop."""
import numpy as np
import pytest

import cases
import pyoracle
import pyssort

pytestmark = pytest.mark.gpu

EDGES = (2, 8, 9, 32, 33, 64, 65, 128, 129, 256, 257, 511, 512, 513, 1023, 1024, 1025, 2047, 2048)
CLASS_MIN_SEGS = 4736  # segments of the first class (257..512) for a launch of its own


def _rows(n, width, alpha, rng):
    """n strings of up to `width` letters out of `alpha`: many ties and duplicates."""
    rows = np.zeros((n, width + 1), dtype=np.uint8)
    rows[:, :width] = rng.integers(97, 97 + alpha, size=(n, width))
    cut = rng.integers(width // 2, width + 1, size=n)
    rows[np.arange(width + 1)[None, :] >= cut[:, None]] = 0
    arena = np.concatenate([rows.ravel(), np.zeros(16, np.uint8)])
    return arena, np.arange(n, dtype=np.uint64) * (width + 1)


def _check_batch(sorter, arena, offs, sizes):
    inst = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
    p, l = sorter.sort_batch_host(arena, offs, inst)
    st = sorter.stats()
    for a, b in zip(inst[:-1], inst[1:]):
        rp, rl = pyoracle.oracle_sort(arena, offs[a:b])
        assert np.array_equal(p[a:b], rp) and np.array_equal(l[a:b], rl), int(b - a)
    return st


@pytest.mark.parametrize("alpha", [2, 26])
def test_class_edges_in_one_launch(sorter, alpha):
    rng = np.random.default_rng(alpha)
    sizes = list(EDGES) * 3
    st = _check_batch(sorter, *_rows(sum(sizes), 18, alpha, rng), sizes)
    assert st.block_fresh >= sum(s for s in sizes if s > 256)
    assert st.partitioned == 0


@pytest.mark.parametrize("cls", [0, 1, 2])
def test_class_edges_in_launches_of_their_own(sorter, cls):
    rng = np.random.default_rng(40 + cls)
    lo, hi = (257, 512) if cls == 0 else (256 << cls, (512 << cls))
    lo += cls > 0
    sizes = [(lo, hi - 1, hi)[i % 3] for i in range((CLASS_MIN_SEGS >> cls) + 1)]
    st = _check_batch(sorter, *_rows(sum(sizes), 18, 3, rng), sizes)
    assert st.block_fresh >= sum(sizes) and st.partitioned == 0


def _tied_runs(size, run, rng):
    """`size` strings: distinct heads of three bytes that use all eight bits, and
    among them four (fewer if they do not fit) heads shared by `run` strings that
    differ in bytes 10 and 11 only."""
    heads = rng.integers(1, 256, size=(size, 3), dtype=np.uint8)
    strings = [bytes(h) + b"mmmmmmm" for h in heads]
    at = rng.permutation(size)
    for g in range(min(4, size // (run + 8))):
        for j in at[g * run:(g + 1) * run]:
            strings[j] = bytes(heads[at[g * run]]) + b"mmmmmmm" + \
                bytes(rng.integers(1, 256, size=2, dtype=np.uint8))
    return strings


@pytest.mark.parametrize("run", [2, 3, 11, 12, 13, 14, 63, 64, 65, 66])
def test_tied_run_lengths(sorter, run):
    """Runs that tie on the packed bits and are out of order: put in order in
    place up to 12 records, by a second sort past that, which counts as a full
    one past 64.  In the one-CTA sort, and in the sorts of a batch."""
    rng = np.random.default_rng(run)
    sizes = [100, 250, 256, 300, 512, 700, 1024, 1500, 2048]
    if run > 20:
        sizes[0] = 200
    all_strings = []
    for n in sizes:
        strings = _tied_runs(n, run, rng)
        all_strings += strings
        arena, offs = cases.arena_of(strings)
        p, l = sorter.sort_host(arena, offs)
        rp, rl = pyoracle.oracle_sort(arena, offs)
        assert np.array_equal(p, rp) and np.array_equal(l, rl), n
        assert sorter.stats().full_sorted == (n if run > 64 else 0), n
    st = _check_batch(sorter, *cases.arena_of(all_strings), sizes)
    assert st.full_sorted == (sum(sizes) if run > 64 else 0)


@pytest.mark.parametrize("groups,per,shared,left", [
    (128, 2, 20, False), (129, 2, 20, True),    # the most segments of a round it keeps
    (8, 20, 400, False), (9, 20, 400, True),    # deep runs: as many as it has warps
    (32, 8, 400, False), (33, 8, 400, True),    # four runs of up to 8 strings to a warp
])
def test_what_the_one_cta_sort_leaves_to_the_general_loop(groups, per, shared, left):
    """Shown by the general loop's first launch, which a sort that ends in the
    one-CTA kernel does not have."""
    rng = np.random.default_rng(groups + per)
    strings = []
    for _ in range(groups):
        s = bytes(rng.integers(97, 123, size=shared, dtype=np.uint8))
        strings += [s + bytes([97 + j]) for j in rng.permutation(per)]
    arena, offs = cases.arena_of(strings)
    with pyssort.Sorter(0) as s:
        s.set_profiling(True)
        p, l = s.sort_host(arena, offs)
        times = s.kernel_times()
    rp, rl = pyoracle.oracle_sort(arena, offs)
    assert np.array_equal(p, rp) and np.array_equal(l, rl)
    assert "tiny" in times
    assert ("classify" in times) == left, sorted(times)
