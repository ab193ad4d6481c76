"""The one-CTA sort of small inputs (at most 2048 strings): rounds run inside
the kernel, rounds handed over to the general loop (many segments, deep
prefixes), and the counters it reports."""
import numpy as np
import pytest

import cases
import pyoracle
import pyssort

pytestmark = pytest.mark.gpu


def _check(sorter, strings):
    arena, offs = cases.arena_of(strings)
    p, l = sorter.sort_host(arena, offs)
    rp, rl = pyoracle.oracle_sort(arena, offs)
    assert np.array_equal(p, rp)
    assert np.array_equal(l, rl)
    return sorter.stats()


@pytest.mark.parametrize("n", [1, 2, 8, 9, 32, 33, 256, 257, 2047, 2048])
def test_sizes(sorter, n):
    rng = np.random.default_rng(n)
    st = _check(sorter, [bytes(rng.integers(97, 99, size=rng.integers(0, 40)).tolist())
                         for _ in range(n)])
    assert st.partitioned == 0
    if n >= 2:
        assert st.live[0] == n and st.rounds >= 1


def test_many_runs_go_on_in_the_general_loop(sorter):
    """1000 pairs that share 600 bytes: more next-round segments than the CTA
    keeps (in-warp refinement resolves them there)."""
    rng = np.random.default_rng(3)
    strings = []
    for _ in range(1000):
        s = bytes(rng.integers(97, 123, size=600).tolist())
        strings += [s + b"b", s + b"a"]
    st = _check(sorter, strings)
    assert st.rounds == 2 or st.warp1_deep > 0


@pytest.mark.parametrize("copies,length", [(40, 1500), (300, 1500), (40, 5000), (300, 5000)])
def test_deep_equal_runs(sorter, copies, length):
    """Runs of more than 32 equal strings take one round per 16 bytes: within the
    kernel's rounds (1500 bytes) and past them (5000 bytes)."""
    st = _check(sorter, [b"x" * length] * copies + [b"x" * (length - 1) + b"y", b"x", b""])
    assert st.rounds >= length // 16


def test_repeated_and_interleaved_contexts():
    """Counters of one sort do not leak into the next, nor between contexts."""
    rng = np.random.default_rng(9)
    sets = [[bytes(rng.integers(97, 100, size=rng.integers(1, 50)).tolist()) for _ in range(n)]
            for n in (5, 2000, 700, 30_000, 12)]
    with pyssort.Sorter(0) as a, pyssort.Sorter(0) as b:
        for k in range(3):
            for s in sets:
                sa, sb = _check(a, s), _check(b, s[::-1])
                assert sa.live[0] == sb.live[0] == len(s)
                assert sa.rounds == sb.rounds


@pytest.mark.parametrize("n", [4096, 4097, 8191, 9215, 9217])
def test_separate_gather(n):
    """The key gather as a kernel of its own at the edges of its 4096-string
    tiles and 1024-string steps, two rounds deep."""
    rng = np.random.default_rng(n)
    strings = [bytes(rng.integers(97, 99, size=rng.integers(0, 24)).tolist()) for _ in range(n)]
    with pyssort.Sorter(0) as s:
        s.set_param(pyssort.SSORT_PARAM_FUSED_GATHER, 0)
        st = _check(s, strings)
    assert st.gather_fused == 0 and st.partitioned > 0


@pytest.mark.parametrize("graph", [0, 1])
def test_batch_with_separate_gather(graph):
    """Large instances whose indices the first level counts, beside small ones
    that read them: several starts, tile remainders and empty instances."""
    rng = np.random.default_rng(17)
    sizes = [5000, 0, 1, 4097, 300, 9217, 2, 2049, 0, 2048, 33]
    inst = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
    strings = [bytes(rng.integers(97, 99, size=rng.integers(0, 24)).tolist())
               for _ in range(int(inst[-1]))]
    arena, offs = cases.arena_of(strings)
    with pyssort.Sorter(0) as s:
        s.set_param(pyssort.SSORT_PARAM_FUSED_GATHER, 0)
        s.set_param(pyssort.SSORT_PARAM_GRAPH, graph)
        p, l = s.sort_batch_host(arena, offs, inst)
    for a, b in zip(inst[:-1], inst[1:]):
        if a == b:
            continue
        rp, rl = pyoracle.oracle_sort(arena, offs[a:b])
        assert np.array_equal(p[a:b], rp) and np.array_equal(l[a:b], rl)
