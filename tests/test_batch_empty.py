"""Batches whose instance table holds long stretches of empty instances: the
results, and the time, which must not grow by a chain of reads over them."""
import numpy as np
import pytest

import pyoracle
import pyssort

pytestmark = pytest.mark.gpu

N = 60_000


def _table(sizes):
    return np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)


@pytest.mark.parametrize("kind", ["ends", "middle", "between", "every_step"])
def test_results(sorter, kind):
    """Empty instances first, last, in the middle, between instances of one or
    two strings, and distances of 0 to 70 instances between neighbours."""
    ss = pyssort.gen_uniform(N, 1, 12, ord("a"), 3, 81)
    rng = np.random.default_rng(82)
    if kind == "ends":
        sizes = [0] * 5000 + [N - 400, 400] + [0] * 5000
    elif kind == "middle":
        sizes = [N // 2 - 1] + [0] * 100_000 + [1, N - N // 2]
    elif kind == "between":
        sizes = np.zeros(200_000, np.int64)
        sizes[np.sort(rng.choice(200_000, N // 3, replace=False))] = 1
        sizes[sizes == 1] += np.arange(N // 3) % 2
        sizes[-1] += N - sizes.sum()
    else:
        sizes = []
        for d in range(71):
            sizes += [0] * d + [1 + d % 5]
        sizes.append(N - sum(sizes))
    inst = _table(sizes)
    assert inst[-1] == N
    p, l = sorter.sort_batch_host(ss.arena, ss.offs, inst)
    full = np.flatnonzero(np.diff(inst.astype(np.int64)) > 2)
    for i in full:
        a, b = int(inst[i]), int(inst[i + 1])
        rp, rl = pyoracle.oracle_sort(ss.arena, ss.offs[a:b])
        assert np.array_equal(p[a:b], rp) and np.array_equal(l[a:b], rl), i
    # every index lies in its own instance
    size = np.repeat(np.diff(inst.astype(np.int64)), np.diff(inst.astype(np.int64)))
    assert (p < size).all()
    first = np.repeat(inst[:-1].astype(np.int64), np.diff(inst.astype(np.int64)))
    assert np.array_equal(np.sort(first + p), np.arange(N))


def test_time_does_not_follow_the_empty_instances():
    """Half a million empty instances between two halves: some 40 table reads and
    a few microseconds more, not one read after the other (50 ms)."""
    torch = pytest.importorskip("torch")
    ss = pyssort.gen_uniform(N, 1, 12, ord("a"), 26, 83)
    A = torch.from_numpy(ss.arena).cuda()
    O = torch.from_numpy(ss.offs.view(np.int64)).cuda()
    p = torch.empty(N, dtype=torch.int32, device="cuda")
    l = torch.empty_like(p)
    best = []
    with pyssort.Sorter(0) as s:
        for empties in (0, 500_000):
            inst = _table([N // 2] + [0] * empties + [N - N // 2])
            I = torch.from_numpy(inst.view(np.int32)).cuda()
            ms = []
            for _ in range(7):
                s.sort_batch_device(A, A.numel(), O, 8, N, I, len(inst) - 1, p, l)
                ms.append(s.stats().device_ms)
            best.append(min(ms))
    assert best[1] < 10 * best[0], best
