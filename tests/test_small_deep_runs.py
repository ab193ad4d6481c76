"""Sorts of at most 2048 strings with many runs that stay equal for long: the
one-CTA sort refines a crowded round (more runs than it has warps) for a few
steps and leaves what is still crowded after it to the general loop."""
import numpy as np
import pytest

import cases
import pyoracle
import pyssort

pytestmark = pytest.mark.gpu


def _groups(groups, per, shared, seed):
    """`per` strings in each of `groups` groups that share `shared` random bytes,
    in random order."""
    rng = np.random.default_rng(seed)
    strings = []
    for _ in range(groups):
        base = bytes(rng.integers(97, 123, size=shared, dtype=np.uint8))
        strings += [base + bytes(rng.integers(97, 123, size=int(rng.integers(0, 9)),
                                              dtype=np.uint8)) for _ in range(per)]
    return [strings[i] for i in rng.permutation(len(strings))]


# runs of up to 8 strings (four to a warp) and of 9 to 32, around 8 warps' worth
# of them, and the most segments the kernel keeps
@pytest.mark.parametrize("groups,per", [(8, 8), (32, 8), (33, 8), (33, 4), (128, 3), (128, 8),
                                        (8, 9), (9, 9), (8, 32), (9, 32), (64, 32), (100, 20),
                                        (128, 16)])
@pytest.mark.parametrize("shared", [30, 50, 400])
@pytest.mark.parametrize("deep", [0, 1, 256])
def test_results(groups, per, shared, deep):
    arena, offs = cases.arena_of(_groups(groups, per, shared, groups * per + shared))
    with pyssort.Sorter(0) as s:
        s.set_param(pyssort.SSORT_PARAM_WARP1_DEEP, deep)
        p, l = s.sort_host(arena, offs)
        st = s.stats()
    rp, rl = pyoracle.oracle_sort(arena, offs)
    assert np.array_equal(p, rp) and np.array_equal(l, rl)
    assert st.live[0] == groups * per and st.partitioned == 0


@pytest.mark.parametrize("groups,per", [(128, 16), (128, 3), (60, 8), (100, 20)])
def test_no_slower_than_the_general_loop(groups, per):
    """The same strings among enough others that the general loop sorts them."""
    torch = pytest.importorskip("torch")
    strings = _groups(groups, per, 1000, 5)
    rng = np.random.default_rng(6)
    others = [bytes(rng.integers(97, 123, size=10, dtype=np.uint8))
              for _ in range(2049 - len(strings))]
    best = []
    with pyssort.Sorter(0) as s:
        for ss in (strings, strings + others):
            arena, offs = cases.arena_of(ss)
            A = torch.from_numpy(arena).cuda()
            O = torch.from_numpy(offs.astype(np.int64)).cuda()
            p = torch.empty(len(ss), dtype=torch.int32, device="cuda")
            ms = []
            for _ in range(9):
                s.sort_device(A, A.numel(), O, 8, len(ss), p, None)
                ms.append(s.stats().device_ms)
            best.append(min(ms))
    assert best[0] < 1.5 * best[1], best
