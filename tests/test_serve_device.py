"""The request server with requests in device memory (their copies run as one
launch): unaligned arenas, offsets of either width, outputs with and without
LCPs, mixed with host requests in one batch."""
import numpy as np
import pytest

import pyssort

pytestmark = pytest.mark.gpu


def test_device_and_host_requests_mixed(sorter):
    torch = pytest.importorskip("torch")
    params = pyssort.batch_instance_params(60, seed=91, lo=1, hi=60_000)
    ss = pyssort.gen_instances(params, seed=92)
    subs = []
    with pyssort.Server(256 << 20, 4_000_000) as srv:
        for i in range(len(params)):
            arena, offs = ss.request(i, (np.uint32, np.uint64)[i % 2])
            n, w = len(offs), offs.dtype.itemsize
            expect = sorter.sort_host(arena.copy(), offs)
            if i % 5 == 4:  # host request
                rid, perm, lcp = srv.submit(arena.copy(), offs)
                subs.append((perm, lcp, expect))
                continue
            skew = (0, 1, 4, 16)[i % 4]  # arena address not 16-byte aligned
            d_arena = torch.zeros(len(arena) + skew, dtype=torch.uint8, device="cuda")
            d_arena[skew:] = torch.from_numpy(arena.copy()).cuda()
            d_offs = torch.from_numpy(offs.view(np.int32 if w == 4 else np.int64)).cuda()
            perm = torch.full((n + 1,), -7, dtype=torch.int32, device="cuda")
            lcp = torch.full((n,), -7, dtype=torch.int32, device="cuda") if i % 3 else None
            torch.cuda.synchronize()
            srv.submit_ptr(d_arena[skew:], len(arena), d_offs, w, n, perm, lcp)
            subs.append((perm, lcp, expect))
        srv.drain()
    torch.cuda.synchronize()
    for perm, lcp, (ep, el) in subs:
        if isinstance(perm, np.ndarray):
            assert np.array_equal(perm, ep) and np.array_equal(lcp, el)
            continue
        got = perm.cpu().numpy()
        assert got[-1] == -7  # nothing past the result
        assert np.array_equal(got[:-1].view(np.uint32), ep)
        if lcp is not None:
            assert np.array_equal(lcp.cpu().numpy().view(np.uint32), el)
