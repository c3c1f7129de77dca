"""The tree's records at the edges of the refit's 256-leaf blocks, and the point queries' shared
walk at the edges of a warp, against the CPU oracle: whole numbers and boxes bit-exact."""
import numpy as np
import pytest

import oracle_py as O
from mguso import lbvh, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt", [1, 2, 3, 255, 256, 257, 511, 513, 4097])
@pytest.mark.parametrize("bits", [30, 63])
def test_records_at_block_edges(ctx, nt, bits):
    import torch
    b = lbvh.Lbvh(ctx)
    for seed, n in ((1, 3 * nt), (2, nt)):  # a larger tree first: the second finds its leftovers
        pos, tris = scenes.triangle_soup(n, seed=seed)
        if seed == 2:
            pos[: 3 * (nt // 2)] = pos[:3].repeat((nt // 2), 0).reshape(-1, 3)[: 3 * (nt // 2)]  # equal codes: a deep tree
        pd, td = torch.from_numpy(pos).cuda(), torch.from_numpy(tris.astype(np.int32)).cuda()
        b.build(pd.data_ptr(), pos.shape[0], td.data_ptr(), n, bits, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        keys, perm, left, right, node = b.download()
        ok, op, ol, orr, on, _ = O.lbvh(pos, tris, bits, 1e-3, cap=1)
        assert np.array_equal(keys, ok) and np.array_equal(perm, op)
        if n > 1:
            assert np.array_equal(left, ol) and np.array_equal(right, orr) and np.array_equal(node, on)


@pytest.mark.parametrize("npts", [1, 3, 4, 31, 33, 127, 129, 9473])
@pytest.mark.parametrize("offset", [0, 1])  # a pair buffer on 8 and on 4 bytes
def test_point_queries_at_warp_edges(ctx, npts, offset):
    import torch
    pos, tris = scenes.triangle_soup(3000, seed=7)
    rng = np.random.default_rng(npts)
    lo, hi = pos.min(0), pos.max(0)
    pts = (lo + (hi - lo) * rng.random((npts, 3), dtype=np.float32)).astype(np.float32)
    if npts > 3:
        pts[1] = np.nan
        pts[2, 0] = np.inf
    dhat = np.float32(0.05)
    tb = pos[tris]
    blo, bhi = tb.min(1), tb.max(1)
    want = []
    for p in range(npts):  # the box test itself, in 32 bits
        ql, qh = pts[p] - dhat, pts[p] + dhat
        hit = np.all((ql <= bhi) & (blo <= qh), axis=1)
        want += [(p, int(t)) for t in np.flatnonzero(hit)]
    b = lbvh.Lbvh(ctx)
    s = torch.cuda.current_stream().cuda_stream
    pd, td, qd = (torch.from_numpy(a).cuda() for a in (pos, tris.astype(np.int32), pts))
    b.build(pd.data_ptr(), pos.shape[0], td.data_ptr(), tris.shape[0], 30, s)
    cap = len(want) + 8
    buf = torch.full((2 * cap + 1 + offset,), -1, dtype=torch.int32, device="cuda")
    cnt = torch.zeros(1, dtype=torch.int64, device="cuda")
    b.query_points(qd.data_ptr(), npts, float(dhat), buf[offset:].data_ptr(), cap, cnt.data_ptr(), s)
    torch.cuda.synchronize()
    assert b.status() == 0 and int(cnt.item()) == len(want)
    got = buf[offset:offset + 2 * len(want)].cpu().numpy().reshape(-1, 2)
    assert sorted(map(tuple, got.tolist())) == sorted(want)


@pytest.mark.parametrize("nt,npts", [(2, 40), (500, 33), (3000, 64)])
def test_queries_that_meet_everything(ctx, nt, npts):
    """Every point meets every triangle, so the walks' node queues fill up and go on node by node."""
    pos, tris = scenes.triangle_soup(nt, seed=11)
    pts = np.concatenate([pos, pos])[:npts] if pos.shape[0] >= npts else np.resize(pos, (npts, 3))
    import torch
    b = lbvh.Lbvh(ctx)
    s = torch.cuda.current_stream().cuda_stream
    pd, td, qd = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (pos, tris.astype(np.int32), pts))
    b.build(pd.data_ptr(), pos.shape[0], td.data_ptr(), nt, 30, s)
    cap = nt * npts
    buf = torch.full((cap, 2), -1, dtype=torch.int32, device="cuda")
    cnt = torch.zeros(1, dtype=torch.int64, device="cuda")
    b.query_points(qd.data_ptr(), npts, 10.0, buf.data_ptr(), cap, cnt.data_ptr(), s)
    torch.cuda.synchronize()
    assert b.status() == 0 and int(cnt.item()) == cap
    key = buf.cpu().numpy().astype(np.int64)
    assert np.array_equal(np.sort(key[:, 0] * nt + key[:, 1]), np.arange(cap))
