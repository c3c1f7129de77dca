"""Trees and queries that take the refit's and the point walk's less usual paths: CTAs that take several
subtrees each, and node queues that fill up and go on node by node."""
import numpy as np
import pytest

import oracle_py as O
from mguso import lbvh

pytestmark = pytest.mark.gpu


def points_as_triangles(c):
    """One triangle of three equal corners per point: its box is the point."""
    c = np.ascontiguousarray(c, np.float32)
    return np.repeat(c, 3, 0), np.arange(3 * len(c), dtype=np.uint32).reshape(-1, 3)


def subtrees(left, right, limit=256):
    """The refit's subtrees of a tree of more than `limit` leaves: the largest with at most that many."""
    count, roots = {}, 0
    order, stack = [], [0]
    while stack:
        n = stack.pop()
        order.append(n)
        stack += [int(c) for c in (left[n], right[n]) if not c >> 31]
    for n in reversed(order):
        count[n] = sum(1 if c >> 31 else count[int(c)] for c in (left[n], right[n]))
    for n in order:
        if count[n] > limit:
            roots += sum(1 for c in (left[n], right[n]) if c >> 31 or count[int(c)] <= limit)
    return roots


@pytest.mark.parametrize("combs", [1, 3])
def test_more_subtrees_than_ctas(ctx, combs):
    """256 primitives at the corner of the box and one at every halving of each axis towards it: every
    level of the tree above the 256 sheds one leaf, so there are ten times as many subtrees as
    CTAs (one for 64 leaves)."""
    import torch
    step = np.concatenate([np.float32(2.0) ** -np.arange(21, dtype=np.float32)[:, None, None] * np.eye(3, dtype=np.float32)])
    c = np.concatenate([np.zeros((256, 3), np.float32)] + [step.reshape(-1, 3)] * combs)
    c = c[np.random.default_rng(1).permutation(len(c))]
    pos, tris = points_as_triangles(c)
    n = len(c)
    b = lbvh.Lbvh(ctx)
    pd, td = torch.from_numpy(pos).cuda(), torch.from_numpy(tris.astype(np.int32)).cuda()
    b.build(pd.data_ptr(), pos.shape[0], td.data_ptr(), n, 63, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    keys, perm, left, right, node = b.download()
    assert subtrees(left, right) > -(-n // 64)
    ok, op, ol, orr, on, _ = O.lbvh(pos, tris, 63, 1e-3, cap=1)
    assert np.array_equal(keys, ok) and np.array_equal(perm, op)
    assert np.array_equal(left, ol) and np.array_equal(right, orr) and np.array_equal(node, on)


def test_full_queues_of_full_warps(ctx):
    """Enough points for 32 of them a warp (16 warps on each of 148 SMs), each of which meets all of 300
    primitives with equal codes and none of the other 99 700: a warp's queue grows by 32 nodes a level of
    a tree 9 levels deep from where the runs begin, past the 256 after which it takes one node at a time."""
    import torch
    rng = np.random.default_rng(3)
    far = rng.random((99700, 3), dtype=np.float32) * np.float32(0.5) + np.float32(0.5)
    near = np.zeros((300, 3), np.float32)
    c = np.concatenate([far, near])
    p = rng.permutation(len(c))
    pos, tris = points_as_triangles(c[p])
    hot = torch.from_numpy(np.sort(np.flatnonzero(p >= len(far)))).cuda()
    npts = 16 * 148 * 32 + 5
    pts = torch.from_numpy(rng.random((npts, 3), dtype=np.float32) * np.float32(0.01)).cuda()
    b = lbvh.Lbvh(ctx)
    s = torch.cuda.current_stream().cuda_stream
    pd, td = torch.from_numpy(pos).cuda(), torch.from_numpy(tris.astype(np.int32)).cuda()
    b.build(pd.data_ptr(), pos.shape[0], td.data_ptr(), len(c), 63, s)
    cap = npts * len(near)
    buf = torch.full((cap, 2), -1, dtype=torch.int32, device="cuda")
    cnt = torch.zeros(1, dtype=torch.int64, device="cuda")
    b.query_points(pts.data_ptr(), npts, 0.05, buf.data_ptr(), cap, cnt.data_ptr(), s)
    torch.cuda.synchronize()
    assert b.status() == 0 and int(cnt.item()) == cap
    q, t = buf[:, 0].long(), torch.searchsorted(hot, buf[:, 1].long())
    assert torch.equal(hot[t.clamp(max=len(near) - 1)], buf[:, 1].long())
    assert torch.equal(torch.sort(q * len(near) + t).values, torch.arange(cap, device="cuda"))
