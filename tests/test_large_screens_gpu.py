"""Sizes at which the constructions and the ground truth work in parts: columns of the
range screen in more than one chunk, row blocks of the k-NN screen in more than one
launch, more queries than a batch holds, more in-neighbours than a list in shared
memory. Compared with float64 sums over all pairs."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _nearest(x, q, k, chunk=100_000):
    """(ids, squared distances) of the k rows of x (device) nearest each row of q."""
    import torch
    dist = torch.full((q.shape[0], 0), 0.0, dtype=torch.float64, device=x.device)
    ids = torch.zeros((q.shape[0], 0), dtype=torch.int64, device=x.device)
    for r0 in range(0, x.shape[0], chunk):
        rows = x[r0:r0 + chunk].double()
        d = torch.stack([(rows - v.double()).square().sum(1) for v in q])
        dist = torch.cat([dist, d], 1)
        ids = torch.cat([ids, torch.arange(r0, r0 + rows.shape[0], device=x.device).expand(q.shape[0], -1)], 1)
        dist, at = dist.topk(min(k, dist.shape[1]), dim=1, largest=False)
        ids = ids.gather(1, at)
    return ids.cpu().numpy(), dist.cpu().numpy()


def test_ground_truth_with_more_than_one_chunk_of_columns():
    """1,690,000 x 256: an operand chunk holds 1,677,696 columns, the last is partly
    filled. The entry lists the answers, so the search's bounds are tight and the
    screen's lists decide."""
    import torch
    from parallel_anns_b200.formats import NSGGraph
    from parallel_anns_b200.searching import Index, ground_truth
    n, d, nq, k = 1_690_000, 256, 70, 10
    gen = torch.Generator(device="cuda").manual_seed(5)
    xt = torch.rand((n, d), generator=gen, device="cuda")
    qt = torch.rand((nq, d), generator=gen, device="cuda")
    ids, dist = _nearest(xt, qt, k)
    x, q = xt.cpu().numpy(), qt.cpu().numpy()
    del xt
    torch.cuda.empty_cache()
    first = np.unique(ids)
    first = first[first != 0]
    off = np.arange(n + 1, dtype=np.int64)
    off[1:] += first.size - 1
    nbrs = np.concatenate([first, (np.arange(1, n) + 1) % n]).astype(np.uint32)
    with Index(0) as ix:
        ix.set_base(x)
        ix.set_graph(NSGGraph(int(first.size), 0, off, nbrs))
        got, gdist = ground_truth(ix, q, k)
    assert np.array_equal(got, ids)
    np.testing.assert_allclose(gdist, dist, rtol=(d + 2) * 2.0 ** -52, atol=0)


def test_build_with_more_than_one_launch_of_row_blocks():
    """2,200,000 x 8: more than 16,384 tiles, so their bounds are made and their row
    blocks screened a part at a time."""
    import torch
    from parallel_anns_b200.graph import build_nsg
    n, d, k = 2_200_000, 8, 8
    x = np.random.default_rng(6).random((n, d), dtype=np.float32)
    _, knn = build_nsg(x, R=6, knn_k=k, with_knn=True)
    assert knn.max() < n and (knn != np.arange(n)[:, None]).all()
    rows = np.random.default_rng(7).permutation(n)[:300]
    xt = torch.from_numpy(x).cuda()
    ids, _ = _nearest(xt, xt[torch.from_numpy(rows).cuda()], k + 1)
    for i, a in enumerate(rows):
        assert np.array_equal(knn[a], ids[i][ids[i] != a][:k]), a


def test_ground_truth_with_more_than_one_batch_of_queries():
    """16,384 queries go through the screen at a time."""
    from parallel_anns_b200.graph import build_nsg
    from parallel_anns_b200.searching import Index, ground_truth
    rng = np.random.default_rng(8)
    x, q = rng.random((5000, 16), dtype=np.float32), rng.random((16_500, 16), dtype=np.float32)
    with Index(0) as ix:
        ix.set_base(x)
        ix.set_graph(build_nsg(x, R=16, knn_k=24))
        ids, dist = ground_truth(ix, q, 10)
    oids, odist = O.ground_truth(x, q, 10)
    assert np.array_equal(ids, oids)
    np.testing.assert_allclose(dist, odist, rtol=18 * 2.0 ** -52, atol=0)


@pytest.mark.parametrize("n", [700, 1500])
def test_reverse_edges_of_a_hub(n):
    """Rows on a sphere, one at its centre and one near that: most lists are pruned to
    the centre, whose in-neighbours pass the 256 that are ranked at once. Every list
    is its pruned one, then the smallest ids of its in-neighbours that it lacks."""
    from parallel_anns_b200.graph import build_nsg_cells
    rng = np.random.default_rng(n)
    k = R = 16
    x = rng.standard_normal((n, 64)).astype(np.float32)
    x /= np.linalg.norm(x, axis=1, keepdims=True)
    x[300], x[301] = 0.0, 0.1 * x[301]
    g, knn = build_nsg_cells(x, R=R, knn_k=k, cells=1, probe=0, sample=n, iters=1, reverse=True, with_knn=True)
    z = x.astype(np.float64)
    pruned, into = [], [[] for _ in range(n)]
    for a in range(n):
        kept = []
        for b in knn[a]:
            if not kept or np.square(z[kept] - z[b]).sum(1).min() >= np.square(z[a] - z[b]).sum():
                kept.append(int(b))
        pruned.append(kept)
        for b in kept:
            into[b].append(a)
    assert len(into[300]) > 256 and len(pruned[300]) < R
    for b in range(n):
        want = pruned[b] + [a for a in into[b] if a not in pruned[b]][:R - len(pruned[b])]
        assert g.nbrs[g.offsets[b]:g.offsets[b + 1]][:len(want)].tolist() == want, b
