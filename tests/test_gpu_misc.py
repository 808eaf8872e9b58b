"""Batched ALS solve, k-means, top-k merge, Gram and the one-launch all-reduce on one GPU."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [8, 32, 50, 128])
def test_als_batched_solve_matches_numpy(k):
    from paracel_b200.ops.als import als_solve
    dev = "cuda:0"
    g = torch.Generator(device=dev).manual_seed(k)
    ni, nu = 500, 300
    H = torch.randn(ni, k, device=dev, generator=g)
    cnt = torch.randint(1, 40, (nu,), device=dev, generator=g)
    cnt[0] = 0                      # a user without ratings keeps a zero factor
    cnt[5] = 9000                   # a heavy user is split over several CTAs
    ptr = torch.zeros(nu + 1, dtype=torch.int64, device=dev)
    ptr[1:] = torch.cumsum(cnt, 0)
    nnz = int(ptr[-1])
    idx = torch.randint(0, ni, (nnz,), device=dev, generator=g).int()
    r = torch.randn(nnz, device=dev, generator=g)
    lam = 0.5
    W = als_solve(ptr, idx, r, H, lam, seg_len=1024)
    torch.cuda.synchronize()
    Hn, pn, idn, rn = H.double().cpu().numpy(), ptr.cpu().numpy(), idx.cpu().numpy(), r.double().cpu().numpy()
    for u in (0, 1, 5, 77, 299):
        Hs = Hn[idn[pn[u]:pn[u + 1]]]
        if Hs.shape[0] == 0:
            assert float(W[u].abs().sum()) == 0.0
            continue
        ref = np.linalg.solve(Hs.T @ Hs + lam * np.eye(k), Hs.T @ rn[pn[u]:pn[u + 1]])
        assert np.allclose(W[u].cpu().numpy(), ref, rtol=2e-3, atol=2e-4), u


def test_kmeans_gpu_matches_numpy_lloyd():
    from paracel_b200.models.kmeans_gpu import KMeansGpu
    dev = "cuda:0"
    g = torch.Generator(device=dev).manual_seed(7)
    k, d, n = 16, 10, 6000
    C0 = 6 * torch.randn(k, d, device=dev, generator=g)
    lab = torch.randint(0, k, (n,), device=dev, generator=g)
    X = C0[lab] + 0.5 * torch.randn(n, d, device=dev, generator=g)
    m = KMeansGpu(k, d, device=dev)
    m.load(X)
    m.fit(6)
    C = m.cluster_centres().double().cpu().numpy()
    Xn = X.double().cpu().numpy()
    Cr = Xn[:k].copy()
    for _ in range(6):
        a = ((Cr * Cr).sum(1)[None, :] - 2 * Xn @ Cr.T).argmin(1)
        for c in range(k):
            if (a == c).any():
                Cr[c] = Xn[a == c].mean(0)
    assert np.allclose(C, Cr, rtol=1e-3, atol=1e-3)
    m.free()


@pytest.mark.parametrize("n,d,k", [(5003, 128, 37), (4001, 64, 5), (3000, 256, 100), (2500, 512, 9),
                                   (3001, 10, 7), (2000, 516, 3), (3, 128, 2)])
def test_kmeans_accumulate_matches_index_add(n, d, k):
    """Per-cluster sums and counts (vector-reduction kernel for d % 4 == 0 and d <= 512, the scalar
    kernel otherwise) against a plain fp64 index_add."""
    from paracel_b200.ops.misc import kmeans_accumulate
    g = torch.Generator(device="cuda").manual_seed(n + d)
    X = torch.randn(n, d, device="cuda", generator=g)
    assign = torch.randint(0, k, (n,), device="cuda", generator=g, dtype=torch.int32)
    sums = torch.zeros(k, d, device="cuda")
    counts = torch.zeros(k, device="cuda")
    kmeans_accumulate(X, assign, sums, counts)
    ref = torch.zeros(k, d, device="cuda", dtype=torch.float64).index_add_(0, assign.long(), X.double())
    cnt = torch.bincount(assign.long(), minlength=k).double()
    assert torch.equal(counts.double(), cnt)
    assert (sums.double() - ref).abs().max().item() < 1e-3


@pytest.mark.parametrize("rows,width,n", [(1000, 128, 3001), (77, 4, 5), (5000, 64, 2500), (300, 200, 1237),
                                          (4096, 512, 700)])
def test_row_table_pull_push_match_torch(rows, width, n):
    """Keyed pull (with snapshot) and the add / scaled_add / max / assign pushes of a row table
    against plain PyTorch indexing in fp64; ids repeat, so pushes to one row accumulate."""
    from paracel_b200.ps.tables import RowTable
    g = torch.Generator(device="cuda").manual_seed(rows + width)
    t = RowTable(rows, width)
    ref = torch.randn(rows, width, device="cuda", generator=g)
    t.shard[:rows] = ref
    ids = torch.randint(0, rows, (n,), device="cuda", generator=g)
    out = torch.empty(n, width, device="cuda")
    snap = torch.empty(n, width, device="cuda")
    t.pull(ids, out, snap)
    t.check()
    assert torch.equal(out, ref[ids]) and torch.equal(snap, ref[ids])
    # add with per-row weights: table += w * (cur - old); old is refreshed to cur
    cur = out + torch.randn(n, width, device="cuda", generator=g)
    w = torch.rand(n, device="cuda", generator=g)
    exp = ref.double().index_add_(0, ids, (cur - snap).double() * w.double()[:, None])
    t.push(ids, cur, snap, w, handler="add", start=n // 3)
    t.check()
    assert (t.shard[:rows].double() - exp).abs().max().item() < 1e-4
    assert torch.equal(snap, cur)
    # scaled add without snapshot: table += scale * cur
    exp = t.shard[:rows].double().index_add_(0, ids, 0.25 * cur.double())
    t.push(ids, cur, None, None, handler="scaled_add", scale=0.25)
    t.check()
    assert (t.shard[:rows].double() - exp).abs().max().item() < 1e-4
    # max
    before = t.shard[:rows].clone()
    exp = before.clone().index_reduce_(0, ids, cur, "amax", include_self=True)
    t.push(ids, cur, None, None, handler="max")
    t.check()
    assert torch.equal(t.shard[:rows], exp)
    # assign on distinct ids
    uids = torch.randperm(rows, device="cuda", generator=g)[: min(rows, n)]
    vals = torch.randn(uids.numel(), width, device="cuda", generator=g)
    t.push(uids, vals, None, None, handler="assign")
    t.check()
    assert torch.equal(t.shard[:rows][uids], vals)
    t.free()


def test_running_topk_and_gram():
    from paracel_b200.ops.misc import RunningTopK, gram
    dev = "cuda:0"
    g = torch.Generator(device=dev).manual_seed(9)
    m, n, k = 300, 1000, 7
    S = torch.randn(m, n, device=dev, generator=g)
    row_ids = torch.arange(m, device=dev) * 3
    col_ids = torch.arange(n, device=dev)
    tk = RunningTopK(row_ids, k, lower=0.5)
    for c0 in range(0, n, 256):           # tiles arrive one after the other
        tk.update(S[:, c0:c0 + 256].contiguous(), col_ids[c0:c0 + 256])
    torch.cuda.synchronize()
    res = tk.result()
    Sm = S.clone()
    Sm[row_ids[:, None] == col_ids[None, :]] = -1e30   # self excluded
    for r in (0, 1, 150, 299):
        vals, idx = torch.topk(Sm[r], k)
        exp = [(int(i), float(v)) for v, i in zip(vals, idx) if v >= 0.5]
        got = res.get(int(row_ids[r]), [])
        assert [i for i, _ in got] == [i for i, _ in exp]
        assert np.allclose([v for _, v in got], [v for _, v in exp])
    H = torch.randn(5000, 50, device=dev, generator=g)
    G = gram(H)
    torch.cuda.synchronize()
    torch.testing.assert_close(G.double(), H.double().T @ H.double(), rtol=1e-4, atol=1e-2)


@pytest.mark.parametrize("n,pitch,k", [(1, 1, 1), (127, 127, 5), (128, 128, 32), (129, 132, 20), (511, 513, 7),
                                       (512, 512, 20), (513, 516, 20), (2051, 2052, 32), (1000, 1003, 1)])
def test_topk_rows_edges_and_ties_match_a_stable_sort(n, pitch, k):
    """Both row layouts (pitch a multiple of four floats or not) at the edges of the 128- and
    512-column steps.  Values are small integers, so most are tied: of equal values the earlier
    column wins, which a stable descending sort gives exactly; each row's own id is left out."""
    from paracel_b200.ops.misc import RunningTopK
    g = torch.Generator(device="cuda").manual_seed(n + pitch + k)
    m = 37
    S = torch.empty(m, pitch, device="cuda")[:, :n]
    S.copy_(torch.randint(-9, 10, (m, n), device="cuda", generator=g).float())
    col_ids = torch.arange(n, device="cuda") + 5
    row_ids = torch.arange(m, device="cuda") * 3
    tk = RunningTopK(row_ids, k, lower=-8.0)
    tk.update(S, col_ids)
    Sm = torch.where((col_ids[None, :] == row_ids[:, None]) | (S < -8.0), torch.full_like(S, -1e30), S)
    val, pos = torch.sort(Sm, dim=1, descending=True, stable=True)
    got = tk.result()
    for r in range(m):
        exp = [(int(col_ids[j]), float(x)) for x, j in zip(val[r, :k], pos[r, :k]) if x > -1e29]
        assert got.get(int(row_ids[r]), []) == exp


def test_device_allreduce_single_rank():
    from paracel_b200.ops.misc import DeviceAllReduce
    ar = DeviceAllReduce(device="cuda:0")
    x = torch.arange(10, dtype=torch.float64, device="cuda:0")
    for _ in range(3):
        y = ar(x)
    torch.cuda.synchronize()
    ar.check()
    assert torch.equal(x, y)
    ar.free()


def test_device_balltree_search_matches_host_tree_and_brute_force():
    import numpy as np
    from paracel_b200.tool.balltree import DeviceBalltree, PyBalltree, PyQuery, balltree_search_with_dp
    rng = np.random.default_rng(4)
    items = rng.standard_normal((6000, 24)) * rng.uniform(0.2, 2.0, (6000, 1))
    tree = PyBalltree(items)
    tree.build()
    dt = DeviceBalltree(tree)
    queries = rng.standard_normal((300, 24))
    k = 7
    idx, sc, vis = dt.search(queries, k)
    torch.cuda.synchronize()
    idx, sc, vis = idx.cpu().numpy(), sc.cpu().numpy(), vis.cpu().numpy()
    exact = (queries @ items.T)
    ref_idx = np.argsort(-exact, axis=1)[:, :k]
    ref_sc = np.take_along_axis(exact, ref_idx, axis=1)
    assert np.allclose(sc, ref_sc, rtol=1e-4, atol=1e-4)          # same scores as brute force
    assert (idx == ref_idx).mean() > 0.995                          # ids differ only on fp32 near-ties
    assert np.all(np.diff(sc, axis=1) <= 1e-6)                      # best first
    assert vis.min() > 0 and vis.max() < tree.node_count            # some balls were pruned
    host = balltree_search_with_dp(PyQuery(list(queries[0]), k), tree)
    assert [i for i, _ in host] == list(idx[0])
    assert abs(tree.last_visited - int(vis[0])) <= 0.05 * tree.last_visited   # same traversal
    # fewer items than k
    small = PyBalltree(items[:3])
    small.build()
    i2, s2, _ = DeviceBalltree(small).search(queries[:2], 5)
    assert (i2[:, 3:] == -1).all().item() and sorted(i2[0, :3].tolist()) == [0, 1, 2]


def _ragged_csr(n, cols, lens, g, weighted=True, lead=0):
    """CSR with the given row lengths; ``lead`` entries before the first row's."""
    ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(lens, 0)
    ptr += lead
    nnz = int(ptr[-1])
    idx = torch.randint(0, cols, (nnz,), device="cuda", generator=g, dtype=torch.int32)
    val = torch.randn(nnz, device="cuda", generator=g) if weighted else None
    return ptr, idx, val


@pytest.mark.parametrize("K", [4, 12, 32, 52, 64, 112, 128])
@pytest.mark.parametrize("shape", ["even", "empty_rows", "one_long_row", "offset_unaligned", "single"])
def test_csr_products_match_fp64(K, shape):
    """Both CSR products, cut by entries: rows cut by segment and block boundaries, runs of empty rows
    longer than a block's row cache, a row far longer than a block, row pointers that do not start at
    zero, arrays off the 16-byte grid.  A sum of n fp32 products is within n 2^-24 of the sum of
    their magnitudes."""
    from paracel_b200.ops.svd import spmm_csr, spmm_csr_t
    g = torch.Generator(device="cuda").manual_seed(K)
    n, N, lead = 3001, 501, 0
    lens = torch.randint(0, 40, (n,), device="cuda", generator=g)
    if shape == "empty_rows":
        n = 9000
        lens = torch.zeros(n, dtype=torch.int64, device="cuda")
        lens[torch.tensor([0, 5, 6, 3000, 3001, 8990], device="cuda")] = torch.tensor([3, 1, 700, 2, 129, 64], device="cuda")
    elif shape == "one_long_row":
        lens[17] = 70_003
    elif shape == "offset_unaligned":
        lead = 37
    elif shape == "single":
        n, lens = 1, torch.tensor([1], device="cuda")
    ptr, idx, val = _ragged_csr(n, N, lens, g, weighted=shape != "even", lead=lead)
    if shape == "offset_unaligned":
        idx, val, ptr = idx[1:], val[1:], ptr - 1
    H = torch.randn(N, K, device="cuda", generator=g)
    W = torch.randn(n, K, device="cuda", generator=g)
    out = spmm_csr(ptr, idx, val, H)
    back = torch.ones(N, K, device="cuda")
    spmm_csr_t(ptr, idx, val, W, back)
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), lens)
    a, b = int(ptr[0]), int(ptr[-1])
    c, v = idx[a:b].long(), torch.ones(b - a, device="cuda").double() if val is None else val[a:b].double()
    for got, dst, src, at, start in ((out, rows, H, c, 0.0), (back, c, W, rows, 1.0)):
        prod = v[:, None] * src.double()[at]
        ref = torch.full(got.shape, start, dtype=torch.float64, device="cuda").index_add_(0, dst, prod)
        mag = torch.full(got.shape, start, dtype=torch.float64, device="cuda").index_add_(0, dst, prod.abs())
        cnt = torch.bincount(dst, minlength=got.shape[0]).double()[:, None] + 2
        assert bool(((got.double() - ref).abs() <= cnt * 2.0 ** -24 * mag).all())


@pytest.mark.parametrize("k", [7, 18, 33, 50, 65, 100, 128])
def test_als_forms_match_fp64_at_their_edges(k):
    """Users on both sides of every form's limits (warp / CTA dual form, k x k form, split users)."""
    from paracel_b200.ops.als import als_solve
    g = torch.Generator(device="cuda").manual_seed(k)
    ni, lam = 700, 0.5
    cnt = [0, 1, 2, 15, 16, 17, 31, 32, 33, 63, 64, 65, 95, 96, 97, 128, 129, 300, 511, 512, 0, 1024, 1025, 2700, 3]
    cnt += [c for c in (k - 1, k, k + 1)]
    ptr = torch.tensor([0] + cnt).cumsum(0).cuda() + 5          # the arrays begin before the first user
    H = torch.randn(ni, k, device="cuda", generator=g)
    idx = torch.randint(0, ni, (int(ptr[-1]),), device="cuda", generator=g).int()
    r = torch.randn(int(ptr[-1]), device="cuda", generator=g)
    W = als_solve(ptr, idx, r, H, lam, seg_len=1024)
    W0 = als_solve(ptr, idx, r, H, 0.0, seg_len=1024)           # without lambda: the k x k form only
    for u, c in enumerate(cnt):
        a, b = int(ptr[u]), int(ptr[u + 1])
        Hs, rs = H[idx[a:b].long()].double(), r[a:b].double()
        if c == 0:
            assert not bool(W[u].any()) and not bool(W0[u].any())
            continue
        for got, l in ((W[u], lam), (W0[u], 0.0)):
            G = Hs.T @ Hs + l * torch.eye(k, device="cuda").double()
            if l == 0.0 and c < 2 * k:
                continue                                        # singular or nearly so
            ref = torch.linalg.solve(G, Hs.T @ rs)
            # backward error of the Gram sums and of the factorisation, both in fp32
            bound = 16 * 2.0 ** -24 * float(torch.linalg.cond(G)) * float(ref.norm())
            assert float((got.double() - ref).norm()) <= bound, (u, c, l)


@pytest.mark.parametrize("width", [4, 124, 128, 132, 1024])
@pytest.mark.parametrize("lead", [0, 1])
def test_int_row_table_pull_push_match_torch(width, lead):
    """Widths around a warp's 128 columns and its four pieces in flight; buffers off 16-byte boundaries."""
    from paracel_b200.ps.tables import RowTable
    g = torch.Generator(device="cuda").manual_seed(width)
    rows, n = 301, 207
    t = RowTable(rows, width, dtype=torch.int32, device="cuda:0")
    t.shard.copy_(torch.randint(-99, 99, (rows, width), device="cuda", generator=g))
    ids = torch.randperm(rows, device="cuda", generator=g)[:n]
    before = t.shard.clone()
    cur, old = (torch.zeros(n, width, dtype=torch.int32, device="cuda") for _ in range(2))
    t.pull(ids, cur, old)
    assert torch.equal(cur, before[ids]) and torch.equal(old, cur)
    new = (cur + torch.randint(-2, 3, cur.shape, device="cuda", generator=g)).int()

    def shifted(x):
        b = torch.zeros(x.numel() + 4, dtype=torch.int32, device="cuda")[lead: lead + x.numel()]
        return b.copy_(x.reshape(-1)).view(x.shape)
    new, old = shifted(new), shifted(old)
    t.push(ids, new, old, refresh_old=False)
    exp = before.clone()
    exp[ids] = new
    assert torch.equal(t.shard, exp) and torch.equal(old, cur)
    t.push(ids, new, old)                      # the same difference again, and old brought up to date
    exp[ids] += new - cur
    assert torch.equal(t.shard, exp) and torch.equal(old, new)
    t.push(ids, new)
    exp[ids] += new
    assert torch.equal(t.shard, exp)
    t.free()


@pytest.mark.parametrize("K", [4, 12, 16, 20, 32, 52, 100, 112])
def test_rows_times_matches_fp64(K):
    """Row counts around 64 and a block's 128 rows, columns around the 16 of a thread row."""
    from paracel_b200.ops.svd import rows_times
    g = torch.Generator(device="cuda").manual_seed(K)
    P = torch.randn(K, K, device="cuda", generator=g)
    for n in (1, 63, 64, 65, 127, 128, 129, 20_011):
        M = torch.randn(n, K, device="cuda", generator=g)
        A, P64 = M.double().abs() @ P.double().abs(), P.double()
        u = 2.0 ** -24 * (K + 1)
        one = rows_times(M, P)
        assert bool(((one.double() - M.double() @ P64).abs() <= u * A).all())
        two = rows_times(M, P, twice=True)
        bound = 2.1 * u * (A @ P64.abs().T)
        assert bool(((two.double() - M.double() @ P64 @ P64.T).abs() <= bound).all())


@pytest.mark.parametrize("n,seed", [(1, 0), (226, 3), (227, 3), (228, 7), (454, 1), (455, 2), (1077, 3), (1078, 4), (1023, 2 ** 32 - 1), (100_003, -5)])
def test_host_rand_is_the_cpu_generators_stream(n, seed):
    from paracel_b200.ops.svd import host_rand
    g = torch.Generator()
    g.manual_seed(seed)
    ref = torch.rand(n, generator=g)
    assert torch.equal(host_rand((n,), seed, "cuda").cpu(), ref)
    assert torch.equal(host_rand((n,), seed, "cuda", 2.0, -1.0).cpu(), ref * 2 - 1)


@pytest.mark.parametrize("d,k", [(4, 1), (4, 3000), (8, 10), (12, 30), (20, 7), (36, 100), (64, 100), (64, 900), (100, 12),
                                 (128, 2), (128, 130), (200, 40), (512, 8)])
def test_kmeans_accumulate_with_few_clusters(d, k):
    """Every group width, on both sides of the limit by which a block keeps its own sums; clusters that
    nobody is in, fewer points than groups."""
    from paracel_b200.ops.misc import kmeans_accumulate
    g = torch.Generator(device="cuda").manual_seed(d * k)
    for n in (1, 5, 1003, 60_001):
        X = torch.randn(n, d, device="cuda", generator=g)
        a = (torch.rand(n, device="cuda", generator=g) ** 2 * k).int().clamp(max=k - 1)
        sums, counts = torch.ones(k, d, device="cuda"), torch.ones(k, device="cuda")
        kmeans_accumulate(X, a, sums, counts)
        ref = torch.ones(k, d, dtype=torch.float64, device="cuda").index_add_(0, a.long(), X.double())
        mag = torch.ones(k, d, dtype=torch.float64, device="cuda").index_add_(0, a.long(), X.double().abs())
        cnt = 1 + torch.bincount(a.long(), minlength=k).double()
        assert torch.equal(counts.double(), cnt)
        assert bool(((sums.double() - ref).abs() <= (cnt[:, None] + 1) * 2.0 ** -24 * mag).all())


def test_similarity_leaves_out_rows_with_negative_ids():
    """A row of B with a negative id is nobody's neighbour and takes no place among the ktop."""
    from paracel_b200.models.similarity_gpu import SimDenseGpu
    g = torch.Generator(device="cuda").manual_seed(5)
    n, d, top = 60, 12, 4
    ids = torch.arange(n, device="cuda")
    ids[::3] = -1 - ids[::3]
    X = torch.randn(n, d, device="cuda", generator=g)
    m = SimDenseGpu(d, ktop=top, simbar=-1.0, device="cuda")
    m.load(ids, X)
    m.solve()
    Xn = X.double() / X.double().norm(dim=1, keepdim=True)
    S = Xn @ Xn.T
    S[:, ids < 0] = -9.0
    S.fill_diagonal_(-9.0)
    order = torch.sort(S, dim=1, descending=True).indices[:, :top]
    assert {r: [c for c, _ in v] for r, v in m.result.items()} == {
        int(ids[r]): [int(ids[c]) for c in order[r]] for r in range(n)}
    m.free()


@pytest.mark.parametrize("copy", [True, False])
def test_svd_of_a_full_rank_matrix_with_and_without_the_transposed_copy(monkeypatch, copy):
    """Row pointers that do not start at zero, empty rows, against an SVD in 64 bits."""
    import paracel_b200.models.svd_gpu as sg
    monkeypatch.setattr(sg, "_transpose_fits", lambda *a: copy)
    g = torch.Generator(device="cuda").manual_seed(8)
    n, N, k, lead = 900, 150, 5, 3
    lens = torch.randint(0, 30, (n,), device="cuda", generator=g)
    ptr, idx, val = _ragged_csr(n, N, lens, g, lead=lead)
    A = torch.zeros(n, N, dtype=torch.float64, device="cuda")
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), lens)
    # a strong rank-5 part, so that the iteration has converged after 30 steps
    U, V = (torch.randn(x, k, dtype=torch.float64, device="cuda", generator=g) for x in (n, N))
    c = idx[lead:].long()
    val[lead:] += (8 * (U[rows] * V[c]).sum(1)).float()
    A.index_put_((rows, c), val[lead:].double(), accumulate=True)
    m = sg.SvdGpu(N, k, iters=30, device="cuda")
    m.load(ptr, idx, val)
    m.solve()
    assert (m.t_ptr is not None) == copy
    Ur, S, Vr = torch.linalg.svd(A, full_matrices=False)
    # Gram matrices in fp32 square the factors' condition: sigma is good to about 2^-24 (s_1 / s_k)^2
    assert bool(((m.sigma.cuda() - S[:k]).abs() <= 64 * 2.0 ** -24 * float(S[0] / S[k - 1]) ** 2 * S[:k]).all())
    P = m.U.double() @ torch.diag(m.sigma.cuda()) @ m.V.double().T
    best = Ur[:, :k] @ torch.diag(S[:k]) @ Vr[:k]
    assert float((P - best).norm()) <= 1e-3 * float(best.norm())
    m.free()


def test_als_accumulators_take_no_more_than_seg_len_ratings_in_a_row():
    """2050 users of 16,300 equal ratings: one fp32 chain over a user's ratings is off by 1.9e-4, chains of
    4096 by at most half a unit of the sum per term, 4096 * 2^-25."""
    from paracel_b200.ops.als import als_solve
    users, n = 2050, 16_300
    r = 1 + 2.0 ** -11 - 2.0 ** -14
    ptr = torch.arange(users + 1, device="cuda") * n
    idx = torch.zeros(users * n, dtype=torch.int32, device="cuda")
    W = als_solve(ptr, idx, torch.full((users * n,), r, device="cuda"), torch.ones(1, 1, device="cuda"), lam=1.0)
    assert float((W.double() / (n * r / (n + 1)) - 1).abs().max()) <= (4096 + 8) * 2.0 ** -25


@pytest.mark.parametrize("d,k,n", [(4, 20, 1200), (16, 40, 7200), (32, 64, 26624), (64, 30, 9450), (100, 30, 9900),
                                   (128, 20, 4400), (256, 12, 4968), (512, 6, 2394)])
def test_kmeans_accumulate_on_both_sides_of_the_point_count_that_picks_its_sums(d, k, n):
    from paracel_b200.ops.misc import kmeans_accumulate
    g = torch.Generator(device="cuda").manual_seed(d + k)
    for m in (n - 1, n):
        X = torch.randn(m, d, device="cuda", generator=g)
        a = torch.randint(0, k, (m,), device="cuda", generator=g, dtype=torch.int32)
        sums, counts = torch.zeros(k, d, device="cuda"), torch.zeros(k, device="cuda")
        kmeans_accumulate(X, a, sums, counts)
        ref = torch.zeros(k, d, dtype=torch.float64, device="cuda").index_add_(0, a.long(), X.double())
        mag = torch.zeros(k, d, dtype=torch.float64, device="cuda").index_add_(0, a.long(), X.double().abs())
        cnt = torch.bincount(a.long(), minlength=k).double()
        assert torch.equal(counts.double(), cnt)
        assert bool(((sums.double() - ref).abs() <= (cnt[:, None] + 1) * 2.0 ** -24 * mag).all())


@pytest.mark.parametrize("k", [30, 64, 96, 128])
def test_gram_chains_are_bounded(k):
    """2.5 M equal rows: a chain of one block's rows, all in one register, is off by 1.1e-4 at k > 64;
    chains of 1280 terms (for k <= 64 a group's share of the block) and of the groups' and blocks' sums by half a
    unit per addition at most, 4.7e-5."""
    from paracel_b200.ops.misc import gram
    n, h = 2_500_000, 1.0 + 2.0 ** -10 + 2.0 ** -13
    G = gram(torch.full((n, k), h, device="cuda"))
    rows = n // 296 + 1
    chain = (1280 + rows // 1280 if k > 64 else rows // (10 if k <= 32 else 3) + 1) + 10 + 296
    assert float((G.double() / (n * h * h) - 1).abs().max()) <= chain * 2.0 ** -25


@pytest.mark.parametrize("n,per,K", [(33_001, 40, 128), (140_003, 7, 32), (90_001, 16, 52), (90_001, 50, 64), (120_001, 200, 128)])
def test_csr_product_writes_every_row_of_a_dirty_output(n, per, K):
    """Outputs beyond 16 MB are cleared by rows: those without entries and those cut by a segment's end
    (of 512 entries in the last case), while the others are stored once."""
    from paracel_b200.ops.svd import spmm_csr
    g = torch.Generator(device="cuda").manual_seed(n)
    lens = torch.full((n,), per, device="cuda")
    lens[::11] = 0
    lens[5], lens[-1] = 3000, 0
    ptr, idx, val = _ragged_csr(n, 701, lens, g)
    H = torch.randn(701, K, device="cuda", generator=g)
    out = torch.full((n, K), float("nan"), device="cuda")
    spmm_csr(ptr, idx, val, H, out)
    assert bool(torch.isfinite(out).all()) and not bool(out[::11].any())
    for r in [1, 4, 5, 6, n // 2, n - 3] + list(range(2000, 2060)):
        a, b = int(ptr[r]), int(ptr[r + 1])
        prod = val[a:b].double()[:, None] * H[idx[a:b].long()].double()
        assert bool(((out[r].double() - prod.sum(0)).abs() <= (b - a + 2) * 2.0 ** -24 * prod.abs().sum(0)).all())


@pytest.mark.parametrize("valued", [True, False])
@pytest.mark.parametrize("logistic", [True, False])
def test_sparse_gradient_of_long_rows(logistic, valued):
    """Rows around the 64 entries of the short form and the 128 a long row keeps in registers, mixed and alone."""
    from paracel_b200.ops.linear import sparse_grad
    g = torch.Generator(device="cuda").manual_seed(9)
    F = 12_000
    for pick in ([63, 64, 65], [127, 128, 129, 1], [65], [400, 0, 128, 256]):
        n = 3001
        lens = torch.tensor(pick, device="cuda")[torch.randint(0, len(pick), (n,), device="cuda", generator=g)]
        ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        ptr[1:] = lens.cumsum(0)
        cols = (torch.rand(int(ptr[-1]), device="cuda", generator=g) ** 3 * F).int().clamp(max=F - 1)
        vals = torch.rand(cols.numel(), device="cuda", generator=g) if valued else None
        v64 = vals.double() if valued else torch.ones(cols.numel(), device="cuda").double()
        theta = 0.05 * torch.randn(F, device="cuda", generator=g)
        y = (torch.rand(n, device="cuda", generator=g) < 0.5).float()
        row = torch.repeat_interleave(torch.arange(n, device="cuda"), lens)
        zero = torch.zeros(n, dtype=torch.float64, device="cuda")
        z = zero.index_add(0, row, v64 * theta.double()[cols.long()])
        zmag = zero.index_add(0, row, v64 * theta.double()[cols.long()].abs())
        r = y.double() - (torch.sigmoid(z) if logistic else z)
        fzero = torch.zeros(F, dtype=torch.float64, device="cuda")
        ref = fzero.index_add(0, cols.long(), r[row] * v64)
        mag = fzero.index_add(0, cols.long(), v64 * (1 + zmag[row]))
        cnt = torch.bincount(cols.long(), minlength=F).double()
        grad, loss = torch.zeros(F, device="cuda"), torch.zeros(1, dtype=torch.float64, device="cuda")
        sparse_grad(ptr, cols, vals, y, theta, grad, loss, logistic=logistic)
        # half a unit of the fixed-point table per term; margins of up to 400 terms; fp32 sums of cnt terms
        bound = (cnt * 2.0 ** -15 if logistic else 0) + (cnt + 420) * 2.0 ** -23 * mag
        assert bool(((grad.double() - ref).abs() <= bound + 1e-30).all()), pick


@pytest.mark.parametrize("spectrum", ["rank 3", "rank 12", "full"])
def test_svd_of_rank_deficient_and_ill_conditioned_matrices(spectrum):
    """Directions of a Gram matrix below its fp32 rounding are noise and must not be inverted.  What is kept
    is good to K 2^-24 (s_1 / s_k)^2, the rounding of the largest eigenvalue against the smallest."""
    from paracel_b200.models.svd_gpu import SvdGpu
    m, n = 80, 30
    for seed in range(8):
        g = torch.Generator().manual_seed(seed)
        if spectrum == "full":
            k = 8
            U = torch.linalg.qr(torch.randn(m, n, dtype=torch.float64, generator=g)).Q
            V = torch.linalg.qr(torch.randn(n, n, dtype=torch.float64, generator=g)).Q
            s = torch.cat([torch.logspace(0, -2, k, dtype=torch.float64),
                           0.003 * 0.8 ** torch.arange(n - k, dtype=torch.float64)])
            M = (U * s) @ V.T
        else:
            k = int(spectrum.split()[1])
            M = torch.randn(m, k, dtype=torch.float64, generator=g) @ torch.randn(k, n, dtype=torch.float64, generator=g)
        ref = torch.linalg.svdvals(M)[:k]
        sv = SvdGpu(n, k, device="cuda", seed=seed)
        sv.load(torch.arange(0, m * n + 1, n), torch.arange(n).repeat(m).int(), M.reshape(-1).float())
        sv.solve()
        assert sv.sigma.numel() == k
        assert bool(((sv.sigma - ref).abs() <= sv.K * 2.0 ** -24 * float(ref[0] / ref[-1]) ** 2 * ref).all()), seed
        sv.free()


@pytest.mark.parametrize("width", [8, 64, 100, 252])
def test_narrow_int_rows_pull_push_match_torch(width):
    """Rows pushed int by int (below 128) and in pieces; pulled one piece per lane up to 128 ints."""
    from paracel_b200.ps.tables import RowTable
    g = torch.Generator(device="cuda").manual_seed(width)
    t = RowTable(500, width, dtype=torch.int32, device="cuda:0")
    t.shard.copy_(torch.randint(-9, 9, (500, width), device="cuda", generator=g))
    before, ids = t.shard.clone(), torch.randperm(500, device="cuda", generator=g)[:333]
    cur, old = (torch.zeros(333, width, dtype=torch.int32, device="cuda") for _ in range(2))
    t.pull(ids, cur, old)
    assert torch.equal(cur, before[ids]) and torch.equal(old, cur)
    new = cur + torch.randint(-2, 3, cur.shape, device="cuda", generator=g, dtype=torch.int32)
    t.push(ids, new, old)
    before[ids] = new
    assert torch.equal(t.shard, before) and torch.equal(old, new)
    t.free()
