"""GPU parity of the exhaustive search (nn_distance, tk_nn_distance):
bit-exact against the oracle's exhaustive search, and identical to the
KD-tree query on the same inputs."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

cuda = torch.device("cuda")


def tk():
    import torch_kdtree_gb300
    return torch_kdtree_gb300


@pytest.mark.parametrize("d", [1, 2, 3, 4, 5, 8, 17, 32, 64, 128])
@pytest.mark.parametrize("k", [1, 3, 16, 32, 100])
def test_exact_mode_matches_oracle(d, k, oracle):
    rng = np.random.default_rng(d * 1000 + k)
    n = 6000 if d <= 32 else 3000
    ref = rng.standard_normal((n, d)).astype(np.float32)
    q = rng.standard_normal((700, d)).astype(np.float32)
    dd, ii = tk().nn_distance(torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda), k)
    bd, bi = oracle.brute(ref, q, k)
    np.testing.assert_array_equal(dd.cpu().numpy(), bd)
    np.testing.assert_array_equal(ii.cpu().numpy(), bi)


@pytest.mark.parametrize("d", [1, 2, 3, 5, 8, 17, 40, 128])
def test_float64(d, oracle):
    """FP64 stays FP64 end to end, at any dimension."""
    rng = np.random.default_rng(40 + d)
    ref = rng.standard_normal((5000, d))
    q = rng.standard_normal((500, d))
    for k in (1, 7, 40):
        dd, ii = tk().nn_distance(torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda), k)
        assert dd.dtype == torch.float64
        bd, bi = oracle.brute(ref, q, k)
        np.testing.assert_array_equal(dd.cpu().numpy(), bd)
        np.testing.assert_array_equal(ii.cpu().numpy(), bi)
    if d in (5, 40):  # gradients in float64 as well
        r = torch.from_numpy(ref).to(cuda).requires_grad_(True)
        qq = torch.from_numpy(q).to(cuda).requires_grad_(True)
        dd, ii = tk().nn_distance(r, qq, 7)
        w = torch.rand_like(dd)
        (dd * w).sum().backward()
        r2 = r.detach().clone().requires_grad_(True)
        q2 = qq.detach().clone().requires_grad_(True)
        ((q2[:, None] - r2[ii.long()]) ** 2).sum(-1).mul(w).sum().backward()
        assert torch.allclose(qq.grad, q2.grad, rtol=1e-12, atol=1e-12)
        assert torch.allclose(r.grad, r2.grad, rtol=1e-12, atol=1e-12)


def test_brute_equals_kdtree():
    g = torch.Generator().manual_seed(3)
    ref = torch.rand(65536, 3, generator=g).to(cuda)
    q = torch.rand(8192, 3, generator=g).to(cuda)
    for k in (1, 16):
        bd, bi = tk().nn_distance(ref, q, k)
        kd, ki = tk().build_kd_tree(ref).query(q, nr_nns_searches=k)
        assert torch.equal(bd, kd) and torch.equal(bi, ki)


def test_duplicates_and_many_slices(oracle):
    """5% exact duplicates; few queries so the reference set is sliced across
    many blocks and the per-slice lists are merged."""
    rng = np.random.default_rng(77)
    ref = rng.standard_normal((200_000, 8)).astype(np.float32)
    m = 10_000
    perm = rng.permutation(len(ref))
    ref[perm[:m]] = ref[perm[m:2 * m]]
    q = ref[rng.integers(0, len(ref), 64)] + np.float32(0)
    dd, ii = tk().nn_distance(torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda), 32)
    bd, bi = oracle.brute(ref, q, 32)
    np.testing.assert_array_equal(dd.cpu().numpy(), bd)
    np.testing.assert_array_equal(ii.cpu().numpy(), bi)


def test_brute_backward_matches_torch():
    g = torch.Generator().manual_seed(5)
    for d in (3, 8, 32):
        ref = torch.randn(4000, d, generator=g).to(cuda).requires_grad_(True)
        q = torch.randn(3000, d, generator=g).to(cuda).requires_grad_(True)
        w = torch.rand(3000, 4, generator=g).to(cuda)
        dists, inds = tk().nn_distance(ref, q, 4)
        (0.5 * (dists * w).sum()).backward()
        q2 = q.detach().clone().requires_grad_(True)
        r2 = ref.detach().clone().requires_grad_(True)
        d2 = torch.sum((q2[:, None] - r2[inds.long()]) ** 2, -1)
        (0.5 * (d2 * w).sum()).backward()
        assert torch.allclose(q.grad, q2.grad, rtol=1e-4, atol=1e-4)
        assert torch.allclose(ref.grad, r2.grad, rtol=1e-4, atol=1e-4)


def test_errors():
    ref = torch.randn(10, 3, device=cuda)
    with pytest.raises(Exception):
        tk().nn_distance(ref, torch.randn(4, 3, device=cuda), 11)
    with pytest.raises(Exception):
        tk().nn_distance(ref, torch.randn(4, 2, device=cuda), 1)
    with pytest.raises(Exception):
        tk().nn_distance(ref, torch.randn(4, 3, device=cuda, dtype=torch.float64), 1)


@pytest.mark.parametrize("mode", ["tf32", "bf16_split"])
@pytest.mark.parametrize("d", [3, 8, 17, 32, 64])
@pytest.mark.parametrize("k", [1, 16, 32])
def test_tensor_core_modes_are_exact(mode, d, k, oracle):
    """Tensor-core candidate search + exact re-rank (+ exact fallback for
    uncertified queries) returns the exact answer, bit for bit."""
    rng = np.random.default_rng(1000 + 10 * d + k)
    ref = rng.standard_normal((20000, d)).astype(np.float32)
    m = 1000
    perm = rng.permutation(len(ref))
    ref[perm[:m]] = ref[perm[m:2 * m]]  # 5% exact duplicates
    q = rng.standard_normal((3000, d)).astype(np.float32)
    dd, ii = tk().nn_distance(torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda), k, mode=mode)
    bd, bi = oracle.brute(ref, q, k)
    np.testing.assert_array_equal(dd.cpu().numpy(), bd)
    np.testing.assert_array_equal(ii.cpu().numpy(), bi)


@pytest.mark.parametrize("mode", ["tf32", "bf16_split"])
@pytest.mark.parametrize("d", [3, 17, 40])
@pytest.mark.parametrize("k", [33, 64])
def test_tensor_core_large_k(mode, d, k, oracle):
    """k above 32: the mma.sync candidate search with a 128-key over-fetch and
    the two-register re-rank; d = 40 also leaves the tcgen05 path's depth."""
    rng = np.random.default_rng(8800 + d + k)
    ref = rng.standard_normal((30000, d)).astype(np.float32)
    ref[rng.permutation(30000)[:500]] = ref[:500]  # exact duplicates
    q = rng.standard_normal((700, d)).astype(np.float32)
    dd, ii = tk().nn_distance(torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda), k, mode=mode)
    bd, bi = oracle.brute(ref, q, k)
    np.testing.assert_array_equal(dd.cpu().numpy(), bd)
    np.testing.assert_array_equal(ii.cpu().numpy(), bi)
    if d == 40:  # too big for the candidate search's shared memory: every query exact
        from torch_kdtree_gb300 import _lib
        from torch_kdtree_gb300._lib import LIB
        from torch_kdtree_gb300.nn_distance import _BRUTE_MODES, _stream_ptr
        m = _BRUTE_MODES[mode]
        r_t, q_t = torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda)
        wsb = LIB.tk_nn_distance_workspace_size(len(ref), len(q), d, k, _lib.TK_F32, m)
        ws = torch.empty(wsb, dtype=torch.uint8, device=cuda)
        d2 = torch.empty(len(q), k, device=cuda)
        i2 = torch.empty(len(q), k, dtype=torch.int32, device=cuda)
        _lib.check(LIB.tk_nn_distance(r_t.data_ptr(), len(ref), q_t.data_ptr(), len(q), d, k, _lib.TK_F32, m,
                                      d2.data_ptr(), i2.data_ptr(), ws.data_ptr(), wsb, _stream_ptr(cuda)))
        torch.cuda.synchronize()
        import ctypes
        flags, rec = ctypes.c_int(-1), ctypes.c_int(-1)
        _lib.check(LIB.tk_nn_distance_report(ws.data_ptr(), len(ref), len(q), d, k, _lib.TK_F32, m,
                                             ctypes.byref(flags), ctypes.byref(rec)))
        assert flags.value == 0 and rec.value == len(q)
        np.testing.assert_array_equal(d2.cpu().numpy(), bd)
        np.testing.assert_array_equal(i2.cpu().numpy(), bi)


@pytest.mark.parametrize("mode", ["tf32", "bf16_split"])
@pytest.mark.parametrize("k", [8, 16, 32])
@pytest.mark.parametrize("data", ["normal", "repeated", "grid"])
def test_tensor_core_sampled_threshold_slices(mode, k, data, oracle):
    """Slices long enough (70,000 refs, 8 slices of ~34 tiles) that the
    candidate kernel first samples a threshold: on N(0,1) data, on 300
    distinct points repeated (every tile overflows the hit buffers and is
    redone in 32-column steps) and on an integer grid (exact distance ties).
    The answer must stay the exhaustive search's, bit for bit."""
    rng = np.random.default_rng(4100 + k)
    d = 16
    if data == "normal":
        ref = rng.standard_normal((70000, d)).astype(np.float32)
    elif data == "repeated":
        ref = rng.standard_normal((300, d)).astype(np.float32)[rng.integers(0, 300, 70000)]
    else:
        ref = rng.integers(-3, 4, (70000, d)).astype(np.float32)
    q = rng.standard_normal((600, d)).astype(np.float32)
    if data == "grid":
        q = np.rint(q)  # integer distances: many exact ties
    dd, ii = tk().nn_distance(torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda), k, mode=mode)
    bd, bi = oracle.brute(ref, q, k)
    np.testing.assert_array_equal(dd.cpu().numpy(), bd)
    np.testing.assert_array_equal(ii.cpu().numpy(), bi)


@pytest.mark.parametrize("mode", ["tf32", "bf16_split"])
@pytest.mark.parametrize("n", [1, 7, 255, 256, 257, 513])
@pytest.mark.parametrize("nq", [1, 5, 129])
def test_tensor_core_edge_sizes(mode, n, nq, oracle):
    """Single, partial and exactly-full 256-reference tiles, query blocks of
    1, 5 and 129 rows (one row past a 128-row block), k up to 32 and at most
    n: slices far too short for the sampled threshold, the last tile's
    column bound, padding rows of both operands."""
    rng = np.random.default_rng(7000 + n + nq)
    d = 12
    ref = rng.standard_normal((n, d)).astype(np.float32)
    q = rng.standard_normal((nq, d)).astype(np.float32)
    for k in sorted({1, min(n, 5), min(n, 32)}):
        dd, ii = tk().nn_distance(torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda), k, mode=mode)
        bd, bi = oracle.brute(ref, q, k)
        np.testing.assert_array_equal(dd.cpu().numpy(), bd)
        np.testing.assert_array_equal(ii.cpu().numpy(), bi)


@pytest.mark.parametrize("mode", ["tf32", "bf16_split"])
def test_tensor_core_fallback_on_massive_ties(mode, oracle):
    """64 distinct points repeated ~300 times: candidate lists cannot separate
    the k-th neighbour from the rest, the certificate fails and the exact
    fallback must produce the answer."""
    rng = np.random.default_rng(7)
    base = rng.standard_normal((64, 16)).astype(np.float32)
    ref = base[rng.integers(0, 64, 20000)]
    q = rng.standard_normal((500, 16)).astype(np.float32)
    dd, ii = tk().nn_distance(torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda), 20, mode=mode)
    bd, bi = oracle.brute(ref, q, 20)
    np.testing.assert_array_equal(dd.cpu().numpy(), bd)
    np.testing.assert_array_equal(ii.cpu().numpy(), bi)


def test_auto_mode_picks_a_mode_and_stays_exact(tmp_path, monkeypatch, oracle):
    """mode="auto" times the modes once (cached) and returns the exact answer."""
    import torch_kdtree_gb300.autotune as at
    from torch_kdtree_gb300 import nn_distance
    monkeypatch.setattr(at, "CACHE_PATH", str(tmp_path / "cache.json"))
    rng = np.random.default_rng(44)
    for d, dtype in ((32, np.float32), (3, np.float32), (3, np.float64)):
        ref = rng.standard_normal((20000, d)).astype(dtype)
        q = rng.standard_normal((700, d)).astype(dtype)
        rt, qt = torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda)
        mode = at.autotune_brute(rt, qt, 8)
        assert mode in (("exact",) if dtype == np.float64 else ("exact", "tf32", "bf16_split"))
        dd, ii = nn_distance(rt, qt, 8, mode="auto")
        bd, bi = oracle.brute(ref, q, 8)
        np.testing.assert_array_equal(dd.cpu().numpy(), bd)
        np.testing.assert_array_equal(ii.cpu().numpy(), bi)
    import json
    assert len(json.load(open(tmp_path / "cache.json"))) == 3


@pytest.mark.parametrize("mode", ["exact", "tf32", "bf16_split"])
def test_infinite_and_overflowing_queries(mode, oracle):
    """Rows whose distances are +inf to every reference (infinite coordinates,
    or squares that overflow) tie at +inf: the k lowest indices, in every mode
    (the tensor-core modes cannot certify them and fall back to exact)."""
    rng = np.random.default_rng(77)
    ref = rng.standard_normal((20000, 8)).astype(np.float32)
    q = rng.standard_normal((600, 8)).astype(np.float32)
    q[3, 0] = np.inf
    q[4, 0] = -np.inf
    q[5, :] = 1e20
    q[6, 0], q[6, 1] = np.inf, -np.inf
    q[7, 0] = 3e19
    dd, ii = tk().nn_distance(torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda), 5, mode=mode)
    bd, bi = oracle.brute(ref, q, 5)
    assert np.isinf(bd[3:8]).all() and (bi[3:8] == np.arange(5)).all()
    np.testing.assert_array_equal(dd.cpu().numpy(), bd)
    np.testing.assert_array_equal(ii.cpu().numpy(), bi)


@pytest.mark.parametrize("mode", ["exact", "tf32", "bf16_split"])
def test_infinite_and_huge_references(mode, oracle):
    """References with infinite coordinates or norms beyond the tensor-core
    range: the tensor-core modes certify nothing and fall back to exact; the
    answers equal the oracle's (such references sit at distance +inf)."""
    rng = np.random.default_rng(78)
    ref = rng.standard_normal((20000, 8)).astype(np.float32)
    ref[5, 2] = np.inf
    ref[9, 0] = -np.inf
    ref[11, :] = 3e19
    q = rng.standard_normal((700, 8)).astype(np.float32)
    q[0, :] = 3e19  # next to ref 11: distance 0 there, +inf to everything else
    dd, ii = tk().nn_distance(torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda), 4, mode=mode)
    bd, bi = oracle.brute(ref, q, 4)
    assert bi[0, 0] == 11 and bd[0, 0] == 0
    np.testing.assert_array_equal(dd.cpu().numpy(), bd)
    np.testing.assert_array_equal(ii.cpu().numpy(), bi)


def test_random_configurations(oracle):
    """A seeded sweep over exhaustive-search shapes: dims 1-64, k up to 64 and
    n, query counts from 1 up, every mode (tensor-core modes for float32),
    duplicates; every answer bit-exact against the oracle."""
    rng = np.random.default_rng(31337)
    for case in range(60):
        d = int(rng.choice([1, 2, 3, 5, 8, 12, 16, 24, 31, 32, 33, 39, 40, 47, 48, 64]))
        n = int(rng.choice([1, 5, 64, 257, 1500, 4000]))
        nq = int(rng.choice([1, 7, 129, 500]))
        k = int(rng.integers(1, min(n, 64) + 1))
        mode = str(rng.choice(["exact", "tf32", "bf16_split"]))
        dtype = np.float64 if (mode == "exact" and rng.random() < 0.3) else np.float32
        ref = (rng.standard_normal((n, d)) * float(rng.choice([1e-2, 1.0, 1e2]))).astype(dtype)
        if n > 10:
            ref[rng.integers(0, n, n // 8)] = ref[rng.integers(0, n, n // 8)]
        q = rng.standard_normal((nq, d)).astype(dtype)
        dd, ii = tk().nn_distance(torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda), k, mode=mode)
        bd, bi = oracle.brute(ref, q, k)
        msg = f"case {case}: d={d} n={n} nq={nq} k={k} {mode} {np.dtype(dtype).name}"
        np.testing.assert_array_equal(dd.cpu().numpy(), bd, err_msg=msg)
        np.testing.assert_array_equal(ii.cpu().numpy(), bi, err_msg=msg)


@pytest.mark.parametrize("mode", ["tf32", "bf16_split"])
@pytest.mark.parametrize("order", ["clustered", "sorted", "one_column"])
@pytest.mark.parametrize("k", [1, 16, 32])
def test_tensor_core_lists_that_fill_up(mode, order, k, oracle):
    """Clouds whose near neighbours are neighbours in memory, or all sit where
    one thread keeps its list: the sampled thresholds let too much through and
    lists are pruned on the way."""
    rng = np.random.default_rng(k)
    n, d, nq = 40_000, 12, 300
    if order == "clustered":
        ref = np.repeat(rng.standard_normal((40, d)) * 8, n // 40, axis=0) + rng.standard_normal((n, d)) * 0.1
    else:
        ref = rng.standard_normal((n, d))
        if order == "sorted":
            ref = ref[np.argsort(ref[:, 0])]
            ref[:, 0] *= 30
        else:  # 157 tiles: every 157th reference shares a tile
            ref[::157] *= 0.01
    ref = ref.astype(np.float32)
    q = (ref[rng.integers(0, n, nq)] + 0.05 * rng.standard_normal((nq, d))).astype(np.float32)
    if order == "one_column":
        q = (0.01 * rng.standard_normal((nq, d))).astype(np.float32)
    bd, bi = oracle.brute(ref, q, k)
    dd, ii = tk().nn_distance(torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda), k, mode=mode)
    np.testing.assert_array_equal(dd.cpu().numpy(), bd)
    np.testing.assert_array_equal(ii.cpu().numpy(), bi)


@pytest.mark.parametrize("n_listed", [3, 300, 2500])
@pytest.mark.parametrize("k", [1, 32, 64])
def test_recomputed_queries(n_listed, k, oracle):
    """Queries without a certificate (their nearest references are all equally
    far) among ordinary ones: few of them take a warp per slice, many the
    tiled kernel."""
    rng = np.random.default_rng(n_listed + k)
    ref = np.concatenate([rng.standard_normal((6000, 8)), np.tile(rng.standard_normal((1, 8)) + 20, (700, 1))])
    ref = ref[rng.permutation(len(ref))].astype(np.float32)
    q = rng.standard_normal((3000, 8)).astype(np.float32)
    hard = rng.permutation(len(q))[:n_listed]
    q[hard] = (20 + 0.1 * rng.standard_normal((n_listed, 8))).astype(np.float32)
    bd, bi = oracle.brute(ref, q, k)
    dd, ii = tk().nn_distance(torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda), k, mode="tf32")
    np.testing.assert_array_equal(dd.cpu().numpy(), bd)
    np.testing.assert_array_equal(ii.cpu().numpy(), bi)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("d", [1, 2, 3])
@pytest.mark.parametrize("data", ["normal", "repeated", "grid", "nan", "inf"])
def test_exact_mode_through_a_tree(dtype, d, data, oracle):
    """Large calls in 1-3 dimensions build a tree for the call; clouds with NaN
    or infinite coordinates are searched exhaustively after all."""
    rng = np.random.default_rng(d)
    n, nq = 20_011, 5_003
    ref = rng.standard_normal((n, d)).astype(dtype)
    q = rng.standard_normal((nq, d)).astype(dtype)
    if data == "repeated":
        ref = ref[rng.integers(0, 50, n)]
    elif data == "grid":
        ref, q = np.round(ref * 2), np.round(q * 2)
    elif data == "nan":
        ref[rng.integers(0, n, 3), rng.integers(0, d, 3)] = np.nan
        q[7, 0] = np.nan
    elif data == "inf":
        ref[rng.integers(0, n, n // 2), 0] = np.inf
        q[:3, 0] = (np.inf, -np.inf, np.nan)
    rt, qt = torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda)
    for k in (1, 5, 17, 100):
        bd, bi = oracle.brute(ref, q, k)
        bi = np.where(bi == 2 ** 31 - 1, -1, bi)  # the oracle's mark of a NaN query's empty slots
        dd, ii = tk().nn_distance(rt, qt, k)
        np.testing.assert_array_equal(dd.cpu().numpy(), bd)
        np.testing.assert_array_equal(ii.cpu().numpy(), bi)


def test_exact_mode_captured_in_a_graph():
    """Every route of the exact mode is device work only."""
    for n, nq, d, k in ((30_000, 30_000, 3, 1), (4_000, 2_000, 16, 8), (300, 50, 3, 2)):
        ref, q = torch.randn(n, d, device=cuda), torch.randn(nq, d, device=cuda)
        want = tk().nn_distance(ref, q, k)
        static_q = torch.zeros_like(q)
        tk().nn_distance(ref, static_q, k)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            dd, ii = tk().nn_distance(ref, static_q, k)
        static_q.copy_(q)
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(dd, want[0]) and torch.equal(ii, want[1])


@pytest.mark.parametrize("mode", ["tf32", "bf16_split"])
@pytest.mark.parametrize("extra", [1, 300, 9000])
@pytest.mark.parametrize("k", [1, 32])
def test_tensor_core_rows_left_over(mode, extra, k, oracle):
    """Row blocks left over after whole waves of blocks are searched in slices
    of their own: a few of them, some, and more than half a wave."""
    rng = np.random.default_rng(extra + k)
    nq = 128 * torch.cuda.get_device_properties(0).multi_processor_count + extra
    ref = rng.standard_normal((9000, 8)).astype(np.float32)
    q = rng.standard_normal((nq, 8)).astype(np.float32)
    bd, bi = oracle.brute(ref, q, k)
    dd, ii = tk().nn_distance(torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda), k, mode=mode)
    np.testing.assert_array_equal(dd.cpu().numpy(), bd)
    np.testing.assert_array_equal(ii.cpu().numpy(), bi)


@pytest.mark.parametrize("n_listed", [1, 32, 33, 200])
@pytest.mark.parametrize("k", [1, 20, 64])
@pytest.mark.parametrize("d", [7, 8])
def test_few_recomputed_queries(n_listed, k, d, oracle):
    """The same with lists at the edges of the block-per-slice search, slices
    that leave warps without a row, and rows read one float at a time."""
    rng = np.random.default_rng(n_listed + k)
    ref = np.concatenate([rng.standard_normal((1000, d)), np.tile(rng.standard_normal((1, d)) + 20, (300, 1))])
    ref = ref[rng.permutation(len(ref))].astype(np.float32)
    q = rng.standard_normal((1000, d)).astype(np.float32)
    hard = rng.permutation(len(q))[:n_listed]
    q[hard] = (20 + 0.1 * rng.standard_normal((n_listed, d))).astype(np.float32)
    bd, bi = oracle.brute(ref, q, k)
    dd, ii = tk().nn_distance(torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda), k, mode="tf32")
    np.testing.assert_array_equal(dd.cpu().numpy(), bd)
    np.testing.assert_array_equal(ii.cpu().numpy(), bi)


@pytest.mark.parametrize("d,mode", [(23, "tf32"), (24, "tf32"), (32, "tf32"), (39, "tf32"), (24, "bf16_split"), (47, "bf16_split")])
@pytest.mark.parametrize("data", ["normal", "repeated", "clusters"])
def test_tensor_core_staged_rerank(d, mode, data, oracle):
    """The re-rank that recomputes the best scores first, at the edges of its
    dimensions: lists of distinct scores, of ties, and of far more than wanted."""
    rng = np.random.default_rng(d)
    n, nq = 20_000, 2_000
    ref = rng.standard_normal((n, d)).astype(np.float32)
    if data == "repeated":
        ref = ref[rng.integers(0, n // 20, n)]
    elif data == "clusters":
        ref = (ref[rng.integers(0, 40, n)] + 0.05 * rng.standard_normal((n, d))).astype(np.float32)
    q = (ref[rng.integers(0, n, nq)] + 0.2 * rng.standard_normal((nq, d))).astype(np.float32)
    for k in (1, 10, 32):
        bd, bi = oracle.brute(ref, q, k)
        dd, ii = tk().nn_distance(torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda), k, mode=mode)
        np.testing.assert_array_equal(dd.cpu().numpy(), bd)
        np.testing.assert_array_equal(ii.cpu().numpy(), bi)


@pytest.mark.parametrize("mode", ["exact", "tf32", "bf16_split"])
@pytest.mark.parametrize("d", [8, 32])
@pytest.mark.parametrize("share", [0.01, 0.1, 0.5])
@pytest.mark.parametrize("value", [np.inf, -np.inf])
def test_many_infinite_references(mode, d, share, value, oracle):
    """References with an infinite coordinate, and nothing else unusual in the
    cloud: many of them, so that whole samples of scores come from such rows."""
    rng = np.random.default_rng(d)
    ref = rng.standard_normal((20_000, d)).astype(np.float32)
    ref[rng.permutation(len(ref))[:int(share * len(ref))], 1] = value
    q = rng.standard_normal((1_000, d)).astype(np.float32)
    for k in (1, 8, 32):
        bd, bi = oracle.brute(ref, q, k)
        assert np.isfinite(bd).all()
        dd, ii = tk().nn_distance(torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda), k, mode=mode)
        np.testing.assert_array_equal(dd.cpu().numpy(), bd)
        np.testing.assert_array_equal(ii.cpu().numpy(), bi)


def test_default_mode_workspace_covers_every_pass():
    """Calls of more queries than one pass over the tensor cores: the size that
    is asked for covers the full passes and the rest, whatever its length."""
    from torch_kdtree_gb300 import _lib
    from torch_kdtree_gb300._lib import LIB
    full = 262_144
    for n, d, k in ((20_000, 32, 8), (20_000, 8, 8), (262_144, 32, 32), (5_000, 16, 1)):
        def size(nq, mode):
            return LIB.tk_nn_distance_workspace_size(n, nq, d, k, _lib.TK_F32, mode)
        one = size(full, _lib.TK_BRUTE_BF16_SPLIT)
        for rest in range(1, full, 128):
            need = size(rest, _lib.TK_BRUTE_BF16_SPLIT)
            assert size(full + rest, _lib.TK_BRUTE_ROUTED) >= max(one, need), (n, d, k, rest)


@pytest.mark.parametrize("nq", [262_144 + 255_000, 262_144 + 1, 2 * 262_144])
def test_default_mode_in_several_passes(nq, oracle):
    rng = np.random.default_rng(nq)
    ref = rng.standard_normal((20_000, 8)).astype(np.float32)
    q = rng.standard_normal((nq, 8)).astype(np.float32)
    dd, ii = tk().nn_distance(torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda), 8)
    rows = np.concatenate([np.arange(100), np.arange(262_044, 262_244) % nq, np.arange(nq - 300, nq)])
    bd, bi = oracle.brute(ref, q[rows], 8)
    np.testing.assert_array_equal(dd.cpu().numpy()[rows], bd)
    np.testing.assert_array_equal(ii.cpu().numpy()[rows], bi)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("nq", [30_000, 400_000])
@pytest.mark.parametrize("k", [1, 4, 8, 16, 20])
def test_nan_queries_through_a_tree(dtype, nq, k):
    """A query with a NaN coordinate has no neighbour, whichever search the
    default mode takes: distance inf, index -1 (the CUDA cores' answer)."""
    from torch_kdtree_gb300.nn_distance import nn_distance_raw
    g = torch.Generator(device=cuda).manual_seed(k)
    for d in (1, 2, 3):
        ref = torch.randn(20_000, d, generator=g, device=cuda, dtype=torch.float64).to(getattr(torch, np.dtype(dtype).name))
        q = torch.randn(nq, d, generator=g, device=cuda, dtype=torch.float64).to(ref.dtype)
        rows = torch.tensor([0, 5, nq // 2, nq - 1], device=cuda)
        q[rows, d - 1] = float("nan")
        dd, ii = tk().nn_distance(ref, q, k)
        assert torch.isinf(dd[rows]).all() and (ii[rows] == -1).all()
        few = torch.cat([rows, torch.arange(1000, 1100, device=cuda)])
        want_d = torch.empty(len(few), k, dtype=ref.dtype, device=cuda)
        want_i = torch.empty(len(few), k, dtype=torch.int32, device=cuda)
        nn_distance_raw(ref, q[few].contiguous(), k, want_d, want_i, "exact")
        assert torch.equal(dd[few], want_d) and torch.equal(ii[few], want_i)


@pytest.mark.parametrize("mode", ["exact", "tf32", "bf16_split"])
@pytest.mark.parametrize("d", [4, 8, 32])
def test_tiny_coordinates(mode, d, oracle):
    """Clouds so small that products of coordinates are subnormal or zero,
    where the relative error bounds of the tensor-core products do not hold."""
    rng = np.random.default_rng(d)
    ref = rng.standard_normal((5_000, d))
    q = rng.standard_normal((500, d))
    for e in np.arange(-23.0, -16.0, 0.25):
        r, p = (ref * 10.0 ** e).astype(np.float32), (q * 10.0 ** e).astype(np.float32)
        bd, bi = oracle.brute(r, p, 8)
        dd, ii = tk().nn_distance(torch.from_numpy(r).to(cuda), torch.from_numpy(p).to(cuda), 8, mode=mode)
        np.testing.assert_array_equal(dd.cpu().numpy(), bd, err_msg=f"1e{e}")
        np.testing.assert_array_equal(ii.cpu().numpy(), bi, err_msg=f"1e{e}")


@pytest.mark.parametrize("n_listed", [257, 1_000, 1_025, 3_000])
@pytest.mark.parametrize("n", [600, 9_000])
@pytest.mark.parametrize("k,d", [(1, 8), (20, 8), (64, 20)])
def test_many_recomputed_queries(n_listed, n, k, d, oracle):
    """Lists of some tiles of queries up to all of them, searched by a block
    per tile and slice, with one slice of the references and with several."""
    rng = np.random.default_rng(n_listed + k)
    ref = np.concatenate([rng.standard_normal((n, d)), np.tile(rng.standard_normal((1, d)) + 20, (400, 1))])
    ref = ref[rng.permutation(len(ref))].astype(np.float32)
    q = rng.standard_normal((3_000, d)).astype(np.float32)
    hard = rng.permutation(len(q))[:n_listed]
    q[hard] = (20 + 0.1 * rng.standard_normal((n_listed, d))).astype(np.float32)
    bd, bi = oracle.brute(ref, q, k)
    for mode in ("tf32", "bf16_split"):
        dd, ii = tk().nn_distance(torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda), k, mode=mode)
        np.testing.assert_array_equal(dd.cpu().numpy(), bd)
        np.testing.assert_array_equal(ii.cpu().numpy(), bi)


@pytest.mark.parametrize("mode", ["exact", "tf32", "bf16_split"])
@pytest.mark.parametrize("d", [4, 8, 32, 39])
@pytest.mark.parametrize("mean", [30.0, -3000.0, "one coordinate"])
def test_clouds_far_from_the_origin(mode, d, mean, oracle):
    """The candidate search takes points relative to the cloud's middle; its
    answers stay exact, and hardly a query needs the exhaustive search."""
    from test_bounded_wait_gpu import run
    rng = np.random.default_rng(d)
    ref = rng.standard_normal((20_000, d))
    q = rng.standard_normal((1_000, d))
    if mean == "one coordinate":
        ref[:, d - 1] += 500
        q[:, d - 1] += 500
    else:
        ref, q = ref + mean, q + mean
    ref, q = ref.astype(np.float32), q.astype(np.float32)
    rt, qt = torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda)
    for k in (1, 8):
        bd, bi = oracle.brute(ref, q, k)
        dd, ii = tk().nn_distance(rt, qt, k, mode=mode)
        np.testing.assert_array_equal(dd.cpu().numpy(), bd)
        np.testing.assert_array_equal(ii.cpu().numpy(), bi)
    if mode == "bf16_split" and mean != -3000.0:
        recomputed = run(rt, qt, 8, mode)[4]
        assert recomputed < len(q) // 10, recomputed


@pytest.mark.parametrize("mode", ["exact", "tf32", "bf16_split"])
@pytest.mark.parametrize("d", [4, 8, 32])
@pytest.mark.parametrize("clusters,apart", [(2, 300.0), (64, 100.0), (64, 10.0), (1000, 100.0)])
def test_distant_clusters(mode, d, clusters, apart, oracle):
    """Clusters whose distances to one another dwarf those within: the lists go
    on by the scores' error where they hold what is there, and rows without a
    chance take no hits; also next to rows of a cloud around the middle."""
    rng = np.random.default_rng(clusters + d)
    n, nq = 20_000, 1_500
    at = (rng.standard_normal((clusters, d)) * apart).astype(np.float32)
    at[0] = 0
    pick = rng.integers(0, clusters, nq)
    pick[: nq // 3] = 0  # whole blocks of rows around the middle
    ref = (at[rng.integers(0, clusters, n)] + rng.standard_normal((n, d))).astype(np.float32)
    q = (at[pick] + rng.standard_normal((nq, d))).astype(np.float32)
    rt, qt = torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda)
    for k in (1, 8, 32):
        bd, bi = oracle.brute(ref, q, k)
        dd, ii = tk().nn_distance(rt, qt, k, mode=mode)
        np.testing.assert_array_equal(dd.cpu().numpy(), bd)
        np.testing.assert_array_equal(ii.cpu().numpy(), bi)


def test_clusters_that_the_lists_hold_are_certified():
    """312 references a cluster, 100 spreads apart: more of them lie within the
    scores' error than the sample's threshold lets through, and fit the lists."""
    from test_bounded_wait_gpu import run
    rng = np.random.default_rng(0)
    at = (rng.standard_normal((64, 8)) * 100).astype(np.float32)
    ref = (at[rng.integers(0, 64, 20_000)] + rng.standard_normal((20_000, 8))).astype(np.float32)
    q = (at[rng.integers(0, 64, 2_000)] + rng.standard_normal((2_000, 8))).astype(np.float32)
    recomputed = run(torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda), 8, "bf16_split")[4]
    assert recomputed < len(q) // 4, recomputed


@pytest.mark.parametrize("mode", ["tf32", "bf16_split"])
def test_tensor_core_modes_in_several_passes(mode, oracle):
    """The modes that name the tensor cores take a million queries a pass: ten
    million ask for no more workspace than that; the report counts all passes."""
    from torch_kdtree_gb300 import _lib
    from torch_kdtree_gb300._lib import LIB
    from torch_kdtree_gb300.nn_distance import _BRUTE_MODES
    from test_bounded_wait_gpu import run
    for d, k in ((8, 1), (32, 32)):
        assert LIB.tk_nn_distance_workspace_size(1_000_000, 10_000_000, d, k, _lib.TK_F32, _BRUTE_MODES[mode]) < 6 << 30
    rng = np.random.default_rng(1)
    nq = (1 << 20) + 1_000
    ref = np.concatenate([rng.standard_normal((2_000, 4)), np.tile(rng.standard_normal((1, 4)) + 20, (700, 1))])
    ref = ref.astype(np.float32)
    q = rng.standard_normal((nq, 4)).astype(np.float32)
    hard = np.concatenate([np.arange(300, 340), np.arange(nq - 50, nq - 20)])  # no certificate: all equally far
    q[hard] = (20 + 0.1 * rng.standard_normal((len(hard), 4))).astype(np.float32)
    dd, ii, rc, flags, recomputed = run(torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda), 2, mode)
    assert rc == 0 and flags == 0 and recomputed >= len(hard)
    rows = np.concatenate([np.arange(250, 450), np.arange((1 << 20) - 100, nq)])
    bd, bi = oracle.brute(ref, q[rows], 2)
    np.testing.assert_array_equal(dd.cpu().numpy()[rows], bd)
    np.testing.assert_array_equal(ii.cpu().numpy()[rows], bi)


@pytest.mark.parametrize("d", [4, 8, 16, 32])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 8, 255, 256, 257, 511, 1023])
def test_nearest_at_the_edges_of_a_tile(d, n, oracle):
    """k = 1 takes eight references at a time: tiles that end anywhere in them."""
    rng = np.random.default_rng(n)
    ref = np.round(rng.standard_normal((n, d)) * 2).astype(np.float32)
    q = np.round(rng.standard_normal((300, d)) * 2).astype(np.float32)
    dd, ii = tk().nn_distance(torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda), 1)
    bd, bi = oracle.brute(ref, q, 1)
    np.testing.assert_array_equal(dd.cpu().numpy(), bd)
    np.testing.assert_array_equal(ii.cpu().numpy(), bi)
