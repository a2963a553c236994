"""GPU tree construction (tk_tree_create_device): the layout must equal the
host build's bit for bit -- point order, original indices, split values and
leaf offsets -- and through it the reference's own layouts (golden fixtures,
whose host-build equality test_abi pins), on tie-free, tie-heavy, signed-zero
and infinite coordinates, every dimension and dtype, and every depth."""
import ctypes

import numpy as np
import pytest
import torch

from golden_util import inputs_of
from test_abi import host_tree, layout_of

pytestmark = pytest.mark.gpu

cuda = torch.device("cuda")


def device_tree(points: np.ndarray, levels: int):
    from torch_kdtree_gb300._lib import LIB
    t = torch.from_numpy(points).to(cuda)
    h = ctypes.c_void_p()
    dt = 0 if points.dtype == np.float32 else 1
    st = LIB.tk_tree_create_device(t.data_ptr(), points.shape[0], points.shape[1], dt, levels, 0,
                                   torch.cuda.current_stream().cuda_stream, ctypes.byref(h))
    return st, h


def both_layouts(points: np.ndarray, levels: int):
    from torch_kdtree_gb300._lib import LIB, check
    n, d = points.shape
    st, hh = host_tree(points, levels)
    check(st)
    st, hd = device_tree(points, levels)
    try:
        check(st)
        return (layout_of(hh, n, d, levels, points.dtype), layout_of(hd, n, d, levels, points.dtype))
    finally:
        LIB.tk_tree_destroy(hh)
        if hd.value:
            LIB.tk_tree_destroy(hd)


def assert_same_layout(points, levels):
    a, b = both_layouts(points, levels)
    for x, y in zip(a, b):
        assert x.dtype == y.dtype
        np.testing.assert_array_equal(x.view(np.uint8), y.view(np.uint8))  # bitwise


def clouds(dtype, d, n, seed):
    rng = np.random.default_rng(seed)
    yield "normal", rng.standard_normal((n, d)).astype(dtype)
    yield "grid", rng.integers(-3, 4, size=(n, d)).astype(dtype)  # heavy coordinate ties
    p = rng.standard_normal((n, d)).astype(dtype)
    p[rng.permutation(n)[: n // 3]] = p[rng.integers(0, n, size=n // 3)]  # exact duplicate points
    yield "dups", p
    z = rng.standard_normal((n, d)).astype(dtype)
    z[rng.random(n) < 0.3, 0] = dtype(0.0)
    z[rng.random(n) < 0.3, 0] = -dtype(0.0)  # signed zeros tie with each other
    yield "signed_zero", z
    w = (rng.standard_normal((n, d)) * 1e3).astype(dtype)
    w[rng.random(n) < 0.02, -1] = np.inf
    w[rng.random(n) < 0.02, 0] = -np.inf
    yield "inf", w


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("d", [1, 2, 3, 4, 5, 8])
def test_device_build_equals_host_build(dtype, d):
    for n in (1, 2, 3, 17, 1000, 65537):
        lmax = max(1, int(np.floor(np.log2(n))) + 1)  # leaf parents need >= 1 point: n >= 2^(L-1)
        for levels in sorted({max(1, min(lmax, x)) for x in (1, 2, 5, lmax - 3, lmax)}):
            for kind, pts in clouds(dtype, d, n, seed=n * 7 + d):
                try:
                    assert_same_layout(pts, levels)
                except AssertionError as e:
                    raise AssertionError(f"{kind} n={n} d={d} L={levels} {dtype.__name__}") from e


def test_device_build_equals_host_build_large():
    from torch_kdtree_gb300.synthetic import cube_and_sphere
    ref, _ = cube_and_sphere(n_ref=1 << 20, n_query=16, seed=3)
    for levels in (13, 16, 19):
        assert_same_layout(ref, levels)


@pytest.mark.parametrize("name", [
    "grid_f32_d1_n1000_q200_k10", "grid_f32_d2_n10000_q300_k20", "grid_f32_d3_n10000_q300_k20",
    "grid_f64_d1_n10000_q300_k20", "grid_f64_d3_n1000_q200_k10", "grid_f32_d3_n30_q20_k5",
    "grid_f64_d2_n5_q5_k1", "levels_f32_d3_n1000_L9", "levels_f32_d3_n1000_L1"])
def test_device_build_matches_reference_layout(name, golden):
    from torch_kdtree_gb300._lib import LIB, check
    case = golden[name]
    ref, _ = inputs_of(case)
    n, d = ref.shape
    L = int(case["levels"])
    st, h = device_tree(ref, L)
    check(st)
    try:
        pts, perm, med, off = layout_of(h, n, d, L, ref.dtype)
    finally:
        LIB.tk_tree_destroy(h)
    np.testing.assert_array_equal(pts, case["structured"])
    np.testing.assert_array_equal(perm, case["perm"])
    np.testing.assert_array_equal(med, case["medians"])
    np.testing.assert_array_equal(off[:-1], case["leaf_off"])


def test_device_built_tree_queries_like_host_built(oracle):
    import torch_kdtree_gb300 as tk
    rng = np.random.default_rng(21)
    ref = rng.standard_normal((50_000, 3)).astype(np.float32)
    q = rng.standard_normal((4000, 3)).astype(np.float32)
    rt, qt = torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda)
    th = tk.build_kd_tree(rt, build="host", levels=12)
    td = tk.build_kd_tree(rt, build="device", levels=12)
    assert th.built_on == "host" and td.built_on == "device"
    assert tk.build_kd_tree(rt).built_on == "device"  # auto picks the GPU for CUDA input
    assert torch.equal(th.shuffled_ind, td.shuffled_ind)
    assert torch.equal(th.structured_points, td.structured_points)
    for k in (1, 16, 100):
        dh, ih = th.query(qt, nr_nns_searches=k)
        dd, id_ = td.query(qt, nr_nns_searches=k)
        assert torch.equal(dh, dd) and torch.equal(ih, id_)
    bd, bi = oracle.brute(ref, q, 16)
    dd, id_ = td.query(qt, nr_nns_searches=16)
    np.testing.assert_array_equal(dd.cpu().numpy(), bd)
    np.testing.assert_array_equal(id_.cpu().numpy(), bi)


def test_device_build_errors():
    from torch_kdtree_gb300._lib import LIB, TK_EINVAL
    import torch_kdtree_gb300 as tk
    pts = np.random.default_rng(0).standard_normal((100, 3)).astype(np.float32)
    st, h = device_tree(pts, 8)  # leaf parents at depth 7 need >= 128 points
    assert st == TK_EINVAL and not h.value
    bad = pts.copy()
    bad[37, 1] = np.nan
    st, h = device_tree(bad, 3)
    assert st == TK_EINVAL and b"NaN" in LIB.tk_last_error()
    host = torch.from_numpy(pts)
    h = ctypes.c_void_p()
    st = LIB.tk_tree_create_device(host.data_ptr(), 100, 3, 0, 3, 0, None, ctypes.byref(h))
    assert st == TK_EINVAL  # host memory is refused
    with pytest.raises(Exception):
        tk.build_kd_tree(torch.from_numpy(bad).to(cuda), levels=3)
    with pytest.raises(Exception):
        tk.build_kd_tree(torch.from_numpy(pts).to(cuda), levels=8)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [1023, 1025, 4095, 4096, 4097, 8191, 8192, 8193, 12289, 16385])
def test_device_build_around_block_capacities(dtype, n):
    """One block sorts and finishes clouds and subtrees of up to 4,096 points;
    radix tiles hold 4,096 (float32) or 2,048 keys, partition tiles 1,024."""
    lmax = int(np.floor(np.log2(n))) + 1
    for d in (1, 2, 3, 5, 8):
        for levels in (1, 3, lmax - 4, lmax):
            for kind, pts in clouds(dtype, d, n, seed=n + d):
                try:
                    assert_same_layout(pts, levels)
                except AssertionError as e:
                    raise AssertionError(f"{kind} n={n} d={d} L={levels} {dtype.__name__}") from e


def test_device_build_one_axis_at_a_time():
    """Above 32M points the axes are sorted and partitioned one after the
    other: two levels of 33.6M points with many ties, against stable sorts."""
    import torch_kdtree_gb300 as tk
    n = 33_600_000
    g = torch.Generator(device=cuda)
    g.manual_seed(5)
    pts = torch.randint(0, 1 << 20, (n, 2), generator=g, device=cuda).float()
    tree = tk.build_kd_tree(pts, levels=2)
    order = torch.sort(pts[:, 0], stable=True).indices
    want = []
    for half in (order[: n // 2], order[n // 2:]):
        ids = half.sort().values
        want.append(ids[torch.sort(pts[ids, 1], stable=True).indices])
    assert torch.equal(tree.shuffled_ind, torch.cat(want))


def test_tree_outlives_its_stream():
    """A tree's memory belongs to the stream it was built on: dropping the tree
    while another stream still queries it must not hand that memory on."""
    import torch_kdtree_gb300 as tk
    ref = torch.randn(300_000, 3, device=cuda)
    q = torch.randn(200_000, 3, device=cuda)
    want_d, want_i = tk.build_kd_tree(ref).query(q, nr_nns_searches=8)
    side = torch.cuda.Stream()
    for _ in range(5):
        tree = tk.build_kd_tree(ref)
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            d, i = tree.query(q, nr_nns_searches=8)
        del tree
        junk = [torch.full((1 << 22,), -1.0, device=cuda) for _ in range(8)]
        torch.cuda.synchronize()
        assert torch.equal(d, want_d) and torch.equal(i, want_i)
        del junk


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("d", [1, 2, 3, 6])
def test_default_depth_tree(dtype, d, oracle, tmp_path):
    """With the default depth the library searches deeper or shallower leaves
    than the layout it reports: the layout stays the host build's, and every
    launch shape, a saved and re-loaded tree and a batch give the exhaustive
    answer."""
    import torch_kdtree_gb300 as tk
    from torch_kdtree_gb300._lib import QueryOpts
    from torch_kdtree_gb300.batched import BatchedKDTrees
    for n in (1, 2, 40, 700, 9000, 300_000):
        for kind, ref in list(clouds(dtype, d, n, seed=n + 3 * d))[:3]:
            q = np.concatenate([ref[:50], np.random.default_rng(n).standard_normal((150, d)).astype(dtype)])
            rt, qt = torch.from_numpy(ref).to(cuda), torch.from_numpy(q).to(cuda)
            tree = tk.build_kd_tree(rt)
            host = tk.build_kd_tree(rt, build="host")
            assert tree.levels == host.levels and tree.built_on == "device"
            assert torch.equal(tree.shuffled_ind, host.shuffled_ind)
            assert torch.equal(tree.structured_points, host.structured_points)
            tree.save(tmp_path / "t.npz")
            loaded = tk.load_kd_tree(tmp_path / "t.npz")
            for k in sorted({1, min(n, 16), min(n, 70)}):
                bd, bi = oracle.brute(ref, q, k)
                for lanes in (0, 1, 4, 32):
                    for traversal in (0, 2):
                        tree.query_opts = QueryOpts.make(threads_per_query=lanes, traversal=traversal)
                        dd, ii = tree.query(qt, nr_nns_searches=k)
                        np.testing.assert_array_equal(dd.cpu().numpy(), bd, err_msg=f"{kind} {n} {k} {lanes}")
                        np.testing.assert_array_equal(ii.cpu().numpy(), bi)
                dd, ii = loaded.query(qt, nr_nns_searches=k)
                np.testing.assert_array_equal(ii.cpu().numpy(), bi)
                bdd, bii = BatchedKDTrees([rt, rt], [k, 1], [len(q), 0]).query([qt, qt[:0]])
                np.testing.assert_array_equal(bii[0].cpu().numpy(), bi)
                np.testing.assert_array_equal(bdd[0].cpu().numpy(), bd)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [4000, 5000, 100_000])
def test_device_build_refuses_nan_at_every_size(dtype, n):
    """NaN coordinates have a place in the sort order, so the passes stay inside
    their arrays and the build ends with the error."""
    import torch_kdtree_gb300 as tk
    from torch_kdtree_gb300._lib import TK_EINVAL
    rng = np.random.default_rng(n)
    for share in (1, n // 3):
        pts = rng.standard_normal((n, 3)).astype(dtype)
        pts[rng.permutation(n)[:share], rng.integers(0, 3, share)] = np.nan
        st, h = device_tree(pts, 9)
        assert st == TK_EINVAL and not h.value
        with pytest.raises(Exception, match="NaN"):
            tk.build_kd_tree(torch.from_numpy(pts).to(cuda))
    good = torch.randn(n, 3, device=cuda)
    d, _ = tk.build_kd_tree(good).query(good[:100])
    assert float(d.max()) == 0.0


@pytest.mark.parametrize("dtype,n", [(np.float32, 131_072), (np.float32, 131_073), (np.float64, 65_536),
                                     (np.float64, 65_537), (np.float32, 2_097_152), (np.float32, 2_097_153)])
def test_device_build_around_scan_limits(dtype, n):
    """Clouds whose radix or level tiles just fit, or no longer fit, the sums
    that the blocks take themselves."""
    rng = np.random.default_rng(n)
    pts = rng.standard_normal((n, 2)).astype(dtype)
    pts[: n // 4] = np.round(pts[: n // 4], 1)
    assert_same_layout(pts, 7)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("d", [1, 2, 3, 5])
@pytest.mark.parametrize("n", [1_000, 4_097, 300_000])
def test_layout_of_a_deeper_image(dtype, d, n):
    """The layout that a default-depth tree reports, put in order from its
    deeper image: the host builder's, with ties, zeros of both signs and
    infinite coordinates."""
    from torch_kdtree_gb300 import build_kd_tree
    rng = np.random.default_rng(d)
    pts = np.round(rng.standard_normal((n, d)) * 50).astype(dtype)
    pts[rng.integers(0, n, n // 10)] *= -0.0
    pts[rng.integers(0, n, 5), 0] = np.inf
    td = build_kd_tree(torch.from_numpy(pts).cuda())
    th = build_kd_tree(torch.from_numpy(pts), device=torch.device("cuda"))
    assert torch.equal(td.shuffled_ind, th.shuffled_ind)
    assert torch.equal(td.structured_points, th.structured_points)


def test_tree_in_a_graph_is_kept_from_its_stream():
    """A query captured on the stream that built the tree may be replayed on
    any other: the tree's memory waits for all of them when it goes."""
    from torch_kdtree_gb300 import build_kd_tree
    from torch_kdtree_gb300.batched import BatchedKDTrees
    s = torch.cuda.Stream()
    ref, q = torch.randn(5_000, 3, device="cuda"), torch.randn(200, 3, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        tree = build_kd_tree(ref)
        batch = BatchedKDTrees([ref], [4], [len(q)])
        want = tree.query(q, 4)
        batch.query_flat(q)
        s.synchronize()
        assert not tree._tree.other_streams and not batch.trees[0]._tree.other_streams
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        got = tree.query(q, 4)
        batch.query_flat(q)
    assert tree._tree.other_streams and batch.trees[0]._tree.other_streams
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    assert torch.equal(batch.out_dists.view(-1, 4), want[0])
