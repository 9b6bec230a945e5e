"""GPU parity tests: every stage of the CUDA tree builder and the whole BUILD_TREE / PREDICT calls
against the CPU oracle on identical seeded inputs, through the C ABI (liblbk.so).

Bars: integer / index results bit-exact; float histograms <= 1e-5 relative (to the largest
magnitude of the histogram); predictions bit-exact (the bar is <= 1e-4)."""
import glob
import os

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lb():
    import legateboost_b200 as lb
    from legateboost_b200 import stages  # noqa: F401

    assert torch.cuda.is_available(), "these tests need a CUDA device"
    lb.library.load()  # fails loudly if liblbk.so is missing
    return lb


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def tree_tuple(t):
    return (t.leaf_value, t.feature, t.split_value)


def to_row_major(bins_p, F):
    """Drops the padding columns of the kernels' layout (rows padded to whole 32-feature groups)."""
    assert bins_p.shape[1] == (F + 31) // 32 * 32
    assert not bins_p[:, F:].any()
    return bins_p[:, :F]


# ---------------------------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("N,F,S", [(1000, 7, 16), (5000, 50, 256), (300, 33, 500), (64, 3, 2048), (2, 1, 256)])
def test_split_proposals_and_bins(lb, oracle, dtype, N, F, S):
    from legateboost_b200 import stages

    rs = np.random.RandomState(N + F)
    X = rs.random((N, F)).astype(dtype)
    X[:, 0] = np.round(X[:, 0] * 3)  # a low-cardinality feature
    for seed in (0, 1872583848):
        want_p, want_rp = oracle.split_proposals(X, S, seed, mode="Q")
        got_p, got_rp = stages.split_proposals(dev(X), S, seed)
        assert np.array_equal(got_rp.cpu().numpy(), want_rp)
        assert np.array_equal(got_p.cpu().numpy(), want_p)
        want_bins = oracle.bin_x(X, want_p, want_rp)
        mb = int(np.diff(want_rp).max())
        bb = 1 if mb <= 256 else 2
        got = stages.bin_matrix(dev(X), got_p, got_rp, bin_bytes=bb)
        assert np.array_equal(to_row_major(got, F).cpu().numpy().astype(np.int16), want_bins)


@pytest.mark.parametrize("N,K", [(1, 1), (1000, 1), (5000, 3), (70000, 2), (1 << 21, 1)])
def test_quantise(lb, oracle, N, K):
    from legateboost_b200 import stages

    rs = np.random.RandomState(N)
    g = rs.normal(size=(N, K)) * 10.0 ** rs.randint(-2, 3, size=(N, K))
    h = rs.random((N, K)) + 1e-8
    want_q, want_scale = oracle.quantise(g, h, seed=1234567)
    gp, root, scale = stages.quantise(dev(g), dev(h), seed=1234567)
    assert np.array_equal(scale.cpu().numpy(), want_scale)
    assert np.array_equal(gp.cpu().numpy().astype(np.int64), want_q)
    assert np.array_equal(root.cpu().numpy(), want_q.sum(axis=0))


@pytest.mark.parametrize("g,h", [
    ([5.0], [0.25]), ([-5.0], [3.0]), ([0.0], [0.0]), ([-0.0, 0.0], [0.0, 1e-290]), ([1e-12, -1e12, 3.5], [1e-8, 1.0, 1e8]),
    ([2.0 ** 30, -(2.0 ** 30)], [1.0, 1.0]), ([1.0, -1.0] * 700, [0.5] * 1400),
])
def test_quantise_whole_numbers_at_the_ends(lb, oracle, g, h):
    """Values that are whole multiples of the scale, the largest magnitudes, zeros of both signs."""
    from legateboost_b200 import stages

    g, h = np.array(g)[:, None], np.array(h)[:, None]
    for seed in (0, 7, 2 ** 31 - 1):
        want_q, want_scale = oracle.quantise(g, h, seed=seed)
        gp, _, scale = stages.quantise(dev(g), dev(h), seed=seed)
        assert np.array_equal(gp.cpu().numpy().reshape(want_q.shape), want_q)
        assert np.array_equal(scale.cpu().numpy(), want_scale)


def test_quantise_row_offset(lb, oracle):
    # the quantised pair depends on the GLOBAL row id: a shard quantised on its own, with the
    # scale of its own |g| sum, must equal the oracle's shard
    from legateboost_b200 import stages

    rs = np.random.RandomState(0)
    g = rs.normal(size=(4000, 2))
    h = np.ones((4000, 2))
    gp, _, scale = stages.quantise(dev(g[1000:3000]), dev(h[1000:3000]), seed=99, row_offset=1000)
    want_q, want_scale = oracle.quantise(g, h, seed=99, rank_off=[0, 1000, 3000, 4000])
    # the oracle takes the max over shards; compare only when this shard carries the max
    single_q, single_scale = oracle.quantise(g[1000:3000], h[1000:3000], seed=99)
    assert np.array_equal(scale.cpu().numpy(), single_scale)
    if np.array_equal(single_scale, want_scale):
        assert np.array_equal(gp.cpu().numpy().astype(np.int64), want_q[1000:3000])


# ---------------------------------------------------------------------------------------------
def _hist_case(rs, N, F, K, n_nodes, nb):
    bins = rs.randint(0, nb, size=(N, F)).astype(np.uint8)
    row_ptr = (np.arange(F + 1) * nb).astype(np.int32)
    node = rs.randint(0, n_nodes, size=N).astype(np.int32) + (n_nodes - 1)
    return bins, row_ptr, node


@pytest.mark.parametrize("N,F,K,n_nodes,nb", [(200000, 128, 1, 128, 256), (50000, 50, 3, 8, 256),
                                              (3000, 100, 1, 64, 7), (100, 5, 2, 4, 256), (70000, 64, 1, 1, 256),
                                              (60000, 70, 2, 5, 200), (90000, 161, 1, 3, 256)])
def test_histogram_int_exact(lb, oracle, N, F, K, n_nodes, nb):
    from legateboost_b200 import stages

    rs = np.random.RandomState(F)
    bins, row_ptr, node = _hist_case(rs, N, F, K, n_nodes, nb)
    q = rs.randint(-(2 ** 20), 2 ** 20, size=(N, K, 2)).astype(np.int32)
    q[:, :, 1] = np.abs(q[:, :, 1])
    want = oracle.histogram_q(bins, row_ptr, q, node, n_nodes - 1, 2 * n_nodes - 1)
    row_index, seg = stages.group_rows(dev(node), n_nodes - 1, n_nodes)
    # grouping is stable: rows ascending inside each node
    ri, sg = row_index.cpu().numpy(), seg.cpu().numpy()
    assert sg[-1] == N
    for j in range(n_nodes):
        r = ri[sg[j]:sg[j + 1]]
        assert np.all(node[r] == j + n_nodes - 1) and np.all(np.diff(r) > 0)
    got = stages.histogram(stages.to_padded_rows(dev(bins)), dev(row_ptr), dev(q), row_index, seg, F, mode=0)
    assert np.array_equal(got.cpu().numpy(), want)
    # the same pairs stored in row_index order (as the tree builder keeps them)
    got = stages.histogram(stages.to_padded_rows(dev(bins)), dev(row_ptr), _by_position(dev(q), row_index), row_index, seg,
                           F, mode=0, pairs_by_position=True, max_abs=_max_abs(q))
    assert np.array_equal(got.cpu().numpy(), want)


def _by_position(pairs, row_index):
    return pairs[row_index.long()].contiguous()


def _max_abs(q):
    return dev(np.abs(q.astype(np.int64)).reshape(-1, 2).max(axis=0).astype(np.int32))


@pytest.mark.parametrize("F,K", [(32, 2), (64, 1)])
def test_histogram_many_large_nodes(lb, oracle, F, K):
    """More large, unequal nodes than resident blocks, some of them empty: the planner cuts the
    larger nodes into chunks that leave partial sums; the sums stay exact."""
    from legateboost_b200 import stages

    N, n_nodes = 6_000_000, 200
    rng = np.random.default_rng(F + K)
    weight = rng.uniform(0.5, 1.5, size=n_nodes)
    weight[[0, 17, 18, 199]] = 0.0  # empty nodes, at both ends and in a row
    edges = np.cumsum(weight / weight.sum())
    node = np.minimum(np.searchsorted(edges, rng.random(N), side="right"), n_nodes - 2).astype(np.int32) + (n_nodes - 1)
    bins = rng.integers(0, 256, size=(N, F), dtype=np.uint8)
    row_ptr = (np.arange(F + 1) * 256).astype(np.int32)
    q = rng.integers(-200, 200, size=(N, K, 2), dtype=np.int32)
    q[:, :, 1] = np.abs(q[:, :, 1])
    want = oracle.histogram_q(bins, row_ptr, q, node, n_nodes - 1, 2 * n_nodes - 1)
    row_index, seg = stages.group_rows(dev(node), n_nodes - 1, n_nodes)
    got = stages.histogram(stages.to_padded_rows(dev(bins)), dev(row_ptr), dev(q), row_index, seg, F, mode=0)
    assert np.array_equal(got.cpu().numpy(), want)


def test_histogram_int_no_wraparound(lb, oracle):
    """Partial sums that exceed int32 in one chunk must still come out exact."""
    from legateboost_b200 import stages

    N, F = 6000, 4
    rs = np.random.RandomState(5)
    bins = np.zeros((N, F), dtype=np.uint8)  # everything in one bin
    row_ptr = (np.arange(F + 1) * 2).astype(np.int32)
    node = np.zeros(N, dtype=np.int32)
    q = np.full((N, 1, 2), 2 ** 30, dtype=np.int32)  # sums reach 6000 * 2^30
    q[::2, 0, 0] *= -1
    q[:, 0, 0] += rs.randint(0, 1000, size=N).astype(np.int32)
    want = oracle.histogram_q(bins, row_ptr, q, node, 0, 1)
    row_index, seg = stages.group_rows(dev(node), 0, 1)
    got = stages.histogram(stages.to_padded_rows(dev(bins)), dev(row_ptr), dev(q), row_index, seg, F, mode=0)
    assert np.array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize("N,F,K,n_nodes", [(200000, 128, 1, 128), (20000, 40, 2, 16)])
def test_histogram_float_tolerance(lb, oracle, N, F, K, n_nodes):
    from legateboost_b200 import stages

    rs = np.random.RandomState(7)
    bins, row_ptr, node = _hist_case(rs, N, F, K, n_nodes, 256)
    gh = np.stack([rs.normal(size=(N, K)), np.ones((N, K))], axis=2).astype(np.float32)
    want = oracle.histogram_d(bins, row_ptr, gh[:, :, 0].copy(), gh[:, :, 1].copy(), node, n_nodes - 1, 2 * n_nodes - 1)
    row_index, seg = stages.group_rows(dev(node), n_nodes - 1, n_nodes)
    got = stages.histogram(stages.to_padded_rows(dev(bins)), dev(row_ptr), dev(gh), row_index, seg, F, mode=1)
    got = got.cpu().numpy()
    scale = np.abs(want).max()
    assert np.abs(got - want).max() <= 1e-5 * scale


def test_histogram_host_buffers(lb, oracle):
    from legateboost_b200 import stages

    rs = np.random.RandomState(11)
    N, F, K, n_nodes = 30000, 64, 1, 8
    bins, row_ptr, node = _hist_case(rs, N, F, K, n_nodes, 256)
    q = rs.randint(-1000, 1000, size=(N, K, 2)).astype(np.int32)
    want = oracle.histogram_q(bins, row_ptr, q, node, n_nodes - 1, 2 * n_nodes - 1)
    row_index, seg = stages.group_rows(dev(node), n_nodes - 1, n_nodes)
    bins_g = stages.to_padded_rows(dev(bins)).cpu().pin_memory()
    got = stages.histogram(bins_g, torch.from_numpy(row_ptr), torch.from_numpy(q).pin_memory(),
                           row_index.cpu(), seg.cpu(), F, mode=0, host=True)
    assert np.array_equal(got.numpy(), want)


# ---------------------------------------------------------------------------------------------
TREE_CASES = [
    # N, F, K, depth, S, dtype, kwargs
    (1000, 10, 1, 4, 64, np.float32, {}),
    (5000, 20, 3, 6, 256, np.float64, {}),
    (300, 5, 2, 8, 16, np.float32, {}),
    (10000, 100, 5, 7, 256, np.float64, {}),
    (20000, 50, 1, 6, 256, np.float32, {}),
    (2000, 33, 1, 5, 500, np.float32, {}),                      # two-byte bins
    (3000, 12, 2, 6, 64, np.float32, {"l1": 0.5, "l2": 2.0, "min_split_gain": 0.01}),
    (2, 1, 1, 12, 256, np.float64, {}),
    (500, 6, 1, 0, 32, np.float32, {}),                          # depth 0: root only
    (4000, 9, 1, 5, 128, np.float32, {"mask": True}),
]


def _run_tree_case(lb, oracle, case, seed, n_ranks=1, trace_nodes=0, hess_small=False):
    from legateboost_b200.tree import build_tree_arrays

    N, F, K, D, S, dt, kw = case
    kw = dict(kw)
    rs = np.random.RandomState(N * 7 + F)
    X = rs.random((N, F)).astype(dt)
    X[:, 0] = np.round(X[:, 0] * 5) / 5
    g = rs.normal(size=(N, K))
    h = rs.random((N, K)) * (1e-3 if hess_small else 1.0) + (0.0 if hess_small else 0.1)
    mask = None
    if kw.pop("mask", False):
        mask = rs.random(F) < 0.5
        mask[0] = True
    want = oracle.build_tree(X, g, h, max_depth=D, split_samples=S, seed=seed, mode="Q", feature_set=mask,
                             trace_nodes=trace_nodes, **kw)
    got = build_tree_arrays(dev(X), dev(g), dev(h), max_depth=D, split_samples=S, seed=seed,
                            feature_set=None if mask is None else torch.from_numpy(mask),
                            row_offset=0, dataset_rows=N, trace_nodes=trace_nodes, **kw)
    return X, want, got


@pytest.mark.parametrize("case", TREE_CASES, ids=[str(c[:5]) for c in TREE_CASES])
def test_build_tree_bit_exact(lb, oracle, case):
    for seed in (2, 1872583848):
        X, want, got = _run_tree_case(lb, oracle, case, seed)
        assert got["B"] == want.B
        assert np.array_equal(got["node_sums"].cpu().numpy(), want.node_sums)
        assert np.array_equal(got["feature"].cpu().numpy(), want.feature)
        assert np.array_equal(got["split_value"].cpu().numpy(), want.split_value)
        assert np.array_equal(got["gain"].cpu().numpy(), want.gain)
        assert np.array_equal(got["leaf_value"].cpu().numpy(), want.leaf_value)
        assert np.array_equal(got["hessian"].cpu().numpy(), want.hessian)


def test_build_tree_histograms_bit_exact(lb, oracle):
    """Every node's histogram as it was when its split was evaluated (scan, write-skip rule,
    sibling subtraction), including a case where quantised hessians of 0 occur."""
    for case, small in (((3000, 8, 2, 5, 32, np.float32, {}), False), ((3000, 8, 2, 5, 32, np.float32, {}), True)):
        D = case[3]
        nodes = 2 ** D - 1
        X, want, got = _run_tree_case(lb, oracle, case, seed=5, trace_nodes=nodes, hess_small=small)
        assert np.array_equal(got["trace_hist"].cpu().numpy(), want.trace_hist)
        assert np.array_equal(got["feature"].cpu().numpy(), want.feature)


def test_scratch_through_the_callers_allocator(lb):
    """lbk_context_set_allocator: with torch's caching allocator behind the callbacks a whole tree is
    built without the library's own pool reserving a byte, and it is the same tree."""
    from legateboost_b200.tree import build_tree_arrays

    N, F, K, D = 50000, 40, 2, 6
    rs = np.random.RandomState(3)
    X, g, h = dev(rs.random((N, F)).astype(np.float32)), dev(rs.normal(size=(N, K))), dev(rs.random((N, K)) + 0.1)
    kw = dict(max_depth=D, split_samples=256, seed=9, row_offset=0, dataset_rows=N, want_leaf=True)
    want = build_tree_arrays(X, g, h, **kw)
    ctx = lb.library.context(X.device.index)
    torch.cuda.synchronize()
    ctx.check(ctx.lib.lbk_context_trim(ctx.handle))
    assert ctx.pool_bytes() == 0
    ctx.use_torch_allocator(True)
    try:
        got = build_tree_arrays(X, g, h, **kw)
        torch.cuda.synchronize()
        assert ctx.pool_bytes() == 0
        assert len(ctx._held) == 0  # everything was given back
    finally:
        ctx.use_torch_allocator(False)
    for name in ("feature", "split_value", "gain", "leaf_value", "hessian", "leaf"):
        assert torch.equal(got[name], want[name]), name
    # the pool is in use again afterwards
    build_tree_arrays(X, g, h, **kw)
    assert ctx.pool_bytes() > 0


@pytest.mark.parametrize("N,F,K,D,S,dtype", [
    (20_000_003, 3, 1, 7, 256, np.float32),   # four bands, one-byte ids, a ragged last chunk
    (10_000_001, 4, 1, 6, 600, np.float64),   # two bands, two-byte ids
    (10_000_001, 5, 2, 5, 64, np.float32),    # two outputs: the pairs are read where they are written
])
def test_trees_of_levels_in_bands(lb, oracle, N, F, K, D, S, dtype):
    """Levels of large matrices are repartitioned in bands of rows, right children from their end: the tree, and with it the
    sums of every node below, are the oracle's bit for bit."""
    from legateboost_b200.tree import build_tree_arrays

    rs = np.random.default_rng(N)
    X = rs.random((N, F), dtype=np.float32).astype(dtype)
    X[:, 1] = np.round(X[:, 1] * 50)
    g, h = rs.random((N, K)) - 0.5 + 0.3 * np.sin(9 * X[:, :1]), rs.random((N, K)) + 0.1
    want = oracle.build_tree(X, g, h, max_depth=D, split_samples=S, seed=3, mode="Q")
    got = build_tree_arrays(dev(X), dev(g), dev(h), max_depth=D, split_samples=S, seed=3, row_offset=0, dataset_rows=N)
    assert (want.feature >= 0).sum() > 2 ** (D - 1)
    for name in ("feature", "split_value", "gain", "leaf_value", "hessian"):
        assert np.array_equal(got[name].cpu().numpy(), getattr(want, name)), name


@pytest.mark.parametrize("N,F,K,D,S,dtype", [
    (50001, 40, 1, 8, 256, np.float32),    # rows of 64 bytes, a last chunk of one row
    (20000, 7, 2, 5, 64, np.float64),      # one group
    (9000, 130, 1, 6, 256, np.float32),    # rows of 160 bytes
    (6000, 300, 1, 4, 128, np.float32),    # rows wider than the tiled form takes
    (7000, 20, 1, 6, 400, np.float32),     # two-byte bins
    (3000, 5, 1, 13, 256, np.float32),     # more nodes than the tiled form takes
])
def test_leaf_record_is_the_walk_of_predict(lb, N, F, K, D, S, dtype):
    """out_leaf (read off the binned matrix) names, for every row, the node whose value predict adds
    for that row when it walks X: leaf_value[out_leaf] == predict(X, tree), bit for bit."""
    from legateboost_b200.tree import build_tree_arrays, predict_arrays

    rs = np.random.RandomState(N % 97)
    X = dev(rs.normal(size=(N, F)).astype(dtype))
    g, h = dev(rs.normal(size=(N, K))), dev(rs.random((N, K)) + 0.05)
    t = build_tree_arrays(X, g, h, max_depth=D, split_samples=S, seed=4, row_offset=0, dataset_rows=N, want_leaf=True)
    # distinct values per node, so that equal predictions mean equal nodes
    M = t["feature"].shape[0]
    values = torch.arange(1, M * K + 1, dtype=torch.float64, device=X.device).reshape(M, K)
    pred = predict_arrays(X, [(values, t["feature"], t["split_value"])])
    leaf = t["leaf"].long()
    assert int(leaf.min()) >= 0 and int(leaf.max()) < M
    assert torch.equal(values[leaf], pred)


def test_peer_barrier_gives_up_and_reports(lb):
    """A peer that never reaches the barrier of the histogram exchange: the barrier kernel's wait is
    bounded (about a second), then it reports through the status word and returns, the call returns
    an error, and the context keeps working.  Emulated on one GPU with a flag that nothing sets."""
    import time
    from legateboost_b200.tree import build_tree_arrays

    ctx = lb.library.context(torch.cuda.current_device())
    stream = torch.cuda.current_stream().cuda_stream
    assert ctx.lib.lbk_selftest_peer_barrier(ctx.handle, 1, stream) == 0
    t0 = time.perf_counter()
    rc = ctx.lib.lbk_selftest_peer_barrier(ctx.handle, 0, stream)
    dt = time.perf_counter() - t0
    assert rc != 0 and b"fault code 41" in ctx.lib.lbk_last_error(ctx.handle)
    assert dt < 20.0
    # the status word was cleared and the device still answers: a present peer passes, a tree builds
    assert ctx.lib.lbk_selftest_peer_barrier(ctx.handle, 1, stream) == 0
    rs = np.random.RandomState(0)
    X, g, h = dev(rs.random((500, 4)).astype(np.float32)), dev(rs.normal(size=(500, 1))), dev(rs.random((500, 1)) + 0.1)
    t = build_tree_arrays(X, g, h, max_depth=2, split_samples=16, seed=1, row_offset=0, dataset_rows=500)
    assert int((t["feature"] >= 0).sum()) >= 1


def test_fixed_sketch_save_and_reuse(lb, oracle):
    """The optional sketch buffer: a saving call gives the oracle's tree, a reusing call with the same
    seed gives it again without reading X, a reusing call with another seed splits on the saved
    proposals only; a buffer without a sketch and a sketch of another shape are errors."""
    from legateboost_b200 import stages
    from legateboost_b200.tree import Sketch, build_tree_arrays

    N, F, K, D, S = 20000, 37, 2, 6, 64
    rs = np.random.RandomState(11)
    X = rs.normal(size=(N, F)).astype(np.float32)
    g = rs.normal(size=(N, K))
    h = rs.uniform(0.5, 2.0, size=(N, K))
    want = oracle.build_tree(X, g, h, max_depth=D, split_samples=S, seed=7, mode="Q")
    dX, dg, dh = dev(X), dev(g), dev(h)
    kw = dict(max_depth=D, split_samples=S, row_offset=0, dataset_rows=N, want_leaf=True)
    sk = Sketch()
    saved = build_tree_arrays(dX, dg, dh, seed=7, sketch=sk, **kw)
    assert sk.key is not None
    reused = build_tree_arrays(dX, dg, dh, seed=7, sketch=sk, **kw)
    for got in (saved, reused):
        for name in ("feature", "split_value", "gain", "leaf_value", "hessian"):
            assert np.array_equal(got[name].cpu().numpy(), getattr(want, name)), name
    assert torch.equal(saved["leaf"], reused["leaf"])
    # another seed on the saved sketch: other roundings, the proposals of seed 7
    other = build_tree_arrays(dX, dg, dh, seed=8, sketch=sk, **kw)
    props, row_ptr = stages.split_proposals(dX, S, 7)
    props, row_ptr = props.cpu().numpy().astype(np.float64), row_ptr.cpu().numpy()
    feat, split = other["feature"].cpu().numpy(), other["split_value"].cpu().numpy()
    assert (feat >= 0).sum() > 10
    for f, v in zip(feat, split):
        if f >= 0:
            assert v in props[row_ptr[f]:row_ptr[f + 1]]
    fresh = build_tree_arrays(dX, dg, dh, seed=8, **{**kw, "want_leaf": False})
    assert not np.array_equal(fresh["split_value"].cpu().numpy(), split)  # seed 8 has proposals of its own
    # errors
    from legateboost_b200 import library as L
    empty = Sketch()
    empty.mode_for(dX, S, L.context(0))
    empty.buffer.zero_()
    empty.key = sk.key  # pretend it was saved
    with pytest.raises(L.LbkError, match="no saved sketch"):
        build_tree_arrays(dX, dg, dh, seed=7, sketch=empty, **kw)
    X36 = dX[:, :36].contiguous()
    wrong = Sketch()
    wrong.buffer, wrong.key = sk.buffer, (lb.tree._tensor_key(X36), S)  # pretend it was saved for X36
    with pytest.raises(L.LbkError, match="another shape"):
        build_tree_arrays(X36, dg, dh, seed=7, sketch=wrong, **kw)


def test_tree_pickle_round_trip(lb):
    """A pickled tree predicts the same bits and leaves the per-fit scratch (leaf record, sketch) behind."""
    import pickle

    rs = np.random.RandomState(2)
    X = dev(rs.normal(size=(4000, 9)).astype(np.float32))
    g, h = dev(rs.normal(size=(4000, 1))), dev(np.ones((4000, 1)))
    t = lb.Tree(max_depth=4, split_samples=32).set_random_state(np.random.RandomState(1))
    t.sketch = lb.Sketch()
    t.fit(X, g, h)
    blob = pickle.dumps(t)
    assert len(blob) < 200_000  # neither the 4000-row leaf record nor the sketch buffer
    u = pickle.loads(blob)
    assert not hasattr(u, "sketch") and getattr(u, "_fit_rows", None) is None
    assert torch.equal(u.predict(X), t.predict(X))
    assert str(u) == str(t)


def test_estimator_fixed_sketch(lb):
    """fixed_sketch=True: the first tree is the one the default driver builds, later trees reuse its
    bins; the model still fits."""
    rs = np.random.RandomState(4)
    X = dev(rs.normal(size=(30000, 20)).astype(np.float32))
    y = X[:, 0] * 2.0 - X[:, 3] + 0.1 * dev(rs.normal(size=30000)).to(torch.float32)
    base = (lb.Tree(max_depth=5, split_samples=64),)
    a = lb.LBRegressor(n_estimators=8, base_models=base, random_state=3).fit(X, y)
    b = lb.LBRegressor(n_estimators=8, base_models=base, random_state=3, fixed_sketch=True).fit(X, y)
    assert torch.equal(a.models_[0].feature, b.models_[0].feature)
    assert torch.equal(a.models_[0].leaf_value, b.models_[0].leaf_value)
    assert all(getattr(t, "sketch", None) is None for t in b.models_)
    err = lambda m: float(((m.predict(X).view(-1) - y.double()) ** 2).mean())
    assert err(b) < 0.5 * float(y.double().var()) and abs(err(b) - err(a)) < 0.2 * err(a) + 1e-3


def test_build_tree_level_batching(lb, oracle):
    """More bins than the 1 GB histogram rule holds on the deepest levels: levels are cut into
    batches and built without parents (reference: test_wide_deep, test_tree.py:218-227)."""
    case = (3000, 500, 1, 10, 256, np.float32, {})
    X, want, got = _run_tree_case(lb, oracle, case, seed=3)
    assert np.array_equal(got["feature"].cpu().numpy(), want.feature)
    assert np.array_equal(got["node_sums"].cpu().numpy(), want.node_sums)
    assert np.array_equal(got["leaf_value"].cpu().numpy(), want.leaf_value)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("S", [3, 100, 256, 300, 512, 700, 2048])
def test_zeros_of_either_sign_among_the_samples(lb, dt, S):
    """-0 and +0 are one candidate, which is +0 whatever comes first; a NaN among the samples counts as +inf."""
    from legateboost_b200 import stages
    from legateboost_b200.tree import build_tree_arrays

    rs = np.random.RandomState(S)
    X = (np.round(rs.normal(size=(3000, 5)) * 5) / 5).astype(dt)
    X[:, 1] = np.where(rs.random(3000) < 0.5, -0.0, X[:, 1])
    X[:, 2] = np.where(X[:, 2] == 0, -0.0, X[:, 2])
    X[:, 3] = -0.0
    X[rs.random(3000) < 0.3, 4] = np.nan
    want, want_ptr = stages.split_proposals(dev(np.where(np.isnan(X), np.inf, X + 0.0).astype(dt)), S, 7)
    p, ptr = stages.split_proposals(dev(X), S, 7)
    words = torch.int32 if dt == np.float32 else torch.int64
    assert torch.equal(ptr, want_ptr) and torch.equal(p.view(words), want.view(words))
    X[:, 4] = rs.random(3000)
    g, h = np.where(X[:, 1:2] > 0, 1.0, -1.0), np.ones((3000, 1))  # (the best split is at zero)
    for N in (3000, 70_000):  # (the one-launch form and the general one)
        big = [dev(np.tile(a, (N // 1000, 1))[:N]) for a in (X, g, h)]
        tree = build_tree_arrays(*big, max_depth=4, split_samples=S, seed=7, row_offset=0, dataset_rows=N)
        v = tree["split_value"].cpu().numpy()
        assert not np.signbit(v[v == 0]).any()
        assert S < 100 or (v[0] == 0 and tree["feature"][0] == 1)


def _random_trees(rs, T, D, features, odd=False):
    """Trees of depth <= D on the given features, splits around U(0, 1); with `odd` infinite and NaN ones too."""
    trees = []
    for _ in range(T):
        M = 2 ** (D + 1) - 1
        f = np.full(M, -1, np.int32)
        f[: M // 2] = rs.choice(features, size=M // 2)
        f[1: M // 2][rs.random(M // 2 - 1) < 0.1] = -1
        for i in range(1, M // 2):
            if f[(i - 1) // 2] < 0:
                f[i] = -1
        v = rs.random(M)
        if odd:
            at = rs.random(M)
            v[at < 0.02], v[(at > 0.02) & (at < 0.03)], v[(at > 0.03) & (at < 0.04)] = np.inf, -np.inf, np.nan
            v[at > 0.9] = np.round(v[at > 0.9] * 4) / 4
        trees.append((dev(rs.normal(size=(M, 1))), dev(f), dev(v)))
    return trees


def _predict_plan(lb, table, X, K, transform):
    """How a prediction is made (lbk_selftest_predict_plan)."""
    import ctypes
    from legateboost_b200 import library as L

    ctx, out = L.context(X.device.index), (ctypes.c_int64 * 8)()
    ctx.check(ctx.lib.lbk_selftest_predict_plan(ctx.handle, X.shape[0], X.shape[1], K, table.n_trees, table.max_nodes, table.total_nodes,
                                                L.LBK_F32 if X.dtype == torch.float32 else L.LBK_F64, transform, out))
    return dict(zip(("threads", "group", "piece", "bytes", "word", "tile_rows", "tile_group", "leaves_with_trees"), out))


def _predict_and_word(lb, table, X, plan, **kw):
    """A prediction whose scratch stays here, and the word in it that says whether the device declined the ranks."""
    ctx, held = lb.library.context(X.device.index), []

    def alloc(user, nbytes, stream):
        held.append(torch.empty(int(nbytes), dtype=torch.uint8, device="cuda"))
        return held[-1].data_ptr()

    cbs = lb.library.ALLOC_FN(alloc), lb.library.RELEASE_FN(lambda user, ptr, stream: None)
    ctx.check(ctx.lib.lbk_context_set_allocator(ctx.handle, cbs[0], cbs[1], None))
    try:
        got = table.predict(X, 1, wait=True, **kw)
        torch.cuda.synchronize()
    finally:
        ctx.use_torch_allocator(False)
    room, = [t for t in held if t.numel() == plan["bytes"]]
    return got, int(room[plan["word"]: plan["word"] + 4].view(torch.int32))


@pytest.mark.parametrize("N,F,T,D,dt,used,what,group,pieces,declined", [
    (1_000_001, 100, 500, 8, np.float32, None, "odd", 4, 1, False),     # a last group of four features, a ragged last tile
    (1_600_003, 100, 500, 8, np.float32, None, "odd", 4, 2, False),     # rows in two pieces
    (1_300_003, 33, 200, 5, np.float64, None, "odd", 4, 1, False),      # a last group of one feature
    (1_200_001, 9, 100, 10, np.float64, None, "odd", 4, 1, False),       # tables of a group in several turns
    (4_000_000, 1, 60, 4, np.float64, None, "", 4, 1, False),           # one feature
    (600_000, 150, 60, 11, np.float64, None, "", 2, 1, False),          # two trees per group
    (600_000, 150, 60, 12, np.float64, None, "", 1, 1, False),          # one
    (800_000, 20, 100, 8, np.float64, [3], "", 4, 1, False),            # all splits on one feature, in chunks; no room for the table
    (400_000, 20, 300, 8, np.float64, [3], "few", 4, 1, False),         # more than there are ranks, of which many are equal
    (300_000, 20, 300, 8, np.float64, [3], "logistic", 4, 1, True),     # more of them than there are ranks
    (1_000_001, 100, 500, 8, np.float32, "3", "odd", 4, 1, True),       # one large table: the ranks would cost more than they give
    (200_000, 330, 300, 8, np.float64, None, "logistic", 4, 1, False),  # rows too wide for the tiled walk
    (200_000, 330, 300, 8, np.float64, [3], "logistic", 4, 1, True),    # ... which are then read through the caches
])
def test_predict_by_ranks(lb, oracle, N, F, T, D, dt, used, what, group, pieces, declined):
    """Large ensembles of one output are walked on ranks, if the device does not find their tables too dear; a few rows at a
    time, where the trees are walked where they lie, give the same bits."""
    from legateboost_b200 import library as L
    from legateboost_b200.tree import TreeTable

    rs = np.random.RandomState(N % 1000 + F)
    X = rs.random((N, F)).astype(dt)
    X[:, 0] = np.round(X[:, 0] * 4) / 4
    if what == "odd":
        for value in (np.nan, np.inf, -np.inf):
            X[rs.randint(N, size=3000), rs.randint(F, size=3000)] = value
        X[-40:] = np.nan
    if used == "3":  # of a hundred splits 41
        used = np.concatenate([np.arange(F), np.full(69, 3)])
    trees = _random_trees(rs, T, D, np.arange(F) if used is None else used, what == "odd")
    if what == "few":
        pool = dev(rs.random(20_000))
        trees = [(v, f, pool[(s * 20_000).long().clamp(0, 19_999)]) for v, f, s in trees]
    table, transform = TreeTable(trees), L.LOGISTIC if what == "logistic" else L.RAW
    init = dev(np.array([0.25])) if what else None
    dX = dev(X)
    plan = _predict_plan(lb, table, dX, 1, transform)
    assert plan["threads"] > 0 and plan["group"] == group and -(-N // plan["piece"]) == pieces
    assert (plan["tile_rows"] == 0) == (F > 320)
    got, word = _predict_and_word(lb, table, dX, plan, init=init, transform=transform)
    assert (word != 0) == declined
    assert torch.equal(table.predict(dX, 1, init=init, transform=transform, wait=True), got)
    edge = min(plan["piece"], N)
    picks = [np.arange(5000), np.arange(N - 5000, N), np.sort(rs.choice(N, 8000, replace=False)), np.arange(edge - 4000, min(edge + 4000, N))]
    for rows in picks:
        rows = dev(rows)
        few = table.predict(dX[rows].contiguous(), 1, init=init, transform=transform, wait=True)
        assert torch.equal(got[rows], few)
    if what == "":
        few = picks[0][:500]
        want = oracle.predict(X[few], [tuple(a.cpu().numpy() for a in t) for t in trees])
        assert np.array_equal(got[few].cpu().numpy(), want)
    # rows that lie apart in memory
    wide = torch.zeros((N, F + 3), dtype=dX.dtype, device="cuda")
    wide[:, 1: F + 1] = dX
    assert torch.equal(table.predict(wide[:, 1: F + 1], 1, init=init, transform=transform, wait=True), got)


def _rank_searches(trees, F, dt):
    """How k_rank_rows finds the ranks of the turns over an ensemble's features: in 3 or 4 steps, by as many as its fullest bucket
    wants ("counted"), or in a table that has no room in shared memory ("where it lies").  Restated from its tables and turns."""
    room = torch.cuda.get_device_properties(0).shared_memory_per_block_optin - 1024 - 16 * 32 * 33 * 4
    f = np.concatenate([t[1].cpu().numpy()[: len(t[1]) // 2] for t in trees])
    s = np.concatenate([t[2].cpu().numpy()[: len(t[2]) // 2] for t in trees])
    fullest, entries = [], []
    for i in range(F):
        v = np.unique(s[f == i]).astype(np.float32 if dt is np.float32 else np.float64)
        entries.append(max(len(v), 1))
        fullest.append(0)
        if len(v):
            lo, hi = np.float32(v[0]), np.float32(v[-1])
            scale = np.float32(len(v)) / (hi - lo) if hi > lo else np.float32(0)
            fullest[-1] = np.bincount(np.minimum(((v.astype(np.float32) - lo) * scale).astype(np.int64), len(v) - 1)).max()

    def table(a, b, pad=0):
        n = sum(entries[a:b])
        return (n + 1) // 2 * 8 + (n + pad * (b - a)) * np.dtype(dt).itemsize

    found = set()
    for g in range(0, F, 32):
        a, end = g, min(g + 32, F)
        while a < end:
            b = a + 1
            while b < end and table(a, b + 1) <= room:
                b += 1
            if b < end:
                b = a + 2 ** int(np.log2(b - a))
            most = max(fullest[a:b])
            if most > 0:
                found.add("where it lies" if table(a, b) > room else "counted" if most >= 16 or table(a, b, 4) > room else 4 if most >= 8 else 3)
            a = b
    return found


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("what,used,searches", [
    ("even", None, (3, 3)), ("any", None, (3, 3)), ("seven", None, (3, 3)), ("fifteen", None, (4, 4)), ("sixteen", None, ("counted", 4)),
    ("sixty", None, ("counted", "counted")), ("skewed", None, ("counted", "counted")), ("one", [3], ("where it lies", "counted"))])
def test_ranks_from_buckets_of_any_size(lb, what, used, searches, dt):
    """Splits evenly apart, by chance, and crowded in buckets of up to so many (one: nearly all of a feature's): the steps of the
    search are another number each time (float32, float64).  A few rows at a time, where trees are walked where they lie, give the same bits."""
    from legateboost_b200 import library as L
    from legateboost_b200.tree import TreeTable

    N, F, T, D = (1_000_003, 60, 300, 8) if dt is np.float32 else (800_011, 20, 70, 8)
    if used is not None and dt is np.float32:  # (of two groups of features the ranks are found too dear)
        F, T = 20, 200
    rs = np.random.RandomState(len(what))
    trees, crowd = [], dict(seven=7, fifteen=15, sixteen=17, sixty=60).get(what)
    for v, f, s in _random_trees(rs, T, D, np.arange(F) if used is None else used):
        s = s.cpu().numpy()
        if what == "even":
            s = np.round(s * 700) / 700
        elif crowd is not None:  # clusters a good deal further apart than a bucket is wide, in a small part of one each
            s = np.floor(s * 40) / 40 + np.floor(rs.random(s.shape) * crowd) * 2e-6
        elif what == "skewed":  # many buckets side by side that are nearly too full to be put in order one by one
            s = np.exp(4 * s)
        elif what == "one":
            s = np.where(rs.random(s.shape) < 0.002, np.sign(s - 0.5) * 1e4, 0.5 + s * 0.02)
        trees.append((v, f, dev(s.astype(dt).astype(np.float64))))
    assert _rank_searches(trees, F, dt) == {searches[0 if dt is np.float32 else 1]}
    table = TreeTable(trees)
    X = np.random.default_rng(len(what)).random((N, F), dtype=dt)
    splits = np.concatenate([t[2].cpu().numpy() for t in trees]).astype(dt)
    X[::2] = splits[rs.randint(len(splits), size=X[::2].shape)]  # ties
    X[rs.randint(N, size=500), rs.randint(F, size=500)] = np.nan
    X[rs.randint(N, size=500), rs.randint(F, size=500)] = np.inf
    dX = dev(X)
    plan = _predict_plan(lb, table, dX, 1, L.RAW)
    assert plan["threads"] > 0
    got, word = _predict_and_word(lb, table, dX, plan)
    assert word == 0  # (the ranks were found and walked on: not declined)
    for rows in (np.arange(8000), np.arange(N - 8000, N), np.sort(rs.choice(N, 8000, replace=False))):
        rows = dev(rows)
        assert torch.equal(got[rows], table.predict(dX[rows].contiguous(), 1, wait=True))


@pytest.mark.parametrize("N,F,K,T,D,dt,with_trees", [
    (20_001, 10, 6, 16, 5, np.float32, True), (100_003, 100, 10, 50, 8, np.float32, True), (9_000, 65, 16, 17, 6, np.float64, True),
    (12_345, 300, 10, 23, 6, np.float32, True), (20_000, 7, 12, 40, 3, np.float64, True),
    (30_000, 33, 10, 50, 8, np.float32, False), (9_999, 20, 10, 20, 9, np.float32, False),  # fewer rows in a block than a tree has leaves
    (20_000, 10, 10, 15, 6, np.float32, False),  # too few trees
])
def test_predict_of_several_outputs_by_tables(lb, oracle, N, F, K, T, D, dt, with_trees):
    """Leaf values that come with the trees (and shapes around them): the bits of the walk in place, a few rows at a time."""
    from legateboost_b200 import library as L
    from legateboost_b200.tree import TreeTable

    rs = np.random.RandomState(N + K)
    X = dev(rs.random((N, F)).astype(dt))
    trees = [(dev(rs.normal(size=(t[1].shape[0], K))),) + t[1:] for t in _random_trees(rs, T, D, np.arange(F))]
    table, init = TreeTable(trees), dev(rs.normal(size=K))
    for transform in (L.RAW, L.SOFTMAX):
        assert _predict_plan(lb, table, X, K, transform)["leaves_with_trees"] == with_trees
        got = table.predict(X, K, init=init, transform=transform, wait=True)
        for rows in (slice(0, 4000), slice(N - 4000, N)):
            assert torch.equal(got[rows], table.predict(X[rows], K, init=init, transform=transform, wait=True))
    want = oracle.predict(X[:300].cpu().numpy(), [tuple(a.cpu().numpy() for a in t) for t in trees])
    assert np.array_equal(table.predict(X, K, wait=True)[:300].cpu().numpy(), want)


@pytest.mark.parametrize("K", [6, 7, 8, 9, 10, 11, 12, 14, 15, 16])
@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_predict_of_even_and_odd_outputs(lb, oracle, K, dt):
    """Leaf values that come with the trees, of an even number of outputs two at a time: the bits of the oracle's sums."""
    from legateboost_b200 import library as L
    from legateboost_b200.tree import TreeTable

    N, F, T, D = 9_003, 11, 17, 5
    rs = np.random.RandomState(K)
    X = rs.random((N, F)).astype(dt)
    trees = [(dev(rs.normal(size=(t[1].shape[0], K))),) + t[1:] for t in _random_trees(rs, T, D, np.arange(F))]
    table, init = TreeTable(trees), dev(rs.normal(size=K))
    assert _predict_plan(lb, table, dev(X), K, L.RAW)["leaves_with_trees"]
    want = oracle.predict(X, [tuple(a.cpu().numpy() for a in t) for t in trees])
    assert np.array_equal(table.predict(dev(X), K, wait=True).cpu().numpy(), want)
    softmax = table.predict(dev(X), K, init=init, transform=L.SOFTMAX, wait=True).cpu().numpy()
    raw = want + init.cpu().numpy()
    e = np.exp(raw - raw.max(axis=1, keepdims=True))
    assert np.allclose(softmax, e / e.sum(axis=1, keepdims=True), rtol=1e-13, atol=0)  # (a few roundings of exp and a sum)


@pytest.mark.parametrize("K", [2, 3, 4, 5, 6, 7, 8, 9, 11, 12, 13, 14, 15, 16, 17])
@pytest.mark.parametrize("T", [5, 16])
def test_predict_of_any_number_of_outputs(lb, oracle, K, T):
    """As many sums as outputs, or one more, with the leaf values apart (few trees, few outputs) or with the trees: the oracle's bits."""
    from legateboost_b200 import library as L
    from legateboost_b200.tree import TreeTable

    N, F, D = 9_001, 12, 6
    rs = np.random.RandomState(100 * T + K)
    X = rs.random((N, F)).astype(np.float32)
    trees = [(dev(rs.normal(size=(t[1].shape[0], K))),) + t[1:] for t in _random_trees(rs, T, D, np.arange(F))]
    table = TreeTable(trees)
    plan = _predict_plan(lb, table, dev(X), K, L.RAW)
    assert plan["tile_rows"] > 0 and plan["leaves_with_trees"] == (T >= 16 and 6 <= K <= 16)
    want = oracle.predict(X, [tuple(a.cpu().numpy() for a in t) for t in trees])
    assert np.array_equal(table.predict(dev(X), K, wait=True).cpu().numpy(), want)


@pytest.mark.parametrize("N,F,K,T,D,dt", [(16, 30, 1, 100, 6, np.float32), (20_001, 40, 10, 20, 6, np.float32), (900_001, 30, 1, 100, 8, np.float64)])
def test_chained_launches_under_capture_and_on_two_streams(lb, N, F, K, T, D, dt):
    """Kernels that may begin as the one before them ends see all that it wrote: in a captured graph, replayed on changing inputs,
    and in calls on two streams at a time."""
    from legateboost_b200.tree import TreeTable

    rs = np.random.RandomState(N % 89)
    trees = [(dev(rs.normal(size=(t[1].shape[0], K))),) + t[1:] for t in _random_trees(rs, T, D, np.arange(F))]
    table = TreeTable(trees)
    inputs = [dev(rs.random((N, F)).astype(dt)) for _ in range(3)]
    want = [table.predict(X, K, wait=True) for X in inputs]
    X, streams = inputs[0].clone(), [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=streams[0]):
        got = table.predict(X * 1, K)
    for given, expected in zip(inputs[::-1], want[::-1]):
        X.copy_(given)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, expected)
    out = []
    for turn in range(6):
        with torch.cuda.stream(streams[turn % 2]):
            out.append(table.predict(inputs[turn % 3] * 1, K))
    torch.cuda.synchronize()
    for turn in range(6):
        assert torch.equal(out[turn], want[turn % 3])


def test_predict_without_room_for_ranks(lb):
    """A caller's allocator that has no 20 MB gets the predictions by the path that needs less."""
    from legateboost_b200.tree import TreeTable

    rs = np.random.RandomState(1)
    X, table = dev(rs.random((500_000, 64))), TreeTable(_random_trees(rs, 64, 8, np.arange(64)))
    want = table.predict(X, 1, wait=True)
    ctx = lb.library.context(X.device.index)
    held, refused = {}, []

    def alloc(user, nbytes, stream):
        if nbytes > 20_000_000:
            refused.append(nbytes)
            return None
        t = torch.empty(int(nbytes), dtype=torch.uint8, device="cuda")
        held[t.data_ptr()] = t
        return t.data_ptr()

    def release(user, ptr, stream):
        held.pop(ptr, None)

    cbs = lb.library.ALLOC_FN(alloc), lb.library.RELEASE_FN(release)
    ctx.check(ctx.lib.lbk_context_set_allocator(ctx.handle, cbs[0], cbs[1], None))
    try:
        got = table.predict(X, 1, wait=True)
        torch.cuda.synchronize()
    finally:
        ctx.use_torch_allocator(False)
    assert len(refused) == 1 and torch.equal(got, want)


@pytest.mark.parametrize("zeros", [False, True])
@pytest.mark.parametrize("N,F,K,D", [(2500, 600, 2, 8), (2500, 600, 2, 10), (700, 1000, 1, 9)])
def test_levels_outside_the_cache(lb, oracle, N, F, K, D, zeros):
    """Levels that the reference builds node by node: derived where every quantised hessian is at least one (in one batch,
    in two, and below a level that was not kept), built where some are 0, which a derived node would show."""
    from legateboost_b200.tree import build_tree_arrays

    rs = np.random.RandomState(N + F + D)
    X = rs.random((N, F)).astype(np.float32)
    X[:, 0] = np.round(X[:, 0] * 5) / 5
    g = rs.normal(size=(N, K))
    h = rs.random((N, K)) + 0.1
    if zeros:
        h[rs.random(N) < 0.3] = 0.0
    want = oracle.build_tree(X, g, h, max_depth=D, split_samples=256, seed=5, mode="Q")
    # (in scratch that holds something: what has to be clear has been cleared)
    dX, dg, dh = dev(X), dev(g), dev(h)
    ctx, held = lb.library.context(dX.device.index), {}

    def alloc(user, nbytes, stream):
        t = torch.full((int(nbytes),), 0x5a, dtype=torch.uint8, device="cuda")
        held[t.data_ptr()] = t
        return t.data_ptr()

    def release(user, ptr, stream):
        held.pop(ptr)

    cbs = lb.library.ALLOC_FN(alloc), lb.library.RELEASE_FN(release)
    ctx.check(ctx.lib.lbk_context_set_allocator(ctx.handle, cbs[0], cbs[1], None))
    try:
        got = build_tree_arrays(dX, dg, dh, max_depth=D, split_samples=256, seed=5, row_offset=0, dataset_rows=N)
        torch.cuda.synchronize()
    finally:
        ctx.use_torch_allocator(False)
    for name in ("feature", "split_value", "node_sums", "gain", "hessian", "leaf_value"):
        assert np.array_equal(got[name].cpu().numpy(), getattr(want, name)), name


def test_levels_outside_the_cache_without_room_for_more(lb):
    """A caller's allocator that has no room for more than the reference's cache, in one piece or in all, gets the tree that
    is built node by node on the levels outside it."""
    from legateboost_b200.tree import build_tree_arrays

    rs = np.random.RandomState(4)
    X, g, h = dev(rs.random((700, 1000)).astype(np.float32)), dev(rs.normal(size=(700, 1))), dev(rs.random((700, 1)) + 0.1)
    build = lambda: build_tree_arrays(X, g, h, max_depth=10, split_samples=256, seed=5, row_offset=0, dataset_rows=700)
    want = build()
    ctx = lb.library.context(X.device.index)

    def build_within(piece, total, but=-1):
        """The most that was lent at a time, how often nothing was, and what was asked for; request `but` is refused anyhow."""
        held, lent, most, refused, asked = {}, [0], [0], [], []

        def alloc(user, nbytes, stream):
            asked.append(nbytes)
            if nbytes > piece or lent[0] + nbytes > total or len(asked) - 1 == but:
                refused.append(nbytes)
                return None
            t = torch.empty(int(nbytes), dtype=torch.uint8, device="cuda")
            held[t.data_ptr()] = t
            lent[0] += nbytes
            most[0] = max(most[0], lent[0])
            return t.data_ptr()

        def release(user, ptr, stream):
            lent[0] -= held.pop(ptr).numel()

        cbs = lb.library.ALLOC_FN(alloc), lb.library.RELEASE_FN(release)
        ctx.check(ctx.lib.lbk_context_set_allocator(ctx.handle, cbs[0], cbs[1], None))
        try:
            got = build()
            torch.cuda.synchronize()
        finally:
            ctx.use_torch_allocator(False)
        assert lent[0] == 0
        for name in ("feature", "split_value", "gain", "hessian", "leaf_value"):
            assert torch.equal(got[name], want[name]), name
        return most[0], len(refused), asked

    everything, refusals, asked = build_within(1 << 62, 1 << 62)
    assert refusals == 0
    least, refusals, _ = build_within(1_000_000_000, 1 << 62)
    assert refusals == 1 and least < everything - 1_000_000_000
    for total in np.linspace(least, everything, 9).astype(np.int64):
        most, refusals, _ = build_within(1 << 62, int(total))
        assert (refusals == 0) == (total == everything) and most <= total
    # every request from the held levels on may be the one that is refused
    first = next(i for i, n in enumerate(asked) if n > 1_000_000_000)
    for but in range(first, len(asked)):
        assert build_within(1 << 62, 1 << 62, but)[1] == 1
    assert len(asked) - first > 3


def test_golden_trees_on_gpu(lb, oracle):
    """The committed golden inputs: the GPU (quantised) tree must predict within 1e-4 of... itself
    via the oracle's Mode Q, and stay close to the reference CPU tree's training loss."""
    from legateboost_b200.tree import build_tree_arrays, predict_arrays

    for path in sorted(glob.glob(os.path.join(HERE, "golden", "tree_*.npz"))):
        z = np.load(path)
        kw = dict(max_depth=int(z["max_depth"]), split_samples=int(z["split_samples"]), seed=int(z["seed"]),
                  l1=float(z["l1"]), l2=float(z["l2"]), min_split_gain=float(z["min_split_gain"]))
        want = oracle.build_tree(z["X"], z["g"], z["h"], mode="Q", **kw)
        got = build_tree_arrays(dev(z["X"]), dev(z["g"]), dev(z["h"]), row_offset=0, dataset_rows=z["X"].shape[0], **kw)
        assert np.array_equal(got["feature"].cpu().numpy(), want.feature)
        assert np.array_equal(got["leaf_value"].cpu().numpy(), want.leaf_value)
        # predict of the reference CPU tree stored in the fixture, evaluated by the GPU kernel
        p = predict_arrays(dev(z["X"]), [(dev(z["leaf_value"]), dev(z["feature"]), dev(z["split_value"]))])
        assert np.array_equal(p.cpu().numpy(), z["pred"])


GOLDEN_Q = sorted(glob.glob(os.path.join(HERE, "golden", "treeq_*.npz")))
SAME_SCALE = {"batching", "deep", "mask", "reg", "rows20k", "softmax10"}


@pytest.mark.parametrize("path", GOLDEN_Q, ids=[os.path.basename(p)[6:-4] for p in GOLDEN_Q])
def test_reference_gpu_vectors_on_gpu(lb, path):
    """liblbk.so against what the reference's own GPU code produced for the same inputs
    (tests/golden/make_golden_q.py).  Bit for bit: bins, feature, split_value, quantised node sums,
    traced histograms, predictions.  The float outputs that pass through the quantiser's scale
    (a float sum whose order the reference leaves to thrust::reduce) or a contracted multiply-add:
    bit for bit equal to the reference built without contraction where the scale is the same
    float (SAME_SCALE), within 1e-12 relative everywhere."""
    import sys

    from legateboost_b200.tree import build_tree_arrays, predict_arrays

    sys.path.insert(0, os.path.join(HERE, "golden"))
    import make_golden_q as G

    z, c = G.load_case(path)
    name = os.path.basename(path)[6:-4]
    tn = int(z["trace_nodes"])
    fs = None if c["feature_set"] is None else torch.from_numpy(np.asarray(c["feature_set"]))
    got = build_tree_arrays(dev(c["X"]), dev(np.asarray(c["g"], dtype=np.float64)), dev(np.asarray(c["h"], dtype=np.float64)),
                            max_depth=c["max_depth"], split_samples=c["split_samples"], seed=c["seed"], l1=c["l1"],
                            l2=c["l2"], min_split_gain=c["min_split_gain"], feature_set=fs, row_offset=0,
                            dataset_rows=c["X"].shape[0], trace_nodes=tn)
    assert got["B"] == int(z["total_bins"])
    assert np.array_equal(got["feature"].cpu().numpy(), z["feature"])
    assert np.array_equal(got["split_value"].cpu().numpy().view(np.int64), z["split_value"].view(np.int64))
    assert np.array_equal(got["node_sums"].cpu().numpy(), z["node_sums"])
    trace = got["trace_hist"].cpu().numpy()
    assert np.array_equal(G.digest(trace), z["trace_digest"])
    assert np.array_equal(trace[:z["trace_hist"].shape[0]], z["trace_hist"])
    for k in ("hessian", "leaf_value", "gain"):
        a = got[k].cpu().numpy()
        assert np.all(np.abs(a - z[k]) <= 1e-12 * np.maximum(np.abs(a), np.abs(z[k]))), k
        if name in SAME_SCALE:
            assert np.array_equal(a.view(np.int64), z[k + "_nofma"].view(np.int64)), k
    pred = predict_arrays(dev(c["X"]), [(dev(z["leaf_value"]), dev(z["feature"]), dev(z["split_value"]))])
    assert np.array_equal(pred.cpu().numpy().view(np.int64), z["pred"].view(np.int64))


# ---------------------------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("N,F,K,T,D", [(1000, 10, 1, 5, 4), (5000, 100, 1, 40, 8), (777, 33, 5, 7, 6), (129, 3, 2, 1, 0)])
def test_predict_bit_exact(lb, oracle, dtype, N, F, K, T, D):
    from legateboost_b200.tree import predict_arrays

    rs = np.random.RandomState(T)
    X = rs.random((N, F)).astype(dtype)
    M = 2 ** (D + 1) - 1
    trees = []
    for _ in range(T):
        feat = rs.randint(0, F, size=M).astype(np.int32)
        feat[2 ** D - 1:] = -1                      # last level are leaves
        feat[rs.random(M) < 0.15] = -1              # some early leaves
        split = rs.random(M)
        leaf = rs.normal(size=(M, K))
        trees.append((leaf, feat, split))
    want = oracle.predict(X, trees)
    got = predict_arrays(dev(X), [(dev(a), dev(b), dev(c)) for a, b, c in trees])
    assert np.array_equal(got.cpu().numpy(), want)


def test_predict_empty_and_batch_sum(lb, oracle):
    from legateboost_b200.tree import predict_arrays

    rs = np.random.RandomState(0)
    X = rs.random((500, 6)).astype(np.float32)
    mk = lambda: (dev(rs.normal(size=(3, 1))), dev(np.array([2, -1, -1], dtype=np.int32)), dev(rs.random(3)))
    a, b = mk(), mk()
    pa, pb = predict_arrays(dev(X), [a]), predict_arrays(dev(X), [b])
    assert torch.equal(predict_arrays(dev(X), [a, b]), pa + pb)
    assert predict_arrays(dev(X[:0]), [a]).shape == (0, 1)


# ---------------------------------------------------------------------------------------------
def test_tree_class_known_answers(lb):
    # reference: test_tree.py:11-21, 64-78, 160-184
    X = dev(np.array([[0.0], [1.0]]))
    g = dev(np.array([[0.0], [-1.0]]))
    h = dev(np.array([[1.0], [1.0]]))
    m = lb.Tree(max_depth=1, l2_regularization=0.0).set_random_state(np.random.RandomState(2)).fit(X, g, h)
    assert np.allclose(m.predict(X).cpu().numpy(), np.array([[0.0], [1.0]]))
    X0 = dev(np.array([[0.0], [0.0]]))
    y = np.array([500.0, 500.0])
    m = lb.Tree(max_depth=0, l2_regularization=10.0).set_random_state(np.random.RandomState(0))
    m.fit(X0, dev(-y[:, None]), dev(np.ones((2, 1))))
    assert np.isclose(m.predict(X0)[0, 0].item(), y.sum() / (y.size + 10.0))
    m = lb.Tree(max_depth=0, l2_regularization=0.0, l1_regularization=1.5).set_random_state(np.random.RandomState(0))
    m.fit(X0, dev(-y[:, None]), dev(np.ones((2, 1))))
    assert np.isclose(m.predict(X0)[0, 0].item(), (y.sum() - 1.5) / y.size)
    assert "leaf=" in str(m) and m == m and (m * 2.0).leaf_value[0, 0].item() == 2 * m.leaf_value[0, 0].item()


def test_tree_class_depth_and_invariants(lb):
    # reference: test_tree.py:24-45 and legateboost/testing/utils.py:22-50
    rs = np.random.RandomState(0)
    X = rs.random((10000, 100))
    for K in (1, 5):
        g = rs.normal(size=(X.shape[0], K))
        h = rs.random(g.shape) + 0.1
        y = -g / h
        metrics = []
        for depth in range(0, 10):
            m = lb.Tree(max_depth=depth).set_random_state(np.random.RandomState(2)).fit(dev(X), dev(g), dev(h))
            p = m.predict(dev(X)).cpu().numpy()
            metrics.append((((p - y) ** 2 * h).sum(axis=0) / h.sum(axis=0)).mean())
            feat, hess, gain = m.feature.cpu().numpy(), m.hessian.cpu().numpy(), m.gain.cpu().numpy()
            split = feat != -1
            assert np.all(hess[split] > 0.0) and np.all(gain[split] > 0.0)
            leaves = (feat == -1) & (hess[:, 0] > 0.0)
            assert np.isclose(hess[leaves].sum(axis=0), hess[0]).all()
        assert all(a - b > -1e-3 for a, b in zip(metrics, metrics[1:])) and metrics[-1] < metrics[0]


def test_max_depth_20_two_rows(lb):
    # reference: test_tree.py:48-61
    X = dev(np.random.RandomState(0).random((2, 1)))
    m = lb.LBRegressor(init=None, base_models=(lb.Tree(max_depth=20),), learning_rate=1.0, n_estimators=1,
                       random_state=0)
    m.fit(X, dev(np.array([500.0, 500.0])))
    assert m[0].feature.shape[0] == 2 ** 21 - 1


def test_estimators_config1_reduced(lb, oracle):
    """Configuration 1 at reduced size: squared error, depth 6, lr 0.1; loss falls every round and
    every tree equals the oracle's tree for the same gradients and seed."""
    rng = np.random.default_rng(0)
    X = rng.random((20000, 50), dtype=np.float32)
    y = (np.sin(6 * X[:, :5]).sum(axis=1) + rng.normal(0, 0.1, size=20000)).astype(np.float32)
    m = lb.LBRegressor(n_estimators=5, learning_rate=0.1, base_models=(lb.Tree(max_depth=6, split_samples=256),),
                       random_state=0, verbose=1)
    m.fit(dev(X), dev(y))
    assert all(a > b for a, b in zip(m.train_metric_, m.train_metric_[1:]))
    # replay round 0 with the oracle
    rs = np.random.RandomState(0)
    seed = rs.randint(0, 2 ** 31)
    y64 = y.astype(np.float64)[:, None]
    g = (np.full_like(y64, y64.mean()) - y64) * 0.1
    want = oracle.build_tree(X, g, np.ones_like(g), max_depth=6, split_samples=256, seed=seed, mode="Q")
    assert np.array_equal(m[0].feature.cpu().numpy(), want.feature)
    assert np.allclose(m[0].leaf_value.cpu().numpy(), want.leaf_value, rtol=1e-9, atol=1e-12)


def test_classifier_multiclass(lb):
    rng = np.random.default_rng(2)
    X = rng.normal(size=(5000, 20)).astype(np.float32)
    W = rng.normal(size=(10, 4))
    y = np.argmax(X[:, :10] @ W + rng.normal(0, 0.5, size=(5000, 4)), axis=1)
    m = lb.LBClassifier(n_estimators=5, base_models=(lb.Tree(max_depth=4),), random_state=1, verbose=1)
    m.fit(dev(X), dev(y))
    assert all(a > b for a, b in zip(m.train_metric_, m.train_metric_[1:]))
    proba = m.predict_proba(dev(X))
    assert torch.allclose(proba.sum(dim=1), torch.ones(5000, dtype=torch.float64, device="cuda"))
    assert (m.predict(dev(X)).cpu().numpy() == y).mean() > 0.5


def test_a_refused_launch_is_the_error_of_its_own_call(lb):
    """More feature groups than a grid is high: the runtime refuses the launch on the host.  The calls that come after it, of
    this library and of torch, do not find that error waiting."""
    from legateboost_b200 import stages

    F = 32 * 65535 + 1
    row_ptr, proposals = torch.arange(F + 1, dtype=torch.int32, device="cuda"), torch.full((F,), np.inf, device="cuda")
    with pytest.raises(lb.library.LbkError, match="invalid"):
        stages.bin_matrix(torch.zeros((1, F), device="cuda"), proposals, row_ptr)
    assert torch.equal(torch.arange(5, device="cuda") + 1, dev(np.arange(1, 6)))
    F = 40
    bins = stages.bin_matrix(torch.zeros((3, F), device="cuda"), proposals[:F], row_ptr[: F + 1])
    assert bins.shape == (3, 64) and not bins.any()


def test_bad_arguments_are_errors(lb):
    from legateboost_b200.tree import build_tree_arrays

    X = dev(np.zeros((10, 3), dtype=np.float32))
    g = dev(np.zeros((10, 1)))
    with pytest.raises(lb.library.LbkError):
        build_tree_arrays(X, g, g, max_depth=2, split_samples=5000, seed=0, row_offset=0, dataset_rows=10)
    with pytest.raises(lb.library.LbkError):
        build_tree_arrays(X, g, g, max_depth=2, split_samples=16, seed=0, row_offset=5, dataset_rows=10)


def test_first_predict_on_the_training_matrix_uses_the_leaf_record(lb):
    """fit() keeps the node every training row ended in; the first predict() on the same, unmodified
    tensor gathers leaf values from it.  It must equal the walk over X bit for bit, must be used
    once, and must not be used after the tensor changed."""
    rs = np.random.RandomState(3)
    for dtype, K, F, S in ((np.float32, 1, 40, 256), (np.float64, 3, 7, 500)):
        X = dev(rs.random((3000, F)).astype(dtype))
        g = dev(rs.normal(size=(3000, K)))
        h = dev(rs.random((3000, K)) + 0.1)
        t = lb.Tree(max_depth=6, split_samples=S).set_random_state(np.random.RandomState(1)).fit(X, g, h)
        assert t._fit_rows is not None
        want = lb.Tree.batch_predict([t], X)
        got = t.predict(X)
        assert t._fit_rows is None
        assert torch.equal(got, want)
        assert torch.equal(t.predict(X), want)           # the walk over X this time
        t.fit(X, g, h)
        X[0, 0] += 1.0                                   # in-place change: the record is stale
        want = lb.Tree.batch_predict([t], X)
        assert torch.equal(t.predict(X), want)
    stump = lb.Tree(max_depth=0).set_random_state(np.random.RandomState(1)).fit(X, g, h)
    assert torch.equal(stump.predict(X), lb.Tree.batch_predict([stump], X))


def _torch_histogram(bins, gpair, node, node_begin, n_nodes, F, n_bins):
    """An independent integer histogram on the device: index_add_ of the pairs at
    node * B + feature * n_bins + bin, a few features at a time (int64, exact)."""
    B = F * n_bins
    out = torch.zeros((n_nodes * B, 2), dtype=torch.int64, device=bins.device)
    base = (node.long() - node_begin) * B
    vals = gpair[:, 0, :].long()
    step = 8
    for f0 in range(0, F, step):
        f1 = min(F, f0 + step)
        idx = base[:, None] + bins[:, f0:f1].long() + (torch.arange(f0, f1, device=bins.device) * n_bins)[None, :]
        out.index_add_(0, idx.reshape(-1), vals[:, None, :].expand(-1, f1 - f0, -1).reshape(-1, 2))
    return out.view(n_nodes, 1, B, 2)


def test_full_size_histogram_exact(lb):
    """The benchmark's own size (10 M x 128, 128 nodes of level 7): every bin of every node equals an
    independent histogram of the same inputs (integer arithmetic: exact)."""
    import bench
    from legateboost_b200 import stages

    n = 10_000_000
    bins, row_ptr, gpair, _, row_index, seg, node, max_abs = bench.hist_inputs(torch, n, 7, torch.device("cuda"))
    hist = stages.histogram(bins, row_ptr, gpair, row_index, seg, bench.HIST_FEATURES, mode=0, max_abs=max_abs)
    n_nodes = seg.shape[0] - 1
    want = _torch_histogram(bins, gpair, node, n_nodes - 1, n_nodes, bench.HIST_FEATURES, bench.HIST_BINS)
    assert torch.equal(hist, want)
    # the same call without the magnitudes handed in (the library finds them) gives the same bits
    assert torch.equal(stages.histogram(bins, row_ptr, gpair, row_index, seg, bench.HIST_FEATURES, mode=0), hist)


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("F", [1, 4, 5, 8, 9, 16, 17, 31, 32, 33, 36, 37, 40, 41, 48, 49, 63, 64, 65, 66, 72, 73, 80, 81, 96, 97, 100, 101, 105, 112, 113, 129])
def test_histogram_of_every_unit_form(lb, F, mode):
    """Units of fewer than 64 features have fewer steps and copies of their words: every number of features at which the
    form changes, against an independent histogram.  The pairs are small whole numbers, whose float32 sums are exact as well."""
    from legateboost_b200 import stages

    N, n_nodes = 17_000_000 // F + 77, 300
    gen = torch.Generator(device="cuda")
    gen.manual_seed(F)
    bins = torch.zeros((N, (F + 31) // 32 * 32), dtype=torch.uint8, device="cuda")
    bins[:, :F] = torch.randint(0, 256, (N, F), dtype=torch.uint8, device="cuda", generator=gen)
    node = (torch.rand(N, device="cuda", generator=gen) ** 3 * n_nodes).to(torch.int32) + (n_nodes - 1)
    pairs = torch.randint(-5, 6, (N, 1, 2), dtype=torch.int32, device="cuda", generator=gen)
    row_index, seg = stages.group_rows(node, n_nodes - 1, n_nodes)
    row_ptr = torch.arange(F + 1, dtype=torch.int32, device="cuda") * 256
    want = _torch_histogram(bins, pairs, node, n_nodes - 1, n_nodes, F, 256)
    cast = torch.float32 if mode else torch.int32
    for by_position in (False, True):
        given = pairs[row_index.long()].contiguous() if by_position else pairs
        max_abs = torch.tensor([5, 5], dtype=torch.int32, device="cuda") if mode == 0 else None
        for merge_tree in (False, True):
            got = stages.histogram(bins, row_ptr, given.to(cast), row_index, seg, F, mode=mode, max_abs=max_abs,
                                   pairs_by_position=by_position, merge_tree=merge_tree)
            assert torch.equal(got, want.to(got.dtype)), (by_position, merge_tree)


@pytest.mark.parametrize("merge_tree", [False, True])
@pytest.mark.parametrize("N,F,K,weights,mode,qmax", [
    (1_500_000, 64, 1, [0.80, 0.0, 0.15, 0.05], 0, 300),    # one node in about 120 pieces (a deep merge tree)
    (1_500_000, 64, 1, [0.80, 0.0, 0.15, 0.05], 0, 5000),   # ... too many rows for 32-bit sums (the tree is climbed
                                                            # two levels, the rest are 64-bit atomics)
    (1_500_000, 64, 1, [0.80, 0.0, 0.15, 0.05], 0, 40000),  # ... (one level only)
    (1_500_000, 64, 1, [0.80, 0.0, 0.15, 0.05], 0, 400000), # ... a piece is flushed several times (no tree)
    (1_500_000, 96, 3, [0.3, 0.3, 0.2, 0.1, 0.1], 0, 300),  # three groups: the second group set is half empty
    (2_000_000, 32, 2, [1.0] * 37, 0, 300),                 # one group per unit (two blocks per SM)
    (1_500_000, 128, 1, [0.55, 0.45], 1, 0),                # float pairs through the same ranges
])
def test_histogram_static_ranges(lb, oracle, N, F, K, weights, mode, qmax, merge_tree):
    """Enough rows for the planner to hand out equal static ranges: nodes reach over range boundaries and their pieces
    add to their histograms with atomics or, as on a rank with peers, meet in merge trees; sums stay exact (floats
    within 1e-5)."""
    from legateboost_b200 import stages

    rng = np.random.default_rng(N + F)
    n_nodes = len(weights)
    edges = np.cumsum(np.asarray(weights) / np.sum(weights))
    node = np.minimum(np.searchsorted(edges, rng.random(N), side="right"), n_nodes - 1).astype(np.int32) + (n_nodes - 1)
    bins = rng.integers(0, 256, size=(N, F), dtype=np.uint8)
    row_ptr = (np.arange(F + 1) * 256).astype(np.int32)
    row_index, seg = stages.group_rows(dev(node), n_nodes - 1, n_nodes)
    if mode == 0:
        q = rng.integers(-qmax, qmax, size=(N, K, 2), dtype=np.int32)
        q[:, :, 1] = np.abs(q[:, :, 1])
        want = oracle.histogram_q(bins, row_ptr, q, node, n_nodes - 1, 2 * n_nodes - 1)
        got = stages.histogram(stages.to_padded_rows(dev(bins)), dev(row_ptr), dev(q), row_index, seg, F, mode=0, merge_tree=merge_tree)
        assert np.array_equal(got.cpu().numpy(), want)
        got = stages.histogram(stages.to_padded_rows(dev(bins)), dev(row_ptr), _by_position(dev(q), row_index), row_index,
                               seg, F, mode=0, pairs_by_position=True, max_abs=_max_abs(q), merge_tree=merge_tree)
        assert np.array_equal(got.cpu().numpy(), want)
    else:
        gh = np.stack([rng.normal(size=(N, K)), np.ones((N, K))], axis=2).astype(np.float32)
        want = oracle.histogram_d(bins, row_ptr, gh[:, :, 0].copy(), gh[:, :, 1].copy(), node, n_nodes - 1, 2 * n_nodes - 1)
        for by_pos in (False, True):
            pairs = _by_position(dev(gh), row_index) if by_pos else dev(gh)
            got = stages.histogram(stages.to_padded_rows(dev(bins)), dev(row_ptr), pairs, row_index, seg, F, mode=1,
                                   pairs_by_position=by_pos, merge_tree=merge_tree)
            err = np.abs(got.cpu().numpy() - want).max()
            assert err <= 1e-5 * np.abs(want).max()


def test_full_size_tree_properties(lb):
    """10 M x 64 rows, depth 8: the node of every training row from the builder equals the walk over
    X; the hessians of the children add up to the parent's (h = 1: the root holds the row count)."""
    n, F = 10_000_000, 64
    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    X = torch.rand((n, F), dtype=torch.float32, device="cuda", generator=gen)
    g = torch.randn((n, 1), dtype=torch.float64, device="cuda", generator=gen)
    h = torch.ones((n, 1), dtype=torch.float64, device="cuda")
    t = lb.Tree(max_depth=8).set_random_state(np.random.RandomState(2)).fit(X, g, h)
    walk = lb.Tree.batch_predict([t], X)
    assert torch.equal(t.predict(X), walk)
    feature = t.feature.cpu().numpy()
    hess = t.hessian.cpu().numpy()[:, 0]
    assert abs(hess[0] - n) <= 1e-6 * n
    split = np.nonzero(feature >= 0)[0]
    assert len(split) > 100
    assert np.allclose(hess[2 * split + 1] + hess[2 * split + 2], hess[split], rtol=1e-12, atol=0)


@pytest.mark.parametrize("dtype,K,D,l1,l2", [(np.float32, 1, 6, 0.0, 1.0), (np.float64, 3, 5, 0.3, 0.5),
                                               (np.float32, 12, 8, 0.0, 1.0)])
def test_update_tree_matches_oracle(lb, oracle, dtype, K, D, l1, l2):
    """Tree.update (UPDATE_TREE): new leaf values and hessians for an unchanged structure.  Float64
    sums in another order than the reference's row loop: 1e-10 relative, hessians included; nodes
    no row reaches get 0."""
    rs = np.random.RandomState(17)
    N, F = 20000, 15
    X = rs.random((N, F)).astype(dtype)
    g = rs.normal(size=(N, K))
    h = rs.random((N, K)) + 0.1
    t = lb.Tree(max_depth=D, split_samples=64, l1_regularization=l1, l2_regularization=l2)
    t.set_random_state(np.random.RandomState(4)).fit(dev(X), dev(g), dev(h))
    feature, split = t.feature.cpu().numpy(), t.split_value.cpu().numpy()
    old_leaf = t.leaf_value.clone()
    g2 = rs.normal(size=(N, K))
    h2 = (rs.random((N, K)) + 0.05) * (rs.random((N, K)) > 0.2)   # some zero hessians
    sub = slice(0, N // 3)                                         # fewer rows: some nodes stay empty
    want_leaf, want_hess = oracle.update_tree(X[sub], g2[sub], h2[sub], feature, split, l1=l1, l2=l2)
    t.update(dev(X[sub]), dev(g2[sub]), dev(h2[sub]))
    assert torch.equal(t.feature.cpu(), torch.from_numpy(feature))
    got_leaf, got_hess = t.leaf_value.cpu().numpy(), t.hessian.cpu().numpy()
    assert np.allclose(got_hess, want_hess, rtol=1e-10, atol=1e-12)
    assert np.allclose(got_leaf, want_leaf, rtol=1e-9, atol=1e-12)
    assert not np.array_equal(got_leaf, old_leaf.cpu().numpy())
    assert np.array_equal(got_leaf == 0.0, want_leaf == 0.0)
    # the updated tree predicts with the new values
    pred = t.predict(dev(X[:100]))
    assert np.allclose(pred.cpu().numpy(), oracle.predict(X[:100], [(got_leaf, feature, split)]), rtol=0, atol=0)
    # an empty shard keeps every node at zero
    t.update(dev(X[:0]), dev(g2[:0]), dev(h2[:0]))
    assert not t.leaf_value.any() and not t.hessian.any()


def test_weighted_gradient_kernels_match_the_array_formulas(lb):
    """lbk_gradient against the reference's chain of array operations (objectives.py:131-135, 489-512,
    legateboost.py:189-224), evaluated with numpy: squared error bit for bit, log loss within the last
    bits of exp / division."""
    from legateboost_b200 import estimator as E

    rs = np.random.RandomState(8)
    N = 5000
    est = lb.LBRegressor(learning_rate=0.3)
    est._obj = E._SquaredError()
    raw, y = rs.normal(size=(N, 3)), rs.normal(size=(N, 3))
    g, h = est._weighted_gradient(dev(y), dev(raw))
    assert np.array_equal(g.cpu().numpy(), (raw - y) * 0.3) and np.array_equal(h.cpu().numpy(), np.ones((N, 3)))
    est._obj = E._LogLoss()
    raw, y = rs.normal(size=(N, 1)) * 4, rs.randint(0, 2, size=(N, 1)).astype(np.float64)
    g, h = est._weighted_gradient(dev(y), dev(raw))
    p = 1.0 / (1.0 + np.exp(-raw))
    assert np.allclose(g.cpu().numpy(), (p - y) * 0.3, rtol=1e-13, atol=1e-16)
    assert np.allclose(h.cpu().numpy(), np.maximum(p * (1 - p), 1e-8), rtol=1e-13)
    for K in (3, 10, 40):
        raw, y = rs.normal(size=(N, K)) * 5, rs.randint(0, K, size=(N, 1)).astype(np.float64)
        raw[0] = 800.0 * np.arange(K)  # far apart: hessians hit the floor
        g, h = est._weighted_gradient(dev(y), dev(raw))
        e = np.exp(raw - raw.max(axis=1, keepdims=True))
        p = e / e.sum(axis=1, keepdims=True)
        want_g = p.copy()
        want_g[np.arange(N), y[:, 0].astype(int)] -= 1.0
        assert np.allclose(g.cpu().numpy(), want_g * 0.3, rtol=1e-12, atol=1e-15)
        assert np.allclose(h.cpu().numpy(), np.maximum(p * (1 - p), 1e-8), rtol=1e-12)
        assert h.min().item() == 1e-8


@pytest.mark.parametrize("N,F,D,S,classes,dtype", [
    (1, 1, 1, 16, 0, np.float32), (500, 10, 4, 256, 0, np.float32),        # one launch per tree, gradients inside
    (16384, 3, 7, 64, 0, np.float64), (4000, 200, 3, 100, 2, np.float32),  # the most rows; more features than SMs
    (1500, 20, 5, 32, 5, np.float32),                                      # ... several outputs: gradients outside
    (16385, 9, 6, 256, 0, np.float32), (20000, 33, 9, 256, 2, np.float32), # the general path
    (3000, 40, 5, 400, 3, np.float64),                                     # ... two-byte bins
])
def test_rounds_in_the_library_match_rounds_from_python(lb, N, F, D, S, classes, dtype):
    """fit() queues whole rounds (`lbk_boost_round`); the same rounds driven tree by tree (gradient, Tree.fit,
    prediction of the leaf record) give the same bits: every step does the same arithmetic."""
    rs = np.random.RandomState(N % 101 + F)
    X = rs.normal(size=(N, F)).astype(dtype)
    X[:, 0] = np.round(X[:, 0] * 2) / 2
    X = dev(X)
    y = dev(rs.normal(size=N)) + 2 * X[:, 0].double() if classes == 0 else dev(rs.randint(0, classes, size=N))
    kw = dict(n_estimators=5, random_state=3, base_models=(
        lb.Tree(max_depth=D, split_samples=S), lb.Tree(max_depth=max(D - 1, 0), split_samples=S, feature_fraction=0.6)))
    kind = lb.LBClassifier if classes else lb.LBRegressor
    a, b = kind(**kw), kind(**kw)
    a._rounds_in_library = lambda: False
    a.fit(X, y)
    b.fit(X, y)
    assert len(a) == len(b) == 5
    for i in range(5):
        for name in ("feature", "split_value", "gain", "leaf_value", "hessian"):
            assert torch.equal(getattr(a[i], name), getattr(b[i], name)), (i, name)
    assert torch.equal(a._train_pred, b._train_pred)
    assert torch.equal(a.predict_raw(X[:50]), b.predict_raw(X[:50]))


def random_trees(rs, F, K, T, D):
    M = 2 ** (D + 1) - 1
    trees = []
    for _ in range(T):
        feat = rs.randint(0, F, size=M).astype(np.int32)
        feat[2 ** D - 1:] = -1
        feat[rs.random(M) < 0.1] = -1
        trees.append((rs.normal(size=(M, K)), feat, rs.normal(size=M)))
    return trees


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("N,F,K,T,D", [
    (8193, 1, 1, 1, 0), (8200, 7, 1, 8, 1), (20011, 100, 1, 17, 8),   # one group, whole groups, a last group of one
    (9001, 5, 1, 3, 10), (9001, 40, 1, 30, 13), (8193, 3, 2, 9, 14),  # narrower groups and blocks for deep trees
    (8193, 425, 1, 17, 6), (8193, 426, 1, 17, 6),                     # the widest rows of a tile, and wider (f64)
    (8193, 851, 1, 17, 6), (8193, 852, 1, 17, 6),                     # ... (f32)
    (8193, 700, 3, 9, 6), (8193, 800, 20, 5, 3), (8193, 1025, 1, 3, 9),
    (8193, 12, 2, 9, 6), (30001, 20, 4, 8, 7), (8193, 3, 5, 16, 5), (8193, 9, 8, 10, 5),  # sums in registers
    (8193, 4, 16, 3, 4), (8193, 4, 17, 11, 4),                        # ... the most of them; in shared memory
    (8193, 60, 1, 16, 6), (8193, 136, 1, 16, 6),                      # 48 KB of dynamic shared memory to the byte (f64, f32)
])
def test_predict_of_many_rows_is_bit_exact(lb, oracle, dtype, N, F, K, T, D):
    """More rows than the one-launch form takes: trees in groups in shared memory, for rows that start on 16 bytes
    and rows that do not, with values that compare false with everything."""
    from legateboost_b200.tree import predict_arrays

    rs = np.random.RandomState(N % 97 + F + K + T + D)
    X = rs.normal(size=(N, F)).astype(dtype)
    X[rs.random((N, F)) < 0.01] = np.nan
    X[rs.random((N, F)) < 0.01] = np.inf
    X[rs.random((N, F)) < 0.01] = -np.inf
    trees = random_trees(rs, F, K, T, D)
    d_trees = [tuple(map(dev, t)) for t in trees]
    want = oracle.predict(X, trees)
    assert np.array_equal(predict_arrays(dev(X), d_trees).cpu().numpy(), want)
    wide = torch.zeros((N, F + 2), dtype=torch.from_numpy(X).dtype, device="cuda")
    wide[:, 1:F + 1] = dev(X)
    assert np.array_equal(predict_arrays(wide[:, 1:F + 1], d_trees).cpu().numpy(), want)


@pytest.mark.parametrize("N,classes,F", [(50, 2, 4), (9000, 2, 4), (50, 3, 4), (9000, 3, 4), (9000, 10, 3), (9000, 20, 4)])
def test_probabilities_are_those_of_the_raw_predictions(lb, N, classes, F):
    rs = np.random.RandomState(classes)
    X = dev(rs.normal(size=(N, F)))
    m = lb.LBClassifier(n_estimators=4, base_models=(lb.Tree(max_depth=3, split_samples=32),), random_state=0)
    m.fit(X, dev(np.arange(N) % classes))
    raw = m.predict_raw(X)
    p = torch.sigmoid(raw) if classes == 2 else torch.softmax(raw, dim=1)
    if classes == 2:
        p = torch.cat([1.0 - p, p], dim=1)
    # exp, a sum of `classes` terms and a division: a few units in the last place
    assert torch.allclose(m.predict_proba(X), p, rtol=(classes + 8) * 2.3e-16, atol=2.3e-16)


def test_an_ensemble_predicts_what_its_trees_hold_now(lb):
    """The device table of the trees' addresses follows every way to change a tree."""
    from legateboost_b200.tree import predict_arrays

    rs = np.random.RandomState(0)
    X = dev(rs.normal(size=(300, 5)))
    m = lb.LBRegressor(n_estimators=3, base_models=(lb.Tree(max_depth=3),), random_state=0).fit(X, dev(rs.normal(size=300)))

    def check():
        want = m.model_init_ + predict_arrays(X, [tree_tuple(t) for t in m])
        assert torch.equal(m.predict_raw(X), want)

    check()
    m[0].leaf_value.mul_(2.0)
    check()
    m[1].leaf_value = m[1].leaf_value * 3.0
    check()
    m[2].leaf_value.data = m[2].leaf_value * 4.0  # the same tensor, other memory
    check()
    m[0].feature.set_(m[0].feature.clone())
    check()
    m.models_.append(m[0] * 0.5)
    check()
    m[3].leaf_value = m[3].leaf_value.repeat(1, 2)
    with pytest.raises(ValueError):
        m.predict_raw(X)


def test_fits_on_several_threads_and_streams(lb):
    """Calls in progress on one device share a context: what their kernels tell the host and where their blocks
    meet belongs to one call."""
    import threading

    rs = np.random.RandomState(0)
    jobs = []
    for i, (N, F, S) in enumerate([(700, 6, 64), (30000, 12, 400), (900, 9, 256), (20000, 5, 600)]):
        jobs.append((dev(rs.normal(size=(N, F))), dev(rs.normal(size=N)), S, i))

    def fit(X, y, S, seed):
        return lb.LBRegressor(n_estimators=4, base_models=(lb.Tree(max_depth=5, split_samples=S),), random_state=seed).fit(X, y)

    want = [fit(*j) for j in jobs]
    torch.cuda.synchronize()
    got, errors = {}, []

    def work(j):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(5):
                    got[j[3]] = fit(*j)
        except Exception as e:  # seen by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
    for j, w in zip(jobs, want):
        for a, b in zip(got[j[3]], w):
            for name in ("feature", "split_value", "leaf_value", "hessian"):
                assert torch.equal(getattr(a, name), getattr(b, name))


@pytest.mark.parametrize("dtype,N,F,S", [
    (np.float64, 1, 1, 512), (np.float64, 1003, 37, 512), (np.float64, 4099, 33, 1024), (np.float64, 2051, 5, 2048),
    (np.float32, 1048583, 1, 1024), (np.float32, 40009, 27, 1000), (np.float32, 131075, 9, 2048), (np.float32, 500, 9, 2048),
])
def test_two_byte_bin_ids_count_the_proposals_below(lb, dtype, N, F, S):
    """The id of a value is the number of proposals below it (0 for a NaN); the padding columns are zero."""
    from legateboost_b200 import stages

    rs = np.random.RandomState(F)
    X = rs.normal(size=(N, F)).astype(dtype)
    X[rs.random((N, F)) < 0.01] = np.inf
    X[rs.random((N, F)) < 0.01] = -np.inf
    sample = dev(rs.normal(size=(4000, F)).astype(dtype))
    proposals, row_ptr = stages.split_proposals(sample, S, 3)
    p, rp = proposals.cpu().numpy(), row_ptr.cpu().numpy()
    X[: min(N, 300)] = p[rp[:-1]]  # values that are proposals
    X[rs.random((N, F)) < 0.01] = np.nan
    got = stages.bin_matrix(dev(X), proposals, row_ptr, 2).cpu().numpy()
    assert not got[:, F:].any()
    for f in range(F):
        x = X[:, f]
        want = np.where(np.isnan(x), 0, np.searchsorted(p[rp[f]:rp[f + 1]], x, side="left"))
        assert np.array_equal(got[:, f], want), f


@pytest.mark.parametrize("N,F,S", [(1, 1, 256), (63, 3, 100), (1025, 33, 256), (40007, 64, 256), (5000, 9, 65)])
@pytest.mark.parametrize("kind", ["uniform", "normal", "lognormal", "crowded", "few", "outliers", "negative_infinity", "nan"])
def test_one_byte_bin_ids_count_the_proposals_below(lb, kind, N, F, S):
    """Whatever the distribution: columns for which the search starts from the bucket table, with three steps or four,
    and columns whose proposals crowd in few buckets or are not in order."""
    from legateboost_b200 import stages

    rs = np.random.RandomState(N % 89 + S)
    make = {
        "uniform": lambda n: rs.random((n, F)), "normal": lambda n: rs.normal(size=(n, F)),
        "lognormal": lambda n: np.exp(1.5 * rs.normal(size=(n, F))), "crowded": lambda n: np.exp(8 * rs.normal(size=(n, F))),
        "few": lambda n: np.round(4 * rs.normal(size=(n, F))), "outliers": lambda n: rs.normal(size=(n, F)) * np.where(rs.random((n, F)) < 0.005, 1e30, 1),
        "negative_infinity": lambda n: np.where(rs.random((n, F)) < 0.01, -np.inf, rs.normal(size=(n, F))),
        "nan": lambda n: np.where(rs.random((n, F)) < 0.01, np.nan, rs.normal(size=(n, F))),
    }[kind]
    proposals, row_ptr = stages.split_proposals(dev(make(3000).astype(np.float32)), S, 3)
    p, rp = proposals.cpu().numpy(), row_ptr.cpu().numpy()
    X = make(N).astype(np.float32)
    X[rs.random((N, F)) < 0.02] = np.inf
    X[rs.random((N, F)) < 0.02] = -np.inf
    for i in range(min(N, 200)):  # the proposals themselves and their neighbours
        at = rp[:-1] + i % np.diff(rp)
        X[i] = p[at] if i % 3 == 0 else np.nextafter(p[at], np.float32(np.inf if i % 3 == 1 else -np.inf))
    X[rs.random((N, F)) < 0.02] = np.nan
    got = stages.bin_matrix(dev(X), proposals, row_ptr, 1).cpu().numpy()
    assert not got[:, F:].any()
    for f in range(F):
        table = np.full(256, np.inf, dtype=np.float32)
        table[: rp[f + 1] - rp[f]] = p[rp[f]:rp[f + 1]]
        want = np.zeros(N, dtype=np.int64)
        for step in (128, 64, 32, 16, 8, 4, 2, 1):  # (also for a table with a NaN in it, where the order of probes matters)
            want += np.where(table[want + step - 1] < X[:, f], step, 0)
        assert np.array_equal(got[:, f], want), f


@pytest.mark.parametrize("offset", [0, 1, 2, 4])
@pytest.mark.parametrize("N", [1, 31, 32, 33, 95, 4737])
def test_one_byte_bin_ids_on_any_boundary(lb, N, offset):
    """Whole and partial tiles of 32 rows; row-major ids that may leave as words of four, and ids that may not."""
    from legateboost_b200 import library as L
    from legateboost_b200 import stages
    from legateboost_b200.tree import _stream_ptr

    F, rs = 41, np.random.RandomState(N)
    proposals, row_ptr = stages.split_proposals(dev(rs.random((2000, F)).astype(np.float32)), 256, 3)
    p, rp = proposals.cpu().numpy(), row_ptr.cpu().numpy()
    X, ctx = rs.random((N, F)).astype(np.float32), L.context(0)
    dX = dev(X)
    room = torch.full((offset + N * 64 + 64,), 255, dtype=torch.uint8, device="cuda")
    ctx.check(ctx.lib.lbk_bin_matrix(ctx.handle, dX.data_ptr(), L.LBK_F32, F, N, F, proposals.data_ptr(), row_ptr.data_ptr(),
                                     room.data_ptr() + offset, 1, _stream_ptr()))
    got = room.cpu().numpy()
    ids = got[offset:offset + N * 64].reshape(N, 64)
    for f in range(F):
        assert np.array_equal(ids[:, f], np.searchsorted(p[rp[f]:rp[f + 1]], X[:, f], side="left")), f
    assert not ids[:, F:].any() and (got[:offset] == 255).all() and (got[offset + N * 64:] == 255).all()


@pytest.mark.parametrize("N,F", [
    (2 * 75776 + 1, 64), (3 * 75776, 33),                       # two tables: 75776 rows a turn of all blocks; a last team of one row
    (2 * 50176 + 97, 75), (5 * 29696 + 31, 160), (40007, 250),  # three, five and eight tables, which do not divide the SMs
])
def test_one_byte_bin_ids_of_several_turns(lb, oracle, N, F):
    """Rows that take every warp through its turns twice and more, row-major and in the feature-major copy that the rows
    are repartitioned by (a wrong id there is a row in a wrong node)."""
    from legateboost_b200 import stages
    from legateboost_b200.tree import build_tree_arrays

    rs = np.random.RandomState(F)
    X = rs.random((N, F)).astype(np.float32)
    dX = dev(X)
    proposals, row_ptr = stages.split_proposals(dX, 256, 3)
    p, rp = proposals.cpu().numpy(), row_ptr.cpu().numpy()
    got = stages.bin_matrix(dX, proposals, row_ptr, 1).cpu().numpy()
    assert not got[:, F:].any()
    for f in range(F):
        assert np.array_equal(got[:, f], np.searchsorted(p[rp[f]:rp[f + 1]], X[:, f], side="left")), f
    g, h = rs.normal(size=(N, 1)) + np.sin(6 * X[:, :1]), np.ones((N, 1))
    want = oracle.build_tree(X, g, h, max_depth=3, split_samples=256, seed=5, mode="Q")
    tree = build_tree_arrays(dX, dev(g), dev(h), max_depth=3, split_samples=256, seed=5, row_offset=0, dataset_rows=N)
    for name in ("feature", "split_value", "gain", "leaf_value", "hessian"):
        assert np.array_equal(tree[name].cpu().numpy(), getattr(want, name)), name


@pytest.mark.parametrize("N,F,S,dt", [
    (250_003, 40, 512, np.float64), (80_001, 39, 2048, np.float64), (250_003, 40, 1000, np.float32), (150_001, 37, 2048, np.float32),
    (30_000, 40, 512, np.float64),  # too few rows for a table of starts
])
@pytest.mark.parametrize("spread", ["even", "crowded"])
def test_two_byte_bin_ids_of_many_rows(lb, oracle, N, F, S, dt, spread):
    """Searches that begin from a table, of three and four steps, and whole ones where proposals crowd together."""
    from legateboost_b200 import stages
    from legateboost_b200.tree import build_tree_arrays

    rs = np.random.RandomState(F + S)
    X = rs.random((N, F)).astype(dt)
    if spread == "crowded":
        X[:, 1::3] = np.exp(4 * rs.normal(size=X[:, 1::3].shape)).astype(dt)
        X[:, 2::3] = np.round(X[:, 2::3] * 700) / 700
        X[:, 3] = 7.0
        X[rs.randint(N, size=20), 4] = 1e30
    proposals, row_ptr = stages.split_proposals(dev(X), S, 3)
    p, rp = proposals.cpu().numpy(), row_ptr.cpu().numpy()
    Z = X.copy()
    for value in (np.nan, np.inf, -np.inf, 0.0):
        Z[rs.randint(N, size=500), rs.randint(F, size=500)] = value
    got = stages.bin_matrix(dev(Z), proposals, row_ptr, 2).cpu().numpy().view(np.uint16)
    assert not got[:, F:].any()
    for f in range(F):
        want = np.where(np.isnan(Z[:, f]), 0, np.searchsorted(p[rp[f]:rp[f + 1]], Z[:, f], side="left"))
        assert np.array_equal(got[:, f], want), f
    g, h = rs.normal(size=(N, 1)) + np.sin(6 * X[:, :1]), np.ones((N, 1))  # (the feature-major copy)
    want = oracle.build_tree(X, g, h, max_depth=2, split_samples=S, seed=5, mode="Q")
    tree = build_tree_arrays(dev(X), dev(g), dev(h), max_depth=2, split_samples=S, seed=5, row_offset=0, dataset_rows=N)
    for name in ("feature", "split_value", "gain", "leaf_value", "hessian"):
        assert np.array_equal(tree[name].cpu().numpy(), getattr(want, name)), name


@pytest.mark.parametrize("N,K", [(1, 3), (255, 23), (257, 24), (1000, 186), (70, 187), (70, 300)])
def test_softmax_gradients_of_whole_and_partial_tiles(lb, N, K):
    """The tiled kernel (256 rows down to 32 per block) and the one for more classes than it takes."""
    from legateboost_b200 import estimator as E

    rs = np.random.RandomState(K)
    est = lb.LBRegressor(learning_rate=0.3)
    est._obj = E._LogLoss()
    raw, y = rs.normal(size=(N, K)) * 5, rs.randint(0, K, size=(N, 1)).astype(np.float64)
    g, h = est._weighted_gradient(dev(y), dev(raw))
    e = np.exp(raw - raw.max(axis=1, keepdims=True))
    p = e / e.sum(axis=1, keepdims=True)
    want_g = p.copy()
    want_g[np.arange(N), y[:, 0].astype(int)] -= 1.0
    tol = (K + 8) * 2.3e-16  # exp, K additions, a division, a product
    assert np.allclose(g.cpu().numpy(), want_g * 0.3, rtol=tol, atol=tol)
    assert np.allclose(h.cpu().numpy(), np.maximum(p * (1 - p), 1e-8), rtol=tol, atol=tol)


@pytest.mark.parametrize("N,F,K,bins,nodes", [
    (131072, 8, 1, 256, 1), (65537, 17, 1, 256, 40), (65537, 17, 1, 256, 60),  # from 2^20 cells on; units around the SMs
    (70001, 9, 2, 256, 5), (131072, 7, 1, 256, 3),                             # several outputs; fewer cells
    (40009, 30, 1, 512, 7), (40009, 30, 1, 300, 64), (40009, 27, 1, 1024, 7),  # two-byte ids
    (300007, 60, 1, 256, 9), (300007, 60, 1, 256, 64),                         # more cells: few units, many units
    (60013, 150, 1, 200, 8),                                                   # many units with rows in them
])
@pytest.mark.parametrize("largest", [1 << 12, 1 << 26])
def test_histograms_of_moderate_matrices(lb, N, F, K, bins, nodes, largest):
    """The forms for up to 3 * 2^24 cells: one copy of the histograms or four, nodes of very different sizes, magnitudes
    for which a block has to empty its 32-bit sums after 31 rows (64-bit atomics) or not before the end."""
    from legateboost_b200 import stages

    rs = np.random.RandomState(N % 97 + F)
    ids = rs.randint(0, bins, size=(N, F))
    ids[:, 0] = np.minimum(ids[:, 0], 2)  # a crowded column
    dt = np.uint8 if bins <= 256 else np.int16
    node = np.minimum(rs.geometric(0.4, size=N) - 1, nodes - 1).astype(np.int32) if nodes < 50 else rs.randint(0, nodes, size=N).astype(np.int32)
    q = rs.randint(-largest, largest, size=(N, K, 2)).astype(np.int32)
    row_ptr = (np.arange(F + 1) * bins).astype(np.int32)
    d_node = dev(node)
    row_index, seg = stages.group_rows(d_node, 0, nodes)
    hist = stages.histogram(stages.to_padded_rows(dev(ids.astype(dt))), dev(row_ptr), dev(q), row_index, seg, F, mode=0)
    want = torch.zeros((nodes * F * bins, K, 2), dtype=torch.int64, device="cuda")
    for f in range(F):
        want.index_add_(0, (d_node.long() * F + f) * bins + dev(ids[:, f]).long(), dev(q).long())
    want = want.view(nodes, F * bins, K, 2).permute(0, 2, 1, 3)
    assert torch.equal(hist, want)


@pytest.mark.parametrize("K", [700, 740, 768, 3072])
def test_many_outputs_at_the_edge_of_default_shared_memory(lb, oracle, K):
    """The per-output tables of the quantiser and of the split search grow past what a launch may use without asking."""
    from legateboost_b200.tree import build_tree_arrays

    rs = np.random.RandomState(K)
    N, D = (40, 2) if K < 3000 else (40, 0)  # (the most outputs that the quantiser takes)
    X = rs.normal(size=(N, 1)).astype(np.float32)
    g, h = rs.normal(size=(N, K)), rs.random((N, K)) + 0.1
    t = build_tree_arrays(dev(X), dev(g), dev(h), max_depth=D, split_samples=8, seed=1, row_offset=0, dataset_rows=N)
    want = oracle.build_tree(X, g, h, max_depth=D, split_samples=8, seed=1, mode="Q")
    for name in ("feature", "split_value", "gain", "leaf_value", "hessian"):
        assert np.array_equal(t[name].cpu().numpy(), getattr(want, name)), name


@pytest.mark.parametrize("N,F,K,D,S,dt", [
    (40_000, 30, 1, 8, 256, np.float32), (40_000, 33, 1, 8, 100, np.float64),  # a warp per feature on the last levels
    (9_000, 60, 1, 8, 700, np.float32), (20_000, 101, 3, 7, 256, np.float32), (4_000, 130, 10, 7, 256, np.float32),
    (33_000, 49, 2, 8, 31, np.float32),
])
def test_wide_levels(lb, oracle, N, F, K, D, S, dt):
    for small in (False, True):
        _, want, got = _run_tree_case(lb, oracle, (N, F, K, D, S, dt, {"mask": small}), seed=D, hess_small=small)
        for name in ("feature", "split_value", "node_sums", "gain", "hessian", "leaf_value"):
            assert np.array_equal(got[name].cpu().numpy(), getattr(want, name)), name


@pytest.mark.parametrize("N,F,K,D,S", [(5_921, 206, 3, 7, 256), (25_053, 51, 1, 9, 256), (60_000, 40, 1, 8, 64), (9_001, 300, 1, 7, 300)])
@pytest.mark.parametrize("pure", [0.0, 0.9])
def test_wide_levels_of_few_nodes(lb, oracle, N, F, K, D, S, pure):
    """Levels that are wide by their nodes, of which some or (rows of which most have the same gradient) few exist."""
    from legateboost_b200.tree import build_tree_arrays

    rs = np.random.RandomState(D)
    X = rs.random((N, F)).astype(np.float32)
    g = rs.normal(size=(N, K))
    g[X[:, 0] < pure] = -1.0  # (nothing is to be gained below the split that takes these apart)
    h = np.ones((N, K))
    want = oracle.build_tree(X, g, h, max_depth=D, split_samples=S, seed=3, mode="Q")
    got = build_tree_arrays(dev(X), dev(g), dev(h), max_depth=D, split_samples=S, seed=3, row_offset=0, dataset_rows=N)
    for name in ("feature", "split_value", "node_sums", "gain", "hessian", "leaf_value"):
        assert np.array_equal(got[name].cpu().numpy(), getattr(want, name)), name


@pytest.mark.parametrize("N,F,K,D,dt", [
    (26_001, 20, 1, 6, np.float32), (32_768, 4, 1, 3, np.float64), (32_769, 4, 1, 3, np.float64),  # many rows; one too many
    (3_000, 64, 1, 9, np.float32), (900, 145, 1, 9, np.float64),  # a warp per pair of nodes, in whole and broken turns
    (300, 12, 1, 11, np.float32), (2_000, 18, 3, 8, np.float32), (700, 9, 10, 5, np.float64),
    (400, 300, 10, 4, np.float32), (12_000, 300, 1, 8, np.float32),  # few rows, but the general path is faster
])
def test_trees_around_the_one_launch_rule(lb, oracle, N, F, K, D, dt):
    for small in (False, True):  # (hessians that quantise to 0: raw bins stay in the scan)
        _, want, got = _run_tree_case(lb, oracle, (N, F, K, D, 256, dt, {}), seed=D, hess_small=small)
        for name in ("feature", "split_value", "node_sums", "gain", "hessian", "leaf_value"):
            assert np.array_equal(got[name].cpu().numpy(), getattr(want, name)), name


@pytest.mark.parametrize("N,F,K,D", [(40, 300, 1, 8), (500, 10, 1, 6), (2000, 3, 3, 7), (16384, 2, 1, 5)])
def test_one_launch_trees_are_the_same_every_time(lb, oracle, N, F, K, D):
    """The blocks of the one-launch tree pick every level's winners for themselves and must agree, whichever of them is
    ahead: one feature or several per block, several blocks per feature."""
    from legateboost_b200.tree import build_tree_arrays

    rs = np.random.RandomState(N)
    X, g, h = rs.normal(size=(N, F)).astype(np.float32), rs.normal(size=(N, K)), rs.random((N, K)) + 0.1
    want = oracle.build_tree(X, g, h, max_depth=D, split_samples=64, seed=9, mode="Q")
    d = [dev(a) for a in (X, g, h)]
    for i in range(50):
        t = build_tree_arrays(*d, max_depth=D, split_samples=64, seed=9, row_offset=0, dataset_rows=N)
        for name in ("feature", "split_value", "gain", "leaf_value", "hessian"):
            assert np.array_equal(t[name].cpu().numpy(), getattr(want, name)), (i, name)


def test_round_after_a_barrier_that_gave_up(lb):
    """The barrier word of a one-launch tree starts below what its blocks can count up to, so that the bounded wait runs
    out (about a second): the fault is reported, and what is queued behind the tree finds no rows' nodes or values that
    were never written (softmax: the leaf values are added by a kernel of its own)."""
    import ctypes as C

    L = lb.library
    rs = np.random.RandomState(0)
    N, F, K, D = 300, 4, 3, 3
    M = 2 ** (D + 1) - 1
    X, y, pred = dev(rs.normal(size=(N, F)).astype(np.float32)), dev(rs.randint(0, K, size=N).astype(np.float64)), dev(rs.normal(size=(N, K)))
    before = pred.clone()
    tree = dict(leaf_value=torch.full((M, K), 7.0, dtype=torch.float64, device="cuda"), feature=torch.full((M,), 3, dtype=torch.int32, device="cuda"))
    for name, shape in (("split_value", M), ("gain", M), ("hessian", M * K)):
        tree[name] = torch.full((shape,), 7.0, dtype=torch.float64, device="cuda")
    word = torch.full((1,), -2 ** 30, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ctx = L.context()
    r = L.BoostRoundArgs()
    a = r.tree
    a.X, a.x_dtype, a.ldx = X.data_ptr(), L.LBK_F32, F
    a.n_local_rows, a.dataset_rows, a.n_features, a.n_outputs = N, N, F, K
    a.max_depth, a.max_nodes, a.split_samples, a.seed, a.l2_regularization = D, M, 16, 1, 1.0
    for name, t in tree.items():
        setattr(a, name, t.data_ptr())
    a.stream = torch.cuda.current_stream().cuda_stream
    r.objective, r.y, r.pred, r.learning_rate, r.zeroed = 1, y.data_ptr(), pred.data_ptr(), 0.5, word.data_ptr()
    ctx.check(ctx.lib.lbk_boost_round(ctx.handle, C.byref(r)))
    with pytest.raises(L.LbkError, match="fault code 51"):
        ctx.check(ctx.lib.lbk_synchronize(ctx.handle, a.stream))
    assert torch.equal(pred, before)
    assert (tree["feature"] == -1).all() and not tree["leaf_value"].any() and not tree["hessian"].any()
    word.zero_()
    ctx.check(ctx.lib.lbk_boost_round(ctx.handle, C.byref(r)))
    ctx.check(ctx.lib.lbk_synchronize(ctx.handle, a.stream))
    assert not torch.equal(pred, before) and (tree["feature"][0] >= 0)


def test_predictions_on_several_threads(lb, oracle):
    """Tiles of different sizes of the same kernel, launched from several threads on one context: the limit of shared
    memory that a function may ask for is the same for all of them."""
    import threading

    from legateboost_b200.tree import predict_arrays

    rs = np.random.RandomState(2)
    jobs = []
    for F, T, D in ((3, 1, 2), (100, 40, 8), (300, 9, 4), (20, 16, 10)):
        X, trees = rs.normal(size=(8200, F)).astype(np.float32), random_trees(rs, F, 1, T, D)
        jobs.append((dev(X), [tuple(map(dev, t)) for t in trees], oracle.predict(X, trees)))
    errors = []

    def work(X, trees, want):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(40):
                    got = predict_arrays(X, trees)
                assert np.array_equal(got.cpu().numpy(), want)
        except Exception as e:  # seen by the main thread
            errors.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_error_texts_of_calls_on_several_threads(lb):
    """A text that is being read is not replaced by another thread's failing call: every thread reads one of the texts
    that were written, whole."""
    import ctypes as C
    import threading

    ctx = lb.library.context()
    seen = set()

    def fail(dtype, n):
        a = lb.library.PredictArgs()
        a.x_dtype, a.n_rows, a.X, a.pred = dtype, 1, 16, 16  # (refused before anything is read)
        for _ in range(n):
            assert ctx.lib.lbk_predict(ctx.handle, C.byref(a)) != 0
            seen.add(ctx.lib.lbk_last_error(ctx.handle))

    fail(9, 1)
    fail(0, 1)
    texts = set(seen)
    assert len(texts) == 2
    threads = [threading.Thread(target=fail, args=(d, 2000)) for d in (9, 0, 9, 0)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert seen == texts


@pytest.mark.parametrize("N,S", [(20000, 64), (20000, 400), (3_400_000, 400), (500, 64)])  # (400: a wait for the width, for the layout)
@pytest.mark.parametrize("fixed_sketch", [False, True])
def test_calls_give_back_the_words_they_borrow(lb, N, S, fixed_sketch):
    import ctypes as C

    from legateboost_b200.tree import build_tree_arrays

    ctx = lb.library.context()

    def lent():
        v = C.c_int(-1)
        ctx.check(ctx.lib.lbk_context_lent_words(ctx.handle, C.byref(v)))
        return v.value

    before = lent()  # (what a call that failed kept)
    rs = np.random.RandomState(0)
    X, y = dev(rs.normal(size=(N, 5)).astype(np.float32)), dev(rs.normal(size=N))
    lb.LBRegressor(n_estimators=7, base_models=(lb.Tree(max_depth=3, split_samples=S),), random_state=0, fixed_sketch=fixed_sketch).fit(X, y)
    build_tree_arrays(X, y[:, None], torch.ones_like(y)[:, None], max_depth=3, split_samples=S, seed=1, row_offset=0, dataset_rows=N)
    assert lent() == before


@pytest.mark.parametrize("K,transform", [(1, "RAW"), (3, "RAW"), (1, "LOGISTIC"), (3, "SOFTMAX")])
@pytest.mark.parametrize("with_init", [False, True])
def test_an_ensemble_without_trees_takes_rows_of_any_width(lb, K, transform, with_init):
    """Through the C ABI: every row is the initial prediction (or 0), transformed; X is not read, so that its width does
    not matter."""
    import ctypes as C

    L = lb.library
    N, F, columns = 9000, 20000, 2 if transform == "LOGISTIC" else K
    X = torch.full((1, F), float("nan"), dtype=torch.float64, device="cuda")  # (a row stands for all of them)
    init = dev(np.linspace(-1.0, 2.0, K))
    pred = torch.full((N, columns + 1), 7.0, dtype=torch.float64, device="cuda")
    a = L.PredictArgs()
    a.X, a.x_dtype, a.ldx, a.n_rows, a.n_features, a.n_outputs = X.data_ptr(), L.LBK_F64, F, N, F, K
    a.pred, a.ldp, a.transform = pred.data_ptr(), columns + 1, getattr(L, transform)
    a.init = init.data_ptr() if with_init else None
    a.stream = torch.cuda.current_stream().cuda_stream
    ctx = L.context()
    ctx.check(ctx.lib.lbk_predict(ctx.handle, C.byref(a)))
    raw = init if with_init else torch.zeros_like(init)
    want = raw if transform == "RAW" else torch.softmax(raw, 0) if transform == "SOFTMAX" else torch.stack([1 - torch.sigmoid(raw[0]), torch.sigmoid(raw[0])])
    assert torch.allclose(pred[:, :columns], want.expand(N, columns), rtol=1e-15 * (K + 8), atol=0)
    assert (pred[:, columns] == 7.0).all()


@pytest.mark.parametrize("N", [500, 30000])
def test_node_sums_go_to_any_array_of_64_bit_numbers(lb, N):
    """The kernels' own 16-byte accesses must not reach an array that is aligned to 8 bytes only."""
    import ctypes as C

    from legateboost_b200.tree import build_tree_arrays

    L = lb.library
    rs = np.random.RandomState(1)
    F, K, D = 6, 2, 4
    M = 2 ** (D + 1) - 1
    X, g, h = dev(rs.normal(size=(N, F)).astype(np.float32)), dev(rs.normal(size=(N, K))), dev(rs.random((N, K)) + 0.1)
    want = build_tree_arrays(X, g, h, max_depth=D, split_samples=32, seed=4, row_offset=0, dataset_rows=N)
    sums = torch.full((M * K * 2 + 2,), -5, dtype=torch.int64, device="cuda")
    assert sums.data_ptr() % 16 == 0
    out = [torch.empty((M * K,), dtype=torch.float64, device="cuda") for _ in range(4)] + [torch.empty((M,), dtype=torch.int32, device="cuda")]
    a = L.BuildTreeArgs()
    a.X, a.x_dtype, a.ldx, a.g, a.h, a.ldg = X.data_ptr(), L.LBK_F32, F, g.data_ptr(), h.data_ptr(), K
    a.n_local_rows, a.dataset_rows, a.n_features, a.n_outputs = N, N, F, K
    a.max_depth, a.max_nodes, a.split_samples, a.seed, a.l2_regularization = D, M, 32, 4, 1.0
    a.leaf_value, a.split_value, a.gain, a.hessian, a.feature = (t.data_ptr() for t in out)
    a.stream = torch.cuda.current_stream().cuda_stream
    a.trace_node_sums = sums.data_ptr() + 8
    ctx = L.context()
    ctx.check(ctx.lib.lbk_build_tree(ctx.handle, C.byref(a)))
    assert torch.equal(sums[1:-1].view(M, K, 2), want["node_sums"])
    assert sums[0] == -5 and sums[-1] == -5


@pytest.mark.parametrize("N,nb", [(20000, 512), (20000, 1024), (3000, 300)])
@pytest.mark.parametrize("allocating", [True, False])
def test_two_byte_histograms_of_arrays_on_any_boundary(lb, N, nb, allocating):
    """Two-byte bins that begin on 2 bytes and histograms that begin on 8: taken as they are."""
    import ctypes as C

    L = lb.library
    rs = np.random.RandomState(nb)
    F, nodes, Fp = 20, 5, 32
    ids = np.zeros((N, Fp), dtype=np.int16)
    ids[:, :F] = rs.randint(0, nb, size=(N, F))
    from legateboost_b200 import stages

    d_node = dev(rs.randint(0, nodes, size=N).astype(np.int32))
    row_index, seg = stages.group_rows(d_node, 0, nodes)
    q, row_ptr = dev(rs.randint(-4000, 4000, size=(N, 1, 2)).astype(np.int32)), dev((np.arange(F + 1) * nb).astype(np.int32))
    want = torch.zeros((nodes * F * nb, 2), dtype=torch.int64, device="cuda")
    for f in range(F):
        want.index_add_(0, (d_node.long() * F + f) * nb + dev(ids[:, f].astype(np.int64)), q[:, 0].long())
    for shift_bins in (0, 1):
        for shift_hist in (0, 1):
            bins = torch.zeros((N * Fp + 8,), dtype=torch.int16, device="cuda")
            bins[shift_bins:N * Fp + shift_bins] = dev(ids.reshape(-1))
            hist = torch.full((nodes * F * nb * 2 + 2,), -7, dtype=torch.int64, device="cuda")
            a = L.HistogramArgs()
            a.bins, a.bin_bytes, a.n_rows, a.n_features = bins.data_ptr() + 2 * shift_bins, 2, N, F
            a.row_ptr, a.total_bins, a.gpair, a.n_outputs = row_ptr.data_ptr(), F * nb, q.data_ptr(), 1
            a.row_index, a.seg, a.n_nodes, a.hist = row_index.data_ptr(), seg.data_ptr(), nodes, hist.data_ptr() + 8 * shift_hist
            a.stream = torch.cuda.current_stream().cuda_stream
            ctx = L.context()
            if allocating:
                ctx.check(ctx.lib.lbk_histogram(ctx.handle, C.byref(a)))
            else:
                assert ctx.lib.lbk_histogram_noalloc(0, C.byref(a)) == 0
            assert torch.equal(hist[shift_hist:shift_hist + want.numel()], want.view(-1))
            assert (hist[shift_hist + want.numel():] == -7).all() and (hist[:shift_hist] == -7).all()


@pytest.mark.parametrize("N", [100, 9000])
def test_queued_predictions_outlive_the_model_and_the_rows(lb, N):
    """A prediction is queued on a stream that is busy; its model and rows, made on another stream, are given up, and their
    memory is asked for again there."""
    rs = np.random.RandomState(N)
    Xt, y = dev(rs.normal(size=(2000, 6))), dev(rs.normal(size=2000))
    X = dev(rs.normal(size=(N, 6)))
    busy = torch.cuda.Stream()
    for K in (1, 3):
        def model():
            base = (lb.Tree(max_depth=4),)
            if K == 1:
                return lb.LBRegressor(n_estimators=5, base_models=base, random_state=0).fit(Xt, y)
            return lb.LBClassifier(n_estimators=5, base_models=base, random_state=0).fit(Xt, y.argsort() % K)

        m = model()
        want = m.predict_raw(X)
        for fresh in (False, True):
            m, rows = model(), X.clone()
            if not fresh:
                m.predict_raw(rows)  # (the table is made on this stream)
            torch.cuda.synchronize()
            with torch.cuda.stream(busy):
                torch.cuda._sleep(200_000_000)
                got = m.predict_raw(rows)
            del m, rows
            junk = [torch.full((n,), float("nan"), dtype=torch.float64, device="cuda") for n in (4, 16, 64, 155, 465, 1000, N * 6) for _ in range(40)]
            torch.cuda.synchronize()
            del junk
            assert torch.equal(got, want), (K, fresh)


def test_a_round_that_fails_waits_for_the_rounds_before_it(lb):
    rs = np.random.RandomState(0)
    X, y = dev(rs.normal(size=(500, 4))), dev(rs.normal(size=500))
    bad = lb.Tree(max_depth=3)
    bad.split_samples = 4096  # (refused by the library, on the host)
    m = lb.LBRegressor(n_estimators=4, base_models=(lb.Tree(max_depth=3), bad), random_state=0)
    lb.LBRegressor(n_estimators=1, base_models=(lb.Tree(max_depth=3),), random_state=0).fit(X, y)
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(200_000_000)
        with pytest.raises(lb.library.LbkError, match="split_samples"):
            m.fit(X, y)
        assert stream.query()
    assert m.models_ == []
    lb.LBRegressor(n_estimators=1, base_models=(lb.Tree(max_depth=3),), random_state=0).fit(X, y)


@pytest.mark.parametrize("N,F,dtype,distinct", [(21001, 7, dtype, distinct) for dtype in (np.float32, np.float64) for distinct in (3, 200, 10 ** 6)] +
                         [(130_001, 37, dtype, distinct) for dtype in (np.float32, np.float64) for distinct in (3, 300, 10 ** 6)] +
                         [(230_001, 75, np.float32, 50), (230_001, 75, np.float32, 10 ** 6)])
def test_fine_bins_of_one_byte_and_of_two(lb, oracle, N, F, dtype, distinct):
    """More than 256 samples, columns whose values ask for ids of one byte and of two: matrices whose ids wait for the
    number of bins, and (above 2^24 cells) one whose whole layout does."""
    from legateboost_b200.tree import build_tree_arrays

    rs = np.random.RandomState(distinct % 97)
    D = 5
    X = np.round(rs.random((N, F)) * distinct).astype(dtype)
    g, h = rs.normal(size=(N, 1)), rs.random((N, 1)) + 0.1
    want = oracle.build_tree(X, g, h, max_depth=D, split_samples=700, seed=11, mode="Q")
    got = build_tree_arrays(dev(X), dev(g), dev(h), max_depth=D, split_samples=700, seed=11, row_offset=0, dataset_rows=N)
    for name in ("feature", "split_value", "gain", "leaf_value", "hessian"):
        assert np.array_equal(got[name].cpu().numpy(), getattr(want, name)), name


@pytest.mark.parametrize("N,F,K", [(30011, 9, 1), (30011, 9, 2), (20003, 40, 3)])
@pytest.mark.parametrize("S", [256, 700])
def test_squared_error_rounds_are_trees_on_their_gradients(lb, N, F, K, S):
    """Rounds read predictions and labels, of one target or several, where trees driven one by one are given (g, h)."""
    rs = np.random.RandomState(K)
    X, y = dev(rs.normal(size=(N, F)).astype(np.float32)), dev(rs.normal(size=(N, K)))
    make = lambda: lb.LBRegressor(n_estimators=3, base_models=(lb.Tree(max_depth=5, split_samples=S),), random_state=5, learning_rate=0.3)
    one_by_one = make()
    one_by_one._weighted_gradient = lambda *a: lb.LBRegressor._weighted_gradient(one_by_one, *a)  # (gradients of one's own are asked for)
    want, got = one_by_one.fit(X, y), make().fit(X, y)
    for a, b in zip(want, got):
        for name in ("feature", "split_value", "gain", "leaf_value", "hessian"):
            assert torch.equal(getattr(a, name), getattr(b, name)), name
    assert torch.equal(want._train_pred, got._train_pred)


@pytest.mark.parametrize("N,F,K,depth", [(17001, 5, 1, 3), (20011, 9, 1, 9), (17003, 6, 1, 10), (6007, 40, 3, 7), (5801, 300, 3, 4), (5801, 33, 10, 7),
                                         (20011, 4, 2, 4), (5801, 9, 24, 3), (5801, 9, 24, 6), (5801, 9, 30, 4)])
def test_rounds_add_the_leaf_values_where_the_leaves_are_found(lb, N, F, K, depth):
    """Leaf tables made by every block and read from memory (more than 1024 values), rows too wide for the tiled walk: the
    kept predictions are those of the trees."""
    rs = np.random.RandomState(depth)
    X = dev(rs.normal(size=(N, F)).astype(np.float32))
    y = dev(rs.normal(size=(N, K))) if K <= 2 else dev(rs.randint(0, K, size=N).astype(np.float64))
    make = lb.LBRegressor if K <= 2 else lb.LBClassifier
    m = make(n_estimators=3, base_models=(lb.Tree(max_depth=depth),), random_state=5).fit(X, y)
    want = m.model_init_.repeat(N, 1)
    for t in m:
        want += lb.Tree.batch_predict([t], X)
    assert torch.equal(m._train_pred, want)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("F,width,offset", [(1, 1, 0), (2, 3, 1), (3, 7, 2), (4, 4, 0), (5, 9, 3), (7, 7, 0), (8, 13, 1), (33, 40, 3), (75, 75, 0)])
def test_predict_rows_on_any_boundary(lb, oracle, dtype, F, width, offset):
    """Rows that begin and end on any value of a 16-byte vector: columns of a wider matrix, odd numbers of columns."""
    rs = np.random.RandomState(F * 7 + offset)
    N, D = 8193 + 37, 5
    M = 2 ** (D + 1) - 1
    wide = rs.normal(size=(N, width)).astype(dtype)
    X = wide[:, offset:offset + F]
    trees = []
    for _ in range(9):
        feature = np.where(np.arange(M) < 2 ** D - 1, rs.randint(0, F, size=M), -1).astype(np.int32)
        trees.append((rs.normal(size=(M, 1)), feature, rs.normal(size=M) * 0.5))
    got = lb.tree.predict_arrays(dev(wide)[:, offset:offset + F], [tuple(dev(a) for a in t) for t in trees])
    assert np.array_equal(got.cpu().numpy(), oracle.predict(np.ascontiguousarray(X), trees))
