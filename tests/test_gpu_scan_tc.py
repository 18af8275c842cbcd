"""The tcgen05 corpus scan at the edges of its tiles and query widths: 128-row tiles, 64 / 128 / 256 query columns, rows of 64 /
128 bf16 or 128 / 256 int8, with and without the sampled pivot, and row scales the int8 filter has to step aside for."""
import numpy as np
import pytest

from oracle import phoenix_oracle as po

pytestmark = pytest.mark.gpu


def _topk(sh, users, k):
    import torch
    B = users.shape[0]
    u = torch.from_numpy(users).cuda()
    sc = torch.empty((B, k), dtype=torch.float32, device="cuda"); ids = torch.empty((B, k), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    sh.topk_device(u, B, k, sc, ids)
    sh.sync()
    return sc.cpu().numpy(), ids.cpu().numpy()


def _users(B, dim, seed):
    u = np.random.default_rng(seed).standard_normal((B, dim)).astype(np.float32)
    return u / np.linalg.norm(u, axis=1, keepdims=True)


@pytest.mark.parametrize("dim", [128, 256])
@pytest.mark.parametrize("N,B,k", [(127, 1, 5), (128, 64, 128), (129, 65, 3), (33000, 1, 50), (40001, 128, 60), (40000, 129, 60), (36900, 250, 17)])
def test_int8_scan_bit_exact(dim, N, B, k):
    """Ids and scores equal the oracle's; some rows have a zero or a negative scale (their order is turned round)."""
    from x_algorithm_b200.engine import dispatch_counts
    from x_algorithm_b200.retrieval import CorpusShard
    r = np.random.default_rng(N + dim)
    q8 = r.integers(-128, 128, size=(N, dim), dtype=np.int8)
    q8[::31] = q8[3]
    scales = (r.random(N, dtype=np.float32) * np.float32(0.01) + np.float32(1e-4)).astype(np.float32)
    scales[::31] = scales[3]
    scales[5::53] = 0.0
    scales[7::59] *= -1.0
    users = _users(B, dim, 2)
    sh = CorpusShard(N, dim, row_offset=11, max_queries=B, max_k=k)
    sh.upload_int8(0, q8, scales)
    sh.set_int8(True)
    before = dispatch_counts()["scan.tcgen05"]
    got_s, got_i = _topk(sh, users, k)
    assert dispatch_counts()["scan.tcgen05"] > before
    want_s, want_i = po.top_k(po.int8_corpus_scores(users, q8, scales), k, row_offset=11)
    np.testing.assert_array_equal(got_i, want_i)
    np.testing.assert_array_equal(got_s, want_s)
    sh.close()


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("N,B,k", [(127, 1, 5), (129, 64, 40), (33000, 65, 30), (50001, 128, 50), (40000, 129, 20)])
def test_bf16_scan_against_64_bit_scores(dim, N, B, k):
    """Every list is ordered, its scores are the bf16 roundings of the rows' own dot products and no row outside it beats
    the last entry by more than a bf16 step (fp32 sums may round to either neighbour: 2^-8 relative)."""
    from x_algorithm_b200.retrieval import CorpusShard
    users = _users(B, dim, 5)
    sh = CorpusShard(N, dim, max_queries=B, max_k=k)
    sh.fill_synthetic(4)
    got_s, got_i = _topk(sh, users, k)
    sh.close()
    corpus = po.bf16_from_bits(po.synthetic_corpus_rows(np.arange(N), dim, 4)).astype(np.float64)
    full = po.bf16_round(users).astype(np.float64) @ corpus.T
    step = 2.0 ** -8
    for b in range(B):
        own = full[b][got_i[b]]
        assert np.all(np.abs(got_s[b] - own) <= step * np.abs(own) + 1e-6)
        key = np.lexsort((got_i[b], -got_s[b].astype(np.float64)))
        np.testing.assert_array_equal(key, np.arange(k))
        assert len(set(got_i[b])) == k
        rest = np.delete(full[b], got_i[b])
        if rest.size:
            assert rest.max() <= got_s[b][-1] + step * abs(got_s[b][-1]) + 1e-6


@pytest.mark.parametrize("B", [16, 64, 200])
def test_int8_scan_of_huge_queries(B):
    """Query scales near the end of fp32's range (the filter's offset times the scale overflows): the list is complete without
    an exact re-run, and equals the oracle's."""
    from x_algorithm_b200.retrieval import CorpusShard
    N, dim, k = 40001, 128, 30
    r = np.random.default_rng(B)
    q8 = r.integers(-127, 128, size=(N, dim), dtype=np.int8)
    scales = (r.random(N, dtype=np.float32) * np.float32(0.01) + np.float32(1e-4)).astype(np.float32)
    users = (_users(B, dim, 7) * np.float32(4e34)).astype(np.float32)
    assert (np.abs(users).max(1) / 127 * np.float64(12582912.0)).min() > 3.5e38
    sh = CorpusShard(N, dim, max_queries=B, max_k=k)
    sh.upload_int8(0, q8, scales)
    sh.set_int8(True)
    got_s, got_i = _topk(sh, users, k)
    assert sh.exact_runs() == 0
    want_s, want_i = po.top_k(po.int8_corpus_scores(users, q8, scales), k)
    sh.close()
    np.testing.assert_array_equal(got_i, want_i)
    np.testing.assert_array_equal(got_s, want_s)


def test_masked_rows_stand_in_front_of_minus_infinity():
    """Fewer eligible rows than k: masked rows fill the list at the bf16 minimum, and an eligible row whose score is -inf comes
    behind them, as in a top-k over all scores."""
    import torch
    from x_algorithm_b200.retrieval import CorpusShard, Retriever
    N, dim, k = 3000, 64, 9
    rows = np.random.default_rng(3).standard_normal((N, dim)).astype(np.float32)
    rows[1234, 0] = -np.inf
    elig = np.zeros(N, bool)
    elig[[7, 1234, 2000, 2999]] = True
    sh = CorpusShard(N, dim, max_queries=2, max_k=k)
    sh.upload(0, po.bf16_bits(rows))
    sh.set_mask(elig)
    users = np.abs(np.random.default_rng(4).standard_normal((2, dim))).astype(np.float32)
    s, i = Retriever([sh]).retrieve(torch.from_numpy(users).cuda(), k)
    s, i = s.cpu().numpy(), i.cpu().numpy()
    sh.close()
    scores = po.bf16_round(users).astype(np.float64) @ po.bf16_round(rows[[7, 2000, 2999]]).astype(np.float64).T
    lowest = np.frombuffer(np.uint32(0xFF7F0000).tobytes(), np.float32)[0]
    for b in range(2):
        order = np.argsort(-scores[b])
        assert list(i[b]) == [[7, 2000, 2999][o] for o in order] + [0, 1, 2, 3, 4] + [1234]
        assert np.all(s[b, 3:8] == lowest) and s[b, 8] == -np.inf


@pytest.mark.parametrize("N,B,k", [(3_000_000, 1, 1), (3_000_000, 1, 900), (400_000, 256, 3), (400_000, 16, 10), (70_000, 3, 1)])
@pytest.mark.parametrize("int8", [False, True])
def test_sampled_pivot_of_short_lists(N, B, k, int8):
    """How many rows the pivot lets through follows the corpus and the batch, not k alone: the lists equal those of the exact
    passes, and no call had to be done again."""
    from x_algorithm_b200.retrieval import CorpusShard
    sh = CorpusShard(N, 128, max_queries=B, max_k=k)
    sh.fill_synthetic(4)
    if int8:
        sh.quantize_int8()
        sh.set_int8(True)
    users = _users(B, 128, 6)
    got_s, got_i = _topk(sh, users, k)
    assert sh.exact_runs() == 0
    sh.set_exact(True)
    want_s, want_i = _topk(sh, users, k)
    sh.close()
    if int8:                                       # integer sums: the same bits
        np.testing.assert_array_equal(got_i, want_i)
        np.testing.assert_array_equal(got_s, want_s)
    else:                                          # the two scans sum in another order: a bf16 step at a rounding edge
        np.testing.assert_allclose(got_s, want_s, rtol=2.0 ** -7)
        assert (got_i == want_i).mean() > 0.9


@pytest.mark.parametrize("dim", [128, 256])
@pytest.mark.parametrize("kind", ["far_apart", "large_sums", "one_scale", "all_below_zero"])
def test_int8_threshold_in_the_sum(dim, kind):
    """Corpora whose thresholds the bias of the int8 sum cannot express, or only coarsely - row scales over six decades, dot products
    beyond its range, sums below zero throughout - and the plain one: lists and scores equal the oracle's, without an exact re-run."""
    from x_algorithm_b200.retrieval import CorpusShard
    N, B, k = 40001, 70, 25
    r = np.random.default_rng(dim)
    scales = np.full(N, 0.01, np.float32)
    if kind == "far_apart":
        scales = (10.0 ** r.uniform(-6, 0, N)).astype(np.float32)
    users = _users(B, dim, 3)
    if kind in ("large_sums", "all_below_zero"):
        q8 = r.integers(60, 128, size=(N, dim), dtype=np.int8)
        users = np.abs(users) if kind == "large_sums" else -np.abs(users)
    else:
        q8 = r.integers(-127, 128, size=(N, dim), dtype=np.int8)
    sh = CorpusShard(N, dim, max_queries=B, max_k=k)
    sh.upload_int8(0, q8, scales)
    sh.set_int8(True)
    got_s, got_i = _topk(sh, users, k)
    assert sh.exact_runs() == 0
    want_s, want_i = po.top_k(po.int8_corpus_scores(users, q8, scales), k)
    sh.close()
    np.testing.assert_array_equal(got_i, want_i)
    np.testing.assert_array_equal(got_s, want_s)


def _int8_equals_the_oracle(N, dim, B, k, users, q8, scales):
    from x_algorithm_b200.retrieval import CorpusShard
    sh = CorpusShard(N, dim, max_queries=B, max_k=k)
    sh.upload_int8(0, q8, scales)
    sh.set_int8(True)
    got_s, got_i = _topk(sh, users, k)
    assert sh.exact_runs() == 0
    want_s, want_i = po.top_k(po.int8_corpus_scores(users, q8, scales), k)
    sh.close()
    np.testing.assert_array_equal(got_i, want_i)
    np.testing.assert_array_equal(got_s, want_s)


@pytest.mark.parametrize("scales,shares", [
    ((1e-39, 1.1e-38, 1.2e-38), (0.2, 0.4, 0.4)),       # below 2^-126 and just above it, in one corpus
    ((1e-40, 9e-40), (0.5, 0.5)),                       # all of them below
    ((1.2e-38, 1e-36), (0.5, 0.5)),                     # small, but none below
    ((1e-44, 1e-30, 1e-3), (0.3, 0.3, 0.4))])
@pytest.mark.parametrize("magnitude", [1e6, 1e14])
def test_int8_row_scales_near_the_smallest(scales, shares, magnitude):
    """Row scales down to the denormals, with queries large enough that their scores are ordinary numbers."""
    N, B, dim, k = 40001, 3, 128, 25
    r = np.random.default_rng(7)
    s = r.choice(np.array(scales, np.float32), size=N, p=shares).astype(np.float32)
    q8 = r.integers(-127, 128, size=(N, dim), dtype=np.int8)
    _int8_equals_the_oracle(N, dim, B, k, (_users(B, dim, 3) * np.float32(magnitude)).astype(np.float32), q8, s)


@pytest.mark.parametrize("scales,magnitude", [((1e36, 1.2e36), 1e-6), ((1e34, 5e37), 1e-5), ((2e38, 3e38), 1e-7), ((1e-3, 3e38), 1e-7)])
def test_int8_row_scales_near_the_largest(scales, magnitude):
    """Row scales so large that a threshold divided by the query's scale, or the reference of the rows' factors, is infinite."""
    N, B, dim, k = 40001, 3, 128, 25
    r = np.random.default_rng(7)
    s = r.choice(np.array(scales, np.float32), size=N).astype(np.float32)
    q8 = r.integers(-127, 128, size=(N, dim), dtype=np.int8)
    users = (_users(B, dim, 3) * np.float32(magnitude)).astype(np.float32)
    assert np.isfinite(po.int8_corpus_scores(users, q8, s)).all()
    _int8_equals_the_oracle(N, dim, B, k, users, q8, s)


@pytest.mark.parametrize("share", [0.15, 0.5, 0.85])
@pytest.mark.parametrize("scale,where", [(1e-12, "end"), (1e-12, "mixed"), (0.0, "end"), (0.0, "mixed"), (-0.0, "mixed")])
def test_int8_shard_with_empty_rows(share, scale, where):
    """Rows of zeros, as the quantiser leaves them (scale 1e-12) or as an uploader marks them, at the end of a shard or all over it."""
    N, B, dim, k = 40001, 70, 128, 25
    r = np.random.default_rng(8)
    q8 = r.integers(-127, 128, size=(N, dim), dtype=np.int8)
    s = (r.random(N, dtype=np.float32) * np.float32(0.01) + np.float32(1e-3)).astype(np.float32)
    empty = np.arange(N) >= int(N * (1 - share)) if where == "end" else r.random(N) < share
    q8[empty] = 0
    s[empty] = scale
    _int8_equals_the_oracle(N, dim, B, k, _users(B, dim, 3), q8, s)


def _median_us(sh, users, k, n=15):
    import torch
    B = users.shape[0]
    u = torch.from_numpy(users).cuda()
    sc = torch.empty((B, k), dtype=torch.float32, device="cuda"); ids = torch.empty((B, k), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    t = []
    for _ in range(n):
        sh.topk_device(u, B, k, sc, ids)
        sh.sync()
        t.append(sh.last_device_ms() * 1e3)
    return float(np.median(t[3:]))


def _int8_shard(N, dim, B, k, change):
    """A quantised synthetic shard with its scales (and empty rows) as `change` leaves them."""
    import torch
    from x_algorithm_b200.retrieval import CorpusShard
    sh = CorpusShard(N, dim, max_queries=B, max_k=k)
    sh.fill_synthetic(4)
    sh.quantize_int8()
    q = torch.empty((N, dim), dtype=torch.int8, device="cuda"); s = torch.empty(N, dtype=torch.float32, device="cuda")
    sh.read_int8_device(0, N, q, s)
    q8, scales = q.cpu().numpy(), s.cpu().numpy()
    change(np.random.default_rng(1), q8, scales)
    sh.upload_int8(0, q8, scales)
    sh.set_int8(True)
    return sh


def _empty_tail(r, q8, scales):
    n = int(0.85 * len(scales)); q8[n:] = 0; scales[n:] = 1e-12


def _half_empty(r, q8, scales):
    rows = r.random(len(scales)) < 0.5; q8[rows] = 0; scales[rows] = 1e-12


def _zero_scales(r, q8, scales):
    scales[r.random(len(scales)) < 0.15] = 0.0


@pytest.mark.parametrize("change", [_empty_tail, _half_empty, _zero_scales])
def test_int8_filter_serves_shards_that_are_not_full(change):
    """Rows that hold nothing do not switch the filter inside the int8 sum off for the others: with it off such a shard takes 1.6 to 1.8
    times as long as a full one, with it 1.0 to 1.1."""
    N, dim, B, k = 4_000_000, 128, 256, 300
    users = _users(B, dim, 3)
    full = _int8_shard(N, dim, B, k, lambda *a: None)
    t_full = _median_us(full, users, k)
    full.close()
    sh = _int8_shard(N, dim, B, k, change)
    # a negative scale that is overwritten leaves no trace
    sh.upload_int8(N - 3, np.ones((1, dim), np.int8), np.full(1, -1.0, np.float32))
    sh.upload_int8(N - 3, np.ones((1, dim), np.int8), np.full(1, 1e-3, np.float32))
    t = _median_us(sh, users, k)
    assert sh.exact_runs() == 0
    sh.close()
    assert t < 1.35 * t_full, f"{t:.0f} us, a full shard {t_full:.0f} us"


def test_int8_negative_scales_come_and_go():
    """A negative scale turns the order of its row round; uploaded anew with a positive one the row is like any other."""
    from x_algorithm_b200.retrieval import CorpusShard
    N, B, dim, k = 40001, 70, 128, 25
    r = np.random.default_rng(9)
    q8 = r.integers(-127, 128, size=(N, dim), dtype=np.int8)
    s = (r.random(N, dtype=np.float32) * np.float32(0.01) + np.float32(1e-3)).astype(np.float32)
    users = _users(B, dim, 3)
    sh = CorpusShard(N, dim, max_queries=B, max_k=k)
    sh.upload_int8(0, q8, s)
    sh.set_int8(True)
    for rows, sign in (((5, 900), -1.0), ((700, 39000), -1.0), ((5, 39000), 1.0)):
        s[rows[0]:rows[1]] = np.abs(s[rows[0]:rows[1]]) * np.float32(sign)
        sh.upload_int8(rows[0], q8[rows[0]:rows[1]], s[rows[0]:rows[1]])
        got_s, got_i = _topk(sh, users, k)
        want_s, want_i = po.top_k(po.int8_corpus_scores(users, q8, s), k)
        np.testing.assert_array_equal(got_i, want_i)
        np.testing.assert_array_equal(got_s, want_s)
    assert sh.exact_runs() == 0
    sh.close()


@pytest.mark.parametrize("B", [5, 70, 128, 200, 256])
@pytest.mark.parametrize("negative", [False, True])
@pytest.mark.parametrize("below", ["all", "some groups", "one query"])
def test_int8_open_groups(B, negative, below):
    """Queries whose scores are all below zero: throughout, in some groups of query columns, one alone; with and without a row whose scale is
    negative.  The bias is left out, switched off by groups, or not there."""
    N, dim, k = 40001, 128, 25
    r = np.random.default_rng(B)
    q8 = r.integers(20, 128, size=(N, dim), dtype=np.int8)
    s = (r.random(N, dtype=np.float32) * np.float32(0.01) + np.float32(1e-3)).astype(np.float32)
    if negative:
        s[[0, 777, N - 1]] *= np.float32(-1)
    users = np.abs(_users(B, dim, 3))
    down = {"all": np.ones(B, bool), "some groups": np.arange(B) % 64 < 40, "one query": np.arange(B) == B // 2}[below]
    users[down] *= -1
    _int8_equals_the_oracle(N, dim, B, k, users, q8, s)


@pytest.mark.parametrize("L", [20_000, 33_000, 36_000, 40_000, 90_000])
@pytest.mark.parametrize("masked", [False, True])
def test_short_list_with_its_rows_in_one_block(L, masked):
    """The rows that matter stand together - a topic's posts uploaded in a row, or a mask that leaves one range: more of them than
    the survivor buffer holds (32768), fewer than a sparse sample would notice.  The pivot still falls among them."""
    from helpers import check_topk_against_scores
    from x_algorithm_b200.retrieval import CorpusShard
    N, dim, k, first = 1_200_000, 64, 10, 500_001
    r = np.random.default_rng(L)
    base = r.standard_normal(dim).astype(np.float32); base /= np.linalg.norm(base)
    x = r.standard_normal((N, dim), dtype=np.float32) * np.float32(0.02)
    if not masked:
        x[first:first + L] = base + r.standard_normal((L, dim), dtype=np.float32) * np.float32(0.02)
    bits = (x.view(np.uint32) >> 16).astype(np.uint16)
    rows = (bits.astype(np.uint32) << 16).view(np.float32)
    sh = CorpusShard(N, dim, max_queries=1, max_k=k)
    sh.upload(0, bits)
    eligible = np.ones(N, bool)
    if masked:
        eligible[:] = False
        eligible[first:first + L] = True
        sh.set_mask(eligible)
    users = po.bf16_round((base + np.float32(0.05) * r.standard_normal(dim).astype(np.float32))[None]).astype(np.float32)
    got_s, got_i = _topk(sh, users, k)
    assert sh.exact_runs() == 0
    scores = np.where(eligible[None], users @ rows.T, np.float32(-100))
    check_topk_against_scores(scores, got_s, got_i, k)
    sh.close()


@pytest.mark.parametrize("through", ["sync", "communicator"])
def test_short_list_among_rows_a_bf16_step_apart(through):
    """A quarter of the corpus scores within a few bf16 steps of each other: a pivot for some hundred rows lets more of them through than the
    survivor buffer holds, one for three times the list does not.  The call is done again with that one, not by the exact passes."""
    import torch
    from helpers import check_topk_against_scores
    from x_algorithm_b200.retrieval import CorpusShard
    N, dim, k, L = 1_200_000, 64, 10, 300_000
    r = np.random.default_rng(2)
    base = r.standard_normal(dim).astype(np.float32)
    x = r.standard_normal((N, dim), dtype=np.float32) * np.float32(0.05)
    x[500_001:500_001 + L] = base + r.standard_normal((L, dim), dtype=np.float32) * np.float32(0.02)
    bits = (x.view(np.uint32) >> 16).astype(np.uint16)
    rows = (bits.astype(np.uint32) << 16).view(np.float32)
    sh = CorpusShard(N, dim, max_queries=1, max_k=k)
    sh.upload(0, bits)
    users = po.bf16_round((base + np.float32(0.1) * r.standard_normal(dim).astype(np.float32))[None]).astype(np.float32)
    if through == "sync":
        got_s, got_i = _topk(sh, users, k)
    else:
        from x_algorithm_b200 import comm as pc
        cm = pc.Communicator(pc.unique_id(), 0, 1, 0)
        u = torch.from_numpy(users).cuda()
        sc = torch.empty((1, k), dtype=torch.float32, device="cuda"); ids = torch.empty((1, k), dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        cm.retrieve_topk(sh, u, 1, k, sc, ids)
        got_s, got_i = sc.cpu().numpy(), ids.cpu().numpy()
        cm.close()
    assert sh.exact_runs() == 0
    check_topk_against_scores(users @ rows.T, got_s, got_i, k, slack=1e-4)
    sh.close()


@pytest.mark.parametrize("k", [1, 10, 60, 150, 220, 300])
def test_short_lists_do_not_run_short(k):
    """However few rows the sample holds for a short list, the pivot leaves enough of them: over 1024 queries (4 calls of 256, where want is
    smallest) no call is done again.  The bound per query is e^-14."""
    import torch
    from x_algorithm_b200.retrieval import CorpusShard
    N, B = 1_000_000, 256
    sh = CorpusShard(N, 64, max_queries=B, max_k=k)
    sh.fill_synthetic(5)
    sc = torch.empty((B, k), dtype=torch.float32, device="cuda"); ids = torch.empty((B, k), dtype=torch.int64, device="cuda")
    for seed in range(4):
        u = torch.from_numpy(_users(B, 64, seed)).cuda()
        torch.cuda.synchronize()
        sh.topk_device(u, B, k, sc, ids)
        assert not sh.finish()
        assert (ids.sort(dim=1).values.diff(dim=1) > 0).all() and (sc.diff(dim=1) <= 0).all()
    sh.close()


# 200000 rows: 1563 tiles; 10 picks for 17 queries expect five rows of a tile to pass, 1000 more than 30
@pytest.mark.parametrize("int8,N,B,k,split", [(True, 3001, 16, 40, True), (True, 3001, 17, 40, False), (True, 200_000, 17, 10, True),
                                              (True, 200_000, 17, 1000, False), (True, 200_000, 16, 1000, True), (True, 200_000, 65, 10, False),
                                              (False, 3001, 16, 40, True), (False, 200_000, 16, 1000, True), (False, 200_000, 17, 10, False)])
def test_scan_shares_its_tiles_by_the_rows_expected_to_pass(int8, N, B, k, split):
    """Both forms of the collect pass, on both sides of the rule that picks them: int8 lists are the exact passes' (whole sums), bf16 lists the other
    form's, to the bit."""
    from x_algorithm_b200.engine import dispatch_counts
    from x_algorithm_b200.retrieval import CorpusShard
    sh = CorpusShard(N, 128, max_queries=max(B, 17), max_k=k)
    sh.fill_synthetic(4)
    if int8:
        sh.quantize_int8()
        sh.set_int8(True)
    before = dispatch_counts()
    got = _topk(sh, _users(B, 128, 9), k)
    after = dispatch_counts()
    assert after["scan.tcgen05"] > before["scan.tcgen05"] and after["topk.exact"] == before["topk.exact"]
    assert (after["form.scan_split"] > before["form.scan_split"]) == split
    if int8:
        sh.set_exact(True)
        want = _topk(sh, _users(B, 128, 9), k)
    else:
        want = _topk(sh, _users(33 - B, 128, 9), k)             # 16 and 17: the first 16 queries are the same
        assert (dispatch_counts()["form.scan_split"] > after["form.scan_split"]) != split
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g[:16] if not int8 else g, w[:16] if not int8 else w)
    sh.close()
