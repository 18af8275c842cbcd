"""The last step of a top-k: lists whose scores the one-histogram pass orders (few binades, few equal scores) and lists that it hands to the
digits (wide ranges, many equal scores, empty slots), against a plain sort by (score descending, row ascending)."""
import numpy as np
import pytest

from oracle import phoenix_oracle as po

pytestmark = pytest.mark.gpu


def scores_of(kind, n, rng):
    """n scores that are bf16 values."""
    if kind == "spread":                      # a few binades, few equal
        return rng.uniform(0.2, 0.9, n)
    if kind == "binades":                     # from 2^-60 up: further down than 255 codes
        return np.exp2(rng.uniform(-60, 0, n))
    if kind == "equal":
        return np.full(n, 0.75)
    if kind == "runs":                        # about 250 of one score
        return 0.5 + np.floor(np.arange(n) / 250) / 256
    if kind == "long runs":                   # more of one score than a code's keys are compared with one another
        return 0.5 + np.floor(np.arange(n) / 300) / 256
    if kind == "negative":
        return -rng.uniform(0.2, 0.9, n)
    if kind == "signs":
        return rng.uniform(-1, 1, n)
    return np.where(rng.random(n) < 0.5, 0.0, rng.uniform(0.1, 1.0, n))     # zeros


@pytest.mark.parametrize("kind", ["spread", "binades", "equal", "runs", "long runs", "negative", "signs", "zeros"])
@pytest.mark.parametrize("n,ks", [(5, (1, 5)), (1000, (1, 31, 999, 1000)), (4097, (700, 1024)), (30001, (1, 1000, 4096))])
def test_select_orders_every_kind_of_list(kind, n, ks):
    """A corpus that fits the survivor buffer: every row is collected, so the list is the select kernel's work alone."""
    import torch
    from x_algorithm_b200.retrieval import CorpusShard
    rng = np.random.default_rng(n)
    c = po.bf16_round(scores_of(kind, n, rng).astype(np.float32))
    c = c[rng.permutation(n)]
    rows = np.zeros((n, 64), np.float32)
    rows[:, 3] = c
    sh = CorpusShard(n, 64, max_queries=3, max_k=max(ks), row_offset=7)
    sh.upload(0, po.bf16_bits(rows))
    users = torch.zeros((3, 64), device="cuda")
    users[:, 3] = torch.tensor([1.0, 0.5, -2.0])
    for k in ks:
        sc = torch.empty((3, k), dtype=torch.float32, device="cuda")
        ids = torch.empty((3, k), dtype=torch.int64, device="cuda")
        sh.topk_device(users, 3, k, sc, ids)
        sh.sync()
        for u, f in enumerate((1.0, 0.5, -2.0)):
            s = (c * np.float32(f)) + np.float32(0)          # exact: a power of two; -0 counts as 0
            order = np.lexsort((np.arange(n), -s))[:k]
            np.testing.assert_array_equal(ids[u].cpu().numpy(), order + 7)
            np.testing.assert_array_equal(sc[u].cpu().numpy(), s[order])
    sh.close()


def test_merge_of_lists_with_empty_slots():
    """Lists of fp32 scores (more than a code's bits), at the bf16 minimum, and with empty slots: best first, empty ones at the end."""
    import torch
    from x_algorithm_b200.retrieval import CorpusShard
    P, B, k = 5, 4, 37
    rng = np.random.default_rng(3)
    sc = rng.uniform(0.5, 0.52, (P, B, k)).astype(np.float32)
    ids = rng.permutation(P * B * k).reshape(P, B, k).astype(np.int64)
    sc[:, 1] = np.float32(-3.3895314e38)                      # all at the bf16 minimum
    ids[1:, 2] = -1                                           # one list only
    ids[:, 3] = -1
    ids[2, 3, :5] = np.arange(5)                              # five entries in all
    ids[3:, 1, 5:] = -1                                       # the minimum beside empty slots
    sh = CorpusShard(64, 64, max_queries=B, max_k=k)
    out_s = torch.empty((B, k), dtype=torch.float32, device="cuda")
    out_i = torch.empty((B, k), dtype=torch.int64, device="cuda")
    sh.merge_device(torch.from_numpy(sc).cuda(), torch.from_numpy(ids).cuda(), P, B, k, out_s, out_i)
    sh.sync()
    for b in range(B):
        s, i = sc[:, b].ravel(), ids[:, b].ravel()
        s, i = s[i >= 0], i[i >= 0]
        order = np.lexsort((i, -s))[:k]
        want_s, want_i = np.full(k, -np.inf, np.float32), np.full(k, -1, np.int64)
        want_s[:len(order)], want_i[:len(order)] = s[order], i[order]
        np.testing.assert_array_equal(out_i[b].cpu().numpy(), want_i)
        np.testing.assert_array_equal(out_s[b].cpu().numpy(), want_s)
    sh.close()


@pytest.mark.parametrize("P,k", [(2, 5), (3, 37), (5, 256)])
def test_merge_of_lists_that_share_entries(P, k):
    """An entry that several lists hold is there as often in the result."""
    import torch
    from x_algorithm_b200.retrieval import CorpusShard
    B = 2
    rng = np.random.default_rng(P)
    one = -np.sort(-rng.uniform(0.5, 0.9, (B, k)).astype(np.float32), axis=1)
    sc = np.ascontiguousarray(np.broadcast_to(one, (P, B, k)))
    ids = np.ascontiguousarray(np.broadcast_to(rng.permutation(B * k).reshape(B, k), (P, B, k))).astype(np.int64)
    sh = CorpusShard(64, 64, max_queries=B, max_k=k)
    out_s = torch.full((B, k), 7.0, dtype=torch.float32, device="cuda")
    out_i = torch.full((B, k), 7, dtype=torch.int64, device="cuda")
    sh.merge_device(torch.from_numpy(sc).cuda(), torch.from_numpy(ids).cuda(), P, B, k, out_s, out_i)
    sh.sync()
    for b in range(B):
        s, i = sc[:, b].ravel(), ids[:, b].ravel()
        order = np.lexsort((i, -s))[:k]
        np.testing.assert_array_equal(out_i[b].cpu().numpy(), i[order])
        np.testing.assert_array_equal(out_s[b].cpu().numpy(), s[order])
    sh.close()
