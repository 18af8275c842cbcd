"""The tcgen05 attention kernels under grouped q heads and the split token layout: the streaming kernel (head dim 128, histories
past 128 keys) and the resident-history kernel (head dim 64), with and without a candidate-only tail, at the edges of the
128-row query tiles and the 64 / 128-key blocks, against the oracle and against the mma.sync kernels."""
import numpy as np
import pytest

from helpers import assert_heads_close, logits_of, make_pair, rel_l2, to_inputs
from oracle import phoenix_oracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,C,dh,hq,hkv,tail", [(129, 1, 64, 4, 2, 1), (128, 129, 64, 4, 1, 0), (127, 40, 128, 4, 1, 1), (200, 130, 128, 2, 2, 2),
                                                (257, 65, 64, 4, 4, 0), (64, 128, 128, 4, 2, 0), (1, 5, 128, 2, 1, 1)])
def test_grouped_heads_and_split_rows(monkeypatch, S, C, dh, hq, hkv, tail):
    from x_algorithm_b200.engine import dispatch_counts
    B = 38 if dh == 64 and S <= 128 else 3              # the resident kernel starts at 148 (batch, head) pairs
    kw = dict(max_batch=B, emb_size=256, num_q_heads=hq, num_kv_heads=hkv, key_size=dh, history_len=S, num_candidates=C, num_layers=2,
              num_candidate_only_layers=tail)
    ocfg, w, rows_fn, eng = make_pair(**kw)
    b = po.make_batch(ocfg, B, seed=S + C, ragged=True)
    before = dispatch_counts()
    got = eng.rank(to_inputs(b))
    ran = {k: v - before[k] for k, v in dispatch_counts().items() if k.startswith("attn.") and v != before[k]}
    assert set(ran) == {"attn.pingpong" if dh == 64 and S <= 128 else "attn.tcgen05"}, ran
    monkeypatch.setenv("PHX_ATTN", "mma")
    other = eng.rank(to_inputs(b))
    eng.close()
    valid = b.cand_post_ids != 0
    assert rel_l2(logits_of(got.log_probs[valid]), logits_of(other.log_probs[valid])) < 1e-2
    few = slice(0, 3)
    bb = po.RankBatch(*(getattr(b, f)[few] for f in ("hist_post_ids", "hist_author_ids", "hist_actions", "hist_surfaces", "cand_post_ids", "cand_author_ids")))
    lp, cont, logits = po.rank_forward(ocfg, w, rows_fn, bb)
    ok = bb.cand_post_ids != 0
    assert_heads_close(got.log_probs[few][ok], got.continuous[few][ok], logits[ok], cont[ok], 2e-2, str(kw))


@pytest.mark.parametrize("dh,S,cap", [(128, 300, -1.0), (64, 600, -1.0), (128, 300, 30.0)])
def test_row_does_not_depend_on_its_neighbours(dh, S, cap):
    """Streaming kernel: other queries beside a candidate (rows of the same warp, some far larger) leave its output bits alone."""
    import torch
    from x_algorithm_b200.engine import dispatch_counts, ranker_attention
    g = torch.Generator(device="cuda").manual_seed(dh + S)
    B, C, H = 2, 32, 4
    q, k, v = (torch.randn(B, S + C, H, dh, device="cuda", generator=g).to(torch.bfloat16) for _ in range(3))
    seg = torch.ones((B, S + C), dtype=torch.int32, device="cuda")
    seg[:, S:] = -1
    before = dispatch_counts()["attn.tcgen05"]
    a, _ = ranker_attention(q, k, v, seg, S, 0.2, cap, 1 if cap > 0 else 0)
    q2 = q.clone()
    q2[:, S + 1::2] *= 6.0
    b, _ = ranker_attention(q2, k, v, seg, S, 0.2, cap, 1 if cap > 0 else 0)
    assert dispatch_counts()["attn.tcgen05"] == before + 2
    assert torch.equal(a[:, S::2], b[:, S::2]) and not torch.equal(a, b)


@pytest.mark.parametrize("dh,B", [(32, 2), (64, 2), (64, 40), (128, 2)])
def test_negative_history_length_is_no_history(dh, B):
    """A candidate without history keys attends to itself alone: its own value row, whatever the sign of the length given."""
    import torch
    from x_algorithm_b200.engine import ranker_attention
    g = torch.Generator(device="cuda").manual_seed(dh + B)
    q, k, v = (torch.randn(B, 131, 4, dh, device="cuda", generator=g).to(torch.bfloat16) for _ in range(3))
    seg = torch.full((B, 131), -1, dtype=torch.int32, device="cuda")
    for hist_len in (0, -1, -200, -(1 << 31)):
        assert torch.equal(ranker_attention(q, k, v, seg, hist_len, 0.2)[0], v)


@pytest.mark.parametrize("S,C,dh,hq,hkv,B", [(128, 512, 64, 8, 8, 4), (128, 500, 64, 8, 4, 4), (128, 512, 64, 8, 8, 5), (200, 40, 64, 4, 2, 3),
                                             (300, 65, 64, 4, 4, 2), (127, 40, 128, 4, 1, 3), (330, 130, 128, 2, 2, 3), (40, 24, 128, 2, 1, 2)])
def test_candidate_only_last_layer_same_bits(monkeypatch, S, C, dh, hq, hkv, B):
    """The last layer over its candidate rows only gives the candidate outputs of the last layer over every row, bit for bit:
    long histories, heads of 128, grouped heads, and a batch whose tiles just fill the SMs with the history tile counted."""
    kw = dict(max_batch=B, emb_size=256, num_q_heads=hq, num_kv_heads=hkv, key_size=dh, history_len=S, num_candidates=C, num_layers=2)
    ocfg, w, rows_fn, eng = make_pair(**kw)
    b = po.make_batch(ocfg, B, seed=S + B, ragged=True)
    got = eng.rank(to_inputs(b)); eng.close()
    monkeypatch.setenv("PHX_LAST_LAYER", "full")
    _, _, _, eng = make_pair(**kw)
    want = eng.rank(to_inputs(b)); eng.close()
    np.testing.assert_array_equal(got.log_probs, want.log_probs)
    np.testing.assert_array_equal(got.continuous, want.continuous)


@pytest.mark.parametrize("S,C,dh,hq,hkv,kw", [(160, 30, 64, 4, 4, {}), (40, 24, 128, 4, 1, {}), (130, 9, 64, 4, 2, dict(qk_norm=True)),
                                              (20, 70, 128, 2, 2, dict(primer_norm=True))])
def test_debug_taps_hold_every_row_in_request_order(monkeypatch, S, C, dh, hq, hkv, kw):
    """phx_debug_read of the trunk is [B, T] with every row taken through every layer, although the engine keeps history and
    candidate rows apart and skips the last layer's history rows: the bits of an engine that does neither."""
    kw = dict(max_batch=3, emb_size=256, num_q_heads=hq, num_kv_heads=hkv, key_size=dh, history_len=S, num_candidates=C, num_layers=2, **kw)
    taps = (("seg", 1, np.int32), ("qkv", (hq + 2 * hkv) * dh, np.uint16), ("attn", hq * dh, np.uint16), ("hidden", 256, np.uint16))

    def read(eng, b):
        first = eng.rank(to_inputs(b))
        out = [eng.debug_read(n, (3, S + C, width), dt) for n, width, dt in taps + taps[-1:]]
        for _ in range(3):                                # replayed launches
            again = eng.rank(to_inputs(b))
        out += [eng.debug_read("hidden", (3, S + C, 256), np.uint16), eng.debug_read("hidden", (S + C + 1, 256), np.uint16)]
        np.testing.assert_array_equal(first.log_probs, again.log_probs)
        eng.close()
        return out

    ocfg, w, rows_fn, eng = make_pair(**kw)
    b = po.make_batch(ocfg, 3, seed=S, ragged=True)
    got = read(eng, b)
    monkeypatch.setenv("PHX_LAST_LAYER", "full")
    _, _, _, eng = make_pair(**kw)
    for a, c in zip(got, read(eng, b)):
        np.testing.assert_array_equal(a, c)


@pytest.mark.parametrize("B,S,C,hkv", [(8, 128, 512, 8), (13, 128, 500, 8), (5, 97, 512, 4), (18, 128, 257, 2)])
def test_fewer_items_than_sms_split_by_tiles(monkeypatch, B, S, C, hkv):
    """The resident-history kernel with fewer (batch, head) pairs than SMs and more query tiles: a CTA's share begins inside one
    item and runs into the next, in full layers and (the last one) without the history tile.  Ragged requests, against the
    mma.sync kernel and the oracle."""
    from x_algorithm_b200.engine import dispatch_counts
    assert B * 8 < 148 <= B * 8 * (1 + -(-C // 128))
    kw = dict(max_batch=B, emb_size=256, num_q_heads=8, num_kv_heads=hkv, key_size=64, history_len=S, num_candidates=C, num_layers=2)
    ocfg, w, rows_fn, eng = make_pair(**kw)
    b = po.make_batch(ocfg, B, seed=S + C, ragged=True)
    before = dispatch_counts()
    got = eng.rank(to_inputs(b))
    ran = {k: v - before[k] for k, v in dispatch_counts().items() if k.startswith("attn.") and v != before[k]}
    assert ran == {"attn.pingpong": 2}, ran
    monkeypatch.setenv("PHX_ATTN", "mma")
    other = eng.rank(to_inputs(b))
    eng.close()
    valid = b.cand_post_ids != 0
    for r in range(B):                                   # request by request: a mixed-up tile cannot hide in the sum
        v = valid[r]
        if v.any():
            assert rel_l2(logits_of(got.log_probs[r][v]), logits_of(other.log_probs[r][v])) < 1e-2, r
    few = slice(B // 2, B // 2 + 2)
    bb = po.RankBatch(*(getattr(b, f)[few] for f in ("hist_post_ids", "hist_author_ids", "hist_actions", "hist_surfaces", "cand_post_ids", "cand_author_ids")))
    lp, cont, logits = po.rank_forward(ocfg, w, rows_fn, bb)
    ok = bb.cand_post_ids != 0
    assert_heads_close(got.log_probs[few][ok], got.continuous[few][ok], logits[ok], cont[ok], 2e-2, str(kw))


@pytest.mark.parametrize("B,S,C,hq,hkv,kind", [(5, 65, 385, 8, 8, "pingpong"), (5, 64, 512, 8, 8, "stream"), (7, 20, 512, 8, 8, "stream"), (4, 65, 384, 8, 8, "stream"),
                                               (19, 64, 385, 8, 2, "pingpong"), (19, 64, 384, 8, 2, "strip"), (19, 65, 64, 8, 2, "pingpong"), (19, 65, 63, 8, 2, "strip"),
                                               (19, 30, 20, 8, 8, "pingpong")])
def test_which_kernel_takes_a_short_history(B, S, C, hq, hkv, kind):
    """Both sides of the lines between the resident-history tcgen05 kernel and the mma.sync kernels at head dim 64; in the
    candidate-only last layer as in the full one."""
    from x_algorithm_b200.engine import dispatch_counts
    kw = dict(max_batch=B, emb_size=128, num_q_heads=hq, num_kv_heads=hkv, key_size=64, history_len=S, num_candidates=C, num_layers=2)
    ocfg, w, rows_fn, eng = make_pair(**kw)
    b = po.make_batch(ocfg, B, seed=S + C)
    before = dispatch_counts()
    eng.rank(to_inputs(b))
    ran = {k: v - before[k] for k, v in dispatch_counts().items() if k.startswith("attn.") and v != before[k]}
    eng.close()
    assert ran == {"attn." + kind: 2}, ran
