"""The streaming attention kernels at the edges of their key blocks and query tiles, and with every kind of row in every place, against a
plain fp32 reference: candidates whose tile is half padding, rows that attend to themselves inside the history, no history at all."""
import math

import pytest

pytestmark = pytest.mark.gpu


def reference(q, k, v, seg, S, scale, cap=lambda x: x):
    import torch
    q, k, v = q.float(), k.float(), v.float()
    g = q.shape[2] // k.shape[2]
    k, v = k.repeat_interleave(g, 2), v.repeat_interleave(g, 2)
    s = cap(torch.einsum("bqhd,bkhd->bhqk", q, k[:, :S]) * scale)
    s = s.masked_fill((seg[:, None, None, :S] != 1), -math.inf)
    own = cap((q * k).sum(-1) * scale).permute(0, 2, 1)[..., None].masked_fill((seg != -1)[:, None, :, None], -math.inf)
    p = torch.nan_to_num(torch.softmax(torch.cat((s, own), -1), -1))
    o = torch.einsum("bhqk,bkhd->bqhd", p[..., :S], v[:, :S]) + p[..., S:].permute(0, 2, 1, 3) * v
    return o * (seg != 0)[:, :, None, None]


@pytest.mark.parametrize("dh,H,Hk", [(128, 4, 2), (64, 4, 4)])
@pytest.mark.parametrize("S,C", [(0, 5), (0, 129), (1, 1), (63, 64), (64, 65), (65, 127), (127, 129), (129, 63), (192, 200), (193, 1), (257, 0), (1025, 130)])
def test_streaming_edges(monkeypatch, dh, H, Hk, S, C):
    import torch
    from x_algorithm_b200.engine import dispatch_counts, ranker_attention
    monkeypatch.setenv("PHX_ATTN", "tcgen05")
    B, T = 3, S + C
    g = torch.Generator(device="cuda").manual_seed(S * 131 + C)
    q, k, v = (torch.randn(B, T, h, dh, device="cuda", generator=g).to(torch.bfloat16) for h in (H, Hk, Hk))
    seg = torch.ones((B, T), dtype=torch.int32, device="cuda")
    seg[:, S:] = -1
    seg[1, S + C // 2:] = 0                       # half of the candidates are padding: whole halves of a tile without a self key
    seg[1, : S // 3] = 0
    seg[2, S // 2: S: 7] = -1                     # rows of the history that are no keys and attend to themselves
    before = dispatch_counts()["attn.tcgen05"]
    got, _ = ranker_attention(q, k, v, seg, S, 1.0 / math.sqrt(dh))
    assert dispatch_counts()["attn.tcgen05"] == before + 1
    want = reference(q, k, v, seg, S, 1.0 / math.sqrt(dh))
    assert bool((got[seg == 0] == 0).all())
    # P and the output are rounded to bf16 (2^-9 each, at most a row's largest |v| in all), scores are fp32 sums of exact products
    assert (got.float() - want).abs().max() <= 2.0 ** -7 * v.float().abs().max()
    assert torch.linalg.norm(got.float() - want) <= 2.0 ** -8 * torch.linalg.norm(want)


@pytest.mark.parametrize("dh,H,Hk", [(128, 8, 2), (64, 8, 8)])
@pytest.mark.parametrize("C", [128, 300, 520])
def test_no_history_rows_without_a_key_are_zero(monkeypatch, dh, H, Hk, C):
    """Without a history nothing but the staging itself waits for a tile's queries to land: whole tiles and warps of rows that are padding, or
    that have no key to attend to, read zero, never what their queries' copy leaves behind."""
    import torch
    from x_algorithm_b200.engine import dispatch_counts, ranker_attention
    monkeypatch.setenv("PHX_ATTN", "tcgen05")
    B = 64
    g = torch.Generator(device="cuda").manual_seed(C + dh)
    q, k, v = (torch.randn(B, C, h, dh, device="cuda", generator=g).to(torch.bfloat16) for h in (H, Hk, Hk))
    seg = torch.zeros((B, C), dtype=torch.int32, device="cuda")            # requests 0, 4, ...: padding alone
    seg[1::4] = 1                                                          # no key, and not their own
    seg[2::4, : C // 3] = -1                                               # then padding, from within a warp's rows on
    seg[3::4, 96:97] = -1                                                  # one row of one warp
    before = dispatch_counts()["attn.tcgen05"]
    for _ in range(5):
        got, _ = ranker_attention(q, k, v, seg, 0, 1.0 / math.sqrt(dh))
        own = v.repeat_interleave(H // Hk, 2) * (seg == -1)[:, :, None, None]      # a row that sees itself alone is its own v
        assert torch.equal(got, own)
    assert dispatch_counts()["attn.tcgen05"] == before + 5


# tiles of 64 / 128 rows on 148 SMs: heads of 128 have one CTA an SM at either height, heads of 64 two
@pytest.mark.parametrize("dh,H,Hk,B,S,C,low", [
    (128, 16, 4, 1, 512, 64, True),      # 144 / 80: one round of either
    (128, 16, 4, 1, 512, 65, False),     # 160 / 80: two rounds against one
    (128, 16, 4, 1, 1022, 64, False),    # 272 / 144
    (128, 8, 2, 5, 300, 148, True),      # 280 / 160: two rounds of either
    (128, 8, 2, 5, 300, 213, False),     # 360 / 200: more than two for every SM
    (64, 8, 8, 1, 257, 2111, True),      # 296 / 152: two low tiles an SM
    (64, 8, 8, 1, 257, 2112, False),     # 304 / 152
    (32, 4, 4, 2, 70, 2223, True)])      # 288 / 144
def test_rows_of_a_tile_follow_the_rounds(monkeypatch, dh, H, Hk, B, S, C, low):
    """The mma.sync kernel's tile height, on both sides of the rule that picks it."""
    import torch
    from x_algorithm_b200.engine import dispatch_counts, ranker_attention
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the tile counts are for 148 SMs")
    monkeypatch.setenv("PHX_ATTN", "mma")
    T = S + C
    g = torch.Generator(device="cuda").manual_seed(T)
    q, k, v = (torch.randn(B, T, h, dh, device="cuda", generator=g).to(torch.bfloat16) for h in (H, Hk, Hk))
    seg = torch.ones((B, T), dtype=torch.int32, device="cuda")
    seg[:, S:] = -1
    seg[:, S - 5: S] = 0
    seg[0, S + C // 2:] = 0
    before = dispatch_counts()
    got, _ = ranker_attention(q, k, v, seg, S, 1.0 / math.sqrt(dh))
    after = dispatch_counts()
    assert after["attn.stream"] == before["attn.stream"] + 1
    assert after["form.attn_low"] == before["form.attn_low"] + (1 if low else 0)
    want = reference(q, k, v, seg, S, 1.0 / math.sqrt(dh))
    assert bool((got[seg == 0] == 0).all())
    assert (got.float() - want).abs().max() <= 2.0 ** -7 * v.float().abs().max()          # as above
    assert torch.linalg.norm(got.float() - want) <= 2.0 ** -8 * torch.linalg.norm(want)


@pytest.mark.parametrize("method", [1, 2])
@pytest.mark.parametrize("dh,H,Hk", [(128, 4, 2), (64, 4, 4)])
@pytest.mark.parametrize("S,C", [(0, 70), (63, 64), (129, 63), (192, 200), (330, 5)])
def test_streaming_with_capped_logits(monkeypatch, S, C, dh, H, Hk, method):
    """Soft sign and tanh at a cap that the larger logits feel, whole and half blocks of keys."""
    import torch
    from x_algorithm_b200.engine import dispatch_counts, ranker_attention
    monkeypatch.setenv("PHX_ATTN", "tcgen05")
    B, T, cap = 2, S + C, 2.0
    g = torch.Generator(device="cuda").manual_seed(S * 131 + C)
    q, k, v = (torch.randn(B, T, h, dh, device="cuda", generator=g).to(torch.bfloat16) for h in (H, Hk, Hk))
    seg = torch.ones((B, T), dtype=torch.int32, device="cuda")
    seg[:, S:] = -1
    seg[1, S // 2: S // 2 + 9] = 0
    before = dispatch_counts()["attn.tcgen05"]
    got, _ = ranker_attention(q, k, v, seg, S, 1.0 / math.sqrt(dh), cap, method)
    assert dispatch_counts()["attn.tcgen05"] == before + 1
    capped = (lambda x: x / (1 + x.abs() / cap)) if method == 1 else (lambda x: cap * torch.tanh(x / cap))
    want = reference(q, k, v, seg, S, 1.0 / math.sqrt(dh), capped)
    assert (got.float() - want).abs().max() <= 2.0 ** -7 * v.float().abs().max()          # as without a cap: the logits stay fp32
    assert torch.linalg.norm(got.float() - want) <= 2.0 ** -8 * torch.linalg.norm(want)


@pytest.mark.parametrize("impl,dh,H,Hk,B,S,C", [
    ("mma", 32, 4, 2, 3, 105, 20), ("mma", 64, 8, 8, 1, 223, 349), ("mma", 128, 4, 1, 2, 300, 40), ("mma", 64, 8, 8, 40, 200, 300), ("mma", 64, 2, 2, 2, 90, 0),
    ("strip", 64, 8, 2, 8, 17, 173), ("strip", 64, 4, 4, 40, 120, 15), ("strip", 64, 4, 1, 25, 128, 428), ("pingpong", 64, 8, 8, 26, 96, 374),
    ("pingpong", 64, 8, 8, 20, 128, 130), ("pingpong", 64, 8, 2, 20, 40, 0), ("resident", 64, 4, 4, 3, 100, 200), ("tcgen05", 64, 8, 8, 2, 200, 60),
    ("tcgen05", 128, 8, 2, 2, 70, 60)])
def test_history_rows_marked_as_candidates_attend_to_themselves(monkeypatch, impl, dh, H, Hk, B, S, C):
    """allowed(q, k) = history key, or the row itself (ranker_attention_utils.py:16-56): also for rows in front of the candidates, whatever tile or
    strip they share, in every kernel."""
    import torch
    from x_algorithm_b200.engine import ranker_attention
    monkeypatch.setenv("PHX_ATTN", impl)
    g = torch.Generator(device="cuda").manual_seed(S * 131 + C)
    T = S + C
    q, k, v = (torch.randn(B, T, h, dh, device="cuda", generator=g).to(torch.bfloat16) for h in (H, Hk, Hk))
    seg = torch.ones((B, T), dtype=torch.int32, device="cuda")
    seg[:, S:] = -1
    r = torch.rand((B, T), device="cuda", generator=g)
    seg[r < 0.3] = 0
    seg[r > 0.9] = -1
    got, _ = ranker_attention(q, k, v, seg, S, 1.0 / math.sqrt(dh))
    want = reference(q, k, v, seg, S, 1.0 / math.sqrt(dh))
    assert bool((got[seg == 0] == 0).all())
    assert (got.float() - want).abs().max() <= 2.0 ** -7 * v.float().abs().max()          # as above
    assert torch.linalg.norm(got.float() - want) <= 2.0 ** -8 * torch.linalg.norm(want)
