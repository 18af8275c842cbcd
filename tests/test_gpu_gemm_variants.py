"""The GEMM variants a call's size picks - one tile per CTA for few tiles, resident A rows for many tiles with a short K - against
the single-CTA kernel, which multiplies and rounds in the same order: the same bits, at the edges of the 128-row and
64 / 128 / 256-column tiles and of the 64-column k-steps, and through the engine for the RoPE, RMSNorm and statistics epilogues."""
import numpy as np
import pytest

from helpers import make_pair, to_inputs
from oracle import phoenix_oracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 64, 64), (127, 72, 8), (129, 512, 2048), (640, 2048, 512), (640, 1536, 520), (1281, 1024, 256),
                                   (20001, 1024, 512), (38000, 512, 448), (19000, 2048, 72)])
@pytest.mark.parametrize("epi", [0, 1, 2])
def test_variants_give_the_same_bits(M, N, K, epi):
    import torch
    from x_algorithm_b200.engine import gemm
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = (torch.randn(M, K, device="cuda", generator=g) * 0.5).to(torch.bfloat16)
    wt = (torch.randn(N, K, device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    r = torch.randn(M, N, device="cuda", generator=g).to(torch.bfloat16) if epi == 1 else None
    c, _ = gemm(a, wt, r, epi, 0)
    one, _ = gemm(a, wt, r, epi, 2)
    assert torch.equal(c, one)


@pytest.mark.parametrize("B,opts", [(1, dict(history_len=31, num_candidates=70)), (5, dict(history_len=32, num_candidates=8)),
                                    (3, dict(emb_size=256, num_q_heads=4, num_kv_heads=2, key_size=64, history_len=40, num_candidates=150)),
                                    (2, dict(emb_size=256, num_q_heads=2, num_kv_heads=1, key_size=128, history_len=40, num_candidates=90)),
                                    (40, dict(emb_size=1024, num_q_heads=4, num_kv_heads=2, key_size=128, history_len=40, num_candidates=90, num_layers=1)),
                                    (90, dict(emb_size=256, num_q_heads=6, num_kv_heads=3, key_size=128, history_len=129, num_candidates=100, num_layers=1)),
                                    (64, dict(emb_size=512, num_q_heads=8, num_kv_heads=8, key_size=64, history_len=100, num_candidates=211, num_layers=1))])
def test_engine_forward_same_bits(monkeypatch, B, opts):
    ocfg, w, rows_fn, eng = make_pair(max_batch=B, **opts)
    b = po.make_batch(ocfg, B, seed=3, ragged=True)
    got = eng.rank(to_inputs(b)); eng.close()
    monkeypatch.setenv("PHX_GEMM", "cta1")
    _, _, _, eng = make_pair(max_batch=B, **opts)
    want = eng.rank(to_inputs(b)); eng.close()
    np.testing.assert_array_equal(got.log_probs, want.log_probs)
    np.testing.assert_array_equal(got.continuous, want.continuous)
