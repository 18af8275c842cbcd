"""Small calls on tiles of 64 rows (long K, few of them): the same bits as the single-CTA kernel at the edges of the 64-row and 64-column
tiles and of the ring, on both sides of the rule that picks them."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 16, 63, 64, 65, 127, 129, 640])
@pytest.mark.parametrize("N,K", [(64, 512), (72, 520), (512, 768), (192, 776), (512, 2048), (512, 504)])
@pytest.mark.parametrize("epi", [0, 1, 2])
def test_low_tiles_give_the_same_bits(M, N, K, epi):
    import torch
    from x_algorithm_b200.engine import dispatch_counts, gemm
    g = torch.Generator(device="cuda").manual_seed(M + 3 * N + K)
    a = (torch.randn(M, K, device="cuda", generator=g) * 0.5).to(torch.bfloat16)
    wt = (torch.randn(N, K, device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    r = torch.randn(M, N, device="cuda", generator=g).to(torch.bfloat16) if epi == 1 else None
    before = dispatch_counts()["gemm.small"]
    got, _ = gemm(a, wt, r, epi, 0)
    assert dispatch_counts()["gemm.small"] == before + 1
    want, _ = gemm(a, wt, r, epi, 2)
    assert torch.equal(got, want)


@pytest.mark.parametrize("B,S,C,D", [(1, 20, 43, 512), (1, 30, 35, 512), (2, 64, 129, 512), (3, 100, 60, 1024)])
def test_low_tiles_in_the_engine(monkeypatch, B, S, C, D):
    """The RoPE, norm and statistics epilogues on tiles of 64 rows: a forward's bits are those of the single-CTA kernel's."""
    import numpy as np
    from helpers import make_pair, to_inputs
    from oracle import phoenix_oracle as po
    out = []
    for mode in (None, "cta1"):
        if mode:
            monkeypatch.setenv("PHX_GEMM", mode)
        ocfg, w, rows_fn, eng = make_pair(max_batch=B, emb_size=D, num_layers=2, num_q_heads=D // 64, num_kv_heads=D // 64, key_size=64,
                                          history_len=S, num_candidates=C)
        out.append(eng.rank(to_inputs(po.make_batch(ocfg, B, seed=3, ragged=True))))
        eng.close()
    np.testing.assert_array_equal(out[0].log_probs, out[1].log_probs)
    np.testing.assert_array_equal(out[0].continuous, out[1].continuous)
