"""Small calls on tiles of 64 rows (long K, few of them) and with the deep ring: the same bits as the single-CTA kernel at the edges of the 64-row and
64-column tiles and of the ring, on both sides of the rules that pick them."""
import pytest

pytestmark = pytest.mark.gpu
FORMS = ("gemm.small", "form.gemm_low", "form.gemm_deep")


def forms_since(before):
    from x_algorithm_b200.engine import dispatch_counts
    now = dispatch_counts()
    return tuple(now[f] - before[f] for f in FORMS)


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
    before = dispatch_counts()
    got, _ = gemm(a, wt, r, epi, 0)
    assert forms_since(before) == ((1, 1, 0) if K >= 512 else (1, 0, 0))       # at most 10 x 8 tiles of 64 x 64
    want, _ = gemm(a, wt, r, epi, 2)
    assert torch.equal(got, want)


@pytest.mark.parametrize("M,N,K,epi,form", [
    (1152, 512, 512, 0, "low"), (1153, 512, 512, 0, "deep"),                  # 144 / 152 tiles of 64 x 64
    (1536, 512, 512, 0, "deep"), (1537, 512, 512, 0, "shallow"),              # 96 / 104 tiles of 128 x 64: two thirds of the SMs
    (1537, 512, 512, 1, "deep"), (1537, 512, 504, 1, "shallow"), (1537, 512, 1016, 2, "shallow"), (1537, 512, 1024, 2, "deep"),
    (3072, 512, 512, 2, "deep"), (3200, 512, 512, 2, "shallow"), (4096, 512, 1024, 0, "deep")])       # 96, 100, 128 tiles of 128 x 128
def test_form_of_a_small_call(M, N, K, epi, form):
    import torch
    from x_algorithm_b200.engine import dispatch_counts, gemm
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the tile counts are for 148 SMs")
    g = torch.Generator(device="cuda").manual_seed(M + K)
    a = (torch.randn(M, K, device="cuda", generator=g) * 0.5).to(torch.bfloat16)
    wt = (torch.randn(N, K, device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    r = torch.randn(M, N, device="cuda", generator=g).to(torch.bfloat16) if epi == 1 else None
    before = dispatch_counts()
    got, _ = gemm(a, wt, r, epi, 0)
    assert forms_since(before) == (1, form == "low", form == "deep")
    want, _ = gemm(a, wt, r, epi, 2)
    assert torch.equal(got, want)


@pytest.mark.parametrize("B,S,C,D", [(1, 20, 43, 512), (1, 30, 35, 512), (2, 64, 129, 512), (3, 100, 60, 1024)])
def test_low_tiles_in_the_engine(monkeypatch, B, S, C, D):
    """The RoPE, norm and statistics epilogues on tiles of 64 rows: a forward's bits are those of the single-CTA kernel's."""
    import numpy as np
    from helpers import make_pair, to_inputs
    from oracle import phoenix_oracle as po
    from x_algorithm_b200.engine import dispatch_counts
    out = []
    for mode in (None, "cta1"):
        if mode:
            monkeypatch.setenv("PHX_GEMM", mode)
        ocfg, w, rows_fn, eng = make_pair(max_batch=B, emb_size=D, num_layers=2, num_q_heads=D // 64, num_kv_heads=D // 64, key_size=64,
                                          history_len=S, num_candidates=C)
        before = dispatch_counts()
        out.append(eng.rank(to_inputs(po.make_batch(ocfg, B, seed=3, ragged=True))))
        small, low, _ = forms_since(before)
        assert (small == low == 0) if mode else (small >= low > 0)
        eng.close()
    np.testing.assert_array_equal(out[0].log_probs, out[1].log_probs)
    np.testing.assert_array_equal(out[0].continuous, out[1].continuous)


def test_low_tiles_follow_the_rows_and_the_buffers():
    """Calls of several sizes on one engine, some from the buffers that a prefetch has filled: the 64-row tiles read the rows of the call."""
    import numpy as np
    import torch
    from helpers import make_pair
    from oracle import phoenix_oracle as po
    from x_algorithm_b200.engine import dispatch_counts
    C, dev = 43, {}
    ocfg, w, rows_fn, eng = make_pair(max_batch=4, emb_size=512, num_layers=2, num_q_heads=8, num_kv_heads=8, key_size=64, history_len=20,
                                      num_candidates=C)
    _, _, _, plain = make_pair(max_batch=4, emb_size=512, num_layers=2, num_q_heads=8, num_kv_heads=8, key_size=64, history_len=20,
                               num_candidates=C)
    for B in (1, 3, 4):
        b = po.make_batch(ocfg, B, seed=B, ragged=True)
        dev[B] = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in
                  (b.hist_post_ids, b.hist_author_ids, b.hist_actions, b.hist_surfaces, b.cand_post_ids, b.cand_author_ids)]

    def forward(e, B):
        lp, co = torch.empty((B, C, ocfg.num_actions), device="cuda"), torch.empty((B, C, ocfg.num_continuous), device="cuda")
        e.rank_device(B, *dev[B], lp, co)
        return lp, co

    sizes = (4, 1, 3, 3, 1, 4)
    before = dispatch_counts()
    got = []
    for i, B in enumerate(sizes):
        got.append(forward(eng, B))
        if i + 1 < len(sizes) and i % 2 == 0:
            eng.rank_prefetch_device(sizes[i + 1], *dev[sizes[i + 1]])
    eng.sync()
    assert forms_since(before)[1] >= len(sizes)
    for B, (lp, co) in zip(sizes, got):
        want = forward(plain, B)
        plain.sync()
        assert torch.equal(lp, want[0]) and torch.equal(co, want[1])
    eng.close()
    plain.close()
