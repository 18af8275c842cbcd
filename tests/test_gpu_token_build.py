"""The plain token build takes 1, 2, 4 or 8 tokens a warp by the call's size; with debug taps the general kernel builds the tokens,
one a warp.  Same sums and roundings: the forwards agree bit for bit, at sizes that leave a partly filled warp, widths that leave
a partly filled 256-column step, every hash count, and packed rows.  The tower's pooling with rows in shared memory and without
against the oracle, and both heads kernels against each other."""
import numpy as np
import pytest

from helpers import assert_heads_close, make_pair, rel_l2, to_inputs
from oracle import phoenix_oracle as po

pytestmark = pytest.mark.gpu
TOL = 2e-2        # bf16 trunk against the oracle: the bound of the other parity tests


@pytest.mark.parametrize("B,S,C,D,H,pack", [
    (1, 9, 5, 128, 2, False), (3, 33, 40, 576, 1, False), (2, 33, 500, 1024, 4, False), (7, 33, 100, 320, 3, True),
    (31, 33, 100, 128, 2, False), (31, 33, 100, 320, 4, True),                       # 4123 tokens: two a warp
    (63, 33, 98, 576, 2, True), (63, 33, 98, 64, 3, False), (63, 33, 98, 256, 1, False),   # 8253: four
    (251, 33, 98, 128, 2, False), (251, 33, 98, 192, 1, True), (251, 33, 98, 64, 4, False)])  # 32881: eight (four of 3-4 hashes)
def test_tokens_a_warp(monkeypatch, B, S, C, D, H, pack):
    kw = dict(max_batch=B, emb_size=D, num_layers=1, num_q_heads=2, num_kv_heads=2, key_size=32, history_len=S, num_candidates=C, num_hashes=H,
              engine_kw=dict(pack_ragged=pack))
    ocfg, w, rows_fn, eng = make_pair(**kw)
    b = po.make_batch(ocfg, B, seed=5, ragged=True)
    got = eng.rank(to_inputs(b))
    eng.close()
    monkeypatch.setenv("PHX_DEBUG_TAPS", "1")
    _, _, _, eng = make_pair(**kw)
    want = eng.rank(to_inputs(b))
    eng.close()
    np.testing.assert_array_equal(got.log_probs, want.log_probs)
    np.testing.assert_array_equal(got.continuous, want.continuous)


@pytest.mark.parametrize("D", [2048, 2112, 2432])
@pytest.mark.parametrize("build", ["plain", "general", "project"])
def test_rows_with_more_than_32_statistics(monkeypatch, D, build):
    """A row's sum of squares goes to slot 0 of D / 64 and the others to zero, all of them: what the forward before left in a slot (the sums of its
    last layer) is no part of the next one's first norm."""
    if build == "general":
        monkeypatch.setenv("PHX_DEBUG_TAPS", "1")
    kw = dict(token_combine="project") if build == "project" else {}
    ocfg, w, rows_fn, eng = make_pair(max_batch=6, emb_size=D, num_layers=1, num_q_heads=2, num_kv_heads=2, key_size=32, history_len=9,
                                      num_candidates=20, **kw)
    a, b = (po.make_batch(ocfg, n, seed=n, ragged=True) for n in (4, 6))
    first = eng.rank(to_inputs(a))
    eng.rank(to_inputs(b))
    again = eng.rank(to_inputs(a))
    np.testing.assert_array_equal(again.log_probs, first.log_probs)
    np.testing.assert_array_equal(again.continuous, first.continuous)
    lp, cont, logits = po.rank_forward(ocfg, w, rows_fn, a)
    valid = a.cand_post_ids != 0
    assert_heads_close(again.log_probs[valid], again.continuous[valid], logits[valid], cont[valid], tol=TOL)
    eng.close()


@pytest.mark.parametrize("S,D,B", [(140, 256, 3), (144, 256, 3), (33, 128, 5), (200, 256, 2)])   # 72 KB of rows and statistics: 142 x 256
def test_pooling_keeps_rows_where_they_fit(S, D, B):
    import torch
    ocfg, w, rows_fn, eng = make_pair(max_batch=B, emb_size=D, num_candidates=0, history_len=S, num_layers=1)
    b = po.make_batch(po.ModelConfig(history_len=S, num_candidates=1), B, seed=5, ragged=True)
    want = po.user_tower(ocfg, w, rows_fn, b)
    users = torch.empty((B, D), dtype=torch.float32, device="cuda")
    dev = [torch.from_numpy(a).cuda() for a in (b.hist_post_ids, b.hist_author_ids, b.hist_actions, b.hist_surfaces)]
    eng.user_tower_device(B, *dev, users)
    eng.sync()
    eng.close()
    ok = b.hist_post_ids[:, 0] != 0
    assert rel_l2(users.cpu().numpy()[ok], want[ok]) < TOL


@pytest.mark.parametrize("D,actions", [(128, 19), (1024, 19), (1664, 30), (2048, 30)])    # the last: too wide for the rows to be staged
def test_heads_with_and_without_staged_rows(D, actions):
    """296 strips of 16 candidates take eight warps a strip with its rows in shared memory, 297 a warp a strip: the same bits."""
    kw = dict(emb_size=D, num_layers=1, num_q_heads=2, num_kv_heads=2, key_size=64, history_len=9, num_candidates=16, num_actions=actions,
              widening_factor=1.0)
    ocfg, w, rows_fn, eng = make_pair(max_batch=297, **kw)
    b = po.make_batch(ocfg, 297, seed=5, ragged=True)
    whole = eng.rank(to_inputs(b))
    part = type(b)(*[np.ascontiguousarray(a[:296]) for a in (b.hist_post_ids, b.hist_author_ids, b.hist_actions, b.hist_surfaces,
                                                            b.cand_post_ids, b.cand_author_ids)])
    some = eng.rank(to_inputs(part))
    eng.close()
    np.testing.assert_array_equal(some.log_probs, whole.log_probs[:296])
    np.testing.assert_array_equal(some.continuous, whole.continuous[:296])


@pytest.mark.parametrize("C", [30, 700])                 # results in one copy; in row chunks
def test_packed_results_are_laid_out_by_the_host(C):
    """Packed calls bring back the valid rows alone: every slot without a candidate reads zero whatever the caller's arrays held, and
    a request's results do not depend on the others' counts (none, one, all of its slots)."""
    import x_algorithm_b200 as px
    B, S = 41, 9
    ocfg, w, rows_fn, eng = make_pair(max_batch=B, emb_size=128, num_layers=1, num_q_heads=2, num_kv_heads=2, key_size=64, history_len=S,
                                      num_candidates=C, engine_kw=dict(pack_ragged=True))
    eng.set_blend(px.blend_spec_from_weights(px.ValueModelWeights(w=dict(po.make_blend_weights(1).w)), px.HEAD_NAMES_19, ocfg.num_actions))
    b = po.make_batch(ocfg, B, seed=5, ragged=True)
    for q, n in ((0, 0), (1, 1), (2, C), (17, 0), (B - 1, 0)):
        b.cand_post_ids[q, :], b.cand_author_ids[q, :] = 7, 9
        b.cand_post_ids[q, n:], b.cand_author_ids[q, n:] = 0, 0
    out = px.RankOutputs(np.full((B, C, ocfg.num_actions), np.nan, np.float32), np.full((B, C, ocfg.num_continuous), np.nan, np.float32),
                         np.full((B, C), np.nan))
    got = eng.rank(to_inputs(b), out)
    names = ("hist_post_ids", "hist_author_ids", "hist_actions", "hist_surfaces", "cand_post_ids", "cand_author_ids")
    for q in range(B):
        one = eng.rank(to_inputs(type(b)(*[np.ascontiguousarray(getattr(b, f)[q:q + 1]) for f in names])))
        n = int((b.cand_post_ids[q] != 0).sum())
        for a, o in ((got.log_probs, one.log_probs), (got.continuous, one.continuous), (got.scores, one.scores)):
            np.testing.assert_array_equal(a[q], o[0])
            assert not np.any(a[q, n:])
    eng.close()


@pytest.mark.parametrize("D,actions", [(1024, 29), (1280, 19), (1536, 19)])
def test_heads_at_one_and_two_strips_an_sm(D, actions):
    """Wide rows: their strips in shared memory while one CTA an SM holds them all (148 strips of 16), four warps a strip up to
    twice that, a warp a strip beyond: the same bits."""
    kw = dict(emb_size=D, num_layers=1, num_q_heads=2, num_kv_heads=2, key_size=64, history_len=9, num_candidates=16, num_actions=actions,
              widening_factor=1.0)
    ocfg, w, rows_fn, eng = make_pair(max_batch=297, **kw)
    b = po.make_batch(ocfg, 297, seed=5, ragged=True)
    whole = eng.rank(to_inputs(b))
    for n in (148, 149, 296):
        part = type(b)(*[np.ascontiguousarray(a[:n]) for a in (b.hist_post_ids, b.hist_author_ids, b.hist_actions, b.hist_surfaces,
                                                               b.cand_post_ids, b.cand_author_ids)])
        some = eng.rank(to_inputs(part))
        np.testing.assert_array_equal(some.log_probs, whole.log_probs[:n])
        np.testing.assert_array_equal(some.continuous, whole.continuous[:n])
    eng.close()


@pytest.mark.parametrize("compute,S,D", [("bf16", 142, 256), ("fp32", 71, 256)])     # the most rows of 512 / 1024 bytes that fit
def test_pooling_bits_with_rows_in_shared_memory_and_without(compute, S, D):
    """One history slot more moves the pooling from rows in shared memory to rows in global memory: users whose last slots are padding
    come out the same to the bit from both."""
    import torch
    B, n = 3, S - 2
    users = []
    for slots in (S, S + 1):
        ocfg, w, rows_fn, eng = make_pair(max_batch=B, emb_size=D, num_q_heads=2, num_kv_heads=2, key_size=32, num_candidates=0,
                                          history_len=slots, num_layers=1, compute=compute)
        b = po.make_batch(po.ModelConfig(history_len=n, num_candidates=1), B, seed=5, ragged=True)
        dev = []
        for a in (b.hist_post_ids, b.hist_author_ids, b.hist_actions, b.hist_surfaces):
            wide = np.zeros((B, slots), a.dtype)
            wide[:, :n] = a
            dev.append(torch.from_numpy(wide).cuda())
        out = torch.empty((B, D), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        eng.user_tower_device(B, *dev, out)
        eng.sync()
        eng.close()
        users.append(out.cpu().numpy())
    assert np.isfinite(users[0]).all() and np.abs(users[0]).max() > 0
    np.testing.assert_array_equal(users[0], users[1])


@pytest.mark.parametrize("S,D", [(9, 256), (71, 256), (72, 256)])
def test_pooling_of_fp32_rows(S, D):
    """The full-precision tower against the oracle's: fp32 sums in another order through one layer, bound of the fp32 parity tests."""
    import torch
    B = 3
    ocfg, w, rows_fn, eng = make_pair(max_batch=B, emb_size=D, num_candidates=0, history_len=S, num_layers=1, compute="fp32")
    b = po.make_batch(po.ModelConfig(history_len=S, num_candidates=1), B, seed=5, ragged=True)
    want = po.user_tower(ocfg, w, rows_fn, b)
    users = torch.empty((B, D), dtype=torch.float32, device="cuda")
    dev = [torch.from_numpy(a).cuda() for a in (b.hist_post_ids, b.hist_author_ids, b.hist_actions, b.hist_surfaces)]
    eng.user_tower_device(B, *dev, users)
    eng.sync()
    eng.close()
    ok = b.hist_post_ids[:, 0] != 0
    assert rel_l2(users.cpu().numpy()[ok], want[ok]) < 1e-5


@pytest.mark.parametrize("C", [30, 700])
def test_packed_batch_without_any_candidate(C):
    """No request has a candidate: nothing comes back, every slot reads zero, and the engine's next call is an ordinary one."""
    import x_algorithm_b200 as px
    B, S = 3, 9
    ocfg, w, rows_fn, eng = make_pair(max_batch=B, emb_size=128, num_layers=2, num_q_heads=2, num_kv_heads=2, key_size=64, history_len=S,
                                      num_candidates=C, engine_kw=dict(pack_ragged=True))
    eng.set_blend(px.blend_spec_from_weights(px.ValueModelWeights(w=dict(po.make_blend_weights(1).w)), px.HEAD_NAMES_19, ocfg.num_actions))
    b = po.make_batch(ocfg, B, seed=5, ragged=True)
    want = eng.rank(to_inputs(b))
    want_lp, want_s = want.log_probs.copy(), want.scores.copy()
    posts, authors = b.cand_post_ids.copy(), b.cand_author_ids.copy()
    b.cand_post_ids[:], b.cand_author_ids[:] = 0, 0
    out = px.RankOutputs(np.full((B, C, ocfg.num_actions), np.nan, np.float32), np.full((B, C, ocfg.num_continuous), np.nan, np.float32),
                         np.full((B, C), np.nan))
    got = eng.rank(to_inputs(b), out)
    assert not got.log_probs.any() and not got.continuous.any() and not got.scores.any()
    b.cand_post_ids[:], b.cand_author_ids[:] = posts, authors
    again = eng.rank(to_inputs(b))
    eng.close()
    assert np.any(want_lp)
    np.testing.assert_array_equal(again.log_probs, want_lp)
    np.testing.assert_array_equal(again.scores, want_s)
