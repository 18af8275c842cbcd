"""History rows of a candidate-only layer go through the QKV projection for their keys and values alone where whole column tiles hold nothing
but query heads: the same results as with every tile, at row counts around the 256-row tiles, split and packed rows.  A debug read still finds
every query row."""
import numpy as np
import pytest

from helpers import make_pair, to_inputs
from oracle import phoenix_oracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hq,hkv", [(8, 2), (8, 4), (4, 4), (6, 1)])
@pytest.mark.parametrize("B,S,C,tail,pack", [(20, 300, 40, 1, False), (32, 256, 20, 2, False), (21, 257, 33, 0, False), (24, 300, 40, 1, True)])
def test_unread_query_tiles_change_nothing(monkeypatch, hq, hkv, B, S, C, tail, pack):
    kw = dict(max_batch=B, emb_size=256, num_layers=2, num_q_heads=hq, num_kv_heads=hkv, key_size=128, history_len=S, num_candidates=C,
              num_candidate_only_layers=tail, engine_kw=dict(pack_ragged=pack))
    from x_algorithm_b200.engine import dispatch_counts
    out = []
    for mode in (None, "cta1"):                       # the single-CTA kernel works on every tile
        if mode:
            monkeypatch.setenv("PHX_GEMM", mode)
        ocfg, w, rows_fn, eng = make_pair(**kw)
        before = dispatch_counts()["form.gemm_kv_only"]
        for seed in (8, 9):                           # the second call meets the buffers of the first
            got = eng.rank(to_inputs(po.make_batch(ocfg, B, seed=seed, ragged=True)))
        # a key head's own query head (4, 4) is half a column tile: nothing to leave out
        left_out = 0 if mode or hq == hkv else 2 * max(tail, 1)
        assert dispatch_counts()["form.gemm_kv_only"] == before + left_out
        out.append(got)
        eng.close()
    assert np.isfinite(out[0].log_probs).all()
    np.testing.assert_array_equal(out[0].log_probs, out[1].log_probs)
    np.testing.assert_array_equal(out[0].continuous, out[1].continuous)


@pytest.mark.parametrize("primer", [False, True])
@pytest.mark.parametrize("tail,pack", [(0, False), (1, False), (2, False), (0, True)])
def test_debug_reads_find_every_query_row(monkeypatch, tail, pack, primer):
    from x_algorithm_b200.engine import plan_ragged
    B, S, C, hq, hkv = 21, 257, 33, 8, 2
    kw = dict(max_batch=B, emb_size=256, num_layers=3, num_q_heads=hq, num_kv_heads=hkv, key_size=128, history_len=S, num_candidates=C,
              num_candidate_only_layers=tail, primer_norm=primer, engine_kw=dict(pack_ragged=pack))
    out = []
    for mode in (None, "cta1"):
        if mode:
            monkeypatch.setenv("PHX_GEMM", mode)
        ocfg, w, rows_fn, eng = make_pair(**kw)
        taps = []
        for seed in (8, 9, 9, 9):                     # the last one replays a graph
            b = po.make_batch(ocfg, B, seed=seed, ragged=True)
            eng.rank(to_inputs(b))
            rows = B * (S + C)
            if pack:
                ho, cc = plan_ragged(b.hist_post_ids, b.cand_post_ids)
                rows = int(ho[-1]) + int(cc[-1])
            first = eng.debug_read("qkv", (rows, (hq + 2 * hkv) * 128), np.uint16) if seed == 9 else None
            if tail == 0 and not pack:                # every row is taken through the last layer, in [B, T] order
                taps += [eng.debug_read("hidden", (rows, 256), np.uint16), eng.debug_read("attn", (rows, hq * 128), np.uint16)]
            taps.append(eng.debug_read("qkv", (rows, (hq + 2 * hkv) * 128), np.uint16))
            if first is not None:
                np.testing.assert_array_equal(first, taps[-1])
        out.append(taps)
        eng.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
