"""History rows of a candidate-only layer go through the QKV projection for their keys and values alone where whole column tiles hold nothing
but query heads: the same results as with every tile, at row counts around the 256-row tiles, split and packed rows."""
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
    out = []
    for mode in (None, "cta1"):                       # the single-CTA kernel works on every tile
        if mode:
            monkeypatch.setenv("PHX_GEMM", mode)
        ocfg, w, rows_fn, eng = make_pair(**kw)
        for seed in (8, 9):                           # the second call meets the buffers of the first
            got = eng.rank(to_inputs(po.make_batch(ocfg, B, seed=seed, ragged=True)))
        out.append(got)
        eng.close()
    assert np.isfinite(out[0].log_probs).all()
    np.testing.assert_array_equal(out[0].log_probs, out[1].log_probs)
    np.testing.assert_array_equal(out[0].continuous, out[1].continuous)
