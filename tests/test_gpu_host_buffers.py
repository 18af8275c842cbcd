"""Host-buffer ranking calls on both sides of the size up to which the device writes its results to pinned memory itself: the same bits as
the same batch from device buffers, call after call on one engine, with other data in between, packed and not."""
import numpy as np
import pytest

from helpers import make_pair, to_inputs
from oracle import phoenix_oracle as po

pytestmark = pytest.mark.gpu


# bytes in and out at the largest batch: 0.01 / 0.01 MB, 0.4 / 0.5, 0.5 / 1.7 (results copied), 0.55 / 0.1, 1.4 / 5.3 (copied)
@pytest.mark.parametrize("B,S,C", [(3, 32, 8), (40, 120, 140), (200, 32, 100), (110, 200, 10), (250, 64, 240)])
@pytest.mark.parametrize("pack", [False, True])
def test_host_buffers_same_bits_as_device_buffers(B, S, C, pack):
    import torch
    import x_algorithm_b200 as px
    from x_algorithm_b200.engine import plan_ragged
    ocfg, w, rows_fn, eng = make_pair(max_batch=B, history_len=S, num_candidates=C, engine_kw=dict(pack_ragged=pack))
    bw = po.make_blend_weights(1)
    eng.set_blend(px.blend_spec_from_weights(px.ValueModelWeights(w=dict(bw.w)), px.HEAD_NAMES_19, ocfg.num_actions))
    for n, seed in ((B, 3), (max(1, B // 3), 4), (B, 5), (B, 5)):          # the last one replays a graph
        b = po.make_batch(ocfg, n, seed=seed, ragged=True)
        if pack:
            b.cand_post_ids[n // 2] = 0                                    # a request without candidates
            b.cand_author_ids[n // 2] = 0
        got = eng.rank(to_inputs(b))
        d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in
             (b.hist_post_ids, b.hist_author_ids, b.hist_actions, b.hist_surfaces, b.cand_post_ids, b.cand_author_ids)]
        lp = torch.full((n, C, ocfg.num_actions), 7.0, device="cuda")
        co = torch.full((n, C, ocfg.num_continuous), 7.0, device="cuda")
        sc = torch.full((n, C), 7.0, dtype=torch.float64, device="cuda")
        if pack:
            ho, cc = plan_ragged(b.hist_post_ids, b.cand_post_ids)
            eng.rank_packed_device(n, *d, torch.from_numpy(ho).cuda(), torch.from_numpy(cc).cuda(), int(ho[-1]), int(cc[-1]), lp, co, sc)
        else:
            eng.rank_device(n, *d, lp, co, sc)
        eng.sync()
        np.testing.assert_array_equal(got.log_probs, lp.cpu().numpy())
        np.testing.assert_array_equal(got.continuous, co.cpu().numpy())
        np.testing.assert_array_equal(got.scores, sc.cpu().numpy())
    eng.close()
