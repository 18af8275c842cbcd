"""The heads kernels that a call's number of candidate rows picks: the same bits for the same rows, whole strips of 16 and partial ones, with
one to 32 outputs, and at widths where a strip's rows no longer stand beside the head matrix."""
import numpy as np
import pytest

from helpers import make_pair, take_requests, to_inputs
from oracle import phoenix_oracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opts,B,C", [(dict(), 240, 31), (dict(num_actions=7), 160, 47), (dict(num_actions=14, num_continuous=2), 500, 17),
                                      (dict(num_actions=30, num_continuous=2), 240, 32),
                                      (dict(emb_size=2432, num_q_heads=2, num_kv_heads=2, key_size=32), 150, 33)])
def test_heads_same_bits_for_any_number_of_rows(opts, B, C):
    """More strips than the small calls' kernel takes, against the same requests a few at a time."""
    assert B * C > 3 * 148 * 16 or "emb_size" in opts
    ocfg, w, rows_fn, eng = make_pair(max_batch=B, num_layers=1, history_len=9, num_candidates=C, **opts)
    b = po.make_batch(ocfg, B, seed=6, ragged=True)
    whole = eng.rank(to_inputs(b))
    for first, n in ((0, 1), (3, 2), (B - 7, 7), (5, 100)):
        part = eng.rank(to_inputs(take_requests(b, list(range(first, first + n)))))
        np.testing.assert_array_equal(part.log_probs, whole.log_probs[first:first + n])
        np.testing.assert_array_equal(part.continuous, whole.continuous[first:first + n])
    eng.close()
