"""The gather-sum for many ids around the size where it takes over, for every hash count and widths that fill, split or overrun a
warp's columns: the same bits as the oracle."""
import numpy as np
import pytest

from helpers import make_pair
from oracle import phoenix_oracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("emb,hashes", [(64, 1), (128, 2), (192, 3), (256, 4), (512, 2), (576, 4)])
def test_many_ids_bit_exact(emb, hashes):
    import torch
    ocfg, w, rows_fn, eng = make_pair(max_batch=1, emb_size=emb, num_hashes=hashes, num_q_heads=emb // 32, num_kv_heads=emb // 32,
                                      history_len=1, num_candidates=1, num_layers=1, table_size=1 << 12)
    rng = np.random.default_rng(emb)
    lay = ocfg.hash_layout()
    for n in ((1 << 12) - 1, 1 << 12, (1 << 12) + 1, 40003):
        ids = rng.integers(-(1 << 40), 1 << 40, size=n)
        ids[::777] = 0
        ids[-1] = 5
        want = po.gather_sum(rows_fn(lay.author_hash(ids)))
        out = torch.full((n + 1, emb), 7, dtype=torch.int16, device="cuda")
        d = torch.from_numpy(ids).cuda()
        torch.cuda.synchronize()
        eng.gather_sum_device(2, d, n, out)
        eng.sync()
        got = out.cpu().numpy()
        np.testing.assert_array_equal(got[:n].view(np.uint16), want)
        assert (got[n] == 7).all()
    eng.close()


@pytest.mark.parametrize("emb,hashes,line", [(64, 1, 8192), (256, 1, 8192), (512, 1, 16384), (256, 2, 4096), (512, 2, 8192), (256, 3, 4096), (512, 4, 6144),
                                             (1024, 4, 12288)])
def test_where_many_ids_begin(emb, hashes, line):
    """Both sides of the line between the two kernels, which lies further out for wide rows and few hashes: the same bits."""
    import torch
    from x_algorithm_b200.engine import dispatch_counts
    ocfg, w, rows_fn, eng = make_pair(max_batch=1, emb_size=emb, num_hashes=hashes, num_q_heads=emb // 32, num_kv_heads=emb // 32,
                                      history_len=1, num_candidates=1, num_layers=1, table_size=1 << 12)
    ids = np.random.default_rng(emb + hashes).integers(-(1 << 40), 1 << 40, size=line)
    want = po.gather_sum(rows_fn(ocfg.hash_layout().author_hash(ids)))
    d = torch.from_numpy(ids).cuda()
    for n, kind in ((line - 1, "gather"), (line, "gather.bulk")):
        out = torch.full((line + 1, emb), 7, dtype=torch.int16, device="cuda")
        torch.cuda.synchronize()
        before = dispatch_counts()
        eng.gather_sum_device(2, d, n, out)
        eng.sync()
        assert {k for k, v in dispatch_counts().items() if v != before[k]} == {kind}
        got = out.cpu().numpy()
        np.testing.assert_array_equal(got[:n].view(np.uint16), want[:n])
        assert (got[n:] == 7).all()
    eng.close()
