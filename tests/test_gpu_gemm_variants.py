"""The GEMM variants a call's size picks - one tile per CTA for few tiles, CTA pairs with 256- or 128-column tiles beyond - against
the single-CTA kernel, which multiplies and rounds in the same order: the same bits, at the edges of the 128-row and
64 / 128 / 256-column tiles and of the 64-column k-steps, and through the engine for the RoPE, RMSNorm and statistics epilogues.
Every case says which kernels it means to run, and they are the ones that ran."""
import ctypes
import ctypes.util

import numpy as np
import pytest

from helpers import make_pair, to_inputs
from oracle import phoenix_oracle as po

pytestmark = pytest.mark.gpu


class ran_gemms:
    """The GEMM variants launched inside the block."""
    def __enter__(self):
        from x_algorithm_b200.engine import dispatch_counts
        self.before = dispatch_counts()
        return self

    def __exit__(self, *exc):
        from x_algorithm_b200.engine import dispatch_counts
        self.kinds = {k[5:] for k, v in dispatch_counts().items() if k.startswith("gemm.") and v != self.before[k]}


@pytest.mark.parametrize("M,N,K,kind", [(1, 64, 64, "small"), (127, 72, 8, "small"), (129, 512, 2048, "small"), (640, 2048, 512, "small"),
                                        (640, 1536, 520, "small"), (1281, 1024, 256, "small"),
                                        (4736, 512, 512, "small"), (4737, 512, 512, "pair256"), (18944, 128, 72, "small"), (18945, 128, 72, "pair128"),
                                        (20001, 1024, 512, "pair256"), (38000, 512, 448, "pair256"), (19000, 2048, 72, "pair256"),
                                        (20001, 128, 512, "pair128"), (7001, 384, 520, "pair128"), (7001, 200, 64, "small"), (12001, 200, 64, "pair128")])
@pytest.mark.parametrize("epi", [0, 1, 2])
def test_variants_give_the_same_bits(monkeypatch, M, N, K, kind, epi):
    import torch
    from x_algorithm_b200.engine import gemm
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = (torch.randn(M, K, device="cuda", generator=g) * 0.5).to(torch.bfloat16)
    wt = (torch.randn(N, K, device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    r = torch.randn(M, N, device="cuda", generator=g).to(torch.bfloat16) if epi == 1 else None
    with ran_gemms() as ran:
        c, _ = gemm(a, wt, r, epi, 0)
    assert ran.kinds == {kind}
    with ran_gemms() as ran:
        one, _ = gemm(a, wt, r, epi, 2)
    assert ran.kinds <= {"cta128", "cta256"}
    assert torch.equal(c, one)
    monkeypatch.setenv("PHX_GEMM", "pair")
    with ran_gemms() as ran:
        two, _ = gemm(a, wt, r, epi, 0)
    assert ran.kinds == {"pair256" if N % 256 == 0 else "pair128"}
    assert torch.equal(two, one)


@pytest.mark.parametrize("rows", [8192, 65536])           # one tile per CTA; CTA pairs
def test_gelu_of_every_value(rows):
    """Every finite bf16 value through the GELU epilogue of each kernel: the value of the scalar formula (the SIMT kernel's), which
    is written in another order; only a zero's sign may differ."""
    import torch
    from x_algorithm_b200.engine import gemm
    v = torch.arange(65536, dtype=torch.int32, device="cuda").to(torch.int16).view(torch.bfloat16)
    v = torch.where(torch.isfinite(v.float()), v, torch.ones_like(v)).reshape(8192, 8).repeat(rows // 8192, 1)
    eye = torch.eye(8, dtype=torch.bfloat16, device="cuda")
    want, _ = gemm(v, eye, None, 2, 1)
    for impl in (0, 2):
        got, _ = gemm(v, eye, None, 2, impl)
        assert torch.equal(got, want)


SMALL, WIDE, NARROW = "small", "pair256", "pair128"


@pytest.mark.parametrize("B,opts,kinds", [
    (1, dict(history_len=31, num_candidates=70), {SMALL}), (5, dict(history_len=32, num_candidates=8), {SMALL}),
    (3, dict(emb_size=256, num_q_heads=4, num_kv_heads=2, key_size=64, history_len=40, num_candidates=150), {SMALL}),
    (2, dict(emb_size=256, num_q_heads=2, num_kv_heads=1, key_size=128, history_len=40, num_candidates=90), {SMALL}),
    (40, dict(emb_size=1024, num_q_heads=4, num_kv_heads=2, key_size=128, history_len=40, num_candidates=90, num_layers=1), {WIDE}),
    (90, dict(emb_size=256, num_q_heads=6, num_kv_heads=3, key_size=128, history_len=129, num_candidates=100, num_layers=1), {WIDE, SMALL}),
    (64, dict(emb_size=512, num_q_heads=8, num_kv_heads=8, key_size=64, history_len=100, num_candidates=211, num_layers=1), {WIDE}),
    # rows enough for pairs where no width is a multiple of 256: heads of 32, and an odd number of 128-column parts
    (40, dict(emb_size=128, num_q_heads=4, num_kv_heads=4, key_size=32, history_len=127, num_candidates=385, num_layers=2), {WIDE, NARROW, SMALL}),
    (40, dict(emb_size=128, num_q_heads=1, num_kv_heads=1, key_size=128, history_len=127, num_candidates=385, num_layers=2), {WIDE, NARROW, SMALL}),
    (40, dict(emb_size=128, num_q_heads=3, num_kv_heads=1, key_size=128, history_len=127, num_candidates=385, num_layers=2), {WIDE, NARROW, SMALL})])
def test_engine_forward_same_bits(monkeypatch, B, opts, kinds):
    ocfg, w, rows_fn, eng = make_pair(max_batch=B, **opts)
    b = po.make_batch(ocfg, B, seed=3, ragged=True)
    with ran_gemms() as ran:
        got = eng.rank(to_inputs(b))
    eng.close()
    assert ran.kinds == kinds
    monkeypatch.setenv("PHX_GEMM", "cta1")
    _, _, _, eng = make_pair(max_batch=B, **opts)
    with ran_gemms() as ran:
        want = eng.rank(to_inputs(b))
    eng.close()
    assert ran.kinds <= {"cta128", "cta256"}
    np.testing.assert_array_equal(got.log_probs, want.log_probs)
    np.testing.assert_array_equal(got.continuous, want.continuous)


@pytest.mark.parametrize("D,hq,hkv,dh,C,mode", [(512, 4, 4, 64, 512, None), (512, 4, 4, 64, 512, "pair"), (512, 4, 4, 64, 512, "cta1"),
                                                (256, 8, 2, 32, 300, None), (256, 4, 1, 128, 300, None), (256, 2, 2, 128, 300, "pair"),
                                                (128, 4, 4, 32, 300, "pair"), (128, 1, 1, 128, 300, "cta1")])
def test_rope_epilogue_rounds_as_stated(monkeypatch, D, hq, hkv, dh, C, mode):
    """The rotated q and k columns against their definition in 64 bits with the epilogue's roundings: (x1, x2) ->
    (fma(x1, c, -fl(x2 s)), fma(x1, s, fl(x2 c))), heads of 128 (.., fma(x2, c, fl(x1 s))), then bf16.  Which product is rounded
    shows in a few columns per million."""
    S = 128
    if mode:
        monkeypatch.setenv("PHX_GEMM", mode)
    kw = dict(max_batch=1, emb_size=D, num_q_heads=hq, num_kv_heads=hkv, key_size=dh, history_len=S, num_candidates=C, num_layers=1)
    width = (hq + 2 * hkv) * dh
    raw = []
    for rotary in (False, True):
        ocfg, w, rows_fn, eng = make_pair(rotary=rotary, **kw)
        eng.rank(to_inputs(po.make_batch(ocfg, 1, seed=3)))
        raw.append(po.bf16_from_bits(eng.debug_read("qkv", (S + C, width), np.uint16)))   # one request: rows in order in any layout
        base = float(ocfg.rope_base)
        eng.close()
    libm = ctypes.CDLL(ctypes.util.find_library("m"))
    for f in (libm.cosf, libm.sinf):
        f.restype, f.argtypes = ctypes.c_float, [ctypes.c_float]
    libm.powf.restype, libm.powf.argtypes = ctypes.c_float, [ctypes.c_float, ctypes.c_float]
    f32, half = np.float32, dh // 2
    inv = [f32(1) / f32(libm.powf(base, float(f32(2 * j) / f32(dh)))) for j in range(half)]
    pos = np.minimum(np.arange(S + C), S)
    tab = [np.array([[f(float(f32(p) * inv[j])) for j in range(half)] for p in range(S + 1)], f32)[pos].astype(np.float64)[:, None, None, :]
           for f in (libm.cosf, libm.sinf)]
    g = hq // hkv
    x, got = (r.reshape(S + C, hkv, g + 2, dh) for r in raw)
    np.testing.assert_array_equal(x[:, :, g + 1], got[:, :, g + 1])                       # v parts pass through
    x1, x2 = (x[:, :, :g + 1, h * half:(h + 1) * half].astype(np.float64) for h in (0, 1))
    fl = lambda v: v.astype(f32).astype(np.float64)
    c, s = tab
    np.testing.assert_array_equal(got[:, :, :g + 1, :half], po.bf16_round((x1 * c - fl(x2 * s)).astype(f32)))
    hi = fl(x1 * s) + x2 * c if dh == 128 else x1 * s + fl(x2 * c)
    np.testing.assert_array_equal(got[:, :, :g + 1, half:], po.bf16_round(hi.astype(f32)))
