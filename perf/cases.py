"""The work that programs on top of this framework have it do, as cases that can be timed and compared: ranking requests
and batches through the engine, the attention layer, the multi-hash embedding gather, the user tower and exhaustive
retrieval, each through its public entry point and over the range of sizes a serving host meets.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) engine / shard handles, weights, tables and inputs on the GPU (or in host buffers where the call
                        takes host buffers)
    run(state)          one pass
    work(case)          bytes and floating-point operations the pass cannot do without
    tolerance(case)     how far another correct implementation at the same precision may be off
    exact(case, seed)   the same results in 64-bit arithmetic, in plain torch
"""
from __future__ import annotations

import math

import numpy as np
import torch

import x_algorithm_b200 as px
from x_algorithm_b200.engine import ranker_attention
from x_algorithm_b200.retrieval import Retriever
from x_algorithm_b200.synthetic import zipf_ids

TABLE_SEED = 7
CORPUS_SEED = 4
ACTION_TYPES, SURFACES, HEADS, CONTINUOUS, HASHES = 8, 4, 19, 1, 2
EPS, ROPE_BASE, DWELL_SCALE, NEGATIVE_OFFSET = 1e-5, 10000.0, 30.0, 0.001


# ---- the cases --------------------------------------------------------------------------------------------------------

def _rank(name, batch, call, *, emb=512, layers=8, heads=8, kv_heads=8, dh=64, history=128, candidates=512, tail=0, log2_rows=18):
    return dict(name=name, kind="rank", call=call, batch=batch, emb=emb, layers=layers, heads=heads, kv_heads=kv_heads, dh=dh,
                history=history, candidates=candidates, tail=tail, log2_rows=log2_rows)


def _attention(name, batch, heads, kv_heads, dh, history, candidates):
    return dict(name=name, kind="attention", batch=batch, heads=heads, kv_heads=kv_heads, dh=dh, history=history, candidates=candidates)


def _retrieve(name, rows, queries, k, int8):
    return dict(name=name, kind="retrieve", rows=rows, dim=128, queries=queries, k=k, int8=int8)


def listed():
    return [
        # one user's feed request at the ranking benchmark's model, host buffers in and out: the latency a caller sees
        _rank("rank_request", 1, "host"),
        # a handful of small requests on the small model: launches and host work are all there is
        _rank("rank_small", 16, "host", emb=128, layers=2, heads=4, kv_heads=4, dh=32, history=32, candidates=8, log2_rows=17),
        # the ranking benchmark's full batch, inputs already on the device: the throughput of a loaded server
        _rank("rank_batch", 256, "device", log2_rows=20),
        # users with uneven histories and candidate counts, run over their valid rows only (two layers of the same model)
        _rank("rank_ragged", 48, "packed", layers=2),
        # a production-like geometry: grouped heads of 128, a history of a thousand posts, few candidates, the last layer on
        # candidate rows only
        _rank("rank_long_history", 8, "device", emb=1024, layers=2, heads=16, kv_heads=4, dh=128, history=1022, candidates=64, tail=1),
        # the attention layer by itself: the ranking model's shape at a medium batch, and a long history with long lists
        _attention("attention_short", 64, 8, 8, 64, 128, 512),
        _attention("attention_long", 32, 16, 16, 128, 1024, 1024),
        # the embedding stage of a training or feature job: millions of ids, four hashes each
        dict(name="gather_sum", kind="gather", ids=1 << 22, width=256, hashes=4, log2_rows=22),
        # the two-tower model's user side for a batch of users
        dict(name="user_tower", kind="tower", batch=256, emb=256, layers=4, heads=4, kv_heads=4, dh=64, history=128, log2_rows=18),
        # retrieval: one user against a small index, a batch of users against one shard, the same with the int8 index
        _retrieve("retrieve_one", 1_000_003, 1, 500, False),
        _retrieve("retrieve_shard", 12_500_000, 256, 1000, False),
        _retrieve("retrieve_shard_int8", 12_500_000, 256, 1000, True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rank", "rank", "rank", "long", "attention", "gather", "tower", "retrieve", "retrieve"])
    if kind == "rank":
        call = rng.choice(["host", "device", "packed"])
        history, candidates, batch = rng.randint(9, 128), _log_int(rng, 5, 512), _log_int(rng, 1, 256)
        if rng.random() < 0.25:
            c = _rank("", batch, call, emb=128, layers=2, heads=4, kv_heads=4, dh=32, history=history, candidates=candidates, log2_rows=17)
        else:
            c = _rank("", batch, call, layers=rng.choice([1, 2, 4, 8]), history=history, candidates=candidates)
    elif kind == "long":
        c = _rank("", _log_int(rng, 1, 16), rng.choice(["host", "device"]), emb=1024, layers=2, heads=16, kv_heads=rng.choice([4, 8, 16]), dh=128,
                  history=rng.randint(129, 1400), candidates=_log_int(rng, 16, 300), tail=rng.choice([0, 1]))
    elif kind == "attention":
        if rng.random() < 0.5:
            heads = rng.choice([4, 8])
            c = _attention("", _log_int(rng, 1, 256), heads, heads, 64, rng.randint(9, 128), _log_int(rng, 8, 512))
        else:
            heads, group = rng.choice([8, 16]), rng.choice([1, 4])
            c = _attention("", _log_int(rng, 1, 24), heads, heads // group, 128, rng.randint(129, 1400), _log_int(rng, 32, 1024))
    elif kind == "gather":
        c = dict(kind="gather", ids=_log_int(rng, 1000, 1 << 22), width=rng.choice([128, 256]), hashes=rng.choice([2, 4]), log2_rows=rng.choice([18, 20, 22]))
    elif kind == "tower":
        c = dict(kind="tower", batch=_log_int(rng, 1, 256), emb=256, layers=4, heads=4, kv_heads=4, dh=64, history=rng.randint(9, 128), log2_rows=18)
    else:
        rows = _log_int(rng, 40_000, 12_500_000)
        c = _retrieve("", rows, _log_int(rng, 1, 256), _log_int(rng, 10, 1000), rng.random() < 0.4)
    c.pop("name", None)
    return c


# ---- inputs -----------------------------------------------------------------------------------------------------------

def _bf16(x):
    return x.to(torch.bfloat16).float()


def _config(case):
    ranks = case["kind"] == "rank"
    return px.PhoenixConfig(
        emb_size=case["emb"], num_layers=case["layers"], num_q_heads=case["heads"], num_kv_heads=case["kv_heads"], key_size=case["dh"],
        widening_factor=4.0, history_len=case["history"], num_candidates=case["candidates"] if ranks else 0, max_batch=case["batch"],
        num_actions=HEADS, num_continuous=CONTINUOUS, num_action_types=ACTION_TYPES, num_surfaces=SURFACES, num_hashes=HASHES,
        table_size=1 << case["log2_rows"], num_candidate_only_layers=case.get("tail", 0) if ranks else 0,
        pack_ragged=ranks and case["call"] == "packed")


def _weights(case, seed):
    """Parameters as float32 CUDA tensors holding bf16 values: matrices N(0, 0.02), norm gains 1 + N(0, 0.05)."""
    g = torch.Generator(device="cuda").manual_seed(1000 + seed)
    D, F = case["emb"], 4 * case["emb"]
    HD, QW = case["heads"] * case["dh"], (case["heads"] + 2 * case["kv_heads"]) * case["dh"]

    def mat(rows, cols, std=0.02):
        return _bf16(torch.randn(rows, cols, device="cuda", generator=g) * std)

    def gain():
        return _bf16(1.0 + 0.05 * torch.randn(D, device="cuda", generator=g))

    w = {"action_table": mat(ACTION_TYPES + 1, D, D ** -0.5), "surface_table": mat(SURFACES + 1, D, D ** -0.5)}
    for i in range(case["layers"]):
        p = f"layer{i}."
        w[p + "pre_attn_norm"], w[p + "w_qkv"], w[p + "w_out"] = gain(), mat(D, QW), mat(HD, D)
        w[p + "pre_ffn_norm"], w[p + "w_up"], w[p + "w_down"] = gain(), mat(D, F), mat(F, D)
    w["final_norm"] = gain()
    w["unembed"], w["cont_unembed"] = mat(D, HEADS), mat(D, CONTINUOUS)
    return w


def _blend():
    """One weight per head: what a product sets once."""
    rng = np.random.Generator(np.random.PCG64(1))
    negative = {"not_interested", "block_author", "mute_author", "report"}
    w = {n: float(-rng.uniform(0.5, 3.0)) if n in negative else float(rng.uniform(0.5, 5.0)) for n in px.HEAD_NAMES_19}
    w["cont_dwell_time"] = float(rng.uniform(0.0, 0.01))
    return px.blend_spec_from_weights(px.ValueModelWeights(w=w), px.HEAD_NAMES_19, HEADS)


def _valid_counts(case):
    """Valid history slots and candidates of every request: spread evenly over [1, S] and [1, C] in a packed batch (the sums
    do not depend on the seed), everything elsewhere."""
    B, S, C = case["batch"], case["history"], case.get("candidates", 0)
    if case.get("call") != "packed":
        return np.full(B, S), np.full(B, C)
    i = np.arange(B)
    return 1 + (i * S) // B, 1 + (i * C) // B


def _batch(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    B, S, C = case["batch"], case["history"], case.get("candidates", 0)
    b = dict(hist_post=zipf_ids((B, S), rng), hist_author=zipf_ids((B, S), rng),
             hist_actions=rng.integers(1, ACTION_TYPES + 1, size=(B, S)).astype(np.int32),
             hist_surfaces=rng.integers(1, SURFACES + 1, size=(B, S)).astype(np.int32),
             cand_post=zipf_ids((B, C), rng), cand_author=zipf_ids((B, C), rng))
    hl, cl = _valid_counts(case)
    hl, cl = rng.permutation(hl), rng.permutation(cl)
    past_h, past_c = np.arange(S)[None, :] >= hl[:, None], np.arange(C)[None, :] >= cl[:, None]
    for n in ("hist_post", "hist_author", "hist_actions", "hist_surfaces"):
        b[n][past_h] = 0
    for n in ("cand_post", "cand_author"):
        b[n][past_c] = 0
    return b


def _engine(case, seed):
    eng = px.PhoenixEngine(_config(case), 0)
    eng.load_weights({n: t.cpu().numpy() for n, t in _weights(case, seed).items()})
    eng.table_fill_synthetic(TABLE_SEED, case["emb"] ** -0.5)
    return eng


def _users(case, seed):
    g = torch.Generator(device="cuda").manual_seed(2000 + seed)
    u = torch.randn(case["queries"], case["dim"], device="cuda", generator=g)
    return u / u.norm(dim=1, keepdim=True)


def _gather_ids(case, seed):
    return zipf_ids((case["ids"],), np.random.Generator(np.random.PCG64(seed)))


def _gather_config(case):
    heads = max(1, case["width"] // 64)
    return px.PhoenixConfig(emb_size=case["width"], num_layers=1, num_q_heads=heads, num_kv_heads=heads, key_size=64, history_len=1,
                            num_candidates=1, max_batch=1, num_hashes=case["hashes"], table_size=1 << case["log2_rows"])


def _qkv(case, seed):
    g = torch.Generator(device="cuda").manual_seed(3000 + seed)
    B, T, dh = case["batch"], case["history"] + case["candidates"], case["dh"]
    q, k, v = ((torch.randn(B, T, h, dh, device="cuda", generator=g) / math.sqrt(dh)).to(torch.bfloat16)
               for h in (case["heads"], case["kv_heads"], case["kv_heads"]))
    seg = torch.ones((B, T), dtype=torch.int32, device="cuda")
    seg[:, case["history"]:] = -1
    return q, k, v, seg


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("rank", "tower"):
        s["eng"] = _engine(case, seed)
        b = _batch(case, seed)
        B, C = case["batch"], case.get("candidates", 0)
        if kind == "tower":
            s["inputs"] = [torch.from_numpy(b[n]).cuda() for n in ("hist_post", "hist_author", "hist_actions", "hist_surfaces")]
            s["users"] = torch.empty((B, case["emb"]), dtype=torch.float32, device="cuda")
            return s
        s["eng"].set_blend(_blend())
        if case["call"] == "device":
            s["inputs"] = [torch.from_numpy(b[n]).cuda() for n in ("hist_post", "hist_author", "hist_actions", "hist_surfaces", "cand_post", "cand_author")]
            s["out"] = (torch.empty((B, C, HEADS), dtype=torch.float32, device="cuda"),
                        torch.empty((B, C, CONTINUOUS), dtype=torch.float32, device="cuda"),
                        torch.empty((B, C), dtype=torch.float64, device="cuda"))
        else:
            s["inputs"] = px.RankInputs(b["hist_post"], b["hist_author"], b["hist_actions"], b["hist_surfaces"], b["cand_post"], b["cand_author"])
            s["out"] = px.RankOutputs(np.empty((B, C, HEADS), np.float32), np.empty((B, C, CONTINUOUS), np.float32), np.empty((B, C), np.float64))
    elif kind == "attention":
        s["q"], s["k"], s["v"], s["seg"] = _qkv(case, seed)
    elif kind == "gather":
        s["eng"] = px.PhoenixEngine(_gather_config(case), 0)
        s["eng"].table_fill_synthetic(TABLE_SEED, case["width"] ** -0.5)
        s["ids"] = torch.from_numpy(_gather_ids(case, seed)).cuda()
        s["out"] = torch.empty((case["ids"], case["width"]), dtype=torch.bfloat16, device="cuda")
    else:
        shard = px.CorpusShard(case["rows"], case["dim"], max_queries=case["queries"], max_k=case["k"])
        shard.fill_synthetic(CORPUS_SEED)
        if case["int8"]:
            shard.quantize_int8()
            shard.set_int8(True)
        s["retriever"] = Retriever([shard])
        s["users"] = _users(case, seed)
    return s


# ---- one pass ---------------------------------------------------------------------------------------------------------

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "rank":
        if case["call"] == "device":
            s["eng"].rank_device(case["batch"], *s["inputs"], *s["out"])
            return s["out"]
        r = s["eng"].rank(s["inputs"], s["out"])
        return r.log_probs, r.continuous, r.scores
    if kind == "tower":
        s["eng"].user_tower_device(case["batch"], *s["inputs"], s["users"])
        return s["users"]
    if kind == "attention":
        return ranker_attention(s["q"], s["k"], s["v"], s["seg"], case["history"], math.sqrt(128.0) / case["dh"])[0]
    if kind == "gather":
        s["eng"].gather_sum_device(1, s["ids"], case["ids"], s["out"])
        return s["out"]
    return s["retriever"].retrieve(s["users"], case["k"])


# ---- what a pass cannot do without ------------------------------------------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind in ("rank", "tower"):
        D, F, HD, QW = case["emb"], 4 * case["emb"], case["heads"] * case["dh"], (case["heads"] + 2 * case["kv_heads"]) * case["dh"]
        KV = 2 * case["kv_heads"] * case["dh"]
        hl, cl = (x.astype(float) for x in _valid_counts(case))
        h, c = hl.sum(), cl.sum()
        L = case["layers"]
        frozen = max(case["tail"], 1) if kind == "rank" else 0    # layers whose history rows nothing reads afterwards
        att_full, att_cand = 4.0 * HD * (hl * hl + cl * (hl + 1)).sum(), 4.0 * HD * (cl * (hl + 1)).sum()
        full = (L - frozen) * (2.0 * (h + c) * D * (QW + HD + 2 * F) + att_full)
        last = frozen * (2.0 * c * D * (QW + HD + 2 * F) + 2.0 * h * D * KV + att_cand)
        heads = 2.0 * c * D * (HEADS + CONTINUOUS)
        weights = 2.0 * L * D * (QW + HD + 2 * F)
        rows = (h + c) * 2 * HASHES * D * 2.0
        ids = h * 24 + c * 16
        out = c * (4.0 * (HEADS + CONTINUOUS) + 8) if kind == "rank" else case["batch"] * D * 4.0
        return dict(bytes=weights + rows + ids + out, flops=full + last + (heads if kind == "rank" else 0.0))
    if kind == "attention":
        B, S, C, H, Hk, dh = case["batch"], case["history"], case["candidates"], case["heads"], case["kv_heads"], case["dh"]
        return dict(bytes=2.0 * B * (S + C) * dh * (2 * H + 2 * Hk) + 4.0 * B * (S + C), flops=4.0 * dh * H * B * (S * S + C * (S + 1.0)))
    if kind == "gather":
        return dict(bytes=case["ids"] * (case["hashes"] * case["width"] * 2.0 + case["width"] * 2.0 + 8.0), flops=case["ids"] * case["hashes"] * float(case["width"]))
    row = case["dim"] + 4.0 if case["int8"] else case["dim"] * 2.0
    return dict(bytes=case["rows"] * row + case["queries"] * (case["dim"] * 4.0 + case["k"] * 12.0), flops=2.0 * case["rows"] * case["dim"] * case["queries"])


def tolerance(case):
    """About four times what the other kernels the library has for the same step (stand-alone norms, other attention and
    scan kernels) were measured to differ by from the default ones: 3.7e-3 for eight layers of the ranking model, 2.3e-3
    for attention, 7e-4 for the tower, whose outputs are 2.4e-3 from the 64-bit result on either side."""
    kind = case["kind"]
    if kind == "rank":
        return {"rel": 1.5e-2}
    if kind in ("attention", "tower"):
        return {"rel": 1e-2}
    if kind == "gather":
        return "exact"            # fixed order of the fp32 sum, one rounding: part of the operator's contract
    if case["int8"]:
        return "exact"            # integer dot products
    return {"rel": 1e-4, "differ": 1e-2}   # scores are rounded to bf16: a sum on the edge of two values moves an id among equals


# ---- the same in 64 bits ----------------------------------------------------------------------------------------------

def _synthetic_rows(rows, width, seed, amp):
    """The synthetic table's rows as bf16 values in float32: a hash of (row, column, seed)."""
    x = (rows[..., None] * width + torch.arange(width, device=rows.device)) & 0xFFFFFFFF
    x ^= seed
    x ^= x >> 16
    x = (x * 0x7FEB352D) & 0xFFFFFFFF
    x ^= x >> 15
    x = (x * 0x846CA68B) & 0xFFFFFFFF
    x = (x ^ (x >> 16)) >> 16
    return _bf16((x.float() - 32768.0) * float(np.float32(amp / 32768.0)))


def _hash_rows(ids, family, offset):
    """Rows of the unified table for int64 ids: wrapping multiply-add, two floored remainders, id 0 -> row 0."""
    out = []
    for scale, bias in zip(family.scales, family.biases):
        raw = torch.remainder(torch.remainder(ids * scale + bias, family.modulus), family.table_size - 1) + 1 + offset
        out.append(torch.where(ids == 0, torch.zeros_like(raw), raw))
    return torch.stack(out, dim=-1)


def _norm64(x, gain):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * gain


def _attend64(q, k, v, seg, S, sm_scale):
    """q [b,T,H,d], k / v [b,T,Hk,d] float64, seg [b,T]: history keys plus, for candidates, their own."""
    H, Hk = q.shape[2], k.shape[2]
    k, v = k.repeat_interleave(H // Hk, dim=2), v.repeat_interleave(H // Hk, dim=2)
    s = torch.einsum("bqhd,bkhd->bhqk", q, k[:, :S]) * sm_scale
    s.masked_fill_((seg[:, None, None, :S] != 1), -math.inf)
    own = ((q * k).sum(-1) * sm_scale).permute(0, 2, 1)[..., None]
    own = own.masked_fill((seg != -1)[:, None, :, None], -math.inf)
    m = torch.maximum(s.amax(-1, keepdim=True), own)
    m = torch.where(torch.isfinite(m), m, torch.zeros_like(m))
    s, own = torch.exp(s - m), torch.exp(own - m)
    l = s.sum(-1, keepdim=True) + own
    o = torch.einsum("bhqk,bkhd->bqhd", s, v[:, :S]) + own.permute(0, 2, 1, 3) * v
    o = o / torch.where(l == 0, torch.ones_like(l), l).permute(0, 2, 1, 3)
    return o * (seg != 0)[:, :, None, None]


def _trunk64(case, w, x, seg, pos, tail):
    H, Hk, dh, S = case["heads"], case["kv_heads"], case["dh"], case["history"]
    b, T, _ = x.shape
    inv = ROPE_BASE ** (-torch.arange(0, dh, 2, device=x.device, dtype=torch.float64) / dh)
    ang = pos.double()[None, :, None, None] * inv
    cos, sin = torch.cos(ang), torch.sin(ang)

    def rope(t):
        a, c = t[..., :dh // 2], t[..., dh // 2:]
        return torch.cat((a * cos - c * sin, c * cos + a * sin), dim=-1)

    for i in range(case["layers"]):
        p = f"layer{i}."
        frozen = x[:, :S] if i >= case["layers"] - tail else None
        qkv = (_norm64(x, w[p + "pre_attn_norm"]) @ w[p + "w_qkv"]).view(b, T, Hk, H // Hk + 2, dh)
        q, k, v = qkv[..., :-2, :].reshape(b, T, H, dh), qkv[..., -2, :], qkv[..., -1, :]
        a = _attend64(rope(q), rope(k), v, seg, S, math.sqrt(128.0) / dh)
        x = x + a.reshape(b, T, H * dh) @ w[p + "w_out"]
        up = _norm64(x, w[p + "pre_ffn_norm"]) @ w[p + "w_up"]
        x = x + torch.nn.functional.gelu(up, approximate="tanh") @ w[p + "w_down"]
        if frozen is not None:
            x = torch.cat((frozen, x[:, S:]), dim=1)
    return x


def _model64(case, seed):
    cfg = _config(case)
    w = {n: t.double() for n, t in _weights(case, seed).items()}
    b = {n: torch.from_numpy(a).cuda() for n, a in _batch(case, seed).items()}
    D, S, C, B = case["emb"], case["history"], case.get("candidates", 0), case["batch"]
    user, item, author, _ = cfg.families()
    off_item = 65 + user.table_size
    off_author = off_item + item.table_size
    T = S + C
    pos = torch.clamp(torch.arange(T, device="cuda"), max=S)
    rows = lambda post, auth: _synthetic_rows(torch.cat((_hash_rows(post, item, off_item), _hash_rows(auth, author, off_author)), -1),
                                              D, TABLE_SEED, D ** -0.5).double().sum(-2)
    step = max(1, int(1.5e9 / (8.0 * max(T * 4 * D, case["heads"] * T * S, T * 4 * D * 4))))
    got = []
    for lo in range(0, B, step):
        c = {n: t[lo:lo + step] for n, t in b.items()}
        x = rows(c["hist_post"], c["hist_author"]) + w["action_table"][c["hist_actions"].long()] + w["surface_table"][c["hist_surfaces"].long()]
        seg = (c["hist_post"] != 0).int()
        if C:
            x = torch.cat((x, rows(c["cand_post"], c["cand_author"])), dim=1)
            seg = torch.cat((seg, -(c["cand_post"] != 0).int()), dim=1)
        x = _trunk64(case, w, x * math.sqrt(D), seg, pos, case.get("tail", 0))
        x = _norm64(x, w["final_norm"])
        if not C:
            valid = (seg == 1).double()[..., None]
            u = (x * valid).sum(1) / valid.sum(1).clamp(min=1.0)
            got.append(u / u.norm(dim=1, keepdim=True).clamp(min=1e-6))
            continue
        cand = x[:, S:]
        lp = torch.nn.functional.logsigmoid(cand @ w["unembed"] * (2.0 * math.sqrt(512.0 / D)))
        cont = torch.sigmoid(cand @ w["cont_unembed"]) * DWELL_SCALE
        spec = _blend()
        cols = torch.cat((lp.exp(), cont), -1)
        sc = sum(cols[..., spec.src[i]] * spec.weight[i] for i in range(spec.num_terms))
        sc = torch.where(sc < 0, (sc + spec.negative_sum) / spec.total_sum * NEGATIVE_OFFSET, sc + NEGATIVE_OFFSET)
        if case["call"] == "packed":       # slots past a request's candidates read zero
            ok = c["cand_post"] != 0
            lp, cont, sc = lp * ok[..., None], cont * ok[..., None], sc * ok
        got.append((lp, cont, sc))
    if not C:
        return torch.cat(got)
    return tuple(torch.cat(t) for t in zip(*got))


def _retrieve64(case, seed):
    """The k best scores per user in 64 bits; the rows they belong to have no such value (ties and near-ties)."""
    u = _users(case, seed).double()
    k = case["k"]
    if case["int8"]:
        us = torch.clamp(u.float().abs().amax(1) / 127.0, min=1e-12)
        u = torch.clamp(torch.round(u.float() / us[:, None]), -127, 127).double()
    best = None
    for lo in range(0, case["rows"], 1 << 19):
        r = torch.arange(lo, min(case["rows"], lo + (1 << 19)), device="cuda")
        raw = _synthetic_rows(r, case["dim"], CORPUS_SEED, 1.0)
        e = _bf16(raw / raw.double().square().sum(1, keepdim=True).clamp(min=1e-12).sqrt().float())
        if case["int8"]:
            rs = torch.clamp(e.abs().amax(1) / 127.0, min=1e-12)
            q = torch.clamp(torch.round(e / rs[:, None]), -127, 127).double()
            s = (u @ q.T) * us.double()[:, None] * rs.double()[None, :]
        else:
            s = u @ e.double().T
        s = s.topk(min(k, s.shape[1]), dim=1).values
        best = s if best is None else torch.cat((best, s), 1).topk(min(k, best.shape[1] + s.shape[1]), dim=1).values
    return best, None


def exact(case, seed):
    kind = case["kind"]
    if kind in ("rank", "tower"):
        return _model64(case, seed)
    if kind == "attention":
        q, k, v, seg = _qkv(case, seed)
        out = []
        step = max(1, int(1.0e9 / (8.0 * case["heads"] * q.shape[1] * case["history"])))
        for lo in range(0, case["batch"], step):
            part = [t[lo:lo + step] for t in (q, k, v)]
            out.append(_attend64(*(t.double() for t in part), seg[lo:lo + step], case["history"], math.sqrt(128.0) / case["dh"]).float())
        return torch.cat(out)
    if kind == "gather":
        user, item, _, _ = _gather_config(case).families()
        ids = torch.from_numpy(_gather_ids(case, seed)).cuda()
        out = torch.empty((case["ids"], case["width"]), dtype=torch.float32, device="cuda")
        for lo in range(0, case["ids"], 1 << 16):
            rows = _hash_rows(ids[lo:lo + (1 << 16)], item, 65 + user.table_size)
            out[lo:lo + (1 << 16)] = _synthetic_rows(rows, case["width"], TABLE_SEED, case["width"] ** -0.5).double().sum(-2).float()
        return out
    return _retrieve64(case, seed)
