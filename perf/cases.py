"""Performance cases: the work a serving program has this library do, at the sizes it meets.

Four kinds, all at the Granite 8B shapes (hidden 4096, MLP 12800, 32 query / 8 KV heads of 128):

  norm     one residual add + RMSNorm with bf16 and FP8 outputs on its own
  glue     the per-layer glue sequence of a batch of token rows whose GEMM and attention outputs
           come from elsewhere (embedding, `layers` x granite4_glue_layer, final norm)
  decode   one decode step: embedding of the newest tokens, two layers with their four FP8
           projections and attention over the int8 paged pool, final norm, lm_head, greedy pick.
           `tree` turns the rows into the verify step of one session's draft tree
  prefill  one layer of a prompt chunk: embedding, QKV projection, RoPE + int8 paged KV write,
           causal attention, O projection, MLP with the fused SwiGLU epilogue

`graph` says whether the program replays a CUDA graph captured once (what a decode loop does in
steady state) or issues the calls one by one (a step whose row count or draft tree is new).
"""
import math

import torch

import granite4_b200  # noqa: F401
from granite4_b200 import capi, glue, kernels as k

S = glue.GraniteShapes()
H, I, D = S.hidden, S.intermediate, S.head_dim
QKV = S.qkv_width
PAGE = 16
MAX_POS = 131072
ATT_SCALE = 1.0 / 128
PROJ = (("qkv", QKV, H), ("o", H, H), ("gate_up", 2 * I, H), ("down", H, I))
LAYERS = 2  # of a decode step
CODE = 448.0 / 5.0  # e4m3 codes of an N(0, 1) tensor whose largest value is 5 sigma


def listed():
    return [
        # the smallest call: one row of the norm between two blocks, f32 in, bf16 and FP8 out
        {"name": "norm_1_row_f32", "kind": "norm", "rows": 1, "cols": 4096, "f32": True},
        # steady-state decoding: one chat session, a busy server, a full batch at long context
        {"name": "decode_1_ctx_1900", "kind": "decode", "rows": 1, "ctx": 1900, "tree": False, "graph": True},
        {"name": "decode_8_ctx_4100", "kind": "decode", "rows": 8, "ctx": 4100, "tree": False, "graph": True},
        {"name": "decode_16_ctx_24000", "kind": "decode", "rows": 16, "ctx": 24000, "tree": False, "graph": True},
        # a step issued call by call: sessions have just joined or left
        {"name": "decode_3_ctx_777_eager", "kind": "decode", "rows": 3, "ctx": 777, "tree": False, "graph": False},
        # speculative decoding: 15 draft-tree rows of one session at 16k context
        {"name": "verify_15_ctx_16384_eager", "kind": "decode", "rows": 15, "ctx": 16384, "tree": True, "graph": False},
        # a short user turn appended to a conversation
        {"name": "prefill_37_at_1203", "kind": "prefill", "rows": 37, "base": 1203},
        # an ordinary prompt
        {"name": "prefill_500", "kind": "prefill", "rows": 500, "base": 0},
        # a chunk of a long document
        {"name": "prefill_1999_at_30000", "kind": "prefill", "rows": 1999, "base": 30000},
        # a long prompt in one chunk
        {"name": "prefill_8192", "kind": "prefill", "rows": 8192, "base": 0},
        # the glue of a small batch through all layers, and of the largest batch a GPU is given
        {"name": "glue_777_rows_40_layers", "kind": "glue", "rows": 777, "layers": 40},
        {"name": "glue_65536_rows_4_layers", "kind": "glue", "rows": 65536, "layers": 4},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("norm", "glue", "decode", "decode", "verify", "prefill", "prefill"))
    if kind == "norm":
        return {"kind": kind, "rows": _log_int(rng, 1, 16384), "cols": 8 * _log_int(rng, 128, 1024), "f32": rng.random() < 0.5}
    if kind == "glue":
        rows = _log_int(rng, 16, 65536)
        return {"kind": kind, "rows": rows, "layers": max(1, min(S.layers, 262144 // rows))}
    if kind == "decode":
        rows = rng.randint(1, 16)
        return {"kind": kind, "rows": rows, "ctx": _log_int(rng, 64, min(100000, 384000 // rows)), "tree": False,
                "graph": rng.random() < 0.6}
    if kind == "verify":
        return {"kind": "decode", "rows": rng.randint(4, 16), "ctx": _log_int(rng, 256, 100000), "tree": True,
                "graph": rng.random() < 0.3}
    rows = _log_int(rng, 17, 8192)
    return {"kind": kind, "rows": rows, "base": rng.choice((0, _log_int(rng, 16, 60000 if rows <= 2048 else 4096)))}


# ---- inputs ---------------------------------------------------------------------------------
_tables = {}


def _rope_tables(dev):
    """One set of RoPE tables for the process, as a program has it."""
    if dev not in _tables:
        _tables[dev] = k.RopeTables(S.rope_theta, D, MAX_POS, dev)
    return _tables[dev]


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=g.device)


def _codes(x):
    """e4m3 codes of an N(0, 1) tensor."""
    return (x * CODE).clamp_(-448.0, 448.0).to(torch.float8_e4m3fn).view(torch.uint8)


def _pages(g, pool_rows, n):
    """Pool rows of n positions in randomly permuted 16-token pages of a pool."""
    perm = torch.randperm(pool_rows // PAGE, generator=g, device=g.device)
    p = torch.arange(n, device=g.device)
    return (perm[p // PAGE] * PAGE + p % PAGE).to(torch.int32)


def _pool(g, rows):
    """An int8 pool already holding keys and values of about N(0, 4) and N(0, 1)."""
    ck = torch.empty(S.kv_heads, rows, D, device=g.device, dtype=torch.int8).random_(-127, 128, generator=g)
    cv = torch.empty_like(ck).random_(-127, 128, generator=g)
    ks = 0.05 + 0.005 * torch.rand(S.kv_heads, rows, generator=g, device=g.device)
    vs = 0.0125 + 0.00125 * torch.rand(S.kv_heads, rows, generator=g, device=g.device)
    return ck, cv, ks, vs


def _layer_weights(g):
    """FP8 weights of one layer and the scales that keep every activation at its usual size:
    queries and keys of about N(0, 4) (attention logits of a few units), all else N(0, 1)."""
    w = {name: _codes(_randn(g, n, kd)) for name, n, kd in PROJ}
    one = 1.0 / CODE
    w["s_qkv"] = (4 * one / math.sqrt(H), 4 * one / math.sqrt(H), one / math.sqrt(H))
    w["s_o"] = w["s_gate_up"] = (one / math.sqrt(H),)
    w["s_down"] = (one / math.sqrt(I),)
    w["norm1"] = (1 + 0.02 * _randn(g, H)).to(torch.bfloat16)
    w["norm2"] = (1 + 0.02 * _randn(g, H)).to(torch.bfloat16)
    return w


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(seed)
    return {"norm": _prepare_norm, "glue": _prepare_glue, "decode": _prepare_decode,
            "prefill": _prepare_prefill}[case["kind"]](case, g, dev)


def _prepare_norm(case, g, dev):
    rows, cols = case["rows"], case["cols"]
    kind = torch.float32 if case["f32"] else torch.bfloat16
    y, res = _randn(g, rows, cols).to(kind), _randn(g, rows, cols).to(kind)
    w = (1 + 0.02 * _randn(g, cols)).to(torch.bfloat16)
    out = {"h": torch.empty(rows, cols, dtype=torch.bfloat16, device=dev),
           "n": torch.empty(rows, cols, dtype=torch.bfloat16, device=dev),
           "codes": torch.empty(rows, cols, dtype=torch.uint8, device=dev),
           "scale": torch.zeros(2, device=dev)}
    rstd = torch.empty(rows, device=dev)

    def step():
        assert k.add_rmsnorm_fp8(y, res, w, S.eps, S.residual_multiplier, h_out=out["h"], n_bf16=out["n"],
                                 n_fp8=out["codes"], scale_amax=out["scale"], rstd=rstd) == 0
        return out
    return step


def _prepare_glue(case, g, dev):
    rows, layers = case["rows"], case["layers"]
    pool = -(-rows // PAGE) * PAGE
    seq = glue.GlueSequence(rows, device=dev, seed=int(torch.randint(1 << 30, (1,), generator=g, device=dev)),
                            layers=layers, pool_rows=pool, max_pos=min(8192, max(rows, 16)))
    seq.set_rows(torch.arange(rows, device=dev) % seq.max_pos, _pages(g, pool, rows))
    emb = (0.02 * _randn(g, 16384, H)).to(torch.bfloat16)
    tok = torch.randint(16384, (rows,), generator=g, device=dev, dtype=torch.int32)
    out = {"hidden": seq.h, "final": seq.out, "q": seq.q_rot, "n_fp8": seq.n_fp8, "act_fp8": seq.act_fp8,
           "scales": seq.scales, "k": seq.cache_k, "v": seq.cache_v, "ks": seq.k_scale, "vs": seq.v_scale}

    def step():
        assert k.embed_gather(tok, emb, S.embedding_multiplier, seq.h) == 0
        seq.run_fast()
        return out
    return step


def _tree(n):
    """Parents of a draft tree of n nodes: a root, then two branches that fan out to depth 7."""
    parent, depth = [-1], [1]
    for i in range(1, n):
        p = max(0, i - 2)
        if depth[p] >= capi.MAX_TREE_DEPTH:
            p = 0
        parent.append(p)
        depth.append(depth[p] + 1)
    return parent


def _prepare_decode(case, g, dev):
    n, ctx, tree = case["rows"], case["ctx"], case["tree"]
    bf = torch.bfloat16
    tables = _rope_tables(dev)
    emb = (0.02 * _randn(g, S.vocab, H)).to(bf)
    w_lm = _codes(emb.float() / 0.02)  # tied lm_head
    w_final = (1 + 0.02 * _randn(g, H)).to(bf)
    layers = [_layer_weights(g) for _ in range(LAYERS)]
    slots = -(-(ctx + 64) // PAGE) * PAGE  # positions a session holds pages for
    sessions = 1 if tree else n
    pool = sessions * slots
    caches = [_pool(g, pool) for _ in range(LAYERS)]
    place = _pages(g, pool, pool)
    tbl = [place[r * slots:(r + 1) * slots].contiguous() for r in range(sessions)]
    toks = [torch.randint(S.vocab, (slots,), generator=g, device=dev, dtype=torch.int32) for _ in range(sessions)]
    desc = capi.MultiRows()
    desc.n = n
    if tree:
        parent = _tree(n)
        tail = torch.zeros(n, capi.MAX_TREE_DEPTH, dtype=torch.int32)
        desc.tree = 1
        for r in range(n):
            chain, a = [], r
            while a >= 0:
                chain.insert(0, ctx + 1 + a)
                a = parent[a]
            tail[r, :len(chain)] = torch.tensor(chain, dtype=torch.int32)
            desc.pos[r], desc.slot[r], desc.tbase[r] = ctx + len(chain), ctx + 1 + r, ctx
        tail = tail.to(dev)
        tbase = torch.full((n,), ctx, dtype=torch.int32, device=dev)
        grp = torch.tensor([r0 | min(4, n - r0) << 8 for r0 in range(0, n, 4)], dtype=torch.int32, device=dev)
    else:
        for r in range(n):  # sessions of unequal length, the longest at ctx
            desc.pos[r] = ctx - (r * ctx) // (2 * n)
    for r in range(n):
        desc.pt[r] = tbl[r % sessions].data_ptr()
        desc.tok[r] = toks[r % sessions].data_ptr()
    where = [(desc.slot[r] if tree else desc.pos[r]) for r in range(n)]
    kv_rows = torch.stack([tbl[r % sessions][p] for r, p in enumerate(where)]).to(torch.int32)
    fresh = k.multi_rows_to_device(desc, dev)
    rows = fresh.clone()
    row_pos = rows[capi.MultiRows.pos.offset:capi.MultiRows.pos.offset + 4 * n].view(torch.int32)
    row_pt = rows[capi.MultiRows.pt.offset:capi.MultiRows.pt.offset + 8 * n].view(torch.int64)
    max_len = min(slots, -(-(ctx + 32) // PAGE) * PAGE)

    hid = torch.empty(n, H, dtype=bf, device=dev)
    n8, a8 = (torch.empty(n, H, dtype=torch.uint8, device=dev) for _ in range(2))
    act8 = torch.empty(n, I, dtype=torch.uint8, device=dev)
    qkv = torch.empty(n, QKV, dtype=bf, device=dev)
    q_rot, att = (torch.empty(n, H, dtype=bf, device=dev) for _ in range(2))
    gu = torch.empty(n, 2 * I, dtype=bf, device=dev)
    logits = torch.empty(n, S.vocab, dtype=bf, device=dev)
    ids = torch.zeros(n, dtype=torch.int32, device=dev)
    sc = torch.zeros(4 * LAYERS + 1, 2, device=dev)
    if tree:
        need = capi.lib().granite4_attn_split_scratch_bytes(S.q_heads, n, max_len)
    else:
        need = k.attn_decode_scratch_bytes(n, 1, S.kv_heads, max_len)
    scratch = torch.empty(max(need, 16), dtype=torch.uint8, device=dev)
    ws = {name: k.gemm_fp8_workspace(n, nn, kd, dev) for name, nn, kd in PROJ + (("lm", S.vocab, H),)}
    lm_scale = (0.02 / CODE,)
    rm = S.residual_multiplier

    def step():
        rows.copy_(fresh)  # the step's descriptor
        rc = k.gpu_multi_embed(rows, n, emb, S.embedding_multiplier, hid)
        for i, w in enumerate(layers):
            ck, cv, ks, vs = caches[i]
            s0, s1, s2, s3 = (sc[4 * i + j] for j in range(4))
            rc |= k.add_rmsnorm_fp8(hid, None, w["norm1"], S.eps, rm, n_fp8=n8, scale_amax=s0)
            rc |= k.gemm_fp8(n8, w["qkv"], qkv, a_scale=s0, w_scales=w["s_qkv"], segs=(H, H + S.kv_heads * D),
                             workspace=ws["qkv"])
            rc |= k.rope_kv_int8_paged(qkv, tables.cos, tables.sin, row_pos, kv_rows, S.q_heads, S.kv_heads, D, pool,
                                       MAX_POS, 1, q_rot, ck, cv, ks, vs)
            if tree:
                rc |= k.attn_split_int8(q_rot, ck, cv, ks, vs, ATT_SCALE, S.q_heads, S.kv_heads, D, pool, att,
                                        max_len=max_len, row_pos=row_pos, row_pt=row_pt, row_grp=grp, row_tbase=tbase,
                                        row_tail=tail, scratch=scratch)
            else:
                rc |= k.attn_decode_int8_paged(q_rot, ck, cv, ks, vs, row_pos, S.q_heads, S.kv_heads, D, pool, max_len,
                                               ATT_SCALE, att, row_pt=row_pt, scratch=scratch)
            rc |= k.fp8_quant(att, a8, s1)
            rc |= k.gemm_fp8(a8, w["o"], hid, a_scale=s1, w_scales=w["s_o"], residual=hid, resid_scale=rm,
                             workspace=ws["o"])
            rc |= k.add_rmsnorm_fp8(hid, None, w["norm2"], S.eps, rm, n_fp8=n8, scale_amax=s2)
            rc |= k.gemm_fp8(n8, w["gate_up"], gu, a_scale=s2, w_scales=w["s_gate_up"], workspace=ws["gate_up"])
            rc |= k.swiglu_fp8(gu[:, :I], gu[:, I:], None, act8, s3, ld=2 * I)
            rc |= k.gemm_fp8(act8, w["down"], hid, a_scale=s3, w_scales=w["s_down"], residual=hid, resid_scale=rm,
                             workspace=ws["down"])
        sf = sc[4 * LAYERS]
        rc |= k.add_rmsnorm_fp8(hid, None, w_final, S.eps, rm, n_fp8=n8, scale_amax=sf)
        rc |= k.gemm_fp8(n8, w_lm, logits, a_scale=sf, w_scales=lm_scale, workspace=ws["lm"])
        if tree:  # the ids of a tree are compared with the drafts before any position advances
            rc |= k.argmax_rows(logits, ids)
        else:
            rc |= k.argmax_advance(logits, rows, ids)
        assert rc == 0
    out = {"hidden": hid, "logits": logits, "ids": ids, "pos": row_pos, "caches": caches}
    if not case["graph"]:
        def eager():
            step()
            return out
        return eager
    side = torch.cuda.Stream(dev)
    side.wait_stream(torch.cuda.current_stream(dev))
    with torch.cuda.stream(side):
        step()
    torch.cuda.current_stream(dev).wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()

    keep = (step, fresh, tbl, toks)

    def replay():
        graph.replay()
        return out
    replay.keep = keep
    return replay


def _prepare_prefill(case, g, dev):
    n, base = case["rows"], case["base"]
    bf = torch.bfloat16
    tables = _rope_tables(dev)
    emb = (0.02 * _randn(g, 16384, H)).to(bf)
    tok = torch.randint(16384, (n,), generator=g, device=dev, dtype=torch.int32)
    w = _layer_weights(g)
    pool = -(-(base + n) // PAGE) * PAGE
    ck, cv, ks, vs = _pool(g, pool)
    pt = _pages(g, pool, pool)
    hid = torch.empty(n, H, dtype=bf, device=dev)
    n8, a8 = (torch.empty(n, H, dtype=torch.uint8, device=dev) for _ in range(2))
    act8 = torch.empty(n, I, dtype=torch.uint8, device=dev)
    act = torch.empty(n, I, dtype=bf, device=dev)
    qkv = torch.empty(n, QKV, dtype=bf, device=dev)
    q_rot, att = (torch.empty(n, H, dtype=bf, device=dev) for _ in range(2))
    s0, s1, s2, s3 = torch.zeros(4, 2, device=dev)
    need = k.attn_decode_scratch_bytes(n, 4, S.kv_heads, base + n) if n <= 64 else 0
    scratch = torch.empty(max(need, 16), dtype=torch.uint8, device=dev)
    ws = {name: k.gemm_fp8_workspace(n, nn, kd, dev) for name, nn, kd in PROJ}
    rm = S.residual_multiplier

    def step():
        rc = k.prefill_embed_rows(tok, 0, n, emb, S.embedding_multiplier, hid)
        rc |= k.add_rmsnorm_fp8(hid, None, w["norm1"], S.eps, rm, n_fp8=n8, scale_amax=s0)
        rc |= k.gemm_fp8(n8, w["qkv"], qkv, a_scale=s0, w_scales=w["s_qkv"], segs=(H, H + S.kv_heads * D),
                         workspace=ws["qkv"])
        rc |= k.prefill_rope_split_append_int8(qkv, tables.cos, tables.sin, base, n, S.q_heads, S.kv_heads, D, pool,
                                               q_rot, ck, cv, ks, vs, pt)
        rc |= k.prefill_attention_int8(q_rot, ATT_SCALE, S.q_heads, S.kv_heads, D, base, pool, att, ck, cv, ks, vs,
                                       pt=pt, scratch=scratch)
        rc |= k.fp8_quant(att, a8, s1)
        rc |= k.gemm_fp8(a8, w["o"], hid, a_scale=s1, w_scales=w["s_o"], residual=hid, resid_scale=rm,
                         workspace=ws["o"])
        rc |= k.add_rmsnorm_fp8(hid, None, w["norm2"], S.eps, rm, n_fp8=n8, scale_amax=s2)
        rc |= k.gemm_fp8(n8, w["gate_up"], act, a_scale=s2, w_scales=w["s_gate_up"], swiglu_scale_amax=s3)
        rc |= k.fp8_encode_with_amax(act, act8, s3)
        rc |= k.gemm_fp8(act8, w["down"], hid, a_scale=s3, w_scales=w["s_down"], residual=hid, resid_scale=rm,
                         workspace=ws["down"])
        assert rc == 0
        return {"hidden": hid, "q": q_rot, "attention": att, "act": act, "k": ck, "v": cv, "ks": ks, "vs": vs}
    return step


# ---- one pass -------------------------------------------------------------------------------
def run(state):
    return state()


# ---- what a pass cannot do without --------------------------------------------------------------
def work(case):
    rows = case["rows"]
    if case["kind"] == "norm":
        c = case["cols"]
        return {"bytes": rows * c * (2 * (4 if case["f32"] else 2) + 2 + 2 + 1) + 2 * c, "flops": 8 * rows * c}
    if case["kind"] == "glue":
        per = glue.bytes_per_row(S)
        layer = 2 * per["add_rmsnorm_fp8"] + per["rope_kv_int8"] + per["swiglu_fp8"]
        return {"bytes": rows * (per["embed"] + case["layers"] * layer + per["final_norm"]), "flops": 0}
    params = sum(n * kd for _, n, kd in PROJ)
    kv_pos = 2 * S.kv_heads * (D + 4)  # bytes of one cache position
    if case["kind"] == "decode":
        ctx = case["ctx"]
        seen = ctx + 1 + rows if case["tree"] else sum(ctx - (r * ctx) // (2 * rows) + 1 for r in range(rows))
        pairs = rows * (ctx + 4) if case["tree"] else seen
        return {"bytes": LAYERS * (params + kv_pos * seen) + S.vocab * H + rows * (4 * H + 2 * S.vocab),
                "flops": 2 * rows * (LAYERS * params + S.vocab * H) + LAYERS * 4 * S.q_heads * D * pairs}
    base = case["base"]
    pairs = rows * base + rows * (rows + 1) // 2
    return {"bytes": params + kv_pos * (base + rows) + rows * 4 * H,
            "flops": 2 * rows * params + 4 * S.q_heads * D * pairs}


def tolerance(case):
    # norm: sums in double and exact rounding, the same bits by contract
    if case["kind"] == "norm":
        return "exact"
    # glue: one bf16 step of a SwiGLU value can move a code, or the tensor's scale with it
    if case["kind"] == "glue":
        return {"rel": 4e-3, "max": 4e-3, "differ": 1e-3}
    # bf16 activations re-quantised to 3-bit mantissas with a per-tensor scale between the GEMMs
    return {"rel": 1e-2, "max": 0.2, "differ": 2e-3}
