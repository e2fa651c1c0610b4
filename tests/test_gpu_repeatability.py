"""A decode or verify layer gives the same bits on every pass, whatever its intermediates held before: the exchange
of partial sums between CTAs, the cluster reductions and the split attention all add in a fixed order, and no op
reads what an earlier pass left."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
H, I, HQ, HK, D = 4096, 12800, 32, 8, 128
QKV = (HQ + 2 * HK) * D


def layer(rows, tree):
    import granite4_b200  # noqa: F401
    from granite4_b200 import capi, kernels as k
    g = torch.Generator(device=DEV).manual_seed(rows)
    bf, ctx, slots = torch.bfloat16, 700, 736
    sessions = 1 if tree else rows
    pool = sessions * slots
    w = {name: torch.randn(n, kd, generator=g, device=DEV).mul_(89.6).clamp_(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8)
         for name, n, kd in (("qkv", QKV, H), ("o", H, H), ("gate_up", 2 * I, H), ("down", H, I))}
    hid0 = torch.randn(rows, H, generator=g, device=DEV).to(bf)
    norm = (1 + 0.02 * torch.randn(H, generator=g, device=DEV)).to(bf)
    ck, cv = (torch.empty(HK, pool, D, dtype=torch.int8, device=DEV).random_(-127, 128, generator=g) for _ in range(2))
    ks, vs = (0.05 + 0.005 * torch.rand(HK, pool, generator=g, device=DEV) for _ in range(2))
    table = torch.randperm(pool, generator=g, device=DEV).int().view(sessions, slots)
    tables = k.RopeTables(1e7, D, 1024, torch.device(DEV))
    if tree:  # a chain of draft rows of one session, each seeing those before it
        slot = torch.arange(rows, device=DEV) + ctx + 1
        pos = (ctx + 1 + torch.arange(rows, device=DEV).clamp_(max=capi.MAX_TREE_DEPTH - 1)).int()
        tail = torch.zeros(rows, capi.MAX_TREE_DEPTH, dtype=torch.int32, device=DEV)
        for r in range(rows):
            n = int(pos[r]) - ctx
            tail[r, :n] = slot[:n].int()
            tail[r, n - 1] = slot[r]
        tbase = torch.full((rows,), ctx, dtype=torch.int32, device=DEV)
        grp = torch.tensor([r | min(4, rows - r) << 8 for r in range(0, rows, 4)], dtype=torch.int32, device=DEV)
        kv_rows = table[0][slot]
    else:
        pos = torch.tensor([ctx - 30 * r for r in range(rows)], dtype=torch.int32, device=DEV)
        kv_rows = torch.stack([table[r][int(pos[r])] for r in range(rows)])
    row_pt = torch.tensor([table[r % sessions].data_ptr() for r in range(rows)], dtype=torch.int64, device=DEV)
    need = (capi.lib().granite4_attn_split_scratch_bytes(HQ, rows, slots) if tree
            else k.attn_decode_scratch_bytes(rows, 1, HK, slots))
    b = {"hid": torch.empty(rows, H, dtype=bf, device=DEV), "qkv": torch.empty(rows, QKV, dtype=bf, device=DEV),
         "q": torch.empty(rows, H, dtype=bf, device=DEV), "att": torch.empty(rows, H, dtype=bf, device=DEV),
         "gu": torch.empty(rows, 2 * I, dtype=bf, device=DEV), "n8": torch.empty(rows, H, dtype=torch.uint8, device=DEV),
         "a8": torch.empty(rows, H, dtype=torch.uint8, device=DEV), "act8": torch.empty(rows, I, dtype=torch.uint8, device=DEV),
         "s": torch.empty(4, 2, device=DEV)}
    scratch = torch.empty(max(need, 16), dtype=torch.uint8, device=DEV)
    sc = 1 / 89.6 / 64

    def step():
        s = b["s"]
        b["hid"].copy_(hid0)
        rc = k.add_rmsnorm_fp8(b["hid"], None, norm, 1e-5, 0.22, n_fp8=b["n8"], scale_amax=s[0])
        rc |= k.gemm_fp8(b["n8"], w["qkv"], b["qkv"], a_scale=s[0], w_scales=(4 * sc, 4 * sc, sc), segs=(H, H + HK * D))
        rc |= k.rope_kv_int8_paged(b["qkv"], tables.cos, tables.sin, pos, kv_rows, HQ, HK, D, pool, 1024, 1, b["q"], ck, cv,
                                   ks, vs)
        if tree:
            rc |= k.attn_split_int8(b["q"], ck, cv, ks, vs, 1 / 128, HQ, HK, D, pool, b["att"], max_len=slots, row_pos=pos,
                                    row_pt=row_pt, row_grp=grp, row_tbase=tbase, row_tail=tail, scratch=scratch)
        else:
            rc |= k.attn_decode_int8_paged(b["q"], ck, cv, ks, vs, pos, HQ, HK, D, pool, slots, 1 / 128, b["att"],
                                           row_pt=row_pt, scratch=scratch)
        rc |= k.fp8_quant(b["att"], b["a8"], s[1])
        rc |= k.gemm_fp8(b["a8"], w["o"], b["hid"], a_scale=s[1], w_scales=(sc,), residual=b["hid"], resid_scale=0.22)
        rc |= k.add_rmsnorm_fp8(b["hid"], None, norm, 1e-5, 0.22, n_fp8=b["n8"], scale_amax=s[2])
        rc |= k.gemm_fp8(b["n8"], w["gate_up"], b["gu"], a_scale=s[2], w_scales=(sc,))
        rc |= k.swiglu_fp8(b["gu"][:, :I], b["gu"][:, I:], None, b["act8"], s[3], ld=2 * I)
        rc |= k.gemm_fp8(b["act8"], w["down"], b["hid"], a_scale=s[3], w_scales=(sc,), residual=b["hid"], resid_scale=0.22)
        assert rc == 0
    return step, {**b, "k": ck, "v": cv, "ks": ks, "vs": vs}, [*b.values(), scratch], (table, row_pt, tables)


@pytest.mark.parametrize("rows,tree", [(1, False), (8, False), (16, False), (4, True), (15, True)])
@pytest.mark.parametrize("graph", [False, True])
def test_a_decode_layer_repeats_to_the_bit(rows, tree, graph):
    step, outputs, poisoned, keep = layer(rows, tree)
    step()
    torch.cuda.synchronize()
    want = {name: t.clone() for name, t in outputs.items()}
    assert want["hid"].isfinite().all()
    run = step
    if graph:
        captured = torch.cuda.CUDAGraph()
        with torch.cuda.graph(captured):
            step()
        run = captured.replay
    differs = torch.zeros(len(want), dtype=torch.int64, device=DEV)
    for i in range(40):
        for t in poisoned:
            t.view(torch.uint8).fill_((0xFF, 0x00, 0x5A, 0x3C)[i % 4])
        for _ in range(1 + i % 2):
            run()
        differs += torch.stack([(outputs[n].view(torch.uint8) != want[n].view(torch.uint8)).sum() for n in want])
    assert not differs.any(), dict(zip(want, differs.tolist()))
    del keep
