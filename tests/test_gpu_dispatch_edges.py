"""Kernel forms at the sizes where the dispatch changes hands and at the edges of their tiles, against
the CPU oracle (the reference's fp32 formulation) or an exact property."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.fixture(scope="module")
def K():
    import granite4_b200  # noqa: F401
    from granite4_b200 import capi, kernels
    capi.lib()
    yield kernels
    assert capi.lib().device_status() == 0


def dev(a):
    a = np.ascontiguousarray(a)
    return torch.from_numpy(a.view(np.int16) if a.dtype == np.uint16 else a).to(DEV)


# exponents of amax: the ends of the range the two-instruction quantiser takes (2^-100 .. 2^100), one
# beyond each, bf16's own ends and ordinary values
@pytest.mark.parametrize("exponent", [1, 26, 27, 28, 124, 127, 136, 226, 227, 228, 254])
def test_fp8_codes_of_every_bf16_value_under_every_amax_mantissa(K, port, exponent):
    """For each of the 128 mantissas of the tensor's largest magnitude: every bf16 value up to it, both
    signs. Codes, scale and amax equal the oracle's (the reference's exact rule), ties included."""
    for m in range(128):
        top = (exponent << 7) | m
        low = max(0, top - 12 * 128 - 127)  # below, every code is zero; keep a few of those too
        mags = np.concatenate([np.arange(low, top + 1), np.arange(0, min(low, 64))]).astype(np.uint16)
        bits = np.concatenate([mags, mags | 0x8000])
        bits = np.concatenate([bits, np.zeros(-len(bits) % 8, np.uint16)])
        want, scale, amax = port.quant_fp8(bits)
        codes = torch.empty(len(bits), dtype=torch.uint8, device=DEV)
        sa = torch.zeros(2, device=DEV)
        assert K.fp8_quant(dev(bits), codes, sa) == 0
        assert sa[1].item() == amax and sa[0].item() == scale
        got = codes.cpu().numpy()
        assert (got == want).all(), (m, (got != want).sum())


def _exact_gemm_case(K, M, N, Kd, kind, pad=0, in_place=False):
    """Codes from {0, +-1, +-2} make every sum exact in f32, so every form of the GEMM must return the
    integer result exactly (bf16: rounded once), whatever order it adds in."""
    g = torch.Generator(device=DEV).manual_seed(M * 7919 + N * 31 + Kd)
    vals = torch.tensor([0x00, 0x38, 0xB8, 0x40, 0xC0], dtype=torch.uint8, device=DEV)  # 0, 1, -1, 2, -2

    def codes(r, c):
        return vals[torch.randint(5, (r, c), generator=g, device=DEV)]
    a, w = codes(M, Kd), codes(N, Kd)
    num = {0x00: 0.0, 0x38: 1.0, 0xB8: -1.0, 0x40: 2.0, 0xC0: -2.0}
    lut = torch.zeros(256, device=DEV)
    for c, v in num.items():
        lut[c] = v
    want = (lut[a.long()].double() @ lut[w.long()].double().T)
    ldc = (N + 7) // 8 * 8 + pad
    buf = torch.full((M, ldc), 7.0, dtype=torch.float32 if kind == "f32" else torch.bfloat16, device=DEV)
    out = buf[:, :N]
    res = None
    if kind == "residual":
        rbuf = torch.randint(-8, 8, (M, ldc), generator=g, device=DEV).to(torch.bfloat16)
        res = rbuf[:, :N]
        want = want * 0.5 + res.double()
        if in_place:
            rbuf[:, N:] = 7.0
            buf, out = rbuf, res
    ws = K.gemm_fp8_workspace(M, N, Kd, DEV)
    assert K.gemm_fp8(a, w, out, residual=res, resid_scale=0.5, workspace=ws) == 0
    want = want.float() if kind == "f32" else want.float().to(torch.bfloat16)
    assert torch.equal(out, want), (M, N, Kd, kind)
    assert (buf[:, N:] == 7.0).all()  # nothing past column N


# row counts at the edges of the forms and of their 128- / 256-row tiles; widths that plan 64, 128 and 192 columns on
# CTA pairs, with ragged last slabs; K of one block, of more blocks than the ring, not a multiple of 128
@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 33, 128, 129, 255, 256, 257, 500])
@pytest.mark.parametrize("N,Kd", [(72, 128), (1000, 1552), (4096, 512), (6144, 256)])
def test_gemm_forms_are_exact_at_their_edges(K, M, N, Kd):
    for kind in ("bf16", "f32", "residual"):
        _exact_gemm_case(K, M, N, Kd, kind, pad=8 if kind == "residual" else 0)


def planned_width(M, N, pairs=74):
    """Columns of a pair tile (csrc/gemm_fp8.cu plan_pair_columns): rounds of tiles over the pairs x measured time."""
    cost = {w: -(-(-(-M // 256) * -(-N // w)) // pairs) * us for w, us in ((256, 0.33), (192, 0.265), (128, 0.19), (64, 0.16))}
    best = 256
    for w in cost:
        best = w if cost[w] < cost[best] * 0.999 else best
    return best


# every width of a pair tile: one round of tiles and several, ragged rows, the last slab of the last tile ragged
@pytest.mark.parametrize("M,N,width", [(500, 8192, 256), (2100, 6144, 256), (512, 9208, 256), (500, 6136, 192),
                                       (300, 4088, 128), (257, 1000, 64)])
def test_gemm_on_cta_pairs_at_every_tile_width(K, M, N, width):
    assert planned_width(M, N) == width
    for kind in ("bf16", "f32", "residual"):
        _exact_gemm_case(K, M, N, 272, kind, pad=8)
    _exact_gemm_case(K, M, N, 272, "residual", pad=8, in_place=True)


@pytest.mark.parametrize("rows", [1, 2, 3, 5, 8, 9, 15, 16, 17])
@pytest.mark.parametrize("cols", [8, 264, 4096, 8184, 8192])
def test_small_norm_quant_and_swiglu_equal_the_oracle(K, port, rows, cols):
    """The one-launch forms of a decode step (one CTA, or one cluster) and the first row count past them."""
    rng = np.random.default_rng(rows * 10007 + cols)

    def bf(shape, sigma=1.0):
        return ((sigma * rng.standard_normal(shape)).astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
    y, res, w = bf((rows, cols)), bf((rows, cols)), bf(cols, 0.1) + 0  # weights of either sign
    h, n = port.add_rmsnorm(y, res, w, 1e-5, 0.22)
    codes, scale, amax = port.quant_fp8(n)
    ho, no = (torch.empty(rows, cols, dtype=torch.int16, device=DEV) for _ in range(2))
    c8 = torch.empty(rows, cols, dtype=torch.uint8, device=DEV)
    sa, rstd = torch.full((2,), 9.0, device=DEV), torch.empty(rows, device=DEV)
    assert K.add_rmsnorm_fp8(dev(y), dev(res), dev(w), 1e-5, 0.22, ho, no, c8, sa, rstd) == 0
    assert (ho.cpu().numpy().view(np.uint16) == h).all() and (no.cpu().numpy().view(np.uint16) == n).all()
    assert (c8.cpu().numpy() == codes).all() and sa[0].item() == scale and sa[1].item() == amax
    cq, sw, aw = port.quant_fp8(y)
    assert K.fp8_quant(dev(y), c8, sa) == 0
    assert (c8.cpu().numpy() == cq).all() and sa[0].item() == sw and sa[1].item() == aw
    act = torch.empty(rows, cols, dtype=torch.int16, device=DEV)
    assert K.swiglu_fp8(dev(y), dev(res), act, c8, sa) == 0
    got = act.cpu().numpy().view(np.uint16)
    want = port.swiglu((y.astype(np.uint32) << 16).view(np.float32), (res.astype(np.uint32) << 16).view(np.float32))
    key = lambda x: np.where(x & 0x8000, -(x.astype(np.int32) & 0x7FFF), x.astype(np.int32))  # noqa: E731
    assert np.abs(key(got) - key(want)).max() <= 1  # the stated 1 bf16 ulp
    cs, ss, as_ = port.quant_fp8(got)
    assert (c8.cpu().numpy() == cs).all() and sa[0].item() == ss and sa[1].item() == as_


# powers of two on the weights: below, inside and above the range of the two-instruction quantiser
@pytest.mark.parametrize("power", [-118, 0, 108])
@pytest.mark.parametrize("rows,cols", [(17, 520), (20, 4096), (33, 4104)])
def test_two_sweep_norm_under_unusual_scales_equals_the_oracle(K, port, rows, cols, power):
    """More than 16 rows with rstd: the encode sweep reads the hidden state and 1/rms, and takes scales outside the
    quantiser's plain range in a loop of its own."""
    rng = np.random.default_rng(rows * 10007 + cols)

    def bf(x):
        return (np.ascontiguousarray(x, np.float32).view(np.uint32) >> 16).astype(np.uint16)
    y, res = bf(rng.standard_normal((rows, cols))), bf(rng.standard_normal((rows, cols)))
    w = bf(np.ldexp(rng.standard_normal(cols), power))
    h, n = port.add_rmsnorm(y, res, w, 1e-5, 0.22)
    codes, scale, amax = port.quant_fp8(n)
    ho, c8 = torch.empty(rows, cols, dtype=torch.int16, device=DEV), torch.empty(rows, cols, dtype=torch.uint8, device=DEV)
    sa, rstd = torch.full((2,), 9.0, device=DEV), torch.empty(rows, device=DEV)
    assert K.add_rmsnorm_fp8(dev(y), dev(res), dev(w), 1e-5, 0.22, ho, None, c8, sa, rstd) == 0
    assert (ho.cpu().numpy().view(np.uint16) == h).all()
    assert (c8.cpu().numpy() == codes).all() and sa[0].item() == scale and sa[1].item() == amax


@pytest.mark.parametrize("M,inter,Kd", [(1, 32, 128), (17, 96, 1552), (37, 1000, 512), (64, 12800, 256), (96, 6144, 256), (128, 200, 4096)])
def test_fused_swiglu_of_few_rows_equals_gemm_then_swiglu(K, M, inter, Kd):
    fused_swiglu_case(K, M, inter, Kd)


# one tile of 256 columns per CTA pair (stored directly), several, tiles of 128 columns (through slabs), the single
# form, ragged edges
@pytest.mark.parametrize("M,inter,Kd,pair", [(700, 3072, 256, True), (1500, 3000, 256, True), (257, 1000, 1552, True), (300, 12800, 256, True),
                                             (500, 96, 128, True), (129, 1000, 512, False), (300, 3072, 256, False)])
def test_fused_swiglu_of_many_rows_equals_gemm_then_swiglu(K, monkeypatch, M, inter, Kd, pair):
    if not pair:
        monkeypatch.setenv("G4_GEMM_PAIR", "0")
    fused_swiglu_case(K, M, inter, Kd)


@pytest.mark.parametrize("M,inter", [(17, 96), (100, 12800), (257, 1000), (300, 12800), (700, 3072)])
def test_fused_swiglu_amax_is_of_the_rows_that_exist(K, M, inter):
    """An infinite activation scale: the stored values and their maximum are infinite, whatever rows past M would be."""
    a, w = (torch.full((r, 128), 0x38, dtype=torch.uint8, device=DEV) for r in (M, 2 * inter))  # all 1.0
    out, slot = torch.empty(M, inter, dtype=torch.bfloat16, device=DEV), torch.full((2,), 9.0, device=DEV)
    inf = torch.tensor([float("inf"), 0.0], device=DEV)
    assert K.gemm_fp8(a, w, out, a_scale=inf, swiglu_scale_amax=slot) == 0
    both = torch.full((M, inter), float("inf"), device=DEV)
    want, c8, sa = torch.empty_like(out), torch.empty(M, inter, dtype=torch.uint8, device=DEV), torch.zeros(2, device=DEV)
    assert K.swiglu_fp8(both, both, want, c8, sa) == 0
    assert torch.equal(out.view(torch.int16), want.view(torch.int16)) and slot[1].item() == sa[1].item() == float("inf")


def fused_swiglu_case(K, M, inter, Kd):
    """Gate and up rows as two parts of one tile: the f32 sums of these integer operands are exact, so the fused
    epilogue has to give the standalone kernel's bits. Ragged last tiles, K of one block to more than the ring,
    a K that is not whole blocks."""
    g = torch.Generator(device=DEV).manual_seed(M * inter + Kd)
    lut = torch.arange(256, dtype=torch.uint8, device=DEV).view(torch.float8_e4m3fn).float()
    pick = (lut.abs() <= 2) & (lut == lut.round()) & ~lut.isnan()
    codes = pick.nonzero().flatten().to(torch.uint8)
    a = codes[torch.randint(len(codes), (M, Kd), generator=g, device=DEV)].contiguous()
    w = codes[torch.randint(len(codes), (2 * inter, Kd), generator=g, device=DEV)].contiguous()
    both = torch.empty(M, 2 * inter, dtype=torch.float32, device=DEV)
    sc = (2.0 ** -6,)
    assert K.gemm_fp8(a, w, both, w_scales=sc, workspace=K.gemm_fp8_workspace(M, 2 * inter, Kd, DEV)) == 0
    assert torch.equal(both, (lut[a.long()].double() @ lut[w.long()].double().T * sc[0]).float())
    out, slot = torch.empty(M, inter, dtype=torch.bfloat16, device=DEV), torch.full((2,), 9.0, device=DEV)
    assert K.gemm_fp8(a, w, out, w_scales=sc, swiglu_scale_amax=slot) == 0
    want, c8, sa = torch.empty_like(out), torch.empty(M, inter, dtype=torch.uint8, device=DEV), torch.zeros(2, device=DEV)
    assert K.swiglu_fp8(both[:, :inter].contiguous(), both[:, inter:].contiguous(), want, c8, sa) == 0
    assert torch.equal(out, want) and slot[1].item() == sa[1].item()


@pytest.mark.parametrize("M,pair", [(129, True), (256, True), (256, False)])
def test_weights_written_on_the_stream_just_before_the_gemm(K, monkeypatch, M, pair):
    """At more than 128 rows W may come from any operation ahead of the call: it is rewritten for every call, once
    with the quantisation of A between (small tensors, whose launches overlap), once as the operation just before.
    The values are codes of themselves (amax 448, scale 1), so each product is a sum of whole numbers."""
    if not pair:
        monkeypatch.setenv("G4_GEMM_PAIR", "0")
    n, kd, rounds = 256, 256, 40
    g = torch.Generator(device=DEV).manual_seed(M)

    def whole(r):
        x = torch.randint(-2, 3, (rounds, r, kd), generator=g, device=DEV).to(torch.bfloat16)
        x[:, 0, 0] = 448.0
        return x
    a, w = whole(M), whole(n)
    a8, w8 = (torch.empty(r, kd, dtype=torch.uint8, device=DEV) for r in (M, n))
    sa, sw = torch.zeros(2, device=DEV), torch.zeros(2, device=DEV)
    out = torch.zeros(2, rounds, M, n, device=DEV)
    for last_is_w in (0, 1):
        for i in range(rounds):
            ops = [(w[i], w8, sw), (a[i], a8, sa)]
            for x, c, s in (reversed(ops) if last_is_w else ops):
                assert K.fp8_quant(x, c, s) == 0
            assert K.gemm_fp8(a8, w8, out[last_is_w, i], a_scale=sa) == 0
    want = torch.matmul(a.double(), w.double().transpose(1, 2)).float()
    assert torch.equal(out[0], want) and torch.equal(out[1], want)
