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
