"""SiLU in the SwiGLU epilogue (`silu_for_bf16`): the bits of the eager chain bf16(g / (1 + expf(-g))) for every finite
bf16 gate.  One GEMM per exponent and sign makes all 128 mantissas (and, below 2^-126, the subnormals) from exact
products; up is the power of two alpha, so SiLU's own bits come out wherever the product neither over- nor underflows."""
import pytest
import torch

pytestmark = pytest.mark.gpu

CODE = {0.5: 1, 1.0: 2, 2.0: 4, 4.0: 6}        # e2m1
SCALE = {1.0: 0x38, 0.25: 0x28, 2.0 ** -6: 0x08}   # ue4m3


def _pack(codes):
    return (codes[:, 0::2] | (codes[:, 1::2] << 4)).contiguous()


def _scales(rows, blocks):
    """One 512-byte atom per 128 rows (K = 64): byte (r % 32) * 16 + (r // 32 % 4) * 4 + block."""
    r = torch.arange(rows)
    out = torch.zeros((rows // 128 + 1) * 512, dtype=torch.uint8)
    for b, v in enumerate(blocks):
        out[(r // 128) * 512 + (r % 32) * 16 + (r // 32 % 4) * 4 + b] = SCALE[v]
    return out


def test_every_finite_gate():
    from arcquant_b200 import ops

    a = torch.zeros((256, 64), dtype=torch.uint8)
    mant = torch.arange(256) % 128
    a[:128, 0] = CODE[4.0]                                         # the leading one (rows 128.. : subnormals)
    for bit, (col, v) in enumerate([(19, 0.5), (18, 1.0), (17, 2.0), (16, 4.0), (3, 0.5), (2, 1.0), (1, 2.0)]):
        a[:, col] = ((mant >> bit) & 1).to(torch.uint8) * CODE[v]
    a[:, 32] = CODE[1.0]
    b = torch.zeros((256, 64), dtype=torch.uint8)                  # 128 gate rows, 128 up rows
    b[:128, 0:4] = CODE[1.0]
    b[:128, 16:20] = CODE[1.0]
    b[128:, 32] = CODE[1.0]
    sfa, sfb = _scales(256, (0.25, 2.0 ** -6, 1.0, 1.0)).cuda(), _scales(256, (1.0, 1.0, 1.0, 1.0)).cuda()
    a, b = _pack(a).cuda(), _pack(b).cuda()
    value = (mant.double() / 128 + (torch.arange(256) < 128)).cuda()
    for e in range(-126, 128):
        for sign in (1.0, -1.0):
            alpha = torch.tensor(sign * 2.0 ** e, dtype=torch.float32, device="cuda")
            got, amax = ops.matmul_swiglu(a, b, sfa, sfb, alpha, None)
            gate = (value * alpha.double()).to(torch.bfloat16)
            gate_up = torch.cat([gate[:, None].expand(256, 128), alpha.to(torch.bfloat16).expand(256, 128)], 1).contiguous()
            want, amax_w = ops.silu_mul(gate_up)
            assert torch.equal(got.view(torch.int16), want.view(torch.int16)), (e, sign)
            assert float(amax) == float(amax_w)
    assert ops.gemm_poll_error() == 0
