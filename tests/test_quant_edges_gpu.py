"""GPU: the quantiser's index lookups and packed arithmetic where they can go wrong - values within an ulp of every codeword
midpoint, scales at the limits of f32 and f16, every dtype, odd lengths and buffers that are not 16-byte aligned - bit for bit
against the CPU specification; and the rotation over shapes that do not fill its blocks."""
import numpy as np
import pytest
import torch

from oracle import attention_ref as ar
from oracle import quant_ref as qr
from tests.util import no_device_error

pytestmark = pytest.mark.gpu


def _check(cuda, x, kind, block, f16):
    from hyprstream_b200 import ops

    codes, amax = ops.quantize_blockwise(x, kind, block, int(f16))
    want, wanta = qr.quantize(x.float().cpu().numpy(), kind, block, f16)
    assert np.array_equal(codes.cpu().numpy(), want)
    assert np.array_equal(amax.cpu().numpy(), wanta)
    for dt in (torch.bfloat16, torch.float16, torch.float32):
        got = ops.dequantize_blockwise(codes, amax, kind, x.numel(), block, dt)
        ref = torch.from_numpy(qr.dequantize(want, wanta, kind, x.numel(), block)).to(dt)
        assert torch.equal(got.cpu(), ref), dt


@pytest.mark.parametrize("kind", [1, 2, 3])
@pytest.mark.parametrize("f16", [False, True])
def test_values_at_every_midpoint(cuda, kind, f16):
    """The f32 midpoint itself, its neighbours and values up to 64 ulp away, in blocks whose largest value is 1 or not a power of two."""
    mid = qr.midpoints(kind).astype(np.float32)
    rows = []
    for amax in (np.float32(1.0), np.float32(0.7), np.float32(3.1), np.float32(-1000.5)):
        a = abs(amax)
        for k in (0, 1, -1, 2, -2, 5, -5, 64, -64):
            v = mid * np.float32(a)
            v = (v.view(np.int32) + np.where(v == 0, 0, k).astype(np.int32)).view(np.float32)
            for i in range(0, len(v), 63):
                rows.append(np.concatenate([[amax], np.resize(v[i:i + 63], 63)]).astype(np.float32))
    x = torch.from_numpy(np.concatenate(rows)).to(cuda)
    _check(cuda, x, kind, 64, f16)


@pytest.mark.parametrize("kind", [1, 2, 3])
@pytest.mark.parametrize("f16", [False, True])
def test_scales_at_the_limits(cuda, kind, f16):
    g = torch.Generator().manual_seed(kind)
    x = torch.rand(12, 64, generator=g) * 1.9 - 0.95
    x = torch.where(x.abs() < 1e-3, 0.5, x)
    x[:, 7] = 1.0
    top = torch.tensor([65504.0, 65519.0, 65521.0, 1e5, 3e38, 1e-40, 2e-39, 3e-39, 6.1e-5, 8.9e-8, 3.1e-8, 1.0])
    _check(cuda, (x * top[:, None]).flatten().to(cuda), kind, 64, f16)


@pytest.mark.parametrize("kind", [1, 2, 3])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("block,n", [(64, 1), (64, 8191), (128, 8193), (256, 24577), (64, 40009)])
def test_odd_lengths_and_alignment(cuda, kind, dt, block, n):
    from hyprstream_b200 import ops

    x = torch.randn(n + 1, generator=torch.Generator().manual_seed(n)).to(dt).to(cuda)
    _check(cuda, x[:n], kind, block, False)
    _check(cuda, x[1:], kind, block, True)  # not 16-byte aligned: element-wise loads
    codes, amax = ops.quantize_blockwise(x[:n], kind, block)
    shifted = torch.empty(codes.numel() + 1, dtype=torch.uint8, device=cuda)[1:]
    shifted.copy_(codes)
    assert torch.equal(ops.dequantize_blockwise(shifted, amax, kind, n, block, dt), ops.dequantize_blockwise(codes, amax, kind, n, block, dt))


@pytest.mark.parametrize("rows,heads,dim,rotary", [(1, 1, 16, 16), (7, 3, 40, 16), (301, 5, 72, 64), (3000, 32, 64, 64), (97, 300, 128, 128), (5, 2, 256, 64)])
def test_rope_block_edges(cuda, rows, heads, dim, rotary):
    from hyprstream_b200 import ops

    g = torch.Generator().manual_seed(rows)
    x = torch.randn(rows, heads, dim, generator=g).bfloat16()
    sin, cos = ar.rope_tables(rotary, 10000.0, 512, torch.bfloat16)
    pos = torch.randint(0, 512, (rows,), generator=g)
    got = ops.rope_apply(x.to(cuda), sin.to(cuda), cos.to(cuda), pos.to(torch.int32).to(cuda), rotary)
    assert torch.equal(got.cpu(), ar.apply_partial_rope(x, sin, cos, pos, rotary))
    no_device_error()
