"""GPU: head_dim 64 prefill on the tcgen05 kernel at the edges of its 128-row tiles and 256-row blocks, behind a prefix, with a
gate, for several query groups; and an output buffer that only the mma.sync kernel can store to."""
import ctypes

import pytest
import torch

from oracle import attention_ref as ar
from tests.util import assert_close_attn, no_device_error

pytestmark = pytest.mark.gpu


def _rand(b, ql, kl, hq, hkv, d, seed):
    g = torch.Generator().manual_seed(seed)
    return tuple(torch.randn(b, n, h, d, generator=g).bfloat16() for n, h in ((ql, hq), (kl, hkv), (kl, hkv)))


@pytest.mark.parametrize("ql,kl", [(2, 2), (127, 127), (128, 128), (129, 129), (255, 300), (257, 257), (5, 1000), (700, 1111)])
@pytest.mark.parametrize("hq,hkv", [(4, 4), (8, 1)])
def test_head_dim_64(cuda, ql, kl, hq, hkv):
    from hyprstream_b200 import ops

    q, k, v = _rand(2, ql, kl, hq, hkv, 64, seed=ql + hq)
    out = ops.prefill_attention(q.to(cuda), k.to(cuda), v.to(cuda))
    torch.cuda.synchronize()
    assert_close_attn(out, ar.attention_fp32(q, k, v), f"{ql} of {kl}")
    no_device_error()


def test_head_dim_64_gate(cuda):
    from hyprstream_b200 import ops

    q, k, v = _rand(1, 300, 300, 4, 2, 64, seed=1)
    gate = torch.randn(1, 300, 4, 64, generator=torch.Generator().manual_seed(2)).bfloat16()
    out = ops.prefill_attention(q.to(cuda), k.to(cuda), v.to(cuda), gate=gate.to(cuda))
    assert_close_attn(out, ar.attention_fp32(q, k, v) * gate.float().sigmoid(), "gated")


@pytest.mark.parametrize("d", [64, 128, 256])
def test_output_aligned_to_four_bytes(cuda, d):
    from hyprstream_b200 import ffi, ops

    q, k, v = (t.to(cuda) for t in _rand(1, 200, 200, 4, 2, d, seed=d))
    want = ops.prefill_attention(q, k, v)
    buf = torch.zeros(q.numel() + 8, dtype=torch.bfloat16, device=cuda)
    out = buf[2:2 + q.numel()]
    ffi.check(ffi.lib.hs_attn_prefill_causal(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), None, 1, 200, 200, 4, 2, d,
                                             ctypes.c_float(d ** -0.5), torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert_close_attn(out.view_as(q), want.float().cpu(), "4-byte aligned output")
    assert buf[:2].abs().sum().item() == 0 and buf[2 + q.numel():].abs().sum().item() == 0
