"""GPU: the tensor-core decode kernel over bf16 caches, for every head_dim and query group it serves, at the edges of its
16-token tiles, of its CTA ranges and of pages that are no multiple of a tile."""
import math

import pytest
import torch

from tests.util import no_device_error

pytestmark = pytest.mark.gpu


def _attend64(q, k, v):
    """q [Hq, D], k / v [L, Hkv, D] -> [Hq, D] in float64."""
    hq, d = q.shape
    g = hq // k.shape[1]
    kk, vv = (t.double().repeat_interleave(g, 1) for t in (k, v))
    p = (torch.einsum("hd,lhd->hl", q.double(), kk) / math.sqrt(d)).softmax(-1)
    return torch.einsum("hl,lhd->hd", p, vv)


def _run(cuda, hq, hkv, d, lens, page_tokens, seed, edit=None):
    from hyprstream_b200 import kv_cache as kc
    from hyprstream_b200 import ops

    g = torch.Generator().manual_seed(seed)
    pool = kc.BlockPool(sum((l + page_tokens - 1) // page_tokens for l in lens) + 1, hkv, d, cuda, kind=0, page_tokens=page_tokens) if page_tokens else None
    caches, kvs = [], []
    for i, l in enumerate(lens):
        k, v = (torch.randn(1, l, hkv, d, generator=g).bfloat16() for _ in range(2))
        if edit:
            edit(k, v)
        c = kc.LayerKVCache.new_paged(1 << 20, pool, owner=i) if pool else kc.LayerKVCache(1 << 20, kc.KVQuantType.NONE, hkv, d, cuda)
        c.update(k.to(cuda), v.to(cuda), 0)
        caches.append(c)
        kvs.append((k[0], v[0]))
    q = torch.randn(len(lens), hq, d, generator=g).bfloat16()
    view, keep = kc.make_view(caches)
    out = ops.decode_attention(q.to(cuda), view, torch.tensor(lens, dtype=torch.int32, device=cuda))
    torch.cuda.synchronize()
    return q, kvs, out.cpu()


@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("g", [1, 2, 4, 8])
@pytest.mark.parametrize("hkv,lens,page_tokens", [(2, [1, 15, 16, 17, 33, 300, 1000], 0), (3, [5, 48, 39, 41, 700], 40), (8, [2500], 256)])
def test_bf16_decode_every_shape(cuda, d, g, hkv, lens, page_tokens):
    q, kvs, out = _run(cuda, hkv * g, hkv, d, lens, page_tokens, seed=d + g)
    for r, (k, v) in enumerate(kvs):
        ref = _attend64(q[r], k, v)
        # one rounding to bf16 (2^-9 of the value) on top of probabilities that carry 16 bits (2^-16 of values up to ~5)
        err = (out[r].double() - ref).abs()
        assert (err <= ref.abs() * 2.0 ** -8 + 5e-4).all(), (lens[r], err.max().item())
    no_device_error()


@pytest.mark.parametrize("g", [2, 8])
def test_bf16_decode_infinite_value(cuda, g):
    """An infinite V element reaches the output of its column as an infinity, and no other column."""
    def edit(k, v):
        v[0, 3, 0, 5] = math.inf
        v[0, 4, 1, 9] = -math.inf
    q, kvs, out = _run(cuda, 2 * g, 2, 128, [20], 0, seed=3, edit=edit)
    o = out[0].float().view(2, g, 128)
    assert (o[0, :, 5] == math.inf).all() and (o[1, :, 9] == -math.inf).all()
    assert torch.isfinite(o).sum().item() == o.numel() - 2 * g
