"""GPU: the tensor-core decode kernel for every kind, head_dim, scale block and query group it serves, at the edges of its 16-token
tiles, of its CTA ranges and of pages that are no multiple of a tile; and code pages that are aligned to words only."""
import ctypes
import math

import pytest
import torch

from oracle import quant_ref as qr
from tests.util import no_device_error

pytestmark = pytest.mark.gpu


def _attend64(q, k, v):
    """q [Hq, D], k / v [L, Hkv, D] -> [Hq, D] in float64."""
    hq, d = q.shape
    g = hq // k.shape[1]
    kk, vv = (t.double().repeat_interleave(g, 1) for t in (k, v))
    p = (torch.einsum("hd,lhd->hl", q.double(), kk) / math.sqrt(d)).softmax(-1)
    return torch.einsum("hl,lhd->hd", p, vv)


def _stored(t, kind, block, sdt):
    """t as a cache of this kind holds it, in float64."""
    codes, amax = qr.quantize(t.float().numpy(), kind, block, bool(sdt))
    idx = torch.from_numpy(codes).long()
    if kind != 1:
        idx = torch.stack((idx >> 4, idx & 15), 1).flatten()
    book = torch.from_numpy(qr.codebook(kind)).double()
    return (book[idx].view(-1, block) * torch.from_numpy(amax.astype("float64"))[:, None]).view(t.shape)


def _run(cuda, hq, hkv, d, lens, page_tokens, seed, edit=None, kind=0, block=64, sdt=0, shard=False):
    from hyprstream_b200 import kv_cache as kc
    from hyprstream_b200 import ops

    g = torch.Generator().manual_seed(seed)
    pool = kc.BlockPool(sum((l + page_tokens - 1) // page_tokens for l in lens) + 1, hkv, d, cuda, kind=kind, block=block, scale_dtype=sdt,
                        page_tokens=page_tokens) if page_tokens else None
    caches, kvs = [], []
    for i, l in enumerate(lens):
        k, v = (torch.randn(1, l, hkv, d, generator=g).bfloat16() for _ in range(2))
        if edit:
            edit(k, v)
        c = kc.LayerKVCache.new_paged(1 << 20, pool, owner=i) if pool else kc.LayerKVCache(
            1 << 20, kc.KVQuantType(kind), hkv, d, cuda, block=block, scale_dtype=sdt)
        c.update(k.to(cuda), v.to(cuda), 0)
        caches.append(c)
        kvs.append((k[0], v[0]) if kind == 0 else tuple(_stored(t, kind, block, sdt) for t in (k[0], v[0])))
    q = torch.randn(len(lens), hq, d, generator=g).bfloat16()
    view, keep = kc.make_view(caches)
    out = ops.decode_attention(q.to(cuda), view, torch.tensor(lens, dtype=torch.int32, device=cuda), shard=shard)
    torch.cuda.synchronize()
    return q, kvs, tuple(t.cpu() for t in out) if shard else out.cpu()


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


@pytest.mark.parametrize("kind", [1, 2, 3])
@pytest.mark.parametrize("d,block,sdt", [(64, 64, 0), (64, 64, 1), (128, 64, 0), (128, 128, 1), (256, 64, 1), (256, 128, 0), (256, 256, 0)])
@pytest.mark.parametrize("g", [1, 2, 4, 8])
@pytest.mark.parametrize("hkv,lens,page_tokens", [(2, [1, 15, 17, 33, 300, 1000], 0), (3, [5, 48, 39, 41, 700], 40)])
def test_code_decode_every_shape(cuda, kind, d, block, sdt, g, hkv, lens, page_tokens):
    q, kvs, out = _run(cuda, hkv * g, hkv, d, lens, page_tokens, seed=d + g + kind, kind=kind, block=block, sdt=sdt)
    # the int8 kernel for 2 x 256 heads (group 8, blocks of 64 and 128) holds P in fp16, whose small values are coarser
    fp16_p = (kind, d, g, hkv) == (1, 256, 8, 2) and block < 256
    for r, (k, v) in enumerate(kvs):
        ref = _attend64(q[r], k, v)
        err = (out[r].double() - ref).abs()
        # one rounding to bf16 (2^-9 of the value) on top of probabilities and table values that carry 16 bits
        assert (err <= ref.abs() * 2.0 ** -8 + (4e-3 if fp16_p else 5e-4)).all(), (lens[r], err.max().item())
    no_device_error()


@pytest.mark.parametrize("kind,d,g", [(1, 64, 4), (2, 128, 2), (3, 64, 8)])
@pytest.mark.parametrize("shift", [4, 8])
def test_pages_aligned_to_words(cuda, kind, d, g, shift):
    """Code pages at an address that is a multiple of 4 (8) bytes only give what aligned ones give, bit for bit."""
    from hyprstream_b200 import ffi, ops

    n, hkv, page = 150, 2, 160
    row = (d if kind == 1 else d // 2) * hkv
    gen = torch.Generator().manual_seed(d)
    kv = [torch.randint(0, 256, (page * row,), generator=gen).to(torch.uint8).to(cuda) for _ in range(2)]
    scales = [(torch.rand(page * hkv * (d // 64), generator=gen) + 0.5).to(cuda) for _ in range(2)]
    q = torch.randn(1, hkv * g, d, generator=gen).bfloat16().to(cuda)
    outs = []
    for by in (0, shift):
        bufs = []
        for t in kv:
            b = torch.zeros(t.numel() + 64, dtype=torch.uint8, device=cuda)
            b[by:by + t.numel()] = t
            bufs.append(b)
        tabs = [torch.tensor([p], dtype=torch.int64, device=cuda) for p in (bufs[0].data_ptr() + by, bufs[1].data_ptr() + by,
                                                                            scales[0].data_ptr(), scales[1].data_ptr())]
        view = ffi.KVView(kind, ffi.SCALE_F32, 64, hkv, d, page, 1, 0, *[t.data_ptr() for t in tabs])
        outs.append(ops.decode_attention(q, view, torch.tensor([n], dtype=torch.int32, device=cuda)))
        torch.cuda.synchronize()
    assert torch.equal(outs[0], outs[1])
    no_device_error()


@pytest.mark.parametrize("hq,hkv,d,rotary", [(32, 8, 128, 128), (4, 2, 64, 64), (16, 2, 256, 64), (3, 3, 128, 0)])
@pytest.mark.parametrize("page_tokens", [0, 40, 256])
def test_bf16_step_writes_its_token(cuda, hq, hkv, d, rotary, page_tokens):
    """decode_append without positions (a batch: the tokens are written first, at seq_lens - 1) leaves the same cache and gives the same
    output as with positions, bit for bit - also where the rotation table ends."""
    from hyprstream_b200 import ffi, kv_cache as kc, ops

    lens = [1, 2, 16, 17, 32, 40, 41, 639]
    g = torch.Generator().manual_seed(d + page_tokens)
    q = torch.randn(len(lens), hq, d, generator=g).bfloat16().to(cuda)
    kn, vn = (torch.randn(len(lens), 1, hkv, d, generator=g).bfloat16().to(cuda) for _ in range(2))
    old = [[torch.randn(1, l, hkv, d, generator=g).bfloat16().to(cuda) for _ in range(2)] for l in lens]
    tables = (None, None) if not rotary else tuple(torch.randn(600, rotary // 2, generator=g).bfloat16().to(cuda) for _ in range(2))
    sl = torch.tensor(lens, dtype=torch.int32, device=cuda)
    results = []
    for dst in (sl - 1, None):
        pool = kc.BlockPool(sum((l + page_tokens - 1) // page_tokens for l in lens), hkv, d, cuda, kind=0, page_tokens=page_tokens) if page_tokens else None
        caches = []
        for i, kv in enumerate(old):
            c = kc.LayerKVCache.new_paged(1 << 20, pool, owner=i) if pool else kc.LayerKVCache(1 << 20, kc.KVQuantType.NONE, hkv, d, cuda)
            c.update(*kv, 0)
            caches.append(c)
        view, keep = kc.make_view(caches)
        out = ops.decode_append(q, kn, vn, view, dst, sl, sin=tables[0], cos=tables[1], rotary_dim=rotary)
        torch.cuda.synchronize()
        err = ffi.take_device_error()
        assert err == (ffi.DEVERR_KV_WRITE_RANGE if rotary else 0)  # position 638 is past the 600 rows of the table
        results.append([out] + [t for c in caches for t in c.get()])
    assert all(torch.equal(a, b) for a, b in zip(*results))


def test_bf16_step_without_room_is_recorded(cuda):
    """A length of 0 and one past the view's pages: recorded, nothing written, the other sequences served."""
    from hyprstream_b200 import ffi, kv_cache as kc, ops

    kc0 = [kc.LayerKVCache(64, kc.KVQuantType.NONE, 2, 64, cuda) for _ in range(3)]
    g = torch.Generator().manual_seed(1)
    for c in kc0:
        c.update(*(torch.randn(1, 64, 2, 64, generator=g).bfloat16().to(cuda) for _ in range(2)), 0)
    before = [t.clone() for c in kc0 for t in c.get()]
    view, keep = kc.make_view(kc0)
    q = torch.randn(3, 4, 64, generator=g).bfloat16().to(cuda)
    kn, vn = (torch.randn(3, 1, 2, 64, generator=g).bfloat16().to(cuda) for _ in range(2))
    out = ops.decode_append(q, kn, vn, view, None, torch.tensor([0, 30, 65], dtype=torch.int32, device=cuda))
    torch.cuda.synchronize()
    assert ffi.take_device_error() == ffi.DEVERR_KV_WRITE_RANGE | ffi.DEVERR_DECODE_RANGE
    after = [t for c in kc0 for t in c.get()]
    assert torch.equal(after[0], before[0]) and torch.equal(after[4], before[4]) and torch.equal(after[5], before[5])
    assert torch.equal(after[2][0, 29], kn[1, 0]) and torch.equal(after[3][0, 29], vn[1, 0])
    assert (out[0] == 0).all() and torch.isfinite(out.float()).all()


@pytest.mark.parametrize("kind,hq,hkv,d", [(0, 32, 8, 128), (0, 4, 2, 64), (0, 16, 2, 256), (1, 8, 2, 64), (2, 32, 8, 128)])
@pytest.mark.parametrize("rows", [1, 2, 9])
@pytest.mark.parametrize("positions", [False, True])
def test_append_over_shared_pages(cuda, kind, hq, hkv, d, rows, positions):
    """New tokens of one sequence handed in as rows (lengths L, L + 1, ... over the same pages): every token is in the cache before any
    row attends, as with the write and the attention called one after the other.  rows = 1: a table that lists the new token's page twice."""
    from hyprstream_b200 import ffi, ops

    page, old, pps = 64, 210, 4
    g = torch.Generator().manual_seed(d + rows)
    rnd = lambda *s: torch.randn(*s, generator=g).bfloat16().to(cuda)  # noqa: E731
    k, v, q = rnd(1, old, hkv, d), rnd(1, old, hkv, d), rnd(rows, hq, d)
    kn, vn = rnd(rows, 1, hkv, d), rnd(rows, 1, hkv, d)
    lens = torch.arange(old + 1, old + 1 + rows, dtype=torch.int32, device=cuda)
    results = []
    for append in (False, True):
        row = {0: 2 * d, 1: d}.get(kind, d // 2) * hkv
        bufs = [torch.zeros(pps, page * row, dtype=torch.uint8, device=cuda) for _ in range(2)]
        bufs += [torch.zeros(pps, page * hkv * (d // 64), device=cuda) for _ in range(2 if kind else 0)]
        tabs = [torch.tensor([[t[i].data_ptr() for i in range(pps)]] * rows, dtype=torch.int64, device=cuda) for t in bufs]
        view = ffi.KVView(kind, ffi.SCALE_F32, 64, hkv, d, page, pps, 0, *[t.data_ptr() for t in tabs], *[None] * (4 - len(tabs)))
        ops.kv_quantize_write(view, k, v, torch.zeros(1, dtype=torch.int32, device=cuda))
        if rows == 1:
            for t in tabs:
                t[0, 0] = t[0, old // page]
        if append:
            out = ops.decode_append(q, kn, vn, view, lens - 1 if positions else None, lens)
        else:
            ops.kv_quantize_write(view, kn, vn, lens - 1)
            out = ops.decode_attention(q, view, lens)
        results.append([out] + bufs)
    assert all(torch.equal(a, b) for a, b in zip(*results))
    no_device_error()


@pytest.mark.parametrize("hq,hkv,d,rotary", [(32, 8, 128, 128), (4, 2, 64, 64), (16, 2, 256, 64), (3, 3, 128, 0)])
@pytest.mark.parametrize("length", [1, 2, 16, 17, 32, 63, 64, 639])
def test_bf16_step_of_one_sequence_writes_its_token(cuda, hq, hkv, d, rotary, length):
    """One sequence in one page: the attention kernel writes the token, and cache and output are those of the two kernels, bit for bit -
    also where the rotation table ends."""
    from hyprstream_b200 import ffi, kv_cache as kc, ops

    g = torch.Generator().manual_seed(d + length)
    rnd = lambda *s: torch.randn(*s, generator=g).bfloat16().to(cuda)  # noqa: E731
    q, kn, vn, old = rnd(1, hq, d), rnd(1, 1, hkv, d), rnd(1, 1, hkv, d), [rnd(1, length, hkv, d) for _ in range(2)]
    tables = (None, None) if not rotary else (rnd(600, rotary // 2), rnd(600, rotary // 2))
    sl = torch.tensor([length], dtype=torch.int32, device=cuda)
    results = []
    for dst in (sl - 1, None):
        c = kc.LayerKVCache(1 << 20, kc.KVQuantType.NONE, hkv, d, cuda)
        c.update(*old, 0)
        view, keep = kc.make_view([c])
        n0 = ffi.launch_count()
        out = ops.decode_append(q, kn, vn, view, dst, sl, sin=tables[0], cos=tables[1], rotary_dim=rotary)
        assert ffi.launch_count() - n0 == (2 if dst is None else 3)
        torch.cuda.synchronize()
        assert ffi.take_device_error() == (ffi.DEVERR_KV_WRITE_RANGE if rotary and length > 600 else 0)
        results.append([out, *c.get()])
    assert all(torch.equal(a, b) for a, b in zip(*results))


@pytest.mark.parametrize("kind,hq,hkv,d", [(0, 8, 2, 128), (1, 8, 2, 64), (2, 32, 8, 64), (1, 32, 8, 128)])
def test_append_with_nothing_to_attend(cuda, kind, hq, hkv, d):
    """Positions given and every length 0: no block of the attention has work, and still what follows on the stream sees the tokens that
    the write kernel in front of it stores."""
    from hyprstream_b200 import kv_cache as kc, ops

    n = 64
    g = torch.Generator().manual_seed(d)
    rnd = lambda *s: torch.randn(*s, generator=g).bfloat16().to(cuda)  # noqa: E731
    kn, vn, q = rnd(n, 1, hkv, d), rnd(n, 1, hkv, d), rnd(n, hq, d)
    dst = torch.arange(n, dtype=torch.int32, device=cuda)
    caches = [[kc.LayerKVCache(64, kc.KVQuantType(kind), hkv, d, cuda) for _ in range(n)] for _ in range(2)]
    for c in caches[0] + caches[1]:
        c._ensure_capacity(64)
    (want, keep0), (got, keep1) = (kc.make_view(c) for c in caches)
    full = torch.full((n,), 64, dtype=torch.int32, device=cuda)
    ops.kv_quantize_write(want, kn, vn, dst)
    ref = ops.kv_gather_dequantize(want, full, 64)
    torch.cuda.synchronize()
    for _ in range(5):
        out = ops.decode_append(q, kn, vn, got, dst, torch.zeros(n, dtype=torch.int32, device=cuda))
        seen = ops.kv_gather_dequantize(got, full, 64)
        assert (out == 0).all() and all(torch.equal(a, b) for a, b in zip(ref, seen))
    no_device_error()


@pytest.mark.parametrize("n", [64, 65, 256, 257, 1025])
def test_many_short_sequences(cuda, n):
    """Batches whose lengths the merge sums warp by warp (up to 64) and block-wide (more), sequences of no tokens among them."""
    from hyprstream_b200 import ffi, ops

    hq, hkv, d, page = 4, 2, 64, 48
    g = torch.Generator(device=cuda).manual_seed(n)
    k, v = (torch.randn(n, page, hkv, d, device=cuda, generator=g).bfloat16() for _ in range(2))
    q = torch.randn(n, hq, d, device=cuda, generator=g).bfloat16()
    lens = torch.randint(0, page + 1, (n,), dtype=torch.int32, device=cuda, generator=g)
    tabs = [t.data_ptr() + torch.arange(n, device=cuda) * (page * hkv * d * 2) for t in (k, v)]
    out = ops.decode_attention(q, ffi.KVView(0, 0, 64, hkv, d, page, 1, 0, *[t.data_ptr() for t in tabs], None, None), lens)
    kk, vv = (t.double().repeat_interleave(hq // hkv, 2) for t in (k, v))
    s = torch.einsum("nhd,nlhd->nhl", q.double(), kk) / math.sqrt(d)
    s.masked_fill_(torch.arange(page, device=cuda) >= lens[:, None, None], -math.inf)
    ref = torch.einsum("nhl,nlhd->nhd", s.softmax(-1).nan_to_num(0.0), vv)  # (no tokens: zeros)
    assert ((out.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 5e-4).all()  # as test_bf16_decode_every_shape
    no_device_error()


@pytest.mark.parametrize("d,g", [(64, 2), (128, 1), (128, 8), (256, 4)])
def test_nf4_decode_infinite_value(cuda, d, g):
    """An infinite V element makes its block's scale infinite and its own code the one of -1: the output of its column is an infinity, the rest
    of the block (0 x infinity) NaN, and nothing else is touched."""
    def edit(k, v):
        v[0, 3, 0, 5] = math.inf
        v[0, 4, 1, d - 1] = -math.inf
    q, kvs, out = _run(cuda, 2 * g, 2, d, [20], 0, seed=4, edit=edit, kind=2)
    o = out[0].float().view(2, g, d)
    assert (o[0, :, 5] == -math.inf).all() and (o[1, :, d - 1] == -math.inf).all()
    assert o[0, :, :64].isnan().sum().item() == o[1, :, d - 64:].isnan().sum().item() == 63 * g
    assert torch.isfinite(o).sum().item() == o.numel() - 2 * 64 * g


@pytest.mark.parametrize("kind,d,block", [(0, 64, 64), (0, 128, 64), (0, 256, 64), (1, 64, 64), (1, 128, 128), (1, 256, 256), (2, 64, 64), (2, 128, 128),
                                          (2, 256, 64), (3, 128, 64)])
@pytest.mark.parametrize("g", [1, 2, 4, 8])
def test_shard_results_in_fp32(cuda, kind, d, block, g):
    """fp32 results (a KV-length shard's output and log-sum-exp) are as near to 64 bits as fp32 weights and table values make them.  A
    score of up to 16 (in powers of two) is rounded to 2^-21, exp2f is good to 2 ulp (2^-22): 7e-7 of a weight at worst, 5e-7 of the
    natural logarithm, and one fp32 rounding of a log-sum-exp below 16 on top (5e-7)."""
    lens = [1, 17, 333, 3000]
    q, kvs, (o, lse) = _run(cuda, 2 * g, 2, d, lens, 0, seed=d + g, kind=kind, block=block, shard=True)
    for r, (k, v) in enumerate(kvs):
        ref = _attend64(q[r], k, v)
        s = torch.einsum("hd,lhd->hl", q[r].double(), k.double().repeat_interleave(g, 1)) / math.sqrt(d)
        assert (o[r].double() - ref).norm() <= 7e-7 * ref.norm(), (lens[r], ((o[r].double() - ref).norm() / ref.norm()).item())
        assert (lse[r].double() - s.logsumexp(-1)).abs().max() <= 1.2e-6, lens[r]


@pytest.mark.parametrize("kind", [0, 1, 2])
def test_append_without_lengths_is_refused_untouched(cuda, kind):
    """Neither positions nor lengths: refused, the cache as it was and no device error left behind."""
    from hyprstream_b200 import ffi, kv_cache as kc, ops

    g = torch.Generator().manual_seed(kind)
    kv = [torch.randn(1, 20, 2, 64, generator=g).bfloat16().to(cuda) for _ in range(2)]
    caches = [kc.LayerKVCache(64, kc.KVQuantType(kind), 2, 64, cuda) for _ in range(2)]
    for c in caches:
        c.update(*kv, 0)
    before = [t.clone() for c in caches for t in c.get()]
    view, keep = kc.make_view(caches)
    x = torch.ones(2, 4, 64, dtype=torch.bfloat16, device=cuda)
    ws = ops.decode_workspace(2, 4, 64, cuda)
    st = ffi.lib.hs_attn_decode_append(x.data_ptr(), x.data_ptr(), x.data_ptr(), ctypes.byref(view), None, None, 2, 4, ctypes.c_float(0.125), None, None, 0, 0,
                                       torch.empty_like(x).data_ptr(), None, ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
    assert st == ffi.HS_ERR_ARG
    torch.cuda.synchronize()
    assert ffi.take_device_error() == 0
    assert all(torch.equal(a, b) for a, b in zip(before, [t for c in caches for t in c.get()]))
