"""GPU: the kernels of a block's decode step may run beside one another; results equal the layers called one by one, also where
layers share buffers (then they take turns), and everything is complete for a kernel behind the block."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

NK, NV, HD, TAPS = 16, 32, 128, 4
CONV = (2 * NK + NV) * HD
HQ, HKV, D, ROT = 16, 2, 256, 64


def _inputs(cuda, n, layers, seed):
    from hyprstream_b200 import ops

    g = torch.Generator(device=cuda).manual_seed(seed)
    r = lambda *s: torch.randn(*s, device=cuda, generator=g)  # noqa: E731
    ls = [ops.GdnLayer((r(CONV, 1, TAPS) * 0.5).bfloat16(), torch.log(torch.rand(NV, device=cuda, generator=g) + 1e-3), r(NV) * 0.3, 1 + 0.1 * r(HD), NK, NV)
          for _ in range(layers)]
    ins = [[r(n, 1, CONV).bfloat16(), r(n, 1, NV, HD).bfloat16(), r(n, 1, NV).bfloat16(), r(n, 1, NV).bfloat16(), r(n, CONV, TAPS - 1).bfloat16(),
            0.1 * r(n, NV, HD, HD)] for _ in range(layers)]
    return ls, ins


@pytest.mark.parametrize("n", [1, 3, 40])
@pytest.mark.parametrize("chained", [False, True])
def test_block_equals_layers_one_by_one(cuda, n, chained):
    from hyprstream_b200 import ffi

    ls, ins = _inputs(cuda, n, 4, seed=n)
    stream = torch.cuda.current_stream().cuda_stream
    results = []
    for whole in (False, True):
        mine = [[t.clone() for t in i] for i in ins]
        ys = [torch.zeros(n, 1, NV, HD, dtype=torch.bfloat16, device=cuda) for _ in ls]
        if chained:  # layer i + 1's gate input is layer i's output
            for i in range(1, len(ls)):
                mine[i][1] = ys[i - 1]
        ws = ls[0].workspace(n, 1, cuda)
        if whole:
            params = (ffi.GdnLayerParams * len(ls))(*[l.params for l in ls])
            ios = (ffi.GdnLayerIO * len(ls))(*[ffi.GdnLayerIO(*[t.data_ptr() for t in m], y.data_ptr()) for m, y in zip(mine, ys)])
            ffi.check(ffi.lib.hs_qwen_block_forward(params, ios, len(ls), None, None, 1, n, 1, ws.data_ptr(), ws.numel(), stream))
        else:
            for l, m, y in zip(ls, mine, ys):
                ffi.check(ffi.lib.hs_gdn_layer_forward(ctypes.byref(l.params), *[t.data_ptr() for t in m], 1, n, 1, y.data_ptr(), ws.data_ptr(), ws.numel(), stream))
        # a kernel behind the block sees every layer's results
        results.append([y + 0 for y in ys] + [t + 0 for m in mine for t in m[4:]])
    assert all(torch.equal(a, b) for a, b in zip(*results))


SHARINGS = ["none", "z of 2 is y of 0", "one rec_state", "one conv_state", "q_proj is y of 0 and 1", "k_proj is y of 2", "v_proj is y of 0", "v_proj is y of 2"]


@pytest.mark.parametrize("n", [1, 3, 40])
@pytest.mark.parametrize("sharing", SHARINGS)
def test_block_with_attention_equals_layers_one_by_one(cuda, n, sharing):
    """Three DeltaNet layers and the attention layer, with a buffer shared between layers that are neighbours or not: outputs, states and
    the cache that the key write may fill beside the other kernels."""
    from hyprstream_b200 import ffi, kv_cache as kc, ops

    ls, ins = _inputs(cuda, n, 3, seed=n + 100)
    g = torch.Generator(device=cuda).manual_seed(n)
    r = lambda *s: torch.randn(*s, device=cuda, generator=g)  # noqa: E731
    attn = ops.QwenAttnLayer(0.1 * r(D), 0.1 * r(D), r(512, ROT // 2).bfloat16(), r(512, ROT // 2).bfloat16(), ROT, HQ, HKV, D)
    old = [[r(1, 300, HKV, D).bfloat16() for _ in range(2)] for _ in range(n)]
    dst = torch.randint(1, 300, (n,), dtype=torch.int32, device=cuda, generator=g)
    proj = [r(n, HQ * 2 * D).bfloat16(), r(n, HKV * D).bfloat16(), r(n, 1, HKV, D).bfloat16()]
    stream = torch.cuda.current_stream().cuda_stream
    results = []
    for whole in (False, True):
        caches = [kc.LayerKVCache(1024, kc.KVQuantType.INT8, HKV, D, cuda, block=128, scale_dtype=1) for _ in range(n)]
        for c, kv in zip(caches, old):
            c.update(*kv, 0)
        view, keep = kc.make_view(caches)
        mine, (q, k, v) = [[t.clone() for t in i] for i in ins], [t.clone() for t in proj]
        ybuf = torch.zeros(3, n, NV * HD, dtype=torch.bfloat16, device=cuda)
        ys = list(ybuf)
        if sharing == "z of 2 is y of 0":
            mine[2][1] = ys[0]
        elif sharing == "one rec_state":
            mine[2][5] = mine[0][5]
        elif sharing == "one conv_state":
            mine[1][4] = mine[0][4]
        elif sharing == "q_proj is y of 0 and 1":  # (as large as two outputs, which lie behind one another)
            q = ybuf[:2]
        elif sharing == "k_proj is y of 2":
            k = ys[2]
        elif sharing.startswith("v_proj"):
            v = ys[int(sharing[-1])]
        ws = torch.empty(max(ls[0].workspace_bytes(n, 1), attn.workspace_bytes(n, 1)), dtype=torch.uint8, device=cuda)
        out = torch.zeros(n, HQ, D, dtype=torch.bfloat16, device=cuda)
        lens = dst + 1
        aio = ffi.QwenAttnIO(q.data_ptr(), k.data_ptr(), v.data_ptr(), ctypes.addressof(view), dst.data_ptr(), dst.data_ptr(), lens.data_ptr(), out.data_ptr())
        if whole:
            params = (ffi.GdnLayerParams * 3)(*[l.params for l in ls])
            ios = (ffi.GdnLayerIO * 3)(*[ffi.GdnLayerIO(*[t.data_ptr() for t in m], y.data_ptr()) for m, y in zip(mine, ys)])
            ffi.check(ffi.lib.hs_qwen_block_forward(params, ios, 3, ctypes.byref(attn.params), ctypes.byref(aio), 1, n, 1, ws.data_ptr(), ws.numel(), stream))
        else:
            for l, m, y in zip(ls, mine, ys):
                ffi.check(ffi.lib.hs_gdn_layer_forward(ctypes.byref(l.params), *[t.data_ptr() for t in m], 1, n, 1, y.data_ptr(), ws.data_ptr(), ws.numel(), stream))
                torch.cuda.synchronize()
            ffi.check(ffi.lib.hs_qwen_attn_layer_forward(ctypes.byref(attn.params), q.data_ptr(), k.data_ptr(), v.data_ptr(), ctypes.byref(view), dst.data_ptr(),
                                                         dst.data_ptr(), lens.data_ptr(), n, 1, out.data_ptr(), ws.data_ptr(), ws.numel(), stream))
        results.append([out + 0, ybuf + 0] + [t + 0 for m in mine for t in m[4:]] + [t for c in caches for t in c.get()])
    assert all(torch.equal(a, b) for a, b in zip(*results))
