"""GPU: the kernels of a block's decode step may run beside one another; results equal the layers called one by one, also when a
layer reads what the layer before it writes (then they take turns), and everything is complete for a kernel behind the block."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

NK, NV, HD, TAPS = 16, 32, 128, 4
CONV = (2 * NK + NV) * HD


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
