"""Prompts give the same bits every time: the order of every sum is fixed by the launch, not by timing, so the bar is equality."""
import numpy as np
import pytest

import lapid_b200 as lp
from lapid_b200 import tp
from lapid_b200.backend import DType, matmul_id_launch
from oracle import oracle as O

pytestmark = pytest.mark.gpu

MIXES = {"q4_k_m": lambda p, i: tp.q4km_format(p, i, 2), "q5_k": lambda p, i: int(DType.Q5K)}


def _weights(be, fmt, n, k, seed, std=0.04):
    import torch
    out = torch.zeros(tp.layout_total(fmt, n, k), dtype=torch.uint8, device="cuda")
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    w = torch.randn(n * k, device="cuda", generator=g).mul_(std)
    torch.cuda.synchronize()
    be.quantize_into(fmt, be.wrap_tensor(w), n, k, be.wrap_tensor(out))
    return out


def _device(**options):
    import torch
    be = lp.Backend(0)
    for key, value in options.items():
        be.set_option(key, value)
    stream = torch.cuda.Stream()
    be.set_stream(stream.cuda_stream)
    return be, stream


def _stack(be, shape, m, mix, fuse_act, weights=None):
    formats = [{p: MIXES[mix](p, i) for p in ("q", "k", "v", "o", "gate", "up", "down")} for i in range(2)]
    if weights is None:
        weights = [{p: _weights(be, f[p], n, k, 500 + 10 * i + j) for j, (p, n, k, _) in enumerate(shape.projections())}
                   for i, f in enumerate(formats)]
    return tp.GpuTpLayers(be, shape, 1, 0, m, weights, formats, fuse_act=fuse_act), weights


@pytest.mark.parametrize("m,layers", [(77, 6), (2048, 2)])
@pytest.mark.parametrize("mix", ["q4_k_m", "q5_k"])
def test_prompt_repeats_bit_for_bit(mix, m, layers):
    """A prompt through layers whose launches have more tiles than SMs (2048 rows) or are split over K (77 rows), twenty times with inputs in turn;
    nothing waits between the launches of a pass, nor between passes."""
    import torch
    be, stream = _device()
    shape = tp.LayerShape(4096, 32, 8, 128, 11008)
    ours, _ = _stack(be, shape, m, mix, False)
    inputs = [torch.from_numpy(O.normal(900 + i, m * shape.d_model).reshape(m, -1)).cuda() for i in range(2)]
    torch.cuda.synchronize()
    outs = []
    with torch.cuda.stream(stream):
        for rep in range(20):
            ours.h.copy_(inputs[rep % 2])
            out = ours.token(layers)
            if rep < 2:
                outs.append(out.clone())
            else:
                outs.append((out != outs[rep % 2]).any())
    stream.synchronize()
    be.synchronize()
    assert torch.isfinite(outs[0]).all() and not torch.equal(outs[0], outs[1])
    assert not any(bool(v) for v in outs[2:]), outs[2:]


def test_expert_prompt_repeats_bit_for_bit():
    """Gate, up, SwiGLU and down of a mixture-of-experts block on the tensor cores, twenty times without a wait in between."""
    import torch
    be, stream = _device()
    t, r, e, n, k = 512, 8, 64, 768, 2048
    fmt = int(DType.Q4K)
    gate, up, down = (_weights(be, fmt, e * a, b, 950 + i) for i, (a, b) in enumerate(((n, k), (n, k), (k, n))))
    x = torch.from_numpy(O.normal(960, t * k).reshape(t, k)).cuda()
    rng = np.random.default_rng(3)
    ids = torch.from_numpy(np.stack([rng.permutation(e)[:r] for _ in range(t)]).astype(np.int32)).cuda()
    mid, out = [torch.zeros(t * r, n, device="cuda") for _ in range(3)], torch.zeros(t * r, k, device="cuda")
    torch.cuda.synchronize()
    bufs = [be.wrap_tensor(v) for v in (x, ids, gate, up, down, *mid, out)]
    first = [matmul_id_launch(fmt, t, r, e, n, k, inputs=(0, 2 + i, 1), output=5 + i) for i in (0, 1)]
    second = [matmul_id_launch(fmt, t * r, 1, e, k, n, inputs=(7, 4, 1), output=8)]
    want, differ = None, []
    with torch.cuda.stream(stream):
        for rep in range(20):
            be.execute_async(first, bufs)
            be.silu_mul(bufs[5], bufs[6], bufs[7], t * r * n)
            be.execute_async(second, bufs)
            if want is None:
                want = out.clone()
            else:
                differ.append((out != want).any())
    stream.synchronize()
    be.synchronize()
    assert torch.isfinite(want).all() and not any(bool(v) for v in differ), differ
