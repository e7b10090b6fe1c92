"""What the order of the kernels on the device must not change: steps captured in a CUDA graph and replayed with new inputs give the bits
of the same step run kernel by kernel (option ``pdl`` = 0: no kernel starts before the one in front of it has finished), and prompts
give the same bits every time. The bar is equality throughout: the order of every sum is fixed by the launch, not by timing."""
import numpy as np
import pytest

import lapid_b200 as lp
from lapid_b200 import tp
from lapid_b200.backend import DType, MatView, gather_launch, matmul_id_launch, matmul_launch
from oracle import oracle as O

pytestmark = pytest.mark.gpu

MIXES = {"q4_k_m": lambda p, i: tp.q4km_format(p, i, 2), "q5_k": lambda p, i: int(DType.Q5K), "q6_k": lambda p, i: int(DType.Q6K),
         "int8": lambda p, i: int(DType.Int8), "int4": lambda p, i: int(DType.Int4), "mxfp4": lambda p, i: int(DType.MXFP4)}


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


def _capture(be, stream, queue):
    """`queue` once plainly (scratch, kernel attributes), then as a graph on the stream."""
    import torch
    with torch.cuda.stream(stream):
        queue()
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        be.set_stream(torch.cuda.current_stream().cuda_stream)
        queue()
    be.set_stream(stream.cuda_stream)
    return graph


def _stack(be, shape, m, mix, fuse_act, weights=None):
    formats = [{p: MIXES[mix](p, i) for p in ("q", "k", "v", "o", "gate", "up", "down")} for i in range(2)]
    if weights is None:
        weights = [{p: _weights(be, f[p], n, k, 500 + 10 * i + j) for j, (p, n, k, _) in enumerate(shape.projections())}
                   for i, f in enumerate(formats)]
    return tp.GpuTpLayers(be, shape, 1, 0, m, weights, formats, fuse_act=fuse_act), weights


@pytest.mark.parametrize("fuse_act", [False, True])
@pytest.mark.parametrize("m", [1, 3, 8])
@pytest.mark.parametrize("mix", list(MIXES))
def test_captured_decode_step_gives_the_bits_of_the_serial_one(mix, m, fuse_act):
    """Six layers: rms_norm -> q, k, v -> o -> rms_norm -> gate, up -> silu_mul -> down. Under capture the first kernel of a list
    requests its weights while the glue kernel or the pre-pass in front of it runs, and the later ones read their quantized activations early."""
    import torch
    serial, s0 = _device(pdl="0")
    be, s1 = _device()
    shape = tp.LayerShape(1024, 8, 2, 128, 2048) if fuse_act or mix not in ("int8", "int4") else tp.LayerShape(960, 8, 2, 120, 1888)  # (ragged widths)
    ref, weights = _stack(serial, shape, m, mix, fuse_act)
    ours, _ = _stack(be, shape, m, mix, fuse_act, weights)
    assert not fuse_act or any(l is not None for ls in ours.act_layouts for l in ls)
    inputs = [torch.from_numpy(O.normal(700 + i, m * shape.d_model).reshape(m, -1)).cuda() for i in range(4)]
    torch.cuda.synchronize()
    graph = _capture(be, s1, lambda: ours.token(6))
    wants = []
    for x in inputs:
        with torch.cuda.stream(s0):
            ref.h.copy_(x)
            wants.append(ref.token(6).clone())
        s0.synchronize()
    for rep in range(40):
        i = rep % len(inputs)
        with torch.cuda.stream(s1):
            ours.h.copy_(inputs[i])
            graph.replay()
            got = ours.hw.clone()
        s1.synchronize()
        assert torch.isfinite(got).all() and torch.equal(got, wants[i]), rep
    serial.synchronize()
    be.synchronize()


@pytest.mark.parametrize("fmt", [DType.Q4K, DType.Q6K, DType.Int8, DType.Iq3Xxs])
@pytest.mark.parametrize("m", [1, 4])
def test_captured_weights_written_between_the_glue_kernel_and_the_list(fmt, m):
    """A list behind a glue kernel may request weights early only when nothing stands between the two: here a copy (then a kernel) rewrites
    the weights there, in every replay with other ones."""
    import torch
    be, stream = _device()
    n, k = 2048, 2048
    if fmt == DType.Iq3Xxs:  # (no quantizer: any bytes are a block)
        a_set = [torch.randint(0, 256, (n * k // 256, 98), dtype=torch.uint8, device="cuda") for _ in range(2)]
        for b in a_set:
            b[:, :2] = torch.full((len(b),), 1e-3, device="cuda").half().view(torch.uint8).view(-1, 2)
        a_set = [torch.cat([b.reshape(-1), b.new_zeros(tp.layout_total(int(fmt), n, k) - b.numel())]) for b in a_set]
    else:
        a_set = [_weights(be, int(fmt), n, k, 800 + i) for i in range(2)]
    source, w = a_set[0].clone(), torch.zeros_like(a_set[0])
    x, normed, out = (torch.from_numpy(O.normal(810, m * k).reshape(m, k)).cuda(), torch.zeros(m, k, device="cuda"), torch.zeros(m, n, device="cuda"))
    layout, nbytes = be.act_layout(matmul_launch(fmt, m, n, k))
    qact = torch.zeros(nbytes, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    bufs = [be.wrap_tensor(t) for t in (normed, w, out, qact, x)]
    plain = [matmul_launch(fmt, m, n, k, inputs=(0, 1), output=2)]
    fused = [matmul_launch(fmt, m, n, k, inputs=(3, 1), output=2, a_quantized=True)]
    wants = []
    with torch.cuda.stream(stream):
        be.rms_norm(bufs[4], bufs[0], m, k, qact=bufs[3], layout=layout)
        for a in a_set:
            w.copy_(a)
            be.execute(plain, bufs)
            wants.append(out.clone())
    stream.synchronize()
    assert not torch.equal(wants[0], wants[1])
    for between in (lambda: w.copy_(source), lambda: torch.add(source, 0, out=w)):
        for ls in (plain, fused):
            def queue():
                be.rms_norm(bufs[4], bufs[0], m, k, qact=bufs[3], layout=layout)
                between()
                be.execute_async(ls, bufs)
            graph = _capture(be, stream, queue)
            second = _capture(be, stream, lambda: be.execute_async(ls, bufs))  # no glue kernel of its own capture in front
            for rep in range(20):
                with torch.cuda.stream(stream):
                    source.copy_(a_set[rep % 2])
                    out.zero_()
                    graph.replay()
                    got = out.clone()
                    w.copy_(a_set[(rep + 1) % 2])
                    second.replay()
                    other = out.clone()
                stream.synchronize()
                assert torch.equal(got, wants[rep % 2]) and torch.equal(other, wants[(rep + 1) % 2]), rep
    be.synchronize()


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


@pytest.mark.parametrize("writer_rows", [8, 40, 300])
@pytest.mark.parametrize("fmt", [DType.Int8, DType.Int4, DType.Q4K, DType.Q5K])
@pytest.mark.parametrize("m", [1, 2, 8, 77, 300])
def test_weights_written_by_an_earlier_launch_of_the_list(fmt, m, writer_rows):
    """A launch of the list (decode or prefill on the tensor cores) stores into the packed bytes of a later launch's weights; the f32
    results are taken as the bytes they are, the scales stay. The later launch's activations are clean, so nothing stands between the
    two kernels of a decode launch; its weights must be the written ones, plain and captured."""
    import torch
    per_block = {DType.Int8: 8, DType.Int4: 4, DType.Q4K: 32, DType.Q5K: 32}[fmt]     # floats that a block's packed values take
    first, pitch = {DType.Q4K: (4, 36), DType.Q5K: (12, 44)}.get(fmt, (0, per_block))  # where they lie: floats before them, from block to block
    k = 1024
    blocks = k // (256 if pitch > per_block else 32)
    n = 4096 if fmt in (DType.Int8, DType.Int4) else 2048
    wn = per_block if pitch > per_block else 1024           # the writer's columns
    rows = n * blocks * per_block // wn                      # ... and the rows that fill every block
    launches = []
    serial, s0 = _device(pdl="0")
    be, s1 = _device()
    w0 = _weights(be, int(fmt), n, k, 990)
    writer = [_weights(be, int(DType.Q4K), wn, 512, 991 + i) for i in range(2)]
    xs = torch.from_numpy(O.normal(992, rows * 512).reshape(rows, 512)).cuda()
    x = torch.from_numpy(O.normal(993, m * k).reshape(m, k)).cuda()
    w, out = w0.clone(), torch.zeros(m, n, device="cuda")
    torch.cuda.synchronize()
    chunk = min(rows, writer_rows)
    # (two blocks of rows are enough: the first fetches of every warp of the later launch lie in them or not)
    for r0 in (0, max(0, rows - chunk)):
        launches.append(matmul_launch(DType.Q4K, chunk, wn, 512, inputs=(0, 1), output=2, a=MatView(r0 * 512, chunk * 512, 512),
                                      out=MatView(first + r0 * wn // per_block * pitch, 0, pitch if pitch > per_block else wn)))
    launches.append(matmul_launch(fmt, m, n, k, inputs=(3, 2), output=4))
    wants = []
    bufs0 = [[serial.wrap_tensor(t) for t in (xs, wr, w, x, out)] for wr in writer]
    for b in bufs0:
        for l in launches:
            serial.execute([l], b)
        wants.append(out.view(torch.int32).clone())
        torch.cuda.synchronize()
    assert not torch.equal(*wants)
    bufs = [[be.wrap_tensor(t) for t in (xs, wr, w, x, out)] for wr in writer]
    graphs = [_capture(be, s1, lambda b=b: be.execute_async(launches, b)) for b in bufs]
    for rep in range(20):
        for run in (lambda: be.execute_async(launches, bufs[rep % 2]), graphs[rep % 2].replay):
            with torch.cuda.stream(s1):
                w.copy_(w0)
                out.zero_()
                run()
                got = out.view(torch.int32).clone()
            s1.synchronize()
            assert torch.equal(got, wants[rep % 2]), rep
    serial.synchronize()
    be.synchronize()


@pytest.mark.parametrize("fmt,m", [(DType.MXFP4, 1), (DType.MXFP4, 3), (DType.MXFP4, 8), (DType.Iq3Xxs, 3), (DType.Iq3Xxs, 8)])
def test_captured_weights_written_between_on_both_kernels(fmt, m):
    """The same for MXFP4 and the i-quants at row counts that take the other of their two kernels."""
    test_captured_weights_written_between_the_glue_kernel_and_the_list(fmt, m)


@pytest.mark.parametrize("fmt", [DType.MXFP4, DType.Iq2Xxs])
@pytest.mark.parametrize("m", [1, 3, 8])
def test_decode_weights_copied_by_a_gather_of_the_list(fmt, m):
    """A Gather (of one f32 row: it copies bytes) writes the weights of two decode launches that share a kernel: they must read the copied ones."""
    import torch
    serial, s0 = _device(pdl="0")
    be, s1 = _device()
    n, k = 2048, 2048
    if fmt == DType.MXFP4:
        sets = [_weights(be, int(fmt), n, k, 1100 + i) for i in range(2)]
    else:
        sets = [torch.randint(0, 256, (n * k // 256, 66), dtype=torch.uint8, device="cuda") for _ in range(2)]
        for b in sets:
            b[:, :2] = torch.full((len(b),), 1e-3, device="cuda").half().view(torch.uint8).view(-1, 2)
        sets = [torch.cat([b.reshape(-1), b.new_zeros(tp.layout_total(int(fmt), n, k) - b.numel())]) for b in sets]
    other = sets[0].clone()
    source, w = sets[0].clone(), torch.zeros_like(sets[0])
    x, outs = torch.from_numpy(O.normal(1110, m * k).reshape(m, k)).cuda(), [torch.zeros(m, n, device="cuda") for _ in range(2)]
    row = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ls = [gather_launch(DType.F32, 1, w.numel() // 4, 1, inputs=(3, 4), output=1), matmul_launch(fmt, m, n, k, inputs=(0, 5), output=6),
          matmul_launch(fmt, m, n, k, inputs=(0, 1), output=2)]
    tensors = (x, w, outs[0], source, row, other, outs[1])
    wants = []
    for a in sets:
        source.copy_(a)
        torch.cuda.synchronize()
        serial.execute(ls, [serial.wrap_tensor(t) for t in tensors])
        wants.append(outs[0].clone())
    assert not torch.equal(*wants)
    bufs = [be.wrap_tensor(t) for t in tensors]
    torch.cuda.synchronize()
    graph = _capture(be, s1, lambda: be.execute_async(ls, bufs))
    for rep in range(20):
        for run in (lambda: be.execute_async(ls, bufs), graph.replay):
            with torch.cuda.stream(s1):
                source.copy_(sets[rep % 2])
                outs[0].zero_()
                run()
                got = outs[0].clone()
            s1.synchronize()
            assert torch.equal(got, wants[rep % 2]), rep
    serial.synchronize()
    be.synchronize()


@pytest.mark.parametrize("how", ["copy", "kernel", "gather"])
@pytest.mark.parametrize("fmt", [DType.Q4K, DType.Q6K])
@pytest.mark.parametrize("m", [77, 300])
def test_prefill_weights_rewritten_right_before_the_launch(fmt, m, how):
    """Weights that a copy or a kernel in front of the list, or a Gather (which copies bytes) in front of the launch, has just rewritten: the tensor-core
    kernel requests packed weights before its dependency wait, and must get the new ones."""
    import torch
    serial, s0 = _device(pdl="0")
    be, s1 = _device()
    n, k = 1024, 2048
    sets = [_weights(be, int(fmt), n, k, 1000 + i) for i in range(2)]
    source, w = sets[0].clone(), torch.zeros_like(sets[0])
    x, out = torch.from_numpy(O.normal(1010, m * k).reshape(m, k)).cuda(), torch.zeros(m, n, device="cuda")
    row = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    launch = matmul_launch(fmt, m, n, k, inputs=(0, 1), output=2)
    ls = [gather_launch(DType.F32, 1, w.numel() // 4, 1, inputs=(3, 4), output=1), launch] if how == "gather" else [launch]
    wants = []
    for a in sets:
        serial.execute([launch], [serial.wrap_tensor(t) for t in (x, a, out)])
        wants.append(out.clone())
        torch.cuda.synchronize()
    assert not torch.equal(*wants)
    bufs = [be.wrap_tensor(t) for t in (x, w, out, source, row)]

    def queue():
        if how == "copy":
            w.copy_(source)
        elif how == "kernel":
            torch.add(source, 0, out=w)
        be.execute_async(ls, bufs)

    graph = _capture(be, s1, queue)
    for rep in range(20):
        for run in (queue, graph.replay):
            with torch.cuda.stream(s1):
                source.copy_(sets[rep % 2])
                w.copy_(sets[(rep + 1) % 2])
                out.zero_()
                run()
                got = out.clone()
            s1.synchronize()
            assert torch.equal(got, wants[rep % 2]), rep
    serial.synchronize()
    be.synchronize()


@pytest.mark.parametrize("m", [77, 300])
def test_prefill_with_a_shared_copy_behind_an_early_decode_launch(m):
    """Two prefill launches of one operand share its bf16 copy; a decode launch between them lets the second start before it has waited itself.
    The copy and both results have the bits of the serial order."""
    import torch
    serial, s0 = _device(pdl="0")
    be, s1 = _device()
    n, k = 1024, 2048
    w1, w2, wd = (_weights(be, int(DType.Q4K), n, k, 1020 + i) for i in range(3))
    inputs = [torch.from_numpy(O.normal(1030 + i, m * k).reshape(m, k)).cuda() for i in range(2)]
    x, xd = torch.zeros(m, k, device="cuda"), torch.from_numpy(O.normal(1040, k).reshape(1, k)).cuda()
    outs = [torch.zeros(r, n, device="cuda") for r in (m, m, 1)]
    torch.cuda.synchronize()
    ls = [matmul_launch(DType.Q4K, m, n, k, inputs=(0, 1), output=5), matmul_launch(DType.Q4K, 1, n, k, inputs=(4, 3), output=7),
          matmul_launch(DType.Q4K, m, n, k, inputs=(0, 2), output=6)]
    tensors = (x, w1, w2, wd, xd, *outs)
    wants = []
    for a in inputs:
        x.copy_(a)
        torch.cuda.synchronize()
        for l in ls:
            serial.execute([l], [serial.wrap_tensor(t) for t in tensors])
        wants.append([o.clone() for o in outs])
        torch.cuda.synchronize()
    bufs = [be.wrap_tensor(t) for t in tensors]
    graph = _capture(be, s1, lambda: be.execute_async(ls, bufs))
    for rep in range(20):
        for run in (lambda: be.execute_async(ls, bufs), graph.replay):
            with torch.cuda.stream(s1):
                x.copy_(inputs[rep % 2])
                for o in outs:
                    o.zero_()
                run()
                got = [o.clone() for o in outs]
            s1.synchronize()
            assert all(torch.equal(a, b) for a, b in zip(got, wants[rep % 2])), rep
    serial.synchronize()
    be.synchronize()


def test_prefill_behind_a_launch_that_takes_long():
    """Two launches share their operand's copy, and the first keeps one SM busy for tens of milliseconds (one tile, K not split): the second, which
    starts beside it, must wait that long for its activations and not give up."""
    import torch
    be, stream = _device(gemm_splitk="0")
    m, n, k = 9, 128, 1 << 24
    w = torch.randint(0, 256, (n * k // 256, 144), dtype=torch.uint8, device="cuda")
    w[:, :4] = torch.full((len(w), 2), 1e-4, device="cuda").half().view(torch.uint8)
    x = torch.randn(m, k, device="cuda")
    outs = [torch.zeros(m, n, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    bufs = [be.wrap_tensor(t) for t in (x, w.reshape(-1), *outs)]
    ls = [matmul_launch(DType.Q4K, m, n, k, inputs=(0, 1), output=2 + i) for i in range(2)]
    be.execute(ls, bufs)
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with torch.cuda.stream(stream):
        start.record()
        be.execute_async(ls[:1], bufs)
        end.record()
    be.execute(ls, bufs)
    assert start.elapsed_time(end) > 20
    assert torch.isfinite(outs[0]).all() and outs[0].any() and torch.equal(*outs)


@pytest.mark.parametrize("chunk", [0, 1, 2])
@pytest.mark.parametrize("m", [77, 300])
def test_prefill_with_uploads_between_the_launches(m, chunk):
    """A prefill step with host buffers: activations and packed weights come up on the copy stream while launches of earlier chunks run; the weights
    that a launch requests before its dependency wait must be the uploaded ones."""
    import torch
    serial, s0 = _device(pdl="0")
    be, s1 = _device()
    n, k = 1024, 2048
    sets = [[_weights(be, int(DType.Q4K), n, k, 1050 + 2 * i + j) for j in range(2)] for i in range(2)]
    xs = [[torch.from_numpy(O.normal(1060 + 2 * i + j, m * k).reshape(m, k)).cuda() for j in range(2)] for i in range(2)]
    dev = [torch.zeros_like(t) for t in (*xs[0], *sets[0])] + [torch.zeros(m, n, device="cuda") for _ in range(3)]
    host = [[t.cpu().pin_memory() for t in (*xs[i], *sets[i])] for i in range(2)]
    outs = [torch.zeros(m, n).pin_memory() for _ in range(3)]
    torch.cuda.synchronize()
    ls = [matmul_launch(DType.Q4K, m, n, k, inputs=(0, 2), output=4), matmul_launch(DType.Q4K, m, n, k, inputs=(0, 3), output=5),
          matmul_launch(DType.Q4K, m, n, k, inputs=(1, 2), output=6)]
    wants = []
    for i in range(2):
        bufs = [serial.wrap_tensor(t) for t in (*xs[i], *sets[i], *dev[4:])]
        for l in ls:
            serial.execute([l], bufs)
        wants.append([t.cpu() for t in dev[4:]])
    bufs = [be.wrap_tensor(t) for t in dev]
    size = [t.numel() * t.element_size() for t in dev]
    for rep in range(20):
        h = host[rep % 2]
        writes = [(b, 0, h[b].data_ptr(), size[b], first) for b, first in ((0, 0), (2, 0), (3, 1), (1, 2))]
        reads = [(4 + i, 0, outs[i].data_ptr(), size[4 + i], i) for i in range(3)]
        be.execute_io(ls, bufs, writes, reads, chunk)
        assert all(torch.equal(a, b) for a, b in zip(outs, wants[rep % 2])), rep
    serial.synchronize()
    be.synchronize()
