"""Workloads of the quantized matmul path: what programs built on this framework have it do.

``listed()`` gives the workloads that are always timed, ``draw(rng)`` more of the same kinds and ranges,
``prepare(case, seed)`` what a program holds before the call (weights, plans, a captured step, inputs),
``run(state)`` one pass through the public entry points, ``work(case)`` the bytes and operations a pass
cannot do without, ``tolerance(case)`` how far another correct implementation may be off.

Kinds (``op``):

  matmul    one projection called by itself: ``Backend.execute`` (waits), any format, activation type and epilogue
  sweep     a step with host buffers: the four projection shapes at one to eight rows, activations copied from and
            results to page-locked host memory, as one ``execute_io`` call
  model     tokens through a decoder: embedding lookup (Gather), the layer stack of ``tp.GpuTpLayers`` and the output
            head. Up to eight rows (decode) the step is captured once in a CUDA graph and replayed, as a serving loop
            does; above (prefill of a prompt) its launches are queued one by one, since prompts differ in length,
            and only the last row goes through the head
  moe       mixture-of-experts blocks (MatMulId): gate and up over the experts each token names, SwiGLU, down
  quantize  a weight matrix on its way in and out: quantize, dequantize, and the import of GGUF blocks for the
            formats that are repacked
"""
import torch

import lapid_b200 as lp
from lapid_b200 import tp
from lapid_b200.backend import DType, Expr, MatView, gather_launch, matmul_id_launch, matmul_launch
from lapid_b200.quant import from_ggml_blocks_into

FMT = {"int8": 4, "int4": 5, "q4_k": 6, "q5_k": 7, "q6_k": 8, "mxfp4": 9, "iq2_xxs": 10, "iq2_s": 11, "iq3_xxs": 12, "iq2_xs": 13}
K_BLOCK = {name: 32 if name in ("int8", "int4", "mxfp4") else 256 for name in FMT}
# i-quant blocks: bytes, and how large a random block's values are over its f16 scale (root mean square)
IQ_BLOCK = {"iq2_xxs": 66, "iq2_s": 82, "iq3_xxs": 98, "iq2_xs": 74}
IQ_RMS = {"iq2_xxs": 57.0, "iq2_s": 57.0, "iq3_xxs": 150.0, "iq2_xs": 57.0}
WEIGHT_STD = 0.02
# what a stack is made of: (most projections, attn_v and the wider ffn_down layers, output head, embedding table)
MIX = {"q4_k_m": ("q4_k", "q6_k", "q6_k", "q4_k"), "q5_k_m": ("q5_k", "q6_k", "q6_k", "q5_k"),
       "int8": ("int8",) * 4, "int4": ("int4", "int4", "int8", "int4"), "mxfp4": ("mxfp4", "mxfp4", "int8", "int8"),
       "iq2": ("iq2_xxs", "iq3_xxs", "q5_k", "q4_k")}
A_DTYPE = {"f32": (DType.F32, torch.float32), "f16": (DType.F16, torch.float16), "bf16": (DType.BF16, torch.bfloat16)}
TENSOR_CORE = ("q4_k", "q5_k", "q6_k")  # above eight rows with bf16 operands; the other formats in exact f32

_stream = None


def stream():
    """The one stream of the program: every state's work is ordered on it."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def listed():
    return [
        # the smallest call: one matrix-vector product, waited for
        {"name": "matvec_q4k", "op": "matmul", "fmt": "q4_k", "m": 1, "n": 4096, "k": 4096, "a": "f32", "epilogue": "none"},
        # a step whose activations live on the host: 16 launches, 1 to 8 rows
        {"name": "sweep_host_q4k", "op": "sweep", "fmt": "q4_k", "d": 4096, "kv": 1024, "ffn": 14336},
        # one token for one user, and for eight at once, through a 32-layer stack in the usual 4-bit mix
        {"name": "decode_q4km_b1", "op": "model", "mix": "q4_k_m", "m": 1, "layers": 32, "d": 4096, "kv": 1024, "ffn": 14336, "vocab": 128256},
        {"name": "decode_q4km_b8", "op": "model", "mix": "q4_k_m", "m": 8, "layers": 32, "d": 4096, "kv": 1024, "ffn": 14336, "vocab": 128256},
        # the 8-bit format with a small batch, on layers whose width is no multiple of 512 and a ragged vocabulary
        {"name": "decode_int8_b3", "op": "model", "mix": "int8", "m": 3, "layers": 12, "d": 2880, "kv": 512, "ffn": 7680, "vocab": 32003},
        # the smallest formats: 2 and 3 bits per weight
        {"name": "decode_iq2_b1", "op": "model", "mix": "iq2", "m": 1, "layers": 8, "d": 4096, "kv": 1024, "ffn": 14336, "vocab": 32000},
        # a short prompt of odd length, and a long one through wide layers
        {"name": "prefill_q4km_m77", "op": "model", "mix": "q4_k_m", "m": 77, "layers": 8, "d": 4096, "kv": 1024, "ffn": 14336, "vocab": 32000},
        {"name": "prefill_q4km_m2048", "op": "model", "mix": "q4_k_m", "m": 2048, "layers": 2, "d": 8192, "kv": 1024, "ffn": 28672, "vocab": 32000},
        # a prompt in the 8-bit format: exact f32 products
        {"name": "prefill_int8_m512", "op": "model", "mix": "int8", "m": 512, "layers": 2, "d": 4096, "kv": 1024, "ffn": 14336, "vocab": 32000},
        # mixture of experts: one token with 6 of 32 experts, a prompt of 512 with 8 of 128
        {"name": "moe_decode_mxfp4", "op": "moe", "fmt": "mxfp4", "t": 1, "r": 6, "e": 32, "n": 2304, "k": 5120, "layers": 4},
        {"name": "moe_prefill_q4k", "op": "moe", "fmt": "q4_k", "t": 512, "r": 8, "e": 128, "n": 768, "k": 2048, "layers": 2},
        # making a model file's matrix and reading it back
        {"name": "quantize_q4k", "op": "quantize", "fmt": "q4_k", "n": 14336, "k": 4096},
    ]


def _log_int(rng, lo, hi, step=1):
    v = lo * (hi / lo) ** rng.random()
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    op = rng.choice(["matmul", "matmul", "sweep", "decode", "decode", "decode", "prefill", "prefill", "moe", "moe", "quantize"])
    if op == "matmul":
        fmt = rng.choice(list(FMT))
        m = _log_int(rng, 1, 700)
        if fmt not in TENSOR_CORE and m > 8:
            m = min(m, 200)
        return {"op": "matmul", "fmt": fmt, "m": m, "n": _log_int(rng, 500, 15000), "k": _log_int(rng, 1024, 14336, K_BLOCK[fmt]),
                "a": rng.choice(list(A_DTYPE)), "epilogue": rng.choice(["none", "bias", "silu"])}
    if op == "sweep":
        return {"op": "sweep", "fmt": rng.choice(["q4_k", "q5_k", "q6_k", "int8", "int4"]), "d": _log_int(rng, 1024, 8192, 256),
                "kv": _log_int(rng, 256, 2048, 64), "ffn": _log_int(rng, 2048, 16384, 256)}
    if op in ("decode", "prefill"):
        mix = rng.choice(list(MIX))
        tc = mix in ("q4_k_m", "q5_k_m")
        d = _log_int(rng, 1024, 8192, 64 if mix in ("int8", "mxfp4", "int4") else 256)
        kv = 64 * _log_int(rng, 4, max(4, d // 256))
        ffn = _log_int(rng, 2 * d, 4 * d, 32 if mix in ("int8", "mxfp4", "int4") else 256)
        vocab = _log_int(rng, 4000, 130000)
        per_layer = 2 * d * d + 2 * kv * d + 3 * d * ffn
        if op == "decode":
            m = rng.randint(1, 8)
            most = int((1.5e9 - d * vocab) / per_layer)
        else:
            m = _log_int(rng, 9, 2048 if tc else 600)
            most = int(min(1.5e9, (1.6e12 if tc else 3e11) / (2 * m)) / per_layer)
        return {"op": "model", "mix": mix, "m": m, "layers": rng.randint(1, max(1, min(16, most))), "d": d, "kv": kv, "ffn": ffn, "vocab": vocab}
    if op == "moe":
        fmt = rng.choice(["mxfp4", "q4_k", "q6_k", "int8", "iq2_xxs", "iq3_xxs"])
        e = rng.choice([8, 16, 32, 60, 64, 128])
        r = rng.randint(1, min(8, e // 2))
        t = rng.choice([1, 1, 2, 5, 8, _log_int(rng, 9, 512 if fmt in TENSOR_CORE else 100)])
        k = _log_int(rng, 1024, 6144, 256)
        n = _log_int(rng, 512, min(14336, int(6e8 / (e * k))), 256)
        return {"op": "moe", "fmt": fmt, "t": t, "r": r, "e": e, "n": n, "k": k, "layers": rng.randint(1, 2)}
    fmt = rng.choice(["q4_k", "q5_k", "q6_k", "int8", "int4", "mxfp4"])
    return {"op": "quantize", "fmt": fmt, "n": _log_int(rng, 500, 14336), "k": _log_int(rng, 1024, 14336 // 4, K_BLOCK[fmt])}


# ---- weights ------------------------------------------------------------------------------------------------
def _weights(be, fmt, n, k, g, std=WEIGHT_STD):
    """A quantized [n, k] matrix of N(0, std) weights on the GPU, from the framework's own quantizer; the i-quants,
    which have none here, are random blocks of about that size (every byte pattern is a valid block)."""
    out = torch.zeros(tp.layout_total(FMT[fmt], n, k), dtype=torch.uint8, device="cuda")
    if fmt in IQ_BLOCK:
        blocks = torch.randint(0, 256, (n * k // 256, IQ_BLOCK[fmt]), dtype=torch.uint8, device="cuda", generator=g)
        d = torch.rand(n * k // 256, device="cuda", generator=g).add_(0.5).mul_(std / IQ_RMS[fmt]).half()
        blocks[:, :2] = d.view(torch.uint8).view(-1, 2)
        out[: blocks.numel()] = blocks.reshape(-1)
        return out
    w = torch.randn(n * k, device="cuda", generator=g).mul_(std)
    torch.cuda.synchronize()
    be.quantize_into(FMT[fmt], be.wrap_tensor(w), n, k, be.wrap_tensor(out))
    be.synchronize()
    return out


def _stack_weights(be, fmt, e, n, k, g):
    """`e` experts' matrices, each at its own multiple of the matrix's bytes."""
    one = tp.layout_total(FMT[fmt], n, k)
    if fmt in ("int8", "int4") or one != n * k // K_BLOCK[fmt] * _block_bytes(fmt):
        return torch.cat([_weights(be, fmt, n, k, g) for _ in range(e)])
    return _weights(be, fmt, e * n, k, g)


def _block_bytes(fmt):
    return {"q4_k": 144, "q5_k": 176, "q6_k": 210, "mxfp4": 17}.get(fmt) or IQ_BLOCK[fmt]


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1009 + 17)
    return g


def _new_backend():
    be = lp.Backend(torch.cuda.current_device())
    be.set_stream(stream().cuda_stream)
    return be


class State:
    """What a program keeps: the device, its buffers and a callable that makes one pass and gives its outputs."""

    def __init__(self, be, call, outputs, keep):
        self.be, self.call, self.outputs, self.keep = be, call, outputs, keep


def _captured(be, queue):
    """`queue` (work of one step) as a CUDA graph on the program's stream."""
    s = stream()
    with torch.cuda.stream(s):
        queue()
    s.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        be.set_stream(torch.cuda.current_stream().cuda_stream)
        queue()
    be.set_stream(s.cuda_stream)

    def replay():
        with torch.cuda.stream(s):
            graph.replay()
    return replay


# ---- one kind each: what is held before the call -------------------------------------------------------------
def _prepare_matmul(c, seed):
    be, g = _new_backend(), _gen(seed)
    m, n, k = c["m"], c["n"], c["k"]
    code, kind = A_DTYPE[c["a"]]
    x = torch.randn(m, k, device="cuda", generator=g).to(kind)
    out = torch.zeros(m, n, device="cuda")
    held = [x, _weights(be, c["fmt"], n, k, g), out]
    more = {}
    if c["epilogue"] != "none":  # a bias over the columns; silu(x w): what stands behind the gate projection
        held.append(torch.randn(n, device="cuda", generator=g))
        more = {"bias_input": 3} if c["epilogue"] == "bias" else {"expr": Expr.silu(Expr.load(0))}
    launches = [matmul_launch(FMT[c["fmt"]], m, n, k, a_dtype=code, inputs=(0, 1), output=2, **more)]
    torch.cuda.synchronize()
    bufs = [be.wrap_tensor(t) for t in held]
    be.prepare(launches)
    return State(be, lambda: be.execute(launches, bufs), out, (held, bufs))


def _sweep_shapes(c):
    return [(m, n, k) for m in (1, 2, 4, 8) for n, k in ((c["d"], c["d"]), (c["kv"], c["d"]), (c["ffn"], c["d"]), (c["d"], c["ffn"]))]


def _prepare_sweep(c, seed):
    be, g = _new_backend(), _gen(seed)
    fmt, shapes = FMT[c["fmt"]], _sweep_shapes(c)
    # every launch has a matrix of its own, as the layers of a model do: their bytes come from HBM
    weights = [_weights(be, c["fmt"], n, k, g) for _, n, k in shapes]
    n_in, n_out = sum(m * k for m, _, k in shapes), sum(m * n for m, n, _ in shapes)
    h_in = torch.randn(n_in, device="cuda", generator=g).cpu().pin_memory()
    h_out = torch.zeros(n_out).pin_memory()
    torch.cuda.synchronize()
    bufs = [be.alloc(n_in * 4), be.alloc(n_out * 4)] + [be.wrap_tensor(w) for w in weights]
    launches, writes, reads, a_at, o_at = [], [], [], 0, 0
    for i, (m, n, k) in enumerate(shapes):
        launches.append(matmul_launch(fmt, m, n, k, inputs=(0, 2 + i), output=1, a=MatView(a_at, m * k, k), out=MatView(o_at, m * n, n)))
        writes.append((0, a_at * 4, h_in.data_ptr() + a_at * 4, m * k * 4, i))
        reads.append((1, o_at * 4, h_out.data_ptr() + o_at * 4, m * n * 4, i))
        a_at, o_at = a_at + m * k, o_at + m * n
    be.prepare(launches)
    return State(be, be.packed_io(launches, bufs, writes, reads), h_out, (weights, h_in, bufs))


def _formats(c):
    """(formats by layer and projection, head, table)."""
    most, wide, head, table = MIX[c["mix"]]
    layers = [{p: wide if tp.q4km_format(p, i, c["layers"]) == tp.Q6_K else most for p in ("q", "k", "v", "o", "gate", "up", "down")}
              for i in range(c["layers"])]
    return layers, head, table


def _layer_shape(c):
    return tp.LayerShape(c["d"], c["d"] // 32, c["kv"] // 32, 32, c["ffn"])


def _prepare_model(c, seed):
    be, g = _new_backend(), _gen(seed)
    m, d, vocab = c["m"], c["d"], c["vocab"]
    decode = m <= 8
    formats, head_fmt, table_fmt = _formats(c)
    shape = _layer_shape(c)
    # the projections that add to the residual stream are scaled by 1 / sqrt(2 layers), as is usual, so that the stream
    # does not grow with depth
    into = WEIGHT_STD / (2 * c["layers"]) ** 0.5
    weights = [{p: _weights(be, f[p], n, k, g, into if p in ("o", "down") else WEIGHT_STD) for p, n, k, _ in shape.projections()} for f in formats]
    head, table = _weights(be, head_fmt, vocab, d, g), _weights(be, table_fmt, vocab, d, g, 2.0)
    ids = torch.randint(0, vocab, (m,), dtype=torch.int32, device="cuda", generator=g)
    rows = m if decode else 1  # of a prompt only the last row is asked for the next token
    logits = torch.zeros(rows, vocab, device="cuda")
    # the glue kernels also write their result quantized for the decode launches behind them where the width allows
    layers = tp.GpuTpLayers(be, shape, 1, 0, m, weights, [{p: FMT[f] for p, f in fs.items()} for fs in formats],
                            fuse_act=decode and d % 1024 == 0 and c["ffn"] % 256 == 0)
    torch.cuda.synchronize()
    bufs = [be.wrap_tensor(t) for t in (table, ids, layers.h, layers.x, head, logits)]
    embed = [gather_launch(FMT[table_fmt], vocab, d, m, inputs=(0, 1), output=2)]
    last = [matmul_launch(FMT[head_fmt], rows, vocab, d, inputs=(3, 4), output=5, a=MatView((m - rows) * d, rows * d, d))]
    be.prepare(embed + last)
    embed, last = be.packed(embed, bufs), be.packed(last, bufs)

    def queue():
        embed()
        layers.token(c["layers"])
        last()
    call = _captured(be, queue) if decode else queue
    return State(be, call, [logits, layers.hw], (weights, head, table, ids, layers, bufs))


def _prepare_moe(c, seed):
    be, g = _new_backend(), _gen(seed)
    t, r, e, n, k, fmt = c["t"], c["r"], c["e"], c["n"], c["k"], FMT[c["fmt"]]
    blocks, keep, outs = [], [], []
    for _ in range(c["layers"]):
        gate, up, down = (_stack_weights(be, c["fmt"], e, a, b, g) for a, b in ((n, k), (n, k), (k, n)))
        x = torch.randn(t, k, device="cuda", generator=g)
        ids = torch.rand(t, e, device="cuda", generator=g).argsort(dim=1)[:, :r].to(torch.int32).contiguous()  # r different experts per token
        mid = [torch.zeros(t * r, n, device="cuda") for _ in range(3)]
        out = torch.zeros(t * r, k, device="cuda")
        torch.cuda.synchronize()
        bufs = [be.wrap_tensor(v) for v in (x, ids, gate, up, down, *mid, out)]
        first = [matmul_id_launch(fmt, t, r, e, n, k, inputs=(0, 2 + i, 1), output=5 + i) for i in (0, 1)]
        second = [matmul_id_launch(fmt, t * r, 1, e, k, n, inputs=(7, 4, 1), output=8)]
        be.prepare(first + second)
        blocks.append((be.packed(first, bufs), bufs, be.packed(second, bufs)))
        keep.append((gate, up, down, x, ids, mid, out))
        outs += mid[:2] + [out]

    def queue():
        for first, bufs, second in blocks:
            first()
            be.silu_mul(bufs[5], bufs[6], bufs[7], t * r * n)
            second()
    call = _captured(be, queue) if t <= 8 else queue
    return State(be, call, outs, (keep, blocks))


def _prepare_quantize(c, seed):
    be, g = _new_backend(), _gen(seed)
    n, k, fmt = c["n"], c["k"], FMT[c["fmt"]]
    total = tp.layout_total(fmt, n, k)
    w = torch.randn(n, k, device="cuda", generator=g).mul_(0.02)
    q, back = torch.zeros(total, dtype=torch.uint8, device="cuda"), torch.zeros(n, k, device="cuda")
    held, bufs = [w, q, back], [be.wrap_tensor(v) for v in (w, q, back)]
    if c["fmt"] in ("int8", "int4"):  # Q8_0 / Q4_0 blocks as a model file holds them: a f16 scale, then the quants
        size = 34 if c["fmt"] == "int8" else 18
        blocks = torch.randint(0, 256, (n * k // 32, size), dtype=torch.uint8, device="cuda", generator=g)
        blocks[:, :2] = torch.rand(n * k // 32, device="cuda", generator=g).mul_(0.001).half().view(torch.uint8).view(-1, 2)
        imported = torch.zeros(total, dtype=torch.uint8, device="cuda")
        held += [blocks, imported]
        bufs += [be.wrap_tensor(blocks), be.wrap_tensor(imported)]
    torch.cuda.synchronize()

    def call():
        be.quantize_into(fmt, bufs[0], n, k, bufs[1])
        be.dequantize_into(fmt, bufs[1], n, k, bufs[2])
        if len(bufs) > 3:
            from_ggml_blocks_into(be, fmt, bufs[3], n * k // 32 * size, n, k, bufs[4])
    return State(be, call, [q, back] + held[4:], (held, bufs))


def prepare(case, seed):
    state = {"matmul": _prepare_matmul, "sweep": _prepare_sweep, "model": _prepare_model, "moe": _prepare_moe,
             "quantize": _prepare_quantize}[case["op"]](case, seed)
    torch.cuda.synchronize()
    return state


def run(state):
    state.call()
    return state.outputs


# ---- what a pass cannot do without ---------------------------------------------------------------------------
def _matrix_bytes(fmt, n, k):
    return tp.layout_total(FMT[fmt], n, k)


def work(case):
    c = case
    if c["op"] == "matmul":
        m, n, k = c["m"], c["n"], c["k"]
        a = m * k * (4 if c["a"] == "f32" else 2)
        return {"bytes": _matrix_bytes(c["fmt"], n, k) + a + 4 * m * n + (4 * n if c["epilogue"] == "bias" else 0), "flops": 2.0 * m * n * k}
    if c["op"] == "sweep":
        s = _sweep_shapes(c)
        return {"bytes": sum(_matrix_bytes(c["fmt"], n, k) + 4 * m * (k + n) for m, n, k in s), "flops": sum(2.0 * m * n * k for m, n, k in s)}
    if c["op"] == "model":
        m, d, vocab = c["m"], c["d"], c["vocab"]
        formats, head, table = _formats(c)
        rows = m if m <= 8 else 1
        shapes = _layer_shape(c).projections()
        b = sum(_matrix_bytes(f[p], n, k) for f in formats for p, n, k, _ in shapes) + _matrix_bytes(head, vocab, d)
        b += m * (_matrix_bytes(table, 1, d) + 4) + 4 * rows * vocab + 4 * m * d  # looked-up rows, indices, logits, residual stream
        return {"bytes": b, "flops": 2.0 * m * c["layers"] * sum(n * k for _, n, k, _ in shapes) + 2.0 * rows * vocab * d}
    if c["op"] == "moe":
        t, r, e, n, k = c["t"], c["r"], c["e"], c["n"], c["k"]
        hit = e * (1.0 - (1.0 - r / e) ** t)  # experts that at least one of t tokens names, on average
        b = hit * 3 * _matrix_bytes(c["fmt"], n, k) + 4 * t * k + 4 * t * r + 4 * t * r * (2 * n + k)
        return {"bytes": b * c["layers"], "flops": 6.0 * t * r * n * k * c["layers"]}
    n, k = c["n"], c["k"]
    q = _matrix_bytes(c["fmt"], n, k)
    b = 4 * n * k + q + 4 * n * k
    if c["fmt"] in ("int8", "int4"):
        b += n * k // 32 * (34 if c["fmt"] == "int8" else 18) + q
    return {"bytes": b, "flops": 1.0 * n * k}


def tolerance(case):
    """What the number formats give, from comparing the path with itself in another order of summation (decode) or with
    its exact f32 form (prefill with bf16 operands), about four times what that shows."""
    c = case
    if c["op"] == "quantize":
        return "exact"  # bytes and dequantized bits are fixed by the formats
    if c["op"] == "sweep" or (c["op"] == "matmul" and (c["m"] <= 8 or c["fmt"] not in TENSOR_CORE)):
        return {"rel": 5e-6, "max": 5e-5}  # exact integer products or f32 products, f32 sums in any order: 1.4e-7 to 3e-7, max 2e-6
    if c["op"] == "matmul":
        return {"rel": 1e-2, "max": 0.05}  # operands rounded to bf16: 2.4e-3, max 1e-2
    if c["op"] == "moe":
        if c["t"] * c["r"] > 8 and c["t"] > 8 and c["fmt"] not in TENSOR_CORE:
            return {"rel": 5e-6, "max": 1e-4}  # f32 throughout
        return {"rel": 1e-2, "max": 0.1}  # two products in a row: bf16 4e-3, max 2e-2; int8 activations whose rounding flips less
    if c["m"] <= 8:
        # a sum that differs in its last bit flips the rounding of an activation to int8 somewhere; over the layers that
        # spreads until two orders of summation differ by the rounding noise itself: 1e-3 to 1.5e-2, max 7e-2
        return {"rel": 0.03, "max": 0.3}
    if c["mix"] in ("q4_k_m", "q5_k_m"):
        return {"rel": 0.02, "max": 0.2}  # bf16 rounding of every product's operands over the layers: 4e-3 to 9e-3, max 4e-2
    return {"rel": 2e-3, "max": 0.03}  # f32 layers; the last row goes through the head with int8 activations, where one flip is 4e-4
