"""Exact-f32 GEMM with producer and consumer warps (csrc/qgemm_f32.cu), which launches with many outputs take: tiles of every width (4 to 8 units of
16 columns, narrower ones, a ragged last one), rows that do not fill a block of 128, the shortest k, every weight format, aligned and unaligned
activations and outputs, a bias, experts.

Exact: an output is one chain of fused multiply-adds over k whatever kernel computes it, so the bits are those of the same rows multiplied sixteen
at a time, which the small tiles do (they are held against the oracle in test_gpu_parity.py)."""
import numpy as np
import pytest

import lapid_b200 as lp
from lapid_b200 import quant
from lapid_b200.backend import MatView, matmul_id_launch, matmul_launch
from oracle import oracle as O

pytestmark = pytest.mark.gpu
FORMATS = [lp.DType.Int8, lp.DType.Int4, lp.DType.MXFP4, lp.DType.Q4K, lp.DType.Q5K, lp.DType.Q6K]


@pytest.fixture(scope="module")
def be():
    be = lp.Backend(0)
    be.set_option("gemm", "f32")
    return be


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("m,n,k,pad,out_pad,bias", [
    (128, 9488, 32, 0, 0, False),     # one round of tiles of four and five units, two steps of k
    (127, 11900, 64, 0, 4, True),     # five and six units, the last one ragged
    (512, 4096, 96, 4, 0, False),     # six and seven
    (100, 18900, 64, 1, 1, True),     # eight; neither operand nor result aligned
    (300, 3000, 64, 0, 0, False),     # tiles narrower than the narrowest loop
    (200, 14336, 32, 0, 0, True),     # two rounds
])
def test_tiles_rows_and_strides(be, fmt, m, n, k, pad, out_pad, bias):
    if int(fmt) in (6, 7, 8):
        k = 256 * -(-k // 256)
    w = np.random.default_rng(m).standard_normal(n * k, dtype=np.float32) * np.float32(0.02)
    rs, os = k + pad, n + out_pad
    bufs = [be.upload(O.normal(40 + m, m * rs)), be.upload(quant.quantize(be, fmt, w, n, k)), be.alloc(m * os * 4), be.upload(O.normal(41, n))]
    more = {"bias_input": 3} if bias else {}
    got = []
    for step in (m, 16):
        bufs[2].write(0, np.full(m * os, -7.0, np.float32))
        be.execute([matmul_launch(fmt, min(step, m - r), n, k, inputs=(0, 1), output=2, a=MatView(r * rs, min(step, m - r) * rs, rs),
                                  out=MatView(r * os, min(step, m - r) * os, os), **more) for r in range(0, m - 8, step)], bufs)
        got.append(bufs[2].download().view(np.uint32).reshape(m, os))
    rows = m - 8 if m % 16 and m % 16 < 9 else m   # (up to eight rows left over would be a decode launch)
    assert np.array_equal(got[0][:rows], got[1][:rows])
    assert np.all(got[0][:, n:].view(np.float32) == -7.0)


@pytest.mark.parametrize("a_dtype", [lp.DType.F16, lp.DType.BF16])
@pytest.mark.parametrize("pad", [0, 1])   # four activations by one load, one by one
def test_half_activations(be, a_dtype, pad):
    """Half activations are widened exactly: the bits of the launch over their f32 values."""
    m, n, k = 130, 7000, 96
    rs = k + pad
    x32 = O.normal(70, m * rs)
    bits = x32.astype(np.float16).view(np.uint16) if a_dtype == lp.DType.F16 else (x32.view(np.uint32) >> 16).astype(np.uint16)
    wide = bits.view(np.float16).astype(np.float32) if a_dtype == lp.DType.F16 else (bits.astype(np.uint32) << 16).view(np.float32)
    w = np.random.default_rng(71).standard_normal(n * k, dtype=np.float32) * np.float32(0.02)
    qb = be.upload(quant.quantize(be, lp.DType.Int8, w, n, k))
    got = []
    for a, code in ((bits.view(np.uint8), a_dtype), (wide, lp.DType.F32)):
        bufs = [be.upload(a), qb, be.alloc(m * n * 4)]
        be.execute([matmul_launch(lp.DType.Int8, m, n, k, a_dtype=code, inputs=(0, 1), output=2, a=MatView(0, m * rs, rs))], bufs)
        got.append(bufs[2].download().view(np.uint32))
    assert np.array_equal(got[0], got[1])


@pytest.mark.parametrize("fmt", [lp.DType.Int8, lp.DType.MXFP4])
def test_experts(be, fmt):
    """Expert-indexed launches of that many rows an expert: the bits of each expert's own product."""
    t, r, e, n, k = 300, 2, 3, 3001, 64
    mats = [quant.quantize(be, fmt, np.random.default_rng(i).standard_normal(n * k, dtype=np.float32) * np.float32(0.02), n, k) for i in range(e)]
    ids = np.array([(i % 2) * 2 for i in range(t * r)], np.int32)   # the middle expert is not used
    bufs = [be.upload(O.normal(50, t * k)), be.upload(np.concatenate(mats)), be.upload(ids.view(np.uint8)), be.alloc(t * r * n * 4), be.alloc(t * n * 4)]
    be.execute([matmul_id_launch(fmt, t, r, e, n, k)], bufs)
    got = bufs[3].download().view(np.uint32).reshape(t, r, n)
    for slot, x in ((0, 0), (1, 2)):
        plain = bufs[:1] + [be.upload(mats[x])] + [bufs[4]]
        be.execute([matmul_launch(fmt, t, n, k, inputs=(0, 1), output=2)], plain)
        assert np.array_equal(got[:, slot], plain[2].download().view(np.uint32).reshape(t, n))
