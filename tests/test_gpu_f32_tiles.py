"""Exact-f32 GEMM (csrc/qgemm_f32.cu): the kernel with producer and consumer warps, which launches with many outputs take, and the larger tiles of the other
one, each fixed by the option ``gemm_f32_tile``. Tiles of every width (1 to 8 units of 16 columns, a ragged last one), rows that do not fill a block of 128,
the shortest k, every weight format, aligned and unaligned activations and outputs, a bias, experts.

Exact: an output is one chain of fused multiply-adds over k whatever kernel computes it, so the bits are those of the same rows multiplied sixteen
at a time on the smallest tiles (they are held against the oracle in test_gpu_parity.py, and here for the i-quants)."""
import numpy as np
import pytest

import lapid_b200 as lp
from lapid_b200 import quant
from lapid_b200.backend import MatView, matmul_id_launch, matmul_launch
from oracle import oracle as O
from tests.refgen import iq_matrix

pytestmark = pytest.mark.gpu
IQ = {lp.DType.Iq2Xxs: 66, lp.DType.Iq2Xs: 74, lp.DType.Iq2S: 82, lp.DType.Iq3Xxs: 98}   # bytes of a block of 256
FORMATS = [lp.DType.Int8, lp.DType.Int4, lp.DType.MXFP4, lp.DType.Q4K, lp.DType.Q5K, lp.DType.Q6K, *IQ]


@pytest.fixture
def be():
    be = lp.Backend(0)
    be.set_option("gemm", "f32")
    return be


def _weights(be, fmt, n, k, seed):
    if fmt in IQ:
        return iq_matrix(fmt, n, k, seed)
    return quant.quantize(be, fmt, np.random.default_rng(seed).standard_normal(n * k, dtype=np.float32) * np.float32(0.02), n, k)


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("m,n,k,pad,out_pad,bias", [
    (128, 9488, 32, 0, 0, False),     # one round of tiles of four and five units, two steps of k
    (127, 11900, 64, 0, 4, True),     # five and six units, the last one ragged
    (512, 4096, 96, 4, 0, False),     # six and seven
    (100, 18900, 64, 1, 1, True),     # eight; neither operand nor result aligned
    (300, 3000, 64, 0, 0, False),     # three and four
    (129, 4000, 32, 0, 0, True),      # one and two
    (200, 14336, 32, 0, 0, True),     # two rounds
    (20, 40, 160, 0, 0, True),        # fewer columns than the narrowest loop has
])
def test_tiles_rows_and_strides(be, oracle, fmt, m, n, k, pad, out_pad, bias):
    if fmt in IQ or int(fmt) in (6, 7, 8):
        k = 256 * -(-k // 256)
    qb, bv = _weights(be, fmt, n, k, m), O.normal(41, n)
    rs, os = k + pad, n + out_pad
    a = O.normal(40 + m, m * rs)
    bufs = [be.upload(a), be.upload(qb), be.alloc(m * os * 4), be.upload(bv)]
    more = {"bias_input": 3} if bias else {}
    got = {}
    for tile, step in (("16", 16), ("128", m), ("64", m), ("32", m)):
        be.set_option("gemm_f32_tile", tile)
        bufs[2].write(0, np.full(m * os, -7.0, np.float32))
        be.execute([matmul_launch(fmt, min(step, m - r), n, k, inputs=(0, 1), output=2, a=MatView(r * rs, min(step, m - r) * rs, rs),
                                  out=MatView(r * os, min(step, m - r) * os, os), **more) for r in range(0, m - 8, step)], bufs)
        got[tile] = bufs[2].download().view(np.uint32).reshape(m, os)
    rows = m - 8 if m % 16 and m % 16 < 9 else m   # (up to eight rows left over would be a decode launch)
    for tile in ("128", "64", "32"):
        assert np.array_equal(got[tile][:rows], got["16"][:rows]), tile
        assert np.all(got[tile][:, n:].view(np.float32) == -7.0), tile
    if fmt in IQ:
        row_bytes = k // 256 * IQ[fmt]
        x = np.ascontiguousarray(a.reshape(m, rs)[:, :k]).reshape(-1)
        for col in (0, n - 1):
            one = np.concatenate([qb[col * row_bytes:(col + 1) * row_bytes], np.zeros(-row_bytes % 256, np.uint8)])
            want, path = oracle.matmul(int(fmt), x, one, 1, k, m=m, bias=bv[col:col + 1] if bias else None)
            assert path == "f32_act" and np.array_equal(got["128"][:, col], want.view(np.uint32)), col


@pytest.mark.parametrize("a_dtype", [lp.DType.F16, lp.DType.BF16])
@pytest.mark.parametrize("pad", [0, 1])   # four activations by one load, one by one
@pytest.mark.parametrize("tile", ["128", "64", "32", "16"])
def test_half_activations(be, a_dtype, pad, tile):
    """Half activations are widened exactly: the bits of the launch over their f32 values."""
    m, n, k = 130, 7000, 96
    rs = k + pad
    x32 = O.normal(70, m * rs)
    bits = x32.astype(np.float16).view(np.uint16) if a_dtype == lp.DType.F16 else (x32.view(np.uint32) >> 16).astype(np.uint16)
    wide = bits.view(np.float16).astype(np.float32) if a_dtype == lp.DType.F16 else (bits.astype(np.uint32) << 16).view(np.float32)
    qb = be.upload(_weights(be, lp.DType.Int8, n, k, 71))
    be.set_option("gemm_f32_tile", tile)
    got = []
    for a, code in ((bits.view(np.uint8), a_dtype), (wide, lp.DType.F32)):
        bufs = [be.upload(a), qb, be.alloc(m * n * 4)]
        be.execute([matmul_launch(lp.DType.Int8, m, n, k, a_dtype=code, inputs=(0, 1), output=2, a=MatView(0, m * rs, rs))], bufs)
        got.append(bufs[2].download().view(np.uint32))
    assert np.array_equal(got[0], got[1])


@pytest.mark.parametrize("tile", ["128", "64", "32", "16"])
@pytest.mark.parametrize("fmt", [lp.DType.Int8, lp.DType.MXFP4, lp.DType.Iq2S])
def test_experts(be, fmt, tile):
    """Expert-indexed launches: the bits of each expert's own product on the smallest tiles."""
    t, r, e, n, k = 300, 2, 3, 3001, 256 if fmt in IQ else 64
    mats = [_weights(be, fmt, n, k, i) for i in range(e)]
    ids = np.array([(i % 2) * 2 for i in range(t * r)], np.int32)   # the middle expert is not used
    bufs = [be.upload(O.normal(50, t * k)), be.upload(np.concatenate(mats)), be.upload(ids.view(np.uint8)), be.alloc(t * r * n * 4), be.alloc(t * n * 4)]
    be.set_option("gemm_f32_tile", tile)
    be.execute([matmul_id_launch(fmt, t, r, e, n, k)], bufs)
    got = bufs[3].download().view(np.uint32).reshape(t, r, n)
    be.set_option("gemm_f32_tile", "16")
    for slot, x in ((0, 0), (1, 2)):
        plain = bufs[:1] + [be.upload(mats[x])] + [bufs[4]]
        be.execute([matmul_launch(fmt, t, n, k, inputs=(0, 1), output=2)], plain)
        assert np.array_equal(got[:, slot], plain[2].download().view(np.uint32).reshape(t, n))
    with pytest.raises(lp.LapidError):
        be.set_option("gemm_f32_tile", "48")
