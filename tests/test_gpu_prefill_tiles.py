"""Tensor-core prefill (csrc/qgemm_tc.cu) at the edges of its tiles: activation rows around the step from one CTA to a pair and between tiles,
weight rows that leave the second CTA of a pair without work, whole tiles beside tiles split over K, and the routing tables that
expert-indexed launches of a list share.

Bar: both operands are rounded to bf16 (2^-9 each) and the sums are f32, so against the exact f32 kernel rel_l2 <= 4e-3 and max_rel <= 3e-2, as
for the other tests of this kernel."""
import numpy as np
import pytest

import lapid_b200 as lp
from lapid_b200 import quant
from lapid_b200.backend import MatView, gather_launch, matmul_id_launch, matmul_launch
from oracle import oracle as O

pytestmark = pytest.mark.gpu
FORMATS = [lp.DType.Q4K, lp.DType.Q5K, lp.DType.Q6K]


@pytest.fixture(scope="module")
def be():
    return lp.Backend(0)


def _close(got, want):
    got, want = got.astype(np.float64), want.astype(np.float64)
    rms = np.sqrt((want ** 2).mean())
    assert np.sqrt(((got - want) ** 2).mean()) / rms <= 4e-3
    assert (np.abs(got - want) / np.maximum(np.abs(want), rms)).max() <= 3e-2


def _both(be, launches, bufs, out):
    """The output buffer's contents from the tensor cores and from the exact f32 kernel."""
    res = []
    for mode in ("tc", "f32"):
        be.set_option("gemm", mode)
        try:
            bufs[out].write(0, np.full(bufs[out].nbytes // 4, -7.0, np.float32))
            be.execute(launches, bufs)
        finally:
            be.set_option("gemm", "tc")
        res.append(bufs[out].download().view(np.float32).copy())
    return res


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("m,n,k,pair", [(m, n, k, pair) for pair in ("-1", "0", "1") for m, n, k in [
    (9, 1, 256), (16, 127, 512), (17, 129, 768), (112, 130, 2048), (128, 300, 1024), (129, 100, 256), (129, 257, 1280), (161, 255, 2048), (256, 513, 512),
    (257, 384, 768), (600, 200, 512)] if pair == "-1" or m > 128])
@pytest.mark.parametrize("ways", ["-1", "0", "3"])
def test_rows_columns_and_splits(be, fmt, m, n, k, ways, pair):
    x, w = O.normal(5000 + m, m * k), O.normal(5001 + n, n * k, 0.05)
    bufs = [be.upload(x), be.upload(quant.quantize(be, fmt, w, n, k)), be.alloc(m * n * 4), be.upload(O.normal(5002, n))]
    for extra in ({}, {"bias_input": 3}):
        be.set_option("gemm_splitk", ways)
        be.set_option("gemm_pair", pair)
        try:
            got, want = _both(be, [matmul_launch(fmt, m, n, k, inputs=(0, 1), output=2, **extra)], bufs, 2)
        finally:
            be.set_option("gemm_splitk", "-1")
            be.set_option("gemm_pair", "-1")
        _close(got, want)


@pytest.mark.parametrize("m", [40, 300])
@pytest.mark.parametrize("fmt", FORMATS)
def test_whole_tiles_beside_split_ones(be, fmt, m):
    """A last round of two tiles of a pair (four of a CTA), split over K, behind a full one; the launch by itself and again give the same bits."""
    import torch
    sms, k = torch.cuda.get_device_properties(0).multi_processor_count, 1024
    n = (sms + 4) * 128 if m <= 128 else (sms // 2 + 2) // 2 * 256   # 300 rows: two activation tiles
    x, w = O.normal(5100, m * k), np.tile(O.normal(5101, 512 * k, 0.05), n // 512 + 1)[: n * k]
    w = (w.reshape(n, k) * (1 + 0.001 * (np.arange(n, dtype=np.float32) % 991))[:, None]).astype(np.float32)
    bufs = [be.upload(x), be.upload(quant.quantize(be, fmt, w, n, k)), be.alloc(m * n * 4)]
    ls = [matmul_launch(fmt, m, n, k, inputs=(0, 1), output=2)]
    got, want = _both(be, ls, bufs, 2)
    _close(got, want)
    be.take_launch_count()
    be.execute(ls, bufs)
    assert be.take_launch_count() == 3   # the copy, the products, the sum of the split tiles
    assert np.array_equal(bufs[2].download().view(np.float32), got)


def test_rows_of_several_batch_entries_in_one_tile(be):
    """A tile's columns cross batch entries whose outputs are strided; nothing outside the views is written."""
    fmt, batch, m, n, k = lp.DType.Q4K, 5, 37, 70, 512
    total = 3 + batch * m * n * 2
    x = O.normal(5200, batch * m * k)
    bufs = [be.upload(x), be.upload(quant.quantize(be, fmt, O.normal(5201, n * k, 0.05), n, k)), be.alloc(total * 4)]
    ls = [matmul_launch(fmt, m, n, k, batch=batch, inputs=(0, 1), output=2, out=MatView(3, n, batch * n))]
    got, want = _both(be, ls, bufs, 2)
    _close(got, want)
    assert np.array_equal(got == -7.0, want == -7.0)


@pytest.mark.parametrize("rewrite", [None, "tokens", "ids"])
def test_expert_indexed_launches_share_their_tables(be, rewrite):
    """Gate and up of one list use the same routing tables and gathered rows; a launch that rewrites the tokens or the ids in between ends that.
    Every result has the bits of the launch run by itself."""
    fmt, t, r, e, n, k = lp.DType.Q4K, 70, 2, 6, 256, 512
    ids = np.stack([np.random.default_rng(i).permutation(e)[:r] for i in range(t)]).astype(np.int32)
    ids[:, 0] = np.where(ids[:, 0] == 3, ids[:, 1] ^ 1, ids[:, 0])
    stacks = [quant.quantize(be, fmt, O.normal(5300 + i, e * n * k, 0.05), e * n, k) for i in range(2)]
    x, y = O.normal(5310, t * k), O.normal(5311, t * k)
    # 0 tokens, 1 ids, 2, 3 stacks, 4, 5 outputs, 6 another operand, 7 the matrix that makes new tokens of it
    bufs = [be.upload(x), be.upload(ids)] + [be.upload(s) for s in stacks] + [be.alloc(t * r * n * 4) for _ in range(2)]
    bufs += [be.upload(y), be.upload(quant.quantize(be, fmt, O.normal(5312, k * k, 0.05), k, k))]
    ls = [matmul_id_launch(fmt, t, r, e, n, k, inputs=(0, 2, 1), output=4), matmul_id_launch(fmt, t, r, e, n, k, inputs=(0, 3, 1), output=5)]
    if rewrite == "tokens":
        ls.insert(1, matmul_launch(fmt, t, k, k, inputs=(6, 7), output=0))
    elif rewrite == "ids":  # a gather of the table's one row: other ids, bit for bit
        other = ids[::-1].copy()
        bufs += [be.upload(other.view(np.float32).reshape(1, -1)), be.upload(np.zeros(1, np.int32))]
        ls.insert(1, gather_launch(lp.DType.F32, 1, t * r, 1, inputs=(8, 9), output=1))
    res, counts = [], []
    for one_list in (False, True):
        bufs[0].write(0, x)
        bufs[1].write(0, ids)
        be.take_launch_count()
        for part in [ls] if one_list else [[l] for l in ls]:
            be.execute(part, bufs)
        counts.append(be.take_launch_count())
        res.append([bufs[i].download().view(np.float32).copy() for i in (4, 5)])
    assert all(np.array_equal(a, b) for a, b in zip(*res))
    assert counts[1] == counts[0] - (0 if rewrite else 2)   # no second route and gather


@pytest.mark.parametrize("m", [9, 130])
@pytest.mark.parametrize("k", [512, 2048])
def test_q6k_infinite_scale_stays_infinite(be, m, k):
    """A Q6_K row whose block scale is infinite gives infinities of the sign of scale times weight, as the exact f32 kernel does (no NaN of its own)."""
    n = 130
    q = quant.quantize(be, lp.DType.Q6K, O.normal(5400, n * k, 0.05), n, k).copy()
    rows = q[: n * k // 256 * 210].reshape(n, k // 256, 210)
    for row, scale, d in ((0, 1, 0x7C00), (1, -3, 0x7C00), (129, 5, 0xFC00)):
        rows[row, :, :192] = 0xFF                    # every value 63 - 32
        rows[row, :, 192:208] = np.uint8(scale & 0xFF)
        rows[row, 0, 208:] = np.frombuffer(np.uint16(d).tobytes(), np.uint8)
    x = np.abs(O.normal(5401, m * k)) + np.float32(0.5)
    bufs = [be.upload(x.astype(np.float32)), be.upload(q), be.alloc(m * n * 4)]
    got, want = _both(be, [matmul_launch(lp.DType.Q6K, m, n, k, inputs=(0, 1), output=2)], bufs, 2)
    got, want = got.reshape(m, n), want.reshape(m, n)
    assert np.isposinf(want[:, 0]).all() and np.isneginf(want[:, [1, 129]]).all()
    assert np.array_equal(got[:, [0, 1, 129]], want[:, [0, 1, 129]])
    _close(got[:, 2:129], want[:, 2:129])


@pytest.mark.parametrize("option,value", [("gemm_splitk", "0"), ("gemm_pair", "0")])
def test_tile_options_belong_to_the_device(be, option, value):
    """An option set on one device leaves the launches of another as they are (the plan of a launch, and with it its part of the scratch, depends on both)."""
    fmt, m, n, k = lp.DType.Q4K, 300, 1024, 4096  # (K split 8 ways in pairs, 6 ways without)
    x, w = O.normal(5500, m * k), O.normal(5501, n * k, 0.05)
    other = lp.Backend(0)
    ls = [matmul_launch(fmt, m, n, k, inputs=(0, 1), output=2)]

    def run(dev):
        bufs = [dev.upload(x), dev.upload(quant.quantize(dev, fmt, w, n, k)), dev.alloc(m * n * 4)]
        dev.take_launch_count()
        dev.execute(ls, bufs)
        return dev.take_launch_count(), bufs[2].download().view(np.float32).copy()

    before = run(be)
    other.set_option(option, value)
    try:
        theirs, after = run(other), run(be)
    finally:
        other.set_option(option, "-1")
    assert before[0] == 3 and after[0] == 3 and np.array_equal(after[1], before[1])
    assert theirs[0] == 2 if option == "gemm_splitk" else not np.array_equal(theirs[1], before[1])  # (the option is not without effect)
    _close(theirs[1], before[1])


@pytest.mark.parametrize("n", [1, 7, 8, 9, 128, 131, 136, 263])
@pytest.mark.parametrize("m,k", [(9, 256), (140, 1792), (300, 2304), (20, 3584)])
def test_q6k_rows_that_are_no_16_byte_multiples(be, m, n, k):
    """Rows come in groups of eight (the second CTA of a pair: of none) and one by one behind the last whole group; every block's place in its
    line differs from row to row."""
    x, w = O.normal(5600 + m, m * k), O.normal(5601 + n, n * k, 0.05)
    bufs = [be.upload(x), be.upload(quant.quantize(be, lp.DType.Q6K, w, n, k)), be.alloc(m * n * 4)]
    got, want = _both(be, [matmul_launch(lp.DType.Q6K, m, n, k, inputs=(0, 1), output=2)], bufs, 2)
    _close(got, want)
