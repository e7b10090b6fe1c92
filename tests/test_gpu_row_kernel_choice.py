"""The two decode kernels of MXFP4 (csrc/row_stream.cuh, csrc/qgemv_mxfp4_mma.cu) and of the i-quants at several rows (csrc/qgemv_iq_rows.cu,
csrc/qgemv_iq.cu): which one a launch takes, both of them at the edges of their shares, and the range and accuracy of their f32 sums.

Bar: integer sums are exact and products the oracle's, f32 terms are added in another order: max_rel <= 2e-5, as for every decode kernel."""
import numpy as np
import pytest

import lapid_b200 as lp
from lapid_b200.backend import matmul_id_launch, matmul_launch
from oracle import oracle as O
from tests.refgen import iq_matrix
from tests.test_gpu_row_kernels import IQ, MX, _max_rel, _weights
from tests.test_gpu_row_kernels import test_mxfp4_shares_steps_and_rows as shares_steps_and_rows

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def be():
    return lp.Backend(0)


@pytest.mark.parametrize("m,n,k", [
    (1, 2300, 1024), (1, 1200, 4096), (2, 2100, 1056), (5, 600, 2880),   # a matrix row for each warp at most; one row, activations not copied
    (2, 1000, 14336), (3, 2048, 8224),                                   # two rows a warp, several warps to a row
])
def test_mxfp4_rows_of_a_warp(be, oracle, m, n, k):
    shares_steps_and_rows(be, oracle, m, n, k)


def _run(be, a, qb, m, n, k):
    bufs = [be.upload(a), be.upload(qb), be.alloc(m * n * 4)]
    be.execute([matmul_launch(MX, m, n, k, inputs=(0, 1), output=2)], bufs)
    return bufs[2].download().view(np.float32)


def test_mxfp4_decode_row_kernel(be, oracle):
    """The MXFP4 row kernel at one to eight rows with one, two and four warps per row and with the launch's own choice,
    against the oracle; the expert-indexed launch included."""
    rng = np.random.default_rng(21)
    for (m, n, k) in [(1, 4096, 4096), (2, 130, 512), (2, 77, 1024), (8, 1030, 14336), (1, 9, 2560), (1, 33, 28672), (2, 700, 7680), (4, 50, 96)]:
        raw = rng.integers(0, 256, n * k // 32 * 17, dtype=np.uint8)
        raw.reshape(-1, 17)[:, 0] = rng.integers(118, 132, n * k // 32, dtype=np.uint8)   # scales around 2^-8
        qb = np.concatenate([raw, np.zeros((-raw.size) % 256, np.uint8)])
        a = O.normal(1900 + m, m * k)
        want, _ = oracle.matmul(O.MXFP4, a, qb, n, k, m=m)
        be.set_option("gemv_mxfp4_mma_rows", "0")       # (the row kernel at every row count)
        for split in ("1", "2", "4", "0"):              # one, two and four warps per row, then the launch's own choice
            be.set_option("gemv_mxfp4_k_split", split)
            assert _max_rel(_run(be, a, qb, m, n, k), want) <= 2e-5, (m, n, k, split)
        be.set_option("gemv_mxfp4_mma_rows", "auto")
    t, r, e, n, k = 3, 2, 4, 200, 1024   # (an expert-indexed launch is one-row work per pair)
    one = oracle.layout(O.MXFP4, n, k).total
    stack = np.zeros(e * one, np.uint8)
    for x in range(e):
        raw = rng.integers(0, 256, n * k // 32 * 17, dtype=np.uint8)
        raw.reshape(-1, 17)[:, 0] = rng.integers(118, 132, n * k // 32, dtype=np.uint8)
        stack[x * one:x * one + raw.size] = raw
    xs = O.normal(1950, t * k)
    ids = np.array([(i * 3 + 1) % e for i in range(t * r)], np.int32)
    want = oracle.matmul_id(O.MXFP4, xs, stack, ids, t, r, e, n, k)
    bufs = [be.upload(xs), be.upload(stack), be.upload(ids.view(np.uint8)), be.alloc(t * r * n * 4)]
    for split in ("1", "2", "0"):
        be.set_option("gemv_mxfp4_k_split", split)
        be.execute([matmul_id_launch(MX, t, r, e, n, k)], bufs)
        assert _max_rel(bufs[3].download().view(np.float32), want) <= 2e-5, split
    be.set_option("gemv_mxfp4_staged", "0")             # (accepted, without effect)


@pytest.mark.parametrize("m,n,k,mma", [
    (3, 1024, 4096, False), (3, 2048, 4096, True), (3, 4097, 4096, False), (3, 2048, 8704, False), (4, 2048, 2048, False), (4, 2304, 5120, True),
    (4, 14336, 512, False), (5, 1024, 2048, False), (5, 2048, 1536, True), (6, 8192, 1024, False), (8, 64, 512, True), (8, 64, 544, False),
])
def test_mxfp4_kernel_choice(oracle, m, n, k, mma):
    """Three to eight rows go to the row kernel or to the tensor cores by size: the bits are those of the kernel named."""
    be = lp.Backend(0)
    qb, a = _weights(MX, n, k, m + n), O.normal(7 + n, m * k)
    bufs = [be.upload(a), be.upload(qb), be.alloc(m * n * 4)]
    got = []
    for option in (None, "1" if mma else "0", "auto"):
        if option:
            be.set_option("gemv_mxfp4_mma_rows", option)
        be.execute([matmul_launch(MX, m, n, k, inputs=(0, 1), output=2)], bufs)
        got.append(bufs[2].download().view(np.uint32).copy())
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
    be.set_option("gemv_mxfp4_mma_rows", "0" if mma else "1")
    be.execute([matmul_launch(MX, m, n, k, inputs=(0, 1), output=2)], bufs)
    other = bufs[2].download().view(np.float32)
    if k % 512 == 0:
        assert not np.array_equal(got[0], other.view(np.uint32))
    assert _max_rel(other, got[0].view(np.float32)) <= 2e-5
    want, _ = oracle.matmul(O.MXFP4, a, qb, n, k, m=m)
    assert _max_rel(got[0].view(np.float32), want) <= 2e-5


@pytest.mark.parametrize("row_kernel", ["1", "2"])   # on csrc/qgemv_iq_rows.cu, on csrc/qgemv_iq.cu
@pytest.mark.parametrize("fmt", [lp.DType.Iq2Xxs, lp.DType.Iq2Xs, lp.DType.Iq2S, lp.DType.Iq3Xxs])
@pytest.mark.parametrize("m,n,k", [
    (8, 3, 256), (8, 150, 1280),                   # one block; a step that is partly there
    (8, 2501, 2304), (8, 33, 13824),               # blocks on odd halves of a word in every other row; more steps than warps
    (3, 2400, 1024), (4, 4097, 2304), (5, 2050, 4352), (6, 1500, 768), (7, 301, 2560),
])
def test_iquants_on_both_kernels(be, oracle, fmt, m, n, k, row_kernel):
    qb, a, bias = iq_matrix(fmt, n, k, m + n), O.normal(7 + n, m * k), O.normal(8 + n, n)
    want, path = oracle.matmul(int(fmt), a, qb, n, k, m=m, bias=bias)
    assert path == "int8_act"
    bufs = [be.upload(a), be.upload(qb), be.alloc(m * n * 4), be.upload(bias)]
    be.set_option("gemv_iq_row_kernel", row_kernel)
    try:
        be.execute([matmul_launch(fmt, m, n, k, inputs=(0, 1), output=2, bias_input=3)], bufs)
    finally:
        be.set_option("gemv_iq_row_kernel", "0")
    assert _max_rel(bufs[2].download().view(np.float32), want) <= 2e-5


def test_iquant_activations_that_do_not_fit(be, oracle):
    """Eight rows of 16640: the row kernel has no room for them, forced or not."""
    m, n, k, fmt = 8, 12, 16640, lp.DType.Iq2Xs
    qb, a = iq_matrix(fmt, n, k, 1), O.normal(9, m * k)
    want, _ = oracle.matmul(int(fmt), a, qb, n, k, m=m)
    bufs = [be.upload(a), be.upload(qb), be.alloc(m * n * 4)]
    for row_kernel in ("1", "0"):
        be.set_option("gemv_iq_row_kernel", row_kernel)
        be.execute([matmul_launch(fmt, m, n, k, inputs=(0, 1), output=2)], bufs)
        assert _max_rel(bufs[2].download().view(np.float32), want) <= 2e-5
    with pytest.raises(lp.LapidError):
        be.set_option("gemv_iq_row_kernel", "3")


@pytest.mark.parametrize("fmt", [MX, lp.DType.Q4K, lp.DType.Q6K, lp.DType.Int8])
def test_expert_launches_share_the_quantized_tokens_whatever_their_size(be, oracle, fmt):
    """gate and up of 8 tokens with 8 slots each: their 64 pairs read more than the L2 holds, so they are two kernels, but the tokens are quantized once."""
    t, r, e, n, k = 8, 8, 8, 2048, 2048   # (each expert eight times: above that the reference multiplies in f32)
    total = oracle.layout(int(fmt), n, k).total
    one = _weights(fmt, n, k, 5) if fmt == MX else oracle.quantize(int(fmt), O.normal(5, n * k, 0.02), n, k)
    stack = np.zeros(e * total, np.uint8)
    for i in range(e):   # every expert another matrix: the first 16 i rows of its quants are zeros
        stack[i * total:i * total + one.size] = one
        stack[i * total:i * total + 16 * i * (one.size // n)] = 0
    ids = np.array([(i // r + i) % e for i in range(t * r)], np.int32)
    x = O.normal(62, t * k)
    bufs = [be.upload(x), be.upload(stack), be.upload(stack), be.upload(ids.view(np.uint8))] + [be.alloc(t * r * n * 4) for _ in range(2)]
    be.take_launch_count()
    be.execute([matmul_id_launch(fmt, t, r, e, n, k, inputs=(0, 1 + i, 3), output=4 + i) for i in (0, 1)], bufs)
    assert be.take_launch_count() == 3
    want = oracle.matmul_id(int(fmt), x, stack, ids, t, r, e, n, k)
    for b in bufs[4:]:
        assert _max_rel(b.download().view(np.float32), want) <= 2e-5


@pytest.mark.parametrize("fmt", [lp.DType.Iq2Xxs, lp.DType.Iq2Xs, lp.DType.Iq2S, lp.DType.Iq3Xxs])
def test_iquant_sums_overflow_no_earlier_than_the_reference(be, oracle, fmt):
    """Activations of one size and with the signs of the weights: the sum, of terms of one sign, is 2e38, and twice that is not finite."""
    m, n, k = 8, 1, 512
    qb = iq_matrix(fmt, n, k, 3)
    w = oracle.dequantize(int(fmt), qb, n, k).reshape(n, k)
    size = 2e38 / np.abs(w[0].astype(np.float64)).sum()
    a = np.tile(np.where(w[0] < 0, -size, size).astype(np.float32), m)
    want, path = oracle.matmul(int(fmt), a, qb, n, k, m=m)
    assert path == "int8_act" and np.isfinite(want).all() and want.max() > 1.9e38
    bufs = [be.upload(a), be.upload(qb), be.alloc(m * n * 4)]
    for row_kernel in ("1", "2", "0"):
        be.set_option("gemv_iq_row_kernel", row_kernel)
        be.execute([matmul_launch(fmt, m, n, k, inputs=(0, 1), output=2)], bufs)
        got = bufs[2].download().view(np.float32)
        assert np.isfinite(got).all() and _max_rel(got, want) <= 2e-5


@pytest.mark.parametrize("fmt,n,k,members,bound", [
    (MX, 1500, 14336, 1, 8.4e-8),      # several warps to a row
    (MX, 4096, 14336, 1, 8.6e-8),      # one warp, fourteen steps
])
def test_f32_sums_are_as_close_to_f64_as_with_more_warps_to_a_row(be, oracle, fmt, n, k, members, bound):
    """One activation row against f64 sums of the same quantized operands. The bounds lie between what these sums show (6.5e-8, 8.2e-8; with two or four
    warps to a row, one chain each: 8.2e-8, 8.3e-8) and one chain over a longer k (8.8e-8, 9.2e-8); 2-norms over all outputs, inputs fixed."""
    a = O.normal(71, k)
    q, d = oracle.quantize_row_sums(a, want_bs=False)[:2]
    x = (np.asarray(q, np.float64).reshape(-1, 32) * np.asarray(d, np.float64).reshape(-1, 1)).reshape(-1)
    ws = [_weights(fmt, n, k, 72 + i) for i in range(members)]
    bufs = [be.upload(a)] + [be.upload(w) for w in ws] + [be.alloc(n * 4) for _ in ws]
    be.execute([matmul_launch(fmt, 1, n, k, inputs=(0, 1 + i), output=1 + members + i) for i in range(members)], bufs)
    off = total = 0.0
    for i, w in enumerate(ws):
        want = oracle.dequantize(int(fmt), w, n, k).reshape(n, k).astype(np.float64) @ x
        off += ((bufs[1 + members + i].download().view(np.float32) - want) ** 2).sum()
        total += (want ** 2).sum()
    assert (off / total) ** 0.5 <= bound
