"""Decode kernels of the formats that become int8 by lookups (MXFP4: csrc/row_stream.cuh, csrc/qgemv_mxfp4.cu; i-quants: csrc/qgemv_iq.cu): shares of the CTAs,
steps of k and batches of rows at their edges, and launches that go out as one because they read the same activations. The Int8 / Int4 kernel
(csrc/qgemv_i8_mma.cu): units of a tile and a chunk that the warps take in order.

Bar: integer sums are exact and products the oracle's, f32 terms are added in another order: max_rel <= 2e-5, as for every decode kernel."""
import numpy as np
import pytest

import lapid_b200 as lp
from lapid_b200.backend import MatView, matmul_id_launch, matmul_launch
from oracle import oracle as O
from tests.refgen import iq_matrix

pytestmark = pytest.mark.gpu
MX, IQ = lp.DType.MXFP4, lp.DType.Iq2Xxs


@pytest.fixture(scope="module")
def be():
    return lp.Backend(0)


def _weights(fmt, n, k, seed):
    if fmt != MX:
        return iq_matrix(fmt, n, k, seed)
    rng = np.random.default_rng(seed)
    raw = rng.integers(0, 256, n * k // 32 * 17, dtype=np.uint8)
    raw.reshape(-1, 17)[:, 0] = rng.integers(118, 132, n * k // 32, dtype=np.uint8)
    return np.concatenate([raw, np.zeros((-raw.size) % 256, np.uint8)])


def _max_rel(got, want):
    got, want = np.asarray(got, np.float64).reshape(-1), np.asarray(want, np.float64).reshape(-1)
    return (np.abs(got - want) / np.maximum(np.abs(want), np.sqrt((want ** 2).mean()))).max()


@pytest.mark.parametrize("m,n,k", [
    (1, 1, 32), (2, 3, 32),            # one unit, fewer rows than CTAs
    (1, 149, 1056), (2, 300, 992),     # one unit more and one fewer than whole steps
    (1, 9473, 96), (2, 9500, 1024),    # four rows a warp, the last ones of a share missing
    (1, 700, 16384), (1, 40, 20480),   # sixteen slices of k and more steps than that
    (1, 5, 230400), (2, 5, 92160),     # activations that do not fit shared memory
    (3, 77, 2880), (8, 40, 160), (8, 33, 23072),
])
def test_mxfp4_shares_steps_and_rows(be, oracle, m, n, k):
    qb, a, bias = _weights(MX, n, k, m + n), O.normal(7 + n, m * k), O.normal(8 + n, n)
    want, path = oracle.matmul(O.MXFP4, a, qb, n, k, m=m, bias=bias)
    assert path == "int8_act"
    bufs = [be.upload(a), be.upload(qb), be.alloc(m * (n + 3) * 4), be.upload(bias)]
    bufs[2].write(0, np.full(m * (n + 3), -7.0, np.float32))
    be.execute([matmul_launch(MX, m, n, k, inputs=(0, 1), output=2, bias_input=3, out=MatView(0, m * (n + 3), n + 3))], bufs)
    got = bufs[2].download().view(np.float32).reshape(m, n + 3)
    assert _max_rel(got[:, :n], want) <= 2e-5 and np.all(got[:, n:] == -7.0)


@pytest.mark.parametrize("fmt", [lp.DType.Iq2Xxs, lp.DType.Iq2Xs, lp.DType.Iq2S, lp.DType.Iq3Xxs])
@pytest.mark.parametrize("m,n,k", [
    (8, 3, 256), (8, 150, 1280),                   # one block; a step that is partly there
    (8, 2501, 2304), (8, 33, 13824),               # blocks on odd halves of a word in every other row; more steps than warps
    (3, 8192, 1024), (4, 4097, 2304), (5, 2050, 4352),   # eight million weights and more
    (8, 12, 16640),                                # activations that do not fit: the other kernel
])
def test_iquants_at_several_rows(be, oracle, fmt, m, n, k):
    qb, a, bias = iq_matrix(fmt, n, k, m + n), O.normal(7 + n, m * k), O.normal(8 + n, n)
    want, path = oracle.matmul(int(fmt), a, qb, n, k, m=m, bias=bias)
    assert path == "int8_act"
    bufs = [be.upload(a), be.upload(qb), be.alloc(m * n * 4), be.upload(bias)]
    be.execute([matmul_launch(fmt, m, n, k, inputs=(0, 1), output=2, bias_input=3)], bufs)
    assert _max_rel(bufs[2].download().view(np.float32), want) <= 2e-5


@pytest.mark.parametrize("fmt", [MX, IQ])
@pytest.mark.parametrize("m", [1, 2, 8])
def test_projections_of_one_operand_go_out_together(be, oracle, fmt, m):
    """q, k, v and a launch that reads what q wrote: three in one kernel, the fourth behind it; ragged member sizes."""
    k, sizes = 1024, (1024, 129, 7)
    a = O.normal(20, m * k)
    ws = [_weights(fmt, n, k, 30 + n) for n in sizes + (50,)]
    bufs = [be.upload(a)] + [be.upload(w) for w in ws] + [be.alloc(m * n * 4) for n in sizes + (50,)]
    ls = [matmul_launch(fmt, m, n, k, inputs=(0, 1 + i), output=5 + i) for i, n in enumerate(sizes)]
    be.execute(ls + [matmul_launch(fmt, m, 50, k, inputs=(5, 4), output=8)], bufs)
    got = [b.download().view(np.float32).copy() for b in bufs[5:]]
    for i, n in enumerate(sizes + (50,)):
        x = a if i < 3 else got[0]
        want = oracle.matmul(int(fmt), x, ws[i], n, k, m=m)[0]
        assert _max_rel(got[i], want) <= 2e-5, i


@pytest.mark.parametrize("fmt", [MX, IQ])
@pytest.mark.parametrize("t,r", [(1, 6), (5, 3)])
def test_expert_launches_of_the_same_tokens_go_out_together(be, oracle, fmt, t, r):
    """gate and up over the same tokens and ids share the quantized tokens and a kernel; other ids, or tokens that the list writes in between, do not."""
    e, n, k = 8, 300, 768
    one = oracle.layout(int(fmt), n, k).total
    stacks = []
    for s in (1, 2):
        st = np.zeros(e * one, np.uint8)
        for x in range(e):
            w = _weights(fmt, n, k, 100 * s + x)
            st[x * one:x * one + w.size] = w
        stacks.append(st)
    x = O.normal(60, t * k)
    ids = np.array([(3 * i + 1) % e for i in range(t * r)], np.int32)
    other = np.array([(5 * i + 2) % e for i in range(t * r)], np.int32)
    w0 = _weights(fmt, k, 256, 9)
    bufs = [be.upload(x), be.upload(stacks[0]), be.upload(stacks[1]), be.upload(ids.view(np.uint8)), be.upload(other.view(np.uint8)),
            be.upload(O.normal(61, t * 256)), be.upload(w0)] + [be.alloc(t * r * n * 4) for _ in range(4)]
    mm = lambda w, i, out: matmul_id_launch(fmt, t, r, e, n, k, inputs=(0, w, i), output=out)
    be.take_launch_count()
    be.execute([mm(1, 3, 7), mm(2, 3, 8)], bufs)
    assert be.take_launch_count() == 2   # the tokens quantized once, one kernel
    be.execute([mm(1, 3, 7), mm(2, 3, 8), mm(1, 4, 9), matmul_launch(fmt, t, k, 256, inputs=(5, 6), output=0), mm(1, 3, 10)], bufs)
    got = [b.download().view(np.float32).copy() for b in bufs[7:]]
    x2 = bufs[0].download().view(np.float32)
    for g, (xs, w, i) in zip(got, [(x, 0, ids), (x, 1, ids), (x, 0, other), (x2, 0, ids)]):
        want = oracle.matmul_id(int(fmt), xs, stacks[w], i, t, r, e, n, k)
        assert _max_rel(g, want) <= 2e-5
    bad = ids.copy()
    bad[-1] = e
    bufs[3].write(0, bad.view(np.uint8))
    with pytest.raises(lp.LapidError) as err:
        be.execute([mm(1, 3, 7), mm(2, 3, 8)], bufs)
    assert err.value.code == "index_out_of_range"


@pytest.mark.parametrize("fmt", [lp.DType.Int8, lp.DType.Int4])
@pytest.mark.parametrize("m,n,k", [
    (1, 33, 32), (3, 40, 288),         # one chunk, two: most warps without a unit
    (2, 11847, 96), (5, 9500, 544),    # several tiles between two barriers, the last of a share alone
    (8, 300, 4128), (4, 2400, 3584),   # more chunks than warps; seven chunks of 512 to eight warps
    (8, 2500, 1024), (3, 100, 8192),   # two chunks; every warp has its place
    (8, 40, 15008), (7, 40, 15616),    # activations that leave room for fewer warps
])
def test_int8_units_of_tiles_and_chunks(be, oracle, fmt, m, n, k):
    qb, a, bias = oracle.quantize(int(fmt), O.normal(n, n * k, 0.02), n, k), O.normal(7 + n, m * k), O.normal(8 + n, n)
    want, path = oracle.matmul(int(fmt), a, qb, n, k, m=m, bias=bias)
    assert path == "int8_act"
    bufs = [be.upload(a), be.upload(qb), be.alloc(m * n * 4), be.upload(bias)]
    be.execute([matmul_launch(fmt, m, n, k, inputs=(0, 1), output=2, bias_input=3)], bufs)
    first = bufs[2].download().view(np.float32).copy()
    assert _max_rel(first, want) <= 2e-5
    be.execute([matmul_launch(fmt, m, n, k, inputs=(0, 1), output=2, bias_input=3)], bufs)
    assert np.array_equal(first, bufs[2].download().view(np.float32))   # the order of the sums does not depend on timing
