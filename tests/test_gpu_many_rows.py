"""The kernels that a prompt's rows take, at the sizes where they can go wrong: edges of the 128-row and 64-deep tiles, remainders, rings that wrap,
grouped heads that do not fill a tile, infinities.  batch_matmul adds in 32 bits: every addition rounds by 2^-24 of the sum so far at most, in either direction,
which for sums of up to 400 terms comes to about sqrt(400) * 2^-24 = 1.2e-6 of sum |terms|; 2e-6 is asked for.  Attention's products on the tensor cores
(csrc/split_gemm.cuh) keep 24 bits of every operand and leave out less than 2^-24 of a term; an accumulator is cut off after 8 additions at most before it
joins a 32-bit sum, so
    |got - exact| <= (2^-24 + 8 * 2^-23 + steps * 2^-24) * sum |terms|
bounds a product of up to `steps` runs of 128 terms: 2e-6 * sum |terms| for sums of up to 2048 terms."""
import numpy as np
import pytest

from oracle import oracle as oc
from oracle.tensor_ref import OracleDevice, OracleTensor
from tests.gpu_common import make_device

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    d = make_device()
    yield d
    d.close()


def tensor(dev, a):
    from crabml_b200 import CudaTensor
    return CudaTensor.new(np.asarray(a, np.float32), list(a.shape), dev)


# ---- rotation of many rows -----------------------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("shape,pos,dims", [([2, 1, 2], 0, 2), ([33, 5, 48], 7, 32), ([300, 3, 128], 100000, 128)])
def test_rotation_of_many_rows_has_the_reference_bits(dev, mode, shape, pos, dims):
    x = np.random.default_rng(0).standard_normal(shape)
    o = OracleTensor.new(x.reshape(-1), shape, OracleDevice()).rope_inplace(mode, pos, dims)
    for _ in range(3):                                     # the staging buffers come round
        np.testing.assert_array_equal(tensor(dev, x).rope_inplace(mode, pos, dims).export().view(np.uint32), o.export().view(np.uint32))


def test_rope_of_positions_asked_for_before_and_not(dev):
    """Runs of positions inside a kept one, behind it, across its end, of other shapes, more than are kept, longer than one may be: the bits of the rows by themselves"""
    rng = np.random.default_rng(3)
    for mode, hd, dims, pos, n in ((0, 64, 64, 0, 40), (0, 64, 64, 5, 30), (0, 64, 64, 40, 24), (0, 64, 64, 30, 60), (0, 64, 32, 3, 20), (1, 64, 64, 3, 20), (0, 128, 128, 7, 20), (0, 64, 64, 900, 33),
                                   (0, 64, 64, 0, 70), (0, 64, 64, 0, 16500), (0, 64, 64, 16490, 12), (0, 64, 64, 899, 2)):
        x = rng.standard_normal((n, 2 * hd)).astype(np.float32)
        got = tensor(dev, x.reshape(n, 2, hd)).rope_inplace(mode, pos, dims).export().reshape(n, 2, hd)
        for r in {0, 1, n // 2, n - 1}:
            one = tensor(dev, x[r:r + 1].reshape(1, 2, hd)).rope_inplace(mode, pos + r, dims).export().reshape(2, hd)
            np.testing.assert_array_equal(got[r].view(np.uint32), one.view(np.uint32))


# ---- softmax: many rows and one row at a time give the same bits ------------------------------------------------------------------------------
@pytest.mark.parametrize("cols", [1, 31, 512, 513, 1025, 2048, 2049])
def test_softmax_of_many_rows_has_the_bits_of_one(dev, cols):
    x = np.random.default_rng(cols).standard_normal((700, cols)).astype(np.float32) * 3
    many = tensor(dev, x).softmax_inplace(1).export().reshape(x.shape)
    for r in (0, 1, 350, 699):
        np.testing.assert_array_equal(many[r].view(np.uint32), tensor(dev, x[r:r + 1]).softmax_inplace(1).export().view(np.uint32))


# ---- batch_matmul of many rows ------------------------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("kind", ["f32", "f16"])
@pytest.mark.parametrize("ab,bb,m,k,n", [(2, 1, 16, 48, 17), (6, 2, 127, 64, 128), (4, 4, 128, 65, 129), (3, 3, 129, 200, 5), (8, 2, 300, 128, 333)])
def test_batch_matmul_of_many_rows(dev, kind, ab, bb, m, k, n):
    from crabml_b200 import CudaTensor, capi
    rng = np.random.default_rng(m)
    a = rng.standard_normal((ab, m, k)).astype(np.float32)
    rows = rng.standard_normal((n, bb, k)).astype(np.float32)          # n cached rows per head, as the key cache holds them
    cache = CudaTensor.alloc([bb, n + 3, k], capi.F16 if kind == "f16" else capi.F32, dev).resize(1, 0)
    cache.concatenate(tensor(dev, rows).transpose([1, 0, 2]), 1)
    if kind == "f16":
        a, rows = a.astype(np.float16).astype(np.float32), rows.astype(np.float16).astype(np.float32)
    head = np.arange(ab) % bb if kind == "f32" else np.arange(ab) // (ab // bb)
    b = rows.transpose(1, 0, 2)[head].astype(np.float64)               # [ab, n, k]
    got = tensor(dev, a).batch_matmul(cache.transpose([0, 2, 1])).export().reshape(ab, m, n)
    want, size = np.einsum("amk,ank->amn", a, b), np.einsum("amk,ank->amn", np.abs(a), np.abs(b))
    assert (np.abs(got - want) <= 2e-6 * size).all()
    if kind == "f32":                                                  # [ab, m, n] x [bb, n, k]: the value product (f16 keeps its own order of sums)
        w = np.abs(rng.standard_normal((ab, m, n))).astype(np.float32)
        got = tensor(dev, w).batch_matmul(cache).export().reshape(ab, m, k)
        want, size = np.einsum("amn,ank->amk", w, b), np.einsum("amn,ank->amk", w, np.abs(b))
        assert (np.abs(got - want) <= 2e-6 * size).all()


@pytest.mark.parametrize("kind", ["f32", "f16"])
@pytest.mark.parametrize("ab,bb,m,k,n", [(2, 1, 4, 1, 1), (2, 2, 9, 31, 33), (4, 2, 64, 128, 32), (6, 3, 65, 67, 63), (8, 2, 130, 160, 129)])
def test_batch_matmul_of_many_rows_has_the_bits_of_one(dev, kind, ab, bb, m, k, n):
    """32-bit sums in the order of a single row's, whatever the number of rows; numbers of very different size on both sides"""
    from crabml_b200 import CudaTensor, capi
    rng = np.random.default_rng(m + k)
    a = (rng.standard_normal((ab, m, k)) * np.exp2(rng.integers(-12, 12, (ab, m, k)))).astype(np.float32)
    cache = CudaTensor.alloc([bb, n + 3, k], capi.F16 if kind == "f16" else capi.F32, dev).resize(1, 0)
    cache.concatenate(tensor(dev, np.abs(rng.standard_normal((n, bb, k)))).transpose([1, 0, 2]), 1)
    for left, right in ((a, cache.transpose([0, 2, 1])), (rng.standard_normal((ab, m, n)), cache)):
        got = tensor(dev, left).batch_matmul(right).export().reshape(ab, m, -1)
        for r in sorted({0, 3, m // 2, m - 1}):
            one = tensor(dev, left[:, r:r + 1]).batch_matmul(right).export().reshape(ab, -1)
            np.testing.assert_array_equal(got[:, r].view(np.uint32), one.view(np.uint32))


def test_batch_matmul_spreads_infinities_like_a_sum_of_products(dev):
    rng = np.random.default_rng(1)
    a, b = rng.standard_normal((1, 40, 70)).astype(np.float32), rng.standard_normal((1, 70, 50)).astype(np.float32)
    a[0, 3, 5], a[0, 7, 9], b[0, 11, 2], b[0, 5, 4] = np.inf, np.nan, -np.inf, 0.0
    with np.errstate(invalid="ignore"):
        want = np.einsum("amk,akn->amn", a.astype(np.float64), b.astype(np.float64))
    got = tensor(dev, a).batch_matmul(tensor(dev, b)).export().reshape(want.shape)
    fine = np.isfinite(want)
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
    np.testing.assert_array_equal(got[~fine & ~np.isnan(want)], want[~fine & ~np.isnan(want)])
    np.testing.assert_allclose(got[fine], want[fine], rtol=0, atol=2e-4)


# ---- attention over a ring ------------------------------------------------------------------------------------------------------------------------
def attend(q, k, v, scale, pos0, window, block, cap, sink):
    """q [T, H, dk]; k, v: row j is position j; -> [T, H, dv] in 64 bits"""
    T, H = q.shape[:2]
    R, out = H // k.shape[1], np.zeros((T, H, v.shape[2]))
    for t in range(T):
        i = pos0 + t
        lo = max(0, i - window + 1) if window else 0
        lo = max(lo, i - i % block) if block else lo
        for h in range(H):
            s = k[lo:i + 1, h // R].astype(np.float64) @ q[t, h].astype(np.float64) * scale
            s = cap * np.tanh(s / cap) if cap else s
            top = max(s.max(), sink[h]) if sink is not None else s.max()
            e = np.exp(s - top)
            out[t, h] = e @ v[lo:i + 1, h // R] / (e.sum() + (np.exp(sink[h] - top) if sink is not None else 0.0))
    return out


CASES = [  # T, pos0, H, G, dk, dv, window, block, cap, sink, latent
    (65, 0, 1, 1, 64, 64, 0, 0, 0.0, False, False),
    (33, 63, 6, 2, 80, 40, 50, 0, 0.0, True, False),          # three heads per key head: 126 of a tile's 128 rows ; a window that ends inside steps
    (130, 129, 2, 2, 128, 128, 0, 0, 5.0, False, False),
    (7, 1000, 10, 1, 36, 132, 64, 0, 0.0, False, False),      # dk not a whole step, dv one column group and four columns
    (200, 100, 4, 4, 64, 200, 0, 96, 0.0, True, False),       # blocks of positions
    (40, 300, 8, 1, 192, 128, 0, 0, 0.0, False, True),        # a key row's first dv columns are its value
    (129, 511, 3, 1, 30, 30, 128, 0, 0.0, False, False),      # rows that cannot be read 16 bytes at a time
]


def rings(k, v, pos, ring):
    """positions pos of k, v in the rows p % ring"""
    kr, vr = np.full((ring,) + k.shape[1:], np.nan, np.float32), None if v is None else np.full((ring,) + v.shape[1:], np.nan, np.float32)
    kr[pos % ring] = k[pos]
    if v is not None:
        vr[pos % ring] = v[pos]
    return kr, vr


@pytest.mark.parametrize("T,pos0,H,G,dk,dv,window,block,cap,sink,latent", CASES)
def test_attention_of_many_rows(dev, T, pos0, H, G, dk, dv, window, block, cap, sink, latent):
    from crabml_b200 import seqops
    rng = np.random.default_rng(T)
    n = pos0 + T
    q, k = rng.standard_normal((T, H, dk)).astype(np.float32), rng.standard_normal((n, G, dk)).astype(np.float32)
    v = k[..., :dv] if latent else rng.standard_normal((n, G, dv)).astype(np.float32)
    sk = rng.standard_normal(H).astype(np.float32) if sink else None
    first = max(0, pos0 - window + 1) if window else 0
    first = max(first, pos0 - pos0 % block) if block else first
    ring = n - first + 5                                       # rows nobody may look at hold NaN
    kr, vr = rings(k, None if latent else v, np.arange(first, n), ring)
    args = dict(window=window, block=block, softcap=cap, sink=None if sk is None else tensor(dev, sk))
    kt, vt = tensor(dev, kr.reshape(ring, -1)), None if latent else tensor(dev, vr.reshape(ring, -1))
    got = seqops.masked_attention_capped(tensor(dev, q.reshape(T, -1)), kt, vt, pos0, H, G, dk, dv, dk ** -0.5, **args).export().reshape(T, H, dv)
    want = attend(q, k, v, dk ** -0.5, pos0, window, block, cap, sk)
    # a score's error moves its weight by as much, the weights' and sums' roundings are a few 2^-24 each: 1e-5 of the values' size
    assert np.abs(got - want).max() <= 1e-5
    # however a portion is cut, a query keeps its bits while both cuts have many rows
    cut = T // 2
    if cut * H > 64 and (T - cut) * H > 64:
        for a, b in ((0, cut), (cut, T)):
            part = seqops.masked_attention_capped(tensor(dev, q[a:b].reshape(b - a, -1)), kt, vt, pos0 + a, H, G, dk, dv, dk ** -0.5, **args).export().reshape(b - a, H, dv)
            np.testing.assert_array_equal(part.view(np.uint32), got[a:b].view(np.uint32))


def test_attention_keeps_an_infinite_value_to_the_queries_that_see_it(dev):
    from crabml_b200 import seqops
    rng = np.random.default_rng(3)
    T, H, d = 96, 2, 64
    q, k, v = (rng.standard_normal((T, H, d)).astype(np.float32) for _ in range(3))
    v[70, 1, 5] = np.inf
    got = seqops.masked_attention(tensor(dev, q.reshape(T, -1)), tensor(dev, k.reshape(T, -1)), tensor(dev, v.reshape(T, -1)), 0, H, H, d, d, d ** -0.5).export().reshape(T, H, d)
    bad = np.zeros(got.shape, bool)
    bad[70:, 1, 5] = True
    assert np.isposinf(got[bad]).all() and np.isfinite(got[:70]).all() and np.isfinite(got[70:, 0]).all()
    assert np.isfinite(np.delete(got[70:, 1], 5, 1)).all()


@pytest.mark.parametrize("window", [256, 512, 1024])
def test_a_windowed_query_keeps_its_bits_wherever_its_call_starts(dev, window):
    """Tiles of queries begin with the call, steps and runs of keys at positions: a query must not see which tile it fell into."""
    from crabml_b200 import seqops
    H, G, d, n = 4, 1, 128, 2012
    rng = np.random.default_rng(window)
    q, k, v = (rng.standard_normal((n, h * d)).astype(np.float32) for h in (H, G, G))
    kt, vt = tensor(dev, k), tensor(dev, v)

    def call(lo, hi):
        return seqops.masked_attention(tensor(dev, q[lo:hi]), kt, vt, lo, H, G, d, d, d ** -0.5, window=window).export().reshape(hi - lo, H * d).view(np.uint32)
    whole = call(1500, n)
    for lo, hi in ((1501, n), (1531, n), (1564, 1700), (1627, n)):
        np.testing.assert_array_equal(call(lo, hi), whole[lo - 1500:hi - 1500])


def test_attention_weighs_scores_of_any_size(dev):
    """Equal scores weigh the same however large they are: exp(score - largest) and no other form of it"""
    from crabml_b200 import seqops
    T, d = 80, 64
    for size in (1.0, 1e10, 1.69e19):
        q, k, v = np.zeros((T, 4), np.float32), np.zeros((T, 4), np.float32), np.random.default_rng(5).standard_normal((T, d)).astype(np.float32)
        q[:, 1], k[:, 1] = size, size
        got = seqops.masked_attention(tensor(dev, q), tensor(dev, k), tensor(dev, v), 0, 1, 1, 4, d, 1.0).export().reshape(T, d)
        want = np.cumsum(v.astype(np.float64), 0) / np.arange(1, T + 1)[:, None]
        assert np.abs(got - want).max() <= 2e-6, size


@pytest.mark.parametrize("bits", [0x3f80ffff, 0x3f807f7f, 0x3f807ebf, 0x3f8101ff, 0x3faaaaab, 0x3fff7fff, 0x3fd5c28f])
def test_attention_scores_of_operands_that_use_all_their_bits(dev, bits):
    """Keys of the odd positions are the nearest bfloat16 number to those of the even ones and lose nothing when they are cut.  A score s of one term: 2^-24 s at
    most is left out, the accumulators cut off twice at 2^-23, the scale rounds once at 2^-24; a weight of two nearly equal ones moves by a quarter of that."""
    from crabml_b200 import seqops
    x = np.array([bits], np.uint32).view(np.float32)[0]
    near = np.array([(bits + 0x8000) & 0xffff0000], np.uint32).view(np.float32)[0]
    T, d = 130, 64
    scale = np.float32(60.0)
    q, k, v = np.full((T, 1), x, np.float32), np.full((T, 1), x, np.float32), np.zeros((T, d), np.float32)
    k[1::2], v[::2] = near, 1.0
    got = seqops.masked_attention(tensor(dev, q), tensor(dev, k), tensor(dev, v), 0, 1, 1, 1, d, scale).export().reshape(T, d)
    want = attend(q[:, None], k[:, None], v[:, None], float(scale), 0, 0, 0, 0.0, None)[:, 0]
    s = float(x) * float(x) * float(scale)
    assert np.abs(got - want).max() <= 0.25 * s * (2.0 ** -24 + 2 * 2.0 ** -23 + 2.0 ** -24) + 4 * 2.0 ** -24


@pytest.mark.parametrize("T,pos0,H,G,d,window,sink", [
    (1, 300, 80, 80, 64, 0, False),               # a decoded token of more heads than 64
    (1, 500, 128, 4, 64, 200, True),              # .. of many heads a key head: four reads of the cache
    (2, 250, 64, 8, 80, 0, False),                # two queries, the last count that goes row by row
    (1, 40000, 8, 1, 64, 0, True),                # a slice of keys that shared memory does not hold: chunks
    (2, 90000, 3, 1, 32, 0, False),               # .. of the kernel that takes four heads together; queries that see different numbers of keys
])
def test_attention_of_few_queries(dev, T, pos0, H, G, d, window, sink):
    from crabml_b200 import seqops
    rng = np.random.default_rng(H)
    n = pos0 + T
    q, k, v = (rng.standard_normal((r, h, d)).astype(np.float32) for r, h in ((T, H), (n, G), (n, G)))
    k[n // 2:] *= 1.5                             # larger scores behind smaller ones
    sk = rng.standard_normal(H).astype(np.float32) if sink else None
    kt, vt, st = tensor(dev, k.reshape(n, -1)), tensor(dev, v.reshape(n, -1)), None if sk is None else tensor(dev, sk)

    def call(a, b):
        qt, launches = tensor(dev, q[a:b].reshape(b - a, -1)), dev.launch_count()
        out = seqops.masked_attention(qt, kt, vt, pos0 + a, H, G, d, d, d ** -0.5, window=window, sink=st)
        assert dev.launch_count() - launches == 2         # scores and values, and no cut of the cache in front of them
        return out.export().reshape(b - a, H, d)
    got = call(0, T)
    # a score's error moves its weight by as much, the weights' and sums' roundings are a few 2^-24 each: 1e-5 of the values' size
    assert np.abs(got - attend(q, k, v, d ** -0.5, pos0, window, 0, 0.0, sk)).max() <= 1e-5
    for t in range(T):                            # a row's bits do not depend on what else the call carries
        np.testing.assert_array_equal(call(t, t + 1)[0].view(np.uint32), got[t].view(np.uint32))


@pytest.mark.parametrize("T,n,H,G,dk,dv,latent", [
    (1, 1, 1, 1, 1, 1, False), (2, 3, 3, 1, 7, 5, False), (3, 130, 8, 8, 33, 34, False),      # rows that are no multiple of 16 bytes
    (1, 127, 4, 1, 128, 128, False), (1, 128, 4, 1, 128, 128, False), (1, 129, 4, 1, 128, 128, False), (2, 129, 4, 1, 128, 128, False),      # one slice, or two
    (1, 700, 2, 1, 64, 64, False), (1, 9000, 2, 1, 16, 16, False),                             # weights in one piece, in several
    (2, 31, 8, 1, 576, 512, True), (1, 32, 5, 1, 576, 512, True), (1, 500, 16, 1, 576, 512, True), (1, 65, 17, 1, 132, 131, True), (1, 1200, 64, 1, 80, 80, False),
    (1, 64, 8, 1, 64, 64, False), (2, 66, 8, 1, 64, 64, False), (1, 32, 16, 1, 64, 80, False), (2, 34, 16, 1, 64, 80, False), (1, 200, 2, 2, 64, 64, False), (1, 46, 1, 1, 576, 512, True),      # one slice, or several
    (1, 13000, 16, 1, 576, 512, True),                                                         # slices too long to stay in shared memory
    (1, 40, 1, 1, 64, 1025, False), (1, 40, 2, 1, 64, 1028, False), (2, 40, 4, 1, 64, 1025, False), (1, 300, 8, 2, 32, 1028, False), (1, 40, 8, 1, 64, 1028, False), (1, 5, 1, 1, 64, 2049, False),      # a last block of few columns
    (1, 300, 9, 1, 256, 256, False), (1, 40, 2, 1, 64, 1500, False), (1, 40, 2, 1, 5000, 64, False), (1, 40, 16, 1, 2000, 40, True)])
def test_attention_of_few_queries_at_the_edges_of_its_slices(dev, T, n, H, G, dk, dv, latent):
    """Edges of slices, tiles and blocks of heads and columns, a ring that wraps around, and the order of a row's sums beside other rows"""
    from crabml_b200 import seqops
    rng = np.random.default_rng(n + H + dk)
    q, k = rng.standard_normal((T, H, dk)).astype(np.float32), rng.standard_normal((n, G, dk)).astype(np.float32)
    v = k[..., :dv] if latent else rng.standard_normal((n, G, dv)).astype(np.float32)
    sk = rng.standard_normal(H).astype(np.float32)
    ring = n + 3                                   # a ring that wraps: position p lies in row p % ring, and positions start at 2 ring - 5
    first = 2 * ring - 5
    order = np.argsort(np.r_[(first + np.arange(n)) % ring, np.setdiff1d(np.arange(ring), (first + np.arange(n)) % ring)])
    kt, vt = (tensor(dev, np.concatenate([x, np.full((3,) + x.shape[1:], np.nan, np.float32)])[order].reshape(ring, -1)) for x in (k, v))
    vt, st = None if latent else vt, tensor(dev, sk)
    window = n - T + 1                             # the first query sees the oldest row

    def call(a, b):
        return seqops.masked_attention(tensor(dev, q[a:b].reshape(b - a, -1)), kt, vt, first + n - T + a, H, G, dk, dv, dk ** -0.5, window=window, sink=st).export().reshape(b - a, H, dv)
    got = call(0, T)
    want = np.stack([attend(q[t:t + 1], k[t:n - T + 1 + t], v[t:n - T + 1 + t], dk ** -0.5, n - T, 0, 0, 0.0, sk)[0] for t in range(T)])
    # as above: 1e-5 of the values' size
    assert np.abs(got - want).max() <= 1e-5
    for t in range(T):
        np.testing.assert_array_equal(call(t, t + 1)[0].view(np.uint32), got[t].view(np.uint32))


@pytest.mark.parametrize("T,n,G,dk,dv", [(2, 18, 1050, 1024, 4096), (1, 2, 33000, 1, 1025)])
def test_attention_of_few_queries_in_portions(dev, T, n, G, dk, dv):
    """Slices of two queries whose sums take 69 MB each, and more blocks of value columns than a grid has units: portions of queries and of heads"""
    from crabml_b200 import seqops
    rng = np.random.default_rng(G)
    q, k, v = (rng.standard_normal(s, np.float32) for s in ((T, G, dk), (n, G, dk), (n, G, dv)))
    kt, vt = tensor(dev, k.reshape(n, -1)), tensor(dev, v.reshape(n, -1))
    qt, launches = tensor(dev, q.reshape(T, -1)), dev.launch_count()
    got = seqops.masked_attention(qt, kt, vt, n - T, G, G, dk, dv, dk ** -0.5)
    assert dev.launch_count() - launches == (4 if T == 2 else 2)
    got = got.export().reshape(T, G, dv)
    for t in range(T):
        seen = n - T + 1 + t
        s = np.einsum("gd,ngd->gn", q[t].astype(np.float64), k[:seen].astype(np.float64)) * dk ** -0.5
        w = np.exp(s - s.max(1, keepdims=True))
        want = np.einsum("gn,ngd->gd", (w / w.sum(1, keepdims=True)).astype(np.float32), v[:seen], optimize=True)
        # scores stay below 7 (one product: below 20, two keys), whose up to 1024 products and sums are off by 2^-24 of 7 a few times over; a weight moves by that share, a result by that share of values below 7.  (Scores
        # of 70, by a scale of 1/2, are off by 1e-5 and with them the results.)
        assert np.abs(got[t] - want).max() <= 1e-5
    one = seqops.masked_attention(tensor(dev, q[T - 1:].reshape(1, -1)), kt, vt, n - 1, G, G, dk, dv, dk ** -0.5).export().reshape(G, dv)
    np.testing.assert_array_equal(one.view(np.uint32), got[T - 1].view(np.uint32))


def test_attention_of_many_rows_over_a_long_cache_takes_its_heads_in_groups(dev):
    """16 heads over 40,000 keys: 820 MB of scores and cut planes where the scores of 33 queries take 84"""
    from crabml_b200 import seqops
    T, pos0, H, d = 33, 40000, 16, 64
    rng = np.random.default_rng(0)
    n = pos0 + T
    q, k, v = (rng.standard_normal((r, H, d)).astype(np.float32) for r in (T, n, n))
    t = [tensor(dev, x.reshape(x.shape[0], -1)) for x in (q, k, v)]
    launches = dev.launch_count()
    out = seqops.masked_attention(*t, pos0, H, H, d, d, d ** -0.5)
    assert dev.launch_count() - launches == 6     # two groups: cut, scores, values
    got = out.export().reshape(T, H, d)
    assert np.abs(got - attend(q, k, v, d ** -0.5, pos0, 0, 0, 0.0, None)).max() <= 1e-5


@pytest.mark.parametrize("pos0,window", [(0, 0), (300, 0), (300, 257), (1000, 700)])
def test_attention_of_more_tiles_than_ctas(dev, pos0, window):
    """A CTA walks over several tiles of scores and of values, of odd and even numbers of steps, skipped ones among them; an infinity in a late one stays there."""
    from crabml_b200 import seqops
    T, H, dk, dv = 512, 16, 192, 200
    rng = np.random.default_rng(pos0 + window)
    n = pos0 + T
    q, k, v = (rng.standard_normal((r, H, d)).astype(np.float32) for r, d in ((T, dk), (n, dk), (n, dv)))
    v[n - 20, H - 1, 3] = np.inf
    got = seqops.masked_attention(tensor(dev, q.reshape(T, -1)), tensor(dev, k.reshape(n, -1)), tensor(dev, v.reshape(n, -1)), pos0, H, H, dk, dv, dk ** -0.5, window=window).export().reshape(T, H, dv)
    bad = np.zeros(got.shape, bool)
    bad[T - 20:, H - 1, 3] = True
    assert np.isposinf(got[bad]).all() and np.isfinite(got[~bad]).all()
    v[n - 20, H - 1, 3] = 0.0
    want = attend(q, k, v, dk ** -0.5, pos0, window, 0, 0.0, None)
    assert np.abs(got - want)[~bad].max() <= 1e-5


# ---- a few activation rows against one quantised matrix ---------------------------------------------------------------------------------------------
@pytest.mark.parametrize("t", [oc.Q4_K, oc.Q5_K, oc.Q6_K])
@pytest.mark.parametrize("m,k,b", [(1, 256, 2), (33, 1024, 3), (40, 2816, 8), (257, 4096, 9), (17, 14336, 31), (16, 40960, 5)])
def test_few_rows_have_the_bits_of_one(dev, t, m, k, b):
    from crabml_b200 import CudaTensor
    from tests.blockgen import random_weight
    rng = np.random.default_rng(m + b)
    w = CudaTensor.from_cpu(random_weight(t, m, k, rng, 0.02), [m, k], t, dev)
    x = rng.standard_normal((b, k)).astype(np.float32)
    got = w.matmul_vec(tensor(dev, x)).export().reshape(b, m)
    for i in range(b):
        np.testing.assert_array_equal(got[i].view(np.uint32), w.matmul_vec(tensor(dev, x[i:i + 1])).export().view(np.uint32))


@pytest.mark.parametrize("m,k,b", [(1, 256, 5), (16, 512, 6), (31, 768, 7), (32, 1280, 8), (47, 1536, 12), (9600, 256, 17), (4800, 2048, 5), (3, 18944, 31)])
def test_few_rows_of_q4_k_have_the_bits_of_one(dev, m, k, b):
    """Edges of the tiles of 16 and 32 rows and of 8 activations, super-blocks fewer than warps and no multiple of 4, more tiles than CTAs"""
    test_few_rows_have_the_bits_of_one(dev, oc.Q4_K, m, k, b)


@pytest.mark.parametrize("m,k,b", [(33, 16896, 8), (1, 17152, 5), (45, 17152, 12), (1217, 17152, 31), (31, 18688, 31), (50, 18688, 7), (20, 18944, 8)])
def test_few_rows_of_q4_k_with_long_activations_have_the_bits_of_one(dev, m, k, b):
    """66 super-blocks are the most that leave room for four stages of weights a warp, 67 to 73 have two (1217 rows: more tiles than CTAs, so the stages fill again), 74 go without the tensor cores"""
    test_few_rows_have_the_bits_of_one(dev, oc.Q4_K, m, k, b)


@pytest.mark.parametrize("t", [oc.Q8_0, oc.Q4_0, oc.Q5_0])
@pytest.mark.parametrize("m,k,b", [(1, 32, 2), (33, 288, 3), (40, 1056, 8), (257, 4096, 9), (17, 14336, 31), (16, 40960, 5)])
def test_few_rows_against_the_oracle(dev, t, m, k, b):
    from tests.test_gpu_matvec import run_case
    run_case(dev, t, m, k, b=b, seed=m + b)


# ---- gated delta rule: any cut of the tokens gives the same bits, columns that do not fill a CTA -------------------------------------------------------
@pytest.mark.parametrize("dk,dv,H,G", [(128, 128, 2, 1), (128, 20, 3, 3), (64, 33, 4, 2), (32, 64, 2, 2), (36, 70, 2, 1)])
def test_delta_rule_however_the_tokens_are_cut(dev, dk, dv, H, G):
    from crabml_b200 import seqops
    rng = np.random.default_rng(dk + dv)
    T = 37
    q, k, v = rng.standard_normal((T, G, dk)) / dk ** 0.5, rng.standard_normal((T, G, dk)), rng.standard_normal((T, H, dv))
    k /= np.linalg.norm(k, axis=-1, keepdims=True)
    a, b, a_log, dt = rng.standard_normal((T, H)), rng.standard_normal((T, H)), np.log(rng.uniform(0.5, 4, H)), rng.uniform(-3, 0, H)
    S0 = rng.standard_normal((H, dk, dv))

    def run(cuts):
        state, outs = tensor(dev, S0.reshape(-1)), []
        for lo, hi in zip(cuts, cuts[1:]):
            t = [tensor(dev, x[lo:hi].reshape(hi - lo, -1)) for x in (q, k, v, a, b)]
            outs.append(seqops.gated_delta_rule(*t, tensor(dev, a_log), tensor(dev, dt), state, H, G, dk, dv).export())
        return np.concatenate(outs).reshape(T, H, dv), state.export().reshape(S0.shape)
    got, end = run([0, T])
    for cuts in ([0, 1, 2, 18, T], [0, 16, 32, T]):
        o, s = run(cuts)
        np.testing.assert_array_equal(o.view(np.uint32), got.view(np.uint32))
        np.testing.assert_array_equal(s.view(np.uint32), end.view(np.uint32))
    S = np.asarray(S0, np.float32).astype(np.float64)
    f = [np.asarray(x, np.float32).astype(np.float64) for x in (q, k, v, a, b, a_log, dt)]
    beta, decay = 1 / (1 + np.exp(-f[4])), np.exp(-np.exp(f[5]) * np.log1p(np.exp(f[3] + f[6])))
    for t in range(T):
        for h in range(H):
            S[h] *= decay[t, h]
            kt = f[1][t, h // (H // G)]
            S[h] += np.outer(kt, beta[t, h] * (f[2][t, h] - S[h].T @ kt))
            # 32-bit sums of dk terms of order one, carried on by a contraction: 1e-5
            assert np.abs(got[t, h] - S[h].T @ f[0][t, h // (H // G)]).max() < 1e-5
    assert np.abs(end - S).max() < 1e-5


# ---- a prompt in one call: the joined steps of a recording device give the bits of the separate ones ----------------------------------------------------
@pytest.mark.parametrize("arch", ["llama", "qwen2"])
@pytest.mark.parametrize("wtype", ["Q8_0", "Q4_0", "Q4_K"])
@pytest.mark.parametrize("tokens", [33, 200])
def test_prompt_recorded_and_eager_agree(arch, wtype, tokens):
    from crabml_b200 import CudaTensor, CudaTensorDevice, capi
    from crabml_b200 import runner as R
    conf = R.LlamaConfig(4, 2, 2, 512, 768, 512, 1000, 1e-5, 128, arch)
    ids = np.random.default_rng(tokens).integers(0, 1000, tokens).tolist()
    got = []
    for lazy in (0, 1, 2):
        d = CudaTensorDevice(0, lazy=lazy)
        w = R.synthetic_weights(d, conf, getattr(capi, wtype), capi.Q8_0, seed=5)
        if arch == "qwen2":
            rng = np.random.default_rng(9)
            for name, n in (("bq", 512), ("bk", 256), ("bv", 256)):
                w[name] = [CudaTensor.from_cpu(rng.standard_normal(n).astype(np.float32), [n], capi.F32, d) for _ in range(2)]
        r = R.LlamaRunner(d, conf, w, 256)
        a = r.forward(ids, 0).copy()
        b = r.forward(ids[:3], tokens).copy()                 # a short portion behind it, and a token
        c = r.forward(ids[:1], tokens + 3).copy()
        got.append(np.stack([a, b, c]))
        r.close()
        del w
        d.close()
    assert np.isfinite(got[0]).all()
    for g in got[1:]:
        np.testing.assert_array_equal(g.view(np.uint32), got[0].view(np.uint32))


@pytest.mark.parametrize("wt,ct", [(oc.Q8_0, oc.Q8_0), (oc.Q4_K, oc.Q6_K)])
@pytest.mark.parametrize("f16_kv", [False, True])
def test_long_tokens_run_in_two_parts_with_the_same_bits(wt, ct, f16_kv):
    """Six layers are recorded as more than one part; the cache's length crosses the 512 positions up to which the persistent kernels' attention keeps an
    exponential per thread.  Every mode reduces in the same order, so the logits are the eager calls' bit for bit."""
    from crabml_b200 import runner as R
    conf = R.LlamaConfig(4, 2, 6, 256, 512, 600, 512, 1e-5, 64)
    prompt = [1 + (7 * i) % 500 for i in range(506)]
    res = {}
    for lazy in (0, 1, 2):
        dev = make_device(lazy=lazy)
        try:
            r = R.LlamaRunner(dev, conf, R.synthetic_weights(dev, conf, wt, ct, seed=3), 600, f16_kv=f16_kv)
            first = [r.forward([t], p).copy() for p, t in enumerate([5, 6, 7])]
            r.forward(prompt, 3)
            before, launches = dev.lazy_stats() if lazy else None, dev.launch_count()
            late = [r.forward([t], 3 + len(prompt) + p).copy() for p, t in enumerate(range(11, 19))]
            res[lazy] = np.stack(first + late)
            if lazy:                                          # two plans a token, captured once or twice (the pool's buffers settle after the prompt), replayed from then on
                st = dev.lazy_stats()
                runs, captures = (st["graph_replays"] + st["graph_captures"] - before["graph_replays"] - before["graph_captures"], st["graph_captures"] - before["graph_captures"])
                assert st["uncached"] == before["uncached"] and runs == 16 and captures <= 4, (before, st)
            if lazy == 2:
                assert dev.launch_count() - launches == 16    # a persistent kernel per part
            r.close()
        finally:
            dev.close()
    assert np.isfinite(res[0]).all() and np.abs(res[0]).max() > 0
    for mode in (1, 2):
        np.testing.assert_array_equal(res[mode].view(np.uint32), res[0].view(np.uint32), err_msg=f"lazy={mode} vs eager")
