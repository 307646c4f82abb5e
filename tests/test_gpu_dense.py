"""Dense quantised GEMM (the reference's gemm_q8_0 / gemm_iq4_xs prefill projections) on the
tensor-core pipeline against the oracle's f64 GEMV, row by row.  f16 operands, x and a weight's scale and product rounded to
2^-11 each: 5e-3 relative for the worst element (row-scaled; about 0.35e-3 as a norm)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 5e-3


@pytest.fixture(scope="module")
def ctx(pkg):
    c = pkg.Context(pkg.synth.Dims(), n_layer=1, max_tokens=1, device=0)
    yield c
    c.close()


@pytest.mark.parametrize("ttype", [8, 23])
@pytest.mark.parametrize("M,K,n", [(512, 256, 1), (1024, 2048, 130), (4096, 2048, 300), (2048, 4096, 64)])
def test_dense_gemm(ctx, orc, syn, ttype, M, K, n):
    W = syn.random_blocks(ttype, M, K, seed=17, tag="dense")
    x = syn.random_x(n, K, seed=18)
    ctx.dense_upload(3, ttype, W, M, K)
    d_x, d_y = ctx.to_device(x), ctx.alloc(n * M * 4)
    ctx.dense_gemm(3, d_x, n, d_y)
    y = d_y.download(np.float32, (n, M))
    rows = sorted(set([0, n - 1, n // 2] + list(range(0, n, max(1, n // 6)))))
    want = np.stack([orc.gemv(ttype, W, x[r], M, K, threads=orc.hardware_threads()) for r in rows])
    assert syn.rel_err_rows(y[rows], want) < TOL
    # a second call with fewer rows reuses the scratch
    ctx.dense_gemm(3, d_x, 1, d_y)
    assert syn.rel_err_rows(d_y.download(np.float32, (1, M)), want[:1]) < TOL
    d_x.free(); d_y.free()


@pytest.mark.parametrize("ttype", [8, 23])
@pytest.mark.parametrize("M,K,n", [(128, 256, 16), (384, 768, 65), (640, 1280, 129), (256, 512, 64), (4480, 256, 257)])
def test_dense_gemm_edges(ctx, orc, syn, ttype, M, K, n):
    """An odd number of 256-column blocks, a lone last row tile, row counts around the 64-row change of accumulator
    sets and the 128-row unit, more units than blocks."""
    W = syn.random_blocks(ttype, M, K, seed=19, tag="dense")
    x = syn.random_x(n, K, seed=20)
    x[n // 2] *= 1e4
    ctx.dense_upload(4, ttype, W, M, K)
    d_x, d_y = ctx.to_device(x), ctx.alloc(n * M * 4)
    ctx.dense_gemm(4, d_x, n, d_y)
    ctx.sync()
    want = orc.gemv(ttype, W, x, M, K, threads=orc.hardware_threads())
    assert syn.rel_err_rows(d_y.download(np.float32, (n, M)), want) < TOL
    d_x.free(); d_y.free()


@pytest.mark.parametrize("ttype,lo,hi", [(8, 6e-8, 1e-6), (23, 6e-8, 1e-6), (23, 1e-5, 1e-4), (8, 300.0, 2000.0), (23, 5.0, 100.0), (8, 2e4, 6.5e4), (23, 2e4, 6.5e4)])
def test_dense_gemm_weight_range(ctx, orc, syn, ttype, lo, hi):
    """Block scales from f16's smallest subnormal to its largest number: weights as f16 operands would overflow above 65504
    (IQ4_XS from d = 16 on, Q8_0 from 512).  Rounding: x 2^-11, a weight's scale and product 2^-11 each."""
    M, K, n = 256, 512, 70
    W = syn.random_blocks(ttype, M, K, seed=21, tag="dense", scale=(lo, hi))
    x = syn.random_x(n, K, seed=22)
    ctx.dense_upload(6, ttype, W, M, K)
    d_x, d_y = ctx.to_device(x), ctx.alloc(n * M * 4)
    ctx.dense_gemm(6, d_x, n, d_y)
    want = orc.gemv(ttype, W, x, M, K, threads=orc.hardware_threads())
    got = d_y.download(np.float32, (n, M)).astype(np.float64)
    # independent roundings of K products: 3 * 2^-11 of the result's size at the very most, as a norm
    assert np.linalg.norm(got - want) < 3 * 2.0**-11 * np.linalg.norm(want)
    assert syn.rel_err_rows(got, want) < 5e-3
    d_x.free(); d_y.free()


@pytest.mark.parametrize("ttype", [8, 23])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 3.4e38])
def test_dense_gemm_extreme_rows(ctx, orc, syn, ttype, value):
    """An infinity, a NaN or an element near the largest float beside ordinary large ones: the outputs that are infinite, NaN and
    finite are those of the f32 formula, and other rows do not notice."""
    M, K, n = 256, 512, 20
    W = syn.random_blocks(ttype, M, K, seed=23, tag="dense", scale=(1e-4, 1e-3))
    x = syn.random_x(n, K, seed=24) * np.float32(1e6)
    x[3, 77] = value
    ctx.dense_upload(7, ttype, W, M, K)
    d_x, d_y = ctx.to_device(x), ctx.alloc(n * M * 4)
    ctx.dense_gemm(7, d_x, n, d_y)
    got, want = d_y.download(np.float32, (n, M)), orc.gemv(ttype, W, x, M, K)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isposinf(got), np.isposinf(want))
    assert np.array_equal(np.isneginf(got), np.isneginf(want))
    live = [r for r in range(n) if r != 3 or np.isfinite(want[3]).all()]
    assert syn.rel_err_rows(got[live], want[live]) < 5e-3
    d_x.free(); d_y.free()


@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("mantissa", [1.0, 2 - 2.0**-9])
def test_tensor_core_accumulation(ctx, syn, sign, mantissa):
    """What the tensor cores lose of a small product beside a large one.  The router's candidate bound allows 2^-22 of the sum a
    column; one product of 64 and 255 of every size below it lose 2^-24 a column at most (measured: 2^-25)."""
    M, K, n = 128, 256, 32
    b = np.zeros((M, K // 32, 34), np.uint8)
    b[:, :, 0:2] = np.array([1], np.float16).view(np.uint8)
    b[:, :, 2:] = 1
    b[:, 0, 2] = 64
    x = np.zeros((n, K), np.float64)
    x[:, 0] = 1
    for j in range(2, n):
        x[j, 1:] = sign * mantissa * 2.0**-min(j, 27)   # f16 operands: normal numbers down to 2^-28 of the row's largest
    ctx.dense_upload(8, 8, b.reshape(-1), M, K)
    d_x, d_y = ctx.to_device(x.astype(np.float32)), ctx.alloc(n * M * 4)
    ctx.dense_gemm(8, d_x, n, d_y)
    want = 64 + x[:, 1:].sum(axis=1)
    err = np.abs(d_y.download(np.float32, (n, M)) - want[:, None]).max(axis=1)
    assert (err <= 255 * 2.0**-24 * np.maximum(64, np.abs(want))).all(), err / (255 * 64 * 2.0**-24)
    d_x.free(); d_y.free()


def test_dense_rejects(ctx, pkg, syn):
    W = syn.random_blocks(8, 128, 256, seed=1)
    d = ctx.alloc(1 << 16)
    with pytest.raises(pkg.QkmError):
        ctx.dense_upload(0, 14, W, 128, 256)          # Q6_K: not a GEMM type
    with pytest.raises(pkg.QkmError):
        ctx.dense_upload(0, 8, W, 100, 256)           # M not a multiple of 128
    with pytest.raises(pkg.QkmError):
        ctx.dense_upload(99, 8, W, 128, 256)
    with pytest.raises(pkg.QkmError):
        ctx.dense_gemm(5, d, 1, d)                    # empty slot
    d.free()
