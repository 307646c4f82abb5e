"""Batched prefill through the tensor-core path (f16 operands, f32 accumulation) against the
f64-accumulating oracle.  Tolerance: 1e-2 on the row-scaled relative error of the worst element (measured: about 4e-3; x, weights
and hidden rows rounded to 2^-11 each, two GEMMs: 0.6e-3 as a norm), expert ids exact,
argmax of every output row unchanged (where the reference itself is not a near-tie)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-2


def run_prefill(pkg, orc, syn, dims, layer, x, tol=TOL):
    T = x.shape[0]
    ref = orc.moe_layer(layer, x, threads=orc.hardware_threads(), want_h=True)
    with pkg.Context(dims, n_layer=1, max_tokens=max(T, 1), device=0) as ctx:
        ctx.upload_layer(0, layer)
        y = ctx.moe_forward_host(0, x, mode=1)
        sel = ctx.last_sel(T)
        y_again = ctx.moe_forward_host(0, x, mode=1)
    assert np.array_equal(sel["ids"][:, :dims.n_used], ref["sel"]["ids"][:, :dims.n_used])
    err = syn.rel_err_rows(y, ref["y"])
    assert err < tol, err
    # argmax of every output row is unchanged wherever the reference's lead over the
    # runner-up is larger than twice the tolerated error (a closer call is a tie at this precision)
    r = ref["y"].astype(np.float64)
    top2 = np.sort(r, axis=1)[:, -2:]
    rms = np.sqrt(np.mean(r * r, axis=1))
    clear = (top2[:, 1] - top2[:, 0]) > 2 * tol * np.maximum(rms, np.abs(top2[:, 1]))
    assert np.array_equal(np.argmax(y, axis=1)[clear], np.argmax(r, axis=1)[clear])
    assert np.array_equal(y, y_again)   # deterministic
    return err


@pytest.mark.parametrize("T", [1, 17, 65, 130, 300])
def test_prefill_full_size(pkg, orc, syn, T):
    """Bench configuration 3 shapes (2048 / 512 / 256 experts / top-8) at small chunk sizes."""
    dims = syn.Dims()
    layer = syn.make_layer(dims, seed=42)
    x = syn.random_x(T, dims.n_embd, seed=77)
    run_prefill(pkg, orc, syn, dims, layer, x)


def test_prefill_operand_precision(pkg, orc, syn):
    """Both expert GEMMs run on f16 operands (x and the hidden rows scaled per row by a power of two,
    the dequantised weights rounded once or twice to f16), so the outputs sit well inside the 1e-2
    budget on the full-size layer."""
    dims = syn.Dims()
    layer = syn.make_layer(dims, seed=42)
    x = syn.random_x(130, dims.n_embd, seed=78)
    x[3] *= 300.0      # rows of very different magnitude: the per-row scales keep their precision
    x[4] *= 1e-4
    err = run_prefill(pkg, orc, syn, dims, layer, x)
    assert err < 7e-3, err


@pytest.mark.parametrize("T", [512, 2048, 4096])
def test_prefill_bench_chunk_sizes(pkg, orc, syn, T):
    """The chunk sizes the prefill figures are quoted on.  Expert ids (tensor-core logits, boundary
    re-evaluated in f64) must equal the f64 router's for EVERY token - the oracle's router alone
    is cheap - including tie / NaN / all-zero rows placed beyond row 1024 where the chunk has
    them.  Outputs: the oracle's full layer on >= 64 sampled rows (selection given) that include
    the first and the last row, rows from every 128-pair N-tile of the busiest expert, and the
    special rows; 1e-2 row-scaled relative."""
    dims = syn.Dims()
    layer = syn.make_layer(dims, seed=42, router_type=syn.F32)
    r = layer.router.view(np.float32).reshape(256, 2048).copy()
    r[200] = r[17]; r[90] = r[17]; r[3] = 0.0; r[4] = 0.0
    r[40] *= 3.0                                    # a busy expert: several N-tiles at the larger chunks
    layer.router = r.reshape(-1).view(np.uint8)
    x = syn.random_x(T, dims.n_embd, seed=79)
    special = []
    if T > 1100:
        x[1030] = r[17] * 50.0; x[1031] = 0.0
        special = [1030, 1031]
    x[T - 1] = r[17] * 50.0
    nthr = orc.hardware_threads()
    want, w64 = orc.route(layer, x, threads=nthr)
    x_nan = None
    if T > 1100:                                    # a NaN row: ids must be 0..7; its output is not compared
        x_nan = 1040
        x[x_nan, 100] = np.nan
        want, w64 = orc.route(layer, x, threads=nthr)
    with pkg.Context(dims, n_layer=1, max_tokens=T, device=0) as ctx:
        ctx.upload_layer(0, layer)
        y = ctx.moe_forward_host(0, x, mode=1)
        sel = ctx.last_sel(T)
    assert np.array_equal(sel["ids"][:, :8], want["ids"][:, :8])
    assert list(sel["ids"][T - 1, :3]) == [17, 90, 200]
    if x_nan is not None:
        assert list(sel["ids"][x_nan, :8]) == list(range(8)) and list(sel["ids"][1031, :8]) == list(range(8))
    ok = np.isfinite(w64[:, :8]).all(axis=1)
    np.testing.assert_allclose(sel["w"][ok, :8], w64[ok, :8], rtol=1e-5, atol=1e-7)
    # rows to check through the whole layer
    ids = want["ids"][:, :8]
    counts = np.bincount(ids.reshape(-1), minlength=256)
    busiest = int(np.argmax(counts))
    toks_busy = np.nonzero((ids == busiest).any(axis=1))[0]      # ascending = pair order inside the expert
    rows = {0, T - 1, *special}
    for tile in range((len(toks_busy) + 127) // 128):            # first and last pair of every N-tile
        seg = toks_busy[tile * 128:(tile + 1) * 128]
        rows.update((int(seg[0]), int(seg[-1])))
    rng = np.random.default_rng(5)
    while len(rows) < 64:
        rows.add(int(rng.integers(0, T)))
    if x_nan is not None:
        rows.discard(x_nan)
    rows = np.array(sorted(rows))
    if T > 1100:
        assert counts[busiest] > 128, "the busy expert should span more than one N-tile"
    ref = orc.moe_layer(layer, x[rows], threads=nthr, sel_in=want[rows])
    err = syn.rel_err_rows(y[rows], ref["y"])
    assert err < TOL, err
    assert np.isfinite(y[np.setdiff1d(np.arange(T), [x_nan] if x_nan is not None else [])]).all()


def test_prefill_hot_expert(pkg, orc, syn):
    """Every token routed to the same experts: more pairs than one block holds (N tiles > 1)."""
    dims = syn.Dims(n_embd=1024, n_ff=512, n_expert=16, n_used=4)
    layer = syn.make_layer(dims, seed=5, router_type=syn.F32)
    r = layer.router.view(np.float32).reshape(16, 1024).copy()
    r[3] *= 40.0; r[7] *= 30.0                      # experts 3 and 7 dominate for most tokens
    layer.router = r.reshape(-1).view(np.uint8)
    x = syn.random_x(150, dims.n_embd, seed=6)
    x[:, :] = np.abs(x) * np.sign(r[3])[None, :] * 0.5 + x * 0.5   # push tokens towards expert 3
    run_prefill(pkg, orc, syn, dims, layer, x)


@pytest.mark.parametrize("gt,dt,n_embd,n_expert,n_used,T", [(18, 23, 512, 4, 1, 520), (23, 14, 1024, 4, 2, 233), (18, 23, 2048, 8, 4, 329), (23, 23, 512, 6, 2, 480), (18, 14, 512, 2, 1, 301)])
def test_prefill_wide_tiles(pkg, orc, syn, gt, dt, n_embd, n_expert, n_used, T):
    """Tiles of 160 pairs (116 to 165 an expert on average): full ones, remainders below and above 64, k-steps that do not divide by three."""
    dims = syn.Dims(n_embd=n_embd, n_ff=512, n_expert=n_expert, n_used=n_used)
    layer = syn.make_layer(dims, seed=7, gateup_type=gt, down_type=dt)
    x = syn.random_x(T, dims.n_embd, seed=8)
    run_prefill(pkg, orc, syn, dims, layer, x)


def _token_errors(y, ref):
    r = ref["y"].astype(np.float64)
    return np.linalg.norm(y - r, axis=1) / np.linalg.norm(r, axis=1)


@pytest.mark.parametrize("gt,dt", [(18, 23), (23, 14)])
@pytest.mark.parametrize("size", [1e4, 1e6])
def test_prefill_large_element_without_weights(pkg, orc, syn, gt, dt, size):
    """x with one large element in 256 columns whose weights are all zero: the products are ordinary and far below what the row
    norms allow, and the hidden rows keep their precision (0.6e-3 to 0.9e-3 for ordinary x; f16 operands)."""
    dims = syn.Dims(n_embd=512, n_ff=512, n_expert=8, n_used=2)
    layer = syn.make_layer(dims, seed=51, gateup_type=gt, down_type=dt)
    for t, elems, size_b in ((layer.gate_exps, 256, syn.BLOCK[gt][1]), (layer.up_exps, 256, syn.BLOCK[gt][1]), (layer.gate_shexp, 32, 34), (layer.up_shexp, 32, 34)):
        t.reshape(-1, dims.n_embd // elems, size_b)[:, :256 // elems, 0:2] = 0   # d of the first 256 columns
    x = syn.random_x(140, dims.n_embd, seed=52)
    x[::3, 5] = size
    ref = orc.moe_layer(layer, x, threads=orc.hardware_threads())
    with pkg.Context(dims, n_layer=1, max_tokens=len(x), device=0) as ctx:
        ctx.upload_layer(0, layer)
        err = _token_errors(ctx.moe_forward_host(0, x, mode=1), ref)
    assert err.max() < 1.5e-3, err


def test_prefill_saturated_gates(pkg, orc, syn):
    """Every gate of every expert between -20 and -45, the shared one too: the hidden values are 1e-8 and less of what the row norms allow.  The
    gates' error (f16 operands, 2^-11 each, 512 products of one sign) enters the exponential: 45 * 2 * 2^-11 at the very most."""
    dims = syn.Dims(n_embd=512, n_ff=512, n_expert=8, n_used=2)
    layer = syn.make_layer(dims, seed=53, gateup_type=23, down_type=23)
    b = layer.gate_exps.reshape(-1, 136)
    b[:, 0:2] = np.array([5.5e-3], np.float16).view(np.uint8)
    b[:, 8:] = 0        # codebook value -127 throughout
    b[:, 2:8] = 0xFF    # sub-block scales 31
    s = layer.gate_shexp.reshape(-1, 34)
    s[:, 2:] = 0x81     # -127
    s[:, 0:2] = np.array([0.17], np.float16).view(np.uint8)
    x = np.abs(syn.random_x(96, dims.n_embd, seed=54)) * np.float32(3e-3)
    ref = orc.moe_layer(layer, x, threads=orc.hardware_threads(), want_h=True)
    assert 0 < np.abs(ref["h"]).max() < 1e-6
    with pkg.Context(dims, n_layer=1, max_tokens=len(x), device=0) as ctx:
        ctx.upload_layer(0, layer)
        err = _token_errors(ctx.moe_forward_host(0, x, mode=1), ref)
    assert err.max() < 45 * 2 * 2.0**-11, err


def test_prefill_norms_beyond_f32(pkg, orc, syn):
    """x of 3e18: its squared norm, and so the bound on the hidden values, passes f32; the hidden values do not."""
    dims = syn.Dims(n_embd=512, n_ff=512, n_expert=8, n_used=2)
    layer = syn.make_layer(dims, seed=55, gateup_type=23, down_type=23)
    for t, size_b in ((layer.gate_exps, 136), (layer.up_exps, 136), (layer.gate_shexp, 34), (layer.up_shexp, 34)):
        v = t.reshape(-1, size_b)
        v[:, 0:2] = (v[:, 0:2].copy().view(np.float16) * np.float16(2.0**-10)).view(np.uint8)
    x = syn.random_x(80, dims.n_embd, seed=56)
    x[10:20] *= np.float32(3e18)
    ref = orc.moe_layer(layer, x, threads=orc.hardware_threads())
    assert np.isfinite(ref["y"]).all()
    with pkg.Context(dims, n_layer=1, max_tokens=len(x), device=0) as ctx:
        ctx.upload_layer(0, layer)
        y = ctx.moe_forward_host(0, x, mode=1)
        live = np.arange(len(x)) if np.isfinite(ref["sel"]["w"]).all() else None
        err = _token_errors(y, ref)
    assert live is not None and err.max() < 2.5e-3, err


@pytest.mark.parametrize("gt,dt", [(18, 23), (23, 14)])
def test_prefill_large_weight_rows(pkg, orc, syn, gt, dt):
    """One gate row and another up row of every expert a thousand times larger than the rest."""
    dims = syn.Dims(n_embd=512, n_ff=512, n_expert=8, n_used=2)
    layer = syn.make_layer(dims, seed=57, gateup_type=gt, down_type=dt)
    for t, r, mats, size_b in ((layer.gate_exps, 3, 8, syn.BLOCK[gt][1]), (layer.up_exps, 7, 8, syn.BLOCK[gt][1]), (layer.gate_shexp, 3, 1, 34), (layer.up_shexp, 7, 1, 34)):
        v = t.reshape(mats, dims.n_ff, -1, size_b)
        v[:, r, :, 0:2] = (v[:, r, :, 0:2].copy().view(np.float16) * np.float16(1000)).view(np.uint8)
    x = syn.random_x(140, dims.n_embd, seed=58)
    ref = orc.moe_layer(layer, x, threads=orc.hardware_threads())
    with pkg.Context(dims, n_layer=1, max_tokens=len(x), device=0) as ctx:
        ctx.upload_layer(0, layer)
        y = ctx.moe_forward_host(0, x, mode=1)
    err = np.linalg.norm(y - ref["y"].astype(np.float64)) / np.linalg.norm(ref["y"].astype(np.float64))
    assert err < 1.5e-3, err


def test_prefill_matches_decode_path(pkg, syn):
    """The two fused paths agree to f16 accuracy on the same inputs."""
    dims = syn.Dims()
    layer = syn.make_layer(dims, seed=8)
    x = syn.random_x(24, dims.n_embd, seed=9)
    with pkg.Context(dims, n_layer=1, max_tokens=24, device=0) as ctx:
        ctx.upload_layer(0, layer)
        yd = ctx.moe_forward_host(0, x, mode=0)
        yp = ctx.moe_forward_host(0, x, mode=1)
    assert syn.rel_err_rows(yp, yd) < TOL


@pytest.mark.parametrize("gt,dt", [(18, 14), (23, 23), (23, 14)])
@pytest.mark.parametrize("T", [70, 200])
def test_prefill_other_type_mixes(pkg, orc, syn, T, gt, dt):
    """Q6_K (14) down tensors and IQ4_XS (23) gate/up tensors: both expert GEMMs on the tensor cores
    (Q6_K / IQ4_XS tiles expanded to f16 in tensor memory)."""
    dims = syn.Dims()
    layer = syn.make_layer(dims, seed=46, router_type=syn.F32, gateup_type=gt, down_type=dt)
    x = syn.random_x(T, dims.n_embd, seed=78)
    run_prefill(pkg, orc, syn, dims, layer, x)
