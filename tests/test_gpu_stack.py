"""Decode stacks whose layers go through each stage of the fused sequence together, against the oracle, layer by layer."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL_F32 = 1e-5   # as the layer-by-layer decode calls: exact integer sums, one f32 rounding per 256 columns


def run_stack(pkg, syn, dims, layers, x, max_tokens=None, y_at=None, runs=None):
    """(y [L][T][n_embd], last layer's selection); y_at: byte offset of the outputs inside the inputs' buffer; runs: how many times layers go
    through the stages together, three or four launches each."""
    L, T = x.shape[:2]
    with pkg.Context(dims, n_layer=L, max_tokens=max_tokens or T, device=0) as ctx:
        for l, layer in enumerate(layers):
            ctx.upload_layer(l, layer)
        if y_at is None:
            d_x, d_y = ctx.to_device(x), ctx.alloc(x.nbytes)
            for _ in range(3):   # counters and tickets are left as they were found
                before = ctx.launch_count()
                ctx.moe_decode_stack(0, L, d_x, T, d_y)
            assert runs is None or 3 * runs <= ctx.launch_count() - before <= 4 * runs
            y = d_y.download(np.float32, x.shape)
        else:
            buf = ctx.to_device(np.concatenate([x.reshape(-1), np.zeros(y_at // 4, np.float32)]))
            ctx.moe_decode_stack(0, L, buf.ptr, T, buf.ptr + y_at)
            y = buf.download(np.float32, x.size + y_at // 4)[y_at // 4:].reshape(x.shape)
        return y, ctx.last_sel(T)


def check(syn, orc, layers, x, y, sel, tol=TOL_F32):
    for l, layer in enumerate(layers):
        ref = orc.moe_layer(layer, x[l], threads=orc.hardware_threads())
        assert syn.rel_err_rows(y[l], ref["y"]) < tol, l
        if l + 1 == len(layers):
            n = layer.dims.n_used
            assert np.array_equal(sel["ids"][:, :n], ref["sel"]["ids"][:, :n])
            np.testing.assert_allclose(sel["w_shared"], ref["sel"]["w_shared"], rtol=1e-6)


# every down kernel (8, other numbers of and more than ten slots; 40 tokens on), router groups of 1, 2, 4 and 8 tokens, odd numbers of tokens, a second
# chunk of six tokens, two to eight column blocks, fewer tiles than teams of warps and many more, shares that begin inside a layer
@pytest.mark.parametrize("n_embd,n_expert,n_used,gt,dt,T,L", [
    (1024, 16, 4, 18, 23, 1, 3), (1024, 16, 4, 18, 23, 2, 3), (1024, 16, 4, 18, 14, 3, 3), (512, 16, 4, 23, 14, 9, 4), (512, 4, 4, 18, 23, 4, 2),
    (2048, 32, 8, 18, 23, 16, 5), (2048, 32, 8, 23, 14, 16, 4), (1024, 512, 10, 23, 23, 5, 2), (512, 32, 15, 18, 14, 3, 2), (512, 20, 1, 18, 23, 33, 3),
    (1024, 8, 8, 18, 14, 64, 2), (512, 24, 6, 23, 23, 70, 3), (512, 8, 2, 18, 23, 1, 30), (512, 16, 8, 18, 14, 2, 9)])
def test_stack_layers_together(pkg, orc, syn, n_embd, n_expert, n_used, gt, dt, T, L):
    dims = syn.Dims(n_embd=n_embd, n_ff=512, n_expert=n_expert, n_used=n_used)
    layers = [syn.make_layer(dims, seed=200, layer=l, router_type=l0, gateup_type=gt, down_type=dt) for l, l0 in enumerate([T & 1] * L)]
    x = np.stack([syn.random_x(T, n_embd, seed=210 + l) for l in range(L)])
    y, sel = run_stack(pkg, syn, dims, layers, x, runs=2 if T > 64 else 1)
    check(syn, orc, layers, x, y, sel)


# router blocks of several pairs of experts: those that keep up to four tokens' x (one, two and four tokens a group) and those that read eight tokens' for
# each pair; the last group and the last block's pairs not full, an odd number of experts, part of the lanes idle (512 columns) and none (2048)
@pytest.mark.parametrize("n_embd,n_expert,T,L", [
    (512, 511, 1, 5), (512, 512, 2, 5), (512, 511, 4, 6), (512, 510, 3, 6), (512, 511, 13, 5), (2048, 64, 64, 10), (512, 511, 6, 6), (512, 256, 8, 10), (512, 255, 21, 5)])
def test_stack_router_blocks_of_several_pairs(pkg, orc, syn, n_embd, n_expert, T, L):
    dims = syn.Dims(n_embd=n_embd, n_ff=512, n_expert=n_expert, n_used=8)
    layers = [syn.make_layer(dims, seed=240, router_type=T & 1)] * L
    x = np.stack([syn.random_x(T, n_embd, seed=250 + l) for l in range(L)])
    y, sel = run_stack(pkg, syn, dims, layers, x, runs=1)
    check(syn, orc, layers, x, y, sel)


def test_stack_of_several_types(pkg, orc, syn):
    """Runs of layers of the same types; a run of one layer."""
    dims = syn.Dims(n_embd=1024, n_ff=512, n_expert=16, n_used=4)
    mixes = [(0, 18, 23), (0, 18, 23), (1, 18, 23), (1, 23, 14), (1, 23, 14), (1, 23, 14), (0, 18, 14)]
    layers = [syn.make_layer(dims, seed=220, layer=l, router_type=r, gateup_type=g, down_type=d) for l, (r, g, d) in enumerate(mixes)]
    x = np.stack([syn.random_x(7, 1024, seed=230 + l) for l in range(len(mixes))])
    y, sel = run_stack(pkg, syn, dims, layers, x, runs=4)
    check(syn, orc, layers, x, y, sel)


def test_stack_more_layers_than_scratch(pkg, orc, syn):
    """64 tokens, 14 layers: more rows than go through together."""
    dims = syn.Dims(n_embd=512, n_ff=512, n_expert=8, n_used=2)
    layers = [syn.make_layer(dims, seed=240, layer=l) for l in range(14)]
    x = np.stack([syn.random_x(64, 512, seed=250 + l) for l in range(14)])
    y, sel = run_stack(pkg, syn, dims, layers, x, runs=2)
    check(syn, orc, layers, x, y, sel)


def test_stack_outputs_that_feed_the_next_layer(pkg, orc, syn):
    """y one layer behind x in the same buffer: layer l + 1 reads what layer l wrote.  And in place: every layer reads its own row first."""
    dims = syn.Dims(n_embd=512, n_ff=512, n_expert=16, n_used=4)
    T, L = 5, 3
    layers = [syn.make_layer(dims, seed=260, layer=l) for l in range(L)]
    x = np.stack([syn.random_x(T, 512, seed=270 + l) for l in range(L)])
    y, _ = run_stack(pkg, syn, dims, layers, x, y_at=T * 512 * 4)
    row = x[0]
    for l in range(L):
        row = orc.moe_layer(layers[l], row, threads=orc.hardware_threads())["y"]
        assert syn.rel_err_rows(y[l], row) < 1e-4   # errors of the layers before go through
        row = y[l]
    y, sel = run_stack(pkg, syn, dims, layers, x, y_at=0)
    check(syn, orc, layers, x, y, sel)


@pytest.mark.parametrize("gt,dt", [(18, 23), (23, 14)])
def test_stack_nonfinite_and_large_rows(pkg, orc, syn, gt, dt):
    """A NaN or an infinity stays in its token; an element of 1e8 where the weights are zero costs the others of its row nothing."""
    dims = syn.Dims(n_embd=1024, n_ff=512, n_expert=16, n_used=4)
    layers = [syn.make_layer(dims, seed=280, layer=l, gateup_type=gt, down_type=dt) for l in range(2)]
    for layer in layers:
        for t, elems, size_b in ((layer.gate_exps, 256, syn.BLOCK[gt][1]), (layer.up_exps, 256, syn.BLOCK[gt][1]), (layer.gate_shexp, 32, 34), (layer.up_shexp, 32, 34)):
            t.reshape(-1, dims.n_embd // elems, size_b)[:, 256 // elems:512 // elems, 0:2] = 0   # d of columns 256 .. 511
    x = np.stack([syn.random_x(9, 1024, seed=290 + l) for l in range(2)])
    x[:, 2, 300] = 1e8
    x[:, 4, 7] = np.nan
    x[:, 5, 900] = np.inf
    y, _ = run_stack(pkg, syn, dims, layers, x)
    ok = np.isfinite(x).all(axis=2)
    for l in range(2):
        ref = orc.moe_layer(layers[l], x[l][ok[l]], threads=orc.hardware_threads())
        assert syn.rel_err_rows(y[l][ok[l]], ref["y"]) < TOL_F32
        assert np.isnan(y[l][~ok[l]]).all()


# 64 tokens and fewer, both down kernels that go by expert and one that does not
@pytest.mark.parametrize("gt,dt,T,L", [(18, 23, 64, 14), (23, 14, 64, 13), (18, 14, 24, 40)])
def test_host_buffers_in_chunks(pkg, orc, syn, gt, dt, T, L):
    """From 1.5 MB of rows on the host-buffer form runs in three chunks of layers that go together, the copies on streams of their own: the bits of the
    layer-by-layer calls, on repeated calls too (scratch and tickets are the chunks' in turn), and fewer layers than chunks need in one."""
    import torch
    dims = syn.Dims(n_embd=512, n_ff=512, n_expert=16, n_used=4)
    x = np.stack([syn.random_x(T, dims.n_embd, seed=300 + l) for l in range(L)])
    assert x.nbytes >= 3 << 19
    layer = syn.make_layer(dims, seed=301, gateup_type=gt, down_type=dt)
    with pkg.Context(dims, n_layer=L, max_tokens=T, device=0) as ctx:
        for l in range(L):
            ctx.upload_layer(l, layer)
        want = np.stack([ctx.moe_forward_host(l, x[l], mode=0) for l in range(L)])
        stream = torch.cuda.Stream(torch.device("cuda", 0))
        ctx.set_stream(stream.cuda_stream)
        for n, chunks in ((L, 3), (L, 3), (5, 1), (L, 3)):
            y = np.zeros_like(x[:n])
            before = ctx.launch_count()
            ctx.moe_decode_stack_host(0, n, x.ctypes.data, T, y.ctypes.data)
            assert 3 * chunks <= ctx.launch_count() - before <= 4 * chunks
            assert np.array_equal(y, want[:n])
        ctx.set_stream(0)
    for l in (0, L // 2, L - 1):
        assert syn.rel_err_rows(want[l], orc.moe_layer(layer, x[l], threads=orc.hardware_threads())["y"]) < TOL_F32


# one token and one pair, an odd and a full batch, every expert chosen by all or by few, the most groups that a layer can have (512 experts, 15 of them
# used), the down kernel that goes by expert (40 tokens on) and those that do not
@pytest.mark.parametrize("n_embd,n_expert,n_used,gt,dt,T", [
    (512, 1, 1, 18, 23, 1), (512, 512, 15, 18, 23, 64), (1024, 512, 10, 23, 14, 63), (2048, 20, 8, 18, 23, 40), (512, 15, 15, 23, 23, 2), (512, 16, 4, 18, 14, 39)])
def test_layer_on_its_own_and_in_a_stack(pkg, orc, syn, n_embd, n_expert, n_used, gt, dt, T):
    """A layer's blocks group its pairs themselves, a stack's router groups them: the same bits, and the oracle's values."""
    dims = syn.Dims(n_embd=n_embd, n_ff=512, n_expert=n_expert, n_used=n_used)
    layers = [syn.make_layer(dims, seed=320, layer=l, gateup_type=gt, down_type=dt) for l in range(2)]
    x = np.stack([syn.random_x(T, n_embd, seed=330 + l) for l in range(2)])
    with pkg.Context(dims, n_layer=2, max_tokens=T, device=0) as ctx:
        for l, layer in enumerate(layers):
            ctx.upload_layer(l, layer)
        d_x, d_y = ctx.to_device(x), ctx.alloc(x.nbytes)
        ctx.moe_decode_stack(0, 2, d_x, T, d_y)
        together = d_y.download(np.float32, x.shape)
        for l in range(2):
            ctx.moe_decode(l, d_x.ptr + l * x[0].nbytes, T, d_y.ptr + l * x[0].nbytes)
        y, sel = d_y.download(np.float32, x.shape), ctx.last_sel(T)
    assert np.array_equal(y, together)
    check(syn, orc, layers, x, y, sel)


def test_stack_scratch_comes_with_the_first_stack(pkg, syn):
    """A context for many layers and slots holds no more at its opening than one for a single layer, but for a few MB; a stack's first call takes the
    rest once, and only once."""
    import torch
    dims = syn.Dims()
    free = lambda: (torch.cuda.synchronize(), torch.cuda.mem_get_info(0)[0])[1]

    def opened(n_layer):
        before = free()
        ctx = pkg.Context(dims, n_layer=n_layer, max_tokens=64, device=0)
        return ctx, before - free()

    torch.zeros(1, device="cuda")
    opened(1)[0].close()   # (what a first context sets up for the process)
    one, few = opened(1)
    one.close()
    ctx, many = opened(40)
    with ctx:
        assert many - few <= 12 << 20, (few, many)
        small = syn.make_layer(dims, seed=340)
        for l in range(2):
            ctx.upload_layer(l, small)
        d = ctx.alloc(2 * 2 * 3 * dims.n_embd * 4)
        at = []
        for _ in range(3):
            ctx.moe_decode_stack(0, 2, d, 3, d.ptr + 2 * 3 * dims.n_embd * 4)
            at.append(free())
        assert at[0] == at[1] == at[2]


@pytest.mark.parametrize("T", [5, 64])
def test_stack_first_called_under_capture(pkg, syn, T):
    """No scratch for several layers yet and none can be had: the layers go one by one, and a replay gives the bits of the call outside."""
    import torch
    dims, L = syn.Dims(n_embd=1024, n_ff=512, n_expert=16, n_used=8), 14
    layer = syn.make_layer(dims, seed=350)
    x = torch.from_numpy(np.stack([syn.random_x(T, dims.n_embd, seed=351 + l) for l in range(L)])).cuda()
    y, z = torch.zeros_like(x), torch.zeros_like(x)
    stream = torch.cuda.Stream()
    with pkg.Context(dims, n_layer=L, max_tokens=64, device=0) as ctx:
        for l in range(L):
            ctx.upload_layer(l, layer)
        torch.cuda.synchronize()
        ctx.set_stream(stream.cuda_stream)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            before = ctx.launch_count()
            ctx.moe_decode_stack(0, L, x.data_ptr(), T, y.data_ptr())
            assert ctx.launch_count() - before >= 3 * L
        for _ in range(2):
            graph.replay()
        torch.cuda.synchronize()
        before = ctx.launch_count()
        ctx.moe_decode_stack(0, L, x.data_ptr(), T, z.data_ptr())
        stream.synchronize()
        assert ctx.launch_count() - before <= 8
        assert torch.isfinite(z).all() and torch.equal(y, z)
        together = torch.cuda.CUDAGraph()
        with torch.cuda.graph(together, stream=stream):   # with the scratch there: the layers together
            before = ctx.launch_count()
            ctx.moe_decode_stack(0, L, x.data_ptr(), T, y.data_ptr())
            assert ctx.launch_count() - before <= 8
        for g in (graph, together, graph, together):
            y.zero_()
            torch.cuda.synchronize()
            g.replay()
            torch.cuda.synchronize()
            assert torch.equal(y, z)
        ctx.set_stream(0)
        del graph, together, g


def test_stack_stage_times(pkg, syn):
    """While stages are timed a stack takes the launches it takes otherwise, and a stage's time is all its runs' together."""
    dims, T, L = syn.Dims(n_embd=512, n_ff=512, n_expert=16, n_used=4), 6, 4
    layers = [syn.make_layer(dims, seed=360, layer=l, down_type=23 if l < 2 else 14) for l in range(L)]   # two runs
    x = np.stack([syn.random_x(T, dims.n_embd, seed=361 + l) for l in range(L)])
    with pkg.Context(dims, n_layer=L, max_tokens=T, device=0) as ctx:
        for l, layer in enumerate(layers):
            ctx.upload_layer(l, layer)
        d_x, d_y = ctx.to_device(x), ctx.alloc(x.nbytes)
        ctx.moe_decode_stack(0, L, d_x, T, d_y)
        want = d_y.download(np.float32, x.shape)
        ctx.profile_enable(True)
        before = ctx.launch_count()
        ctx.moe_decode_stack(0, L, d_x, T, d_y)
        assert ctx.launch_count() - before == 6
        ms = ctx.profile_read()
        assert set(ms) == {"moe.route", "moe.gu", "moe.dn"} and all(0 < v < 100 for v in ms.values())
        ctx.profile_enable(False)
        assert np.array_equal(d_y.download(np.float32, x.shape), want)
