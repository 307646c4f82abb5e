"""Many calls on the same rows give the same bits: the kernels that stream weights through rings of bulk copies.  A ring stage that was filled again
while the last reads of it were still under way showed as one wrong 16-row tile of a hidden row in some ten thousand launches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gt,dt,T", [(18, 23, 64), (18, 14, 64), (23, 14, 16), (18, 23, 39)])
def test_decode_stack_same_bits_every_time(pkg, syn, gt, dt, T):
    import torch
    dims = syn.Dims(n_embd=2048, n_ff=512, n_expert=96, n_used=8)
    L = 10
    made = [syn.make_layer(dims, seed=300, layer=l, gateup_type=gt, down_type=dt) for l in range(2)]
    x = torch.from_numpy(np.stack([syn.random_x(T, dims.n_embd, seed=310 + l) for l in range(L)])).cuda()
    y = torch.empty_like(x)
    stream = torch.cuda.Stream()
    with pkg.Context(dims, n_layer=L, max_tokens=T, device=0) as ctx:
        for l in range(L):
            ctx.upload_layer(l, made[l % 2])
        torch.cuda.synchronize()
        ctx.set_stream(stream.cuda_stream)
        ctx.moe_decode_stack(0, L, x.data_ptr(), T, y.data_ptr())
        stream.synchronize()
        first = y.clone()
        assert torch.isfinite(first).all()
        torch.cuda.synchronize()
        for i in range(400):
            ctx.moe_decode_stack(0, L, x.data_ptr(), T, y.data_ptr())
            stream.synchronize()
            assert torch.equal(y, first), f"call {i}: {int((y != first).sum())} values differ"
        ctx.set_stream(0)


# a block-wide ring whose stages come back by mbarrier (Q6_K, IQ4_XS), rings that are filled again behind a barrier (Q8_0, IQ3_XXS); many tiles a block
@pytest.mark.parametrize("ttype,M,K", [(8, 60016, 2048), (14, 60016, 2048), (23, 60016, 2048), (23, 30000, 4096), (18, 60016, 2048)])
def test_large_gemv_same_bits_every_time(pkg, orc, syn, ttype, M, K):
    import torch
    w, x = syn.random_blocks(ttype, M, K, seed=320 + ttype), syn.random_x(1, K, seed=321)
    y = torch.empty(M, device="cuda")
    with pkg.Context(syn.Dims(), n_layer=1, max_tokens=1, device=0) as ctx:
        d_w, d_x = ctx.to_device(w), ctx.to_device(x)
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        ctx.set_stream(stream.cuda_stream)
        ctx.gemv(ttype, d_w, d_x, y.data_ptr(), M, K, 1)
        stream.synchronize()
        first = y.clone()
        assert syn.rel_err_rows(first.cpu().numpy()[None, :4096], orc.gemv(ttype, w[:4096 * syn.row_bytes(ttype, K)], x, 4096, K)) < 1e-5
        torch.cuda.synchronize()
        for i in range(400):
            ctx.gemv(ttype, d_w, d_x, y.data_ptr(), M, K, 1)
            stream.synchronize()
            assert torch.equal(y, first), f"call {i}: {int((y != first).sum())} values differ"
        ctx.set_stream(0)
