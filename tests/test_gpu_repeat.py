"""Many decode calls on the same rows give the same bits.  A ring stage that was filled again while the last reads of it were still under way showed
as one wrong 16-row tile of a hidden row in some ten thousand launches."""
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
