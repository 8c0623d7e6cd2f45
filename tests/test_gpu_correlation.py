"""Planar parameter-gradient kernels at the edges of their ranges: planes around a tile, halo tiles in both
directions, partial channel groups, every layout and type, deep and shallow pyramids, no level at all;
against autograd through the oracle in fp64."""
import pytest
import torch

from conftest import max_err
from oracle import wtconv_torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,C,H,W,L,K,layout,dtype", [
    (3, 5, 2, 3, 1, 5, "nchw", torch.float32), (2, 12, 8, 8, 3, 3, "nchw", torch.float32), (2, 9, 33, 31, 4, 7, "nchw", torch.float32),
    (1, 3, 150, 142, 5, 5, "nchw", torch.float32), (1, 8, 90, 131, 3, 3, "cl", torch.float32), (5, 24, 56, 56, 5, 5, "cl", torch.bfloat16),
    (2, 19, 29, 30, 2, 7, "cl", torch.float16), (9, 40, 7, 7, 2, 5, "cl", torch.bfloat16), (2, 4, 16, 20, 0, 3, "nchw", torch.float32),
    (2, 7, 64, 64, 1, 5, "nchw", torch.bfloat16), (20, 3, 17, 40, 3, 5, "strided", torch.float32),
])
def test_parameter_gradients(B, C, H, W, L, K, layout, dtype):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    import wtconv_b200
    g = torch.Generator().manual_seed(H * 100 + W + L)
    params = wtconv_torch.random_params(C, K, L, ndim=2, bias=True, seed=H + W)
    m = wtconv_b200.WTConv2d(C, C, kernel_size=K, bias=True, wt_levels=L)
    sd = m.state_dict()
    m.load_state_dict({**sd, **{k: torch.as_tensor(v).float().reshape(sd[k].shape) for k, v in params.items() if "filter" not in k}})
    m = m.cuda()
    x = torch.randn(B, C, H, W, generator=g).to(dtype)
    gy = torch.randn(B, C, H, W, generator=g).to(dtype)

    def place(t):
        t = t.cuda()
        if layout == "cl":
            return t.contiguous(memory_format=torch.channels_last)
        if layout == "strided":
            big = torch.zeros(B, C, H + 3, W + 1, device="cuda", dtype=dtype)
            big[:, :, 2:H + 2, 1:] = t
            return big[:, :, 2:H + 2, 1:]
        return t

    m(place(x)).backward(place(gy))
    names = [n for n, _ in m.named_parameters() if "filter" not in n]
    pd = {n: p.detach().cpu().double().requires_grad_(True) for n, p in m.named_parameters() if "filter" not in n}
    yr = wtconv_torch.wtconv2d_forward(x.double(), pd)
    refs = torch.autograd.grad(yr, [pd[n] for n in names], gy.double())
    got = dict(m.named_parameters())
    for n, r in zip(names, refs):
        err = max_err(got[n].grad.double().cpu().numpy(), r.numpy())
        assert err <= 1e-5, f"{n}: {err:.3e}"     # the sums are fp32 whatever the activations' type
