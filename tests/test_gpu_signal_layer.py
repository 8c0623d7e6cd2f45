"""Register-resident 1-D kernels at the edges of their ranges: five levels, pooled outputs, lengths around
a warp's segment and below one, unaligned rows; forward, input gradient and parameter gradients against
autograd through the oracle in fp64."""
import pytest
import torch

from conftest import max_err
from oracle import wtconv_torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,C,N,L,K,stride,dtype", [
    (2, 3, 897, 5, 5, 1, torch.float32), (1, 2, 31, 5, 7, 1, torch.float32), (3, 5, 4097, 5, 3, 2, torch.float32),
    (2, 3, 448, 4, 5, 2, torch.float32), (2, 3, 449, 4, 7, 4, torch.float32), (1, 1, 17, 2, 5, 8, torch.float32),
    (3, 2, 1000, 3, 7, 3, torch.float32), (40, 9, 130, 0, 5, 1, torch.float32), (2, 4, 2048, 5, 5, 2, torch.bfloat16),
    (5, 700, 64, 1, 1, 1, torch.float16), (3, 3, 961, 4, 5, 1, torch.bfloat16), (4, 3, 3333, 5, 7, 1, torch.float16),
    (2, 5, 1922, 3, 5, 1, torch.bfloat16), (3, 3, 449, 1, 7, 1, torch.bfloat16),
])
def test_forward_and_gradients(B, C, N, L, K, stride, dtype):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    import wtconv_b200
    g = torch.Generator().manual_seed(N + L)
    params = wtconv_torch.random_params(C, K, L, ndim=1, bias=True, seed=N)
    m = wtconv_b200.WTConv1d(C, C, kernel_size=K, stride=stride, bias=True, wt_levels=L)
    m.load_state_dict({**m.state_dict(), **{k: torch.as_tensor(v).float().reshape(m.state_dict()[k].shape) for k, v in params.items() if "filter" not in k}})
    m = m.cuda()
    x = torch.randn(B, C, N, generator=g).to(dtype)
    gy = torch.randn(B, C, N // stride, generator=g).to(dtype)
    xt = x.cuda().requires_grad_(True)
    y = m(xt)
    y.backward(gy.cuda())
    names = [n for n, _ in m.named_parameters() if "filter" not in n]
    pd = {n: p.detach().cpu().double().requires_grad_(True) for n, p in m.named_parameters() if "filter" not in n}
    xr = x.double().requires_grad_(True)
    yr = wtconv_torch.wtconv1d_forward(xr, pd, stride=stride)
    refs = torch.autograd.grad(yr, [xr] + [pd[n] for n in names], gy.double())
    tol = 1e-5 if dtype == torch.float32 else 2e-2
    assert max_err(y.detach().double().cpu().numpy(), yr.detach().numpy()) <= tol
    assert max_err(xt.grad.double().cpu().numpy(), refs[0].numpy()) <= tol
    got = dict(m.named_parameters())
    for n, r in zip(names, refs[1:]):
        err = max_err(got[n].grad.double().cpu().numpy(), r.numpy())
        assert err <= (1e-4 if dtype == torch.float32 else 2e-2), f"{n}: {err:.3e}"
