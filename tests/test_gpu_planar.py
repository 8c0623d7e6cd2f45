"""Planar forward kernels at the edges of their ranges: planes around one tile, whole planes and halo tiles in both
directions, partial channel groups, strides, every layout and type, pyramids with and without small levels;
against the float64 oracle (16-bit types: the same-type oracle's tolerance)."""
import pytest
import torch

from conftest import max_err
from oracle import wtconv_torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,C,H,W,L,K,stride,layout,dtype", [
    (2, 3, 1, 1, 1, 3, 1, "nchw", torch.float32), (3, 5, 8, 8, 3, 5, 1, "nchw", torch.float32), (2, 9, 9, 7, 2, 7, 1, "nchw", torch.float32),
    (1, 33, 64, 66, 5, 5, 1, "nchw", torch.bfloat16), (700, 4, 28, 28, 4, 5, 1, "nchw", torch.float32), (2, 6, 31, 130, 2, 3, 3, "nchw", torch.float32),
    (1, 4, 300, 258, 5, 5, 1, "nchw", torch.float32), (1, 2, 140, 500, 1, 7, 2, "nchw", torch.float16), (2, 7, 129, 65, 0, 5, 1, "nchw", torch.float32),
    (2, 24, 57, 64, 5, 7, 1, "cl", torch.float32), (1, 40, 150, 90, 4, 7, 1, "cl", torch.bfloat16), (5, 17, 20, 20, 3, 5, 1, "cl", torch.float32),
    (40, 64, 14, 14, 3, 3, 1, "cl", torch.float16), (3, 72, 56, 57, 4, 3, 1, "cl", torch.float32), (2, 16, 33, 47, 3, 5, 2, "cl", torch.float32),
    (1, 24, 70, 200, 3, 3, 2, "cl", torch.float32), (2, 8, 130, 131, 3, 3, 1, "cl", torch.float32),
])
def test_planar_forward(B, C, H, W, L, K, stride, layout, dtype):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    import wtconv_b200
    params = wtconv_torch.random_params(C, K, L, ndim=2, bias=True, seed=H + W)
    m = wtconv_b200.WTConv2d(C, C, kernel_size=K, stride=stride, bias=True, wt_levels=L)
    sd = m.state_dict()
    m.load_state_dict({**sd, **{k: torch.as_tensor(v).float().reshape(sd[k].shape) for k, v in params.items() if "filter" not in k}})
    m = m.cuda()
    x = torch.randn(B, C, H, W, generator=torch.Generator().manual_seed(H * W)).to(dtype)
    xt = x.cuda()
    if layout == "cl":
        xt = xt.contiguous(memory_format=torch.channels_last)
    with torch.no_grad():
        y = m(xt).double().cpu()
    n = min(B, 3)                       # samples are independent: the first ones and the last against the oracle
    pick = sorted(set(range(n)) | {B - 1})
    pd = {k: p.detach().cpu().double() for k, p in m.named_parameters() if "filter" not in k}
    with torch.no_grad():
        ref = wtconv_torch.wtconv2d_forward(x[pick].double(), pd, stride=stride)
    assert max_err(y[pick].numpy(), ref.numpy()) <= (1e-5 if dtype == torch.float32 else 2e-2)
