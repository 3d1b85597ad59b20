"""Router of 2..8 rows against float64: one and several 16-row groups, the widest and the narrowest H, one and two column tiles."""

import pytest
import torch

from nexrt_b200.ops.lib import check, load, ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,rows_pad,M", [(128, 16, 2), (1024, 32, 5), (4096, 528, 4), (4096, 528, 8), (3968, 48, 7), (256, 16, 8)])
def test_router_rows(H, rows_pad, M):
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(H + M)
    x = torch.randn(8, H, device=dev, generator=g).to(torch.bfloat16)
    ln = 1 + 0.1 * torch.randn(H, device=dev, generator=g)
    w = (torch.randn(rows_pad, H, device=dev, generator=g) * 0.03).to(torch.bfloat16)
    cols = torch.zeros(16, H, dtype=torch.bfloat16, device=dev)
    partial, planes = torch.zeros(4, M, rows_pad, device=dev), torch.zeros(24, H, dtype=torch.uint8, device=dev)
    check(load().nexrt_moe_router_rows(ptr(x), ptr(ln), ptr(w), ptr(cols), ptr(partial), ptr(planes), rows_pad, H, M, 1e-6, torch.cuda.current_stream().cuda_stream),
          "moe_router_rows")
    torch.cuda.synchronize()
    xd = x[:M].double()
    xn = xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-6) * ln.double()
    # hi + lo leaves 2^-17 of a value; fp32 sums
    bound = 2.0**-15 * (xn.abs() @ w.double().abs().T)
    assert ((partial.double().sum(0) - xn @ w.double().T).abs() <= bound).all()
    t = planes[: 3 * M].view(torch.float8_e4m3fn).double().view(M, 3, H)
    assert ((t[:, 0] + t[:, 1] / 16 + t[:, 2] / 256) / 2 - xn).abs().max() <= 2.0**-11 * xn.abs().max()
    assert not planes[3 * M :].any()
