"""Out-projection of 1..8 rows: the form that makes the input's terms in every CTA and the one with a staging kernel in front,
against float64.  K from one 128-wide block to the widest that fits with eight rows; output groups from fewer than one per
warp set to several per CTA."""

import pytest
import torch

from nexrt_b200.ops.lib import check, load, ptr
from nexrt_b200.parallel.channel import LLChannel
from nexrt_b200.quant import dequantize_blockwise, quantize_blockwise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1, 4])
@pytest.mark.parametrize("K,M,H", [(128, 1, 144), (128, 8, 16), (384, 3, 1024), (1024, 1, 4096), (1024, 2, 4096), (1024, 8, 4096), (1152, 5, 272),
                                   (2048, 6, 4096), (4096, 1, 4096), (4096, 7, 4096), (8192, 1, 4096), (8192, 4, 4096), (8192, 8, 4096)])
def test_out_projection_rows(mode, K, M, H):
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(K + M + mode)
    wq, ws = quantize_blockwise(torch.randn(H, K, device=dev, generator=g) * 0.03)
    inp = torch.randn(8, K, device=dev, generator=g) * torch.logspace(-3, 3, 8, device=dev)[:, None]
    inp[0, 64:] *= 1e-6                                             # blocks far below their row's scale
    z = torch.randn(8, K, device=dev, generator=g)
    gnorm = 1 + 0.1 * torch.randn(128, device=dev, generator=g)
    x0 = torch.randn(8, H, device=dev, generator=g).to(torch.bfloat16)
    lib, st = load(), torch.cuda.current_stream().cuda_stream
    ch = LLChannel(dev, 1, 0, 8 * H)
    planes, descale = torch.zeros(24, K, dtype=torch.uint8, device=dev), torch.zeros(8, device=dev)
    a = inp[:M].double()
    if mode == 1:
        h = a.view(M, -1, 128)
        h = h * torch.rsqrt(h.square().mean(-1, keepdim=True) + 1e-6) * gnorm.double()
        a = (h * torch.nn.functional.silu(z[:M].double()).view(M, -1, 128)).reshape(M, K)
    y = a @ dequantize_blockwise(wq, ws).double().T
    want = y + (0 if mode & 4 else x0[:M].double())
    # bf16 result: half a unit in the last of 8 significant bits, up to 2^-8 of the value; three e4m3 terms: 2^-12 of the row's largest magnitude per input value, which the sums over
    # K values of random sign leave below 2^-12 * sqrt(K) * |a|_max * rms(w)
    bound = 2.0**-8 * want.abs() * 1.01 + 4 * 2.0**-12 * a.abs().amax(1, keepdim=True) * K**0.5 * 0.03
    for staged in (False, True):
        x = x0.clone()
        if staged:
            e = lib.nexrt_oproj_rows_allreduce(ptr(inp), ptr(z), ptr(gnorm), ptr(wq), ptr(ws), ptr(x), ptr(planes), ptr(descale), H, K, M, mode, 1e-6, 128, ch.ref, 0,
                                               None, 0, 148, st)
        else:
            e = lib.nexrt_oproj_allreduce(ptr(inp), ptr(z), ptr(gnorm), ptr(wq), ptr(ws), ptr(x), H, K, M, mode, 1e-6, 128, ch.ref, 0, None, 0, 148, st)
        check(e, "oproj")
        torch.cuda.synchronize()
        assert torch.equal(x[M:], x0[M:])
        assert ((x[:M].double() - want).abs() <= bound).all(), ((x[:M].double() - want).abs() / bound).max()
