"""Fronts of 2..8 rows (terms made once, weights streamed once) against float64: fewer row groups than CTAs, exactly one round of
CTAs and several, one and two K steps of the register ring, rings that wrap."""

import pytest
import torch

from nexrt_b200.ops.lib import check, load, ptr
from nexrt_b200.quant import dequantize_blockwise, quantize_blockwise
from nexrt_b200.runtime.control import CTL_WORDS, Ctl

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rows(g, M, H):
    x = torch.randn(8, H, device=DEV, generator=g).to(torch.bfloat16)
    ln = 1 + 0.1 * torch.randn(H, device=DEV, generator=g)
    xd = x[:M].double()
    return x, ln, xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-6) * ln.double()


def _close(got, want, xn, what):
    # three e4m3 terms leave 2^-12 of an input value, at least 2^-13 of one (the terms' fixed scale), random over the K products
    bound = 4 * 2.0**-12 * xn.abs().amax() * xn.shape[1] ** 0.5 * 0.03 + 1e-5 * want.abs().max()
    assert (got.double() - want).abs().max() <= bound, (what, (got.double() - want).abs().max(), bound)


@pytest.mark.parametrize("H,nqk,nv,M,C0", [(256, 1, 1, 2, 0), (1024, 1, 2, 5, 14), (4096, 2, 8, 8, 979), (4096, 2, 8, 3, 1), (4096, 8, 32, 2, 40), (4096, 8, 32, 6, 29), (4096, 2, 8, 2, 13)])
def test_gdn_front_rows(H, nqk, nv, M, C0):
    g = torch.Generator(device=DEV).manual_seed(H + nv + M)
    C, R, ring = (2 * nqk + nv) * 128, (2 * nqk + 2 * nv) * 128, 16
    wq, ws = quantize_blockwise(torch.randn(R, H, device=DEV, generator=g) * 0.03)
    ba = (torch.randn(2 * nv, H, device=DEV, generator=g) * 0.03).to(torch.bfloat16)
    conv = torch.randn(C, 4, device=DEV, generator=g)
    a_log, dt = torch.randn(nv, device=DEV, generator=g), torch.randn(nv, device=DEV, generator=g)
    x, ln, xn = _rows(g, M, H)
    ctl = torch.zeros(CTL_WORDS, dtype=torch.int32, device=DEV)
    ctl[Ctl.COMMITTED_LEN] = C0
    hist = torch.randn(ring, C, device=DEV, generator=g)
    if C0 == 0:
        hist.zero_()
    rings = hist.clone()
    z = lambda *s: torch.zeros(*s, device=DEV)
    qkv, zz, beta, gg = z(8, C), z(8, R - C), z(8, nv), z(8, nv)
    cols = torch.zeros(16, H, dtype=torch.float16, device=DEV)
    check(load().nexrt_gdn_front_rows(ptr(x), ptr(ln), ptr(wq), ptr(ws), ptr(ba), ptr(conv), ptr(a_log), ptr(dt), ptr(ctl), ptr(rings), ptr(qkv), ptr(zz), ptr(beta),
                                      ptr(gg), ptr(cols), H, R, C, nv, M, ring, 1e-6, torch.cuda.current_stream().cuda_stream), "gdn_front_rows")
    torch.cuda.synchronize()
    pre = xn @ dequantize_blockwise(wq, ws).double().T
    slots = [(C0 + m) % ring for m in range(M)]
    _close(rings[slots], pre[:, :C], xn, "history")
    keep = [s for s in range(ring) if s not in slots]
    assert torch.equal(rings[keep], hist[keep])
    win = torch.cat([hist[[(C0 - 3 + j) % ring for j in range(3)]].double(), pre[:, :C]])
    out = torch.stack([(win[m : m + 4].T * conv.double()).sum(1) for m in range(M)])
    _close(qkv[:M], torch.nn.functional.silu(out), xn * 4, "conv")
    _close(zz[:M], pre[:, C:], xn, "z")
    b = xn @ ba.double().T
    assert (beta[:M].double() - torch.sigmoid(b[:, :nv])).abs().max() < 1e-5
    want = -a_log.double().exp() * torch.nn.functional.softplus(b[:, nv:] + dt.double())
    assert ((gg[:M].double() - want).abs() <= 1e-5 * want.abs() + 1e-6).all()
    assert not qkv[M:].any() and not zz[M:].any() and not beta[M:].any()


@pytest.mark.parametrize("H,hd,nq,ngate,kvh,M,C0", [(256, 128, 1, 1, 1, 2, 0), (4096, 256, 4, 4, 1, 8, 100), (4096, 256, 16, 4, 1, 3, 7), (4096, 256, 32, 32, 2, 7, 28), (4096, 256, 4, 4, 1, 2, 30)])
def test_attn_front_rows(H, hd, nq, ngate, kvh, M, C0):
    g = torch.Generator(device=DEV).manual_seed(H + nq + M)
    R, cache = (nq + ngate + 2 * kvh) * hd, C0 + 4          # the last rows of a step may lie past the end of the cache
    wq, ws = quantize_blockwise(torch.randn(R, H, device=DEV, generator=g) * 0.03)
    x, ln, xn = _rows(g, M, H)
    ctl = torch.zeros(CTL_WORDS, dtype=torch.int32, device=DEV)
    ctl[Ctl.COMMITTED_LEN] = C0
    z = lambda *s: torch.zeros(*s, device=DEV)
    q, gate, k, v = z(8, nq, hd), z(8, ngate, hd), z(8, kvh, hd), z(kvh, cache, hd).to(torch.bfloat16)
    cols = torch.zeros(16, H, dtype=torch.float16, device=DEV)
    check(load().nexrt_attn_front_rows(ptr(x), ptr(ln), ptr(wq), ptr(ws), ptr(ctl), ptr(q), ptr(gate), ptr(k), ptr(v), ptr(cols), H, hd, nq, ngate, kvh, M, cache, 1e-6,
                                       torch.cuda.current_stream().cuda_stream), "attn_front_rows")
    torch.cuda.synchronize()
    pre = xn @ dequantize_blockwise(wq, ws).double().T
    heads = pre[:, : (nq + ngate) * hd].view(M, nq + ngate, hd)
    wq_, wg_ = (heads[:, 0::2], heads[:, 1::2]) if nq == ngate else (heads[:, :nq], heads[:, nq:])
    _close(q[:M], wq_, xn, "q")
    _close(gate[:M], wg_, xn, "gate")
    kv = pre[:, (nq + ngate) * hd :].view(M, 2, kvh, hd)
    _close(k[:M], kv[:, 0], xn, "k")
    n = min(M, 4)
    got, want = v[:, C0 : C0 + n].double(), kv[:n, 1].transpose(0, 1)
    assert ((got - want).abs() <= 2.0**-8 * want.abs() + 1e-2).all()
    assert not v[:, :C0].any() and not q[M:].any()
