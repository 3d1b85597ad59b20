"""Shared memory of the row kernels.  Layout of the CUDA-core forms: what lies behind the partial sums starts on a 16-byte boundary,
whatever the numbers of rows, CTAs and threads (the layout function is compiled for the host).  Size: launches whose dynamic
memory alone stays within the default limit of 48 KB and whose static memory takes them over it."""

import shutil
import subprocess

import pytest

from nexrt_b200 import build as B

PROGRAM = r"""
#include "gemv_cta.cuh"
#include <cstdio>
int main() {
    const int threads[] = {128, 256, 512}, ctas[] = {1, 7, 132, 148, 1024}, per_chunk[] = {8, 16};
    int bad = 0;
    for (int H = 256; H <= 4096; H += 256)
        for (int t : threads)
            for (int e : per_chunk)
                for (int mb : {1, 4})
                    for (int n : ctas)
                        for (int rows = 16; rows <= 4096; rows += 113) {
                            const nexrt::GemvGeom g = nexrt::gemv_geom(H / e, t);
                            const int nrows = (rows + n - 1) / n;
                            const size_t f = nexrt::gemv_part_floats(nrows, mb, g), need = static_cast<size_t>(nrows) * g.wpr * mb;
                            if (f % 4 || f < need || f > need + 3) ++bad;
                        }
    std::printf("%d\n", bad);
    return 0;
}
"""


def test_partial_sums_end_on_a_16_byte_boundary(tmp_path):
    nvcc = B.nvcc_path()
    if shutil.which(nvcc) is None:
        pytest.skip("no nvcc on this machine")
    src = tmp_path / "layout.cu"
    src.write_text(PROGRAM)
    subprocess.run([nvcc, *B.ARCH_FLAGS, "-std=c++17", "-I", str(B.CSRC), "-o", str(tmp_path / "layout"), str(src)], check=True, capture_output=True)
    assert subprocess.run([str(tmp_path / "layout")], check=True, capture_output=True, text=True).stdout.strip() == "0"


# ---- the kernels themselves, at odd numbers of partial sums per CTA -----------------------------------------------------
def _setup(H, R, seed):
    import torch
    from nexrt_b200.quant import dequantize_blockwise, quantize_blockwise

    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(1, H, device="cuda", generator=g).to(torch.bfloat16)
    ln = 1 + 0.1 * torch.randn(H, device="cuda", generator=g)
    wq, ws = quantize_blockwise(torch.randn(R, H, device="cuda", generator=g) * 0.03)
    xd = x.double()
    return g, x, ln, wq, ws, xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-6) * ln.double(), dequantize_blockwise(wq, ws).double()


def _close(got, xn, w):
    # fp32 norm, products and sums of up to 2^11 terms
    assert ((got.double() - xn @ w.T).abs() <= 1e-5 * (xn.abs() @ w.abs().T)).all()


@pytest.mark.gpu
@pytest.mark.parametrize("H,n_cta", [(256, 512), (256, 74), (1280, 74), (256, 171)])
def test_attn_front(H, n_cta):
    import torch
    from nexrt_b200.ops.lib import check, load, ptr
    from nexrt_b200.runtime.control import CTL_WORDS

    hd, R = 128, 512
    assert H % 512 and -(-R // n_cta) % 2
    g, x, ln, wq, ws, xn, w = _setup(H, R, H + n_cta)
    z = lambda *s: torch.zeros(*s, device="cuda")
    q, gate, k, v, ctl = z(1, hd), z(1, hd), z(1, hd), z(1, 4, hd).to(torch.bfloat16), torch.zeros(CTL_WORDS, dtype=torch.int32, device="cuda")
    check(load().nexrt_attn_front(ptr(x), ptr(ln), ptr(wq), ptr(ws), ptr(ctl), ptr(q), ptr(gate), ptr(k), ptr(v), H, hd, 1, 1, 1, 1, 4, 1e-6, n_cta,
                                  torch.cuda.current_stream().cuda_stream), "attn_front")
    torch.cuda.synchronize()
    _close(torch.cat([q, gate, k], 1), xn, w[:384])
    want = xn @ w[384:].T
    assert ((v[0, 0].double() - want[0]).abs() <= 2.0**-8 * want[0].abs() + 1e-5).all()


@pytest.mark.gpu
@pytest.mark.parametrize("H,n_cta", [(256, 148), (768, 171), (256, 512)])
def test_gdn_front(H, n_cta):
    import torch
    from nexrt_b200.ops.lib import check, load, ptr
    from nexrt_b200.runtime.control import CTL_WORDS

    R, C, nv, ring = 512, 384, 1, 16
    g, x, ln, wq, ws, xn, w = _setup(H, R, H + n_cta)
    ba = (torch.randn(2 * nv, H, device="cuda", generator=g) * 0.03).to(torch.bfloat16)
    conv, z = torch.randn(C, 4, device="cuda", generator=g), lambda *s: torch.zeros(*s, device="cuda")
    rings, qkv, zz, beta, gg, ctl = z(ring, C), z(1, C), z(1, R - C), z(1, nv), z(1, nv), torch.zeros(CTL_WORDS, dtype=torch.int32, device="cuda")
    check(load().nexrt_gdn_front(ptr(x), ptr(ln), ptr(wq), ptr(ws), ptr(ba), ptr(conv), ptr(z(nv)), ptr(z(nv)), ptr(ctl), ptr(rings), ptr(qkv), ptr(zz), ptr(beta), ptr(gg),
                                 H, R, C, nv, 1, ring, 1e-6, 0, n_cta, torch.cuda.current_stream().cuda_stream), "gdn_front")
    torch.cuda.synchronize()
    _close(rings[:1], xn, w[:C])
    _close(zz, xn, w[C:])
    assert (beta.double() - torch.sigmoid(xn @ ba[:1].double().T)).abs().max() < 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("H", [256, 768])
def test_router_and_gate_up(H):
    import torch
    from nexrt_b200.ops.lib import check, load, ptr

    E, topk, I, n_cta = 128, 3, 128, 148
    S, R = topk + 1, 2 * I
    g, x, ln, wq, ws, xn, w = _setup(H, (E + 1) * R, H)
    rw = (torch.randn(E + 1, H, device="cuda", generator=g) * 0.03).to(torch.bfloat16)
    z, st = lambda *s, **k: torch.zeros(*s, device="cuda", **k), torch.cuda.current_stream().cuda_stream
    logits, ids, wts, ticket, gu = z(1, E + 1), z(1, S, dtype=torch.int32), z(1, S), z(1, dtype=torch.int32), z(S, R)
    check(load().nexrt_moe_router(ptr(x), ptr(ln), ptr(rw), ptr(logits), ptr(ids), ptr(wts), ptr(ticket), None, 0, H, E, topk, 1, 1e-6, n_cta, None, st), "router")
    check(load().nexrt_moe_l1(ptr(x), ptr(ln), ptr(wq), ptr(ws), ptr(ids), ptr(gu), H, I, S, 1, 1e-6, E, n_cta, st), "l1")
    torch.cuda.synchronize()
    _close(logits, xn, rw.double())
    picked = ids[0].tolist()
    assert picked[-1] == E and sorted(picked[:-1]) == sorted(logits[0, :E].topk(topk).indices.tolist())
    for s, e in enumerate(picked):
        _close(gu[s : s + 1], xn, w[e * R : (e + 1) * R])


@pytest.mark.gpu
@pytest.mark.parametrize("H,hd,heads,n_cta", [(2304, 128, 2, 27),       # 32 bytes of dynamic memory below 48 KB
                                              (4096, 256, 4, 148)])     # the model's width, above it
def test_attn_front_of_two_rows_at_the_default_limit(H, hd, heads, n_cta):
    import torch
    from nexrt_b200.ops.lib import check, load, ptr
    from nexrt_b200.quant import dequantize_blockwise, quantize_blockwise
    from nexrt_b200.runtime.control import CTL_WORDS

    M, kvh = 2, 1 if heads == 4 else 2
    R = (2 * heads + 2 * kvh) * hd
    g = torch.Generator(device="cuda").manual_seed(H)
    x = torch.randn(M, H, device="cuda", generator=g).to(torch.bfloat16)
    ln = 1 + 0.1 * torch.randn(H, device="cuda", generator=g)
    wq, ws = quantize_blockwise(torch.randn(R, H, device="cuda", generator=g) * 0.03)
    z = lambda *s: torch.zeros(*s, device="cuda")
    q, gate, k, v, ctl = z(M, heads, hd), z(M, heads, hd), z(M, kvh, hd), z(kvh, 4, hd).to(torch.bfloat16), torch.zeros(CTL_WORDS, dtype=torch.int32, device="cuda")
    check(load().nexrt_attn_front(ptr(x), ptr(ln), ptr(wq), ptr(ws), ptr(ctl), ptr(q), ptr(gate), ptr(k), ptr(v), H, hd, heads, heads, kvh, M, 4, 1e-6, n_cta,
                                  torch.cuda.current_stream().cuda_stream), "attn_front")
    torch.cuda.synchronize()
    xd = x.double()
    xn, w = xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-6) * ln.double(), dequantize_blockwise(wq, ws).double()
    pre = (xn @ w.T)[:, : (2 * heads + kvh) * hd].view(M, 2 * heads + kvh, hd)
    got = torch.cat([torch.stack([q, gate], 2).view(M, 2 * heads, hd), k], 1).double()
    assert ((got - pre).abs() <= 1e-5 * (xn.abs() @ w.abs().T)[:, : (2 * heads + kvh) * hd].view(pre.shape)).all()      # fp32, as above
