"""Decode attention with a cache long enough for the streaming form, against float64: short contexts and long ones, at the edges of its
16-key tiles, with fewer tiles than rings and more, one to several row groups and passes; and caches and contexts at the lines between
the forms: where the cache's length chooses, where the committed length chooses on the device, and steps that end past the cache."""

import pytest
import torch

from nexrt_b200.ops.lib import check, load, ptr
from nexrt_b200.runtime.control import CTL_WORDS, Ctl

pytestmark = pytest.mark.gpu
DEV, HD, ROT = "cuda", 256, 64


@pytest.mark.parametrize("M,nq,kvh", [(1, 4, 1), (2, 4, 1), (3, 4, 1), (8, 4, 1), (1, 8, 1), (5, 8, 1), (1, 32, 2), (8, 32, 2), (8, 8, 4)])
@pytest.mark.parametrize("C0", [5, 1023, 1040, 1301, 4095, 4097, 9999, 20000])
def test_long_context_decode(M, nq, kvh, C0):
    _check_decode(M, nq, kvh, C0, max(C0, 6000) + M + 3)


# The cluster kernel alone for caches of up to 2048 rows (one row of 16 heads: 3072, of 2 x 16: 11264), the streaming form alone behind
# them; one row of more than eight heads launches both for longer caches, and the committed length decides.
@pytest.mark.parametrize("M,nq,kvh,keys,cache", [(1, 4, 1, 1, 2049), (8, 4, 1, 8, 2049), (2, 8, 1, 17, 2049), (3, 4, 1, 2047, 2048), (3, 4, 1, 2048, 2048), (3, 4, 1, 2049, 2048),
                                                 (3, 4, 1, 2047, 2049), (3, 4, 1, 2048, 2049), (3, 4, 1, 2049, 2049), (3, 4, 1, 2050, 2049), (8, 4, 1, 4100, 4096),
                                                 (3, 8, 2, 2049, 2049), (3, 8, 2, 2051, 2049), (8, 32, 2, 8, 64), (8, 32, 2, 66, 64),
                                                 (1, 16, 1, 1, 3073), (1, 16, 1, 3072, 3072), (1, 16, 1, 3071, 3073), (1, 16, 1, 3072, 3073), (1, 16, 1, 3073, 3073),
                                                 (1, 32, 2, 1, 11265), (1, 32, 2, 11264, 11264), (1, 32, 2, 11263, 11265), (1, 32, 2, 11264, 11265), (1, 32, 2, 11265, 11265),
                                                 (1, 32, 2, 12345, 20000)])
def test_lines_between_the_forms(M, nq, kvh, keys, cache):
    _check_decode(M, nq, kvh, keys - M, cache)


@pytest.mark.parametrize("hd,nq,kvh,M,keys", [(256, 4, 1, 1, 2048), (256, 8, 1, 1, 2048), (256, 4, 1, 8, 2048), (256, 16, 1, 1, 3072), (256, 16, 1, 3, 2048), (256, 32, 2, 1, 11264),
                                              (256, 16, 1, 4, 0), (256, 32, 2, 2, 0), (256, 8, 1, 8, 0), (128, 4, 1, 1, 2**31 - 1)])
def test_keys_of_the_cluster_kernel(hd, nq, kvh, M, keys):
    assert load().nexrt_attn_cluster_keys(hd, nq, kvh, M, ROT) == keys


def _check_decode(M, nq, kvh, C0, cache):
    g = torch.Generator(device=DEV).manual_seed(M * 1000 + nq + C0)
    n_splits, G, end = 148 // kvh, nq // kvh, min(C0 + M, cache)
    rn = lambda *s: torch.randn(*s, device=DEV, generator=g)
    q, gate, k, qn, kn = rn(8, nq, HD), rn(8, nq, HD), rn(8, kvh, HD), 1 + 0.1 * rn(HD), 1 + 0.1 * rn(HD)
    kc, vc = rn(kvh, cache, HD).to(torch.bfloat16), rn(kvh, cache, HD).to(torch.bfloat16)
    kc[:, C0:] = float("nan")                                  # rows of the future: never read
    vc[:, C0 + M :] = float("nan")
    inv = 1.0 / (1e7 ** (torch.arange(0, ROT, 2, dtype=torch.float32) / ROT)).to(DEV)
    ang = torch.arange(cache + M, dtype=torch.float32, device=DEV)[:, None] * inv[None, :]
    whole = torch.stack([ang.cos(), ang.sin()], -1)
    rope = whole[:cache].contiguous()
    ctl = torch.zeros(CTL_WORDS, dtype=torch.int32, device=DEV)
    ctl[Ctl.COMMITTED_LEN] = C0
    ws_acc, ws_ml = torch.full((kvh, n_splits, 8 * G, HD), float("nan"), device=DEV), torch.full((kvh, n_splits, 8 * G, 2), float("nan"), device=DEV)
    ticket, out = torch.zeros(kvh, dtype=torch.int32, device=DEV), torch.zeros(8, nq * HD, device=DEV)
    for flags in (8, 0, 16, 8 | 32):                            # the last two: the caller names the side of the line, rightly or not
        out.zero_()
        kcc = kc.clone()
        check(load().nexrt_attn_decode(ptr(q), ptr(gate), ptr(k), ptr(qn), ptr(kn), ptr(inv), ptr(rope), ptr(ctl), ptr(kcc), ptr(vc), ptr(ws_acc), ptr(ws_ml), ptr(ticket),
                                       ptr(out), HD, nq, nq, kvh, M, cache, ROT, n_splits, 1e-6, flags, 0, 0, 0, 1, 0, None, 0,
                                       torch.cuda.current_stream().cuda_stream), "attn_decode")
        torch.cuda.synchronize()
        norm = lambda x, w: x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * w.double()

        def rot(x):
            c, s = whole[C0 : C0 + M, :, 0].double()[:, None], whole[C0 : C0 + M, :, 1].double()[:, None]
            a, b = x[..., : ROT // 2], x[..., ROT // 2 : ROT]
            return torch.cat([a * c - b * s, b * c + a * s, x[..., ROT:]], -1)

        qd, kd = rot(norm(q[:M].double(), qn)), rot(norm(k[:M].double(), kn))
        new, kd = kcc[:, C0:end].double(), kd.transpose(0, 1)[:, : end - C0]
        assert ((new - kd).abs() <= 2.0**-8 * kd.abs() + 1e-5).all()
        assert torch.equal(kcc[:, :C0], kc[:, :C0])
        K, V = torch.cat([kc[:, :C0].double(), new], 1), vc[:, :end].double()
        sc = torch.einsum("mhgd,hkd->mhgk", qd.view(M, kvh, G, HD), K) / 16.0
        sc = sc.masked_fill(torch.arange(end, device=DEV) > torch.arange(C0, C0 + M, device=DEV)[:, None, None, None], -float("inf"))
        p = torch.softmax(sc, -1)
        ctx = torch.einsum("mhgk,hkd->mhgd", p, V).reshape(M, nq, HD) * torch.sigmoid(gate[:M].double())
        # Q and P are bf16 hi + lo (2^-17), everything else fp32: errors stay below 2^-14 of sum p |v|
        bound = 2.0**-14 * torch.einsum("mhgk,hkd->mhgd", p, V.abs()).reshape(M, nq, HD) + 1e-6
        err = (out[:M].view(M, nq, HD).double() - ctx).abs()
        assert (err <= bound).all(), (err / bound).max()
        assert not out[M:].any()
