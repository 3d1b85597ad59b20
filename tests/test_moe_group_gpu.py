"""Grouped experts of a prefill chunk: the plan against a host sort, the persistent GEMM against float64, with experts nobody is
routed to, experts of more pairs than one item holds, CTAs with no, one and many tiles, and one and several K blocks; the activation
of the pairs; and the whole block from the rows to what is added to the residual."""

import pytest
import torch

from nexrt_b200.ops.lib import check, load, ptr
from nexrt_b200.quant import dequantize_blockwise, quantize_blockwise

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _ids(g, T, S, E, skew):
    """Distinct routed experts per row, the shared expert (id E) last; ``skew``: every row picks the same ones."""
    rows = [torch.randperm(E, generator=g)[: S - 1].sort().values if not (skew and t) else None for t in range(T)]
    return torch.stack([torch.cat([r if r is not None else rows[0], torch.tensor([E])]) for r in rows]).to(torch.int32)


@pytest.mark.parametrize("T,S,E,R,K,terms,skew", [(16, 2, 1, 128, 128, 1, False), (16, 5, 16, 512, 1024, 3, False), (24, 11, 512, 256, 512, 3, False),
                                                  (64, 11, 40, 256, 384, 2, False), (128, 11, 512, 4096, 128, 3, False), (128, 4, 12, 256, 256, 1, True),
                                                  (128, 11, 30, 1024, 256, 3, True)])
def test_plan_and_group_gemm(T, S, E, R, K, terms, skew):
    g = torch.Generator().manual_seed(T + S + E)
    ids = _ids(g, T, S, E, skew)
    lib, st, pairs, n_total, NP = load(), torch.cuda.current_stream().cuda_stream, T * S, E + 1, 32 // terms
    i32 = lambda *s: torch.full(s, -1, dtype=torch.int32, device=DEV)
    items, n_items, pair_row, out_row = i32(pairs, 4), i32(1), i32(pairs), i32(pairs)
    check(lib.nexrt_moe_plan(ptr(ids.to(DEV)), ptr(items), ptr(n_items), ptr(pair_row), ptr(out_row), S, T, n_total, terms, st), "plan")
    want = sorted((int(ids[m, s]), m, s) for m in range(T) for s in range(S))
    assert pair_row.tolist() == [m for _, m, _ in want]
    assert out_row.tolist() == [s * T + m for _, m, s in want]
    tiles, first = [], 0
    for e in range(n_total):
        n = sum(1 for w in want if w[0] == e)
        tiles += [[e, first + i, min(NP, n - i), 0] for i in range(0, n, NP)]
        first += n
    assert int(n_items.item()) == len(tiles) and items[: len(tiles)].tolist() == tiles

    gd = torch.Generator(device=DEV).manual_seed(K + R)
    wq, ws = quantize_blockwise(torch.randn(n_total, R, K, device=DEV, generator=gd) * 0.03)
    xq = (torch.randn(terms * T, K, device=DEV, generator=gd) * 100).to(torch.float8_e4m3fn)
    sx = torch.rand(terms * T, K // 128, device=DEV, generator=gd) * 0.02 + 0.001
    xp, sp = torch.zeros(terms * pairs, K, dtype=torch.uint8, device=DEV), torch.zeros(pairs, K // 128, device=DEV)
    check(lib.nexrt_moe_gather(ptr(xq), ptr(sx), ptr(pair_row), ptr(xp), ptr(sp), pairs, T, K, terms, st), "gather")
    rows = pair_row.long()
    assert torch.equal(sp, sx[rows])
    assert torch.equal(xp.view(pairs, terms, K), torch.stack([xq.view(torch.uint8)[p * T + rows] for p in range(terms)], 1))
    x = sum(xq.double().view(terms, T, K)[p][rows] * 16.0**-p for p in range(terms)) * sp.double().repeat_interleave(128, 1)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    for mapped in (False, True):
        out = torch.full((pairs, R), float("nan"), device=DEV)
        check(lib.nexrt_moe_group_gemm(ptr(wq), ptr(ws), ptr(xp), ptr(sp), ptr(out), ptr(items), ptr(n_items), ptr(out_row) if mapped else None, pairs, n_total, R, K,
                                       terms, ptr(status), st), "group_gemm")
        torch.cuda.synchronize()
        assert int(status.item()) == 0
        got = out[out_row.long()] if mapped else out
        for e in range(n_total):
            sel = [i for i, w in enumerate(want) if w[0] == e]
            if sel:
                w = dequantize_blockwise(wq[e], ws[e]).double()
                y, mag = x[sel] @ w.T, x[sel].abs() @ w.abs().T
                assert ((got[sel].double() - y).abs() <= 1e-5 * mag).all(), (e, ((got[sel].double() - y).abs() / mag).max())   # fp32 sums of up to K exact products


def _plan(lib, ids, S, T, n_total, terms, st):
    i32 = lambda *s: torch.full(s, -1, dtype=torch.int32, device=DEV)
    items, n_items, pair_row, out_row = i32(T * S, 4), i32(1), i32(T * S), i32(T * S)
    check(lib.nexrt_moe_plan(ptr(ids), ptr(items), ptr(n_items), ptr(pair_row), ptr(out_row), S, T, n_total, terms, st), "plan")
    return items, n_items, pair_row, out_row


# relative error of a value written as 1, 2 or 3 e4m3 terms with a scale per 128 of them: 2^-4, 2^-8, 2^-12 of the largest
TOL = {1: 0.04, 2: 3e-3, 3: 2e-4}


@pytest.mark.parametrize("T,S,E,I,terms", [(16, 2, 4, 128, 1), (17, 5, 16, 128, 3), (24, 3, 40, 384, 2), (128, 11, 512, 128, 3), (64, 11, 512, 1024, 3)])
def test_pair_act(T, S, E, I, terms):
    g = torch.Generator().manual_seed(T + I)
    lib, st, pairs = load(), torch.cuda.current_stream().cuda_stream, T * S
    *_, pair_row, out_row = _plan(lib, _ids(g, T, S, E, False).to(DEV), S, T, E + 1, terms, st)
    gd = torch.Generator(device=DEV).manual_seed(T)
    gu, wts = torch.randn(pairs, 2 * I, device=DEV, generator=gd), torch.rand(T, S, device=DEV, generator=gd) + 0.01
    gu[:, : I // 2] *= 1e-3                                      # blocks of other magnitudes
    hq, hs = torch.zeros(terms * pairs, I, dtype=torch.float8_e4m3fn, device=DEV), torch.zeros(pairs, I // 128, device=DEV)
    check(lib.nexrt_moe_pair_act(ptr(gu), ptr(out_row), ptr(wts), ptr(hq), ptr(hs), I, S, T, terms, st), "pair_act")
    torch.cuda.synchronize()
    slot, row = out_row.long() // T, out_row.long() % T
    assert torch.equal(row, pair_row.long())
    want = torch.nn.functional.silu(gu[:, :I].double()) * gu[:, I:].double() * wts[row, slot].double()[:, None]
    got = sum(hq.double().view(pairs, terms, I)[:, p] * 16.0**-p for p in range(terms)) * hs.double().repeat_interleave(128, 1)
    err = (got - want).view(-1, 128).norm(dim=1) / want.view(-1, 128).norm(dim=1)      # every pair and block by itself
    assert err.max() <= TOL[terms], err.max()


@pytest.mark.parametrize("T,S,E,H,I,terms", [(16, 3, 8, 256, 128, 1), (64, 11, 512, 512, 128, 3), (128, 11, 64, 256, 256, 2), (64, 5, 12, 1024, 384, 3)])
def test_rows_to_residual(T, S, E, H, I, terms):
    from nexrt_b200.ops.tc_gemm import act_quant

    g = torch.Generator().manual_seed(H + I)
    gd = torch.Generator(device=DEV).manual_seed(H + I)
    lib, st, pairs, n_total = load(), torch.cuda.current_stream().cuda_stream, T * S, E + 1
    ids = _ids(g, T, S, E, False).to(DEV)
    x, wts = torch.randn(T, H, device=DEV, generator=gd), torch.rand(T, S, device=DEV, generator=gd)
    w13, s13 = quantize_blockwise(torch.randn(n_total, 2 * I, H, device=DEV, generator=gd) * 0.05)
    w2, s2 = quantize_blockwise(torch.randn(n_total, H, I, device=DEV, generator=gd) * 0.05)
    xq, sx = act_quant(x, terms=terms)
    items, n_items, pair_row, out_row = _plan(lib, ids, S, T, n_total, terms, st)
    f8, f32 = lambda *s: torch.zeros(*s, dtype=torch.float8_e4m3fn, device=DEV), lambda *s: torch.full(s, float("nan"), device=DEV)
    xp, sp, gu, hq, hs, y, out = f8(terms * pairs, H), f32(pairs, H // 128), f32(pairs, 2 * I), f8(terms * pairs, I), f32(pairs, I // 128), f32(S * T, H), f32(T, H)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    check(lib.nexrt_moe_gather(ptr(xq), ptr(sx), ptr(pair_row), ptr(xp), ptr(sp), pairs, T, H, terms, st), "gather")
    check(lib.nexrt_moe_group_gemm(ptr(w13), ptr(s13), ptr(xp), ptr(sp), ptr(gu), ptr(items), ptr(n_items), None, pairs, n_total, 2 * I, H, terms, ptr(status), st), "up")
    check(lib.nexrt_moe_pair_act(ptr(gu), ptr(out_row), ptr(wts), ptr(hq), ptr(hs), I, S, T, terms, st), "pair_act")
    check(lib.nexrt_moe_group_gemm(ptr(w2), ptr(s2), ptr(hq), ptr(hs), ptr(y), ptr(items), ptr(n_items), ptr(out_row), pairs, n_total, H, I, terms, ptr(status), st), "down")
    check(lib.nexrt_planes_residual(None, ptr(y), ptr(out), T * H, S, st), "planes_sum")
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    want = torch.zeros(T, H, dtype=torch.float64, device=DEV)
    for e in range(n_total):
        row, slot = (ids == e).nonzero(as_tuple=True)
        if len(row):
            u = x[row].double() @ dequantize_blockwise(w13[e], s13[e]).double().T
            h = torch.nn.functional.silu(u[:, :I]) * u[:, I:] * wts[row, slot].double()[:, None]
            want.index_add_(0, row, h @ dequantize_blockwise(w2[e], s2[e]).double().T)
    # the rounding of the rows reaches gate and up, that of h comes on top
    err = (out.double() - want).norm(dim=1) / want.norm(dim=1)
    assert err.max() <= 4 * TOL[terms], err.max()
