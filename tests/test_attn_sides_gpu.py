"""One row of sixteen heads with a cache on both sides of the attention line: ``generate`` crosses it on two graphs, each with one of the
forms alone, and gives the tokens of the graph in which the device chooses."""

from dataclasses import replace

import pytest
import torch

from nexrt_b200.attn import FullAttn
from nexrt_b200.config import rank_shard_config
from nexrt_b200.decode_engine import DecodeEngine
from nexrt_b200.runtime.context import FAR, NEAR
from nexrt_b200.weights import random_rank_model

pytestmark = pytest.mark.gpu


def test_generate_across_the_line():
    dev = torch.device("cuda", 0)
    cfg = replace(rank_shard_config(), name="sixteen-heads", n_q_heads=16, n_experts=32, vocab=4096, max_context=3072)
    eng = DecodeEngine(0, 1, dev, ext=random_rank_model(cfg, 1, 0, dev, seed=3), cfg=cfg, max_rows=1, cache_len=3200)
    line, new = 3072, 12
    attn = next(m for m in eng.mixers if isinstance(m, FullAttn))
    assert eng.ctx.lib.nexrt_attn_cluster_keys(256, 16, 1, 1, cfg.rotary_dim) == line
    g = torch.Generator(device=dev).manual_seed(1)
    k, v = (torch.randn(1, line, 256, device=dev, generator=g).to(torch.bfloat16) for _ in range(2))
    out = {}
    for start in (line - 6, line - new, line):          # across the line, on its near side, beyond it
        for plain in (True, False):
            eng.graphs.clear()
            eng.reset(first_token=7, committed_len=start)
            attn.load_kv(k[:, :start], v[:, :start])
            out[plain] = eng.generate(eng.capture(1) if plain else None, max_new=new)
            want = {(1, False)} if plain else {(1, False, NEAR)} if start + new <= line else {(1, False, FAR)} if start == line else {(1, False, NEAR), (1, False, FAR)}
            assert set(eng.graphs) == want
            assert eng.status_max() == 0 and eng.ctx.attn_side == 0
        assert out[True] == out[False] and len(out[True]) == new
