"""The kernel instantiations the 8-GPU deployment runs, against the fp32 oracle, on one GPU.

Every other numerics test uses the shrunk geometry (hidden 1024, head_dim 128, 16 experts top-4, vocab 4096).  The
deployment at tensor-parallel 8 launches different template instances and shapes: head_dim-256 attention with 4 query
heads on one kv head, the 528-row router with top-10, K = 4096 projection fronts, 8 gated-delta-net value heads, the
31 040-row vocabulary shard.  ``rank_shard_config`` is a two-layer model whose global shapes are exactly one rank's
shard, so running it at tp = 1 executes those instances; the oracle keeps the 513 experts in FP8 and dequantises only
the ones a token selects.  (The reference checks its full-size kernels against torch references with real weights,
``nex_n2_5_pro/gdn.py:327-408`` and the other block mains; this is the checkpoint-free form.)
"""

import pytest
import torch

from nexrt_b200.config import rank_shard_config
from nexrt_b200.models.reference import RefModel, robust_prompt, synthetic_prompt
from nexrt_b200.testing import gather_logits

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return float((a - b).norm() / b.norm().clamp_min(1e-12))


@pytest.fixture(scope="module")
def setup():
    from nexrt_b200.decode_engine import DecodeEngine
    from nexrt_b200.weights import random_checkpoint, shard_model

    cfg = rank_shard_config()
    dev = torch.device("cuda", torch.cuda.current_device())
    ckpt_gpu = random_checkpoint(cfg, seed=3, device=dev)        # generated on the device: 3 x 513 expert matrices per layer
    model = shard_model(ckpt_gpu, cfg, 1, 0, dev)
    ckpt = {k: v.cpu() for k, v in ckpt_gpu.items()}
    del ckpt_gpu
    ref = RefModel(cfg, ckpt)
    eng = DecodeEngine(0, 1, dev, ext=model, cfg=cfg, max_rows=8, cache_len=512)
    eng.head.enable_logits()
    return cfg, ref, eng


def _check(got, want, tol=2e-2):
    assert rel_l2(got, want) < tol, rel_l2(got, want)
    top = int(got.argmax())
    assert top == int(want.argmax()) or float(want.max() - want[top]) < 0.05


def test_one_row_steps_at_deployment_shapes(setup):
    cfg, ref, eng = setup
    # top-10 of 512 random experts: the 10th and 11th logits are close for most tokens, and picking the other one moves the
    # output by several per cent - a property of random weights, not of the kernels.  Take the prompt whose oracle run
    # stays furthest from such ties.
    prompt, margin = robust_prompt(ref, cfg.vocab, 8, seeds=range(1, 13))
    ref.reset()
    eng.reset(first_token=prompt[0])
    for tok in prompt:
        eng.set_rows([tok])
        eng.set_forced_commit(1)
        eng.step(1)
        _check(gather_logits(eng, 1)[0], ref.step(tok))
    ctl = eng.read_ctl()
    assert ctl["committed_len"] == len(prompt) and ctl["status"] == 0


@pytest.mark.parametrize("rows", [2, 4, 8])     # 2: the ragged end of a prompt
def test_verify_rows_at_deployment_shapes(setup, rows):
    """The speculative verifiers' row counts (tcgen05 experts, wide fronts, multi-row attention)."""
    cfg, ref, eng = setup
    prompt, margin = robust_prompt(ref, cfg.vocab, 2 * rows, seeds=range(20, 28))
    ref.reset()
    want = torch.stack([ref.step(t) for t in prompt])
    eng.reset(first_token=prompt[0])
    got = []
    for i in range(0, len(prompt), rows):
        eng.set_rows(prompt[i : i + rows])
        eng.set_forced_commit(rows)
        eng.step(rows)
        got.append(gather_logits(eng, rows))
    got = torch.cat(got)
    for g, w in zip(got, want):
        _check(g, w)
    assert eng.read_ctl()["status"] == 0


def test_graph_replay_at_deployment_shapes(setup):
    """Captured one-row graph: same tokens as the eager steps from the same boundary (programmatic launch, early reads
    of the committed length, cluster attention and the routed expert pair all inside one graph)."""
    cfg, ref, eng = setup
    prompt = synthetic_prompt(cfg.vocab, 16, seed=7)
    first = eng.prefill(prompt, chunk=8)
    state = eng.export_state()
    eager = []
    for _ in range(5):
        eng.step(1)
        eager.append(eng.read_ctl()["emitted"][0])
    eng.load_prefill(state)
    assert eng.read_ctl()["pending"] == first
    assert eng.generate(max_new=5) == eager


def test_prompt_that_ends_on_two_rows(setup):
    """A prompt of 8 n + 2 tokens: the last prefill step has two rows.  Same logits as the oracle's last token."""
    cfg, ref, eng = setup
    prompt, margin = robust_prompt(ref, cfg.vocab, 10, seeds=range(30, 38))
    ref.reset()
    want = [ref.step(t) for t in prompt][-1]
    eng.prefill(prompt, chunk=8)
    _check(gather_logits(eng, 2)[1], want)
    assert eng.read_ctl()["committed_len"] == len(prompt)
