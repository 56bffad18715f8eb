"""Block prefill of models with sparse MLPs and latent attention (tokens sorted by expert, grouped projections, the
latent attention of several positions per block) against the token-by-token prefill through the decode step."""
import dataclasses
import os
import threading

import numpy as np
import pytest

from nerva_b200 import ops, synth
from nerva_b200.session import CudaHfDecodeSequenceLoop, CudaHfDecodeSequenceSession, SmokeStatus

pytestmark = pytest.mark.gpu

# Both prefills round the projections' inputs and the cached rows to bf16; they differ in the order of fp32 sums, which
# moves single roundings: the bound that the token-by-token sessions are held to against the oracle.
LOGIT_ATOL = 2e-2

# widths that are no multiple of a tile: 128 rows, 64 columns, 256 rows of the down projection
MOE = synth.DecoderConfig("moe", layers=2, hidden=320, heads=8, kv_heads=2, head_dim=64, intermediate=1024, vocab=2048,
                          rope_theta=1e6, qk_norm=True, num_experts=12, top_k=3, moe_intermediate=136,
                          shared_intermediate=0, norm_topk_prob=True)
MOE_SHARED = dataclasses.replace(MOE, hidden=512, num_experts=40, top_k=5, moe_intermediate=256, shared_intermediate=72)
# a step's activations of all experts exceed shared memory: the down projection goes in passes
MOE_WIDE = dataclasses.replace(MOE, layers=1, hidden=1600, intermediate=5120, num_experts=16, top_k=12, moe_intermediate=5120,
                               shared_intermediate=2056)
LATENT = dataclasses.replace(synth.DEEPSEEK_V2_LITE, layers=3, vocab=4096, hidden=512, heads=4, kv_heads=4, head_dim=64,
                             intermediate=1024, num_experts=8, top_k=2, moe_intermediate=128, shared_intermediate=256,
                             kv_lora_rank=128, qk_nope_head_dim=64, qk_rope_head_dim=32)
LATENT_256 = dataclasses.replace(LATENT, heads=5, kv_heads=5, head_dim=64, kv_lora_rank=256, qk_nope_head_dim=72,
                                 qk_rope_head_dim=24)
FULL = dataclasses.replace(synth.DEEPSEEK_V2_LITE, layers=2, vocab=4096)

_checkpoints = {}


def _checkpoint(cfg):
    key = (cfg.name, cfg.hidden, cfg.kv_lora_rank, cfg.num_experts)
    if key not in _checkpoints:
        _checkpoints[key] = synth.dense_checkpoint(cfg, fill=ops.synth_normal_bf16)
    return _checkpoints[key]


def _start(session, prompt, by_decode=False):
    if by_decode:
        os.environ["NERVA_B200_PREFILL"] = "decode"
    try:
        start, loop = CudaHfDecodeSequenceLoop.start(session, prompt)
    finally:
        os.environ.pop("NERVA_B200_PREFILL", None)
    assert start.status == SmokeStatus.OK, start.error
    return start, loop


def _steps_apart(a, b):
    fa, fb = synth.bf16_to_f32(a), synth.bf16_to_f32(b)
    top = max(float(np.abs(fa).max()), float(np.abs(fb).max()))
    return 0.0 if top == 0.0 else float(np.abs(fa - fb).max() / 2.0 ** (np.floor(np.log2(top)) - 7))


@pytest.mark.parametrize("cfg,count", [(MOE, 2), (MOE, 7), (MOE, 129), (MOE_SHARED, 9), (MOE_SHARED, 300), (MOE_WIDE, 5), (LATENT, 4),
                                       (LATENT, 35), (LATENT, 257), (LATENT_256, 66), (FULL, 33), (FULL, 210)])
def test_block_prefill_matches_prefill_by_decode(built_lib, cfg, count):
    checkpoint = _checkpoint(cfg)
    prompt = synth.uniform_u32(3, synth.T_PROMPT, count, cfg.vocab)
    block, serial = (CudaHfDecodeSequenceSession(checkpoint, count + 8) for _ in range(2))
    assert block.status == SmokeStatus.OK, block.error
    # pages out of order
    block.set_kv_block_table(synth.permutation(5, synth.T_PAGE_TABLE, (count + 8 + 15) // 16))
    start_b, loop_b = _start(block, prompt)
    start_s, loop_s = _start(serial, prompt, by_decode=True)
    assert start_b.graph_replays == 0 and start_s.graph_replays == count
    assert np.abs(block.read_logits() - serial.read_logits()).max() <= LOGIT_ATOL
    # one rounding step in the first layer; behind it a stream that has already moved by one
    for layer, steps in ((0, 1.0), (cfg.layers - 1, 2.0)):
        for token in sorted({0, count // 2, count - 1}):
            assert _steps_apart(block.read_kv_row(layer, token, 0), serial.read_kv_row(layer, token, 0)) <= steps
    assert loop_b.advance(4).tokens == loop_s.advance(4).tokens
    block.destroy()
    serial.destroy()


@pytest.mark.parametrize("cfg", [MOE_SHARED, LATENT])
def test_block_prefill_behind_a_context_and_in_threads(built_lib, cfg):
    """append after a prompt gives the logits of the whole prompt; forks in threads share the workspace in turn."""
    checkpoint = _checkpoint(cfg)
    session = CudaHfDecodeSequenceSession(checkpoint, 320)
    prompts = [synth.uniform_u32(11 + i, synth.T_PROMPT, 150 + 31 * i, cfg.vocab) for i in range(3)]
    want = []
    for prompt in prompts:
        want.append(session.append(prompt, want=[70, len(prompt) - 1], reset=True))
    head = session.append(prompts[0][:64], want=[63], reset=True)
    tail = session.append(prompts[0][64:], want=[6, len(prompts[0]) - 65])
    assert np.abs(tail - want[0]).max() <= LOGIT_ATOL and np.isfinite(head).all()
    forks = [session.fork_shared_weights() for _ in prompts]
    got = [None] * len(forks)

    def work(i):
        for _ in range(3):
            got[i] = forks[i].append(prompts[i], want=[70, len(prompts[i]) - 1], reset=True)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(forks))]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    for fork in forks:
        fork.destroy()
    session.destroy()
