"""A cached value that is not finite spoils the positions that attend to it and no others: prompts in blocks with one token
whose value overflows, beside the same prompt with an ordinary token there.

Ordinary embeddings are zero in the first channel (the first two, behind a norm that takes the mean away), the token BAD is
nothing else; one value feature per KV head reads that channel with a weight near the largest bf16 number, so it is zero for
all tokens but BAD, and infinite for BAD."""
import dataclasses

import numpy as np
import pytest

from nerva_b200 import ops, synth
from nerva_b200.session import CudaHfDecodeSequenceSession, SmokeStatus
from tests import vamidra_models as M
from tests.test_gpu_sparse_prefill import LATENT, LATENT_256, MOE

pytestmark = pytest.mark.gpu

AT = 150  # the position; BAD and GOOD are the tokens there, in no other place
BAD, GOOD = 7, 8
HUGE = 3e38
HUGE_BITS = int(synth.f32_to_bf16(np.array([HUGE], np.float32))[0])
ONE = int(synth.f32_to_bf16(np.array([1.0], np.float32))[0])


def _dense(name, **fields):
    return dataclasses.replace(synth.DecoderConfig(name, layers=2, hidden=512, heads=8, kv_heads=2, head_dim=128, intermediate=768,
                                                   vocab=2048), **fields)


DECODERS = {
    "128 wide": _dense("a"), "64 wide": _dense("b", head_dim=64), "a head per KV head": _dense("c", heads=4, kv_heads=4),
    "experts": MOE, "latent 128": LATENT, "latent 256": LATENT_256,
    "latent 512": dataclasses.replace(LATENT, layers=2, heads=16, kv_heads=16, kv_lora_rank=512, qk_nope_head_dim=128, qk_rope_head_dim=64),
}


def _overflowing(cfg):
    ck = synth.dense_checkpoint(cfg, fill=ops.synth_normal_bf16)
    embed = ck.embeddings.reshape(cfg.vocab, cfg.hidden)
    embed[:, 0] = 0
    embed[BAD] = 0
    embed[BAD, 0] = ONE
    layer = ck.layers[0]
    if cfg.kv_lora_rank:
        latent = layer["w_kv_a"].reshape(-1, cfg.hidden)
        latent[3] = 0
        latent[3, 0] = ONE
        layer["kv_a_norm"][3] = HUGE_BITS
    else:
        value = layer["w_v"].reshape(cfg.kv_heads, cfg.head_dim, cfg.hidden)
        value[:, 3] = 0
        value[:, 3, 0] = HUGE_BITS
    return ck


def _logits(session, vocab, count, first, token):
    """Logits of all positions, the first `first` of them in a portion of their own."""
    prompt = synth.uniform_u32(5, synth.T_PROMPT, count, vocab)
    prompt[(prompt == BAD) | (prompt == GOOD)] = 9
    prompt[AT] = token
    head = session.append(prompt[:first], range(first), reset=True) if first else np.zeros((0, vocab), np.float32)
    return np.concatenate([head, session.append(prompt[first:], range(count - first), reset=first == 0)])


def _check(session, vocab, count, first, sees):
    want, got = (_logits(session, vocab, count, first, token) for token in (GOOD, BAD))
    assert np.isfinite(want).all()
    same = np.array([np.array_equal(a, b) for a, b in zip(got, want)])
    assert (same == ~sees).all(), np.flatnonzero(same == sees)


@pytest.mark.parametrize("first", [0, 70, 131])
@pytest.mark.parametrize("name", sorted(DECODERS))
def test_earlier_positions_stay(built_lib, name, first):
    cfg = DECODERS[name]
    s = CudaHfDecodeSequenceSession(_overflowing(cfg), 256)
    assert s.status == SmokeStatus.OK, s.error
    _check(s, cfg.vocab, 203, first, np.arange(203) >= AT)
    s.destroy()


@pytest.mark.parametrize("window,keep", [(1000, 0), (20, 0), (37, 160), (130, 3)])
@pytest.mark.parametrize("dim", [64, 128])
def test_positions_that_the_window_has_left_stay(built_lib, dim, window, keep):
    """One layer: a position is spoiled if it sees AT, and otherwise as if an ordinary token stood there."""
    cfg = M.config([M.attention(ff=0, heads=4, kv_heads=2, dim=dim, vdim=dim, window=window, keep=keep, cap=0.0)], width=128)
    w = M.weights(cfg)
    w["embed"][:, :2] = 0.0
    w["embed"][BAD] = 0.0
    w["embed"][BAD, 0] = 1.0
    w["l0.norm1"][:2] = 1.0
    value = w["l0.mix.v"].reshape(2, dim, 128)
    value[:, 3] = 0.0
    value[:, 3, :2] = M.round_bf16(np.array([HUGE / 3, -HUGE / 3], np.float32))  # times (1 - mean) / deviation > 11
    s = CudaHfDecodeSequenceSession(M.checkpoint(cfg, w), 320, compute="bfloat16")
    assert s.status == SmokeStatus.OK, s.error
    at = np.arange(310)
    for first in (0, 90):
        _check(s, cfg["vocab"], 310, first, (at >= AT) & ((at - AT < window) | (AT < keep)))
    s.destroy()
