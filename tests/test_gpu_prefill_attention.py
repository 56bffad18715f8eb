"""Prefill attention on 128-row tiles (prefill_attention.cu): prompts and portions around its tile edges, against the
token-by-token prefill through the decode step.  (Windows, kept positions, caps and gates: the vuvolix and vamidra tests.)"""
import os

import numpy as np
import pytest

from nerva_b200 import ops, synth
from nerva_b200.session import CudaHfDecodeSequenceLoop, CudaHfDecodeSequenceSession, SmokeStatus

pytestmark = pytest.mark.gpu

LOGIT_ATOL = 2e-2  # the stated bound of logits at this width and depth: both paths round the same values to bf16

SHAPES = [(8, 2, 128), (6, 2, 64), (16, 1, 128), (4, 4, 64)]  # heads, KV heads, head size: 4, 3, 16 and 1 heads per KV head


def _checkpoint(heads, kv_heads, dim):
    cfg = synth.DecoderConfig("prefill", layers=2, hidden=512, heads=heads, kv_heads=kv_heads, head_dim=dim,
                              intermediate=768, vocab=2048)
    return cfg, synth.dense_checkpoint(cfg, fill=ops.synth_normal_bf16)


def _by_decode(ck, prompt, context):
    os.environ["NERVA_B200_PREFILL"] = "decode"
    try:
        s = CudaHfDecodeSequenceSession(ck, context)
        summary, _ = CudaHfDecodeSequenceLoop.start(s, prompt)
        assert summary.status == SmokeStatus.OK, summary.error
        return s.read_logits()
    finally:
        os.environ.pop("NERVA_B200_PREFILL", None)


@pytest.mark.parametrize("heads,kv_heads,dim", SHAPES)
def test_tile_prefill_matches_prefill_by_decode(built_lib, heads, kv_heads, dim):
    cfg, ck = _checkpoint(heads, kv_heads, dim)
    for tokens in (64, 127, 128, 129, 385):
        prompt = synth.uniform_u32(5, synth.T_PROMPT, tokens, cfg.vocab)
        want = _by_decode(ck, prompt, 512)
        s = CudaHfDecodeSequenceSession(ck, 512)
        s.set_kv_block_table(synth.permutation(3, synth.T_PAGE_TABLE, 32))
        got = s.append(prompt, want=[tokens - 1], reset=True)[0]
        assert np.abs(got - want).max() <= LOGIT_ATOL, tokens
        # the same tokens in two portions, the second on tiles that start in the middle of the cache
        if tokens == 385:
            s.append(prompt[:101], reset=True)
            again = s.append(prompt[101:], want=[tokens - 102])[0]
            assert np.abs(again - want).max() <= LOGIT_ATOL
        s.destroy()
