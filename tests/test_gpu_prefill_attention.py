"""Prefill attention on 128-row tiles (prefill_attention.cu): prompts and portions around its tile edges, against the
token-by-token prefill through the decode step.  (Windows, kept positions, caps and gates: the vuvolix and vamidra tests.)"""
import os

import numpy as np
import pytest

from nerva_b200 import ops, synth
from nerva_b200.session import CudaHfDecodeSequenceLoop, CudaHfDecodeSequenceSession, SmokeStatus

pytestmark = pytest.mark.gpu

LOGIT_ATOL = 2e-2  # the stated bound of logits at this width and depth: both paths round the same values to bf16

# heads, KV heads, head size: 4, 3, 8 and 1 heads per KV head (more than 8 keep a decoder off blocks)
SHAPES = [(8, 2, 128), (6, 2, 64), (16, 2, 128), (4, 4, 64)]


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
        assert s.create_result.prefill_chunk_tokens > 1  # the prompt goes in blocks
        s.set_kv_block_table(synth.permutation(3, synth.T_PAGE_TABLE, 32))
        got = s.append(prompt, want=[tokens - 1], reset=True)[0]
        assert np.abs(got - want).max() <= LOGIT_ATOL, tokens
        # the same tokens in two portions, the second on tiles that start in the middle of the cache
        if tokens == 385:
            s.append(prompt[:101], reset=True)
            again = s.append(prompt[101:], want=[tokens - 102])[0]
            assert np.abs(again - want).max() <= LOGIT_ATOL
        s.destroy()


@pytest.mark.parametrize("heads,dim,mixer", [(16, 64, {}), (12, 128, {}), (24, 64, {"window": 90, "keep": 5, "cap": 6.0})])
def test_many_query_heads_of_one_key_head(built_lib, heads, dim, mixer):
    """More than 8 heads per KV head reach the tiles through the models described layer by layer."""
    from tests import vamidra_models as M
    from tests import vamidra_oracle as O
    shape = {"window": 1000, "keep": 0, "cap": 0.0, **mixer}
    cfg = M.config([M.attention(ff=0, heads=heads, kv_heads=1, dim=dim, vdim=dim, **shape)], width=128)
    w = M.weights(cfg)
    tokens = M.tokens(cfg, 200)
    s = CudaHfDecodeSequenceSession(M.checkpoint(cfg, w), 208, compute="bfloat16")
    got = s.append(tokens, range(200), reset=True)
    assert M.worst_position(got, O.forward(cfg, w, tokens)) < 2 * M.TOLERANCE["bfloat16"]
    s.destroy()


@pytest.mark.parametrize("first,sizes", [(0, (64, 79, 80, 81, 96)), (120, (64, 65, 75, 76)), (420, (16, 39, 40, 41))])
def test_rows_around_where_tiles_begin(built_lib, first, sizes):
    """Portions of fewer rows go row by row, the more keys there are the fewer: 80 of a new prompt, 40 behind 400 keys."""
    from tests import vamidra_models as M
    from tests import vamidra_oracle as O
    cfg, ck = _checkpoint(8, 2, 128)
    windowed = M.config([M.attention(ff=0, dim=64, vdim=64, window=450, keep=3, cap=0.0), M.attention(ff=0, dim=128, vdim=128, window=300)],
                        width=128)
    w = M.weights(windowed)
    dense = CudaHfDecodeSequenceSession(ck, 512)
    layers = CudaHfDecodeSequenceSession(M.checkpoint(windowed, w), 512, compute="bfloat16")
    longest = first + max(sizes)
    prompt, tokens = synth.uniform_u32(5, synth.T_PROMPT, longest, cfg.vocab), M.tokens(windowed, longest)
    oracle = O.forward(windowed, w, tokens)
    for rows in sizes:
        want = _by_decode(ck, prompt[:first + rows], 512)
        if first:
            dense.append(prompt[:first], reset=True)
            layers.append(tokens[:first], reset=True)
        got = dense.append(prompt[first:first + rows], want=[rows - 1], reset=first == 0)[0]
        assert np.abs(got - want).max() <= LOGIT_ATOL, rows
        got = layers.append(tokens[first:first + rows], range(rows), reset=first == 0)
        assert M.worst_position(got, oracle[first:first + rows]) < 2 * M.TOLERANCE["bfloat16"], rows
    dense.destroy()
    layers.destroy()
