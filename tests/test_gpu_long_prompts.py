"""Prompts of more positions than one block carries (2048): what one block leaves for the next (cached rows, recurrent state,
the place of wanted logits, the latent attention's first position).  A prompt in one call is cut into blocks of equal size,
a multiple of 16; given as portions of exactly those sizes it takes the same launches and has to give the same bits."""
import os

import numpy as np
import pytest

from nerva_b200 import ops, synth
from nerva_b200.session import CudaHfDecodeSequenceLoop, CudaHfDecodeSequenceSession, SmokeStatus
from tests import vamidra_models as M
from tests import vamidra_oracle as O
from tests.test_gpu_sparse_prefill import LATENT, MOE

pytestmark = pytest.mark.gpu

CONTEXT = 4128
DENSE = synth.DecoderConfig("long", layers=2, hidden=256, heads=4, kv_heads=2, head_dim=64, intermediate=512, vocab=1024)
LOGIT_ATOL = 2e-2  # the bound of the other prefill tests


def _cuts(count):
    blocks = -(-count // 2048)
    size = -(-count // blocks) + 15 & ~15
    return [min(size, count - at) for at in range(0, count, size)]


def _places(count):
    edges = np.cumsum(_cuts(count))
    near = {int(e) + d for e in edges for d in (-17, -2, -1, 0, 1, 18)}
    return sorted({0, 40, count - 1} | {p for p in near if p < count})


@pytest.fixture(scope="module")
def models(built_lib):
    cfg = M.config([M.space(ff=0, heads=4, groups=2, state=32, norm_groups=2), M.attention(window=500, keep=4, dim=64, vdim=64)])
    return {"dense": synth.dense_checkpoint(DENSE, fill=ops.synth_normal_bf16),
            "experts": synth.dense_checkpoint(MOE, fill=ops.synth_normal_bf16),
            "latent": synth.dense_checkpoint(LATENT, fill=ops.synth_normal_bf16),
            "state space": M.checkpoint(cfg, M.weights(cfg))}


def _open(checkpoint, **kw):
    s = CudaHfDecodeSequenceSession(checkpoint, CONTEXT, **kw)
    assert s.status == SmokeStatus.OK, s.error
    assert s.create_result.prefill_chunk_tokens == 2048
    return s


def test_the_cuts_are_those_of_the_library():
    assert _cuts(2047) == [2047] and _cuts(2048) == [2048]
    assert _cuts(2049) == [1040, 1009] and _cuts(4100) == [1376, 1376, 1348]


@pytest.mark.parametrize("count", [2047, 2048, 2049, 4100])
@pytest.mark.parametrize("name", ["dense", "experts", "latent", "state space"])
def test_blocks_of_a_prompt_are_portions(models, name, count):
    ck = models[name]
    vocab = ck.config.vocab
    tokens = synth.uniform_u32(5, synth.T_PROMPT, count, vocab)
    s = _open(ck)
    places = _places(count)
    whole = s.append(tokens, want=places, reset=True)
    last = s.read_logits()
    at, parts = 0, []
    for n in _cuts(count):
        here = [p - at for p in places if at <= p < at + n]
        parts.append(s.append(tokens[at:at + n], want=here, reset=at == 0))
        at += n
    assert np.isfinite(whole).all()
    assert np.array_equal(np.concatenate(parts), whole)
    assert np.array_equal(whole[-1], last) or np.abs(whole[-1] - last).max() <= LOGIT_ATOL  # block head, step head
    # what the prompt left behind carries on as it does behind the portions
    more = synth.uniform_u32(6, synth.T_PROMPT, 20, vocab)
    again = s.append(more, want=[0, 19])
    s.append(tokens, reset=True)
    assert np.array_equal(s.append(more, want=[0, 19]), again)
    s.destroy()


@pytest.mark.parametrize("name", ["dense", "latent"])
def test_long_prompts_match_the_prefill_by_decode(models, name):
    ck = models[name]
    tokens = synth.uniform_u32(7, synth.T_PROMPT, 2300, ck.config.vocab)
    block, serial = _open(ck), _open(ck)
    CudaHfDecodeSequenceLoop.start(block, tokens)
    os.environ["NERVA_B200_PREFILL"] = "decode"
    try:
        CudaHfDecodeSequenceLoop.start(serial, tokens)
    finally:
        os.environ.pop("NERVA_B200_PREFILL", None)
    assert np.abs(block.read_logits() - serial.read_logits()).max() <= LOGIT_ATOL
    block.destroy()
    serial.destroy()


def test_a_long_prompt_of_a_state_space_model_follows_the_oracle(built_lib):
    cfg = M.config([M.space(ff=0, heads=2, vdim=16, groups=1, state=16, norm_groups=1), M.attention(ff=0, window=100, keep=2)], width=64)
    w = M.weights(cfg)
    tokens = M.tokens(cfg, 2200)
    s = CudaHfDecodeSequenceSession(M.checkpoint(cfg, w), 2208, compute="bfloat16")
    places = _places(2200)
    got = s.append(tokens, places, reset=True)
    assert M.worst_position(got, O.forward(cfg, w, tokens)[places]) < 2 * M.TOLERANCE["bfloat16"]
    s.destroy()


def test_fused_row_attention_of_more_rows_than_have_partials(models):
    """NERVA_B200_ROW_ATTENTION=fused: 600 rows go in parts of 256 that share the split attention's partials."""
    ck = models["dense"]
    tokens = synth.uniform_u32(8, synth.T_PROMPT, 600, ck.config.vocab)
    places = [0, 255, 256, 257, 511, 512, 599]
    tiles = _open(ck)
    want = tiles.append(tokens, want=places, reset=True)
    os.environ["NERVA_B200_ROW_ATTENTION"] = "fused"
    try:
        rows = _open(ck)
    finally:
        os.environ.pop("NERVA_B200_ROW_ATTENTION", None)
    got = rows.append(tokens, want=places, reset=True)
    assert np.abs(got - want).max() <= LOGIT_ATOL
    assert np.array_equal(got, rows.append(tokens, want=places, reset=True))
    tiles.destroy()
    rows.destroy()
