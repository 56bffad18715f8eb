"""A page table that is set while other work is queued on the default stream is the one that the next request uses."""
import numpy as np
import pytest

from nerva_b200 import ops, synth
from nerva_b200.session import CudaHfDecodeSequenceSession, SmokeStatus

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads", [(4, 2), (16, 1)])  # a prompt in blocks, token by token
def test_table_set_behind_a_busy_default_stream(built_lib, heads, kv_heads):
    import torch
    cfg = synth.DecoderConfig("table", layers=1, hidden=256, heads=heads, kv_heads=kv_heads, head_dim=128, intermediate=256, vocab=512)
    ck = synth.dense_checkpoint(cfg, fill=ops.synth_normal_bf16)
    prompt = synth.uniform_u32(5, synth.T_PROMPT, 96, cfg.vocab)
    got = []
    for busy in (False, True):
        s = CudaHfDecodeSequenceSession(ck, 128)
        assert s.status == SmokeStatus.OK, s.error
        if busy:
            torch.cuda._sleep(400_000_000)  # cycles: a fifth of a second, and the copy of a table is small enough to be queued
        s.set_kv_block_table(synth.permutation(3, synth.T_PAGE_TABLE, 8))
        s.append(prompt[:48], reset=True)
        torch.cuda.synchronize()
        got.append(s.append(prompt[48:], want=[0, 47]))
        s.destroy()
    assert np.array_equal(got[0], got[1])
