"""Sessions on a device with little memory left: the block workspace takes shorter chunks instead of failing the create."""
import dataclasses

import numpy as np
import pytest

from nerva_b200 import ops, synth
from nerva_b200.session import CudaHfDecodeSequenceSession, SmokeStatus
from tests.test_gpu_sparse_prefill import MOE_SHARED

pytestmark = pytest.mark.gpu

DENSE = synth.DecoderConfig("tight", layers=1, hidden=4096, heads=32, kv_heads=8, head_dim=128, intermediate=12288, vocab=512)


@pytest.mark.parametrize("cfg", [DENSE, dataclasses.replace(MOE_SHARED, layers=1)], ids=["dense", "experts"])
def test_create_with_room_for_short_chunks_only(built_lib, cfg):
    import torch
    ck = synth.dense_checkpoint(cfg, fill=ops.synth_normal_bf16)
    prompt = synth.uniform_u32(5, synth.T_PROMPT, 700, cfg.vocab)

    def free():
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        return torch.cuda.mem_get_info()[0]

    def chunk_and_logits():
        s = CudaHfDecodeSequenceSession(ck, 4096)
        assert s.status == SmokeStatus.OK, s.error
        left, chunk = free(), int(s.create_result.prefill_chunk_tokens)
        got = s.append(prompt, want=[5, 255, 256, 699], reset=True)
        s.destroy()
        return chunk, got, left

    warm, want, _ = chunk_and_logits()
    before = free()
    full, _, after = chunk_and_logits()
    assert warm == full == 2048
    took = before - after
    spare = 120 << 20 if cfg is DENSE else 25 << 20  # of what the long chunks' workspace takes
    filler = torch.empty(free() - (took - spare), dtype=torch.uint8, device="cuda")
    chunk, got, _ = chunk_and_logits()
    del filler
    free()
    assert 256 <= chunk < 2048
    assert np.abs(got - want).max() <= 2e-2
