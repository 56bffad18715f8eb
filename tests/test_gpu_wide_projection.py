"""The block projection of more than 256 tokens (pairs of SMs, gemm_wide.cu) through the per-operator C ABI, against a
64-bit product of the same bf16 operands."""
import numpy as np
import pytest

from nerva_b200 import ops, synth

pytestmark = pytest.mark.gpu

# fp32 sums of bf16 products in the MMA's own order: the bound of the other projection tests, whose operands
# (weights N(0, 0.02), activations N(0, 1)) and inner sizes are the same
PROJ_ATOL = 2e-3


@pytest.mark.parametrize("rows,cols,tokens", [
    (256, 64, 257),                      # one weight tile, one slice, the fewest tokens
    (37, 512, 288), (257, 192, 300),     # ragged rows: less than a block's half, one row into the next tile
    (768, 512, 511), (512, 1536, 513),   # one token on either side of two full tiles
    (6144, 4096, 640), (4096, 12288, 1500), (24576, 4096, 300),  # more tiles than pairs, several waves
    (1000, 1408, 2048), (130, 64, 2049),
    # 65 to 256 tokens of matrices with many rows, and one row tile fewer than that takes
    (24576, 4096, 65), (13825, 128, 100), (16384, 64, 256), (13824, 128, 100),
])
def test_wide_projection_matches_a_64_bit_product(built_lib, rows, cols, tokens):
    import torch
    w = ops.synth_normal_bf16(0, 77, rows * cols, 0.02)
    x = ops.synth_normal_bf16(0, synth.T_ACTIVATION, tokens * cols, 1.0)
    y, _ = ops.projection(w, x, rows, cols, tokens=tokens)

    def wide(bits, shape):
        return torch.from_numpy(bits.view(np.int16)).cuda().view(torch.bfloat16).view(shape).double()

    ref = (wide(x, (tokens, cols)) @ wide(w, (rows, cols)).T).cpu().numpy()
    assert np.isfinite(y).all()
    assert np.abs(y - ref).max() <= PROJ_ATOL
    again, _ = ops.projection(w, x, rows, cols, tokens=tokens)
    assert np.array_equal(y, again)
