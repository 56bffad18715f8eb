"""The epilogues of the block projections (gate/up pairs, residuals added in place, both at once) at the edges of their
groups of 16 tokens and 32 rows, on the split kernel and on pairs of SMs."""
import numpy as np
import pytest

from nerva_b200 import ops, synth

pytestmark = pytest.mark.gpu


def _picked(rng, rows, cols):
    """A matrix whose row r is 1 at one column and 0 elsewhere: every sum is one value of x, exact in any order."""
    w = np.zeros((rows, cols), np.float32)
    w[np.arange(rows), rng.integers(0, cols, rows)] = 1.0
    return w


# (rows, stored rows, tokens): on the split kernel (up to 64 tokens, and up to 256 of few rows) and on pairs of SMs
SHAPES = [(64, 0, 2), (130, 0, 17), (1000, 0, 33), (1536, 0, 65), (2048, 0, 255),
          (96, 32, 3), (1090, 64, 63), (1154, 1120, 129), (33, 33, 15), (1001, 1001, 241), (97, 97, 31),
          (14336, 0, 100), (14400, 64, 67), (14337, 14337, 113), (2048, 0, 257), (1090, 64, 289), (1001, 1001, 2049)]


@pytest.mark.parametrize("rows,stored,tokens", SHAPES)
@pytest.mark.parametrize("activation", [0, 1])
def test_epilogues_are_those_of_fp32(built_lib, rows, stored, tokens, activation):
    """Gates from -1e20 to 1e20 and infinite ones too: the activation is v / (1 + exp(-u)) in fp32, its quotient rounded to nearest.
    Sums are exact, so a residual's sum is one fp32 addition; a gated value is compared by bits with torch's fp32 functions."""
    import torch
    cols, rng = 128, np.random.default_rng(rows + tokens)
    w = _picked(rng, rows, cols)
    x = rng.standard_normal((tokens, cols)) * np.exp2(rng.integers(-6, 8, (tokens, cols)))
    special = [-90.0, -88.5, -104.0, -1e20, 1e20, 90.0, 0.0, -0.0, 1e-30, -1e-30, -17.0, 3e38]
    x[np.arange(tokens), rng.integers(0, cols, tokens)] = np.resize(special, tokens)
    if tokens > 4:
        x[1, 5], x[3, 7] = np.inf, -np.inf  # other columns of these tokens: 0 * inf
    xb = synth.f32_to_bf16(x.astype(np.float32))
    residual = rng.standard_normal((tokens, stored)).astype(np.float32)
    out, gated = ops.block_projection(synth.f32_to_bf16(w), xb, rows, cols, tokens, residual, activation)
    xv = torch.from_numpy(synth.bf16_to_f32(xb).reshape(tokens, cols)).cuda()
    y = (xv.double() @ torch.from_numpy(w).cuda().double().T).float()
    want = (y[:, :stored] + torch.from_numpy(residual).cuda()).cpu().numpy()
    assert np.array_equal(out, want, equal_nan=True)
    gate, up = y[:, stored::2], y[:, stored + 1::2]
    u = 1.5957691216057308 * torch.addcmul(gate, 0.044715 * gate * gate, gate) if activation == 1 else gate
    act = gate / (1.0 + torch.exp(-u)) * up
    got = torch.from_numpy(gated.view(np.int16)).cuda().view(torch.bfloat16)
    number = ~torch.isnan(act)  # (the codec of the stores, like the reference's, does not keep every NaN one)
    if activation == 0:
        assert torch.equal(got[number], act.to(torch.bfloat16)[number])
    else:  # the cubic's fused multiply-add rounds once where torch's may round twice: a unit of bf16 at most
        a, b = got[number].float(), act.to(torch.bfloat16)[number].float()
        assert (((a - b).abs() <= b.abs() * 2.0 ** -7 + 1e-37) | (a == b)).all()
