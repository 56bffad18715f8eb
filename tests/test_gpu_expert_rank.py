"""A rank of an expert-parallel step on one GPU: which of the chosen experts it computes, and what it pushes into the ranks'
receive buffers, against the same sums in 64 bits.  No rank waits for another here."""
import numpy as np
import pytest

from nerva_b200 import ops, synth

pytestmark = pytest.mark.gpu


def _weights(seed, shape, std, mean=0.0):
    w = synth.f32_to_bf16((np.random.default_rng(seed).standard_normal(shape) * std + mean).astype(np.float32)).reshape(shape)
    return w, synth.bf16_to_f32(w).astype(np.float64).reshape(shape)


def _silu(x):
    return x / (1.0 + np.exp(-x))


# experts, top_k, hidden, intermediate, shared intermediate (of all ranks), ranks
@pytest.mark.parametrize("experts,top_k,hidden,inter,shared,world", [
    (8, 3, 512, 128, 0, 1), (8, 3, 512, 128, 256, 2), (16, 1, 320, 136, 0, 4),  # three of the four ranks hold none of one
    (12, 5, 1032, 72, 96, 2), (16, 12, 512, 5120, 512, 2),                     # a partial piece; several passes
    (64, 6, 2048, 1408, 2816, 8),
])
@pytest.mark.parametrize("norm_topk", [False, True])
def test_ranks_add_up_to_the_whole_layer(built_lib, experts, top_k, hidden, inter, shared, world, norm_topk):
    rng = np.random.default_rng(hidden + top_k)
    h = rng.standard_normal(hidden).astype(np.float32)
    norm, norm_v = _weights(1, hidden, 0.1, 1.0)
    router, router_v = _weights(2, (experts, hidden), 2.0 * hidden ** -0.5)
    gate_up, gate_up_v = _weights(3, (experts, 2, inter, hidden), hidden ** -0.5)
    down, down_v = _weights(4, (experts, hidden, inter), inter ** -0.5)
    sh = [_weights(5 + i, s, hidden ** -0.5) for i, s in enumerate([(shared, hidden), (shared, hidden), (hidden, shared)])]
    x = h.astype(np.float64) / np.sqrt(np.mean(h.astype(np.float64) ** 2) + 1e-6) * norm_v
    p = np.exp(router_v @ x - (router_v @ x).max())
    p /= p.sum()
    chosen = np.argsort(-p, kind="stable")[:top_k]
    weight = p[chosen] / (p[chosen].sum() if norm_topk else 1.0)
    held, part = experts // world, shared // world
    empty = 0
    for rank in range(world):
        want = np.zeros(hidden)
        for e, w in zip(chosen, weight):
            if rank * held <= e < (rank + 1) * held:
                want += w * (down_v[e] @ (_silu(gate_up_v[e, 0] @ x) * (gate_up_v[e, 1] @ x)))
        empty += not want.any()
        own = slice(rank * part, (rank + 1) * part)
        if shared:
            want += sh[2][1][:, own] @ (_silu(sh[0][1][own] @ x) * (sh[1][1][own] @ x))
        mine = slice(rank * held, (rank + 1) * held)
        got = ops.sparse_mlp_rank(h, norm, router, gate_up[mine], down[mine],
                                  (sh[0][0][own], sh[1][0][own], sh[2][0][:, own]) if shared else None,
                                  top_k=top_k, norm_topk=norm_topk, expert_base=rank * held, rank=rank, world=world)
        # two projections behind each other in fp32: sums of n <= 5120 random terms, each with a relative rounding error of
        # 2^-24 per addition along a chain of n / 256 (a lane's), so below 1e-5 of the output's size
        assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
    if top_k == 1:
        assert empty == world - 1
