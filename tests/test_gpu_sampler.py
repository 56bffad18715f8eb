"""GPU parity of the temperature / top-k / top-p sampler: the kernel against the reference's own
sampler kernel (compiled from the reference checkout into oracle/_ref, token for token), against
the CPU oracle, and inside the resident decode session."""
import numpy as np
import pytest

from nerva_b200 import ops, synth
from nerva_b200.session import (CudaHfDecodeSequenceLoop, CudaHfDecodeSequenceSession, SmokeStatus, sampler_config)

pytestmark = pytest.mark.gpu

# (temperature, top_p, top_k): arg-max, Gumbel-max, top-p only, top-k only, both, clamped top-k
CONFIGS = [(0.0, 1.0, 0), (0.7, 1.0, 1), (1.0, 1.0, 0), (0.7, 0.9, 0), (1.3, 1.0, 40), (0.8, 0.95, 50),
           (1.0, 0.3, 2), (2.0, 1.0, 128), (1.0, 0.999, 4000)]
NEAR_TIE = 1e-4  # oracle decisions closer than this (relative) may fall the other way on the device


def _logit_sets():
    rng = np.random.default_rng(17)
    out = {}
    out["vocab151936"] = (rng.standard_normal(151936) * 2.5).astype(np.float32)
    out["vocab32000_peaked"] = (rng.standard_normal(32000) * 6.0).astype(np.float32)
    ties = np.round(rng.standard_normal(5000) * 2.0).astype(np.float32)  # thousands of exact ties
    out["ties"] = ties
    small = rng.standard_normal(37).astype(np.float32)  # fewer candidates than the top-k ceiling
    out["vocab37"] = small
    holes = (rng.standard_normal(3000) * 3.0).astype(np.float32)
    bad = rng.choice(3000, 2950, replace=False)
    holes[bad[:1000]] = np.inf
    holes[bad[1000:2000]] = -np.inf
    holes[bad[2000:]] = np.nan  # 50 finite candidates left
    out["holes"] = holes
    out["nothing_finite"] = np.full(500, -np.inf, dtype=np.float32)
    out["negative"] = (-np.abs(rng.standard_normal(9000)) * 40.0 - 5.0).astype(np.float32)
    out["one"] = np.array([0.25], dtype=np.float32)
    return out


@pytest.mark.parametrize("name", list(_logit_sets()))
def test_kernel_matches_reference_kernel(built_lib, oracle_mod, name):
    if oracle_mod.ref_sampler_lib() is None:
        pytest.skip("the reference sampler was not compiled (no reference checkout at build time)")
    logits = _logit_sets()[name]
    checked = 0
    for temperature, top_p, top_k in CONFIGS:
        for position in (0, 1, 7, 4095):
            for seed in (0, 0x9E3779B97F4A7C15, 12345):
                want = oracle_mod.ref_sample_token(logits, position, temperature, top_p, top_k, seed)
                got = ops.sample_token(logits, position, temperature, top_p, top_k, seed)
                assert got == want, (name, temperature, top_p, top_k, position, seed)
                checked += 1
    assert checked == len(CONFIGS) * 12


@pytest.mark.parametrize("name", list(_logit_sets()))
def test_kernel_matches_oracle(built_lib, oracle_mod, name):
    logits = _logit_sets()[name]
    exact = total = 0
    for temperature, top_p, top_k in CONFIGS:
        for position in range(12):
            want, margin = oracle_mod.sample_token(logits, position, temperature, top_p, top_k, 777)
            got = ops.sample_token(logits, position, temperature, top_p, top_k, 777)
            total += 1
            exact += int(got == want)
            if margin > NEAR_TIE:
                assert got == want, (name, temperature, top_p, top_k, position, margin)
    assert exact >= 0.97 * total


def _arranged(kind, count):
    """The kernel's cluster takes index i in slice i % 8192 // 32 (of fewer than 8192 logits: i % 256); the bound of its list
    comes from the slices' maxima."""
    rng = np.random.default_rng(count)
    out = (rng.standard_normal(count) * 3.0).astype(np.float32)
    index = np.arange(count)
    few = np.isin(index % 8192 // 32 if count >= 8192 else index % 256, (3, 4, 250))
    if kind == "few slices":  # hold all of the largest: more keys reach the bound than the list takes
        out[few] += 40.0
    elif kind == "finite in few slices":  # fewer maxima than candidates: no bound
        out[~few] = np.nan
    elif kind == "ascending":
        out.sort()
    return out


@pytest.mark.parametrize("kind", ["random", "few slices", "finite in few slices", "ascending"])
@pytest.mark.parametrize("count", [2, 128, 255, 1024, 1025, 4064, 4065, 8191, 8192, 8193, 65537, 151936])
def test_candidates_at_the_edges_of_slices(built_lib, oracle_mod, kind, count):
    logits = _arranged(kind, count)
    for temperature, top_p, top_k in [(1.0, 1.0, 0), (0.9, 0.95, 0), (1.5, 1.0, 128), (0.7, 0.9, 50), (1.0, 0.5, 2)]:
        for position in range(4):
            want, margin = oracle_mod.sample_token(logits, position, temperature, top_p, top_k, 31)
            got = ops.sample_token(logits, position, temperature, top_p, top_k, 31)
            if margin > NEAR_TIE:
                assert got == want, (temperature, top_p, top_k, position, margin)


def test_rejects_bad_configurations(built_lib):
    logits = np.zeros(8, dtype=np.float32)
    for temperature, top_p in ((-1.0, 1.0), (np.nan, 1.0), (np.inf, 1.0), (1.0, 0.0), (1.0, 1.5), (1.0, np.nan)):
        with pytest.raises(RuntimeError):
            ops.sample_token(logits, 0, temperature, top_p, 0, 0)


@pytest.mark.parametrize("config", [(0.9, 0.95, 0), (1.0, 1.0, 0), (1.2, 1.0, 20)])
def test_session_samples_what_the_oracle_samples_from_its_logits(built_lib, oracle_mod, tiny_checkpoint, config):
    """Every sampled token of a resident session equals the oracle's draw from the logits the
    session itself produced at that position, and the next step consumes that token."""
    cfg = synth.TINY_QWEN3
    temperature, top_p, top_k = config
    prompt = synth.prompt_ids(cfg)[:9]
    s = CudaHfDecodeSequenceSession(tiny_checkpoint, 64)
    assert s.status == SmokeStatus.OK, s.error
    sampler = sampler_config(temperature, top_p, top_k, seed=4242)
    start, loop = CudaHfDecodeSequenceLoop.start(s, prompt, sampler=sampler)
    assert start.status == SmokeStatus.OK, start.error
    tokens = []
    for i in range(24):
        out = loop.advance(1)
        assert out.status == SmokeStatus.OK, out.error
        logits = s.read_logits()
        want, margin = oracle_mod.sample_token(logits, len(prompt) - 1 + i, temperature, top_p, top_k, 4242)
        if margin > NEAR_TIE:
            assert out.tokens[0] == want, (i, margin)
        tokens.append(out.tokens[0])
    assert len(set(tokens)) > 4  # not the arg-max cycle
    # the same request through run() reproduces the sequence (seeded), another seed does not
    again = s.run(prompt, 24, sampler=sampler)
    assert again.status == SmokeStatus.OK and again.tokens == tokens
    other = s.run(prompt, 24, sampler=sampler_config(temperature, top_p, top_k, seed=4243))
    assert other.status == SmokeStatus.OK and other.tokens != tokens
    # and the arg-max sampler still gives the arg-max sequence afterwards
    greedy = s.run(prompt, 8)
    assert greedy.status == SmokeStatus.OK
    fresh = CudaHfDecodeSequenceSession(tiny_checkpoint, 64)
    assert fresh.run(prompt, 8).tokens == greedy.tokens
    fresh.destroy()
    s.destroy()


def test_fork_continues_the_sampled_sequence(built_lib, tiny_checkpoint):
    cfg = synth.TINY_QWEN3
    prompt = synth.prompt_ids(cfg)[:5]
    s = CudaHfDecodeSequenceSession(tiny_checkpoint, 48)
    sampler = sampler_config(1.0, 0.9, 0, seed=9)
    start, loop = CudaHfDecodeSequenceLoop.start(s, prompt, sampler=sampler)
    assert start.status == SmokeStatus.OK, start.error
    head = loop.advance(6).tokens
    child = s.fork_shared_weights()
    assert child.status == SmokeStatus.OK, child.error
    tail_parent = loop.advance(10).tokens
    tail_child = CudaHfDecodeSequenceLoop(child).advance(10).tokens
    assert tail_child == tail_parent
    assert len(head) == 6 and len(tail_parent) == 10
    child.destroy()
    s.destroy()


def test_one_kernel_engine_refuses_sampling(built_lib, tiny_checkpoint):
    prompt = synth.prompt_ids(synth.TINY_QWEN3)[:4]
    try:
        s = CudaHfDecodeSequenceSession(tiny_checkpoint, 32, engine=1)
    except RuntimeError:
        pytest.skip("the one-kernel engine is unavailable for this shape")
    assert s.status == SmokeStatus.OK
    out = s.run(prompt, 4, sampler=sampler_config())
    assert out.status != SmokeStatus.OK and "engine 0" in out.error
    assert s.run(prompt, 4).status == SmokeStatus.OK  # arg-max still runs on it
    s.destroy()
