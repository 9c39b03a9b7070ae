"""The talker whose stacks exceed the L2 and that runs as a chain of kernels: what test_talker_gpu.py asks of the persistent
kernel's models, asked of it."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def chain_config(**generation):
    """The `mid` talker with 188 MB of stack weights."""
    from pega_omni_b200.config import presets
    base = presets["mid"]()
    cfg = dataclasses.replace(base, talker=dataclasses.replace(base.talker, hidden_size=1024, intermediate_size=3072,
                                                               num_hidden_layers=6, num_attention_heads=16,
                                                               num_key_value_heads=8, head_dim=128))
    return cfg.with_generation(**generation)


def make(cfg=None, seed=3, max_batch=16, std=0.02, **kw):
    from pega_omni_b200.model import Limits, Model
    from pega_omni_b200.synthetic import random_checkpoint
    cfg = cfg or chain_config()
    ck = random_checkpoint(cfg, seed=seed, std=std, device="cuda")
    return cfg, ck, Model.load(0, ck, cfg, Limits(max_batch=max_batch, max_tokens=2048, kv_gib=0.5), **kw)


def prompts_for(cfg, lens, seed=0):
    from pega_omni_b200.model import Prompt
    rng = np.random.default_rng(seed)
    return [Prompt(rng.integers(0, cfg.text_vocab_size, n).tolist(), np.where(rng.random(n) < 0.3, rng.integers(0, 64, n), -1).tolist()) for n in lens]


def draws_for(rng, n):
    from pega_omni_b200.model import Draw
    return [Draw(u) for u in rng.random((n, 16)).tolist()]


def test_trace_writes_a_line_per_kernel(built_lib, tmp_path):
    cfg, _, m = make()
    rng, path = np.random.default_rng(1), tmp_path / "trace.txt"
    seqs = [m.open(9, 32) for _ in range(3)]
    m.start(list(zip(seqs, prompts_for(cfg, [9] * 3), draws_for(rng, 3))))
    plain, ms = m.run_ticks(seqs, [draws_for(rng, 3) for _ in range(2)])
    assert not path.exists()
    m.trace(path)
    m.run_ticks(seqs, [draws_for(rng, 3) for _ in range(4)])
    kernels = m.stats().last_call_launches // 4
    lines = [x.split() for x in path.read_text().splitlines()]
    assert lines[0][:2] == ["kernel", "what"] and len(lines) == kernels + 1
    names = {x[1] for x in lines[1:]}
    assert {"rope_attend", "gemm", "norm_gemm", "norm_gemm_swiglu", "launch_sample_next"} <= names
    dur, end = [int(x[5]) for x in lines[1:]], [int(x[6]) for x in lines[1:]]
    assert min(dur) >= 0 and end == list(np.cumsum(dur)) and 0.5 * min(ms) < end[-1] * 1e-6 < 10 * max(ms)
    path.unlink()
    m.trace(None)
    m.run_ticks(seqs, [draws_for(rng, 3) for _ in range(2)])
    assert not path.exists() and m.stats().last_call_launches // 2 == kernels
    m.close()


def test_predictor_wider_than_a_draw_holds(built_lib):
    """A predictor of 4,352 channels: its rows do not come out of the draw, and its logits are those of the per-op kernels."""
    from pega_omni_b200.model import Draw
    base = chain_config()
    cfg = dataclasses.replace(base, predictor=dataclasses.replace(base.predictor, hidden_size=4352, num_hidden_layers=1))
    rng = np.random.default_rng(2)
    forced = rng.integers(0, 64, (3, 3, 16)).astype(np.int32)
    forced[:, :, cfg.num_code_groups:] = 0
    got = []
    for tick_kernel in (True, False):
        _, _, m = make(cfg, max_batch=4, std=0.01, tick_kernel=tick_kernel)
        seqs, prompts, rows = [m.open(7, 8) for _ in range(3)], prompts_for(cfg, [7] * 3), []
        for t in range(3):
            draws = [Draw([0.5] * 16, list(forced[t, s])) for s in range(3)]
            out = m.start(list(zip(seqs, prompts, draws))) if t == 0 else m.step(list(zip(seqs, draws)))
            assert (out.codes == forced[t]).all()
            rows.append(np.stack([np.concatenate([m.talker_logits(s), m.predictor_logits(s).ravel()]) for s in range(3)]))
        got.append(np.stack(rows))
        m.close()
    a, b = got
    step = np.exp2(np.floor(np.log2(np.maximum(np.abs(b), 2.0))) - 7)
    assert float((np.abs(a - b) / step).max()) <= 2.0


# ---- the persistent kernel's tests, on this model in the place of `tiny128` ------------------------------------------

@pytest.fixture
def as_tiny(monkeypatch):
    from pega_omni_b200.config import presets
    monkeypatch.setitem(presets, "tiny128", chain_config)
    import test_talker_gpu as same
    return same


def test_runs_as_a_chain(built_lib):
    cfg, _, m = make()
    rng, seqs = np.random.default_rng(0), [m.open(9, 4)]
    m.start(list(zip(seqs, prompts_for(cfg, [9]), draws_for(rng, 1))))
    m.step(list(zip(seqs, draws_for(rng, 1))))
    assert m.stats().last_call_launches > 100
    m.close()


def test_teacher_forced_logits_match_oracle(built_lib, oracle_lib):
    """Both sides store logits as bf16: at most two of its steps apart (one logit of mid's width, summed over 3,072 channels in
    another order, lands 1.5 steps away across a binade), cosine 0.9999."""
    from pega_omni_b200.model import Draw
    cfg, ck, m = make()
    o = oracle_lib.CpuOracle(cfg, ck)
    lens, frames = [9, 33, 17], 6
    prompts = prompts_for(cfg, lens, seed=1)
    forced = np.random.default_rng(5).integers(0, 2048, (frames, 3, 16)).astype(np.int32)
    seqs, sids = [m.open(n, 8) for n in lens], [o.open(n, 8) for n in lens]
    for t in range(frames):
        draws = [Draw([0.5] * 16, list(forced[t, s])) for s in range(3)]
        if t == 0:
            m.start(list(zip(seqs, prompts, draws)))
            o.start(sids, prompts, draws)
        else:
            m.step(list(zip(seqs, draws)))
            o.step(sids, draws)
        for s in range(3):
            for a, b in [(m.talker_logits(s), o.talker_logits(s))] + list(zip(m.predictor_logits(s), o.predictor_logits(s))):
                step = np.exp2(np.floor(np.log2(np.maximum(np.abs(b), 2.0))) - 7)
                assert float((np.abs(a - b) / step).max()) <= 2.0, (t, s)
                assert float(a @ b / (np.linalg.norm(a) * np.linalg.norm(b))) >= 0.9999, (t, s)
    m.close()


def test_greedy_agreement_over_512_frames(as_tiny, built_lib, oracle_lib):
    as_tiny.test_greedy_agreement_over_512_frames(built_lib, oracle_lib)


def test_in_loop_sampler_is_exact_on_its_own_logits(as_tiny, built_lib, oracle_lib):
    as_tiny.test_in_loop_sampler_is_exact_on_its_own_logits(built_lib, oracle_lib)


def test_lockstep_streams_bit_identical_and_late_joiner_agrees(as_tiny, built_lib):
    as_tiny.test_lockstep_streams_bit_identical_and_late_joiner_agrees(built_lib)


def test_run_ticks_equals_steps(as_tiny, built_lib):
    as_tiny.test_run_ticks_equals_steps(built_lib)


def test_philox_mode_matches_oracle_stream(as_tiny, built_lib, oracle_lib):
    as_tiny.test_philox_mode_matches_oracle_stream(built_lib, oracle_lib)


def forced_logits(m, n, frames, forced):
    from pega_omni_b200.model import Draw
    cfg_prompts = prompts_for(m.config, [4 + s % 5 for s in range(n)])
    seqs, rows = [m.open(len(p), frames + 1) for p in cfg_prompts], []
    for t in range(frames):
        draws = [Draw([0.5] * 16, list(forced[t, s])) for s in range(n)]
        out = m.start(list(zip(seqs, cfg_prompts, draws))) if t == 0 else m.step(list(zip(seqs, draws)))
        assert (out.codes == forced[t]).all()
        rows.append(np.stack([np.concatenate([m.talker_logits(s), m.predictor_logits(s).ravel()]) for s in range(0, n, 13)]))
    return np.stack(rows)


def test_free_draws_give_the_rows_of_forced_ones(built_lib):
    """The codes a free call drew, forced upon another model: the same logits, so the draw left the rows of its own codes."""
    from pega_omni_b200.model import Draw
    cfg, _, m = make()
    rng, n = np.random.default_rng(4), 5
    prompts = prompts_for(cfg, [8 + s for s in range(n)])
    seqs, frames = [m.open(len(p), 8) for p in prompts], []
    for t in range(5):
        draws = draws_for(rng, n)
        out = m.start(list(zip(seqs, prompts, draws))) if t == 0 else m.step(list(zip(seqs, draws)))
        frames.append((out.codes.copy(), [np.concatenate([m.talker_logits(s), m.predictor_logits(s).ravel()]) for s in range(n)]))
    m.close()
    _, _, m = make(tick_kernel=False)
    seqs = [m.open(len(p), 8) for p in prompts]
    for t, (codes, logits) in enumerate(frames):
        draws = [Draw([0.5] * 16, codes[s].tolist()) for s in range(n)]
        m.start(list(zip(seqs, prompts, draws))) if t == 0 else m.step(list(zip(seqs, draws)))
        for s in range(n):
            b = np.concatenate([m.talker_logits(s), m.predictor_logits(s).ravel()])
            step = np.exp2(np.floor(np.log2(np.maximum(np.abs(b), 2.0))) - 7)
            assert float((np.abs(logits[s] - b) / step).max()) <= 2.0, (t, s)
    m.close()


def test_more_than_128_sessions_agree_with_per_op_kernels(built_lib):
    """A bucket of 256: the predictor's first pass has 512 rows, and its rows no longer come out of the draw."""
    n, frames, got = 140, 3, []
    forced = np.random.default_rng(6).integers(0, 2048, (frames, n, 16)).astype(np.int32)
    for tick_kernel in (True, False):
        cfg, _, m = make(max_batch=n, tick_kernel=tick_kernel)
        hi = min(cfg.talker.vocab_size - cfg.control_tokens, cfg.predictor.vocab_size)
        got.append(forced_logits(m, n, frames, forced % hi))
        m.close()
    step = np.exp2(np.floor(np.log2(np.maximum(np.abs(got[1]), 2.0))) - 7)
    assert float((np.abs(got[0] - got[1]) / step).max()) <= 2.0
