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
