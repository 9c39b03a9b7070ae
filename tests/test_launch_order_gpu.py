"""Kernels launched early (programmatic dependent launch) give what the same kernels give one after the other, bit for bit:
every model's calls as a replayed graph here against a process in which each launch is waited for."""
import dataclasses
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]


def chain_config():
    """The `mid` talker with stacks beyond the 126 MB of L2, which run as a chain of kernels."""
    from pega_omni_b200.config import presets
    base = presets["mid"]()
    return dataclasses.replace(base, talker=dataclasses.replace(base.talker, hidden_size=1024, intermediate_size=3072,
                                                                num_hidden_layers=6, num_attention_heads=16,
                                                                num_key_value_heads=8, head_dim=128))


def talker(n, graphs):
    from pega_omni_b200.model import Draw, Limits, Model, Prompt
    from pega_omni_b200.synthetic import random_checkpoint
    cfg = chain_config()
    m = Model.load(0, random_checkpoint(cfg, seed=5, device="cuda"), cfg, Limits(max_batch=max(n, 8), max_tokens=2048, kv_gib=0.5), use_graphs=graphs)
    rng = np.random.default_rng(n)
    prompts = [Prompt(rng.integers(0, cfg.text_vocab_size, 5 + (37 * s) % 61).tolist(), [-1] * (5 + (37 * s) % 61)) for s in range(n)]
    seqs, out = [m.open(len(p), 24) for p in prompts], []
    for t in range(20):
        draws = [Draw(rng.random(16).tolist()) for _ in range(n)]
        got = m.start(list(zip(seqs, prompts, draws))) if t == 0 else m.step(list(zip(seqs, draws)))
        out += [got.codes.astype(np.float32).ravel()] + [np.concatenate([m.talker_logits(s), m.predictor_logits(s).ravel()]) for s in range(0, n, 7)]
    m.close()
    return out


def duplex(n, graphs):
    from pega_omni_b200.duplex import PRESETS, Model, Prompt, Step, random_checkpoint
    c = PRESETS["duplex-mid"]
    m = Model.load(0, random_checkpoint(c, seed=6), c, max_sessions=max(n, 4), max_prefill=2048, use_graphs=graphs)
    rng, out = np.random.default_rng(n), []
    sessions = [m.open() for _ in range(n)]
    prompts = [Prompt(rng.integers(0, c.card, (3 + i % 9, 17)).astype(np.int32), rng.integers(0, c.card, 17).tolist(), rng.integers(0, c.card, 7).tolist()) for i in range(n)]
    m.start(list(zip(sessions, prompts)))
    for t in range(20):
        got = m.tick([(s, Step(caller=rng.integers(0, c.card, 8).tolist(), seed=t * 1000 + i)) for i, s in enumerate(sessions)])
        out += [got.emitted.astype(np.float32).ravel()] + [np.concatenate([m.text_logits(i), m.audio_logits(i).ravel()]) for i in range(0, n, 7)]
    m.close()
    return out


def higgs(n, graphs):
    from pega_omni_b200.higgs import CODEBOOKS, HIGGS_PRESETS, HiggsDraw, HiggsModel, higgs_random_checkpoint
    c = HIGGS_PRESETS["higgs-mid"]
    m = HiggsModel.load(0, higgs_random_checkpoint(c, seed=7), c, max_batch=max(n, 4), max_tokens=2048, kv_gib=0.5, use_graphs=graphs)
    rng, out = np.random.default_rng(n), []
    prompts = [rng.integers(0, c.body.vocab_size, 4 + (23 * i) % 50).astype(np.int32) for i in range(n)]
    seqs = [m.open(len(p), 24) for p in prompts]
    for t in range(20):
        draws = [HiggsDraw(rng.random(CODEBOOKS).tolist()) for _ in range(n)]
        got = m.start(list(zip(seqs, prompts, draws))) if t == 0 else m.step(list(zip(seqs, draws)))
        out += [np.asarray(got.rows, np.float32).ravel()] + [m.logits(i).astype(np.float32).ravel() for i in range(0, n, 7)]
    m.close()
    return out


def codec(n, graphs):
    from pega_omni_b200.codec import CODEC_PRESETS, Codec, codec_random_checkpoint
    c = CODEC_PRESETS["qwen3-tts-12hz"]
    m = Codec(c, codec_random_checkpoint(c, seed=8), max_batch=n, use_graphs=graphs)
    rng = np.random.default_rng(n)
    streams = [m.open() for _ in range(n)]
    out = [m.decode(streams, rng.integers(0, c.codebook_size, (n, 16)).astype(np.int32)).copy() for _ in range(90)]
    m.close()
    return out


CALLS = {"talker": (talker, [1, 6, 40]), "duplex": (duplex, [1, 6, 40]), "higgs": (higgs, [1, 6, 40]), "codec": (codec, [1, 3, 64])}


def results(what, graphs):
    call, batches = CALLS[what]
    return {str(n): np.concatenate([np.ravel(x) for x in call(n, graphs)]) for n in batches}


@pytest.mark.parametrize("what", list(CALLS))
def test_launched_early_equals_one_after_the_other(built_lib, tmp_path, what):
    serial = tmp_path / "serial.npz"
    env = dict(os.environ, CUDA_LAUNCH_BLOCKING="1", PYTHONPATH=str(ROOT))
    subprocess.run([sys.executable, __file__, what, str(serial)], env=env, cwd=ROOT, check=True, timeout=300)
    want = np.load(serial)
    for n, got in results(what, True).items():
        assert np.isfinite(want[n]).all()
        assert np.array_equal(got, want[n]), (n, int((got != want[n]).sum()), float(np.abs(got - want[n]).max()))


if __name__ == "__main__":  # the process in which every launch is waited for
    np.savez(sys.argv[2], **results(sys.argv[1], False))
