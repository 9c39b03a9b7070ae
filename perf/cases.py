"""The work a serving program has this library do, as measurable cases.

Every case is one call of a model shell on a live batch, the way an engine drives it:

  talker-step    one decode tick of the Qwen3-TTS talker: the talker pass and its 15 code-predictor passes
  talker-start   admission of new requests: leases, prompt prefill, the first frame (time to first audio)
  duplex-tick    one 80 ms tick of live PersonaPlex conversations (Helium, then the depformer)
  higgs-step     one decode step of the Higgs-style model, with or without its audio-FFN adapter
  codec-decode   one frame of every stream through the streaming codec decoder, host codes to host samples

The models have the architectures of this repository's presets and random weights; the model of the latest case is kept
loaded, as a server keeps it. What a pass gives back are tokens (or samples), so the heads are made peaked: the row of
token j points along the embedding of the token that j follows. A trained model's draws are mostly decided by a wide
margin too, while a random head's nearly flat logits would turn on the last bit of a sum.
"""
from __future__ import annotations

import dataclasses
import math

import numpy as np
import torch

from pega_omni_b200.codec import CODEC_PRESETS, Codec, codec_random_checkpoint
from pega_omni_b200.config import presets
from pega_omni_b200.duplex import DEP_STEPS, PRESETS as DUPLEX_PRESETS, Model as DuplexModel, Prompt as DuplexPrompt, Step
from pega_omni_b200.duplex import random_checkpoint as duplex_random_checkpoint
from pega_omni_b200.higgs import CODEBOOKS, HIGGS_PRESETS, HiggsDraw, HiggsModel, higgs_random_checkpoint
from pega_omni_b200.model import Draw, Limits, Model, Prompt
from pega_omni_b200.synthetic import random_checkpoint

LEASE = 640        # frames (rows) a sequence may generate before its request ends and the next one takes its place
STATES = 4         # batches that may be alive at once
MAX_TOKENS = 8192  # prompt tokens of one start call (the shells' default limit)

TALKER = presets["qwen3-tts-1.7b"]()
TALKER_NUCLEUS = TALKER.with_generation(sampler="philox", top_p=0.95)
DUPLEX = dataclasses.replace(DUPLEX_PRESETS["personaplex-7b"], context=1000)  # 80 s of conversation per lease
HIGGS = HIGGS_PRESETS["higgs-4b"]
CODEC = CODEC_PRESETS["qwen3-tts-12hz"]
SPREAD = 3.0       # standard deviation of the logits of the tokens that do not follow


# ---- cases ---------------------------------------------------------------------------------------------------------

def listed():
    return [
        # one speaker, the interactive case: latency of a frame
        {"name": "talker-step-1", "kind": "talker-step", "sessions": 1, "prompt_min": 128, "prompt_max": 128, "nucleus": False},
        # a quiet server with the library's own random stream and a nucleus filter
        {"name": "talker-step-8-nucleus", "kind": "talker-step", "sessions": 8, "prompt_min": 32, "prompt_max": 256, "nucleus": True},
        # the configuration the headline metric is quoted on
        {"name": "talker-step-64", "kind": "talker-step", "sessions": 64, "prompt_min": 128, "prompt_max": 128, "nucleus": False},
        # a full server, prompts of the session sweep
        {"name": "talker-step-128-ragged", "kind": "talker-step", "sessions": 128, "prompt_min": 32, "prompt_max": 512, "nucleus": False},
        # one new request: time to first audio
        {"name": "talker-start-1", "kind": "talker-start", "sessions": 1, "prompt_min": 77, "prompt_max": 77, "nucleus": False},
        # a burst of requests that fills a start call
        {"name": "talker-start-28-ragged", "kind": "talker-start", "sessions": 28, "prompt_min": 32, "prompt_max": 512, "nucleus": False},
        # one live conversation
        {"name": "duplex-tick-1", "kind": "duplex-tick", "sessions": 1, "rows": 250},
        # a busy server
        {"name": "duplex-tick-64", "kind": "duplex-tick", "sessions": 64, "rows": 250},
        # a few generations, and the full batch with the audio-FFN adapter
        {"name": "higgs-step-3", "kind": "higgs-step", "sessions": 3, "prompt_min": 100, "prompt_max": 300, "adapter": False},
        {"name": "higgs-step-32-adapter", "kind": "higgs-step", "sessions": 32, "prompt_min": 256, "prompt_max": 256, "adapter": True},
        # audio of one speaker, and of the headline batch
        {"name": "codec-decode-1", "kind": "codec-decode", "sessions": 1, "age": 100},
        {"name": "codec-decode-64", "kind": "codec-decode", "sessions": 64, "age": 100},
    ]


def _spread(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["talker-step"] * 4 + ["talker-start"] * 2 + ["duplex-tick"] * 2 + ["higgs-step"] * 2 + ["codec-decode"] * 2)
    if kind == "talker-start":
        lo = _spread(rng, 16, 256)
        hi = _spread(rng, lo, 512)
        return {"kind": kind, "sessions": _spread(rng, 1, max(1, min(64, MAX_TOKENS * 9 // 10 // hi))), "prompt_min": lo, "prompt_max": hi, "nucleus": False}
    if kind == "talker-step":
        lo = _spread(rng, 16, 256)
        return {"kind": kind, "sessions": _spread(rng, 1, 128), "prompt_min": lo, "prompt_max": _spread(rng, lo, 512), "nucleus": rng.random() < 0.25}
    if kind == "duplex-tick":
        return {"kind": kind, "sessions": _spread(rng, 1, 64), "rows": _spread(rng, 40, 250)}
    if kind == "higgs-step":
        lo = _spread(rng, 64, 256)
        return {"kind": kind, "sessions": _spread(rng, 1, 32), "prompt_min": lo, "prompt_max": _spread(rng, lo, 400), "adapter": rng.random() < 0.5}
    return {"kind": kind, "sessions": _spread(rng, 1, 64), "age": _spread(rng, 4, 200)}


def _lengths(case):
    """Prompt lengths of a case's sessions: evenly over its range, in a fixed mixed order."""
    n, lo, hi = case["sessions"], case["prompt_min"], case["prompt_max"]
    step = next(k for k in range(max(1, round(0.618 * n)), n + 2) if math.gcd(k, n) == 1)
    return [lo + (hi - lo) * (i * step % n) // max(1, n - 1) for i in range(n)]


# ---- models (loaded once, kept while cases of the same model follow one another) -----------------------------------

class _Loaded:
    def __init__(self, model):
        self.model, self.served = model, []  # every request's handle, as a request log keeps them

    def __del__(self):  # the last batch of the model is gone
        self.model.close()


_loaded = {}


def _keep(key, load):
    if key not in _loaded:
        _loaded.clear()
        torch.cuda.empty_cache()
        _loaded[key] = _Loaded(load())
        torch.cuda.empty_cache()
    return _loaded[key]


def _following(table, count, logits_std):
    """Head rows for tokens 0..count-1: token (3 c + 1) mod count follows token c."""
    after = (3 * torch.arange(count, device=table.device) + 1) % count
    head = torch.empty_like(table[:count])
    head[after] = table[:count]
    rms = head.float().square().mean().sqrt()
    return head * (logits_std / (rms * head.shape[1] ** 0.5)).to(head.dtype)


def _load_talker(cfg):
    ck = random_checkpoint(cfg, seed=0, std=0.01, device="cuda", embed_std=1.0)
    usable = cfg.talker.vocab_size - cfg.control_tokens
    first = ck["talker.model.codec_embedding.weight"]
    ck["talker.codec_head.weight"][:usable] = _following(first[:usable].float(), usable, SPREAD).bfloat16()
    project = ck["talker.code_predictor.small_to_mtp_projection.weight"].float()
    for g in range(cfg.num_code_groups - 1):  # head g draws the code that follows the previous group's
        table = first if g == 0 else ck[f"talker.code_predictor.model.codec_embedding.{g - 1}.weight"]
        rows = table[:cfg.predictor.vocab_size].float() @ project.T
        ck[f"talker.code_predictor.lm_head.{g}.weight"] = _following(rows, cfg.predictor.vocab_size, SPREAD).bfloat16()
    return Model.load(0, ck, cfg, Limits(max_batch=STATES * 128, max_tokens=MAX_TOKENS, kv_gib=60.0))


def _load_duplex():
    c = DUPLEX
    ck = duplex_random_checkpoint(c, seed=0, std=0.01, device="cuda")
    ck["h.text_linear"] = _following(ck["h.text_emb"].float(), c.text_vocab, SPREAD).bfloat16()
    # a text token stands for the audio code of the same number modulo the codebook
    ck["d.text_emb"] = ck["d.text_emb"][:c.card].repeat(-(-(c.text_vocab + 1) // c.card), 1)[:c.text_vocab + 1].contiguous()
    books = [ck["d.text_emb"]] + list(ck["d.emb"].view(DEP_STEPS - 1, c.card + 1, c.dep_dim))
    ck["d.heads"] = torch.cat([_following(b.float(), c.card, SPREAD).bfloat16() for b in books])
    model = DuplexModel.load(0, ck, c, max_sessions=STATES * 64)
    model.warmup()
    return model


def _load_higgs(adapter):
    c = dataclasses.replace(HIGGS, audio_adapter=adapter)
    ck = higgs_random_checkpoint(c, seed=0, std=0.01, device="cuda", embed_std=1.0)
    # the head is the embedding table itself, so a code is followed by itself; the final norm's gain sets the logits' scale
    ck["body.norm.weight"].fill_(SPREAD / c.body.hidden_size ** 0.5)
    kv_gib = 2.0 * STATES * 16 * (400 + LEASE) * c.body.kv_bytes_per_token() / 2 ** 30
    model = HiggsModel.load(0, ck, c, max_batch=STATES * 32, max_tokens=MAX_TOKENS, kv_gib=kv_gib)
    model.warmup()
    return model


def _load_codec():
    # gentler periodic activations than the preset's (log-scale frequencies): the waveform stays inside the clamp, as
    # speech does, and a rounding in an early layer is not blown up by the later ones
    ck = {k: v - 1.0 if k.endswith(".alpha") else v for k, v in codec_random_checkpoint(CODEC, seed=0).items()}
    model = Codec(CODEC, ck, max_batch=64, streams=STATES * 64)
    model.warmup()
    return model


# ---- states --------------------------------------------------------------------------------------------------------

def _talker_prompts(case, rng):
    """Text ids on every row; the codec track carries codes from the middle of the prompt on."""
    out = []
    for n in _lengths(case):
        codec = rng.integers(0, 2048, n)
        codec[:n // 2] = -1
        out.append(Prompt(rng.integers(0, TALKER.text_vocab_size, n).tolist(), codec.tolist()))
    return out


def _talker_draws(rng, n):
    return [Draw(u) for u in rng.random((n, 16)).tolist()]


class _Talker:
    """`frames` > 0: a batch in mid-generation; 0: requests that wait to be admitted."""

    def __init__(self, case, seed, frames):
        cfg = TALKER_NUCLEUS if case["nucleus"] else TALKER
        self.kept = _keep(("talker", case["nucleus"]), lambda: _load_talker(cfg))
        self.model = self.kept.model
        rng = np.random.default_rng(seed)
        self.prompts, self.frames, self.seqs, self.at = _talker_prompts(case, rng), frames, [], 0
        self.first = _talker_draws(rng, case["sessions"])
        self.draws = [_talker_draws(rng, case["sessions"]) for _ in range(16 if frames else 0)]
        self.seeds = rng.integers(0, 2 ** 62, case["sessions"]).tolist() if case["nucleus"] else None
        if frames:
            self.admit()

    def admit(self):
        self.seqs = [self.model.open(len(p), max(1, self.frames)) for p in self.prompts]
        self.kept.served += self.seqs
        if self.seeds:
            for s, seed in zip(self.seqs, self.seeds):
                self.model.seed(s, seed)
        rows, codes, tokens = [], [], 0
        for row in zip(self.seqs, self.prompts, self.first):
            if tokens + len(row[1]) > MAX_TOKENS:
                codes.append(self.model.start(rows).codes)
                rows, tokens = [], 0
            rows.append(row)
            tokens += len(row[1])
        codes.append(self.model.start(rows).codes)
        self.left = self.frames - 1
        return codes[0] if len(codes) == 1 else np.concatenate(codes)

    def leave(self):
        for s in self.seqs:
            self.model.release(s)
        self.seqs = []

    def step(self):
        if self.left < 1:
            self.leave()
            self.admit()
        self.left -= 1
        self.at += 1
        return self.model.step(list(zip(self.seqs, self.draws[self.at % len(self.draws)]))).codes

    def start(self):
        codes = self.admit()
        self.leave()
        return codes

    def __del__(self):
        self.leave()


class _Duplex:
    """Conversations that share four personas (their prompts are the same for every caller), each with its own caller."""

    def __init__(self, case, seed):
        self.kept = _keep(("duplex",), _load_duplex)
        self.model = self.kept.model
        n, c, rng = case["sessions"], DUPLEX, np.random.default_rng(seed)
        fixed = np.random.default_rng(case["rows"])
        personas = [np.concatenate([fixed.integers(0, c.text_vocab, (case["rows"], 1)), fixed.integers(0, c.card, (case["rows"], 16))], 1) for _ in range(4)]
        self.sessions = [self.model.open() for _ in range(n)]
        prompts = [DuplexPrompt(personas[i % 4], [int(rng.integers(0, c.text_vocab))] + rng.integers(0, c.card, 16).tolist(), rng.integers(0, c.card, 7).tolist())
                   for i in range(n)]
        for at in range(0, n, 8):  # 2,048 prompt rows at most in one call
            self.model.start(list(zip(self.sessions[at:at + 8], prompts[at:at + 8])))
        self.steps = [[Step(caller=rng.integers(0, c.card, 8).tolist(), seed=int(rng.integers(0, 2 ** 62))) for _ in range(n)] for _ in range(16)]
        self.at = 0

    def tick(self):
        self.at += 1
        return self.model.tick(list(zip(self.sessions, self.steps[self.at % len(self.steps)]))).emitted

    def __del__(self):
        for s in self.sessions:
            self.model.release(s)


class _Higgs:
    """Generations past the delay pattern's ramp: all eight codebooks are drawn."""

    def __init__(self, case, seed):
        self.kept = _keep(("higgs", case["adapter"]), lambda: _load_higgs(case["adapter"]))
        self.model = self.kept.model
        n, rng = case["sessions"], np.random.default_rng(seed)
        self.prompts = [rng.integers(0, HIGGS.body.vocab_size, k).astype(np.int32) for k in _lengths(case)]
        self.ramp = [[HiggsDraw([0.5] * CODEBOOKS, r) for r in rng.integers(0, 1024, (n, CODEBOOKS)).tolist()] for _ in range(CODEBOOKS)]
        self.draws = [[HiggsDraw(u) for u in rng.random((n, CODEBOOKS)).tolist()] for _ in range(16)]
        self.seqs, self.at = [], 0
        self.admit()

    def admit(self):
        self.seqs = [self.model.open(len(p), LEASE) for p in self.prompts]
        for at in range(0, len(self.seqs), 16):
            self.model.start(list(zip(self.seqs, self.prompts, self.ramp[0]))[at:at + 16])
        for row in self.ramp[1:]:
            self.model.step(list(zip(self.seqs, row)))
        self.left = LEASE - CODEBOOKS

    def leave(self):
        for s in self.seqs:
            self.model.release(s)
        self.seqs = []

    def step(self):
        if self.left < 1:
            self.leave()
            self.admit()
        self.left -= 1
        self.at += 1
        out = self.model.step(list(zip(self.seqs, self.draws[self.at % len(self.draws)])))
        return {"rows": out.rows, "ended": out.ended}

    def __del__(self):
        self.leave()


class _Codec:
    """Streams that have played `age` frames (the attention window is full after 72)."""

    def __init__(self, case, seed):
        self.kept = _keep(("codec",), _load_codec)
        self.model = self.kept.model
        n, rng = case["sessions"], np.random.default_rng(seed)
        self.frames = list(rng.integers(0, CODEC.codebook_size, (24, n, 16)).astype(np.int32))
        self.streams = [self.model.open() for _ in range(n)]
        self.at = 0
        for _ in range(case["age"]):
            self.decode()

    def decode(self):
        self.at += 1
        return self.model.decode(self.streams, self.frames[self.at % len(self.frames)])

    def __del__(self):
        for s in self.streams:
            s.close()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "talker-step":
        return _Talker(case, seed, LEASE).step
    if kind == "talker-start":
        return _Talker(case, seed, 0).start
    if kind == "duplex-tick":
        return _Duplex(case, seed).tick
    if kind == "higgs-step":
        return _Higgs(case, seed).step
    return _Codec(case, seed).decode


def run(state):
    return state()


# ---- what a pass cannot do without ---------------------------------------------------------------------------------

def _stack(c, layers=None):
    return (c.num_hidden_layers if layers is None else layers) * c.layer_weight_bytes() // 2  # parameters


def work(case):
    """Every weight once (bf16), every key and value that is attended to once, the new ones written; the heads' and
    projections' multiply-adds per row."""
    n, kind = case["sessions"], case["kind"]
    if kind.startswith("talker"):
        t, p, g = TALKER.talker, TALKER.predictor, TALKER.num_code_groups
        tail = t.vocab_size * t.hidden_size + _stack(p) + p.hidden_size * t.hidden_size + (g - 1) * p.vocab_size * p.hidden_size
        # the first frame's head, its 15 predictor passes over 16 rows, 15 heads
        tail_macs = n * (t.vocab_size * t.hidden_size + g * (_stack(p) + p.hidden_size * t.hidden_size) + (g - 1) * p.vocab_size * p.hidden_size)
        lens = _lengths(case)
        kv, qd = t.kv_bytes_per_token(), t.num_attention_heads * t.head_dim
        if kind == "talker-start":
            rows = sum(lens)
            pairs = sum(k * (k + 1) // 2 for k in lens)
            macs = rows * (_stack(t) + 2 * t.hidden_size ** 2) + t.num_hidden_layers * 2 * qd * pairs + tail_macs
            return {"bytes": 2 * (_stack(t) + 2 * t.hidden_size ** 2 + tail) + rows * (kv + 4 * t.hidden_size), "flops": 2 * macs}
        pairs = sum(k + 2 for k in lens)
        macs = n * _stack(t) + t.num_hidden_layers * 2 * qd * pairs + tail_macs
        return {"bytes": 2 * (_stack(t) + tail) + kv * (pairs + n), "flops": 2 * macs}
    if kind == "duplex-tick":
        c = DUPLEX
        weights, pairs = c.tick_weight_bytes(), n * (case["rows"] + 2)
        return {"bytes": weights + c.layers * c.heads * 2 * 132 * (pairs + n), "flops": weights * n + 4 * c.layers * c.dim * pairs}
    if kind == "higgs-step":
        c = dataclasses.replace(HIGGS, audio_adapter=case["adapter"])
        b, weights, pairs = c.body, c.step_weight_bytes(), sum(k + CODEBOOKS + 1 for k in _lengths(case))
        qd = b.num_attention_heads * b.head_dim
        return {"bytes": weights + b.kv_bytes_per_token() * (pairs + n), "flops": weights * n + 4 * b.num_hidden_layers * qd * pairs}
    window = CODEC.num_hidden_layers * CODEC.num_attention_heads * CODEC.head_dim * 2 * 2 * min(case["age"] + 1, CODEC.sliding_window)
    return {"bytes": CODEC.weight_bytes() + n * (window + 4 * CODEC.samples_per_frame), "flops": n * CODEC.flops_per_frame()}


def tolerance(case):
    if case["kind"] == "codec-decode":
        return {"rel": 0.025}  # some forty bf16 layers deep: two summation orders in the GEMMs differ by 0.015 to 0.017
    return "exact"
