"""The kernels of the decode chains and of the prompts, at the sizes where they can go wrong: the row counts at which
another kernel takes over, ragged tiles and K splits, the smallest and largest team of an attention item. Products are
checked against fp32 torch, attention in one kernel against the separate rotation and attention kernels."""
import dataclasses

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops(built_lib):
    from pega_omni_b200.ops import Ops
    o = Ops(0)
    yield o
    o.close()


def rand(shape, seed, scale=1.0):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return (torch.randn(shape, generator=g, device="cuda") * scale).to(torch.bfloat16)


def close(got, want, steps=2.0, floor=0.05):
    """Within `steps` bf16 steps of the fp32 value; `floor`: the size of what was rounded on the way, where sums cancel."""
    g, w = got.float(), want.float()
    bad = ~((g - w).abs() <= steps * 2.0 ** -7 * w.abs().clamp_min(floor))  # NaN is a difference
    assert not bad.any(), (int(bad.sum()), float((g - w).abs().max()))


def product(x, w):
    return x.float() @ w.float().T


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


# rows: the warp-level kernel up to eight, then tcgen05 with M = 64, 128, two row tiles, SM pairs
@pytest.mark.parametrize("rows", [1, 7, 8, 9, 16, 17, 64, 65, 128, 129, 256, 257, 300])
@pytest.mark.parametrize("n,k,epilogue", [(200, 128, 0), (1000, 1088, 1), (4096, 64, 2), (24, 6144, 0)])
def test_chain_gemm(ops, rows, n, k, epilogue):
    w, x, bias = rand((n, k), 1, k ** -0.5), rand((rows, k), 2), rand((n,), 3)
    y = torch.full((rows + 1, n), 7.0, dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    ops.chain_gemm(w, x, y[:rows], bias=bias if epilogue else None, epilogue=epilogue)
    ops.sync()
    want = product(x, w).bfloat16().float()
    if epilogue:
        want = (want + bias.float()).bfloat16().float()
    if epilogue == 2:
        want = torch.nn.functional.silu(want)
    close(y[:rows], want, floor=4.0 if epilogue else 0.05)
    assert (y[rows] == 7.0).all()  # nothing past the last row


def test_a_gemm_waits_for_the_call_that_makes_its_bias(ops):
    """The second call's bias is the first one's output, which takes a few CTAs some time; nobody waits in between."""
    w1, x1, w2, x2 = rand((64, 32768), 151, 32768 ** -0.5), rand((16, 32768), 152), rand((64, 64), 153, 0.125), rand((16, 64), 154)
    outs = []
    for wait in (True, False):
        made = torch.zeros((16, 64), dtype=torch.bfloat16, device="cuda")
        y = torch.zeros((16, 64), dtype=torch.bfloat16, device="cuda")
        torch.cuda.synchronize()
        ops.chain_gemm(w1, x1, made)
        if wait:
            ops.sync()
        ops.chain_gemm(w2, x2, y, bias=made[15], epilogue=1)
        ops.sync()
        outs.append(y)
    assert torch.equal(outs[0], outs[1])


# few rows whose share of a CTA's shared memory, or whose weights, the tcgen05 kernel takes: both sides of either line
@pytest.mark.parametrize("rows,n,k", [(5, 48, 4288), (5, 48, 4352), (8, 48, 2560), (8, 48, 2752), (8, 48, 11264), (2, 8208, 8192), (3, 8208, 8192),
                                      (3, 8176, 8192)])
def test_chain_gemm_of_few_long_rows(ops, rows, n, k):
    test_chain_gemm(ops, rows, n, k, 0)


@pytest.mark.parametrize("k", [64, 4096])
def test_swiglu_of_few_long_rows_at_any_address(ops, k):
    """The tcgen05 kernel refuses an activation row that vector stores cannot take: few rows stay with the other one."""
    w, x = rand((64, k), 51, k ** -0.5), rand((8, k), 52)
    y = torch.zeros(8 * 32 + 1, dtype=torch.bfloat16, device="cuda")[1:].view(8, 32)
    torch.cuda.synchronize()
    ops.chain_gemm(w, x, y, swiglu=True)
    ops.sync()
    gate, up = product(x, w[:32]).bfloat16().float(), product(x, w[32:]).bfloat16().float()
    close(y, torch.nn.functional.silu(gate).bfloat16().float() * up, steps=3.0)


# the tcgen05 epilogue's fragments: rows that end inside one, columns that leave a warp of a pair without any, one to four sums
@pytest.mark.parametrize("rows", [10, 24, 25, 57, 73, 121])
@pytest.mark.parametrize("n,k", [(199, 64), (176, 192), (40, 320), (8, 1024)])
def test_chain_gemm_fragments(ops, rows, n, k):
    w, x = rand((n, k), 41, k ** -0.5), rand((rows, k), 42)
    y = torch.full((rows + 1, n), 7.0, dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    ops.chain_gemm(w, x, y[:rows])
    ops.sync()
    close(y[:rows], product(x, w))
    assert (y[rows] == 7.0).all()


@pytest.mark.parametrize("rows", [1, 9, 17, 128, 129, 257])
@pytest.mark.parametrize("inter,k", [(256, 64), (3072, 1024), (4096, 576)])
def test_chain_swiglu(ops, rows, inter, k):
    """The last tile may hold fewer channels than the others."""
    w, x = rand((2 * inter, k), 4, k ** -0.5), rand((rows, k), 5)
    y = torch.zeros((rows, inter), dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    ops.chain_gemm(w, x, y, swiglu=True)
    ops.sync()
    gate, up = product(x, w[:inter]).bfloat16().float(), product(x, w[inter:]).bfloat16().float()
    close(y, torch.nn.functional.silu(gate).bfloat16().float() * up, steps=3.0)


@pytest.mark.parametrize("rows", [1, 2, 4, 5, 8, 9, 17, 130, 256])
@pytest.mark.parametrize("d,k,n", [(1024, 3072, 512), (2560, 64, 200), (64, 2048, 96), (4096, 128, 64)])
def test_chain_norm_gemm(ops, rows, d, k, n):
    """Split sums, the add + norm over them (folded into the next product or on its own) and that product."""
    w1, x, res, gain = rand((d, k), 6, k ** -0.5), rand((rows, k), 7), rand((rows, d), 8), rand((d,), 9, 0.2) + 1
    w2, y = rand((n, d), 10, d ** -0.5), torch.zeros((rows, n), dtype=torch.bfloat16, device="cuda")
    v = product(x, w1).bfloat16().float() + res.float()
    h = (v * torch.rsqrt((v * v).mean(1, keepdim=True) + 1e-6) * gain.float()).bfloat16()
    torch.cuda.synchronize()
    ops.chain_norm_gemm(w1, x, res, gain, 1e-6, w2, y)
    ops.sync()
    close(res, v, floor=4.0)
    close(y, product(h, w2), floor=4.0)


def paged(lens, seed, spare=3):
    """Shuffled pages of sequences that hold lens[s] tokens: (pos, slot, indptr, pages, page count)."""
    rng = np.random.default_rng(seed)
    count = sum((n + 15) // 16 for n in lens) + spare
    perm, at = rng.permutation(count), 0
    pos, slot, indptr, pages = [], [], [0], []
    for n in lens:
        mine = [int(p) for p in perm[at:at + (n + 15) // 16]]
        at += len(mine)
        pages += mine
        indptr.append(len(pages))
        pos.append(n - 1)
        slot.append(mine[(n - 1) // 16] * 16 + (n - 1) % 16)
    return i32(pos), i32(slot), i32(indptr), i32(pages), count


# up to 148 (sequence, kv head) items a team has eight warps, up to 444 four, beyond that three
@pytest.mark.parametrize("hq,hk,d", [(16, 8, 128), (4, 4, 64), (5, 1, 128), (8, 2, 64), (8, 1, 128)])
@pytest.mark.parametrize("sessions", [1, 40, 160])
def test_decode_attention_in_one_kernel(ops, hq, hk, d, sessions):
    lens = [[1, 16, 17, 129, 300][s % 5] for s in range(sessions)]
    pos, slot, indptr, pages, count = paged(lens, sessions)
    qkv, qn, kn = rand((sessions, (hq + 2 * hk) * d), 11), rand((d,), 12, 0.2) + 1, rand((d,), 13, 0.2) + 1
    kv = rand((count, hk, 2, 16, d), 14)
    a, b = (torch.zeros((sessions, hq * d), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    kv_b, qkv_b = kv.clone(), qkv.clone()
    torch.cuda.synchronize()
    ops.decode_attend(qkv, qn, kn, kv, count, pos, slot, indptr, pages, hq, hk, d, 1e-6, 1e6, a)
    ops.rope_attend(qkv_b, qn, kn, kv_b, count, pos, slot, None, indptr, pages, hq, hk, d, 1e-6, 1e6, b)
    ops.sync()
    assert torch.equal(kv, kv_b)
    close(a, b, steps=1.5, floor=0.25)


# around the counts at which the warps of a team change: 148, 444 and 592 items on 148 SMs
@pytest.mark.parametrize("items", [147, 149, 443, 445, 500, 591, 593])
@pytest.mark.parametrize("hq,hk,d", [(2, 1, 128), (4, 1, 64), (5, 1, 128)])
def test_decode_attention_teams(ops, hq, hk, d, items):
    test_decode_attention_in_one_kernel(ops, hq, hk, d, items)


# two, four and eight columns a thread, rows that end inside a warp of each; one sum, of products that are one k-block long
@pytest.mark.parametrize("rows", [9, 250])
@pytest.mark.parametrize("d", [1984, 2048, 2112, 4096, 4160])
def test_chain_norm_columns(ops, rows, d):
    test_chain_norm_gemm(ops, rows, d, 64, 64)


# every count of sums by every count of columns a thread (the last by the rows, too)
@pytest.mark.parametrize("lm", [False, True])
@pytest.mark.parametrize("splits", [1, 2, 4, 8])
@pytest.mark.parametrize("rows,d", [(9, 1984), (250, 2048), (9, 2112), (256, 4096), (9, 4160), (5, 8192), (257, 1024)])
def test_add_norm_of_split_sums(ops, rows, d, splits, lm):
    g = torch.Generator(device="cuda").manual_seed(d + splits)
    part = torch.randn((splits, rows, d), generator=g, device="cuda")
    res, gain = rand((rows, d), 171), rand((d,), 172, 0.2) + 1
    total = part[0].clone()
    for p in part[1:]:
        total += p
    v = res.float() + total.bfloat16().float()
    if lm:
        v = v.bfloat16().float()
    out = torch.zeros((rows, d), dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    ops.add_norm_sum(part, res, gain, out, 1e-6, lm=lm)
    ops.sync()
    assert torch.equal(res, v.bfloat16())
    close(out, v * torch.rsqrt((v * v).mean(1, keepdim=True) + 1e-6) * gain.float(), steps=1.0)


@pytest.mark.parametrize("heads,sessions", [(4, 1), (4, 37), (32, 5), (16, 16)])
def test_fp8_ring_attention_in_one_kernel(ops, heads, sessions):
    """Positions before, at and past the end of a ring of 40 tokens."""
    context, per = 40, 3
    rng = np.random.default_rng(heads + sessions)
    pages = rng.permutation(sessions * per)
    at = [[0, 15, 16, 39, 40, 55, 131][s % 7] for s in range(sessions)]
    slot = [int(pages[s * per + (p % context) // 16]) * 16 + p % context % 16 for s, p in enumerate(at)]
    block = heads * (2 * 16 * 128 + 2 * 16 * 4)
    kv = torch.zeros(sessions * per, block, dtype=torch.uint8, device="cuda")
    coef, scale = float(np.float32(-np.log(10000.0) * 2.0 / 128)), 128 ** -0.5
    indptr, table = i32([s * per for s in range(sessions + 1)]), i32(pages.tolist())
    for p in range(context):  # fills the rings through the separate kernels
        qkv = rand((sessions, 3 * heads * 128), 100 + p)
        where = i32([int(pages[s * per + p // 16]) * 16 + p % 16 for s in range(sessions)])
        out = torch.zeros((sessions, heads * 128), dtype=torch.bfloat16, device="cuda")
        torch.cuda.synchronize()
        ops.lm_rope_attend(qkv, kv, sessions * per, i32([p] * sessions), where, None, indptr, table, heads, coef, scale, context, out)
        ops.sync()
    qkv = rand((sessions, 3 * heads * 128), 99)
    qkv_b, kv_b = qkv.clone(), kv.clone()
    a, b = (torch.zeros((sessions, heads * 128), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    ops.lm_decode_attend(qkv, kv, sessions * per, i32(at), i32(slot), indptr, table, heads, coef, scale, context, a)
    ops.lm_rope_attend(qkv_b, kv_b, sessions * per, i32(at), i32(slot), None, indptr, table, heads, coef, scale, context, b)
    ops.sync()
    assert torch.equal(kv, kv_b)
    close(a, b, steps=1.5, floor=0.25)


# one, two, eight and sixteen warps an item, and a last CTA that is not full (four, and more than one page a warp: further down)
@pytest.mark.parametrize("heads,sessions", [(4, 296), (1, 1187), (3, 231), (32, 19), (4, 73), (1, 147)])
def test_fp8_ring_attention_teams(ops, heads, sessions):
    test_fp8_ring_attention_in_one_kernel(ops, heads, sessions)


# sixteen, eight, four, two warps an item and one, which stores whole rows as vectors where it may
@pytest.mark.parametrize("per_sm", [1, 2, 4, 8, 9])
def test_fp8_ring_attention_into_rows_at_any_address(ops, per_sm):
    sessions, context = per_sm * torch.cuda.get_device_properties(0).multi_processor_count, 16
    kv = torch.zeros(sessions, 1, 2 * 16 * 128 + 2 * 16 * 4, dtype=torch.uint8, device="cuda")
    qkv, table = rand((sessions, 3 * 128), 141), i32(list(range(sessions)))
    at, slot, indptr = i32([3] * sessions), i32([16 * s + 3 for s in range(sessions)]), i32(list(range(sessions + 1)))
    outs = []
    for offset in (0, 1):
        out = torch.zeros(sessions * 128 + 1, dtype=torch.bfloat16, device="cuda")[offset:offset + sessions * 128].view(sessions, 128)
        torch.cuda.synchronize()
        ops.lm_decode_attend(qkv, kv, sessions, at, slot, indptr, table, 1, -0.14, 0.1, context, out)
        ops.sync()
        outs.append(out)
    close(outs[1], outs[0], steps=1.0, floor=1e-3)  # (one warp's sums merged by two)
    assert outs[0].any()


@pytest.mark.parametrize("top", [2.0 ** -130, 2.0 ** -113, 2.0 ** -112, 1.5 * 2.0 ** 113, 2.0 ** 114, 2.0 ** 115])
def test_fp8_ring_attention_of_a_query_of_any_size(ops, top):
    """Queries whose largest element is near either end of f32: the sums of the scalar kernel are finite, and so are these."""
    heads, sessions, per, context = 4, 3, 2, 32
    at, table, indptr = i32([7, 31, 50]), i32([4, 1, 0, 2, 5, 3]), i32([0, 2, 4, 6])
    slot = i32([4 * 16 + 7, 2 * 16 + 15, 3 * 16 + 2])
    kv = torch.zeros(sessions * per, heads, 2 * 16 * 128 + 2 * 16 * 4, dtype=torch.uint8, device="cuda")
    kv[:, :, :4096] = (rand((sessions * per, heads, 4096), 131).float() * 0.5).to(torch.float8_e4m3fn).view(torch.uint8)
    kv[:, :, 4096:] = torch.full((sessions * per, heads, 32), 0.01, device="cuda").view(torch.uint8)
    x = torch.randn((sessions, 3 * heads * 128), generator=torch.Generator().manual_seed(7)).clamp(-2, 2)
    q = x[:, :heads * 128].view(sessions, heads, 64, 2)
    q[:, :, 5] = torch.tensor([4.0, 0.0])
    q *= top / 4.0  # rotation keeps a pair's length: 2^0 to 2^-0.5 of it is in its larger element
    qkv = x.to(torch.bfloat16).cuda()
    qkv_b, kv_b = qkv.clone(), kv.clone()
    a, b = (torch.zeros((sessions, heads * 128), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    coef = float(np.float32(-np.log(10000.0) * 2.0 / 128))
    ops.lm_decode_attend(qkv, kv, sessions * per, at, slot, indptr, table, heads, coef, 128 ** -0.5, context, a)
    ops.lm_rope_attend(qkv_b, kv_b, sessions * per, at, slot, None, indptr, table, heads, coef, 128 ** -0.5, context, b)
    ops.sync()
    assert torch.equal(kv, kv_b) and torch.isfinite(b.float()).all()
    close(a, b, steps=1.5, floor=1e-3)


@pytest.mark.parametrize("vocab", [1, 2047, 2048, 2049, 32768, 40001])
def test_duplex_sampler_takes_the_largest(ops, vocab):
    """top_k = 1 leaves the largest logit whatever the noise, at both ends of each register budget."""
    rows = 5
    logits = rand((rows, vocab), vocab, 3.0)
    top = torch.randint(0, vocab, (rows,), generator=torch.Generator().manual_seed(vocab))
    logits[torch.arange(rows), top.cuda()] = 40.0
    force = torch.full((rows, 9), -1, dtype=torch.int32, device="cuda")
    force[2, 3] = 0
    drawn = torch.full((rows, 9), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ops.lm_sample(logits, 0.8, 1, force, i32([[r, 7] for r in range(rows)]), 3, drawn)
    ops.sync()
    want = top.clone()
    want[2] = 0
    assert drawn[:, 3].cpu().tolist() == want.tolist()


# 96 channels take zero-filled boxes; one stream leaves most of a 128-row tile empty; 70 streams fill several tiles
@pytest.mark.parametrize("n", [1, 3, 70])
@pytest.mark.parametrize("T,C,N,taps,dil,kind", [(4, 4096, 64, 1, 1, 1), (32, 128, 256, 7, 9, 2), (160, 192, 200, 7, 3, 0),
                                                 (128, 96, 96, 7, 1, 2), (2, 64, 24, 1, 1, 0), (64, 96, 96, 1, 1, 1)])
def test_codec_conv(ops, n, T, C, N, taps, dil, kind):
    P = (taps - 1) * dil + T
    w, x, bias = rand((N, taps * C), 20, (taps * C) ** -0.5), rand((n, P, C), 21), rand((N,), 22)
    y = rand((n * T, N), 23)
    alpha, inv_b = torch.rand(N, device="cuda") + 0.5, torch.rand(N, device="cuda") + 0.5
    cols = torch.stack([x[:, j * dil:j * dil + T] for j in range(taps)], 2).reshape(n * T, taps * C)
    want = product(cols, w)
    if kind == 1:
        want = want + y.float()
    if kind == 2:
        want = want.bfloat16().float() + bias.float()
        want = want + inv_b * torch.sin(alpha * want) ** 2
    torch.cuda.synchronize()
    ops.codec_conv(w, C, taps, dil, x, T, n, y, epilogue=kind, bias=bias, alpha=alpha, inv_b=inv_b)
    ops.sync()
    close(y, want, floor=4.0)


@pytest.mark.parametrize("sessions", [1, 5, 20])
def test_talker_as_a_chain_agrees_with_per_op_kernels(built_lib, sessions, predictor={}, ticks=4, max_tokens=2048):
    """Stacks too large for the L2 run as chains: forced frames give the logits of the per-op kernels."""
    from pega_omni_b200.config import presets
    from pega_omni_b200.model import Draw, Limits, Model, Prompt
    from pega_omni_b200.synthetic import random_checkpoint
    base = presets["mid"]()
    cfg = dataclasses.replace(base, talker=dataclasses.replace(base.talker, hidden_size=1024, intermediate_size=3072,
                                                               num_hidden_layers=6, num_attention_heads=16,
                                                               num_key_value_heads=8, head_dim=128),
                              predictor=dataclasses.replace(base.predictor, **predictor))
    ck = random_checkpoint(cfg, seed=3, device="cuda")
    rng = np.random.default_rng(sessions)
    lens = [9 + (31 * s) % 90 for s in range(sessions)]
    prompts = [Prompt(list(rng.integers(0, cfg.text_vocab_size, n)), [-1] * n) for n in lens]
    hi = min(cfg.talker.vocab_size - cfg.control_tokens, cfg.predictor.vocab_size)
    forced = rng.integers(0, hi, (ticks, sessions, 16)).astype(np.int32)
    forced[:, :, cfg.num_code_groups:] = 0
    got = []
    for tick_kernel in (True, False):
        m = Model.load(0, ck, cfg, Limits(max_batch=max(sessions, 8), max_tokens=max_tokens, kv_gib=0.5), tick_kernel=tick_kernel)
        seqs, rows = [m.open(n, 8) for n in lens], []
        for t in range(ticks):
            draws = [Draw([0.5] * 16, list(forced[t, s])) for s in range(sessions)]
            out = m.start(list(zip(seqs, prompts, draws))) if t == 0 else m.step(list(zip(seqs, draws)))
            assert (out.codes == forced[t]).all()
            rows.append(np.stack([np.concatenate([m.talker_logits(s), m.predictor_logits(s).ravel()]) for s in range(sessions)]))
        assert m.stats().last_call_launches > 1
        got.append(np.stack(rows))
        m.close()
    a, b = got
    step = np.exp2(np.floor(np.log2(np.maximum(np.abs(b), 2.0))) - 7)
    assert float((np.abs(a - b) / step).max()) <= 2.0


# More than 444 rows and kv heads: the longest rows' attention starts first. Buckets of 64 (one wave of three-warp CTAs) and 128
# rows, with padding; prompts of one to seven pages in no order of length, which changes between the ticks of the replayed graph.
@pytest.mark.parametrize("sessions", [60, 70])
def test_talker_rows_started_by_length_agree_with_per_op_kernels(built_lib, sessions):
    pages = [[(9 + (31 * s) % 90 + t) // 16 for s in range(sessions)] for t in range(5)]
    orders = [sorted(range(sessions), key=lambda s: -p[s]) for p in pages]  # as the staged inputs have it, ties as they come
    assert all(o != list(range(sessions)) for o in orders) and orders[2] != orders[3] != orders[4]
    test_talker_as_a_chain_agrees_with_per_op_kernels(built_lib, sessions, ticks=6, max_tokens=8192)


# a frame's attention: head widths and query heads a kv head, one row a sequence and the first two
@pytest.mark.parametrize("hq,hk,d", [(4, 4, 64), (8, 4, 64), (8, 2, 128), (5, 1, 128), (16, 2, 64)])
def test_frame_attention_agrees_with_per_op_kernels(built_lib, hq, hk, d):
    test_talker_as_a_chain_agrees_with_per_op_kernels(built_lib, 19, dict(num_attention_heads=hq, num_key_value_heads=hk, head_dim=d))


@pytest.mark.parametrize("bad", [-9, (1 << 20) + 9])  # tokens 7 and 9, which no other row writes
def test_a_row_without_a_page_stores_nothing(ops, bad):
    """A slot outside the pool is reported; the pages, page 0 among them, keep what the other rows need."""
    from pega_omni_b200.ops import OpsError
    hq, hk, d, lens, lost = 4, 2, 128, [17, 5, 33], 1
    pos, slot, indptr, pages, count = paged(lens, 3)
    wrong = slot.clone()
    wrong[lost] = bad
    qkv, qn, kn = rand((3, (hq + 2 * hk) * d), 31), rand((d,), 32, 0.2) + 1, rand((d,), 33, 0.2) + 1
    kv = rand((count, hk, 2, 16, d), 34)
    own = (int(slot[lost]) // 16, slice(None), slice(None), int(slot[lost]) % 16)
    want, before = kv.clone(), kv[own].clone()
    out = torch.zeros((3, hq * d), dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    ops.decode_attend(qkv, qn, kn, want, count, pos, slot, indptr, pages, hq, hk, d, 1e-6, 1e6, out)
    ops.sync()
    want[own] = before
    torch.cuda.synchronize()
    ops.decode_attend(qkv, qn, kn, kv, count, pos, wrong, indptr, pages, hq, hk, d, 1e-6, 1e6, out)
    with pytest.raises(OpsError):
        ops.sync()
    assert torch.equal(kv, want)


@pytest.mark.parametrize("in_one", [True, False])
def test_a_ring_row_without_a_page_stores_nothing(ops, in_one):
    from pega_omni_b200.ops import OpsError
    heads, context, sessions = 2, 32, 3
    table, indptr = i32([4, 1, 0, 2, 5, 3]), i32([0, 2, 4, 6])
    at, slot = i32([3, 20, 9]), i32([4 * 16 + 3, 2 * 16 + 4, 1 << 20])
    qkv = rand((sessions, 3 * heads * 128), 41)
    kv = torch.zeros(6, heads, 2 * 16 * 128 + 2 * 16 * 4, dtype=torch.uint8, device="cuda")
    out = torch.zeros((sessions, heads * 128), dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    if in_one:
        ops.lm_decode_attend(qkv, kv, 6, at, slot, indptr, table, heads, -0.14, 0.1, context, out)
    else:
        ops.lm_rope_attend(qkv, kv, 6, at, slot, None, indptr, table, heads, -0.14, 0.1, context, out)
    with pytest.raises(OpsError):
        ops.sync()
    assert not kv[[0, 1, 3, 5]].any() and kv[4].any() and kv[2].any()


def test_decode_attention_calls_one_behind_the_other(ops):
    """A call's own token is a key of the next call, made without waiting for it."""
    hq, hk, d, n = 4, 2, 128, 40
    qkv = [rand((1, (hq + 2 * hk) * d), 50 + t) for t in range(n)]
    qn, kn, pages = rand((d,), 48, 0.2) + 1, rand((d,), 49, 0.2) + 1, i32([2, 0, 1])
    at = [(i32([t]), i32([int(pages[t // 16]) * 16 + t % 16]), i32([0, 3])) for t in range(n)]
    outs = []
    for wait in (True, False):
        kv = torch.zeros((3, hk, 2, 16, d), dtype=torch.bfloat16, device="cuda")
        out = torch.zeros((n, hq * d), dtype=torch.bfloat16, device="cuda")
        torch.cuda.synchronize()
        for t, (pos, slot, indptr) in enumerate(at):
            ops.decode_attend(qkv[t], qn, kn, kv, 3, pos, slot, indptr, pages, hq, hk, d, 1e-6, 1e6, out[t:t + 1])
            if wait:
                ops.sync()
        ops.sync()
        outs.append(out)
    assert torch.equal(outs[0], outs[1])


def attention64(q, kv, pages, length, hq, hk, d):
    """One row in float64 from the bf16 queries, keys and values the kernels read."""
    block = kv[pages.long()].double()
    k, v = (block[:, :, i].permute(1, 0, 2, 3).reshape(hk, -1, d)[:, :length] for i in range(2))
    p = torch.softmax(torch.einsum("hgd,hld->hgl", q.double().reshape(hk, hq // hk, d), k) / d ** 0.5, -1)
    return torch.einsum("hgl,hld->hgd", p, v).reshape(hq * d)


# Outputs that are not the bf16 nearest to float64's: an error of a few f32 ulp (2^-22) moves a value over a rounding boundary
# (2^-8 apart) in one of 2^13 cases, four times that where values cancel - 0.05 %. Sixteen-bit probabilities (2^-17): 0.2 %.
NOT_NEAREST = 5e-4


@pytest.mark.parametrize("hq,hk,d", [(16, 8, 128), (20, 4, 128), (8, 8, 64)])
@pytest.mark.parametrize("prompt", [False, True])
def test_attention_keeps_f32_probabilities(ops, hq, hk, d, prompt):
    n, length = (256, 256) if prompt else (96, 200)
    per = (length + 15) // 16
    rng = np.random.default_rng(d)
    table = rng.permutation(per if prompt else n * per).reshape(-1, per)
    at = list(range(n)) if prompt else [length - 1 - s % 9 for s in range(n)]
    page = [table[0] if prompt else table[s] for s in range(n)]
    pos, slot = i32(at), i32([int(page[s][at[s] // 16]) * 16 + at[s] % 16 for s in range(n)])
    qkv, qn, kn = rand((n, (hq + 2 * hk) * d), 61), rand((d,), 62, 0.2) + 1, rand((d,), 63, 0.2) + 1
    kv = rand((table.size, hk, 2, 16, d), 64)
    out, scalar = (torch.zeros((n, hq * d), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    q, kv2 = qkv.clone(), kv.clone()
    each, lists = i32([s * per for s in range(n + 1)]), i32(np.concatenate(page).tolist())
    torch.cuda.synchronize()
    ops.rope_attend(q, qn, kn, kv2, table.size, pos, slot, None, each, lists, hq, hk, d, 1e-6, 1e6, scalar)
    if prompt:
        ops.rope_attend(qkv, qn, kn, kv, table.size, pos, slot, i32([0] * n), i32([0, per]), i32(page[0].tolist()), hq, hk, d, 1e-6, 1e6, out)
    else:
        ops.decode_attend(qkv, qn, kn, kv, table.size, pos, slot, each, lists, hq, hk, d, 1e-6, 1e6, out)
    ops.sync()
    assert torch.equal(kv, kv2)
    want = torch.stack([attention64(q[s, :hq * d].reshape(hq, d), kv2, torch.tensor(page[s], device="cuda"), at[s] + 1, hq, hk, d) for s in range(n)])
    for got in (scalar, out):
        assert float((got != want.to(torch.bfloat16)).double().mean()) <= NOT_NEAREST


@pytest.mark.parametrize("rows", [1, 40, 300])
def test_swiglu_of_every_gate(ops, rows):
    """Each finite bf16 as the gate, the up channel 1: the result nearest to float64's, the last f32 bit apart at a tie."""
    v = torch.arange(0, 65536, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    v = v[torch.isfinite(v.float())].cuda()
    w = torch.zeros((2 * len(v), 64), dtype=torch.bfloat16, device="cuda")
    w[:len(v), 0], w[len(v):, 1] = v, 1
    x = torch.zeros((rows, 64), dtype=torch.bfloat16, device="cuda")
    x[:, :2] = 1
    y = torch.zeros((rows, len(v)), dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    ops.chain_gemm(w, x, y, swiglu=True)
    ops.sync()
    want = v.double() * torch.sigmoid(v.double())
    assert (y == y[0]).all()
    assert int((y[0] != want.to(torch.bfloat16)).sum()) <= 1
    # half a bf16 step of the value and 2^-22 of it for the f32 arithmetic; below the smallest normal f32 a step is fixed
    assert ((y[0].double() - want).abs() <= want.abs() * (2.0 ** -8 + 2.0 ** -22) + 2.0 ** -134).all()


def ring64(q, kv, pages, length, heads, scale):
    """One row of the FP8 ring in float64, from the bf16 query and the bytes and scales the kernels read."""
    block = kv[pages.long()].view(-1, heads, 2 * 16 * 128 + 2 * 16 * 4)
    byte = block[:, :, :4096].reshape(-1, heads, 2, 16, 128).view(torch.float8_e4m3fn).double()
    scales = block[:, :, 4096:].contiguous().view(torch.float32).view(-1, heads, 2, 16).double()
    k, v = ((byte[:, :, i] * scales[:, :, i, :, None]).permute(1, 0, 2, 3).reshape(heads, -1, 128)[:, :length] for i in range(2))
    p = torch.softmax(torch.einsum("hd,hld->hl", q.double().reshape(heads, 128), k) * scale, -1)
    return torch.einsum("hl,hld->hd", p, v).reshape(heads * 128)


# Both sides of the item counts at which the warps an item change (16, 8, 4, 2 and 1 of them, from few items to many), a last CTA
# that is not full among them. Full rings are 63 pages, so that every warp of sixteen takes three at least; the row's own page is
# the first, one in the middle and the last, of rings that are not full, full and wrapped. Token scales differ by 2^9 (keys, which
# keeps the scores below ten, as f32 sums need) and 2^16 (values); what lies behind a row's end is NaN; some queries are zero.
@pytest.mark.parametrize("heads", [1, 4])
@pytest.mark.parametrize("per_sm,more", [(1, 0), (1, 1), (2, 0), (2, 1), (4, 0), (4, 1), (8, 0), (8, 1)])
def test_fp8_ring_attention_keeps_f32_weights(ops, per_sm, more, heads):
    context, per = 1000, 63
    sessions = per_sm * torch.cuda.get_device_properties(0).multi_processor_count // heads + more
    rng = np.random.default_rng(sessions)
    table = rng.permutation(sessions * per).reshape(sessions, per)
    at = [[0, 5, 15, 16, 40, 255, 256, 500, 991, 992, 999, 1000, 1007, 1008, 1500, 1991, 1999, 2000, 2640][s % 19] for s in range(sessions)]
    slot = [int(table[s, p % context // 16]) * 16 + p % context % 16 for s, p in enumerate(at)]
    pages, indptr = torch.tensor(table, device="cuda"), i32([s * per for s in range(sessions + 1)])
    g = torch.Generator(device="cuda").manual_seed(sessions)
    kv = torch.empty((sessions * per, heads, 2 * 16 * 128 + 2 * 16 * 4), dtype=torch.uint8, device="cuda")
    for i in range(0, sessions * per, 4096):
        part = kv[i:i + 4096]
        part[:, :, :4096] = (torch.randn((len(part), heads, 4096), generator=g, device="cuda") * 40).to(torch.float8_e4m3fn).view(torch.uint8)
        e = torch.rand((len(part), heads, 32), generator=g, device="cuda")
        e[:, :, :16] = e[:, :, :16] * 9 - 14.5
        e[:, :, 16:] = e[:, :, 16:] * 16 - 14
        part[:, :, 4096:] = torch.exp2(e).view(torch.uint8)
    ends = torch.tensor([min(p + 1, context) for p in at], device="cuda")
    behind = torch.arange(per * 16, device="cuda").view(1, per, 16) >= ends.view(-1, 1, 1)  # [session, page, token]
    s_at, p_at, t_at = behind.nonzero(as_tuple=True)

    def plant(pool):
        lost = pages[s_at, p_at]
        for i in range(2):
            pool[:, :, :4096].view(-1, heads, 2, 16, 128)[lost, :, i, t_at] = 0x7f
            pool[:, :, 4096 + 64 * i:4160 + 64 * i].view(torch.int32)[lost, :, t_at] = 0x7fc00000
    qkv = rand((sessions, 3 * heads * 128), 161)
    qkv[7::19, :heads * 128] = 0
    qkv_b, kv_b = qkv.clone(), kv.clone()
    a, b = (torch.zeros((sessions, heads * 128), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    plant(kv)  # (the scalar kernel wants numbers there)
    torch.cuda.synchronize()
    coef, scale, lists = float(np.float32(-np.log(10000.0) * 2.0 / 128)), 128 ** -0.5, i32(table.ravel().tolist())
    ops.lm_decode_attend(qkv, kv, sessions * per, i32(at), i32(slot), indptr, lists, heads, coef, scale, context, a)
    ops.lm_rope_attend(qkv_b, kv_b, sessions * per, i32(at), i32(slot), None, indptr, lists, heads, coef, scale, context, b)
    ops.sync()
    rows = rng.permutation(sessions)[:160]
    want = torch.stack([ring64(qkv_b[s, :heads * 128], kv_b, pages[s], min(at[s] + 1, context), heads, scale) for s in rows])
    close(a, b, steps=1.5, floor=0.25)
    plant(kv_b)
    assert torch.equal(kv, kv_b)
    # as NOT_NEAREST, for scores up to ten instead of two or three: twice the error, two to four times the rounding boundaries crossed
    for got in (a, b):
        assert float((got[torch.tensor(rows, device="cuda")] != want.to(torch.bfloat16)).double().mean()) <= 2 * NOT_NEAREST


@pytest.mark.parametrize("lens,broken", [([10, 9], 0), ([10, 9], 1), ([33, 5, 40], 1), ([3, 3, 3, 3], 2)])
def test_prompts_of_a_tile_do_not_touch_one_another(ops, lens, broken):
    """One sequence's values are infinite: the others, in the same tiles of rows, give what they give beside a sound one."""
    hq, hk, d, n = 4, 2, 128, sum(lens)
    per = [(x + 15) // 16 for x in lens]
    first = np.cumsum([0] + per)
    table = np.random.default_rng(n).permutation(int(first[-1]))
    where = [(s, t) for s, x in enumerate(lens) for t in range(x)]
    pos, seq = i32([t for _, t in where]), i32([s for s, _ in where])
    slot = i32([int(table[first[s] + t // 16]) * 16 + t % 16 for s, t in where])
    qkv, qn, kn = rand((n, (hq + 2 * hk) * d), 71), rand((d,), 72, 0.2) + 1, rand((d,), 73, 0.2) + 1
    outs = []
    for bad in (False, True):
        x = qkv.clone()
        if bad:
            x[seq == broken, (hq + hk) * d:] = float("inf")
        kv = torch.zeros((len(table), hk, 2, 16, d), dtype=torch.bfloat16, device="cuda")
        out = torch.zeros((n, hq * d), dtype=torch.bfloat16, device="cuda")
        torch.cuda.synchronize()
        ops.rope_attend(x, qn, kn, kv, len(table), pos, slot, seq, i32(first.tolist()), i32(table.tolist()), hq, hk, d, 1e-6, 1e6, out)
        ops.sync()
        outs.append(out)
    others = seq != broken
    assert torch.equal(outs[0][others], outs[1][others])


@pytest.mark.parametrize("dim", [128, 320, 2112, 4160, 8192])
def test_norms_of_rows_that_end_inside_a_warp(ops, dim):
    x, y, gain = rand((3, dim), 81), rand((3, dim), 82), rand((dim,), 83, 0.2) + 1
    out, res, out2 = (torch.zeros((3, dim), dtype=torch.bfloat16, device="cuda") for _ in range(3))
    res2 = y.clone()
    torch.cuda.synchronize()
    ops.norm_copy(x, gain, out, res, 1e-6)
    ops.add_norm(x, res2, gain, out2, 1e-6)
    ops.sync()

    def norm(v):
        return v * torch.rsqrt((v * v).mean(1, keepdim=True) + 1e-6) * gain.float()
    close(out, norm(x.float()), steps=1.0)
    close(out2, norm(x.float() + y.float()), steps=1.0)
    if dim >= 256:
        z = y.clone()
        torch.cuda.synchronize()
        ops.lm_norm(x, gain, out, 1e-6)
        ops.lm_norm(z, gain, out2, 1e-6, y=x)
        ops.sync()
        close(out, norm(x.float()), steps=1.0)
        close(out2, norm((x.float() + y.float()).bfloat16().float()), steps=1.0)


@pytest.mark.parametrize("vocab", [2047, 2048, 2049, 32768, 40001])
@pytest.mark.parametrize("top_k", [1, 5, 250])
def test_duplex_sampler_keeps_the_top_k(ops, vocab, top_k):
    """Nearly flat logits, where the noise decides: every draw is one of the top k (ties with the k-th included) and the one
    the host's restatement of the hash and the score takes (`__logf` against `logf` may move a near-tie)."""
    from oracle import duplex as O
    rows, col = 64, 2
    logits = (torch.rand((rows, vocab), generator=torch.Generator().manual_seed(vocab + top_k)) * 0.5 - 0.25).to(torch.bfloat16).cuda()
    force = torch.full((rows, 9), -1, dtype=torch.int32, device="cuda")
    drawn = torch.full((rows, 9), -7, dtype=torch.int32, device="cuda")
    seeds = [[r * 7919 + 1, r % 3] for r in range(rows)]
    torch.cuda.synchronize()
    ops.lm_sample(logits, 0.8, top_k, force, i32(seeds), col, drawn)
    ops.sync()
    got, host = drawn[:, col].cpu().numpy(), logits.float().cpu().numpy()
    kth = np.sort(host, axis=1)[:, -top_k]
    assert (host[np.arange(rows), got] >= kth).all()
    want = np.array([O.sample(host[r], 0.8, top_k, seeds[r][0], seeds[r][1], col) for r in range(rows)])
    assert (got == want).sum() >= rows - 1, (got, want)


@pytest.mark.parametrize("vocab", [16, 1000, 2048, 3072, 4093])
@pytest.mark.parametrize("top_k,top_p", [(50, 1.0), (0, 1.0), (40, 0.8), (1, 1.0)])
def test_rows_without_a_penalty_draw_what_the_general_path_draws(ops, vocab, top_k, top_p):
    """Unpenalised rows take sixteen-bit keys; a penalty of 1 over an empty bitmap takes the general path on the same logits,
    infinities, NaN, ties and one-signed rows among them. Also from an address that vector loads cannot take."""
    if top_p < 1 and top_k <= 0:
        pytest.skip("refused")
    rows, group = 64, 3
    x = rand((rows, vocab), vocab + top_k, 2.0)
    x[1], x[2], x[3] = -x[1].abs() - 1, 0.0, -float("inf")
    x[4, 3], x[5, 3], x[6, 3] = float("nan"), float("inf"), -float("inf")
    x[7] = torch.where(torch.arange(vocab, device="cuda") % 2 == 0, x[7].abs(), -x[7].abs())
    x[8], x[9, :] = (x[8] * 4).round() / 4, torch.tensor(-0.0, device="cuda")
    x[10, ::5], x[11, : vocab // 2] = float("nan"), -float("inf")
    x[12] = x[12] * 1e30
    x[13] = -x[13].abs() - 1
    x[13, :3] = x[13, :3].abs()
    bits = x.view(torch.int16)
    bits[14, 3], bits[15, 3], bits[16, ::5] = 0x7fc0, 0x7fc0 - 0x8000, 0x7fff  # NaN of either sign
    odd = torch.empty(rows * vocab + 1, dtype=torch.bfloat16, device="cuda")[1:].view(rows, vocab).copy_(x)
    stride = 4 * (16 + (vocab + 31) // 32 + 1) + 8
    stride = (stride + 255) // 256 * 256
    frames, uniforms = i32([2] * rows), torch.rand((rows, 16), generator=torch.Generator().manual_seed(vocab)).cuda()
    force, lines = torch.full((rows, 16), -1, dtype=torch.int32, device="cuda"), i32(list(range(rows)))
    got = []
    for logits, penalize in ((x, 1), (x, 0), (odd, 0)):
        state = torch.zeros((rows, stride // 4), dtype=torch.int32, device="cuda")
        codes = torch.full((rows, 16), -9, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        ops.sample(logits, 0.9, top_k, top_p, 1.0, 0, 0, -1, 0, frames, uniforms, force, state, lines, stride, penalize, 0, codes, group)
        ops.sync()
        got.append(codes[:, group].tolist())
    assert got[0] == got[1] == got[2]


@pytest.mark.parametrize("prompt", [False, True])
def test_attention_from_addresses_that_vector_loads_cannot_take(ops, prompt):
    hq, hk, d, n = 4, 2, 128, 20
    pos, slot = i32(list(range(n))), i32(list(range(n)))
    seq, indptr, pages = (i32([0] * n), i32([0, 2]), i32([0, 1])) if prompt else (None, i32([2 * s for s in range(n + 1)]), i32([0, 1] * n))
    x, qn, kn = rand((n, (hq + 2 * hk) * d), 91), rand((d,), 92, 0.2) + 1, rand((d,), 93, 0.2) + 1

    def at(offset, like):
        return torch.empty(like.numel() + 8, dtype=torch.bfloat16, device="cuda")[offset:offset + like.numel()].view(like.shape).copy_(like)
    got = []
    for offset in (0, 1):
        qkv, out = at(offset, x), at(offset, torch.zeros((n, hq * d), dtype=torch.bfloat16, device="cuda"))
        kv = torch.zeros((2, hk, 2, 16, d), dtype=torch.bfloat16, device="cuda")
        torch.cuda.synchronize()
        ops.rope_attend(qkv, qn, kn, kv, 2, pos, slot, seq, indptr, pages, hq, hk, d, 1e-6, 1e6, out)
        ops.sync()
        got.append((qkv, out, kv))
    for a, b in zip(*got):
        assert torch.equal(a, b)


def test_operands_that_vector_accesses_cannot_take_are_refused(ops):
    from pega_omni_b200.ops import OpsError
    w, x = rand((128, 64), 1), rand((300, 64), 2)
    y = torch.zeros(300 * 64 + 1, dtype=torch.bfloat16, device="cuda")[1:].view(300, 64)
    for rows in (40, 300):
        with pytest.raises(OpsError):
            ops.chain_gemm(w, x[:rows], y[:rows], swiglu=True)
    qkv = torch.zeros(3 * 2 * 128 + 1, dtype=torch.bfloat16, device="cuda")[1:].view(1, -1)
    kv = torch.zeros(1, 2, 2 * 16 * 128 + 2 * 16 * 4, dtype=torch.uint8, device="cuda")
    out = torch.zeros((1, 256), dtype=torch.bfloat16, device="cuda")
    for call in (ops.lm_decode_attend, lambda q, k, n, p, s, *rest: ops.lm_rope_attend(q, k, n, p, s, None, *rest)):
        with pytest.raises(OpsError):
            call(qkv, kv, 1, i32([0]), i32([0]), i32([0, 1]), i32([0]), 2, -0.14, 0.1, 16, out)
    ops.sync()
