"""The work a serving engine has the paged-KV path do, as cases that can be timed one by one.

A case is one engine step (or the part of it that this library does): every layer's K/V append and
attention over a fragmented block pool, with the planning and index building that come once a step.

  decode   one new token per sequence: the split-K plan from the host copy of the positions, then
           one captured graph of all layers (plan upload, append and attention), replayed
  engine   what an unmodified llm-engine runs through the exported launchers: per layer the append and
           ONE attention call over prefill slices and decode tokens together; a decode-only step is
           captured, a step with prefill slices (whose shape is never the same twice) is launched
  prefill  chunks of prompts: per layer rope and append in one pass, then the prefill kernel
  prefix   sequences that share a cached prompt: one wave of copy-on-write block copies over every
           pool, the step's index arrays built on the device, then the captured layers
  copy     the block copies alone

Head counts are those of Qwen2.5-0.5B (14 query heads, 2 kv heads, 64 dims) and TinyLlama-1.1B (32, 4,
64), the two models the benchmark configurations use, and a generic (32, 8, 128).  Lengths follow the
case alone, so that every seed costs the same; values, tables and the order of the lengths follow
the seed.  Pools hold what the step needs and a sixteenth more, in shuffled order.
"""
import importlib

import numpy as np
import torch

pkv = importlib.import_module("llm-engine_b200")

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
QWEN = {"q_heads": 14, "kv_heads": 2, "head_dim": 64}
TINY = {"q_heads": 32, "kv_heads": 4, "head_dim": 64}
WIDE = {"q_heads": 32, "kv_heads": 8, "head_dim": 128}


def _case(kind, heads, dtype, layers, block=16, seqs=0, ctx=(0, 0), chunks=0, new=(0, 0), past=0, shared=0, lengths=1):
    """seqs sequences decode one token each over ctx = (shortest, longest) cached tokens (lengths spread
    over their logarithm, `shared` leading tokens in common); chunks sequences bring new = (shortest,
    longest) prompt tokens each on top of up to `past` cached ones."""
    return {"kind": kind, **heads, "dtype": dtype, "layers": layers, "block": block, "seqs": seqs, "ctx_lo": ctx[0],
            "ctx_hi": ctx[1], "chunks": chunks, "new_lo": new[0], "new_hi": new[1], "past_hi": past, "shared": shared,
            "lengths": lengths}


def listed():
    return [
        # a chat with one user: nothing but latency, 24 dependent layers
        {"name": "decode_one", **_case("decode", QWEN, "bf16", 24, seqs=1, ctx=(333, 333))},
        # a moderately loaded server (benchmark configuration 2)
        {"name": "decode_64", **_case("decode", QWEN, "bf16", 24, seqs=64, ctx=(256, 2048), lengths=2)},
        # a full server with very different histories (benchmark configuration 3, six of its 22 layers)
        {"name": "decode_256", **_case("decode", TINY, "bf16", 6, seqs=256, ctx=(128, 8192), lengths=3)},
        # an odd batch on wider heads and larger blocks
        {"name": "decode_37_wide", **_case("decode", WIDE, "f16", 8, block=32, seqs=37, ctx=(100, 6000), lengths=4)},
        # fp32 K/V, the precision the reference's CPU engine checks against (configuration 1, all layers)
        {"name": "decode_f32", **_case("decode", QWEN, "f32", 24, seqs=8, ctx=(64, 512), lengths=5)},
        # the unmodified engine in a decode-only step
        {"name": "engine_decode", **_case("engine", TINY, "f16", 22, seqs=48, ctx=(32, 1500), lengths=6)},
        # the unmodified engine with two prompts being prefilled next to running sequences
        {"name": "engine_mixed", **_case("engine", QWEN, "f16", 24, seqs=20, ctx=(100, 2000), chunks=2, new=(300, 300), past=1200, lengths=7)},
        # a few fresh prompts of everyday length arriving together
        {"name": "prefill_prompts", **_case("prefill", QWEN, "f16", 24, chunks=9, new=(17, 400), lengths=8)},
        # chunked prefill of 32 sequences (benchmark configuration 4, four layers)
        {"name": "prefill_chunks", **_case("prefill", QWEN, "bf16", 4, chunks=32, new=(512, 512), past=1536, lengths=9)},
        # the last chunk of one long document
        {"name": "prefill_long", **_case("prefill", TINY, "bf16", 4, chunks=1, new=(2048, 2048), past=6144, lengths=10)},
        # prefix cache: first divergent step of 128 sequences behind a common prompt (configuration 5)
        {"name": "prefix_step", **_case("prefix", TINY, "bf16", 22, seqs=128, ctx=(544, 768), shared=512, lengths=11)},
        # copy-on-write alone: 127 forked sequences, each with its own block to leave, on every layer's pools
        {"name": "copy_wave", **_case("copy", TINY, "bf16", 22, seqs=128, ctx=(544, 768), shared=512, lengths=11)},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "engine", "engine", "prefill", "prefill", "prefix", "copy"])
    lengths = rng.randrange(1, 1 << 20)
    if kind == "prefill":
        heads = rng.choice([QWEN, TINY])
        new_hi = _log_int(rng, 16, 2048)
        c = _case(kind, heads, rng.choice(["bf16", "f16"]), 24, chunks=_log_int(rng, 1, 32),
                  new=(max(1, new_hi // rng.randrange(1, 24)), new_hi), past=rng.choice([0, _log_int(rng, 16, 6144)]), lengths=lengths)
    elif kind == "engine":
        hi = _log_int(rng, 64, 4096)
        c = _case(kind, rng.choice([QWEN, TINY]), "f16", 22, seqs=_log_int(rng, 1, 128), ctx=(max(1, hi // rng.randrange(1, 32)), hi), lengths=lengths)
        if rng.random() < 0.6:
            c.update(chunks=rng.randrange(1, 5), new_hi=_log_int(rng, 17, 512), past_hi=rng.choice([0, 300, 1200]))
            c["new_lo"] = max(1, c["new_hi"] // rng.randrange(1, 5))
    elif kind in ("prefix", "copy"):
        shared = 16 * _log_int(rng, 4, 512)
        c = _case(kind, TINY, "bf16", 22, seqs=_log_int(rng, 2, 128), ctx=(shared + 17, shared + _log_int(rng, 32, 256)), shared=shared, lengths=lengths)
    else:
        hi = _log_int(rng, 64, 8192)
        dtype = rng.choice(["bf16", "bf16", "f16", "f32"])
        c = _case(kind, rng.choice([QWEN, TINY, WIDE]), dtype, 24, block=rng.choice([16, 16, 32]),
                  seqs=_log_int(rng, 1, 32 if dtype == "f32" else 256), ctx=(max(1, hi // rng.randrange(1, 64)), hi), lengths=lengths)
    # as many layers as cost no more than the largest listed cases do
    while c["layers"] > 1 and not _affordable(c):
        c["layers"] -= 1
    while not _affordable(c):
        for k in ("seqs", "chunks"):
            c[k] = (c[k] + 1) // 2 if c[k] > 1 else c[k]
    return c


def _affordable(c):
    w = work(c)
    rows = c["layers"] * int(_lengths(c)[1].sum())
    pools = c["layers"] * 2 * _pool_blocks(c) * c["block"] * c["kv_heads"] * c["head_dim"]
    return w["bytes"] <= (2e8 if c["dtype"] == "f32" else 2.4e9) and w["flops"] <= 4.5e11 and rows <= 70000 and pools <= 1.9e9


def _lengths(c):
    """(cached tokens, new tokens, sharing) per sequence: prompt chunks first, then decode tokens."""
    rng = np.random.default_rng(c["lengths"])

    def spread(lo, hi, n):
        lo, hi = max(1, lo), max(1, lo, hi)
        return np.clip(np.round(np.exp(rng.uniform(np.log(lo), np.log(hi + 0.49), size=n))), lo, hi).astype(np.int64)

    new = np.concatenate([spread(c["new_lo"], c["new_hi"], c["chunks"]), np.ones(c["seqs"], np.int64)])
    past = rng.integers(0, c["past_hi"] + 1, size=c["chunks"]) if c["chunks"] != 1 else np.full(1, c["past_hi"])
    return np.concatenate([past.astype(np.int64), spread(c["ctx_lo"], c["ctx_hi"], c["seqs"])]), new


def _pool_blocks(c):
    ctx, new = _lengths(c)
    n = int(((ctx + new + c["block"] - 1) // c["block"]).sum()) - max(0, c["seqs"] - 1) * (c["shared"] // c["block"]) + c["seqs"]
    return n + n // 16 + 4


def work(c):
    """K and V of every attended token read once per kv head, q read and the result written, new K/V rows
    read and written to the pool, tables read; products of Q K^T and P V over the visible pairs."""
    ctx, new = _lengths(c)
    e, kv_dim, q_dim, n = (4 if c["dtype"] == "f32" else 2), c["kv_heads"] * c["head_dim"], c["q_heads"] * c["head_dim"], int(new.sum())
    forks, block_bytes = max(0, c["seqs"] - 1), 2 * c["block"] * kv_dim * e
    copies = {"prefix": (forks + 1) * block_bytes, "copy": 2 * forks * block_bytes}.get(c["kind"], 0)
    if c["kind"] == "copy":
        return {"bytes": c["layers"] * copies, "flops": 0}
    held = int((ctx + new).sum()) - max(0, c["seqs"] - 1) * c["shared"]
    rope = 2 * n * q_dim * e if c["kind"] == "prefill" else 0
    per_layer = 2 * held * kv_dim * e + 2 * n * q_dim * e + 4 * n * kv_dim * e + rope + copies
    tables = 4 * int(((ctx + new + c["block"] - 1) // c["block"]).sum()) + 16 * n
    pairs = int((new * ctx + new * (new + 1) // 2).sum())
    return {"bytes": c["layers"] * (per_layer + tables), "flops": c["layers"] * 4 * c["head_dim"] * c["q_heads"] * pairs}


def tolerance(c):
    if c["kind"] == "copy":
        return "exact"
    # four times what the path is off an fp64 evaluation of the same inputs: 2.4e-7, 2.9e-4 and 2.35e-3 at most
    return {"f32": {"rel": 1e-6}, "f16": {"rel": 1.1e-3}, "bf16": {"rel": 9.5e-3}}[c["dtype"]]


class _State:
    pass


def prepare(c, seed):
    s = _State()
    rng = np.random.default_rng([seed, c["lengths"]])
    gen = torch.Generator(device="cuda").manual_seed(seed * 1000003 + c["lengths"])
    ctx, new = _lengths(c)
    for part in (slice(0, c["chunks"]), slice(c["chunks"], None)):
        order = rng.permutation(len(ctx[part]))
        ctx[part], new[part] = ctx[part][order], new[part][order]
    bs, L, S, dt = c["block"], c["layers"], len(ctx), DTYPES[c["dtype"]]
    qh, kvh, hd = c["q_heads"], c["kv_heads"], c["head_dim"]
    nb, kv_dim, n = _pool_blocks(c), kvh * hd, int(new.sum())
    s.case, s.heads, s.n, s.bs, s.nb, s.L, s.scale = c, (qh, kvh, hd), n, bs, nb, L, hd ** -0.5
    # block tables dealt from a shuffled pool; sequences behind a common prompt start with its blocks
    ids = rng.permutation(nb).astype(np.int32)
    common, at, tables = c["shared"] // bs, c["shared"] // bs, []
    for k in (ctx + new + bs - 1) // bs:
        tables.append(np.concatenate([ids[:common], ids[at:at + k - common]]))
        at += k - common
    def normal(*shape):
        return torch.randn(shape, generator=gen, device="cuda", dtype=dt)

    def ints(a):
        return torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).cuda()

    s.pools = normal(L, 2, nb * bs, kv_dim)
    # copy-on-write: every sequence but the first moves its last, shared block to a free one
    own = [int(t[-1]) for t in tables]
    if c["kind"] in ("prefix", "copy"):
        for i in range(1, S):
            tables[i][-1] = ids[at]
            at += 1
        first = c["kind"] == "prefix"     # all behind one prompt leave the same block; forks of many, each its own
        s.pairs = ints([[own[0] if first else own[i], int(t[-1])] for i, t in enumerate(tables) if i > 0])
        s.pool_ptrs = torch.tensor([s.pools[l, i].data_ptr() for l in range(L) for i in (0, 1)], dtype=torch.int64, device="cuda")
        if c["kind"] == "copy":
            return s
    s.q, s.k, s.v = normal(L, n, qh * hd), normal(L, n, kv_dim), normal(L, n, kv_dim)
    s.out = torch.zeros_like(s.q)
    if c["kind"] == "prefix":
        s.ctx = ctx
        s.last = [(i, len(t) - 1, int(t[-1])) for i, t in enumerate(tables)]
        s.packer = pkv.DeviceStepPacker(S, max(len(t) for t in tables), bs, n, sum(len(t) for t in tables))
        for i, t in enumerate(tables):
            s.packer.set_table(i, t)
        s.packer.pack([(i, int(p), 1) for i, p in enumerate(ctx)], check=True)
        p = s.packer
        s.index = (p.tables, p.table_offset, p.token_seq, p.positions)
        s.slots = p.slots
    else:
        rows = np.repeat(np.arange(S), new)
        pos = np.concatenate([np.arange(a, a + b) for a, b in zip(ctx, new)]).astype(np.int32)
        idx = pkv.pack_step([tables[r] for r in rows], pos, bs, tok_keys=rows + 1)
        s.slots = ints(idx.slots)
        s.index = (ints(idx.block_tables), ints(idx.table_offset), ints(idx.token_seq), ints(idx.token_pos))
        s.host_pos = idx.token_pos
    if c["kind"] == "engine":
        s.workspace = torch.empty(pkv.mixed_workspace_bytes(n, *s.heads), dtype=torch.uint8, device="cuda")
    elif c["kind"] == "prefill":
        s.chunks = (ints(np.cumsum(new) - new), ints(new), ints(ctx))
        s.n_seqs, s.max_new = S, int(new.max())
        inv = 10000.0 ** (-torch.arange(0, hd, 2, device="cuda", dtype=torch.float64) / hd)
        angle = torch.arange(int((ctx + new).max()), device="cuda", dtype=torch.float64)[:, None] * inv
        s.cos, s.sin = angle.cos().float().contiguous(), angle.sin().float().contiguous()
    else:
        s.plan = pkv.DecodePlan(n, *s.heads, num_blocks=nb)
    if c["kind"] in ("decode", "prefix") or (c["kind"] == "engine" and c["chunks"] == 0):
        # a server captures the layers of a decode step once per batch size; the first call on a
        # device (look-ups, attributes) comes before the capture
        if c["kind"] == "decode":
            s.image = s.plan.build_host_image(s.host_pos)
        _layers(s)
        torch.cuda.synchronize()
        s.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s.graph):
            _layers(s)
        s.replayed = torch.cuda.Event()
        s.replayed.record()
    return s


def _layers(s):
    """Every layer's append and attention, on the current stream."""
    c = s.case
    kind, (qh, kvh, hd) = c["kind"], s.heads
    if kind == "decode":
        s.plan.workspace[:s.image].copy_(s.plan.staging[:s.image], non_blocking=True)
    elif kind == "prefix":
        s.plan.build_device(s.index[3][:s.n])
    for l in range(s.L):
        kc, vc, q, k, v, out = s.pools[l, 0], s.pools[l, 1], s.q[l], s.k[l], s.v[l], s.out[l]
        if kind == "prefix" or (kind == "decode" and c["dtype"] != "f32"):
            s.plan.append_attention(q, k, v, s.slots, kc, vc, *s.index, out, s.bs, s.scale)
        elif kind == "decode":
            pkv.launch_store_kv(k, v, s.slots, kc, vc, s.n, kvh * hd)
            s.plan.attention(q, kc, vc, *s.index, out, s.bs, s.scale)
        elif kind == "engine":
            pkv.launch_store_kv(k, v, s.slots, kc, vc, s.n, kvh * hd)
            pkv.launch_attention_mixed(q, kc, vc, *s.index, out, s.n, qh, kvh, hd, s.bs, s.scale, s.workspace)
        else:
            # q is rotated in place, as the forward pass has it: it comes fresh from a projection every
            # step there, and here from the pass before
            pkv.launch_rope_store_kv(q, k, v, s.index[3], s.cos, s.sin, s.slots, kc, vc, s.n, qh, kvh, hd)
            pkv.launch_attention_prefill(q, kc, vc, s.index[0], s.index[1], *s.chunks, out, s.n, s.n_seqs, s.max_new, qh, kvh, hd,
                                         s.bs, s.nb, s.scale)


def run(s):
    c = s.case
    if c["kind"] in ("prefix", "copy"):
        pkv.launch_copy_blocks_layers(s.pool_ptrs, 2 * s.L, s.pairs, s.pairs.shape[0], s.bs * c["kv_heads"] * c["head_dim"] * 2)
        if c["kind"] == "copy":
            return s.pools
        for row, index, block in s.last[1:]:
            s.packer.set_block(row, index, block)
        s.packer.pack([(i, int(p), 1) for i, p in enumerate(s.ctx)])
    elif c["kind"] == "decode":
        s.replayed.synchronize()      # the plan's staging buffer belongs to the last replay until it has run
        s.plan.build_host_image(s.host_pos)
    if c["kind"] in ("decode", "prefix") or (c["kind"] == "engine" and c["chunks"] == 0):
        s.graph.replay()
        s.replayed.record()
    else:
        _layers(s)
    return {"out": s.out, "pools": s.pools, "q": s.q} if c["kind"] == "prefill" else {"out": s.out, "pools": s.pools}
