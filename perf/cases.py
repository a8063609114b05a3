"""The work that users of this library have it do, as measurable cases.

A case is one call (or one short run of calls) of the public entry points on inputs that a decoding program has in hand:
quantised weights, a key/value cache with its block table, a decode stack.  Sizes are those of the benchmark
configurations (hidden 4096, intermediate 14336, 32 query / 8 kv heads of 128, pages of 16 tokens, contexts up to 8192),
of the reference's own benchmark commands (intermediate 11008, group size 32), and odd ones in between.

Activations and K/V are N(0, 1), weights N(0, 0.02) quantised affine per group; everything is made on the GPU from a
seed.  Lengths of ragged batches are spread evenly over their range, in an order drawn from the seed, so that the bytes
of a pass are known.
"""
import importlib
import math

import torch

import __graft_entry__

__graft_entry__.load_package()


def _module(name):
    return importlib.import_module("mlx_metal_kernels_b200." + name)


quant_ops = _module("ops.quant_ops")
mlp_ops = _module("ops.mlp_block_ops")
paged_quantized_ops = _module("ops.paged_quantized_kv_ops")
gqa_ops = _module("ops.gqa_ops")
sparse_ops = _module("ops.sparse_attention_ops")
stack_mod = _module("stack")
synth = _module("synth")

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
HEAD_DIM, PAGE = 128, 16
STACK_VOCAB = 1024        # rows of the embedding table: only the rows of the given token ids are read
STACK_STEPS = 4           # decode steps of one pass of a stack case


def listed():
    return [
        # one projection of one token (the attention output projection of an 8B-sized model): the smallest call
        dict(name="matvec_q4_b1", op="matvec", bits=4, batch=1, n=4096, k=4096, group=64, dtype="fp16"),
        # an 8-bit up projection for a small batch of sequences
        dict(name="matvec_q8_b8", op="matvec", bits=8, batch=8, n=14336, k=4096, group=64, dtype="fp16"),
        # a projection whose sizes fit no tile, in bf16, with the default group size
        dict(name="matvec_q4_b3_odd_bf16", op="matvec", bits=4, batch=3, n=5003, k=2592, group=32, dtype="bf16"),
        # the MLP block of one decoded token, of a full decode batch, and of a chunk of prompt tokens
        dict(name="mlp_q4_b1", op="mlp", bits=4, batch=1, tokens=1, hidden=4096, inter=14336, group=64, dtype="fp16"),
        dict(name="mlp_q4_b32", op="mlp", bits=4, batch=32, tokens=1, hidden=4096, inter=14336, group=64, dtype="fp16"),
        dict(name="mlp_q4_prompt256", op="mlp", bits=4, batch=4, tokens=64, hidden=4096, inter=11008, group=32, dtype="fp16"),
        # decode attention of a serving batch with ragged contexts over shuffled pages, and of a single sequence
        dict(name="attention_q4_b16_ragged", op="attention", bits=4, batch=16, min_len=1024, max_len=8192, q_heads=32, kv_heads=8,
             group=32, dtype="fp16", window=0),
        dict(name="attention_q8_b1", op="attention", bits=8, batch=1, min_len=4096, max_len=4096, q_heads=32, kv_heads=8,
             group=32, dtype="fp16", window=0),
        # decode attention over pages that are not quantised
        dict(name="attention_pages_bf16_b16", op="attention_pages", batch=16, min_len=1024, max_len=4096, q_heads=32, kv_heads=8,
             dtype="bf16"),
        # the key/value pages of freshly computed prompts: quantised into the cache, and read back
        dict(name="kv_pages_q8", op="kv_pages", bits=8, pages=2048, kv_heads=8, group=32, dtype="fp16"),
        # decode steps of the whole stack: one sequence, and a full batch
        dict(name="stack_b1", op="stack", batch=1, context=4096, layers=32),
        dict(name="stack_b32", op="stack", batch=32, context=4096, layers=32),
    ]


def _log_int(rng, lo, hi, multiple=1):
    """An integer in [lo, hi], spread over the logarithm, rounded down to a multiple."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, v)) // multiple * multiple


def draw(rng):
    op = rng.choice(["matvec", "matvec", "mlp", "mlp", "attention", "attention", "attention_pages", "kv_pages", "stack"])
    dtype = rng.choice(["fp16", "fp16", "bf16"])
    bits = rng.choice([4, 4, 8])
    if op == "matvec":
        group = rng.choice([32, 64, 64, 128])
        return dict(op=op, bits=bits, batch=_log_int(rng, 1, 64), n=_log_int(rng, 1024, 16384),
                    k=_log_int(rng, 1024, 14336, group), group=group, dtype=dtype)
    if op == "mlp":
        batch, tokens = rng.choice([(_log_int(rng, 1, 64), 1), (_log_int(rng, 1, 4), _log_int(rng, 8, 64))])
        return dict(op=op, bits=bits, batch=batch, tokens=tokens, hidden=_log_int(rng, 1024, 4096, 128),
                    inter=_log_int(rng, 2816, 14336, 128), group=rng.choice([32, 64, 64, 128]), dtype=dtype)
    if op in ("attention", "attention_pages"):
        batch = _log_int(rng, 1, 32)
        kv_heads = rng.choice([2, 4, 8, 8])
        longest = _log_int(rng, 128, 8192)
        case = dict(op=op, batch=batch, min_len=max(1, longest // rng.choice([1, 4, 8])), max_len=longest,
                    q_heads=kv_heads * rng.choice([1, 4, 4, 8]), kv_heads=kv_heads, dtype=dtype)
        if op == "attention":
            case.update(bits=bits, group=rng.choice([32, 32, 64]), window=rng.choice([0, 0, 1024]))
        return case
    if op == "kv_pages":
        return dict(op=op, bits=bits, pages=_log_int(rng, 16, 2048), kv_heads=rng.choice([2, 4, 8]), group=rng.choice([32, 64]),
                    dtype=dtype)
    return dict(op=op, batch=_log_int(rng, 1, 32), context=_log_int(rng, 256, 4096), layers=rng.choice([4, 8, 16]))


# ---- inputs ---------------------------------------------------------------------------------------------------------
class _Source:
    """Random tensors on the GPU from one seed."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, *shape, dtype=torch.float16, std=1.0):
        return (torch.randn(shape, generator=self.gen, device="cuda") * std).to(dtype)

    def weight(self, n, k, bits, group):
        w = torch.randn((n, k), generator=self.gen, device="cuda") * 0.02
        return synth.quantize_affine(w, bits, group)

    def order(self, n):
        return torch.randperm(n, generator=self.gen, device="cuda")


def _lengths(case):
    b, lo, hi = case["batch"], case["min_len"], case["max_len"]
    return [hi] if b == 1 else [lo + (hi - lo) * i // (b - 1) for i in range(b)]


def _block_table(case, src):
    """(block table [B, max_blocks], lengths [B], pages in the pool): pages of all sequences shuffled over one pool."""
    lengths = torch.tensor(_lengths(case), dtype=torch.int32, device="cuda")[src.order(case["batch"])].contiguous()
    blocks = (lengths + PAGE - 1) // PAGE
    max_blocks = (case["max_len"] + PAGE - 1) // PAGE
    total = sum((n + PAGE - 1) // PAGE for n in _lengths(case))
    pool = total + total // 16 + 1
    col = torch.arange(max_blocks, device="cuda").reshape(1, -1)
    used = col < blocks.reshape(-1, 1)
    rank = torch.cumsum(used.reshape(-1), 0).reshape(used.shape) - 1
    table = torch.where(used, src.order(pool)[rank.clamp(0)], -1).to(torch.int32)
    return table.contiguous(), lengths, pool


def prepare(case, seed):
    src = _Source(seed)
    return globals()["_prepare_" + case["op"]](case, src, seed)


def _prepare_matvec(case, src, seed):
    w, s, z = src.weight(case["n"], case["k"], case["bits"], case["group"])
    x = src.normal(case["batch"], case["k"], dtype=DTYPES[case["dtype"]])
    return dict(op="matvec", fn=quant_ops.q4_matvec_decode if case["bits"] == 4 else quant_ops.q8_matvec_decode, x=x, w=w, s=s, z=z,
                group=case["group"])


def _prepare_mlp(case, src, seed):
    shape = (case["batch"], case["tokens"], case["hidden"])
    dtype = DTYPES[case["dtype"]]
    mats = [src.weight(n, k, case["bits"], case["group"])
            for n, k in ((case["inter"], case["hidden"]), (case["inter"], case["hidden"]), (case["hidden"], case["inter"]))]
    norm = (1.0 + src.normal(case["hidden"], dtype=torch.float32, std=0.1)).to(torch.float16)
    return dict(op="mlp", x=src.normal(*shape, dtype=dtype), residual=src.normal(*shape, dtype=dtype), norm=norm, mats=mats,
                bits=case["bits"], group=case["group"])


def _prepare_attention(case, src, seed):
    table, lengths, pool = _block_table(case, src)
    shape = (pool, PAGE, case["kv_heads"], HEAD_DIM)
    (kq, ks), (vq, vs) = (synth.quantize_kv_symmetric(src.normal(*shape, dtype=torch.float32), case["bits"], case["group"])
                          for _ in range(2))
    cache = paged_quantized_ops.PagedQuantizedKVCache(
        k_pages_q=kq, v_pages_q=vq, k_scales=ks, v_scales=vs, block_table=table, lengths=lengths, bits=case["bits"],
        page_size=PAGE, group_size=case["group"], original_page_shape=shape)
    q = src.normal(case["batch"], 1, case["q_heads"], HEAD_DIM, dtype=DTYPES[case["dtype"]])
    pattern = None
    if case["window"]:
        pattern = sparse_ops.SparseAttentionPattern("sliding_window_sink", window_size=case["window"], sink_tokens=4)
    return dict(op="attention", q=q, cache=cache, pattern=pattern)


def _prepare_attention_pages(case, src, seed):
    table, lengths, pool = _block_table(case, src)
    dtype = DTYPES[case["dtype"]]
    k, v = (src.normal(pool, PAGE, case["kv_heads"], HEAD_DIM, dtype=dtype) for _ in range(2))
    q = src.normal(case["batch"], 1, case["q_heads"], HEAD_DIM, dtype=dtype)
    return dict(op="attention_pages", q=q, k=k, v=v, table=table, lengths=lengths)


def _prepare_kv_pages(case, src, seed):
    shape = (case["pages"], PAGE, case["kv_heads"], HEAD_DIM)
    k, v = (src.normal(*shape, dtype=DTYPES[case["dtype"]]) for _ in range(2))
    table = torch.arange(case["pages"], dtype=torch.int32, device="cuda").reshape(1, -1)
    lengths = torch.tensor([case["pages"] * PAGE], dtype=torch.int32, device="cuda")
    config = paged_quantized_ops.PagedQuantizedKVConfig(bits=case["bits"], page_size=PAGE, group_size=case["group"])
    return dict(op="kv_pages", k=k, v=v, table=table, lengths=lengths, config=config)


def _prepare_stack(case, src, seed):
    cfg = stack_mod.StackConfig(n_layers=case["layers"], vocab=STACK_VOCAB)
    layers = [stack_mod.random_layer(cfg, seed + 7919 * i, "cuda") for i in range(case["layers"])]
    embedding = src.normal(STACK_VOCAB, cfg.hidden)
    stack = stack_mod.DecodeStack(cfg, layers, torch.ones(cfg.hidden, dtype=torch.float16, device="cuda"), embedding,
                                  case["batch"], case["context"] + STACK_STEPS + PAGE, "cuda")
    stack.set_context(case["context"], seed)
    stack.capture()
    ids = torch.randint(0, STACK_VOCAB, (STACK_STEPS, case["batch"]), generator=src.gen, device="cuda")
    return dict(op="stack", stack=stack, ids=ids, context=case["context"])


# ---- one pass -------------------------------------------------------------------------------------------------------
def run(state):
    return globals()["_run_" + state["op"]](state)


def _run_matvec(st):
    return st["fn"](st["x"], st["w"], st["s"], st["z"], group_size=st["group"], backend="cuda")


def _run_mlp(st):
    (gw, gs, gz), (uw, us, uz), (dw, ds, dz) = st["mats"]
    return mlp_ops.quantized_mlp_block(st["x"], st["residual"], st["norm"], gw, gs, uw, us, dw, ds, gate_zeros=gz, up_zeros=uz,
                                       down_zeros=dz, bits=st["bits"], group_size=st["group"], backend_preset="cuda")


def _run_attention(st):
    if st["pattern"] is not None:
        return paged_quantized_ops.sparse_paged_quantized_kv_gqa_decode_attention(st["q"], st["cache"], st["pattern"])
    return paged_quantized_ops.paged_quantized_kv_gqa_decode_attention(st["q"], st["cache"], backend="cuda")


def _run_attention_pages(st):
    return gqa_ops.paged_gqa_decode_attention(st["q"], st["k"], st["v"], st["table"], st["lengths"])


def _run_kv_pages(st):
    cache = paged_quantized_ops.quantize_kv_pages(st["k"], st["v"], st["table"], st["lengths"], st["config"])
    k, v = paged_quantized_ops.dequantize_kv_pages(cache)
    return cache.k_pages_q, cache.v_pages_q, cache.k_scales, cache.v_scales, k, v


def _run_stack(st):
    """A few decode steps from the same context: the rows of each step, and the cache of the last layers, which holds
    the tokens that were appended."""
    stack = st["stack"]
    stack.positions.fill_(st["context"])
    stack.lengths.fill_(st["context"] + 1)
    hidden = [stack.step(ids).clone() for ids in st["ids"]]
    caches = [(c.k_codes, c.v_codes, c.k_scales, c.v_scales) for c in stack.caches[-8:]]
    return {"hidden": hidden, "caches": caches}


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
def _matrix_bytes(n, k, bits, group):
    return n * k * bits // 8 + n * -(-k // group) * 4


def work(case):
    op = case["op"]
    if op == "matvec":
        b, n, k = case["batch"], case["n"], case["k"]
        return {"bytes": _matrix_bytes(n, k, case["bits"], case["group"]) + 2 * b * (k + n), "flops": 2 * b * n * k}
    if op == "mlp":
        rows, h, m = case["batch"] * case["tokens"], case["hidden"], case["inter"]
        weights = 2 * _matrix_bytes(m, h, case["bits"], case["group"]) + _matrix_bytes(h, m, case["bits"], case["group"])
        return {"bytes": weights + 2 * h + 3 * 2 * rows * h, "flops": 6 * rows * h * m}
    if op in ("attention", "attention_pages"):
        window = case.get("window", 0)
        tokens = sum(min(n, window + 4) if window else n for n in _lengths(case))
        if op == "attention":
            row = 2 * case["kv_heads"] * (HEAD_DIM * case["bits"] // 8 + HEAD_DIM // case["group"] * 2)
        else:
            row = 2 * case["kv_heads"] * HEAD_DIM * 2
        q_bytes = 2 * 2 * case["batch"] * case["q_heads"] * HEAD_DIM
        return {"bytes": tokens * row + tokens // PAGE * 4 + q_bytes, "flops": 4 * tokens * case["q_heads"] * HEAD_DIM}
    if op == "kv_pages":
        values = 2 * case["pages"] * PAGE * case["kv_heads"] * HEAD_DIM
        coded = values * case["bits"] // 8 + values // case["group"] * 2
        return {"bytes": 2 * values + 2 * coded + 2 * values, "flops": 4 * values}
    cfg = stack_mod.StackConfig()
    b, ctx = case["batch"], case["context"]
    shapes = ((cfg.hidden + 2 * cfg.n_kv_heads * cfg.head_dim, cfg.hidden), (cfg.hidden, cfg.hidden), (cfg.intermediate, cfg.hidden),
              (cfg.intermediate, cfg.hidden), (cfg.hidden, cfg.intermediate))
    weights = sum(_matrix_bytes(n, k, cfg.bits, cfg.group_size) for n, k in shapes)
    kv = b * ctx * 2 * cfg.n_kv_heads * (cfg.head_dim + cfg.head_dim // cfg.kv_group_size * 2)
    flops = 2 * b * sum(n * k for n, k in shapes) + 4 * b * ctx * cfg.n_heads * cfg.head_dim
    return {"bytes": STACK_STEPS * case["layers"] * (weights + kv), "flops": STACK_STEPS * case["layers"] * flops}


def tolerance(case):
    """fp16 results of one contraction agree to 1e-3 (weights rounded to fp16 or not, fp32 sums), a block of two to
    2e-3; bf16 results to 6e-3 and 1e-2.  Quantised pages and their dequantisation are exact.  Through the layers of a
    stack the fp16 roundings add up to 1e-2, and a code of an appended row may then fall on the other side of a tie."""
    op = case["op"]
    if op == "kv_pages":
        return "exact"
    if op == "stack":
        return {"rel": 1e-2, "differ": 5e-3 if case["context"] < 1024 else 1e-3}
    fp16 = case["dtype"] == "fp16"
    if op == "mlp":
        return {"rel": 2e-3 if fp16 else 1e-2}
    return {"rel": 1e-3 if fp16 else 6e-3}
