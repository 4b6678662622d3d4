"""Timed cases of the numeric backend: what its users run, through the public entry points.

Six kinds of work, each with the sizes, formats and options it meets in use:

  prefill   flash-attention prefill (`attention_fa`): a short prompt, a chunk of a prompt behind an already cached
            prefix, the batch of long sequences of the benchmark, and the f32 attention block
  decode    flash-decoding (`attention_fd`): one sequence, and a serving batch over long KV caches
  gemm      a projection region with its epilogue (`gemm_epilogue`): a few token rows, ordinary and ragged sizes, 8192^3
  layer     decoder layer forward (`ShardedDecoderLayer.forward_fused`, one shard): one prompt, a batch of sequences
  commands  the command-level seam on host storage, as the functional model calls it: a GEMM, an elementwise, a convert
            and a reduce command, each consuming the result of the one before
  program   replay of per-Tile target modules (`TileProgram.run`): the online-attention command run on 1 to 16 Tiles

`listed()` gives fixed representatives; `draw()` gives further cases of the same ranges.
"""
import math

import numpy as np
import torch

from vibe_compiler_b200 import _abi as abi
from vibe_compiler_b200.backend import B200TargetModelBackend, FormalGemmOperation, NumericTensor, PhysicalTensorDescriptor
from vibe_compiler_b200.decoder_layer import LayerConfig, LayerWeights, ShardedDecoderLayer, layer_flops
from vibe_compiler_b200.tile_program import TileProgram

_DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
_FORMATS = {"bf16": abi.BF16, "f16": abi.F16, "f32": abi.F32}
_EPILOGUES = {"none": abi.EPI_NONE, "bias": abi.EPI_BIAS, "bias_gelu": abi.EPI_BIAS_GELU, "swiglu": abi.EPI_SWIGLU}
# (query heads, KV heads): the benchmark's multi-head and grouped forms, the 28-head block, narrow shards of them
_HEADS = ((32, 32), (32, 8), (28, 4), (28, 28), (16, 4), (8, 2), (8, 8))

_MAX_PREFILL_FLOPS = 4 * 128 * 4 * 32 * 4096 * 4097 // 2
_MAX_DECODE_KEYS = 64 * 8 * 32768          # (batch, KV head, key) triples of the largest decode
_MAX_GEMM = 8192 ** 3
_MAX_TOKENS = 8 * 2048

_backend_of_process = None


def _backend():
    """One backend per process, as a program holds it."""
    global _backend_of_process
    if _backend_of_process is None:
        _backend_of_process = B200TargetModelBackend(torch.cuda.current_device())
    return _backend_of_process


# ---------------------------------------------------------------------------------------------------------- the cases
def _prefill(name, batch, q_heads, kv_heads, q_len, prefix, head_dim, dtype, causal, lse, token_major):
    case = dict(kind="prefill", batch=batch, q_heads=q_heads, kv_heads=kv_heads, q_len=q_len, prefix=prefix, head_dim=head_dim,
                dtype=dtype, causal=causal, lse=lse, token_major=token_major)
    return dict(case, name=name) if name else case


def _decode(name, batch, q_heads, kv_heads, capacity, length, dtype, lse):
    case = dict(kind="decode", batch=batch, q_heads=q_heads, kv_heads=kv_heads, capacity=capacity, length=length, dtype=dtype, lse=lse)
    return dict(case, name=name) if name else case


def _gemm(name, m, n, k, dtype, epilogue, out, lhs_t, rhs_t):
    case = dict(kind="gemm", m=m, n=n, k=k, dtype=dtype, epilogue=epilogue, out=out, lhs_transposed=lhs_t, rhs_transposed=rhs_t)
    return dict(case, name=name) if name else case


def _layer(name, batch, seq, dtype, wide, offset):
    case = dict(kind="layer", batch=batch, seq=seq, dtype=dtype, wide=wide, position_offset=offset)
    return dict(case, name=name) if name else case


def _commands(name, m, k, n, dtype, tensor_policy):
    case = dict(kind="commands", m=m, k=k, n=n, dtype=dtype, tensor_policy=tensor_policy)
    return dict(case, name=name) if name else case


def _program(name, tiles, blocks):
    case = dict(kind="program", tiles=tiles, blocks=blocks)
    return dict(case, name=name) if name else case


def listed():
    return [
        # A single short chat prompt, grouped heads: latency of one small prefill.
        _prefill("prefill_short_prompt", 1, 32, 8, 333, 0, 128, "bf16", True, False, False),
        # Chunked prefill: 1000 new tokens behind 2051 cached ones, two sequences, rows for the output projection.
        _prefill("prefill_chunk_behind_prefix", 2, 28, 4, 1000, 2051, 128, "f16", True, False, True),
        # The benchmark's batch of long sequences, with the log-sum-exp a later merge needs.
        _prefill("prefill_long_batch", 4, 32, 32, 4096, 0, 128, "bf16", True, True, False),
        # The f32 attention block the reference's CPU path can run as well.
        _prefill("prefill_f32_block", 1, 8, 8, 512, 0, 64, "f32", False, True, False),
        # One sequence being decoded in the middle of its cache: the smallest call, launches and host work count.
        _decode("decode_one_sequence", 1, 28, 4, 2048, 1537, "f16", False),
        # A serving batch over long caches (the benchmark's decode).
        _decode("decode_long_batch", 64, 32, 8, 32768, 32768, "bf16", True),
        # The fused QKV projection of sixteen token rows: weights read once for a few rows.
        _gemm("gemm_few_rows", 16, 6144, 4096, "bf16", "none", "bf16", False, False),
        # The benchmark's GEMM region: bias + GELU + narrowing.
        _gemm("gemm_square_bias_gelu", 8192, 8192, 8192, "bf16", "bias_gelu", "bf16", False, False),
        # One prompt through a full-width decoder layer.
        _layer("layer_one_prompt", 1, 1000, "bf16", True, 0),
        # The benchmark's decoder layer: eight sequences of 2048 tokens.
        _layer("layer_batch", 8, 2048, "bf16", True, 0),
        # Command-level seam: the four commands of a small projection on host storage, ragged channels.
        _commands("commands_projection", 256, 512, 520, "bf16", True),
        # A compiled attention program on the full 16-Tile grid.
        _program("program_attention_16_tiles", 16, 8),
    ]


def _log_int(rng, low, high, multiple=1):
    value = math.exp(rng.uniform(math.log(low), math.log(high)))
    return min(high, max(low, int(round(value / multiple)) * multiple))


def _draw_prefill(rng):
    while True:
        if rng.random() < 0.25:   # the f32 block and its neighbours
            heads = rng.choice((4, 8, 16))
            return _prefill(None, rng.choice((1, 1, 2)), heads, heads, _log_int(rng, 48, 1024), 0, rng.choice((64, 64, 128)), "f32",
                            rng.random() < 0.5, rng.random() < 0.5, False)
        q_heads, kv_heads = rng.choice(_HEADS)
        batch, q_len = rng.choice((1, 1, 2, 3, 4)), _log_int(rng, 48, 4096)
        prefix = _log_int(rng, 16, 4096) if rng.random() < 0.35 else 0
        case = _prefill(None, batch, q_heads, kv_heads, q_len, prefix, 128, rng.choice(("bf16", "bf16", "f16")),
                        rng.random() < 0.8, rng.random() < 0.4, rng.random() < 0.4)
        if _prefill_flops(case) <= _MAX_PREFILL_FLOPS:
            return case


def _draw_decode(rng):
    while True:
        q_heads, kv_heads = rng.choice(_HEADS)
        batch = _log_int(rng, 1, 64)
        length = _log_int(rng, 64, 1 << 20) if batch == 1 else _log_int(rng, 64, 32768)
        capacity = length + (_log_int(rng, 16, 2048) if rng.random() < 0.5 else 0)
        if batch * kv_heads * capacity <= _MAX_DECODE_KEYS:
            return _decode(None, batch, q_heads, kv_heads, capacity, length, rng.choice(("bf16", "bf16", "f16")), rng.random() < 0.4)


def _draw_gemm(rng):
    while True:
        epilogue = rng.choice(("none", "none", "bias", "bias_gelu", "swiglu"))
        m = _log_int(rng, 8, 8192, 8)
        n, k = _log_int(rng, 256, 28672, 32 if epilogue == "swiglu" else 8), _log_int(rng, 256, 14336, 8)
        dtype = rng.choice(("bf16", "bf16", "f16"))
        out = "f32" if epilogue != "swiglu" and rng.random() < 0.2 else dtype
        if m * n * k <= _MAX_GEMM:
            return _gemm(None, m, n, k, dtype, epilogue, out, rng.random() < 0.15, rng.random() < 0.4)


def draw(rng):
    kind = rng.choice(("prefill",) * 4 + ("decode",) * 2 + ("gemm",) * 2 + ("layer",) * 2 + ("commands", "program"))
    if kind == "prefill":
        return _draw_prefill(rng)
    if kind == "decode":
        return _draw_decode(rng)
    if kind == "gemm":
        return _draw_gemm(rng)
    if kind == "layer":
        batch = rng.choice((1, 1, 2, 3, 4, 8))
        seq = _log_int(rng, 16, min(4096, _MAX_TOKENS // batch), 8)
        return _layer(None, batch, seq, rng.choice(("bf16", "bf16", "f16")), rng.random() < 0.75, rng.choice((0, 0, 777)))
    if kind == "commands":
        return _commands(None, _log_int(rng, 33, 700), _log_int(rng, 64, 1024), _log_int(rng, 33, 1024), rng.choice(("bf16", "f16")),
                         rng.random() < 0.6)
    return _program(None, rng.randint(1, 16), rng.randint(1, 12))


# ---------------------------------------------------------------------------------------------------------- inputs
def _normal(gen, shape, dtype, std=1.0):
    return (torch.randn(shape, device="cuda", generator=gen, dtype=torch.float32 if dtype == torch.float32 else dtype) * std)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return _PREPARE[case["kind"]](case, seed, gen)


def run(state):
    return _RUN[state["kind"]](state)


def _prepare_prefill(c, seed, gen):
    dtype, d = _DTYPES[c["dtype"]], c["head_dim"]
    keys = c["prefix"] + c["q_len"]
    return dict(kind="prefill", backend=_backend(), q=_normal(gen, (c["batch"], c["q_heads"], c["q_len"], d), dtype),
                k=_normal(gen, (c["batch"], c["kv_heads"], keys, d), dtype), v=_normal(gen, (c["batch"], c["kv_heads"], keys, d), dtype),
                lse=torch.empty(c["batch"], c["q_heads"], c["q_len"], device="cuda") if c["lse"] else None,
                scale=d ** -0.5, causal=c["causal"], query_start=c["prefix"], token_major=c["token_major"])


def _run_prefill(s):
    out = s["backend"].attention_fa(s["q"], s["k"], s["v"], s["scale"], s["causal"], lse=s["lse"], query_start=s["query_start"],
                                    token_major_out=s["token_major"])
    return (out,) if s["lse"] is None else (out, s["lse"])


def _prepare_decode(c, seed, gen):
    dtype = _DTYPES[c["dtype"]]
    cache = (c["batch"], c["kv_heads"], c["capacity"], 128)
    return dict(kind="decode", backend=_backend(), q=_normal(gen, (c["batch"], c["q_heads"], 1, 128), dtype), k=_normal(gen, cache, dtype),
                v=_normal(gen, cache, dtype), lse=torch.empty(c["batch"], c["q_heads"], 1, device="cuda") if c["lse"] else None,
                scale=128 ** -0.5, length=c["length"])


def _run_decode(s):
    out = s["backend"].attention_fd(s["q"], s["k"], s["v"], s["scale"], lse=s["lse"], key_end=s["length"])
    return (out,) if s["lse"] is None else (out, s["lse"])


def _prepare_gemm(c, seed, gen):
    dtype = _DTYPES[c["dtype"]]

    def uniform(*shape):
        return torch.rand(shape, device="cuda", generator=gen, dtype=torch.float32).mul_(2).sub_(1).to(dtype)
    a = uniform(*((c["k"], c["m"]) if c["lhs_transposed"] else (c["m"], c["k"])))
    b = uniform(*((c["n"], c["k"]) if c["rhs_transposed"] else (c["k"], c["n"])))
    if c["epilogue"] == "swiglu":   # activations of a layer: gate and up values around one
        b *= 2.0 * c["k"] ** -0.5
    bias = _normal(gen, (c["n"],), torch.float32, 0.02) if c["epilogue"] in ("bias", "bias_gelu") else None
    return dict(kind="gemm", backend=_backend(), a=a, b=b, bias=bias, epilogue=_EPILOGUES[c["epilogue"]], out_dtype=_DTYPES[c["out"]],
                lhs_transposed=c["lhs_transposed"], rhs_transposed=c["rhs_transposed"])


def _run_gemm(s):
    return s["backend"].gemm_epilogue(s["a"], s["b"], s["bias"], epilogue=s["epilogue"], out_dtype=s["out_dtype"],
                                      lhs_transposed=s["lhs_transposed"], rhs_transposed=s["rhs_transposed"])


def _layer_config(c):
    return LayerConfig() if c["wide"] else LayerConfig(d_model=512, q_heads=4, kv_heads=2, ffn=768)


def _prepare_layer(c, seed, gen):
    cfg, dtype = _layer_config(c), _DTYPES[c["dtype"]]

    def w(*shape):
        return _normal(gen, shape, dtype, 0.02)
    hd = cfg.head_dim
    weights = LayerWeights(norm1=1.0 + w(cfg.d_model), wq=w(cfg.d_model, cfg.q_heads * hd), wk=w(cfg.d_model, cfg.kv_heads * hd),
                           wv=w(cfg.d_model, cfg.kv_heads * hd), wo=w(cfg.q_heads * hd, cfg.d_model), norm2=1.0 + w(cfg.d_model),
                           wgate=w(cfg.d_model, cfg.ffn), wup=w(cfg.d_model, cfg.ffn), wdown=w(cfg.ffn, cfg.d_model))
    layer = ShardedDecoderLayer(_backend(), cfg, weights)
    return dict(kind="layer", layer=layer, x=_normal(gen, (c["batch"], c["seq"], cfg.d_model), dtype), offset=c["position_offset"])


def _run_layer(s):
    return s["layer"].forward_fused(s["x"], position_offset=s["offset"])


def _prepare_commands(c, seed, gen):
    rng = np.random.default_rng(seed)
    dtype, fmt = _DTYPES[c["dtype"]], _FORMATS[c["dtype"]]
    m, k, n = c["m"], c["k"], c["n"]

    def tensor(key):   # physical storage holding values of U[-1, 1]
        count = B200TargetModelBackend.physical_bytes(key) // 2
        return NumericTensor(key, torch.from_numpy(rng.uniform(-1, 1, count).astype(np.float32)).to(dtype).view(torch.uint8).numpy())

    def blank(key):
        return NumericTensor(key, np.zeros(B200TargetModelBackend.physical_bytes(key), dtype=np.uint8))
    keys = {name: PhysicalTensorDescriptor(f, abi.LAYOUT_CX, shape) for name, f, shape in (
        ("lhs", fmt, [m, k]), ("rhs", fmt, [k, n]), ("product", fmt, [m, n]), ("wide", abi.F32, [m, n]), ("sums", abi.F32, [1, n]))}
    return dict(kind="commands", backend=_backend(), operation=FormalGemmOperation(keys["lhs"], keys["rhs"], keys["product"], m, k, n),
                lhs=tensor(keys["lhs"]), rhs=tensor(keys["rhs"]), residual=tensor(keys["product"]), product=blank(keys["product"]),
                wide=blank(keys["wide"]), sums=blank(keys["sums"]), widen=155 if c["dtype"] == "bf16" else 161, dtype=dtype,
                policy=abi.GEMM_TENSOR if c["tensor_policy"] else abi.GEMM_FORMAL)


def _run_commands(s):
    be = s["backend"]
    product = be.try_execute(s["operation"], s["lhs"], s["rhs"], s["product"], policy=s["policy"])
    total = be.execute_elementwise("add", [product.destination, s["residual"]], s["product"])
    wide = be.execute_convert(s["widen"], total.destination, s["wide"])
    sums = be.execute_reduce("sum", "trailing1", wide.destination, s["sums"])
    values = [torch.from_numpy(product.destination.storage).view(s["dtype"]), torch.from_numpy(total.destination.storage).view(s["dtype"])]
    return values + [wide.destination.storage.view(np.float32), sums.destination.storage.view(np.float32)]


_BLOCK = 16384   # bytes of a 64 x 64 f32 matrix
_DMA = "i32 {0}, i32 {0}, i32 0, i32 0, i32 0, i32 1, i32 1, i32 1, i32 5, i32 0"


def _attention_module(tile, tiles, blocks):
    """One Tile's module: online attention of its 64 queries over `blocks` blocks of 64 keys, head dimension 64, f32, in the
    transposed form (the queries are the 64 channels). Per block: scores, scaling, row maximum, new maximum, norm, rescaled
    sum, probabilities, row sum, new sum, rescaled accumulator, PV product with the accumulator as partial sum."""
    q, k, v, s, p, acc, scaled = 0, 16384, 32768, 49152, 65536, 98304, 114688
    m_old, m_tile, m_new, diff, norm, total, rescaled, p_sum, inverse = (81920 + 256 * i for i in range(9))
    full, vector = "i32 4096, i32 5", "i32 64, i32 5"
    same, unit = "i32 0, i32 0, i32 0, i32 1", "i32 64, i32 0, i32 0, i32 1"
    one = _DMA.format(_BLOCK)
    call = "  call void @wafer_tx81_"
    lines = ["define void @entry(i64 %0, i64 %1, i64 %2, i64 %3) {", f"  %qsrc = add i64 %0, {tile * _BLOCK}", f"  %odst = add i64 %3, {tile * _BLOCK}",
             f"{call}rdma(i64 %qsrc, i64 {q}, {one})", f"{call}memset(i64 {m_old}, i32 -8388608, i32 64, i32 5, i32 0)",
             f"{call}memset(i64 {total}, i32 0, i32 64, i32 5, i32 0)", f"{call}memset(i64 {acc}, i32 0, i32 4096, i32 5, i32 0)",
             "  br label %head", "head:", "  %j = phi i64 [ 0, %4 ], [ %next, %body ]", f"  %more = icmp ult i64 %j, {blocks}",
             "  br i1 %more, label %body, label %done", "body:", f"  %off = mul i64 %j, {_BLOCK}", "  %ksrc = add i64 %1, %off",
             "  %vsrc = add i64 %2, %off", f"{call}rdma(i64 %ksrc, i64 {k}, {one})", f"{call}rdma(i64 %vsrc, i64 {v}, {one})",
             f"{call}gemm_oriented(i64 {k}, i64 {q}, i64 {s}, i64 0, i32 64, i32 64, i32 64, i32 1, i32 5, i32 5, i32 13, i32 0, i32 1, i32 0)",
             f"{call}elementwise_mul(i64 {s}, i64 1040187392, i64 {s}, {full}, i32 0, i32 1, i32 0, i32 1)",   # * 0.125
             f"{call}reduce_max(i64 {s}, i64 {m_tile}, i32 1, i32 1, i32 1, i32 64, i32 64, i32 5, i32 1)",
             f"{call}elementwise_max(i64 {m_old}, i64 {m_tile}, i64 {m_new}, {vector}, {same})",
             f"{call}elementwise_sub(i64 {m_old}, i64 {m_new}, i64 {diff}, {vector}, {same})",
             f"{call}elementwise_exp(i64 {diff}, i64 {norm}, {vector}, i32 1)",
             f"{call}elementwise_mul(i64 {total}, i64 {norm}, i64 {rescaled}, {vector}, {same})",
             f"{call}elementwise_sub(i64 {s}, i64 {m_new}, i64 {p}, {full}, {unit})",
             f"{call}elementwise_exp(i64 {p}, i64 {p}, {full}, i32 1)",
             f"{call}reduce_sum(i64 {p}, i64 {p_sum}, i32 1, i32 1, i32 1, i32 64, i32 64, i32 5, i32 1)",
             f"{call}elementwise_add(i64 {rescaled}, i64 {p_sum}, i64 {total}, {vector}, {same})",
             f"{call}elementwise_mul(i64 {acc}, i64 {norm}, i64 {scaled}, {full}, {unit})",
             f"{call}gemm_oriented(i64 {v}, i64 {p}, i64 {acc}, i64 {scaled}, i32 64, i32 64, i32 64, i32 1, i32 5, i32 5, i32 5, i32 1, i32 0, i32 0)",
             f"{call}elementwise_max(i64 {m_new}, i64 {m_new}, i64 {m_old}, {vector}, {same})",
             "  %next = add nuw i64 %j, 1", "  br label %head", "done:", f"{call}elementwise_recip(i64 {total}, i64 {inverse}, {vector}, i32 1)",
             f"{call}elementwise_mul(i64 {acc}, i64 {inverse}, i64 {scaled}, {full}, {unit})", f"{call}wdma(i64 {scaled}, i64 %odst, {one})",
             "  ret void", "}", "!wafer.target.tile_id = !{!2}", "!wafer.target.entry_arguments = !{!10, !11, !12, !13}", f"!2 = !{{i64 {tile}}}"]
    for i, (kind, ordinal, count, access) in enumerate((("input", 0, tiles, "read"), ("input", 1, blocks, "read"), ("input", 2, blocks, "read"),
                                                        ("output", 0, tiles, "write"))):
        lines.append(f'!{10 + i} = !{{i64 {i}, !"external-{kind}", i64 {ordinal}, !"", !"f32", !"tensor", i64 {count * _BLOCK}, i64 {count * 4096}, '
                     f'!"{access}-only", i64 {count * 64}, i64 64, i64 0}}')
    return "\n".join(lines) + "\n"


def _prepare_program(c, seed, gen):
    rng = np.random.default_rng(seed)
    modules = [_attention_module(tile, c["tiles"], c["blocks"]) for tile in range(c["tiles"])]
    inputs = [rng.standard_normal((64 * count, 64)).astype(np.float32) for count in (c["tiles"], c["blocks"], c["blocks"])]
    return dict(kind="program", program=TileProgram(modules, _backend(), spm_bytes=1 << 17), inputs=inputs)


def _run_program(s):
    outputs, _ = s["program"].run(s["inputs"])
    return [bits.view(np.float32) for bits in outputs]


_PREPARE = {"prefill": _prepare_prefill, "decode": _prepare_decode, "gemm": _prepare_gemm, "layer": _prepare_layer,
            "commands": _prepare_commands, "program": _prepare_program}
_RUN = {"prefill": _run_prefill, "decode": _run_decode, "gemm": _run_gemm, "layer": _run_layer, "commands": _run_commands,
        "program": _run_program}


# ---------------------------------------------------------------------------------------------------------- what a pass needs
def _prefill_flops(c):
    keys, rows = c["prefix"] + c["q_len"], c["q_len"]
    pairs = rows * c["prefix"] + rows * (rows + 1) // 2 if c["causal"] else rows * keys
    return 4 * c["head_dim"] * c["batch"] * c["q_heads"] * pairs


def work(case):
    c, kind = case, case["kind"]
    if kind == "prefill":
        width = 4 if c["dtype"] == "f32" else 2
        keys = c["prefix"] + c["q_len"]
        values = c["batch"] * c["head_dim"] * (2 * c["q_heads"] * c["q_len"] + 2 * c["kv_heads"] * keys)
        return {"bytes": values * width + (4 * c["batch"] * c["q_heads"] * c["q_len"] if c["lse"] else 0), "flops": _prefill_flops(c)}
    if kind == "decode":
        values = 128 * c["batch"] * (2 * c["kv_heads"] * c["length"] + 2 * c["q_heads"])
        return {"bytes": 2 * values + (4 * c["batch"] * c["q_heads"] if c["lse"] else 0), "flops": 4 * 128 * c["batch"] * c["q_heads"] * c["length"]}
    if kind == "gemm":
        columns = c["n"] // 2 if c["epilogue"] == "swiglu" else c["n"]
        size = 2 * (c["m"] * c["k"] + c["k"] * c["n"]) + (4 if c["out"] == "f32" else 2) * c["m"] * columns
        return {"bytes": size + (4 * c["n"] if c["epilogue"] in ("bias", "bias_gelu") else 0), "flops": 2 * c["m"] * c["n"] * c["k"]}
    if kind == "layer":
        cfg = _layer_config(c)
        weights = cfg.d_model * (2 * (cfg.q_heads + cfg.kv_heads) * cfg.head_dim + 3 * cfg.ffn + 2)
        return {"bytes": 2 * (weights + 2 * c["batch"] * c["seq"] * cfg.d_model), "flops": layer_flops(cfg, c["batch"], c["seq"])}
    if kind == "commands":
        m, k, n = c["m"], c["k"], c["n"]
        # host storage in and out of each command: product, sum (two operands), widening, column sums
        return {"bytes": 2 * (m * k + k * n + m * n) + 2 * 3 * m * n + 6 * m * n + 4 * (m * n + n), "flops": 2 * m * n * k + 2 * m * n}
    return {"bytes": _BLOCK * (2 * c["tiles"] + 2 * c["blocks"]), "flops": 4 * 64 * 64 * 64 * c["tiles"] * c["blocks"]}


def tolerance(case):
    c, kind = case, case["kind"]
    if kind == "prefill":
        return {"rel": {"bf16": 1e-2, "f16": 2e-3, "f32": 1e-5}[c["dtype"]]}
    if kind == "decode":
        return {"rel": {"bf16": 1e-2, "f16": 2e-3}[c["dtype"]]}
    if kind == "gemm":
        return {"rel": {"bf16": 1e-2, "f16": 2e-3, "f32": 1e-5}[c["out"]]}
    if kind == "layer":
        return {"rel": {"bf16": 1e-2, "f16": 2e-3}[c["dtype"]]}
    if kind == "commands" and c["tensor_policy"]:
        return {"rel": {"bf16": 1e-2, "f16": 2e-3}[c["dtype"]]}
    return "exact"   # the bit-exact command families
