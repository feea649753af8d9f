"""The work this framework is measured on: what a decode server has it do, through its public entry points.

    layer      one decode step of a whole sparse-attention MoE layer (DecoderLayer), a CUDA-graph replay: the call a
               server makes per layer and token
    indexer    paged index scores (FP8 or MXFP4 keys) and the top-k selection over them
    gemm       one block-scaled projection: FP8 with general or power-of-two scales, NVFP4, FP8 x FP4, BF16
    attention  sparse MLA decode attention over a sliding window and the selected compressed records
    quant      RMSNorm + FP8 quantisation of the hidden rows, then partial RoPE + FP8 quantisation of the query heads

"graph" says how a program calls the operators of a case: captured once and replayed, as a server does with the steps
it repeats, or as plain calls.  All inputs are made on the GPU from the seed.
"""
import torch

import wuda_b200 as wuda
from wuda_b200 import layer_setup

HIDDEN = 7168
# the projections of the block-scaled GEMM sweep: (N, K)
PROJECTIONS = ((24576, 7168), (7168, 16384), (2112, 7168), (4096, 7168))
FORMATS = ("fp8", "fp8_pow2", "nvfp4", "fp8_fp4", "bf16")


def listed():
    return [
        # a single user's token: eight experts stream, everything else is latency
        dict(name="layer_b1_ctx4096", kind="layer", batch=1, context=4096, fp4=False),
        # the headline configuration: 64 requests at 32 K tokens
        dict(name="layer_b64_ctx32768", kind="layer", batch=64, context=32768, fp4=False),
        # the largest batch a step takes, an odd context, the indexer in its MXFP4 form
        dict(name="layer_b128_ctx50003_fp4", kind="layer", batch=128, context=50003, fp4=True),
        # the benchmark's indexer step: two query rows per request, 16 K to 64 K entries
        dict(name="indexer_b64_n2", kind="indexer", batch=64, next_n=2, lo=16384, hi=65536, topk=2048, fp4=False, graph=True),
        # a few short requests, called directly
        dict(name="indexer_b4_short", kind="indexer", batch=4, next_n=1, lo=1, hi=4096, topk=2048, fp4=False, graph=False),
        # an odd batch of mixed lengths over MXFP4 keys
        dict(name="indexer_b37_fp4", kind="indexer", batch=37, next_n=1, lo=1000, hi=33000, topk=1024, fp4=True, graph=True),
        # the widest projection at the usual batch, general scales
        dict(name="gemm_fp8_m64", kind="gemm", format="fp8", m=64, n=24576, k=7168, graph=True),
        # the output projection at the largest batch, power-of-two scales as the checkpoints hold them
        dict(name="gemm_fp8_pow2_m256", kind="gemm", format="fp8_pow2", m=256, n=7168, k=16384, graph=False),
        # NVFP4 at two requests' worth of a batch of 64
        dict(name="gemm_nvfp4_m128", kind="gemm", format="nvfp4", m=128, n=24576, k=7168, graph=True),
        # one token through the smallest projection, called directly
        dict(name="gemm_fp8_m1", kind="gemm", format="fp8", m=1, n=2112, k=7168, graph=False),
        # the attention of the headline configuration
        dict(name="attention_b64", kind="attention", batch=64, heads=128, lo=16384, hi=65536, topk=2048, graph=True),
        # norm / RoPE / quantisation of a 256-token batch, called directly
        dict(name="quant_t256", kind="quant", tokens=256, pow2=False, graph=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(("layer", "indexer", "gemm", "gemm", "attention", "quant"))
    if kind == "layer":
        return dict(kind=kind, batch=_log_int(rng, 1, 128), context=_log_int(rng, 1000, 50000), fp4=rng.random() < 0.3)
    if kind == "indexer":
        fp4 = rng.random() < 0.4
        hi = _log_int(rng, 1024, 65536)
        return dict(kind=kind, batch=_log_int(rng, 1, 128 if fp4 else 64), next_n=1 if fp4 else rng.choice((1, 2)),
                    lo=max(1, hi // rng.choice((1, 2, 4, 16))), hi=hi, topk=rng.choice((512, 1024, 2048)), fp4=fp4,
                    graph=rng.random() < 0.5)
    if kind == "gemm":
        fmt = rng.choice(FORMATS)
        n, k = rng.choice(PROJECTIONS)
        if rng.random() < 0.5:      # other widths: multiples of 64 rows, of 256 columns
            n = 64 * _log_int(rng, 16, 384)
            k = 256 * _log_int(rng, 4, min(64, 24576 * 7168 // (256 * n)))
        return dict(kind=kind, format=fmt, m=_log_int(rng, 1, 128 if fmt == "bf16" else 256), n=n, k=k,
                    graph=rng.random() < 0.5)
    if kind == "attention":
        hi = _log_int(rng, 2048, 65536)
        return dict(kind=kind, batch=_log_int(rng, 1, 128), heads=rng.choice((64, 128)), lo=max(1, hi // rng.choice((1, 4))),
                    hi=hi, topk=rng.choice((512, 1024, 2048)), graph=rng.random() < 0.5)
    return dict(kind=kind, tokens=_log_int(rng, 1, 256), pow2=rng.random() < 0.5, graph=rng.random() < 0.5)


# ---------------------------------------------------------------- what a program holds before the call

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randint(g, lo, hi, *shape, dtype=torch.int32):
    return torch.randint(lo, hi, shape, generator=g, device="cuda", dtype=dtype)


def _prepare_layer(c, seed):
    layer, slots, x = layer_setup.build_random_layer(c["batch"], c["context"], seed=seed, indexer_fp4=c["fp4"])
    layer.prepare(slots)
    layer.capture(x, c["batch"])
    return dict(layer=layer, x=x)


def _contexts(c, g):
    """Lengths of the requests: uniform in [lo, hi], the longest at hi."""
    ctx = _randint(g, c["lo"], c["hi"] + 1, c["batch"])
    ctx[int(_randint(g, 0, c["batch"], 1))] = c["hi"]
    return ctx


def _pages_of(ctx, per_page, g):
    """A shuffled block table [batch, pages of the longest] over exactly the pages the requests need."""
    need = (ctx + per_page - 1) // per_page
    first = torch.cumsum(need, 0) - need
    total = int(need.sum())
    shuffled = torch.randperm(total, generator=g, device="cuda").int()
    at = torch.arange(int(need.max()), device="cuda")[None, :]
    table = torch.where(at < need[:, None], shuffled[(first[:, None] + at).clamp_max(total - 1)], -1)
    return table.int().contiguous(), total


def _prepare_indexer(c, seed):
    g = _generator(seed)
    batch, next_n, epb = c["batch"], c["next_n"], 64
    rows = batch * next_n
    ctx = _contexts(c, g)
    table, total = _pages_of(ctx, epb, g)
    lens = (ctx[:, None] - next_n + 1 + torch.arange(next_n, device="cuda")).clamp_min(0).int().contiguous()
    weights = torch.randn(rows, 64, generator=g, device="cuda") / 8
    if c["fp4"]:     # MXFP4 of normal values: fp4_act_quant's codes and exponent bytes
        pages = torch.empty(total, epb * 68, dtype=torch.uint8, device="cuda")
        codes, sf = wuda.fp4_act_quant(torch.randn(total * epb, 128, generator=g, device="cuda").bfloat16(), 32)
        pages[:, :epb * 64] = codes.view(torch.uint8).view(total, epb * 64)
        pages[:, epb * 64:] = sf.view(torch.uint8).view(total, epb * 4)
        q, q_sf = wuda.fp4_act_quant(torch.randn(rows * 64, 128, generator=g, device="cuda").bfloat16(), 32)
        q = q.view(torch.uint8).view(torch.int8).view(rows, 64, 64)
        q_sf = q_sf.view(torch.uint8).view(torch.int32).view(rows, 64)
    else:            # e4m3 of normal values, one fp32 scale per token
        pages = torch.empty(total, epb * 132, dtype=torch.uint8, device="cuda")
        for at in range(0, total, 8192):
            part = pages[at:at + 8192]
            keys = torch.randn(part.size(0), epb * 128, generator=g, device="cuda").to(torch.float8_e4m3fn)
            part[:, :epb * 128] = keys.view(torch.uint8)
        scales = torch.rand(total, epb, generator=g, device="cuda") * 0.09 + 0.01
        pages[:, epb * 128:] = scales.view(torch.uint8)
        q, q_sf = torch.randn(rows, 64, 128, generator=g, device="cuda").to(torch.float8_e4m3fn), None
    width = (c["hi"] + 255) // 256 * 256
    logits = torch.full((rows, width), float("-inf"), device="cuda")
    out = torch.empty(rows, c["topk"], dtype=torch.int32, device="cuda")

    def call():
        if c["fp4"]:
            wuda.mqa_logits_fp4_decode_out(q, q_sf, pages, weights, lens, table, logits, c["hi"], epb)
        else:
            wuda.mqa_logits_fp8_decode_out(q, pages, weights, lens, table, None, logits, epb, next_n=next_n)
        wuda.topk_v2_transform(logits, lens.view(-1), table, out, epb, rows_per_table_row=next_n)
        return logits, out

    return _captured(c, call)


def _fp8_weight(n, k, g, pow2):
    """N(0, 0.02) weights as e4m3 with one fp32 scale per 128 x 128 block."""
    rows = (n + 127) // 128 * 128
    w = torch.zeros(rows, k, device="cuda")
    w[:n] = torch.randn(n, k, generator=g, device="cuda") * 0.02
    v = w.view(rows // 128, 128, k // 128, 128)
    s = v.abs().amax(dim=(1, 3)).clamp_min(1e-4) / 448
    if pow2:
        s = torch.exp2(torch.ceil(torch.log2(s)))
    w = (v / s[:, None, :, None]).clamp_(-448, 448).view(rows, k)[:n].to(torch.float8_e4m3fn)
    return w.contiguous(), s.contiguous()


def _nvfp4(x):
    """Packed e2m1 codes, tensor-core-ordered ue4m3 scale bytes and the tensor's fp32 scale of x [rows, k]."""
    rows, k = x.shape
    gs = float(x.abs().max()) / (448 * 6)
    pad = (rows + 127) // 128 * 128
    codes = torch.empty(rows, k // 2, dtype=torch.uint8, device="cuda")
    sf = torch.zeros(pad, k // 16, dtype=torch.uint8, device="cuda")
    bounds = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], device="cuda")
    for at in range(0, rows, 4096):
        v = x[at:at + 4096].float().view(-1, k // 16, 16)
        s8 = (v.abs().amax(-1) / 6 / gs).clamp_max(448).to(torch.float8_e4m3fn)
        sf[at:at + v.size(0)] = s8.view(torch.uint8)
        y = torch.where(s8.float()[..., None] > 0, v / (s8.float()[..., None] * gs), 0.0)
        code = torch.bucketize(y.abs(), bounds).to(torch.uint8)
        code |= ((y < 0) & (code != 0)).to(torch.uint8) << 3
        code = code.view(-1, k // 2, 2)
        codes[at:at + v.size(0)] = code[..., 0] | code[..., 1] << 4
    packed = sf.view(pad // 128, 4, 32, k // 256, 4, 4).permute(0, 3, 4, 2, 1, 5).contiguous().view(-1)
    return codes, packed, gs


def _prepare_gemm(c, seed):
    g = _generator(seed)
    m, n, k, fmt = c["m"], c["n"], c["k"], c["format"]
    x = torch.randn(m, k, generator=g, device="cuda").bfloat16()
    if fmt in ("fp8", "fp8_pow2"):
        a, a_s = wuda.act_quant(x, 128, "ue8m0" if fmt == "fp8_pow2" else None)
        w, w_s = _fp8_weight(n, k, g, fmt == "fp8_pow2")
        return _captured(c, lambda: wuda.fp8_gemm(a, a_s, w, w_s, pow2_scales=fmt == "fp8_pow2"))
    weight = torch.randn(n, k, generator=g, device="cuda").mul_(0.02).bfloat16()
    if fmt == "nvfp4":
        a, a_sf, a_gs = _nvfp4(x)
        w, w_sf, w_gs = _nvfp4(weight)
        return _captured(c, lambda: wuda.nvfp4_gemm(a, a_sf, a_gs, w, w_sf, w_gs))
    if fmt == "fp8_fp4":
        a, a_s = wuda.act_quant(x, 128, "ue8m0")
        w, w_s = wuda.fp4_act_quant(weight, 32)
        return _captured(c, lambda: wuda.fp4_gemm(a, a_s, w, w_s))
    return _captured(c, lambda: wuda.bf16_gemm(x, weight))


def _prepare_attention(c, seed):
    g = _generator(seed)
    batch, epb = c["batch"], 64
    ctx = _contexts(c, g)
    entries = (ctx // 4).clamp_min(1)
    table, total = _pages_of(entries, epb, g)
    pools = [layer_setup.model1_pool(pages, per, seed + i) for i, (pages, per) in enumerate(((batch, 256), (total, epb)))]
    swa, cmp = (p.as_strided((p.size(0), per, 1, 584), (p.size(1), 584, 584, 1)) for p, per in zip(pools, (256, epb)))
    # the window: the last 128 tokens in a ring of 128, in the request's page of the window pool
    swa_len = ctx.clamp_max(128).int()
    at = torch.arange(128, device="cuda")[None, :]
    ring = (ctx[:, None] - swa_len[:, None] + at) % 128
    swa_idx = torch.where(at < swa_len[:, None], ring + 256 * torch.arange(batch, device="cuda")[:, None], -1).int().contiguous()
    # the selection: distinct entries of the request in no order, through its page table
    cmp_len = entries.clamp_max(c["topk"]).int()
    most = int(entries.max())
    pick = torch.rand(batch, most, generator=g, device="cuda")
    pick = pick.masked_fill_(torch.arange(most, device="cuda") >= entries[:, None], 2.0).argsort(1)[:, :c["topk"]]
    sel = torch.full((batch, c["topk"]), -1, dtype=torch.int32, device="cuda")
    keep = torch.arange(pick.size(1), device="cuda") < cmp_len[:, None]
    sel[:, :pick.size(1)] = torch.where(keep, torch.gather(table, 1, pick.div(epb, rounding_mode="floor").clamp_max(table.size(1) - 1))
                                        * epb + pick % epb, -1).int()
    q = torch.randn(batch, c["heads"], 512, generator=g, device="cuda").bfloat16()
    sink = torch.randn(c["heads"], generator=g, device="cuda")
    return _captured(c, lambda: wuda.sparse_mla_decode(q, swa, swa_idx, swa_len, cmp, sel, cmp_len, sink))


def _prepare_quant(c, seed):
    g = _generator(seed)
    t = c["tokens"]
    x = torch.randn(t, HIDDEN, generator=g, device="cuda").bfloat16()
    gamma = (torch.randn(HIDDEN, generator=g, device="cuda") * 0.1 + 1).bfloat16()
    heads = torch.randn(t, 128, 192, generator=g, device="cuda").bfloat16()
    pos = _randint(g, 0, 65536, t, dtype=torch.int64)
    angle = torch.outer(torch.arange(65536, device="cuda").float(), 10000 ** (-torch.arange(0, 64, 2, device="cuda").float() / 64))
    cos, sin = angle.cos().contiguous(), angle.sin().contiguous()
    fmt = "ue8m0" if c["pow2"] else None

    def call():
        y16, y8, s = wuda.rmsnorm_quant(x, gamma, 1e-6, scale_fmt=fmt)
        _, q8, qs = wuda.rope_quant(heads, pos, cos, sin, 64, scale_fmt=fmt)
        return y16, y8, s, q8, qs

    return _captured(c, call)


def _captured(c, call):
    """The call itself, or a CUDA graph of it made after one plain call."""
    if not c["graph"]:
        return dict(call=call)
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = call()
    return dict(graph=graph, out=out, call=call)


def prepare(case, seed):
    return dict(layer=_prepare_layer, indexer=_prepare_indexer, gemm=_prepare_gemm, attention=_prepare_attention,
                quant=_prepare_quant)[case["kind"]](case, seed)


def run(state):
    if "layer" in state:
        layer = state["layer"]
        out, cache = layer.replay(), layer.attn.cache
        # the residual streams, and the state rings and record pools that the step wrote into
        return out, cache.main_state, cache.idx_state, cache.swa_pool, cache.cmp_pool, cache.idx_pool
    if "graph" in state:
        state["graph"].replay()
        return state["out"]
    return state["call"]()


# ---------------------------------------------------------------- what a pass cannot do without

def _work_layer(c):
    m, entries = c["batch"], c["context"] // 4
    experts, topk = 256, 8
    active = experts * (1 - (1 - topk / experts) ** m)
    index_record = 68 if c["fp4"] else 132
    cache = m * (entries * index_record + (128 + min(2048, entries)) * 584)
    rows = m * 4 * HIDDEN * 2 * 2
    keys = 128 + min(2048, entries)
    # every dense weight once per token (experts: the eight chosen ones), index scores, attention
    dense = layer_setup.layer_weight_bytes(experts_active=0)
    params = dense - 2624 * HIDDEN - experts * HIDDEN - 2 * 24 * 4 * HIDDEN * 3
    flops = 2 * m * (params + topk * 3 * HIDDEN * 2048) + 2 * m * entries * 64 * 128 + 4 * m * keys * 128 * 512
    return dict(bytes=layer_setup.layer_weight_bytes(experts_active=active) + cache + rows, flops=flops)


def _mean_length(c):
    return (c["hi"] + (c["batch"] - 1) * (c["lo"] + c["hi"]) / 2) / c["batch"]


def _work_indexer(c):
    tokens, rows = c["batch"] * _mean_length(c), c["batch"] * c["next_n"]
    query = 64 * 64 + 64 * 4 if c["fp4"] else 64 * 128
    return dict(bytes=tokens * (68 if c["fp4"] else 132) + tokens * c["next_n"] * 4 + rows * (query + 64 * 4 + c["topk"] * 4),
                flops=2 * 64 * 128 * tokens * c["next_n"])


def _work_gemm(c):
    m, n, k = c["m"], c["n"], c["k"]
    tiles = (n + 127) // 128
    per_weight, per_act = dict(fp8=(1, 1 + 1 / 32), fp8_pow2=(1, 1 + 1 / 32), nvfp4=(9 / 16, 9 / 16), fp8_fp4=(17 / 32, 1 + 1 / 32),
                               bf16=(2, 2))[c["format"]]
    scales = tiles * (k // 128) * 4 if c["format"] in ("fp8", "fp8_pow2") else 0
    return dict(bytes=n * k * per_weight + scales + m * k * per_act + m * n * 2, flops=2 * m * n * k)


def _work_attention(c):
    def selected(ctx):
        return min(c["topk"], max(ctx // 4, 1)) + min(ctx, 128)

    steps = 64
    mean = sum(selected(c["lo"] + (c["hi"] - c["lo"]) * i // steps) for i in range(steps + 1)) / (steps + 1)
    keys = selected(c["hi"]) + (c["batch"] - 1) * mean
    return dict(bytes=keys * (584 + 4) + 2 * c["batch"] * c["heads"] * 512 * 2, flops=4 * keys * c["heads"] * 512)


def _work_quant(c):
    t = c["tokens"]
    hidden = t * HIDDEN * (2 + 2 + 1) + t * (HIDDEN // 128) * 4 + HIDDEN * 2
    query = t * 24576 * (2 + 1) + t * (24576 // 128) * 4 + t * (8 + 2 * 32 * 4)
    return dict(bytes=hidden + query, flops=t * (HIDDEN * 6 + 24576 * 4))


def work(case):
    return dict(layer=_work_layer, indexer=_work_indexer, gemm=_work_gemm, attention=_work_attention,
                quant=_work_quant)[case["kind"]](case)


def tolerance(case):
    """About four times what one correct pass differs from another (sums in another order, or in 64 bits)."""
    kind = case["kind"]
    if kind == "layer":         # other sums in the front and shared projections: 2.4e-3, 0.13 (FP8 codes at a tie)
        return {"rel": 1e-2, "max": 0.5, "differ": 1e-4}
    if kind == "indexer":       # fp32 sums of exact products; the selection may differ at a tie
        return {"rel": 1e-5, "max": 1e-4, "differ": 1e-3}
    if kind == "gemm":          # bf16 outputs against sums in 64 bits: 1.7e-3, 3.9e-3
        return {"rel": 7e-3, "max": 1.6e-2}
    if kind == "attention":     # 16-bit probabilities and bf16 outputs
        return {"rel": 8e-3, "max": 5e-2}
    return {"rel": 2e-3, "max": 0.15}   # an e4m3 code is up to 1/8 from the next
