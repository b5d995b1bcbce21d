"""What a user of this framework has it do, at the sizes it is used at: grouped MXFP8 quantisation, the two grouped
GEMMs, and the expert-parallel MoE layer on one GPU — each through its public entry point.

Row counts per expert come from three kinds of routing: "zipf" (skewed, Zipf(1.2) popularity), "uniform" (random
top-8 of a batch) and "classes" (70/15/10/5 % of the experts with 1-32 / 32-64 / 64-128 / 128-1024 rows, the mix of
the SM100 benchmark of the operators).  A case fixes the multiset of row counts; the seed decides which expert has
which count, and all values.
"""
import math
import socket

import numpy as np
import torch

import expert_specialization_moe_b200 as es

TOPK = 8
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


# ---- the cases -----------------------------------------------------------------------------------------------------
def listed():
    return [
        # one decode step's activations before the expert GEMM: 64 tokens x top-8, hidden 7168 — latency counts
        {"name": "quant_decode", "op": "quant", "experts": 256, "rows": 512, "k": 7168, "routing": "zipf",
         "dtype": "bf16"},
        # a prefill's activations (4096 tokens x top-8): bound by memory
        {"name": "quant_prefill", "op": "quant", "experts": 256, "rows": 32768, "k": 7168, "routing": "zipf",
         "dtype": "bf16"},
        # SiLU * mul and requantisation between the two expert GEMMs, 16384 tokens x top-8 with intermediate size 768
        {"name": "silu_prefill", "op": "silu", "experts": 128, "rows": 131072, "k": 768, "routing": "uniform",
         "dtype": "bf16"},
        # smallest GEMM call: 8 tokens x top-8 on a tensor-parallel gate_up shard
        {"name": "mm_decode_small", "op": "mm", "experts": 128, "rows": 64, "n": 768, "k": 4096, "routing": "uniform",
         "dtype": "bf16"},
        # decode down-projection, skewed routing, 64 tokens x top-8
        {"name": "mm_decode_down", "op": "mm", "experts": 256, "rows": 512, "n": 7168, "k": 2048, "routing": "zipf",
         "dtype": "bf16"},
        # tensor-parallel down-projection (short K) on mixed row counts
        {"name": "mm_mixed_down", "op": "mm", "experts": 256, "rows": 0, "n": 7168, "k": 256, "routing": "classes",
         "dtype": "bf16"},
        # expert-parallel gate_up with 16 local experts on mixed row counts, fp16 output
        {"name": "mm_mixed_gate_up", "op": "mm", "experts": 16, "rows": 0, "n": 4096, "k": 7168, "routing": "classes",
         "dtype": "fp16"},
        # prefill, gate_up of a small-expert model, balanced routing: 256 rows for every expert on average
        {"name": "mm_prefill_balanced", "op": "mm", "experts": 128, "rows": 32768, "n": 1536, "k": 2048,
         "routing": "uniform", "dtype": "bf16"},
        # prefill, gate_up of a large model, skewed routing: the largest call
        {"name": "mm_prefill_skewed", "op": "mm", "experts": 256, "rows": 32768, "n": 4096, "k": 7168,
         "routing": "zipf", "dtype": "bf16"},
        # block-scaled (fp32 scales) down-projection, batch 512 x top-8
        {"name": "bw_decode_down", "op": "bw", "experts": 256, "rows": 4096, "n": 7168, "k": 256, "routing": "uniform",
         "dtype": "bf16"},
        # block-scaled gate_up, batch 3072 x top-8: 192 rows per expert on average, fp16 output
        {"name": "bw_prefill_gate_up", "op": "bw", "experts": 128, "rows": 24576, "n": 768, "k": 4096,
         "routing": "uniform", "dtype": "fp16"},
        # the whole expert-parallel layer in a group of one GPU: route, dispatch with quantisation, gate_up, SiLU * mul,
        # down with the combine in its epilogue, weighted sum
        {"name": "layer_prefill", "op": "layer", "experts": 128, "tokens": 16384, "hidden": 2048, "inter": 768},
    ]


def draw(rng):
    def loguni(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    def mult(lo, hi, step=128):
        return max(1, round(loguni(lo, hi) / step)) * step

    op = rng.choice(["quant", "silu", "mm", "mm", "mm", "mm", "bw", "bw", "layer"])
    if op == "layer":
        case = {"op": op, "experts": rng.choice([32, 64, 128]), "tokens": int(loguni(16, 8192)),
                "hidden": mult(1024, 4096), "inter": mult(256, 1536)}
        while case["experts"] * 3 * case["hidden"] * case["inter"] > 8e8:
            case["inter"] = max(128, case["inter"] // 256 * 128)
        return case
    while True:
        case = {"op": op, "experts": int(loguni(8, 320)), "rows": int(loguni(32, 65536)),
                "routing": rng.choice(["zipf", "uniform", "classes"]), "dtype": rng.choice(["bf16", "bf16", "fp16"])}
        if op in ("mm", "bw"):
            case["n"] = mult(256, 7168)
        case["k"] = mult(256, 7168)
        rows = int(counts_of(case).sum())
        n = case.get("n", 0)
        if case["routing"] == "classes":
            case["rows"] = 0
        # at most about the work of the largest listed case of the kind
        if op in ("quant", "silu") and rows * case["k"] * (1 if op == "quant" else 2) > 2.4e8:
            continue
        if op in ("mm", "bw") and (case["experts"] * n * case["k"] > 4e9 or rows * (case["k"] + 2 * n) > 6e8):
            continue
        if op in ("mm", "bw") and rows * n * case["k"] > (6e11 if op == "mm" else 1.5e11):
            continue
        return case


def counts_of(case):
    """The multiset of row counts of a case, as an int64 array of one count per expert."""
    e, t = case["experts"], case["rows"]
    rng = np.random.default_rng([e, case["k"], case.get("n", 0)])
    if case["routing"] == "classes":
        u = rng.random(e)
        lo = np.where(u <= 0.7, 1, np.where(u <= 0.85, 32, np.where(u <= 0.95, 64, 128)))
        hi = np.where(u <= 0.7, 32, np.where(u <= 0.85, 64, np.where(u <= 0.95, 128, 1024)))
        return rng.integers(lo, hi + 1).astype(np.int64)
    if case["routing"] == "zipf":
        p = np.arange(1, e + 1, dtype=np.float64) ** -1.2
    else:
        p = np.ones(e)
    return rng.multinomial(t, p / p.sum()).astype(np.int64)


# ---- plain tensor arithmetic the inputs are made with (nothing of the framework) ----------------------------------
def _align128(x):
    return (x + 127) // 128 * 128


def _swizzle(sf):
    """[rows, K/32] scale bytes, rows a multiple of 128 -> the flat layout of 512-byte atoms."""
    r, kb = sf.shape
    return sf.view(r // 128, 4, 32, kb // 4, 4).permute(0, 3, 2, 1, 4).contiguous().view(r, kb)


def _mx_quant(x):
    """[rows, K] -> e4m3 values of x / scale and the UE8M0 scale byte of every 32 values: the smallest power of two
    that brings the block's largest magnitude to at most 448."""
    r, k = x.shape
    b = x.float().view(r, k // 32, 32)
    amax = b.abs().amax(-1)
    mant, ex = torch.frexp(amax / 448.0)
    ex = torch.where(mant == 0.5, ex - 1, ex).clamp(-127, 127)
    ex = torch.where(amax == 0, torch.full_like(ex, -127), ex)
    q = (b * torch.exp2(-ex.float()).unsqueeze(-1)).to(torch.float8_e4m3fn).view(r, k)
    return q, (ex + 127).to(torch.uint8)


def _mx_dequant64(q, sf):
    r, k = q.shape
    return (q.double().view(r, k // 32, 32) * torch.exp2(sf.double() - 127.0).unsqueeze(-1)).view(r, k)


def _mx_weights(gen, e, n, k, std):
    """e4m3 weights [e, n, k] and their row-major scale bytes [e, n, k/32], a few experts at a time."""
    w = torch.empty((e, n, k), dtype=torch.float8_e4m3fn, device="cuda")
    sf = torch.empty((e, n, k // 32), dtype=torch.uint8, device="cuda")
    step = max(1, (1 << 28) // (n * k))
    for i in range(0, e, step):
        c = min(step, e - i)
        q, s = _mx_quant(torch.randn((c * n, k), generator=gen, device="cuda").mul_(std).to(torch.bfloat16))
        w[i:i + c] = q.view(c, n, k)
        sf[i:i + c] = s.view(c, n, k // 32)
    return w, sf


def _activations(gen, rows, k, dtype, outliers):
    x = torch.randn((rows, k), generator=gen, device="cuda")
    if outliers:      # a percent of the values stand out fifty times, as activations' outlier channels do
        x *= torch.where(torch.rand((rows, k), generator=gen, device="cuda") < 0.01, 50.0, 1.0)
    return x.to(dtype)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * seed + 17)


class _Lists:
    """Problem list of a call: row counts, first rows and first scale rows per expert."""

    def __init__(self, case, seed):
        c = counts_of(case)
        np.random.default_rng(seed).shuffle(c)
        self.counts = c
        self.rows = int(c.sum())
        eo = np.concatenate([[0], np.cumsum(c)[:-1]])
        mp = _align128(c)
        bo = np.concatenate([[0], np.cumsum(mp)[:-1]])
        self.first, self.sf_first, self.sf_rows = eo, bo, int(mp.sum())
        ps = np.stack([c, np.full_like(c, case.get("n", 0)), np.full_like(c, case["k"])], 1)
        self.ps, self.eo, self.bo = (torch.from_numpy(np.ascontiguousarray(a).astype(np.int32)).cuda()
                                     for a in (ps, eo, bo))
        # scale row of every row of the batch
        self.sf_row_of = torch.from_numpy(np.concatenate(
            [np.arange(m) + b for m, b in zip(c, bo)] or [np.zeros(0, np.int64)])).cuda()


def _block_cast(x, rows_per_block):
    """fp32-scaled e4m3: one scale per rows_per_block x 128 block, amax / 448."""
    r, k = x.shape
    b = x.view(r // rows_per_block, rows_per_block, k // 128, 128)
    s = b.abs().float().amax(dim=(1, 3), keepdim=True).clamp(1e-4) / 448.0
    return (b / s).to(torch.float8_e4m3fn).view(r, k), s.view(r // rows_per_block, k // 128)


# ---- a call's inputs, the call, and what it cannot do without --------------------------------------------------
def _mm_inputs(case, seed):
    g, lists = _gen(seed), _Lists(case, seed)
    w, sfw = _mx_weights(g, case["experts"], case["n"], case["k"], 0.02)
    a, sf = _mx_quant(_activations(g, lists.rows, case["k"], torch.bfloat16, False))
    return lists, a, sf, w, sfw


def _bw_inputs(case, seed):
    g, lists = _gen(seed), _Lists(case, seed)
    e, n, k = case["experts"], case["n"], case["k"]
    w = torch.empty((e, n, k), dtype=torch.float8_e4m3fn, device="cuda")
    sw = torch.empty((e, n // 128, k // 128), device="cuda")
    step = max(1, (1 << 28) // (n * k))
    for i in range(0, e, step):
        c = min(step, e - i)
        q, s = _block_cast(torch.randn((c * n, k), generator=g, device="cuda"), 128)
        w[i:i + c], sw[i:i + c] = q.view(c, n, k), s.view(c, n // 128, k // 128)
    a, sa = _block_cast(_activations(g, lists.rows, k, torch.bfloat16, False).float(), 1)
    return lists, a, sa.contiguous(), w, sw


def _layer_inputs(case, seed):
    g = _gen(seed)
    e, t, h, i = case["experts"], case["tokens"], case["hidden"], case["inter"]
    w1 = (torch.randn((e, 2 * i, h), generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    w2 = (torch.randn((e, h, i), generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    x = torch.randn((t, h), generator=g, device="cuda").to(torch.bfloat16)
    prob = torch.softmax(torch.randn((t, e), generator=g, device="cuda"), -1)
    wts, ids = torch.topk(prob, TOPK, dim=-1)
    return x, ids.contiguous(), (wts / wts.sum(-1, keepdim=True)).contiguous(), w1, w2


def _group_of_one():
    import torch.distributed as dist
    if not dist.is_initialized():
        torch.cuda.set_device(0)
        with socket.socket() as s:
            s.bind(("127.0.0.1", 0))
            port = s.getsockname()[1]
        dist.init_process_group("nccl", init_method=f"tcp://127.0.0.1:{port}", rank=0, world_size=1,
                                device_id=torch.device("cuda", 0))


def prepare(case, seed):
    op = case["op"]
    if op in ("quant", "silu"):
        lists, dt = _Lists(case, seed), DTYPES[case["dtype"]]
        x = _activations(_gen(seed), lists.rows, case["k"] * (2 if op == "silu" else 1), dt, op == "quant")
        codes = torch.empty((lists.rows, case["k"]), dtype=torch.uint8, device="cuda").view(torch.float8_e4m3fn)
        sf = torch.empty((max(lists.sf_rows, 128), case["k"] // 32), dtype=torch.uint8, device="cuda")
        fn = es.es_sm100_mxfp8_blockscaled_grouped_quant if op == "quant" else es.es_sm100_mxfp8_silu_mul_grouped_quant
        return {"op": op, "fn": fn, "args": (x, lists.ps, lists.eo, lists.bo, codes, sf),
                "out": [codes.view(torch.uint8), sf[:lists.sf_rows]]}
    if op == "mm":
        lists, a, sf, w, sfw = _mm_inputs(case, seed)
        e, n, k = w.shape
        sfa = torch.zeros((max(lists.sf_rows, 128), k // 32), dtype=torch.uint8, device="cuda")
        sfa[lists.sf_row_of] = sf
        d = torch.empty((lists.rows, n), dtype=DTYPES[case["dtype"]], device="cuda")
        args = (d, a, w.transpose(1, 2), _swizzle(sfa), _swizzle(sfw.view(e * n, k // 32)), lists.ps, lists.eo, lists.bo)
        return {"op": op, "fn": es.es_sm100_mxfp8_blockscaled_grouped_mm, "args": args, "out": d}
    if op == "bw":
        lists, a, sa, w, sw = _bw_inputs(case, seed)
        e, n, k = w.shape
        d = torch.empty((lists.rows, n), dtype=DTYPES[case["dtype"]], device="cuda")
        ld = torch.full((e,), k, dtype=torch.int64, device="cuda")
        args = (d, a, w.transpose(1, 2), sa, sw.transpose(1, 2), ld, ld, torch.full_like(ld, n), lists.ps, lists.eo,
                torch.empty(1024, dtype=torch.uint8, device="cuda"))
        return {"op": op, "fn": es.es_fp8_blockwise_scaled_grouped_mm, "args": args, "out": d}
    from expert_specialization_moe_b200 import expert_parallel as ep
    _group_of_one()
    x, ids, wts, w1, w2 = _layer_inputs(case, seed)
    shard = ep.ExpertShard(w1, w2)
    fx = ep.FusedExchange(case["experts"], TOPK, case["tokens"], case["hidden"], x.device)
    out = torch.empty_like(x)
    return {"op": op, "fn": fx.forward, "args": (x, ids, wts, shard, True, out), "out": out}


def run(state):
    state["fn"](*state["args"])
    return state["out"]


def work(case):
    op = case["op"]
    if op == "layer":
        e, t, h, i = case["experts"], case["tokens"], case["hidden"], case["inter"]
        used = min(e, t * TOPK)
        return {"bytes": used * 3 * h * i * (1 + 1 / 32) + 2 * t * h * 2 + t * TOPK * 12, "flops": 6 * t * TOPK * h * i}
    c, k = counts_of(case), case["k"]
    rows, padded, used = int(c.sum()), int(_align128(c).sum()), int((c > 0).sum())
    lists = case["experts"] * 20
    if op in ("quant", "silu"):
        per = 2 if op == "quant" else 4
        return {"bytes": rows * k * (per + 1) + padded * k // 32 + lists, "flops": 0}
    n = case["n"]
    scales = (rows + used * n) * k / 32 if op == "mm" else (rows + used * n / 128) * k / 128 * 4
    return {"bytes": used * n * k + rows * k + 2 * rows * n + scales + lists, "flops": 2 * rows * n * k}


def tolerance(case):
    # codes and scale bytes are the same bytes in every correct implementation
    if case["op"] in ("quant", "silu"):
        return "exact"
    # two roundings of the intermediate (bf16, then e4m3 with its scale) decide differently where the sums before them
    # differ in the last bit (1.8e-2 from the same layer with its intermediate rounded once, from 64 bits to e4m3)
    if case["op"] == "layer":
        return {"rel": 3e-2}
    # sums of e4m3 products in 32 bits; one rounding to the output's type decides differently now and then
    return {"rel": 4e-3, "max": 2e-2} if case["dtype"] == "bf16" else {"rel": 1e-3, "max": 5e-3}


def exact(case, seed):
    op = case["op"]
    w = work(case)
    if op in ("quant", "silu") or w["flops"] > 3e14:
        return None                 # bytes are compared as they are; a GEMM beyond this takes too long in 64 bits
    if op == "layer":
        return _exact_layer(case, seed)
    lists, a, sa, wt, sw = (_mm_inputs if op == "mm" else _bw_inputs)(case, seed)
    e, n, k = wt.shape
    d = torch.empty((lists.rows, n), dtype=torch.float64, device="cuda")
    for x in range(e):
        m, r = int(lists.counts[x]), int(lists.first[x])
        if m == 0:
            continue
        if op == "mm":
            af, wf = _mx_dequant64(a[r:r + m], sa[r:r + m]), _mx_dequant64(wt[x], sw[x])
        else:
            af = a[r:r + m].double() * sa[r:r + m].double().repeat_interleave(128, 1)
            wf = wt[x].double() * sw[x].double().repeat_interleave(128, 0).repeat_interleave(128, 1)
        d[r:r + m] = af @ wf.t()
    return d


def _exact_layer(case, seed):
    x, ids, wts, w1, w2 = _layer_inputs(case, seed)
    i = case["inter"]
    xq = _mx_dequant64(*_mx_quant(x))
    out = torch.zeros(x.shape, dtype=torch.float64, device="cuda")
    for e in range(case["experts"]):
        tok, j = torch.nonzero(ids == e, as_tuple=True)
        if tok.numel() == 0:
            continue
        h = xq[tok] @ _mx_dequant64(*_mx_quant(w1[e])).t()
        act = h[:, :i] / (1 + torch.exp(-h[:, :i])) * h[:, i:]
        act = _mx_dequant64(*_mx_quant(act))
        y = act @ _mx_dequant64(*_mx_quant(w2[e])).t()
        out.index_add_(0, tok, wts[tok, j].double().unsqueeze(1) * y)
    return out
