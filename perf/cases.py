"""What a user of this library has it do, as timed cases: decode and speculative-verify attention over the paged FP4 cache
(UltraQuant and NVFP4), tree drafts, a layer's step (append the new tokens, then verify), and the append of a whole prompt.

Sizes are those of bench.py's configurations and of the tests, or generic ones between them; every case goes through the
public Python entry points (`all_quant_b200.uq_cuda`, `all_quant_b200.vllm_adapter`) with device-resident inputs, the way an
engine calls them.  Keys carry a lognormal(0, 0.5) multiplier per channel, values and queries are N(0, 1), the cache is
written by the library's own append, physical pages are a random permutation (as in bench.py).
"""
import random

import torch

from all_quant_b200 import uq_cuda, vllm_adapter

# the per-tensor scales of an NVFP4 cache: a block maximum of 32 (keys) / 8 (values) sits at the top of the e4m3 range
K_TS, V_TS = 32.0 / (6 * 448), 8.0 / (6 * 448)
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def _attention(name, B, ctx, K, HQ, HKV, D=128, PAGE=64, fmt=0, call="decode", rotate=False, scratch=True, lens_seed=7):
    """An attention case.  ctx: one length for all sequences, or (shortest, longest) of a ragged batch.  call: `decode`
    (uq_decode_cuda), `tree` (uq_tree_decode) or `step` (append of the K new tokens of every sequence, then the engine
    adapter's verify).  scratch: the caller keeps a workspace and an output, as a serving loop does; without it the call
    allocates both, as the plain one-line call does."""
    lo, hi = (ctx, ctx) if isinstance(ctx, int) else ctx
    case = {"kind": "attention", "B": B, "ctx_lo": lo, "ctx_hi": hi, "K": K, "HQ": HQ, "HKV": HKV, "D": D, "PAGE": PAGE, "fmt": fmt,
            "call": call, "rotate": rotate, "scratch": scratch, "lens_seed": lens_seed}
    return {"name": name, **case} if name else case


def _append(name, T, HKV, D=128, PAGE=64, fmt=0, dtype="bf16", rotate=False):
    """The append-quantize of T new tokens, keys and values, into a cache of about that size."""
    case = {"kind": "append", "T": T, "HKV": HKV, "D": D, "PAGE": PAGE, "fmt": fmt, "dtype": dtype, "rotate": rotate}
    return {"name": name, **case} if name else case


def listed():
    return [
        # the smallest call: two short chats, four drafts; launches and latency are all there is
        _attention("verify_short_b2_k4", 2, (777, 1000), 4, 8, 2, scratch=False),
        # one layer of a small engine step with Hadamard-rotated keys: append, rotate the queries, verify
        _attention("step_rotated_b4_2k_k2", 4, (1024, 2048), 2, 32, 8, call="step", rotate=True),
        # small heads and an engine's smallest pages: head_dim 64, 16-token pages, odd draft count
        _attention("verify_d64_page16_b16_4k_k3", 16, (1024, 4096), 3, 32, 8, D=64, PAGE=16),
        # one layer of a 7B-shaped verify step: append 8 drafts per sequence, then verify them
        _attention("step_b8_12k_k8", 8, (8192, 16384), 8, 32, 8, call="step"),
        # plain decode of a long-context batch: one query token, eight query rows per cache head
        _attention("decode_b8_32k_k1", 8, 32768, 1, 64, 8),
        # the headline: eight drafts at 32 K tokens, the whole 64-row tile in use
        _attention("verify_b8_32k_k8", 8, 32768, 8, 64, 8),
        # a tree of sixteen drafts (the most a mask holds): 128 query rows per cache head
        _attention("tree_b4_8k_k16", 4, (4096, 8192), 16, 64, 8, call="tree", scratch=False),
        # the NVFP4 cache in a mid-size batch
        _attention("nvfp4_b8_16k_k4", 8, (8192, 16384), 4, 64, 8, fmt=1),
        # one very long sequence with large heads
        _attention("verify_d256_b1_131k_k8", 1, 131072, 8, 32, 4, D=256),
        # the largest: a ragged serving batch whose cache is ten times the L2
        _attention("verify_ragged_b32_64k_k8", 32, (4096, 65536), 8, 64, 8),
        # prefill's write: a batch of prompts appended in one call, a token count that is no multiple of anything
        _append("append_prompt_40001", 40001, 8),
        # the same for the NVFP4 cache, a shorter prompt
        _append("append_prompt_nvfp4_12289", 12289, 8, fmt=1),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    if rng.random() < 0.25:
        fmt = rng.choice([0, 0, 1])
        return _append(None, _log_int(rng, 16, 49152), rng.choice([2, 4, 8]), D=rng.choice([64, 128, 128, 256]), PAGE=rng.choice([16, 32, 64, 128]),
                       fmt=fmt, dtype=rng.choice(["bf16", "bf16", "fp16", "fp32"]), rotate=fmt == 0 and rng.random() < 0.25)
    call = rng.choice(["decode"] * 4 + ["step", "tree"])
    D = rng.choice([64, 128, 128, 128, 256])
    HKV, G = rng.choice([1, 2, 4, 8]), rng.choice([1, 2, 4, 8, 8])
    K = rng.choice([1, 1, 2, 3, 4, 5, 6, 8, 8, 16])
    fmt = rng.choice([0, 0, 0, 1]) if call == "decode" else 0
    B = _log_int(rng, 1, 32)
    hi = _log_int(rng, 128, 131072)
    # no more cache than the largest listed case has (and half of it where the query rows need two launches)
    most = 32 * 34816 * 8 * 128 // (2 if K * G > 64 else 1)
    hi = max(128, min(hi, most // (B * HKV * D)))
    lo = max(K, hi // rng.choice([1, 2, 4, 16]))
    return _attention(None, B, (lo, hi), K, HKV * G, HKV, D=D, PAGE=rng.choice([16, 32, 64, 64, 128]), fmt=fmt, call=call,
                      rotate=call == "step" and rng.random() < 0.3, scratch=rng.random() < 0.6, lens_seed=rng.randrange(1 << 16))


def _lens(case):
    r = random.Random(case["lens_seed"])
    return [r.randint(case["ctx_lo"], case["ctx_hi"]) for _ in range(case["B"])]


def _empty_cache(pages, HKV, PAGE, D, fmt):
    new = lambda row: torch.zeros(pages, HKV, PAGE, row, dtype=torch.uint8, device="cuda")
    scales = D // (16 if fmt else 32)
    return new(D // 2), new(scales), new(D // 2), new(scales)


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    HKV, D, PAGE, fmt = case["HKV"], case["D"], case["PAGE"], case["fmt"]
    chan = torch.exp(0.5 * torch.randn(1, HKV, D, generator=g, device="cuda"))

    def tokens(n, dtype=torch.bfloat16):
        k = torch.randn(n, HKV, D, generator=g, device="cuda") * chan
        return k.to(dtype), torch.randn(n, HKV, D, generator=g, device="cuda").to(dtype)

    def write(cache, k, v, slots):
        if fmt:
            uq_cuda.append_kv_nvfp4(*cache, k, v, slots, K_TS, V_TS)
        else:
            uq_cuda.append_kv(*cache, k, v, slots, rotate_k=case["rotate"])

    if case["kind"] == "append":
        T = case["T"]
        pages = -(-T // PAGE)
        cache = _empty_cache(pages, HKV, PAGE, D, fmt)
        key, value = tokens(T, DTYPES[case["dtype"]])
        perm = torch.randperm(pages, generator=g, device="cuda")
        pos = torch.arange(T, device="cuda")
        slots = perm[pos // PAGE] * PAGE + pos % PAGE
        return {"case": case, "cache": cache, "key": key, "value": value, "slots": slots}

    B, K, HQ = case["B"], case["K"], case["HQ"]
    lens = _lens(case)
    npg = [-(-n // PAGE) for n in lens]
    cache = _empty_cache(sum(npg), HKV, PAGE, D, fmt)
    perm = torch.randperm(sum(npg), generator=g, device="cuda").to(torch.int32)
    bt = torch.zeros(B, max(npg), dtype=torch.int32, device="cuda")
    new_k, new_v, new_slots, first = [], [], [], 0
    for b, n in enumerate(lens):
        bt[b, :npg[b]] = perm[first:first + npg[b]]
        first += npg[b]
        k, v = tokens(n)
        pos = torch.arange(n, device="cuda")
        slots = bt[b].long()[pos // PAGE] * PAGE + pos % PAGE
        write(cache, k, v, slots)
        new_k.append(k[n - K:])
        new_v.append(v[n - K:])
        new_slots.append(slots[n - K:])
    q = torch.randn(B, K, HQ, D, generator=g, device="cuda").bfloat16()
    st = {"case": case, "cache": cache, "q": q, "bt": bt, "sl": torch.tensor(lens, dtype=torch.int32, device="cuda"), "ws": None, "out": None}
    if case["scratch"]:
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        nsplit = uq_cuda.auto_nsplit(B, HKV, bt.shape[1], sms, K, HQ // HKV)
        st["ws"] = torch.empty(uq_cuda.workspace_floats(B, K, HQ, HKV, D, nsplit), dtype=torch.float32, device="cuda")
        st["out"] = torch.empty_like(q)
    if case["call"] == "step":
        # the engine's varlen layout, and the newest K tokens of every sequence with their slots
        st["q"] = q.view(B * K, HQ, D)
        st["out"] = None if st["out"] is None else st["out"].view(B * K, HQ, D)
        st["new"] = (torch.cat(new_k), torch.cat(new_v), torch.cat(new_slots))
    if case["call"] == "tree":
        r = random.Random(seed)
        parents = [[-1] + [r.randrange(max(0, j - 4), j) for j in range(1, K)] for _ in range(B)]
        st["mask"] = uq_cuda.parents_to_mask(parents).cuda()
    return st


def run(st):
    case, cache = st["case"], st["cache"]
    if case["kind"] == "append":
        if case["fmt"]:
            uq_cuda.append_kv_nvfp4(*cache, st["key"], st["value"], st["slots"], K_TS, V_TS)
        else:
            uq_cuda.append_kv(*cache, st["key"], st["value"], st["slots"], rotate_k=case["rotate"])
        return cache
    if case["call"] == "step":
        vllm_adapter.append_kv(*cache, *st["new"], rotate_k=case["rotate"])
        out = vllm_adapter.uq_verify_attention(st["q"], *cache, st["bt"], st["sl"], case["K"], workspace=st["ws"], out=st["out"], rotate_q=case["rotate"])
        return (out,) + tuple(cache)
    if case["call"] == "tree":
        return uq_cuda.uq_tree_decode(st["q"], *cache, st["bt"], st["sl"], st["mask"], workspace=st["ws"], out=st["out"])
    ts = {"fmt": 1, "k_ts": K_TS, "v_ts": V_TS} if case["fmt"] else {}
    return uq_cuda.uq_decode_cuda(st["q"], *cache, st["bt"], st["sl"], workspace=st["ws"], out=st["out"], **ts)


def work(case):
    HKV, D = case["HKV"], case["D"]
    row = D // 2 + D // (16 if case["fmt"] else 32)   # one key or value of one head in the cache
    if case["kind"] == "append":
        size = 4 if case["dtype"] == "fp32" else 2
        return {"bytes": case["T"] * (2 * HKV * (D * size + row) + 8), "flops": 0}
    lens, B, K, HQ = _lens(case), case["B"], case["K"], case["HQ"]
    n = sum(lens)
    by = n * HKV * 2 * row + 2 * (B * K * HQ * D * 2) + 4 * B + 4 * sum(-(-m // case["PAGE"]) for m in lens)
    if case["call"] == "step":
        by += B * K * (2 * HKV * (D * 2 + row) + 8)
    return {"bytes": by, "flops": 4 * n * HQ * K * D}


def tolerance(case):
    if case["kind"] == "append":
        return "exact"
    # Against the same attention in 64 bits (cache dequantised exactly), the cases above and drawn ones show a relative error of
    # 1.6e-3 .. 1.7e-3 - the bf16 rounding of the result itself, 1.62e-3 .. 1.71e-3 - and a largest one of 4.5e-3: about four times that.
    return {"rel": 7e-3, "max": 2e-2}
