"""The work whose speed matters here, as calls of the public Python entry points: sparse-MLA decode on fp8 and bf16
caches, causal prefill, the v4 form (attention sink, second pool), the index-list producer, the cache write and the
host-buffer serving step.

A case is a dict of plain values.  `listed()` are the ones that are followed; `draw()` gives others of the same ranges.
Sizes are those of the benchmark configurations, the tests and the harness of this repository, and odd ones between.
"""
import math
import random

import torch

from opfoundry_b200 import api, workloads

SCALE = 1.0 / math.sqrt(192.0)
PAGE = 64


def listed():
    return [
        # one sequence, one token: the latency of a single user's decode step
        decode("decode_fp8_b1", fp8=True, B=1, kv_len=32768),
        # a small serving batch: fewer sequences than CTA pairs, so lists are split and merged
        decode("decode_fp8_b16", fp8=True, B=16, kv_len=32768),
        # the serving batch of the headline benchmark: 128 heads, 5 % of the slots padding
        decode("decode_fp8_b64", fp8=True, B=64, kv_len=32768),
        # one rank of a head-sharded (TP8) deployment with one MTP token: 16 heads, half of the sequences share a list
        decode("decode_fp8_mtp_tp8", fp8=True, B=128, H=16, s_q=2, share=True, kv_len=16384, pad=0.0),
        # the small bf16 configuration: two sequences, 16 heads, contiguous cache
        decode("decode_bf16_b2_h16", fp8=False, B=2, H=16, kv_len=4096, paged=False, pad=0.0),
        # prefill of a 4096-token prompt, 128 heads: the largest case
        prefill("prefill_bf16_4096", T=4096),
        # a later chunk of a prompt of odd length on half of the heads, odd top-k (chunked prefill, TP2)
        prefill("prefill_bf16_chunk", T=3001, q_begin=1733, H=64, topk=1500),
        # v4-style prefill: attention sink per head and the chunk's own rows in a second pool
        prefill("prefill_v4_sink_pool", T=2048, q_begin=1024, topk=640, pool=512, sink=True),
        # index lists of a decode batch from the indexer's scores
        dict(name="topk_select_decode", kind="select", rows=64, kv_len=32768, topk=2048, causal=False),
        # index lists of a prefill chunk: causal valid lengths, many rows
        dict(name="topk_select_prefill", kind="select", rows=2048, kv_len=8192, topk=2048, causal=True),
        # quantised cache write of a prefill chunk to scattered pages
        dict(name="pack_fp8_rows", kind="pack", rows=8192, scatter=True),
        # the serving step on pinned host buffers, copies overlapped with the kernels
        decode("decode_fp8_host_step", kind="host", fp8=True, B=64, kv_len=32768, chunks=8, lanes=4),
    ]


def decode(name, *, fp8, B, kv_len, H=128, topk=2048, s_q=1, share=False, paged=True, pad=0.05, kind="decode", chunks=1, lanes=1):
    return dict(name=name, kind=kind, fp8=fp8, B=B, H=H, kv_len=kv_len, topk=topk, s_q=s_q, share=share, paged=paged, pad=pad,
                chunks=chunks, lanes=lanes)


def prefill(name, *, T, q_begin=0, H=128, topk=2048, pool=0, sink=False):
    return dict(name=name, kind="prefill", T=T, q_begin=q_begin, H=H, topk=topk, pool=pool, sink=sink)


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: the kinds of work above with sizes over their whole range."""
    what = rng.choice(["fp8", "fp8", "fp8", "mtp", "bf16", "prefill", "prefill", "v4", "select", "select", "pack", "host"])
    if what == "fp8":
        c = decode("", fp8=True, B=_log_int(rng, 1, 160), H=rng.choice([128, 128, 128, 64]), kv_len=PAGE * _log_int(rng, 32, 512),
                   topk=rng.choice([2048, 2048, 1024, _log_int(rng, 100, 2047)]), pad=rng.choice([0.0, 0.05, 0.2]))
    elif what == "mtp":
        c = decode("", fp8=True, B=_log_int(rng, 4, 128), H=rng.choice([16, 32, 64, 128]), s_q=2, share=rng.random() < 0.7,
                   kv_len=PAGE * _log_int(rng, 64, 256), pad=0.0)
    elif what == "bf16":
        c = decode("", fp8=False, B=_log_int(rng, 1, 64), H=rng.choice([16, 64, 128]), kv_len=PAGE * _log_int(rng, 40, 256),
                   topk=rng.choice([2048, _log_int(rng, 100, 2047)]), paged=rng.random() < 0.7, pad=rng.choice([0.0, 0.05]))
    elif what == "prefill":
        T = _log_int(rng, 96, 4096)
        c = prefill("", T=T, q_begin=rng.choice([0, 0, int(T * rng.uniform(0.2, 0.8))]), H=rng.choice([128, 128, 64, 16]),
                    topk=rng.choice([2048, 2048, _log_int(rng, 200, 2047)]))
    elif what == "v4":
        T = _log_int(rng, 256, 3000)
        c = prefill("", T=T, q_begin=T // 2, topk=rng.choice([640, _log_int(rng, 300, 2048)]), pool=rng.choice([0, _log_int(rng, 64, 1024)]), sink=True)
    elif what == "select":
        causal = rng.random() < 0.5
        c = dict(name="", kind="select", rows=_log_int(rng, 64, 3000) if causal else _log_int(rng, 1, 160),
                 kv_len=_log_int(rng, 3000, 10000) if causal else _log_int(rng, 4096, 131072),
                 topk=rng.choice([2048, 2048, _log_int(rng, 64, 2047)]), causal=causal)
    elif what == "pack":
        c = dict(name="", kind="pack", rows=_log_int(rng, 1, 60000), scatter=rng.random() < 0.5)
    else:
        chunks = rng.choice([1, 4, 8])
        c = decode("", kind="host", fp8=True, B=8 * rng.randint(2, 10), kv_len=PAGE * _log_int(rng, 64, 512), chunks=chunks,
                   lanes=rng.choice([1, 2, 4]) if chunks > 1 else 1)
    del c["name"]
    return c


# ------------------------------------------------------------------ what a program has in hand before the call
def prepare(case, seed):
    s = {"decode": _prepare_decode, "host": _prepare_decode, "prefill": _prepare_prefill, "select": _prepare_select, "pack": _prepare_pack}[case["kind"]](case, seed)
    s["case"] = case
    return s


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _shared(case, seed):
    """Per sequence, whether its query rows carry one list (a coin flip by the seed)."""
    r = random.Random(seed)
    return [case["share"] and r.random() < 0.5 for _ in range(case["B"])]


def _prepare_decode(case, seed):
    B, H, topk, s_q, kv_len = case["B"], case["H"], case["topk"], case["s_q"], case["kv_len"]
    g = _gen(seed)
    rows = B * s_q
    if case["fp8"]:
        kv = workloads.make_fp8_cache(B * kv_len, seed + 1)
    else:
        kv = torch.randn(B * kv_len, api.D_QK, generator=g, device="cuda").to(torch.bfloat16)
    table = torch.randperm(B * kv_len // PAGE, generator=g, device="cuda").to(torch.int32).view(B, -1).contiguous() if case["paged"] else None
    q = torch.randn(rows, H, api.D_QK, generator=g, device="cuda").to(torch.bfloat16)
    idx = torch.full((rows, topk), -1, dtype=torch.int32, device="cuda")
    sel = workloads.unique_topk(rows, kv_len, topk, g, "cuda")
    idx[:, :sel.shape[1]] = sel
    if int(case["pad"] * topk):
        idx[:, topk - int(case["pad"] * topk):] = -1
    shared = _shared(case, seed)
    for b in range(B):
        if shared[b]:
            idx[b * s_q:(b + 1) * s_q] = idx[b * s_q].clone()
    s = dict(q=q, kv=kv, idx=idx, kw=dict(block_table=table, page_block_size=PAGE, kv_batch_stride_rows=0 if case["paged"] else kv_len),
             out=torch.empty(rows, H, api.D_V, dtype=torch.bfloat16, device="cuda"), lse=torch.empty(rows, H, device="cuda"))
    if case["kind"] == "decode":
        s["plan"] = api.mla_decode_plan_create(rows, H, topk, s_q, mtp_shared=shared if any(shared) else None)
        return s
    # the serving step: this step's queries and lists in pinned host memory, results wanted there
    per = rows // case["chunks"]
    if case["lanes"] > 1:
        sms = torch.cuda.get_device_properties(0).multi_processor_count // case["lanes"] // 2 * 2
        s["lane_plans"] = [api.mla_decode_plan_create(per, H, topk, s_q, num_sms=sms) for _ in range(case["lanes"])]
    else:
        s["lane_plans"] = None
    s["plan"] = s["lane_plans"][0] if s["lane_plans"] else api.mla_decode_plan_create(per, H, topk, s_q)
    s["q_host"], s["idx_host"] = q.cpu().pin_memory(), idx.cpu().pin_memory()
    s["out_host"] = torch.empty(rows, H, api.D_V, dtype=torch.bfloat16).pin_memory()
    s["lse_host"] = torch.empty(rows, H).pin_memory()
    s["args"] = api.make_args(q, kv, idx, s["plan"], SCALE, out=s["out"], lse=s["lse"], **s["kw"])
    return s


def _prefill_lists(case, g):
    """Query t attends to min(t + 1, slots) positions drawn from [0, t]; with a second pool the slots after them hold
    up to pool / 4 rows of the pool.  Returns (lists, valid lengths, first slot of the second pool)."""
    T, t0, topk, pool = case["T"], case["q_begin"], case["topk"], case["pool"]
    nq = T - t0
    n2 = min(pool // 4, topk // 2) if pool else 0
    k1 = topk - n2
    t = torch.arange(t0, T, device="cuda")
    n1 = torch.minimum(t + 1, torch.tensor(k1, device="cuda"))
    idx = torch.full((nq, topk), -1, dtype=torch.int32, device="cuda")
    for r0 in range(0, nq, 1024):
        r1 = min(nq, r0 + 1024)
        keys = torch.rand(r1 - r0, T, generator=g, device="cuda")
        keys[torch.arange(T, device="cuda")[None, :] > t[r0:r1, None]] = 2.0   # positions after t sort last
        k = min(k1, T)
        sel = keys.topk(k, dim=1, largest=False).indices.to(torch.int32)
        idx[r0:r1, :k] = torch.where(torch.arange(k, device="cuda")[None, :] < n1[r0:r1, None], sel, torch.full_like(sel, -1))
    if n2:
        ext = torch.rand(nq, pool, generator=g, device="cuda").argsort(dim=1)[:, :n2].to(torch.int32)
        idx.scatter_(1, n1[:, None] + torch.arange(n2, device="cuda")[None, :], ext)
    return idx, n1 + n2, n1.to(torch.int32)


def _prepare_prefill(case, seed):
    T, H, nq = case["T"], case["H"], case["T"] - case["q_begin"]
    g = _gen(seed)
    kv = torch.randn(T, api.D_QK, generator=g, device="cuda").to(torch.bfloat16)
    q = torch.randn(nq, H, api.D_QK, generator=g, device="cuda").to(torch.bfloat16)
    idx, valid, split = _prefill_lists(case, g)
    s = dict(q=q, kv=kv, idx=idx, out=torch.empty(nq, H, api.D_V, dtype=torch.bfloat16, device="cuda"), lse=torch.empty(nq, H, device="cuda"),
             plan=api.mla_decode_plan_create(nq, H, case["topk"], nq, valid_len_hint=valid.cpu().numpy()))
    s["sink"] = torch.randn(H, generator=g, device="cuda") if case["sink"] else None
    s["kv2"] = torch.randn(case["pool"], api.D_QK, generator=g, device="cuda").to(torch.bfloat16) if case["pool"] else None
    s["split"] = split if case["pool"] else None
    return s


def _valid_lengths(case):
    """Row i of a causal chunk sees the positions up to its own; the chunk is the end of the sequence."""
    return [max(1, case["kv_len"] - case["rows"] + i + 1) if case["causal"] else case["kv_len"] for i in range(case["rows"])]


def _prepare_select(case, seed):
    scores = torch.randn(case["rows"], case["kv_len"], generator=_gen(seed), device="cuda")
    valid = torch.tensor(_valid_lengths(case), dtype=torch.int32, device="cuda") if case["causal"] else None
    return dict(scores=scores, valid=valid, out=torch.empty(case["rows"], case["topk"], dtype=torch.int32, device="cuda"))


def _prepare_pack(case, seed):
    g, n = _gen(seed), case["rows"]
    return dict(latent=torch.randn(n, api.D_V, generator=g, device="cuda"),
                rope=torch.randn(n, api.D_ROPE, generator=g, device="cuda").to(torch.bfloat16),
                out=torch.zeros(n, api.FP8_ROW_BYTES, dtype=torch.uint8, device="cuda"),
                dst=torch.randperm(n, generator=g, device="cuda") if case["scatter"] else None)


# ------------------------------------------------------------------ one pass
def run(s):
    kind = s["case"]["kind"]
    if kind == "decode":
        return api.mla_decode_launch_pipeline(s["q"], s["kv"], s["idx"], s["plan"], SCALE, out=s["out"], lse=s["lse"], check=False, **s["kw"])
    if kind == "prefill":
        if s["sink"] is not None or s["kv2"] is not None:
            return api.mla_v4_launch_pipeline(s["q"], s["kv"], s["idx"], s["plan"], SCALE, attn_sink=s["sink"], kv2=s["kv2"],
                                              pool_split=s["split"], out=s["out"], lse=s["lse"], check=False)
        return api.sparse_mla_prefill(s["q"], s["kv"], s["idx"], s["plan"], SCALE, out=s["out"], lse=s["lse"], check=False)
    if kind == "select":
        return api.topk_select(s["scores"], s["case"]["topk"], s["valid"], out=s["out"])
    if kind == "pack":
        return api.pack_fp8_rows(s["latent"], s["rope"], out=s["out"], dst_rows=s["dst"])
    api.mla_decode_step_host(s["args"], s["q_host"], s["idx_host"], s["out_host"], s["lse_host"], num_chunks=s["case"]["chunks"], lane_plans=s["lane_plans"])
    return s["out_host"], s["lse_host"]


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "select":
        n = sum(_valid_lengths(case))
        return {"bytes": 4 * n + 4 * case["rows"] * case["topk"], "flops": 0}
    if kind == "pack":
        return {"bytes": case["rows"] * (4 * api.D_V + 2 * api.D_ROPE + api.FP8_ROW_BYTES + (8 if case["scatter"] else 0)), "flops": 0}
    H, topk = case["H"], case["topk"]
    if kind == "prefill":
        rows = case["T"] - case["q_begin"]
        n2 = min(case["pool"] // 4, topk // 2) if case["pool"] else 0
        pairs = sum(min(t + 1, topk - n2) + n2 for t in range(case["q_begin"], case["T"]))
        cache = (case["T"] + case["pool"]) * api.BF16_ROW_BYTES     # every row is read once; it stays in L2
    else:
        rows = case["B"] * case["s_q"]
        n = min(topk - int(case["pad"] * topk), case["kv_len"])
        pairs = rows * n
        # distinct cache rows of a sequence: one list's when shared, else at most all of them
        row_bytes = api.FP8_ROW_BYTES if case["fp8"] else api.BF16_ROW_BYTES
        lists = case["s_q"] * (0.5 if case["share"] else 1.0) + (0.5 if case["share"] else 0.0)
        cache = case["B"] * min(lists * n, case["kv_len"]) * row_bytes
    q_and_out = rows * H * (2 * api.D_QK + 2 * api.D_V + 4)
    return {"bytes": cache + q_and_out + 4 * rows * topk, "flops": 2 * H * (api.D_QK + api.D_V) * pairs}


def tolerance(case):
    """Lists and packed bytes are exact.  The attention rounds P and the output to bf16 around fp32 sums: against the same
    attention in 64 bits `out` is off by 0.9e-3 to 2.2e-3 (2-norm, twelve rows of every listed case) and lse by 8e-7; four
    times the former is stated."""
    if case["kind"] in ("select", "pack"):
        return "exact"
    return {"rel": 8e-3}
