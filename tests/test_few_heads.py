"""Items of at most 32 tile rows, most of which run on a kernel of their own (slots on the rows of the tensor-core tile, the pair
splits the slots; items that are short on average stay on the 128-row kernel, and with an fp8 cache those of more than 16 rows): edges of its 48-slot
tiles and of its 16- and 32-row forms, moving references, sink and second pool.  (17 to 32 rows of an fp8 cache at the edges of the other kernel's
tiles are in test_paired_fp8.)"""
import math

import numpy as np
import pytest

from helpers import TOL_BF16, TOL_FP8, check_lse, check_out, few_heads_form
from opfoundry_b200 import api, synth

pytestmark = pytest.mark.gpu

SCALE = 1.0 / math.sqrt(192.0)


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("B,H,topk", [(2, 1, 1), (2, 16, 2), (3, 16, 95), (2, 16, 96), (2, 17, 97), (2, 32, 193), (1, 7, 1000), (40, 16, 300), (40, 16, 700)])
def test_tile_edges(built_lib, oracle, fp8, B, H, topk):
    from gpu_util import run_gpu, run_oracle
    case = synth.make_decode_case(B, H, 1024, topk, fp8=fp8, paged=fp8, pad_frac=0.1 if topk > 90 else 0.0, scatter_pad=True, seed=H + topk)
    case["indices"][0] = -1     # a query without any position
    g_out, g_lse, _ = run_gpu(case, SCALE)
    r_out, r_lse = run_oracle(oracle, case, SCALE)
    check_out(g_out, r_out, **(TOL_FP8 if fp8 else TOL_BF16))
    check_lse(g_lse, r_lse)


@pytest.mark.parametrize("H,s_q", [(8, 2), (8, 3), (8, 4), (16, 2)])
def test_stacked_rows(built_lib, oracle, H, s_q):
    from gpu_util import run_gpu, run_oracle
    case = synth.make_decode_case(5, H, 2048, 700, s_q=s_q, fp8=True, paged=True, share_mtp="coin", seed=3 * H + s_q)
    case["mtp_shared"][:2] = [True, False]
    case["indices"][:s_q] = case["indices"][0]
    g_out, g_lse, _ = run_gpu(case, SCALE, mtp_shared=case["mtp_shared"])
    r_out, r_lse = run_oracle(oracle, case, SCALE)
    check_out(g_out, r_out, **TOL_FP8)
    check_lse(g_lse, r_lse)


@pytest.mark.parametrize("H", [16, 32])
def test_references_move(built_lib, oracle, H):
    """Scores that grow along the list: the reference maxima move in later tiles and the sums so far are rescaled."""
    from gpu_util import run_gpu, run_oracle
    case = synth.make_decode_case(2, H, 1024, 600, seed=H)
    case["indices"] = np.sort(case["indices"], axis=1)
    f = (case["kv"].astype(np.uint32) << 16).view(np.float32).reshape(2, 1024, 576) * np.linspace(0.1, 16.0, 1024, dtype=np.float32)[None, :, None]
    f[:, :, :512] /= np.linspace(0.1, 16.0, 1024, dtype=np.float32)[None, :, None] ** 0.5
    case["kv"] = synth.f32_to_bf16_bits(f.reshape(case["kv"].shape))
    g_out, g_lse, _ = run_gpu(case, SCALE)
    r_out, r_lse = run_oracle(oracle, case, SCALE)
    check_out(g_out, r_out, **TOL_BF16)
    check_lse(g_lse, r_lse)


@pytest.mark.parametrize("H", [16, 24])
def test_sink_and_second_pool(built_lib, oracle, H):
    import torch
    from opfoundry_b200 import api
    from test_v4_ext import _make
    case, idx, split, kv2, sink = _make(T=120, H=H, topk=100, rows2=32, seed=H)
    idx[7] = -1
    bf = lambda a: torch.from_numpy(a.view(np.int16)).cuda().view(torch.bfloat16)
    plan = api.mla_decode_plan_create(120, H, 100, 120, valid_len_hint=(idx >= 0).sum(1))
    out, lse = api.mla_v4_launch_pipeline(bf(case["q"]), bf(case["kv"]), torch.from_numpy(idx).cuda(), plan, SCALE, attn_sink=torch.from_numpy(sink).cuda(),
                                          kv2=bf(kv2), pool_split=torch.from_numpy(split).cuda())
    r_out, r_lse = oracle.sparse_mla_v4(case["q"], case["kv"], idx, SCALE, attn_sink=sink, kv2=kv2, pool_split=split, s_q=120)
    check_out(out.view(torch.int16).cpu().numpy().view(np.uint16), r_out, **TOL_BF16)
    check_lse(lse.cpu().numpy(), r_lse)


EDGES = [1, 2, 3, 31, 47, 48, 49, 94, 95, 96, 97, 98, 143, 144, 145, 192, 193, 0]   # a CTA takes half of the slots, 48 a tile


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("H", [1, 16, 17, 32])
def test_tile_edges_among_long_items(built_lib, oracle, H, fp8):
    """Items at the edges of the 48-slot tiles, in one list with items long enough for the few-heads kernel."""
    from gpu_util import run_gpu, run_oracle
    lens = np.array([x for n in EDGES for x in (n, 1100)] + [1100] * (0 if H <= 16 else 42), np.int32)
    case = synth.make_decode_case(len(lens), H, 1216, 1100, fp8=fp8, paged=fp8, seed=H)
    for r, n in enumerate(lens):
        case["indices"][r, n:] = -1
    kw = dict(num_sms=14, valid_len_hint=lens)
    assert few_heads_form(api.plan_host(len(lens), H, 1100, **kw), fp8) == (16 if H <= 16 else 0 if fp8 else 32)
    g_out, g_lse, _ = run_gpu(case, SCALE, **kw)
    r_out, r_lse = run_oracle(oracle, case, SCALE)
    check_out(g_out, r_out, **(TOL_FP8 if fp8 else TOL_BF16))
    check_lse(g_lse, r_lse)


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("H,topk", [(16, 96), (16, 128), (32, 128), (32, 500)])
def test_short_items_stay_on_the_128_row_kernel(built_lib, H, topk, fp8):
    """There a head's result does not depend on the other heads, so it has the bits that it has among 64 heads."""
    from gpu_util import run_gpu
    case = synth.make_decode_case(40, 64, 1024, topk, fp8=fp8, paged=fp8, seed=topk)
    few = dict(case, q=np.ascontiguousarray(case["q"][:, :H]))
    w_out, w_lse, _ = run_gpu(case, SCALE)
    g_out, g_lse, _ = run_gpu(few, SCALE)
    assert np.array_equal(g_out, w_out[:, :H]) and np.array_equal(g_lse, w_lse[:, :H])


def _moving_references(B, H, topk, *, s_q, fp8, share, seed):
    """Scores that grow along the sorted lists by the rope columns alone, so V keeps its size: the largest score of a head, in
    powers of two, rises to about a hundred, and its reference maximum moves again and again in both halves of an item."""
    case = synth.make_decode_case(B, H, topk + 64, topk, s_q=s_q, fp8=fp8, paged=fp8, seed=seed)
    case["indices"] = np.sort(case["indices"], axis=1)
    if share:
        for b in range(0, B, 2):
            case["indices"][b * s_q:(b + 1) * s_q] = case["indices"][b * s_q]
    n = case["kv"].shape[0]
    pos = np.tile(np.arange(n // B, dtype=np.float32), B) * (B / n)     # a row's place in its sequence, 0 to 1
    if fp8:
        rows = (case["block_table"].reshape(-1)[:, None] * 64 + np.arange(64)).reshape(-1)
        pos[rows] = pos.copy()
        rope = case["kv"][:, 528:].copy().view(np.uint16)
    else:
        rope = case["kv"][:, 512:]
    bits = synth.f32_to_bf16_bits((rope.astype(np.uint32) << 16).view(np.float32) * (0.05 + 80.0 * pos)[:, None])
    if fp8:
        case["kv"][:, 528:] = bits.view(np.uint8).reshape(n, 128)
    else:
        case["kv"][:, 512:] = bits
    return case


def _moves(case, half_slots, fp8):
    """How often a head's reference moves in each half of the first item, tile by tile, as the kernel moves it: the most of any head."""
    q = (case["q"][0].astype(np.uint32) << 16).view(np.float32)[:, 512:]
    idx = case["indices"][0]
    rows = case["block_table"][0][idx // 64] * 64 + idx % 64 if fp8 else idx
    rope = np.ascontiguousarray(case["kv"][rows][:, 528:]).view(np.uint16) if fp8 else case["kv"][rows][:, 512:]
    y = (rope.astype(np.uint32) << 16).view(np.float32) @ q.T * (SCALE * 1.4427)      # the other columns add a few units at most
    out = []
    for part in (y[:half_slots], y[half_slots:]):
        ref, n = part[:48].max(axis=0), np.zeros(q.shape[0], int)
        for t in range(48, len(part), 48):
            top = part[t:t + 48].max(axis=0)
            n += top > ref + 8
            ref = np.where(top > ref + 8, top, ref)
        out.append(int(n.max()))
    return out


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("H,s_q,share", [(16, 1, False), (32, 1, False), (16, 2, True)])
def test_many_long_items_per_list(built_lib, oracle, H, s_q, share, fp8):
    """Lists of several items of a dozen tiles per CTA: the rings and the parities of the barriers wrap many times, references
    move several times in an item, and (share) stacked items of 32 rows and single ones of 16 follow one another in a list."""
    from gpu_util import run_gpu, run_oracle
    B, topk = 8 // s_q + 4, 1216
    case = _moving_references(B, H, topk, s_q=s_q, fp8=fp8, share=share, seed=H + s_q)
    assert min(_moves(case, topk // 2, fp8)) >= 4
    shared = [share and b % 2 == 0 for b in range(B)]
    kw = dict(num_sms=4, mtp_shared=shared if share else None)
    assert few_heads_form(api.plan_host(B * s_q, H, topk, s_q, **kw), fp8) == (16 if H * s_q == 16 else 0 if fp8 else 32)
    g_out, g_lse, plan = run_gpu(case, SCALE, **kw)
    works, indptr = plan.read_works()
    lists = [works[a:b] for a, b in zip(indptr, indptr[1:])]
    assert max(len(x) for x in lists) >= 4 and max(w.k_end - w.k_begin for w in works) >= 2 * 8 * 48
    if share:
        assert any(len({w.stacked_rows for w in x}) > 1 for x in lists)
    r_out, r_lse = run_oracle(oracle, case, SCALE)
    check_out(g_out, r_out, **(TOL_FP8 if fp8 else TOL_BF16))
    check_lse(g_lse, r_lse)


@pytest.mark.parametrize("H,s_q", [(8, 2), (8, 4), (16, 2)])
def test_stacked_rows_of_a_bf16_cache(built_lib, oracle, H, s_q):
    from gpu_util import run_gpu, run_oracle
    case = synth.make_decode_case(5, H, 2048, 900, s_q=s_q, share_mtp="coin", seed=5 * H + s_q)
    case["mtp_shared"][:2] = [True, False]
    case["indices"][:s_q] = case["indices"][0]
    kw = dict(mtp_shared=case["mtp_shared"])
    assert few_heads_form(api.plan_host(5 * s_q, H, 900, s_q, **kw), fp8=False) == (16 if H * s_q == 16 else 32)
    g_out, g_lse, _ = run_gpu(case, SCALE, **kw)
    r_out, r_lse = run_oracle(oracle, case, SCALE)
    check_out(g_out, r_out, **TOL_BF16)
    check_lse(g_lse, r_lse)


@pytest.mark.parametrize("H,B", [(16, 2), (24, 2), (16, 90)])
def test_sink_with_an_fp8_cache(built_lib, oracle, H, B):
    import torch
    from gpu_util import to_dev
    topk = 1000
    case = synth.make_decode_case(B, H, 1024, topk, fp8=True, paged=True, seed=H + B)
    case["indices"][0] = -1      # nothing but the sink
    sink = np.random.default_rng(H).normal(0.0, 2.0, H).astype(np.float32)
    assert few_heads_form(api.plan_host(B, H, topk)) == (16 if H <= 16 else 0)
    d = to_dev(case)
    out, lse = api.mla_v4_launch_pipeline(d["q"], d["kv"], d["indices"], api.mla_decode_plan_create(B, H, topk), SCALE, attn_sink=torch.from_numpy(sink).cuda(),
                                          block_table=d["block_table"], page_block_size=64)
    r_out, r_lse = oracle.sparse_mla_v4(case["q"], case["kv"], case["indices"], SCALE, attn_sink=sink, kv_is_fp8=True, block_table=case["block_table"],
                                        page_block_size=64)
    check_out(out.view(torch.int16).cpu().numpy().view(np.uint16), r_out, **TOL_FP8)
    check_lse(lse.cpu().numpy(), r_lse)


@pytest.mark.parametrize("B,H,s_q,fp8,share", [(2, 16, 1, True, False), (90, 16, 1, False, False), (3, 24, 1, True, False), (40, 16, 2, True, True), (4, 64, 1, True, False),
                                                (4, 64, 1, False, False), (74, 128, 1, False, False), (40, 64, 2, False, True), (5, 48, 2, False, True)])
def test_rows_go_to_every_peer(built_lib, B, H, s_q, fp8, share):
    """The gathered buffers of two destinations on this GPU (the other rank's arrival is set beforehand, so nothing is waited
    for): both hold this rank's heads, bit for bit what the call without peers gives, and nothing else is written."""
    import ctypes as C
    import torch
    from gpu_util import to_dev
    topk, H_all, h0, T = 1500, 4 * H, H, B * s_q
    case = synth.make_decode_case(B, H, 2048, topk, s_q=s_q, fp8=fp8, paged=fp8, share_mtp="coin" if share else None, seed=B)
    plan = api.mla_decode_plan_create(T, H, topk, s_q, mtp_shared=case["mtp_shared"] if share else None)
    d = to_dev(case)
    kw = dict(block_table=d["block_table"], page_block_size=case["page_block_size"], kv_batch_stride_rows=case["kv_batch_stride_rows"])
    want_out, want_lse = api.mla_decode_launch_pipeline(d["q"], d["kv"], d["indices"], plan, SCALE, **kw)
    outs = [torch.full((T, H_all, 512), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    lses = [torch.full((T, H_all), 7.0, device="cuda") for _ in range(2)]
    flags = torch.zeros(2, api.MAX_PEERS, dtype=torch.int32, device="cuda")
    flags[0, 1] = 1
    a = api.make_args(d["q"], d["kv"], d["indices"], plan, SCALE, out=outs[0][:, h0:h0 + H], lse=None, **kw)
    po = api.PeerOutputs()
    po.num_peers, po.my_rank, po.lse_stride_row, po.step = 2, 0, H_all, 1
    for r in range(2):
        po.out[r], po.lse[r], po.flags[r] = outs[r].data_ptr() + h0 * 1024, lses[r].data_ptr() + h0 * 4, flags[r].data_ptr()
    torch.cuda.synchronize()
    api._check(api.lib().dsa_v32_decode_pipeline_allgather(C.byref(a), C.byref(po), api._stream()), "dsa_v32_decode_pipeline_allgather")
    api._check(api.lib().dsa_v32_device_status(C.byref(a), api._stream()), "dsa_v32_device_status")
    for o, l in zip(outs, lses):
        assert torch.equal(o[:, h0:h0 + H].view(torch.int16), want_out.view(torch.int16)) and torch.equal(l[:, h0:h0 + H], want_lse)
        assert torch.all(o[:, :h0] == 7) and torch.all(o[:, h0 + H:] == 7) and torch.all(l[:, :h0] == 7) and torch.all(l[:, h0 + H:] == 7)
    assert flags[:, 0].tolist() == [1, 1]


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("B,fp8,H", [(2, False, 16), (2, True, 16), (90, False, 16), (90, True, 16), (2, False, 72), (74, False, 128)])
def test_infinite_and_nan_sinks(built_lib, B, fp8, H, value):
    """A row without positions is zeros whatever its sink is, also when the pieces are merged; an infinite sink takes all of
    a row's weight, a NaN is no term (both as in the 128-row kernel)."""
    import torch
    from gpu_util import to_dev
    topk = 1000
    case = synth.make_decode_case(B, H, 1024, topk, fp8=fp8, paged=fp8, seed=B)
    case["indices"][0] = -1
    case["indices"][1, :500] = -1      # nothing in the first CTA's half
    d = to_dev(case)
    plan = api.mla_decode_plan_create(B, H, topk)
    kw = dict(block_table=d["block_table"], page_block_size=case["page_block_size"], kv_batch_stride_rows=case["kv_batch_stride_rows"])
    run = lambda sink: api.mla_v4_launch_pipeline(d["q"], d["kv"], d["indices"], plan, SCALE, attn_sink=torch.tensor(sink, device="cuda"), **kw)
    sink = [0.5] * H
    sink[1::2] = [value] * (H // 2)
    out, lse = run(sink)
    assert torch.all(out[0] == 0) and torch.all(lse[0, 1::2] == float("inf"))
    if value == float("inf"):
        if plan.info.num_partials:     # (the merge has no finite reference for a piece of infinite weight)
            return
        assert torch.all(out[:, 1::2] == 0) and torch.all(lse[:, 1::2] == float("inf"))
    else:
        w_out, w_lse = run([0.5, -float("inf")] * (H // 2))
        assert torch.equal(out[1:], w_out[1:]) and torch.equal(lse[1:], w_lse[1:])
