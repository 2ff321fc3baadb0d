"""The 128-row kernel (one pair MMA over the two CTAs of a cluster, 64 tile rows and 32 of a tile's 64 slots each): edges of its
tiles and row halves, lists of many short items (the ring of stages that Q and the tiles share), moving references, stacked rows."""
import math

import numpy as np
import pytest

from helpers import TOL_BF16, TOL_FP8, check_lse, check_out, few_heads_form
from opfoundry_b200 import api, synth
from test_few_heads import _moving_references

pytestmark = pytest.mark.gpu

SCALE = 1.0 / math.sqrt(192.0)


def _compare(oracle, case, **kw):
    from gpu_util import run_gpu, run_oracle
    T, H = case["q"].shape[:2]
    assert few_heads_form(api.plan_host(T, H, case["topk"], case["s_q"], **kw), case["fp8"]) == 0
    g_out, g_lse, plan = run_gpu(case, SCALE, **kw)
    r_out, r_lse = run_oracle(oracle, case, SCALE)
    check_out(g_out, r_out, **(TOL_FP8 if case["fp8"] else TOL_BF16))
    check_lse(g_lse, r_lse)
    return plan


EDGES = [1, 2, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 191, 193, 255, 256, 257, 321, 0]


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("H,num_sms", [(33, 2), (64, 4), (72, 6), (128, 2), (128, 148), (200, 4)])
def test_tile_edges_in_lists_of_short_items(built_lib, oracle, H, num_sms, fp8):
    lens = np.array(EDGES + EDGES[::-1], np.int32)
    case = synth.make_decode_case(len(lens), H, 512, 321, fp8=fp8, paged=fp8, seed=H + num_sms)
    for r, n in enumerate(lens):
        case["indices"][r, n:] = -1
    _compare(oracle, case, num_sms=num_sms, valid_len_hint=lens)


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("H,s_q", [(64, 1), (128, 1), (64, 2)])
def test_references_move_in_long_items(built_lib, oracle, H, s_q, fp8):
    B, topk = 6, 1216
    case = _moving_references(B, H, topk, s_q=s_q, fp8=fp8, share=s_q > 1, seed=H + s_q)
    _compare(oracle, case, num_sms=4, mtp_shared=[b % 2 == 0 for b in range(B)] if s_q > 1 else None)


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("H,s_q", [(24, 4), (40, 3), (64, 2), (56, 2)])
def test_stacked_rows_over_both_ctas(built_lib, oracle, H, s_q, fp8):
    """Stacked query rows that end inside, at and beyond the 64 tile rows of a CTA, among items of a single row."""
    case = synth.make_decode_case(7, H, 1024, 200, s_q=s_q, fp8=fp8, paged=fp8, share_mtp="coin", seed=H + s_q)
    case["mtp_shared"][:2] = [True, False]
    case["indices"][:s_q] = case["indices"][0]
    plan = _compare(oracle, case, num_sms=6, mtp_shared=case["mtp_shared"])
    assert any(w.stacked_rows > 1 for w in plan.read_works()[0])


@pytest.mark.parametrize("T,H,topk,strides", [(1, 128, 512, (1 << 41, 576, 1)), (1, 64, 100, (1 << 50, 576, 1)), (40, 1, 64, (576, 1 << 41, 1)), (1, 1, 31, (1 << 45, 1 << 41, 1))])
def test_any_stride_of_a_single_row_or_head(built_lib, T, H, topk, strides):
    """A stride that nothing follows is not used, so it may be larger than a tensor map takes."""
    import torch
    case = synth.make_decode_case(T, H, 1024, topk, seed=H)
    bf = lambda a: torch.from_numpy(a.view(np.int16)).cuda().view(torch.bfloat16)
    q, kv, idx = bf(case["q"]), bf(case["kv"]), torch.from_numpy(case["indices"]).cuda()
    plan = api.mla_decode_plan_create(T, H, topk)
    kw = dict(kv_batch_stride_rows=1024)
    want, want_lse = api.mla_decode_launch_pipeline(q, kv, idx, plan, SCALE, **kw)
    out, lse = api.mla_decode_launch_pipeline(q.as_strided((T, H, 576), strides), kv, idx, plan, SCALE, **kw)
    assert torch.equal(out.view(torch.int16), want.view(torch.int16)) and torch.equal(lse, want_lse)


@pytest.mark.parametrize("T,H,strides", [(1, 128, (1 << 40, 576, 1)), (1, 8, (1 << 40, 576, 1)), (3, 1, (576, 1 << 41, 1)), (1, 40, (1 << 39, 576, 1))])
def test_strides_beyond_a_tensor_map_stay_refused_with_an_fp8_cache(built_lib, T, H, strides):
    """Whichever kernel the number of heads would lead to."""
    from gpu_util import to_dev
    case = synth.make_decode_case(T, H, 1024, 100, fp8=True, paged=True, seed=H)
    d = to_dev(case)
    plan = api.mla_decode_plan_create(T, H, 100)
    with pytest.raises(api.DsaError):
        api.mla_decode_launch_pipeline(d["q"].as_strided((T, H, 576), strides), d["kv"], d["indices"], plan, SCALE, block_table=d["block_table"], page_block_size=64)


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("B,H", [(3, 128), (80, 72)])
def test_repeated_launches_give_the_same_bits(built_lib, B, H, fp8):
    """Split items with their merge, and whole items several to a list: which warp sums what is fixed by the plan."""
    from gpu_util import run_gpu
    case = synth.make_decode_case(B, H, 1024, 700, fp8=fp8, paged=fp8, pad_frac=0.1, seed=B)
    first = run_gpu(case, SCALE, num_sms=40)
    assert (first[2].info.num_partials > 0) == (B == 3)
    for _ in range(5):
        out, lse, _ = run_gpu(case, SCALE, num_sms=40)
        assert np.array_equal(out, first[0]) and np.array_equal(lse, first[1])


@pytest.mark.parametrize("what", ["sink", "pool", "both"])
@pytest.mark.parametrize("B,H,s_q,num_sms", [(3, 128, 1, 0), (5, 40, 1, 24), (6, 24, 4, 60), (7, 64, 2, 6)])
def test_sink_and_second_pool_of_split_and_stacked_items(built_lib, oracle, B, H, s_q, num_sms, what):
    """Pieces (the sink counts once, in the piece that starts the list; the second pool begins inside a piece or between two) and
    stacked rows, which share a list and the slot where the second pool begins."""
    import torch
    topk, T = 900, B * s_q
    case = synth.make_decode_case(B, H, 1024, topk, s_q=s_q, pad_frac=0.1, scatter_pad=True, share_mtp="coin" if s_q > 1 else None, seed=H + B)
    rng = np.random.default_rng(H)
    idx, rows2 = case["indices"], 96
    split = np.repeat(rng.choice([0, 1, 63, 128, 500, 640, topk - 1, topk], B), s_q).astype(np.int32)
    split[:s_q] = 321
    sink = (rng.normal(size=H) * 3.0).astype(np.float32)
    kv2 = synth.normal_bf16(H, "kv2", (rows2, 576))
    if what == "sink":
        kv2 = split = None
    else:
        for b in range(B):     # rows of the second pool, one list for a sequence's rows where they share it
            for r in range(b * s_q, (b + 1) * s_q):
                if s_q > 1 and r > b * s_q and case["mtp_shared"][b]:
                    idx[r] = idx[b * s_q]
                else:
                    idx[r, split[r]:] = rng.integers(-1, rows2, topk - split[r])
    idx[T - 1] = -1            # no position
    shared = case["mtp_shared"].astype(bool).copy() if s_q > 1 else None
    if s_q > 1:
        shared[B - 1] = False
    if what == "pool":
        sink = None
    kw = dict(num_sms=num_sms, mtp_shared=shared)
    plan = api.mla_decode_plan_create(T, H, topk, s_q, **kw)
    works = plan.read_works()[0]
    assert plan.info.num_partials > 0 and (s_q == 1 or any(w.stacked_rows > 1 for w in works))
    bf = lambda a: torch.from_numpy(a.view(np.int16)).cuda().view(torch.bfloat16)
    dev = lambda a: None if a is None else torch.from_numpy(a).cuda()
    out, lse = api.mla_v4_launch_pipeline(bf(case["q"]), bf(case["kv"]), dev(idx), plan, SCALE, attn_sink=dev(sink), kv2=None if kv2 is None else bf(kv2),
                                          pool_split=dev(split), kv_batch_stride_rows=1024)
    r_out, r_lse = oracle.sparse_mla_v4(case["q"], case["kv"], idx, SCALE, attn_sink=sink, kv2=kv2, pool_split=split, s_q=s_q, kv_batch_stride_rows=1024)
    check_out(out.view(torch.int16).cpu().numpy().view(np.uint16), r_out, **TOL_BF16)
    check_lse(lse.cpu().numpy(), r_lse)
