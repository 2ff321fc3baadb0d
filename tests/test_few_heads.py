"""Items of at most 32 tile rows, most of which run on a kernel of their own (slots on the rows of the tensor-core tile, the pair
splits the slots; items that are short on average stay on the 128-row kernel): edges of its 48-slot tiles and of its 16- and
32-row forms, moving references, sink and second pool."""
import math

import numpy as np
import pytest

from helpers import TOL_BF16, TOL_FP8, check_lse, check_out, few_heads_form
from opfoundry_b200 import api, synth

pytestmark = pytest.mark.gpu

SCALE = 1.0 / math.sqrt(192.0)


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("B,H,topk", [(2, 1, 1), (2, 16, 2), (3, 16, 95), (2, 16, 96), (2, 17, 97), (2, 32, 193), (1, 7, 1000), (40, 16, 300)])
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
    assert few_heads_form(api.plan_host(len(lens), H, 1100, **kw)) == (16 if H <= 16 else 32)
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
