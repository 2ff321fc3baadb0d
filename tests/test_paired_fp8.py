"""The 128-row kernel of an fp8 cache: Q as a sum of an e5m2 and an e4m3 number per row factor, V scaled to f16 with one exponent per scale group
for a tile, which moves with the largest scale.  Tile edges, split and stacked items are in test_paired_heads."""
import math

import numpy as np
import pytest

from helpers import TOL_FP8, check_lse, check_out, few_heads_form
from opfoundry_b200 import api, synth

pytestmark = pytest.mark.gpu

SCALE = 1.0 / math.sqrt(192.0)


def _bf16(x):
    return (np.ascontiguousarray(x, np.float32).view(np.uint32) >> 16).astype(np.uint16)


def _f32(bits):
    return (bits.astype(np.uint32) << 16).view(np.float32)


def _case(seed, H=72, topk=321, B=3):
    return synth.make_decode_case(B, H, 512, topk, fp8=True, paged=True, seed=seed)


def _scales(case):
    return case["kv"][:, 512:528].view(np.float32)


def _check(oracle, case, rel=4e-3):
    """Against the oracle relative to each query row's largest output: P, V and the output are rounded to 11, 11 and 8 significant bits, the last of
    these to half of 2^-7 of a value."""
    from gpu_util import run_gpu, run_oracle
    g_out, g_lse, _ = run_gpu(case, SCALE, num_sms=4)
    r_out, r_lse = run_oracle(oracle, case, SCALE)
    g, r = _f32(g_out), _f32(r_out)
    assert np.isfinite(g).all()
    assert (np.abs(g - r) <= rel * np.abs(r).max(axis=-1, keepdims=True) + 2.0 ** -8 * np.abs(r)).all()
    check_lse(g_lse, r_lse)


@pytest.mark.parametrize("factor", [2.0 ** -60, 2.0 ** -20, 2.0 ** 12, 2.0 ** 40])
def test_caches_far_from_one(built_lib, oracle, factor):
    """All scales times a power of two, Q times its inverse: the scores stay, the output is that many times larger or smaller."""
    case = _case(5)
    kv = case["kv"].copy()
    kv[:, 512:528].view(np.float32)[:] *= np.float32(factor)
    q = _f32(case["q"]).copy()
    q[..., :512] *= np.float32(1.0 / factor)
    _check(oracle, dict(case, kv=kv, q=_bf16(q)))


def test_the_exponent_of_v_moves_within_an_item(built_lib, oracle):
    """Slots in order of growing scale: 2^30 from the first tile's rows to the last one's, in steps of which some exceed the 2^7 that pass without a move;
    the latent part of Q is zero, so every row counts."""
    case = _case(6, topk=512, B=2)
    kv, q, idx = case["kv"].copy(), _f32(case["q"]).copy(), case["indices"]
    q[..., :512] = 0.0
    for b in range(idx.shape[0]):
        pos = idx[b]
        blocks = case["block_table"][b]
        page = case["page_block_size"]
        rows = blocks[pos // page] * page + pos % page
        steps = np.array([0, 3, 6, 8, 17, 17, 29, 30], np.float32)[np.arange(512) // 64]
        kv[rows, 512:528] = (kv[rows, 512:528].copy().view(np.float32) * np.exp2(steps - 15)[:, None]).astype(np.float32).view(np.uint8)
    _check(oracle, dict(case, kv=kv, q=_bf16(q)))


def test_rows_of_zeros_and_of_very_different_size(built_lib, oracle):
    """Query rows of zeros, with one element far above the others, and with all elements tiny; cache rows whose scales are zero."""
    case = _case(7)
    q, kv = _f32(case["q"]).copy(), case["kv"].copy()
    q[:, 0] = 0.0
    q[:, 1, :512] = 0.0
    q[:, 2, 5] = 60.0
    q[:, 3, :512] *= 2.0 ** -90
    q[:, 4] *= 2.0 ** -140
    kv[::7, 512:528] = 0
    _check(oracle, dict(case, kv=kv, q=_bf16(q)))


def test_nan_codes_and_scales_reach_only_their_own_queries(built_lib):
    """The e4m3 NaN code or a NaN scale in a row makes the queries that select it NaN and no others."""
    from gpu_util import run_gpu
    case = _case(8, topk=100)
    kv, idx = case["kv"].copy(), case["indices"]
    clean, _, _ = run_gpu(case, SCALE)
    pos, page = int(idx[1, 70]), case["page_block_size"]
    row = int(case["block_table"][1][pos // page]) * page + pos % page
    for poison in (lambda r: r.__setitem__(130, 0x7F), lambda r: r[512:516].view(np.float32).__setitem__(0, np.nan)):
        bad = kv.copy()
        poison(bad[row])
        out, _, _ = run_gpu(dict(case, kv=bad), SCALE)
        assert np.isnan(_f32(out)[1]).any(axis=-1).all()
        np.testing.assert_array_equal(out[[0, 2]], clean[[0, 2]])


@pytest.mark.parametrize("num_sms", [6, 148])
def test_sinks_far_above_the_scores(built_lib, num_sms):
    """A sink 10 nats above a row's lse leaves e^-10 of its output, one 85 or 300 above it next to nothing, and lse is theirs (whole and split items)."""
    import torch
    from gpu_util import to_dev
    H, topk = 48, 700
    case = synth.make_decode_case(3, H, 1024, topk, fp8=True, paged=True, seed=9)
    d = to_dev(case)
    plan = api.mla_decode_plan_create(3, H, topk, num_sms=num_sms)
    assert (plan.info.num_partials > 0) == (num_sms == 148)
    kw = dict(block_table=d["block_table"], page_block_size=case["page_block_size"], kv_batch_stride_rows=case["kv_batch_stride_rows"])
    run = lambda sink: [x.float() for x in api.mla_v4_launch_pipeline(d["q"], d["kv"], d["indices"], plan, SCALE, attn_sink=sink, **kw)]
    out0, lse0 = run(torch.full((H,), -float("inf"), device="cuda"))
    above = torch.tensor([10.0, 85.0, 300.0] * (H // 3), device="cuda")
    sink = lse0[0] + above      # of query row 0
    out, lse = run(sink)
    assert torch.isfinite(out).all() and torch.isfinite(lse).all()
    torch.testing.assert_close(lse[0], torch.logaddexp(lse0[0], sink), rtol=1e-5, atol=1e-3)
    weight = torch.sigmoid(lse0[0] - sink)[:, None]
    scale = out0[0].abs().amax(dim=1, keepdim=True) * weight
    assert ((out[0] - out0[0] * weight).abs() <= 1e-2 * scale + 1e-37).all()


def _in_list_order(case):
    """Cache rows that a query's list names, slot by slot."""
    idx, page = case["indices"], case["page_block_size"]
    return [case["block_table"][b][idx[b] // page] * page + idx[b] % page for b in range(idx.shape[0])]


def _check_groups(oracle, case, rel=4e-3):
    """As _check, but each group of 128 columns against its own largest output, so that a small group counts as much as a large one."""
    from gpu_util import run_gpu, run_oracle
    g_out, g_lse, _ = run_gpu(case, SCALE, num_sms=4)
    r_out, r_lse = run_oracle(oracle, case, SCALE)
    g, r = [_f32(x).reshape(x.shape[0], x.shape[1], 4, 128) for x in (g_out, r_out)]
    assert np.isfinite(g).all()
    assert (np.abs(g - r) <= rel * np.abs(r).max(axis=-1, keepdims=True) + 2.0 ** -8 * np.abs(r)).all()
    check_lse(g_lse, r_lse)


@pytest.mark.parametrize("amax", [1e-2, 1e-3, 1e-4, 1e-5, 1e-7])
def test_rows_of_zeros_from_the_cache_writer_beside_small_ones(built_lib, oracle, amax):
    """The cache writer gives a group of zeros the scale 1: it must not take precision from the other rows, whose scales are far smaller."""
    case = _case(10)
    latent = synth.stream(10, "kv").standard_normal(size=(case["kv"].shape[0], 512), dtype=np.float32) * np.float32(amax)
    for rows in _in_list_order(case):
        latent[rows[0]] = 0.0
        latent[rows[5], 128:256] = 0.0      # a row with one such group
    kv = synth.pack_fp8_rows(latent, np.ascontiguousarray(case["kv"][:, 528:]).view(np.uint16))
    _check_groups(oracle, dict(case, kv=kv))


@pytest.mark.parametrize("power", [-30, -60])
@pytest.mark.parametrize("where", ["first tile", "here and there", "with other groups of scale 0"])
def test_rows_of_zeros_whose_scale_is_far_above_all_others(built_lib, oracle, power, where):
    """Scales of 2^power, and rows of zeros of scale 1, which set no exponent that the others could not leave."""
    case = _case(19, topk=500, B=2)
    kv = case["kv"].copy()
    scales, q = kv[:, 512:528].copy().view(np.float32) * np.float32(2.0 ** power), _f32(case["q"]).copy()
    q[..., :512] *= np.float32(2.0 ** -power)
    for rows in _in_list_order(case):
        zeros = rows[:64] if where == "first tile" else rows[::9]
        kv[zeros, :512], scales[zeros] = 0, 1.0
        if where == "with other groups of scale 0":
            scales[zeros, 1:] = 0.0
    kv[:, 512:528] = scales.view(np.uint8).reshape(-1, 16)
    _check_groups(oracle, dict(case, kv=kv, q=_bf16(q)))


@pytest.mark.parametrize("power", [-12, -24, -36])
def test_one_group_far_smaller_than_the_others(built_lib, oracle, power):
    case = _case(11)
    kv = case["kv"].copy()
    kv[:, 512:528].view(np.float32)[:, 2] *= np.float32(2.0 ** power)
    _check_groups(oracle, dict(case, kv=kv))


@pytest.mark.parametrize("power", [-12, -20, -30, None])
def test_groups_small_by_turns(built_lib, oracle, power):
    """Some rows have one group far smaller (None: of scale 0) than their others, other rows another: neither takes bits from the large ones.
    (Against 64 bits the kernel is up to 2.0e-3 of a group's largest output off here, the oracle, which rounds P to 8 bits, 4.0e-3: together 6e-3.)"""
    case = _case(17)
    kv = case["kv"].copy()
    scales, factor = kv[:, 512:528].view(np.float32), np.float32(0.0 if power is None else 2.0 ** power)
    scales[::3, 0] *= factor
    scales[1::3, 1] *= factor
    _check_groups(oracle, dict(case, kv=kv), rel=6e-3)


@pytest.mark.parametrize("power", [-14, -22, -30, -38])
@pytest.mark.parametrize("mixed", [False, True])
def test_small_rows_that_carry_the_weight(built_lib, oracle, power, mixed):
    """The rows with next to no weight (2^-60 and less) have the large scales, those that make the result the small ones: at the start of the list, or in every tile."""
    case = _case(12, topk=512, B=2)
    kv, q = case["kv"].copy(), _f32(case["q"]).copy()
    rope = _f32(np.ascontiguousarray(kv[:, 528:]).view(np.uint16)).copy()
    q[..., 512] = 24.0
    rope[:, 0] = 0.0
    for rows in _in_list_order(case):
        few = rows[::7] if mixed else rows[:64]
        rope[few, 0] = -32.0        # 24 x -32 / sqrt(192) = -55 nats
        rest = np.setdiff1d(rows, few)
        kv[rest, 512:528] = (kv[rest, 512:528].copy().view(np.float32) * np.float32(2.0 ** power)).view(np.uint8)
    kv[:, 528:] = _bf16(rope).view(np.uint8).reshape(kv.shape[0], 128)
    _check_groups(oracle, dict(case, kv=kv, q=_bf16(q)))


@pytest.mark.parametrize("power", [8, 9, 11, 14, 20, 30])
@pytest.mark.parametrize("H,columns,num_sms", [(72, 1, 4), (72, 200, 148), (128, 3, 148), (40, 1, 148), (48, 200, 4)])
def test_elements_of_q_far_above_the_others(built_lib, oracle, power, H, columns, num_sms):
    """Columns of Q that are 2^power times the others and that the cache holds zeros in: what is left of the row decides, and has all its bits.  In some
    heads only, whole and split; lse to 2e-5: at most 16 elements lie below what the two parts hold, each rounded to 2^-22 of 2^9.5 (2^-12.5), which is
    2^-12.5 / sqrt(3) x 4 / sqrt(192) = 3e-5 of a score, and lse averages over more than four of them."""
    from gpu_util import run_gpu, run_oracle
    case = _case(13, H=H, topk=500 if num_sms == 148 else 321)
    q, kv = _f32(case["q"]).copy(), case["kv"].copy()
    heads = [0, 3, 31, 32, H - 1] + ([63, 64] if H > 64 else [])
    q[:, heads, 7:7 + columns] *= np.float32(2.0 ** power)
    kv[:, 7:7 + columns] = 0
    case = dict(case, kv=kv, q=_bf16(q))
    g_out, g_lse, plan = run_gpu(case, SCALE, num_sms=num_sms)
    assert (plan.info.num_partials > 0) == (num_sms == 148)
    r_out, r_lse = run_oracle(oracle, case, SCALE)
    check_out(g_out, r_out, **TOL_FP8)
    assert np.abs(g_lse - r_lse).max() < 2e-5
    again = run_gpu(case, SCALE, num_sms=num_sms)
    assert np.array_equal(again[0], g_out) and np.array_equal(again[1], g_lse)


def test_stacked_rows_with_elements_far_above_the_others(built_lib, oracle):
    """Both forms of the softmax warps in one list, stacked and single rows."""
    from gpu_util import run_gpu, run_oracle
    case = synth.make_decode_case(9, 24, 1024, 300, s_q=2, fp8=True, paged=True, seed=15)
    shared = [b % 2 == 0 for b in range(9)]
    q, kv, idx = _f32(case["q"]).copy(), case["kv"].copy(), case["indices"]
    for b in range(0, 9, 2):
        idx[2 * b + 1] = idx[2 * b]
    q[6:, ::5, 300] *= np.float32(2.0 ** 15)
    kv[:, 300] = 0
    case = dict(case, kv=kv, q=_bf16(q))
    g_out, g_lse, _ = run_gpu(case, SCALE, num_sms=4, mtp_shared=shared)
    r_out, r_lse = run_oracle(oracle, case, SCALE)
    check_out(g_out, r_out, **TOL_FP8)
    assert np.abs(g_lse - r_lse).max() < 2e-5


@pytest.mark.parametrize("B,H", [(2, 72), (2, 24), (74, 128)])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_a_row_without_positions_under_an_infinite_or_nan_sink(built_lib, B, H, value):
    """Zeros and +inf, whole or merged (the other kernels are in test_few_heads)."""
    import torch
    from gpu_util import to_dev
    case = synth.make_decode_case(B, H, 1024, 1000, fp8=True, paged=True, seed=B)
    case["indices"][0] = -1
    d = to_dev(case)
    plan = api.mla_decode_plan_create(B, H, 1000)
    assert (plan.info.num_partials > 0) == (B == 2)
    out, lse = api.mla_v4_launch_pipeline(d["q"], d["kv"], d["indices"], plan, SCALE, attn_sink=torch.full((H,), value, device="cuda"), block_table=d["block_table"],
                                          page_block_size=case["page_block_size"], kv_batch_stride_rows=case["kv_batch_stride_rows"])
    assert torch.all(out[0] == 0) and torch.all(lse[0] == float("inf"))


@pytest.mark.parametrize("B,H,num_sms", [(3, 72, 148), (3, 24, 148), (3, 16, 148), (3, 16, 2), (3, 72, 2)])
def test_infinite_sinks_on_a_bf16_cache(built_lib, B, H, num_sms):
    """An infinite sink takes all of a row's weight, whole or merged."""
    import torch
    from gpu_util import run_gpu, to_dev
    case = synth.make_decode_case(B, H, 1024, 900, seed=16)
    clean_out, clean_lse, plan = run_gpu(case, SCALE, num_sms=num_sms)
    assert (plan.info.num_partials > 0) == (num_sms == 148)
    d = to_dev(case)
    sink = torch.tensor([float("inf") if h % 2 else -float("inf") for h in range(H)], device="cuda")
    out, lse = api.mla_v4_launch_pipeline(d["q"], d["kv"], d["indices"], plan, SCALE, attn_sink=sink, kv_batch_stride_rows=1024)
    assert torch.all(out[:, 1::2] == 0) and torch.all(lse[:, 1::2] == float("inf"))
    np.testing.assert_array_equal(out[:, ::2].cpu().view(torch.int16).numpy().view(np.uint16), clean_out[:, ::2])


@pytest.mark.parametrize("B,H,num_sms", [(3, 72, 148), (3, 24, 148), (3, 16, 148), (3, 16, 2), (3, 72, 2)])
def test_nan_in_a_row_of_a_bf16_cache(built_lib, B, H, num_sms):
    """A NaN in a row of the cache reaches out and lse of its queries, whole or merged."""
    from gpu_util import run_gpu
    case = synth.make_decode_case(B, H, 1024, 900, seed=16)
    clean_out, clean_lse, plan = run_gpu(case, SCALE, num_sms=num_sms)
    assert (plan.info.num_partials > 0) == (num_sms == 148)
    kv = case["kv"].copy()
    kv[1024 + case["indices"][1, 800], 300] = 0x7FC0
    out, lse, _ = run_gpu(dict(case, kv=kv), SCALE, num_sms=num_sms)
    assert np.isnan(_f32(out)[1]).any(axis=-1).all() and np.isnan(lse[1]).all()
    np.testing.assert_array_equal(out[[0, 2]], clean_out[[0, 2]])
    np.testing.assert_array_equal(lse[[0, 2]], clean_lse[[0, 2]])


@pytest.mark.parametrize("H,topk,num_sms", [(72, 100, 2), (72, 700, 148), (24, 700, 148), (24, 100, 2), (16, 700, 148), (16, 700, 2), (16, 100, 2)])
@pytest.mark.parametrize("poison", ["code", "scale", "rope"])
def test_nan_in_a_row_reaches_out_and_lse_on_every_route(built_lib, H, topk, num_sms, poison):
    """The e4m3 NaN code, a NaN scale or a NaN in the rope of a row makes out and lse of the queries that select it NaN, whole or split, whatever the number of heads."""
    from gpu_util import run_gpu
    case = synth.make_decode_case(3, H, 1024, topk, fp8=True, paged=True, seed=14)
    kv, idx = case["kv"].copy(), case["indices"]
    clean_out, clean_lse, plan = run_gpu(case, SCALE, num_sms=num_sms)
    assert (plan.info.num_partials > 0) == (num_sms == 148)
    pos, page = int(idx[1, 70]), case["page_block_size"]
    row = int(case["block_table"][1][pos // page]) * page + pos % page
    if poison == "code":
        kv[row, 130] = 0xFF if H == 72 else 0x7F
    elif poison == "scale":
        kv[row, 516:520].view(np.float32)[0] = np.nan
    else:
        kv[row, 540:542].view(np.uint16)[0] = 0x7FC0
    out, lse, _ = run_gpu(dict(case, kv=kv), SCALE, num_sms=num_sms)
    assert np.isnan(_f32(out)[1]).any(axis=-1).all() and np.isnan(lse[1]).all()
    np.testing.assert_array_equal(out[[0, 2]], clean_out[[0, 2]])
    np.testing.assert_array_equal(lse[[0, 2]], clean_lse[[0, 2]])


@pytest.mark.parametrize("H,s_q,num_sms", [(17, 1, 2), (24, 1, 148), (32, 1, 6), (16, 2, 4), (8, 3, 148)])
def test_17_to_32_rows(built_lib, oracle, H, s_q, num_sms):
    """Heads or stacked rows that the few-heads kernel would take from a bf16 cache, at the edges of this kernel's tiles of 64 slots."""
    from gpu_util import run_gpu, run_oracle
    edges = [1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 191, 193, 257, 321, 1100]
    lens = np.repeat(np.array(edges + edges[::-1], np.int32), s_q)
    T = len(lens)
    case = synth.make_decode_case(T // s_q, H, 1216, 1100, s_q=s_q, fp8=True, paged=True, seed=H)
    for r, n in enumerate(lens):
        if r % s_q:
            case["indices"][r] = case["indices"][r - r % s_q]
        case["indices"][r, n:] = -1
    kw = dict(num_sms=num_sms, valid_len_hint=lens, mtp_shared=[True] * (T // s_q) if s_q > 1 else None)
    assert few_heads_form(api.plan_host(T, H, 1100, s_q, **kw)) == 0
    g_out, g_lse, plan = run_gpu(case, SCALE, **kw)
    assert s_q == 1 or any(w.stacked_rows == s_q for w in plan.read_works()[0])
    r_out, r_lse = run_oracle(oracle, case, SCALE)
    check_out(g_out, r_out, **TOL_FP8)
    check_lse(g_lse, r_lse)


@pytest.mark.parametrize("H,num_sms", [(72, 4), (24, 148)])
@pytest.mark.parametrize("power", [20, 27, 40])
def test_scores_beyond_the_resolution_of_their_reference(built_lib, H, num_sms, power):
    """Scores of 2^power and more: the largest one's row is the output (or a mean of rows whose scores fp32 does not tell apart), and out and lse are finite."""
    from gpu_util import run_gpu
    case = _case(18, H=H, topk=500)
    q = (_f32(case["q"]) * np.float32(2.0 ** power)).astype(np.float32)
    out, lse, _ = run_gpu(dict(case, q=_bf16(q)), SCALE, num_sms=num_sms)
    g, qd = _f32(out), _f32(_bf16(q)).astype(np.float64)
    assert np.isfinite(g).all() and np.isfinite(lse).all()
    from opfoundry_b200.synth import bf16_bits_to_f32
    import torch
    for b, rows in enumerate(_in_list_order(case)):
        kv = torch.from_numpy(case["kv"][rows])
        v = (kv[:, :512].view(torch.float8_e4m3fn).double() * kv[:, 512:528].contiguous().view(torch.float32).double().repeat_interleave(128, 1)).numpy()
        rope = bf16_bits_to_f32(np.ascontiguousarray(case["kv"][rows][:, 528:]).view(np.uint16))
        s = qd[b] @ np.concatenate([v, rope], axis=1).T * SCALE
        order = np.sort(s, axis=1)
        clear = order[:, -1] - order[:, -2] > 1e-6 * np.abs(qd[b]).max() * 576      # to the rounding of the sums
        assert clear.sum() > H // 2
        want = v[s.argmax(axis=1)]
        assert (np.abs(g[b] - want) <= 1e-2 * np.abs(want) + 1e-3)[clear].all()
        assert (np.abs(lse[b] - s.max(axis=1)) <= 1e-6 * np.abs(qd[b]).max() * 576)[clear].all()


@pytest.mark.parametrize("B,H,s_q", [(3, 24, 1), (80, 40, 1), (3, 72, 1), (74, 128, 1), (40, 32, 2)])
def test_residuals_with_peers_and_a_sink(built_lib, B, H, s_q):
    """Rows of Q with residuals, which wait in this GPU's rows of the gathered buffer: both peers' buffers hold the bits of the call without peers, nothing else is
    written; and the sink's weight is that of the call without one."""
    import ctypes as C
    import torch
    from gpu_util import to_dev
    topk, T = 700, B * s_q
    case = synth.make_decode_case(B, H, 1024, topk, s_q=s_q, fp8=True, paged=True, share_mtp="coin" if s_q > 1 else None, seed=B)
    q = _f32(case["q"]).copy()
    q[:, ::3, 9] *= np.float32(2.0 ** 16)
    kv = case["kv"].copy()
    kv[:, 9] = 0
    plan = api.mla_decode_plan_create(T, H, topk, s_q, mtp_shared=case["mtp_shared"] if s_q > 1 else None)
    d = to_dev(dict(case, q=_bf16(q), kv=kv))
    kw = dict(block_table=d["block_table"], page_block_size=64)
    want_out, want_lse = api.mla_decode_launch_pipeline(d["q"], d["kv"], d["indices"], plan, SCALE, **kw)
    outs = [torch.full((T, 3 * H, 512), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    lses = [torch.full((T, 3 * H), 7.0, device="cuda") for _ in range(2)]
    flags = torch.zeros(2, api.MAX_PEERS, dtype=torch.int32, device="cuda")
    flags[0, 1] = 1
    a = api.make_args(d["q"], d["kv"], d["indices"], plan, SCALE, out=outs[0][:, H:2 * H], lse=None, **kw)
    po = api.PeerOutputs()
    po.num_peers, po.my_rank, po.lse_stride_row, po.step = 2, 0, 3 * H, 1
    for r in range(2):
        po.out[r], po.lse[r], po.flags[r] = outs[r].data_ptr() + H * 1024, lses[r].data_ptr() + H * 4, flags[r].data_ptr()
    torch.cuda.synchronize()
    api._check(api.lib().dsa_v32_decode_pipeline_allgather(C.byref(a), C.byref(po), api._stream()), "dsa_v32_decode_pipeline_allgather")
    api._check(api.lib().dsa_v32_device_status(C.byref(a), api._stream()), "dsa_v32_device_status")
    for o, l in zip(outs, lses):
        assert torch.equal(o[:, H:2 * H].view(torch.int16), want_out.view(torch.int16)) and torch.equal(l[:, H:2 * H], want_lse)
        assert torch.all(o[:, :H] == 7) and torch.all(o[:, 2 * H:] == 7) and torch.all(l[:, :H] == 7) and torch.all(l[:, 2 * H:] == 7)
    sink = want_lse.mean(dim=0).contiguous()
    out, lse = api.mla_v4_launch_pipeline(d["q"], d["kv"], d["indices"], plan, SCALE, attn_sink=sink, **kw)
    torch.testing.assert_close(lse, torch.logaddexp(want_lse, sink[None]), rtol=1e-5, atol=1e-4)
    weight = torch.sigmoid(want_lse - sink[None])[..., None]
    ref = want_out.float() * weight
    assert ((out.float() - ref).abs() <= 2.0 ** -7 * ref.abs() + 1e-3 * ref.abs().amax(dim=-1, keepdim=True)).all()
