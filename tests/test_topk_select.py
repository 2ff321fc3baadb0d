"""The index-list producer (dsa_v32_topk_select) against a numpy selection on the same scores: exact sets,
ties at the threshold resolved toward the lower position, -1 padding, NaN never preferred; and its output
driving the attention (select -> gather -> attend) against the oracle."""
import math

import numpy as np
import pytest
import torch

from opfoundry_b200 import api, synth

pytestmark = pytest.mark.gpu


def numpy_select(scores, topk, valid_len):
    total_q, kv_len = scores.shape
    out = np.full((total_q, topk), -1, np.int32)
    for q in range(total_q):
        n = kv_len if valid_len is None else int(valid_len[q])
        s = scores[q, :n].astype(np.float64)
        s[np.isnan(s)] = -np.inf
        order = np.lexsort((np.arange(n), -s))          # by score descending, then position ascending
        k = min(topk, n)
        out[q, :k] = np.sort(order[:k])
    return out


@pytest.mark.parametrize("kv_len,topk", [(4096, 2048), (32768, 2048), (1000, 64), (517, 600), (70000, 512)])
def test_select_matches_numpy(built_lib, kv_len, topk):
    g = torch.Generator(device="cuda")
    g.manual_seed(kv_len + topk)
    total_q = 12
    scores = torch.randn(total_q, kv_len, generator=g, device="cuda")
    scores[1] = torch.round(scores[1] * 2) / 2                       # heavy ties
    scores[2] = 0.0                                                   # all equal
    scores[3, ::7] = float("nan")
    scores[4] = -scores[4].abs()                                      # all negative
    scores[5, :10] = float("inf")
    valid = torch.full((total_q,), kv_len, dtype=torch.int32, device="cuda")
    valid[6], valid[7], valid[8], valid[9] = 0, 1, min(topk, kv_len) - 1 if topk > 1 else 1, min(kv_len, topk + 1)
    got = api.topk_select(scores, topk, valid).cpu().numpy()
    want = numpy_select(scores.cpu().numpy(), topk, valid.cpu().numpy())
    assert np.array_equal(got, want)
    got2 = api.topk_select(scores, topk).cpu().numpy()
    assert np.array_equal(got2, numpy_select(scores.cpu().numpy(), topk, None))


def test_select_then_attend(built_lib, oracle):
    """Lists produced on the device feed the attention kernel directly; the oracle gets the same lists."""
    from gpu_util import to_dev
    from helpers import TOL_FP8, check_lse, check_out
    B, H, kv_len, topk = 4, 128, 2048, 512
    case = synth.make_decode_case(B, H, kv_len, topk, fp8=True, paged=True, seed=31)
    d = to_dev(case)
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    scores = torch.randn(B, kv_len, generator=g, device="cuda")
    valid = torch.tensor([kv_len, 300, kv_len, 1500], dtype=torch.int32, device="cuda")
    idx = api.topk_select(scores, topk, valid)
    plan = api.mla_decode_plan_create(B, H, topk, 1, valid_len_hint=[min(topk, int(v)) for v in valid.cpu()])
    scale = 1.0 / math.sqrt(192.0)
    out, lse = api.mla_decode_launch_pipeline(d["q"], d["kv"], idx, plan, scale, block_table=d["block_table"], page_block_size=64)
    torch.cuda.synchronize()
    r_out, r_lse = oracle.sparse_mla(case["q"], case["kv"], idx.cpu().numpy(), scale, kv_is_fp8=True,
                                     block_table=case["block_table"], page_block_size=64)
    check_out(out.view(torch.int16).cpu().numpy().view(np.uint16), r_out, **TOL_FP8)
    check_lse(lse.cpu().numpy(), r_lse)


@pytest.mark.parametrize("rows,kv_len,topk,stride", [
    (2, 4095, 7, 4095),          # one CTA per row, rows that are not 16-byte aligned
    (300, 8192, 2048, 8192),     # many rows: the small CTAs, a full register file
    (3, 8193, 2048, 8196),       # the first length above it
    (1, 131072, 2048, 131072),   # eight CTAs per row
    (300, 20001, 500, 20004),    # many long rows: the large CTAs
    (2, 300001, 2048, 300004),   # more than eight CTAs hold in registers: the slices are read again
])
def test_select_over_the_slices(built_lib, rows, kv_len, topk, stride):
    """Every way a row is cut over CTAs and registers, with values that fall into one bin of the first pass (more than
    the candidate list holds), ties over slice borders, and lengths that end inside a slice."""
    g = torch.Generator(device="cuda")
    g.manual_seed(kv_len)
    buf = torch.randn(rows, stride, generator=g, device="cuda")
    scores = buf[:, :kv_len]
    scores[0] = 1.0 + torch.randint(0, 1000, (kv_len,), generator=g, device="cuda") * 2.0 ** -20   # one 12-bit bin, heavy ties
    if rows > 1:
        scores[1] = torch.round(scores[1])
    valid = torch.randint(topk, kv_len + 1, (rows,), generator=g, device="cuda").to(torch.int32)
    valid[0] = kv_len
    got = api.topk_select(scores, topk, valid).cpu().numpy()
    check = sorted({0, 1 % rows, rows // 2, rows - 1})
    want = numpy_select(scores[check].cpu().numpy(), topk, valid[check].cpu().numpy())
    assert np.array_equal(got[check], want)


def test_time_follows_the_rows_own_length(built_lib):
    """Short rows in a buffer made for long ones (a serving batch) take a small multiple of their time in a narrow buffer (a
    CTA that makes, counts and tests keys for the whole width took 14 times as long), and give the same lists."""
    g = torch.Generator(device="cuda")
    g.manual_seed(11)
    wide = torch.randn(300, 131072, generator=g, device="cuda")
    narrow = wide[:, :3000].contiguous()
    valid = torch.randint(2100, 3001, (300,), generator=g, device="cuda").to(torch.int32)

    def best(scores):
        out = api.topk_select(scores, 2048, valid)
        times = []
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(20):
                api.topk_select(scores, 2048, valid, out=out)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times), out

    t_wide, o_wide = best(wide)
    t_narrow, o_narrow = best(narrow)
    assert torch.equal(o_wide, o_narrow)
    assert t_wide < 6 * t_narrow, (t_wide, t_narrow)


@pytest.mark.parametrize("rows,kv_len", [(64, 32768), (300, 20004), (40, 131072), (2, 300004)])
def test_lengths_at_the_edges_of_rounds_and_slices(built_lib, rows, kv_len):
    """Rows of one buffer that end around a round of a CTA's registers (2048 or 4096 positions), around what one CTA holds
    (8192 or 32768) and around a slice."""
    edges = [n + d for n in (2048, 4096, 6144, 8192, 12288, 16384, 32768, 32768 + 4096, 65536, 131072, kv_len) for d in (-3, -1, 0, 1, 2)]
    edges = [n for n in edges if 0 < n <= kv_len]
    topk = 300
    g = torch.Generator(device="cuda")
    g.manual_seed(kv_len)
    for i0 in range(0, len(edges), rows):
        lens = (edges[i0:i0 + rows] * rows)[:rows]
        scores = torch.round(torch.randn(rows, kv_len, generator=g, device="cuda") * 64) / 64
        valid = torch.tensor(lens, dtype=torch.int32, device="cuda")
        got = api.topk_select(scores, topk, valid).cpu().numpy()
        n = min(rows, len(edges) - i0)
        assert np.array_equal(got[:n], numpy_select(scores[:n].cpu().numpy(), topk, np.array(lens[:n])))
