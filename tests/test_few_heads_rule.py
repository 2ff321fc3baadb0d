"""Which kernel the items of a plan run on for either cache type (the last two words of the plan's header)."""
import numpy as np
import pytest

from opfoundry_b200 import api


@pytest.mark.parametrize("H,topk,fp8,bf16", [(16, 152, 0, 0), (16, 160, 16, 0), (16, 511, 16, 0), (16, 512, 16, 16), (1, 2048, 16, 16), (17, 767, 0, 0), (17, 768, 0, 32), (33, 2048, 0, 0)])
def test_whole_items(built_lib, H, topk, fp8, bf16):
    blob = api.plan_host(296, H, topk, num_sms=148)
    assert np.frombuffer(blob, np.int32, 2, 112).tolist() == [fp8, bf16]


@pytest.mark.parametrize("H,fp8,bf16", [(16, 16, 16), (24, 0, 32), (40, 0, 0)])
def test_pieces_of_split_items(built_lib, H, fp8, bf16):
    blob = api.plan_host(2, H, 2048, num_sms=148)
    assert np.frombuffer(blob, np.int32, 2, 112).tolist() == [fp8, bf16]
