"""CPU: calls with fake tensors never reach the native host path."""
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

import flash_attn_npu_v3 as fa3
from flash_b200 import lib as L


@pytest.mark.parametrize("inside", [True, False])
def test_planned_call_on_fake_tensors(inside):
    """A plan's bytes are not read while the call is only being traced for its shapes."""
    mode = FakeTensorMode()
    with mode:
        q = torch.empty((2, 1, 8, 128), dtype=torch.bfloat16, device="cuda")
        kc = torch.empty((2, 256, 2, 128), dtype=torch.bfloat16, device="cuda")
        lens = torch.empty((2,), dtype=torch.int32, device="cuda")
        meta = torch.empty((L.PLAN_BYTES,), dtype=torch.uint8, device="cuda")
    call = lambda: fa3.flash_attn_with_kvcache(q, kc, kc, cache_seqlens=lens, scheduler_metadata=meta, return_softmax_lse=True)
    if inside:
        with mode:
            out, lse, *_ = call()
    else:
        out, lse, *_ = call()
    assert out.shape == q.shape and out.dtype == q.dtype and lse.shape == (2, 8, 1)
