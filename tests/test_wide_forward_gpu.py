"""GPU: prefill of head dims above 128, where two threads share a query row, 64 keys of a block each: last blocks that end in, at
and behind the first thread's half, windows that leave one half without keys, rows that see nothing, more tiles than SMs.
Inputs are N(0, 1); tolerances are the rules of precision.py."""
import pytest
import torch

import parity_util as U
from flash_b200 import lib as L
from flash_b200 import ops
from oracle import api as OA

pytestmark = pytest.mark.gpu
BF, FP = torch.bfloat16, torch.float16


@pytest.mark.parametrize("dtype,d,b,s_q,s_k,h,hk,causal,window,softcap", [
    (BF, 256, 1, 128, 1, 2, 1, False, (-1, -1), 0.0), (FP, 256, 1, 129, 64, 2, 2, False, (-1, -1), 0.0),
    (BF, 192, 2, 130, 65, 4, 2, True, (-1, -1), 0.0),      # rows that see no key
    (BF, 256, 1, 300, 449, 2, 1, True, (-1, -1), 30.0), (FP, 136, 1, 257, 575, 4, 1, False, (20, 10), 0.0),
    (BF, 256, 1, 400, 400, 2, 1, True, (30, 0), 0.0), (BF, 256, 3, 640, 640, 16, 4, True, (-1, -1), 0.0)])
def test_two_threads_per_row(dtype, d, b, s_q, s_k, h, hk, causal, window, softcap):
    g = torch.Generator().manual_seed(d + s_q + s_k)
    q, k, v = U.normal((b, s_q, h, d), dtype, g), U.normal((b, s_k, hk, d), dtype, g), U.normal((b, s_k, hk, d), dtype, g)
    out, lse, pl = ops.attention_forward(q.cuda(), k.cuda(), v.cuda(), softmax_scale=d ** -0.5, causal=causal, window_left=window[0],
                                         window_right=window[1], softcap=softcap, return_plan=True)
    assert pl.kernel == L.KERNEL_TCGEN05 and pl.block_m == 128
    go, gl = OA.flash_attn_func(q, k, v, causal=causal, window_size=window, softcap=softcap)
    U.check_rules(out, lse, go, gl, tag=f"d {d} {s_q} x {s_k}")


@pytest.mark.parametrize("d", [64, 72, 128, 200, 256])
@pytest.mark.parametrize("where", ["rows", "base", "batch"])
def test_output_rows_off_the_sector_boundary(d, where):
    """Output rows that do not start on 32-byte boundaries (or are no whole sectors long) give the same bits, and what lies around
    them stays as it was."""
    g = torch.Generator().manual_seed(d)
    b, n, h = 2, 300, 3
    q, k, v = (U.normal((b, n, h, d), BF, g).cuda() for _ in range(3))
    want, _ = ops.attention_forward(q, k, v, softmax_scale=d ** -0.5, causal=True)
    pad = {"rows": 8, "base": 16, "batch": 16}[where]  # elements behind each row
    buf = torch.full((b * n * h * (d + pad) + 64,), 7.0, dtype=BF, device="cuda")
    first, per = (8, n * h * (d + pad)) if where == "base" else (0, n * h * (d + pad) + (8 if where == "batch" else 0))
    view = buf.as_strided((b, n, h, d), (per, h * (d + pad), d + pad, 1), first)
    out, _, pl = ops.attention_forward(q, k, v, softmax_scale=d ** -0.5, causal=True, out=view, return_plan=True)
    assert pl.kernel == L.KERNEL_TCGEN05 and torch.equal(out, want)
    view.fill_(7.0)
    assert bool((buf == 7.0).all())
