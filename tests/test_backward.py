"""Backward (dQ, dK, dV).

CPU: the oracle (oracle/bwd.py) reproduces the fixtures under tests/golden/bwd/, which hold outputs of the
reference's own backward golden (tests/fa_small_op_golden.py, generated by tests/golden/make_golden_bwd.py).
GPU: the CUDA backward through the drop-in autograd API against the oracle, with the tolerance of the
reference's backward tests (tests/test_flash_attn_npu_v2_bwd.py:31-32,42-46: rtol = atol = 1e-2) and the same input
distribution (2 * (rand - 0.5), seeded)."""
import glob
import itertools
import json
import os

import numpy as np
import pytest
import torch

from oracle import api as OA
from oracle import bwd as OB

HERE = os.path.dirname(os.path.abspath(__file__))
FIXTURES = sorted(glob.glob(os.path.join(HERE, "golden", "bwd", "*.npz")))
BF, FP = torch.bfloat16, torch.float16
RTOL = ATOL = 1e-2


def _load(path):
    z = np.load(path)
    meta = json.loads(str(z["meta"]))
    t = {}
    for key in z.files:
        if key == "meta":
            continue
        x = torch.from_numpy(np.ascontiguousarray(z[key]))
        t[key] = x.view(torch.bfloat16) if meta["dtypes"][key] == "bf16" else x
    return meta, t


@pytest.mark.parametrize("path", FIXTURES, ids=lambda p: os.path.basename(p)[:-4])
def test_oracle_reproduces_reference_backward_golden(path):
    meta, t = _load(path)
    kw = dict(softmax_scale=meta["scale"], causal=meta["causal"], window=tuple(meta["window"]),
              softcap=meta.get("softcap", 0.0))
    if meta["varlen"]:
        dq, dk, dv = OB.attention_varlen_backward(t["q"], t["k"], t["v"], t["dout"], t["lse"], t["cu_seqlens_q"],
                                                  t["cu_seqlens_k"], **kw)
    else:
        dq, dk, dv = OB.attention_backward(t["q"], t["k"], t["v"], t["dout"], t["lse"], **kw)
    for name, got in (("dq", dq), ("dk", dk), ("dv", dv)):
        # the same float64 arithmetic: at most one rounding of the 16-bit result apart
        torch.testing.assert_close(got.float(), t[name].float(), rtol=2 ** -7, atol=1e-4, msg=lambda m: f"{name}: {m}")


def test_fixtures_exist():
    assert len(FIXTURES) >= 5


def _rand(shape, dtype, g):
    return (2.0 * (torch.rand(shape, generator=g) - 0.5)).to(dtype)


def _check(name, got, want):
    torch.testing.assert_close(got.float().cpu(), want.float(), rtol=RTOL, atol=ATOL, msg=lambda m: f"{name}: {m}")


BSND_CASES = [
    # dtype, b, s_q, s_k, h, h_k, d, causal, window
    (BF, 2, 128, 128, 4, 4, 64, False, (-1, -1)),
    (BF, 2, 256, 256, 4, 2, 128, True, (-1, -1)),
    (FP, 1, 200, 333, 6, 2, 64, True, (-1, -1)),
    (FP, 2, 100, 100, 2, 1, 128, False, (-1, -1)),
    (BF, 1, 512, 512, 2, 2, 128, True, (-1, -1)),
    (BF, 1, 256, 256, 2, 2, 64, False, (64, 32)),
    (FP, 1, 300, 260, 4, 4, 128, True, (100, 0)),
    (BF, 1, 64, 64, 3, 3, 96, True, (-1, -1)),
    (FP, 1, 77, 190, 2, 2, 40, False, (-1, -1)),
    # head dims of the reference's varlen backward table (tests/test_flash_attn_npu_v2_bwd.py:233-236)
    (FP, 1, 333, 400, 5, 1, 192, False, (-1, -1)),
    (FP, 1, 500, 560, 5, 1, 256, True, (-1, -1)),
    (BF, 1, 311, 700, 5, 1, 111, True, (-1, -1)),
    (BF, 2, 130, 130, 2, 2, 256, False, (50, 20)),
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", BSND_CASES, ids=lambda c: "-".join(str(x).replace("torch.", "") for x in c))
def test_backward_dense(case):
    import flash_attn_npu_v2 as fa2
    dtype, b, s_q, s_k, h, h_k, d, causal, window = case
    g = torch.Generator().manual_seed(42)
    q, k, v = _rand((b, s_q, h, d), dtype, g), _rand((b, s_k, h_k, d), dtype, g), _rand((b, s_k, h_k, d), dtype, g)
    dout = _rand((b, s_q, h, d), dtype, g)
    scale = d ** -0.5
    qg, kg, vg = [t.cuda().requires_grad_(True) for t in (q, k, v)]
    out, lse, _ = fa2.flash_attn_func(qg, kg, vg, softmax_scale=scale, causal=causal, window_size=window,
                                      return_attn_probs=True)
    dq, dk, dv = torch.autograd.grad(out, (qg, kg, vg), dout.cuda())
    gq, gk, gv = OB.attention_backward(q, k, v, dout, lse.detach().cpu(), softmax_scale=scale, causal=causal, window=window)
    assert dq.shape == q.shape and dk.shape == k.shape and dv.shape == v.shape
    _check("dq", dq, gq)
    _check("dk", dk, gk)
    _check("dv", dv, gv)


@pytest.mark.gpu
@pytest.mark.parametrize("causal,window,d", [(True, (-1, -1), 64), (False, (-1, -1), 128), (True, (80, 0), 128)])
def test_backward_varlen_ragged(causal, window, d):
    import flash_attn_npu_v2 as fa2
    g = torch.Generator().manual_seed(7)
    lq, lk = [70, 0, 130, 1, 257], [100, 5, 130, 33, 300]
    cq = torch.tensor([0] + list(itertools.accumulate(lq)), dtype=torch.int32)
    ck = torch.tensor([0] + list(itertools.accumulate(lk)), dtype=torch.int32)
    h, h_k = 4, 2
    q, k, v = _rand((sum(lq), h, d), BF, g), _rand((sum(lk), h_k, d), BF, g), _rand((sum(lk), h_k, d), BF, g)
    dout = _rand((sum(lq), h, d), BF, g)
    scale = d ** -0.5
    qg, kg, vg = [t.cuda().requires_grad_(True) for t in (q, k, v)]
    out, lse, _ = fa2.flash_attn_varlen_func(qg, kg, vg, cq.cuda(), ck.cuda(), max(lq), max(lk), softmax_scale=scale,
                                             causal=causal, window_size=window, return_attn_probs=True)
    dq, dk, dv = torch.autograd.grad(out, (qg, kg, vg), dout.cuda())
    gq, gk, gv = OB.attention_varlen_backward(q, k, v, dout, lse.detach().cpu(), cq, ck, softmax_scale=scale,
                                              causal=causal, window=window)
    _check("dq", dq, gq)
    _check("dk", dk, gk)
    _check("dv", dv, gv)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,causal,window", [(FP, True, (-1, -1)), (BF, False, (-1, -1)), (BF, True, (128, 64))])
def test_backward_softcap(dtype, causal, window):
    """softcap = 30 like the reference's backward tables (tests/test_flash_attn_npu_v2_bwd.py:156-159,196-199)."""
    import flash_attn_npu_v2 as fa2
    g = torch.Generator().manual_seed(5)
    b, s, h, h_k, d = 2, 320, 4, 2, 128
    q, k, v, dout = _rand((b, s, h, d), dtype, g), _rand((b, s, h_k, d), dtype, g), _rand((b, s, h_k, d), dtype, g), _rand((b, s, h, d), dtype, g)
    scale = d ** -0.5
    qg, kg, vg = [t.cuda().requires_grad_(True) for t in (q, k, v)]
    out, lse, _ = fa2.flash_attn_func(qg, kg, vg, softmax_scale=scale, causal=causal, window_size=window, softcap=30.0,
                                      return_attn_probs=True)
    dq, dk, dv = torch.autograd.grad(out, (qg, kg, vg), dout.cuda())
    gq, gk, gv = OB.attention_backward(q, k, v, dout, lse.detach().cpu(), softmax_scale=scale, causal=causal, window=window,
                                       softcap=30.0)
    _check("dq", dq, gq)
    _check("dk", dk, gk)
    _check("dv", dv, gv)


@pytest.mark.gpu
def test_backward_through_packed_api_and_module_bwd():
    """kv-packed wrapper is differentiable; the extension-level ``bwd`` has the reference's positional signature."""
    import flash_attn_npu_arch22_v2 as ext
    import flash_attn_npu_v2 as fa2
    g = torch.Generator().manual_seed(3)
    b, s, h, d = 1, 192, 2, 64
    q, kv, dout = _rand((b, s, h, d), FP, g), _rand((b, s, 2, h, d), FP, g), _rand((b, s, h, d), FP, g)
    qg, kvg = q.cuda().requires_grad_(True), kv.cuda().requires_grad_(True)
    out = fa2.flash_attn_kvpacked_func(qg, kvg, causal=True)
    dq, dkv = torch.autograd.grad(out, (qg, kvg), dout.cuda())
    out2, lse2, _, _ = ext.fwd(q.cuda(), kv[:, :, 0].cuda().contiguous(), kv[:, :, 1].cuda().contiguous(), None, None, 0.0,
                               d ** -0.5, True, -1, -1, 0.0, False, None)
    dq2, dk2, dv2, _ = ext.bwd(dout.cuda(), q.cuda(), kv[:, :, 0].cuda().contiguous(), kv[:, :, 1].cuda().contiguous(), out2,
                               lse2, None, None, None, None, 0.0, d ** -0.5, True, -1, -1, 0.0, False, None, None)
    assert torch.equal(dq, dq2) and torch.equal(dkv[:, :, 0], dk2) and torch.equal(dkv[:, :, 1], dv2)
    with pytest.raises(RuntimeError):  # dropout stays refused, as in the forward
        ext.bwd(dout.cuda(), q.cuda(), q.cuda(), q.cuda(), out2, lse2, None, None, None, None, 0.1, 1.0, True, -1, -1, 0.0,
                False, None, None)


@pytest.mark.gpu
def test_backward_v3_api_dense_and_varlen():
    """The FA3-style package is differentiable through the same kernels."""
    import flash_attn_npu_v3 as fa3
    g = torch.Generator().manual_seed(11)
    b, s, h, h_k, d = 2, 160, 4, 2, 128
    q, k, v, dout = _rand((b, s, h, d), BF, g), _rand((b, s, h_k, d), BF, g), _rand((b, s, h_k, d), BF, g), _rand((b, s, h, d), BF, g)
    qg, kg, vg = [t.cuda().requires_grad_(True) for t in (q, k, v)]
    out, lse = fa3.flash_attn_func(qg, kg, vg, causal=True, return_attn_probs=True)
    dq, dk, dv = torch.autograd.grad(out, (qg, kg, vg), dout.cuda())
    gq, gk, gv = OB.attention_backward(q, k, v, dout, lse.detach().cpu(), softmax_scale=d ** -0.5, causal=True)
    _check("dq", dq, gq); _check("dk", dk, gk); _check("dv", dv, gv)
    lq = [100, 60, 160]
    cq = torch.tensor([0] + list(itertools.accumulate(lq)), dtype=torch.int32)
    qv_, kv_, vv_, dv_ = [t.reshape(b * s, -1, d)[:sum(lq)].contiguous() for t in (q, k, v, dout)]
    qg, kg, vg = [t.cuda().requires_grad_(True) for t in (qv_, kv_, vv_)]
    out, lse = fa3.flash_attn_varlen_func(qg, kg, vg, cq.cuda(), cq.cuda(), max(lq), max(lq), causal=True,
                                          return_attn_probs=True)
    dq, dk, dv = torch.autograd.grad(out, (qg, kg, vg), dv_.cuda())
    gq, gk, gv = OB.attention_varlen_backward(qv_, kv_, vv_, dv_, lse.detach().cpu(), cq, cq, softmax_scale=d ** -0.5, causal=True)
    _check("dq", dq, gq); _check("dk", dk, gk); _check("dv", dv, gv)


# ---------------------------------------------------------------------------------------------------------------
# The tcgen05 kernels (head dim 128, no softcap) forced through the operator-level call, against the oracle.
# ---------------------------------------------------------------------------------------------------------------
TC5_CASES = [
    # dtype, b, s_q, s_k, h, h_k, causal, window [, head dim (128)]
    (BF, 1, 128, 128, 1, 1, False, (-1, -1)),      # one block of each
    (BF, 2, 640, 640, 4, 1, True, (-1, -1)),       # group of 4 query heads per kv head
    (FP, 1, 130, 1000, 2, 2, True, (-1, -1)),      # few query rows at the end of a long key range
    (BF, 1, 900, 200, 2, 1, True, (-1, -1)),       # more query rows than keys: the first 700 rows see nothing
    (BF, 1, 515, 515, 2, 2, False, (200, 100)),    # two-sided window, ragged last blocks
    (BF, 2, 400, 400, 4, 2, True, (-1, -1), 64),   # the 64-column tiles
    (FP, 1, 300, 333, 2, 2, False, (-1, -1), 64),
    (BF, 1, 333, 400, 3, 1, True, (-1, -1), 96),   # between the two tile widths: zero columns beyond the head dim
    (FP, 1, 200, 260, 2, 2, True, (100, 0), 40),
    (BF, 1, 260, 260, 2, 1, False, (-1, -1), 112),
    (FP, 2, 384, 384, 2, 2, False, (380, 63)),     # a left side that hardly binds (a negative literal means different
                                                    # things to the reference's forward and backward goldens: not exercised)
    (BF, 1, 1536, 1536, 2, 2, True, (300, 0)),     # sliding window: key blocks most query blocks never see
    (BF, 1, 64, 64, 2, 2, True, (-1, -1)),         # less than a block
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", TC5_CASES, ids=lambda c: "-".join(str(x).replace("torch.", "") for x in c))
def test_tcgen05_backward_dense(case):
    from flash_b200 import lib as L
    from flash_b200 import ops
    dtype, b, s_q, s_k, h, h_k, causal, window = case[:8]
    d = case[8] if len(case) > 8 else 128
    g = torch.Generator().manual_seed(1234)
    q, k, v = _rand((b, s_q, h, d), dtype, g), _rand((b, s_k, h_k, d), dtype, g), _rand((b, s_k, h_k, d), dtype, g)
    dout = _rand((b, s_q, h, d), dtype, g)
    kw = dict(softmax_scale=d ** -0.5, causal=causal, window_left=window[0], window_right=window[1])
    out, lse = ops.attention_forward(q.cuda(), k.cuda(), v.cuda(), **kw)
    dq, dk, dv = ops.attention_backward(dout.cuda(), q.cuda(), k.cuda(), v.cuda(), out, lse, kernel=2, **kw)
    torch.cuda.synchronize()
    assert L.load().fa_b200_check_status(torch.cuda.current_stream().cuda_stream) == 0
    gq, gk, gv = OB.attention_backward(q, k, v, dout, lse.cpu(), softmax_scale=d ** -0.5, causal=causal, window=window)
    _check("dq", dq, gq)
    _check("dk", dk, gk)
    _check("dv", dv, gv)
    # no atomics anywhere: a second run gives the same bits, and the automatic choice is this pair of kernels
    again = ops.attention_backward(dout.cuda(), q.cuda(), k.cuda(), v.cuda(), out, lse, kernel=2, **kw)
    auto = ops.attention_backward(dout.cuda(), q.cuda(), k.cuda(), v.cuda(), out, lse, **kw)
    for a, c, e in zip((dq, dk, dv), again, auto):
        assert torch.equal(a, c) and torch.equal(a, e)
    # the mma.sync kernel computes the same thing (dQ through fp32 atomics: equal up to summation order)
    other = ops.attention_backward(dout.cuda(), q.cuda(), k.cuda(), v.cuda(), out, lse, kernel=1, **kw)
    for name, a, c in zip(("dq", "dk", "dv"), (dq, dk, dv), other):
        torch.testing.assert_close(a.float(), c.float(), rtol=RTOL, atol=ATOL, msg=lambda m: f"{name} between the kernels: {m}")


@pytest.mark.gpu
@pytest.mark.parametrize("causal,window", [(True, (-1, -1)), (False, (-1, -1)), (False, (150, 40))])
def test_tcgen05_backward_packed_sequences(causal, window):
    """Packed input whose sequences include an empty one, one shorter than a block on either side, one with more query
    rows than keys and one far longer than the others (so that most key blocks of the grid do not exist for most
    sequences)."""
    from flash_b200 import lib as L
    from flash_b200 import ops
    g = torch.Generator().manual_seed(77)
    d, h, h_k = 128, 4, 2
    lq, lk = [70, 0, 130, 1, 400, 257, 1100], [100, 5, 130, 33, 90, 300, 1250]
    cq = torch.tensor([0] + list(itertools.accumulate(lq)), dtype=torch.int32)
    ck = torch.tensor([0] + list(itertools.accumulate(lk)), dtype=torch.int32)
    q, k, v = _rand((sum(lq), h, d), BF, g), _rand((sum(lk), h_k, d), BF, g), _rand((sum(lk), h_k, d), BF, g)
    dout = _rand((sum(lq), h, d), BF, g)
    kw = dict(softmax_scale=d ** -0.5, causal=causal, window_left=window[0], window_right=window[1], cu_seqlens_q=cq.cuda(),
              cu_seqlens_k=ck.cuda(), max_seqlen_q=max(lq), max_seqlen_k=max(lk))
    out, lse = ops.attention_forward(q.cuda(), k.cuda(), v.cuda(), **kw)
    dq = torch.full_like(q, float("nan")).cuda()  # every element must be written, zeros included
    dk, dv = torch.full_like(k, float("nan")).cuda(), torch.full_like(v, float("nan")).cuda()
    ops.attention_backward(dout.cuda(), q.cuda(), k.cuda(), v.cuda(), out, lse, dq=dq, dk=dk, dv=dv, kernel=2, **kw)
    torch.cuda.synchronize()
    assert L.load().fa_b200_check_status(torch.cuda.current_stream().cuda_stream) == 0
    gq, gk, gv = OB.attention_varlen_backward(q, k, v, dout, lse.cpu(), cq, ck, softmax_scale=d ** -0.5, causal=causal,
                                              window=window)
    _check("dq", dq, gq)
    _check("dk", dk, gk)
    _check("dv", dv, gv)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,causal,window", [(FP, True, (-1, -1)), (BF, False, (-1, -1)), (BF, True, (128, 64))])
def test_tcgen05_backward_softcap(dtype, causal, window):
    """softcap = 30 like the reference's backward tables (tests/test_flash_attn_npu_v2_bwd.py:156-159,196-199), on the
    tcgen05 forward and backward kernels."""
    from flash_b200 import lib as L
    from flash_b200 import ops
    g = torch.Generator().manual_seed(5)
    b, s, h, h_k, d = 2, 320, 4, 2, 128
    q, k, v, dout = _rand((b, s, h, d), dtype, g), _rand((b, s, h_k, d), dtype, g), _rand((b, s, h_k, d), dtype, g), _rand((b, s, h, d), dtype, g)
    kw = dict(softmax_scale=d ** -0.5, causal=causal, window_left=window[0], window_right=window[1], softcap=30.0)
    out, lse, plan = ops.attention_forward(q.cuda(), k.cuda(), v.cuda(), return_plan=True, **kw)
    assert plan.kernel == L.KERNEL_TCGEN05
    go, gl = OA.flash_attn_func(q, k, v, softmax_scale=d ** -0.5, causal=causal, window_size=window, softcap=30.0)
    _check("out", out, go)
    _check("lse", lse, gl)
    dq, dk, dv = ops.attention_backward(dout.cuda(), q.cuda(), k.cuda(), v.cuda(), out, lse, kernel=2, **kw)
    torch.cuda.synchronize()
    assert L.load().fa_b200_check_status(torch.cuda.current_stream().cuda_stream) == 0
    gq, gk, gv = OB.attention_backward(q, k, v, dout, lse.cpu(), softmax_scale=d ** -0.5, causal=causal, window=window, softcap=30.0)
    _check("dq", dq, gq)
    _check("dk", dk, gk)
    _check("dv", dv, gv)


@pytest.mark.gpu
def test_tcgen05_backward_refuses_what_it_does_not_cover():
    from flash_b200 import ops
    g = torch.Generator().manual_seed(5)
    d = 192
    q, k, v, dout = [_rand((1, 128, 2, d), BF, g).cuda() for _ in range(4)]
    out, lse = ops.attention_forward(q, k, v, softmax_scale=d ** -0.5)
    with pytest.raises(RuntimeError, match="tcgen05 backward covers"):
        ops.attention_backward(dout, q, k, v, out, lse, softmax_scale=d ** -0.5, kernel=2)
    ops.attention_backward(dout, q, k, v, out, lse, softmax_scale=d ** -0.5)  # the other kernel takes it
    with pytest.raises(RuntimeError, match="kernel must be"):
        ops.attention_backward(dout, q, k, v, out, lse, softmax_scale=d ** -0.5, kernel=7)


@pytest.mark.gpu
@pytest.mark.parametrize("d", [64, 72, 128, 192, 256])
@pytest.mark.parametrize("where", ["rows", "base"])
def test_gradient_rows_off_the_sector_boundary(d, where):
    """Gradient rows that do not start on 32-byte boundaries (or are no whole sectors long) get the same bits, and what lies around
    them stays as it was."""
    from flash_b200 import ops
    g = torch.Generator().manual_seed(d)
    b, n, h = 2, 200, 2
    q, k, v, dout = (torch.randn(b, n, h, d, generator=g).to(torch.bfloat16).cuda() for _ in range(4))
    kw = dict(softmax_scale=d ** -0.5, causal=True)
    out, lse = ops.attention_forward(q, k, v, **kw)
    want = ops.attention_backward(dout, q, k, v, out, lse, **kw)
    pad, first = (8, 0) if where == "rows" else (16, 8)
    bufs = [torch.full((b * n * h * (d + pad) + 64,), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(3)]
    views = [x.as_strided((b, n, h, d), (n * h * (d + pad), h * (d + pad), d + pad, 1), first) for x in bufs]
    ops.attention_backward(dout, q, k, v, out, lse, dq=views[0], dk=views[1], dv=views[2], **kw)
    for buf, view, x in zip(bufs, views, want):
        assert torch.equal(view, x)
        view.fill_(7.0)
        assert bool((buf == 7.0).all())


@pytest.mark.gpu
@pytest.mark.parametrize("d,s,s_k,h,h_k,causal", [
    (64, 130, 130, 1, 1, True), (64, 700, 700, 30, 30, True), (128, 128, 128, 2, 2, True), (128, 1100, 1100, 20, 20, True),
    (64, 4096, 128, 32, 1, False), (128, 4096, 128, 32, 1, False)])
def test_what_follows_the_backward_follows_both_kernels(d, s, s_k, h, h_k, causal):
    """The dQ kernel starts beside the dK / dV kernel: fewer work items than SMs, and more; and one dK / dV item of 2048 units, which
    is at work long after the other SMs are through with all of dQ (head dim 64: 1150 us, and 19 for a dQ kernel by itself, which starts
    some 10 us later).  Inputs are overwritten right behind the call, in stream order; the same through a captured graph."""
    from flash_b200 import ops
    g = torch.Generator().manual_seed(s)
    q, k, v, dout = (torch.randn(1, n, heads, d, generator=g).to(torch.bfloat16).cuda() for n, heads in ((s, h), (s_k, h_k), (s_k, h_k), (s, h)))
    kw = dict(softmax_scale=d ** -0.5, causal=causal)
    out, lse = ops.attention_forward(q, k, v, **kw)
    want = ops.attention_backward(dout, q, k, v, out, lse, **kw)
    torch.cuda.synchronize()
    for _ in range(20):
        x = [t.clone() for t in (dout, q, k, v)]
        got = ops.attention_backward(*x, out, lse, **kw)
        for t in x:
            t.fill_(float("nan"))
        for a, b in zip(got, want):
            assert torch.equal(a, b)
    x = [t.clone() for t in (dout, q, k, v)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = ops.attention_backward(*x, out, lse, **kw)
        for t in x:
            t.fill_(float("nan"))
    for _ in range(3):
        for t, src in zip(x, (dout, q, k, v)):
            t.copy_(src)
        graph.replay()
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("over", ["q", "dout", "columns of q", "packed q"])
def test_dq_over_an_input(d, over):
    """dQ may be written over q or dout, or over some of their columns: the dQ kernel reads its own rows before it writes them, and does
    not start beside a dK / dV kernel that still reads them (one item of 2048 units, see above).  The same bits as apart."""
    from flash_b200 import ops
    g = torch.Generator().manual_seed(d)
    s, s_k, h = 4096, 128, 32
    wide = torch.randn(1, s, h, d + 16, generator=g).to(torch.bfloat16).cuda()
    q, k, v, dout = (torch.randn(1, n, heads, d, generator=g).to(torch.bfloat16).cuda() for n, heads in ((s, h), (s_k, 1), (s_k, 1), (s, h)))
    kw = dict(softmax_scale=d ** -0.5, causal=False)
    if over == "columns of q":
        q = wide[..., :d]
    if over == "packed q":
        q, k, v, dout = (t[0] for t in (q, k, v, dout))
        cu = [torch.tensor([0, 1000, n], dtype=torch.int32).cuda() for n in (s, s_k)]
        cu[1][1] = 1
        kw.update(cu_seqlens_q=cu[0], cu_seqlens_k=cu[1], max_seqlen_q=s - 1000, max_seqlen_k=s_k - 1)
    out, lse = ops.attention_forward(q, k, v, **kw)
    want = ops.attention_backward(dout, q, k, v, out, lse, **kw)
    dq = {"q": q, "dout": dout, "columns of q": wide[..., 16:], "packed q": q}[over]
    got = ops.attention_backward(dout, q, k, v, out, lse, dq=dq, **kw)
    for a, b in zip(got, want):
        assert torch.equal(a, b)
