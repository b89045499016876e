"""GPU: the edges of the ranges that the planner's kernel choices cover, against the oracle: tile remainders, head dims
between the tile widths, the smallest and largest row counts, single sequences cut over the whole grid.  Inputs are
N(0, 1); tolerances are the rules of precision.py (rtol = atol = 1e-2 for 16-bit outputs, and the 99.5 % rule)."""
import pytest
import torch

import parity_util as U
from flash_b200 import lib as L
from flash_b200 import ops
from oracle import api as OA

pytestmark = pytest.mark.gpu
BF, FP = torch.bfloat16, torch.float16


def _cuda(t):
    return None if t is None else t.cuda()


def _cache(g, dtype, b, room, hk, d, page):
    """(k, v, block table or None): contiguous rows, or pages of a shuffled pool."""
    if not page:
        return U.normal((b, room, hk, d), dtype, g), U.normal((b, room, hk, d), dtype, g), None
    per = -(-room // page)
    bt = torch.randperm(b * per, generator=g).view(b, per).to(torch.int32)
    return U.normal((b * per, page, hk, d), dtype, g), U.normal((b * per, page, hk, d), dtype, g), bt


@pytest.mark.parametrize("page", [0, 128])
@pytest.mark.parametrize("dtype,d,window", [(BF, 128, -1), (FP, 64, -1), (BF, 192, 100)])
def test_packed_queries_against_a_cache_on_tcgen05(dtype, d, window, page):
    import flash_attn_npu_v3 as fa3
    g = torch.Generator().manual_seed(d + page)
    h, hk = 4, 2
    q_lens, k_lens = [1, 127, 128, 129, 257], [1, 500, 128, 640, 300]
    b, room = len(q_lens), 640
    cq = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32)
    q = U.normal((sum(q_lens), h, d), dtype, g)
    kc, vc, bt = _cache(g, dtype, b, room, hk, d, page)
    lens = torch.tensor(k_lens, dtype=torch.int32)
    out, lse, *_ = fa3.flash_attn_with_kvcache(q.cuda(), kc.cuda(), vc.cuda(), cache_seqlens=lens.cuda(), page_table=_cuda(bt),
                                               cu_seqlens_q=cq.cuda(), max_seqlen_q=max(q_lens), causal=True,
                                               window_size=(window, -1), return_softmax_lse=True)
    for i in range(b):
        rows = slice(int(cq[i]), int(cq[i + 1]))
        ki, vi, bi = (kc, vc, bt[i:i + 1]) if page else (kc[i:i + 1], vc[i:i + 1], None)
        # a left window counts from the call's longest sequence; none of these windows covers it
        go, gl = OA.flash_attn_with_kvcache(q[rows].unsqueeze(0), ki, vi, cache_seqlens=lens[i:i + 1], block_table=bi, causal=True,
                                            window_size=(window if window < k_lens[i] - 1 else -1, -1))
        U.check_rules(out[rows].unsqueeze(0), lse[:, rows].unsqueeze(0), go, gl, tag=f"sequence {i}")


@pytest.mark.parametrize("softcap", [0.0, 30.0])
@pytest.mark.parametrize("kind", ["dense", "packed", "chunk", "decode"])
def test_negative_softmax_scale(kind, softcap):
    g = torch.Generator().manual_seed(3)
    n, h, hk, d, scale = 1 if kind == "decode" else 300, 4, 2, 128, -0.5
    m = 600 if kind in ("chunk", "decode") else n
    q, k, v = U.normal((n, h, d), BF, g), U.normal((m, hk, d), BF, g), U.normal((m, hk, d), BF, g)
    cq, ck, lens = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in ([0, n], [0, m], [m]))
    kw = dict(softmax_scale=scale, causal=True, softcap=softcap)
    if kind == "dense":
        out, lse = ops.attention_forward(q[None].cuda(), k[None].cuda(), v[None].cuda(), **kw)
    elif kind == "packed":
        out, lse = ops.attention_forward(q.cuda(), k.cuda(), v.cuda(), cu_seqlens_q=cq, cu_seqlens_k=ck, max_seqlen_q=n, max_seqlen_k=m, **kw)
    elif kind == "chunk":
        out, lse = ops.attention_forward(q.cuda(), k[None].cuda(), v[None].cuda(), cu_seqlens_q=cq, max_seqlen_q=n, seqused_k=lens, **kw)
    else:
        out, lse = ops.attention_forward(q[None].cuda(), k[None].cuda(), v[None].cuda(), seqused_k=lens, **kw)
    kk, vv = (t.double().repeat_interleave(h // hk, 1).transpose(0, 1) for t in (k, v))
    x = q.double().transpose(0, 1) @ kk.transpose(1, 2) * scale
    if softcap:
        x = softcap * torch.tanh(x / softcap)
    x = x.masked_fill(torch.ones(n, m, dtype=torch.bool).triu(1 + m - n), float("-inf"))
    torch.testing.assert_close(out.cpu().double().view(n, h, d), (torch.softmax(x, 2) @ vv).transpose(0, 1), rtol=1e-2, atol=1e-2)
    torch.testing.assert_close(lse.cpu().double().view(h, n), torch.logsumexp(x, 2), rtol=1e-2, atol=1e-2)


@pytest.mark.parametrize("dtype,d", [(FP, 64), (FP, 128), (BF, 256)])
def test_softcap_of_packed_queries_against_a_cache(dtype, d):
    """Capped scores as exact as on the kernels that served these calls before (1 - 2 / (e^2y + 1): a few units of 2^-24
    of the cap, times log2 e).  Scores reach the cap here; the LSE shows their error without the rounding of P.  Sums of
    fp32 products: sqrt(d) * 2^-24 of the largest partial sums (about 100), 1e-4 in all; tanh.approx gives 3e-4 and more."""
    g = torch.Generator().manual_seed(d)
    n, h, hk, cap = 700, 4, 2, 50.0
    q, k, v = U.normal((n, h, d), dtype, g) * 6, U.normal((1, n, hk, d), dtype, g), U.normal((1, n, hk, d), dtype, g)
    cq, lens = torch.tensor([0, n], dtype=torch.int32), torch.tensor([n], dtype=torch.int32)
    out, lse, pl = ops.attention_forward(q.cuda(), k.cuda(), v.cuda(), cu_seqlens_q=cq.cuda(), max_seqlen_q=n, seqused_k=lens.cuda(),
                                         softmax_scale=d ** -0.5, causal=True, softcap=cap, return_plan=True)
    assert pl.kernel == L.KERNEL_TCGEN05
    kk, vv = (t[0].double().repeat_interleave(h // hk, 1).transpose(0, 1) for t in (k, v))
    x = cap * torch.tanh(q.double().transpose(0, 1) @ kk.transpose(1, 2) * d ** -0.5 / cap)
    x = x.masked_fill(torch.ones(n, n, dtype=torch.bool).triu(1), float("-inf"))
    want = torch.logsumexp(x, 2)
    assert float((lse.cpu().double() - want).abs().max()) < 1e-4
    torch.testing.assert_close(out.cpu().double(), (torch.softmax(x, 2) @ vv).transpose(0, 1), rtol=1e-2, atol=1e-2)


@pytest.mark.parametrize("d,h,hk,rows,keys,kernel", [
    (64, 4, 2, 1279, 4096, L.KERNEL_MMA), (64, 4, 2, 1280, 4096, L.KERNEL_TCGEN05), (128, 8, 1, 383, 8192, L.KERNEL_MMA),
    (128, 8, 1, 384, 8192, L.KERNEL_TCGEN05), (96, 8, 8, 287, 2048, L.KERNEL_MMA), (96, 8, 8, 287, 1920, L.KERNEL_TCGEN05),
    (256, 4, 1, 255, 4096, L.KERNEL_MMA), (256, 4, 1, 256, 4096, L.KERNEL_TCGEN05)])
def test_few_packed_rows_against_many_keys(d, h, hk, rows, keys, kernel):
    """Both sides of the line where a chunk is too small to fill the chip with tiles."""
    g = torch.Generator().manual_seed(rows)
    q, (kc, vc, bt) = U.normal((rows, h, d), BF, g), _cache(g, BF, 1, keys, hk, d, 128)
    lens = torch.tensor([keys - 5], dtype=torch.int32)
    cq = torch.tensor([0, rows], dtype=torch.int32)
    out, lse, pl = ops.attention_forward(q.cuda(), kc.cuda(), vc.cuda(), seqused_k=lens.cuda(), block_table=bt.cuda(), cu_seqlens_q=cq.cuda(),
                                         max_seqlen_q=rows, softmax_scale=d ** -0.5, causal=True, return_plan=True)
    assert pl.kernel == kernel and (kernel == L.KERNEL_TCGEN05 or pl.num_splits > 1)
    go, gl = OA.flash_attn_with_kvcache(q.unsqueeze(0), kc, vc, cache_seqlens=lens, block_table=bt, causal=True)
    U.check_rules(out.unsqueeze(0), lse.unsqueeze(0), go, gl, tag=f"d {d} rows {rows} keys {keys}")


@pytest.mark.parametrize("page", [0, 128])
@pytest.mark.parametrize("rows", [1, 16, 17, 32])
@pytest.mark.parametrize("d", [64, 72, 96, 128, 136, 192, 256])
def test_decode_kernel_every_head_dim(d, rows, page):
    """1 to 32 packed rows per kv head; new tokens appended with rotary; lengths around the key blocks' edges."""
    import flash_attn_npu_v2 as fa2
    g = torch.Generator().manual_seed(d * 100 + rows)
    dtype = BF if rows % 2 else FP
    hk, group, s_q = 2, {1: 1, 16: 8, 17: 17, 32: 8}[rows], {1: 1, 16: 2, 17: 1, 32: 4}[rows]
    new, room = s_q, 520
    lens = torch.tensor([0, 1, 127, 128, 300, room - new], dtype=torch.int32)
    b = lens.numel()
    rotary = d // 16 * 16
    q = U.normal((b, s_q, hk * group, d), dtype, g)
    kc, vc, bt = _cache(g, dtype, b, room, hk, d, page)
    k, v = U.normal((b, new, hk, d), dtype, g), U.normal((b, new, hk, d), dtype, g)
    cos, sin = U.rotary_tables(room, rotary, dtype)
    kc_o, vc_o, kc_g, vc_g = kc.clone(), vc.clone(), kc.cuda(), vc.cuda()
    plan = ops.attention_forward(q.cuda(), kc.cuda(), vc.cuda(), k_new=k.cuda(), v_new=v.cuda(), seqused_k=lens.cuda(),
                                 block_table=_cuda(bt), rotary_cos=cos.cuda(), rotary_sin=sin.cuda(), causal=True, return_plan=True)[2]
    assert plan.kernel == L.KERNEL_DECODE
    go, gl = OA.flash_attn_with_kvcache(q, kc_o, vc_o, k, v, rotary_cos=cos, rotary_sin=sin, cache_seqlens=lens, block_table=bt,
                                        causal=True, rotary_interleaved=False)
    out, lse = fa2.flash_attn_with_kvcache(q.cuda(), kc_g, vc_g, k.cuda(), v.cuda(), rotary_cos=cos.cuda(), rotary_sin=sin.cuda(),
                                           cache_seqlens=lens.cuda(), block_table=_cuda(bt), causal=True,
                                           rotary_interleaved=False, return_softmax_lse=True)
    assert torch.equal(kc_g.cpu().view(torch.int16), kc_o.view(torch.int16)) and torch.equal(vc_g.cpu().view(torch.int16), vc_o.view(torch.int16))
    U.check_rules(out, lse, go, gl, tag=f"d {d} rows {rows}")


@pytest.mark.parametrize("b,hk,d,keys", [(1, 1, 128, 40000), (1, 1, 256, 9001), (2, 1, 64, 20001), (1, 8, 128, 2048), (3, 4, 128, 512)])
def test_few_sequences_are_cut_over_the_grid(b, hk, d, keys):
    """One unit over up to the whole grid: up to ~300 partials, the merge of more than 32 among them."""
    g = torch.Generator().manual_seed(keys)
    h = 4 * hk
    q, kc, vc = U.normal((b, 1, h, d), BF, g), U.normal((b, keys, hk, d), BF, g), U.normal((b, keys, hk, d), BF, g)
    lens = torch.tensor([keys, 1, keys // 3][:b], dtype=torch.int32)
    out, lse, pl = ops.attention_forward(q.cuda(), kc.cuda(), vc.cuda(), seqused_k=lens.cuda(), softmax_scale=d ** -0.5, causal=True,
                                         return_plan=True)
    assert pl.kernel == L.KERNEL_DECODE and pl.num_splits > 1
    go, gl = OA.flash_attn_with_kvcache(q, kc, vc, cache_seqlens=lens, causal=True)
    U.check_rules(out, lse, go, gl, tag=f"b {b} hk {hk} d {d} keys {keys}")


@pytest.mark.parametrize("n", [32, 33, 300, 1000])
@pytest.mark.parametrize("d", [4, 128, 256, 300])
def test_merge_of_many_partials(n, d):
    """fp32 partials, fp32 result: the merge's own rounding only, sqrt(n) terms of 2^-24 and two exponentials of 2^-22."""
    g = torch.Generator().manual_seed(n + d)
    o, lse = torch.randn((n, 2, 3, 2, d), generator=g), torch.randn((n, 2, 3, 2), generator=g) * 3
    lse[::3, 0, 1] = float("-inf")
    lse[:, 1, 2, 1] = float("-inf")
    o[:, 1, 2, 1] = float("nan")  # an empty partial's values are never read
    out, l = ops.combine(o.cuda(), lse.cuda())
    w = torch.softmax(lse.double(), 0).nan_to_num(0.0)
    want = (w.unsqueeze(-1) * o.double().nan_to_num(0.0)).sum(0)
    torch.testing.assert_close(out.cpu().double(), want, rtol=1e-5, atol=1e-5)
    want_l = torch.logsumexp(lse.double(), 0)
    want_l[want_l == float("-inf")] = float("inf")
    torch.testing.assert_close(l.cpu().double(), want_l, rtol=1e-5, atol=1e-5)


def _backward_inputs(g, dtype, rows_q, rows_k, h, hk, d):
    """2 (rand - 0.5), the distribution that the reference's backward tolerance (rtol = atol = 1e-2) is meant for."""
    r = lambda *s: (2.0 * (torch.rand(s, generator=g) - 0.5)).to(dtype)
    return r(*rows_q, h, d), r(*rows_k, hk, d), r(*rows_k, hk, d), r(*rows_q, h, d)


def _check_gradients(got, want):
    for name, a, b in zip(("dq", "dk", "dv"), got, want):
        torch.testing.assert_close(a.float().cpu(), b.float(), rtol=1e-2, atol=1e-2, msg=lambda m: f"{name}: {m}")
    assert L.load().fa_b200_check_status(torch.cuda.current_stream().cuda_stream) == 0


@pytest.mark.parametrize("dtype,b,s_q,s_k,h,hk,d,causal,window,softcap", [
    (BF, 1, 64, 64, 1, 1, 256, False, (-1, -1), 0.0), (FP, 2, 1, 129, 2, 1, 256, True, (-1, -1), 0.0),
    (BF, 1, 257, 191, 4, 2, 136, True, (-1, -1), 0.0), (BF, 1, 500, 500, 3, 3, 192, True, (-1, -1), 0.0),
    (FP, 1, 333, 400, 5, 1, 200, False, (-1, -1), 30.0), (BF, 2, 300, 460, 2, 2, 256, False, (70, 40), 0.0),
    (FP, 1, 640, 640, 2, 1, 192, True, (128, 0), 0.0), (BF, 1, 1100, 1100, 2, 1, 256, True, (-1, -1), 30.0)])
def test_wide_head_backward(dtype, b, s_q, s_k, h, hk, d, causal, window, softcap):
    """Head dims 129 .. 256 on the tcgen05 kernel: units and blocks cut off, rows without keys, grouped heads, windows."""
    from oracle import bwd as OB
    g = torch.Generator().manual_seed(d + s_q)
    q, k, v, dout = _backward_inputs(g, dtype, (b, s_q), (b, s_k), h, hk, d)
    kw = dict(softmax_scale=d ** -0.5, causal=causal, window_left=window[0], window_right=window[1], softcap=softcap)
    out, lse = ops.attention_forward(q.cuda(), k.cuda(), v.cuda(), **kw)
    grads = [torch.full_like(t, float("nan")).cuda() for t in (q, k, v)]  # every element must be written, zeros included
    n0 = L.load().fa_b200_launch_count()
    ops.attention_backward(dout.cuda(), q.cuda(), k.cuda(), v.cuda(), out, lse, dq=grads[0], dk=grads[1], dv=grads[2], **kw)
    assert L.load().fa_b200_launch_count() - n0 == 2  # rowsum and the one persistent kernel
    _check_gradients(grads, OB.attention_backward(q, k, v, dout, lse.cpu(), softmax_scale=d ** -0.5, causal=causal, window=window,
                                                  softcap=softcap))


@pytest.mark.parametrize("d,causal", [(192, True), (256, False)])
def test_wide_head_backward_packed(d, causal):
    from oracle import bwd as OB
    g = torch.Generator().manual_seed(d)
    lq, lk, h, hk = [130, 0, 1, 64, 300], [200, 77, 5, 64, 280], 4, 2
    cq, ck = [torch.tensor([0] + list(torch.tensor(x).cumsum(0)), dtype=torch.int32) for x in (lq, lk)]
    q, k, v, dout = _backward_inputs(g, BF, (sum(lq),), (sum(lk),), h, hk, d)
    kw = dict(softmax_scale=d ** -0.5, causal=causal, cu_seqlens_q=cq.cuda(), cu_seqlens_k=ck.cuda(), max_seqlen_q=max(lq), max_seqlen_k=max(lk))
    out, lse = ops.attention_forward(q.cuda(), k.cuda(), v.cuda(), **kw)
    grads = [torch.full_like(t, float("nan")).cuda() for t in (q, k, v)]
    ops.attention_backward(dout.cuda(), q.cuda(), k.cuda(), v.cuda(), out, lse, dq=grads[0], dk=grads[1], dv=grads[2], **kw)
    _check_gradients(grads, OB.attention_varlen_backward(q, k, v, dout, lse.cpu(), cq, ck, softmax_scale=d ** -0.5, causal=causal,
                                                         window=(-1, -1)))


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("dtype,d", [(BF, 128), (FP, 64), (BF, 256)])
def test_packed_tiles_of_more_than_32_sequences(dtype, d, causal):
    """Tiles are drawn by level and batch entry, 32 entries at a time: empty sequences, sequences of one tile and of several,
    lengths at the tiles' edges, keys longer and shorter than the queries, an entry count that is not a multiple of 32."""
    import flash_attn_npu_v2 as fa2
    g = torch.Generator().manual_seed(d + causal)
    h, hk = 4, 2
    q_lens = ([0, 1, 127, 128, 129, 255, 256, 257, 513, 3] * 4)[:37]
    k_lens = [n + x if n else 0 for n, x in zip(q_lens, [0, 5, 300, 0, 640, 1, 0, 128, 77, 0] * 4)]
    k_lens[7] = 200  # fewer keys than queries
    cq, ck = (torch.tensor([0] + list(torch.tensor(x).cumsum(0)), dtype=torch.int32) for x in (q_lens, k_lens))
    q = U.normal((sum(q_lens), h, d), dtype, g)
    k, v = U.normal((sum(k_lens), hk, d), dtype, g), U.normal((sum(k_lens), hk, d), dtype, g)
    out, lse, *_ = fa2.flash_attn_varlen_func(q.cuda(), k.cuda(), v.cuda(), cq.cuda(), ck.cuda(), max(q_lens), max(k_lens),
                                              causal=causal, return_attn_probs=True)
    for i, n in enumerate(q_lens):
        if not n:
            continue
        rq, rk = slice(int(cq[i]), int(cq[i + 1])), slice(int(ck[i]), int(ck[i + 1]))
        go, gl = OA.flash_attn_func(q[rq].unsqueeze(0), k[rk].unsqueeze(0), v[rk].unsqueeze(0), causal=causal)
        U.check_rules(out[rq].unsqueeze(0), lse[:, rq].unsqueeze(0), go, gl, tag=f"sequence {i}")


def test_head_chunks_of_a_large_cache():
    """A cache too large for L2 runs its heads in chunks (here 8 and 4 of 12 query heads)."""
    import flash_attn_npu_v2 as fa2
    g = torch.Generator().manual_seed(5)
    b, s_q, h, hk, d, room = 3, 300, 12, 6, 128, 16384
    lens = torch.tensor([300, 700, 2049], dtype=torch.int32)
    kc, vc = torch.zeros((b, room, hk, d), dtype=BF), torch.zeros((b, room, hk, d), dtype=BF)
    kc[:, :2049], vc[:, :2049] = U.normal((b, 2049, hk, d), BF, g), U.normal((b, 2049, hk, d), BF, g)
    q = U.normal((b, s_q, h, d), BF, g)
    out, lse = fa2.flash_attn_with_kvcache(q.cuda(), kc.cuda(), vc.cuda(), cache_seqlens=lens.cuda(), causal=True, return_softmax_lse=True)
    go, gl = OA.flash_attn_with_kvcache(q, kc[:, :2049].contiguous(), vc[:, :2049].contiguous(), cache_seqlens=lens, causal=True)
    U.check_rules(out, lse, go, gl, tag="head chunks")


@pytest.mark.parametrize("d", [192, 256])
def test_wide_head_backward_short_items(d):
    """More items than SMs, most of one or two units: a CTA's dV items end while their tiles are still arriving, and the dQ
    items behind them must wait for their own.  Every repetition gives the same bits."""
    from oracle import bwd as OB
    g = torch.Generator().manual_seed(d)
    lens = ([1, 128, 64, 65, 17, 127, 129, 100] * 10)[:75]
    h, hk = 4, 2
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32)
    q, k, v, dout = _backward_inputs(g, BF, (sum(lens),), (sum(lens),), h, hk, d)
    kw = dict(softmax_scale=d ** -0.5, causal=True, cu_seqlens_q=cu.cuda(), cu_seqlens_k=cu.cuda(), max_seqlen_q=max(lens),
              max_seqlen_k=max(lens))
    qg, kg, vg, dg = q.cuda(), k.cuda(), v.cuda(), dout.cuda()
    out, lse = ops.attention_forward(qg, kg, vg, **kw)
    grads = ops.attention_backward(dg, qg, kg, vg, out, lse, **kw)
    for _ in range(20):
        again = [torch.full_like(t, float("nan")) for t in (qg, kg, vg)]
        ops.attention_backward(dg, qg, kg, vg, out, lse, dq=again[0], dk=again[1], dv=again[2], **kw)
        assert all(torch.equal(a, b) for a, b in zip(grads, again))
    _check_gradients(grads, OB.attention_varlen_backward(q, k, v, dout, lse.cpu(), cu, cu, softmax_scale=d ** -0.5, causal=True,
                                                         window=(-1, -1)))


@pytest.mark.parametrize("dtype,d,causal", [(BF, 128, True), (FP, 64, False)])
def test_backward_of_many_short_sequences(dtype, d, causal):
    """Several hundred packed sequences of 1 - 128 rows: every dQ item has one key block, so the products of an item may
    run while the elementwise warps still finish the item before."""
    from oracle import bwd as OB
    g = torch.Generator().manual_seed(d)
    lens = [1 + (37 * i) % 128 for i in range(400)]
    h, hk = 4, 2
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32)
    q, k, v, dout = _backward_inputs(g, dtype, (sum(lens),), (sum(lens),), h, hk, d)
    kw = dict(softmax_scale=d ** -0.5, causal=causal, cu_seqlens_q=cu.cuda(), cu_seqlens_k=cu.cuda(), max_seqlen_q=max(lens),
              max_seqlen_k=max(lens))
    out, lse = ops.attention_forward(q.cuda(), k.cuda(), v.cuda(), **kw)
    grads = [torch.full_like(t, float("nan")).cuda() for t in (q, k, v)]
    ops.attention_backward(dout.cuda(), q.cuda(), k.cuda(), v.cuda(), out, lse, dq=grads[0], dk=grads[1], dv=grads[2], **kw)
    _check_gradients(grads, OB.attention_varlen_backward(q, k, v, dout, lse.cpu(), cu, cu, softmax_scale=d ** -0.5, causal=causal,
                                                         window=(-1, -1)))


SCHEDULES = {"plain": (dict(num_splits=1), 1, 1), "splits": (dict(num_splits=2), 2, 2), "shared": (dict(), 2, 5)}  # arguments, launches, least splits


@pytest.mark.parametrize("schedule", SCHEDULES)
@pytest.mark.parametrize("rows", [1, 16])
@pytest.mark.parametrize("d", [64, 72, 96, 128, 136, 192, 256])
def test_decode_kernel_without_clusters(monkeypatch, d, rows, schedule):
    """Up to 16 packed rows on one CTA per unit, on key splits with partials and on equal shares of all blocks; new tokens appended
    with rotary; lengths around the key blocks' edges."""
    monkeypatch.setenv("FA_B200_DECODE_CLUSTER", "0")
    g = torch.Generator().manual_seed(d * 100 + rows)
    dtype = BF if rows % 2 else FP
    hk, group, s_q = 2, {1: 1, 16: 8}[rows], {1: 1, 16: 2}[rows]
    new, room = s_q, 1300
    lens = torch.tensor([0, 1, 127, 128, 700, room - new], dtype=torch.int32)
    b, rotary = lens.numel(), d // 16 * 16
    q, (kc, vc, _) = U.normal((b, s_q, hk * group, d), dtype, g), _cache(g, dtype, b, room, hk, d, 0)
    k, v = U.normal((b, new, hk, d), dtype, g), U.normal((b, new, hk, d), dtype, g)
    cos, sin = U.rotary_tables(room, rotary, dtype)
    kw, launches, least = SCHEDULES[schedule]
    kc_g, vc_g = kc.cuda(), vc.cuda()
    n0 = L.load().fa_b200_launch_count()
    out, lse, pl = ops.attention_forward(q.cuda(), kc_g, vc_g, k_new=k.cuda(), v_new=v.cuda(), seqused_k=lens.cuda(), rotary_cos=cos.cuda(),
                                         rotary_sin=sin.cuda(), rotary_interleaved=False, causal=True, softmax_scale=d ** -0.5, return_plan=True, **kw)
    assert L.load().fa_b200_launch_count() - n0 == launches == pl.launches
    assert pl.kernel == L.KERNEL_DECODE and pl.config == 3 and pl.num_splits >= least and (pl.blocks_per_split == 0) == (schedule == "shared")
    go, gl = OA.flash_attn_with_kvcache(q, kc, vc, k, v, rotary_cos=cos, rotary_sin=sin, cache_seqlens=lens, causal=True,
                                        rotary_interleaved=False)  # appends to kc, vc
    assert torch.equal(kc_g.cpu().view(torch.int16), kc.view(torch.int16)) and torch.equal(vc_g.cpu().view(torch.int16), vc.view(torch.int16))
    U.check_rules(out, lse, go, gl, tag=f"d {d} rows {rows} {schedule}")


@pytest.mark.parametrize("schedule", SCHEDULES)
def test_alibi_without_clusters(monkeypatch, schedule):
    monkeypatch.setenv("FA_B200_DECODE_CLUSTER", "0")
    g = torch.Generator().manual_seed(5)
    b, h, hk, d, room = 3, 6, 3, 128, 1300
    q, kc, vc = U.normal((b, 2, h, d), FP, g), U.normal((5, room, hk, d), FP, g), U.normal((5, room, hk, d), FP, g)
    lens, idx = torch.tensor([10, 1250, 640], dtype=torch.int32), torch.tensor([4, 0, 2], dtype=torch.int32)
    slopes = torch.rand(b, h, generator=g) * 0.3
    kw, launches, _ = SCHEDULES[schedule]
    for causal in (False, True):
        out, lse, pl = ops.attention_forward(q.cuda(), kc.cuda(), vc.cuda(), seqused_k=lens.cuda(), cache_batch_idx=idx.cuda(), causal=causal,
                                             alibi_slopes=slopes.cuda(), softmax_scale=d ** -0.5, return_plan=True, **kw)
        assert pl.kernel == L.KERNEL_DECODE and pl.config == 3 and pl.launches == launches
        go, gl = OA.flash_attn_with_kvcache(q, kc, vc, cache_seqlens=lens, cache_batch_idx=idx, causal=causal, alibi_slopes=slopes)
        U.check_rules(out, lse, go, gl, tag=f"alibi {schedule}")


@pytest.mark.parametrize("b,hk,d,keys", [(1, 8, 128, 4500), (1, 8, 128, 2048), (3, 4, 128, 512)])
def test_short_sequences_are_cut_over_the_grid_without_clusters(monkeypatch, b, hk, d, keys):
    """Partials and a merge where clusters are switched off, up to and behind the range that they take."""
    monkeypatch.setenv("FA_B200_DECODE_CLUSTER", "0")
    n0 = L.load().fa_b200_launch_count()
    test_few_sequences_are_cut_over_the_grid(b, hk, d, keys)
    assert L.load().fa_b200_launch_count() - n0 == 2


@pytest.mark.parametrize("d,h", [(128, 32), (192, 24)])
def test_backward_item_order_of_streams_beyond_l2(d, h):
    """The causal backward takes a pair at a time when the streamed tensors exceed 88 MB, and the blocks of all pairs together below:
    a head's gradients are the same to the bit."""
    g = torch.Generator().manual_seed(d)
    b, s, part = 1, 8192, 8
    assert 4 * b * s * h * d > 88 << 20 >= 4 * b * s * part * d
    q, k, v, dout = (t.cuda() for t in _backward_inputs(g, BF, (b, s), (b, s), h, h, d))
    kw = dict(softmax_scale=d ** -0.5, causal=True)
    out, lse = ops.attention_forward(q, k, v, **kw)
    grads = ops.attention_backward(dout, q, k, v, out, lse, **kw)
    for h0 in range(0, h, part):
        at = [t[:, :, h0:h0 + part].contiguous() for t in (dout, q, k, v, out)]
        some = ops.attention_backward(*at, lse[:, h0:h0 + part].reshape(-1).view(b, part, s), **kw)
        for all_heads, x in zip(grads, some):
            assert torch.equal(all_heads[:, :, h0:h0 + part], x), h0


@pytest.mark.parametrize("d", [64, 128, 256])
def test_calls_that_start_under_one_another(d):
    """Kernels that are launched to start under the end of the one in front: a chain in which every call reads what the call before
    wrote (its output as q, its keys in the cache) gives the bits of the same chain with a synchronisation behind every call, back to
    back and in a CUDA graph."""
    import flash_attn_npu_v2 as fa2
    g = torch.Generator().manual_seed(d)
    b, s, h, hk, room = 2, 100, 8, 2, 6000  # 100 rows: the mma.sync kernel, 32 CTAs; the caches: equal shares and key splits
    q0, k0, v0 = (U.normal((b, s, n, d), BF, g).cuda() for n in (h, hk, hk))
    kc0, vc0 = (U.normal((b, room, hk, d), BF, g).cuda() for _ in range(2))
    lens, short = (torch.tensor(t, dtype=torch.int32).cuda() for t in ([5900, 3000], [300, 20]))

    def chain(sync):
        wait = torch.cuda.synchronize if sync else (lambda: None)
        kc, vc, x, seen = kc0.clone(), vc0.clone(), q0, []
        for n in range(6):
            x = fa2.flash_attn_func(x, k0, v0, causal=True); wait()
            row = x[:, n:n + 1].contiguous()
            new = row[:, :, ::4].contiguous()
            row = fa2.flash_attn_with_kvcache(row, kc, vc, new, new, cache_seqlens=lens + n, causal=True); wait()           # appends
            row = fa2.flash_attn_with_kvcache(row, kc, vc, cache_seqlens=lens + n + 1, causal=True, num_splits=3); wait()
            row = fa2.flash_attn_with_kvcache(row, kc[:, :512], vc[:, :512], cache_seqlens=short, causal=True); wait()      # clusters
            x = x + row
            seen.append(row)
        return [x, kc, vc] + seen

    want = [t.clone() for t in chain(True)]
    for got in (chain(False), chain(False)):
        assert all(torch.equal(a, c) for a, c in zip(want, got))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = chain(False)
    for _ in range(3):
        graph.replay()
        assert all(torch.equal(a, c) for a, c in zip(want, got))


@pytest.mark.parametrize("s_q,s_k,causal,window", [
    (128, 1, False, (-1, -1)), (128, 128, True, (-1, -1)), (129, 129, True, (-1, -1)), (256, 256, False, (-1, -1)),
    (257, 385, True, (-1, -1)), (300, 200, True, (-1, -1)),  # rows that see no key
    (513, 513, True, (100, 0)), (400, 640, False, (200, 130)),
    (256, 1500, False, (-1, -1)), (700, 1100, True, (-1, -1))])  # many blocks between two tiles' last ones
def test_two_p_buffers_over_many_tiles(s_q, s_k, causal, window):
    """Head dim 64: tiles of one, two and more key blocks, sub-tiles of unequal length, one tile after another on every SM (two P
    buffers with a barrier each for the P.V that has read them, and factors that alternate between two rows across tiles; the
    softmax warps look at one phase of those barriers a tile, the more the blocks the more pass unseen)."""
    g = torch.Generator().manual_seed(s_q + s_k)
    b, h, hk = 5, 64, 4
    q, k, v = U.normal((b, s_q, h, 64), FP, g), U.normal((b, s_k, hk, 64), FP, g), U.normal((b, s_k, hk, 64), FP, g)
    out, lse, pl = ops.attention_forward(q.cuda(), k.cuda(), v.cuda(), softmax_scale=0.125, causal=causal, window_left=window[0],
                                         window_right=window[1], return_plan=True)
    assert pl.kernel == L.KERNEL_TCGEN05 and b * h > 2 * 148
    go, gl = OA.flash_attn_func(q, k, v, causal=causal, window_size=window)
    U.check_rules(out, lse, go, gl, tag=f"{s_q} x {s_k}")
