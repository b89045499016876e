"""GPU: decode calls of few units and short ranges, whose key splits are the CTAs of one thread-block cluster: head dims between
the tile widths, cluster sizes 2, 4 and 8, ranges that leave CTAs without keys, empty sequences, appended tokens, windows, softcap.
Inputs are N(0, 1); tolerances are the rules of precision.py."""
import pytest
import torch

import parity_util as U
from flash_b200 import lib as L
from flash_b200 import ops
from oracle import api as OA

pytestmark = pytest.mark.gpu
BF, FP = torch.bfloat16, torch.float16


def test_splits_that_are_asked_for_are_kept():
    import flash_attn_npu_v3 as fa3
    g = torch.Generator().manual_seed(1)
    q, k, v = U.normal((1, 1, 8, 128), BF, g), U.normal((1, 1024, 2, 128), BF, g), U.normal((1, 1024, 2, 128), BF, g)
    lens = torch.tensor([1000], dtype=torch.int32)
    go, gl = OA.flash_attn_with_kvcache(q, k, v, cache_seqlens=lens, causal=True)
    for splits, launches in ((0, 1), (1, 1), (3, 2)):
        n0 = L.load().fa_b200_launch_count()
        out, lse, *_ = fa3.flash_attn_with_kvcache(q.cuda(), k.cuda(), v.cuda(), cache_seqlens=lens.cuda(), causal=True, num_splits=splits,
                                                   return_softmax_lse=True)
        assert L.load().fa_b200_launch_count() - n0 == launches
        U.check_rules(out, lse, go, gl, tag=f"splits {splits}")


@pytest.mark.parametrize("dtype,d,b,hk,group,s_q,room,page,append,window,softcap,cluster", [
    (BF, 128, 1, 8, 4, 1, 2048, 0, False, -1, 0.0, 8),
    (FP, 64, 3, 4, 8, 2, 700, 128, True, -1, 0.0, 4),      # 16 rows; sequences with fewer blocks than CTAs
    (BF, 256, 5, 6, 2, 1, 1000, 256, True, 300, 0.0, 2),   # a window
    (BF, 96, 16, 4, 1, 3, 513, 0, False, -1, 30.0, 2),
    (FP, 136, 4, 2, 4, 4, 130, 128, False, 40, 0.0, 2),    # a range of two key blocks
    (BF, 128, 2, 2, 16, 1, 129, 0, True, -1, 0.0, 2)])
def test_clustered_decode(dtype, d, b, hk, group, s_q, room, page, append, window, softcap, cluster):
    import flash_attn_npu_v2 as fa2
    g = torch.Generator().manual_seed(d * 10 + b)
    new = s_q if append else 0
    lens = torch.tensor(([room - new, 0, 1, 127, 64, room // 2] * 3)[:b], dtype=torch.int32)
    q = U.normal((b, s_q, hk * group, d), dtype, g)
    if page:
        per = -(-room // page)
        bt = torch.randperm(b * per, generator=g).view(b, per).to(torch.int32)
        shape = (b * per, page, hk, d)
    else:
        bt, shape = None, (b, room, hk, d)
    kc, vc = U.normal(shape, dtype, g), U.normal(shape, dtype, g)
    kn, vn = (U.normal((b, new, hk, d), dtype, g), U.normal((b, new, hk, d), dtype, g)) if new else (None, None)
    dev = lambda t: None if t is None else t.cuda()  # noqa: E731
    kc_o, vc_o, kc_g, vc_g = kc.clone(), vc.clone(), kc.cuda(), vc.cuda()
    kw = dict(causal=True, window_size=(window, -1), softcap=softcap)
    go, gl = OA.flash_attn_with_kvcache(q, kc_o, vc_o, kn, vn, cache_seqlens=lens, block_table=bt, **kw)
    pl = ops.attention_forward(q.cuda(), kc.cuda(), vc.cuda(), k_new=dev(kn), v_new=dev(vn), seqused_k=lens.cuda(), block_table=dev(bt),
                               causal=True, window_left=window, softcap=softcap, return_plan=True)[2]
    assert pl.kernel == L.KERNEL_DECODE and pl.config == 3 + 256 * cluster and pl.grid == b * hk * cluster
    n0 = L.load().fa_b200_launch_count()
    for _ in range(2):  # the appended rows are written again with the same values
        out, lse = fa2.flash_attn_with_kvcache(q.cuda(), kc_g, vc_g, dev(kn), dev(vn), cache_seqlens=lens.cuda(), block_table=dev(bt),
                                               return_softmax_lse=True, **kw)
        U.check_rules(out, lse, go, gl, tag=f"d {d} b {b}")
    assert L.load().fa_b200_launch_count() - n0 == 2  # no merge launch
    assert torch.equal(kc_g.cpu().view(torch.int16), kc_o.view(torch.int16)) and torch.equal(vc_g.cpu().view(torch.int16), vc_o.view(torch.int16))


@pytest.mark.parametrize("b,hk,room,lens,window,cluster", [
    (1, 8, 32768, [30000], 1024, True), (4, 8, 400, [400, 3, 250, 399], -1, True), (1, 8, 2048, [2000], -1, True),
    (1, 8, 2048, [2000], -1, False), (4, 8, 400, [400, 3, 250, 399], -1, False), (3, 2, 600, [0, 0, 0], -1, True)])
def test_a_plan_runs_what_it_says(monkeypatch, b, hk, room, lens, window, cluster):
    """A planned call makes the plan's launches and gives the bits of the call that is planned on the spot, for plans with clusters and
    for plans that were made without them."""
    import ctypes as C
    import flash_attn_npu_v3 as fa3
    g = torch.Generator().manual_seed(room)
    d, h = 128, 4 * hk
    q, k, v = U.normal((b, 1, h, d), BF, g).cuda(), U.normal((b, room, hk, d), BF, g).cuda(), U.normal((b, room, hk, d), BF, g).cuda()
    lens_g = torch.tensor(lens, dtype=torch.int32).cuda()
    if not cluster:
        monkeypatch.setenv("FA_B200_DECODE_CLUSTER", "0")
    kw = dict(cache_seqlens=lens_g, causal=True, window_size=(window, -1), return_softmax_lse=True)
    plan = fa3.get_scheduler_metadata(b, 1, room, h, hk, d, lens_g, qkv_dtype=BF, causal=True, window_size=(window, -1))
    raw, pl = bytes(plan.cpu().numpy().tobytes()), L.FwdPlan()
    L.check(L.load().fa_b200_plan_decode(raw, len(raw), C.byref(pl)))
    want = fa3.flash_attn_with_kvcache(q, k, v, **kw)[:2]
    monkeypatch.delenv("FA_B200_DECODE_CLUSTER", raising=False)
    n0 = L.load().fa_b200_launch_count()
    got = fa3.flash_attn_with_kvcache(q, k, v, scheduler_metadata=plan, **kw)[:2]
    assert L.load().fa_b200_launch_count() - n0 == pl.launches
    assert (pl.config // 256 > 1) == cluster
    for x, y in zip(want, got):
        assert torch.equal(x, y)
    go, gl = OA.flash_attn_with_kvcache(q.cpu(), k.cpu(), v.cpu(), cache_seqlens=lens_g.cpu(), causal=True, window_size=(window, -1))
    U.check_rules(got[0], got[1], go, gl, tag=f"planned {b} {room}")
