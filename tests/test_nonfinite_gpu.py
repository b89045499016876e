"""GPU: a NaN or an infinite score among the keys that a row sees makes the row's output and LSE NaN, whichever way the decode call
is shared out; the other rows and heads do not notice, to the bit.  Which rows are affected is asked of the oracle."""
import pytest
import torch

import parity_util as U
from flash_b200 import lib as L
from flash_b200 import ops
from oracle import api as OA

pytestmark = pytest.mark.gpu
BF, FP = torch.bfloat16, torch.float16
NAN, INF = float("nan"), float("inf")
ROUTES = {  # sequences, kv heads, keys of the longest, arguments, launches
    "plain": (2, 2, 500, dict(num_splits=1), 1),
    "cluster": (2, 2, 500, dict(), 1),
    "splits": (2, 2, 500, dict(num_splits=3), 2),
    "shared": (4, 4, 4500, dict(), 2),               # equal shares of all blocks, merge of up to 32 partials
    "shared_many": (2, 1, 9000, dict(), 2),          # ... of more
    "mma_splits": (2, 2, 500, dict(kernel=L.KERNEL_MMA, num_splits=3), 2),
    "mma_plain": (2, 2, 500, dict(kernel=L.KERNEL_MMA, num_splits=1), 1)}


@pytest.mark.parametrize("fault", ["key", "query", "score"])
@pytest.mark.parametrize("dtype,d", [(BF, 64), (FP, 128), (BF, 256)])
@pytest.mark.parametrize("route", ROUTES)
def test_nonfinite_rows_stay_nonfinite(route, dtype, d, fault):
    b, hk, keys, kw, launches = ROUTES[route]
    g = torch.Generator().manual_seed(d + keys)
    q, k, v = U.normal((b, 1, 4 * hk, d), dtype, g), U.normal((b, keys, hk, d), dtype, g), U.normal((b, keys, hk, d), dtype, g)
    lens = torch.tensor([keys - 3 - i for i in range(b)], dtype=torch.int32)
    q[..., 7] = q[..., 7].abs() + 0.5  # an infinite element of K becomes a score of +inf

    def call(q, k):
        n0 = L.load().fa_b200_launch_count()
        got = ops.attention_forward(q.cuda(), k.cuda(), v.cuda(), seqused_k=lens.cuda(), softmax_scale=d ** -0.5, causal=True, **kw)
        assert L.load().fa_b200_launch_count() - n0 == launches
        return [t.cpu() for t in got]

    out0, lse0 = call(q, k)
    if fault == "query":
        q[0, 0, 1, 5] = NAN
    else:
        k[0, keys // 3, 0, 7] = NAN if fault == "key" else INF
    out, lse = call(q, k)
    go, gl = OA.flash_attn_with_kvcache(q, k, v, cache_seqlens=lens, causal=True)
    bad = gl.isnan()
    assert int(bad.sum()) == (1 if fault == "query" else 4)
    assert torch.equal(lse.isnan(), bad) and torch.equal(out.isnan(), go.isnan()), f"{route} {fault}"
    ok = ~bad.transpose(1, 2)  # (b, 1, h)
    assert torch.equal(lse[~bad], lse0[~bad]) and torch.equal(out[ok].view(torch.int16), out0[ok].view(torch.int16))


def test_merge_of_nonfinite_partials():
    """The merge by itself, up to 32 partials and more: a NaN among empty partials, and every partial NaN."""
    for n in (2, 32, 33, 300):
        g = torch.Generator().manual_seed(n)
        o, lse = torch.randn((n, 1, 1, 5, 64), generator=g), torch.randn((n, 1, 1, 5), generator=g)
        lse[:, 0, 0, 0] = -INF
        lse[n - 1, 0, 0, 0] = NAN   # all the others are empty
        lse[n // 2, 0, 0, 1] = NAN
        lse[:, 0, 0, 2] = NAN
        lse[:, 0, 0, 3] = -INF      # a row without keys
        for partial in (False, True):
            out, l = [t.cpu() for t in ops.combine(o.cuda(), lse.cuda(), partial_out=partial)]
            assert out[0, 0, :3].isnan().all() and l[0, 0, :3].isnan().all(), n
            assert torch.equal(out[0, 0, 3], torch.zeros(64)) and float(l[0, 0, 3]) == (-INF if partial else INF)
            want = (torch.softmax(lse[:, 0, 0, 4].double(), 0)[:, None] * o[:, 0, 0, 4].double()).sum(0)
            torch.testing.assert_close(out[0, 0, 4].double(), want, rtol=1e-5, atol=1e-5)
