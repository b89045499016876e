"""GPU: calls that the native host path (csrc/torch_binding.cpp) must leave to the registered operators."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _qkv(seed=0, s=64, grad=False):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn((2, s, 4, 64), generator=g, device="cuda", dtype=BF, requires_grad=grad) for _ in range(3)]


@pytest.mark.parametrize("api", ["flash_attn_npu_v2", "flash_attn_npu_v3"])
def test_trace_records_the_attention(api):
    """A traced function computes attention of the inputs it is called with."""
    fa = pytest.importorskip(api)
    fns = [lambda q, k, v: fa.flash_attn_func(q, k, v, causal=True)]
    if api.endswith("v3"):  # (the cache call of v2 is not a registered operator)
        fns.append(lambda q, k, v: fa.flash_attn_with_kvcache(q, k, v, causal=True))
    for fn in fns:
        traced = torch.jit.trace(fn, tuple(_qkv(1)), check_trace=False)
        q, k, v = _qkv(2)
        assert torch.equal(traced(q, k, v), fn(q, k, v))


@pytest.mark.parametrize("requires_grad", [False, True])
@pytest.mark.parametrize("api", ["flash_attn_npu_v2", "flash_attn_npu_v3"])
def test_forward_mode_differentiation_is_refused(api, requires_grad):
    """There is no jvp: a dual tensor raises instead of losing its tangent."""
    import torch.autograd.forward_ad as fwAD
    fa = pytest.importorskip(api)
    for which in range(3):
        with fwAD.dual_level(), pytest.raises(NotImplementedError, match="jvp"):
            ts = _qkv(3, grad=requires_grad)
            ts[which] = fwAD.make_dual(ts[which], torch.ones_like(ts[which]))
            fa.flash_attn_func(*ts, causal=True)


def test_kvcache_call_on_inputs_that_require_grad():
    """v3: the call has no autograd formula.  Its output requires a gradient and the backward says so; it is not detached."""
    import flash_attn_npu_v3 as fa3
    q, k, v = _qkv(4)
    q.requires_grad_(True)
    out = fa3.flash_attn_with_kvcache(q, k, v, causal=True)
    assert out.requires_grad
    with pytest.raises(RuntimeError, match="no autograd formula"):
        out.sum().backward()
    with torch.no_grad():
        assert torch.equal(fa3.flash_attn_with_kvcache(q, k, v, causal=True), out)


def test_workspace_that_does_not_fit_is_an_out_of_memory_error():
    """The partials of a split call are allocated through a callback of the C library; its failure is torch's own error."""
    import flash_attn_npu_v2 as fa2
    g = torch.Generator(device="cuda").manual_seed(5)
    q = torch.randn((16, 4, 64, 128), generator=g, device="cuda", dtype=BF)  # 64 splits: 135 MB of partials
    k, v = (torch.randn((16, 8192, 8, 128), generator=g, device="cuda", dtype=BF) for _ in range(2))
    lens = torch.full((16,), 8192, dtype=torch.int32, device="cuda")
    call = lambda: fa2.flash_attn_with_kvcache(q, k, v, cache_seqlens=lens, causal=True, num_splits=64)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    try:
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (60 << 20)) / total)
        with pytest.raises(torch.cuda.OutOfMemoryError):
            call()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.isfinite(call().float()).all()
