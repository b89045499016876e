"""B200 backend of the flash_attn_npu_v2 / flash_attn_npu_v3 drop-in modules.

``ops.attention_forward`` / ``ops.combine`` wrap the C ABI of libfa_b200.so;
``_native`` is the native host path of the public calls (csrc/torch_binding.cpp);
``dist`` holds the multi-GPU helpers (sharding, cross-GPU merge of partials).
"""
from . import lib, ops  # noqa: F401

lib.load()  # no fallback: fail at import when libfa_b200.so (or the host path linked against it) is missing
from . import _native  # noqa: E402,F401

__all__ = ["lib", "ops"]
