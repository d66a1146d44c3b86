"""The library of the text decoders' kernel units is whole by itself: it links, loads and exports what its callers declare."""
import ctypes


def test_text_units_load_by_themselves(tmp_path):
    from inference_b200 import _native
    from inference_b200._native import build

    srcs = [build.CSRC / "kernels" / f"{u}.cu" for u in build.TEXT_UNITS]
    lib = ctypes.CDLL(str(build._build_kernel_lib(srcs, tmp_path / "libswb200_text.so", False)))     # undefined symbols raise here
    _native._declare_kernels(lib)
    for name in ("swb_gemm_bf16_act", "swb_gemm_bf16_gated", "swb_gemm_bf16_routed", "swb_moe_combine", "swb_attn_varlen_causal"):
        assert hasattr(lib, name), name
