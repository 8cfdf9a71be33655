"""ctypes loader of libf3d_b200.so and the prototypes of its C ABI (include/f3d_b200.h).

There is no CPU fallback: if the shared library is missing or a call fails, a RuntimeError is raised.
"""
from __future__ import annotations

import ctypes
import importlib.machinery
import importlib.util
import os
from ctypes import c_char_p, c_float, c_int, c_uint32, c_uint64, c_void_p
from pathlib import Path

LIB_PATH = Path(__file__).resolve().parent / "libf3d_b200.so"

_u32, _vp, _int, _f32 = c_uint32, c_void_p, c_int, c_float


class XfmrBlock(ctypes.Structure):
    """f3d_xfmr_block of include/f3d_b200.h."""
    _fields_ = [(n, c_void_p) for n in ("norm_w", "norm_b", "qkv_w", "qkv_b", "proj_w", "proj_b", "ln2_w", "ln2_b", "fc1_w",
                                        "fc1_b", "fc2_w", "fc2_b", "qkv_colsum", "fc1_colsum", "scopes")] + [
                (n, c_float) for n in ("norm_eps", "ln2_eps")] + [
                (n, c_int) for n in ("heads", "hidden", "num_scopes", "scope_size", "bucket")]


class XfmrSaved(ctypes.Structure):
    """f3d_xfmr_saved of include/f3d_b200.h."""
    _fields_ = [(n, c_void_p) for n in ("x", "n1", "qkv", "attn", "lse", "mid", "n2", "hid", "out")]


class XfmrGrads(ctypes.Structure):
    """f3d_xfmr_grads of include/f3d_b200.h."""
    _fields_ = [(n, c_void_p) for n in ("qkv_wt", "proj_wt", "fc1_wt", "fc2_wt", "norm_w", "norm_b", "qkv_w", "qkv_b", "proj_w", "proj_b",
                                        "ln2_w", "ln2_b", "fc1_w", "fc1_b", "fc2_w", "fc2_b", "grad_x", "g_pre", "g_mid", "g_qkv")] + [
                ("covered", c_int)]


# name -> (restype, argtypes); mirrors include/f3d_b200.h declaration by declaration
PROTOTYPES = {
    "f3d_last_error": (c_char_p, []),
    "f3d_version": (_int, []),
    "f3d_init_device": (_int, [_int]),
    "f3d_set_sync": (_int, [_int]),
    "f3d_get_sync": (_int, []),
    "f3d_set_seed": (_int, [c_uint64]),
    "f3d_get_seed": (c_uint64, []),
    "f3d_set_scene_base": (_int, [_u32]),
    "f3d_get_scene_base": (_u32, []),
    "f3d_release_workspaces": (_int, []),
    "f3d_launch_count": (ctypes.c_ulonglong, []),
    "f3d_batch_psh_scatter_pad_hash": (_int, [_vp, _vp, _vp, _vp, _vp, _u32, _u32, _u32, _u32, _u32, _u32, _u32,
                                              _vp, _vp, _vp, _vp, _vp, _u32, _f32, _u32, _int, _vp]),
    "f3d_batch_psh_scatter_pad_hash_noalloc": (_int, [_vp, _vp, _vp, _vp, _vp, _u32, _u32, _u32, _u32, _u32, _u32, _u32,
                                                      _vp, _vp, _vp, _vp, _vp, _u32, _f32, _u32, _int, _vp]),
    "f3d_batch_bucket_sanitizer_cpu": (_int, [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _u32, _u32, _u32, _u32]),
    "f3d_batch_subbuck_reduce": (_int, [_vp, _vp, _vp, _u32, _u32, _u32, _u32, _u32, _vp, _vp, _vp, _vp, _vp, _vp, _vp,
                                        _vp, _u32, _u32, _u32, _int, _u32, _u32, _int, _vp]),
    "f3d_batch_subbuck_reduce_backward": (_int, [_vp, _vp, _vp, _vp, _u32, _u32, _u32, _int, _u32, _u32, _int, _vp]),
    "f3d_additive_unpool_fwd": (_int, [_vp, _vp, _vp, _vp, _u32, _u32, _u32, _u32, _int, _u32, _int, _vp]),
    "f3d_additive_unpool_bwd": (_int, [_vp, _vp, _vp, _vp, _u32, _u32, _u32, _int, _u32, _int, _vp]),
    "f3d_device_status": (_int, [_int]),
    "f3d_linear_bf16": (_int, [_vp, _vp, _vp, _vp, _vp, _int, _int, _int, _int, _int, _int, _vp]),
    "f3d_linear_dtype": (_int, [_vp, _vp, _vp, _vp, _vp, _int, _int, _int, _int, _int, _int, _int, _vp]),
    "f3d_buck_swin_fwd_dtype": (_int, [_vp, _vp, _vp, _vp, _vp, _vp, _int, _int, _int, _int, _int, _int, _u32, _int, _int, _vp]),
    "f3d_linear_fused": (_int, [_vp, _vp, _vp, _vp, _vp, _int, _int, _int, _int, _int, _int, _vp, _vp, _f32, _vp, _int, _vp]),
    "f3d_bbox_f16": (_int, [_vp, _vp, _vp, _u32, _int, _vp]),
    "f3d_clear_unlisted": (_int, [_vp, _vp, _int, _int, c_uint64, _int, _int, _u32, _int, _vp]),
    "f3d_row_stats_bf16": (_int, [_vp, _vp, _u32, _u32, _int, _vp]),
    "f3d_xfmr_stack_bf16": (_int, [ctypes.POINTER(XfmrBlock), _int, _vp, _vp, _vp, _vp, c_uint64, _u32, _u32, _int, _vp]),
    "f3d_xfmr_stack_scratch": (c_uint64, [_u32, _u32, _u32]),
    "f3d_xfmr_block_fwd_bf16": (_int, [ctypes.POINTER(XfmrBlock), ctypes.POINTER(XfmrSaved), _u32, _u32, _int, _vp]),
    "f3d_xfmr_block_bwd_bf16": (_int, [ctypes.POINTER(XfmrBlock), ctypes.POINTER(XfmrSaved), ctypes.POINTER(XfmrGrads), _vp, _vp, c_uint64, _u32,
                                       _u32, _int, _vp]),
    "f3d_xfmr_block_bwd_scratch": (c_uint64, [_u32, _u32, _u32, _u32]),
    "f3d_linear_swiglu_bwd_bf16": (_int, [_vp, _vp, _vp, _vp, _vp, _int, _int, _int, _int, _vp]),
    "f3d_mlp_swiglu_bwd_bf16": (_int, [_vp, _vp, _vp, _vp, _vp, _vp, _int, _int, _int, _int, _vp]),
    "f3d_layernorm_bwd_add_bf16": (_int, [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _u32, _u32, _f32, _int, _vp]),
    "f3d_gemm_sm_bf16": (_int, [_vp, _vp, _vp, _int, _int, _int, _int, _vp]),
    "f3d_buck_swin_fwd": (_int, [_vp, _vp, _vp, _vp, _vp, _vp, _int, _int, _int, _int, _int, _int, _u32, _int, _vp]),
    "f3d_layernorm_bf16": (_int, [_vp, _vp, _vp, _vp, _u32, _u32, _f32, _int, _int, _vp]),
    "f3d_coord_embed_bf16": (_int, [_vp, _vp, _vp, _vp, _u32, _u32, _int, _vp]),
    "f3d_layernorm_bwd_bf16": (_int, [_vp, _vp, _vp, _vp, _vp, _vp, _u32, _u32, _f32, _int, _vp]),
    "f3d_swiglu_bwd_bf16": (_int, [_vp, _vp, _vp, c_uint64, _u32, _int, _vp]),
    "f3d_colsum_bf16": (_int, [_vp, _vp, c_uint64, _u32, _int, _vp]),
    "f3d_gelu_bwd_bf16": (_int, [_vp, _vp, _vp, c_uint64, _int, _int, _vp]),
    "f3d_coord_embed_bwd": (_int, [_vp, _vp, _vp, _vp, _u32, _u32, _int, _vp]),
    "f3d_linear_wgrad_split_bf16": (_int, [_vp, _vp, _vp, _vp, _int, _int, _int, _int, _int, _vp]),
    "f3d_linear_wgrad_bf16": (_int, [_vp, _vp, _vp, _vp, _int, _int, _int, _int, _vp]),
    "f3d_linear_ksplit_bf16": (_int, [_vp, _vp, _vp, _vp, _vp, _int, _int, _int, _int, _int, _vp]),
    "f3d_collate_points_f32": (_int, [_vp, _vp, _vp, c_uint64, _u32, _int, _vp]),
    "f3d_scatter_index": (_int, [_vp, _vp, _vp, _vp, _vp, _vp, _u32, _u32, _u32, _u32, _int, _vp]),
    "f3d_gather_rows": (_int, [_vp, _vp, _vp, c_uint64, _u32, _u32, _int, _vp]),
    "f3d_buck_swin_bwd": (_int, [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _int, _int, _int, _int, _int, _int,
                                 _u32, _int, _vp]),
}

_lib = None


def load() -> ctypes.CDLL:
    """Load the library once; raise loudly when it has not been built."""
    global _lib
    if _lib is not None:
        return _lib
    if not LIB_PATH.exists():
        raise RuntimeError(
            f"{LIB_PATH} is missing: build it with `python -m flash3dtransformer_b200.build` "
            "(there is no CPU or PyTorch fallback for these operators)")
    lib = ctypes.CDLL(os.fspath(LIB_PATH))
    for name, (res, args) in PROTOTYPES.items():
        fn = getattr(lib, name)          # AttributeError if the symbol is not exported
        fn.restype = res
        fn.argtypes = args
    _lib = lib
    return lib


class _NoHost:
    """Stands in for the host module where it was not built: every call goes through ctypes."""

    @staticmethod
    def _none(*_):
        return None

    linear = swin_fwd = scatter = index = bbox = empties = _none


_host = None


def host():
    """The module of csrc/host: operator calls with their checks in native code.  A function returns the status of the call, or
    None for arguments that it leaves to the checks in Python."""
    global _host
    if _host is None:
        lib = load()
        try:
            loader = importlib.machinery.ExtensionFileLoader("_f3d_host", os.fspath(LIB_PATH.with_name("_f3d_host.so")))
            mod = importlib.util.module_from_spec(importlib.util.spec_from_loader("_f3d_host", loader))
            loader.exec_module(mod)
            mod.bind(*[ctypes.cast(getattr(lib, n), c_void_p).value for n in (
                "f3d_linear_dtype", "f3d_buck_swin_fwd_dtype", "f3d_batch_psh_scatter_pad_hash", "f3d_scatter_index", "f3d_bbox_f16")])
            _host = mod
        except ImportError:                  # not built, or built for another torch
            _host = _NoHost
    return _host


def is_loaded() -> bool:
    return _lib is not None


def last_error() -> str:
    msg = load().f3d_last_error()
    return msg.decode("utf-8", "replace") if msg else ""


def check(status: int, what: str) -> None:
    """Turn a negative status into the RuntimeError the reference's bindings raise (std::runtime_error in
    src/common/runtime.h:36-86 surfaces as RuntimeError through pybind11)."""
    if status != 0:
        raise RuntimeError(f"{what}: {last_error()} (status {status})")
