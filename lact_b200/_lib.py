"""ctypes binding of liblact_b200.so (the C ABI in include/lact_b200.h).

There is no fallback: if the shared library is missing, loading raises and every op fails.
"""
from __future__ import annotations

import ctypes as C
import os
from typing import Optional

import torch

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(PKG_DIR, "liblact_b200.so")
OPS_PATH = os.path.join(PKG_DIR, "liblact_b200_torch.so")

LACT_F32, LACT_BF16 = 0, 1
RENORM_NONE, RENORM_EPS_OUTSIDE, RENORM_EPS_INSIDE = 0, 1, 2


class ScanConfig(C.Structure):
    _fields_ = [(n, C.c_int64) for n in ("B", "L", "D", "H", "out_len")] + [
        (n, C.c_int32) for n in ("act_dtype", "lr_dtype", "mom_dtype", "w_dtype", "use_momentum", "use_muon",
                                 "ns_steps", "ns_const_coeffs", "ns_concat", "ns_gram_right", "renorm", "prenorm",
                                 "prenorm_bf16", "overwrite_quirk")] + [("w_scale", C.c_float)] + [
        (n, C.c_int64) for n in ("q_bs", "q_ts", "k_bs", "k_ts", "v_bs", "v_ts", "o_bs", "o_ts")]


class ScanIO(C.Structure):
    _fields_ = [(n, C.c_void_p) for n in ("w0", "w1", "w2", "q", "k", "v", "lr0", "lr1", "lr2", "momentum", "m0_in",
                                          "m1_in", "m2_in", "o", "w0_out", "w1_out", "w2_out", "m0_out", "m1_out",
                                          "m2_out", "state_dump", "ns_trace", "shadow_dump")]


ERR_CONFIG = -5  # LACT_ERR_CONFIG


class BmmDesc(C.Structure):
    """lact_bmm_desc of the C header."""
    _fields_ = ([(n, C.c_void_p) for n in ("a0", "b0", "a1", "b1", "c")] +
                [(n, C.c_int64) for n in ("a0_ld", "a0_bs", "b0_ld", "b0_bs", "a1_ld", "a1_bs", "b1_ld", "b1_bs",
                                          "c_ld", "c_bs", "batch", "M", "N", "K")] +
                [(n, C.c_int32) for n in ("a0_mn", "b0_mn", "a1_mn", "b1_mn", "c_dtype", "accumulate")])


class NsBwdGroup(C.Structure):
    """lact_ns_bwd_group of the C header."""
    _fields_ = [("du", C.c_void_p), ("g", C.c_void_p), ("dg", C.c_void_p), ("trace", C.c_void_p),
                ("trace_bytes", C.c_size_t), ("partials", C.c_void_p), ("nmat", C.c_int64), ("rows", C.c_int64),
                ("cols", C.c_int64)]


_lib: Optional[C.CDLL] = None


def _declare(lib: C.CDLL) -> None:
    vp, i32, i64, f32 = C.c_void_p, C.c_int32, C.c_int64, C.c_float
    szp = C.POINTER(C.c_size_t)
    lib.lact_version.restype = C.c_int
    lib.lact_error_string.restype = C.c_char_p
    lib.lact_error_string.argtypes = [C.c_int]
    lib.lact_read_status.argtypes = [vp, vp]
    lib.lact_stream_sync_count.restype = C.c_int64
    lib.lact_set_wait_limit_ns.argtypes = [C.c_uint64]
    lib.lact_debug_wait_timeout.argtypes = [vp, vp]
    lib.lact_static_status.argtypes = [vp]
    lib.lact_launch_count.restype = C.c_int64
    lib.lact_profile_enable.argtypes = [C.c_int]
    lib.lact_profile_enable.restype = C.c_int
    lib.lact_profile_num_classes.restype = C.c_int
    lib.lact_profile_class_name.argtypes = [C.c_int]
    lib.lact_profile_class_name.restype = C.c_char_p
    lib.lact_profile_read.argtypes = [C.POINTER(C.c_double), C.POINTER(C.c_int64)]
    lib.lact_profile_read.restype = C.c_int
    lib.lact_scan_workspace_bytes.argtypes = [C.POINTER(ScanConfig), i32, C.POINTER(i32), C.POINTER(i64),
                                              C.POINTER(i64), szp]
    lib.lact_scan_ns_trace_bytes.argtypes = [C.POINTER(ScanConfig), szp, szp]
    lib.lact_scan_ns_trace_bytes.restype = C.c_int
    lib.lact_ns_trace_result_offset.argtypes = [i64, i64, i64, i32, szp]
    lib.lact_ns_trace_result_offset.restype = C.c_int
    lib.lact_scan_fwd.argtypes = [C.POINTER(ScanConfig), C.POINTER(ScanIO), i32, C.POINTER(i32), C.POINTER(i64),
                                  C.POINTER(i64), C.POINTER(i64), vp, C.c_size_t, vp]
    lib.lact_scan_f32_workspace_bytes.argtypes = lib.lact_scan_workspace_bytes.argtypes
    lib.lact_scan_f32_fwd.argtypes = lib.lact_scan_fwd.argtypes
    lib.lact_swiglu_ffn_workspace_bytes.argtypes = [i64, i64, i64, i64, szp]
    lib.lact_swiglu_ffn_fwd.argtypes = [vp, vp, vp, vp, i64, i64, i64, i64, vp, C.c_size_t, vp]
    lib.lact_static_scratch_bytes.restype = C.c_size_t
    lib.lact_swiglu_ffn_fwd_static.argtypes = [vp, vp, vp, vp, i64, i64, i64, i64, vp]
    lib.lact_swiglu_ffn_fwd_static.restype = C.c_int
    lib.lact_fw_grad_workspace_bytes.argtypes = [i64, i64, i64, i64, szp]
    lib.lact_fw_grad.argtypes = [vp, vp, vp, vp, vp, vp, vp, i32, vp, vp, i64, i64, i64, i64, vp, C.c_size_t, vp]
    lib.lact_newton_schulz_workspace_bytes.argtypes = [i64, i64, i64, szp]
    lib.lact_newton_schulz.argtypes = [vp, i32, vp, i64, i64, i64, i32, i32, vp, C.c_size_t, vp]
    lib.lact_l2_norm_add.argtypes = [vp, i32, vp, i32, vp, vp, i32, i64, i64, i64, f32, vp]
    lib.lact_prenorm_momentum_l2norm.argtypes = [vp, vp, vp, vp, vp, vp, vp, vp, i64, i64, i64, f32, vp]
    lib.lact_bmm_bf16.argtypes = [vp, i32, vp, i32, vp, i32, i64, i64, i64, i64, vp, vp]
    lib.lact_bmm2_bf16.argtypes = [vp, i32, vp, i32, vp, i32, vp, i32, vp, i32, i32, i64, i64, i64, i64, vp, vp]
    lib.lact_bmm2_strided_bf16.argtypes = [vp, i32, i64, i64, vp, i32, i64, i64, vp, i32, i64, i64, vp, i32, i64, i64, vp,
                                           i32, i64, i64, i32, i64, i64, i64, i64, vp, vp]
    lib.lact_qkv_prologue.argtypes = [vp, vp, vp, i64, i64, i64, i64, i64, i64, vp, vp, vp, i64, i64, i64, i64, i32, i32, vp]
    lib.lact_qkv_prologue_rope.argtypes = [vp, vp, vp, i64, i64, i64, i64, i64, i64, vp, vp, vp, i64, i64, i64, i64, i32, i32,
                                           vp, vp, i64, i64, i64, vp, vp]
    lib.lact_qkv_prologue_rope.restype = C.c_int
    lib.lact_lr_prologue.argtypes = [vp, i32, i64, f32, vp, i32, i64, vp, vp, vp, vp, i64, i64, i64, vp]
    lib.lact_out_epilogue.argtypes = [vp, vp, vp, i64, vp, i64, vp, i64, i64, i64, i64, i64, f32, vp]
    lib.lact_swiglu_bwd_planes.argtypes = [vp, vp, vp, vp, vp, i32, f32, vp, vp, i64, i64, vp]
    lib.lact_fw_grad_bwd_pointwise.argtypes = [vp] * 7 + [i32, f32] + [vp] * 7 + [i64] * 5 + [i32, vp]
    lib.lact_renorm_bwd.argtypes = [vp, vp, i32, vp, vp, vp, vp, vp, i64, i64, i32, vp]
    lib.lact_ns_norm_bwd.argtypes = [vp, vp, vp, i64, i64, vp]
    lib.lact_momentum_bwd_slices.restype = C.c_int
    lib.lact_qkv_prologue_bwd.argtypes = [vp] * 3 + [i64] * 6 + [vp] * 6 + [i64] * 4 + [i32, i32, vp, vp, i64, i64, i64, vp, vp]
    lib.lact_out_epilogue_bwd_blocks.restype = C.c_int
    lib.lact_out_epilogue_bwd.argtypes = [vp, vp, vp, i64, vp, i64, vp, vp, vp, i64, i64, i64, i64, f32, vp]
    lib.lact_swa_fwd.argtypes = [vp, vp, vp, vp] + [i64] * 14 + [f32, vp, vp, vp, vp]
    lib.lact_swa_fwd_split_bytes.argtypes = [i64] * 6 + [szp, C.POINTER(i64)]
    lib.lact_swa_fwd_split.argtypes = [vp, vp, vp, vp] + [i64] * 14 + [f32, vp, vp, vp, vp, C.c_size_t, vp, vp]
    lib.lact_swa_bwd.argtypes = [vp] * 10 + [i64] * 16 + [f32, vp, vp, vp]
    lib.lact_bmm_group_bf16.argtypes = [C.POINTER(BmmDesc), i32, vp, vp]
    lib.lact_bmm_group_split_bytes.argtypes = [C.POINTER(BmmDesc), i32, szp, C.POINTER(i64)]
    lib.lact_bmm_group_split_bf16.argtypes = [C.POINTER(BmmDesc), i32, vp, vp, C.c_size_t, vp, vp]
    lib.lact_fw_grad_pointwise.argtypes = [vp, vp, vp, i64, i64, vp, i64, i64, vp, vp, vp, i32, i64, f32, vp, vp, i64, i64,
                                           i64, i64, vp, vp]
    lib.lact_ns_trace_bwd_fused.argtypes = [C.POINTER(NsBwdGroup), i32, i32, i32, i32, vp, vp]
    lib.lact_ns_norm_bwd.restype = C.c_int
    lib.lact_momentum_bwd.argtypes = [vp, vp, vp, vp, vp, vp, vp, vp, vp, vp, i64, i64, i64, i32, vp]
    lib.lact_momentum_bwd.restype = C.c_int
    lib.lact_ns_trace_bytes.argtypes = [i64, i64, i64, i32, C.POINTER(C.c_size_t)]
    lib.lact_ns_trace_fwd.argtypes = [vp, i32, vp, i64, i64, i64, i32, i32, i32, vp, C.c_size_t, vp, vp]
    lib.lact_ns_trace_bwd.argtypes = [vp, vp, i64, i64, i64, i32, i32, i32, vp, C.c_size_t, vp, vp]
    lib.lact_sgemm_f32.argtypes = [vp, i32, vp, i32, vp, i32, vp, i64, i64, i64, i64, vp]
    lib.lact_swiglu_planes_f32.argtypes = [vp, vp, vp, vp, vp, i32, f32, vp, vp, i64, i64, vp]
    lib.lact_add_renorm.argtypes = [vp, vp, vp, vp, vp, vp, i64, i64, i64, i32, i32, i32, i32, vp]
    for name in ("lact_read_status", "lact_set_wait_limit_ns", "lact_debug_wait_timeout", "lact_static_status",
                 "lact_scan_workspace_bytes", "lact_scan_fwd", "lact_scan_f32_workspace_bytes", "lact_scan_f32_fwd", "lact_swiglu_ffn_workspace_bytes",
                 "lact_swiglu_ffn_fwd", "lact_fw_grad_workspace_bytes", "lact_fw_grad",
                 "lact_newton_schulz_workspace_bytes", "lact_newton_schulz", "lact_l2_norm_add",
                 "lact_prenorm_momentum_l2norm", "lact_bmm_bf16", "lact_bmm2_bf16", "lact_bmm2_strided_bf16", "lact_swiglu_bwd_planes",
                 "lact_fw_grad_bwd_pointwise", "lact_renorm_bwd", "lact_sgemm_f32", "lact_swiglu_planes_f32",
                 "lact_add_renorm", "lact_qkv_prologue", "lact_lr_prologue", "lact_out_epilogue", "lact_ns_trace_bytes", "lact_ns_trace_fwd", "lact_ns_trace_bwd"):
        getattr(lib, name).restype = C.c_int


def lib() -> C.CDLL:
    """Loads the shared library (once).  Raises if it has not been built."""
    global _lib
    if _lib is None:
        if not os.path.exists(LIB_PATH):
            raise ImportError(f"{LIB_PATH} is missing: build it with `python -m lact_b200.build` "
                              "(there is no fallback implementation)")
        handle = C.CDLL(LIB_PATH)
        _declare(handle)
        _lib = handle
    return _lib


# The registered operators (torch.ops.lact_b200) live in a second library on top of the first.
_ops_loaded = False
_ops_lib: Optional[C.CDLL] = None


def load_ops() -> None:
    """Loads the operator library (once) and registers its shape-only implementations.  Raises if it has not been built."""
    global _ops_loaded, _ops_lib
    if _ops_loaded:
        return
    lib()
    if not os.path.exists(OPS_PATH):
        raise ImportError(f"{OPS_PATH} is missing: build it with `python -m lact_b200.build` "
                          "(there is no fallback implementation)")
    from . import build
    if not build.built_for_this_torch(OPS_PATH):
        raise ImportError(f"{OPS_PATH} was built for another PyTorch than {torch.__version__}: rebuild it with "
                          "`python -m lact_b200.build`")
    torch.ops.load_library(OPS_PATH)
    from . import _fakes
    _fakes.register()
    _ops_lib = C.CDLL(OPS_PATH)
    _ops_lib.lact_torch_take_status.argtypes = [C.c_int]
    _ops_lib.lact_torch_take_status.restype = C.c_int
    _ops_lib.lact_torch_prepare_status.argtypes = [C.c_int]
    _ops_lib.lact_torch_prepare_status.restype = C.c_int
    _ops_lib.lact_torch_set_error_type.argtypes = [C.py_object]
    _ops_lib.lact_torch_set_error_type.restype = None
    _ops_lib.lact_torch_set_error_type(LactError)   # what a device status or a CUDA error is raised as
    _ops_loaded = True


def call(op, *args):
    """One operator call; with LACT_B200_SYNC_CHECK=1 it is waited for and its status checked."""
    out = op(*args)
    if SYNC_CHECK and not torch.compiler.is_compiling() and not torch.cuda.is_current_stream_capturing():
        synchronize_and_check()
    return out


class LactError(RuntimeError):
    pass


def check(rc: int, what: str) -> None:
    if rc == 0:
        return
    msg = lib().lact_error_string(rc).decode()
    if rc in (-1, -2, -3, -5, -6):
        raise ValueError(f"{what}: {msg} (code {rc})")
    raise LactError(f"{what}: {msg} (code {rc})")


def dtype_code(t: torch.Tensor) -> int:
    if t.dtype == torch.float32:
        return LACT_F32
    if t.dtype == torch.bfloat16:
        return LACT_BF16
    raise TypeError(f"unsupported dtype {t.dtype}: expected float32 or bfloat16")


def stream_ptr() -> int:
    return torch.cuda.current_stream().cuda_stream


# LACT_B200_SYNC_CHECK=1 waits for the device and checks its status after every operator call, backwards included, outside
# stream captures (debugging).
SYNC_CHECK = os.environ.get("LACT_B200_SYNC_CHECK", "0") == "1"


def workspace(nbytes: int, device: torch.device) -> torch.Tensor:
    """Scratch for one call on the current stream, from PyTorch's caching allocator (stream-ordered: giving it back right
    after the call has been enqueued is safe)."""
    prepare_status(device)
    return torch.empty(max(nbytes, 1 << 20), dtype=torch.uint8, device=device)


def on_16_bytes(t: torch.Tensor) -> torch.Tensor:
    """`t` (contiguous), copied if it starts off a 16-byte boundary (a view into a packed buffer): kernels read it 16 bytes
    at a time."""
    return t if t.data_ptr() % 16 == 0 else t.clone(memory_format=torch.contiguous_format)


_prepared = set()   # devices whose failures have a place to be reported in


def prepare_status(device: torch.device) -> None:
    """Before a library call that is not a registered operator: its kernels find the word that failures are left in."""
    index = device.index if device.index is not None else torch.cuda.current_device()
    if index not in _prepared:
        load_ops()
        check(_ops_lib.lact_torch_prepare_status(index), "lact_status_host_word")
        _prepared.add(index)


def _take_status(index: int) -> None:
    load_ops()
    st = _ops_lib.lact_torch_take_status(index)
    if st != 0:
        raise LactError("device status: " + lib().lact_error_string(st).decode() + f" (code {st})")


def mark_pending(ws: torch.Tensor) -> None:
    """Called after a library call has been enqueued with `ws` as its workspace.  Kernels that give up leave their status
    in a word of mapped host memory (`lact_status_host_word`): reading it here raises for any EARLIER call that has
    failed by now, without copies, events or waits."""
    if SYNC_CHECK and not torch.cuda.is_current_stream_capturing():
        read_status(ws)
    _take_status(ws.device.index)


def read_status(ws: torch.Tensor) -> None:
    """Synchronises the current stream and raises if the workspace's status word is non-zero."""
    rc = lib().lact_read_status(ws.data_ptr(), stream_ptr())
    if rc != 0:
        raise LactError("device status: " + lib().lact_error_string(rc).decode() + f" (code {rc})")


def synchronize_and_check() -> None:
    """Waits for the work enqueued so far and raises if any call recorded a device-side error (a bounded wait that ran
    out).  The op calls themselves never wait."""
    if not _ops_loaded or not torch.cuda.is_initialized():
        return
    for idx in range(torch.cuda.device_count()):
        if torch.cuda.device_count() > 1 and torch.cuda.memory_reserved(idx) == 0:
            continue
        torch.cuda.synchronize(idx)
        _take_status(idx)


def stream_sync_count() -> int:
    """cudaStreamSynchronize calls made inside the library in this process so far."""
    return int(lib().lact_stream_sync_count())


def nvtx_enable(on: bool = True) -> None:
    """NVTX ranges around every kernel launch of the library (named after the kernel class) on / off."""
    check(lib().lact_nvtx_enable(1 if on else 0), "lact_nvtx_enable")


def launch_count() -> int:
    """Kernels launched by the library in this process so far."""
    return int(lib().lact_launch_count())


def profile_enable(on: bool) -> None:
    lib().lact_profile_enable(int(on))


def profile_read() -> dict:
    """{class name: (total ms, launches)} for launches recorded since the last read."""
    n = lib().lact_profile_num_classes()
    ms = (C.c_double * n)()
    cnt = (C.c_int64 * n)()
    check(lib().lact_profile_read(ms, cnt), "lact_profile_read")
    return {lib().lact_profile_class_name(i).decode(): (ms[i], int(cnt[i])) for i in range(n) if cnt[i]}
