"""ctypes binding of `libcagnet_b200.so` (the C ABI declared in include/cagnet_b200.h).

There is no fallback: if the library has not been built, or a call fails, this raises.
"""
import ctypes
import os

_HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(_HERE, "libcagnet_b200.so")

_vp, _i32, _i64, _f32, _f64, _sz, _cp = (ctypes.c_void_p, ctypes.c_int32, ctypes.c_int64, ctypes.c_float,
                                         ctypes.c_double, ctypes.c_size_t, ctypes.c_char_p)

# name -> (restype, argtypes); mirrors include/cagnet_b200.h one to one
PROTOTYPES = {
    "cagnet_version": (_i32, []),
    "cagnet_last_error_string": (_cp, []),
    "cagnet_set_param": (_i32, [_cp, _i32]),
    "cagnet_get_param": (_i32, [_cp]),
    "cagnet_coo2csr_i32": (_i32, [_vp, _i64, _i32, _vp, _vp]),
    "cagnet_check_csr_i32": (_i32, [_vp, _vp, _vp, _i32, _i32, _i64, _vp, _vp]),
    "cagnet_spmm_plan_bytes": (_sz, [_i32, _i64]),
    "cagnet_spmm_plan_i32": (_i32, [_vp, _i32, _i64, _vp, _sz, _vp]),
    "cagnet_spmm_csr_f32": (_i32, [_vp, _vp, _vp, _i32, _i32, _i64, _vp, _i64, _vp, _i64, _i32, _f32, _vp, _vp]),
    "cagnet_spmm_noalloc_max_nnz": (_i64, []),
    "cagnet_spmm_csr_f32_noalloc": (_i32, [_vp, _vp, _vp, _i32, _i32, _i64, _vp, _i64, _vp, _i64, _i32, _f32, _vp]),
    "cagnet_spmm_split_plan_bytes": (_sz, [_i64]),
    "cagnet_spmm_split_plan_i32": (_i32, [_vp, _vp, _vp, _vp, _i32, _i64, _vp, _sz, _vp]),
    "cagnet_spmm_block_workspace_bytes": (_sz, [_vp, _vp, _i64, _i32]),
    "cagnet_spmm_block_launches": (_i32, [_vp, _i64, _i32]),
    "cagnet_spmm_block_f32": (_i32, [_vp, _vp, _i64, _vp, _i64, _i32, _f32, _vp, _sz, _vp]),
    "cagnet_check_coo_i32": (_i32, [_vp, _vp, _i32, _i32, _i64, _vp, _vp]),
    "cagnet_spmm_coo_workspace_bytes": (_sz, [_i32, _i64, _vp, _i64, _i32]),
    "cagnet_spmm_coo_f32": (_i32, [_vp, _vp, _vp, _i32, _i32, _i64, _vp, _i64, _vp, _i64, _i32, _vp, _vp, _sz, _vp]),
    "cagnet_tile_count_i32": (_i32, [_vp, _vp, _i32, _vp, _vp, _i32, _i32, _vp, _vp]),
    "cagnet_tile_fill_i32": (_i32, [_vp, _vp, _vp, _i32, _vp, _vp, _i32, _i32, _vp, _vp, _vp, _vp, _vp, _vp]),
    "cagnet_tile_core_workspace_bytes": (_sz, [_i32, _i32, _i32]),
    "cagnet_tile_core_f32": (_i32, [_vp, _vp, _vp, _vp, _i32, _i32, _vp, _i32, _vp, _i32, _vp, _vp, _vp, _vp, _i64, _vp,
                                    _i64, _i32, _vp, _sz, _vp]),
    "cagnet_tile_core_error": (_i32, []),
    "cagnet_core_gemm_workspace_bytes": (_sz, [_i32, _i32, _i32]),
    "cagnet_core_gemm_f32": (_i32, [_vp, _i64, _vp, _i32, _vp, _i32, _vp, _i64, _vp, _i64, _i32, _vp, _sz, _vp]),
    "cagnet_core_gemm_tc_available": (_i32, []),
    "cagnet_core_gemm_tc_workspace_bytes": (_sz, [_i32, _i32, _i32]),
    "cagnet_split_tf32_f32": (_i32, [_vp, _i64, _vp, _vp, _vp]),
    "cagnet_gather_split_rows_f32": (_i32, [_vp, _i64, _vp, _i32, _i32, _vp, _i64, _vp]),
    "cagnet_core_gemm_tc_f32": (_i32, [_vp, _vp, _i64, _i32, _i32, _vp, _i64, _vp, _i32, _vp, _sz, _vp]),
    "cagnet_add_rows3_f32": (_i32, [_vp, _i64, _vp, _i32, _i32, _vp, _i64, _vp]),
    "cagnet_core_gemm_int_available": (_i32, []),
    "cagnet_core_gemm_int_workspace_bytes": (_sz, [_i32, _i32, _i32]),
    "cagnet_gather_scale_split3_bf16": (_i32, [_vp, _i64, _vp, _vp, _i32, _i32, _vp, _i64, _vp]),
    "cagnet_core_gemm_int_bf16": (_i32, [_vp, _i64, _i32, _i32, _vp, _i64, _vp, _i32, _vp, _sz, _vp]),
    "cagnet_add_rows_scaled3_f32": (_i32, [_vp, _i64, _vp, _vp, _i32, _i32, _vp, _i64, _vp]),
    "cagnet_gemm_nn_f32": (_i32, [_vp, _i64, _vp, _i64, _i32, _vp, _i64, _i64, _i32, _i32, _i32, _vp, _i64, _vp]),
    "cagnet_gemm_tn_workspace_bytes": (_sz, [_i64, _i32, _i32]),
    "cagnet_gemm_tn_f32": (_i32, [_vp, _i64, _vp, _i64, _vp, _i64, _i64, _i32, _i32, _f32, _vp, _sz, _vp]),
    "cagnet_row_reduce_f32": (_i32, [_vp, _i64, _i64, _i32, _i32, _vp, _vp, _vp]),
    "cagnet_log_softmax_apply_f32": (_i32, [_vp, _i64, _vp, _vp, _vp, _i64, _i64, _i32, _vp]),
    "cagnet_log_softmax_bwd_apply_f32": (_i32, [_vp, _i64, _vp, _i64, _vp, _vp, _i64, _i64, _i32, _vp]),
    "cagnet_relu_fwd_f32": (_i32, [_vp, _i64, _vp, _i64, _i64, _i32, _vp]),
    "cagnet_relu_bwd_f32": (_i32, [_vp, _i64, _vp, _i64, _vp, _i64, _i64, _i32, _vp]),
    "cagnet_log_softmax_fwd_f32": (_i32, [_vp, _i64, _vp, _i64, _i64, _i32, _vp]),
    "cagnet_log_softmax_bwd_f32": (_i32, [_vp, _i64, _vp, _i64, _vp, _i64, _i64, _i32, _vp]),
    "cagnet_nll_workspace_bytes": (_sz, [_i64]),
    "cagnet_nll_masked_f32": (_i32, [_vp, _i64, _vp, _vp, _i64, _i32, _i32, _i32, _f32, _f32, _vp, _vp, _i64, _vp,
                                     _sz, _vp]),
    "cagnet_nll_softmax_bwd_f32": (_i32, [_vp, _i64, _vp, _vp, _i64, _i32, _i32, _i32, _f32, _vp, _i64,
                                          ctypes.POINTER(_i32), _vp, _sz, _vp]),
    "cagnet_gemm_tn_partials2_f32": (_i32, [_vp, _vp, _i64, ctypes.POINTER(_i32), _vp]),
    "cagnet_gemm_tn_partials_f32": (_i32, [_vp, _i64, _vp, _i64, _i64, _i32, _i32, _vp, _sz, _vp, _vp]),
    "cagnet_log_softmax_nll_f32": (_i32, [_vp, _i64, _i64, _i32, _vp, _vp, _i32, _i32, _f32, _vp, _i64, _vp, _i64,
                                          ctypes.POINTER(_i32), _vp, _sz, _vp]),
    "cagnet_gemm_nll_f32": (_i32, [_vp, _i64, _vp, _i64, _i64, _i32, _i32, _vp, _vp, _i32, _i32, _f32, _vp, _i64, _vp, _i64,
                                   ctypes.POINTER(_i32), ctypes.POINTER(_i32), _vp, _sz, _vp]),
    "cagnet_epoch_tail_f32": (_i32, [_vp] * 10 + [_f64, _f64, _f64, _f64, _i64, _vp, _i32, _f32, _vp, _vp]),
}



class TnSum(ctypes.Structure):
    """`cagnet_tn_sum` of include/cagnet_b200.h, field for field."""
    _fields_ = [("partials", _vp), ("chunks", _i32), ("K", _i32), ("N", _i32), ("transposed", _i32)]


class Block(ctypes.Structure):
    """`cagnet_block` of include/cagnet_b200.h, field for field."""
    _fields_ = ([("n", _i32), ("m", _i32), ("nnz", _i64), ("rowptr", _vp), ("col", _vp), ("val", _vp), ("plan", _vp),
                 ("hub_rows", _i32), ("max_row", _i32), ("split", _vp), ("rows", _vp), ("empty", _vp), ("nrows", _i32),
                 ("nempty", _i32), ("tiles", _i32), ("panels", _i32), ("ctas", _i32), ("joins", _i32), ("tile_kbs", _i32),
                 ("reserved", _i32), ("tile_nnz", _i64), ("tile_work", _i64)] +
                [(name, _vp) for name in ("tile_bits", "tile_kb", "panel_ptr", "cta_ptr", "join_list", "tile_cols",
                                          "panel_rows", "panel_scale", "col_scale", "rest")])


_lib = None


def lib():
    """The loaded library; raises RuntimeError with build instructions if it is missing."""
    global _lib
    if _lib is None:
        if not os.path.exists(LIB_PATH):
            raise RuntimeError(
                "cagnet_b200: native library %s is missing; build it with `python -m cagnet_b200.build` "
                "(there is no CPU or PyTorch fallback)" % LIB_PATH)
        handle = ctypes.CDLL(LIB_PATH)
        for name, (res, args) in PROTOTYPES.items():
            fn = getattr(handle, name)
            fn.restype, fn.argtypes = res, args
        _lib = handle
    return _lib


_host = None


def host():
    """The native host path (csrc/host.cpp), a Python extension beside the library."""
    global _host
    if _host is None:
        lib()
        try:
            import torch  # noqa: F401  (its libraries are what the extension links against)
            from . import _host as module
        except ImportError as e:
            raise RuntimeError("cagnet_b200: native host module is missing or does not load (%s); build it with "
                               "`python -m cagnet_b200.build`" % e) from e
        _host = module
    return _host


def check(status, what=""):
    if status != 0:
        msg = lib().cagnet_last_error_string()
        raise RuntimeError("cagnet_b200 %s failed with status %d: %s" % (what, status, msg.decode() if msg else "?"))


def set_param(name, value):
    check(lib().cagnet_set_param(name.encode(), int(value)), "set_param")


def get_param(name):
    return lib().cagnet_get_param(name.encode())
