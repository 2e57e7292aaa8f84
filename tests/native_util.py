"""The kernels that have no entry point of their own, called through the symbols of the built library on torch buffers."""
import ctypes as C


class PrefillAttn(C.Structure):  # prism::PrefillAttn, common.cuh
    _fields_ = [("qkv", C.c_void_p), ("stride", C.c_uint32), ("kc", C.c_void_p), ("vc", C.c_void_p), ("cache_rows", C.c_uint64), ("out", C.c_void_p),
                ("nh", C.c_uint32), ("nkv", C.c_uint32), ("hd", C.c_uint32), ("T", C.c_uint32), ("n_seq", C.c_uint32), ("pos0", C.c_uint32),
                ("seq0", C.c_uint32), ("seq_rows", C.c_uint32), ("max_seq", C.c_uint32), ("rope_k", C.c_uint32), ("rope_base", C.c_float),
                ("page_tbl", C.c_void_p), ("page_shift", C.c_uint32), ("tbl_stride", C.c_uint32)]


def _call(backend, symbol, *args):
    import torch

    torch.cuda.synchronize()
    f = getattr(backend.L, symbol)
    f.restype = C.c_int
    backend._ck(f(backend.ctx, *args))
    backend.synchronize()


def prompt_attention(backend, qkv, kc, vc, nh, nkv, hd, T, pos0=0, n_seq=1, rope_k=1, rope_base=1e4, page_tbl=None, page=0):
    """qkv [n_seq * T, (nh + 2 nkv) hd] fp16 (q is rotated in place), kc / vc: [rows, nkv hd] fp16 caches of equal sequences, or
    of pages.  Returns [n_seq * T, nh hd]."""
    import torch

    out = torch.empty(n_seq * T, nh * hd, dtype=torch.float16, device="cuda")
    rows = kc.shape[0] // n_seq if page_tbl is None else page_tbl.shape[1] * page
    a = PrefillAttn(qkv.data_ptr(), qkv.shape[1], kc.data_ptr(), vc.data_ptr(), kc.shape[0], out.data_ptr(), nh, nkv, hd, T, n_seq, pos0, 0, rows, rows,
                    rope_k, rope_base, 0 if page_tbl is None else page_tbl.data_ptr(), page.bit_length() - 1 if page else 0,
                    0 if page_tbl is None else page_tbl.shape[1])
    _call(backend, "_ZN5prism19launch_prefill_attnEP14prism_cuda_ctxRKNS_11PrefillAttnE", C.byref(a))
    return out
