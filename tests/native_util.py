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


def _tensor(backend, handle):
    f = backend.L._ZN5prism10get_tensorEP14prism_cuda_ctxi
    f.restype, f.argtypes = C.c_void_p, [C.c_void_p, C.c_int32]
    return C.c_void_p(f(backend.ctx, handle))


def gemm_tc5(backend, handle, x, y, resid=None):
    """y = x W^T by the tcgen05 GEMM whatever the engine would choose; resid (y itself, say) is added after the rounding of the product."""
    _call(backend, "_ZN5prism15launch_gemm_tc5EP14prism_cuda_ctxRKNS_9LutTensorEPKtjPtS6_", _tensor(backend, handle), C.c_void_p(x.data_ptr()),
          C.c_uint32(x.shape[0]), C.c_void_p(y.data_ptr()), C.c_void_p(resid.data_ptr()) if resid is not None else None)


def gemm_add(backend, handle, x, h):
    """h += x W^T, rounded after the product and after the sum."""
    import torch

    tmp = torch.empty_like(h)
    _call(backend, "_ZN5prism15launch_gemm_addEP14prism_cuda_ctxRKNS_9LutTensorEPKtjPtS7_", _tensor(backend, handle), C.c_void_p(x.data_ptr()),
          C.c_uint32(x.shape[0]), C.c_void_p(h.data_ptr()), C.c_void_p(tmp.data_ptr()))


def gemm_swiglu(backend, gate, up, x, out, fused):
    """out = silu(x Wg^T) * (x Wu^T), rounded after each; by one kernel, or as the engine chooses."""
    import torch

    a = [_tensor(backend, gate), _tensor(backend, up), C.c_void_p(x.data_ptr()), C.c_uint32(x.shape[0]), C.c_void_p(out.data_ptr())]
    if fused:
        return _call(backend, "_ZN5prism17launch_swiglu_tc5EP14prism_cuda_ctxRKNS_9LutTensorES4_PKtjPt", *a)
    u = torch.empty_like(out)
    _call(backend, "_ZN5prism18launch_gemm_swigluEP14prism_cuda_ctxRKNS_9LutTensorES4_PKtjPtS7_", *a, C.c_void_p(u.data_ptr()))


def linear_few_tokens(backend, handle, x, y, resid=None, up=None, norm_eps=-1.0):
    """y = x W^T of 1..32 rows by the register-palette kernel: plain, with a residual, or silu(gate) * up; rows of y may be apart."""
    mode = 2 if up is not None else 0 if resid is None else 1
    _call(backend, "_ZN5prism15launch_gemm_regEP14prism_cuda_ctxNS_8GemvModeERKNS_9LutTensorEPS4_PKtjPtjS8_jf", C.c_int(mode), _tensor(backend, handle),
          _tensor(backend, up) if up is not None else None, C.c_void_p(x.data_ptr()), C.c_uint32(x.stride(0)), C.c_void_p(y.data_ptr()),
          C.c_uint32(y.stride(0)), C.c_void_p(resid.data_ptr()) if resid is not None else None, C.c_uint32(x.shape[0]), C.c_float(norm_eps))


class DenseSeg(C.Structure):  # prism::DenseSeg, dense.cuh
    _fields_ = [("row0", C.c_uint32), ("rows", C.c_uint32), ("inp", C.c_uint32), ("k", C.c_uint32), ("act", C.c_uint32), ("mul", C.c_float), ("bias", C.c_void_p)]


class DenseLinear(C.Structure):
    _fields_ = [("w", C.c_void_p), ("k_pad", C.c_uint32), ("n_tiles", C.c_uint32), ("n_segs", C.c_uint32), ("experts", C.c_uint32), ("seg", DenseSeg * 12)]


class DenseOut(C.Structure):
    _fields_ = [("p", C.c_void_p), ("pitch", C.c_uint32), ("store", C.c_uint32)]


class DenseIn(C.Structure):
    _fields_ = [("x", C.c_void_p), ("pitch", C.c_uint32), ("f32", C.c_uint32), ("norm_w", C.c_void_p), ("n_norm", C.c_uint32), ("eps", C.c_float),
                ("gate", C.c_void_p), ("gate_pitch", C.c_uint32), ("x2", C.c_void_p), ("pitch2", C.c_uint32)]


def dense_layout(w):
    """[rows of whole tiles of 128, k of whole 64s] bf16 in the device layout of a dense weight."""
    rows, k = w.shape
    return w.reshape(rows // 128, 128, k // 8, 8).permute(0, 2, 1, 3).contiguous()


def dense_stream(backend, packed, k_pad, segs, x, outs, x2=None):
    """The streaming linear of few rows.  segs: dicts of DenseSeg fields; outs: (tensor, store) per segment."""
    l = DenseLinear(packed.data_ptr(), k_pad, packed.shape[0], len(segs), 1)
    for i, s in enumerate(segs):
        l.seg[i] = DenseSeg(s["row0"], s["rows"], s.get("inp", 0), s.get("k", 0), s.get("act", 0), s.get("mul", 1.0), s["bias"].data_ptr() if s.get("bias") is not None else None)
    o = (DenseOut * len(outs))(*[DenseOut(t.data_ptr(), t.stride(0), store) for t, store in outs])
    i = DenseIn(x=x.data_ptr(), pitch=x.stride(0), x2=x2.data_ptr() if x2 is not None else None, pitch2=x2.stride(0) if x2 is not None else 0)
    _call(backend, "_ZN5prism19launch_dense_streamEP14prism_cuda_ctxRKNS_11DenseLinearERKNS_7DenseInEPKNS_8DenseOutEj", C.byref(l), C.byref(i), o, C.c_uint32(x.shape[0]))


def few_tokens_taken(backend, handle, x, y):
    """y = x W^T where the register-palette kernel is the engine's choice for it; whether it is."""
    takes = C.c_bool(False)
    _call(backend, "_ZN5prism15gemm_few_tokensEP14prism_cuda_ctxNS_8GemvModeERKNS_9LutTensorEPS4_PKtjPtjS8_jfPb", C.c_int(0), _tensor(backend, handle), None,
          C.c_void_p(x.data_ptr()), C.c_uint32(x.stride(0)), C.c_void_p(y.data_ptr()), C.c_uint32(y.stride(0)), None, C.c_uint32(x.shape[0]), C.c_float(-1.0), C.byref(takes))
    return takes.value
