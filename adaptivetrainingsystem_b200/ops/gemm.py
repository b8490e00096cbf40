"""bf16 GEMMs on the tcgen05 kernel (``csrc/gemm_tcgen05.cu``) and their PyTorch definitions.

Naming: ``nt`` = A[M,K] · B[N,K]ᵀ, ``nn`` = A[M,K] · B[K,N], ``tn`` = A[K,M]ᵀ · B[K,N]; all row-major.
These are the three products of a linear layer (forward, input gradient, weight gradient); none needs a
transposed copy because the kernel reads either operand K-major or MN-major.

Grouped forms work on the expert capacity layout ``[E, C, *]`` with a device-side ``counts[E]`` (rows of
group ``e`` actually used; pad rows up to the next multiple of 128 must be zero).
"""
from __future__ import annotations

import contextlib
import ctypes
import os
from typing import Optional

import torch

from . import _lib

EPI_STORE, EPI_ADDC, EPI_F32, EPI_SWIGLU, EPI_SWIGLU_BWD = 0, 1, 2, 3, 4

_c_int, _c_ll, _c_f, _vp = ctypes.c_int, ctypes.c_longlong, ctypes.c_float, ctypes.c_void_p
_configured = False


class _Skinny(ctypes.Structure):   # csrc/skinny.cuh
    _fields_ = [("T", _c_int), ("N", _c_int), ("K", _c_int), ("mode", _c_int), ("up_offset", _c_int), ("act_cols", _c_int), ("head_dim", _c_int), ("alpha", _c_f), ("a1", _c_f), ("a2", _c_f),
                ("ldx", _c_int), ("out", _vp), ("ldo", _c_ll), ("add", _vp), ("ldadd", _c_ll), ("bias", _vp), ("x", _vp), ("w1", _vp), ("b1", _vp), ("w2", _vp),
                ("b2", _vp), ("pos", _vp), ("next_w", _vp), ("next_out", _vp), ("next_parts", _vp), ("scale_parts", _vp), ("scale_n", _c_int), ("scale_inv", _c_f),
                ("scale_eps", _c_f), ("status", _vp), ("w_ready", _c_int)]


class StreamStep(ctypes.Structure):   # csrc/stream_step.cuh
    _fields_ = [("scale_parts", _vp), ("scale_n", _c_int), ("scale_inv", _c_f), ("scale_eps", _c_f), ("next_w", _vp), ("next_out", _vp), ("next_parts", _vp),
                ("pos", _vp), ("cos_t", _vp), ("sin_t", _vp), ("act_cols", _c_int), ("head_dim", _c_int)]


def stream_step(K: int, scale=None, next_norm=None, rope=None) -> Optional[StreamStep]:
    """``scale`` = (sums of squares [M, n], eps), ``next_norm`` = (weight, rows [M, N], sums of squares [M, N / 16]), ``rope`` = (cos, sin, positions [M]
    int32, rotated columns, head width) of a streaming product with ``K`` terms; the tensors outlive the launch's call."""
    if scale is None and next_norm is None and rope is None:
        return None
    step = StreamStep()
    if scale is not None:
        step.scale_parts, step.scale_n, step.scale_inv, step.scale_eps = scale[0].data_ptr(), scale[0].shape[1], 1.0 / K, scale[1]
    if next_norm is not None:
        step.next_w, step.next_out, step.next_parts = (t.data_ptr() for t in next_norm)
    if rope is not None:
        step.cos_t, step.sin_t, step.pos = (t.data_ptr() for t in rope[:3])
        step.act_cols, step.head_dim = rope[3:]
    return step


def _fn():
    global _configured
    lib = _lib.cuda_lib()
    if not _configured:
        lib.ats_gemm_bf16.restype = _c_int
        lib.ats_gemm_bf16.argtypes = [
            _vp, _c_ll, _c_ll, _c_ll, _c_int,  # A
            _vp, _c_ll, _c_ll, _c_ll, _c_int,  # B
            _vp, _c_int, _vp, _c_int, _vp, _c_int,  # D, C, aux
            _c_int, _c_int, _c_int, _c_f, _c_int, _c_int, _c_int,  # M N K alpha beta epilogue up_offset
            _c_int, _c_int, _vp,  # groups ragged counts
            _c_int, _c_int, _c_int, _c_int,  # group coordinate shifts
            _c_ll, _c_ll, _c_ll,  # d_gs c_gs aux_gs
            _c_int, _c_int, _c_int, _vp, _c_int, _c_int,  # b_div k_segs seg_stride d_table k_split scatter_rows
            _vp, _c_int, _vp]  # status, max_ctas, stream
        lib.ats_splitk_reduce.restype = _c_int
        lib.ats_splitk_reduce.argtypes = [_vp, _c_int, _c_ll, _c_ll, _vp, _vp, _vp]
        lib.ats_gemm_skinny.restype = _c_int
        lib.ats_gemm_skinny.argtypes = [_vp, _c_ll, _vp, _c_ll, _c_ll, ctypes.POINTER(_Skinny), _c_int, _vp]
        lib.ats_chain_launches.restype = None
        lib.ats_chain_launches.argtypes = [_c_int]
        lib.ats_gemm_set_pair.restype = None
        lib.ats_gemm_set_pair.argtypes = [_c_int]
        if os.environ.get("ATS_GEMM_PAIR") is not None:
            lib.ats_gemm_set_pair(int(os.environ["ATS_GEMM_PAIR"]))
        lib.ats_gemm_set_wide_stores.restype = None
        lib.ats_gemm_set_wide_stores.argtypes = [_c_int]
        if os.environ.get("ATS_GEMM_WIDE_STORES") is not None:
            lib.ats_gemm_set_wide_stores(int(os.environ["ATS_GEMM_WIDE_STORES"]))
        _configured = True
    return lib.ats_gemm_bf16


def set_pair_kernels(on: bool) -> None:
    """Products with at least 256 rows run on pairs of CTAs (``tcgen05.mma.cta_group::2``, the default) or on single CTAs."""
    _fn()
    _lib.cuda_lib().ats_gemm_set_pair(int(bool(on)))


def _raw(a, a_rows, a_cols, lda, a_mn, b, b_rows, b_cols, ldb, b_mn, d, ldd, c, ldc, aux, ldaux,
         M, N, K, alpha=1.0, beta=0, epilogue=EPI_STORE, up_offset=0, groups=1, ragged=0, counts=None,
         a_gs_mn=0, a_gs_k=0, b_gs_mn=0, b_gs_k=0, d_gs=0, c_gs=0, aux_gs=0, max_ctas=0,
         b_div=1, k_segs=1, seg_stride=0, d_table=None, k_split=1, scatter_rows=0):
    dev = a.device
    # (addresses as integers: the function's argument types are declared, and a c_void_p per tensor is a third of the call's host time)
    err = _fn()(a.data_ptr(), a_rows, a_cols, lda, a_mn, b.data_ptr(), b_rows, b_cols, ldb, b_mn,
                None if d is None else d.data_ptr(), ldd, None if c is None else c.data_ptr(), ldc, None if aux is None else aux.data_ptr(), ldaux,
                M, N, K, alpha, beta, epilogue, up_offset, groups, ragged, None if counts is None else counts.data_ptr(),
                a_gs_mn, a_gs_k, b_gs_mn, b_gs_k, d_gs, c_gs, aux_gs,
                b_div, k_segs, seg_stride, None if d_table is None else d_table.data_ptr(), k_split, scatter_rows,
                _lib.status_tensor(dev).data_ptr(), max_ctas, _lib.stream_ptr(dev))
    _lib.check(err, "ats_gemm_bf16")


def _check2d(t: torch.Tensor) -> torch.Tensor:
    if t.dim() != 2:
        raise ValueError("expected a 2-D tensor")
    if t.stride(1) != 1 or (t.stride(0) % 8) or (t.data_ptr() % 16):
        t = t.contiguous()
    return t


# Skinny products (a decode step: M = batch rows, few 256-column output tiles) would occupy N / 256 of the 148 SMs and stream
# the weight at a fraction of HBM bandwidth; their reduction dimension is split over the SMs instead: bf16 products by a kernel of their own
# (``csrc/gemm_skinny.cu``), 8-bit ones over groups of the grouped kernel, every group writing an fp32 partial product that a small
# reduction folds.  ATS_SPLIT_K=0 switches it off.
SPLIT_K_SKINNY = os.environ.get("ATS_SPLIT_K", "1") == "1"


def _skinny_splits(M: int, N: int, K: int) -> int:
    if M > 128 or K < 2048:
        return 1
    tiles = (N + 255) // 256
    s = 1
    while s * 2 * tiles <= 160 and K % (s * 2 * 64) == 0 and K // (s * 2) >= 512 and s < 16:
        s *= 2
    return s


def _gemm_nt_split_k(a, b, out, add, alpha, splits):
    M, K = a.shape
    N = b.shape[0]
    kp = K // splits
    part = torch.empty(splits, M, N, dtype=torch.float32, device=a.device)
    _raw(a, M, K, a.stride(0), 0, b, N, K, b.stride(0), 0, part, N, None, 0, None, 0, M, N, kp, alpha=alpha, beta=0,
         epilogue=EPI_F32, groups=splits, a_gs_k=kp, b_gs_k=kp, d_gs=M * N)
    if out is None:
        out = torch.empty(M, N, dtype=a.dtype, device=a.device)
    if out.is_contiguous() and (add is None or add.is_contiguous()):
        _fold_partials(part, splits, M * N, 1, out, add)  # one launch: sum of the slices (+ residual) -> bf16
        return out
    res = part.sum(0)
    if add is not None:
        res += add
    out.copy_(res)
    return out


@contextlib.contextmanager
def chained_launches(on: bool = True):
    """Kernels launched inside (by this thread) may start while the kernel before them still runs, and the decode products fetch their first
    weights, the decode attention its first cached keys, then.  For a decode step: no kernel launched inside may write a parameter, a packed
    4-bit copy of one, a length, or a cached row below its sequence's length (the row at the length is the step's own).  A product whose weight
    is the result of a kernel (:func:`_weight_ready`) waits for it."""
    if not on or not torch.cuda.is_available():
        yield
        return
    _fn()
    lib = _lib.cuda_lib()
    lib.ats_chain_launches(1)   # counted per thread
    try:
        yield
    finally:
        lib.ats_chain_launches(0)


def _weight_ready(w: torch.Tensor) -> bool:
    """Whether ``w`` certainly holds its values before a chained step begins: a parameter itself, not a view or a copy of one, nor a matrix that
    a kernel writes (a dequantised weight, a gathered shard)."""
    return isinstance(w, torch.nn.Parameter) and getattr(w, "_ats_z3", None) is None


SK_PART, SK_STORE, SK_F32, SK_SWIGLU, SK_SILU, SK_GELU, SK_DYT, SK_ROPE = range(8)


def skinny_ok(a: torch.Tensor, w: torch.Tensor, n: Optional[int] = None) -> bool:
    """Whether ``a`` [T, K] @ ``w`` [N, K]^T runs on the decode kernel (``csrc/gemm_skinny.cu``), where the product is a stream of the weight; ``n``:
    the outputs of a gate / up pair.  The lines are where the general kernel with its fold becomes the faster one (us, decode kernel / general):

    * up to 32 rows hardly ever (2048 x 2048, one row 6.6 / 14.3; 32000 x 2048, 16 rows 24 / 32; 128256 x 384, 32 rows 30.4 / 27.4);
    * up to 64 rows with very many outputs, where a CTA walks its whole tile alone: 32000 x 2048 27.6 / 29.0, 128256 x 1024 61 / 54; pairs: 64 rows
      8192 x 2048 19.4 / 22.0, 11008 x 2048 25.3 / 24.1; 48 rows 14336 x 2048 26.7 / 27.0, 28672 x 2048 51 / 47; and with pairs over short
      reductions, whose epilogue is the longer part: 64 rows 256 x 256 9.0 / 8.5, 256 x 512 8.1 / 9.7; 48 rows 14336 x 136 12.7 / 10.9;
    * up to 128 rows, where one CTA fills an SM and four slices are the most, with many outputs (8192 x 2048, 128 rows 19.9 / 19.7), one or two
      tiles or a reduction long for their number (1024 x 8192 20.6 / 19.1, 2048 x 4096 16.4 / 17.4), and short reductions (2048 x 512
      13.6 / 10.3, 2048 x 1024 11.4 / 12.8; pairs 2816 x 512 12.1 / 10.5, 2816 x 1024 13.4 / 14.4)."""
    T, K, N = a.shape[0], a.shape[-1], w.shape[0] if n is None else n
    if not (SPLIT_K_SKINNY and a.dim() == 2 and 1 <= T <= 128 and K % 8 == 0 and N % 8 == 0):
        return False
    if T <= 32:
        return T <= 16 or N <= 65536 or K >= 768
    if T <= 64:
        if n is None:
            return N <= 32768
        return N <= (14336 if T <= 48 else 8192) and (K >= 512 or (T <= 48 and 128 <= N <= 8192))
    if N > 4096:
        return False
    if n is None:
        return N >= 128 and K <= max(4096, 4 * N) and (K >= 1024 or T <= 80)
    return K >= 1024 or (K >= 512 and T <= 80)


def skinny_fits(T: int, N: int, K: int) -> bool:
    """The same for a product whose decode kernel also saves a launch (a rotation, a norm) and fetches its first weights early: a captured step of
    four 4096-wide layers with 28672 inner columns and 64 rows takes 792 us, with the lines of :func:`skinny_ok` for the pairs 844.  Beyond 64 rows
    the reduction must not be long for the outputs (1024-wide layers with 28672 inner columns, 96 rows: 416 us, 476 without that)."""
    return SPLIT_K_SKINNY and K % 8 == 0 and N % 8 == 0 and (1 <= T <= 64 or (T <= 128 and N <= 4096 and K <= max(4096, 4 * N)))


def skinny_splits(T: int, N: int, K: int, width: int = 128) -> int:
    """Reduction slices of a decode product: as many as there are CTA slots (two per SM; one beyond 64 rows, whose rings are larger), but no
    slice below four 64-element blocks, where start-up and the sum of the slices cost more than the further SMs bring, and at most eight (a
    cluster; four beyond 64 rows, where clusters of eight whole SMs leave the rest of a processing cluster idle).  Clusters of three and more
    do not find all slots: 88 x 3 and 64 x 4 CTAs run at once, 96 x 3 and 74 x 4 in two waves (64 rows, us with two / three / four slices:
    11264 x 1536 15.5 / 14.2 / 20.1, 12288 x 1536 15.8 / 21.4 / 20.5, 8192 x 1536 14.2 / 13.2 / 12.2, 9472 x 1536 14.4 / 13.5 / 19.3)."""
    tiles, slots, most = (N + width - 1) // width, 296 if T <= 64 else 148, 8 if T <= 64 else 4
    s = max(1, min(most, slots // tiles, (K + 63) // 64 // 4))
    if s > 2:
        s = max(2, min(s, slots * 264 // 296 // tiles))
    return s if s <= 4 else 4 if s < 8 else 8


_STREAM_MODES = (SK_STORE, SK_SWIGLU, SK_ROPE)


def stream_fits(T: int, N: int, K: int, mode: int = SK_STORE, head_dim: int = 0) -> bool:
    """Whether a decode product runs on the streaming kernel (``csrc/gemv_bf16.cu``); ``N``: the outputs.  The lines are where a CTA per tile no longer
    has an SM to itself, or its warps walk a long reduction alone where the decode kernel cuts it over clusters (us in a chain of launches, decode
    kernel / streaming kernel; one to eight rows, then sixteen):

    * up to 148 tiles of 16 outputs: 2048 x 2048 4.5 / 2.9, 5.0 / 3.8; 2048 x 5632 8.0 / 5.9, 8.3 / 7.3; 2368 x 14336 15.5 / 13.3, 15.9 / 15.2, but
      with sixteen rows 1024 x 14336 12.1 / 12.8; more tiles: 3072 x 5632 9.0 / 10.0, 9.4 / 12.8;
    * up to 148 pairs of tiles of rotated heads: 2560 x 2048 5.2 / 3.7, 5.6 / 4.6; 4608 x 4096 11.0 / 8.7, 12.0 / 9.4; more: 6144 x 2048 7.6 / 8.1;
    * up to 296 pairs of gate and up tiles, whose CTAs have half the warps: 2816 x 1024 4.8 / 3.3, 5.1 / 4.1; 4736 x 2048 9.3 / 7.5, 9.7 / 9.0; longer
      reductions: 2048 x 4096 8.7 / 9.3, 9.0 / 11.0; more: 5632 x 2048 9.4 / 10.0."""
    if not (SPLIT_K_SKINNY and 1 <= T <= 16 and N % 16 == 0 and K % 64 == 0 and mode in _STREAM_MODES):
        return False
    if mode == SK_ROPE:
        return head_dim >= 32 and head_dim % 32 == 0 and N % head_dim == 0 and N <= 148 * 32 and K <= 4096
    if mode == SK_SWIGLU:
        return N <= 296 * 16 and K <= 2048
    return N <= 148 * 16 and K <= (14336 if T <= 8 else 8192)


def norm_parts(T: int, N: int, K: int) -> int:
    """Sums of squares that :func:`skinny` leaves for each row of a ``SK_STORE`` product with an RMSNorm behind it."""
    return N // 16 if stream_fits(T, N, K) else (N + 127) // 128


def skinny(a: torch.Tensor, w: torch.Tensor, out: torch.Tensor, mode: int, n: Optional[int] = None, splits: Optional[int] = None, add: Optional[torch.Tensor] = None,
           alpha: float = 1.0, up_offset: int = 0, act_cols: int = 0, bias: Optional[torch.Tensor] = None, x: Optional[torch.Tensor] = None, chain=None,
           head_dim: int = 0, pos: Optional[torch.Tensor] = None, next_norm=None, scale=None) -> None:
    """One launch of the decode kernel or, by the lines of :func:`stream_fits`, of the streaming one; ``chain`` = (w1, b1, a1, w2, b2, a2) of the residual step ``SK_DYT``; for ``SK_ROPE``
    w1 and w2 are the cosine and sine tables, ``pos`` the positions (int32) and ``act_cols`` the rotated columns.  ``next_norm`` = (weight, rows
    [T, N], sums of squares [T, norm_parts]) of an RMSNorm that follows ``SK_STORE``; ``scale`` = (sums of squares, eps): ``a`` came from such a product."""
    _fn()
    a, w = _check2d(a), _check2d(w)
    (T, K), N = a.shape, w.shape[0] if n is None else n
    if splits is None:
        stream = (alpha == 1.0 and stream_fits(T, N, K, mode, head_dim) and (mode != SK_SWIGLU or (add is None and up_offset == N and w.shape[0] == 2 * N))
                  and (next_norm is None or next_norm[2].shape[1] == N // 16) and (mode != SK_ROPE or (add is None and act_cols % head_dim == 0)))
        splits = 0 if stream else skinny_splits(T, N, K, 64 if mode == SK_SWIGLU else 128)
    w1, b1, a1, w2, b2, a2 = chain if chain is not None else (None, None, 0.0, None, None, 0.0)

    def at(t):
        return None if t is None else t.data_ptr()
    args = _Skinny(T, N, K, mode, up_offset, act_cols, head_dim, alpha, a1, a2, 0 if x is None else x.stride(0), at(out), out.stride(-2), at(add), 0 if add is None else add.stride(0),
                   at(bias), at(x), at(w1), at(b1), at(w2), at(b2), at(pos), *(map(at, next_norm) if next_norm is not None else (None,) * 3),
                   *((at(scale[0]), scale[0].shape[1], 1.0 / K, scale[1]) if scale is not None else (None, 0, 0.0, 0.0)), at(_lib.status_tensor(a.device)), int(_weight_ready(w)))
    _lib.check(_lib.cuda_lib().ats_gemm_skinny(a.data_ptr(), a.stride(0), w.data_ptr(), w.stride(0), w.shape[0], ctypes.byref(args), splits, _lib.stream_ptr(a.device)),
               "ats_gemm_skinny")


def skinny_partials(a: torch.Tensor, w: torch.Tensor) -> torch.Tensor:
    """-> the slices [splits, T, N] in fp32, for a fold that works on whole rows."""
    T, K = a.shape
    splits = skinny_splits(T, w.shape[0], K)
    part = torch.empty(splits, T, w.shape[0], dtype=torch.float32, device=a.device)
    skinny(a, w, part, SK_PART, splits=splits)
    return part


def _fold_partials(part: torch.Tensor, splits: int, n_inner: int, n_outer: int, out: torch.Tensor, add: Optional[torch.Tensor] = None) -> None:
    """out[o, :] = sum over the ``splits`` fp32 partial blocks of problem ``o`` (+ add), written as bf16."""
    _fn()
    _lib.check(_lib.cuda_lib().ats_splitk_reduce(_lib.ptr(part), splits, n_inner, n_outer, _lib.ptr(out), _lib.ptr(add),
                                                 _lib.stream_ptr(part.device)), "splitk_reduce")


def _addressable(t: Optional[torch.Tensor], M: int, N: int, dtype) -> bool:
    """Whether the epilogues can read or write ``t`` in place: [M, N] of their type, adjacent columns, 16-byte aligned rows."""
    return (t is None or (t.dtype == dtype and t.shape == (M, N) and t.stride(1) == 1 and t.stride(0) % 8 == 0 and t.data_ptr() % 16 == 0))


def gemm_nt(a: torch.Tensor, b: torch.Tensor, out: Optional[torch.Tensor] = None,
            add: Optional[torch.Tensor] = None, alpha: float = 1.0, out_fp32: bool = False,
            accumulate: bool = False, max_ctas: int = 0) -> torch.Tensor:
    """a[M,K] @ b[N,K]^T (+ add).  ``out_fp32`` writes (or accumulates into) an fp32 matrix."""
    if not _lib.use_cuda_kernels(a):
        r = (a.float() @ b.float().t()) * alpha
        if add is not None:
            r = r + add.float()
        if out_fp32:
            if out is not None:
                out.copy_(out + r if accumulate else r)
                return out
            return r
        r = r.to(a.dtype)
        if out is not None:
            out.copy_(r)
            return out
        return r
    a, b = _check2d(a), _check2d(b)
    M, K = a.shape
    N = b.shape[0]
    dtype = torch.float32 if out_fp32 else a.dtype
    if N % 8 == 0 and not (_addressable(out, M, N, dtype) and _addressable(add, M, N, a.dtype)):
        # transposed, expanded over the columns, oddly pitched, of another type or of more dimensions: the fp32 product, then torch
        with torch.no_grad():
            res = gemm_nt(a, b, alpha=alpha, out_fp32=True, max_ctas=max_ctas)
            if add is not None:
                res += add.reshape(M, N) if add.numel() == M * N else add
            if out is None:
                return res.to(dtype)
            dst = out.view(M, N)
            dst.copy_(dst + res if accumulate and out_fp32 else res)
        return out
    if out is None:
        out = torch.empty(M, N, dtype=dtype, device=a.device)
    if skinny_ok(a, b) and not accumulate and not max_ctas and (add is None or not out_fp32):
        skinny(a, b, out, SK_F32 if out_fp32 else SK_STORE, add=add, alpha=alpha)
        return out
    splits = _skinny_splits(M, N, K) if not out_fp32 and SPLIT_K_SKINNY else 1
    if splits > 1:
        return _gemm_nt_split_k(a, b, out, add, alpha, splits)
    epi = EPI_F32 if out_fp32 else (EPI_ADDC if add is not None else EPI_STORE)
    _raw(a, M, K, a.stride(0), 0, b, N, K, b.stride(0), 0, out, out.stride(0), add, add.stride(0) if add is not None else 0,
         None, 0, M, N, K, alpha=alpha, beta=int(accumulate), epilogue=epi, max_ctas=max_ctas)
    return out


def gemm_nn(a: torch.Tensor, b: torch.Tensor, out: Optional[torch.Tensor] = None,
            add: Optional[torch.Tensor] = None, alpha: float = 1.0, max_ctas: int = 0) -> torch.Tensor:
    """a[M,K] @ b[K,N] (+ add)."""
    if not _lib.use_cuda_kernels(a):
        r = (a.float() @ b.float()) * alpha
        if add is not None:
            r = r + add.float()
        r = r.to(a.dtype)
        if out is not None:
            out.copy_(r)
            return out
        return r
    a, b = _check2d(a), _check2d(b)
    M, K = a.shape
    N = b.shape[1]
    if out is None:
        out = torch.empty(M, N, dtype=a.dtype, device=a.device)
    _raw(a, M, K, a.stride(0), 0, b, K, N, b.stride(0), 1, out, out.stride(0), add, add.stride(0) if add is not None else 0,
         None, 0, M, N, K, alpha=alpha, epilogue=EPI_ADDC if add is not None else EPI_STORE, max_ctas=max_ctas)
    return out


def _tn_splits(M: int, N: int, K: int, clusters: int = 74) -> int:
    """Reduction slices for a weight-gradient product whose 256 x 256 tiles fill the CTA pairs badly (e.g. 80 tiles on 74 pairs run
    two waves at 0.54 utilisation).  Modelled time = waves / slices + the fold of the fp32 partials; returns the best slice count
    (1 = do not split).  Only long reductions are worth it."""
    if M < 256 or K < 8192 or os.environ.get("ATS_WGRAD_SPLIT_K", "1") != "1":
        return 1
    tiles = ((M + 255) // 256) * ((N + 255) // 256)
    if tiles >= 4 * clusters:
        return 1
    wave_us = 256 * 256 * K * 2 / 18.9e6   # one wave of full tiles at the sustained rate of a CTA pair
    best, best_t = 1, -(-tiles // clusters) * wave_us
    for s in (2, 3, 4):
        if K % (64 * s) or K // s < 2048:
            continue
        fold_us = ((2 * s * 4 + 4) * M * N) / 6.5e6
        t = -(-(tiles * s) // clusters) * wave_us / s + fold_us
        if t < 0.93 * best_t:
            best, best_t = s, t
    return best


class ScatterTarget:
    """Destination of a weight-gradient product whose rows are owned by different ranks (ZeRO-3 row shards): ``table`` is a
    device int64 tensor with the address of every owner's fp32 gradient rows, ``rows`` the number of rows per owner.  Passed
    as ``out`` to :func:`gemm_tn`, which then adds its result into the owners' buffers from the GEMM epilogue (reduce-scatter
    fused into the product; always accumulating -- the owners zero their shards once per optimiser step)."""

    def __init__(self, table: torch.Tensor, rows: int, shape):
        self.table, self.rows, self.shape = table, rows, tuple(shape)

    def view(self, *shape):
        return self


def gemm_tn(a: torch.Tensor, b: torch.Tensor, out: Optional[torch.Tensor] = None, accumulate: bool = False,
            alpha: float = 1.0, out_fp32: bool = False, max_ctas: int = 0) -> torch.Tensor:
    """a[K,M]^T @ b[K,N]; ``accumulate`` adds into ``out``."""
    if isinstance(out, ScatterTarget):
        a, b = _check2d(a), _check2d(b)
        K, M = a.shape
        N = b.shape[1]
        assert (M, N) == tuple(out.shape) and _lib.use_cuda_kernels(a)
        _raw(a, K, M, a.stride(0), 1, b, K, N, b.stride(0), 1, None, N, None, 0, None, 0, M, N, K, alpha=alpha, beta=1,
             epilogue=EPI_F32, max_ctas=max_ctas, d_table=out.table, scatter_rows=out.rows)
        return out
    if not _lib.use_cuda_kernels(a):
        r = (a.float().t() @ b.float()) * alpha
        if out is not None:
            if accumulate:
                r = r + out.float()
            out.copy_(r.to(out.dtype))
            return out
        return r if out_fp32 else r.to(a.dtype)
    a, b = _check2d(a), _check2d(b)
    K, M = a.shape
    N = b.shape[1]
    if out is None:
        out = torch.empty(M, N, dtype=torch.float32 if out_fp32 else a.dtype, device=a.device)
        accumulate = False
    fp32 = out.dtype == torch.float32
    splits = _tn_splits(M, N, K) if (not fp32 and out.is_contiguous() and alpha == 1.0) else 1
    if splits > 1:
        # the reduction (tokens) is cut into slices that run as groups with fp32 partial outputs; one launch folds them (+ the
        # gradient accumulated so far) into the bf16 result
        kp = K // splits
        part = torch.empty(splits, M, N, dtype=torch.float32, device=a.device)
        _raw(a, K, M, a.stride(0), 1, b, K, N, b.stride(0), 1, part, N, None, 0, None, 0, M, N, kp, epilogue=EPI_F32, groups=splits,
             a_gs_k=kp, b_gs_k=kp, d_gs=M * N, max_ctas=max_ctas)
        _fold_partials(part, splits, M * N, 1, out, out if accumulate else None)
        return out
    epi = EPI_F32 if fp32 else (EPI_ADDC if accumulate else EPI_STORE)
    _raw(a, K, M, a.stride(0), 1, b, K, N, b.stride(0), 1, out, out.stride(0),
         out if (accumulate and not fp32) else None, out.stride(0), None, 0, M, N, K, alpha=alpha,
         beta=int(accumulate), epilogue=epi, max_ctas=max_ctas)
    return out


def gemm_nt_swiglu(a: torch.Tensor, w_gate_up: torch.Tensor, out: Optional[torch.Tensor] = None,
                   pre_act: Optional[torch.Tensor] = None, max_ctas: int = 0) -> torch.Tensor:
    """h = silu(a @ Wg^T) * (a @ Wu^T) with ``w_gate_up = [Wg; Wu]`` of shape [2I, K].  ``pre_act`` ([M, 2I])
    receives the gate/up pre-activations when the backward pass needs them."""
    inter = w_gate_up.shape[0] // 2
    if not _lib.use_cuda_kernels(a):
        gu = (a.float() @ w_gate_up.float().t()).to(a.dtype)
        if pre_act is not None:
            pre_act.copy_(gu)
        g, u = gu.float().chunk(2, dim=-1)
        r = (torch.nn.functional.silu(g) * u).to(a.dtype)
        if out is not None:
            out.copy_(r)
            return out
        return r
    a, w = _check2d(a), _check2d(w_gate_up)
    M, K = a.shape
    if out is None:
        out = torch.empty(M, inter, dtype=a.dtype, device=a.device)
    if pre_act is None and not max_ctas and skinny_ok(a, w, inter):
        skinny(a, w, out, SK_SWIGLU, n=inter, up_offset=inter)
        return out
    _raw(a, M, K, a.stride(0), 0, w, 2 * inter, K, w.stride(0), 0, out, out.stride(0), None, 0,
         pre_act, pre_act.stride(0) if pre_act is not None else 0, M, inter, K, epilogue=EPI_SWIGLU,
         up_offset=inter, max_ctas=max_ctas)
    return out


def swiglu_bwd_reference(pre: torch.Tensor, dh: torch.Tensor):
    """(dgu [.., 2I], h [.., I]) of h = silu(gate) * up from the saved pre-activations [.., 2I] and dh [.., I], in fp32."""
    g, u = pre.float().chunk(2, dim=-1)
    sg = torch.sigmoid(g)
    dhf = dh.float()
    return torch.cat([dhf * u * (sg + g * sg * (1 - sg)), dhf * g * sg], dim=-1).to(pre.dtype), (g * sg * u).to(pre.dtype)


def gemm_nn_swiglu_bwd(dy: torch.Tensor, w_down: torch.Tensor, pre: torch.Tensor):
    """dy [M, H] · w_down [H, I] = dh, pushed through the SwiGLU backward in the GEMM epilogue: -> (dgu [M, 2I], h [M, I])
    from the saved pre-activations ``pre`` [M, 2I]; dh is never written."""
    inter = w_down.shape[1]
    if not _lib.use_cuda_kernels(dy):
        return swiglu_bwd_reference(pre, (dy.float() @ w_down.float()).to(dy.dtype))
    dy, w = _check2d(dy), _check2d(w_down)
    M, H = dy.shape
    assert pre.is_contiguous() and pre.shape == (M, 2 * inter)
    dgu = torch.empty_like(pre)
    h = torch.empty(M, inter, dtype=pre.dtype, device=pre.device)
    _raw(dy, M, H, dy.stride(0), 0, w, H, inter, w.stride(0), 1, dgu, 2 * inter, h, inter, pre, 2 * inter, M, inter, H,
         epilogue=EPI_SWIGLU_BWD, up_offset=inter)
    return dgu, h


# ----------------------------------------------------------------------------------------------------------
# grouped (expert) products on the capacity layout
# ----------------------------------------------------------------------------------------------------------
def _ref_mask(counts: torch.Tensor, cap: int) -> torch.Tensor:
    return (torch.arange(cap, device=counts.device)[None, :] < counts[:, None].long())


def pack_kmajor(w: torch.Tensor) -> torch.Tensor:
    """[.., N, K] weight -> the same shape with the elements stored tile by tile ([N / 128][K / 64][128][64]): every
    128 x 64 box the GEMM loads is then 16 KB of consecutive memory, which lets a weight that is read once per step (decode)
    stream at close to HBM speed instead of touching 128 bytes per DRAM page.  Needs N % 128 == 0 and K % 64 == 0."""
    *lead, N, K = w.shape
    if N % 128 or K % 64:
        raise ValueError("pack_kmajor needs N % 128 == 0 and K % 64 == 0")
    t = w.reshape(-1, N // 128, 128, K // 64, 64).permute(0, 1, 3, 2, 4).contiguous()
    return t.view(*lead, N, K)


def unpack_kmajor(w: torch.Tensor) -> torch.Tensor:
    """Inverse of :func:`pack_kmajor`."""
    *lead, N, K = w.shape
    t = w.reshape(-1, N // 128, K // 64, 128, 64).permute(0, 1, 3, 2, 4).contiguous()
    return t.view(*lead, N, K)


def grouped_nt(x: torch.Tensor, w: torch.Tensor, counts: torch.Tensor, swiglu: bool = False,
               pre_act: Optional[torch.Tensor] = None, out: Optional[torch.Tensor] = None, b_div: int = 1,
               d_table: Optional[torch.Tensor] = None, packed: bool = False, k_split: int = 1, fold=None) -> torch.Tensor:
    """x[G,C,K] · w[E,N,K]^T -> [G,C,N] (or [G,C,N/2] through SwiGLU) for the first counts[g] rows of every
    group; group g uses weight g // b_div (G = E * b_div: several token blocks per expert, one per source rank).
    Rows beyond the padded count are left untouched.  ``d_table`` (int64 [G]) redirects the output of group g to
    an arbitrary base address (a buffer on a peer GPU).  ``packed``: ``w`` is stored as :func:`pack_kmajor` leaves it."""
    Gn, C, K = x.shape
    N = w.shape[1]
    if not _lib.use_cuda_kernels(x):
        if packed:
            w = unpack_kmajor(w)
        wx = w.repeat_interleave(b_div, dim=0) if b_div > 1 else w
        y = torch.einsum("eck,enk->ecn", x.float(), wx.float()).to(x.dtype)
        mask = _ref_mask(counts, C)[..., None]
        y = torch.where(mask, y, torch.zeros_like(y))
        if swiglu:
            if pre_act is not None:
                pre_act.copy_(y)
            g, u = y.float().chunk(2, dim=-1)
            y = (torch.nn.functional.silu(g) * u).to(x.dtype)
        if out is not None:
            out.copy_(y)
            return out
        return y
    assert x.is_contiguous() and w.is_contiguous() and C % 128 == 0
    n_out = N // 2 if swiglu else N
    if out is None and d_table is None:
        out = torch.empty(Gn, C, n_out, dtype=x.dtype, device=x.device)
    if k_split > 1:
        # few output tiles and a long reduction (the down projection of a decode step): the reduction is cut into k_split
        # slices, every (group, slice) pair is a work item with an fp32 partial block, and one small launch folds the slices
        assert not swiglu and d_table is None and pre_act is None and K % (64 * k_split) == 0 and out.is_contiguous()
        part = torch.empty(Gn * k_split, C, N, dtype=torch.float32, device=x.device)
        _raw(x, Gn * C, K, K, 0, w, w.shape[0] * N, K, K, 2 if packed else 0, part, N, None, 0, None, 0, C, N, K // k_split,
             epilogue=EPI_F32, groups=Gn * k_split, ragged=1, counts=counts, a_gs_mn=C, b_gs_mn=N, d_gs=C * N, b_div=b_div,
             k_split=k_split)
        # ``fold(part, k_split, n_inner, n_outer, out)`` replaces the plain fold (e.g. one that also signals the peers that will read out)
        (fold or _fold_partials)(part, k_split, C * N, Gn, out)
        return out
    _raw(x, Gn * C, K, K, 0, w, w.shape[0] * N, K, K, 2 if packed else 0, out, n_out, None, 0, pre_act,
         N if pre_act is not None else 0,
         C, n_out, K, epilogue=EPI_SWIGLU if swiglu else EPI_STORE, up_offset=N // 2 if swiglu else 0,
         groups=Gn, ragged=1, counts=counts, a_gs_mn=C, b_gs_mn=N, d_gs=C * n_out,
         aux_gs=C * N if pre_act is not None else 0, b_div=b_div, d_table=d_table)
    return out


def grouped_nn(dy: torch.Tensor, w: torch.Tensor, counts: torch.Tensor, out: Optional[torch.Tensor] = None,
               b_div: int = 1, d_table: Optional[torch.Tensor] = None) -> torch.Tensor:
    """dy[G,C,N] · w[E,N,K] -> [G,C,K] (input gradient of grouped_nt)."""
    Gn, C, N = dy.shape
    K = w.shape[2]
    if not _lib.use_cuda_kernels(dy):
        wx = w.repeat_interleave(b_div, dim=0) if b_div > 1 else w
        y = torch.einsum("ecn,enk->eck", dy.float(), wx.float()).to(dy.dtype)
        y = torch.where(_ref_mask(counts, C)[..., None], y, torch.zeros_like(y))
        if out is not None:
            out.copy_(y)
            return out
        return y
    assert dy.is_contiguous() and w.is_contiguous() and C % 128 == 0
    if out is None and d_table is None:
        out = torch.empty(Gn, C, K, dtype=dy.dtype, device=dy.device)
    _raw(dy, Gn * C, N, N, 0, w, w.shape[0] * N, K, K, 1, out, K, None, 0, None, 0, C, K, N,
         groups=Gn, ragged=1, counts=counts, a_gs_mn=C, b_gs_k=N, d_gs=C * K, b_div=b_div, d_table=d_table)
    return out


def grouped_nn_swiglu_bwd(dy: torch.Tensor, w: torch.Tensor, counts: torch.Tensor, pre: torch.Tensor, b_div: int = 1):
    """Backward through ``h = silu(gate) * up`` fused into the product ``dh = dy · w``: dy [G,C,N], w [E,N,I], pre [G,C,2I]
    (saved gate / up pre-activations) -> (dgu [G,C,2I], h [G,C,I]); dh itself is never written.  Rows beyond the padded
    count of a group are left untouched.  With 16-byte accesses this epilogue (two reads and three stores per element,
    one row per thread) slowed the step by 2.5 %, because every access filled half an L2 sector and the requests crowded out the
    operand loads; with 32-byte loads and stores it is 1 % faster than GEMM + streaming element-wise kernel."""
    Gn, C, N = dy.shape
    inter = w.shape[2]
    if not _lib.use_cuda_kernels(dy):
        return swiglu_bwd_reference(pre, grouped_nn(dy, w, counts, b_div=b_div))
    assert dy.is_contiguous() and w.is_contiguous() and pre.is_contiguous() and C % 128 == 0
    dgu = torch.empty_like(pre)
    h = torch.empty(Gn, C, inter, dtype=pre.dtype, device=pre.device)
    _raw(dy, Gn * C, N, N, 0, w, w.shape[0] * N, inter, inter, 1, dgu, 2 * inter, h, inter, pre, 2 * inter, C, inter, N,
         epilogue=EPI_SWIGLU_BWD, up_offset=inter, groups=Gn, ragged=1, counts=counts, a_gs_mn=C, b_gs_k=N, d_gs=C * 2 * inter,
         c_gs=C * inter, aux_gs=C * 2 * inter, b_div=b_div)
    return dgu, h


def grouped_tn(dy: torch.Tensor, x: torch.Tensor, counts: torch.Tensor, out: Optional[torch.Tensor] = None,
               accumulate: bool = False, k_segs: int = 1) -> torch.Tensor:
    """dy[G,C,N]^T · x[G,C,K] -> [G / k_segs, N, K] (weight gradient of grouped_nt): expert e reduces over the used
    rows of its k_segs consecutive token blocks."""
    Gn, C, N = dy.shape
    K = x.shape[2]
    E = Gn // k_segs
    if not _lib.use_cuda_kernels(dy):
        mask = _ref_mask(counts, C)[..., None].float()
        r = torch.einsum("ecn,eck->enk", (dy.float() * mask).reshape(E, k_segs * C, N), (x.float() * mask).reshape(E, k_segs * C, K))
        if out is not None:
            if accumulate:
                r = r + out.float()
            out.copy_(r.to(out.dtype))
            return out
        return r.to(dy.dtype)
    assert dy.is_contiguous() and x.is_contiguous() and C % 128 == 0
    if out is None:
        out = torch.empty(E, N, K, dtype=dy.dtype, device=dy.device)
        accumulate = False
    _raw(dy, Gn * C, N, N, 1, x, Gn * C, K, K, 1, out, K, out if accumulate else None, K, None, 0, N, K, C,
         epilogue=EPI_ADDC if accumulate else EPI_STORE, groups=E, ragged=2, counts=counts,
         a_gs_k=k_segs * C, b_gs_k=k_segs * C, d_gs=N * K, c_gs=N * K, k_segs=k_segs, seg_stride=C)
    return out
