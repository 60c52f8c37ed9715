"""ctypes binding of the sm_100a kernel library (libmlb_cuda.so).

Every function takes torch CUDA tensors (bf16 activations / parameters, fp32 statistics, gradients and
optimizer state), checks dtype / contiguity, and launches on the current torch stream.  Nothing here falls
back to PyTorch: if the library cannot be loaded the import fails.
"""
from __future__ import annotations

import ctypes as C
import importlib.util
import os
import subprocess
import sys
import threading
import warnings
from functools import lru_cache

import torch

from .. import build as _build

_i32, _i64, _f32, _vp = C.c_int, C.c_long, C.c_float, C.c_void_p


class Address(int):
    """Device memory by its address, where an entry point of the extension module takes no tensor: an untyped buffer, a part of a workspace."""


NONE = Address(0)      # an optional tensor that is not there

# Entry points that the extension module has, by the C type of each parameter.  b bf16, f fp32, i int32, u bytes: tensors, or an Address; n int,
# l long, d float; s the current stream
_KINDS = {
    "linear_fwd": "bbbnnnnnns", "linear_fwd_posembed": "bbbbnnnnnnns", "linear_fwd_rope": "bbbnnnnnnffnns",
    "linear_fwd_swiglu": "bbbbnnnnnns", "linear_dx": "bbbnnnnnns", "linear_dx_delta": "bbbbfnnnnnnnns", "linear_dw": "fbbnnnnnns",
    "gemm": "bbbnnnnnnnnns", "gemm_dw_direct": "nnn", "linear_fwd_fp8": "buunnnnnnds", "capture_id": "s", "zero": "bls",
    "cast_f2b": "bflds", "colsum_splits": "ln", "colsum": "bblnfs", "rmsnorm_fwd": "bfbblnds", "add_rmsnorm_fwd": "bbfbbblnds",
    "rmsnorm_fwd_fp8": "bufbblndds", "rmsnorm_bwd_blocks": "l", "rmsnorm_bwd": "bfbbbfblnfis", "rmsnorm_bwd_cast": "bbbbbfblnfs",
    "layernorm_fwd": "bffbbblnds", "layernorm_bwd2": "bbbnbbbfflnfs", "swiglu_fwd": "bblns", "swiglu_fwd_fp8": "bublnds",
    "swiglu_bwd": "bbblns", "rope": "bfflnnnds", "rope_copy": "bbfflnnnns", "kv_group_sum": "bblnnns", "attn_fwd": "bfbnnnns",
    "attn_bwd_scratch_bytes": "nnnn", "attn_bwd": "bbbbffbnnnnffs", "attn_bwd_have_delta": "bbbbffbnnnnffs",
    "attn_bidir_fwd": "bfbnnnns", "attn_bidir_bwd": "bbbbffnnnns", "ce_mean": "fffbbilns", "ce_fwd_bwd": "fbilnldns",
    "scale_dev": "bbfls", "embed_fwd": "bbilnns", "embed_bwd": "fbilnnnns", "adamw": "fbffflddddddddfs", "sum_scale": "fflds"}
_CTYPES = {"n": _i32, "l": _i64, "d": _f32}      # (else a pointer)


@lru_cache(maxsize=1)
def lib():
    ext = _build.external_lib("libmlb_cuda.so")
    if ext is None and not _build.is_fresh(_build.CUDA_LIB, _build.cuda_hash()):
        if _build.CUDA_LIB.exists() and _build._nvcc() is None:
            pass  # no compiler on this machine: use the library that travelled with the tree
        else:
            _build.build_cuda()
    L = C.CDLL(str(ext or _build.CUDA_LIB))
    sig = {
        "mlb_gemm_force_simt": [_i32],
        "mlb_gemm_set_max_ctas": [_i32],
        "mlb_gemm_set_splits": [_i32],
        "mlb_gemm_use_3d_maps": [_i32],
        "mlb_gemm_use_pairs": [_i32],
        "mlb_gemm_epilogue_mode": [_i32],
        "mlb_gemm_streamk": [_i32],
        "mlb_gemm_tile_order": [_i32],
        "mlb_gemm_streamk_groups": [_i32],
        "mlb_attn_force_simt": [_i32],
        "mlb_attn_fwd_mode": [_i32],
        "mlb_attn_fwd_balance": [_i32],
        "mlb_ce_mode": [_i32],
        "mlb_set_prefix": [_vp, _vp, _i32, _i32, _i32, _i32, _vp],
        "mlb_gather_prefix_grad": [_vp, _vp, _i32, _i32, _i32, _i32, _vp],
        "mlb_fp8_qdq": [_vp, _vp, _i64, _f32, _vp],
        "mlb_ce_chunk_stats": [_vp, _vp, _vp, _vp, _vp, _i64, _i32, _i64, _i32, _vp],
        "mlb_ce_chunk_grad": [_vp, _vp, _vp, _vp, _vp, _vp, _i64, _i32, _i64, _i32, _f32, _vp],
        "mlb_cast_b2f": [_vp, _vp, _i64, _f32, _vp],
        "mlb_scale_f32": [_vp, _i64, _f32, _vp],
        "mlb_residual_add": [_vp, _vp, _vp, _i64, _vp],
        "mlb_patchify": [_vp, _vp, _i32, _i32, _i32, _i32, _i32, _vp],
        "mlb_add_posembed": [_vp, _vp, _i64, _i32, _i32, _vp],
        "mlb_posembed_grad": [_vp, _vp, _i64, _i32, _i32, _vp],
        "mlb_linear_fwd_gather": [_vp, _vp, _i32, _i32, _i32, _i32, _i32, _vp, _i64, _vp, _i64, _i32, _vp, _vp, C.c_double, _vp],
        "mlb_layernorm_bwd": [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _i64, _i32, _vp],
        "mlb_linear_fwd_fp8_rope": [_vp, _vp, _vp, _i32, _i32, _i32, _i32, _i32, _i32, _f32, _vp, _vp, _i32, _i32, _vp],
        "mlb_linear_fwd_fp8_swiglu": [_vp, _vp, _vp, _vp, _i32, _i32, _i32, _i32, _i32, _i32, _f32, _vp],
        "mlb_add_rmsnorm_fwd_fp8": [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _i64, _i32, _f32, _f32, _vp],
        "mlb_cast_bf16_fp8": [_vp, _vp, _i64, _f32, _vp],
        "mlb_adamw_fp8": [_vp] * 6 + [_i64] + [_f32] * 9 + [_vp, _vp],
    }
    sig.update({"mlb_" + name: [_CTYPES.get(k, _vp) for k in kinds] for name, kinds in _KINDS.items()})
    for name, args in sig.items():
        fn = getattr(L, name)
        fn.argtypes = args
        fn.restype = _i32
    L.mlb_attn_bwd_scratch_bytes.restype = _i64
    L.mlb_capture_id.restype = C.c_ulonglong
    for tag in ("gemm", "attn", "elementwise", "comm"):
        for pre in ("mlb_get_error_", "mlb_clear_error_"):
            if hasattr(L, pre + tag):
                getattr(L, pre + tag).restype = _i32
                getattr(L, pre + tag).argtypes = []
    L.mlb_attn_dynamic.argtypes = [_i32]
    L.mlb_attn_dynamic.restype = None
    if os.environ.get("ENTROPY_ATTN_DYNAMIC", "") == "1":
        L.mlb_attn_dynamic(1)
    return L


@lru_cache(maxsize=1)
def bridge():
    """The operators' host path as an extension module on this library's kernels (csrc/torch/bridge.cpp), or None where it cannot be
    built or loaded with this torch: ops/autograd.py and the functions below then call the same kernels from Python."""
    lib()
    try:
        spec = importlib.util.spec_from_file_location("mlb_torch", str(_build.build_torch()))
        m = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(m)
        m.bind(str(_build.external_lib("libmlb_cuda.so") or _build.CUDA_LIB), sys.modules[__name__])
    except (OSError, subprocess.CalledProcessError, ImportError, RuntimeError) as e:      # (ImportError: another torch's; RuntimeError: bind)
        warnings.warn(f"libmlb_torch.so cannot be built or loaded ({e}): operators run through Python, several times slower per call")
        return None
    return m


def gemm_autotune(on: bool):
    """Per-shape plan cache of the GEMMs (the reference's ENTROPY_AUTOTUNE, train/gemm.cuh): on = the first call of a shape
    outside graph capture times this library's own forms (tile, tile order, epilogue, stream-K) and later calls use the
    fastest; off = static heuristics."""
    L = lib()
    L.mlb_gemm_autotune.argtypes = [_i32]
    L.mlb_gemm_autotune.restype = None
    L.mlb_gemm_autotune(1 if on else 0)


def gemm_plans():
    """The plan cache as a list of dicts (form: bit 2 = A MN-major, bit 1 = B MN-major, bit 0 = fp32 add-reduce)."""
    L = lib()
    L.mlb_gemm_plan_count.restype = _i32
    L.mlb_gemm_plan_count.argtypes = []
    L.mlb_gemm_plan_get.restype = _i32
    L.mlb_gemm_plan_get.argtypes = [_i32, C.POINTER(C.c_int)]
    out = []
    buf = (C.c_int * 10)()
    for i in range(L.mlb_gemm_plan_count()):
        if L.mlb_gemm_plan_get(i, buf) == 0:
            out.append(dict(form=buf[0], M=buf[1], N=buf[2], K=buf[3], tile=("pair", "model", "1cta")[buf[4]],
                            order=buf[5], epilogue=("tma", "warps")[buf[6]], streamk=buf[7], groups=buf[8], us=buf[9]))
    return out


def attn_dynamic(on: bool):
    """The persistent attention kernels draw their work items from a counter in device memory (on) instead of following
    the table built on the host (off, the default; ENTROPY_ATTN_DYNAMIC=1 turns it on at load).  Measured: alone the
    table is 4 us (forward) and 10 us (backward) per call ahead, and with the gradient kernels running behind backward
    on 4 GPUs the step is 17.4-17.6 ms with the table against 17.7-17.8 ms with the counter, so nothing selects the
    counter by itself; it needs no table for a shape met for the first time during graph capture."""
    lib().mlb_attn_dynamic(1 if on else 0)


LAUNCHES = 0  # number of kernel-launching calls made through this module (bench.py reports it)


def _st():
    # the current stream's handle without a Stream object around it (that costs more than the rest of a call's arguments)
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def _chk(rc, name):
    global LAUNCHES
    LAUNCHES += 1
    if rc != 0:
        raise RuntimeError(f"{name} failed: code {rc} ({_cuda_err(rc)})")


def _cuda_err(rc):
    if rc == -2:
        return f"tensor map refused, driver code {lib().mlb_tmap_error()}"
    try:
        return torch.cuda.cudart().cudaGetErrorString(rc) if rc > 0 else "library error"
    except Exception:
        return "?"


def get_error() -> int:
    """Non-zero if a kernel gave up on a bounded wait: (code << 24) | detail, see csrc/common.cuh."""
    L = lib()
    for tag in ("gemm", "attn", "elementwise", "comm"):
        if hasattr(L, "mlb_get_error_" + tag):
            v = getattr(L, "mlb_get_error_" + tag)()
            if v:
                return v
    return 0


_ERR_CODES = {1: "an mbarrier wait inside a kernel's pipeline ran out", 2: "a wait on a peer's or the host's flag ran out",
              3: "an index was out of range"}
_ERR_BOUNDS = {0xE1: "token id outside the vocabulary (embedding forward)", 0xE2: "token id outside the vocabulary (embedding backward)",
               0xCE: "target outside the vocabulary (cross-entropy)",
               0xA1: "shared memory of the attention backward (head size 128) does not start on a 1024-byte boundary",
               0xA2: "shared memory of the attention backward (head size 64) does not start on a 1024-byte boundary"}


def describe_error(err: int) -> str:
    """The error word in words: (code << 24) | detail, see csrc/common.cuh."""
    code, detail = err >> 24, err & 0xFFFFFF
    text = _ERR_CODES.get(code, f"code {code}")
    if code == 3 and detail in _ERR_BOUNDS:
        return f"{text}: {_ERR_BOUNDS[detail]}"
    return f"{text}, detail {detail:#x}"


def read_errors_async(host_words: torch.Tensor):
    """The four error words copied into `host_words` (pinned int32[4]) behind the current stream's work, without a
    synchronisation of their own: a caller that synchronises the stream anyway (to read a loss) checks them for free."""
    L = lib()
    base = host_words.data_ptr()
    for i, tag in enumerate(("gemm", "attn", "elementwise", "comm")):
        fn = getattr(L, "mlb_read_error_async_" + tag)
        fn.argtypes = [_vp, _vp]
        fn.restype = _i32
        _chk(fn(base + 4 * i, _st()), "read_error_async")


def clear_error():
    L = lib()
    for tag in ("gemm", "attn", "elementwise", "comm"):
        if hasattr(L, "mlb_clear_error_" + tag):
            getattr(L, "mlb_clear_error_" + tag)()


def _b(t, name="tensor"):
    assert t.is_cuda and t.dtype == torch.bfloat16 and t.is_contiguous(), f"{name}: need contiguous CUDA bf16"
    return t.data_ptr()


def _f(t, name="tensor"):
    assert t.is_cuda and t.dtype == torch.float32 and t.is_contiguous(), f"{name}: need contiguous CUDA fp32"
    return t.data_ptr()


def _i(t, name="tensor"):
    assert t.is_cuda and t.dtype == torch.int32 and t.is_contiguous(), f"{name}: need contiguous CUDA int32"
    return t.data_ptr()


class _Ctypes:
    """The entry points as the extension module has them, through ctypes."""

    def __getattr__(self, name):
        fn, kinds, to = getattr(lib(), name), _KINDS[name[4:]], {"b": _b, "f": _f, "i": _i, "u": _u8}

        def call(*args):
            a = [to[k](x) if k in to and type(x) is not Address else x for k, x in zip(kinds, args, strict=kinds[-1] != "s")]
            return fn(*a, _st()) if kinds[-1] == "s" else fn(*a)

        setattr(self, name, call)
        return call


_E = None


def _entries():
    global _E
    if _E is None:
        _E = bridge() or _Ctypes()
    return _E


_scratch = threading.local()


def _capture_id(st):
    """Number of the graph capture the stream takes part in, 0 outside one."""
    return lib().mlb_capture_id(st) if torch._C._cuda_isCurrentStreamCapturing() else 0


def scratch(key, numel, dtype, device, zero=False):
    """Workspace kept from call to call: of the calling thread, on its current stream (another thread or stream may be in the middle
    of the same sequence of kernels), and inside a graph capture of that capture (its replays run when and where they like;
    zero-filled ones are zeroed by every replay).  Grows; what it grew out of goes back to the allocator."""
    st = _st()
    cap = _capture_id(st)
    tensors = getattr(_scratch, "tensors", None)
    if tensors is None or (cap and cap != _scratch.capture):      # (an earlier capture is over: its graph owns its memory)
        _scratch.capture = cap
        tensors = _scratch.tensors = {k: t for k, t in (tensors or {}).items() if k[4] == 0}
    k = (key, device, dtype, st, cap)
    t = tensors.get(k)
    if t is None or t.numel() < numel:
        t = tensors[k] = (torch.zeros if zero else torch.empty)(numel, dtype=dtype, device=device)
    return t


# ------------------------------------------------------------------ linear
def linear_fwd(out, x, W):
    M, K = x.shape
    N = W.shape[0]
    _chk(_entries().mlb_linear_fwd(out, x, W, M, N, K, out.stride(0), x.stride(0), W.stride(0)), "linear_fwd")


def linear_fwd_rope(out, x, W, cos, sin, T, rope_cols):
    """out = x . W^T with rotary embedding applied to output columns [0, rope_cols) in the GEMM epilogue (heads of 64
    columns, position = row % T).  Returns False when the shape does not take that path (nothing was launched)."""
    M, K = x.shape
    N = W.shape[0]
    fn = _entries().mlb_linear_fwd_rope
    rc = fn(out, x, W, M, N, K, out.stride(0), x.stride(0), W.stride(0), cos, sin, T, rope_cols)
    if rc == -7:
        return False
    _chk(rc, "linear_fwd_rope")
    return True


def linear_fwd_swiglu(gu, sw, x, W):
    """gu[M, 2I] = x . W^T (W = [W_gate; W_up]) and sw[M, I] = silu(gate) * up out of the same GEMM's epilogue.  Returns
    False when the shape does not take that path (nothing was launched): the caller then runs the product and the
    SwiGLU kernel one after the other."""
    M, K = x.shape
    I = sw.shape[1]
    if W.shape[0] != 2 * I or gu.shape[1] != 2 * I or sw.stride(0) != I:
        return False
    fn = _entries().mlb_linear_fwd_swiglu
    rc = fn(gu, sw, x, W, M, I, K, gu.stride(0), x.stride(0), W.stride(0))
    if rc == -7:
        return False
    _chk(rc, "linear_fwd_swiglu")
    return True


def linear_fwd_posembed(out, x, W, pos, period):
    """out = x . W^T + pos[row % period] with the add on the fp32 accumulators in the GEMM epilogue.  Returns False when
    the shape does not take that path (nothing was launched)."""
    M, K = x.shape
    N = W.shape[0]
    if pos.shape[-1] != N or not pos.is_contiguous():
        return False
    fn = _entries().mlb_linear_fwd_posembed
    rc = fn(out, x, W, pos, period, M, N, K, out.stride(0), x.stride(0), W.stride(0))
    if rc == -7:
        return False
    _chk(rc, "linear_fwd_posembed")
    return True


def linear_dx(dx, dout, W):
    M, N = dout.shape
    K = W.shape[1]
    _chk(_entries().mlb_linear_dx(dx, dout, W, M, N, K, dx.stride(0), dout.stride(0), W.stride(0)), "linear_dx")


def linear_dw(dW, dout, x):
    M, N = dout.shape
    K = x.shape[1]
    _chk(_entries().mlb_linear_dw(dW, dout, x, M, N, K, dW.stride(0), dout.stride(0), x.stride(0)), "linear_dw")


def linear_bias_fwd(out, x, W, b):
    """out = x . W^T + b: the position-table epilogue with a period of one row; where the shape does not take it the bias is added
    behind the product."""
    if not linear_fwd_posembed(out, x, W, b.view(1, -1), 1):
        linear_fwd(out, x, W)
        out += b


def linear_dw_cast(dW, dout, x):
    """dW (bf16, overwritten) = dout^T . x with fp32 accumulation and one rounding.  Either one product that stores bf16, or the
    add-reduce product into a zeroed fp32 buffer and a cast: the second cuts the reduction over the rows up to fill the machine,
    the first saves two launches and 14 bytes per element of dW.  The library's estimate of both decides."""
    if dW.dtype == torch.bfloat16 and (_entries().mlb_gemm_dw_direct(dout.shape[1], x.shape[1], dout.shape[0]) or dW.numel() == 0):
        return gemm(dW, dout, x, True, True, False)
    acc = torch.empty(dW.shape, dtype=torch.float32, device=dW.device)
    zero_(acc)
    linear_dw(acc, dout, x)
    cast(dW, acc)


def gemm(out, A, B, a_mn=False, b_mn=False, accumulate=False):
    """D[M,N] = sum_k A(m,k) B(n,k).  A is [M,K] (a_mn=False) or stored transposed [K,M] (a_mn=True); B likewise with N.
    `out` is bf16 (overwritten) or, with accumulate=True, fp32 (added to)."""
    M, K = (A.shape[1], A.shape[0]) if a_mn else A.shape
    N = B.shape[1] if b_mn else B.shape[0]
    _chk(_entries().mlb_gemm(Address(out.data_ptr()), A, B, M, N, K, out.stride(0), A.stride(0), B.stride(0), int(a_mn), int(b_mn),
                        int(accumulate)), "gemm")


def linear_fwd_gather(out, x, N, K, unit_dst, w_off, src_table, shard_elems, world, flags, ctr, spin_limit_s=20.0):
    """out = x . W^T with W = unit_dst[w_off : w_off + N*K] viewed [N, K]; the same launch all-gathers the whole sharded
    unit into unit_dst from the ranks' shards (device pointer table `src_table`).  Cooperative launch."""
    fn = lib().mlb_linear_fwd_gather
    M = x.shape[0]
    _chk(fn(_b(out), _b(x), M, N, K, out.stride(0), x.stride(0), _b(unit_dst), w_off, src_table.data_ptr(), shard_elems, world,
            _i(flags), _i(ctr), spin_limit_s, _st()), "linear_fwd_gather")


# ------------------------------------------------------------------ attention
def attn_fwd(out, lse, qkv, B, T, H, hd):
    _chk(_entries().mlb_attn_fwd(out, lse, qkv, B, T, H, hd), "attn_fwd")


FUSED_ATTN_BWD = True   # head size 64: single fused backward kernel (False = separate dK/dV and dQ kernels)
FUSED_ATTN_BWD_MAX_SCRATCH = 4 << 30   # bytes of dQ partials (grows with B*T*T) the fused backward may use


def linear_dx_delta(dx, dout, W, o, B, T, H):
    """dx[M, C] = dout[M, N] . W[N, C] for the attention output projection (C = H * 64) with the attention backward's
    delta[b, h, t] = sum_c dx[row, h*64 + c] * o[row, h*64 + c] written by the same kernel's epilogue into the scratch that
    attn_bwd(..., have_delta=True) reads.  Returns False when the shape does not take that path (nothing was launched)."""
    M, N = dout.shape
    Cc = W.shape[1]
    if Cc != H * 64 or M != B * T or dx.stride(0) != Cc or o.stride(0) != Cc:
        return False
    delta = scratch("attn_delta", B * H * T, torch.float32, dout.device)
    fn = _entries().mlb_linear_dx_delta
    rc = fn(dx, dout, W, o, delta, T, H, M, N, Cc, dx.stride(0), dout.stride(0), W.stride(0))
    if rc == -7:
        return False
    _chk(rc, "linear_dx_delta")
    return True


def attn_bwd(dqkv, dout, qkv, out, lse, B, T, H, hd, rope=None, have_delta=False):
    """rope=(cos, sin): ask the kernel to apply RoPE's backward rotation to dQ/dK in its epilogue.
    have_delta: linear_dx_delta has just written this call's delta term, the pass over dO and O is left out.
    Returns True if it did (tensor-core path), False if the caller still has to call rope_bwd."""
    delta = scratch("attn_delta", B * H * T, torch.float32, qkv.device)
    part = NONE
    if hd == 64 and FUSED_ATTN_BWD:
        # per-(query tile, key tile) bf16 partials of dQ; past FUSED_ATTN_BWD_MAX_SCRATCH the two-kernel backward runs
        nbytes = _entries().mlb_attn_bwd_scratch_bytes(B, T, H, hd)
        if 0 < nbytes <= FUSED_ATTN_BWD_MAX_SCRATCH:
            part = torch.empty(nbytes // 2, dtype=torch.bfloat16, device=qkv.device)      # (too large to be kept per stream)
    cp, sp = (NONE, NONE) if rope is None else rope
    fn = _entries().mlb_attn_bwd
    if have_delta:
        fn = _entries().mlb_attn_bwd_have_delta
    rc = fn(dqkv, dout, qkv, out, lse, delta, part, B, T, H, hd, cp, sp)
    global LAUNCHES
    LAUNCHES += 2 if have_delta else 3
    if rc < 0 or rc > 1:
        raise RuntimeError(f"attn_bwd failed: code {rc}")
    return rc == 1


def attn_bidir_fwd(out, lse, qkv, B, T, H, hd):
    fn = _entries().mlb_attn_bidir_fwd
    _chk(fn(out, lse, qkv, B, T, H, hd), "attn_bidir_fwd")


def attn_bidir_bwd(dqkv, dout, qkv, out, lse, B, T, H, hd):
    delta = scratch("attn_delta", B * H * T, torch.float32, qkv.device)
    fn = _entries().mlb_attn_bidir_bwd
    _chk(fn(dqkv, dout, qkv, out, lse, delta, B, T, H, hd), "attn_bidir_bwd")


# ------------------------------------------------------------------ embedding
def embed_fwd(out, wte, ids):
    _chk(_entries().mlb_embed_fwd(out, wte, ids, ids.numel(), wte.shape[1], wte.shape[0]), "embed_fwd")


def embed_bwd(dwte, dout, ids, T, n_pre):
    _chk(_entries().mlb_embed_bwd(dwte, dout, ids, ids.numel(), dwte.shape[1], dwte.shape[0], T, n_pre), "embed_bwd")


def set_prefix(x, prefix, B, T, n_pre):
    _chk(lib().mlb_set_prefix(_b(x), _b(prefix), B, T, n_pre, x.shape[-1], _st()), "set_prefix")


def gather_prefix_grad(dprefix, dresid, B, T, n_pre):
    _chk(lib().mlb_gather_prefix_grad(_b(dprefix), _b(dresid), B, T, n_pre, dresid.shape[-1], _st()), "gather_prefix_grad")


# ------------------------------------------------------------------ norms
def rmsnorm_fwd(out, rstd, x, w, eps):
    rows, Cc = x.shape
    _chk(_entries().mlb_rmsnorm_fwd(out, rstd, x, w, rows, Cc, eps), "rmsnorm_fwd")


def add_rmsnorm_fwd(resid, out, rstd, a, b, w, eps):
    rows, Cc = a.shape
    _chk(_entries().mlb_add_rmsnorm_fwd(resid, out, rstd, a, b, w, rows, Cc, eps), "add_rmsnorm_fwd")


def layernorm_fwd(out, mean, rstd, x, w, b, eps):
    rows, Cc = x.shape
    fn = _entries().mlb_layernorm_fwd
    _chk(fn(out, mean, rstd, x, w, NONE if b is None else b, rows, Cc, eps), "layernorm_fwd")


def _partial(numel, device):
    # of the caching allocator, per call: calls on different streams do not share it
    return torch.empty(numel, dtype=torch.float32, device=device)


def layernorm_bwd(dx, dw, db, dy, x, w, mean, rstd):
    rows, Cc = x.shape
    L = lib()
    part = _partial(L.mlb_rmsnorm_bwd_blocks(rows) * 2 * Cc, x.device)
    d = _f(db) if db is not None else None
    rc = L.mlb_layernorm_bwd2(_b(dx), _f(dw), d, 0, _b(dy), _b(x), _b(w), _f(mean), _f(rstd), rows, Cc, part.data_ptr(), _st())
    if rc == -7:      # a width those kernels do not take
        rc = L.mlb_layernorm_bwd(_b(dx), _f(dw), d, _b(dy), _b(x), _b(w), _f(mean), _f(rstd), rows, Cc, _st())
    _chk(rc, "layernorm_bwd")


def layernorm_bwd_cast(dx, dw, db, dy, x, w, mean, rstd):
    """layernorm_bwd with dw (and db) in bf16, overwritten."""
    rows, Cc = x.shape
    L = _entries()
    part = _partial(L.mlb_rmsnorm_bwd_blocks(rows) * 2 * Cc, x.device)
    rc = L.mlb_layernorm_bwd2(dx, dw, NONE if db is None else db, 1, dy, x, w, mean, rstd, rows, Cc, part)
    if rc == -7:
        aw, ab = torch.zeros_like(dw, dtype=torch.float32), torch.zeros_like(dw, dtype=torch.float32)
        layernorm_bwd(dx, aw, ab, dy, x, w, mean, rstd)
        dw.copy_(aw)
        if db is not None:
            db.copy_(ab)
        return
    _chk(rc, "layernorm_bwd_cast")


def rmsnorm_bwd_cast(dx, dw, dy, x, w, rstd, add=None):
    """rmsnorm_bwd with dw in bf16, overwritten."""
    rows, Cc = x.shape
    L = _entries()
    part = _partial(L.mlb_rmsnorm_bwd_blocks(rows) * Cc, x.device)
    rc = L.mlb_rmsnorm_bwd_cast(dx, dw, dy, x, w, rstd, NONE if add is None else add, rows, Cc, part)
    if rc == -7:
        acc = torch.zeros_like(dw, dtype=torch.float32)
        rmsnorm_bwd(dx, acc, dy, x, w, rstd, add)
        dw.copy_(acc)
        return
    _chk(rc, "rmsnorm_bwd_cast")


def colsum(out, x):
    """out[N] (bf16) = sum of x[M, N] over its rows, in fp32."""
    M, N = x.shape
    L = _entries()
    part = _partial(L.mlb_colsum_splits(M, N) * N, x.device)
    rc = L.mlb_colsum(out, x, M, N, part)
    if rc == -7:
        out.copy_(x.sum(0))
        return
    _chk(rc, "colsum")


def rmsnorm_bwd(dx, dw, dy, x, w, rstd, add=None):
    rows, Cc = x.shape
    L = _entries()
    blocks = L.mlb_rmsnorm_bwd_blocks(rows)
    # 32 words of tickets, zero between calls, then the partial sums
    ws = scratch("rms_bwd", 32 + (blocks + 16) * Cc, torch.float32, x.device, zero=True)
    _chk(L.mlb_rmsnorm_bwd(dx, dw, dy, x, w, rstd, NONE if add is None else add, rows, Cc, ws, NONE), "rmsnorm_bwd")


# ------------------------------------------------------------------ rope / swiglu / CE / AdamW
def rope_fwd(qkv, cos, sin, B, T, H, hd):
    _chk(_entries().mlb_rope(qkv, cos, sin, B * T, T, H, hd, 1.0), "rope_fwd")


def _heads(name, full, grouped, B, T, H, hd, Hkv):
    """Both tensors hold what the kernels will read and write of them."""
    if Hkv < 1 or H % Hkv or full.numel() != B * T * 3 * H * hd or grouped.numel() != B * T * (H + 2 * Hkv) * hd:
        raise ValueError(f"{name}: {tuple(full.shape)} and {tuple(grouped.shape)} are not {B * T} rows of {H} + 2 x {Hkv} heads of {hd}")


def rope_copy(out, qkv, cos, sin, B, T, H, hd, Hkv=None):
    _heads("rope_copy", out, qkv, B, T, H, hd, H if Hkv is None else Hkv)
    rc = _entries().mlb_rope_copy(out, qkv, cos, sin, B * T, T, H, H if Hkv is None else Hkv, hd)
    if rc == -7:      # a head size or alignment that kernel does not take: heads laid out first, then rotated in place
        N, rep = B * T, 1 if Hkv is None else H // Hkv
        o, x = out.view(N, 3 * H, hd), qkv.view(N, -1, hd)
        o[:, :H] = x[:, :H]
        o[:, H:] = x[:, H:].repeat_interleave(rep, 1)
        return rope_fwd(out, cos, sin, B, T, H, hd)
    _chk(rc, "rope_copy")


def kv_group_sum(out, dqkv, B, T, H, hd, Hkv):
    _heads("kv_group_sum", dqkv, out, B, T, H, hd, Hkv)
    rc = _entries().mlb_kv_group_sum(out, dqkv, B * T, H, Hkv, hd)
    if rc == -7:
        o, x = out.view(B * T, -1, hd), dqkv.view(B * T, 3 * H, hd)
        o[:, :H] = x[:, :H]
        o[:, H:] = x[:, H:].reshape(B * T, 2 * Hkv, H // Hkv, hd).sum(2)
        return
    _chk(rc, "kv_group_sum")


def rope_bwd(dqkv, cos, sin, B, T, H, hd):
    _chk(_entries().mlb_rope(dqkv, cos, sin, B * T, T, H, hd, -1.0), "rope_bwd")


def swiglu_fwd(out, gu):
    rows, I2 = gu.shape
    _chk(_entries().mlb_swiglu_fwd(out, gu, rows, I2 // 2), "swiglu_fwd")


def swiglu_bwd(dgu, dout, gu):
    rows, I2 = gu.shape
    _chk(_entries().mlb_swiglu_bwd(dgu, dout, gu, rows, I2 // 2), "swiglu_bwd")


def ce_fwd_bwd(losses, logits, tgt, dscale, V_valid=None, threads=512):
    rows, V = logits.shape
    _chk(_entries().mlb_ce_fwd_bwd(losses, logits, tgt, rows, V if V_valid is None else V_valid, logits.stride(0),
                              dscale, threads), "ce_fwd_bwd")


def ce_mean(loss, losses, dlogits, logits, tgt):
    rows, V = logits.shape
    if rows == 0:
        return loss.zero_()
    stats = torch.empty(2, dtype=torch.float32, device=logits.device)
    d = NONE if dlogits is None else dlogits
    rc = _entries().mlb_ce_mean(loss, losses, stats, d, logits, tgt, rows, V)
    if rc == -7:      # misaligned rows: through an aligned copy
        work = logits.clone() if dlogits is None else dlogits.copy_(logits)
        rc = _entries().mlb_ce_mean(loss, losses, stats, NONE if dlogits is None else work, work, tgt, rows, V)
    _chk(rc, "ce_mean")


def scale_dev(out, x, s):
    _chk(_entries().mlb_scale_dev(out, x, s, out.numel()), "scale_dev")


def ce_chunk_stats(rowmax, rowsum, tgt_logit, chunk, tgt, off):
    rows, n = chunk.shape
    _chk(lib().mlb_ce_chunk_stats(_f(rowmax), _f(rowsum), _f(tgt_logit), _b(chunk), _i(tgt), rows, n, chunk.stride(0), off, _st()),
         "ce_chunk_stats")


def ce_chunk_grad(losses, chunk, tgt, rowmax, rowsum, tgt_logit, off, dscale):
    rows, n = chunk.shape
    _chk(lib().mlb_ce_chunk_grad(_f(losses), _b(chunk), _i(tgt), _f(rowmax), _f(rowsum), _f(tgt_logit), rows, n, chunk.stride(0),
                                 off, dscale, _st()), "ce_chunk_grad")


def adamw(master, params, grads, m, v, lr, b1, b2, eps, wd, bc1, bc2, grad_scale=1.0, dev_hyper=None):
    """dev_hyper: optional CUDA fp32[4] = {lr, 1/bc1, 1/bc2, grad_scale} read by the kernel instead of the scalar
    arguments (lets a captured graph follow the optimizer step count)."""
    n = master.numel()
    pp = NONE if (params is None or params.data_ptr() == master.data_ptr()) else params
    hp = NONE if dev_hyper is None else dev_hyper
    _chk(_entries().mlb_adamw(master, pp, grads, m, v, n, lr, b1, b2, eps, wd, bc1, bc2, grad_scale, hp), "adamw")


# ------------------------------------------------------------------ vision / utilities
def patchify(out, pixels, patch):
    B, Cin, Hh, Ww = pixels.shape
    _chk(lib().mlb_patchify(_b(out), _f(pixels), B, Cin, Hh, Ww, patch, _st()), "patchify")


def add_posembed(x, pos, n_patch):
    NP, vC = x.shape
    _chk(lib().mlb_add_posembed(_b(x), _b(pos), NP, n_patch, vC, _st()), "add_posembed")


def posembed_grad(dpos, dx, n_patch):
    NP, vC = dx.shape
    _chk(lib().mlb_posembed_grad(_f(dpos), _b(dx), NP, n_patch, vC, _st()), "posembed_grad")


def residual_add(out, a, b):
    _chk(lib().mlb_residual_add(_b(out), _b(a), _b(b), out.numel(), _st()), "residual_add")


def cast(out, x, scale=1.0):
    n = out.numel()
    if out.dtype == torch.bfloat16 and x.dtype == torch.float32:
        _chk(lib().mlb_cast_f2b(_b(out), _f(x), n, scale, _st()), "cast_f2b")
    elif out.dtype == torch.float32 and x.dtype == torch.bfloat16:
        _chk(lib().mlb_cast_b2f(_f(out), _b(x), n, scale, _st()), "cast_b2f")
    else:
        raise TypeError(f"cast {x.dtype} -> {out.dtype} is not a kernel of this library")


# ------------------------------------------------------------------ 8-bit forward (E4M3 storage, tcgen05 kind::f8f6f4)
def _u8(t, name="tensor"):
    assert t.is_cuda and t.dtype == torch.uint8 and t.is_contiguous(), f"{name}: expected contiguous CUDA uint8 (E4M3 bytes)"
    return t.data_ptr()


def linear_fwd_fp8(out, x8, W8, out_scale):
    """out[M,N] (bf16) = out_scale * x8 . W8^T with E4M3 operands.  Returns False when the shape does not take the
    8-bit tensor-core path (nothing was launched)."""
    M, K = x8.shape
    N = W8.shape[0]
    fn = _entries().mlb_linear_fwd_fp8
    rc = fn(out, x8, W8, M, N, K, out.stride(0), x8.stride(0), W8.stride(0), out_scale)
    if rc == -7:
        return False
    _chk(rc, "linear_fwd_fp8")
    return True


def linear_fwd_fp8_rope(out, x8, W8, out_scale, cos, sin, T, rope_cols):
    M, K = x8.shape
    N = W8.shape[0]
    fn = lib().mlb_linear_fwd_fp8_rope
    rc = fn(_b(out), _u8(x8), _u8(W8), M, N, K, out.stride(0), x8.stride(0), W8.stride(0), out_scale, _f(cos), _f(sin), T, rope_cols, _st())
    if rc == -7:
        return False
    _chk(rc, "linear_fwd_fp8_rope")
    return True


def linear_fwd_fp8_swiglu(gu, sw, x8, W8, out_scale):
    M, K = x8.shape
    I = sw.shape[1]
    if W8.shape[0] != 2 * I or gu.shape[1] != 2 * I or sw.stride(0) != I:
        return False
    fn = lib().mlb_linear_fwd_fp8_swiglu
    rc = fn(_b(gu), _b(sw), _u8(x8), _u8(W8), M, I, K, gu.stride(0), x8.stride(0), W8.stride(0), out_scale, _st())
    if rc == -7:
        return False
    _chk(rc, "linear_fwd_fp8_swiglu")
    return True


def rmsnorm_fwd_fp8(out, out8, rstd, x, w, eps, scale):
    rows, Cc = x.shape
    fn = _entries().mlb_rmsnorm_fwd_fp8
    _chk(fn(out, out8, rstd, x, w, rows, Cc, eps, scale), "rmsnorm_fwd_fp8")


def add_rmsnorm_fwd_fp8(resid, out, out8, rstd, a, b, w, eps, scale):
    rows, Cc = a.shape
    fn = lib().mlb_add_rmsnorm_fwd_fp8
    _chk(fn(_b(resid), _b(out), _u8(out8), _f(rstd), _b(a), _b(b), _b(w), rows, Cc, eps, scale, _st()), "add_rmsnorm_fwd_fp8")


def swiglu_fwd_fp8(out, out8, gu, scale):
    rows, I2 = gu.shape
    fn = _entries().mlb_swiglu_fwd_fp8
    _chk(fn(out, out8, gu, rows, I2 // 2, scale), "swiglu_fwd_fp8")


def cast_bf16_fp8(out8, x, scale):
    fn = lib().mlb_cast_bf16_fp8
    _chk(fn(_u8(out8), _b(x), x.numel(), scale, _st()), "cast_bf16_fp8")


def adamw_fp8(master, params, params8, grads, m, v, lr, b1, b2, eps, wd, bc1, bc2, grad_scale, w_scale, dev_hyper=None):
    """AdamW that also writes the E4M3 copy of the updated weights (x w_scale) the 8-bit forward reads."""
    fn = lib().mlb_adamw_fp8
    hp = _f(dev_hyper) if dev_hyper is not None else None
    _chk(fn(_f(master), _b(params), _u8(params8), _f(grads), _f(m), _f(v), master.numel(), lr, b1, b2, eps, wd, bc1, bc2, grad_scale,
            w_scale, hp, _st()), "adamw_fp8")


def fp8_qdq(out, x, scale=1.0):
    _chk(lib().mlb_fp8_qdq(_b(out), _b(x), x.numel(), scale, _st()), "fp8_qdq")


def sum_scale(out, x, scale):
    """out[0] = scale * sum(x) on the device (x fp32, contiguous)."""
    fn = _entries().mlb_sum_scale
    _chk(fn(out, x, x.numel(), scale), "sum_scale")


def zero_(x):
    fn = _entries().mlb_zero
    assert x.is_cuda and x.is_contiguous()
    _chk(fn(Address(x.data_ptr()), x.numel() * x.element_size()), "zero")
    global LAUNCHES
    LAUNCHES -= 1          # a memset node, not a kernel of this library: not part of the launch count


def scale_(x, s):
    _chk(lib().mlb_scale_f32(_f(x), x.numel(), s, _st()), "scale_f32")
