"""Host-side mirror of nanochat-cpp's MXFP8 Linear interface over libmxb200.so.

Same names, argument meaning and error behaviour as the reference's fp8.h / mx_gemm.h (file:line cited per
function, paths within nanochat-cpp), with torch tensors used only as owners of device memory. Every call
goes to the CUDA library through the C ABI; nothing here computes on the CPU and nothing falls back. The functions a
model calls per layer (Linear, q/k/v, MLP, loss, residual step, weight refresh) run their host side in
csrc/torch_engine.cpp; the single-kernel ones below go through ctypes.
"""
from __future__ import annotations

import ctypes
import enum
from dataclasses import dataclass
from typing import List, Optional, Sequence

import torch

from . import capi
from .capi import MxOut, check, lib
from . import _torch_engine as native  # after capi, which builds and loads libmxb200.so

__all__ = [
    "Fp8Tensor", "Fp8WeightCache", "MxGemmBackend", "set_mx_gemm_backend", "mx_gemm_backend", "mx_fits",
    "empty_mx", "empty_mx_scale", "mx_out", "mx_outs", "quantize_mx", "quantize_mx_into", "quantize_mx_batch_into",
    "quantize_mx_relu_square_bwd", "residual_norm_mx", "residual_norm_mx_fits", "quantize_fp8_weight", "mx_qkv_weights", "mx_gemm", "mx_gemm_out",
    "mx_gemm_f32", "mx_gemm_relu_square", "mx_gemm_relu_square_bwd", "mx_grad_direct", "mx_grad_weights", "fp8_matmul", "fp8_qkv", "fp8_relu_square_mlp", "relu_square_mlp_mx", "fp8_eligible",
    "softcap_ce_loss", "softcap_ce_grad_mx", "softcap_cross_entropy",
    "SCALE_REFERENCE", "SCALE_OCP_FLOOR",
]

SCALE_REFERENCE = capi.SCALE_REFERENCE
SCALE_OCP_FLOOR = capi.SCALE_OCP_FLOOR
E4M3 = torch.float8_e4m3fn
E8M0 = torch.float8_e8m0fnu


class MxGemmBackend(enum.Enum):
    """src/nanochat/model/fp8/mx_gemm.h:9 has {Cublas, Cutlass}; this library is the third value a
    ``--gemm=b200`` flag would select. It is the only one implemented here."""
    B200 = "b200"


_backend = MxGemmBackend.B200


def set_mx_gemm_backend(backend: MxGemmBackend) -> None:
    """src/nanochat/model/fp8/mx_gemm.cpp:134-136. Anything but B200 raises: there is no other backend."""
    global _backend
    if backend is not MxGemmBackend.B200:
        raise ValueError("only MxGemmBackend.B200 exists in this library")
    _backend = backend


def mx_gemm_backend() -> MxGemmBackend:
    return _backend


@dataclass
class Fp8Tensor:
    """A quantized 2-D tensor: data (R, C) scaled along its rows, data_t (C, R) scaled along its own rows,
    swizzled E8M0 scales for each (src/nanochat/model/fp8/fp8.h:68-77)."""
    data: Optional[torch.Tensor] = None
    data_t: Optional[torch.Tensor] = None
    inv_scale: Optional[torch.Tensor] = None
    inv_scale_t: Optional[torch.Tensor] = None


def mx_fits(rows: int, cols: int) -> bool:
    """src/nanochat/model/fp8/fp8.h:86-88."""
    return rows % 128 == 0 and cols % 128 == 0


def fp8_eligible(in_features: int, out_features: int) -> bool:
    """src/nanochat/model/fp8/fp8.h:127-130."""
    return in_features % 16 == 0 and out_features % 16 == 0 and min(in_features, out_features) >= 128


def _stream() -> int:
    return torch.cuda.current_stream().cuda_stream


def _require_cuda(t: torch.Tensor, what: str) -> None:
    if not t.is_cuda:
        raise RuntimeError(f"{what}: expected a CUDA tensor; this engine has no CPU path")


def empty_mx_scale(rows: int, cols: int, device) -> torch.Tensor:
    """src/nanochat/model/fp8/fp8.cpp:113-115."""
    return torch.empty(rows * cols // 32, dtype=E8M0, device=device)


def empty_mx(R: int, C: int, device, rows: bool = True, cols: bool = True) -> Fp8Tensor:
    """src/nanochat/model/fp8/fp8.cpp:122-133."""
    q = Fp8Tensor()
    if rows:
        q.data = torch.empty((R, C), dtype=E4M3, device=device)
        q.inv_scale = empty_mx_scale(R, C, device)
    if cols:
        q.data_t = torch.empty((C, R), dtype=E4M3, device=device)
        q.inv_scale_t = empty_mx_scale(C, R, device)
    return q


def mx_out(data: torch.Tensor, scale: torch.Tensor, row: int = 0, col: int = 0) -> MxOut:
    """The kernels' view of MX data (R, ld) from (row, col) on; row, col % 128 == 0
    (src/nanochat/model/fp8/fp8.cpp:117-120)."""
    if row % 128 or col % 128:
        raise RuntimeError("mx_out: row and col must be multiples of 128")
    ld = data.size(1)
    tiles = ld // 128
    return MxOut(data.data_ptr() + row * ld + col, ld, scale.data_ptr() + ((row // 128) * tiles + col // 128) * 512, tiles)


def mx_outs(q: Fp8Tensor):
    """src/nanochat/model/fp8/fp8.cpp:135-142."""
    out = mx_out(q.data, q.inv_scale) if q.data is not None else MxOut(None, 0, None, 0)
    out_t = mx_out(q.data_t, q.inv_scale_t) if q.data_t is not None else MxOut(None, 0, None, 0)
    return out, out_t


def quantize_mx_into(x: torch.Tensor, relu_square: bool, out: MxOut, out_t: MxOut,
                     scale_rule: int = SCALE_REFERENCE) -> None:
    """quantize_mx of x into given buffers (src/nanochat/model/fp8/fp8.cpp:144-153)."""
    _require_cuda(x, "quantize_mx")
    if not (x.dim() == 2 and x.is_contiguous() and mx_fits(x.size(0), x.size(1))
            and x.dtype in (torch.bfloat16, torch.float32) and (not relu_square or x.dtype == torch.bfloat16)):
        raise RuntimeError("MX: expected an aligned, contiguous 2D tensor with dims % 128")
    check(lib.mxb200_quantize_mx(x.data_ptr(), int(x.dtype == torch.bfloat16), x.size(0), x.size(1), out, out_t,
                                 capi.PROLOGUE_RELU_SQUARE if relu_square else capi.PROLOGUE_NONE, scale_rule,
                                 _stream()), "quantize_mx")


def quantize_mx_batch_into(jobs: Sequence[tuple], scale_rule: int = SCALE_REFERENCE) -> None:
    """quantize_mx_into(x, False, out, out_t) for every (x, out, out_t) of jobs, all bf16 or all fp32, in as few
    launches as possible: the same bytes as one call each. For runs of small tensors, e.g. the parts of the merged
    q/k/v weight (src/nanochat/model/fp8/fp8.cpp:155-171) or a model's weights after an optimizer step."""
    native.quantize_mx_batch_into(jobs, scale_rule)


def quantize_mx(x: torch.Tensor, rows: bool = True, cols: bool = True, relu_square: bool = False,
                scale_rule: int = SCALE_REFERENCE) -> Fp8Tensor:
    """MXFP8 E4M3 of a contiguous 2-D bf16 or fp32 x (src/nanochat/model/fp8/fp8.h:82-84,
    fp8.cpp:538-549)."""
    _require_cuda(x, "quantize_mx")
    q = empty_mx(x.size(0), x.size(1), x.device, rows, cols)
    out, out_t = mx_outs(q)
    quantize_mx_into(x, relu_square, out, out_t, scale_rule)
    return q


def quantize_mx_relu_square_bwd(g: torch.Tensor, h: torch.Tensor, rows: bool = True, cols: bool = True,
                                scale_rule: int = SCALE_REFERENCE) -> Fp8Tensor:
    """MX of dh = bf16(h > 0 ? g * 2h : 0) without writing dh
    (src/nanochat/model/fp8/fp8_kernel.h:41-43; caller fp8.cpp:318-323)."""
    _require_cuda(g, "quantize_mx_relu_square_bwd")
    if not (g.shape == h.shape and g.dtype == h.dtype == torch.bfloat16 and g.is_contiguous() and h.is_contiguous()
            and mx_fits(g.size(0), g.size(1))):
        raise RuntimeError("MX: expected two contiguous bf16 2D tensors of one shape with dims % 128")
    q = empty_mx(g.size(0), g.size(1), g.device, rows, cols)
    out, out_t = mx_outs(q)
    check(lib.mxb200_quantize_mx_relu_square_bwd(g.data_ptr(), h.data_ptr(), g.size(0), g.size(1), out, out_t,
                                                 scale_rule, _stream()), "quantize_mx_relu_square_bwd")
    return q


def residual_norm_mx_fits(rows: int, cols: int) -> bool:
    """Whether residual_norm_mx handles (rows, cols): both % 128 and cols within the kernel's row-in-registers limit
    (the reference's is 1536, src/nanochat/model/ops/residual_norm_kernel.h:15; this kernel's is 2048)."""
    return mx_fits(rows, cols) and cols <= 2048


def residual_norm_mx(x: torch.Tensor, r: Optional[torch.Tensor] = None, x0: Optional[torch.Tensor] = None,
                     lr: Optional[torch.Tensor] = None, l0: Optional[torch.Tensor] = None, layer: int = 0,
                     gate_cols: int = 0, eps: float = torch.finfo(torch.float32).eps, out: Optional[tuple] = None):
    """Forward of the reference's fused residual step with MX output (src/nanochat/model/ops/residual_norm.cpp:36-96,
    the `mx` branch): s = x + r, res = lr[layer] * s + l0[layer] * x0 (with the op path's bf16 roundings),
    n = rms_norm(res). Returns (res, n, n_mx, rstd, s): n holds only its first gate_cols columns; n_mx is
    quantize_mx(n) in both layouts, bit for bit; s is None unless both r and x0 are given. out: a tuple this function
    returned earlier for the same shapes and inputs present, whose buffers are written again instead of new ones."""
    _require_cuda(x, "residual_norm_mx")
    cols = x.size(-1)
    rows = x.numel() // cols
    if not (x.dtype == torch.bfloat16 and x.is_contiguous() and residual_norm_mx_fits(rows, cols)
            and 0 <= gate_cols <= cols):
        raise RuntimeError("residual_norm_mx: shape")
    for t in (r, x0):
        if t is not None and not (t.dtype == torch.bfloat16 and t.is_contiguous() and t.shape == x.shape):
            raise RuntimeError("residual_norm_mx: expected contiguous bf16 of x's shape")
    blend = x0 is not None
    if blend and not (lr is not None and l0 is not None and lr.dtype == l0.dtype == torch.float32
                      and 0 <= layer < lr.numel() == l0.numel() and lr.is_contiguous() and l0.is_contiguous()):
        raise RuntimeError("residual_norm_mx: the blend needs fp32 lambdas")
    if out is None:
        res, n, data, data_t, scale, scale_t, rstd, s = native.residual_norm_mx(x, r, x0, lr, l0, layer, gate_cols, eps)
        return res, n, Fp8Tensor(data, data_t, scale, scale_t), rstd, s
    res, n, n_mx, rstd, s = out
    if not (res.shape == x.shape and n.shape == x.shape and rstd.numel() == rows and n_mx.data.shape == (rows, cols)
            and (s is not None) == (r is not None and blend)):
        raise RuntimeError("residual_norm_mx: out does not match")
    out, out_t = mx_outs(n_mx)
    args = capi.ResidualNormMx(x.data_ptr(), r.data_ptr() if r is not None else None,
                               x0.data_ptr() if blend else None,
                               lr.data_ptr() + 4 * layer if blend else None, l0.data_ptr() + 4 * layer if blend else None,
                               s.data_ptr() if s is not None else None, res.data_ptr(), n.data_ptr(), rstd.data_ptr(),
                               rows, cols, eps, out, out_t, gate_cols)
    check(lib.mxb200_residual_norm_mx_fwd(ctypes.byref(args), _stream()), "residual_norm_mx")
    return res, n, n_mx, rstd, s


class Fp8WeightCache(native.WeightCache):
    """FP8 copies of weights, remade only when a weight changes: in-place updates bump the tensor's version
    (src/nanochat/model/fp8/fp8.h:18-38, fp8.cpp:516-536). `get(kind, weights, make)` returns make()'s list, kept while
    `enabled` and until another kind or weight is asked for."""

    def __init__(self, enabled: bool = False):
        super().__init__(enabled)

    def __reduce__(self):  # a copy starts empty
        return type(self), (self.enabled,), vars(self) or None


def _weight_source(cache, *weights):
    """What the native functions take for the quantized copy of (merged) weights: None or the native cache itself, or the
    four tensors that the get() of any other cache, or of a subclass, returns."""
    if cache is None or getattr(type(cache), "get", None) is native.WeightCache.get:
        return cache
    if len(weights) == 3:
        return list(mx_qkv_weights(*weights, cache))
    return _mx_list(quantize_fp8_weight(*weights, cache))


def quantize_fp8_weight(w: torch.Tensor, cache: Optional[Fp8WeightCache] = None) -> Fp8Tensor:
    """A weight's E4M3 copy under MX, from cache while w is unchanged
    (src/nanochat/model/fp8/fp8.cpp:551-558)."""
    def make():
        q = quantize_mx(w.detach().contiguous())
        return [q.data, q.data_t, q.inv_scale, q.inv_scale_t]
    v = cache.get(1, [w], make) if cache is not None else make()
    return Fp8Tensor(v[0], v[1], v[2], v[3])


def mx_qkv_weights(wq: torch.Tensor, wk: torch.Tensor, wv: torch.Tensor, cache: Optional[Fp8WeightCache] = None):
    """Merged q/k/v weights: {w_cat (n, C), w_cat^T (C, n), their scales}; each part quantized into its row
    range of one buffer (src/nanochat/model/fp8/fp8.cpp:155-171)."""
    C = wq.size(1)
    n = wq.size(0) + wk.size(0) + wv.size(0)

    def make():
        out = [torch.empty((n, C), dtype=E4M3, device=wq.device), torch.empty((C, n), dtype=E4M3, device=wq.device),
               empty_mx_scale(n, C, wq.device), empty_mx_scale(C, n, wq.device)]
        row, jobs = 0, []
        for w in (wq, wk, wv):
            if w.size(1) != C:
                raise RuntimeError("q/k/v weights must share the input dim")
            jobs.append((w.detach().contiguous(), mx_out(out[0], out[2], row, 0), mx_out(out[1], out[3], 0, row)))
            row += w.size(0)
        if len({j[0].dtype for j in jobs}) == 1:
            quantize_mx_batch_into(jobs)  # the three parts in one launch
        else:
            for x, o, o_t in jobs:
                quantize_mx_into(x, False, o, o_t)
        return out
    return cache.get(1, [wq, wk, wv], make) if cache is not None else make()


# ------------------------------------------------------------------------------------------------ GEMMs

_workspaces: dict = {}


def _workspace(device, nbytes: int) -> torch.Tensor:
    """Split-K scratch, grown on demand and kept per (device, stream): split-K GEMMs on different streams may
    overlap on the GPU and must not share their K slices, while launches on one stream are ordered
    and reuse theirs (the reference's cuBLASLt path likewise borrows torch's per-stream workspace,
    src/nanochat/model/fp8/mx_gemm.cpp:236-237). A replaced tensor is handed back to the caching allocator, which
    keeps it for the stream it was allocated on until that stream's queued work has run."""
    index = device.index if device.index is not None else torch.cuda.current_device()
    key = (index, torch.cuda.current_stream(index).cuda_stream)
    ws = _workspaces.get(key)
    if ws is None or ws.numel() < nbytes:
        ws = torch.empty(max(nbytes, 1 << 20), dtype=torch.uint8, device=device)
        _workspaces[key] = ws
    return ws


def _check_operands(a, a_scale, b, b_scale, what):
    for t in (a, a_scale, b, b_scale):
        _require_cuda(t, what)
    if not (a.dim() == 2 and b.dim() == 2 and a.is_contiguous() and b.is_contiguous() and a.dtype == E4M3
            and b.dtype == E4M3 and a.size(1) == b.size(1)):
        raise RuntimeError(f"{what}: shape mismatch")
    M, N, K = a.size(0), b.size(0), a.size(1)
    if a_scale.numel() != M * K // 32 or b_scale.numel() != N * K // 32:
        raise RuntimeError(f"{what}: expected e4m3 operands with their MX scales")
    return M, N, K


def mx_gemm_out(out: torch.Tensor, a: torch.Tensor, a_scale: torch.Tensor, b: torch.Tensor, b_scale: torch.Tensor,
                resid: Optional[torch.Tensor] = None, splits: Optional[int] = None) -> None:
    """mx_gemm into out, bf16 or fp32 (src/nanochat/model/fp8/mx_gemm.h:26-27, mx_gemm.cpp:164-173).
    resid: optional bf16 (M, N) residual fused into the bf16 epilogue. splits: None lets the library decide."""
    M, N, K = _check_operands(a, a_scale, b, b_scale, "mx_gemm")
    if not (out.is_contiguous() and out.size(0) == M and out.size(1) == N and out.dtype in (torch.bfloat16, torch.float32)):
        raise RuntimeError("mx_gemm: shape mismatch")
    kind = capi.OUT_BF16 if out.dtype == torch.bfloat16 else capi.OUT_F32
    if resid is not None and not (kind == capi.OUT_BF16 and resid.shape == out.shape and resid.dtype == torch.bfloat16
                                  and resid.is_contiguous()):
        raise RuntimeError("mx_gemm: the residual must be a contiguous bf16 tensor of the output's shape")
    s = lib.mxb200_gemm_splits(M, N, K) if splits is None else splits
    rp = resid.data_ptr() if resid is not None else None
    if s <= 1:
        if kind == capi.OUT_BF16:
            st = lib.mxb200_gemm_bf16(a.data_ptr(), a_scale.data_ptr(), b.data_ptr(), b_scale.data_ptr(), out.data_ptr(),
                                      rp, M, N, K, _stream())
        else:
            st = lib.mxb200_gemm_f32(a.data_ptr(), a_scale.data_ptr(), b.data_ptr(), b_scale.data_ptr(), out.data_ptr(),
                                     M, N, K, None, 0, _stream())
    else:
        nbytes = lib.mxb200_gemm_workspace_bytes(M, N, K, s)
        ws = _workspace(out.device, nbytes)
        st = lib.mxb200_gemm_splitk(a.data_ptr(), a_scale.data_ptr(), b.data_ptr(), b_scale.data_ptr(), out.data_ptr(),
                                    kind, rp, M, N, K, None, 0, s, ws.data_ptr(), ws.numel(), _stream())
    check(st, "mx_gemm")


def mx_gemm(a: torch.Tensor, a_scale: torch.Tensor, b: torch.Tensor, b_scale: torch.Tensor,
            out_dtype: torch.dtype = torch.bfloat16, resid: Optional[torch.Tensor] = None,
            splits: Optional[int] = None) -> torch.Tensor:
    """a (M, K) . b (N, K)^T as out_dtype (src/nanochat/model/fp8/mx_gemm.h:18-24, mx_gemm.cpp:154-162)."""
    out = torch.empty((a.size(0), b.size(0)), dtype=out_dtype, device=a.device)
    mx_gemm_out(out, a, a_scale, b, b_scale, resid, splits)
    return out


def mx_gemm_f32(a: torch.Tensor, a_scale: torch.Tensor, b: torch.Tensor, b_scale: torch.Tensor, out: torch.Tensor,
                accumulate: bool, alpha: Optional[torch.Tensor] = None, splits: Optional[int] = None) -> None:
    """out (M, N) fp32 (+)= alpha * a . b^T; alpha a device fp32 scalar (None: 1)
    (src/nanochat/model/fp8/mx_gemm.h:44-50, mx_gemm.cpp:214-319)."""
    M, N, K = _check_operands(a, a_scale, b, b_scale, "mx_gemm_f32")
    if not (out.is_cuda and out.is_contiguous() and out.dtype == torch.float32 and out.size(0) == M and out.size(1) == N):
        raise RuntimeError("mx_gemm_f32: expected a contiguous fp32 (M, N) output")
    if alpha is not None and not (alpha.is_cuda and alpha.dtype == torch.float32 and alpha.numel() == 1):
        raise RuntimeError("mx_gemm_f32: alpha must be a device fp32 scalar")
    ap = alpha.data_ptr() if alpha is not None else None
    s = lib.mxb200_gemm_splits(M, N, K) if splits is None else splits
    if s <= 1:
        st = lib.mxb200_gemm_f32(a.data_ptr(), a_scale.data_ptr(), b.data_ptr(), b_scale.data_ptr(), out.data_ptr(),
                                 M, N, K, ap, int(accumulate), _stream())
    else:
        nbytes = lib.mxb200_gemm_workspace_bytes(M, N, K, s)
        ws = _workspace(out.device, nbytes)
        st = lib.mxb200_gemm_splitk(a.data_ptr(), a_scale.data_ptr(), b.data_ptr(), b_scale.data_ptr(), out.data_ptr(),
                                    capi.OUT_F32, None, M, N, K, ap, int(accumulate), s, ws.data_ptr(), ws.numel(),
                                    _stream())
    check(st, "mx_gemm_f32")


def _check_mx_out(t: torch.Tensor, scale: torch.Tensor, rows: int, cols: int, what: str) -> None:
    """src/nanochat/model/fp8/mx_gemm.cpp:125-130."""
    if not (t.is_cuda and t.is_contiguous() and t.dtype == E4M3 and t.size(0) == rows and t.size(1) == cols
            and scale.numel() == rows * cols // 32):
        raise RuntimeError(f"{what}: expected e4m3 ({rows}, {cols}) with its MX scales")


def mx_gemm_relu_square(h: torch.Tensor, q: torch.Tensor, q_scale: torch.Tensor, q_t: torch.Tensor,
                        q_t_scale: torch.Tensor, a: torch.Tensor, a_scale: torch.Tensor, b: torch.Tensor,
                        b_scale: torch.Tensor) -> bool:
    """h = mx_gemm(a, ..., bf16) into h and q = quantize_mx(h, True, True, True) into q, q_t (N, M) in one GEMM
    (src/nanochat/model/fp8/mx_gemm.h:29-35, mx_gemm.cpp:175-192). Returns True, as the reference does when its
    fused backend applies; there is no unfused fallback to report here."""
    M, N, K = _check_operands(a, a_scale, b, b_scale, "mx_gemm_relu_square")
    if not (h.is_cuda and h.is_contiguous() and h.dtype == torch.bfloat16 and h.size(0) == M and h.size(1) == N):
        raise RuntimeError("mx_gemm_relu_square: shape mismatch")
    _check_mx_out(q, q_scale, M, N, "mx_gemm_relu_square")
    _check_mx_out(q_t, q_t_scale, N, M, "mx_gemm_relu_square")
    check(lib.mxb200_gemm_relu_square(a.data_ptr(), a_scale.data_ptr(), b.data_ptr(), b_scale.data_ptr(), h.data_ptr(),
                                      q.data_ptr(), q_scale.data_ptr(), q_t.data_ptr(), q_t_scale.data_ptr(), M, N, K,
                                      _stream()), "mx_gemm_relu_square")
    return True


def mx_gemm_relu_square_bwd(a: torch.Tensor, a_scale: torch.Tensor, b: torch.Tensor, b_scale: torch.Tensor,
                            h: torch.Tensor, dh: torch.Tensor, dh_scale: torch.Tensor, dh_t: torch.Tensor,
                            dh_t_scale: torch.Tensor) -> bool:
    """relu^2's backward from its dgrad GEMM in one GEMM: ga = mx_gemm(a, ..., bf16) (not written) and h (M, N) bf16
    -> quantize_mx_relu_square_bwd's outputs (src/nanochat/model/fp8/mx_gemm.h:37-42, mx_gemm.cpp:194-212)."""
    M, N, K = _check_operands(a, a_scale, b, b_scale, "mx_gemm_relu_square_bwd")
    if not (h.is_cuda and h.is_contiguous() and h.dtype == torch.bfloat16 and h.size(0) == M and h.size(1) == N):
        raise RuntimeError("mx_gemm_relu_square_bwd: shape mismatch")
    _check_mx_out(dh, dh_scale, M, N, "mx_gemm_relu_square_bwd")
    _check_mx_out(dh_t, dh_t_scale, N, M, "mx_gemm_relu_square_bwd")
    check(lib.mxb200_gemm_relu_square_bwd(a.data_ptr(), a_scale.data_ptr(), b.data_ptr(), b_scale.data_ptr(),
                                          h.data_ptr(), dh.data_ptr(), dh_scale.data_ptr(), dh_t.data_ptr(),
                                          dh_t_scale.data_ptr(), M, N, K, _stream()), "mx_gemm_relu_square_bwd")
    return True


# ------------------------------------------------------------------------------------------------ Linear

def mx_grad_direct(w: torch.Tensor) -> bool:
    """Whether backward may write w's gradient straight into w.grad: a contiguous fp32 leaf that requires
    grad (src/nanochat/model/fp8/fp8.h:114-116)."""
    return w.is_leaf and w.requires_grad and w.dtype == torch.float32 and w.is_contiguous()


def mx_grad_weights(go_t: torch.Tensor, go_scale_t: torch.Tensor, in_t: torch.Tensor, in_scale_t: torch.Tensor,
                    ws: Sequence[torch.Tensor], alpha: Optional[torch.Tensor] = None) -> None:
    """dW = alpha * go_t (n, N) . in_t (C, N)^T into the .grad of ws, whose rows concatenate to n: allocated (=)
    when undefined, else accumulated (+=). Several ws share one buffer, so one GEMM serves
    (src/nanochat/model/fp8/fp8.h:118-125, fp8.cpp:470-514)."""
    n, C = go_t.size(0), in_t.size(0)
    if sum(w.size(0) for w in ws) != n or any(w.size(1) != C for w in ws):
        raise RuntimeError("mx_grad_weights: weight rows must concatenate to the gradient's")
    merged = None
    if all(w.grad is not None for w in ws):
        g0 = ws[0].grad
        base = g0.data_ptr()
        contiguous, row = True, 0
        for w in ws:
            contiguous &= w.grad.data_ptr() == base + row * C * 4 and w.grad.is_contiguous() and w.grad.dtype == torch.float32
            row += w.size(0)
        if contiguous and len(ws) > 1 and g0._base is not None and g0._base.numel() == n * C:
            merged = g0._base.view(n, C)
        elif contiguous and len(ws) == 1:
            merged = g0
    if merged is not None:
        mx_gemm_f32(go_t, go_scale_t, in_t, in_scale_t, merged, True, alpha)
        return
    buf = torch.empty((n, C), dtype=torch.float32, device=go_t.device)
    mx_gemm_f32(go_t, go_scale_t, in_t, in_scale_t, buf, False, alpha)
    row = 0
    for w in ws:
        part = buf.narrow(0, row, w.size(0))
        if w.grad is None:
            w.grad = part  # row blocks of one buffer, as the reference's merged q/k/v
        else:
            w.grad.add_(part)
        row += w.size(0)


def _mx_list(q: Optional[Fp8Tensor]):
    return None if q is None else [q.data, q.data_t, q.inv_scale, q.inv_scale_t]


def fp8_qkv(x_2d: torch.Tensor, wq: torch.Tensor, wk: torch.Tensor, wv: torch.Tensor, gate_cols: int = 0,
            cache: Optional[Fp8WeightCache] = None, x_mx: Optional[Fp8Tensor] = None):
    """Attention's c_q, c_k, c_v as fp8_matmuls of the same x_2d (N, in) bf16, merged
    (src/nanochat/model/fp8/fp8.h:58-66, MX branch). Returns (q, k, v), views of one (N, q + k + v) buffer, plus
    x_2d[:, :gate_cols] when gate_cols > 0 (the value-embedding gate's input; its gradient is added to dx in the
    same pass). x_mx: x_2d already quantized in both layouts (residual_norm_mx), as the reference's attention path
    takes it (src/nanochat/model/attention/mx_attention.h:20, mx_attention.cpp:45); x_2d then carries autograd and the
    gate's columns only."""
    if x_mx is not None and (x_mx.data is None or x_mx.data_t is None):
        raise RuntimeError("fp8_qkv: x_mx needs both layouts")
    return tuple(native.fp8_qkv(x_2d, wq, wk, wv, gate_cols, _weight_source(cache, wq, wk, wv), _mx_list(x_mx)))


def relu_square_mlp_mx(N: int, cin: int, w_fc: torch.Tensor, w_proj: torch.Tensor) -> bool:
    """Whether fp8_relu_square_mlp of an (N, in) input runs under MX: every dim % 128
    (src/nanochat/model/fp8/fp8.h:56-58)."""
    return (mx_fits(N, cin) and mx_fits(w_fc.size(0), w_fc.size(1)) and mx_fits(w_proj.size(0), w_proj.size(1))
            and w_fc.size(1) == cin and w_proj.size(1) == w_fc.size(0))


def fp8_relu_square_mlp(x_2d: torch.Tensor, w_fc: torch.Tensor, w_proj: torch.Tensor,
                        fc_cache: Optional[Fp8WeightCache] = None, proj_cache: Optional[Fp8WeightCache] = None,
                        x_mx: Optional[Fp8Tensor] = None) -> torch.Tensor:
    """The MLP's c_proj(relu(c_fc(x)).square()) with both matmuls as fp8_matmul, bit for bit as long as in and out are below
    4096, from where a GEMM may be cut into K slices but the fused ones are not (src/nanochat/model/fp8/fp8.h:46-54). x_2d (N, in) bf16, w_fc (hidden, in), w_proj (out, hidden) -> (N, out).
    x_mx: x_2d already quantized in both layouts (residual_norm_mx); x_2d then only carries autograd."""
    if x_mx is not None and (x_mx.data is None or x_mx.data_t is None):
        raise RuntimeError("fp8_relu_square_mlp: x_mx needs both layouts")
    return native.fp8_relu_square_mlp(x_2d, w_fc, w_proj, _weight_source(fc_cache, w_fc),
                                      _weight_source(proj_cache, w_proj), _mx_list(x_mx))


def fp8_matmul(input_2d: torch.Tensor, weight: torch.Tensor, cache: Optional[Fp8WeightCache] = None) -> torch.Tensor:
    """input_2d (N, in) bf16, weight (out, in) -> (N, out) bf16 under the MX recipe
    (src/nanochat/model/fp8/fp8.h:40-44, fp8.cpp:566-571). Dims must be % 128: the reference falls back to its
    tensorwise recipe otherwise, which is outside this library."""
    if cache is not None and type(cache) is not Fp8WeightCache:
        cache = _weight_source(cache, weight)
    return native.fp8_matmul(input_2d, weight, cache)


# ------------------------------------------------------------------------------------------------ chunked lm_head loss

def softcap_ce_loss(logits: torch.Tensor, targets: torch.Tensor, vocab: int, softcap: float,
                    loss: Optional[torch.Tensor] = None, lse: Optional[torch.Tensor] = None):
    """Per row of bf16 logits (rows, padded): lse of the soft-capped logits and loss = lse - capped[target]; rows with
    target < 0 get loss 0 (src/nanochat/model/ops/softcap_ce_kernel.h:13-22 with grad = false). Returns (loss, lse),
    written into the given fp32 tensors when present."""
    _require_cuda(logits, "softcap_ce_loss")
    rows, padded = logits.shape
    if not (logits.dtype == torch.bfloat16 and logits.stride(1) == 1 and targets.dtype == torch.int64
            and targets.is_contiguous() and targets.numel() == rows):
        raise RuntimeError("softcap_ce_loss: expected bf16 logits (rows, padded) and int64 targets (rows)")
    loss = torch.empty(rows, dtype=torch.float32, device=logits.device) if loss is None else loss
    lse = torch.empty(rows, dtype=torch.float32, device=logits.device) if lse is None else lse
    check(lib.mxb200_softcap_ce_loss(logits.data_ptr(), rows, logits.stride(0), targets.data_ptr(), vocab, padded,
                                     softcap, loss.data_ptr(), lse.data_ptr(), _stream()), "softcap_ce_loss")
    return loss, lse


def softcap_ce_grad_mx(logits: torch.Tensor, targets: torch.Tensor, lse: torch.Tensor, vocab: int, softcap: float,
                       out: MxOut, out_t: MxOut, grad_scale: Optional[torch.Tensor] = None,
                       num_valid: Optional[torch.Tensor] = None, scale_rule: int = SCALE_REFERENCE) -> None:
    """The loss's gradient with respect to the logits, MX-quantized (as quantize_mx of its bf16) into out / out_t
    without being written, from the logits and softcap_ce_loss's lse
    (src/nanochat/model/ops/softcap_ce_kernel.h:24-29). grad_scale: fp32 (rows) or one element (every row);
    num_valid: int64 scalar on the device that divides the scale."""
    _require_cuda(logits, "softcap_ce_grad_mx")
    rows, padded = logits.shape
    stride = 0
    if grad_scale is not None:
        if grad_scale.dtype != torch.float32 or not grad_scale.is_contiguous():
            raise RuntimeError("softcap_ce_grad_mx: grad_scale must be contiguous fp32")
        stride = 1 if grad_scale.dim() == 1 and grad_scale.numel() == rows and rows > 1 else 0
    if num_valid is not None and num_valid.dtype != torch.int64:
        raise RuntimeError("softcap_ce_grad_mx: num_valid must be int64")
    check(lib.mxb200_softcap_ce_grad_mx(logits.data_ptr(), rows, logits.stride(0), targets.data_ptr(), lse.data_ptr(),
                                        vocab, padded, softcap,
                                        grad_scale.data_ptr() if grad_scale is not None else None, stride,
                                        num_valid.data_ptr() if num_valid is not None else None, out, out_t,
                                        scale_rule, _stream()), "softcap_ce_grad_mx")


def softcap_cross_entropy(x: torch.Tensor, weight: torch.Tensor, targets: torch.Tensor, vocab_size: int,
                          softcap: float, chunk_rows: int, reduction: str = "mean",
                          cache: Optional[Fp8WeightCache] = None) -> torch.Tensor:
    """lm_head + logit softcap + cross-entropy a chunk of rows at a time under the MX recipe, so that the full
    (N, vocab) logits never exist (src/nanochat/model/ops/softcap_ce.h:16-24, recipe Mx). x: (N, C) bf16; weight:
    (V_padded, C) fp32 lm_head weight; targets: (N) int64, -1 = ignored; logits are cropped to vocab_size and capped as
    softcap * tanh(z / softcap); mean divides by the number of targets that are not ignored. MX needs N, C, chunk_rows
    and V_padded % 128 (the reference falls back to other recipes otherwise, which are outside this library)."""
    if x.dim() != 2 or targets.dim() != 1 or targets.size(0) != x.size(0):
        raise ValueError("softcap_cross_entropy expects x (N, C) and targets (N)")
    if chunk_rows < 1:
        raise ValueError("chunk_rows must be positive")
    if not x.is_cuda or x.dtype != torch.bfloat16:
        raise ValueError("softcap_cross_entropy expects bf16 CUDA activations")
    if reduction not in ("mean", "sum", "none"):
        raise ValueError("reduction must be mean, sum or none")
    if not (mx_fits(x.size(0), x.size(1)) and chunk_rows % 128 == 0 and weight.size(0) % 128 == 0
            and weight.size(0) >= vocab_size and weight.size(1) == x.size(1)):
        raise RuntimeError("softcap_cross_entropy: MX needs N, C, chunk_rows and the padded vocab % 128")
    return native.softcap_cross_entropy(x, weight, targets, int(vocab_size), float(softcap), int(chunk_rows),
                                        ("mean", "sum", "none").index(reduction), _weight_source(cache, weight))
