"""Tensor-level operator interface: one function per C entry point, same name without the
`fluke_` prefix, same argument meaning and the same error behaviour (void functions exit the
process on a bad dimension, int functions raise on a non-zero return). Inputs must be
contiguous CUDA tensors; nothing here computes on the host. The work of a call (checks, output
allocation, the C call) is done by the extension module (csrc/native_ops.cpp); what is not called
per step goes through ctypes.
"""
import ctypes

import torch

from . import lib as _lib

TX_DIMS = dict(d_model=512, dim_feedforward=2048, nhead=8, head_dim=64)


def _L():
    return _lib.load()


class _Native:
    """The extension module, loaded (and built if it is missing) at the first call of an operator."""

    def __getattr__(self, name):
        fn = getattr(_lib.native(), name)
        setattr(self, name, fn)
        return fn


_N = _Native()


def _dev(*ts):
    for t in ts:
        if t is None:
            continue
        if not t.is_cuda:
            raise RuntimeError("fluke_b200.ops needs CUDA tensors (there is no CPU fallback)")
        if not t.is_contiguous():
            raise RuntimeError("fluke_b200.ops needs contiguous tensors")


def _p(t):
    return 0 if t is None else t.data_ptr()


def _check(rc, what):
    if rc != 0:
        raise RuntimeError(f"{what} failed: rc={rc} {_L().fluke_last_error().decode()}")


def set_stream(stream=None):
    """Route later launches to `stream` (torch.cuda.Stream) or back to the legacy default stream."""
    _L().fluke_set_stream(0 if stream is None else stream.cuda_stream)


# ---- memory-bound kernels -----------------------------------------------------------------

def rmsnorm(x, residual, weight, alpha, eps, out=None):
    return _N.rmsnorm(x, residual, weight, alpha, eps, out)


def rmsnorm_quant_int8(x, weight, residual_i8, residual_scale, alpha, eps):
    """In place on (residual_i8, residual_scale)."""
    return _N.rmsnorm_quant(x, weight, residual_i8, residual_scale, alpha, eps, False)


def rmsnorm_quant_fp8(x, weight, residual_u8, residual_scale, alpha, eps):
    return _N.rmsnorm_quant(x, weight, residual_u8, residual_scale, alpha, eps, True)


def quant_int8(x, out=None, scale=None):
    return _N.quant(x, out, scale, False)


def quant_fp8(x, out=None, scale=None):
    return _N.quant(x, out, scale, True)


def dequant_transpose(x, scale, fp8=False):
    """[T,N,C] int8 / e4m3 bytes -> f16 [N,T,C]."""
    return _N.dequant_transpose(x, scale, fp8)


def rotary_emb_(x_ptr, sin, cos, batch, seq_len, n_heads, head_dim, width, sb, ss, sh):
    """In place on the f16 tensor starting at device address x_ptr (strides in elements)."""
    _N.rotary_emb(x_ptr, sin, cos, batch, seq_len, n_heads, head_dim, width, sb, ss, sh)


def rotary_qkv_(qkv, sin, cos, width):
    """Rotate the q and k chunks of qkv [N, seq, 3, heads, head_dim] in place, passing the full
    qkv strides (the call pattern of test/test_rotary_gpu.py:26-38)."""
    return _N.rotary_qkv(qkv, sin, cos, width)


def silu_mul(x):
    return _N.silu_mul(x)


def flstm_step(scratch, ih_t, cell, hh_next=None):
    return _N.flstm_step(scratch, ih_t, cell, hh_next)


# ---- fused transformer kernels ------------------------------------------------------------

def int8_select(device_index=0, max_seq=2048, **dims):
    d = dict(TX_DIMS, **dims)
    b = _L().fluke_int8_select(device_index, _lib.fluke_dims_t(d["d_model"], d["dim_feedforward"],
                                                               d["nhead"], d["head_dim"], max_seq))
    return b  # None when unsupported (the caller keeps fp16, as with the reference)


def fp8_select(device_index=0, max_seq=2048, **dims):
    d = dict(TX_DIMS, **dims)
    return _L().fluke_fp8_select(device_index, _lib.fluke_dims_t(d["d_model"], d["dim_feedforward"],
                                                                d["nhead"], d["head_dim"], max_seq))


def qkv_rotary_i8(backend, a_i8, wqkv_i8, scale_a, scale_b, sin, cos, seqlen, out=None):
    return _N.qkv_rotary(backend, a_i8, wqkv_i8, scale_a, scale_b, sin, cos, seqlen, out, 0, wqkv_i8.size(0))


def gated_mlp_i8(backend, a_i8, gate_i8, up_i8, scale_a, scale_gate, scale_up, out=None):
    return _N.gated_mlp(backend, a_i8, gate_i8, up_i8, scale_a, scale_gate, scale_up, out, 0, gate_i8.size(0))


def qkv_rotary_fp8(backend, a_fp8, w_fp8, scale_a, scale_b, sin, cos, seqlen, plain=False, out=None):
    """w_fp8: PRESHUFFLED bytes (plain=False, the reference ABI) or row-major [N,K] (plain=True)."""
    return _N.qkv_rotary(backend, a_fp8, w_fp8, scale_a, scale_b, sin, cos, seqlen, out, 2 if plain else 1,
                         3 * TX_DIMS["d_model"])


def gated_mlp_fp8(backend, a_fp8, gate_fp8, up_fp8, scale_a, scale_gate, scale_up, plain=False, out=None):
    return _N.gated_mlp(backend, a_fp8, gate_fp8, up_fp8, scale_a, scale_gate, scale_up, out, 2 if plain else 1,
                        TX_DIMS["dim_feedforward"])


# ---- base GEMMs (additive) ----------------------------------------------------------------

def gemm_i8(a_i8, b_i8, scale_a, scale_b, const_scale_a=0.0):
    return _N.gemm_i8(a_i8, b_i8, scale_a, scale_b, const_scale_a)


def gemm_i8_s32(a_i8, b_i8):
    _dev(a_i8, b_i8)
    m, k = a_i8.shape
    n = b_i8.size(0)
    out = torch.empty(m, n, dtype=torch.int32, device=a_i8.device)
    _check(_L().fluke_gemm_i8_s32_gpu(_p(out), _p(a_i8), _p(b_i8), m, n, k), "fluke_gemm_i8_s32_gpu")
    return out


def gemm_fp8(a_fp8, b_fp8_nk, scale_a, scale_b):
    return _N.gemm_fp8(a_fp8, b_fp8_nk, scale_a, scale_b)


def fp8_unshuffle(w_preshuffled, n, k):
    _dev(w_preshuffled)
    out = torch.empty(n, k, dtype=torch.uint8, device=w_preshuffled.device)
    _check(_L().fluke_fp8_unshuffle_gpu(_p(out), _p(w_preshuffled), n, k), "fluke_fp8_unshuffle_gpu")
    return out


# ---- factored LSTM (additive) ---------------------------------------------------------------

def down_proj_i8(a_i8, w_i8, scale_a, scale_b, out=None):
    """f16 [M,N] = int8 GEMM * (sa*sb); scale_a None = the fixed 1/127 of an int8 hidden state."""
    return _N.down_proj(a_i8, w_i8, scale_a, scale_b, out, False)


def down_proj_fp8(a_fp8, w_fp8_nk, scale_a, scale_b, out=None):
    """f16 [M,N] = (e4m3 GEMM * sa[m]) * sb[n]; a_fp8 [M,K], w_fp8_nk [N,K] as uint8 e4m3 bytes."""
    return _N.down_proj(a_fp8, w_fp8_nk, scale_a, scale_b, out, True)


def factored_lstm_step_i8(A, W4, bias4, c, h_out=None, fp8_export_name=False):
    """A f16 [B,Kc]; W4 f16 [4H,Kc] (gate-major i,f,g,o); bias4 f32 [4H]; c f32 [B,H] in place."""
    return _N.lstm_step(A, W4, bias4, c, h_out, fp8_export_name)


def factored_lstm_layer_i8(x_i8, x_scale, dn_ih, dn_ih_scale, dn_hh, dn_hh_scale, w_up, bias, c, h,
                           reverse=False, h_out=None, workspace=None, phase_mask=7):
    """One layer over x_i8 [T,B,H]; c (f32 [B,H]) and h (int8 [B,H]) are state, updated in place.
    phase_mask != 7 launches only some kernel classes (timing aid, see fluke.h)."""
    _dev(x_i8, x_scale, dn_ih, dn_ih_scale, dn_hh, dn_hh_scale, w_up, bias, c, h)
    t, b, hd = x_i8.shape
    r = dn_ih.size(0)
    need = _L().fluke_factored_lstm_layer_workspace(t, b, hd, r)
    if workspace is None or workspace.numel() < need:
        workspace = torch.empty(need, dtype=torch.uint8, device=x_i8.device)
    h_out = torch.empty(t, b, hd, dtype=torch.int8, device=x_i8.device) if h_out is None else h_out
    layer = _lib.fluke_flstm_layer_t(t, b, hd, r, 1 if reverse else 0, _p(x_i8), _p(x_scale),
                                     _p(dn_ih), _p(dn_ih_scale), _p(dn_hh), _p(dn_hh_scale),
                                     _p(w_up), _p(bias), _p(c), _p(h), _p(h_out),
                                     _p(workspace), workspace.numel())
    if phase_mask == 7:
        _check(_L().fluke_factored_lstm_layer_i8_gpu(ctypes.byref(layer)), "fluke_factored_lstm_layer_i8_gpu")
    else:
        _check(_L().fluke_factored_lstm_layer_phases_gpu(ctypes.byref(layer), phase_mask),
               "fluke_factored_lstm_layer_phases_gpu")
    return h_out
