"""Tensor-level calls into libbm_b200 (torch supplies device memory and the CUDA stream only).

Every function validates dtypes / contiguity on the host, fills the C args struct with raw device
pointers and launches on torch's current stream.  Outputs are freshly allocated, like the tensors a
Burn backend returns from the reference's slot (src/mamba2/ssd/serial_recalculated/serial_recalculated.rs:86-98).
The work of a call is done by the native module (csrc/host/native.cpp); the functions here own names, defaults and
documentation.
"""
import torch

from . import _ffi, _native

_native.init(_ffi.LIB_PATH, _ffi.BmError)

PATHS = {"auto": _ffi.BM_PATH_AUTO, "exact": _ffi.BM_PATH_EXACT, "tensor": _ffi.BM_PATH_TENSOR,
         "tensor_single": _ffi.BM_PATH_TENSOR_SINGLE, "tensor_pair": _ffi.BM_PATH_TENSOR_PAIR}


def last_workspace_status():
    """Device status word left by the most recent SSD launch on the current device and stream, or BM_ERR_TIMEOUT when a wait of
    a decode step on the device ran out and that has not been raised yet (synchronises); 0 when there is nothing to report."""
    return _native.workspace_status()


def ssd2_fwd(x, dt, a, b, c, d=None, h0=None, chunk_len=256, path="auto", dt_bias=None, dt_limit=(0.0, 65504.0),
             z=None, return_chunk_states=False, check_status=False, debug_reserved=0):
    """Mamba-2 chunked SSD forward.  x [b,s,h,p], dt [b,s,h] f32, a [h] f32, b/c [b,s,g,r], d [h] f32,
    h0 [b,h,p,r] f32 -> (y [b,s,h,p], h_final [b,h,p,r] f32[, chunk_states [b,n,h,p,r]]).
    `debug_reserved` goes into the args struct's `reserved` field (0 in production)."""
    return _native.ssd2_fwd(x, dt, a, b, c, d, h0, dt_bias, z, chunk_len, PATHS[path], dt_limit[0], dt_limit[1],
                            return_chunk_states, check_status, debug_reserved, False)


def step2(state, x, dt, a, b, c, d=None, dt_bias=None, dt_limit=(0.0, 65504.0), z=None):
    """Mamba-2 recurrent step; `state` [b,h,p,r] f32 is updated in place.  Returns y [b,h,p]."""
    return _native.step2(state, x, dt, a, b, c, d, dt_bias, z, dt_limit[0], dt_limit[1])


def conv_step(window, xin, weight, bias=None, splits=None):
    """Causal depthwise conv, one token: slides `window` [b,v,k] f32 in place, returns silu(conv) [b,v] -- or, with
    splits = (split_x, split_bc, split_bc), the three tensors (x [b,split_x], B, C [b,split_bc]).  `xin` [b,v] may be
    a column slice of a wider row."""
    sx, sbc, sbc2 = (-1, 0, 0) if splits is None else splits
    return _native.conv_step(window, xin, weight, bias, sx, sbc, sbc2)


DIV_EPS = {torch.float32: 8.1584695e-8, torch.bfloat16: 2.0885676e-5}   # src/utils/mod.rs:50-95


def conv1d_silu_fwd(xbc, weight, bias=None, window=None, splits=None, want_window=True):
    """Prefill causal depthwise conv + bias + SiLU.  xbc [b, s, v] (may be a column slice), weight [v, k] f32,
    window [b, v, k] f32 or None -> (out [b,s,v] or (x, B, C) when splits = (split_x, split_bc, split_bc), new_window)."""
    sx, sbc, sbc2 = (-1, 0, 0) if splits is None else splits
    return _native.conv1d_silu_fwd(xbc, weight, bias, window, want_window, sx, sbc, sbc2)


def rmsnorm_gated(x, z, gamma, norm_before_gate=False, eps=None):
    """RmsNormGated over the last axis (z = None: plain RmsNorm).  x / z [..., d] (may be column slices), gamma [d]."""
    return _native.rmsnorm_gated(x, z, gamma, norm_before_gate, DIV_EPS[x.dtype] if eps is None else eps)


def mamba3_bc_prep(b_raw, c_raw, b_gamma, c_gamma, b_bias, c_bias, angles=None, rope_dim=None, pairwise=None, ngroups=1,
                   eps=None):
    """Mamba-3 B / C from the raw projection columns to what the SSD slot takes: RMS norm over r, group -> head
    expansion, + bias[h, m, r], rotation by the cumulative angles.  b_raw / c_raw [b, s, m * g * r] (may be column
    slices of the projection output), gammas [r] f32, biases [h, m, r] f32, angles [b, s, h, rope_dim / 2] f32 or
    None -> (B, C) [b, s, m, h, r] in the activations' dtype."""
    return _native.mamba3_bc_prep(b_raw, c_raw, b_gamma, c_gamma, b_bias, c_bias, angles, -1 if rope_dim is None else rope_dim,
                                  -1 if pairwise is None else pairwise, ngroups, DIV_EPS[b_raw.dtype] if eps is None else eps)


def selscan1_fwd(u, delta, a, b, c, d=None, z=None, h0=None, delta_bias=None, delta_softplus=False, serial=False):
    """Mamba-1 selective scan.  u/delta/z [b,s,i], a [i,r] f32, b/c [b,s,r] -> (y [b,s,i], h_final [b,i,r] f32).
    The sequence-parallel kernels (bm_selscan1_fwd_ws) are used unless `serial` asks for the kernels that walk
    the sequence in order and need no workspace (bm_selscan1_fwd)."""
    return _native.selscan1_fwd(u, delta, a, b, c, d, z, h0, delta_bias, delta_softplus, serial)


def step1(state, u, delta, a, b, c, d=None, z=None, delta_bias=None, delta_softplus=False):
    """Mamba-1 recurrent step; `state` [b,i,r] f32 updated in place.  Returns y [b,i]."""
    return _native.step1(state, u, delta, a, b, c, d, z, delta_bias, delta_softplus)


SSD3_TENSOR_PATH = True   # bm_ssd3_*_fwd have a tensor-core path (bf16, P 64, N 128, MIMO rank 1 / 2 / 4)


def ssd3_single_fwd(v, da, b, c, gamma, scale, h0=None, chunk_len=64, angles=None, rope_dim=0, path="auto", check_status=False):
    """Mamba-3 single-pass SSD.  v [b,s,m,h,p], da/gamma/scale [b,s,h] f32, b/c [b,s,m,h,r]."""
    return _native.ssd3_fwd(True, v, da, b, c, gamma, scale, h0, angles, chunk_len, rope_dim, PATHS[path], check_status)


def ssd3_double_fwd(v, da, b, c, h0=None, chunk_len=64, angles=None, rope_dim=0, path="auto", check_status=False):
    """Generic MIMO SSD on pre-scaled v (one pass of Mamba-3's double-SSD pathway)."""
    return _native.ssd3_fwd(False, v, da, b, c, None, None, h0, angles, chunk_len, rope_dim, PATHS[path], check_status)


def angle_cumsum(rot, dt, prev=None, rng=2.0):
    """theta [b,s,h,a] = prev + cumsum_s(dt * range * pi * tanh(rot)); also returns wrap(theta[:, -1])."""
    return _native.angle_cumsum(rot, dt, prev, rng)


def step3(state, k_state, v_state, angle, x, b, c, rot, dt, alpha, beta, gamma, mimo_x=None, rope_dim=None, rng=2.0):
    """Mamba-3 recurrent step; state / k_state / v_state / angle are updated in place.  Returns y [b,m,h,p]."""
    return _native.step3(state, k_state, v_state, angle, x, b, c, rot, dt, alpha, beta, gamma, mimo_x,
                         -1 if rope_dim is None else rope_dim, rng)


def ssd2_fwd_noalloc(x, dt, a, b, c, d=None, h0=None, chunk_len=256, dt_bias=None, dt_limit=(0.0, 65504.0), z=None):
    """bm_ssd2_fwd_noalloc: the exact Mamba-2 SSD forward with the library's built-in scratch instead of
    a workspace -- this wrapper still allocates the outputs, the library call itself allocates nothing.
    Raises BmError(BM_ERR_WORKSPACE_TOO_SMALL) when the problem needs more scratch than the built-in
    array holds.  Calls share that array: do not overlap them on different streams."""
    return _native.ssd2_fwd(x, dt, a, b, c, d, h0, dt_bias, z, chunk_len, _ffi.BM_PATH_EXACT, dt_limit[0], dt_limit[1],
                            False, False, 0, True)


def ssd2_bwd(x, dt, a, b, c, d, h0, dy, dh_final=None, chunk_len=256, path="auto", check_status=False):
    """Mamba-2 SSD backward (recompute).  Returns dict(dx, ddt, da, db, dc, dd, dh0), all float32;
    db / dc are per group.  path: "auto" (tensor-core kernel for bf16, headdim 64, state_rank 128), "exact", "tensor"."""
    return _native.ssd2_bwd(x, dt, a, b, c, d, h0, dy, dh_final, chunk_len, PATHS[path], check_status)


def ssd3_bwd(v, da, b, c, gamma, scale, h0, dy, dh_final=None, chunk_len=64, single=True, path="auto", check_status=False):
    """Mamba-3 SSD backward.  single: returns also dgamma / dscale.  All gradients float32.
    path: "auto" (tensor-core kernel for bf16, headdim 64, state_rank 128, MIMO rank 1 / 2 / 4), "exact", "tensor"."""
    return _native.ssd3_bwd(single, v, da, b, c, gamma if single else None, scale if single else None, h0, dy, dh_final, chunk_len,
                            PATHS[path], check_status)
