"""Workspace sizes the library asks for (host only): what the path that serves the call needs, and not what another would."""
import ctypes as C

import pytest

P, R = 64, 128


def _state(b, s, h, q, m=1):
    """Bytes of one float32 state per chunk of q steps."""
    return b * -(-s // q) * h * P * R * 4


def _bwd2(bm, path="auto", **kw):
    f = bm._ffi
    d = dict(batch=3, seqlen=1999, nheads=32, headdim=P, state_rank=R, ngroups=2, chunk_len=256, dtype=f.BM_DTYPE_BF16, path=bm.ops.PATHS[path])
    d.update(kw)
    return bm.lib.bm_ssd2_bwd_workspace_bytes(C.byref(f.Ssd2BwdArgs(**d))), d


def _bwd3(bm, path="auto", **kw):
    f = bm._ffi
    d = dict(batch=16, seqlen=2048, nheads=32, headdim=P, state_rank=R, mimo_rank=4, chunk_len=64, dtype=f.BM_DTYPE_BF16, path=bm.ops.PATHS[path])
    d.update(kw)
    return bm.lib.bm_ssd3_bwd_workspace_bytes(C.byref(f.Ssd3BwdArgs(**d))), d


@pytest.mark.parametrize("shape", [dict(batch=8, seqlen=4096, nheads=80), dict(), dict(batch=1, seqlen=1, nheads=4), dict(chunk_len=16)])
def test_backward_on_the_tensor_cores_asks_for_its_own_need(bm, shape):
    """Its layout: the state entering every 128-row tile, final state, per-SM slots, and what the state chain needs."""
    n, d = _bwd2(bm, **shape)
    tiles = _state(d["batch"], d["seqlen"], d["nheads"], 128)
    assert tiles <= n <= 1.1 * tiles + (32 << 20)
    assert n == _bwd2(bm, path="tensor", **shape)[0]


@pytest.mark.parametrize("shape", [dict(), dict(batch=2, seqlen=65, mimo_rank=1), dict(seqlen=100, mimo_rank=2, chunk_len=8)])
def test_mamba3_backward_on_the_tensor_cores_asks_for_its_own_need(bm, shape):
    n, d = _bwd3(bm, **shape)
    tiles = _state(d["batch"], d["seqlen"] * d["mimo_rank"], d["nheads"], 128)
    assert tiles <= n <= 1.1 * tiles + (32 << 20)
    assert n == _bwd3(bm, path="tensor", **shape)[0]


def test_exact_backward_still_asks_for_the_exact_need(bm):
    n, d = _bwd2(bm, path="exact")
    assert n >= 2 * _state(d["batch"], d["seqlen"], d["nheads"], 64)
    assert _bwd2(bm, headdim=32)[0] == _bwd2(bm, path="exact", headdim=32)[0]   # a shape the tensor kernel does not cover


@pytest.mark.parametrize("q", [65, 67, 127, 130, 254, 257])
def test_chunk_states_at_a_chunk_length_without_large_divisors(bm, q):
    """No divisor fills half a tile: the states live in the caller's buffer, and the workspace is two scalars per step."""
    f = bm._ffi
    a = f.Ssd2FwdArgs(batch=1, seqlen=4096, nheads=8, headdim=P, state_rank=R, ngroups=1, chunk_len=q, dtype=f.BM_DTYPE_F32, path=f.BM_PATH_EXACT,
                      chunk_states=0x1000)
    assert bm.lib.bm_ssd2_fwd_workspace_bytes(C.byref(a)) <= 2 * (8 * (4096 + q) * 4 + 256)
    a.chunk_len = 192   # 3 x 64: chunks of one full tile, their states beside the caller's
    assert bm.lib.bm_ssd2_fwd_workspace_bytes(C.byref(a)) >= _state(1, 4096, 8, 64)
