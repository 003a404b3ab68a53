"""The float32 path with less workspace than it asks for: its chunks grow towards the caller's length, and down to the size that
chunks of the caller's length need every call is served.  Tolerances as for the tile edges of the same kernels: 1e-5 forward, 1e-4
for gradients."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import inputs, mamba2
from oracle.numerics import rel_l2

pytestmark = pytest.mark.gpu


def _problem(b, s, h, p, r, m=None, seed=1):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = lambda *z, k=1.0: k * torch.randn(*z, generator=gen, device="cuda")
    dt = 0.01 + 0.05 * torch.rand(b, s, h, generator=gen, device="cuda")
    lead = (b, s) if m is None else (b, s, m)
    g = 1 if m is None else h
    t = dict(dt=dt, x=n(*lead, h, p), b=n(*lead, g, r, k=r ** -0.5), c=n(*lead, g, r, k=r ** -0.5), h0=n(b, h, p, r, k=0.1), dy=n(*lead, h, p),
             a=-1 - 3 * torch.rand(h, generator=gen, device="cuda"), d=n(h), dhf=n(b, h, p, r))
    t["da"], t["gamma"], t["scale"] = dt * t["a"], 0.4 * dt, 0.9 * dt
    return t


def _per_chunk(b, s, h, p, r, q):
    """Bytes of one scalar per step, one state per chunk, one scalar per chunk."""
    up = lambda n: (n + 255) // 256 * 256
    nc = -(-s // q)
    return up(b * h * nc * q * 4), up(b * nc * h * p * r * 4), up(b * h * nc * 4)


def _run(lib_call, args, nbytes):
    ws = torch.full((nbytes,), 255, dtype=torch.uint8, device="cuda")
    return lib_call(C.byref(args), ws.data_ptr(), nbytes, torch.cuda.current_stream().cuda_stream)


def _close(a, b, tol):
    return (a - b).norm() <= tol * b.norm()


@pytest.mark.parametrize("states", [False, True])
@pytest.mark.parametrize("s,r,q", [(500, 64, 256), (777, 128, 300)])
def test_mamba2_forward(bm, s, r, q, states):
    f, b, h, p = bm._ffi, 2, 3, 64
    t = _problem(b, s, h, p, r)
    want = bm.ops.ssd2_fwd(t["x"], t["dt"], t["a"], t["b"], t["c"], t["d"], t["h0"], chunk_len=q, path="exact", return_chunk_states=states)
    got = [torch.full_like(w, float("nan")) for w in want]
    a = f.Ssd2FwdArgs(batch=b, seqlen=s, nheads=h, headdim=p, state_rank=r, ngroups=1, chunk_len=q, dtype=f.BM_DTYPE_F32, path=f.BM_PATH_EXACT,
                      y=got[0].data_ptr(), h_final=got[1].data_ptr(), chunk_states=got[2].data_ptr() if states else None,
                      **{k: t[k].data_ptr() for k in ("x", "dt", "a", "b", "c", "d", "h0")})
    most = bm.lib.bm_ssd2_fwd_workspace_bytes(C.byref(a))
    scan, st, _ = _per_chunk(b, s, h, p, r, q)
    least = 2 * scan + (0 if states else st)
    assert least < most
    for n in (least, (least + most) // 2, most):
        assert _run(bm.lib.bm_ssd2_fwd, a, n) == 0
        assert all(_close(x, w, 1e-5) for x, w in zip(got, want))
        for x in got:
            x.fill_(float("nan"))
    assert _run(bm.lib.bm_ssd2_fwd, a, least - 256) == f.BM_ERR_WORKSPACE_TOO_SMALL


@pytest.mark.parametrize("s,r,q,p", [(500, 64, 256, 64), (200, 128, 130, 40)])
def test_mamba2_backward(bm, s, r, q, p):
    f, b, h = bm._ffi, 2, 3
    t = _problem(b, s, h, p, r)
    want = bm.ops.ssd2_bwd(t["x"], t["dt"], t["a"], t["b"], t["c"], t["d"], t["h0"], t["dy"], t["dhf"], chunk_len=q, path="exact")
    got = {k: torch.full_like(v, float("nan")) for k, v in want.items()}
    a = f.Ssd2BwdArgs(batch=b, seqlen=s, nheads=h, headdim=p, state_rank=r, ngroups=1, chunk_len=q, dtype=f.BM_DTYPE_F32, path=f.BM_PATH_EXACT,
                      dh_final=t["dhf"].data_ptr(), **{k: v.data_ptr() for k, v in got.items()},
                      **{k: t[k].data_ptr() for k in ("x", "dt", "a", "b", "c", "d", "h0", "dy")})
    most = bm.lib.bm_ssd2_bwd_workspace_bytes(C.byref(a))
    scan, st, end = _per_chunk(b, s, h, p, r, q)
    least = 6 * scan + 2 * st + end + (b * s * h * 4 + 255) // 256 * 256   # the accumulators of the kernels for long chunks
    assert least < most
    for n in (least, (least + most) // 2, most):
        assert _run(bm.lib.bm_ssd2_bwd, a, n) == 0
        assert all(_close(got[k], want[k], 1e-4) for k in want)
        for x in got.values():
            x.fill_(float("nan"))
    assert _run(bm.lib.bm_ssd2_bwd, a, least - 256) == f.BM_ERR_WORKSPACE_TOO_SMALL


@pytest.mark.parametrize("single", [False, True])
def test_mamba3(bm, single):
    f, b, s, h, p, r, m, q = bm._ffi, 1, 150, 2, 64, 64, 2, 128
    t = _problem(b, s, h, p, r, m)
    t["v"] = t.pop("x")
    co = (t["gamma"], t["scale"]) if single else ()
    fwd = bm.ops.ssd3_single_fwd if single else bm.ops.ssd3_double_fwd
    want = fwd(t["v"], t["da"], t["b"], t["c"], *co, h0=t["h0"], chunk_len=q, path="exact")
    grads = bm.ops.ssd3_bwd(t["v"], t["da"], t["b"], t["c"], t["gamma"], t["scale"], t["h0"], t["dy"], t["dhf"], chunk_len=q, single=single, path="exact")
    got = [torch.full_like(w, float("nan")) for w in want]
    gg = {k: torch.full_like(v, float("nan")) for k, v in grads.items()}
    common = dict(batch=b, seqlen=s, nheads=h, headdim=p, state_rank=r, mimo_rank=m, chunk_len=q, dtype=f.BM_DTYPE_F32, path=f.BM_PATH_EXACT,
                  **{k: t[k].data_ptr() for k in ("v", "da", "b", "c", "h0") + (("gamma", "scale") if single else ())})
    af = f.Ssd3FwdArgs(y=got[0].data_ptr(), h_final=got[1].data_ptr(), **common)
    ab = f.Ssd3BwdArgs(dy=t["dy"].data_ptr(), dh_final=t["dhf"].data_ptr(), **common, **{k: v.data_ptr() for k, v in gg.items()})
    scan, st, end = _per_chunk(b, s, h, p, r, q)
    name = "single" if single else "double"
    assert 2 * scan + st < bm.lib.bm_ssd3_fwd_workspace_bytes(C.byref(af))
    assert _run(getattr(bm.lib, f"bm_ssd3_{name}_fwd"), af, 2 * scan + st) == 0
    assert all(_close(x, w, 1e-5) for x, w in zip(got, want))
    assert 6 * scan + 2 * st + end < bm.lib.bm_ssd3_bwd_workspace_bytes(C.byref(ab))
    assert _run(getattr(bm.lib, f"bm_ssd3_{name}_bwd"), ab, 6 * scan + 2 * st + end) == 0
    assert all(_close(gg[k], grads[k], 1e-4) for k in grads)


def test_a_call_runs_where_memory_does_not_hold_what_it_asks_for(bm):
    b, s, h, q = 2, 4096, 16, 256
    t = _problem(b, s, h, 64, 128)
    call = lambda: bm.ops.ssd2_fwd(t["x"], t["dt"], t["a"], t["b"], t["c"], t["d"], t["h0"], chunk_len=q, path="exact")
    want = call()
    torch.cuda.synchronize()
    side = torch.cuda.Stream()   # its workspace does not exist yet
    side.wait_stream(torch.cuda.current_stream())
    states = b * (s // 64) * h * 64 * 128 * 4   # 64 MB for chunks of 64, 16 MB for the caller's
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    outputs = sum(w.numel() * w.element_size() for w in want)
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + outputs + 0.6 * states) / total)
    try:
        with torch.cuda.stream(side):
            got = call()
            assert bm.ops.last_workspace_status() == 0
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    torch.cuda.synchronize()
    assert all(_close(x, w, 1e-5) for x, w in zip(got, want))


@pytest.mark.parametrize("q", [65, 130, 257])
def test_chunk_states_at_a_chunk_length_without_large_divisors(bm, q):
    """The caller's chunks, several tiles each, against the float64 oracle."""
    cfg = inputs.ssd2_prefill(seed=q, batch=2, seqlen=300, nheads=2, headdim=64, state_rank=64, ngroups=1, h0_std=0.1)
    w = {k: v.astype(np.float64) for k, v in cfg.items()}
    want = mamba2.ssd_serial(w["x"], w["dt"], w["a"], w["b"], w["c"], w["d"], w["h0"], q, return_chunk_states=True)
    t = {k: torch.from_numpy(np.ascontiguousarray(v, dtype=np.float32)).cuda() for k, v in cfg.items()}
    got = bm.ops.ssd2_fwd(t["x"], t["dt"], t["a"], t["b"], t["c"], t["d"], t["h0"], chunk_len=q, path="exact", return_chunk_states=True)
    assert all(rel_l2(g.cpu().numpy(), v) <= 1e-5 for g, v in zip(got, want))
