"""A bounded wait that runs out in a decode step: the projection's sums become NaN, the kernel ends, and the host raises it once."""
import ctypes as C

import pytest
import torch

from test_gpu_decode_chain import _stack

pytestmark = pytest.mark.gpu


# K blocks of 64: fewer than the 12 (or, above 74 column tiles, 6) stages, and more than they hold
@pytest.mark.parametrize("batch,k,n,planes", [(1, 128, 128, 1), (8, 2048, 136, 2), (3, 1536, 9600, 1)])
def test_projection_that_gives_up(bm, batch, k, n, planes):
    lib = C.CDLL(bm._ffi.LIB_PATH)
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    gen = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(planes, batch, k, generator=gen, device="cuda").to(torch.bfloat16)
    w = torch.randn(k, n, generator=gen, device="cuda").to(torch.bfloat16)
    ns = lib.bmx_decode_slices(batch, k, n)
    assert ns > 0
    part, status = torch.zeros(ns, batch, n, device="cuda"), torch.zeros(4, dtype=torch.int32, device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())
    call = lambda stall: lib.bmx_decode_linear(ptr(x), planes, ptr(w), ptr(part), batch, k, n, ns, ptr(status), 1, stall, stream)
    assert call(1) == 0
    torch.cuda.synchronize()
    assert part.isnan().all() and status.tolist() == [bm._ffi.BM_ERR_TIMEOUT, 0, 0, 0]
    status.zero_()
    assert call(0) == 0
    torch.cuda.synchronize()
    want = x.double().sum(0) @ w.double()
    assert status.tolist() == [0] * 4
    assert (part.double().sum(0) - want).norm() <= 1e-5 * want.norm()   # float32 sums of k exact products


def test_a_step_reports_a_wait_that_ran_out_once(bm):
    blocks, norms, gen = _stack(bm, 2, 256, 1, seed=9)
    x = torch.randn(2, 256, generator=gen, device="cuda").to(torch.bfloat16)
    caches = [k.zero_cache(2) for k in blocks]
    lib = C.CDLL(bm._ffi.LIB_PATH)
    lib.bmx_chain_status.restype = C.POINTER(C.c_int32)
    word = lib.bmx_chain_status(torch.cuda.current_device())
    step = lambda **kw: bm.mamba2.stack_step(blocks, norms, caches, x, **kw)
    step(check_status=True)
    before = [c.ssm_bhpr.clone() for c in caches]
    word[0] = bm._ffi.BM_ERR_TIMEOUT   # what a projection that gives up leaves
    with pytest.raises(bm.BmError) as e:
        step()
    assert e.value.code == bm._ffi.BM_ERR_TIMEOUT
    assert all(torch.equal(a, c.ssm_bhpr) for a, c in zip(before, caches))   # raised before anything was launched
    step(check_status=True)
    blocks[0].step(x, blocks[0].zero_cache(2), check_status=True)
    word[0] = bm._ffi.BM_ERR_TIMEOUT
    assert bm.ops.last_workspace_status() == bm._ffi.BM_ERR_TIMEOUT and bm.ops.last_workspace_status() == 0
