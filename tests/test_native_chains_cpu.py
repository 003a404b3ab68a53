"""Which calls the native block chains take (csrc/host/native.cpp), as far as it shows without a GPU: a chain declines by
returning None before it touches the device, and its kernels' entry points refuse missing pointers.

The operands are tensors that say they live on a GPU: plain ones over host memory, or a subclass without any storage.  A chain
that took one of these calls would fail at its first allocation here."""
import ctypes as C

import pytest
import torch

BF, F = torch.bfloat16, torch.float32


class NoStorage(torch.Tensor):
    """Like a quantised weight that keeps its parts elsewhere and dispatches on its type."""

    @staticmethod
    def __new__(cls, shape, dtype):
        return torch.Tensor._make_wrapper_subclass(cls, shape, dtype=dtype, device="cuda:0")

    @classmethod
    def __torch_dispatch__(cls, func, types, args=(), kwargs=None):
        raise AssertionError(f"{func} reached a tensor without storage")


_KEEP = []   # the host memory behind the plain operands


def _plain(shape, dtype, device="cuda:0"):
    host = torch.zeros(shape, dtype=dtype)
    _KEEP.append(host)
    storage = torch._C._construct_storage_from_data_pointer(host.data_ptr(), torch.device(device), host.nbytes)
    return torch._C._construct_CUDA_Tensor_From_Storage_And_Metadata(
        dict(dtype=dtype, size=host.size(), stride=host.stride(), storage_offset=0), storage)


def _m2(make, odd):
    """(layer tuple, x, residual) of a Mamba-2 step: operand number `odd` made by `make`."""
    dm, h, p, v = 128, 8, 32, 256 + 2 * 128
    n = 256 + v + h
    specs = [((dm, n), BF), ((v, 4), F), ((v,), F), ((h,), F), ((h,), F), ((h,), F), ((256,), BF), ((256, dm), BF), ((2, v, 4), F), ((2, h, p, 128), F),
             ((dm,), BF), ((2, dm), BF), ((2, dm), BF)]
    t = [(make if k == odd else _plain)(*s) for k, s in enumerate(specs)]
    return tuple(t[:11]) + (h, 1, False, 0.0, 1e4), t[11], t[12]


def _m3(make, odd):
    """(block tuple, u [b, d_model], caches, u [b, s, d_model]) of a Mamba-3 block: operand number `odd` made by `make`."""
    dm, h, p, r, m = 64, 4, 32, 32, 2
    n = 2 * h * p + 2 * m * r + 3 * h + r // 2
    specs = [((dm, n), F), ((h,), F), ((h,), F), ((r,), F), ((r,), F), ((h, m, r), F), ((h, m, r), F), ((h * p, dm), F), ((h, m, p), F), ((h, m, p), F), ((h, m, p), F),
             ((2, dm), F), ((2, h, p, r), F), ((2, m, h, r), F), ((2, h, p), F), ((2, h, r // 2), F), ((2, 1, dm), F)]
    t = [(make if k == odd else _plain)(*s) for k, s in enumerate(specs)]
    return tuple(t[:11]) + (h, r, 1, m, r, 2.0, 0.0, 1e4, 1e-4, 1e-7), t[11], t[12:16], t[16]


def _calls(bm, kind, make=_plain, odd=-1):
    """The chain calls that read operand number `odd`."""
    native = bm.mamba2._native
    if kind == "m2":
        layer, x, res = _m2(make, odd)
        if odd == 12:   # a residual is for a step without layer norm
            return [lambda: native.m2_decode([layer[:10] + (None,) + layer[11:]], x, res, 1e-5)]
        return [lambda: native.m2_decode([layer], x, None, 1e-5)]
    block, u, caches, seq = _m3(make, odd)
    step, forward = (lambda: native.m3_step(block, u, *caches)), (lambda: native.m3_forward(block, seq, *caches, 64))
    return [step] if odd == 11 else [forward] if odd == 16 else [step, forward]


@pytest.mark.skipif(torch.cuda.is_available(), reason="the calls would run, on host memory")
@pytest.mark.parametrize("kind", ["m2", "m3"])
def test_the_calls_below_are_ones_the_chains_take(bm, kind):
    """All operands plain: the chain goes on to the device, which is not there."""
    for call in _calls(bm, kind):
        with pytest.raises(RuntimeError):
            call()


OPERANDS = [("m2", k) for k in range(13)] + [("m3", k) for k in range(17)]


@pytest.mark.parametrize("kind,odd", OPERANDS)
def test_chains_leave_tensors_without_storage_to_the_general_form(bm, kind, odd):
    assert all(call() is None for call in _calls(bm, kind, NoStorage, odd))


@pytest.mark.parametrize("kind,odd", [("m2", 0), ("m2", 8), ("m2", 11), ("m3", 1), ("m3", 11), ("m3", 13)])
def test_chains_leave_python_subclasses_and_lazy_negations_to_the_general_form(bm, kind, odd):
    class Named(torch.Tensor):
        pass
    for make in (lambda s, d: _plain(s, d).as_subclass(Named), lambda s, d: torch._neg_view(_plain(s, d))):
        assert all(call() is None for call in _calls(bm, kind, make, odd))


@pytest.mark.parametrize("kind,odd", OPERANDS)
def test_chains_leave_operands_on_two_devices_to_the_general_form(bm, kind, odd):
    """torch refuses such a call in the general form; a chain would read another device's address."""
    assert all(call() is None for call in _calls(bm, kind, lambda s, d: _plain(s, d, "cuda:1"), odd))


def test_entry_points_of_the_chain_kernels_refuse_missing_pointers(bm):
    """A zeroed argument block (all pointers NULL) is refused on the host; nothing is launched."""
    lib, zeros = C.CDLL(bm._ffi.LIB_PATH), C.create_string_buffer(1024)
    null = bm._ffi.BM_ERR_NULL_POINTER
    p, buf = C.c_void_p, C.c_void_p(4096)
    assert lib.bmx_m3_coefficients(zeros, *[buf] * 6, p()) == null
    assert lib.bmx_m3_seed(zeros, *[buf] * 6, p()) == null
    assert lib.bmx_m3_tail(zeros, *[buf] * 5, p()) == null
    assert lib.bmx_m3_step(zeros, *[buf] * 5, p()) == null
    assert lib.bmx_decode_linear(buf, 1, p(), buf, 1, 128, 128, 1, buf, 1, 0, p()) == null
    assert lib.bmx_decode_norm(buf, p(), p(), p(), p(), C.c_float(1e-5), p(), p(), buf, 1, 1, 128, 1, p()) == null
    assert lib.bmx_decode_mixer(zeros, p()) == null
    assert lib.bmx_decode_state(zeros, zeros, 0, p()) == null
    assert lib.bmx_decode_gated_norm(zeros, zeros, 1, p()) == null
