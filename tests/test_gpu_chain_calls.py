"""Ways of making a step that the native chains have to serve like the general form: inference mode, caches and activations that are
not 16-byte aligned or not dense, a side thread with a stream of its own, weights that are Parameters, operands of a subclass."""
import threading

import pytest
import torch

from test_gpu_decode_chain import _stack
from test_gpu_mamba3_native import _block, _cache, _close

pytestmark = pytest.mark.gpu


def _m2(bm, batch=2):
    blocks, norms, gen = _stack(bm, 2, 256, 1, seed=11)
    rn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    x = rn(batch, 256).to(torch.bfloat16)
    caches = [bm.Mamba2Cache(0.1 * rn(batch, k.conv_dim, 4), 0.1 * rn(batch, k.nheads, 64, 128)) for k in blocks]
    fresh = lambda f=torch.clone: [bm.Mamba2Cache(f(c.conv_bvk), f(c.ssm_bhpr)) for c in caches]
    return blocks, norms, x, fresh


def _run(bm, blocks, norms, caches, x):
    out = bm.mamba2.stack_step(blocks, norms, caches, x)
    return [out] + [t for c in caches for t in (c.conv_bvk, c.ssm_bhpr)]


def _off_by_one(t):
    """The same values one element past an aligned base."""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    return buf[1:].view(t.shape).copy_(t)


def _same(a, b, tol=0.0):
    return all((x.float() - y.float()).norm() <= tol * y.float().norm() for x, y in zip(a, b))


def test_inference_mode_and_parameters(bm):
    blocks, norms, x, fresh = _m2(bm)
    want = _run(bm, blocks, norms, fresh(), x)
    with torch.inference_mode():
        assert _same(_run(bm, blocks, norms, fresh(), x.clone()), want)
    for k in blocks:
        k.w_in, k.w_out = torch.nn.Parameter(k.w_in), torch.nn.Parameter(k.w_out)
    with torch.no_grad():
        assert _same(_run(bm, blocks, norms, fresh(), x), want)
    assert _run(bm, blocks, norms, fresh(), x)[0].requires_grad   # gradients asked for: the general form, which records them


def test_unaligned_and_strided_operands(bm):
    blocks, norms, x, fresh = _m2(bm)
    want = _run(bm, blocks, norms, fresh(), x)
    wide = torch.zeros(2, 512, dtype=x.dtype, device="cuda")
    wide[:, 128:384] = x
    assert _same(_run(bm, blocks, norms, fresh(), wide[:, 128:384]), want, 1e-2)   # bf16 in another order of rounding
    assert _same(_run(bm, blocks, norms, fresh(), _off_by_one(x)), want, 1e-2)
    with pytest.raises(bm.BmError) as e:   # kernels read caches in 16-byte vectors, in either form
        _run(bm, blocks, norms, fresh(_off_by_one), x)
    assert e.value.code == bm._ffi.BM_ERR_BAD_ALIGNMENT
    blk, n = _block(bm, 2, 64, 32, 16, 32, seed=3)
    c, u = _cache(blk, n, 2), n(2, 64)
    fresh3 = lambda: {k: v.clone() for k, v in c.items()}
    want3, _ = blk.step_double_ssd(u, fresh3())
    assert _close(blk.step_double_ssd(_off_by_one(u), fresh3())[0], want3)


def test_a_side_thread_with_its_own_stream(bm):
    blocks, norms, x, fresh = _m2(bm)
    blk, n = _block(bm, 4, 64, 32, 16, 32, seed=7)
    c, u = _cache(blk, n, 2), n(2, 64)
    want, want3 = _run(bm, blocks, norms, fresh(), x), blk.step_double_ssd(u, {k: v.clone() for k, v in c.items()})[0]
    torch.cuda.synchronize()
    bad = []

    def work():
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            for _ in range(50):
                got = _run(bm, blocks, norms, fresh(), x)
                got3 = blk.step_double_ssd(u, {k: v.clone() for k, v in c.items()})[0]
                stream.synchronize()
                if not (_same(got, want) and torch.equal(got3, want3)):
                    bad.append(1)

    threads = [threading.Thread(target=work) for _ in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


class Scaled(torch.Tensor):
    """A weight kept as int8 and a scale, like weight-only quantisation: it serves the products and has no values of its own."""

    @staticmethod
    def __new__(cls, q, scale):
        t = torch.Tensor._make_wrapper_subclass(cls, q.shape, dtype=torch.bfloat16, device=q.device)
        t.q, t.scale = q, scale
        return t

    @classmethod
    def __torch_dispatch__(cls, func, types, args=(), kwargs=None):
        assert func in (torch.ops.aten.mm.default, torch.ops.aten.addmm.default, torch.ops.aten.detach.default), func
        if func is torch.ops.aten.detach.default:
            return cls(args[0].q, args[0].scale)
        return func(*[a.q.to(torch.bfloat16) * a.scale if isinstance(a, cls) else a for a in args], **(kwargs or {}))


@pytest.mark.parametrize("batch", [2, 9])
def test_weights_that_bring_their_own_products(bm, batch):
    blocks, norms, x, fresh = _m2(bm, batch)
    for k in blocks:
        for name in ("w_in", "w_out"):
            q = (getattr(k, name).float() * 512).round().clamp(-127, 127).to(torch.int8)
            setattr(k, name, Scaled(q, torch.tensor(1 / 512, dtype=torch.bfloat16, device="cuda")))
    got = _run(bm, blocks, norms, fresh(), x)
    for k in blocks:
        k.w_in, k.w_out = (w.q.to(torch.bfloat16) * w.scale for w in (k.w_in, k.w_out))
    assert _same(got, _run(bm, blocks, norms, fresh(), x), 1e-2)
