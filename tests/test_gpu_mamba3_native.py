"""The native Mamba-3 block (kernels around the slot, fused step) against the same block as torch ops around the library's
entry points, at sizes where its kernels branch.  float32: sums of at most a few hundred terms in another order, sines of the
same angles: 2e-5 relative."""
import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = 2e-5


def _block(bm, m, d_model, r, p, rope, seed, g=1, mimo_x=True):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = lambda *s, k=1.0: k * torch.randn(*s, generator=gen, device="cuda")
    di = 2 * d_model
    h = di // p
    mimo = lambda: None if m == 1 else 0.5 + n(h, m, p, k=0.2)
    w_in = n(d_model, 2 * di + 2 * m * g * r + 3 * h + max(rope // 2, 1), k=d_model ** -0.5)
    return bm.Mamba3(w_in, n(h) - 3, n(h), 1 + n(r, k=0.1), 1 + n(r, k=0.1), n(h, m, r, k=0.3), n(h, m, r, k=0.3), n(di, d_model, k=di ** -0.5),
                     nheads=h, state_rank=r, ngroups=g, mimo_rank=m, rope_dim=rope, mimo_x=mimo() if mimo_x else None, mimo_z=mimo(), mimo_o=mimo()), n


def _cache(blk, n, b):
    h, p, r = blk.nheads, blk.per_head_dim, blk.state_rank
    return dict(ssm=n(b, h, p, r, k=0.1), k=n(b, blk.mimo_rank, h, r, k=0.1), v=n(b, h, p), angle=n(b, h, blk.num_rope_angles))


def _close(a, b):
    return (a - b).norm() <= TOL * b.norm().clamp_min(1e-20)


@pytest.mark.parametrize("b,m,d_model,r,p,rope,g", [
    (2, 4, 64, 128, 64, 128, 2),    # few pairs: a cluster of four CTAs per (batch, head)
    (1, 1, 96, 32, 48, 16, 1),      # three CTAs, partial rotation, rows shorter than a warp
    (80, 4, 128, 64, 64, 64, 1),    # a wave of pairs: one CTA each
    (75, 2, 128, 128, 32, 0, 1),    # no rotation, warps without rows
    (160, 1, 64, 20, 64, 20, 1),    # a state rank that is no multiple of 16
])
def test_fused_step_matches_the_unfused_block(bm, monkeypatch, b, m, d_model, r, p, rope, g):
    blk, n = _block(bm, m, d_model, r, p, rope, seed=b, g=g, mimo_x=b != 2)
    cache = _cache(blk, n, b)
    twin = {k: v.clone() for k, v in cache.items()}
    us = [n(b, d_model) for _ in range(2)]
    got = [blk.step_double_ssd(u, cache)[0] for u in us]
    monkeypatch.setattr(bm.mamba3._native, "m3_step", lambda *a: None)
    want = [blk.step_double_ssd(u, twin)[0] for u in us]
    for x, y in list(zip(got, want)) + [(cache[k], twin[k]) for k in cache]:
        assert _close(x, y)


@pytest.mark.parametrize("s,m,r,p,rope,with_cache", [(1, 4, 32, 16, 32, True), (37, 1, 16, 20, 8, True), (65, 2, 64, 64, 0, False), (130, 4, 128, 64, 128, False)])
def test_native_forward_matches_the_unfused_block(bm, monkeypatch, s, m, r, p, rope, with_cache):
    blk, n = _block(bm, m, 40 if p == 20 else 64, r, p, rope, seed=s)
    u, cache = n(2, s, blk.w_in.shape[0]), None
    if with_cache:
        cache = _cache(blk, n, 2)
    got, gc = blk.forward_single_ssd(u, cache)
    monkeypatch.setattr(bm.mamba3._native, "m3_forward", lambda *a: None)
    want, wc = blk.forward_single_ssd(u, cache)
    assert _close(got, want)
    for k in wc:
        assert gc[k].shape == wc[k].shape and _close(gc[k], wc[k])


@pytest.mark.parametrize("value", [float("nan"), float("inf"), float("-inf")])
@pytest.mark.parametrize("where", ["dt_bias", "dd_dt", "dd_A", "lambda", "rot"])
def test_infinities_and_nan_reach_the_output_as_in_the_unfused_block(bm, monkeypatch, where, value):
    """One head's scalar (or one angle) is infinite or NaN: clamps keep NaN, and every value that stays finite is the same."""
    blk, n = _block(bm, 2, 64, 32, 16, 32, seed=4)
    at = {"dd_dt": sum(blk.splits[:4]), "dd_A": sum(blk.splits[:5]), "lambda": sum(blk.splits[:6]), "rot": sum(blk.splits[:7])}
    if where == "dt_bias":
        blk.dt_bias[1] = value
    else:
        blk.w_in[3, at[where] + 1] = value
    cache, u = _cache(blk, n, 2), n(2, 9, 64)
    fresh = lambda: {k: v.clone() for k, v in cache.items()}
    run = lambda: [blk.forward_single_ssd(u, fresh()), blk.step_double_ssd(u[:, 0].contiguous(), fresh())]
    got = run()
    monkeypatch.setattr(bm.mamba3._native, "m3_forward", lambda *a: None)
    monkeypatch.setattr(bm.mamba3._native, "m3_step", lambda *a: None)
    for (go, gc), (wo, wc) in zip(got, run()):
        for a, b in [(go, wo)] + [(gc[k], wc[k]) for k in wc]:
            assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isinf(), b.isinf())
            ok = b.isfinite()
            assert not ok.any() or _close(a[ok], b[ok])


@pytest.mark.parametrize("given", [("k", "v", "angle"), ("ssm", "v", "angle"), ("ssm", "k", "v")])
def test_a_cache_without_one_of_its_tensors_is_refused(bm, given):
    blk, n = _block(bm, 2, 64, 32, 16, 32, seed=2)
    cache = {k: t for k, t in _cache(blk, n, 2).items() if k in given}
    with pytest.raises(KeyError):
        blk.forward_single_ssd(n(2, 5, 64), cache)
    with pytest.raises(KeyError):
        blk.step_double_ssd(n(2, 64), cache)
    for dropped in set(("ssm", "k", "v", "angle")) - set(given):   # there, but None
        with pytest.raises((AttributeError, TypeError)):
            blk.forward_single_ssd(n(2, 5, 64), {**cache, dropped: None})
