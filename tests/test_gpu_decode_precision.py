"""One decode step of a stack against the float64 oracle, and against the error that the same step made of single kernels and torch
products has: the chain may not be the less exact of the two.  (The other tests of the chain compare the two with each other.)"""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from oracle import mamba2 as o2
from oracle.numerics import rel_l2, rms_norm

from test_gpu_decode_chain import _stack, _unfused

pytestmark = pytest.mark.gpu
BF16_ROUNDING = 2.0 ** -7 / 12 ** 0.5   # rms of rounding to 8 significant bits, for a significand of 1


def _oracle(blocks, norms, caches, x):
    f64 = lambda t: t.double().cpu().numpy()
    x = f64(x)
    out = []
    for blk, gamma, c in zip(blocks, norms, caches):
        w = SimpleNamespace(w_in=f64(blk.w_in), conv_w=f64(blk._conv_w32), conv_b=f64(blk._conv_b32), dt_bias=f64(blk.dt_bias), a_log=f64(blk.a_log),
                            d=f64(blk.d), norm_gamma=f64(blk.norm_gamma), w_out=f64(blk.w_out), d_inner=blk.d_inner, conv_dim=blk.conv_dim,
                            ngroups=blk.ngroups, state_rank=blk.state_rank, nheads=blk.nheads, per_head_dim=blk.per_head_dim, dt_limit=blk.dt_limit)
        y, conv, ssm = o2.block_step(w, rms_norm(x, f64(gamma), "bf16"), f64(c.conv_bvk), f64(c.ssm_bhpr), dtype_name="bf16")
        x = x + y
        out += [conv, ssm]
    return [x] + out


# (batch, d_model, groups, layers, head width): streaming projections with the fused mixer and with the kernels apart (320 pairs),
# either side of the batch that takes library products, two slices of five K blocks (d_model 320; rows in whole 16-byte vectors ask
# for a multiple of eight heads)
@pytest.mark.parametrize("batch,d_model,g,layers,p", [(1, 768, 1, 6, 64), (3, 320, 1, 3, 16), (8, 256, 2, 4, 64), (8, 320, 1, 4, 16), (9, 256, 1, 4, 64),
                                                      (70, 256, 4, 3, 64)])
def test_the_chain_is_no_less_exact_than_the_single_kernels(bm, batch, d_model, g, layers, p):
    blocks, norms, gen = _stack(bm, layers, d_model, g, seed=batch + d_model, headdim=p)
    rn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    caches = [bm.Mamba2Cache(0.1 * rn(batch, k.conv_dim, 4), 0.1 * rn(batch, k.nheads, p, 128)) for k in blocks]
    twin = [bm.Mamba2Cache(c.conv_bvk.clone(), c.ssm_bhpr.clone()) for c in caches]
    x = rn(batch, d_model).to(torch.bfloat16)
    want = _oracle(blocks, norms, caches, x)
    err = lambda out, cs: [rel_l2(t.double().cpu().numpy(), w) for t, w in zip([out] + [t for c in cs for t in (c.conv_bvk, c.ssm_bhpr)], want)]
    out = bm.mamba2._native.m2_decode([k._chain(c, n) for k, c, n in zip(blocks, caches, norms)], x, None, bm.ops.DIV_EPS[torch.bfloat16])
    assert out is not None   # the chain, and not the form it is compared with
    got = err(out, caches)
    apart = x
    for blk, gamma, c in zip(blocks, norms, twin):
        apart = _unfused(bm, blk, bm.mamba2.rms_norm(apart, gamma), c, apart)
    single = err(apart, twin)
    # per tensor, with room for another order of the same roundings; what neither rounds to bf16 sits at float32's level
    assert all(a <= 1.1 * b + 2e-5 for a, b in zip(got, single)), (got, single)
    if batch <= 8 and batch * blocks[0].nheads < 296:
        # nothing but the output is rounded to bf16: projections of operands in two planes (16 bits), sums and streams in float32
        assert got[0] <= BF16_ROUNDING and max(got[1:]) <= 5e-5, got
