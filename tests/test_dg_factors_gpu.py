# -*- coding: utf-8 -*-
"""The residual on 1D operator factors and, for element matrices without that
structure, the dense one: both against the FP64 oracle on the same matrices,
on a ragged mesh (one full element block and one of 4), with every boundary
point evaluated, for every SIMT launch shape."""

import numpy as np
import pytest
import torch

from frfs_b200 import mesh as mgen
from frfs_b200.shapes import QuadShape
from helpers import dg_setup, rel_err
from oracle import vhs as ovhs
from test_dg_gpu import TOL, _cfg, _states, _system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('precision', ['double', 'single'])
@pytest.mark.parametrize('order', [1, 2, 3])
@pytest.mark.parametrize('dense', [None, 'M0', 'M3', 'M1 - M3*M2'])
def test_factored_and_dense_residual(precision, order, dense, monkeypatch):
    exact = QuadShape.opmat

    def opmat(self, expr):
        m = exact(self, expr)
        if expr == dense:
            rng = np.random.default_rng(order)
            m = m + 0.05*np.max(np.abs(m))*rng.standard_normal(m.shape)
        return m
    monkeypatch.setattr(QuadShape, 'opmat', opmat)
    cfg = _cfg(precision, 'dgfs-wall-diffuse', 'dgfs-wall-specular', order)
    m = mgen.quad_box(9, 4, 0.0, 1.0, 0.0, 0.75, periodic_x=True, jitter=0.2,
                      seed=order)
    dg, sh, geo, vm = dg_setup(cfg, m)
    u = _states(vm, sh.nupts, geo.neles, seed=order)
    be, s = _system(cfg, m, u)
    # without 1D factors a handle starts on the dense shape without prefetch
    assert (s._dg_shape == 0) == (dense is not None)
    u_used = s.bank[0].get().astype(np.float64)
    uf = dg.disu(u_used)
    dg.update_bc(uf)
    ref = dg.rhs(u_used, uf)
    for i, v in enumerate(s.dg_variants()):
        if v['tensor_cores']:
            continue
        s.select_dg(i)
        s.bank[1].data.zero_()
        s.updatebc(0.0, 0, 1, 0, 0)
        s.rhs(0.0, 0, 1, 0, 0)
        torch.cuda.synchronize()
        assert rel_err(s.face_values(), uf) < TOL[precision], i
        assert rel_err(s.bank[1].get(), ref) < TOL[precision], (i, v)


@pytest.mark.parametrize('order', [1, 2, 3])
def test_small_terms_are_added_first(order):
    """alpha A + beta B + gamma (R + C) rounds at the size of f once per
    full-size term.  f varies by 10 % in space, so |gamma R| < 2e-4 f at
    gamma = 1e-6 (R <= 2 c f / h, c < 7, 2/h = 18) and R's own round-off, 1e-6
    of it, is 2e-10 f: 1/300 of the spacing of f's values, which can move one
    value in 300 (and the oracle's rounding of the sum as many); one rounding
    at the size of f more moves every fourth or so."""
    cfg = _cfg('single', 'dgfs-outlet', 'dgfs-outlet', order)
    m = mgen.quad_box(9, 4, 0.0, 1.0, 0.0, 0.75, periodic_x=True, jitter=0.2,
                      seed=order)
    dg, sh, geo, vm = dg_setup(cfg, m)
    rng = np.random.default_rng(order)
    shape = (sh.nupts, 1, geo.neles)
    u = ovhs.maxwellian(vm.cv(), 1.0, [0.2, -0.1, 0.0], 0.9)[None, :, None] * \
        rng.uniform(0.95, 1.05, shape)
    be, s = _system(cfg, m, u)
    s.bank[1].set(100*u*rng.uniform(0.5, 1.5, u.shape))
    u0, c = (s.bank[i].get().astype(np.float64) for i in (0, 1))
    uf = dg.disu(u0)
    dg.update_bc(uf)
    f32 = lambda x: x.astype(np.float32).astype(np.float64)
    small = f32(1e-6*(dg.rhs(u0, uf) + c))
    first, second = f32(u0 + small), f32(0.5*u0 + f32(0.5*c + small))
    for i, v in enumerate(s.dg_variants()):
        if v['tensor_cores']:
            continue
        s.select_dg(i)
        s.updatebc(0.0, 0, 2, 0, 0)
        for want, args in ((first, (1.0, 0, 0.0, None)),
                           (second, (0.5, 1, 0.5, 0))):
            s.rk_stage(0, 2, *args, 1e-6, 1, interp=False)
            torch.cuda.synchronize()
            assert np.mean(s.bank[2].get() == want) > 0.98, (i, v)
