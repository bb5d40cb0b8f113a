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
