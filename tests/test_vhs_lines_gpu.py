# -*- coding: utf-8 -*-
"""The single-CTA and two-CTA collision kernels at the sizes where their work
split changes: one point (its radial nodes spread over CTAs), a ragged bank
whose points are still split, and one with more points than CTAs, against
the FP64 oracle; a point's value does not depend on the launch it is part
of."""

import numpy as np
import pytest

from helpers import config, oracle_for, random_states, rel_err
from oracle import vhs as ovhs
from test_vhs_gpu import FP32_TOL, FP64_TOL, _bank, _model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('neles', [1, 33, 450])
@pytest.mark.parametrize('project', [0, 1])
@pytest.mark.parametrize('name,precision,kw', [
    ('channel-n32', 'single', dict(Nv=8, Nrho=3, M=6)),
    ('channel-n32', 'single', dict(Nv=16, Nrho=5, M=6)),
    ('channel-n32', 'single', dict(Nv=24, Nrho=2, M=6)),
    ('channel-n32', 'double', dict(Nv=16, Nrho=2, M=6)),
    ('channel-n32', 'double', dict(Nv=16, Nrho=5, M=6)),
    ('channel-n32', 'double', dict(Nv=24, Nrho=3, M=6)),
    ('channel-n32', 'single', dict(Nv=32, Nrho=2, M=6)),
])
def test_line_kernels_across_splits(name, precision, kw, project, neles):
    cfg = config(name, precision, **kw)
    cfg.set('backend-b200', 'vhs-project', project)
    be, vm, sm = _model(cfg)
    ovm, pre, prefac = oracle_for(cfg)
    base = random_states(vm.cv(), 3, seed=neles)
    f = base[np.arange(neles) % 3][None]
    fin, fout = _bank(be, vm, f)
    fu = fin.get().astype(np.float64)
    tol = FP64_TOL if precision == 'double' else FP32_TOL
    shapes = [i for i, v in enumerate(sm.variants())
              if v['exchange'] in ('single-cta', 'pair')]
    assert shapes
    for i in shapes:
        sm.select(i)
        sm.fs_all(fin, fout)
        sm.status()
        Q = fout.get()[0]
        # equal states give equal values wherever their point runs
        for e in range(neles):
            np.testing.assert_array_equal(Q[:, e], Q[:, e % 3])
        for e in range(min(3, neles)):
            Qo = ovhs.vhs_Q(fu[0, :, e], ovm, pre, prefac)
            if project:
                Qo = ovhs.project_conservative(Qo, vm.cv())
            assert rel_err(Q[:, e], Qo) < tol, (i, e)
        _, one = _bank(be, vm, f)
        sm.fs(fin, one, neles - 1, 0)
        np.testing.assert_array_equal(one.get()[0, :, neles - 1],
                                      Q[:, neles - 1])


@pytest.mark.parametrize('precision,Nv,P,M', [
    ('single', 16, 8, 6), ('single', 24, 12, 16), ('double', 16, 8, 6)])
def test_split_rule_does_not_change_values(precision, Nv, P, M):
    """Banks on both sides of each wave of split and whole items: every
    point equals the value it has in a launch of its own."""
    cfg = config('channel-n32', precision, Nv=Nv, Nrho=P, M=M)
    be, vm, sm = _model(cfg)
    neles = 150
    base = random_states(vm.cv(), 3, seed=Nv)
    fin, ref = _bank(be, vm, base[np.arange(neles) % 3][None])
    for pt in range(3):
        sm.fs_range(fin, ref, pt, 1)
    want = ref.get()[0, :, :3]
    for n in (18, 37, 49, 55, 56, 74, 75, 90, 91, 147, 148, 149):
        _, out = _bank(be, vm, base[np.arange(neles) % 3][None])
        sm.fs_range(fin, out, 0, n)
        sm.status()
        got = out.get()[0]
        for e in range(n):
            np.testing.assert_array_equal(got[:, e], want[:, e % 3])
