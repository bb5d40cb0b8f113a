# -*- coding: utf-8 -*-
"""Round-off of the FP32 collision operator.

Near equilibrium Q is 1e-6 to 1e-2 of the gain and the loss it is the
difference of, and round-off of 3e-7 of the gain is percents of it: there, a
change in the order of the transforms' operations changes Q.  The golden
values are those of the scalar mixed-radix kernels (N = 24 on one CTA, N = 32 on
two, N = 16 the cluster exchange).
"""

import os

import numpy as np
import pytest

from conftest import GOLDEN
from helpers import config, oracle_for
from oracle import vhs as ovhs
from test_vhs_gpu import _bank, _model

pytestmark = pytest.mark.gpu

GRIDS = {16: (8, 6), 24: (12, 16), 32: (16, 24)}


def _cfg(Nv):
    P, M = GRIDS[Nv]
    cfg = config('channel-n32', 'single', Nv=Nv, Nrho=P, M=M)
    cfg.set('backend-b200', 'vhs-project', 0)
    if Nv < 24:
        cfg.set('velocity-mesh', 'dev', 4.8)
    return cfg


def bumps(Nv):
    """Two smooth bumps made of products alone: the same bits everywhere."""
    i = np.arange(Nv) + 0.5

    def one(a, n):
        t = np.maximum(1 - ((i - a*Nv)/(n*Nv))**2, 0)
        t = t*t
        return t*t

    def three(a, b, c, n):
        return (one(a, n)[:, None, None]*one(b, n)[None, :, None] *
                one(c, n)[None, None, :]).ravel()
    return (0.75*three(0.5, 0.4375, 0.5625, 0.40625) +
            0.5*three(0.5625, 0.5, 0.46875, 0.34375))


def sampled(Q):
    return Q[::{16: 1, 24: 5, 32: 11}[round(len(Q)**(1/3))]]


@pytest.mark.parametrize('Nv', sorted(GRIDS))
def test_values_keep_their_rounding(Nv):
    """To 5e-8 of the gain: transforms with other roundings give values 1.6e-7
    to 2.1e-7 away (FP32 round-off itself), a rare last bit far less."""
    cfg = _cfg(Nv)
    be, vm, sm = _model(cfg)
    fin, fout = _bank(be, vm, bumps(Nv)[None, None])
    sm.fs_all(fin, fout)
    sm.status()
    f = fin.get()[0, :, 0].astype(np.float64)
    Q = sampled(fout.get()[0, :, 0]).astype(np.float64)
    gain, _ = ovhs.vhs_Q_gain_loss(f, *oracle_for(cfg))
    want = np.load(os.path.join(GOLDEN, 'vhs_q_fp32.npz'))[f'n{Nv}']
    off = np.linalg.norm(Q - want)/np.linalg.norm(sampled(gain))
    assert off < 5e-8, off
