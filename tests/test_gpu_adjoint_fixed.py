"""The backward pass at the edges of the fixed-point step adjoint's range (st_fixed.cuh):
steps above a quarter radian, strong and steep fields, pulses of either sign of w, a
zero pulse with its gradients asked for.  Loss weights of 2^-850 leave the range of the
fixed-point form, so that every step runs in FP64, and gradients are linear in the
weights: 2^850 times those gradients agree with the ones of the plain weights to 1e-9
of the largest of their parameter (FP64's own error is near 1e-11 with a pulse)."""
from __future__ import annotations

import math

import numpy as np
import pytest

import spintrack as st
from spintrack.adjoint import NUM_THETA

pytestmark = pytest.mark.gpu

G = np.random.default_rng(3).normal(0.0, 1e-9, 9)
BASE = dict(numParticles=40, dist="M", T=4.2, diffuse=0.2, gas_coll=False, gravity=True, Gx=G[0:3], Gy=G[3:6], Gz=G[6:9],
            E=(0.0, 0.0, 75e5), B0=(3e-6, 0.0, 0.0), yi=(0.0, 0.0, 1.0), tf=0.02, ioutInt=0.01, seed=5, rtol=1e-12, atol=1e-12,
            h=1e-3, hmax=1.0, hmin=1e-8)
CASES = {
    "plain": dict(),
    "loose": dict(rtol=1e-6, atol=1e-6),
    "strong": dict(B0=(1e-4, 1e-5, 0.0), tf=0.004, ioutInt=0.002),
    "steep": dict(Gx=(1e-5, 2e-5, 0.0), Gy=(0.0, -1e-5, 1e-5), Gz=(3e-6, 0.0, 0.0)),
    "pulse": dict(a=5e-6, w=2 * math.pi * 1000.0, hmax=1e-4),
    "pulse_back": dict(a=5e-6, w=-2 * math.pi * 1000.0, hmax=1e-4),
    "zero_pulse": dict(a=0.0, w=2 * math.pi * 1000.0, hmax=1e-4),
    "norm": dict(yi=(60.0, -80.0, 35.0), atol=1e-10),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_gradients_agree_with_fp64(gpu, name):
    import torch
    opt = st.derive(st.make_options(**{**BASE, **CASES[name]}))
    dev = torch.device("cuda", 0)
    w = torch.tensor(np.random.default_rng(2).normal(size=(opt.numParticles, 3)), dtype=torch.float64, device=dev)
    out = []
    with st.Particles(opt) as p:
        for scale in (1.0, 2.0 ** -850):
            ws = (w * scale).contiguous()
            grad = torch.empty(p.n, NUM_THETA, dtype=torch.float64, device=dev)
            p.init_particles()
            p.adjoint_record(st.num_windows(opt))
            torch.cuda.synchronize()
            p.adjoint_backward(ws.data_ptr(), grad.data_ptr(), pulse="pulse" in name)
            torch.cuda.synchronize()
            out.append((grad / scale).cpu().numpy())
    assert np.isfinite(out[0]).all()
    top = np.abs(out[1]).max(axis=0)
    assert (top[:15] > 0).all()
    assert (np.abs(out[0] - out[1]) <= 1e-9 * top).all()
