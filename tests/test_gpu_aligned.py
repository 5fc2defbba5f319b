"""Fields along each axis and spins along or across them (the grades of st_fixed.cuh).

Gradients: with a loss along the field, spins that start along it leave products of small components only.  Loss
weights of 2^-850 leave the range of the fixed-point form, so that every step runs in FP64: 2^850 times those
gradients agree with the plain ones to 1e-9 of the largest of their parameter.

Forward: counts and spins are the oracle's (1e-9), for a field along x precession turns those of a run whose steps are all
FP64 (any beta but 0 makes them so; 1e-300 changes no step size), and every kernel and variant gives the same bits."""
from __future__ import annotations

import math

import numpy as np
import pytest

import spintrack as st
from spintrack.adjoint import NUM_THETA

pytestmark = pytest.mark.gpu

G = np.random.default_rng(3).normal(0.0, 1e-9, 9)


def options(axis, small=1.0, E=75e5, **kw):
    B0, yi = [0.0, 0.0, 0.0], [0.0, 0.0, 0.0]
    B0[axis] = 3e-6
    g = G * small
    base = dict(numParticles=40, dist="M", T=4.2, diffuse=0.2, gas_coll=False, gravity=True, Gx=g[0:3], Gy=g[3:6], Gz=g[6:9],
                B0=B0, yi=yi, E=tuple(E if c == (axis + 2) % 3 else 0.0 for c in range(3)), tf=0.02, ioutInt=0.01, seed=5,
                rtol=1e-12, atol=1e-12, h=1e-3, hmax=1.0, hmin=1e-8)
    base.update(kw)
    if not any(base["yi"]):
        base["yi"][axis] = 1.0
    return st.derive(st.make_options(**base))


GRADIENTS = {
    "along_1e-4": dict(E=0.0), "along_1e-5": dict(E=0.0, small=0.1), "along_1e-6": dict(E=0.0, small=0.01),
    "along_motional": dict(), "against": dict(yi=[-1.0, 0.0, 0.0]), "across": dict(yi=[0.0, 0.6, 0.8]), "tilted": dict(yi=[1.0, 1e-3, 0.0]),
}


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("name", sorted(GRADIENTS))
def test_gradients_of_a_loss_along_the_field(gpu, name, axis):
    import torch
    kw = dict(GRADIENTS[name])
    if "yi" in kw:
        kw["yi"] = [kw["yi"][(c - axis) % 3] for c in range(3)]
    opt = options(axis, **kw)
    dev = torch.device("cuda", 0)
    w = torch.zeros(opt.numParticles, 3, dtype=torch.float64, device=dev)
    w[:, axis] = 1.0
    out = []
    with st.Particles(opt) as p:
        for scale in (1.0, 2.0 ** -850):
            ws = (w * scale).contiguous()
            grad = torch.empty(p.n, NUM_THETA, dtype=torch.float64, device=dev)
            p.init_particles()
            p.adjoint_record(st.num_windows(opt))
            torch.cuda.synchronize()
            p.adjoint_backward(ws.data_ptr(), grad.data_ptr())
            torch.cuda.synchronize()
            out.append((grad / scale).cpu().numpy())
    assert np.isfinite(out[0]).all()
    top = np.abs(out[1]).max(axis=0)
    assert (top[9:12] > 0).all()
    assert (np.abs(out[0] - out[1]) <= 1e-9 * top).all()


FORWARD = {
    "along": dict(), "across": dict(yi=[0.0, 1.0, 0.0]), "minus_zero": dict(yi=[0.0, -1.0, -0.0]), "tilted": dict(yi=[0.6, 0.0, -0.8]),
    "pulse": dict(yi=[0.0, -0.6, 0.8], a=5e-6, w=2 * math.pi * 1000.0, hmax=1e-4), "gas": dict(gas_coll=True, T=0.4, yi=[1.0, 1e-4, 0.0]),
}


def run(opt, kernel, variant=-1):
    import torch
    with st.Particles(opt) as p:
        if variant >= 0:
            p.set_launch_config(variant, 0)
        p.init_particles()
        p.run_windows(0, st.num_windows(opt), kernel)
        phase = torch.empty(p.n, dtype=torch.float64, device="cuda")
        p.gather_phase(phase.data_ptr())
        torch.cuda.synchronize()
        return p.output_data(), phase.cpu().numpy()


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("name", sorted(FORWARD))
def test_each_axis(gpu, oracle, name, axis):
    from _oracle import Options
    kw = dict(FORWARD[name])
    if "yi" in kw:
        kw["yi"] = [kw["yi"][(c - axis) % 3] for c in range(3)]
    opt = options(axis, **kw)
    oracle.set_math_mode(oracle.MATH_CR)
    try:
        _, ref = oracle.run_sample(Options.from_buffer_copy(bytes(opt)), 0, opt.numParticles)
    finally:
        oracle.set_math_mode(oracle.MATH_LIBM)
    got, phase = run(opt, st.KERNEL_PERSISTENT, 6)
    for f in ("fail", "n_coll", "n_bounce", "n_steps"):
        np.testing.assert_array_equal(got[f], ref[f], err_msg=f)
    assert np.max(np.abs(got["S"] - ref["S"])) <= 1e-9
    if axis == 0:
        # the phase counts whole turns: an error there is 2 pi; the across part may be 1e-4 of the spin.  (About another
        # axis than the field's the spin does not turn one way: it passes the cut near y = 0, where a step's end decides.)
        _, phase64 = run(options(axis, **dict(kw, beta=1e-300)), st.KERNEL_PERSISTENT, 6)
        assert np.max(np.abs(phase - phase64)) <= 1e-4
    for kernel, variant in ((st.KERNEL_PLAIN, -1), (st.KERNEL_PERSISTENT, 0), (st.KERNEL_PERSISTENT, 14), (st.KERNEL_PERSISTENT, 17)):
        again, phase2 = run(opt, kernel, variant)
        for f in got:
            np.testing.assert_array_equal(again[f], got[f], err_msg=f"{kernel} {variant} {f}")
        np.testing.assert_array_equal(phase2, phase)
