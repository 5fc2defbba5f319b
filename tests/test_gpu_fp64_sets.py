"""Runs in which no set steps in fixed point (beta, an absolute tolerance far below the relative one, RK45) have kernels of
their own: every variant's output is the plain kernel's, bit for bit, also where such sets share a context with
fixed-point ones, and st_set_params changes over in both directions."""
from __future__ import annotations

import numpy as np
import pytest

import spintrack as st
from spintrack import _capi
from spintrack.adjoint import NUM_THETA

pytestmark = pytest.mark.gpu

G = np.random.default_rng(8).normal(0.0, 1e-9, 9)
BASE = dict(numParticles=70, dist="M", T=0.4, gravity=True, diffuse=0.2, Gx=G[0:3], Gy=G[3:6], Gz=G[6:9], E=(0.0, 0.0, 75e5),
            B0=(3e-6, 0.0, 0.0), yi=(0.0, 0.0, 1.0), tf=0.02, ioutInt=0.01, seed=17, rtol=1e-12, atol=1e-12, hmax=1.0, hmin=1e-8)
CASES = {
    "beta": dict(beta=0.04), "atol_small": dict(atol=1e-16), "atol_zero": dict(atol=0.0, rtol=1e-10, yi=(0.3, 0.4, 0.5)),
    "rk45": dict(integratorType=1, tf=2e-5, ioutInt=1e-5), "norm": dict(yi=(3000.0, 0.0, 4000.0), atol=1e-13),
    "trajectory_only": dict(integratorType=9),
    "radians": dict(rtol=1e-5, atol=1e-5, gas_coll=False), "fixed_step_radians": dict(fixedStepSize=True, h=4e-3, nmax=20),
    "hmin_long": dict(hmin=3e-4), "hmin_past_collisions": dict(T=1.39, tf=2e-6, ioutInt=1e-6),
}


def options(**kw):
    return st.derive(st.make_options(**{**BASE, **kw}))


def run(opts, kernel, variant=-1):
    with st.Particles(opts) as p:
        if variant >= 0:
            try:
                p.set_launch_config(variant, 0)
            except st.SpinTrackError:
                return None  # no such kernel for these types
        p.init_particles()
        p.run_windows(0, 2, kernel)
        return p.output_data()


def same(a, b, what):
    for f in a:
        np.testing.assert_array_equal(a[f], b[f], err_msg=f"{what} {f}")


@pytest.mark.parametrize("gas", [False, True])
@pytest.mark.parametrize("name", sorted(CASES))
def test_every_variant_matches_plain(gpu, name, gas):
    opt = options(**{"gas_coll": gas, **CASES[name]})
    ref = run(opt, st.KERNEL_PLAIN)
    ran = 0
    for v in range(_capi.load().st_launch_variant_count()):
        got = run(opt, st.KERNEL_PERSISTENT, v)
        if got is not None:
            same(got, ref, st.variant_name(v))
            ran += 1
    assert ran >= 18


def test_mixed_with_fixed_point_sets(gpu):
    sets = [options(), options(beta=0.04, seed=400), options(atol=1e-16, seed=500)]
    got = run(sets, st.KERNEL_PERSISTENT)
    parts = [run(o, st.KERNEL_PLAIN) for o in sets]
    same(got, {f: np.concatenate([p[f] for p in parts]) for f in got}, "mixed")


def test_set_params_changes_over(gpu):
    a, b = options(), options(beta=0.04)
    with st.Particles(a) as p:
        for opt in (a, b, a):
            p.set_params([opt])
            for _ in range(2):  # the second from a captured graph
                p.init_particles()
                p.run_windows(0, 2)
                same(p.output_data(), run(opt, st.KERNEL_PLAIN), "set_params")


@pytest.mark.parametrize("gas", [False, True])
def test_record_and_backward(gpu, gas):
    import torch
    grads = []
    for kw in (dict(), dict(beta=1e-300)):  # the second steps in FP64 with the same step sizes
        with st.Particles(options(gas_coll=gas, **kw)) as p:
            w = torch.ones(p.n, 3, dtype=torch.float64, device="cuda")
            grad = torch.empty(p.n, NUM_THETA, dtype=torch.float64, device="cuda")
            p.init_particles()
            p.adjoint_record(2)
            p.adjoint_backward(w.data_ptr(), grad.data_ptr())
            torch.cuda.synchronize()
            grads.append(grad.cpu().numpy())
    top = np.abs(grads[1]).max(axis=0)
    assert (np.abs(grads[0] - grads[1]) <= 1e-9 * top).all()


def test_split_waits_for_a_long_segment(gpu):
    """One segment of twenty million fixed steps keeps a consumer for longer than the producers' idle limit."""
    opt = options(numParticles=3, tf=0.04, ioutInt=0.02, diffuse=0.1, gas_coll=False, fixedStepSize=True, h=2e-3, nmax=20000000, beta=1e-300)
    ref = run(opt, st.KERNEL_PERSISTENT, 3)
    same(run(opt, st.KERNEL_PERSISTENT, 14), ref, "split")
