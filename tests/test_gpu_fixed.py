"""DOP853 segments at the edges of the fixed-point step's range (st_fixed.cuh):
steps that start above one radian, loose tolerances, absolute tolerances far
from the relative ones, a beta controller, fixed steps, spins of other norms
and directions, pulses of either sign of w, starts before time zero, no field at
all.  Inside the range or not (those steps run in FP64), counts equal the
oracle's and spins agree to 1e-9 of the spin's norm, for both kernels."""
from __future__ import annotations

import math

import numpy as np
import pytest

import spintrack as st

pytestmark = pytest.mark.gpu

G = np.random.default_rng(8).normal(0.0, 1e-9, 9)
BASE = dict(numParticles=33, dist="M", T=0.4, gas_coll=False, gravity=True, diffuse=0.1, Gx=G[0:3], Gy=G[3:6], Gz=G[6:9],
            E=(0.0, 0.0, 75e5), B0=(3e-6, 0.0, 0.0), yi=(0.0, 0.0, 1.0), t0=0.0, tf=0.04, ioutInt=0.02, seed=17, rtol=1e-12,
            atol=1e-12, h=1e-3, hmax=1.0, hmin=1e-8)
CASES = {
    "strong_field": dict(B0=(1e-4, 2e-5, 0.0), tf=0.01, ioutInt=0.005),
    "loose": dict(rtol=1e-3, atol=1e-3),
    "steep_gradient": dict(Gx=(1e-5, 2e-5, 0.0), Gy=(0.0, -1e-5, 1e-5), Gz=(3e-6, 0.0, 0.0), tf=0.01, ioutInt=0.005),
    "atol_large": dict(rtol=1e-12, atol=1e-9),
    "atol_zero": dict(rtol=1e-10, atol=0.0, yi=(0.3, 0.4, 0.5)),
    "rtol_zero": dict(rtol=0.0, atol=1e-12),
    "beta": dict(beta=0.04),
    "fixed_step": dict(fixedStepSize=True, h=5e-5),
    "fixed_step_coarse": dict(fixedStepSize=True, h=2e-3),
    "norm_large": dict(yi=(60.0, -80.0, 35.0), atol=1e-10),
    "norm_small": dict(yi=(0.0, 3e-4, -4e-4)),
    "pulse_back": dict(a=5e-6, w=-2 * math.pi * 1000.0, hmax=1e-4, t0=-0.02, tf=0.02),
    "pulse_free": dict(a=4e-6, w=2 * math.pi * 300.0),
    "constant_pulse": dict(a=1e-6, w=0.0),
    "no_field": dict(B0=(0.0, 0.0, 0.0), E=(0.0, 0.0, 0.0), Gx=(0.0, 0.0, 0.0), Gy=(0.0, 0.0, 0.0), Gz=(0.0, 0.0, 0.0)),
    "keep_step": dict(keepStepSize=True, gas_coll=True),
    "no_gravity": dict(gravity=False, hmax=2e-5),
}


@pytest.mark.parametrize("kernel", [st.KERNEL_PERSISTENT, st.KERNEL_PLAIN], ids=["persistent", "plain"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_edges_of_the_fixed_point_range(gpu, oracle, name, kernel):
    from _oracle import Options
    opt = st.derive(st.make_options(**{**BASE, **CASES[name]}))
    oracle.set_math_mode(oracle.MATH_CR)
    try:
        _, ref = oracle.run_sample(Options.from_buffer_copy(bytes(opt)), 0, opt.numParticles)
    finally:
        oracle.set_math_mode(oracle.MATH_LIBM)
    with st.Particles(opt) as p:
        p.init_particles()
        p.run_windows(0, st.num_windows(opt), kernel)
        got = p.output_data()
    for f in ("fail", "n_coll", "n_bounce", "n_steps"):
        np.testing.assert_array_equal(got[f], ref[f], err_msg=f)
    assert np.array_equal(np.isnan(got["S"]), np.isnan(ref["S"]))
    norm = math.sqrt(opt.yi.x ** 2 + opt.yi.y ** 2 + opt.yi.z ** 2)
    m = ~np.isnan(ref["S"])
    # the two follow the same tolerance with step sequences that differ in the last bits of h
    assert np.max(np.abs(got["S"][m] - ref["S"][m])) <= 1e-9 * norm
