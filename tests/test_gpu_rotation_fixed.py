"""Quaternion steppers' segments at the edges of the fixed-point step's range (st_fixed.cuh): steps
small and above four radians, strong fields, pulses.
In range or not (those steps run in FP64), spins agree with the oracle's to 1e-9 of
the spin's norm per window, and the trajectory's counts are the oracle's, for both
kernels."""
from __future__ import annotations

import math

import numpy as np
import pytest

import spintrack as st

pytestmark = pytest.mark.gpu

G = np.random.default_rng(9).normal(0.0, 1e-9, 9)
BASE = dict(numParticles=33, dist="M", T=0.4, gas_coll=False, gravity=True, diffuse=0.1, Gx=G[0:3], Gy=G[3:6], Gz=G[6:9],
            E=(0.0, 0.0, 75e5), B0=(3e-6, 0.0, 0.0), yi=(0.0, 0.0, 1.0), t0=0.0, tf=0.02, ioutInt=0.01, seed=19, rtol=1e-12,
            atol=1e-12, h=1e-3, hmax=1.0, hmin=1e-10, integratorType=3)
CASES = {
    "rk45q": dict(integratorType=3, rtol=1e-9, tf=0.002, ioutInt=0.001),
    "rk45q_strong": dict(integratorType=3, rtol=1e-9, B0=(1e-4, 1e-5, 0.0), tf=0.0004, ioutInt=0.0002),
    "rk45q_pulse": dict(integratorType=3, rtol=1e-9, a=5e-6, w=-2 * math.pi * 1000.0, tf=0.002, ioutInt=0.001),
    "rkf45q": dict(integratorType=5, rtol=1e-6, tf=2e-5, ioutInt=1e-5),
    "rkf45q_coarse": dict(integratorType=5, rtol=3e-1, hmax=1e-3, tf=0.002, ioutInt=0.001),
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
    for f in ("fail", "n_coll", "n_bounce"):
        np.testing.assert_array_equal(got[f], ref[f], err_msg=f)
    norm = math.sqrt(opt.yi.x ** 2 + opt.yi.y ** 2 + opt.yi.z ** 2)
    np.testing.assert_allclose(got["S"], ref["S"], rtol=0, atol=1e-9 * norm)
