"""Particles of few segments: a ring holds many of them, and lanes must not take them all ahead while others go
without.  65,536 RKF45 particles of seven segments on some 38,000 lanes: the trajectory-ahead kernel takes about as long as
the flattened one, whose lanes take a particle when they are free (1.8 times as long when rings were filled)."""
from __future__ import annotations

import time

import numpy as np
import pytest

import spintrack as st

pytestmark = pytest.mark.gpu

G = np.random.default_rng(3).normal(0.0, 1e-9, 9)


def test_last_particles_are_dealt_evenly(gpu):
    opt = st.derive(st.make_options(numParticles=65536, dist="M", T=4.2, gas_coll=False, gravity=True, diffuse=0.1, Gx=G[0:3], Gy=G[3:6],
                                    Gz=G[6:9], E=(0.0, 0.0, 75e5), B0=(3e-6, 0.0, 0.0), yi=(0.0, 0.0, 1.0), tf=0.005, ioutInt=0.005,
                                    seed=5, rtol=1e-3, atol=1e-12, integratorType=4))
    names = {st.variant_name(v): v for v in range(25) if st.variant_name(v) != "?"}
    took, out = {}, {}
    with st.Particles(opt) as p:
        for name in ("flat_b64_m4", "ahead_b64_m4_q64_s1"):
            p.set_launch_config(names[name], 0)
            best = 1e9
            for _ in range(3):
                p.init_particles()
                t = time.perf_counter()
                p.run_windows(0, 1)
                best = min(best, time.perf_counter() - t)
            took[name], out[name] = best, p.output_data()
    for f, v in out["flat_b64_m4"].items():
        np.testing.assert_array_equal(v, out["ahead_b64_m4_q64_s1"][f], err_msg=f)
    assert took["ahead_b64_m4_q64_s1"] < 1.4 * took["flat_b64_m4"], took
