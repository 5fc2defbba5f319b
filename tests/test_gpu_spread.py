"""Particle counts at the edges of the lane spreading (spread_lanes: 2 warps per
SM before warps fill up): a particle's result does not depend on how many lanes
of its warp work, so every count's output is that of the full ensemble's first
particles, bit for bit, in every kernel and variant."""
from __future__ import annotations

import numpy as np
import pytest

import spintrack as st

pytestmark = pytest.mark.gpu

BASE = dict(dist="M", T=0.4, diffuse=0.3, E=(0.0, 0.0, 75e5), B0=(3e-6, 0.0, 0.0), yi=(0.0, 0.0, 1.0), t0=0.0, tf=0.004,
            ioutInt=0.002, seed=29, rtol=1e-10, atol=1e-10, hmax=1.0, hmin=1e-9)


def run(n, kernel, variant=-1, **kw):
    opt = st.derive(st.make_options(**{**BASE, **kw, "numParticles": n}))
    with st.Particles(opt) as p:
        if variant >= 0:
            p.set_launch_config(variant, 0)
        p.init_particles()
        p.run_windows(0, st.num_windows(opt), kernel)
        return p.output_data()


@pytest.mark.parametrize("gas", [False, True])
@pytest.mark.parametrize("integrator", [0, 1, 2])
def test_counts_at_the_edges(gpu, gas, integrator):
    import torch
    warps = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    kw = dict(gas_coll=gas, integratorType=integrator)
    if integrator == 1:
        kw.update(tf=2e-5, ioutInt=1e-5)
    full = run(32 * warps, st.KERNEL_PERSISTENT, 0, **kw)
    for n in (1, 31, warps - 1, warps, warps + 1, 3 * warps + 1, 31 * warps, 31 * warps + 1):
        for kernel, variant in ((st.KERNEL_PLAIN, -1), (st.KERNEL_PERSISTENT, 0), (st.KERNEL_PERSISTENT, 5), (st.KERNEL_PERSISTENT, 6)):
            got = run(n, kernel, variant, **kw)
            for f in full:
                np.testing.assert_array_equal(got[f], full[f][:n], err_msg=f"{n} {kernel} {variant} {f}")
