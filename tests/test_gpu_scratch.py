"""Device memory of the trajectory-ahead kernel's rings: a context holds what its own launch configuration needs, and where
that does not fit it runs with fewer blocks, with the same results."""
from __future__ import annotations

import numpy as np
import pytest

import spintrack as st
from spintrack.adjoint import NUM_THETA

pytestmark = pytest.mark.gpu

G = np.random.default_rng(3).normal(0.0, 1e-9, 9)
MB = 2 ** 20


def options(n=60000):
    return st.derive(st.make_options(numParticles=n, dist="M", T=4.2, gas_coll=False, gravity=True, diffuse=0.1, Gx=G[0:3], Gy=G[3:6],
                                     Gz=G[6:9], E=(0.0, 0.0, 75e5), B0=(3e-6, 0.0, 0.0), yi=(0.0, 0.0, 1.0), tf=0.004, ioutInt=0.002,
                                     seed=5, rtol=1e-10, atol=1e-10))


def variant(name):
    return next(v for v in range(25) if st.variant_name(v) == name)


def run(p):
    p.init_particles()
    p.run_windows(0, 2)
    return p.output_data()


def test_rings_of_the_configuration_in_use(gpu):
    import torch
    with st.Particles(options(100)) as p:  # the library's own start-up allocations
        p.set_launch_config(variant("ahead_b64_m4_q32_s4"), 0)
        run(p)
    with st.Particles(options()) as p:
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        p.set_launch_config(variant("ahead_b64_m4_q32_s4"), 0)
        run(p)
        used = before - torch.cuda.mem_get_info()[0]
    # 256 lanes per SM of 32 records and five states, 112 bytes each, and a graph
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert used <= 256 * sms * 37 * 112 + 32 * MB, used / MB


def test_short_of_memory(gpu):
    import torch
    opt = options()
    with st.Particles(opt) as ref, st.Particles(opt) as p:
        ref.set_launch_config(variant("ahead_b64_m4_q128_s4"), 0)  # 580 MB of rings on 152 SMs
        want = run(ref)
        ref.close()
        p.set_launch_config(variant("ahead_b64_m4_q128_s4"), 0)
        p.init_particles()
        torch.cuda.synchronize()
        hold = torch.empty(torch.cuda.mem_get_info()[0] - 400 * MB, dtype=torch.uint8, device="cuda")
        try:
            for _ in range(2):  # the second time without another try for the whole
                got = run(p)
                for f in want:
                    np.testing.assert_array_equal(got[f], want[f], err_msg=f)
        finally:
            del hold
            torch.cuda.empty_cache()


def test_record_short_of_memory(gpu):
    import torch
    opt = options(45000)
    grads = []
    for short in (False, True):
        with st.Particles(opt) as p:
            w = torch.ones(p.n, 3, dtype=torch.float64, device="cuda")
            grad = torch.empty(p.n, NUM_THETA, dtype=torch.float64, device="cuda")
            p.init_particles()
            torch.cuda.synchronize()
            hold = torch.empty(torch.cuda.mem_get_info()[0] - 900 * MB, dtype=torch.uint8, device="cuda") if short else None
            try:
                p.adjoint_record(2, tape_bytes=512 * MB)
                p.adjoint_backward(w.data_ptr(), grad.data_ptr())
                torch.cuda.synchronize()
                grads.append(grad.cpu().numpy())
            finally:
                del hold
                torch.cuda.empty_cache()
    np.testing.assert_array_equal(grads[0], grads[1])
