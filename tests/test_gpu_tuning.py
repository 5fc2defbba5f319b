"""The launch configuration that one context tuned serves later contexts of the process only where they share what the
choice hangs on: not across gas and no gas, and not across the edge of the lane spreading (62 particles per SM), from
which on the warp-specialised variants are no candidates."""
from __future__ import annotations

import numpy as np
import pytest

import spintrack as st

pytestmark = pytest.mark.gpu

G = np.random.default_rng(3).normal(0.0, 1e-9, 9)
BASE = dict(dist="M", gravity=True, diffuse=0.1, Gx=G[0:3], Gy=G[3:6], Gz=G[6:9], E=(0.0, 0.0, 75e5), B0=(3e-6, 0.0, 0.0),
            yi=(0.0, 0.0, 1.0), tf=0.05, ioutInt=0.05, seed=5, rtol=1e-12, atol=1e-12, hmax=1.0, hmin=1e-8)


def choice(**kw):
    opt = st.derive(st.make_options(**{**BASE, **kw}))
    with st.Particles(opt) as p:
        p.init_particles()
        p.run_windows(0, st.num_windows(opt))
        return st.variant_name(p.launch_config()[0])


def test_gas_is_tuned_by_itself(gpu):
    choice(numParticles=300, T=4.2, gas_coll=False)  # a warp-specialised variant wins (4.6 ms against 5.2)
    # with gas it takes nearly three times as long as the best
    assert not choice(numParticles=300, T=0.4, gas_coll=True).startswith("split")


@pytest.mark.parametrize("diffuse", [0.1, 0.11], ids=["small_first", "large_first"])
def test_edge_of_the_spreading(gpu, diffuse):
    import torch
    edge = 62 * torch.cuda.get_device_properties(0).multi_processor_count
    counts = [edge, edge + 1] if diffuse == 0.1 else [edge + 1, edge]
    names = {n: choice(numParticles=n, T=4.2, gas_coll=False, diffuse=diffuse, tf=0.004, ioutInt=0.002) for n in counts}
    assert not names[edge + 1].startswith("split")


def test_short_windows_are_ranked_as_they_come(gpu):
    # three windows of 12 ms: the variants with six blocks per SM lose a third, in a single window they lead
    name = choice(numParticles=67001, T=4.2, gas_coll=False, dist="C", integratorType=2, tf=0.0367, ioutInt=0.0367 / 3)
    assert "_m4_" in name or "_b256_m1_" in name, name
