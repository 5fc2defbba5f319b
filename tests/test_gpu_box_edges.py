"""A box edge below zero: every position is out of bounds, so each particle stops at its
first event with failure 1, as the reference's sanity check has it, in every kernel."""
from __future__ import annotations

import numpy as np
import pytest

import spintrack as st

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("edge", [0, 1, 2])
@pytest.mark.parametrize("kernel", [st.KERNEL_PERSISTENT, st.KERNEL_PLAIN], ids=["persistent", "plain"])
def test_negative_edge_stops_every_particle(gpu, oracle, kernel, edge):
    from _oracle import Options
    L = [0.4, 0.3, 0.5]
    L[edge] = -L[edge]
    opt = st.derive(st.make_options(numParticles=37, L=tuple(L), gas_coll=False, tf=0.02, ioutInt=0.01, seed=3))
    _, ref = oracle.run_sample(Options.from_buffer_copy(bytes(opt)), 0, opt.numParticles)
    assert np.all(ref["fail"] == 1)
    with st.Particles(opt) as p:
        p.init_particles()
        p.run_windows(0, st.num_windows(opt), kernel)
        got = p.output_data()
    for f in ("fail", "n_steps", "n_bounce", "n_coll"):
        np.testing.assert_array_equal(got[f], ref[f], err_msg=f)
