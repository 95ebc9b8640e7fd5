"""Brownian redraws shared by a block of the first step, against the flush at the end of a run, which draws
per nucleotide: a run of n steps and n runs of one step end in the same bits.  Sizes at the edges of a warp
and of a block of 64 nucleotides; redraws in every step (blocks held to an even share per SM) and in every
third; in graphs (drawn before the wait for the forces) and single steps (after it).  (Not backend_precision =
float, whose flush makes its half kick in FP64 and so ends a rounding apart.)
"""
import numpy as np
import pytest

from oxdna_gb300 import MDSystem, dna2_settings, md_settings
from oxdna_gb300 import generate as G
from oxdna_gb300 import io as oxio

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "double"])
@pytest.mark.parametrize("n", [2, 31, 33, 64, 65, 127, 200])
def test_shared_redraws_match_single_ones(n, precision):
    s = G.system_for_config(1, seed=n, scale=(n + 40) / 40000.0)
    n3, n5 = s.top.n3[:n].copy(), s.top.n5[:n].copy()
    n3[n3 >= n] = -1
    n5[n5 >= n] = -1
    top = oxio.Topology(n3, n5, s.top.btype[:n], s.top.type[:n], np.zeros(n, np.int32), 1)
    for every in (1, 3):
        ends = []
        for chunks in ([1] * 10, [10]):
            m = MDSystem(s.box, top, dna2_settings(s.T, 0.5),
                         md_settings(precision=precision, dt=0.002, thermostat="john", newtonian_steps=every, pt=0.4, seed=9,
                                     steps_per_graph=5))
            m.set_state(s.pos[:n], s.quats()[:n], s.vel[:n], s.L[:n])
            start = m.get_state()["vel"]
            for c in chunks:
                m.run(c)
            ends.append(m.get_state())
            m.close()
        for key in ("pos", "quat", "vel", "Lmom"):
            assert np.array_equal(ends[0][key], ends[1][key]), (every, key)
        assert not np.array_equal(ends[0]["vel"], start)
