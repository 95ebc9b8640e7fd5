"""The double engine's kept FP64 frames: made by the first step, made anew by a sort, and read by every
force kernel.  A sorted run stays bit-identical to an unsorted one, and the forces of the state that a run
ends in are the FP64 oracle's, to 1e-10 of max(1, |F|_inf) (a few hundred roundings of 1e-16 of forces that
cancel to ~1e-3 of their terms).  Sizes below, at and above a group of 32 nucleotides and a block.
"""
import numpy as np
import pytest

import oracle
from oxdna_gb300 import MDSystem, dna2_settings, md_settings
from oxdna_gb300 import generate as G
from oxdna_gb300 import io as oxio

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 120, 680])
def test_frames_follow_steps_and_sorts(n):
    s = G.system_for_config(1, seed=n, scale=n / 40000.0)
    states = []
    for kw in (dict(), dict(sort_every=1), dict(sort_every=1, sort_order="cells")):
        m = MDSystem(s.box, s.top, dna2_settings(s.T, 0.5),
                     md_settings(precision="double", dt=0.003, thermostat="john", newtonian_steps=3, pt=0.2, seed=5,
                                 steps_per_graph=10, verlet_skin=0.03, **kw))
        m.set_state(s.pos, s.quats(), s.vel, s.L)
        m.run(57)
        F, T, _, _ = m.compute_forces()
        states.append((m.get_state(), F, T))
        assert m.info()["rebuilds"] >= 2
        m.close()
    st, F, T = states[0]
    for other, Fo, To in states[1:]:
        for key in ("pos", "quat", "vel", "Lmom"):
            assert np.array_equal(st[key], other[key]), key
        assert np.array_equal(F, Fo) and np.array_equal(T, To)
    a1, a2, a3 = oxio.quat_to_frame(st["quat"])
    p = oracle.make_params(oracle.make_settings(s.T, 0.5))
    rc, Fr, Tr, _, _ = oracle.forces(p, st["pos"], a1, a2, a3, s.top.n3, s.top.n5, s.top.type, s.top.btype, s.box)
    for got, want in ((F, Fr), (T, Tr)):
        err = np.abs(got - want).max(1) / np.maximum(1.0, np.abs(want).max(1))
        assert err.max() <= 1e-10, err.argmax()
