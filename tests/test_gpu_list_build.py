"""The one-kernel list build over the forms it takes: cells filled by one block (systems of up to 4096
nucleotides) or by the grid in phases, whole builds and rebuilds of single systems of a batch.

A batch that holds a system above the one-block limit fills all its cells in phases; the same systems
alone take the one-block form where they are small.  Rows are identical entry for entry either way, so
the trajectories are bit-identical (Brownian; the skin is narrow, so that systems go stale one by one).
"""
import numpy as np
import pytest

from oxdna_gb300 import MDSystem, dna2_settings, md_settings
from oxdna_gb300 import generate as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(4200, 40, 680), (4080, 40, 120), (40, 40)])
def test_partial_rebuilds_of_a_batch_match_the_systems_alone(sizes):
    systems = [G.system_for_config(1, seed=60 + k, scale=n / 40000.0) for k, n in enumerate(sizes)]
    assert [s.N for s in systems] == list(sizes)
    kw = dict(dt=0.003, thermostat="john", newtonian_steps=7, pt=0.2, verlet_skin=0.03)
    b = MDSystem([s.box for s in systems], [s.top for s in systems], [dna2_settings(s.T, 0.5) for s in systems],
                 md_settings(seed=5, **kw))
    b.set_state(*[np.concatenate(x) for x in zip(*[(s.pos, s.quats(), s.vel, s.L) for s in systems])])
    b.run(101)
    sb, rows_b, builds = b.get_state(), b.neighbours(), b.info()["rebuilds"]
    alone = 0
    for k, s in enumerate(systems):
        lo, hi = b.offsets[k], b.offsets[k + 1]
        m = MDSystem(s.box, s.top, dna2_settings(s.T, 0.5), md_settings(seed=5 + k, **kw))
        m.set_state(s.pos, s.quats(), s.vel, s.L)
        m.run(101)
        sm, rows = m.get_state(), m.neighbours()
        for key in ("pos", "quat", "vel", "Lmom"):
            assert np.array_equal(sb[key][lo:hi], sm[key]), (k, key)
        assert np.array_equal(rows_b[0][lo:hi], rows[0]), k
        for i in range(s.N):
            assert np.array_equal(rows_b[1][lo + i, :rows[0][i]] - lo, rows[1][i, :rows[0][i]]), (k, i)
        alone += m.info()["rebuilds"]
        m.close()
    # systems were rebuilt apart from each other
    assert builds < alone
    b.close()


def test_batches_beyond_a_blocks_systems_match_the_systems_alone():
    # more systems than a block has threads: the rows go through all nucleotides and test each
    one = [G.system_for_config(1, seed=70 + k, scale=40 / 40000.0) for k in range(3)]
    n = 1030
    kw = dict(dt=0.003, thermostat="john", newtonian_steps=7, pt=0.2, verlet_skin=0.03)
    s = [one[k % 3] for k in range(n)]
    b = MDSystem([x.box for x in s], [x.top for x in s], [dna2_settings(x.T, 0.5) for x in s], md_settings(seed=5, **kw))
    b.set_state(*[np.concatenate(x) for x in zip(*[(x.pos, x.quats(), x.vel, x.L) for x in s])])
    b.run(41)
    sb, rows_b = b.get_state(), b.neighbours()
    for k in (0, 511, 1023, 1024, 1029):
        m = MDSystem(s[k].box, s[k].top, dna2_settings(s[k].T, 0.5), md_settings(seed=5 + k, **kw))
        m.set_state(s[k].pos, s[k].quats(), s[k].vel, s[k].L)
        m.run(41)
        sm, rows = m.get_state(), m.neighbours()
        lo, hi = b.offsets[k], b.offsets[k + 1]
        for key in ("pos", "quat", "vel", "Lmom"):
            assert np.array_equal(sb[key][lo:hi], sm[key]), (k, key)
        assert np.array_equal(rows_b[0][lo:hi], rows[0]), k
        m.close()
    assert b.info()["rebuilds"] >= 2
    b.close()
