"""Step graphs of any length: the Bussi draws of all steps of a graph are made by one launch, which has to take
more steps than a grid's second dimension holds (65,535).  The draws depend on the seed and the step alone,
so a run is the same, bit for bit, however many steps its graphs hold."""
import numpy as np
import pytest

from oxdna_gb300 import MDSystem, dna2_settings, md_settings
from oxdna_gb300 import generate as G

pytestmark = pytest.mark.gpu


def test_graph_of_more_steps_than_a_grid_dimension():
    s = G.system_for_config(0, seed=3)
    n, states = 65536 + 4, []
    for steps in (64, n):
        m = MDSystem(s.box, s.top, dna2_settings(s.T, 0.5),
                     md_settings(dt=0.002, thermostat="bussi", newtonian_steps=1, seed=4, steps_per_graph=steps))
        m.set_state(s.pos, s.quats(), s.vel, s.L)
        m.run(n)
        states.append(m.get_state())
        m.close()
    for k in ("pos", "quat", "vel", "Lmom"):
        assert np.array_equal(states[0][k], states[1][k]), k
