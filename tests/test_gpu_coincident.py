"""Nucleotides on top of one another have no finite energy: no term may leave them out, so that a broken
configuration shows in every precision, in the total and in the Debye-Hueckel and excluded-volume sums."""
import numpy as np
import pytest

from oxdna_gb300 import MDSystem, dna2_settings, md_settings
from oxdna_gb300 import io as oxio

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "float", "double"])
def test_coincident_nucleotides(precision):
    n = 4
    pos = np.array([[1.0, 2.0, 3.0], [1.0, 2.0, 3.0], [9.0, 9.0, 9.0], [9.0, 9.0, 15.0]])
    none, zero = np.full(n, -1, np.int32), np.zeros(n, np.int32)
    m = MDSystem(30.0, oxio.Topology(none, none, zero, zero, np.arange(n, dtype=np.int32), n), dna2_settings(0.1, 0.5),
                 md_settings(precision=precision))
    m.set_state(pos, np.tile([0.0, 0.0, 0.0, 1.0], (n, 1)), np.zeros((n, 3)), np.zeros((n, 3)))
    F, T, E, split = m.compute_forces()
    split = np.ravel(split)
    assert not np.isfinite(split[7]) and not np.isfinite(split[3])
    assert not np.isfinite(E[0]) and not np.isfinite(E[1])
    assert np.all(np.isfinite(F[2:])) and np.all(np.isfinite(E[2:]))
    m.close()
