"""Debye-Hueckel from fixed-point sites: their unit, box / 2^32, is no FP32 number, and rounded it would scale
every distance of a box by the same factor.  A solution of duplexes in the middle of the box has the same
Debye-Hueckel energy in any larger box, so the energies in boxes whose unit (or its square) rounds badly are
compared with that in a box of 128, whose unit is exact.  What may differ are the roundings of single pairs: of a
site half a unit and of a pair's FP32 operations a few 6e-8 of its energy, at random, some thousands of pairs, so
well under 4e-8 of the sum; the rounded unit itself would shift it by (1 + kappa r) / 2 of its square's error,
1e-7 and more."""
import numpy as np
import pytest

from oxdna_gb300 import MDSystem, dna2_settings, md_settings
from oxdna_gb300 import generate as G

pytestmark = pytest.mark.gpu


def _square_error(box):
    unit = np.float32(box / 2.0 ** 32)
    return abs(float(unit * unit) / (box / 2.0 ** 32) ** 2 - 1.0)


def test_energy_does_not_depend_on_the_box():
    s = G.system_for_config(1, seed=12, scale=0.03)
    pos = s.pos - s.pos.mean(0)
    assert 2.0 * np.abs(pos).max() + 8.0 < 128.0  # nothing near a face
    boxes = [b for b in np.linspace(130.0, 900.0, 40001) if _square_error(b) > 1.5e-7][::4][:12]
    assert len(boxes) >= 6
    energy = []
    for box in [128.0] + boxes:
        m = MDSystem(float(box), s.top, dna2_settings(s.T, 0.2), md_settings())
        m.set_state(pos, s.quats(), s.vel, s.L)
        energy.append(float(np.ravel(m.compute_forces()[3])[7]))
        m.close()
    shift = np.abs(np.array(energy[1:]) / energy[0] - 1.0)
    assert shift.max() < 4e-8, shift
