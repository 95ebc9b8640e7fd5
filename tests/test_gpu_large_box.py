"""FP32 engines in boxes on both sides of the largest one whose sites are kept in fixed point (2,048), and far
beyond it, with coordinates many boxes away: forces, torques and energies are the double engine's.

Clusters in a large box: forces and torques off by no more than twice what they are off in an ordinary box.  Contacts at the edge: pairs whose backbone sites are within 1e-5 to 4e-5 of the
excluded volume's cutoff, where its force is 0.02 to 0.1 (a slope of 2 eps b, about 3,600); a pair that the screen
misses is off by that
(in the largest of the boxes a fixed-point separation of them rounds up past the margin), while FP32 makes an error of 3,600 times the refined distance's 1e-8 and of the 1e-7 of a
Debye-Hueckel force below 0.1, together below 1e-4."""
import numpy as np
import pytest

from oxdna_gb300 import MDSystem, dna2_settings, md_settings
from oxdna_gb300 import generate as G
from oxdna_gb300 import io as oxio

pytestmark = pytest.mark.gpu

RC1 = 0.711879214356  # backbone-backbone cutoff of the excluded volume


def _both(box, top, T, state, **kw):
    out = []
    for precision in ("mixed", "double"):
        m = MDSystem(box, top, dna2_settings(T, 0.5), md_settings(dt=0.003, precision=precision, **kw))
        m.set_state(*state)
        out.append(m.compute_forces())
        if kw.get("thermostat") is None:
            m.run(20)
            out[-1] = out[-1] + (m.get_state()["pos"],)
        m.close()
    return out


@pytest.mark.parametrize("box", [2048.0, 2048.5, 30000.0, 100000.0])
def test_clusters_in_a_large_box(box):
    s = G.system_for_config(1, seed=31, scale=0.05)
    state = s.pos, s.quats(), s.vel, s.L
    a, b = _both(256.0, s.top, s.T, state)
    ordinary = [np.abs(a[k] - b[k]).max() for k in (0, 1)]
    rng = np.random.default_rng(1)
    shift = np.floor(rng.uniform(-20, 20, (s.N // 40, 3))) * box  # whole molecules, other images
    pos = s.pos + np.repeat(shift, 40, axis=0) + box * 0.5 - s.box / 2  # the cluster across a corner of the box
    a, b = _both(box, s.top, s.T, (pos,) + state[1:])
    for k in (0, 1):
        # (hi + lo keeps a coordinate of 20 boxes to 2^-48 of itself)
        assert np.abs(a[k] - b[k]).max() < 2.0 * ordinary[k] + 3600 * 20 * box * 2.0 ** -47
    assert np.abs(a[4] - b[4]).max() < 1e-3


@pytest.mark.parametrize("box", [600.0, 2048.0, 2049.0, 20000.0, RC1 * 2.0 ** 32 / 7500.3])
def test_contacts_at_the_edge(box):
    n = 1500
    rng = np.random.default_rng(2)
    side = 12
    cell = np.array(np.unravel_index(np.arange(n), (side, side, side))).T * (box / side)
    first = cell + rng.uniform(0.5, 0.7, (n, 3)) * (box / side)
    first[::10] = np.floor(first[::10] / (box / 2)) * (box / 2) - 0.3  # across faces and signs
    first[::10] += 4.0 * np.array(np.unravel_index(np.arange(len(first[::10])), (6, 6, 6))).T
    gap = RC1 * (1.0 - rng.uniform(1e-5, 4e-5, n))
    pos = np.empty((2 * n, 3))
    pos[0::2] = first
    pos[1::2] = first + np.array([0.0, 0.0, 1.0]) * gap[:, None]  # along a3: the other sites are out of reach
    quat = np.tile([0.0, 0.0, 0.0, 1.0], (2 * n, 1))
    none = np.full(2 * n, -1, np.int32)
    zero = np.zeros(2 * n, np.int32)
    top = oxio.Topology(none, none, zero, zero, np.arange(2 * n, dtype=np.int32), 2 * n)
    vel = np.zeros((2 * n, 3))
    a, b = _both(box, top, 0.1, (pos, quat, vel, vel), thermostat="no")
    assert np.ravel(b[3])[3] > 0.0  # there are contacts
    assert (np.abs(b[0][:, 2]) > 1e-2).mean() > 0.9
    # (hi + lo keeps a coordinate to 2^-48 of itself)
    assert np.abs(a[0] - b[0]).max() < 1e-4 + 3600 * box * 2.0 ** -46
