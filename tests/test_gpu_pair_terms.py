"""The pair-term blocks (hydrogen bonding, cross and coaxial stacking by eight lanes per term) on crowded
random states, where a group of 32 nucleotides owns from no pair to several hundred live ones, pairs
have two terms at once and every angular factor is met on both sides of its range.

Half of the nucleotides come as pairs at hydrogen-bonding or stacking distance, turned a little; the
others anywhere, with no bonds.  Checked against the FP64 oracle, per nucleotide relative to max(1,
|F|_inf): the double engine to 1e-10 (a few hundred roundings of 1e-16 of forces that cancel to ~1e-3 of
their terms), the mixed engine to 1e-5, the bound of its forces everywhere else.  Sizes at the edges of
the groups (one, 32 +- 1) and of the chunks of queued items.
"""
import numpy as np
import pytest

import oracle
from oxdna_gb300 import MDSystem, dna2_settings, md_settings
from oxdna_gb300 import generate as G
from oxdna_gb300 import io as oxio

pytestmark = pytest.mark.gpu


def crowded(n, box, seed):
    rng = np.random.default_rng(seed)
    pos = rng.uniform(0, box, (n, 3))
    frames = np.array([G.random_rotation(rng) for _ in range(n)])
    base = rng.integers(0, 4, n)
    for k in range(0, n - 1, 4):
        v = rng.normal(size=3) * 0.35
        K = np.array([[0, -v[2], v[1]], [v[2], 0, -v[0]], [-v[1], v[0], 0]])
        t = np.linalg.norm(v)
        turn = np.eye(3) + np.sin(t) / t * K + (1 - np.cos(t)) / t**2 * K @ K
        facing = k % 8 == 0  # across a base pair, or stacked on top of each other
        frames[k + 1] = frames[k] @ np.diag([-1.0, 1.0, -1.0] if facing else [1.0, 1.0, 1.0]) @ turn
        pos[k + 1] = pos[k] + frames[k] @ (np.array([1.2, 0, 0] if facing else [0, 0, 0.42]) + rng.normal(size=3) * 0.1)
        base[k + 1] = 3 - base[k]
    none = np.full(n, -1, np.int32)
    top = oxio.Topology(none, none, base.astype(np.int32), base.astype(np.int32), np.zeros(n, np.int32), 1)
    return pos, frames[:, :, 0], frames[:, :, 1], frames[:, :, 2], top


@pytest.mark.parametrize("precision,tol", [("double", 1e-10), ("mixed", 1e-5)])
@pytest.mark.parametrize("n,box", [(2, 9.0), (31, 9.0), (33, 9.0), (64, 9.0), (129, 9.0), (600, 11.0), (1500, 11.0)])
def test_crowded_pairs_match_the_oracle(n, box, precision, tol):
    pos, a1, a2, a3, top = crowded(n, box, 100 + n)
    q = oxio.frame_to_quat(a1, a2, a3)
    a1, a2, a3 = oxio.quat_to_frame(q)
    m = MDSystem(box, top, dna2_settings(0.1, 0.5), md_settings(precision=precision))
    m.set_state(pos, q, np.zeros((n, 3)), np.full((n, 3), 1e-3))
    F, T, _, split = m.compute_forces()
    Fs, Ts, _ = m.get_forces()  # the MD step's variant, without energies
    m.close()
    p = oracle.make_params(oracle.make_settings(0.1, 0.5))
    rc, Fo, To, so, _ = oracle.forces(p, pos, a1, a2, a3, top.n3, top.n5, top.type, top.btype, box)
    for got, want in ((F, Fo), (T, To), (Fs, Fo), (Ts, To)):
        err = np.abs(got - want).max(1) / np.maximum(1.0, np.abs(want).max(1))
        assert err.max() <= tol, err.argmax()
    # hydrogen bonding, cross stacking, coaxial stacking, each a sum of n or so terms of order one
    assert np.abs(split[4:7] - so[4:7]).max() <= tol * max(1.0, np.abs(so[4:7]).max())
    if n >= 129:
        assert np.all(so[4:7] != 0.0)
