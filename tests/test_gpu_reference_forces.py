"""Forces on the reference's device layout at every lane count (32, 16 and 8 lanes per nucleotide, by the
number of nucleotides) and at the edges of a block's 4, 8 or 16 nucleotides, rows of either stride, added
to what the buffers held.

The oracle gets the FP32 positions and quaternions that the kernel gets (the forces of generated strands
move by 2e-4 when their positions are rounded to FP32).  A separation still carries the rounding of one
minimum image, and the stiffest term (FENE) amplifies it: normwise 1e-4 and per nucleotide 1e-3 of
max(|F|, 0.1 RMS |F|), as for every force of this layout.
"""
import ctypes as C

import numpy as np
import pytest

import oracle
from gpu_util import force_errors
from oxdna_gb300 import _abi, dna2_settings
from oxdna_gb300 import generate as G
from oxdna_gb300 import io as oxio

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,rows_first", [(40, True), (1000, False), (2420, True), (2460, False),
                                          (4840, True), (4880, False), (4680, True), (4720, False),
                                          (9360, True), (9400, True), (9400, False), (12040, False)])
def test_forces_match_the_oracle(n, rows_first):
    s = G.system_for_config(1, seed=n, scale=n / 40000.0)
    # the last strand's tail cut off: a ragged number of nucleotides, its end unpaired
    N = s.N - 3
    n3, n5 = s.top.n3[:N].copy(), s.top.n5[:N].copy()
    n3[n3 >= N] = -1
    n5[n5 >= N] = -1
    box = s.box
    pos, q = (x[:N].astype(np.float32).astype(np.float64) for x in (s.pos, s.quats()))
    p = oracle.make_params(oracle.make_settings(s.T, 0.5))
    a1, a2, a3 = oxio.quat_to_frame(q)
    rc, Fo, To, so, _ = oracle.forces(p, pos, a1, a2, a3, n3, n5, s.top.type[:N], s.top.btype[:N], box)

    pairs = np.asarray(oracle.pairs_within(pos, box, p.rcut))
    i, j = pairs.T
    pairs = pairs[(n3[i] != j) & (n5[i] != j)]
    pairs = np.concatenate([pairs, pairs[:, ::-1]])
    pairs = pairs[np.argsort(pairs[:, 0], kind="stable")]
    count = np.bincount(pairs[:, 0], minlength=N).astype(np.int32)
    width = int(count.max()) + 1
    matrix = np.zeros((N, width), np.int32)
    matrix[pairs[:, 0], np.arange(len(pairs)) - np.repeat(np.cumsum(count) - count, count)] = pairs[:, 1]
    p4 = np.zeros((N, 4), np.float32)
    p4[:, :3] = pos
    p4[:, 3] = ((s.top.btype[:N].astype(np.int32) << 22) | np.arange(N, dtype=np.int32)).view(np.float32)
    d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in
         (p4, q.astype(np.float32), np.stack([n3, n5], 1).astype(np.int32),
          matrix if rows_first else matrix.T, count)]
    F = torch.full((N, 4), 0.25, dtype=torch.float32, device="cuda")
    T = torch.full((N, 4), -0.5, dtype=torch.float32, device="cuda")
    L, h = _abi.lib(), C.c_void_p()
    _abi.check(L.oxgb_dna2_create(C.byref(dna2_settings(s.T, 0.5)), C.byref(h)))
    strides = (width, 1) if rows_first else (1, N)
    _abi.check(L.oxgb_dna2_compute_forces(h, N, box, d[0].data_ptr(), d[1].data_ptr(), F.data_ptr(), T.data_ptr(),
                                          d[2].data_ptr(), d[3].data_ptr(), d[4].data_ptr(), width, *strides, None))
    torch.cuda.synchronize()
    _abi.check(L.oxgb_dna2_destroy(h))
    F, T = F.cpu().numpy().astype(np.float64), T.cpu().numpy().astype(np.float64)
    for got, want in ((F[:, :3] - 0.25, Fo), (T[:, :3] + 0.5, To)):
        worst, norm = force_errors(got, want)
        assert norm <= 1e-4 and worst <= 1e-3, (worst, norm)
    assert abs((F[:, 3] - 0.25).sum() / 2 - so.sum()) <= 1e-4 * abs(so).sum()
    # the hydrogen-bonding energy is stored, not added
    assert abs(T[:, 3].sum() / 2 - so[4]) <= 1e-4 * max(1.0, abs(so[4]))
