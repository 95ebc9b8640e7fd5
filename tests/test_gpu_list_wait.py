"""A list build that gives up at its barrier: it ends, it is reported, and nothing of it reaches later builds.

The wait is made to run out by its limit (no polls at all: whoever arrives at the barrier before the last
block leaves).  Until the status has been read every further build ends the same way; after that the next
one is whole, so its rows, and an engine's trajectory from the same state, are those of an undisturbed run,
entry for entry and bit for bit.  A build by one block has no barrier and cannot give up.
"""
import ctypes as C

import numpy as np
import pytest

from oxdna_gb300 import MDSystem, _abi, dna2_settings, md_settings
from oxdna_gb300 import generate as G

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

E_CUDA = 2


class _View:
    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<i4", "data": (int(ptr), False), "version": 3,
                                         "strides": None}


def _system(n):
    return G.system_for_config(1, seed=80, scale=n / 40000.0)


# cells by one block (up to 4,096 nucleotides) and by the grid
@pytest.mark.parametrize("n", [1000, 6000, 16000])
def test_plain_list(n):
    s = _system(n)
    L = _abi.lib()
    p = np.zeros((s.N, 4), np.float32)
    p[:, :3] = s.pos
    p[:, 3] = ((s.top.btype.astype(np.int32) << 22) | np.arange(s.N, dtype=np.int32)).view(np.float32)
    pos, bonds = torch.from_numpy(p).cuda(), torch.from_numpy(np.stack([s.top.n3, s.top.n5], 1).astype(np.int32)).cuda()
    at = torch.zeros_like(pos)
    v = C.c_void_p()
    _abi.check(L.oxgb_verlet_create(s.N, s.box, 3.2638, 0.05, 1, 0, C.byref(v)))
    nb, nnb, most = C.c_void_p(), C.c_void_p(), C.c_int()
    _abi.check(L.oxgb_verlet_buffers(v, C.byref(nb), C.byref(nnb), C.byref(most), None))
    rows = torch.as_tensor(_View(nb.value, (most.value, s.N)), device="cuda")
    counts = torch.as_tensor(_View(nnb.value, (s.N,)), device="cuda")

    def build():
        _abi.check(L.oxgb_verlet_update(v, pos.data_ptr(), at.data_ptr(), bonds.data_ptr(), None))
        torch.cuda.synchronize()

    def result():
        return rows.cpu().numpy().copy(), counts.cpu().numpy().copy()

    build()
    assert L.oxgb_verlet_status(v) == 0
    want = result()
    for _ in range(2):
        _abi.check(L.oxgb_verlet_set_list_wait(v, -1))
        build()
        _abi.check(L.oxgb_verlet_set_list_wait(v, 0))
        build()  # kept out: the status has not been read
        assert L.oxgb_verlet_status(v) == E_CUDA and b"list build" in L.oxgb_last_error()
        rows.fill_(-7)
        counts.fill_(-7)
        build()
        assert L.oxgb_verlet_status(v) == 0
        got = result()
        assert np.array_equal(want[1], got[1])
        valid = np.arange(most.value)[:, None] < want[1]
        assert np.array_equal(want[0][valid], got[0][valid])
    _abi.check(L.oxgb_verlet_destroy(v))


def _engine(systems, **kw):
    one = len(systems) == 1
    pick = (lambda x: x[0]) if one else list
    m = MDSystem(pick([s.box for s in systems]), pick([s.top for s in systems]),
                 pick([dna2_settings(s.T, 0.5) for s in systems]),
                 md_settings(dt=0.003, thermostat="john", newtonian_steps=7, pt=0.2, seed=5, verlet_skin=0.03, **kw))
    return m, [np.concatenate(x) for x in zip(*[(s.pos, s.quats(), s.vel, s.L) for s in systems])]


@pytest.mark.parametrize("sizes,kw", [((1000,), {}), ((6000,), {}), ((4200, 680), {}), ((1000, 680), {}),
                                      ((6000,), dict(sort_every=1)), ((1000,), dict(sort_every=1, sort_order="cells")),
                                      ((1000,), dict(precision="double"))])
def test_engine(sizes, kw):
    systems = [_system(n) for n in sizes]
    a, state = _engine(systems, **kw)
    a.set_state(*state)
    a.run(57)
    want = a.get_state()
    assert a.info()["rebuilds"] >= 3
    a.close()
    b, _ = _engine(systems, **kw)
    b.set_state(*state)
    L = _abi.lib()
    for _ in range(2):
        _abi.check(L.oxgb_md_set_list_wait(b.handle, -1))
        with pytest.raises(_abi.OxgbError, match="list build"):
            b.run(57)
        with pytest.raises(_abi.OxgbError, match="list build"):
            b.set_state(*state)
        _abi.check(L.oxgb_md_set_list_wait(b.handle, 0))
        if "sort_every" in kw:
            with pytest.raises(_abi.OxgbError):
                b.run(1)  # it may have stopped between the two halves of a move
        b.set_state(*state)
        b.run(57)
        got = b.get_state()
        # (the draws follow the step count, which went on: a state is compared from the same step only)
        assert all(np.all(np.isfinite(got[k])) for k in got)
    b.close()
    # the same after a failure before the first step
    c, _ = _engine(systems, **kw)
    _abi.check(L.oxgb_md_set_list_wait(c.handle, -1))
    with pytest.raises(_abi.OxgbError, match="list build"):
        c.set_state(*state)
    _abi.check(L.oxgb_md_set_list_wait(c.handle, 0))
    c.set_state(*state)
    c.run(57)
    got = c.get_state()
    for k in ("pos", "quat", "vel", "Lmom"):
        assert np.array_equal(want[k], got[k]), k
    c.close()
