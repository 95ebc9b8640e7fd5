"""Engines and lists beside other work on the GPU.

A kernel that holds an SM for long (one block, on a stream of its own) must not hold up a list build, nor
the steps of an engine: they have to finish while it is still running, and their results must be those of
the GPU to themselves, bit for bit, whichever blocks a build was shared by.  The same for two engines whose
steps run at the same time.  Sizes with cells by one block (up to 4,096 nucleotides) and by the grid, and builds of one, of some
and of as many blocks as there are SMs.
"""
import ctypes as C
import threading

import numpy as np
import pytest

from oxdna_gb300 import MDSystem, _abi, dna2_settings, md_settings
from oxdna_gb300 import generate as G

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

CYCLES = 1_000_000_000  # half a second and more
KEYS = ("pos", "quat", "vel", "Lmom")


class _Busy:
    """some streams with a one-block kernel each, running until the block is left"""

    def __init__(self, n=6):
        self.streams = [torch.cuda.Stream() for _ in range(n)]

    def __enter__(self):
        torch.cuda.synchronize()
        for s in self.streams:
            with torch.cuda.stream(s):
                torch.cuda._sleep(CYCLES)
        return self

    def running(self):
        return not any(s.query() for s in self.streams)

    def __exit__(self, *exc):
        torch.cuda.synchronize()


def _engine(n, seed=81, **kw):
    s = G.system_for_config(1, seed=seed, scale=n / 40000.0)
    m = MDSystem(s.box, s.top, dna2_settings(s.T, 0.5),
                 md_settings(dt=0.003, thermostat="john", newtonian_steps=7, pt=0.2, seed=5, verlet_skin=0.03, **kw))
    m.set_state(s.pos, s.quats(), s.vel, s.L)
    return m


@pytest.mark.parametrize("n,kw", [(40, {}), (1000, {}), (16000, {}), (40000, {}), (40000, dict(sort_every=1)),
                                  (4000, dict(precision="double"))])
def test_steps_go_on_beside_a_long_kernel(n, kw):
    a = _engine(n, **kw)
    a.run(16)
    a.run(64)
    want, builds = a.get_state(), a.info()["rebuilds"]
    a.close()
    b = _engine(n, **kw)
    b.run(16)
    with _Busy() as busy:
        b.run(64)
        assert busy.running()
    got = b.get_state()
    assert b.info()["rebuilds"] == builds >= 3
    for k in KEYS:
        assert np.array_equal(want[k], got[k]), k
    b.close()


@pytest.mark.parametrize("n", [1000, 16000, 40000])
def test_a_plain_list_is_built_beside_a_long_kernel(n):
    s = G.system_for_config(1, seed=82, scale=n / 40000.0)
    p = np.zeros((s.N, 4), np.float32)
    p[:, :3] = s.pos
    p[:, 3] = ((s.top.btype.astype(np.int32) << 22) | np.arange(s.N, dtype=np.int32)).view(np.float32)
    pos, bonds = torch.from_numpy(p).cuda(), torch.from_numpy(np.stack([s.top.n3, s.top.n5], 1).astype(np.int32)).cuda()
    at = torch.zeros_like(pos)
    L = _abi.lib()
    v = C.c_void_p()
    _abi.check(L.oxgb_verlet_create(s.N, s.box, 3.2638, 0.05, 1, 0, C.byref(v)))
    nb, nnb, most = C.c_void_p(), C.c_void_p(), C.c_int()
    _abi.check(L.oxgb_verlet_buffers(v, C.byref(nb), C.byref(nnb), C.byref(most), None))

    class View:
        def __init__(self, ptr, shape):
            self.__cuda_array_interface__ = {"shape": shape, "typestr": "<i4", "data": (int(ptr), False), "version": 3,
                                             "strides": None}

    rows = torch.as_tensor(View(nb.value, (most.value, s.N)), device="cuda")
    counts = torch.as_tensor(View(nnb.value, (s.N,)), device="cuda")
    st = torch.cuda.Stream()

    def build():
        _abi.check(L.oxgb_verlet_update(v, pos.data_ptr(), at.data_ptr(), bonds.data_ptr(), st.cuda_stream))
        st.synchronize()

    torch.cuda.synchronize()
    build()
    want = rows.cpu().numpy().copy(), counts.cpu().numpy().copy()
    with _Busy() as busy:
        for _ in range(3):
            build()
        assert busy.running()
    assert L.oxgb_verlet_status(v) == 0
    assert np.array_equal(want[1], counts.cpu().numpy())
    valid = np.arange(most.value)[:, None] < want[1]
    assert np.array_equal(want[0][valid], rows.cpu().numpy()[valid])
    _abi.check(L.oxgb_verlet_destroy(v))


@pytest.mark.parametrize("n", [1000, 16000, 40000])
def test_two_engines_at_once(n):
    want = []
    for seed in (81, 83):
        m = _engine(n, seed)
        m.run(16)
        m.run(400)
        want.append(m.get_state())
        m.close()
    m = [_engine(n, seed) for seed in (81, 83)]
    for e in m:
        e.run(16)
    failed = []

    def go(e):
        try:
            e.run(400)
        except Exception as x:  # (reported by the main thread)
            failed.append(x)

    threads = [threading.Thread(target=go, args=(e,)) for e in m]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    for e, w in zip(m, want):
        got = e.get_state()
        for k in KEYS:
            assert np.array_equal(w[k], got[k]), k
        e.close()
