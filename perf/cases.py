"""The work that users of this framework have it do, as cases whose time can be measured.

Five kinds of case, each through the entry points that a user's program calls:

* ``md``: a program steps one system (``MDSystem.run``) and takes a frame of the trajectory;
* ``batch``: a parallel-tempering program steps many independent systems in one engine and reads
  their energies, which decide the swaps;
* ``score``: a program uploads a configuration and asks for its forces, torques and energies;
* ``forces``, ``list``, ``order``: a host program on the reference's own device layout calls the
  interaction, the Verlet list and the order parameters of the C ABI on device buffers.

Systems are solutions of duplexes or of single strands on a lattice of random orientations, thermally
perturbed, or a melt of long random-walk strands; all are made from the seed alone.

The mixed engine computes its forces in FP32, so the state that a run ends in is determined to FP32:
a frame is taken as FP32 values, the precision trajectories are analysed in (FP64 for the double
engine).  The FP32 engine's forces, torques and energies come back as the FP32 values they are.
"""

import ctypes as C
import itertools
import math

import numpy as np
import torch

from oxdna_gb300 import MDSystem, _abi, dna2_settings, md_settings
from oxdna_gb300 import generate, io as oxio

KELVIN = 0.1 / 300.0  # simulation units of temperature in a kelvin


def listed():
    return [
        # one 12-bp duplex in vacuum: the smallest call, nothing but launches and latency
        dict(name="duplex 24 nt NVE", kind="md", mol="duplex", length=12, count=1, density=0.003, precision="mixed",
             thermostat="no", every=1, dt=0.005, salt=0.5, steps=200, sort=0, tuned=False),
        # a small assembly at the default settings: what most single runs look like
        dict(name="duplexes 1k Brownian", kind="md", mol="duplex", length=13, count=41, density=0.01, precision="mixed",
             thermostat="john", every=103, dt=0.003, salt=0.5, steps=200, sort=0, tuned=False),
        # the 40,000-nt duplex solution, Bussi thermostat every step
        dict(name="duplexes 40k Bussi", kind="md", mol="duplex", length=20, count=1000, density=0.01, precision="mixed",
             thermostat="bussi", every=1, dt=0.003, salt=0.5, steps=100, sort=0, tuned=False),
        # the largest ordinary run: a quarter of a million nucleotides of free strands, shapes autotuned
        dict(name="strands 250k Brownian", kind="md", mol="strand", length=23, count=10870, density=0.02,
             precision="mixed", thermostat="john", every=103, dt=0.003, salt=0.5, steps=100, sort=0, tuned=True),
        # relaxation of a generated melt of 1000-nt strands: backbone force capped, momenta refreshed often
        dict(name="melt 32k relaxation", kind="md", mol="walk", length=1000, count=32, density=0.02, precision="mixed",
             thermostat="john", every=1, dt=0.003, salt=0.5, steps=50, sort=0, tuned=False),
        # double precision, as parity runs use it
        dict(name="duplexes 4k double", kind="md", mol="duplex", length=17, count=119, density=0.01, precision="double",
             thermostat="no", every=1, dt=0.003, salt=0.5, steps=16, sort=0, tuned=False),
        # parallel tempering: 96 duplex and fragment systems of 16 to 4000 nt on a temperature ladder
        dict(name="batch of 96 systems", kind="batch", systems=96, low=16, high=4000, steps=100, tuned=True),
        # a configuration uploaded and evaluated once (analysis, FFS restarts)
        dict(name="score 10k", kind="score", mol="strand", length=19, count=527, density=0.02, precision="mixed",
             salt=0.3),
        # the interaction layer under a host program's own step loop, small and ordinary
        dict(name="forces 1k", kind="forces", mol="duplex", length=16, count=31, density=0.01, salt=0.5),
        dict(name="forces 40k", kind="forces", mol="duplex", length=20, count=1000, density=0.01, salt=0.5),
        # the list layer under the same loop
        dict(name="list 120k", kind="list", mol="strand", length=21, count=5715, density=0.02, salt=0.5, skin=0.05),
        # order parameters of forward flux sampling, between two force calls
        dict(name="order parameters 3k pairs", kind="order", mol="duplex", length=20, count=150, density=0.01, salt=0.5,
             pairs=3001),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case: sizes log-uniform from one duplex to a quarter of a million nucleotides."""
    kind = rng.choice(["md", "md", "md", "md", "batch", "score", "forces", "forces", "list", "order"])
    if kind == "batch":
        low = rng.randint(16, 64)
        return dict(kind=kind, systems=rng.randint(5, 120), low=low, high=rng.randint(low + 1, 3000),
                    steps=rng.randint(20, 100), tuned=rng.random() < 0.5)
    mol = rng.choice(["duplex", "strand"])
    length = rng.randint(8, 30)
    n = _log(rng, 24, 60000 if kind in ("score", "forces") else 240000)
    density = round(rng.uniform(0.005, 0.02), 4)
    salt = rng.choice([0.2, 0.3, 0.5, 0.5, 1.0])
    if kind == "md":
        precision = rng.choice(["mixed"] * 6 + ["float", "double"])
        if precision == "double":
            n = min(n, 6000)
        if rng.random() < 0.1:
            mol, length, n = "walk", rng.randint(200, 1000), min(n, 30000)
        count = max(1, round(n / (length * (2 if mol == "duplex" else 1))))
        size = count * length * (2 if mol == "duplex" else 1)
        thermostat = "john" if mol == "walk" else rng.choice(["no", "john", "bussi"])
        every = 1 if mol == "walk" else rng.choice([1, 103]) if thermostat == "bussi" else rng.choice([1, 53, 103])
        most = 16 if precision == "double" else max(20, min(200, int(2e7 / size)))
        return dict(kind=kind, mol=mol, length=length, count=count, density=0.02 if mol == "walk" else density,
                    precision=precision, thermostat=thermostat, every=every, dt=rng.choice([0.002, 0.003]), salt=salt,
                    steps=rng.randint(max(2, most // 3), most),
                    sort=rng.choice([0, 0, 0, 1]) if precision == "mixed" and size < 60000 else 0,
                    tuned=rng.random() < 0.3 and precision != "double")
    count = max(1, round(n / (length * (2 if mol == "duplex" else 1))))
    case = dict(kind=kind, mol=mol, length=length, count=count, density=density, salt=salt)
    if kind == "score":
        case["precision"] = rng.choice(["mixed", "mixed", "double"])
        if case["precision"] == "double":
            case["count"] = min(count, 150)
    if kind == "list":
        case["skin"] = rng.choice([0.05, 0.1, 0.2])
    if kind == "order":
        case["pairs"] = int(_log(rng, 10, 20000))
    return case


# ---------------------------------------------------------------- systems


def _helix(n, phase, z0, up):
    """centres, a1, a3 of one strand of the ideal B helix"""
    k = np.arange(n) if up else -np.arange(n)
    phi = phase + k * math.radians(34.8)
    u = np.stack([np.cos(phi), np.sin(phi), np.zeros(n)], 1)
    pos = 0.6 * u
    pos[:, 2] = z0 + 0.3897 * k
    return pos, -u, np.tile([0.0, 0.0, -1.0 if up else 1.0], (n, 1))


def _rotations(rng, n):
    """n uniformly distributed rotation matrices"""
    q = rng.normal(size=(n, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    x, y, z, w = q.T
    return np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                     2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                     2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], 1).reshape(n, 3, 3)


def _turns(rng, n, size):
    """n rotation matrices by small angles of standard deviation `size` about each axis"""
    v = rng.normal(size=(n, 3)) * size
    t = np.linalg.norm(v, axis=1)[:, None, None]
    k = np.zeros((n, 3, 3))
    k[:, 0, 1], k[:, 0, 2], k[:, 1, 2] = -v[:, 2], v[:, 1], -v[:, 0]
    k -= k.transpose(0, 2, 1)
    return np.eye(3) + np.sinc(t / np.pi) * k + (1 - np.cos(t)) / np.maximum(t * t, 1e-30) * (k @ k)


def _quaternions(m):
    """(x, y, z, w) of the rotation matrices whose columns are the body axes"""
    t = np.stack([1 + m[:, 0, 0] - m[:, 1, 1] - m[:, 2, 2], 1 - m[:, 0, 0] + m[:, 1, 1] - m[:, 2, 2],
                  1 - m[:, 0, 0] - m[:, 1, 1] + m[:, 2, 2], 1 + m[:, 0, 0] + m[:, 1, 1] + m[:, 2, 2]], 1)
    xy, xz, yz = m[:, 0, 1] + m[:, 1, 0], m[:, 0, 2] + m[:, 2, 0], m[:, 1, 2] + m[:, 2, 1]
    wx, wy, wz = m[:, 2, 1] - m[:, 1, 2], m[:, 0, 2] - m[:, 2, 0], m[:, 1, 0] - m[:, 0, 1]
    rows = np.stack([np.stack([t[:, 0], xy, xz, wx], 1), np.stack([xy, t[:, 1], yz, wy], 1),
                     np.stack([xz, yz, t[:, 2], wz], 1), np.stack([wx, wy, wz, t[:, 3]], 1)], 1)
    q = rows[np.arange(len(m)), np.argmax(t, 1)]
    return q / np.linalg.norm(q, axis=1, keepdims=True)


class _System:
    """a generated system: box, FP64 state, topology arrays, temperature"""

    def __init__(self, box, pos, axes, n3, n5, base, strand, T, rng):
        n = len(pos)
        self.box, self.T, self.N = float(box), T, n
        self.pos, self.quat = pos, _quaternions(axes)
        self.vel, self.L = rng.normal(size=(n, 3)) * math.sqrt(T), rng.normal(size=(n, 3)) * math.sqrt(T)
        self.n3, self.n5, self.base, self.strand = (np.asarray(a, np.int32) for a in (n3, n5, base, strand))

    def topology(self):
        return oxio.Topology(self.n3, self.n5, self.base, self.base.copy(), self.strand, int(self.strand[-1]) + 1)

    def state(self):
        return self.pos, self.quat, self.vel, self.L


def _solution(rng, mol, lengths, density, T):
    """Molecules of the given lengths, one to a lattice cell wide enough for any orientation, in random
    orientations, every nucleotide displaced and turned a little (as by thermal motion)."""
    longest, count = int(max(lengths)), len(lengths)
    sizes = np.asarray(lengths) * (2 if mol == "duplex" else 1)
    side = math.ceil(round(count ** (1 / 3), 9))
    # a molecule and its sites fit into a sphere of this diameter; the box also has to be wider than
    # twice the interaction's range at the lowest salt
    room = math.hypot(0.3897 * longest, 2.0) + 1.2
    cell = max(float(np.mean(sizes) / density) ** (1 / 3), room, 11.0 / side)
    spots = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    spots = spots[np.sort(rng.permutation(len(spots))[:count])]
    turn = _rotations(rng, count)
    pos, axes, n3, n5, base, strand = [], [], [], [], [], []
    first, strands, done = 0, 0, 0
    for n, same in itertools.groupby(int(v) for v in lengths):
        c = len(list(same))  # c molecules of this length at once
        p, a1, a3 = _helix(n, 0.0, 0.0, True)
        b = rng.integers(0, 4, (c, n))
        ends = [n]
        if mol == "duplex":
            q, c1, c3 = _helix(n, (n - 1) * math.radians(34.8) + math.pi, (n - 1) * 0.3897, False)
            p, a1, a3, b = np.vstack([p, q]), np.vstack([a1, c1]), np.vstack([a3, c3]), np.hstack([b, 3 - b[:, ::-1]])
            ends = [n, 2 * n]
        size = len(p)
        i = np.arange(c * size).reshape(c, size) + first
        up, down = i + 1, i - 1
        up[:, np.array(ends) - 1] = -1
        down[:, [0] + ends[:-1]] = -1
        R = turn[done:done + c]
        pos.append(((p - p.mean(0)) @ R.transpose(0, 2, 1) + (spots[done:done + c, None] + 0.5) * cell).reshape(-1, 3))
        axes.append((R[:, None] @ np.stack([a1, np.cross(a3, a1), a3], 2)).reshape(-1, 3, 3))
        n3.append(up.ravel()), n5.append(down.ravel()), base.append(b.ravel())
        which = np.searchsorted(ends, np.arange(size), side="right")
        strand.append((strands + len(ends) * np.arange(c)[:, None] + which).ravel())
        strands, first, done = strands + c * len(ends), first + c * size, done + c
    pos, axes = np.concatenate(pos), np.concatenate(axes)
    pos += rng.normal(size=pos.shape) * 0.01
    axes = _turns(rng, len(pos), 0.03) @ axes
    return _System(side * cell, pos, axes, *(np.concatenate(a) for a in (n3, n5, base, strand)), T, rng)


def _melt(rng, count, length, density, T):
    """Self-avoiding random-walk strands: one cell of four strands, repeated over the box with bases and
    momenta of its own in every copy."""
    group = min(4, count)
    cell = (group * length / density) ** (1 / 3)
    mols = generate.random_walk_melt(group, length, cell, rng)
    p = np.concatenate([m.pos for m in mols])
    a1, a2, a3 = oxio.orthonormal_frame(np.concatenate([m.a1 for m in mols]), np.concatenate([m.a3 for m in mols]))
    side = max(1, round((count / group) ** (1 / 3)))
    shifts = np.stack(np.meshgrid(*[np.arange(side) * cell] * 3, indexing="ij"), -1).reshape(-1, 3)
    copies = len(shifts)
    pos = (p[None] + shifts[:, None]).reshape(-1, 3)
    axes = np.tile(np.stack([a1, a2, a3], 2), (copies, 1, 1))
    n = len(pos)
    i = np.arange(n)
    n3, n5 = np.where(i % length == length - 1, -1, i + 1), np.where(i % length == 0, -1, i - 1)
    return _System(side * cell, pos, axes, n3, n5, rng.integers(0, 4, n), i // length, T, rng)


def _system(case, seed):
    rng = np.random.default_rng(int(seed))
    if case["mol"] == "walk":
        return _melt(rng, case["count"], case["length"], case["density"], 300 * KELVIN)
    return _solution(rng, case["mol"], [case["length"]] * case["count"], case["density"], 300 * KELVIN)


def _batch(case, seed):
    """Independent systems of log-uniform sizes, duplexes of at most 50 bp as fragments, 280 to 360 K."""
    rng = np.random.default_rng(int(seed))
    sizes = np.geomspace(case["low"], case["high"], case["systems"])
    sizes = np.random.default_rng(case["systems"]).permutation(sizes)  # in no order along the ladder
    out = []
    for k, target in enumerate(sizes):
        bp = max(8, int(target) // 2)
        parts = [50] * (bp // 50) + ([bp % 50] if bp % 50 >= 8 else [])
        T = 280 * KELVIN * (360 / 280) ** (k / max(1, case["systems"] - 1))
        out.append(_solution(rng, "duplex", parts, 0.005, T))
    return out


# ---------------------------------------------------------------- what a program has in hand


class _Device:
    """device memory of an engine or a handle, as a torch tensor, which keeps its owner"""

    def __init__(self, owner, ptr, shape, kind):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": kind, "data": (int(ptr), False), "version": 3,
                                         "strides": None}


def _view(owner, ptr, shape, kind):
    return torch.as_tensor(_Device(owner, ptr, shape, kind), device="cuda")


class _Handles:
    """handles of the C ABI, given back with the state"""

    def __init__(self):
        self.dna, self.verlet = C.c_void_p(), C.c_void_p()

    def __del__(self):
        try:
            if self.verlet:
                _abi.lib().oxgb_verlet_destroy(self.verlet)
            if self.dna:
                _abi.lib().oxgb_dna2_destroy(self.dna)
        except Exception:
            pass


def _engine(case, systems, seed, **kw):
    capped = dict(mbf_fmax=5.0) if case.get("mol") == "walk" else {}
    one = len(systems) == 1
    pick = (lambda v: v[0]) if one else list
    e = MDSystem(pick([s.box for s in systems]), pick([s.topology() for s in systems]),
                 pick([dna2_settings(s.T, case.get("salt", 0.5), **capped) for s in systems]),
                 md_settings(seed=int(seed) % 100003, autotune=case.get("tuned", False), **kw))
    return e, [np.concatenate(a) for a in zip(*[s.state() for s in systems])]


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("md", "batch"):
        if kind == "md":
            kw = dict(dt=case["dt"], thermostat=case["thermostat"], newtonian_steps=case["every"],
                      precision=case["precision"], sort_every=case["sort"])
            if case["mol"] == "walk":
                kw["pt"] = 0.1
            systems = [_system(case, seed)]
        else:
            kw = dict(dt=0.003, thermostat="bussi", newtonian_steps=1, bussi_tau=1000.0, steps_per_graph=25)
            systems = _batch(case, seed)
        e, state = _engine(case, systems, seed, **kw)
        e.set_state(*state)
        out = dict(case=case, engine=e)
        if case.get("precision") != "double" and not case.get("sort"):
            # the engine's own buffers, for a frame without a copy to the host
            p = [C.c_void_p() for _ in range(6)]
            _abi.check(_abi.lib().oxgb_md_device_buffers(e.handle, *[C.byref(x) for x in p]))
            out["state"] = [_view(e, x.value, (e.N, 4), "<f8") for x in p[:4]]
            out["forces"] = [_view(e, x.value, (e.N, 4), "<f4") for x in p[4:]]
            out["frame"] = [torch.zeros((e.N, 4), device="cuda") for _ in range(6)]
            torch.cuda.synchronize()
            out["stream"] = torch.cuda.ExternalStream(e.stream)
        return out
    s = _system(case, seed)
    if kind == "score":
        e, state = _engine(case, [s], seed, precision=case["precision"])
        e.set_state(*state)
        return dict(case=case, engine=e, input=state)
    # the reference's device layout: float4 positions with btype << 22 | index in w, float4 quaternions
    L = _abi.lib()
    h = _Handles()
    pos = torch.zeros((s.N, 4), device="cuda")
    pos[:, :3] = torch.from_numpy(s.pos.astype(np.float32)).cuda()
    pos[:, 3] = torch.from_numpy(((s.base << 22) | np.arange(s.N, dtype=np.int32)).view(np.float32)).cuda()
    quat = torch.from_numpy(s.quat.astype(np.float32)).cuda()
    out = dict(case=case, N=s.N, box=s.box, pos=pos, quat=quat, handles=h)
    _abi.check(L.oxgb_dna2_create(C.byref(dna2_settings(s.T, case["salt"])), C.byref(h.dna)))
    if kind == "order":
        # the base pairs that a simulation watches: paired nucleotides, and others by the way
        rng = np.random.default_rng(int(seed) + 1)
        m = case["length"] * (2 if case["mol"] == "duplex" else 1)
        first = rng.integers(0, s.N, case["pairs"])
        second = first - first % m + (m - 1 - first % m)
        second = np.where((rng.random(case["pairs"]) < 0.3) | (second == first), (first + 1) % s.N, second)
        out["one"], out["two"] = (torch.from_numpy(a.astype(np.int32)).cuda() for a in (first, second))
        out["hb"], out["dist"] = (torch.zeros(case["pairs"], device="cuda") for _ in range(2))
        out["near"] = torch.zeros(case["pairs"], dtype=torch.bool, device="cuda")
        return out
    out["bonds"] = torch.from_numpy(np.stack([s.n3, s.n5], 1)).contiguous().cuda()
    out["list_pos"] = torch.zeros_like(pos)
    rcut = C.c_double()
    _abi.check(L.oxgb_dna2_get_rcut(h.dna, C.byref(rcut)))
    _abi.check(L.oxgb_verlet_create(s.N, s.box, rcut.value, case.get("skin", 0.05), 1, 0, C.byref(h.verlet)))
    rows, counts, most, side = C.c_void_p(), C.c_void_p(), C.c_int(), C.c_int()
    _abi.check(L.oxgb_verlet_buffers(h.verlet, C.byref(rows), C.byref(counts), C.byref(most), C.byref(side)))
    out["rows"] = _view(h, rows.value, (most.value, s.N), "<i4")
    out["counts"] = _view(h, counts.value, (s.N,), "<i4")
    out["rows"].zero_()
    if kind == "forces":
        _abi.check(L.oxgb_verlet_update(h.verlet, pos.data_ptr(), out["list_pos"].data_ptr(), out["bonds"].data_ptr(),
                                        torch.cuda.current_stream().cuda_stream))
        out["F"], out["T"] = torch.zeros((s.N, 4), device="cuda"), torch.zeros((s.N, 4), device="cuda")
        torch.cuda.synchronize()
        _abi.check(L.oxgb_verlet_status(h.verlet))
    torch.cuda.synchronize()
    return out


# ---------------------------------------------------------------- one pass


def run(state):
    case, L = state["case"], _abi.lib()
    kind = case["kind"]
    if kind in ("md", "batch"):
        e = state["engine"]
        e.run(case["steps"])
        out = {}
        if kind == "batch":
            out["U"], out["Kt"], out["Kr"] = (x.astype(np.float32) for x in e.energies())
        if "state" not in state:
            st = e.get_state()
            return st if case["precision"] == "double" else {k: v.astype(np.float32) for k, v in st.items()}
        with torch.cuda.stream(state["stream"]):  # in order with the engine's own work
            for to, x in zip(state["frame"], state["state"] + state["forces"]):
                to.copy_(x)
        pos, vel, mom, quat, F, T = state["frame"]
        return dict(out, pos=pos[:, :3], vel=vel[:, :3], Lmom=mom[:, :3], quat=quat, F=F[:, :3], T=T[:, :3])
    if kind == "score":
        e = state["engine"]
        e.set_state(*state["input"])
        F, T, E, split = e.compute_forces()
        if case["precision"] == "double":
            return dict(F=F, T=T, E=E, split=split)
        return dict(F=F.astype(np.float32), T=T.astype(np.float32), E=E.astype(np.float32), split=split.astype(np.float32))
    stream = torch.cuda.current_stream().cuda_stream
    h = state["handles"]
    at = [state[k].data_ptr() for k in ("pos", "quat")]
    if kind == "order":
        who = [state["one"].data_ptr(), state["two"].data_ptr(), case["pairs"]]
        _abi.check(L.oxgb_dna2_hb_op_precalc(h.dna, state["box"], *at, *who, state["hb"].data_ptr(), stream))
        _abi.check(L.oxgb_dna2_near_hb_op_precalc(h.dna, state["box"], *at, *who, state["near"].data_ptr(), stream))
        _abi.check(L.oxgb_dna2_dist_op_precalc(h.dna, state["box"], *at, *who, state["dist"].data_ptr(), stream))
        return dict(hb=state["hb"], near=state["near"], dist=state["dist"])
    if kind == "list":
        _abi.check(L.oxgb_verlet_update(h.verlet, at[0], state["list_pos"].data_ptr(), state["bonds"].data_ptr(), stream))
        return dict(rows=state["rows"], counts=state["counts"], positions=state["list_pos"][:, :3])
    state["F"].zero_()
    state["T"].zero_()
    _abi.check(L.oxgb_dna2_compute_forces(h.dna, state["N"], state["box"], *at, state["F"].data_ptr(), state["T"].data_ptr(),
                                          state["bonds"].data_ptr(), state["rows"].data_ptr(), state["counts"].data_ptr(),
                                          state["rows"].shape[0], 1, state["N"], stream))
    return dict(F=state["F"], T=state["T"])


def work(case):
    """What a pass cannot do without.  A step reads and writes the FP64 state (13 numbers) and takes about
    1000 FP32 operations per nucleotide of a single strand and 2500 of a duplex (pairs in range counted once);
    a pass of the device-layout calls reads and writes their buffers."""
    kind = case["kind"]
    if kind == "batch":
        n = 0.5 * case["systems"] * (case["high"] - case["low"]) / math.log(case["high"] / case["low"]) * 2
        return dict(bytes=208.0 * n * case["steps"], flops=2500.0 * n * case["steps"])
    pair = case["mol"] == "duplex"
    n = case["count"] * case["length"] * (2 if pair else 1)
    each = 2500.0 if pair else 1000.0
    # neighbours of a nucleotide within the list's radius, as the density and the strand itself give them
    near = (25.0 if pair else 9.0) + case["density"] * 150.0
    if kind == "md":
        return dict(bytes=208.0 * n * case["steps"], flops=each * n * case["steps"])
    if kind == "score":
        return dict(bytes=(104.0 + 28.0) * n, flops=each * n)
    if kind == "forces":
        return dict(bytes=(72.0 + 64.0 + 4.0 * near) * n, flops=each * n)
    if kind == "list":
        return dict(bytes=(16.0 + 8.0 + 16.0 + 4.0 + 4.0 * near) * n, flops=20.0 * near * n)
    return dict(bytes=(64.0 + 8.0 + 9.0) * case["pairs"], flops=300.0 * case["pairs"])


# ---------------------------------------------------------------- the model in 64 bits, by automatic differentiation

_F = lambda *v: [float(np.float32(x)) for x in v]  # noqa: E731  (the model's constants are FP32 literals)
_PI = float(np.float32(math.pi))


def _angle(a, b):
    """the angle between vectors, well conditioned at every angle"""
    x = torch.linalg.cross(a, b)
    return torch.atan2((x * x).sum(-1).sqrt(), (a * b).sum(-1))


def _f1(r, eps, a, rc, r0, blow, bhigh, rlow, rhigh, rclow, rchigh):
    shift = (1 - math.exp(float(np.float32(-(np.float32(rc) - np.float32(r0)) * np.float32(a))))) ** 2
    zero = torch.zeros_like(r)
    mid = eps * (1 - torch.exp(-(r - r0) * a)) ** 2 - eps * shift
    f = torch.where((r > rlow) & (r <= rhigh), mid, zero)
    f = torch.where((r > rhigh) & (r < rchigh), eps * bhigh * (r - rchigh) ** 2, f)
    return torch.where((r > rclow) & (r <= rlow), eps * blow * (r - rclow) ** 2, f)


def _f2(r, k, rc, r0, blow, rlow, rclow, bhigh, rhigh, rchigh):
    zero = torch.zeros_like(r)
    f = torch.where((r > rlow) & (r <= rhigh), k / 2 * ((r - r0) ** 2 - (rc - r0) ** 2), zero)
    f = torch.where((r > rhigh) & (r < rchigh), k * bhigh * (r - rchigh) ** 2, f)
    return torch.where((r > rclow) & (r <= rlow), k * blow * (r - rclow) ** 2, f)


def _f4(t, a, b, t0, ts, tc):
    d = (t - t0).abs()
    return torch.where(d < tc, torch.where(d > ts, b * (tc - d) ** 2, 1 - a * d * d), torch.zeros_like(t))


def _f5(x):
    a, b, xc, xs = _F(2.0, 10.9032, -0.769231, -0.65)
    f = torch.where(x < 0, 1 - a * x * x, torch.ones_like(x))
    return torch.where(x <= xc, torch.zeros_like(x), torch.where(x < xs, b * (xc - x) ** 2, f))


_ST4, _ST5 = _F(1.3, 6.4381, 0, 0.8, 0.961538), _F(0.9, 3.89361, 0, 0.95, 1.16959)
_HB1, _HB4 = _F(1.5, 4.16038, 0, 0.7, 0.952381), _F(0.46, 0.133855, _PI, 0.7, 3.10559)
_HB7 = _F(4.0, 17.0526, _PI * 0.5, 0.45, 0.555556)
_CR1 = _F(2.25, 7.00545, np.float32(_PI) - np.float32(2.35), 0.58, 0.766284)
_CR2, _CR4 = _F(1.7, 6.2469, 1.0, 0.68, 0.865052), _F(1.5, 2.59556, 0, 0.65, 1.02564)
_CR7 = _F(1.7, 6.2469, 0.875, 0.68, 0.865052)
_CX1 = _F(2.0, 10.9032, np.float32(_PI) - np.float32(0.25), 0.65, 0.769231)
_HYDR = _F(8, 0.75, 0.4, -126.243, -7.87708, 0.34, 0.7, 0.276908, 0.783775)
_STCK = _F(6, 0.9, 0.4, -68.1857, -3.12992, 0.32, 0.75, 0.23239, 0.956)
_CRST = _F(47.5, 0.675, 0.575, -0.888889, 0.495, 0.45, -0.888889, 0.655, 0.7)
_CXST = _F(58.5, 0.6, 0.4, -2.13158, 0.22, 0.177778, -2.13158, 0.58, 0.6222222)
_EXCL = [_F(0.70, 0.675, 892.016223343, 0.711879214356), _F(0.33, 0.32, 4119.70450017, 0.335388426126),
         _F(0.515, 0.50, 1707.30627298, 0.52329943261)]


def _excluded(d, which):
    sigma, rstar, b, rc = _EXCL[which]
    r2 = (d * d).sum(-1)
    keep = r2 < rc * rc
    r = torch.where(keep, r2, torch.ones_like(r2)).sqrt()
    lj = (sigma * sigma / (r * r)) ** 3
    e = torch.where(r > rstar, 2.0 * b * (r - rc) ** 2, 8.0 * (lj * lj - lj))
    return torch.where(keep, e, torch.zeros_like(e))


def _debye(T, salt):
    q = 0.0543
    high = 3.0 * 0.3616455 * math.sqrt(T / float(np.float32(0.1))) / math.sqrt(float(np.float32(salt)))
    lam = 0.3616455 * math.sqrt(T / 0.1) / math.sqrt(float(np.float32(salt)))
    b = -(math.exp(-high / lam) * q * q * (high + lam) ** 2) / (-4 * high ** 3 * lam * lam * q)
    return q, lam, high, b, high * (q * high + 3 * q * lam) / (q * (high + lam))


class _Model:
    """oxDNA2 (average sequence) of one system: energies of every pair, forces and torques."""

    def __init__(self, box, n3, n5, base, T, salt):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        to = lambda a: torch.from_numpy(np.asarray(a, np.int64)).to(self.dev)  # noqa: E731
        self.box, self.T, self.debye = box, T, _debye(T, salt)
        self.n3, self.n5, self.base = to(n3), to(n5), to(base)
        self.end = (self.n3 < 0) | (self.n5 < 0)
        self.p = torch.nonzero(self.n3 >= 0)[:, 0]
        self.q = self.n3[self.p]

    def frame(self, q):
        x, y, z, w = q.unbind(-1)
        xx, yy, zz, ww, xy, xz, xw, yz, yw, zw = x * x, y * y, z * z, w * w, x * y, x * z, x * w, y * z, y * w, z * w
        return (torch.stack([xx - yy - zz + ww, 2 * (xy + zw), 2 * (xz - yw)], -1),
                torch.stack([2 * (xy - zw), -xx + yy - zz + ww, 2 * (yz + xw)], -1),
                torch.stack([2 * (xz + yw), 2 * (yz - xw), -xx - yy + zz + ww], -1))

    def near(self, x, reach):
        """the unordered non-bonded pairs whose centres are within `reach`"""
        got = []
        for a in range(0, len(x), 1000):
            d = x[a:a + 1000, None] - x[None, a:]
            d -= torch.round(d / self.box) * self.box
            i, j = torch.nonzero((d * d).sum(-1) < reach * reach, as_tuple=True)
            i, j = i + a, j + a
            keep = (j > i) & (self.n3[i] != j) & (self.n5[i] != j)
            got.append(torch.stack([i[keep], j[keep]]))
        return torch.cat(got, 1)

    def energies(self, x, frame, pairs):
        """[(i, j, energy)] by term: FENE, bonded excluded volume, stacking, excluded volume, hydrogen bonding, cross
        stacking, coaxial stacking, Debye-Hueckel"""
        a1, a2, a3 = frame
        m1, m2, back0 = _F(-0.34, 0.3408, -0.4)
        s_stack, s_base = _F(0.34, 0.4)
        back, stack, base = a1 * m1 + a2 * m2, a1 * s_stack, a1 * s_base
        dot = lambda u, v: (u * v).sum(-1)  # noqa: E731
        p, q = self.p, self.q
        r = x[q] - x[p]
        d = (r + back[q] - back[p]).norm(dim=-1) - float(np.float32(0.7564))
        out = [(p, q, -torch.log(1 - d * d / 0.0625))]
        out.append((p, q, _excluded(r + base[q] - base[p], 1) + _excluded(r + back[q] - base[p], 2) +
                    _excluded(r + base[q] - back[p], 2)))
        ref = r + (a1[q] - a1[p]) * back0
        rs = r + stack[q] - stack[p]
        fact, eps0 = _F(2.6717, 1.3523)
        e = _f1(rs.norm(dim=-1), eps0 + fact * self.T, *_STCK)
        e = e * _f4(_angle(a3[p], a3[q]), *_ST4) * _f4(_angle(a3[p], -rs), *_ST5) * _f4(_angle(-a3[q], rs), *_ST5)
        out.append((p, q, e * _f5(dot(a2[p], ref) / ref.norm(dim=-1)) * _f5(dot(a2[q], ref) / ref.norm(dim=-1))))
        i, j = pairs
        r = x[j] - x[i]
        r = r - torch.round(r.detach() / self.box) * self.box
        out.append((i, j, _excluded(r + base[j] - base[i], 1) + _excluded(r + base[j] - back[i], 2) +
                    _excluded(r + back[j] - base[i], 2) + _excluded(r + back[j] - back[i], 0)))

        def inside(rv, lo, hi, also=None):
            n = rv.detach().norm(dim=-1)
            k = (n > lo) & (n < hi)
            return torch.nonzero(k if also is None else k & also)[:, 0]

        rb = r + base[j] - base[i]
        k = inside(rb, _HYDR[7], _HYDR[8], self.base[i] + self.base[j] == 3)
        u, v, w = i[k], j[k], rb[k]
        e = _f1(w.norm(dim=-1), _F(1.0678)[0], *_HYDR)
        e = e * _f4(_angle(a1[u], -a1[v]), *_HB1) * _f4(_angle(-a1[v], w), *_HB1) * _f4(_angle(a1[u], w), *_HB1)
        out.append((u, v, e * _f4(_angle(a3[u], a3[v]), *_HB4) * _f4(_angle(-a3[v], w), *_HB7) * _f4(_angle(a3[u], w), *_HB7)))
        k = inside(rb, _CRST[5], _CRST[8])
        u, v, w = i[k], j[k], rb[k]
        both = lambda t, c: _f4(t, *c) + _f4(math.pi - t, *c)  # noqa: E731
        e = _f2(w.norm(dim=-1), *_CRST)
        e = e * _f4(_angle(a1[u], -a1[v]), *_CR1) * _f4(_angle(-a1[v], w), *_CR2) * _f4(_angle(a1[u], w), *_CR2)
        out.append((u, v, e * both(_angle(a3[u], a3[v]), _CR4) * both(_angle(-a3[v], w), _CR7) * both(_angle(a3[u], w), _CR7)))
        rk = r + stack[j] - stack[i]
        k = inside(rk, _CXST[5], _CXST[8])
        u, v, w = i[k], j[k], rk[k]
        t1 = _angle(a1[u], -a1[v])
        sb = float(np.float32(_PI) - np.float32(0.1) * (np.float32(_PI) - (np.float32(_PI) - np.float32(0.25))))
        f1 = _f4(t1, *_CX1) + 20.0 * torch.clamp(t1 - sb, min=0.0) ** 2
        e = _f2(w.norm(dim=-1), *_CXST) * f1 * _f4(_angle(a3[u], a3[v]), *_ST4)
        out.append((u, v, e * both(_angle(a3[u], w), _ST5) * both(_angle(-a3[v], w), _ST5)))
        pre, lam, high, b, rc = self.debye
        rk = r + back[j] - back[i]
        k = inside(rk, 0.0, rc)
        u, v, n = i[k], j[k], rk[k].norm(dim=-1)
        e = torch.where(n < high, torch.exp(-n / lam) * pre / n, b * (n - rc) ** 2)
        out.append((u, v, e * (1 - 0.5 * self.end[u]) * (1 - 0.5 * self.end[v])))
        return out

    def forces(self, x, quat, pairs):
        """forces, body-frame torques, per-nucleotide energies (each pair's on both), hydrogen bonding's, terms"""
        x = x.detach().requires_grad_(True)
        frame = [a.detach().requires_grad_(True) for a in self.frame(quat)]
        terms = self.energies(x, frame, pairs)
        g = torch.autograd.grad(sum(e.sum() for _, _, e in terms), [x] + frame)
        lab = -sum(torch.linalg.cross(a.detach(), d) for a, d in zip(frame, g[1:]))
        body = torch.stack([(a.detach() * lab).sum(-1) for a in frame], -1)
        per = torch.zeros(len(x), dtype=torch.float64, device=x.device)
        hb = torch.zeros_like(per)
        for k, (i, j, e) in enumerate(terms):
            for t in (per, hb) if k == 4 else (per,):
                t.index_add_(0, i, e.detach())
                t.index_add_(0, j, e.detach())
        return -g[0], body, per, hb, torch.stack([e.detach().sum() for _, _, e in terms])

    def reach(self):
        return 2 * math.hypot(0.34, 0.3408) + self.debye[4] + 0.01


def _model(s, salt):
    return _Model(s.box, s.n3, s.n5, s.base, s.T, salt)


def exact(case, seed):
    """What run() returns, in 64 bits by automatic differentiation of the model's energy.  None for the
    thermostatted runs, whose values are those of the engine's own random stream, and for the list's whole
    numbers."""
    kind = case["kind"]
    if kind in ("batch", "list") or kind == "md" and (case["thermostat"] != "no" or case["mol"] == "walk"):
        return None
    s = _system(case, seed)
    m = _model(s, case["salt"])
    to = lambda a: torch.from_numpy(np.asarray(a, np.float64)).to(m.dev)  # noqa: E731
    if kind == "order":
        x, q = to(s.pos.astype(np.float32)), to(s.quat.astype(np.float32))
        rng = np.random.default_rng(int(seed) + 1)
        n = case["length"] * (2 if case["mol"] == "duplex" else 1)
        first = rng.integers(0, s.N, case["pairs"])
        second = first - first % n + (n - 1 - first % n)
        second = np.where((rng.random(case["pairs"]) < 0.3) | (second == first), (first + 1) % s.N, second)
        i, j = (torch.from_numpy(a).to(m.dev) for a in (first, second))
        frame = m.frame(q)
        r = x[j] - x[i]
        r = r - torch.round(r / s.box) * s.box + _F(0.4)[0] * (frame[0][j] - frame[0][i])
        hb = torch.zeros(len(i), dtype=torch.float64, device=m.dev)
        # the energies of the listed pairs, each a pair of its own
        terms = m.energies(x, frame, torch.stack([i, j]))
        u, v, e = terms[4]
        at = {}
        for a, b, c in zip(u.tolist(), v.tolist(), e.tolist()):
            at[a, b] = c
        hb = torch.tensor([at.get(k, 0.0) for k in zip(first.tolist(), second.tolist())], dtype=torch.float64)
        return dict(hb=hb, near=None, dist=r.norm(dim=-1))
    if kind == "forces":
        x, q = to(s.pos.astype(np.float32)), to(s.quat.astype(np.float32))
        F, T, E, hb, _ = m.forces(x, q, m.near(x, m.reach()))
        return dict(F=torch.cat([F, E[:, None]], 1), T=torch.cat([T, hb[:, None]], 1))
    x, q, v, L = (to(a) for a in s.state())
    q = q / q.norm(dim=-1, keepdim=True)
    if kind == "score":
        F, T, E, _, split = m.forces(x, q, m.near(x, m.reach()))
        return dict(F=F, T=T, E=E, split=split)
    if s.N > 20000 and case["precision"] != "double":
        return None  # over 20 seconds
    dt, half = case["dt"], 0.5 * case["dt"]
    pairs, at = m.near(x, m.reach() + 0.8), x
    F, T = m.forces(x, q, pairs)[:2]
    for _ in range(case["steps"]):
        v, L = v + half * F, L + half * T
        x = x + dt * v
        n = L.norm(dim=-1, keepdim=True)
        u = torch.cat([torch.sin(half * n) / n * L, torch.cos(half * n)], 1)
        qv, qw, uv, uw = q[:, :3], q[:, 3:], u[:, :3], u[:, 3:]
        q = torch.cat([qw * uv + uw * qv + torch.linalg.cross(qv, uv), qw * uw - (qv * uv).sum(-1, keepdim=True)], 1)
        q = q / q.norm(dim=-1, keepdim=True)
        if float((x - at).norm(dim=-1).max()) > 0.2:
            pairs, at = m.near(x, m.reach() + 0.8), x
        F, T = m.forces(x, q, pairs)[:2]
        v, L = v + half * F, L + half * T
    out = dict(pos=x, quat=q, vel=v, Lmom=L)
    return out if case["precision"] == "double" or case["sort"] else dict(out, F=F, T=T)
