"""Performance cases of the LULESH step: what a program that uses this library
has it do, through the public entry points, from the smallest call to a mesh
well beyond the L2.

A case is one of six kinds of call:

  sedov   a set (single domain, tp^3 subdomains, mixed precision) restarted
          from a state the program holds and advanced by some cycles
  mesh    the same for an unstructured mesh read from an lmesh file
  force   lulesh_volume_force_noalloc on the caller's own arrays
  batch   uneven jobs created, run in one graph launch and read back
  serve   a burst of jobs through a running server

The restart state is a blast in mid-flight: the mesh displaced and moving
radially, energy and pressure falling off from the origin, with smooth
seeded perturbations, so that every element is at work (a run's first cycles
have all but a few elements at rest).  It is computed here, in torch, from the
seed alone.  `exact` advances the same state with a plain torch FP64 restatement
of the Lagrange step.
"""
import ctypes
import math
import os
import random
import sys
import tempfile

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "cuda-ipc-benchmarks_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

F64 = torch.float64
EDGE = 1.125  # edge of the Sedov cube
NODE = ("x", "y", "z", "xd", "yd", "zd")
ELEM = ("e", "p", "q", "v", "ss")
T0, DT0 = 1.0e-3, 1.0e-7  # time and dt a restart begins from (dt then grows by 1.2 a cycle)


def _sedov(name, nx, cycles, tp=1, mixed=False, staged=False, host=False, regions=11, balance=1,
           cost=1):
    return {"name": name, "kind": "sedov", "nx": nx, "cycles": cycles, "tp": tp, "mixed": mixed,
            "staged": staged, "host": host, "regions": regions, "balance": balance, "cost": cost}


def listed():
    return [
        # the smallest runs: a 1,000-element mesh, every kernel a handful of blocks
        _sedov("sedov-10", 10, 32),
        # the reference's verification size (-s 30, 11 regions)
        _sedov("sedov-30", 30, 32),
        # LULESH's own default mesh, each cycle driven from the host as the
        # reference drives it (time state in, time state and status out)
        _sedov("sedov-45-host", 45, 16, host=True),
        # the headline mesh, one domain of a million elements
        _sedov("sedov-100", 100, 12),
        # an odd edge past the L2, with many regions and a costly EOS
        _sedov("sedov-133-regions", 133, 6, regions=20, balance=2, cost=4),
        # the largest: four million elements, 2.3 GB of state
        _sedov("sedov-160", 160, 4),
        # the headline mesh as 2x2x2 subdomains of -s 50
        _sedov("subdomains-2x50", 50, 12, tp=2),
        # mixed precision at its own benchmark size
        _sedov("mixed-120", 120, 8, mixed=True),
        # an unstructured mesh: warped, nodes and elements renumbered
        {"name": "mesh-40", "kind": "mesh", "nx": 40, "cycles": 16},
        # nodal forces for a caller that owns all arrays, the largest it may pass
        {"name": "force-32", "kind": "force", "nx": 32},
        # a parameter study: uneven jobs in one batch, created, run and read back
        {"name": "batch-12", "kind": "batch", "jobs": 12, "its": 50, "pick": 0},
        # a burst of requests at a server that stays up
        {"name": "serve-24", "kind": "serve", "jobs": 24, "its": 160, "pick": 0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["single", "sub", "mixed", "mesh", "force", "batch", "serve"],
                       [8, 3, 2, 2, 2, 1, 1])[0]
    if kind == "force":
        return {"kind": "force", "nx": _log_int(rng, 3, 32)}
    if kind == "mesh":
        return {"kind": "mesh", "nx": _log_int(rng, 6, 40), "cycles": rng.randint(8, 16)}
    if kind == "batch":
        return {"kind": "batch", "jobs": rng.randint(4, 12), "its": rng.randint(20, 50),
                "pick": rng.randint(1, 10 ** 6)}
    if kind == "serve":
        return {"kind": "serve", "jobs": rng.randint(8, 24), "its": rng.randint(80, 160),
                "pick": rng.randint(1, 10 ** 6)}
    tp = rng.choice([2, 2, 3]) if kind == "sub" else 1
    nx = _log_int(rng, 5, {1: 160, 2: 60, 3: 40}[tp])
    if kind == "mixed":
        nx = _log_int(rng, 8, 130)
    zones = (nx * tp) ** 3
    cycles = max(4, min(32, int(1.5e7 / zones)))
    c = _sedov("", nx, cycles, tp=tp, mixed=kind == "mixed", staged=tp > 1 and rng.random() < 0.3,
               host=tp == 1 and zones < 10 ** 6 and rng.random() < 0.25,
               regions=rng.randint(5, 20), balance=rng.choice([1, 2, 4]),
               cost=rng.choice([1, 2, 4]))
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# meshes and the state of a blast in mid-flight


def _device():
    return torch.device("cuda", torch.cuda.current_device())


class _Mesh:
    """A hex mesh on the device: reference coordinates [3,N], nodes [8,E], face
    links [6,E] (itself where there is none), plus whether each face is a
    symmetry plane (minus side) or a free surface (plus side)."""

    def __init__(self, xyz, nodes, links, symm_face, free_face, symm_node):
        self.xyz, self.nodes, self.links = xyz, nodes, links
        self.symm_face, self.free_face, self.symm_node = symm_face, free_face, symm_node


def _box(nx):
    """The Sedov cube of edge nx, in the numbering of a structured run."""
    dev, en = _device(), nx + 1
    c = EDGE * torch.arange(en, dtype=F64, device=dev) / float(nx)
    xyz = torch.stack([c.repeat(en * en), c.repeat_interleave(en).repeat(en),
                       c.repeat_interleave(en * en)])
    a = torch.arange(nx, device=dev)
    ex, ey, ez = a.repeat(nx * nx), a.repeat_interleave(nx).repeat(nx), a.repeat_interleave(nx * nx)
    n0 = (ez * en + ey) * en + ex
    p = en * en
    nodes = torch.stack([n0, n0 + 1, n0 + en + 1, n0 + en,
                         n0 + p, n0 + p + 1, n0 + p + en + 1, n0 + p + en])
    i = torch.arange(nx ** 3, device=dev)
    links, symm, free = [], [], []
    for pos, stride in ((ex, 1), (ey, nx), (ez, nx * nx)):
        links += [torch.where(pos == 0, i, i - stride), torch.where(pos == nx - 1, i, i + stride)]
        symm.append(pos == 0)
        free.append(pos == nx - 1)
    return _Mesh(xyz, nodes, torch.stack(links), torch.stack(symm), torch.stack(free),
                 xyz == 0.0)


def _warped(nx, seed):
    """A curvilinear, renumbered box (host arrays: it is written to a file):
    coordinates [N,3], nodes [E,8], links [E,6], symmetry sets, free set."""
    m = _box(nx)
    xyz = m.xyz.cpu().numpy().T
    u = xyz / EDGE
    bump = np.sin(np.pi * u)
    warped = xyz.copy()
    for a in range(3):
        b, c = (a + 1) % 3, (a + 2) % 3
        warped[:, a] += 0.03 * EDGE * bump[:, a] * np.sin(2 * np.pi * u[:, b]) * np.cos(np.pi * u[:, c])
    rng = np.random.default_rng(seed)
    npm, epm = rng.permutation(xyz.shape[0]), rng.permutation(m.nodes.shape[1])
    out = np.empty_like(warped)
    out[npm] = warped
    nodes = np.empty((m.nodes.shape[1], 8), dtype=np.int64)
    nodes[epm] = npm[m.nodes.cpu().numpy().T]
    links = np.empty((m.nodes.shape[1], 6), dtype=np.int64)
    links[epm] = epm[m.links.cpu().numpy().T]
    sets = [np.sort(npm[np.nonzero(xyz[:, a] == 0.0)[0]]) for a in range(3)]
    free = np.sort(npm[np.nonzero((xyz == EDGE).any(axis=1))[0]])
    return out, nodes, links, sets, free, epm, m


def _mesh_on_device(w):
    xyz, nodes, links, sets, _, epm, box = w
    dev = _device()
    e = torch.from_numpy(epm).to(dev)
    symm_face, free_face = torch.empty_like(box.symm_face), torch.empty_like(box.free_face)
    symm_face[:, e] = box.symm_face
    free_face[:, e] = box.free_face
    symm_node = torch.zeros(3, xyz.shape[0], dtype=torch.bool, device=dev)
    for a in range(3):
        symm_node[a, torch.from_numpy(sets[a]).to(dev)] = True
    return _Mesh(torch.from_numpy(np.ascontiguousarray(xyz.T)).to(dev),
                 torch.from_numpy(np.ascontiguousarray(nodes.T)).to(dev),
                 torch.from_numpy(np.ascontiguousarray(links.T)).to(dev), symm_face, free_face,
                 symm_node)


def _cross(a, b):
    return torch.stack([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2],
                        a[0] * b[1] - a[1] * b[0]])


def _dot(a, b):
    return (a * b).sum(0)


def _volume(P):
    """Volume of the hexahedra with corners P [3,8,E]."""
    def d(i, j):
        return P[:, i] - P[:, j]

    return (_dot(d(3, 1) + d(7, 2), _cross(d(6, 3), d(2, 0))) +
            _dot(d(4, 3) + d(5, 7), _cross(d(6, 4), d(7, 0))) +
            _dot(d(1, 4) + d(2, 5), _cross(d(6, 1), d(5, 0)))) / 12.0


def _blast(mesh, seed):
    """The state the runs restart from, on `mesh`: {field: tensor}."""
    r = random.Random(1000003 * (seed + 1))
    front, e1, v0 = r.uniform(0.45, 0.65), r.uniform(4e3, 6e3), r.uniform(40.0, 60.0)
    push = r.uniform(0.04, 0.08)
    amp = [r.uniform(-1.0, 1.0) for _ in range(9)]
    X0 = mesh.xyz
    s = (X0 * X0).sum(0) / front ** 2
    u = math.pi / EDGE * X0
    wob = torch.stack([torch.sin(u[a]) * (amp[3 * a] * torch.cos(u[(a + 1) % 3]) +
                                          amp[3 * a + 1] * torch.cos(2 * u[(a + 2) % 3]) +
                                          amp[3 * a + 2]) for a in range(3)])
    X = X0 * (1.0 + push * torch.exp(-s)) + 0.002 * wob
    V = v0 / front * X0 * torch.exp(-0.5 * s * s) + 0.02 * v0 * wob
    volo = _volume(X0[:, mesh.nodes])
    v = _volume(X[:, mesh.nodes]) / volo
    c = X0[:, mesh.nodes].mean(1)
    sc = (c * c).sum(0) / front ** 2
    e = e1 * (torch.exp(-3.0 * sc) + 1e-3) * (1.0 + 0.05 * torch.sin(7.0 * c[0] + 5.0 * c[1]) *
                                              torch.cos(6.0 * c[2] + amp[0]))
    p = (2.0 / 3.0) / v * e
    q = 0.1 * p * torch.exp(-sc)
    ss = torch.sqrt((2.0 / 3.0) * e + v * v * (2.0 / 3.0) / v * p)
    return {"x": X[0], "y": X[1], "z": X[2], "xd": V[0], "yd": V[1], "zd": V[2],
            "e": e, "p": p, "q": q, "v": v, "ss": ss, "volo": volo}


def _split(f, nx, tp, nodal):
    """A field over the whole cube as [tp^3, n]: each subdomain's own elements
    or nodes, subdomain r at (r % tp, r / tp % tp, r / tp^2)."""
    if tp == 1:
        return f.reshape(1, -1)
    g = f.reshape((nx * tp + int(nodal),) * 3)
    w = nx + int(nodal)
    return torch.stack([g[pl * nx:pl * nx + w, ro * nx:ro * nx + w, co * nx:co * nx + w].reshape(-1)
                        for pl in range(tp) for ro in range(tp) for co in range(tp)])


# ---------------------------------------------------------------------------
# a set's device arrays as tensors


class _View(ctypes.Structure):  # lulesh_domain_view
    _fields_ = ([(n, ctypes.c_int) for n in (
        "numElem numNode padded_numElem sizeX sizeY sizeZ colLoc rowLoc planeLoc tp numReg allElem "
        "numSymmX numSymmY numSymmZ").split()] +
        [(n, ctypes.c_void_p) for n in (
            "nodelist lxim lxip letam letap lzetam lzetap elemBC nodeElemCount nodeElemStart "
            "nodeElemCornerList symmX symmY symmZ matElemlist regCSR regReps regNumList "
            "regElemlist regSorted e p q ql qq v volo delv vdov arealg ss elemMass x y z xd yd zd "
            "xdd ydd zdd fx fy fz nodalMass").split()])
    # the transients that follow in the C struct
    _fields_ += [(n, ctypes.c_void_p) for n in (
        "vnew delx_xi delx_eta delx_zeta delv_xi delv_eta delv_zeta fx_elem fy_elem fz_elem").split()]


class _Pointer:
    """Device memory of a set; a tensor made of it keeps the set."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False),
                                         "version": 3, "strides": None}


def _arrays(s):
    """{field: [tensor per domain]} over the set's own device memory."""
    out = {f: [] for f in NODE + ELEM}
    for d in range(s.num_domains):
        w = _View()
        assert s.lib.lulesh_domain_view_get(s.h, d, ctypes.byref(w)) == 0
        for f in out:
            n = w.numNode if f in NODE else w.numElem
            out[f].append(torch.as_tensor(_Pointer(s, getattr(w, f), n), device=_device()))
    return out


def _together(s, parts):
    """The domains' arrays of one field as one [ndom, n] tensor: a strided view
    where they lie at a constant distance in the set's arena, else None."""
    if len(parts) == 1:
        return parts[0].reshape(1, -1)
    step = parts[1].data_ptr() - parts[0].data_ptr()
    if any(b.data_ptr() - a.data_ptr() != step for a, b in zip(parts, parts[1:])) or step % 8:
        return None
    span = step // 8 * (len(parts) - 1) + parts[0].numel()
    flat = torch.as_tensor(_Pointer(s, parts[0].data_ptr(), span), device=_device())
    return flat.as_strided((len(parts), parts[0].numel()), (step // 8, 1))


def _in_single(outs):
    """A mixed-precision run's fields are good to FP32 and handed on as such.
    All but q: it switches on where an element starts to compress, and FP32
    puts elements at rest on either side of that switch."""
    return [o.float() for f, o in zip(NODE + ELEM, outs) if f != "q"]


_streams = {}


def _stream():
    """The program's compute stream: one for all of its sets."""
    d = torch.cuda.current_device()
    if d not in _streams:
        _streams[d] = torch.cuda.Stream()
    return _streams[d]


# ---------------------------------------------------------------------------
# the cases


def _jobs(case, seed):
    """The jobs of a batch or a burst: sizes and regions by the case, cycle
    budgets by the seed (their sum stays within one cycle a job)."""
    import lulesh_b200 as L

    rng = random.Random(7919 * case["pick"] + case["jobs"])
    lo, hi = (10, 48) if case["kind"] == "batch" else (8, 64)
    shapes = [(_log_int(rng, lo, hi), rng.randint(5, 20),
               rng.choice([1, 2, 4]) if case["kind"] == "batch" else 1,
               rng.choice([1, 2, 4]) if case["kind"] == "batch" else 1) for _ in range(case["jobs"])]
    r = random.Random(104729 * (seed + 1))
    return [L.JobSpec(s, reg, b, c, case["its"] + r.randint(-2, 2)) for s, reg, b, c in shapes]


def _zones(case):
    if case["kind"] in ("batch", "serve"):
        rng = random.Random(7919 * case["pick"] + case["jobs"])
        lo, hi = (10, 48) if case["kind"] == "batch" else (8, 64)
        total = 0
        for _ in range(case["jobs"]):
            total += _log_int(rng, lo, hi) ** 3 * case["its"]
            rng.randint(5, 20)
            if case["kind"] == "batch":
                rng.choice([1, 2, 4]), rng.choice([1, 2, 4])
        return total
    return (case["nx"] * case.get("tp", 1)) ** 3 * case.get("cycles", 1)


def prepare(case, seed):
    import lulesh_b200 as L

    dev = _device()
    if case["kind"] == "force":
        st = _blast(_box(case["nx"]), seed)
        # a caller's own masses: density 1
        ins = [st[f].contiguous() for f in NODE] + [st["volo"], st["v"], st["p"], st["q"], st["ss"],
                                                    st["volo"].clone()]
        n = (case["nx"] + 1) ** 3
        outs = [torch.empty(n, dtype=F64, device=dev) for _ in range(3)]
        bad = torch.zeros(1, dtype=torch.int32, device=dev)
        return {"kind": "force", "lib": L.load_library(), "nx": case["nx"], "ins": ins,
                "outs": outs, "bad": bad}
    if case["kind"] == "batch":
        return {"kind": "batch", "L": L, "jobs": _jobs(case, seed)}
    if case["kind"] == "serve":
        # the slots, workers and cycles per step of serving.run_served
        srv = L.Server(max_jobs=4096, cycles_per_step=64, prepare_threads=8)
        return {"kind": "serve", "srv": srv, "jobs": _jobs(case, seed)}

    nx, tp = case["nx"], case.get("tp", 1)
    if case["kind"] == "mesh":
        import lmesh

        w = _warped(nx, seed)
        mesh = _mesh_on_device(w)
        fd, path = tempfile.mkstemp(suffix=".lmesh")
        os.close(fd)
        try:
            lmesh.write(path, lmesh.LMesh(w[0], w[1], w[2], tuple(w[3]), w[4]))
            s = L.LuleshSet.from_mesh(path)
        finally:
            os.unlink(path)
    else:
        mesh = _box(nx * tp)
        flags = (L.FLAG_MIXED if case["mixed"] else 0) | (L.FLAG_COMM_STAGED if case["staged"] else 0)
        s = L.LuleshSet(nx=nx, tp=tp, numReg=case["regions"], balance=case["balance"],
                        cost=case["cost"], flags=flags)
    s.set_stream(_stream().cuda_stream)
    st = _blast(mesh, seed)
    views = _arrays(s)
    dst, src = [], []
    for f in NODE + ELEM:
        whole = _split(st[f], nx, tp, f in NODE) if tp > 1 else st[f].reshape(1, -1)
        for d, t in enumerate(views[f]):
            dst.append(t)
            src.append(whole[d].contiguous().clone())
    outs = [_together(s, views[f]) for f in NODE + ELEM]
    torch.cuda.synchronize()
    state = {"kind": "sedov", "set": s, "stream": _stream(), "dst": dst, "src": src, "outs": outs,
             "views": views, "cycles": case["cycles"], "host": case.get("host", False),
             "single": case.get("mixed", False), "staged": case.get("staged", False),
             "begin": L.JobState(time=T0, deltatime=DT0)}
    # the set has run before it is restarted (its first cycle ever takes dt as given)
    with torch.cuda.stream(state["stream"]):
        torch._foreach_copy_(dst, src)
    s.host_cycle(state["begin"])
    return state


def run(state):
    if state["kind"] == "force":
        ptr = [ctypes.c_void_p(t.data_ptr()) for t in state["ins"]]
        st = state["lib"].lulesh_volume_force_noalloc(
            state["nx"], *ptr, 3.0, *[ctypes.c_void_p(t.data_ptr()) for t in state["outs"]],
            ctypes.c_void_p(state["bad"].data_ptr()),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert st == 0
        return state["outs"] + [state["bad"]]
    if state["kind"] == "batch":
        jobs = state["jobs"]
        with state["L"].LuleshSet.batch(jobs) as s:
            s.set_tuning(elem_block=64, node_block=128, order=0, graph_cycles=8)
            s.run_graph()
            return [s.field("e", j) for j in range(len(jobs))]
    if state["kind"] == "serve":
        srv, jobs = state["srv"], state["jobs"]
        ids = [srv.submit(j) for j in jobs]
        done = {}
        while len(done) < len(jobs):
            srv.step()
            for r in srv.poll():
                done[r["id"]] = r
        return [np.array([done[i]["origin_energy"] for i in ids]),
                np.array([done[i]["time"] for i in ids]),
                np.array([done[i]["cycle"] for i in ids], dtype=np.int64)]
    s = state["set"]
    with torch.cuda.stream(state["stream"]):
        torch._foreach_copy_(state["dst"], state["src"])
        s.host_cycle(state["begin"])  # sets the clock, then the first cycle
        if state["host"]:
            for _ in range(state["cycles"] - 1):
                s.host_cycle()
        else:
            s.step(state["cycles"] - 1)
        outs = [o if o is not None else torch.stack(state["views"][f])
                for f, o in zip(NODE + ELEM, state["outs"])]
        return _in_single(outs) if state["single"] else outs


def work(case):
    """Bytes that have to cross each of a cycle's four grid-wide dependencies
    (each array once: force 120, node update 128, kinematics 144, EOS 168 per
    element) and FP64 operations of the step's sums and products, per element
    and cycle; for the force call its inputs and outputs."""
    n = _zones(case)
    if case["kind"] == "force":
        return {"bytes": 8.0 * (6 * n + 6 * (case["nx"] + 1) ** 3 + 3 * (case["nx"] + 1) ** 3),
                "flops": 1000.0 * n}
    return {"bytes": 560.0 * n, "flops": 2000.0 * n}


# ---------------------------------------------------------------------------
# the same in plain torch, 64 bits

_FACES = ((0, 1, 2, 3), (0, 4, 5, 1), (1, 5, 6, 2), (2, 6, 7, 3), (3, 7, 4, 0), (4, 7, 6, 5))
_SIDES = ((0, 1, 2, 3), (4, 5, 6, 7), (0, 1, 5, 4), (1, 2, 6, 5), (2, 3, 7, 6), (3, 0, 4, 7))
_VDER = ((0, 1, 2, 3, 4, 5, 7), (3, 0, 1, 2, 7, 4, 6), (2, 3, 0, 1, 6, 7, 5), (1, 2, 3, 0, 5, 6, 4),
         (4, 7, 6, 5, 0, 3, 1), (5, 4, 7, 6, 1, 0, 2), (6, 5, 4, 7, 2, 1, 3), (7, 6, 5, 4, 3, 2, 0))
_MODES = ((1, 1, -1, -1, -1, -1, 1, 1), (1, -1, -1, 1, -1, 1, 1, -1),
          (1, -1, 1, -1, 1, -1, 1, -1), (-1, 1, -1, 1, 1, -1, 1, -1))
_CORNER = ((-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1),
           (-1, -1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1))


def _corner_forces(P, V, volo, v, p, q, ss, mass, hgcoef=3.0):
    """Stress and Flanagan-Belytschko hourglass forces [3,8,E]."""
    det = volo * v
    dv = torch.empty_like(P)
    for out, *n in _VDER:
        a = [P[:, i] for i in n]
        s = _cross(a[1] + a[2], a[0] + a[1]) + _cross(a[0] + a[4], a[3] + a[4]) - \
            _cross(a[2] + a[5], a[3] + a[5])
        dv[:, out] = s / 12.0
    g = torch.tensor(_MODES, dtype=F64, device=P.device)
    h = torch.einsum("mk,cke->cme", g, P)
    hg = g[:, :, None] - torch.einsum("cke,cme->mke", dv, h) / det
    s = torch.einsum("mke,cke->cme", hg, V)
    coef = -hgcoef * 0.01 * ss * mass / det.pow(1.0 / 3.0)
    f = coef * torch.einsum("mke,cme->cke", hg, s)
    sig = -(p + q)
    for a, b, c, d in _FACES:
        t0 = 0.5 * (P[:, d] + P[:, c] - P[:, b] - P[:, a])
        t1 = 0.5 * (P[:, c] + P[:, b] - P[:, d] - P[:, a])
        area = -0.25 * sig * _cross(t0, t1)
        for k in (a, b, c, d):
            f[:, k] += area
    return f


def _derivs(A):
    """(d/dxi, d/deta, d/dzeta) at the centre of corner values A [3,8,E]."""
    sg = torch.tensor(_CORNER, dtype=F64, device=A.device)
    return [0.125 * torch.einsum("k,cke->ce", sg[:, a], A) for a in range(3)]


def _limited(d, lm, lp, symm, free):
    norm = 1.0 / (d + 1.0e-36)
    m = torch.where(symm, d, d[lm]) * norm
    q = torch.where(free, torch.zeros_like(d), d[lp]) * norm
    phi = torch.minimum(torch.minimum(0.5 * (m + q), 2.0 * m), 2.0 * q)
    return phi.clamp(0.0, 1.0)


def _pressure(e, comp):
    bvc = (2.0 / 3.0) * (comp + 1.0)
    p = bvc * e
    p = torch.where(p.abs() < 1e-7, torch.zeros_like(p), p)
    return p.clamp(min=0.0), bvc


def _sound(e, vol, bvc, p):
    s = (2.0 / 3.0) * e + vol * vol * bvc * p
    return torch.where(s <= .1111111e-36, torch.full_like(s, .3333333e-18),
                       torch.sqrt(s.clamp(min=.1111111e-36)))


def _cut(e):
    return torch.where(e.abs() < 1e-7, torch.zeros_like(e), e).clamp(min=-1e15)


def _leapfrog(mesh, st, mass_n, mass_e, dt):
    """One Lagrange step of `st` in place; the next step's Courant and hydro dt."""
    X = torch.stack([st["x"], st["y"], st["z"]])
    V = torch.stack([st["xd"], st["yd"], st["zd"]])
    volo = st["volo"]
    f = _corner_forces(X[:, mesh.nodes], V[:, mesh.nodes], volo, st["v"], st["p"], st["q"],
                       st["ss"], mass_e)
    F = torch.zeros_like(X)
    F.index_add_(1, mesh.nodes.reshape(-1), f.reshape(3, -1))
    del f
    acc = torch.where(mesh.symm_node, torch.zeros_like(F), F / mass_n)
    V = V + acc * dt
    V = torch.where(V.abs() < 1e-7, torch.zeros_like(V), V)
    X = X + V * dt
    st["x"], st["y"], st["z"], st["xd"], st["yd"], st["zd"] = [*X, *V]

    P, W = X[:, mesh.nodes], V[:, mesh.nodes]
    vol = _volume(P)
    vnew = vol / volo
    delv = vnew - st["v"]
    area = None
    for a, b, c, d in _SIDES:
        t = 4.0 * _cross(P[:, c] - P[:, a], P[:, d] - P[:, b]).square().sum(0)
        area = t if area is None else torch.maximum(area, t)
    length = 4.0 * vol / torch.sqrt(area)
    jv = _derivs(W)
    j = [a - 0.5 * dt * b for a, b in zip(_derivs(P), jv)]
    cof = [_cross(j[1], j[2]), _cross(j[2], j[0]), _cross(j[0], j[1])]
    vdov = sum(_dot(c, w) for c, w in zip(cof, jv)) / _dot(j[0], cof[0])
    jx = [2.0 * a for a in _derivs(P)]
    delx, delw = [], []
    for a, b, c in ((1, 2, 0), (2, 0, 1), (0, 1, 2)):  # xi, eta, zeta
        n = _cross(jx[a], jx[b])
        delx.append(vol / torch.sqrt(n.square().sum(0) + 1e-36))
        delw.append(_dot(n, 2.0 * jv[c]) / (vol + 1e-36))
    del P, W, cof, j, jx

    phi = [_limited(delw[a], mesh.links[2 * a], mesh.links[2 * a + 1], mesh.symm_face[a],
                    mesh.free_face[a]) for a in range(3)]
    dx = [(w * x).clamp(max=0.0) for w, x in zip(delw, delx)]
    rho = mass_e / (volo * vnew)
    zero = torch.zeros_like(vol)
    ql = torch.where(vdov > 0, zero, -0.5 * rho * sum(d * (1.0 - h) for d, h in zip(dx, phi)))
    qq = torch.where(vdov > 0, zero,
                     (2.0 / 3.0) * rho * sum(d * d * (1.0 - h * h) for d, h in zip(dx, phi)))

    vc, pq = vnew.clamp(1e-9, 1e9), st["p"] + st["q"]
    comp = 1.0 / vc - 1.0
    half = 1.0 / (vc - 0.5 * delv) - 1.0
    grow = delv > 0
    e = (st["e"] - 0.5 * delv * pq).clamp(min=-1e15)
    ph, bvc = _pressure(e, half)
    vh = 1.0 / (1.0 + half)
    qn = torch.where(grow, zero, _sound(e, vh, bvc, ph) * ql + qq)
    e = _cut(e + 0.5 * delv * (3.0 * pq - 4.0 * (ph + qn)))
    p, bvc = _pressure(e, comp)
    qt = torch.where(grow, zero, _sound(e, vc, bvc, p) * ql + qq)
    e = _cut(e - (7.0 * pq - 8.0 * (ph + qn) + (p + qt)) * delv / 6.0)
    p, bvc = _pressure(e, comp)
    q2 = _sound(e, vc, bvc, p) * ql + qq
    qn = torch.where(grow, qn, torch.where(q2.abs() < 1e-7, zero, q2))
    ss = _sound(e, vc, bvc, p)
    st["e"], st["p"], st["q"], st["ss"] = e, p, qn, ss
    st["v"] = torch.where((vnew - 1.0).abs() < 1e-10, torch.ones_like(vnew), vnew)

    on = vdov != 0.0
    big = torch.full_like(vol, 1e20)
    hydro = torch.where(on, 0.1 / (vdov.abs() + 1e-20), big).min()
    dtf = ss * ss + torch.where(vdov < 0, 256.0 * length * length * vdov * vdov, zero)
    courant = torch.where(on, length / torch.sqrt(dtf), big).min()
    return float(courant), float(hydro)


def _advance(mesh, st, cycles, time, dt, first_as_given):
    """`cycles` steps, dt by the time increment's rule; `first_as_given`: a run's
    very first cycle takes dt as it is, a restarted set's grows it by 1.2."""
    volo = st["volo"]
    mass_n = torch.zeros(mesh.xyz.shape[1], dtype=F64, device=volo.device)
    mass_n.index_add_(0, mesh.nodes.reshape(-1), (volo / 8.0).repeat(8))
    courant = hydro = 1e20
    for k in range(cycles):
        target = 1e-2 - time
        if not (k == 0 and first_as_given):
            new = 1e20
            if courant < new:
                new = courant / 2.0
            if hydro < new:
                new = hydro * 2.0 / 3.0
            if new >= dt:
                new = dt if new / dt < 1.1 else min(new, 1.2 * dt)
            dt = min(new, 1e-2)
        if dt < target < 4.0 * dt / 3.0:
            target = 2.0 * dt / 3.0
        dt = min(dt, target)
        time += dt
        courant, hydro = _leapfrog(mesh, st, mass_n, volo, dt)
    return time


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        return None  # thousands of cycles of dozens of meshes
    if kind == "batch":
        outs = []
        for j in _jobs(case, seed):
            mesh = _box(j.nx)
            st = {f: torch.zeros(mesh.xyz.shape[1] if f in NODE else mesh.nodes.shape[1], dtype=F64,
                                 device=_device()) for f in NODE + ELEM}
            st["x"], st["y"], st["z"] = mesh.xyz.clone()
            st["volo"] = _volume(mesh.xyz[:, mesh.nodes])
            st["v"] += 1.0
            deposit = 3.948746e7 * (j.nx / 45.0) ** 3
            st["e"][0] = deposit
            dt = 0.5 * float(st["volo"][0]) ** (1.0 / 3.0) / math.sqrt(2.0 * deposit)
            _advance(mesh, st, j.its, 0.0, dt, True)
            outs.append(st["e"].cpu().numpy())
        return outs
    if kind == "force":
        mesh = _box(case["nx"])
        st = _blast(mesh, seed)
        X = torch.stack([st["x"], st["y"], st["z"]])
        V = torch.stack([st["xd"], st["yd"], st["zd"]])
        f = _corner_forces(X[:, mesh.nodes], V[:, mesh.nodes], st["volo"], st["v"], st["p"],
                           st["q"], st["ss"], st["volo"])
        F = torch.zeros_like(X)
        F.index_add_(1, mesh.nodes.reshape(-1), f.reshape(3, -1))
        return [F[0], F[1], F[2], None]
    nx, tp = case["nx"], case.get("tp", 1)
    mesh = _mesh_on_device(_warped(nx, seed)) if kind == "mesh" else _box(nx * tp)
    st = _blast(mesh, seed)
    _advance(mesh, st, case["cycles"], T0, DT0, False)
    outs = [_split(st[f], nx, tp, f in NODE) for f in NODE + ELEM]
    return _in_single(outs) if case.get("mixed") else outs
