"""What a user has this framework do, as a list of measurable cases.

Every case goes through the public entry points: ``Monodomain.solve`` (whole
simulations), ``Monodomain.step`` (the time step a program drives itself),
``Monodomain.assemble``, ``Monodomain.phie_recovery`` and ``MonodomainBatch``.
``prepare`` makes the mesh, the conductivities and the stimuli on the GPU and
loads them into the simulator objects; ``run`` is the call.

Launch shapes stay at the library's defaults (``autotune=False``): the tuner's
choice is kept in a file per machine, and a timing run inside the measured call
would be measured too.

``exact`` restates the discretised equations in 64 bits with plain torch: P1
matrices, the ionic models with their lookup tables, and linear systems solved
to convergence.  The library stops its solver at the caller's tolerance, so the
distance to ``exact`` is that truncation plus the rounding of its 32-bit state.
"""
import math
from functools import lru_cache

import numpy as np
import torch

CHI, CM, THETA = 140.0, 0.01, 0.5
N_STATES = {"ms": 1, "ttp": 18, "crn": 19}


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest calls: a block of tissue of a thousand nodes, a millisecond-scale run; launches and latency
        _solve("solve_ttp_cube_9", "cube", 9, "ttp", cell="EPI", steps=1000),
        # the 20^3 Mitchell-Schaeffer cube of the repository's first configuration (1 mm spacing, one face paced)
        _solve("solve_ms_cube_20", "cube", 20, "ms", h=1.0, steps=2000),
        # a median serving request: about 50,000 nodes, ten Tusscher-Panfilov
        _solve("solve_ttp_cube_36", "cube", 36, "ttp", steps=1000),
        # the headline configuration's mesh and model, a million nodes, the start of its run
        _solve("solve_ttp_cube_100", "cube", 100, "ttp", steps=1000),
        # an atrial shell as a mesh generator numbers it (neighbours far apart in memory), Courtemanche
        _solve("solve_crn_ico_6", "ico", 6, "crn", dt=0.02, steps=1000),
        # the same at the size of the repository's precision study
        _solve("solve_crn_ico_7", "ico", 7, "crn", dt=0.02, steps=600),
        # a quarter of a million nodes solved tightly and without the extrapolated guess: many CG passes a step
        _solve("solve_ms_cube_63_tight", "cube", 63, "ms", steps=250, tol=1e-8, guess=False, frames=False),
        # a program that drives the time step itself, as the reference's step() allows: one call, one answer
        dict(name="step_ttp_cube_36", kind="step", mesh="cube", n=36, h=0.25, model="ttp", cell="ENDO", dt=0.01, tol=1e-5),
        # many small simulations at once: cubes of 16 to 64 nodes an edge, two models, as the batched configuration
        dict(name="batch_cubes_24", kind="batch", count=24, lo=15, hi=63, models="ms ttp", shells=False, steps=200, tol=1e-5),
        # a serving mix: cubes and shells, all three models
        dict(name="batch_mixed_12", kind="batch", count=12, lo=20, hi=40, models="ms ttp crn", shells=True, steps=300, tol=1e-5),
        # matrices of a new mesh: pattern, element integrals, gather, system values
        dict(name="assemble_cube_80", kind="assemble", mesh="cube", n=80, h=0.25, dt=0.01),
        # extracellular potentials after a run: a Poisson-like solve for every frame, tens of CG passes each
        dict(name="phie_cube_40", kind="phie", mesh="cube", n=40, h=0.25, frames=8, tol=1e-5, max_iter=400),
    ]


def _solve(name, mesh, n, model, h=0.25, dt=0.01, steps=1000, cell="ENDO", tol=1e-5, guess=True, frames=True):
    c = dict(kind="solve", mesh=mesh, n=n, h=h, model=model, cell=cell, dt=dt, steps=steps, tol=tol, guess=guess, frames=frames)
    return dict(c, name=name) if name else c


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: node counts spread over the logarithm of the range, any model, both meshes."""
    kind = rng.choice(["solve"] * 6 + ["step", "batch", "assemble", "phie"])
    nodes = _log(rng, 700, 1_000_000)
    n = max(8, min(99, int(round(nodes ** (1 / 3))) - 1))
    if kind == "solve":
        model = rng.choice(["ms", "ttp", "crn"])
        shell = rng.random() < 0.3
        level = max(3, min(7, int(round(math.log(nodes / 10, 4)))))
        size = 10 * 4 ** level + 2 if shell else (n + 1) ** 3
        steps = max(60, min(1500, int(6e8 / size)))
        tol = rng.choice([1e-5, 1e-5, 1e-5, 1e-6, 1e-8])
        if tol < 1e-5:
            steps = max(60, steps // 3)
        return _solve(None, "ico" if shell else "cube", level if shell else n, model, h=rng.choice([0.2, 0.25, 0.4]),
                      dt=rng.choice([0.01, 0.02]), steps=steps + rng.randrange(40), cell=rng.choice(["ENDO", "EPI"]),
                      tol=tol, guess=rng.random() < 0.8, frames=rng.random() < 0.7)
    if kind == "step":
        model = rng.choice(["ms", "ttp", "crn"])
        return dict(kind="step", mesh="cube", n=n, h=0.25, model=model, cell="ENDO", dt=0.01, tol=1e-5)
    if kind == "batch":
        hi = rng.randrange(24, 56)
        return dict(kind="batch", count=rng.randrange(5, 24), lo=rng.randrange(10, 20), hi=hi,
                    models=rng.choice(["ms ttp", "ms ttp crn", "ttp"]), shells=rng.random() < 0.5,
                    steps=rng.randrange(100, 220), tol=1e-5)
    if kind == "assemble":
        return dict(kind="assemble", mesh="cube", n=max(10, n), h=0.25, dt=0.01)
    return dict(kind="phie", mesh="cube", n=max(10, min(48, n)), h=0.25, frames=rng.randrange(3, 9), tol=1e-5, max_iter=400)


def _bytes_flops(nodes, nnz, model, steps):
    s = N_STATES[model] + 1
    # a time step reads M, K and the pattern, reads and writes the ionic state and V, AT and RT
    per_step = 12 * nnz + nodes * (8 * s + 36)
    arithmetic = nodes * {"ms": 30, "ttp": 330, "crn": 330}[model] + 2 * nnz * 5
    return steps * per_step, steps * arithmetic


def work(case):
    if case["kind"] == "batch":
        got = [_bytes_flops(*_size(p["mesh"], p["n"])[:2], p["model"], case["steps"]) for p in _parts(case, 0)]
        return {"bytes": sum(b for b, _ in got), "flops": sum(f for _, f in got)}
    nodes, nnz, elems, k = _size(case["mesh"], case["n"])
    if case["kind"] in ("solve", "step"):
        b, f = _bytes_flops(nodes, nnz, case["model"], case.get("steps", 1))
        return {"bytes": b, "flops": f}
    mesh = 12 * nodes + elems * (4 * k + 4 * 3 + 8)
    if case["kind"] == "assemble":   # mesh in; row pointers, columns, M, K, A, K' and 1/diag out
        return {"bytes": mesh + 4 * nodes + 20 * nnz, "flops": elems * 250}
    # frames in, potentials out, the matrices once for each frame
    return {"bytes": mesh + case["frames"] * (8 * nodes + 12 * nnz), "flops": case["frames"] * nnz * 2 * 60}


def tolerance(case):
    # Measured against the library's other ionic instances (IEEE instead of hardware division) and the inner
    # products summed over another number of blocks: V 1e-6, activation times 5e-6 and one step of dt, which is
    # 1e-3 of the run's length; the matrices and the single solves against exact().  A step whose residual lies on the solver's
    # tolerance may take a pass more or less, which moves V by up to that tolerance (1e-5 of its norm).
    if case["kind"] == "assemble":
        return {"rel": 1e-6, "max": 1e-5}
    if case["kind"] == "phie":
        return {"rel": 1e-4, "max": 1e-3}
    if case["kind"] == "step":
        return {"rel": 5e-5, "max": 1e-3}
    return {"rel": 1e-4, "max": max(5e-3, 4.0 / case["steps"])}


# ---------------------------------------------------------------- meshes
def _size(mesh, n):
    """(nodes, non-zeros, elements, nodes per element)"""
    if mesh == "cube":
        nodes = (n + 1) ** 3
        return nodes, nodes + 2 * (3 * n * (n + 1) ** 2 + 3 * n * n * (n + 1) + n ** 3), 6 * n ** 3, 4
    return 10 * 4 ** n + 2, 10 * 4 ** n + 2 + 60 * 4 ** n, 20 * 4 ** n, 3


@lru_cache(maxsize=64)
def _cube(n):
    """Node indices (i, j, k) and the six tetrahedra of every cell (around its main diagonal)."""
    g = torch.arange(n + 1, device="cuda")
    ijk = torch.stack(torch.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    c = torch.arange(n, device="cuda")
    i, j, k = (t.reshape(-1) for t in torch.meshgrid(c, c, c, indexing="ij"))
    v = [((i + a) * (n + 1) + j + b) * (n + 1) + k + d
         for a, b, d in ((0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1))]
    tets = [(0, 1, 2, 6), (0, 2, 3, 6), (0, 3, 7, 6), (0, 7, 4, 6), (0, 4, 5, 6), (0, 5, 1, 6)]
    return ijk, torch.stack([torch.stack([v[q] for q in t], -1) for t in tets], 1).reshape(-1, 4).to(torch.int32)


@lru_cache(maxsize=8)
def _sphere(level):
    """Unit icosphere: midpoints are numbered as they appear, so neighbours end up far apart."""
    p = (1 + 5 ** 0.5) / 2
    v = np.array([(-1, p, 0), (1, p, 0), (-1, -p, 0), (1, -p, 0), (0, -1, p), (0, 1, p), (0, -1, -p), (0, 1, -p),
                  (p, 0, -1), (p, 0, 1), (-p, 0, -1), (-p, 0, 1)], dtype=np.float64)
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    f = np.array([(0, 11, 5), (0, 5, 1), (0, 1, 7), (0, 7, 10), (0, 10, 11), (1, 5, 9), (5, 11, 4), (11, 10, 2),
                  (10, 7, 6), (7, 1, 8), (3, 9, 4), (3, 4, 2), (3, 2, 6), (3, 6, 8), (3, 8, 9), (4, 9, 5),
                  (2, 4, 11), (6, 2, 10), (8, 6, 7), (9, 8, 1)])
    for _ in range(level):
        e = np.stack([f[:, [0, 1]], f[:, [1, 2]], f[:, [2, 0]]], 1).reshape(-1, 2)
        e.sort(axis=1)
        uniq, first, inv = np.unique(e[:, 0] * len(v) + e[:, 1], return_index=True, return_inverse=True)
        order = np.argsort(first)
        rank = np.argsort(order)
        mid = v[e[first[order], 0]] + v[e[first[order], 1]]
        m = (len(v) + rank[inv]).reshape(-1, 3)
        v = np.concatenate([v, mid / np.linalg.norm(mid, axis=1, keepdims=True)])
        f = np.concatenate([np.stack([f[:, 0], m[:, 0], m[:, 2]], 1), np.stack([f[:, 1], m[:, 1], m[:, 0]], 1),
                            np.stack([f[:, 2], m[:, 2], m[:, 1]], 1), m], 0)
    return torch.from_numpy(v).cuda(), torch.from_numpy(f.astype(np.int32)).cuda()


def _tissue(part, seed):
    """Mesh, fibres, regions, conductivities and stimulus of one simulation, from the seed."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rnd = np.random.default_rng(seed)
    scale = float(rnd.uniform(0.8, 1.25))
    if part["mesh"] == "cube":
        n, h = part["n"], part["h"]
        ijk, elems = _cube(n)
        # a tenth of the spacing off the lattice: no two elements alike, as in a generated mesh
        nodes = ((ijk + 0.2 * (torch.rand(ijk.shape, generator=gen, device="cuda", dtype=torch.float64) - 0.5)) * h).float()
        centre = nodes[elems.long()].mean(1)
        # fibre angle turning by 120 degrees from one wall to the other
        th = (centre[:, 2] / (n * h) - 0.5) * (2 * math.pi / 3) + float(rnd.uniform(-0.3, 0.3))
        fibres = torch.stack([torch.cos(th), torch.sin(th), torch.zeros_like(th)], 1)
        regions = (1 + (centre[:, 0] > 0.5 * n * h)).int()
        cond = [([1], 0.5272 * scale, 0.2076 * scale, 1.0732, 0.4227), ([2], 0.9074 * scale, 0.3332 * scale, 1.8, 0.7)]
        corner = rnd.integers(0, 2, 3)
        if part["model"] == "ms":   # one face
            axis = int(rnd.integers(0, 3))
            paced = ijk[:, axis] == (n if corner[axis] else 0)
        else:                       # a block of nodes in a corner
            paced = torch.ones(len(ijk), dtype=torch.bool, device="cuda")
            for a in range(3):
                paced &= (ijk[:, a] >= n - 4) if corner[a] else (ijk[:, a] <= 4)
        pulse = (0.0, 1.0, 100.0)
    else:
        unit, elems = _sphere(part["n"])
        nodes = (25.0 * unit).float()
        c = unit[elems.long()].mean(1)
        c = c / c.norm(dim=1, keepdim=True)
        ref = torch.zeros_like(c)
        ref[:, 2] = (c[:, 2].abs() < 0.9).double()
        ref[:, 0] = 1.0 - ref[:, 2]
        e1 = torch.linalg.cross(c, ref)
        e1 = e1 / e1.norm(dim=1, keepdim=True)
        th = (torch.rand(len(c), generator=gen, device="cuda", dtype=torch.float64) * (2 * math.pi))[:, None]
        fibres = (torch.cos(th) * e1 + torch.sin(th) * torch.linalg.cross(c, e1)).float()
        regions = torch.ones(len(elems), device="cuda", dtype=torch.int32)
        cond = [([1], 0.4 * scale, 0.1 * scale, 0.8, 0.3)]
        axis = int(rnd.integers(0, 3))
        paced = unit[:, axis] > 0.97
        pulse = (0.0, 2.0, 50.0)
    return dict(nodes=nodes, elems=elems, regions=regions, fibres=fibres, cond=cond, paced=paced, pulse=pulse)


def _parts(case, seed):
    """The simulations of a batch: sizes fixed by the case, models in turn."""
    sizes = random_sizes(case["count"], case["lo"], case["hi"])
    models = case["models"].split()
    out = []
    for k, n in enumerate(sizes):
        shell = case["shells"] and k % 2 == 1
        out.append(dict(mesh="ico" if shell else "cube", n=(5 if n < (case["lo"] + case["hi"]) // 2 else 6) if shell else n, h=0.25,
                        model=models[k % len(models)], cell="ENDO", dt=0.01, steps=case["steps"], tol=case["tol"]))
    return out


def random_sizes(count, lo, hi):
    return [int(v) for v in np.random.default_rng(2024).integers(lo, hi + 1, size=count)]


# ---------------------------------------------------------------- the calls
def _simulator(part, t, extracellular=False):
    from torchcor_b200.ionic import CourtemancheRamirezNattel, ModifiedMS2v, TenTusscherPanfilov
    from torchcor_b200.simulator import Monodomain
    dt = part["dt"]
    if part["model"] == "ttp":
        ionic = TenTusscherPanfilov(part["cell"], dt, device="cuda")
    elif part["model"] == "crn":
        ionic = CourtemancheRamirezNattel(dt, device="cuda")
    else:
        ionic = ModifiedMS2v(dt, device="cuda")
    sim = Monodomain(ionic, T=(part["steps"] + 0.5) * dt, dt=dt, device="cuda")
    sim.load_device_arrays(t["nodes"], t["elems"], t["regions"], t["fibres"])
    for ids, il, it, el, et in t["cond"]:
        sim.add_conductivity(ids, il, it, *((el, et) if extracellular else ()))
    start, duration, intensity = t["pulse"]
    sim.add_stimulus(None, start, duration, intensity, region=torch.nonzero(t["paced"])[:, 0].cpu().numpy())
    return sim


def _wave(t, seed, frames):
    """Membrane potentials of a front crossing the tissue."""
    rnd = np.random.default_rng(seed + 5)
    x = t["nodes"].double()
    d = torch.tensor(rnd.normal(size=3), device="cuda")
    s = x @ (d / d.norm())
    s = (s - s.min()) / (s.max() - s.min())
    at = torch.linspace(0.15, 0.85, frames, device="cuda", dtype=torch.float64)[:, None]
    return (-85.0 + 105.0 * torch.sigmoid((at - s) / 0.04)).float()


def prepare(case, seed):
    if case["kind"] == "batch":
        parts = _parts(case, seed)
        return dict(case=case, sims=[_simulator(p, _tissue(p, seed * 1000 + k)) for k, p in enumerate(parts)])
    part = dict(case)
    if case["kind"] in ("assemble", "phie"):
        part.update(model="ms", dt=case.get("dt", 0.01), steps=100)
    if case["kind"] == "step":
        part.update(steps=60000)
    t = _tissue(part, seed)
    st = dict(case=case, sim=_simulator(part, t, extracellular=case["kind"] == "phie"))
    if case["kind"] == "phie":
        st["vm"] = _wave(t, seed, case["frames"])
    if case["kind"] == "step":
        st["sim"].prepare(case["tol"], case["tol"], 100, snapshot_interval=st["sim"].T)
        st["u"] = _wave(t, seed, 1)[0].contiguous()
    return st


def _activation(sim):
    """Activation times, the end of the run where the front has not come yet: a map as it is drawn, in which a
    node on the threshold at the last step counts a step early or late and not as a node without a time."""
    at = sim.activation_time
    return torch.where(at < 0, sim.nt * sim.dt, at)


def run(state):
    c = state["case"]
    if c["kind"] == "batch":
        from torchcor_b200.simulator import MonodomainBatch
        batch = MonodomainBatch("cuda", max_sims=64)
        for sim in state["sims"]:
            sim.prepare(c["tol"], c["tol"], 100, snapshot_interval=sim.T)
            batch.add(sim)
        batch.run()
        return {k: torch.cat([f(s).reshape(-1) for s in state["sims"]]) for k, f in (
            ("AT", _activation), ("RT", lambda s: s.repolarization_time), ("Vm", lambda s: s.current_solution()),
            ("state", lambda s: s.ionic_model.state[:, : s.n_nodes]))}
    sim = state["sim"]
    if c["kind"] == "assemble":
        s = sim.assemble()
        return {"rowptr": s.rowptr, "col": s.col, "M": s.m_val, "K": s.k_val, "A": s.a_val, "D": s.d_inv[: s.n]}
    if c["kind"] == "phie":
        return {"phi": sim.phie_recovery(a_tol=c["tol"], r_tol=c["tol"], max_iter=c["max_iter"], Vm=state["vm"])}
    if c["kind"] == "step":
        u = sim.step(state["u"], c["dt"], c["tol"], c["tol"], 100)[0]
        return {"Vm": u, "state": sim.ionic_model.state[:, : sim.n_nodes]}
    sim.solve(c["tol"], c["tol"], 100, linear_guess=c["guess"], snapshot_interval=1 if c["frames"] else sim.T,
              verbose=False, autotune=False)
    out = {"AT": _activation(sim), "RT": sim.repolarization_time, "Vm": sim.current_solution(),
           "state": sim.ionic_model.state[:, : sim.n_nodes]}
    if c["frames"]:
        out["frames"] = sim.solutions
    return out


# ---------------------------------------------------------------- the same in 64 bits
def _elements(t, sl, st):
    """(Ke, Me) of every element: P1 stiffness with sigma = st I + (sl - st) f f^T, consistent mass."""
    x = t["nodes"].double()[t["elems"].long()]
    f = t["fibres"].double()
    k = x.shape[1]
    edges = x[:, 1:] - x[:, :1]                                    # rows: edge vectors
    gram = edges @ edges.transpose(1, 2)
    measure = torch.linalg.det(gram).abs().sqrt() / (6.0 if k == 4 else 2.0)
    grad = torch.linalg.solve(gram, edges)                         # gradients of nodes 1.. (tangential for shells)
    grad = torch.cat([-grad.sum(1, keepdim=True), grad], 1)
    gf = (grad * f[:, None, :]).sum(-1)
    ke = st[:, None, None] * (grad @ grad.transpose(1, 2)) + (sl - st)[:, None, None] * gf[:, :, None] * gf[:, None, :]
    me = (torch.ones(k, k, device=x.device, dtype=x.dtype) + torch.eye(k, device=x.device, dtype=x.dtype)) / (20.0 if k == 4 else 12.0)
    return measure[:, None, None] * ke, measure[:, None, None] * me


def _sparse(t, blocks):
    """CSR (rowptr, col) and one value array for each set of element matrices."""
    el, n = t["elems"].long(), t["nodes"].shape[0]
    k = el.shape[1]
    key = (el[:, :, None] * n + el[:, None, :]).reshape(-1)
    uniq, inv = torch.unique(key, return_inverse=True)
    vals = [torch.zeros(len(uniq), device="cuda", dtype=torch.float64).index_add_(0, inv, b.reshape(-1)) for b in blocks]
    row, col = uniq // n, uniq % n
    ptr = torch.zeros(n + 1, device="cuda", dtype=torch.int64)
    ptr[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    return ptr, row, col, vals


def _sigmas(t, extracellular):
    il, it, el, et = (torch.zeros(len(t["regions"]), device="cuda", dtype=torch.float64) for _ in range(4))
    for ids, a, b, c, d in t["cond"]:
        for r in ids:
            m = t["regions"] == r
            for v, w in ((il, a), (it, b), (el, c), (et, d)):
                v[m] = float(np.float32(w))
    return (il, it, el, et) if extracellular else (il, it)


def _csr(ptr, col, val):
    n = len(ptr) - 1
    return torch.sparse_csr_tensor(ptr.int(), col.int(), val, size=(n, n))


def _cg(a, d, b, x, its=500):
    """Jacobi-PCG to convergence (checked every few passes)."""
    r = b - a @ x
    z = d * r
    p = z.clone()
    rz = torch.dot(r, z)
    stop = 1e-22 * torch.dot(b, d * b) + 1e-300
    for k in range(its):
        ap = a @ p
        alpha = rz / torch.dot(p, ap)
        x = x + alpha * p
        r = r - alpha * ap
        z = d * r
        new = torch.dot(r, z)
        if k % 4 == 3 and bool(new <= stop):
            break
        p = z + (new / rz) * p
        rz = new
    return x


def _join(tissues):
    """Several meshes as one (block-diagonal) system."""
    off, out = 0, dict(nodes=[], elems=[], regions=[], fibres=[], paced=[])
    for t in tissues:
        out["nodes"].append(t["nodes"])
        out["elems"].append(t["elems"].long() + off)
        off += len(t["nodes"])
        for k in ("regions", "fibres", "paced"):
            out[k].append(t[k])
    return {k: torch.cat(v) for k, v in out.items()}


def _matrices(t):
    sl, st = _sigmas(t, False)
    return _sparse(t, _elements(t, sl, st))


def _simulate(parts, tissues, frame_every):
    """AT, RT, V, state and frames of simulations of one model, side by side in one system."""
    model, cell, dt, steps = (parts[0][k] for k in ("model", "cell", "dt", "steps"))
    mats = [_matrices(t) for t in tissues]
    off = np.cumsum([0] + [len(t["nodes"]) for t in tissues])
    nz = np.cumsum([0] + [len(m[2]) for m in mats])
    ptr = torch.cat([m[0][(0 if k == 0 else 1):] + int(nz[k]) for k, m in enumerate(mats)])
    row = torch.cat([m[1] + int(off[k]) for k, m in enumerate(mats)])
    col = torch.cat([m[2] + int(off[k]) for k, m in enumerate(mats)])
    kv, mv = (torch.cat([m[3][j] for m in mats]) for j in (0, 1))
    kv = kv / CHI
    av = CM * mv + THETA * dt * kv
    diag = torch.zeros(int(off[-1]), device="cuda", dtype=torch.float64)
    diag[row[row == col]] = av[row == col]
    a, m, k = _csr(ptr, col, av), _csr(ptr, col, mv), _csr(ptr, col, (1 - THETA) * dt * kv)
    d = 1.0 / diag
    stim = torch.cat([t["paced"].double() * t["pulse"][2] for t in tissues])
    until = torch.cat([torch.full((len(t["nodes"]),), t["pulse"][1], device="cuda", dtype=torch.float64) for t in tissues])
    last = float(until.max())
    ionic = {"ms": MS, "ttp": TTP, "crn": CRN}[model](dt, cell)
    u, s = ionic.initial(int(off[-1]))
    at, rt = torch.full_like(u, -1.0), torch.full_like(u, -1.0)
    frames, prev, t = [u.clone()], u, 0.0
    for n in range(1, steps + 1):
        t += dt
        b = CM * u + dt * ionic.step(u, s) / 100.0
        if t <= last:
            b = b + dt * torch.where(t <= until, stim, 0.0) / 100.0
        new = _cg(a, d, m @ b - k @ u, 2 * u - prev)
        prev, u = u, new
        at = torch.where((u > 0) & (at == -1), t, at)
        rt = torch.where((at > 0) & (rt == -1) & (u < -70), t, rt)
        if frame_every and n % frame_every == 0:
            frames.append(u)
    return torch.where(at < 0, steps * dt, at), rt, u, s, frames, off


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        parts = _parts(case, seed)
        tissues = [_tissue(p, seed * 1000 + k) for k, p in enumerate(parts)]
        got = [None] * len(parts)
        for model in sorted({p["model"] for p in parts}):
            at = [k for k, p in enumerate(parts) if p["model"] == model]
            a, r, u, s, _, off = _simulate([parts[k] for k in at], [tissues[k] for k in at], 0)
            for j, k in enumerate(at):
                w = slice(int(off[j]), int(off[j + 1]))
                got[k] = (a[w], r[w], u[w], s[:, w].reshape(-1))
        return {n: torch.cat([g[j] for g in got]) for j, n in enumerate(("AT", "RT", "Vm", "state"))}
    part = dict(case)
    if kind in ("assemble", "phie"):
        part.update(model="ms")
    t = _tissue(part, seed)
    if kind == "assemble":
        ptr, row, col, (kv, mv) = _matrices(t)
        kv = kv / CHI
        av = CM * mv + THETA * case["dt"] * kv
        return {"rowptr": None, "col": None, "M": mv, "K": kv, "A": av, "D": 1.0 / av[row == col]}
    if kind == "phie":
        il, it, el, et = _sigmas(t, True)
        ptr, row, col, (kie, ki) = _sparse(t, [_elements(t, il + el, it + et)[0], _elements(t, il, it)[0]])
        a, m, d = _csr(ptr, col, kie), _csr(ptr, col, ki), 1.0 / kie[row == col]
        out, x = [], torch.zeros(len(d), device="cuda", dtype=torch.float64)
        for v in _wave(t, seed, case["frames"]).double():
            x = _cg(a, d, -(m @ v), x, 2000)
            x = x - x.mean()
            out.append(x)
        return {"phi": torch.stack(out)}
    if kind == "step":
        u = _wave(t, seed, 1)[0].double()
        ionic = {"ms": MS, "ttp": TTP, "crn": CRN}[case["model"]](case["dt"], case["cell"])
        _, s = ionic.initial(len(u))
        ptr, row, col, (kv, mv) = _matrices(t)
        kv, dt = kv / CHI, case["dt"]
        av = CM * mv + THETA * dt * kv
        b = CM * u + dt * ionic.step(u, s) / 100.0 + dt * t["paced"].double() * t["pulse"][2] / 100.0
        b = _csr(ptr, col, mv) @ b - (1 - THETA) * dt * (_csr(ptr, col, kv) @ u)
        return {"Vm": _cg(_csr(ptr, col, av), 1.0 / av[row == col], b, u), "state": s}
    if case["steps"] * _size(case["mesh"], case["n"])[0] > 1.2e9:
        return None   # longer than a few seconds in plain torch
    a, r, u, s, frames, _ = _simulate([part], [t], int(1 / case["dt"]) if case["frames"] else 0)
    out = {"AT": a, "RT": r, "Vm": u, "state": s}
    if case["frames"]:
        out["frames"] = torch.stack(frames)
    return out


def _full(rows, n):
    return torch.tensor(rows, device="cuda", dtype=torch.float64)[:, None].expand(-1, n).clone()


def _grid(lo, hi, res):
    return torch.arange(lo, hi, res, device="cuda", dtype=torch.float64)


def _clean(tab):
    """A grid point on a removable singularity takes the mean of its neighbours."""
    bad = ~torch.isfinite(tab)
    return torch.where(bad, 0.5 * (tab.roll(1, 0) + tab.roll(-1, 0)), tab)


def _look(x, tab, lo, hi, res):
    x = x.clamp(lo, hi)
    i = ((x - lo) / res).long().clamp(0, len(tab) - 2)
    w = ((x - (lo + i * res)) / res)[:, None]
    return ((1 - w) * tab[i] + w * tab[i + 1]).T


class MS:
    """Two-variable Mitchell-Schaeffer, dimensional."""

    def __init__(self, dt, cell):
        self.dt = dt

    def initial(self, n):
        return _full([-80.0], n)[0], _full([1.0], n)

    def step(self, V, s):
        x, h = (V + 80.0) / 100.0, s[0].clone()
        dv = 100.0 * (h * x * (x - 0.13) * (1.0 - x) / 0.1 - (1.0 - h) * x / 9.0)
        s[0] = h + self.dt * torch.where(x > 0.13, -h / 120.0, (1.0 - h) / 100.0)
        return dv


def _gates(dt, pairs):
    cols = []
    for inf, tau in pairs:
        cols += [-inf * torch.expm1(-dt / tau), torch.exp(-dt / tau)]
    return cols


class TTP:
    """ten Tusscher-Panfilov 2006 as openCARP discretises it (tables over V, CaSS and V - EK)."""
    RTF = 8314.472 * 310.0 / 96485.3415

    def __init__(self, dt, cell):
        self.dt, self.gks, self.gto = dt, 0.392, 0.294 if cell == "EPI" else 0.073
        E, F = torch.exp, 1.0 / self.RTF
        c = _grid(1e-5, 10.0, 1e-5)
        q = 1 + (c / 0.05) ** 2
        self.cass = torch.stack(_gates(dt, [(0.6 / q + 0.4, 80.0 / q + 2.0)]), 1)
        V = _grid(-800.0, 800.0, 0.05)
        low = V < -40.0
        h_inf = 1 / (1 + E((V + 71.55) / 7.43)) ** 2
        a_h = torch.where(low, 0.057 * E(-(V + 80) / 6.8), 0.0)
        b_h = torch.where(low, 2.7 * E(0.079 * V) + 3.1e5 * E(0.3485 * V), 0.77 / (0.13 * (1 + E(-(V + 10.66) / 11.1))))
        a_j = torch.where(low, (-2.5428e4 * E(0.2444 * V) - 6.948e-6 * E(-0.04391 * V)) * (V + 37.78) / (1 + E(0.311 * (V + 79.23))), 0.0)
        b_j = torch.where(low, 0.02424 * E(-0.01052 * V) / (1 + E(-0.1378 * (V + 40.14))), 0.6 * E(0.057 * V) / (1 + E(-0.1 * (V + 32))))
        t_d = (1.4 / (1 + E((-35 - V) / 13)) + 0.25) * (1.4 / (1 + E((V + 5) / 5))) + 1 / (1 + E((50 - V) / 20))
        t_f = 1102.5 * E(-(V + 27) ** 2 / 225) + 200 / (1 + E((13 - V) / 10)) + 180 / (1 + E((V + 30) / 10)) + 20
        t_f2 = 562 * E(-(V + 27) ** 2 / 240) + 31 / (1 + E((25 - V) / 10)) + 80 / (1 + E((V + 30) / 10))
        t_m = (0.1 / (1 + E((V + 35) / 5)) + 0.1 / (1 + E((V - 50) / 200))) / (1 + E((-60 - V) / 5))
        t_r = 9.5 * E(-(V + 40) ** 2 / 1800) + 0.8
        t_s = 1000 * E(-(V + 67) ** 2 / 1000) + 8 if cell == "ENDO" else 85 * E(-(V + 45) ** 2 / 320) + 5 / (1 + E((V - 20) / 5)) + 3
        t_x1 = 450 / (1 + E((-45 - V) / 10)) * 6 / (1 + E((V + 30) / 11.5))
        t_x2 = 3 / (1 + E((-60 - V) / 20)) * 1.12 / (1 + E((V - 60) / 20))
        t_xs = 1400 / torch.sqrt(1 + E((5 - V) / 6)) / (1 + E((V - 35) / 15)) + 80
        den = 1000.0 / (87.5 ** 3 + 140.0 ** 3) / (1.38 + 2.0) / (1 + 0.1 * E(-0.65 * V * F))
        self.v = torch.stack(_gates(dt, [
            (1 / (1 + E((-8 - V) / 7.5)), t_d), (1 / (1 + E((V + 20) / 7)), t_f), (0.67 / (1 + E((V + 35) / 7)) + 0.33, t_f2),
            (h_inf, 1 / (a_h + b_h)), (h_inf, 1 / (a_j + b_j)), (1 / (1 + E((-56.86 - V) / 9.03)) ** 2, t_m),
            (1 / (1 + E((20 - V) / 6)), t_r), (1 / (1 + E((V + 20) / 5)), t_s), (1 / (1 + E((-26 - V) / 7)), t_x1),
            (1 / (1 + E((V + 88) / 24)), t_x2), (1 / (1 + E((-5 - V) / 14)), t_xs)]) + [
            den * 2.0 * E(0.35 * V * F), den * E(-0.65 * V * F) * 140.0 ** 3 * 2.5, 0.25 * E(2 * (V - 15) * F),
            1 / (1 + 0.1245 * E(-0.1 * V * F) + 0.0353 * E(-V * F)), 1 / (1 + E((25 - V) / 5.98))], 1)
        a = 0.1 / (1 + E(0.06 * (V - 200)))
        b = (3 * E(0.0002 * (V + 100)) + E(0.1 * (V - 10))) / (1 + E(-0.5 * V))
        self.k1 = (a / (a + b))[:, None]
        self.v, self.k1 = _clean(self.v), _clean(self.k1)

    def initial(self, n):
        #           CaSR  CaSS  Cai   D  F  F2 FCaSS  H     J   Ki     M    Nai  R   R_  S   Xr1 Xr2 Xs
        return _full([-86.2], n)[0], _full([1.3, 7e-5, 7e-5, 0., 1., 1., 1., 0.75, 0.75, 138.3, 0., 7.67, 0., 1., 1., 0., 1., 0.], n)

    def step(self, V, s):
        casr, cass, cai, D, F, F2, FC, H, J, ki, M, nai, R, R_, S, X1, X2, Xs = s.clone()
        g, dt, rtf, fc = _look(V, self.v, -800.0, 800.0, 0.05), self.dt, self.RTF, 96485.3415
        cg = _look(cass, self.cass, 1e-5, 10.0, 1e-5)
        log = torch.log
        eca, ek, ena = 0.5 * rtf * log(2.0 / cai), rtf * log(5.4 / ki), rtf * log(140.0 / nai)
        eks = rtf * log((5.4 + 0.03 * 140.0) / (ki + 0.03 * nai))
        x = 2 * (V - 15.0) / rtf
        a1 = 3.98e-5 * fc / rtf * 4.0 * torch.where(V == 15.0, 0.5 / rtf, (V - 15.0) / torch.expm1(x))
        vk = V - ek
        ipca, ikr, iks = 0.1238 * cai / (0.0005 + cai), 0.153 * X1 * X2 * vk, self.gks * Xs * Xs * (V - eks)
        ina, inak = 14.838 * M ** 3 * H * J * (V - ena), 2.724 * (5.4 / 6.4) * nai / (nai + 40.0) * g[25]
        ibca, ibna, ipk, ito = 0.000592 * (V - eca), 0.00029 * (V - ena), 0.0146 * g[26] * vk, self.gto * R * S * vk
        ical = D * F * F2 * FC * (a1 * g[24] * cass - a1 * 2.0)
        inaca = g[22] * nai ** 3 - g[23] * cai
        ik1 = 5.405 * _look(vk, self.k1, -800.0, 800.0, 0.05)[0] * vk
        ion = ikr + iks + ik1 + ito + ina + ibna + ical + ibca + inak + inaca + ipca + ipk
        vc, vsr, vss, cap = 0.016404, 0.001094, 0.00005468, 0.185
        leak, up, xfer = 0.00036 * (casr - cai), 0.006375 / (1 + 0.00025 ** 2 / cai ** 2), 0.0038 * (cass - cai)
        kc = 2.5 - 1.5 / (1 + (1.5 / casr) ** 2)
        inv = cap / (vc * fc)
        s[0] = casr + dt * (up - leak) / (1 + 10.0 * 0.3 / (casr + 0.3) ** 2)
        s[1] = cass + dt * (-xfer * vc / vss - ical * cap / (2 * vss * fc)) / (1 + 0.4 * 0.00025 / (cass + 0.00025) ** 2)
        s[2] = cai + dt * (xfer - (ibca + ipca - 2 * inaca) * inv / 2 - (up - leak) * vsr / vc) / (1 + 0.2 * 0.001 / (cai + 0.001) ** 2)
        s[9] = ki - dt * (ik1 + ito + ikr + iks - 2 * inak + ipk) * inv
        s[11] = nai - dt * (ina + ibna + 3 * inak + 3 * inaca) * inv
        s[13] = R_ + dt * (0.005 * (1 - R_) - 0.045 * kc * cass * R_)
        for k, row in enumerate((3, 4, 5, 7, 8, 10, 12, 14, 15, 16, 17)):
            s[row] = g[2 * k] + g[2 * k + 1] * s[row]
        s[6] = cg[0] + cg[1] * FC
        return -ion


class CRN:
    """Courtemanche-Ramirez-Nattel 1998 as openCARP discretises it (tables over V, Cai and the release flux)."""

    def __init__(self, dt, cell):
        self.dt = dt
        E, R, T, F = torch.exp, 8.3143, 310.0, 96.4867
        self.rtf = rtf = R * T / F
        con = _grid(3e-4, 30.0, 3e-4) / 1000
        self.ca = torch.stack([
            0.005 / (1 + 0.00092 / con),
            (0.07 * 0.0005 / (con + 0.0005) ** 2 + 0.05 * 0.00238 / (con + 0.00238) ** 2 + 1) / 0.00705882352941176 / 1000,
            0.275 * con / (0.0005 + con) - 0.00113 * rtf / 2 * torch.log(1.8 / con), con,
            -1 / (1 + con / 0.00035) * math.expm1(-dt / 2.0)], 1)
        V = _grid(-200.0, 200.0, 0.1)
        low = V < -40.0
        e_na = rtf * math.log(140.0 / 11.2)
        a_h = torch.where(low, 0.135 * E((V + 80) / -6.8), 0.0)
        b_h = torch.where(low, 3.56 * E(0.079 * V) + 3.1e5 * E(0.35 * V), 1 / 0.13 / (1 + E(-(V + 10.66) / 11.1)))
        a_j = torch.where(low, (-127140 * E(0.2444 * V) - 3.474e-5 * E(-0.04391 * V)) * (V + 37.78) / (1 + E(0.311 * (V + 79.23))), 0.0)
        b_j = torch.where(low, 0.1212 * E(-0.01052 * V) / (1 + E(-0.1378 * (V + 40.14))), 0.3 * E(-2.535e-7 * V) / (1 + E(-0.1 * (V + 32))))
        a_m, b_m = 0.32 * (V + 47.13) / (1 - E(-0.1 * (V + 47.13))), 0.08 * E(-V / 11)
        oa = 0.65 / (E((V + 10) / -8.5) + E((30 - V) / 59)) + 0.65 / (2.5 + E((V + 82) / 17))
        oi = 1 / (18.53 + E((V + 113.7) / 10.95)) + 1 / (35.56 + E(-(V + 1.26) / 7.44))
        ui = 1 / (21 + E((V - 185) / -28)) + E((V - 158) / 16)
        xr = 0.0003 * (V + 14.1) / (1 - E((V + 14.1) / -5)) + 7.3898e-5 * (V - 3.3328) / (E((V - 3.3328) / 5.1237) - 1)
        xs = 4e-5 * (V - 19.9) / (1 - E((19.9 - V) / 17)) + 3.5e-5 * (V - 19.9) / (E((V - 19.9) / 9) - 1)
        t_d = (1 - E(-(V + 10) / 6.24)) / 0.035 / (V + 10) / (1 + E(-(V + 10) / 6.24))
        t_f = 9 / (0.0197 * E(-0.0337 ** 2 * (V + 10) ** 2) + 0.02)
        t_w = 6 * (1 - E((7.9 - V) / 5)) / (1 + 0.3 * E((7.9 - V) / 5)) / (V - 7.9)
        sig = (math.exp(140.0 / 67.3) - 1) / 7
        nak = 0.6 / (1 + 0.1245 * E(-0.1 * V / rtf) + 0.0365 * sig * E(-V / rtf)) / (1 + (10.0 / 11.2) ** 1.5) * 5.4 / 6.9
        ex = 1600.0 / (669921.875 + 140.0 ** 3) / (1.38 + 1.8) / (1 + 0.1 * E(-0.65 * V / rtf))
        rate = lambda a, b: (a / (a + b), 1 / (a + b))  # noqa: E731
        self.v = _clean(torch.stack(_gates(dt, [
            (1 / (1 + E(-(V + 10) / 8)), t_d), (1 / (1 + E((V + 28) / 6.9)), t_f), rate(a_h, b_h), rate(a_j, b_j), rate(a_m, b_m),
            (1 / (1 + E(-(V + 20.47) / 17.54)), 1 / oa / 3), (1 / (1 + E((V + 43.1) / 5.3)), 1 / oi / 3),
            (1 / (1 + E((V + 30.3) / -9.6)), 1 / oa / 3), (1 / (1 + E((V - 99.45) / 27.48)), 1 / ui / 3),
            (1 - 1 / (1 + E((40 - V) / 17)), t_w), (1 / (1 + E((V + 14.1) / -6.5)), 1 / xr),
            (1 / torch.sqrt(1 + E((V - 19.9) / -12.7)), 0.5 / xs)]) + [
            0.1238 * (V - 65), 7.8 * (V - e_na), ex * E(0.35 * V / rtf) * 11.2 ** 3 * 1.8, ex * E(-0.65 * V / rtf) * 140.0 ** 3 / 1000,
            0.005 + 0.05 / (1 + E((15 - V) / 13)), 0.00113 * V, 0.000674 * (V - e_na), nak], 1))
        fn = _grid(-2e-11, 10e-11, 2e-15)
        k = 1 / (1 + E((3.4175e-13 - fn) / 13.67e-16))
        t_v = 1.91 + 2.09 * k
        v_inf = 1 - 1 / (1 + E((6.835e-14 - fn) / 13.67e-16))
        self.fn = torch.stack([-k * math.expm1(-dt / 8.0), -v_inf * torch.expm1(-dt / t_v), E(-dt / t_v)], 1)

    def initial(self, n):
        #      Ca_rel Ca_up Cai    Ki     d        f      f_Ca   h      j      m        oa       oi     u   ua       ui     v   w      xr       xs
        rows = [1.49, 1.49, 0.102, 139.0, 1.37e-4, 0.999, 0.775, 0.965, 0.978, 2.91e-3, 3.04e-2, 0.999, 0., 4.96e-3, 0.999, 1., 0.999, 3.29e-5, 1.87e-2]
        return _full([-81.2], n)[0], _full(rows, n)

    def step(self, V, s):
        rel, up, cai, ki, d, f, fca, h, j, m, oa, oi, u, ua, ui, v, w, xr, xs = s.clone()
        g, c, dt, E = _look(V, self.v, -200.0, 200.0, 0.1), _look(cai, self.ca, 3e-4, 30.0, 3e-4), self.dt, torch.exp
        vk = V - self.rtf * torch.log(5.4 / ki)
        ical, ina, inaca = g[24] * d * f * fca, g[25] * m ** 3 * h * j, g[26] - cai * g[27]
        ik1, ikr = 0.09 * vk / (1 + E(0.07 * (V + 80))), 0.0294 * vk / (1 + E((V + 15) / 22.4)) * xr
        iks, ikur, ito = 0.129 * vk * xs ** 2, g[28] * vk * ua ** 3 * ui, 0.1652 * vk * oa ** 3 * oi
        ipca = c[2] + g[29]
        ion = ina + ik1 + ito + ikur + ikr + iks + ical + ipca + inaca + g[30] + g[31]
        tr, irel = (up - rel) / 180.0, u * u * v * 30.0 * w * (rel - c[3])
        dup = c[0] - 0.005 / 15.0 * up
        s[0] = rel + dt * (tr - irel) / (1 + 8.0 / (rel + 0.8) ** 2)
        s[1] = up + dt * (dup - tr * 0.0869565217391304)
        s[2] = cai + dt * (0.00537112496043221 * (2 * inaca - ipca - ical) - 11.5 * dup + irel) / c[1]
        s[3] = ki - dt * (ito + ikr + ikur + iks + ik1 - 2 * g[31]) / (96.4867 * 13668.0)
        q = _look(9.648e-13 * irel - 2.5910306809e-13 * (ical - 0.4 * inaca), self.fn, -2e-11, 10e-11, 2e-15)
        for k, row in enumerate((4, 5, 7, 8, 9, 10, 11, 13, 14, 16, 17, 18)):
            s[row] = g[2 * k] + g[2 * k + 1] * s[row]
        s[6] = c[4] + math.exp(-dt / 2.0) * fca
        s[12] = q[0] + math.exp(-dt / 8.0) * u
        s[15] = q[1] + q[2] * v
        return -ion
