"""The work a user of this framework has it do, as measurable cases.

Four paths, each through its public entry points: the demag solve (``Problem.solve_u``), the energy
and gradient (``make_energy_kernels``), one field step of a hysteresis loop (``make_minimizer``) and
the warm-start network (``learned.UNet``).  Meshes are the graded cubes and the voxelised ellipsoids
of ``synthetic``.  A hysteresis loop keeps one mesh and its handle over hundreds of field steps, so
the handle belongs to the case; the magnetisation, the initial guess and the network's input belong
to the seed.
"""

from __future__ import annotations

import dataclasses
import functools
import math

import numpy as np
import torch

from mumag_matrixfree2_gb300 import fem_utils, learned
from mumag_matrixfree2_gb300 import synthetic as syn
from mumag_matrixfree2_gb300.cuda_backend import problem_for_geom
from mumag_matrixfree2_gb300.energy_kernels import make_energy_kernels
from mumag_matrixfree2_gb300.minimizers import make_minimizer
from mumag_matrixfree2_gb300.poisson_solve import make_solve_U

TOL = 1e-10  # relative residual of every demag solve, as in the hysteresis loops
WEIGHTS_SEED = 3  # the network's weights are the case's, its input is the seed's


def _cube(L, h, r, n_air, box):
    return {"mesh": "cube", "L": L, "h": h, "r": r, "n_air": n_air, "box": box}


CUBE8 = _cube(8.0, 2.0, 1.3, 3, 24.0)  # 1,331 nodes
CUBE40 = _cube(40.0, 2.0, 1.2, 9, 200.0)  # 59,319 nodes
CUBE80 = _cube(80.0, 1.6, 1.15, 10, 200.0)  # 357,911 nodes
CUBE120 = _cube(120.0, 1.2, 1.2, 8, 240.0)  # 1,601,613 nodes
PARTICLE = {"mesh": "ellipsoid", "a": 7.3, "b": 11.9, "c": 18.4}  # a ragged voxelised body, three different axes


def listed():
    return [
        # the smallest solve: launches and waits, no bandwidth
        {"name": "solve_cube8_fp64", "path": "solve", **CUBE8, "precision": "fp64", "start": "zero", "arrays": "device"},
        # a small magnet, called with host arrays as the reference's solve_U is
        {"name": "solve_cube40_fp64_host", "path": "solve", **CUBE40, "precision": "fp64", "start": "zero",
         "arrays": "host"},
        # the headline solve in the plain method and with the FP32 V-cycle
        {"name": "solve_cube80_fp64", "path": "solve", **CUBE80, "precision": "fp64", "start": "zero", "arrays": "device"},
        {"name": "solve_cube80_fp32v", "path": "solve", **CUBE80, "precision": "fp32_precond", "start": "zero",
         "arrays": "device"},
        # one particle of a batch in iterative refinement, warm-started from the previous state's potential
        {"name": "solve_particle_mixed", "path": "solve", **PARTICLE, "precision": "mixed", "start": "previous",
         "arrays": "device"},
        # the largest magnet
        {"name": "solve_cube120_fp64", "path": "solve", **CUBE120, "precision": "fp64", "start": "zero",
         "arrays": "device"},
        # energy evaluations of the line search: FP64, and float-float as the mixed modes take them
        {"name": "energy_cube120_ff", "path": "energy", **CUBE120, "precision": "fp32_precond"},
        {"name": "energy_cube80_fp64", "path": "energy", **CUBE80, "precision": "fp64"},
        # whole field steps: the loop's default method, one particle of a batch, a quasi-Newton method
        {"name": "step_cube80_fp64", "path": "minimize", **CUBE80, "precision": "fp64", "method": "pcohen_hs",
         "B_T": -3.0},
        {"name": "step_particle_fp32v", "path": "minimize", **PARTICLE, "precision": "fp32_precond",
         "method": "pcohen_hs", "B_T": 1.0},
        {"name": "step_cube40_lbfgs", "path": "minimize", **CUBE40, "precision": "fp64", "method": "lbfgs", "B_T": -2.0},
        # the warm-start network's training pass (forward, loss, gradients) at its training size
        {"name": "network_32x8", "path": "network", "grid": 32, "batch": 8},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _draw_mesh(rng, most_cells):
    """A cube of 3 .. 90 cells or an ellipsoid of the batch's sizes; at most most_cells cells an axis."""
    if rng.random() < 0.4:
        return {"mesh": "ellipsoid", **{k: round(_log(rng, 5.0, 25.0), 2) for k in "abc"}}
    n_air = rng.randint(3, 10)
    cells = int(_log(rng, 3, most_cells - 2 * n_air + 0.99))
    h = round(rng.uniform(1.0, 2.4), 2)
    L = round(cells * h, 2)
    return _cube(L, h, round(rng.uniform(1.1, 1.3), 2), n_air, round(L * rng.uniform(1.6, 3.0) + 8.0 * h, 2))


def draw(rng):
    """One more case of the same ranges: every path, size, precision, start and kind of arrays."""
    path = rng.choice(["solve"] * 5 + ["energy"] * 2 + ["minimize"] * 3 + ["network"])
    if path == "network":
        grid = 8 * rng.randint(2, 8)
        return {"path": path, "grid": grid, "batch": rng.randint(1, 2 if grid > 48 else 4 if grid > 32 else 8)}
    precision = rng.choice(["fp64", "fp64", "fp32_precond", "mixed"])
    if path == "solve":
        return {"path": path, **_draw_mesh(rng, 112), "precision": precision, "start": rng.choice(["zero", "previous"]),
                "arrays": rng.choice(["device", "host"])}
    if path == "energy":
        return {"path": path, **_draw_mesh(rng, 112), "precision": precision}
    return {"path": path, **_draw_mesh(rng, 56), "precision": rng.choice(["fp64", "fp32_precond"]),
            "method": rng.choice(["pcohen_hs", "pcohen_hs", "pcohen", "lbfgs"]), "B_T": rng.choice([4.0, 1.0, 0.0, -2.0, -3.0])}


# ------------------------------------------------------------------------------------------------
# handles and inputs
# ------------------------------------------------------------------------------------------------
MESH_KEYS = {"cube": ("L", "h", "r", "n_air", "box"), "ellipsoid": ("a", "b", "c")}
EASY_AXIS = (math.sin(0.06), 0.0, math.cos(0.06))  # the particle's


def _mesh_key(case):
    return (case["mesh"], *(case[k] for k in MESH_KEYS[case["mesh"]]))


def _raw_mesh(key):
    """(knt, ijk, materials) of a mesh key."""
    if key[0] == "cube":
        _, L, h, r, n_air, box = key
        knt, ijk = syn.box_mesh(syn.BoxWorkload("case", L=L, h=h, r=r, n_air=n_air, box=box))
        return knt, ijk, syn.reduced_materials([syn.Material(), syn.AIR])
    mat = syn.Material(Js=1.3, A=8e-12, K1=4.3e6, axis=EASY_AXIS)
    knt, ijk = syn.ellipsoid_mesh(syn.Particle(*key[1:], mat))
    return knt, ijk, syn.reduced_materials([mat, syn.AIR])


@functools.lru_cache(maxsize=1)
def _setup(key):
    knt, ijk, (A, K1, Js, k, Js_ref) = _raw_mesh(key)
    return fem_utils.prepare(knt, ijk, A, K1, Js, k), Js_ref


@functools.lru_cache(maxsize=1)
def _handle(key, precision):
    """The mesh and its device problem with the solver, as a hysteresis loop builds them once."""
    s, Js_ref = _setup(key)
    s = dataclasses.replace(s, geom=dataclasses.replace(s.geom))  # a geometry carries its problems
    prob = problem_for_geom(s.geom, s.A_lookup, s.K1_lookup, s.Js_lookup, s.k_easy, s.V_mag, s.M_nodal, s.boundary_mask)
    make_solve_U(s.geom, s.Js_lookup, precond_type="amgcl", cg_tol=TOL, boundary_mask=s.boundary_mask,
                 precision=precision, problem=prob)
    return s, Js_ref, prob


@functools.lru_cache(maxsize=1)
def _network(grid, batch):
    return learned.UNet(grid, batch, learned.init_params(WEIGHTS_SEED))


def _magnetisation(knt, seed, step=0):
    """A state of the sweep: a tilted, slowly varying direction with a little noise, normalised; the
    next step of the same sweep differs by a few degrees."""
    rng = np.random.default_rng(seed)
    tilt, turn = rng.uniform(0.05, 1.2) + 0.05 * step, rng.uniform(0.0, 2.0 * np.pi)
    q = rng.standard_normal((2, 3))
    q *= (rng.uniform(1.0, 4.0, (2, 1)) / np.linalg.norm(q, axis=1, keepdims=True)) / max(1e-9, float(np.abs(knt).max()))
    phase = rng.uniform(0.0, 2.0 * np.pi, 2)
    noise = rng.uniform(-0.01, 0.01, knt.shape)
    th = tilt + 0.3 * np.sin(knt @ q[0] * np.pi + phase[0])
    ph = turn + 0.3 * np.sin(knt @ q[1] * np.pi + phase[1])
    m = np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)], 1) + noise
    return m / np.linalg.norm(m, axis=1, keepdims=True)


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    t.copy_(torch.from_numpy(np.ascontiguousarray(a)))
    return t.numpy()


def prepare(case, seed):
    path = case["path"]
    if path == "network":
        net = _network(case["grid"], case["batch"])
        gen = torch.Generator(device="cuda").manual_seed(seed)
        shape = (case["batch"], case["grid"] ** 3)
        x = torch.randn((*shape, 4), generator=gen, device="cuda") * 0.5
        x[..., 3] = 0.0  # the potential channel is off by default
        t = torch.randn(shape, generator=gen, device="cuda") * 0.5
        return {"path": path, "net": net, "x": x, "t": t, "y": torch.empty(shape, device="cuda")}
    key = _mesh_key(case)
    s, Js_ref, prob = _handle(key, case["precision"])
    if path == "minimize":
        minimize = make_minimizer(s.geom, s.A_lookup, s.K1_lookup, s.Js_lookup, s.k_easy, s.V_mag, s.node_volumes,
                                  s.M_nodal, make_solve_U(s.geom, s.Js_lookup, problem=prob), TOL, method=case["method"],
                                  boundary_mask=s.boundary_mask)
        m0 = torch.from_numpy(syn.initial_state(s.N, seed=seed)).cuda()
        B = case["B_T"] / Js_ref * syn.tilted_field_direction(1.0)
        return {"path": path, "minimize": minimize, "m0": m0, "B": B}
    m = _magnetisation(s.knt, seed)
    if path == "energy":
        kernels = make_energy_kernels(s.geom, s.A_lookup, s.K1_lookup, s.Js_lookup, s.k_easy, s.V_mag, s.M_nodal,
                                      boundary_mask=s.boundary_mask)
        R = float(np.abs(s.knt).max())
        U = np.prod(np.cos(0.5 * np.pi * s.knt / np.abs(s.knt).max(0)), axis=1) * (s.knt @ m.mean(0)) * (8.0 / R)
        return {"path": path, "energy_and_grad": kernels[0], "m": torch.from_numpy(m).cuda(),
                "U": torch.from_numpy(U).cuda(), "B": np.array([0.01, -0.02, -0.3])}
    if case["start"] == "previous":
        x0 = _potential(key, _magnetisation(s.knt, seed, step=-1), 1e-12)
    else:
        x0 = torch.zeros(s.N, dtype=torch.float64, device="cuda")
    if case["arrays"] == "host":
        return {"path": path, "prob": prob, "m": _pinned(m), "x0": _pinned(x0.cpu().numpy()),
                "out": _pinned(np.zeros(s.N))}
    return {"path": path, "prob": prob, "m": torch.from_numpy(m).cuda(), "x0": x0, "out": None}


def run(state):
    path = state["path"]
    if path == "solve":
        if state["out"] is not None:
            return state["prob"].solve_u(state["m"], state["x0"], TOL, out=state["out"])[0]
        U = state["x0"].clone()
        torch.cuda.current_stream().synchronize()  # the solve runs on the problem's own stream
        return state["prob"].solve_u(state["m"], U, TOL)[0]
    if path == "energy":
        E, g = state["energy_and_grad"](state["m"], state["U"], state["B"])
        return {"E": E, "g": g}
    if path == "minimize":
        m, U, info = state["minimize"](state["m0"], state["B"], tau_f=1e-8, eps_a=1e-6, pc_iters=10, pc_auto=True,
                                       pc_stagnation_nu=0.01, verbose=False)
        return {"m": m, "U": U, "E": info["E"]}
    net = state["net"]
    torch.cuda.current_stream().synchronize()  # the network runs on its own stream
    net.forward_dev(state["x"], state["y"])
    loss = net.backward_dev(state["t"])
    return {"y": state["y"], "loss": loss, "grads": net.get_grads()}


# ------------------------------------------------------------------------------------------------
# the work of a pass
# ------------------------------------------------------------------------------------------------
def _counts(case):
    """(nodes, magnetic nodes) of a mesh, from its cells."""
    if case["mesh"] == "cube":
        nc = max(1, math.ceil(case["L"] / case["h"]))
        return (nc + 2 * case["n_air"] + 1) ** 3, (nc + 1) ** 3
    h, r, box = 1.5, 1.2, 5.0 * max(case["a"], case["b"], case["c"])
    n, mag = 1, 4.0 / 3.0 * math.pi
    for k in "abc":
        nc = math.ceil(2.0 * case[k] / h)
        air = math.ceil(math.log(1.0 + 0.5 * (box - nc * h) * (r - 1.0) / (h * r)) / math.log(r))
        n *= nc + 2 * max(1, air) + 1
        mag *= case[k] / h + 0.5
    return n, int(mag)


ROW = 15  # entries of a row of a mesh operator (six tetrahedra a cell: 14 neighbours and the node)
PCG = 16  # V-cycle PCG iterations of a cold solve at TOL (12 to 18 over these meshes)
FIELD_STEP = (4, 8, 10)  # minimizer iterations, trial states with a demag solve, iterations of each solve
CHANNELS = [(0, 16, 16)] * 4 + [(1, 16, 32), (1, 32, 32), (1, 32, 32), (1, 32, 16), (2, 32, 64), (2, 64, 64),
                                (2, 64, 64), (2, 64, 32), (3, 64, 128), (3, 128, 128), (3, 128, 64)]


def work(case):
    """Inputs once, outputs once, and the operator once: an iterative path's operator could stay on
    the chip.  Flops: two a stored entry for the products that the method's iterations consist of."""
    if case["path"] == "network":
        v = case["batch"] * case["grid"] ** 3
        fwd = sum(2.0 * 27 * ci * co * v / 8 ** lvl for lvl, ci, co in CHANNELS)
        params = sum(27 * ci * co + co for _, ci, co in CHANNELS)
        return {"bytes": v * 4.0 * (4 + 1 + 1) + 2.0 * 4.0 * params, "flops": 3.0 * fwd}
    n, mag = _counts(case)
    if case["path"] == "energy":
        return {"bytes": mag * ROW * 44.0 + n * 8.0 * 7, "flops": mag * ROW * 2.0 * 7}
    poisson = n * ROW * 12.0 + n * 8.0 * 5
    products = n * ROW * 2.0 * 3  # direction, residual, smoothing; the coarse levels come on top
    if case["path"] == "solve":
        return {"bytes": poisson, "flops": PCG * products}
    its, trials, pcg = FIELD_STEP
    return {"bytes": poisson + mag * ROW * 44.0 + n * 8.0 * 7,
            "flops": trials * (pcg * products + mag * ROW * 2.0 * 7) + its * 10 * mag * ROW * 2.0 * 4}


# ------------------------------------------------------------------------------------------------
# the same values in 64 bits, by plain element loops
# ------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=1)
def _elements(key):
    knt, ijk, (A, K1, Js, k, _) = _raw_mesh(key)
    dev = torch.device("cuda")
    x = torch.from_numpy(knt).to(dev)
    conn = torch.from_numpy(ijk[:, :4].astype(np.int64)).to(dev)
    mat = torch.from_numpy(ijk[:, 4].astype(np.int64) - 1).to(dev)
    p = x[conn]
    a, b, c = p[:, 1] - p[:, 0], p[:, 2] - p[:, 0], p[:, 3] - p[:, 0]
    det = (a * torch.linalg.cross(b, c)).sum(1, keepdim=True)
    g1, g2, g3 = torch.linalg.cross(b, c) / det, torch.linalg.cross(c, a) / det, torch.linalg.cross(a, b) / det
    grad = torch.stack([-(g1 + g2 + g3), g1, g2, g3], 1)
    lim = x.abs().amax(0)
    inner = ((x.abs() < lim * (1 - 1e-12)).all(1)).double()  # the potential is held on the box faces
    tab = lambda v: torch.as_tensor(np.asarray(v, np.float64), device=dev)[mat]  # noqa: E731
    return {"n": x.shape[0], "conn": conn, "grad": grad, "V": det.abs().squeeze(1) / 6.0, "inner": inner,
            "A": tab(A), "K1": tab(K1), "Js": tab(Js), "axis": tab(k)}


def _to_nodes(el, v):
    out = torch.zeros((el["n"], *v.shape[2:]), dtype=torch.float64, device=v.device)
    return out.index_add_(0, el["conn"].reshape(-1), v.reshape(-1, *v.shape[2:]))


@functools.lru_cache(maxsize=1)
def _stiffness(key):
    el = _elements(key)
    Ke = el["V"][:, None, None] * (el["grad"] @ el["grad"].transpose(1, 2))
    free = el["inner"][el["conn"]]
    Ke = Ke * free[:, :, None] * free[:, None, :]
    rows = el["conn"][:, :, None].expand(-1, 4, 4).reshape(-1)
    cols = el["conn"][:, None, :].expand(-1, 4, 4).reshape(-1)
    at = torch.arange(el["n"], device=rows.device)
    fixed = (1.0 - el["inner"]) + 1e-12 * el["inner"]
    A = torch.sparse_coo_tensor(torch.stack([torch.cat([rows, at]), torch.cat([cols, at])]),
                                torch.cat([Ke.reshape(-1), fixed]), (el["n"], el["n"])).coalesce()
    i, j = A.indices()
    diag = torch.zeros(el["n"], dtype=torch.float64, device=i.device)
    diag[i[i == j]] = A.values()[i == j]
    return A.to_sparse_csr(), diag


def _potential(key, m, tol):
    """A U = D m by conjugate gradients with the diagonal as preconditioner."""
    el = _elements(key)
    A, diag = _stiffness(key)
    m = torch.as_tensor(m, dtype=torch.float64, device="cuda")
    msum = m[el["conn"]].sum(1)
    b = _to_nodes(el, (el["V"] * el["Js"])[:, None] * 0.25 * torch.einsum("eai,ei->ea", el["grad"], msum))
    x = torch.zeros_like(b)
    r = b.clone()
    z = r / diag
    p = z.clone()
    rz = torch.dot(r, z)
    stop = tol * float(b.norm())
    for it in range(20000):
        Ap = A @ p
        alpha = rz / torch.dot(p, Ap)
        x += alpha * p
        r -= alpha * Ap
        if it % 40 == 39 and float(r.norm()) <= stop:
            break
        z = r / diag
        new = torch.dot(r, z)
        p = z + (new / rz) * p
        rz = new
    return x


def _energy(key, m, U, B):
    el = _elements(key)
    me, Ue, grad, V = m[el["conn"]], U[el["conn"]], el["grad"], el["V"]
    exch = torch.einsum("eai,eci->eac", grad, torch.einsum("ebi,ebc->eci", grad, me)) * (2.0 * el["A"] * V)[:, None, None]
    along = torch.einsum("ebc,ec->eb", me, el["axis"])
    along = (along.sum(1, keepdim=True) + along) * (-2.0 * el["K1"] * V / 20.0)[:, None]
    demag = (2.0 * el["Js"] * V / 4.0)[:, None] * torch.einsum("ebi,eb->ei", grad, Ue)
    g = _to_nodes(el, exch + along[:, :, None] * el["axis"][:, None, :] + demag[:, None, :])
    zeeman = _to_nodes(el, (0.25 * el["Js"] * V)[:, None].expand(-1, 4))[:, None] * (-2.0 * B)
    V_mag = V[el["Js"] > 0].sum()
    return float(0.5 * (m * (g + 2.0 * zeeman)).sum() / V_mag), (g + zeeman) / V_mag


def _network_pass(case, state):
    """The network without any rounding: output channel 0, loss and gradients by autograd."""
    F = torch.nn.functional
    params = {k: torch.from_numpy(v).cuda().double().requires_grad_(True)
              for k, v in learned.init_params(WEIGHTS_SEED).items()}
    G, nb = case["grid"], case["batch"]

    def conv(name, h, relu=True):
        w = params[name + ".w"]
        w5 = w.reshape(3, 3, 3, w.shape[1], w.shape[2]).permute(4, 3, 0, 1, 2)
        h = F.conv3d(h, w5, params[name + ".b"], padding=1)
        return torch.relu(h) if relu else h

    def up(h):
        return F.interpolate(h, scale_factor=2, mode="nearest")

    h = torch.zeros((nb, 16, G, G, G), dtype=torch.float64, device="cuda")
    h[:, :4] = state["x"].double().reshape(nb, G, G, G, 4).permute(0, 4, 1, 2, 3)
    s0 = conv("e0b", conv("e0a", h))
    s1 = conv("e1b", conv("e1a", F.avg_pool3d(s0, 2)))
    s2 = conv("e2b", conv("e2a", F.avg_pool3d(s1, 2)))
    h = conv("b3c", conv("b3b", conv("b3a", F.avg_pool3d(s2, 2))))
    h = conv("d2b", conv("d2a", up(h) + s2))
    h = conv("d1b", conv("d1a", up(h) + s1))
    y = conv("d0b", conv("d0a", up(h) + s0), relu=False)[:, 0].reshape(nb, -1)
    loss = ((y - state["t"].double()) ** 2).mean()
    loss.backward()
    return {"y": y.detach(), "loss": float(loss.detach()), "grads": {k: v.grad for k, v in params.items()}}


def exact(case, seed):
    """What run returns, in 64 bits.  A field step's result is one of many states within its stopping
    test, and the path of its decisions is the method's own: no value for it."""
    if case["path"] == "minimize":
        return None
    if case["path"] == "network":
        return _network_pass(case, prepare(case, seed))
    key = _mesh_key(case)
    _handle.cache_clear()  # room for the element arrays
    m = _magnetisation(_raw_mesh(key)[0], seed)
    if case["path"] == "solve":
        U = _potential(key, m, 1e-14)
        return U.cpu().numpy() if case["arrays"] == "host" else U
    state = prepare(case, seed)
    E, g = _energy(key, state["m"], state["U"], torch.from_numpy(state["B"]).cuda())
    return {"E": E, "g": g}
