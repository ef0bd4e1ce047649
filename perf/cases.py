"""Timing cases of the MPM engine: what a simulation program has it do, through its public entry points.

A case runs a rollout from a saved state: the particle state is put back (x, v into the bound
buffers, F and C through ``set_particle_state``), a number of substeps runs, and the whole updated
state is returned.  The saved states are those of a simulation under way (a smooth velocity field,
deformed F, a C that belongs to the velocities), made from the seed.  ``exact`` is the same map in
64-bit floating point, written out with plain torch.

All scenes of the process share one stream, as a program with one simulation loop has it.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cressim-mpm_b200"))

import crmpm_b200 as cb  # noqa: E402
from crmpm_b200 import adjoint, meshes, scenes  # noqa: E402

DEVICE = "cuda:0"
_stream = None


def _sim_stream():
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream(device=DEVICE)
    return _stream


# ---------------------------------------------------------------------------------------------
# Cases


def listed():
    return [
        # The smallest scene of the benchmark, driven as a scene object drives a solver: one step()
        # per substep, 11 substeps a frame.  Launch latency decides.
        dict(name="drop_frame_4k", kind="drop", solver="mls", cells=8, ppc=8, material="neohookean", calls="step", substeps=11),
        # An ordinary body of odd size and of the other stress model.
        dict(name="drop_odd_85k", kind="drop", solver="mls", cells=23, ppc=7, material="corotational", calls="many", substeps=10),
        # The standard MPM solver (momentum and force passes) on a mid-sized body.
        dict(name="standard_64k", kind="drop", solver="standard", cells=20, ppc=8, material="neohookean", calls="many", substeps=10),
        # A tissue patch of ragged size: walls at four sides and a probe.
        dict(name="slab_ragged_173k", kind="slab", nx=37, ny=11, nz=53, ppc=8, option="", substeps=10),
        # The benchmark's tissue slab at full size.
        dict(name="slab_1600k", kind="slab", nx=100, ny=20, nz=100, ppc=8, option="", substeps=10),
        # A frame of a patch with its particles read back to pinned host memory for display.
        dict(name="slab_readback_200k", kind="slab", nx=50, ny=10, nz=50, ppc=8, option="readback", substeps=10),
        # Reproducible substeps, as regression runs use them.
        dict(name="slab_deterministic_230k", kind="slab", nx=60, ny=12, nz=40, ppc=8, option="deterministic", substeps=10),
        # PB-MPM on a small body, the solver's default iteration count.
        dict(name="pb_small_9k", kind="pb", nx=16, ny=9, nz=8, ppc=8, iterations=10, blade=False, substeps=4),
        # The benchmark's cutting workload: one step of 20 iterations with a slicer in the slab.
        dict(name="pb_cut_540k", kind="pb", nx=75, ny=12, nz=75, ppc=8, iterations=20, blade=True, substeps=1),
        # A batch of independent scenes of uneven sizes, as sampling-based planners run them.
        dict(name="batch_64_scenes", kind="batch", scenes=64, nmin=2000, nmax=64000, substeps=10),
        # Material identification: forward trajectory, loss, and the gradients by the adjoint.
        dict(name="identify_64k", kind="identify", cells=20, ppc=8, substeps=40, interval=20),
        # Signed distance grid of a triangle mesh (an instrument loaded into a scene).
        dict(name="sdf_5120_triangles", kind="sdf", subdivisions=4, radius=0.3, cell=0.005),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["drop", "drop", "slab", "slab", "slab", "pb", "pb", "batch", "identify", "sdf"])
    if kind == "drop":
        return dict(kind=kind, solver=rng.choice(["mls", "mls", "standard"]), cells=_log_int(rng, 6, 40), ppc=rng.randint(4, 9),
                    material=rng.choice(["neohookean", "corotational", "linear"]), calls=rng.choice(["step", "many"]),
                    substeps=rng.randint(1, 12))
    if kind == "slab":
        return dict(kind=kind, nx=_log_int(rng, 9, 99), ny=_log_int(rng, 4, 20), nz=_log_int(rng, 9, 99), ppc=rng.randint(5, 8),
                    option=rng.choice(["", "", "readback", "deterministic"]), substeps=rng.randint(2, 10))
    if kind == "pb":
        return dict(kind=kind, nx=_log_int(rng, 6, 74), ny=_log_int(rng, 4, 12), nz=_log_int(rng, 6, 74), ppc=rng.randint(5, 8),
                    iterations=rng.randint(4, 20), blade=rng.random() < 0.5, substeps=1)
    if kind == "batch":
        n = _log_int(rng, 2, 60)
        return dict(kind=kind, scenes=n, nmin=_log_int(rng, 1000, 4000), nmax=_log_int(rng, 8000, 60000), substeps=rng.randint(2, 10))
    if kind == "identify":
        k = rng.randint(4, 20)
        return dict(kind=kind, cells=_log_int(rng, 5, 19), ppc=rng.randint(6, 8), substeps=2 * k, interval=k)
    return dict(kind=kind, subdivisions=rng.randint(1, 4), radius=rng.uniform(0.1, 0.3), cell=rng.uniform(0.006, 0.02))


# ---------------------------------------------------------------------------------------------
# Inputs

_MATERIALS = {"neohookean": scenes.MAT_NEOHOOKEAN, "corotational": scenes.MAT_COROTATIONAL, "linear": scenes.MAT_LINEAR_ELASTIC}


def _seed(case, seed):
    return 7919 * (int(seed) + 1) + len(case["kind"])


def _scene(case, seed):
    """The scene (a list of scenes for a batch) of a case: particles jittered by the seed."""
    kind, s = case["kind"], _seed(case, seed)
    if kind == "drop":
        cell = 0.05 if case["cells"] <= 10 else 0.02  # the cube drop's and the material cube's cell sizes
        sc = scenes.cube_drop(seed=s, side=case["cells"] * cell, cell=cell, ppc=case["ppc"],
                              solver=scenes.SOLVER_STANDARD if case["solver"] == "standard" else scenes.SOLVER_MLS,
                              material=_MATERIALS[case["material"]])
        sc.pos_mass[:, 1] -= np.float32(0.5 - case["cells"] * cell / 2 - 0.5 * cell)  # half a cell above the ground
        return sc
    if kind == "slab":
        c = 0.01
        sx, sy, sz = case["nx"] * c, case["ny"] * c, case["nz"] * c
        # The grid's planes lie a fraction of a cell off the shapes' faces, and the walls have
        # friction instead of holding every node that approaches them: else rounding decides about
        # nodes that lie on a face or hardly move.
        sc = scenes.tissue_slab(seed=s, size=(sx, sy, sz), cell=c, ppc=case["ppc"],
                                bounds_min=(-sx / 2 - 0.0963, -0.1, -sz / 2 - 0.0963),
                                bounds_max=(sx / 2 + 0.1037, sy + 0.3, sz / 2 + 0.1037))
        sc.shapes.params0[:4, 1:3] = (1.0, 0.5)
        return sc
    if kind == "pb":
        c = 0.008
        sx, sy, sz = case["nx"] * c, case["ny"] * c, case["nz"] * c
        sc = scenes.pb_cutting(seed=s, size=(sx, sy, sz), cell=c, ppc=case["ppc"], iterations=case["iterations"],
                               depth=min(0.05, sy / 2), bounds_min=(-sx / 2 - 0.1, -sy - 0.0987, -sz / 2 - 0.1),
                               bounds_max=(sx / 2 + 0.1, 0.2, sz / 2 + 0.1))
        if case["blade"]:
            sc.shapes.position[1, :3] += np.float32([0.37 * c, 0.21 * c, 0.3 * c])  # off the planes of grid nodes
        else:
            sc.shapes.shape_ids = sc.shapes.shape_ids[:1].copy()
        return sc
    if kind == "batch":
        # bodies and probes by the case, the particles' places by the seed
        out = scenes.batched_scenes(seed=case["scenes"], num_scenes=case["scenes"], nmin=case["nmin"], nmax=case["nmax"])
        rng = np.random.default_rng(s)
        for sc in out:
            sc.pos_mass[:, :3] += (sc.cell_size * rng.uniform(-0.3, 0.3, size=(sc.n, 3))).astype(np.float32)
        return out
    return scenes.material_cube(seed=s, side=case["cells"] * 0.02, ppc=case["ppc"], v0=(0.0, -4.0, 0.0), drop=0.01)


# mean velocity of the saved state: bodies fall onto the ground, slabs sag
_DRIFT = {"drop": (0.1, -1.0, 0.05), "slab": (0.0, -0.3, 0.0), "pb": (0.02, -0.1, 0.01), "batch": (0.05, -0.5, 0.0)}


def _field(x, rng, amplitude, wavelength):
    """A smooth vector field of four plane waves at positions x: values [n, 3] and gradients
    [n, 3, 3] (component, axis)."""
    val = torch.zeros_like(x)
    grad = torch.zeros((x.shape[0], 3, 3), dtype=x.dtype, device=x.device)
    for _ in range(4):
        k = rng.normal(size=3)
        k = torch.tensor(2 * math.pi / wavelength * k / np.linalg.norm(k), dtype=x.dtype, device=x.device)
        a = torch.tensor(amplitude * rng.normal(size=3), dtype=x.dtype, device=x.device)
        ph = x @ k + rng.uniform(0, 2 * math.pi)
        val += torch.sin(ph)[:, None] * a
        grad += torch.cos(ph)[:, None, None] * (a[:, None] * k[None, :])
    return val, grad


def _saved_state(case, seed, pos_mass, cell):
    """x [n, 4], v [n, 4], F [n, 9], C [n, 9] (float32, column-major matrices) of a simulation under way."""
    rng = np.random.default_rng(_seed(case, seed) + 1)
    x4 = torch.from_numpy(pos_mass).to(DEVICE)
    x = x4[:, :3].double()
    n = x.shape[0]
    vel, dvel = _field(x, rng, 0.05, 20 * cell)
    _, dev = _field(x, rng, 0.05 * cell, 20 * cell)
    v4 = torch.zeros((n, 4), device=DEVICE)
    v4[:, :3] = vel + torch.tensor(_DRIFT[case["kind"]], dtype=x.dtype, device=DEVICE)
    F = torch.eye(3, device=DEVICE, dtype=x.dtype) + dev
    C = (cell * dvel).transpose(1, 2)  # C(r, c) = cell * dv_c / dx_r, the solvers' APIC matrix
    col = lambda m: m.transpose(1, 2).reshape(n, 9).float().contiguous()  # noqa: E731
    return x4, v4, col(F), col(C)


def _identify_inputs(case, seed, sc):
    """Initial velocities, targets at the captured substeps and the guess of E and nu."""
    rng = np.random.default_rng(_seed(case, seed) + 2)
    caps = [case["substeps"] // 2, case["substeps"]]
    x = torch.from_numpy(sc.pos_mass[:, :3]).to(DEVICE).double()
    v0 = torch.from_numpy(sc.vel[:, :3].copy()).to(DEVICE)
    v0 += 0.05 * _field(x, rng, 1.0, 0.4)[0].float()
    # targets of a much softer body: one that goes on falling, with some measurement error
    targets = torch.stack([x + v0.double() * (sc.dt * t) + _field(x, rng, 0.001, 0.5)[0] for t in caps]).float()
    return caps, v0, targets, 8e3 * rng.uniform(0.9, 1.1), 0.25 * rng.uniform(0.9, 1.1)


def _mesh(case, seed):
    """A closed, slightly dented sphere mesh in a box of fixed size (host arrays, as a mesh file
    gives them)."""
    P, T = meshes.icosphere(case["radius"], case["subdivisions"])
    rng = np.random.default_rng(_seed(case, seed))
    k = rng.normal(size=(3, 3)) * 4.0
    dent = 1.0 + 0.05 * np.sin(P.astype(np.float64) / case["radius"] @ k.T + rng.uniform(0, 6, size=3)).sum(1, keepdims=True)
    P = P * dent
    lo, hi = P.min(0), P.max(0)
    return (((P - lo) / (hi - lo) * 2 - 1) * case["radius"]).astype(np.float32), T


_FATTEN = 0.02


def prepare(case, seed):
    if case["kind"] == "sdf":
        P, T = _mesh(case, seed)
        return dict(case=case, points=P, triangles=T)
    sc = _scene(case, seed)
    if case["kind"] == "batch":
        ds = cb.DeviceBatch(sc, device=DEVICE, stream=_sim_stream())
        sc = ds.scene
    else:
        det = case.get("option") == "deterministic"
        ds = cb.DeviceScene(sc, device=DEVICE, stream=_sim_stream(), compute_initial=not det)
        if det:
            ds.solver.set_option(cb.OPT_DETERMINISTIC, 1)
            ds.compute_initial_data()
    st = dict(case=case, ds=ds)
    if case["kind"] == "identify":
        caps, v0, targets, E, nu = _identify_inputs(case, seed, sc)
        st["run"] = adjoint.Trajectory(ds, case["substeps"], caps, case["interval"])
        st["v0"] = v0.requires_grad_(True)
        st["targets"] = targets
        st["E"] = torch.tensor(E, dtype=torch.float32, device=DEVICE, requires_grad=True)
        st["nu"] = torch.tensor(nu, dtype=torch.float32, device=DEVICE, requires_grad=True)
    else:
        st["x0"], st["v0"], st["F0"], st["C0"] = _saved_state(case, seed, sc.pos_mass, float(sc.cell_size))
        st["F"], st["C"] = torch.empty_like(st["F0"]), torch.empty_like(st["C0"])
        if case.get("option") == "readback":
            st["host_x"] = torch.empty((sc.n, 4), dtype=torch.float32, pin_memory=True)
            st["host_v"] = torch.empty((sc.n, 4), dtype=torch.float32, pin_memory=True)
    torch.cuda.synchronize()
    return st


def run(state):
    case = state["case"]
    if case["kind"] == "sdf":
        return cb.build_sdf(state["points"], state["triangles"], case["cell"], _FATTEN, device=DEVICE).data
    if case["kind"] == "identify":
        E, nu, v0, traj = state["E"], state["nu"], state["v0"], state["run"]
        for t in (E, nu, v0):
            t.grad = None
        lam, mu = adjoint.lame(E, nu)
        pos = adjoint.trajectory(traj, lam.expand(traj.n), mu.expand(traj.n), v0)
        loss = adjoint.position_mse(pos, state["targets"])
        loss.backward()
        return dict(positions=pos.detach(), loss=loss.detach(), grad_E=E.grad, grad_nu=nu.grad, grad_v0=v0.grad)
    ds = state["ds"]
    n = ds.scene.n
    with torch.cuda.stream(ds.stream):
        ds.pos.copy_(state["x0"])
        ds.vel.copy_(state["v0"])
    ds.solver.set_particle_state(n, state["F0"].data_ptr(), state["C0"].data_ptr(), 0)
    x, v = ds.pos, ds.vel
    if case.get("calls") == "step":
        for _ in range(case["substeps"]):
            ds.solver.step()
    elif case.get("option") == "readback":
        x, v = state["host_x"], state["host_v"]
        ds.solver.advance((case["substeps"] - 0.5) * ds.scene.dt, x.data_ptr(), v.data_ptr())
    else:
        ds.solver.step_many(case["substeps"])
    ds.solver.copy_particle_state(n, state["F"].data_ptr(), state["C"].data_ptr(), 0)
    return dict(x=x, v=v, F=state["F"], C=state["C"])


# ---------------------------------------------------------------------------------------------
# Work


def _particles(case):
    if case["kind"] in ("drop", "identify"):
        return case["cells"] ** 3 * case["ppc"]
    if case["kind"] == "batch":  # the mean of the log-uniform sizes
        lo, hi = case["nmin"], max(case["nmax"], case["nmin"] + 1)
        return case["scenes"] * (hi - lo) / math.log(hi / lo)
    return case["nx"] * case["ny"] * case["nz"] * case["ppc"]


def work(case):
    """Per substep and particle: x, v, F, C read and written once, mass with x, V0 and the material
    read; per touched node 64 B.  The saved state in and out adds 136 B per particle each way."""
    if case["kind"] == "sdf":
        lo = 2 * (case["radius"] + _FATTEN) / case["cell"] + 1
        nodes, tris = lo ** 3, 20 * 4 ** case["subdivisions"]
        return {"bytes": 16 * nodes + 36 * tris, "flops": 120 * nodes * math.log2(tris)}
    n = _particles(case)
    nodes = n / case.get("ppc", 8) * 1.25
    inner = case["substeps"]
    state = 2 * 104 * n
    if case["kind"] == "pb":
        it = case["iterations"]
        # v and C change in each iteration, x and F once in the step
        return {"bytes": inner * (it * (104 * n + 64 * nodes) + 104 * n) + state, "flops": inner * it * 1400 * n}
    if case["kind"] == "identify":
        # forward, recomputed forward, reverse (reads the state and its adjoint, writes the adjoint)
        return {"bytes": inner * (2 * (200 * n + 64 * nodes) + 300 * n + 96 * nodes), "flops": inner * 4000 * n}
    return {"bytes": inner * (200 * n + 64 * nodes) + state, "flops": inner * 900 * n}


# ---------------------------------------------------------------------------------------------
# The same map in 64 bits


def _qrot(q, v):
    u, w = q[:3].expand_as(v), q[3]
    t = 2 * torch.cross(u, v, dim=-1)
    return v + w * t + torch.cross(u, t, dim=-1)


def _norm(v):
    s = (v * v).sum(-1)
    return torch.where(s > 0, torch.sqrt(torch.where(s > 0, s, torch.ones_like(s))), torch.zeros_like(s))


class _Exact:
    """MLS, standard and PB-MPM substeps of one scene in float64 (box, sphere, plane and quad
    slicer shapes, kinematic contact)."""

    def __init__(self, sc, device):
        f = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=device)  # noqa: E731
        self.sc, self.dev = sc, device
        self.n = [int(d) for d in sc.grid_dims()]
        self.gmin, self.gmax = f(sc.grid_min), f(sc.grid_max)
        self.dx = float(np.float32(sc.cell_size))
        self.inv = float(np.float32(1) / np.float32(sc.cell_size))
        self.dt, self.g = float(np.float32(sc.dt)), f(sc.gravity)
        self.m = f(sc.pos_mass[:, 3])
        self.lam, self.mu = f(sc.mat_params[:, 0]), f(sc.mat_params[:, 1])
        self.mat = int(sc.mat_type[0])
        self.pb, self.std = sc.solver_type == scenes.SOLVER_PB, sc.solver_type == scenes.SOLVER_STANDARD
        st = sc.shapes
        self.shapes = []
        for i in st.shape_ids:
            g = st.geom_idx[i]
            q = f(st.rotation[i])
            self.shapes.append(dict(type=int(st.geom_type[g]), gp=f(st.geom_params[g]), pos=f(st.position[i, :3]), q=q,
                                    qi=q * f([-1, -1, -1, 1]), par=[float(v) for v in st.params0[i]],
                                    vel=f(st.lin_vel[i, :3] * (st.shape_type[i] != scenes.SHAPE_STATIC))))
        self.blades = [s for s in self.shapes if s["type"] == scenes.GEOM_QUAD_SLICER]
        a = torch.arange(27, device=device)
        self.off = torch.stack([a // 9, (a // 3) % 3, a % 3], -1)

    def stencil(self, x):
        sp = (x - self.gmin) * self.inv
        base = torch.floor(sp.detach() - 0.5).long()
        fx = sp - base
        w1 = torch.stack([0.5 * (1.5 - fx) ** 2, 0.75 - (fx - 1) ** 2, 0.5 * (fx - 0.5) ** 2], 1)  # [n, 3 (offset), 3]
        d1 = torch.stack([fx - 1.5, 2 * (1 - fx), fx - 0.5], 1)
        o = self.off
        W = [w1[:, o[:, d], d] for d in range(3)]
        node = base[:, None, :] + o[None]
        lim = torch.tensor(self.n, device=self.dev)
        ok = ((node >= 0) & (node < lim)).all(-1)
        idx = torch.where(ok, (node[..., 2] * self.n[1] + node[..., 1]) * self.n[0] + node[..., 0], 0)
        d = (o[None] - fx[:, None, :])  # [n, 27, 3], node units
        w = torch.where(ok, W[0] * W[1] * W[2], 0.0)
        gw = None
        if self.std:
            D = [d1[:, o[:, k], k] for k in range(3)]
            gw = torch.stack([D[0] * W[1] * W[2], W[0] * D[1] * W[2], W[0] * W[1] * D[2]], -1) * ok[..., None]
        return idx, w, d, gw

    def volumes(self, x):
        idx, w, _, _ = self.stencil(x)
        mass = torch.zeros(self.n[0] * self.n[1] * self.n[2], dtype=x.dtype, device=self.dev)
        mass.index_add_(0, idx.reshape(-1), (w * self.m[:, None]).reshape(-1))
        return self.m / ((mass[idx] * w).sum(1) / self.dx ** 3)

    def cut(self, x, d):
        """Cut bits [n, 27] of the slicers and the side normals of the cut nodes."""
        cut, nrm = None, None
        for s in self.blades:
            side = lambda p: _qrot(s["qi"], p - s["pos"])  # noqa: E731
            r1, r2 = side(x)[:, None, :], side((x[:, None, :] + d * self.dx).reshape(-1, 3)).reshape(d.shape)
            on = lambda r: (r[..., 0].abs() <= s["gp"][0]) & (r[..., 2].abs() <= s["gp"][1])  # noqa: E731
            c = on(r1) & on(r2) & (torch.signbit(r1[..., 1]) != torch.signbit(r2[..., 1]))
            g = torch.zeros_like(d)
            g[..., 1] = torch.where(torch.signbit(r2[..., 1]), -1.0, 1.0)
            cut, nrm = (c, g) if cut is None else (cut | c, torch.where(cut[..., None], nrm, g))
        return cut, nrm

    def distance(self, s, p):
        """Distance and unit normal of shape s at points p."""
        lp = _qrot(s["qi"], p - s["pos"])
        gp = s["gp"]
        if s["type"] == scenes.GEOM_PLANE:
            g = torch.zeros_like(lp)
            g[:, 1] = 1
            dist = lp[:, 1]
        elif s["type"] == scenes.GEOM_SPHERE:
            r = _norm(lp)
            g, dist = lp / r.clamp_min(1e-30)[:, None], r - gp[0]
        elif s["type"] == scenes.GEOM_BOX:
            pen = lp.abs() - gp[:3]
            q = pen.clamp_min(0)
            l, top = _norm(q), pen.max(1)
            inner = torch.nn.functional.one_hot(top.indices, 3).to(lp.dtype)
            g = torch.where(lp < 0, -1.0, 1.0) * torch.where(top.values[:, None] > 0, q / l.clamp_min(1e-30)[:, None], inner)
            dist = l + top.values.clamp_max(0)
        else:  # quad slicer
            g = torch.zeros_like(lp)
            g[:, 1] = torch.where(torch.signbit(lp[:, 1]), -1.0, 1.0)
            on = (lp[:, 0].abs() <= gp[0]) & (lp[:, 2].abs() <= gp[1])
            dist = torch.where(on, lp[:, 1].abs(), torch.full_like(lp[:, 1], 1e30))
        return dist - s["par"][3], _qrot(s["q"], g)

    def grid(self, mom, mass, force):
        """Node velocities after division, contact and the boundary band."""
        live = mass >= (1e-8 if self.pb else 1e-4)
        if force is not None:
            mom = mom + force * (self.dt * live)[:, None]
        idx = torch.nonzero(live.detach())[:, 0]
        m, v = mass[idx], mom[idx] / mass[idx][:, None]
        ijk = torch.stack([idx % self.n[0], (idx // self.n[0]) % self.n[1], idx // (self.n[0] * self.n[1])], -1)
        pos = ijk * self.dx + self.gmin + v * self.dt
        for s in self.shapes:
            dist, nrm = self.distance(s, pos)
            rel = v - s["vel"]
            vn = (rel * nrm).sum(-1)
            tang = rel - nrm * vn[:, None]
            fc = (s["par"][2] * vn / (_norm(tang) + 1.1920928955078125e-07)).clamp_min(-1.0)
            hit = (dist < s["par"][0]) & (vn < 0)
            v = torch.where(hit[:, None], (tang + tang * fc[:, None]) * s["par"][1] + s["vel"], v)
        band = torch.stack([(ijk[:, d] < 2) | (ijk[:, d] > self.n[d] - 3) for d in range(3)], -1)
        v = torch.where(band, torch.zeros_like(v), v)
        return mom.index_copy(0, idx, v)

    def stress(self, F):
        I = torch.eye(3, dtype=F.dtype, device=self.dev)
        if self.mat == scenes.MAT_NEOHOOKEAN:
            J = torch.linalg.det(F).clamp_min(1e-6)
            return self.mu[:, None, None] * (F @ F.transpose(1, 2) - I) + (self.lam * torch.log(J))[:, None, None] * I
        E = 0.5 * (F.transpose(1, 2) @ F - I)
        tr = E.diagonal(dim1=1, dim2=2).sum(-1)
        return F @ (2 * self.mu[:, None, None] * E + (self.lam * tr)[:, None, None] * I) @ F.transpose(1, 2)

    def constrained(self, F, C):
        """PB-MPM's material constraint: C moved toward the target's.  The polar factor and F^-1 both
        come transposed, as the solver defines them."""
        I = torch.eye(3, dtype=F.dtype, device=self.dev)
        t = (I + C * self.dt) @ F
        R = t
        for _ in range(12):  # Newton's iteration for the polar factor
            R = 0.5 * (R + torch.linalg.inv(R).transpose(1, 2))
        det = torch.linalg.det(t)
        q = 1 / (torch.sign(det) * torch.sqrt(det.abs().clamp(0.1, 1000.0)))
        tgt = R.transpose(1, 2) * self.mu[:, None, None] + t * (q * (1 - self.mu))[:, None, None]
        return C + (tgt @ torch.linalg.inv(F).transpose(1, 2) - I - C * self.dt) * self.lam[:, None, None]

    def transfer(self, st, v, m, A, F, V0, cut, nrm):
        """P2G, grid update and G2P's sums: v' and the velocity moment matrix."""
        idx, w, d, gw = st
        nodes = self.n[0] * self.n[1] * self.n[2]
        wp = w if cut is None else torch.where(cut, 0.0, w)
        kick = v if (self.pb or self.std) else v + self.g * self.dt
        mom = (kick * m[:, None])[:, None, :].expand(-1, 27, -1)
        if A is not None:
            mom = mom + torch.einsum("pij,pnj->pni", A, d * self.dx)
        mom = mom * wp[..., None]
        flat = idx.reshape(-1)
        z = torch.zeros((nodes, 3), dtype=v.dtype, device=self.dev)
        P = z.index_add(0, flat, mom.reshape(-1, 3))
        M = z[:, 0].index_add(0, flat, (wp * m[:, None]).reshape(-1))
        force = None
        if self.std:
            a = -V0[:, None, None] * self.stress(F)
            fn = torch.einsum("pij,pnj->pni", a, gw) + self.g * (w * m[:, None])[..., None]
            force = z.index_add(0, flat, fn.reshape(-1, 3))
        nv = self.grid(P, M, force)[idx]
        if cut is not None:
            nv = torch.where(cut[..., None], kick[:, None, :] - nrm * (2 * (kick[:, None, :] * nrm).sum(-1, keepdim=True)), nv)
        va = (nv * w[..., None]).sum(1)
        T = torch.einsum("pni,pnj->pij", nv, gw) if self.std else 4 * torch.einsum("pni,pnj->pij", d * w[..., None], nv)
        return va, T

    def advect(self, x, v):
        x = torch.maximum(torch.minimum(x + v * self.dt, self.gmax), self.gmin)
        for s in self.shapes:
            dist, nrm = self.distance(s, x)
            x = x - nrm * torch.where(dist < 0, dist, torch.zeros_like(dist))[:, None]
        return x

    def step(self, x, v, F, C, V0):
        st = self.stencil(x)
        cut, nrm = self.cut(x, st[2]) if self.blades else (None, None)
        I = torch.eye(3, dtype=x.dtype, device=self.dev)
        m = self.m
        if self.pb:
            for _ in range(self.sc.iterations):
                C = self.constrained(F, C)
                v, C = self.transfer(st, v, m, C * m[:, None, None], F, V0, cut, nrm)
            x = self.advect(x, v)
            v = v + self.g * self.dt
        else:
            A = None if self.std else self.stress(F) * (-self.dt * 4 * self.inv ** 2 * V0)[:, None, None] + C * m[:, None, None]
            v, T = self.transfer(st, v, m, A, F, V0, cut, nrm)
            x = self.advect(x, v)
            if self.std:
                return x, v, (I + T * self.dt) @ F, C
            C = T
        return x, v, (I + C * self.dt) @ F, C


def _exact_scene(case, sc, state, device):
    ex = _Exact(sc, device)
    x4, v4, F, C = state
    n = x4.shape[0]
    mat = lambda a: a.double().reshape(n, 3, 3).transpose(1, 2)  # noqa: E731
    x, v, F, C = x4[:, :3].double(), v4[:, :3].double(), mat(F), mat(C)
    V0 = ex.volumes(torch.as_tensor(sc.pos_mass[:, :3], device=device).double())
    for _ in range(case["substeps"]):
        x, v, F, C = ex.step(x, v, F, C, V0)
    col = lambda a: a.transpose(1, 2).reshape(n, 9)  # noqa: E731
    return dict(x=torch.cat([x, x4[:, 3:].double()], 1), v=torch.cat([v, torch.zeros_like(v[:, :1])], 1), F=col(F), C=col(C))


def _exact_identify(case, seed):
    sc = _scene(case, seed)
    caps, v0, targets, E, nu = _identify_inputs(case, seed, sc)
    ex = _Exact(sc, DEVICE)
    E = torch.tensor(float(np.float32(E)), dtype=torch.float64, device=DEVICE, requires_grad=True)
    nu = torch.tensor(float(np.float32(nu)), dtype=torch.float64, device=DEVICE, requires_grad=True)
    v0 = v0.double().requires_grad_(True)
    n = v0.shape[0]
    lam, mu = E * nu / ((1.0 + nu) * (1.0 - 2.0 * nu)), E / (2.0 * (1.0 + nu))
    ex.lam, ex.mu = lam.expand(n), mu.expand(n)
    x = torch.as_tensor(sc.pos_mass[:, :3], device=DEVICE).double()
    V0 = ex.volumes(x)
    F = torch.eye(3, dtype=x.dtype, device=DEVICE).expand(n, 3, 3)
    C, v, out = torch.zeros_like(F), v0, []
    for t in range(1, case["substeps"] + 1):
        x, v, F, C = ex.step(x, v, F, C, V0)
        if t in caps:
            out.append(x)
    pos = torch.stack(out)
    loss = ((pos - targets.double()) ** 2).mean(dim=(1, 2)).sum()
    loss.backward()
    return dict(positions=pos.detach(), loss=loss.detach(), grad_E=E.grad, grad_nu=nu.grad, grad_v0=v0.grad)


def _exact_sdf(case, seed):
    """Distances by testing every triangle, signs by the winding number, gradients by differences."""
    P32, T = _mesh(case, seed)
    cell = np.float32(case["cell"])
    one = np.float32(1e-4)
    lower = (np.minimum(P32.min(0), np.float32(0)) - one) - np.float32(_FATTEN)
    upper = (np.maximum(P32.max(0), np.float32(0)) + one) + np.float32(_FATTEN)
    nx, ny, nz = (int(v) for v in ((upper - lower) / cell + np.float32(1.0)))
    P = torch.as_tensor(P32, device=DEVICE).double()
    a, b, c = (P[torch.as_tensor(T[:, k].astype(np.int64), device=DEVICE)] for k in range(3))
    nrm = torch.cross(b - a, c - a, dim=1)
    n2 = (nrm * nrm).sum(1)
    ax = [torch.arange(n, device=DEVICE, dtype=torch.float64) * float(cell) + float(lower[d]) for d, n in enumerate((nx, ny, nz))]
    z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    q = torch.stack([x, y, z], -1).reshape(-1, 3)
    dist = torch.empty(q.shape[0], dtype=torch.float64, device=DEVICE)
    dot = lambda u, v: (u * v).sum(-1)  # noqa: E731
    step = max(1, (1 << 24) // T.shape[0])
    for i in range(0, q.shape[0], step):
        p = q[i:i + step, None, :]
        inside, best, corner = None, None, [a - p, b - p, c - p]
        h = dot(corner[0], nrm)
        for u, v, s in ((a, b, 0), (b, c, 1), (c, a, 2)):
            e, w = v - u, -corner[s]
            t = (dot(w, e) / dot(e, e)).clamp(0, 1)
            r = w - t[..., None] * e
            d2 = dot(r, r)
            best = d2 if best is None else torch.minimum(best, d2)
            side = dot(w, torch.cross(nrm, e, dim=1)) >= 0
            inside = side if inside is None else inside & side
        best = torch.where(inside, h * h / n2, best).min(1).values
        la, lb, lc = (torch.sqrt(dot(v, v)) for v in corner)
        den = la * lb * lc + dot(corner[0], corner[1]) * lc + dot(corner[1], corner[2]) * la + dot(corner[2], corner[0]) * lb
        # corner triple product: a . (b x c) of the corners equals h
        wind = torch.atan2(h, den).sum(1) / (2 * math.pi)
        dist[i:i + step] = torch.where(wind > 0.5, -1.0, 1.0) * torch.sqrt(best)
    w = dist.reshape(nz, ny, nx)
    g = torch.stack(list(reversed(torch.gradient(w, spacing=float(cell)))), -1)
    s = (g * g).sum(-1, keepdim=True)
    g = torch.where(s > 0, g / torch.sqrt(torch.where(s > 0, s, torch.ones_like(s))), g)
    return torch.cat([g, w[..., None]], -1)


def exact(case, seed):
    if case["kind"] == "sdf":
        return _exact_sdf(case, seed)
    if case["kind"] == "identify":
        return _exact_identify(case, seed)
    sc = _scene(case, seed)
    if case["kind"] != "batch":
        return _exact_scene(case, sc, _saved_state(case, seed, sc.pos_mass, float(sc.cell_size)), DEVICE)
    merged = scenes.make_batch(sc)
    state = _saved_state(case, seed, merged.merged.pos_mass, float(merged.merged.cell_size))
    parts = [_exact_scene(case, one, [t[merged.slice(i)] for t in state], DEVICE) for i, one in enumerate(sc)]
    return {k: torch.cat([p[k] for p in parts]) for k in parts[0]}
