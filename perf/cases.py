"""What the reconstruction library is measured on: complete passes through its public entry points.

A case is one call as a user's program makes it: a cloud in, a mesh out, through the Python binding or
the C ABI; several clouds in one call; a sparse system given as CSR; a training run of the learned
preconditioner.  Every size stands for clouds the library is used on, from a few thousand points (a
preview, where launches and host round trips count) to 30 million (a large scan).
"""
from __future__ import annotations

import ctypes
import math
import os

import numpy as np
import torch

import poissonrecon_gpu_gb300 as pg
from poissonrecon_gpu_gb300 import shapes

CHECKPOINT = os.path.join(os.path.dirname(os.path.abspath(pg.__file__)), "weights", "lpc_ellipsoids_d9.bin")
REFERENCE, RELATIVE = "reference", "relative"     # CG stopping rules (absolute 1e-5, relative 1e-6)
OPTIONS = ("weld", "density_weights", "cascadic", "learned", "refine", "stable_basis")


def _cloud(name, shape, n, depth, api, solve, *options):
    case = {"name": name, "kind": "cloud", "shape": shape, "n": n, "depth": depth, "api": api, "solve": solve}
    case.update({o: o in options for o in OPTIONS})
    return case


def listed():
    return [
        # a preview of a small object in an interactive tool: the smallest call, all latency
        _cloud("sphere_5k_d6", "sphere", 5_000, 6, "python", REFERENCE),
        # the reference program's own configuration (maxDepth 8, its CG schedule), called from C
        _cloud("sphere_50k_d8", "sphere", 50_000, 8, "c_host", REFERENCE),
        # a scan of a few objects solved with the learned preconditioner and the FP64 residual check
        _cloud("ellipsoids_61k_d9_learned", "ellipsoids", 61_007, 9, "python", RELATIVE, "learned", "refine"),
        # a cloud that is sparse for its octree: most of the surface lies in coarse leaves
        _cloud("superquadric_100k_d10", "superquadric", 100_003, 10, "python", RELATIVE),
        # an unevenly sampled scan with every quality option: density weights, coarse-to-fine solve,
        # closed-form basis, one vertex per edge
        _cloud("torus_200k_d9_options", "torus", 200_001, 9, "python", RELATIVE, "weld", "density_weights",
               "cascadic", "stable_basis"),
        # the ordinary scan (the benchmark's workload): host buffers in, host mesh out
        _cloud("torus_1m_d10", "torus", 1_000_000, 10, "c_host", RELATIVE),
        # a dense scan with fine surface detail, already on the GPU (another stage produced it)
        _cloud("displaced_4m_d11", "displaced_sphere", 4_194_301, 11, "c_device", RELATIVE),
        # the largest: a 30M-point scan at maxDepth 12
        _cloud("displaced_30m_d12", "displaced_sphere", 30_000_000, 12, "c_device", RELATIVE),
        # a data set of uneven objects in one call (points per cloud spread over two decades)
        {"name": "batch_16_superquadrics", "kind": "batch", "clouds": 16, "n_min": 5_000, "n_max": 500_000,
         "depth_min": 7, "depth_max": 10},
        # a caller's own symmetric system through the CSR solver: the 27-point stencil on a box
        {"name": "csr_915k_rows", "kind": "csr", "nx": 97, "ny": 85, "nz": 111},
        # fine-tuning the preconditioner on recorded solves: a resume from the shipped checkpoint
        {"name": "train_40_steps", "kind": "train", "shapes": 3, "points": 40_009, "depth": 8, "rows": 512,
         "batch": 16_384, "steps": 40},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["cloud", "batch", "csr", "train"], [7, 1, 1, 1])[0]
    if kind == "batch":
        hi = _logint(rng, 20_000, 500_000)
        return {"kind": "batch", "clouds": rng.randint(2, 24), "n_min": 5_000, "n_max": hi, "depth_min": 7,
                "depth_max": rng.randint(8, 10)}
    if kind == "csr":
        return {"kind": "csr", "nx": _logint(rng, 9, 120), "ny": _logint(rng, 9, 120), "nz": _logint(rng, 9, 120)}
    if kind == "train":
        return {"kind": "train", "shapes": rng.randint(1, 3), "points": _logint(rng, 20_000, 100_000),
                "depth": rng.randint(7, 9), "rows": _logint(rng, 64, 768), "batch": _logint(rng, 1_000, 20_000),
                "steps": rng.randint(10, 60)}
    n = _logint(rng, 1_000, 20_000_000)
    shape = "displaced_sphere" if n > 1_000_000 else rng.choice(["sphere", "torus", "ellipsoids", "superquadric"])
    # the tree's finest cells hold between one point in a few and a few points each
    depth = min(12, max(5, round(0.5 * math.log2(n) + rng.uniform(-1.0, 1.6))))
    options = []
    solve = rng.choice([REFERENCE, RELATIVE])
    for o, p in (("weld", 0.25), ("density_weights", 0.2), ("stable_basis", 0.25)):
        if rng.random() < p:
            options.append(o)
    if solve == RELATIVE and n <= 2_000_000 and rng.random() < 0.4:
        options += rng.choice([["cascadic"], ["learned", "refine"], ["refine"]])
    apis = ["python", "c_host", "c_device"] if n <= 1_000_000 else ["c_host", "c_device"]
    case = _cloud("", shape, n, depth, rng.choice(apis), solve, *options)
    del case["name"]
    return case


class _MeshBuffers:
    """The caller's own mesh, in arrays it keeps from call to call: the library's arrays are valid until
    the next call only.  'area' bounds the triangles in units of 4^depth; what a mesh leaves free is 0."""

    def __init__(self, depth, area):
        cap = 1024 + int(area * 4 ** depth)
        self.vertices = torch.zeros((cap, 3), dtype=torch.float32)
        self.triangles = torch.zeros((cap, 3), dtype=torch.int32)

    def take(self, vertices, triangles):
        self.vertices[:len(vertices)].copy_(torch.from_numpy(vertices))
        self.triangles[:len(triangles)].copy_(torch.from_numpy(triangles))
        return {"n_vertices": len(vertices), "n_triangles": len(triangles), "vertices": self.vertices,
                "triangles": self.triangles}


class _Context:
    """A reconstruction context held by a caller of the C ABI."""

    def __init__(self, case):
        self.lib = ctypes.CDLL(pg.LIB_PATH)
        for name, (res, args) in pg.SIGNATURES.items():
            f = getattr(self.lib, name)
            f.restype, f.argtypes = res, args
        p = pg.Params()
        self.call("prgpu_params_default", ctypes.byref(p))
        p.depth = case["depth"]
        if case["solve"] == RELATIVE:
            p.solve_mode, p.cg_tol = pg.SOLVE_RELATIVE, 1e-6
        for o in OPTIONS:
            setattr(p, o, int(case[o]))
        self.ctx = ctypes.c_void_p()
        self.call("prgpu_create", ctypes.byref(p), ctypes.byref(self.ctx))
        if case["learned"]:
            self.call("prgpu_load_preconditioner", self.ctx, CHECKPOINT.encode())
        self.mesh = pg.Mesh()

    def call(self, name, *args):
        rc = getattr(self.lib, name)(*args)
        if rc not in (0, 5):                      # 5: the solver's iteration cap, results written
            raise RuntimeError("%s: %d %s" % (name, rc, self.lib.prgpu_last_error().decode()))

    def mesh_arrays(self):
        """The library's own mesh arrays: valid until the next call on this context."""
        m = self.mesh
        if not m.n_triangles:
            return np.zeros((0, 3), np.float32), np.zeros((0, 3), np.int32)
        return (np.ctypeslib.as_array(m.vertices, (m.n_vertices, 3)),
                np.ctypeslib.as_array(m.triangles, (m.n_triangles, 3)))

    def __del__(self):
        if getattr(self, "ctx", None) and self.ctx.value:
            self.lib.prgpu_destroy(self.ctx)
            self.ctx = ctypes.c_void_p()


# room kept for a mesh, in triangles per 4^depth
ROOM = {"sphere": 9.0, "displaced_sphere": 8.0, "torus": 7.0, "ellipsoids": 9.0, "superquadric": 9.0}


def _points(shape, n, seed):
    if shape == "sphere":
        return shapes.sphere(n, seed=seed)
    if shape == "torus":
        return shapes.torus(n, seed=seed)
    if shape == "ellipsoids":
        return shapes.ellipsoid_union(seed, n_min=n, n_max=n)
    if shape == "superquadric":
        return shapes.superquadric(seed, n_min=n, n_max=n)
    return shapes.displaced_sphere(n, seed=seed, device="cuda")


def _line():
    """1-D stencils (neighbour, centre) of stiffness and mass, whose products form the matrix:
    small integers, so the float32 matrix is exact."""
    return (-1.0, 2.0), (1.0, 4.0)


def _csr_rhs(case, seed):
    """A right-hand side that lives near a surface, as the divergence of a sampled normal field does."""
    rng = np.random.default_rng(seed)
    shape = (case["nx"], case["ny"], case["nz"])
    g = np.meshgrid(*[(np.arange(m) + 0.5) / m - 0.5 for m in shape], indexing="ij")
    rad = np.sqrt(g[0] ** 2 + g[1] ** 2 + g[2] ** 2)
    b = np.where(np.abs(rad - 0.35) < 1.5 / min(shape), rng.standard_normal(shape), 0.0)
    return (100.0 * b).astype(np.float32)


def _csr_matrix(case):
    """The 27-point stencil K*M*M + M*K*M + M*M*K on the box, as CSR in device memory."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    (k1, k0), (m1, m0) = _line()
    row = torch.arange(nx * ny * nz, device="cuda")
    ix, iy, iz = row // (ny * nz), (row // nz) % ny, row % nz
    cols, vals, oks = [], [], []
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                k = [k0 if d == 0 else k1 for d in (dx, dy, dz)]
                m = [m0 if d == 0 else m1 for d in (dx, dy, dz)]
                v = k[0] * m[1] * m[2] + m[0] * k[1] * m[2] + m[0] * m[1] * k[2]
                ok = ((ix + dx >= 0) & (ix + dx < nx) & (iy + dy >= 0) & (iy + dy < ny)
                      & (iz + dz >= 0) & (iz + dz < nz))
                cols.append(row + (dx * ny + dy) * nz + dz)
                vals.append(torch.full((len(row),), v, dtype=torch.float32, device="cuda"))
                oks.append(ok)
    ok = torch.stack(oks, 1)
    ptr = torch.zeros(len(row) + 1, dtype=torch.int32, device="cuda")
    ptr[1:] = torch.cumsum(ok.sum(1), 0).to(torch.int32)
    return ptr, torch.stack(cols, 1)[ok].to(torch.int32).contiguous(), torch.stack(vals, 1)[ok].contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        # the sizes follow a golden-ratio sequence over their logarithm, the depths take turns
        lo, hi, span = math.log(case["n_min"]), math.log(case["n_max"]), case["depth_max"] - case["depth_min"] + 1
        ns = [int(math.exp(lo + (hi - lo) * ((k + 1) * 0.6180339887 % 1.0))) for k in range(case["clouds"])]
        clouds = [_points("superquadric", n, seed * 1000 + k) for k, n in enumerate(ns)]
        depths = [case["depth_min"] + k % span for k in range(case["clouds"])]
        return {"case": case, "rec": pg.Reconstructor(depth=8, solve_mode=pg.SOLVE_RELATIVE, cg_tol=1e-6),
                "clouds": clouds, "depths": depths, "out": [_MeshBuffers(d, ROOM["superquadric"]) for d in depths]}
    if kind == "csr":
        b = torch.from_numpy(_csr_rhs(case, seed)).cuda().flatten()
        ptr, col, val = _csr_matrix(case)
        x = torch.zeros_like(b)
        torch.cuda.synchronize()
        return {"case": case, "ptr": ptr, "col": col, "val": val, "b": b, "x": x}
    if kind == "train":
        trainer = pg.Trainer(seed=seed)
        rec = pg.Reconstructor(depth=case["depth"], solve_mode=pg.SOLVE_RELATIVE, cg_tol=1e-6)
        for k in range(case["shapes"]):
            rec.set_points(*_points("ellipsoids", case["points"], seed * 1000 + k))
            rec.build_octree()
            rec.compute_rhs()
            trainer.record(rec, rows_per_depth=case["rows"])
        rec.close()
        return {"case": case, "trainer": trainer}
    xyz, nrm = _points(case["shape"], case["n"], seed)
    state = {"case": case, "n": len(xyz), "out": _MeshBuffers(case["depth"], ROOM[case["shape"]])}
    if case["api"] == "python":
        state["xyz"], state["nrm"] = xyz, nrm
        state["rec"] = pg.Reconstructor(
            depth=case["depth"], solve_mode=pg.SOLVE_RELATIVE if case["solve"] == RELATIVE else pg.SOLVE_REFERENCE,
            cg_tol=1e-6 if case["solve"] == RELATIVE else 1e-5, weld=case["weld"],
            density_weights=case["density_weights"], cascadic=case["cascadic"], refine=case["refine"],
            stable_basis=case["stable_basis"], preconditioner=CHECKPOINT if case["learned"] else None)
        return state
    state["ctx"] = _Context(case)
    xyz, nrm = torch.from_numpy(xyz), torch.from_numpy(nrm)
    if case["api"] == "c_host":                   # page-locked, as a streaming reader keeps them
        state["xyz"], state["nrm"] = xyz.pin_memory(), nrm.pin_memory()
    else:
        state["xyz"], state["nrm"] = xyz.cuda(), nrm.cuda()
        torch.cuda.synchronize()
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        meshes = state["rec"].reconstruct_batch(state["clouds"], state["depths"])
        return [out.take(v, f) for out, (v, f) in zip(state["out"], meshes)]
    if kind == "csr":
        n, nnz = state["b"].numel(), state["val"].numel()
        pg.solverCG_DeviceToDevice(n, nnz, state["ptr"].data_ptr(), state["col"].data_ptr(), state["val"].data_ptr(),
                                   state["b"].data_ptr(), state["x"].data_ptr())
        return {"x": state["x"]}
    if kind == "train":
        t = state["trainer"]
        t.load(CHECKPOINT)
        loss = t.train(case["steps"], batch=case["batch"], lr=1e-4)
        return {"params": t.params(), "loss": loss}
    if case["api"] == "python":
        return state["out"].take(*state["rec"].reconstruct(state["xyz"], state["nrm"]))
    c = state["ctx"]
    px, pn, n = state["xyz"].data_ptr(), state["nrm"].data_ptr(), state["n"]
    if case["api"] == "c_host":
        c.call("prgpu_reconstruct", c.ctx, px, pn, n, ctypes.byref(c.mesh))
        return state["out"].take(*c.mesh_arrays())
    iso = ctypes.c_float(0)
    c.call("prgpu_set_points_device", c.ctx, px, pn, n)
    c.call("prgpu_build_octree", c.ctx)
    c.call("prgpu_compute_rhs", c.ctx)
    c.call("prgpu_solve", c.ctx)
    c.call("prgpu_eval_points", c.ctx, ctypes.byref(iso))
    c.call("prgpu_extract_mesh", c.ctx)
    c.call("prgpu_get_mesh", c.ctx, ctypes.byref(c.mesh))
    return dict(state["out"].take(*c.mesh_arrays()), iso=iso.value)


def _cloud_work(n, depth, area):
    """Points in, mesh out; the splat's and the evaluation's products at the points.  A surface of
    'area' (in units of the cube's face) has about 'area' * 4^depth triangles and two thirds as many
    vertices, 12 bytes each."""
    triangles = area * 4.0 ** depth
    return {"bytes": 24.0 * n + 20.0 * triangles, "flops": n * (27.0 * 8 + 27.0 * 4 * (depth + 1))}


AREA = {"sphere": 6.1, "displaced_sphere": 6.1, "torus": 2.9, "ellipsoids": 4.0, "superquadric": 3.0}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        n = (case["n_max"] - case["n_min"]) / math.log(case["n_max"] / case["n_min"])
        per = [_cloud_work(n, d, AREA["superquadric"]) for d in range(case["depth_min"], case["depth_max"] + 1)]
        return {k: case["clouds"] * sum(p[k] for p in per) / len(per) for k in ("bytes", "flops")}
    if kind == "csr":
        n = case["nx"] * case["ny"] * case["nz"]
        iters = 1.5 * max(case["nx"], case["ny"], case["nz"])
        return {"bytes": n * (27.0 * 8 + 4 + 8), "flops": iters * n * (2.0 * 27 + 10)}
    if kind == "train":
        # forward, weight gradients and error propagation of the two 64 x 64 layers
        rows = float(case["steps"] * case["batch"])
        return {"bytes": rows * 132.0, "flops": rows * 2.0 * 64 * 64 * 5}
    return _cloud_work(case["n"], case["depth"], AREA[case["shape"]])


def exact(case, seed):
    """The CSR system's solution in 64 bits: the matrix is a sum of products of 1-D stencils, which
    the sine vectors diagonalise.  A mesh and trained weights have no such value."""
    if case["kind"] != "csr":
        return None
    (k1, k0), (m1, m0) = _line()
    x = _csr_rhs(case, seed).astype(np.float64)
    basis, lk, lm = [], [], []
    for m in x.shape:
        j = np.arange(1, m + 1)
        basis.append(np.sqrt(2.0 / (m + 1)) * np.sin(np.pi * np.outer(j, j) / (m + 1)))
        lk.append(k0 + 2 * k1 * np.cos(np.pi * j / (m + 1)))
        lm.append(m0 + 2 * m1 * np.cos(np.pi * j / (m + 1)))

    def transform(a):
        for s in basis:                           # each axis in turn; the axes rotate back into place
            a = np.tensordot(a, s, axes=(0, 0))
        return a

    lam = (lk[0][:, None, None] * lm[1][None, :, None] * lm[2][None, None, :]
           + lm[0][:, None, None] * lk[1][None, :, None] * lm[2][None, None, :]
           + lm[0][:, None, None] * lm[1][None, :, None] * lk[2][None, None, :])
    return {"x": transform(transform(x) / lam).ravel()}
