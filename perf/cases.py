"""Performance cases of the matrix-free multigrid path: the work a user's program has it do.

Every case is one pass through the public classes of hyteg_b200 on the unit box split into
nx x ny x nz sub-cubes of six tetrahedra (PrimitiveStorage.cuboid), each refined `level` times:

  vcycle          one V(3,3) cycle from a zero start (the preconditioner of an outer iteration)
  solve           twelve FP32 cycles in FP64 defect correction, one coefficient per macro-cell
  cg              ten CG iterations from a zero start (the Krylov path: apply, dots, updates)
  apply, residual the P1 operator; form 0 is the Laplace, form 1 the mass operator
  sor             one forward and one backward sweep (the symmetric smoother)
  transfers       restriction of a residual, prolongation and add of a correction
  p2_apply        the P2 operator; `level` is the P2 level (its lattice has level + 1)
  p2_sor          one forward and one backward P2 sweep
  p2_vcycle       one P2 V(3,3) cycle from a zero start
  stokes_apply    the Taylor-Hood block operator
  stokes_minres   twenty preconditioned MINRES iterations from a zero start

Vectors are uniform in [-1, 1), the right-hand sides of the benchmark and of the solve server.
Outputs are the level buffers of the result; where an operation leaves the copies of a DoF at
other macro-primitives undefined, the pass ends with the halo exchange a reader would call.
"""
import functools
import math

import torch

import hyteg_b200 as hg

F64, F32 = "f64", "f32"
DTYPE = {F64: "float64", F32: "float32"}
NEVER = 1e-300  # a tolerance that no residual meets: the number of iterations is fixed


def _case(kind, n, level, dtype=F64, **more):
    return dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], level=level, dtype=dtype, **more)


def listed():
    return [
        # the benchmark's step: the 48-tetrahedron cube at level 8, smoother schedules tuned once
        dict(_case("vcycle", (2, 2, 2), 8, tuned=True), name="vcycle_f64_l8"),
        # the cycle inside mixed-precision defect correction, library defaults
        dict(_case("vcycle", (2, 2, 2), 7, F32, tuned=False), name="vcycle_f32_l7"),
        # the smallest request of the solve server: one sub-cube, launches and latency count
        dict(_case("vcycle", (1, 1, 1), 4, tuned=False), name="vcycle_f64_1cube_l4"),
        # a variable-coefficient solve as the server runs it, 3^3 sub-cubes
        dict(_case("solve", (3, 3, 3), 5), name="solve_mixed_27cubes_l5"),
        # Krylov iterations without multigrid
        dict(_case("cg", (2, 2, 2), 6), name="cg_f64_l6"),
        # operator evaluations of the largest size (matrix-free apply inside any outer method)
        dict(_case("apply", (2, 2, 2), 8, form=0), name="apply_f64_l8"),
        # the smoother by itself, forward and backward, library defaults
        dict(_case("sor", (2, 2, 2), 7), name="sor_f64_l7"),
        # the grid transfers of the largest cycle
        dict(_case("transfers", (2, 2, 2), 8), name="transfers_f64_l8"),
        # quadratic elements: operator, cycle
        dict(_case("p2_apply", (2, 2, 2), 6), name="p2_apply_f64_l6"),
        dict(_case("p2_vcycle", (2, 2, 2), 5), name="p2_vcycle_f64_l5"),
        # Taylor-Hood Stokes: operator, preconditioned Krylov iterations
        dict(_case("stokes_apply", (2, 2, 2), 5), name="stokes_apply_f64_l5"),
        dict(_case("stokes_minres", (2, 2, 2), 4), name="stokes_minres_f64_l4"),
    ]


# smallest level, and the largest size in unknowns (nx ny nz 8^level), of the drawn cases
_RANGE = {
    "vcycle": (2, 8 ** 9), "solve": (3, 27 * 8 ** 5), "cg": (2, 8 ** 8), "apply": (2, 8 ** 9), "residual": (2, 8 ** 9),
    "sor": (2, 8 ** 9), "transfers": (2, 8 ** 9), "p2_apply": (1, 8 ** 7), "p2_sor": (1, 8 ** 7),
    "p2_vcycle": (1, 8 ** 6), "stokes_apply": (1, 8 ** 6), "stokes_minres": (2, 8 ** 5),
}


def draw(rng):
    kind = rng.choice(sorted(_RANGE))
    low, most = _RANGE[kind]
    while True:
        n = (rng.randint(1, 4), rng.randint(1, 4), rng.randint(1, 4))
        cubes = n[0] * n[1] * n[2]
        top = int(math.log(most / cubes, 8) + 1e-9)
        if top >= low and cubes <= 27:
            break
    dtype = F64 if kind in ("solve", "cg", "p2_vcycle", "stokes_apply", "stokes_minres") else rng.choice((F64, F64, F32))
    case = _case(kind, n, rng.randint(low, top), dtype)
    if kind == "vcycle":
        case["tuned"] = rng.random() < 0.5
    if kind in ("apply", "residual"):
        case["form"] = rng.choice((0, 0, 1))
    return case


@functools.lru_cache(maxsize=1)
def _stream():
    """The stream of the program: every storage works on it, so passes follow one another."""
    return torch.cuda.Stream()


class _Buffer:
    """A level buffer on the device as torch sees it (no copy). The tensor keeps this object, and
    with it the function and its storage, alive."""

    def __init__(self, f, level):
        self.function = f
        n = f.storage.level_size(level)
        kind = "<f8" if f.dtype.itemsize == 8 else "<f4"
        self.__cuda_array_interface__ = dict(shape=(n,), typestr=kind, data=(f.device_ptr(level), False), version=3)


def _out(f, level):
    return torch.as_tensor(_Buffer(f, level), device="cuda")


def _coefficients(case):
    """Smooth positive diffusion coefficient, one value per macro-cell."""
    n = 6 * case["nx"] * case["ny"] * case["nz"]
    return [1.0 + 0.5 * math.sin(0.7 * i) for i in range(n)]


def prepare(case, seed):
    kind, L, dt = case["kind"], case["level"], DTYPE[case["dtype"]]
    p2 = kind.startswith(("p2", "stokes"))
    top = L + 1 if p2 else L
    st = hg.PrimitiveStorage.cuboid((0, 0, 0), (1, 1, 1), case["nx"], case["ny"], case["nz"], top)
    st.set_stream(_stream().cuda_stream)
    s = dict(case=case, kind=kind, level=L, storage=st)
    seed = 64 * int(seed)

    def p1(name, low=L, random=None, high=L):
        f = hg.P1Function(name, st, low, high, dtype=dt)
        if random is not None:
            f.fill_random(seed + random, high)
        return f

    def quadratic(name, low=L, random=None):
        f = hg.P2Function(name, st, low, L, dtype=dt)
        if random is not None:
            f.fill_random(seed + random, L)
        return f

    if kind == "vcycle":
        s.update(A=hg.P1ConstantLaplaceOperator(st, 0, L), x=p1("x", 0), b=p1("b", 0, random=1))
        s["solver"] = hg.GeometricMultigridSolver(st, hg.SORSmoother(1.0), hg.CGSolver(st, 0, 0),
                                                  hg.P1toP1LinearRestriction(), hg.P1toP1LinearProlongation(), 0, L,
                                                  3, 3, dtype=dt)
        if case["tuned"]:
            st.autotune_sor(2, L, dtype=dt)
    elif kind == "solve":
        st.set_cell_coefficients(_coefficients(case))
        s.update(A=hg.P1ConstantLaplaceOperator(st, 0, L), x=p1("x"), b=p1("b", random=1))
        s["solver"] = hg.GeometricMultigridSolver(st, hg.SORSmoother(1.0), hg.CGSolver(st, 0, 0),
                                                  hg.P1toP1LinearRestriction(), hg.P1toP1LinearProlongation(), 0, L,
                                                  3, 3, dtype="float32")
    elif kind == "cg":
        s.update(A=hg.P1ConstantLaplaceOperator(st, L, L), x=p1("x"), b=p1("b", random=1),
                 solver=hg.CGSolver(st, L, L, maxIter=10))
    elif kind in ("apply", "residual"):
        op = hg.P1ConstantMassOperator if case["form"] else hg.P1ConstantLaplaceOperator
        s.update(A=op(st, L, L), x=p1("x", random=1), b=p1("b", random=2), y=p1("y"))
    elif kind == "sor":
        s.update(A=hg.P1ConstantLaplaceOperator(st, L, L), x=p1("x", random=1), b=p1("b", random=2))
    elif kind == "transfers":
        s.update(r=p1("r", L - 1, random=1), x=p1("x", L - 1, random=2),
                 R=hg.P1toP1LinearRestriction(), P=hg.P1toP1LinearProlongation())
        s["x"].fill_random(seed + 3, L - 1)
    elif kind in ("p2_apply", "p2_sor"):
        s.update(A=hg.P2ConstantLaplaceOperator(st, L, L), x=quadratic("x", random=1), y=quadratic("y", random=2))
    elif kind == "p2_vcycle":
        A = hg.P2ConstantLaplaceOperator(st, 0, L)
        s.update(A=A, x=quadratic("x", 0), b=quadratic("b", 0, random=1),
                 solver=hg.P2GeometricMultigridSolver(st, A, 0, L, 3, 3))
    else:
        s["S"] = hg.P2P1TaylorHoodStokesOperator(st, 0 if kind == "stokes_minres" else L, L)
        s.update(u=[quadratic("u", random=1 + k) for k in range(3)], f=[quadratic("f", random=4 + k) for k in range(3)],
                 p=p1("p", random=7), g=p1("g"))
    st.synchronize()
    return s


def run(s):
    kind, L = s["kind"], s["level"]
    if kind in ("vcycle", "cg"):
        s["x"].interpolate(0.0, L)
        s["solver"].solve(s["A"], s["x"], s["b"], L)
        s["x"].communicate(L)
        return _out(s["x"], L)
    if kind == "solve":
        s["x"].interpolate(0.0, L)
        s["solver"].solve_to(s["A"], s["x"], s["b"], L, NEVER, 12)
        s["x"].communicate(L)
        return _out(s["x"], L)
    if kind == "apply":
        s["A"].apply(s["x"], s["y"], L, hg.Inner)
        return _out(s["y"], L)
    if kind == "residual":
        s["A"].residual(s["x"], s["b"], s["y"], L, hg.Inner)
        return _out(s["y"], L)
    if kind == "sor":
        s["A"].smooth_sor(s["x"], s["b"], 1.0, L, hg.Inner)
        s["A"].smooth_sor_backwards(s["x"], s["b"], 1.0, L, hg.Inner)
        s["x"].communicate(L)
        return _out(s["x"], L)
    if kind == "transfers":
        s["R"].restrict(s["r"], L, hg.Inner)
        s["P"].prolongateAndAdd(s["x"], L - 1, hg.Inner)
        return {"coarse": _out(s["r"], L - 1), "fine": _out(s["x"], L)}
    if kind == "p2_apply":
        s["A"].apply(s["x"], s["y"], L)
        return _out(s["y"].v, L + 1)
    if kind == "p2_sor":
        s["A"].smooth_sor(s["x"], s["y"], 1.0, L)
        s["A"].smooth_sor_backwards(s["x"], s["y"], 1.0, L)
        return _out(s["x"].v, L + 1)
    if kind == "p2_vcycle":
        s["x"].interpolate(0.0, L)
        s["solver"].solve(s["x"], s["b"], L)
        return _out(s["x"].v, L + 1)
    if kind == "stokes_apply":
        s["S"].apply(s["u"], s["p"], s["f"], s["g"], L)
        return {"v": [_out(f.v, L + 1) for f in s["f"]], "q": _out(s["g"], L)}
    for f in s["u"]:
        f.interpolate(0.0, L)
    s["p"].interpolate(0.0, L)
    s["S"].minres(s["u"], s["p"], s["f"], s["g"], L, max_iter=20, tol=NEVER)
    for f in s["u"]:
        f.communicate(L)
    s["p"].communicate(L)
    return {"u": [_out(f.v, L + 1) for f in s["u"]], "p": _out(s["p"], L)}


def _inner(case, level):
    n = 2 ** level
    return (case["nx"] * n - 1) * (case["ny"] * n - 1) * (case["nz"] * n - 1)


def work(case):
    """Bytes and operations of one pass: per operation each vector read once and written once."""
    kind, L = case["kind"], case["level"]
    size = 8 if case["dtype"] == F64 else 4
    p1 = [max(_inner(case, k), 0) for k in range(L + 2)]
    n, m = p1[L], p1[L + 1]
    stencil, row2 = 29, 57.5  # flops of a 15-point row, and of a P2 row on average
    if kind == "apply":
        return {"bytes": 2 * size * n, "flops": stencil * n}
    if kind == "residual":
        return {"bytes": 3 * size * n, "flops": (stencil + 1) * n}
    if kind == "sor":
        return {"bytes": 2 * 3 * size * n, "flops": 2 * (stencil + 3) * n}
    if kind == "transfers":
        return {"bytes": size * (3 * n + 2 * p1[L - 1]), "flops": 16 * p1[L - 1] + 3 * n}
    if kind in ("vcycle", "solve"):  # six sweeps, the residual, the restriction, the prolongation per level
        cycle = [sum(p1[1:L + 1]), sum(p1[0:L])]
        moved, flops = (6 * 3 + 3 + 1 + 2) * cycle[0] + 2 * cycle[1], (7 * stencil + 25) * cycle[0]
        if kind == "vcycle":
            return {"bytes": size * moved, "flops": flops}
        return {"bytes": 12 * (4 * moved + 8 * 5 * n), "flops": 12 * (flops + 35 * n)}
    if kind == "cg":  # apply, two fused updates, the dots with them
        return {"bytes": 8 * 11 * 10 * n, "flops": 10 * (stencil + 10) * n}
    if kind == "p2_apply":
        return {"bytes": 2 * size * m, "flops": row2 * m}
    if kind == "p2_sor":
        return {"bytes": 2 * 3 * size * m, "flops": 2 * (row2 + 3) * m}
    if kind == "p2_vcycle":
        cycle = [sum(p1[2:L + 2]), sum(p1[1:L + 1])]
        return {"bytes": size * ((6 * 3 + 3 + 1 + 2) * cycle[0] + 2 * cycle[1]), "flops": (7 * row2 + 40) * cycle[0]}
    apply_bytes, apply_flops = size * (6 * m + 2 * n), (3 * row2 + 50) * m + 390 * n
    if kind == "stokes_apply":
        return {"bytes": apply_bytes, "flops": apply_flops}
    cycles = 3 * ((4 * 3 + 3 + 1 + 2) * sum(p1[2:L + 2]) + 2 * sum(p1[1:L + 1]))  # three V(2,2)
    return {"bytes": 21 * apply_bytes + size * (21 * cycles + 20 * 3 * 14 * m),
            "flops": 21 * apply_flops + 21 * 3 * (5 * row2 + 40) * sum(p1[2:L + 2])}


# ---------------------------------------------------------------------------------------------
# The same outputs in 64 bits from element matrices. Every micro-vertex of the box is a point of
# one dense (nx N + 1) x (ny N + 1) x (nz N + 1) grid, so a DoF vector is a grid and an operator
# is a sum over the micro-tetrahedra of the macro-cells.
# ---------------------------------------------------------------------------------------------
# tetrahedra of a sub-cube by hexahedron corner, the corners' positions, and the six kinds of
# micro-tetrahedra of a refined one with the reduction of their index range
_TETS = ((4, 5, 7, 3), (0, 3, 1, 4), (4, 1, 5, 3), (5, 6, 7, 2), (1, 3, 2, 5), (7, 2, 3, 5))
_CORNERS = ((0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1))
_MICRO = ((((0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1)), 0), (((1, 0, 0), (1, 1, 0), (0, 1, 0), (1, 0, 1)), 1),
          (((1, 0, 0), (0, 1, 0), (1, 0, 1), (0, 0, 1)), 1), (((1, 1, 0), (1, 1, 1), (0, 1, 1), (1, 0, 1)), 2),
          (((1, 0, 1), (0, 1, 1), (0, 0, 1), (0, 1, 0)), 1), (((0, 1, 0), (1, 1, 0), (1, 0, 1), (0, 1, 1)), 1))
_PAIRS = ((0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3))


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Box:
    """Macro-mesh of the box: vertices on the integer grid, cells, faces and edges by vertex IDs."""

    def __init__(self, nx, ny, nz):
        self.n = (nx, ny, nz)
        vid = lambda i, j, k: (k * (ny + 1) + j) * (nx + 1) + i  # noqa: E731
        self.pos = [(i, j, k) for k in range(nz + 1) for j in range(ny + 1) for i in range(nx + 1)]
        self.cells = sorted(tuple(vid(i + _CORNERS[c][0], j + _CORNERS[c][1], k + _CORNERS[c][2]) for c in t)
                            for k in range(nz) for j in range(ny) for i in range(nx) for t in _TETS)
        self.edges = sorted({tuple(sorted((c[a], c[b]))) for c in self.cells for a, b in _PAIRS})
        self.faces = sorted({tuple(sorted(c[i] for i in range(4) if i != o)) for c in self.cells for o in range(4)})
        self.verts = [(v,) for v in range(len(self.pos))]

    def around(self, kind, prims):
        """Per primitive the IDs of the neighbours of a higher kind that hold it."""
        own = [set(p) for p in prims]
        at = {}
        for i, p in enumerate(kind):
            for v in p:
                at.setdefault(v, []).append(i)
        return [sorted(set.intersection(*(set(at[v]) for v in p))) if p else [] for p in own]


@functools.lru_cache(maxsize=4)
def _box(nx, ny, nz):
    return _Box(nx, ny, nz)


class _Level:
    """One refinement level of a box: grid, level-buffer slots, micro-tetrahedra."""

    def __init__(self, box, level):
        self.box, self.L, self.N = box, level, 2 ** level
        self.dim = [k * self.N + 1 for k in box.n]
        self.step = (1, self.dim[0], self.dim[0] * self.dim[1])
        self.points = self.dim[0] * self.dim[1] * self.dim[2]

    def at(self, v):
        return sum(self.N * p * s for p, s in zip(self.box.pos[v], self.step))

    def along(self, a, b):
        return sum((q - p) * s for p, q, s in zip(self.box.pos[a], self.box.pos[b], self.step))

    @functools.lru_cache(maxsize=8)
    def _simplex(self, count, dims):
        """(x, y, z) with x + y + z < count in the layout's order (x fastest), the first `dims` of them."""
        d = _device()
        r = torch.arange(max(count, 0), device=d)
        if dims == 1:
            return (r,)
        if dims == 2:
            y, x = torch.meshgrid(r, r, indexing="ij")
            keep = x + y < count
            return x[keep], y[keep]
        parts = [self._simplex(count - z, 2) for z in range(count)]
        zs = [torch.full_like(p[0], z) for z, p in enumerate(parts)]
        if not parts:
            return r, r, r
        return torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts]), torch.cat(zs)

    def slots(self):
        """Grid point of every slot of the level buffer (-1: padding); owned slots; per owned slot
        the macro-primitive's number and its SOR colour."""
        box, N, w = self.box, self.N, self.N + 1
        where, owned, prim, colour = [], [], [], []
        first = {k: o for k, o in zip("vefc", (0, len(box.verts), len(box.verts) + len(box.edges),
                                               len(box.verts) + len(box.edges) + len(box.faces)))}

        def put(point, own, who, col):
            where.append(point)
            owned.append(own if torch.is_tensor(own) else torch.full_like(point, own, dtype=torch.bool))
            prim.append(torch.full_like(point, who, dtype=torch.int32))
            colour.append(col.to(torch.int8) if torch.is_tensor(col) else torch.full_like(point, col, dtype=torch.int8))

        x, y, z = self._simplex(w, 3)
        inside, col = (x > 0) & (y > 0) & (z > 0) & (x + y + z < N), (x + 2 * y + 3 * z) % 4
        for i, c in enumerate(box.cells):
            put(self.at(c[0]) + x * self.along(c[0], c[1]) + y * self.along(c[0], c[2]) + z * self.along(c[0], c[3]),
                inside, first["c"] + i, col)
            pad = -len(x) % 32
            if pad:
                put(torch.full((pad,), -1, device=x.device), False, 0, 0)
        fc, ef, ec = (box.around(box.cells, box.faces), box.around(box.faces, box.edges),
                      box.around(box.cells, box.edges))
        ve = box.around(box.edges, box.verts)
        x, y = self._simplex(w, 2)
        gx, gy = self._simplex(w - 1, 2)
        for i, f in enumerate(box.faces):
            a, b = self.along(f[0], f[1]), self.along(f[0], f[2])
            put(self.at(f[0]) + x * a + y * b, (x > 0) & (y > 0) & (x + y < N), first["f"] + i, (x + 2 * y) % 3)
            for c in fc[i]:
                o = next(v for v in box.cells[c] if v not in f)
                put(self.at(f[0]) + gx * a + gy * b + self.along(f[0], o), False, 0, 0)
        x = torch.arange(w, device=gx.device)
        for i, e in enumerate(box.edges):
            a = self.along(e[0], e[1])
            put(self.at(e[0]) + x * a, (x > 0) & (x < N), first["e"] + i, x % 2)
            for f in ef[i]:
                o = next(v for v in box.faces[f] if v not in e)
                put(self.at(e[0]) + x[:-1] * a + self.along(e[0], o), False, 0, 0)
            for c in ec[i]:
                o, q = [v for v in box.cells[c] if v not in e]
                put(self.at(e[0]) + x[:-2] * a + self.along(e[0], o) + self.along(e[0], q), False, 0, 0)
        for v in range(len(box.verts)):
            put(torch.tensor([self.at(v)], device=x.device), True, first["v"] + v, 0)
            for e in ve[v]:
                a, b = box.edges[e]
                put(torch.tensor([self.at(v) + self.along(v, b if a == v else a)], device=x.device), False, 0, 0)
        return tuple(torch.cat(p) for p in (where, owned, prim, colour))

    def inner(self):
        """Grid points off the boundary of the box."""
        keep = torch.zeros(tuple(reversed(self.dim)), dtype=torch.bool, device=_device())
        keep[1:-1, 1:-1, 1:-1] = True
        return keep.reshape(-1)

    def micro(self, quadratic=False):
        """Per (macro-cell, kind of micro-tetrahedron): grid points of its nodes and coordinates of
        its vertices relative to the first. Quadratic nodes (vertices, then edge midpoints) live on
        this level's grid, the tetrahedra on the next coarser one."""
        n, two = (self.N // 2, 2) if quadratic else (self.N, 1)
        for i, c in enumerate(self.box.cells):
            d = [self.along(c[0], c[k]) for k in (1, 2, 3)]
            p = [torch.tensor([float(self.box.pos[c[k]][e]) / self.box.n[e] for e in range(3)], dtype=torch.float64)
                 for k in range(4)]
            frame = torch.stack([p[k] - p[0] for k in (1, 2, 3)]) / n  # rows: one step in x, y, z
            for corners, less in _MICRO:
                x, y, z = self._simplex(n - less, 3)
                if not len(x):
                    continue
                base = self.at(c[0]) + two * (x * d[0] + y * d[1] + z * d[2])
                nodes = [two * sum(o * s for o, s in zip(v, d)) for v in corners]
                if quadratic:
                    nodes += [(nodes[a] + nodes[b]) // 2 for a, b in _PAIRS]
                xyz = torch.tensor(corners, dtype=torch.float64) @ frame
                yield i, base, nodes, xyz


def _gradients(xyz):
    """Gradients of the barycentric coordinates and the volume of a tetrahedron."""
    J = (xyz[1:] - xyz[0]).T
    G = torch.linalg.inv(J)
    return torch.cat([-G.sum(0, keepdim=True), G]), abs(float(torch.linalg.det(J))) / 6


def _laplace(xyz):
    G, vol = _gradients(xyz)
    return vol * G @ G.T


def _mass(xyz):
    _, vol = _gradients(xyz)
    return vol / 20 * (torch.ones(4, 4, dtype=torch.float64) + torch.eye(4, dtype=torch.float64))


def _quadrature(xyz):
    """Four points of degree two: weights, barycentric coordinates, gradients of the ten basis functions."""
    G, vol = _gradients(xyz)
    b = (5 - math.sqrt(5)) / 20
    for q in range(4):
        lam = torch.full((4,), b, dtype=torch.float64)
        lam[q] = 1 - 3 * b
        rows = [(4 * lam[i] - 1) * G[i] for i in range(4)] + [4 * (lam[i] * G[j] + lam[j] * G[i]) for i, j in _PAIRS]
        yield vol / 4, lam, torch.stack(rows)


def _laplace2(xyz):
    return sum(w * g @ g.T for w, _, g in _quadrature(xyz))


def _divergence(xyz):
    """[k][pressure vertex][velocity node]: -int psi_i d(phi_j)/dx_k."""
    return sum(-w * torch.einsum("i,jk->kij", lam, g) for w, lam, g in _quadrature(xyz))


def _apply(level, u, element, coefficient=None, quadratic=False):
    y = torch.zeros_like(u)
    for c, base, nodes, xyz in level.micro(quadratic):
        K = element(xyz) * (coefficient[c] if coefficient else 1.0)
        at = [base + o for o in nodes]
        v = torch.stack([u[i] for i in at])
        for i, row in zip(at, K.to(u.device) @ v):
            y.index_add_(0, i, row)
    return y


class _Sweep:
    """The multicolour SOR: vertices, edges, faces, cells in this order (reversed backwards), the
    colours of a kind one after another. A row reads its primitive's closure as it is, anything
    beyond it as of the sweep's start (backwards: as of the start of the kind's phase)."""

    def __init__(self, level, where, owned, prim, colour):
        d, box = _device(), level.box
        self.points = level.points
        self.prim = torch.zeros(level.points, dtype=torch.int64, device=d)
        self.prim[where[owned]] = prim[owned].long()
        col = torch.zeros(level.points, dtype=torch.int64, device=d)
        col[where[owned]] = colour[owned].long()
        prims = [frozenset(p) for k in (box.verts, box.edges, box.faces, box.cells) for p in k]
        kind = torch.tensor([len(p) for p in prims], device=d)[self.prim]
        self.closure = torch.tensor([[q <= p for q in prims] for p in prims], device=d)
        inner = level.inner()
        self.phases = [[inner & (kind == k) & (col == c) for c in range(n)] for k, n in ((1, 1), (2, 2), (3, 3), (4, 4))]
        at, mats = [], []
        for _, base, nodes, xyz in level.micro():
            at.append(torch.stack([base + o for o in nodes], 1))
            mats.append(_laplace(xyz).to(d).expand(len(base), 4, 4))
        self.at, self.K = torch.cat(at), torch.cat(mats)
        self.diagonal = torch.zeros(level.points, dtype=torch.float64, device=d)
        self.diagonal.index_add_(0, self.at.reshape(-1), torch.diagonal(self.K, dim1=1, dim2=2).reshape(-1))

    def product(self, rows, u, old):
        touched = rows[self.at].any(1)
        at, K = self.at[touched], self.K[touched]
        p = self.prim[at]
        v = torch.where(self.closure[p[:, :, None], p[:, None, :]], u[at][:, None, :], old[at][:, None, :])
        y = torch.zeros_like(u)
        y.index_add_(0, at.reshape(-1), (K * v).sum(2).reshape(-1))
        return y

    def __call__(self, u, f, backwards=False):
        u, start = u.clone(), u.clone()
        for phase in reversed(self.phases) if backwards else self.phases:
            if backwards:
                start = u.clone()
            for rows in reversed(phase) if backwards else phase:
                if bool(rows.any()):
                    r = f - self.product(rows, u, start)
                    u = torch.where(rows, u + r / torch.where(rows, self.diagonal, 1.0), u)
        return u


def _midpoints(coarse, fine):
    """Fine grid points of the midpoints of the coarse micro-edges, their coarse ends, how often each occurs."""
    cut = lambda v: sum((v // s % d) * 2 * t for s, d, t in zip(coarse.step, coarse.dim, fine.step))  # noqa: E731
    ends = [[], []]
    for _, base, nodes, _ in coarse.micro():
        for a, b in _PAIRS:
            ends[0].append(base + nodes[a])
            ends[1].append(base + nodes[b])
    a, b = torch.cat(ends[0]), torch.cat(ends[1])
    key = torch.unique(torch.stack([torch.minimum(a, b), torch.maximum(a, b)], 1), dim=0)
    a, b = key[:, 0], key[:, 1]
    return a, b, (cut(a) + cut(b)) // 2, cut


def _prolong(coarse, fine, u):
    a, b, mid, cut = _midpoints(coarse, fine)
    v = torch.zeros(fine.points, dtype=u.dtype, device=u.device)
    v[cut(torch.arange(coarse.points, device=u.device))] = u
    v[mid] = 0.5 * (u[a] + u[b])
    return v


def _restrict(coarse, fine, v):
    a, b, mid, cut = _midpoints(coarse, fine)
    u = v[cut(torch.arange(coarse.points, device=v.device))].clone()
    u.index_add_(0, a, 0.5 * v[mid])
    u.index_add_(0, b, 0.5 * v[mid])
    return u


def _mix(z):
    """One step of splitmix64 on 64-bit integers held as signed ones."""
    z = z + -7046029254386353131
    for shift, factor in ((30, -4658895280553007687), (27, -7723592293110705685)):
        z = (z ^ (z >> shift & (1 << 64 - shift) - 1)) * factor
    return z ^ (z >> 31 & (1 << 33) - 1)


def _random(level, table, seed, dtype=F64):
    """The grid a function holds after fill_random(seed): a value of the owner slot's number."""
    where, owned = table[:2]
    slot = torch.nonzero(owned).reshape(-1)
    key = _mix(torch.tensor([seed], device=slot.device))
    u = (_mix(key ^ slot) >> 11 & (1 << 53) - 1).double() / 2 ** 53
    g = torch.zeros(level.points, dtype=torch.float64, device=slot.device)
    v = -1 + 2 * u
    g[where[slot]] = v.float().double() if dtype == F32 else v
    return g


def _whole(table, grid):
    """Level buffer with every slot holding its grid point's value."""
    where = table[0]
    return torch.where(where >= 0, grid[where.clamp(min=0)], 0.0)


def _owned(table, grid, others=0.0):
    """Level buffer with the grid's values at the owned slots only."""
    where, owned = table[:2]
    return torch.where(owned, grid[where.clamp(min=0)], others)


def _cycle(levels, sweeps, f, L):
    """V(3,3) from a zero start; the coarsest level solved exactly."""
    u = torch.zeros_like(f)
    level = levels[L]
    if L == 0:
        free = torch.nonzero(level.inner()).reshape(-1)
        if len(free):
            cols = []
            for i in free:
                e = torch.zeros_like(f)
                e[i] = 1
                cols.append(_apply(level, e, _laplace)[free])
            u[free] = torch.linalg.solve(torch.stack(cols, 1), f[free])
        return u
    inner = level.inner()
    for _ in range(3):
        u = sweeps[L](u, f)
    # the boundary rows of the residual vector are never written and stay zero
    r = torch.where(inner, f - _apply(level, u, _laplace), 0.0)
    e = _cycle(levels, sweeps, _restrict(levels[L - 1], level, r), L - 1)
    u = torch.where(inner, u + _prolong(levels[L - 1], level, e), u)
    for _ in range(3):
        u = sweeps[L](u, f)
    return u


def exact(case, seed):
    kind, L, dt = case["kind"], case["level"], case["dtype"]
    seed, gpu = 64 * int(seed), torch.cuda.is_available()
    size = case["nx"] * case["ny"] * case["nz"] * 8 ** (L + (1 if kind.startswith(("p2", "stokes")) else 0))
    most = {"apply": 8 ** 9, "residual": 8 ** 9, "transfers": 8 ** 7, "sor": 8 ** 7, "vcycle": 8 ** 6, "cg": 8 ** 7,
            "p2_apply": 8 ** 8, "stokes_apply": 8 ** 7}.get(kind, 0)  # the others: the whole multigrid again, over 20 s
    if size > (most if gpu else most // 64):
        return None
    box = _box(case["nx"], case["ny"], case["nz"])
    if kind.startswith(("p2", "stokes")):
        level = _Level(box, L + 1)
        table, inner = level.slots(), level.inner()
        if kind == "p2_apply":
            y = _apply(level, _random(level, table, seed + 1, dt), _laplace2, quadratic=True)
            return _whole(table, torch.where(inner, y, _random(level, table, seed + 2, dt)))
        coarse = _Level(box, L)
        ctable = coarse.slots()
        u = [_random(level, table, seed + 1 + k) for k in range(3)]
        p = _random(coarse, ctable, seed + 7)
        v = [_apply(level, g, _laplace2, quadratic=True) for g in u]
        q = torch.zeros_like(p)
        for (_, base, nodes, xyz), (_, cbase, cnodes, _) in zip(level.micro(True), coarse.micro()):
            D = _divergence(xyz).to(p.device)
            at, pat = [base + o for o in nodes], [cbase + o for o in cnodes[:4]]
            pv = torch.stack([p[i] for i in pat])
            for k in range(3):
                for i, row in zip(at, D[k].T @ pv):
                    v[k].index_add_(0, i, row)
                for i, row in zip(pat, D[k] @ torch.stack([u[k][j] for j in at])):
                    q.index_add_(0, i, row)
        return {"v": [_whole(table, torch.where(inner, v[k], _random(level, table, seed + 4 + k))) for k in range(3)],
                "q": _whole(ctable, q)}
    level = _Level(box, L)
    table, inner = level.slots(), level.inner()
    if kind in ("apply", "residual"):
        y = _apply(level, _random(level, table, seed + 1, dt), _mass if case["form"] else _laplace)
        if kind == "residual":
            y = _random(level, table, seed + 2, dt) - y
        return _owned(table, torch.where(inner, y, 0.0))
    if kind == "transfers":
        coarse = _Level(box, L - 1)
        ctable = coarse.slots()
        r, x = _random(level, table, seed + 1, dt), _random(level, table, seed + 2, dt)
        c = torch.where(coarse.inner(), _restrict(coarse, level, r), 0.0)
        fine = torch.where(inner, x + _prolong(coarse, level, _random(coarse, ctable, seed + 3, dt)), x)
        # the copies of the fine function hold what the random fill's exchange left there
        return {"coarse": _owned(ctable, c), "fine": _owned(table, fine, _whole(table, x))}
    if kind == "sor":
        sweep = _Sweep(level, *table)
        u, f = _random(level, table, seed + 1, dt), _random(level, table, seed + 2, dt)
        return _whole(table, sweep(sweep(u, f), f, backwards=True))
    f = _random(level, table, seed + 1, dt if kind == "vcycle" else F64)
    if kind == "cg":
        x = torch.zeros_like(f)
        r = torch.where(inner, f, 0.0)
        p, rr = r.clone(), float(r @ r)
        for _ in range(10):
            ap = torch.where(inner, _apply(level, p, _laplace), 0.0)
            a = rr / float(p @ ap)
            x, r = x + a * p, r - a * ap
            new = float(r @ r)
            if math.sqrt(new) < 1e-16:
                break
            p, rr = r + new / rr * p, new
        return _whole(table, x)
    levels = [_Level(box, k) for k in range(L + 1)]
    sweeps = [_Sweep(v, *(table if v.L == L else v.slots())) if v.L else None for v in levels]
    levels[L] = level
    return _whole(table, _cycle(levels, sweeps, f, L))
