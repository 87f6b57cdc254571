"""The work that programs have this library do, as cases that can be timed and compared.

A case is a plain dict.  Its "kind" says which part of a program it is:

  step     blocks of whole electrostatic steps (charge density, Poisson
           multigrid, push, re-sort) between two reads of the energies, in 2-D
           and 3-D, both precisions, periodic and bounded
  solve    one Poisson solve from a zero guess through a solver handle
  spline   a B-spline gradient gather and deposit of all positions
  restart  particles in arbitrary order loaded, sorted, deposited, binned, pushed
           in the potential of a checkpoint and exported: the first push of a run
  adjoint  forward and backward pass of a differentiable run

Every random array is made on the GPU from the seed alone.  The step cases
return fields, densities and energies of the state that they leave; FP64 ones
in a periodic box, where no particle leaves, return the particles too.  In mixed precision the particles themselves cannot
be compared one by one: a potential that differs in its last bits moves a few
of 10^8 particles over a cell face, and the order of a sorted state shifts.
The density after several steps depends on every position and velocity, and
the restart cases, whose potential is an input, return every particle.
"""
import math

import numpy as np
import torch

import psum_b200 as P
from psum_b200.adjoint import ElectrostaticLoss, ElectrostaticRun

MASS_RATIO = 1836.0
CHUNK = 1 << 24   # particles per piece of the 64-bit comparison


# --------------------------------------------------------------------- cases --
def _step(**k):
    case = dict(kind="step", nz=0, periodic=True, species=1, precision="mixed", sort=1, steps=4, profile="uniform",
                pusher="leapfrog", dt=0.1, tol=1e-8, order=1, fma=False)
    case.update(k)
    return case


def listed():
    return [
        # a 64 x 64-node periodic FP64 plasma (1 % density mode): the smallest run, where launches and latency count;
        # one block of steps is the interval after which it re-sorts
        _step(name="step_2d_fp64_64", nx=64, ny=64, ppc=64, precision="fp64", sort=20, steps=20, tol=1e-10,
              profile="mode1"),
        # the bench's plasma: two species between grounded, absorbing walls, re-sorted every step
        _step(name="step_2d_bounded_1025", nx=1025, ny=1025, ppc=256, periodic=False, species=2),
        # two electron beams through a 3-D periodic box, 32 particles per cell, re-sorted every step
        _step(name="step_3d_beams_128", nx=128, ny=128, nz=128, ppc=32, dt=0.05, profile="beams"),
        # the FP64 run that the mixed one is compared with: in-place push, re-sort every fourth step
        _step(name="step_2d_fp64_513", nx=513, ny=513, ppc=64, periodic=False, species=2, precision="fp64", sort=4,
              fma=True),
        # a dense blob drifting through a 3-D box: clustered load, restarted from its snapshot every block
        _step(name="step_3d_blob_128", nx=128, ny=128, nz=128, ppc=8, profile="blob"),
        # the potential of a bounded 2-D plasma (PSuM's usual field solve), mixed precision
        dict(name="solve_2d_1025", kind="solve", nx=1025, ny=1025, nz=0, periodic=False, precision="mixed", tol=1e-8),
        # a 3-D periodic potential of mean zero
        dict(name="solve_3d_128", kind="solve", nx=128, ny=128, nz=128, periodic=True, precision="mixed", tol=1e-8),
        # a small FP64 solve in a 3-D box with grounded walls and unequal sides
        dict(name="solve_3d_fp64_33", kind="solve", nx=33, ny=41, nz=29, periodic=False, precision="fp64", tol=1e-10),
        # third-order shapes on a 1024 x 1024-node grid, 64 particles per cell stored cell by cell
        dict(name="spline_2d_order3", kind="spline", nx=1024, ny=1024, nz=0, ppc=64, order=3, sorted=True),
        # second-order shapes in 3-D
        dict(name="spline_3d_order2", kind="spline", nx=97, ny=97, nz=97, ppc=16, order=2, sorted=True),
        # particles of a 3-D run in arbitrary order: load, sort, deposit, bin, first push, export
        dict(name="restart_3d_16m", kind="restart", nx=128, ny=128, nz=128, n=1 << 24, precision="mixed"),
        # Landau damping, 64 electrons per cell, differentiated with respect to initial velocities and an external field
        dict(name="adjoint_2d_256", kind="adjoint", nx=256, ny=256, ppc=64, steps=20, tol=1e-10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, dim, lo, hi, periodic):
    """Nodes per axis, within a factor of 1.6 of each other; a wrapping axis is
    halved level by level, so its count is a multiple of a power of two."""
    first = _log_int(rng, lo, hi)
    side = [first] + [max(lo, min(hi, int(first * math.exp(rng.uniform(-0.5, 0.5))))) for _ in range(dim - 1)]
    if periodic:
        unit = 16 if dim == 3 or hi <= 256 else 32
        side = [max(unit, k // unit * unit) for k in side]
    return side + [0] * (3 - dim)


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["step", "step", "step", "step", "solve", "solve", "spline", "spline", "restart", "adjoint"])
    fp64 = rng.random() < 0.3
    if kind == "step":
        periodic = rng.random() < 0.5
        three = rng.random() < 0.45
        species = 1 if periodic else 2
        most = (3 << 24) // species if not fp64 else (1 << 24) // species   # particles per species
        side = _sides(rng, 3, 24, 128, periodic) if three else _sides(rng, 2, 48, 1025, periodic)
        nodes = side[0] * side[1] * max(1, side[2])
        ppc = max(4, min(_log_int(rng, 8, 256), most // nodes))
        sort = rng.choice([1, 1, 1, 4]) if not fp64 else rng.choice([4, 20])
        return _step(nx=side[0], ny=side[1], nz=side[2], ppc=ppc, periodic=periodic, species=species,
                     precision="fp64" if fp64 else "mixed", sort=sort, fma=fp64 and rng.random() < 0.5,
                     profile=rng.choice(["uniform", "mode1", "beams"]) if periodic else "uniform",
                     dt=0.05, pusher=rng.choice(["leapfrog", "leapfrog", "boris"]),
                     order=rng.choice([1, 1, 1, 1, 2, 3]))
    if kind == "solve":
        periodic = rng.random() < 0.4
        side = _sides(rng, 2, 33, 1025, periodic) if rng.random() < 0.5 else _sides(rng, 3, 17, 128, periodic)
        return dict(kind="solve", nx=side[0], ny=side[1], nz=side[2], periodic=periodic,
                    precision="fp64" if fp64 else "mixed", tol=1e-10 if fp64 else 1e-8)
    if kind == "spline":
        side = _sides(rng, 2, 32, 1024, False) if rng.random() < 0.6 else _sides(rng, 3, 16, 97, False)
        nodes = side[0] * side[1] * max(1, side[2])
        ppc = max(2, min(_log_int(rng, 4, 128), (1 << 25) // nodes))
        return dict(kind="spline", nx=side[0], ny=side[1], nz=side[2], ppc=ppc, order=rng.choice([1, 2, 3, 4]),
                    sorted=rng.random() < 0.7)
    if kind == "restart":
        side = _sides(rng, 2, 48, 1025, False) if rng.random() < 0.5 else _sides(rng, 3, 24, 128, False)
        return dict(kind="restart", nx=side[0], ny=side[1], nz=side[2], n=_log_int(rng, 1 << 15, 1 << 24),
                    precision="fp64" if fp64 else "mixed")
    side = _sides(rng, 2, 32, 256, True)
    return dict(kind="adjoint", nx=side[0], ny=side[1], ppc=rng.choice([16, 32, 64]), steps=rng.choice([5, 10, 20]), tol=1e-10)


# ------------------------------------------------------------------ geometry --
def _nodes(case):
    return (case["nx"], case["ny"]) + ((case["nz"],) if case.get("nz") else ())


def _box(case):
    """Cells, lower and upper corner (unit spacing).  Periodic boxes follow the
    wrapping-node idiom: n nodes, n - 1 cells, lower corner at half a cell, period n."""
    n = _nodes(case)
    lo = 0.5 if case.get("periodic", True) else 0.0
    return tuple(k - 1 for k in n), (lo,) * len(n), tuple(lo + k - 1 for k in n)


def _depth(case):
    """Levels below the finest: halve while every axis keeps eight nodes (a
    wrapping axis must stay even to be halved)."""
    n, depth, periodic = list(_nodes(case)), 0, case.get("periodic", True)
    while min(n) >= 8 and depth < 5 and not (periodic and any(k % 2 for k in n)):
        n = [k // 2 if periodic else (k + 1) // 2 for k in n]
        depth += 1
    return max(1, depth)


def _problem(case, pinned=False):
    """Grid, solver options and fixed nodes: grounded walls, or a periodic box
    whose potential has mean zero or is pinned at one node."""
    n = _nodes(case)
    cells, lo, hi = _box(case)
    grid = P.simple_grid(lo, hi, cells)
    three = len(n) == 3
    opts = (f"I {n[0]} J {n[1]} K {n[2] if three else 1} depth {_depth(case)} pre_relax 2 post_relax 2 "
            f"max_cycles 40 correction_interval 2 tol {case['tol']}")
    if case.get("periodic", True):
        opts += " periodic_I 1 periodic_J 1" + (" periodic_K 1" if three else "") + ("" if pinned else " null_space 1")
        return grid, opts, [P.Dirichlet_nodes(grid, [(0,) * len(n)], 0.0)] if pinned else []
    wall = np.flatnonzero(_walls(n))
    return grid, opts, [(wall.astype(np.uint64), np.zeros(wall.size))]


def _walls(n):
    wall = np.ones(n, bool)
    wall[tuple(slice(1, -1) for _ in n)] = False
    return wall.reshape(-1)


def _solver(case, pinned=False):
    """The Poisson solver a run keeps."""
    grid, opts, fixed = _problem(case, pinned)
    ps = P.Poisson_solver_3d() if grid.dim == 3 else P.Poisson_solver_2d()
    ps.set_options(opts)
    ps.init("cuda_multigrid64_gpu" if case["precision"] == "fp64" else "cuda_multigrid32f_gpu", grid, ps.Cartesian,
            fixed, 1.0)
    ps.make_righthand_item()
    return ps


def _mode1(u, L, amp):
    """Positions with density 1 + amp cos(2 pi x / L), from uniform ones."""
    k = 2 * math.pi / L
    x = u.clone()
    for _ in range(12):
        x -= (x + amp / k * torch.sin(k * x) - u) / (1 + amp * torch.cos(k * x))
    return torch.remainder(x, L)


def _species(case):
    """(charge, mass, thermal velocity) per species."""
    return [(-1.0, 1.0, 1.0), (1.0, MASS_RATIO, 1.0 / math.sqrt(MASS_RATIO))][:case.get("species", 1)]


def _particles(case, seed):
    """FP64 positions and velocities of every species, and the particle weight
    that makes the mean density one."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    n = _nodes(case)
    cells, lo, _ = _box(case)
    width = [float(k) for k in (n if case.get("periodic", True) else cells)]
    count = int(np.prod(width)) * case["ppc"]
    out = []
    for _, _, vth in _species(case):
        pos = torch.empty((len(n), count), dtype=torch.float64, device="cuda")
        vel = torch.empty((3, count), dtype=torch.float64, device="cuda")
        vel.normal_(0.0, vth, generator=gen)
        profile = case.get("profile", "uniform")
        if profile == "blob":
            pos.normal_(0.0, 1.0, generator=gen)
            for a in range(len(n)):
                pos[a].mul_(0.05 * width[a]).add_(width[a] / 2)
            vel[2] += 2.0
        else:
            pos.uniform_(0.0, 1.0, generator=gen)
            for a in range(len(n)):
                pos[a].mul_(width[a])
            if profile == "mode1":
                pos[0] = _mode1(pos[0], width[0], 0.05 if case["kind"] == "adjoint" else 0.01)
            elif profile == "beams":
                vel[0, :count // 2] += 5.0
                vel[0, count // 2:] -= 5.0
        for a in range(len(n)):
            if case.get("periodic", True):
                torch.remainder(pos[a], width[a], out=pos[a])
            pos[a].add_(lo[a])
        out.append((pos, vel))
    return out, float(np.prod(width)) / count


# ------------------------------------------------------------------- prepare --
def prepare(case, seed):
    return {"step": _prepare_step, "solve": _prepare_solve, "spline": _prepare_spline, "restart": _prepare_restart,
            "adjoint": _prepare_adjoint}[case["kind"]](case, seed)


def _context(case):
    cells, lo, hi = _box(case)
    return P.ParticleContext(cells, lo, hi, (int(case.get("periodic", True)),) * len(cells),
                             P.FP64 if case["precision"] == "fp64" else P.MIXED)


def _pinned(case):
    return case["periodic"] and not case["nz"]


def _prepare_step(case, seed):
    parts, weight = _particles(case, seed)
    ctx = _context(case)
    ctx.set_options(f"sort_interval {case['sort']} diagnostics 1" + (f" interp_order {case['order']}" if case["order"] > 1 else "")
                    + (" fp64_fma 1" if case["fma"] else ""))
    ids = []
    for (q, m, _), (pos, vel) in zip(_species(case), parts):
        ids.append(ctx.add_species(q, m, weight, pos.shape[1]))
        ctx.load(ids[-1], pos, vel)
    del parts, pos, vel
    torch.cuda.empty_cache()
    ctx.sort()
    ctx.deposit()
    # 2-D periodic runs pin one node, 3-D ones take the potential of mean zero
    solver = _solver(case, pinned=_pinned(case))
    stream = torch.cuda.Stream()
    ctx.set_stream(stream)
    nodes = int(np.prod(_nodes(case)))
    field = lambda: torch.zeros(nodes, dtype=torch.float64, device="cuda")   # noqa: E731
    s = dict(case=case, ctx=ctx, ids=ids, solver=solver, stream=stream, rho=field(), phi=field(),
             density=[field() for _ in ids])
    if case["profile"] == "blob":
        s["snapshot"] = torch.empty(ctx.state_bytes(ids[0]), dtype=torch.uint8, device="cuda")
        ctx.save_state(ids[0], s["snapshot"])
    torch.cuda.synchronize()
    return s


def _charge(case, seed):
    """The right-hand side of a plasma: a smooth charge and particle noise."""
    n = _nodes(case)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    rho = torch.randn(n, generator=gen, device="cuda", dtype=torch.float64) * 0.1
    smooth = torch.ones((), dtype=torch.float64, device="cuda")
    for a, k in enumerate(n):
        x = torch.arange(k, dtype=torch.float64, device="cuda") / k
        phase = torch.rand((), generator=gen, device="cuda", dtype=torch.float64)
        smooth = smooth * torch.cos(2 * math.pi * (x + phase)).reshape([-1 if b == a else 1 for b in range(len(n))])
    return (rho + smooth).reshape(-1).contiguous()


def _prepare_solve(case, seed):
    rho = _charge(case, seed)
    return dict(case=case, solver=_solver(case), rho=rho, b=torch.empty_like(rho), x=torch.empty_like(rho))


def _prepare_spline(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    n = _nodes(case)
    cells, lo, hi = _box(case)
    count = int(np.prod(cells)) * case["ppc"]
    pos = torch.rand((len(n), count), generator=gen, device="cuda", dtype=torch.float64)
    if case["sorted"]:
        cell = torch.arange(count, device="cuda") // case["ppc"]
        for a in reversed(range(len(n))):
            pos[a] += cell % cells[a]
            cell = cell // cells[a]
    else:
        for a in range(len(n)):
            pos[a] *= cells[a]
    for a in range(len(n)):
        pos[a] += lo[a]
    nodes = int(np.prod(n))
    return dict(case=case, grid=P.simple_grid(lo, hi, cells), pos=pos,
                phi=torch.randn(nodes, generator=gen, device="cuda", dtype=torch.float64),
                rho=torch.zeros(nodes, dtype=torch.float64, device="cuda"),
                scratch=torch.empty(nodes, dtype=torch.int64, device="cuda"))


def _restart_particles(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    n = _nodes(case)
    pos = torch.rand((len(n), case["n"]), generator=gen, device="cuda", dtype=torch.float64)
    for a in range(len(n)):
        pos[a].mul_(float(n[a])).add_(0.5)
    vel = torch.randn((3, case["n"]), generator=gen, device="cuda", dtype=torch.float64)
    return pos, vel


def _restart_potential(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed + 1)
    return torch.randn(int(np.prod(_nodes(case))), generator=gen, device="cuda", dtype=torch.float64)


def _prepare_restart(case, seed):
    pos, vel = _restart_particles(case, seed)
    cells = _box(case)[0]
    ctx = _context(case)
    sp = ctx.add_species(-1.0, 1.0, 1.0, case["n"])
    ref_cells = int(np.prod(cells))
    new = lambda n, t: torch.empty(n, dtype=t, device="cuda")   # noqa: E731
    return dict(case=case, ctx=ctx, sp=sp, pos=pos, vel=vel, keys=new(case["n"], torch.int64),
                counts=new(ref_cells, torch.int64), offsets=new(ref_cells, torch.int64),
                perm=torch.zeros(case["n"], dtype=torch.int64, device="cuda"),
                density=new(int(np.prod(_nodes(case))), torch.float64), phi=_restart_potential(case, seed))


def _adjoint_inputs(case, seed):
    parts, weight = _particles(dict(case, periodic=True, species=1, profile="mode1"), seed)
    pos, vel = parts[0]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed + 1)
    phi_ext = torch.randn(case["nx"] * case["ny"], generator=gen, device="cuda", dtype=torch.float64) * 0.01
    return pos, vel.to(torch.float32), phi_ext, weight


def _prepare_adjoint(case, seed):
    pos, vel, phi_ext, weight = _adjoint_inputs(case, seed)
    grid, opts, fixed = _problem(case, pinned=True)
    run = ElectrostaticRun(grid, (1, 1), [(-1.0, 1.0, weight, pos)], fixed, opts, 0.1, case["steps"],
                           checkpoint_every=10, precision=P.MIXED, background=1.0)
    return dict(case=case, run=run, vel=vel, phi_ext=phi_ext)


# ----------------------------------------------------------------------- run --
FIELD_B = (0.0, 0.0, 0.5)


def run(s):
    return {"step": _run_step, "solve": _run_solve, "spline": _run_spline, "restart": _run_restart,
            "adjoint": _run_adjoint}[s["case"]["kind"]](s)


def _run_step(s):
    """A block of steps, then the fields and energies a program records."""
    case, ctx = s["case"], s["ctx"]
    with torch.cuda.stream(s["stream"]):
        if "snapshot" in s:
            s["rho"].zero_()
            s["phi"].zero_()
            ctx.restore_state(s["ids"][0], s["snapshot"])
            ctx.deposit()
        background = 1.0 if case["species"] == 1 else 0.0
        pusher = P.BORIS if case["pusher"] == "boris" else P.LEAPFROG
        for _ in range(case["steps"]):
            ctx.step(s["solver"].backend, background, s["rho"], s["phi"], case["dt"], pusher, FIELD_B)
        out = {"rho": s["rho"], "phi": s["phi"], "energy": _energies(ctx.step_diagnostics(1.0))}
        if case["order"] == 1:   # with B-spline shapes a step leaves no CIC deposit to read
            for sp, d in zip(s["ids"], s["density"]):
                ctx.density(sp, d)
            out["density"] = s["density"]
        if case["precision"] == "fp64" and case["periodic"]:
            out["particles"] = [ctx.get_state_device(sp) for sp in s["ids"]]
        return out


def _energies(d):
    return np.array(list(d["kinetic"]) + [d["field"]])


def _run_solve(s):
    """b is the solve's scratch (its sources are applied in place)."""
    stream = torch.cuda.current_stream()
    s["b"].copy_(s["rho"])
    s["x"].zero_()
    s["solver"].backend.solve_async(s["b"], s["x"], stream)
    return {"phi": s["x"]}


def _run_spline(s):
    order = s["case"]["order"]
    grad = P.interp_diff_B_spline(order, s["grid"], s["pos"], s["phi"])
    s["rho"].zero_()
    P.add_back_B_spline(order, s["grid"], s["pos"], 0.25, s["rho"], scratch=s["scratch"])
    return {"gradient": grad, "rho": s["rho"]}


def _run_restart(s):
    ctx, sp = s["ctx"], s["sp"]
    ctx.load(sp, s["pos"], s["vel"])
    ctx.sort()
    ctx.deposit()
    ctx.density(sp, s["density"])
    inside = ctx.bin(sp, s["keys"], s["counts"], s["offsets"], s["perm"])
    ctx.push(s["phi"], 0.05)
    ctx.sort()
    pos, vel = ctx.get_state_device(sp)
    return {"density": s["density"], "keys": s["keys"], "counts": s["counts"], "offsets": s["offsets"],
            "perm": s["perm"], "inside": inside, "pos": pos, "vel": vel}


def _run_adjoint(s):
    v = s["vel"].clone().requires_grad_(True)
    pe = s["phi_ext"].clone().requires_grad_(True)
    loss = ElectrostaticLoss.apply(s["run"], pe, v)
    loss.backward()
    return {"loss": loss.detach(), "velocity_gradient": v.grad, "field_gradient": pe.grad}


# ----------------------------------------------------------- work, tolerance --
def work(case):
    """Bytes of one read of every input and one write of every output; of a
    step, one read and one write of every particle's state and of the fields."""
    nodes = int(np.prod(_nodes(case)))
    dim = len(_nodes(case))
    kind = case["kind"]
    if kind == "solve":
        return {"bytes": nodes * 16, "flops": 0}
    if kind == "spline":
        n = int(np.prod(_box(case)[0])) * case["ppc"]
        taps = (case["order"] + 1) ** dim
        return {"bytes": n * (8 * dim + 8 * dim) + nodes * 16, "flops": n * taps * (2 * dim + 2)}
    if kind == "restart":
        fp64 = case["precision"] == "fp64"
        stored = 8 * (dim + 3) if fp64 else 4 * (dim + 3)
        n = case["n"]
        return {"bytes": n * (8 * (dim + 3) + 2 * stored + 8 * (dim + 3) + 16) + nodes * 32, "flops": 0}
    width = _nodes(case) if case.get("periodic", True) else _box(case)[0]
    n = int(np.prod(width)) * case["ppc"] * case.get("species", 1)
    state = (4 * (dim + 3) + 4) if case.get("precision", "mixed") == "mixed" else (8 * (dim + 3) + 4)
    passes = case["steps"] * (2 if kind == "adjoint" else 1)
    fields = nodes * 8 * (3 + case.get("species", 1))
    return {"bytes": passes * (2 * n * state + fields), "flops": 0}


def tolerance(case):
    kind = case["kind"]
    fp64 = case.get("precision") == "fp64"
    if kind == "solve":
        # solves of different rounding that meet the same residual bound (measured against a direct solve: 3e-11 at 1e-8)
        return {"rel": 1e-8 if fp64 else 1e-6}
    if kind == "spline":
        return {"rel": 1e-10}   # the deposit's fixed point: 3e-12 against 64 bits
    if kind == "restart":
        return "exact"          # integers, and particles in an order that every bit of their positions decides
    if kind == "adjoint":
        return {"rel": 5e-4}    # FP32 adjoint arrays: 1.2e-4 against 64 bits
    if fp64:                    # the potential's residual bound
        return {"rel": 1e-6 if case["tol"] > 1e-9 else 1e-8}
    # FP32 offsets and velocities: 2e-7 against 64 bits, and 7e-5 where a dense blob explodes over many cells
    return {"rel": 3e-4 if case["profile"] == "blob" else 1e-5}


# --------------------------------------------------------------------- exact --
def exact(case, seed):
    return {"step": _exact_step, "solve": _exact_solve, "spline": _exact_spline, "restart": _exact_restart,
            "adjoint": _exact_adjoint}[case["kind"]](case, seed)


def _eigen(n, periodic):
    """Eigenvalues of -d2/dx2 (unit spacing) per axis, summed over the grid."""
    total = torch.zeros((), dtype=torch.float64, device="cuda")
    for a, k in enumerate(n):
        if periodic:
            m = torch.arange(k, dtype=torch.float64, device="cuda")
            e = 4 * torch.sin(math.pi * m / k) ** 2
        else:
            m = torch.arange(1, k - 1, dtype=torch.float64, device="cuda")
            e = 4 * torch.sin(math.pi * m / (2 * (k - 1))) ** 2
        total = total + e.reshape([-1 if b == a else 1 for b in range(len(n))])
    return total


def _sine(v, axis):
    """Discrete sine transform (type I) along one axis; its own inverse up to 2 / (n + 1)."""
    v = v.movedim(axis, -1)
    n = v.shape[-1]
    z = torch.zeros(v.shape[:-1] + (1,), dtype=v.dtype, device=v.device)
    odd = torch.cat([z, v, z, -v.flip(-1)], dim=-1)
    return (-0.5 * torch.fft.fft(odd, dim=-1).imag[..., 1:n + 1]).movedim(-1, axis)


def _poisson(rho, n, periodic, pinned):
    """-laplace(phi) = rho in 64 bits: Fourier (periodic) or sine (grounded walls) series."""
    r = rho.reshape(n)
    if periodic:
        if pinned:   # the pinned node's own equation is dropped: its charge follows from neutrality
            r = r.reshape(-1).clone()
            r = torch.cat([-r[1:].sum().reshape(1), r[1:]]).reshape(n)
        f = torch.fft.fftn(r)
        e = _eigen(n, True).clone()
        e.view(-1)[0] = 1.0
        f = f / e
        f = f * (torch.arange(f.numel(), device="cuda") > 0).reshape(n)
        phi = torch.fft.ifftn(f).real
        if pinned:
            phi = phi - phi.reshape(-1)[0]
        return phi.reshape(-1)
    inner = r[tuple(slice(1, -1) for _ in n)]
    f = inner
    for a in range(len(n)):
        f = _sine(f, a)
    f = f / _eigen(n, False)
    for a in range(len(n)):
        f = _sine(f, a) * (2.0 / (n[a] - 1))
    phi = torch.zeros(n, dtype=torch.float64, device="cuda")
    phi[tuple(slice(1, -1) for _ in n)] = f
    return phi.reshape(-1)


def _exact_solve(case, seed):
    return {"phi": _poisson(_charge(case, seed), _nodes(case), case["periodic"], pinned=False)}


def _shape(t, order):
    """Centred cardinal B-spline of degree `order` at t (Cox-de Boor)."""
    if order == 0:
        return ((t >= -0.5) & (t < 0.5)).to(t.dtype)
    h = (order + 1) / 2
    return ((t + h) * _shape(t + 0.5, order - 1) + (h - t) * _shape(t - 0.5, order - 1)) / order


def _weights(s, order):
    """Base node and weights (values, derivatives) along one axis at s (cell units)."""
    base = torch.floor(s) - (order - 1) // 2 if order % 2 else torch.floor(s + 0.5) - order // 2
    w, d = [], []
    for k in range(order + 1):
        t = s - (base + k)
        if order == 1:
            w.append((1 - t) if k == 0 else (1 + t))
            d.append(torch.full_like(t, -1.0 if k == 0 else 1.0))
        else:
            w.append(_shape(t, order))
            d.append(_shape(t + 0.5, order - 1) - _shape(t - 0.5, order - 1))
    return base.long(), w, d


def _taps(order, dim):
    return np.ndindex(*([order + 1] * dim))


def _node(bases, tap, n):
    i = 0
    for a, k in enumerate(n):
        i = i * k + torch.remainder(bases[a] + tap[a], k)
    return i


def _gradient(s, phi, n, order):
    axes = [_weights(s[a], order) for a in range(len(n))]
    g = torch.zeros_like(s)
    for tap in _taps(order, len(n)):
        f = phi[_node([x[0] for x in axes], tap, n)]
        for a in range(len(n)):
            term = f
            for b in range(len(n)):
                term = term * (axes[b][2] if b == a else axes[b][1])[tap[b]]
            g[a] += term
    return g


def _deposit(s, out, n, order, weight):
    axes = [_weights(s[a], order) for a in range(len(n))]
    for tap in _taps(order, len(n)):
        w = torch.full_like(s[0], weight)
        for a in range(len(n)):
            w = w * axes[a][1][tap[a]]
        out.index_add_(0, _node([x[0] for x in axes], tap, n), w)


def _exact_spline(case, seed):
    s = _prepare_spline(case, seed)
    n = _nodes(case)
    lo = _box(case)[1]
    taps = (case["order"] + 1) ** len(n)
    if s["pos"].shape[1] * taps > 2.5e9:
        return None
    grad, rho = torch.empty_like(s["pos"]), s["rho"]
    for i in range(0, s["pos"].shape[1], CHUNK // 4):
        u = torch.stack([s["pos"][a, i:i + CHUNK // 4] - lo[a] for a in range(len(n))])
        grad[:, i:i + CHUNK // 4] = _gradient(u, s["phi"], n, case["order"])
        _deposit(u, rho, n, case["order"], 0.25)
    return {"gradient": grad, "rho": rho}


def _exact_restart(case, seed):
    """The density of the loaded particles and, in FP64, the pushed particles
    sorted by cell (stable).  FP32 offsets put some particles on the other side
    of a cell face, so a mixed state has another order than the 64-bit one."""
    pos, vel = _restart_particles(case, seed)
    n = _nodes(case)
    rho = torch.zeros(int(np.prod(n)), dtype=torch.float64, device="cuda")
    u, v = pos - 0.5, vel
    _deposit(u, rho, n, 1, 1.0)
    out = {"density": rho, "keys": None, "counts": None, "offsets": None, "perm": None, "inside": None, "pos": None,
           "vel": None}
    if case["precision"] == "fp64":
        width = torch.tensor([float(k) for k in n], device="cuda").double()[:, None]
        for pushed in (False, True):
            if pushed:
                u, v = _push(u, v, _restart_potential(case, seed), n, dict(dt=0.05, order=1, pusher="leapfrog"), -1.0)
                u = torch.remainder(u, width)
            key = torch.zeros_like(u[0], dtype=torch.int64)
            for a, k in enumerate(n):
                key = key * k + torch.floor(u[a]).long()
            order = torch.argsort(key, stable=True)
            u, v = u[:, order], v[:, order]
        out.update(pos=u + 0.5, vel=v)
    return out


def _push(u, v, phi, n, case, q_m):
    """One kick and move (cell units = length units here); Boris rotation about FIELD_B."""
    dt = case["dt"]
    e = -_gradient(u, phi, n, case["order"])
    kick = torch.zeros_like(v)
    kick[:len(n)] = e * (q_m * dt)
    if case["pusher"] == "boris":
        half = v + 0.5 * kick
        t = torch.tensor(FIELD_B, dtype=torch.float64, device="cuda").mul(0.5 * q_m * dt)
        sv = 2 * t / (1 + (t * t).sum())
        cross = lambda p, b: torch.stack([p[1] * b[2] - p[2] * b[1], p[2] * b[0] - p[0] * b[2],   # noqa: E731
                                          p[0] * b[1] - p[1] * b[0]])
        prime = half + cross(half, t)
        v = half + cross(prime, sv) + 0.5 * kick
    else:
        v = v + kick
    return u + dt * v[:len(n)], v


def _exact_step(case, seed):
    """The step in 64 bits with a direct Poisson solve."""
    n = _nodes(case)
    lo = _box(case)[1]
    width = torch.tensor([float(k) for k in (n if case["periodic"] else _box(case)[0])], device="cuda").double()[:, None]
    parts, weight = _particles(case, seed)
    if sum(p.shape[1] for p, _ in parts) * case["steps"] * (case["order"] + 1) ** len(n) > 9e9:
        return None
    parts = [(p.sub_(lo[0]), v) for p, v in parts]
    nodes = int(np.prod(n))

    def density(pos, order):
        d = torch.zeros(nodes, dtype=torch.float64, device="cuda")
        for i in range(0, pos.shape[1], CHUNK):
            _deposit(pos[:, i:i + CHUNK], d, n, order, weight)
        return d

    for _ in range(case["steps"]):
        rho = torch.full((nodes,), 1.0 if case["species"] == 1 else 0.0, dtype=torch.float64, device="cuda")
        for (q, _, _), (pos, _) in zip(_species(case), parts):
            rho += q * density(pos, case["order"])
        phi = _poisson(rho, n, case["periodic"], pinned=_pinned(case))
        kinetic, moved = [], []
        for (q, m, _), (pos, vel) in zip(_species(case), parts):
            for i in range(0, pos.shape[1], CHUNK):
                pos[:, i:i + CHUNK], vel[:, i:i + CHUNK] = _push(pos[:, i:i + CHUNK], vel[:, i:i + CHUNK], phi, n,
                                                                 case, q / m)
            if case["periodic"]:
                torch.remainder(pos, width, out=pos)
            else:
                keep = ((pos >= 0) & (pos < width)).all(0)
                pos, vel = pos[:, keep], vel[:, keep]
            kinetic.append(0.5 * m * weight * float(sum((vel[c] * vel[c]).sum() for c in range(3))))
            moved.append((pos, vel))
        parts = moved
    p = phi.reshape(n)
    field = 0.0
    for a in range(len(n)):
        d = torch.roll(p, -1, a) - p
        if not case["periodic"]:
            d = d.narrow(a, 0, n[a] - 1)
        field += 0.5 * float((d * d).sum())
    # the right-hand side as the solve leaves it: fixed values put in, or the mean taken out
    if not case["periodic"]:
        rho[torch.from_numpy(_walls(n)).cuda()] = 0.0
    elif _pinned(case):
        rho[0] = 0.0
    else:
        rho -= rho.mean()
    out = {"rho": rho, "phi": phi, "energy": np.array(kinetic + [field])}
    if case["order"] == 1:
        out["density"] = [density(pos, 1) for pos, _ in parts]
    if case["precision"] == "fp64" and case["periodic"]:
        out["particles"] = None   # stored in the order of the last re-sort
    return out


def _exact_adjoint(case, seed):
    """Gradients of the 64-bit run by automatic differentiation."""
    pos, vel, phi_ext, weight = _adjoint_inputs(case, seed)
    if pos.shape[1] * case["steps"] > 1e8:
        return None
    n = _nodes(case)
    v = vel.double().requires_grad_(True)
    pe = phi_ext.clone().requires_grad_(True)
    u, w = pos - 0.5, v
    dt = 0.1
    width = torch.tensor([[float(k)] for k in n], dtype=torch.float64, device="cuda")

    def field(u):
        axes = [_weights(u[a], 1) for a in range(2)]
        rho = torch.full((n[0] * n[1],), 1.0, dtype=torch.float64, device="cuda")
        for tap in _taps(1, 2):
            rho = rho.index_add(0, _node([x[0] for x in axes], tap, n), -weight * axes[0][1][tap[0]] * axes[1][1][tap[1]])
        return _poisson(rho, n, True, pinned=True) + pe

    for _ in range(case["steps"]):
        phi = field(u)
        axes = [_weights(u[a], 1) for a in range(2)]
        gx = gy = 0.0
        for tap in _taps(1, 2):
            f = phi[_node([x[0] for x in axes], tap, n)]
            gx = gx + f * axes[0][2][tap[0]] * axes[1][1][tap[1]]
            gy = gy + f * axes[0][1][tap[0]] * axes[1][2][tap[1]]
        w = torch.cat([w[:2] + dt * torch.stack([gx, gy]), w[2:]])   # q/m = -1, E = -gradient
        u = torch.remainder(u + dt * w[:2], width)
    p = field(u).reshape(n)
    loss = sum(((torch.roll(p, -1, a) - p) ** 2).sum() for a in range(2))
    loss.backward()
    return {"loss": loss.detach(), "velocity_gradient": v.grad, "field_gradient": pe.grad}
