"""The performance cases: what a particle-in-cell program has this library do
for it, through the public Python binding (`minipic_b200`).

All cases run on Kuhn meshes of the 0.1 m box (n^3 hexes of 6 tets, optionally
minus a centred r = 0.02 m sphere at -10 V), O+ ions with a 7 km/s drift and a
0.1 eV Maxwellian, n0 = 1e10 m^-3, kTe = 2 eV: the benchmark configurations'
plasma.  Kinds:

  push     InjectIons + MoveParticles: one batch of inlet ions appended, one
           push + walk + density scatter; the tet re-sort every 10 steps.  The
           population is seeded at the beam's steady state and stays there, so
           a pass is one step of a running simulation.
  newton   FESolver::computePhi, the Lapack method: one Newton step of the
           Poisson-Boltzmann problem from a given potential and ion density
           (noise: volts of fluctuation on the potential; the density's
           relative fluctuation is twice the number).
  gs       the same with the reference's Gauss-Seidel inner solver.
  sparse   the same on a mesh past dense storage (sparse K, conjugate gradients).
  adjoint  K push + scatter steps forward and their vector-Jacobian product.
  step     a whole time step: injection, push, Newton step, updateEf.

`run` returns the library's own device buffers where it has them (node density,
potential, field) and the step's counts.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mini-fem-pic-main_b200"))
import minipic_b200 as mp  # noqa: E402
from minipic_b200 import adjoint as mp_adjoint  # noqa: E402
from minipic_b200 import kuhn  # noqa: E402

L = 0.1                      # box length [m]
SPHERE = (50.0, 50.0, 50.0, 20.0)  # centre, radius [mm]
SPHERE_PHI = -10.0           # [V]
WALL_PHI = -5.0              # [V] on x = L (0 V on x = 0)
N0 = 1e10                    # electron and plasma density [m^-3]
KTE = 2.0                    # [eV]
DRIFT = 7000.0               # [m/s]
QE, AMU, EPS0 = 1.602e-19, 1.660538921e-27, 8.8541878e-12
MASS = 16 * AMU
QM = QE / MASS
SIGMA = math.sqrt(0.1 * QE / MASS)  # 0.1 eV Maxwellian, per component
BATCHES = 8                  # inlet batches a push state cycles through


def listed():
    return [
        # the small FP64 configuration's step: 50k ions, launches and latency
        dict(name="push_fp64_8h_50k", kind="push", n=8, sphere=False, ions=50_000, form="fp64", dt=1e-7),
        # the FP64 throughput configuration
        dict(name="push_fp64_20h_2M", kind="push", n=20, sphere=False, ions=2_000_000, form="fp64", dt=5e-8),
        # the same in the mixed-precision particle form
        dict(name="push_mixed_20h_2M", kind="push", n=20, sphere=False, ions=2_000_000, form="mixed", dt=5e-8),
        # the headline's population: many more ions than the caches hold, a cavity
        dict(name="push_mixed_sphere32h_48M", kind="push", n=32, sphere=True, ions=48_000_000, form="mixed", dt=5e-8),
        # field solve of the small configuration: 567 unknowns
        dict(name="newton_fp64_8h", kind="newton", n=8, sphere=False, form="fp64", noise=0.05),
        # field solve of the FP64 throughput configuration: 8,379 unknowns
        dict(name="newton_fp64_20h", kind="newton", n=20, sphere=False, form="fp64", noise=0.05),
        # the headline's field solve: 32,244 unknowns
        dict(name="newton_mixed_sphere32h", kind="newton", n=32, sphere=True, form="mixed", noise=0.05),
        # the reference's Gauss-Seidel method at a size where its test asks for many sweeps
        dict(name="gs_12h", kind="gs", n=12, sphere=False, form="fp64", noise=0.05),
        # a mesh that dense storage cannot hold: 255,822 unknowns
        dict(name="sparse_sphere64h", kind="sparse", n=64, sphere=True, form="fp64", noise=0.05),
        # the adjoint configuration: 20 steps, a checkpoint every 5
        dict(name="adjoint_16h_1M", kind="adjoint", n=16, ions=1_000_000, steps=20, every=5, dt=1e-7),
        # whole steps: the small configuration and the headline
        dict(name="step_fp64_8h_50k", kind="step", n=8, sphere=False, ions=50_000, form="fp64", dt=1e-7),
        dict(name="step_mixed_sphere32h_48M", kind="step", n=32, sphere=True, ions=48_000_000, form="mixed", dt=5e-8),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(("push", "push", "newton", "newton", "gs", "sparse", "adjoint", "step"))
    form = rng.choice(("fp64", "mixed"))
    noise = round(rng.uniform(0.01, 0.1), 4)
    if kind == "gs":
        return dict(kind=kind, n=rng.randint(5, 15), sphere=False, form="fp64", noise=noise)
    if kind == "sparse":
        n = round(_log(rng, 12, 60))
        return dict(kind=kind, n=n, sphere=rng.random() < 0.5, form="fp64", noise=noise)
    if kind == "adjoint":
        return dict(kind=kind, n=rng.randint(6, 20), ions=round(_log(rng, 2e4, 1.5e6)), steps=rng.randint(5, 20),
                    every=rng.randint(2, 8), dt=rng.choice((5e-8, 1e-7)))
    n = round(_log(rng, 5, 32 if form == "mixed" else 24))
    sphere = n >= 10 and rng.random() < 0.5
    if kind == "newton":
        return dict(kind=kind, n=n, sphere=sphere, form=form, noise=noise)
    ions = round(_log(rng, 8e3, 3e7 if kind == "push" else 5e6))
    return dict(kind=kind, n=n, sphere=sphere, ions=ions, form=form, dt=rng.choice((5e-8, 1e-7)))


# ---- what a program sets up once ---------------------------------------------------

@functools.lru_cache(maxsize=24)
def _deck(n, sphere):
    """The mesh as a program holds it after reading its files."""
    kd = kuhn.build(n, sphere=SPHERE if sphere else None)
    mesh = mp.Mesh.build(kd.nodes_mm / 1000.0, kd.tets, kd.inlet_nodes, kd.inlet_tris,
                         np.concatenate([kd.wall_nodes, kd.sphere_nodes]), device=0)
    params = mp.Parameters(plasma_den=N0, ion_velocity=DRIFT, electron_temperature=KTE / mp.KB,
                           wall_potential=-WALL_PHI, plasma_species="Oxygen", fesolver_method=mp.LAPACK)
    deck = mp.Deck(params, mesh, kd.sphere_nodes)
    return kd, deck, deck.fe_desc_arrays(SPHERE_PHI if sphere else None)


class _Buffer:
    """A context's FP64 device vector, for torch."""

    def __init__(self, ctx, name):
        ptr, n = ctx.device_buffer(name)
        self.ctx = ctx
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f8", data=(ptr, False), version=3)


def _view(ctx, name):
    return torch.as_tensor(_Buffer(ctx, name), device="cuda")


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uniform(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _hex(pos, n):
    """Hex corner, fractions inside it, and the fractions' descending order, of points pos [3][m]."""
    f = pos / (L / n)
    c = f.floor().long().clamp(0, n - 1)
    fr = f - c
    return c, fr, torch.argsort(fr, dim=0, descending=True, stable=True)


_PERM = [-1] * 27
for _i, _p in enumerate(kuhn.PERMS):
    _PERM[9 * _p[0] + 3 * _p[1] + _p[2]] = _i


def _cell(kd, pos):
    """Tet of each point (-1 in the cavity)."""
    n = kd.n
    c, _, o = _hex(pos, n)
    perm = torch.tensor(_PERM, device="cuda")[9 * o[0] + 3 * o[1] + o[2]]
    at = torch.as_tensor(kd.hexperm_to_tet, device="cuda")
    return at[(c[0] + n * c[1] + n * n * c[2]) * 6 + perm].int()


def _beam(kd, g, ions):
    """pos [3][m], vel [3][m], cell [m] of about `ions` ions (a full box's worth) of the free-streaming beam
    at steady state: an ion is there if the straight line back to the inlet stays inside the mesh."""
    out = []
    done = 0
    while done < ions:
        m = min(ions - done, 8_000_000)
        done += m
        pos = _uniform(g, 3, m) * ((1 - 2e-6) * L) + 1e-6 * L
        vel = _normal(g, 3, m) * SIGMA
        vel[0] += DRIFT
        back = pos[0] / vel[0]
        keep = vel[0] > 0
        for k in (1, 2):
            from_ = pos[k] - vel[k] * back
            keep &= (from_ >= 0) & (from_ <= L)
        if kd.sphere_nodes.size:
            rel = pos - 0.5 * L
            t = ((rel * vel).sum(0) / (vel * vel).sum(0)).clamp(min=0)
            t = torch.minimum(t, back)
            keep &= (rel - vel * t).square().sum(0) > (SPHERE[3] / 1000.0 + 0.6 * L / kd.n) ** 2
        pos, vel = pos[:, keep], vel[:, keep]
        cell = _cell(kd, pos)
        inside = cell >= 0
        out.append((pos[:, inside], vel[:, inside], cell[inside]))
    return [torch.cat(x, dim=-1).contiguous() for x in zip(*out)]


def _inlet(kd, g, count):
    """A batch of ions on the inlet face."""
    pos = _uniform(g, 3, count) * ((1 - 2e-6) * L) + 1e-6 * L
    pos[0] = 0
    vel = _normal(g, 3, count) * SIGMA
    vel[0] = DRIFT + vel[0].abs()
    return pos, vel, _cell(kd, pos)


def _per_step(case):
    """Specific weight of the ions (a full box holds case["ions"]), and how many enter a step."""
    spwt = N0 * L ** 3 / case["ions"]
    return spwt, max(1, round(N0 * DRIFT * L * L * case["dt"] / spwt))


def _ramp(deck):
    """The vacuum potential between inlet and wall, at the nodes."""
    return WALL_PHI * deck.mesh.node_pos[:, 0] / L


def _potential(deck, fe, seed, noise):
    """A Newton state near the solution: (node potential, its unknowns)."""
    rng = np.random.default_rng(seed)
    uh = _ramp(deck) + noise * rng.standard_normal(deck.mesh.n_nodes)
    ID = fe["ID"]
    uh = np.where(ID >= 0, uh, fe["g"])
    d = np.zeros(fe["neq"])
    d[ID[ID >= 0]] = uh[ID >= 0]
    return uh, d


def _particles(case, seed):
    """Inputs of a particle case, on the GPU: population, inlet batches, per-tet field."""
    kd, deck, fe = _deck(case["n"], case["sphere"])
    g = _gen(seed)
    pop = _beam(kd, g, case["ions"])
    _, count = _per_step(case)
    batches = [_inlet(kd, g, count) for _ in range(BATCHES)]
    return kd, deck, fe, pop, batches


def _field(deck, seed):
    """Per-tet field of the ramp plus 20 V/m of fluctuation (numpy, [n_tets][3])."""
    rng = np.random.default_rng(seed + 77)
    ef = 20.0 * rng.standard_normal((deck.mesh.n_tets, 3))
    ef[:, 0] -= WALL_PHI / L
    return ef


def _load_particles(ctx, case, pop):
    n = pop[2].numel()
    if case["sphere"]:
        # an ion that steps into the cavity lies in no tet: its walk ends at the hop limit
        ctx.set_walk_limit(256)
        ctx.set_walk_policy(mp.WALK_LIMIT_ABSORB)
    ctx.set_track_ids(False)
    ctx.set_sort_period(10)
    ctx.reserve(int(1.25 * n) + 4096)
    ctx.append_device(pop[0].data_ptr(), pop[1].data_ptr(), pop[2].data_ptr(), n)
    ctx.sort_by_tet()
    if case["form"] == "mixed":
        ctx.set_form(mp.MIXED)


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, k=0)
    form = mp.MIXED if case.get("form") == "mixed" else mp.FP64
    if kind == "adjoint":
        kd, deck, fe = _deck(case["n"], False)
        slots = _adjoint_slots(case, seed)
        ctx = mp.Context(deck.mesh)
        dirs = deck.mesh.inlet_normal[0]
        adj = mp_adjoint.Adjoint(ctx, case["steps"], case["every"], QM, MASS, case["dt"], _per_step(case)[0], dirs,
                                 mp_adjoint.wall_nodes_of(deck.mesh), nx=fe["nx"])
        for first, injected, pos, vel, cell in slots:
            adj.add_particles(first, injected, pos.T.cpu().numpy(), vel.T.cpu().numpy(), cell.cpu().numpy())
        rng = np.random.default_rng(seed + 5)
        dev = lambda a: torch.as_tensor(a, device="cuda")  # noqa: E731
        nn = deck.mesh.n_nodes
        s |= dict(ctx=ctx, adj=adj, phi=dev(_adjoint_phi(deck, seed)), den=dev(np.zeros(nn)),
                  phi_bar=dev(np.zeros(nn)), den_bar=dev(rng.standard_normal(nn) / N0))
        torch.cuda.synchronize()
        return s
    kd, deck, fe = _deck(case["n"], case["sphere"])
    ctx = mp.Context(deck.mesh)
    s |= dict(ctx=ctx, deck=deck, form=form)
    if kind == "sparse":
        ctx.set_fe_storage(mp.FE_SPARSE)
    if kind != "push":
        ctx.fe_setup(**fe)
        s |= {k: _view(ctx, k) for k in ("d", "F1", "uh", "ef")}
    s["den"] = _view(ctx, "den")
    if kind in ("push", "step"):
        _, _, _, pop, batches = _particles(case, seed)
        torch.cuda.synchronize()
        _load_particles(ctx, case, pop)
        s |= dict(batches=batches, spwt=_per_step(case)[0])
        if kind == "push":
            ctx.fe_set("ef", _field(deck, seed))
        else:
            uh, d = _potential(deck, fe, seed, 0.05)
            ctx.fe_set("d", d)
            ctx.update_ef(uh)
            s["inj"] = mp.Injector(deck.mesh, seed=seed % 2 ** 31)
            s["seed"] = int(seed)
    else:
        g = _gen(seed)
        s["den"].copy_(N0 * (1 + 2 * case["noise"] * _normal(g, deck.mesh.n_nodes)).clamp(min=0))
        _, d = _potential(deck, fe, seed, case["noise"])
        s["d0"] = torch.as_tensor(d, device="cuda") if kind != "gs" else torch.zeros_like(s["d"])
    torch.cuda.synchronize()
    return s


METHOD = {"newton": mp.LAPACK, "step": mp.LAPACK, "gs": mp.GAUSS_SEIDEL, "sparse": mp.SPARSE_CG}


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "adjoint":
        _, st = s["adj"].forward(s["phi"], DRIFT, den_out=s["den"])
        _, v_bar = s["adj"].backward(s["den_bar"], 1e6, phi_bar_out=s["phi_bar"])
        return dict(den=s["den"], flux=st.flux, phi_bar=s["phi_bar"], v_bar=v_bar, alive=st.alive, exits=st.wall_exits)
    if kind in ("push", "step"):
        if kind == "step" and case["sphere"]:
            ctx.inject_device(s["inj"], N0, DRIFT, case["dt"], s["spwt"], SIGMA, QM, s["seed"], s["k"])
        else:
            pos, vel, cell = s["batches"][s["k"] % BATCHES]
            ctx.append_device(pos.data_ptr(), vel.data_ptr(), cell.data_ptr(), cell.numel(), True, QM,
                              0.5 * case["dt"])
        st = ctx.push(QM, case["dt"], s["spwt"])
        s["k"] += 1
        out = dict(den=s["den"], before=st.n_before, after=st.n_after, hops=st.total_hops)
        if kind == "push":
            return out
    else:
        out = {}
        s["d"].copy_(s["d0"])
    # a fresh assembly of the load vector, as FESolver::startAssembly leaves it
    s["F1"].zero_()
    torch.cuda.current_stream().synchronize()  # the context has a stream of its own
    st = ctx.compute_phi(METHOD[kind], s["form"])
    out |= dict(d=s["d"], uh=s["uh"])
    if kind == "gs":
        out["sweeps"] = st.linear_iterations
    if kind == "step":
        ctx.update_ef()
        out["ef"] = s["ef"]
    return out


# ---- the adjoint's inputs ----------------------------------------------------------

def _adjoint_phi(deck, seed):
    x, y, z = (deck.mesh.node_pos[:, k] / L for k in range(3))
    amp = 0.5 + 0.1 * np.random.default_rng(seed).standard_normal()
    return WALL_PHI * x + amp * np.sin(np.pi * x) * np.sin(np.pi * y) * np.sin(np.pi * z)


def _adjoint_slots(case, seed):
    """(first step, injected, pos, vel, cell): the initial population and a batch for each step, whose
    velocities are the thermal part alone."""
    kd, _, _ = _deck(case["n"], False)
    g = _gen(seed)
    out = [(0, False, *_beam(kd, g, case["ions"]))]
    _, count = _per_step(case)
    for k in range(case["steps"]):
        pos, vel, cell = _inlet(kd, g, count)
        vel[0] -= DRIFT
        out.append((k, True, pos, vel, cell))
    return out


# ---- work --------------------------------------------------------------------------

def _counts(case):
    n = case["n"]
    nodes, tets, unknowns = (n + 1) ** 3, 6 * n ** 3, (n - 1) * (n + 1) ** 2
    if case.get("sphere"):
        out = 1 - 4 / 3 * math.pi * (SPHERE[3] / 100) ** 3
        nodes, tets, unknowns = round(nodes * out), round(tets * out), round(unknowns * out * 0.97)
    return nodes, tets, unknowns


def work(case):
    kind = case["kind"]
    nodes, tets, unknowns = _counts(case)
    size, record = (4, 96) if case.get("form") == "mixed" else (8, 192)
    particles = newton = dict(bytes=0, flops=0)
    if kind in ("push", "step"):
        # position, velocity, tet: in and out; the tets' records and the density once
        m = case["ions"]
        particles = dict(bytes=m * 2 * (6 * size + 4) + tets * record + nodes * 8, flops=m * 70)
    if kind == "adjoint":
        # a slot's state in, its weights out, and once more for the reverse pass
        m = case["ions"]
        return dict(bytes=2 * (m * 52 + tets * 192 + nodes * 16), flops=m * case["steps"] * 200)
    if kind != "push":
        # K's nonzeros (value and column), the load's tets, d, F0, F1 and the density in, d, F1 and uh out;
        # a solution touches every nonzero at least once
        nnz = 15 * unknowns
        newton = dict(bytes=nnz * 12 + tets * 24 + unknowns * 48 + nodes * 24, flops=nnz * 4 + unknowns * 40)
        if kind == "step":
            newton["bytes"] += tets * (16 + 96 + 24)
    return {k: particles[k] + newton[k] for k in ("bytes", "flops")}


# ---- the same results in plain 64-bit torch ------------------------------------------

def _scatter(pos, n, den):
    """Adds the barycentric weights of points pos [3][m] of the box's Kuhn mesh to den [(n+1)^3]."""
    step = torch.tensor([1, n + 1, (n + 1) ** 2], device="cuda")
    for p in pos.split(8_000_000, dim=1):
        c, fr, o = _hex(p, n)
        f = torch.gather(fr, 0, o)
        at = (c * step[:, None]).sum(0)
        w = (1 - f[0], f[0] - f[1], f[1] - f[2], f[2])
        for k in range(4):
            den.index_add_(0, at, w[k])
            if k < 3:
                at = at + step[o[k]]


def _inside(pos):
    return ((pos >= 0) & (pos <= L)).all(0)


def _node_volume(deck):
    con = torch.as_tensor(deck.mesh.con, device="cuda").long()
    x = torch.as_tensor(deck.mesh.node_pos, device="cuda")[con]
    vol = torch.linalg.det(x[:, 1:] - x[:, :1]).abs() / 6
    out = torch.zeros(deck.mesh.n_nodes, dtype=torch.float64, device="cuda")
    for a in range(4):
        out.index_add_(0, con[:, a], vol / 4)
    return out


def _exact_push(kd, deck, case, pop, batch, ef):
    """(density, ions before, after) of one step of the box; ef [n_tets][3]."""
    spwt, _ = _per_step(case)
    pos, vel, cell = pop
    bpos, bvel, bcell = batch
    bvel = bvel - QM * ef[bcell.long()].T * (0.5 * case["dt"])
    pos, vel, cell = torch.cat([pos, bpos], 1), torch.cat([vel, bvel], 1), torch.cat([cell, bcell])
    pos = pos + (vel + QM * ef[cell.long()].T * case["dt"]) * case["dt"]
    keep = _inside(pos)
    den = torch.zeros(deck.mesh.n_nodes, dtype=torch.float64, device="cuda")
    _scatter(pos[:, keep], case["n"], den)
    return den * spwt / _node_volume(deck), cell.numel(), int(keep.sum())


def _shape(deck):
    """Gradients [n_tets][4][3] of the tets' linear shape functions and det J, in FESolver's convention."""
    con = torch.as_tensor(deck.mesh.con, device="cuda").long()
    x = torch.as_tensor(deck.mesh.node_pos, device="cuda")[con]
    J = (x[:, :3] - x[:, 3:]).transpose(1, 2)  # dx_i/dxi_j
    inv = torch.linalg.inv(J)
    return con, torch.cat([inv, -inv.sum(1, keepdim=True)], 1), torch.linalg.det(J)


class _Field:
    """K, F0 and the quadrature weights of the Poisson-Boltzmann problem (K as row, column, value)."""

    def __init__(self, deck, fe):
        con, nx, det = _shape(deck)
        self.ID = torch.as_tensor(fe["ID"], device="cuda").long()
        self.g = torch.as_tensor(fe["g"], device="cuda")
        self.neq = n = fe["neq"]
        LM = self.ID[con]
        self.F0 = torch.zeros(n, dtype=torch.float64, device="cuda")
        self.w = torch.zeros_like(self.F0)  # sum of the quadrature weights of an unknown's shape functions
        row, col, val = [], [], []
        for a in range(4):
            ok = LM[:, a] >= 0
            # FESolver integrates its load terms over the unit cube
            self.w.index_add_(0, LM[ok, a], (0.5 if a < 3 else -0.5) * det[ok])
            for b in range(4):
                ke = 8 * (nx[:, a] * nx[:, b]).sum(1) * det
                both = ok & (LM[:, b] >= 0)
                row.append(LM[both, a])
                col.append(LM[both, b])
                val.append(ke[both])
                self.F0.index_add_(0, LM[ok, a], -(ke * self.g[con[:, b]])[ok])
        self.K = torch.sparse_coo_tensor(torch.stack([torch.cat(row), torch.cat(col)]), torch.cat(val), (n, n)).coalesce()
        self.con, self.nx = con, nx

    def terms(self, den, d):
        """G = K d - F0 - F1 and FP of J = K - diag(FP)."""
        ex = torch.exp(d / KTE)
        node = torch.zeros(self.neq, dtype=torch.float64, device="cuda")
        node[self.ID[self.ID >= 0]] = den[self.ID >= 0]
        F1 = QE / EPS0 * (node + N0 * ex) * self.w
        FP = -QE / EPS0 * N0 * ex / KTE * self.w
        return torch.mv(self.K, d) - self.F0 - F1, FP

    def dense(self, FP):
        J = self.K.to_dense()
        J.diagonal().sub_(FP)
        return J

    def uh(self, d):
        u = self.g.clone()
        u[self.ID >= 0] += d[self.ID[self.ID >= 0]]
        return u

    def ef(self, uh):
        return -(self.nx * uh[self.con][:, :, None]).sum(1)


def _newton(f, den, d):
    """d after one Newton step with an accurate linear solve."""
    G, FP = f.terms(den, d)
    Jv = lambda v: torch.mv(f.K, v) - FP * v  # noqa: E731
    if f.neq <= 33_000:
        lu = torch.linalg.lu_factor(f.dense(FP))
        solve = lambda r: torch.linalg.lu_solve(*lu, r[:, None])[:, 0]  # noqa: E731
    else:
        diag = torch.zeros_like(d)
        i, v = f.K.indices(), f.K.values()
        on = i[0] == i[1]
        diag[i[0][on]] = v[on]
        diag -= FP

        def solve(r):  # preconditioned conjugate gradients
            x, stop = torch.zeros_like(r), 1e-13 * float(r.norm())
            z = r / diag
            p, rz = z, torch.dot(r, z)
            for it in range(4000):
                q = Jv(p)
                a = rz / torch.dot(p, q)
                x, r = x + a * p, r - a * q
                if it % 25 == 0 and float(r.norm()) <= stop:
                    break
                z = r / diag
                rz, old = torch.dot(r, z), rz
                p = z + (rz / old) * p
            return x
    y = solve(G)
    y = y + solve(G - Jv(y))
    return d - y


def _gauss_seidel(f, den, d):
    """d after the step whose solver is Gauss-Seidel from zero, checked after sweeps 1, 26, 51, ..."""
    G, FP = f.terms(den, d)
    J = f.dense(FP)
    U = torch.triu(J, 1)
    y = torch.zeros_like(G)
    for it in range(3000):
        y = torch.linalg.solve_triangular(J, (G - torch.mv(U, y))[:, None], upper=False)[:, 0]
        if it % 25 == 0 and float((G - torch.mv(J, y)).norm()) / f.neq < 1e-4:
            return d - y, it
    return None


def exact(case, seed):
    kind = case["kind"]
    if case.get("sphere") and kind in ("push", "step"):
        return None  # where a walk meets the cavity, the ion's end is the walk's, not geometry's
    kd, deck, fe = _deck(case["n"], bool(case.get("sphere")))
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    if kind == "push":
        _, _, _, pop, batches = _particles(case, seed)
        den, before, after = _exact_push(kd, deck, case, pop, batches[0],
                                         torch.as_tensor(_field(deck, seed), device="cuda"))
        return dict(den=den, before=before, after=after, hops=None)
    f = _Field(deck, fe)
    if kind == "step":
        uh, d = _potential(deck, fe, seed, 0.05)
        _, _, _, pop, batches = _particles(case, seed)
        den, before, after = _exact_push(kd, deck, case, pop, batches[0], f.ef(torch.as_tensor(uh, device="cuda")))
        d = _newton(f, den, torch.as_tensor(d, device="cuda"))
        uh = f.uh(d)
        return dict(den=den, before=before, after=after, hops=None, d=d, uh=uh, ef=f.ef(uh).reshape(-1))
    den = N0 * (1 + 2 * case["noise"] * _normal(_gen(seed), deck.mesh.n_nodes)).clamp(min=0)
    d = torch.as_tensor(_potential(deck, fe, seed, case["noise"])[1], device="cuda")
    if kind == "gs":
        got = _gauss_seidel(f, den, torch.zeros_like(d))
        return None if got is None else dict(d=got[0], uh=f.uh(got[0]), sweeps=got[1])
    d = _newton(f, den, d)
    return dict(d=d, uh=f.uh(d))


def _exact_adjoint(case, seed):
    """The forward's density; the exits' faces, and with them the rest, are the walk's."""
    kd, deck, _ = _deck(case["n"], False)
    con, nx, _ = _shape(deck)
    phi = torch.as_tensor(_adjoint_phi(deck, seed), device="cuda")
    ef = -(nx * phi[con][:, :, None]).sum(1)
    kick = QM * case["dt"]
    pos = vel = None
    slots = _adjoint_slots(case, seed)
    for k in range(case["steps"]):
        for first, injected, p, v, c in slots:
            if first != k:
                continue
            if injected:
                v = v.clone()
                v[0] += DRIFT
                v = v - 0.5 * kick * ef[c.long()].T
            pos, vel = (p, v) if pos is None else (torch.cat([pos, p], 1), torch.cat([vel, v], 1))
        vel = vel + kick * ef[_cell(kd, pos).long()].T
        pos = pos + vel * case["dt"]
        keep = _inside(pos)
        pos, vel = pos[:, keep], vel[:, keep]
    den = torch.zeros(deck.mesh.n_nodes, dtype=torch.float64, device="cuda")
    _scatter(pos, case["n"], den)
    return dict(den=den * _per_step(case)[0] / _node_volume(deck), flux=None, phi_bar=None, v_bar=None,
                alive=int(keep.sum()), exits=None)
