"""The work that a user of this package has it do, as timed cases.

The package solves the vertical columns of a TIE-GCM grid: batches of
tridiagonal and block-tridiagonal systems (Plan, trsolv_dev, blksolve_dev,
and solve_host on host arrays), the column routines that assemble and solve
them (dt_ng, minor_ng, comp_ng, settei_ng, oplus_ng) and one whole
dynamics_ng step of those routines (DynamicsStep).  A case is one call, or
the few calls a time step makes, on one of the model's grids:

  solve     one batch of systems through trsolv_dev / blksolve_dev
  plan      every system of a step of one workload (its grid, or the grid and
            its nests with their sub-steps) through one Plan
  host      the same systems of one grid on page-locked host arrays (solve_host)
  routine   one column routine with its post-solve steps, fields on the device
  dynamics  one dynamics_ng step as a CUDA graph, on a nest or the global grid

Grids are the model's: 29, 57 or 113 levels, 5 to 0.625 degree global grids
and nests of a few thousand columns with two ghost points on each side.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch


def _package():
    """The package directory's name is no Python identifier: load it by path."""
    name = "tiegcm_ng_b200"
    if name not in sys.modules:
        root = os.path.join(os.getcwd(), "tiegcm3.0_ng_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(root, "__init__.py"),
                                                      submodule_search_locations=[root])
        sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[name])
    return sys.modules[name]


tg = _package()
synth, batch, dynamics = tg.synth, tg.batch, tg.dynamics
DZ = {29: 0.5, 57: 0.25, 113: 0.125}     # level spacing in scale heights
DS, DS2 = 0.95, 0.5 * (1.0 - 0.95)       # the model's time-filter weights
PROFILES = 1024                          # distinct synthetic columns of a routine's fields


def listed():
    return [
        # one temperature solve of the 5 degree model: the smallest call, all latency
        dict(name="solve_5deg", what="solve", nlon=72, nlat=36, ghost=0, nk=29, block=0, column=False, refine=False),
        # the O2/O/He block solve of comp_ng on a nest, upper boundary row included
        dict(name="blocks3_nest1", what="solve", nlon=97, nlat=65, ghost=2, nk=57, block=3, column=False,
             refine=False),
        # the column step of the 2.5 degree grid: seven scalar systems and one 2x2 block system
        dict(name="step_2.5deg", what="plan", grid="global2.5", nests=0, block=2, refine=False),
        # the same on the 1.25 degree grid with 113 levels and diffusion over seven decades
        dict(name="step_1.25deg", what="plan", grid="global1.25", nests=0, block=2, refine=False),
        # the 2.5 degree grid and its three nests, up to 16 sub-steps of each in one batch
        dict(name="nested", what="plan", grid="global2.5", nests=16, block=2, refine=False),
        # the mixed-precision path of the same systems
        dict(name="nested_refine", what="plan", grid="global2.5", nests=4, block=2, refine=True),
        # a Fortran caller's whole column step of one nest: host arrays in, host arrays out
        dict(name="host_nest2", what="host", nlon=65, nlat=49, ghost=2, nk=57, block=2),
        # single routines: the 1.25 degree grid, the 2.5 degree grid, a nest
        dict(name="minor_1.25deg", what="routine", routine="minor", nlon=288, nlat=144, nk=113),
        dict(name="comp_1.25deg", what="routine", routine="comp", nlon=288, nlat=144, nk=113),
        dict(name="settei_2.5deg", what="routine", routine="settei", nlon=144, nlat=72, nk=57),
        # a whole step of the innermost nest, which runs 512 times per model step
        dict(name="dynamics_nest3", what="dynamics", nlon=52, nlat=33, nk=57, ring=False),
        # a whole step of the 2.5 degree global grid with its polar filter
        dict(name="dynamics_2.5deg", what="dynamics", nlon=144, nlat=72, nk=57, ring=True),
    ]


def draw(rng):
    def span(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    what = rng.choice(["solve", "plan", "host", "routine", "routine", "routine", "dynamics"])
    nk = rng.choice([29, 57, 57, 113])
    if what == "solve":
        return dict(what=what, nlon=span(30, 288), nlat=span(16, 144), ghost=rng.choice([0, 2]), nk=nk,
                    block=rng.choice([0, 0, 2, 3]), column=rng.random() < 0.2, refine=rng.random() < 0.2)
    if what == "plan":
        grid = rng.choice(["global5", "global2.5", "global2.5", "global2.5", "global1.25"])
        nests = rng.randint(1, 16) if grid == "global2.5" else 0
        return dict(what=what, grid=grid, nests=nests, block=rng.choice([0, 2, 2, 3] if nests < 12 else [0, 2]),
                    refine=rng.random() < (0.3 if nests < 5 else 0.))
    if what == "host":
        return dict(what=what, nlon=span(24, 72), nlat=span(16, 52), ghost=2, nk=rng.choice([29, 57]),
                    block=rng.choice([0, 2, 3]))
    if what == "routine":
        return dict(what=what, routine=rng.choice(["dt", "minor", "comp", "settei", "oplus"]),
                    nlon=span(40, 288), nlat=span(24, 144), nk=nk)
    if rng.random() < 0.2:
        return dict(what=what, nlon=72, nlat=36, nk=29, ring=True)
    return dict(what=what, nlon=span(36, 120), nlat=span(24, 70), nk=rng.choice([29, 57]), ring=False)


# ---- what a caller has in hand ---------------------------------------------
def _ncol(case):
    g = 2 if case["what"] in ("routine", "dynamics") else case["ghost"]
    return (case["nlon"] + 2 * g) * (case["nlat"] + 2 * g)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


LAWS = {"global5": dict(d0_range=(1e-3, 1e-2), loss=("uniform", 0.0, 1e-3), d_span=None),
        "global2.5": dict(d0_range=(1e-4, 1e-1), loss=("lognormal", -6.0, 2.0), d_span=None),
        "global1.25": dict(d0_range=(1e-4, 1e-1), loss=("lognormal", -6.0, 2.0), d_span=(1e-5, 1e2))}


def _grids(case):
    """(nlon, nlat, ghost, nk, sub-steps) of a plan case's grids."""
    if case["grid"] == "global5":
        return [(72, 36, 0, 29, 1)]
    if case["grid"] == "global1.25":
        return [(288, 144, 0, 113, 1)]
    nests = [(97, 65, 2, 57, min(4, case["nests"])), (65, 49, 2, 57, case["nests"]), (52, 33, 2, 57, case["nests"])]
    return [(144, 72, 0, 57, 1)] + (nests if case["nests"] else [])


def _solve_state(case, seed):
    nk, ncol, B = case["nk"], _ncol(case), case["block"]
    law = LAWS["global5" if nk == 29 else "global2.5"]
    ld = ncol if case["column"] else batch.pad_ld(ncol)
    g, dz = _gen(seed), DZ[nk]
    make = (lambda: batch.gen_scalar_device(nk, ncol, ld, dz, g, device="cuda", **law)) if not B else \
        (lambda: batch.gen_block_device(B, nk, ncol, ld, dz, g, device="cuda", **law))
    a, b, c, f = make()
    s = dict(a=a, b=b, c=c, f=f, ratio=None, add=None)
    if B == 3:           # comp_ng's upper boundary row u(nk) = ratio*u(nk-1) + add
        s["ratio"] = torch.empty((B, ld), dtype=torch.float64, device="cuda").uniform_(0.5, 1.5, generator=g)
        s["add"] = torch.empty((B, ld), dtype=torch.float64, device="cuda").uniform_(-0.1, 0.1, generator=g)
    if case["column"]:   # the Fortran order: level fastest within a column
        for k in ("a", "b", "c", "f", "ratio", "add"):
            s[k] = None if s[k] is None else s[k].movedim(-1, 0).contiguous()
    s["x"] = torch.zeros_like(s["f"])
    return s


def _plan_state(case, seed):
    law, B, g = LAWS[case["grid"]], case["block"], _gen(seed)
    segs, outs = [], []
    for nlon, nlat, ghost, nk, nsub in _grids(case):
        ncol = (nlon + 2 * ghost) * (nlat + 2 * ghost)
        ld, dz = batch.pad_ld(ncol), DZ[nk]
        nsys = 1 if case["grid"] == "global5" else 7
        x = torch.zeros((nsub, nsys, nk, ld), dtype=torch.float64, device="cuda")
        u = torch.zeros((nsub, nk, B, ld), dtype=torch.float64, device="cuda") if B else None
        for sub in range(nsub):
            for i in range(nsys):
                a, b, c, f = batch.gen_scalar_device(nk, ncol, ld, dz, g, device="cuda", **law)
                segs.append(dict(kind=tg.TG_KIND_SCALAR, nk=nk, k2=nk, ncol=ncol, ld=ld, a=a, b=b, c=c, f=f,
                                 x=x[sub, i]))
            if B:
                a, b, c, f = batch.gen_block_device(B, nk, ncol, ld, dz, g, device="cuda", **law)
                segs.append(dict(kind=B, nk=nk, k2=nk, ncol=ncol, ld=ld, a=a, b=b, c=c, f=f, x=u[sub]))
        outs += [v[..., :ncol] for v in (x, u) if v is not None]
    return dict(segs=segs, outs=outs)


def _host_state(case, seed):
    nk, ncol, B = case["nk"], _ncol(case), case["block"]
    law = dict(d0_range=(1e-4, 1e-1), loss=("lognormal", -6.0, 2.0))
    made = [(0, synth.scalar_system(nk, ncol, DZ[nk], 100 * seed + i, **law)) for i in range(7)]
    if B:
        made.append((B, synth.block_system(B, nk, ncol, DZ[nk], 100 * seed + 50, **law)))
    # one page-locked arena, every array on a 256-byte boundary, each system's solution after its inputs
    sizes = [(v.nbytes + 255) // 256 * 256 for _, arrs in made for v in (*arrs, arrs[3])]
    arena = torch.empty(sum(sizes), dtype=torch.uint8, pin_memory=True)
    buf, off, systems = arena.numpy(), 0, []
    for kind, arrs in made:
        views = []
        for v in (*arrs, np.zeros_like(arrs[3])):
            w = np.ndarray(v.shape, dtype=np.float64, buffer=buf, offset=off, order="F")
            np.copyto(w, v)
            views.append(w)
            off += (v.nbytes + 255) // 256 * 256
        systems.append(dict(kind=kind, a=views[0], b=views[1], c=views[2], f=views[3], x=views[4]))
    return dict(arena=arena, systems=systems)


def _fields(host, ncol, ld, nk, seed):
    """A routine's fields on the device, level-major with column stride ld:
    every column is one of the synthetic profiles, the same one in all fields."""
    pick = torch.randint(0, PROFILES, (ncol,), generator=_gen(seed), device="cuda")
    out = {}
    for k, v in host.items():
        v = np.asarray(v)
        if k in ("expz", "difk", "dift", "zpint"):
            out[k] = torch.from_numpy(np.ascontiguousarray(v)).cuda()
            continue
        v = np.moveaxis(v, 1, 2) if k == "fs" else v
        t = torch.from_numpy(np.ascontiguousarray(v)).cuda()
        out[k] = torch.zeros((*t.shape[:-1], ld), dtype=torch.float64, device="cuda")
        out[k][..., :ncol] = t[..., pick]
    return out


def _routine_state(case, seed):
    nk, ncol, r = case["nk"], _ncol(case), case["routine"]
    ld, dz, g = batch.pad_ld(ncol), DZ[nk], _gen(seed + 1)
    made = getattr(synth, r + "_inputs")(nk, PROFILES, dz, seed)
    host = dict(made[0], qtotal0=made[2]) if r == "settei" else made[0]
    F = _fields(host, ncol, ld, nk, seed)
    z = lambda *n: torch.zeros((*n, nk, ld), dtype=torch.float64, device="cuda")  # noqa: E731
    near = lambda t, e: t * torch.empty_like(t).uniform_(1 - e, 1 + e, generator=g)  # noqa: E731
    s = dict(F=F, C=made[1], ld=ld, x=z(), nm=z())
    mask = dynamics.Grid(nk, case["nlon"], case["nlat"], dz).boundary_mask()
    mask = torch.from_numpy(np.pad(mask, (0, ld - ncol))).cuda()
    cur = {"dt": "tn", "minor": "ftm1_smooth", "oplus": "op"}.get(r)
    if cur:
        s["post"] = dict(cur=near(F[cur], 0.02) if r == "minor" else F[cur], prev=near(F[cur], 0.01), nm_upd=s["nm"],
                         bnd_mask=mask, bnd=near(F[cur], 0.03), dtsmooth=DS, dtsmooth_div2=DS2)
    if r == "oplus":
        s.update(xiop2p=z(), xiop2d=z(), Fe=z(), Fn=z())
    if r == "settei":
        s.update(ti=z(), qtotal=z())
    if r == "comp":
        s["x"] = z(3)
    return s


_capture_stream = None


def _dynamics_state(case, seed):
    global _capture_stream
    if _capture_stream is None:
        _capture_stream = torch.cuda.Stream()
    grid, ring = _dyn_grid(case)
    step = dynamics.DynamicsStep(grid, dynamics.synthetic_inputs(grid, seed), ring=ring)
    _capture_stream.wait_stream(torch.cuda.current_stream())
    step.capture(_capture_stream)
    torch.cuda.current_stream().wait_stream(_capture_stream)
    return dict(step=step, ncol=grid.ncol)


def _dyn_grid(case):
    nlon, nlat, nk = case["nlon"], case["nlat"], case["nk"]
    if case["ring"]:
        return dynamics.Grid(nk, nlon, nlat, DZ[nk]), synth.RING_CHUNKS[(nlon, nlat)]
    return dynamics.Grid(nk, nlon, nlat, DZ[nk], lat0_deg=20.0, dlat_deg=0.15625), None


def prepare(case, seed):
    what = case["what"]
    if what == "plan":
        s = _plan_state(case, seed)
        s["plan"] = tg.Plan(s["segs"], tg.TG_PREC_F32_REFINE if case["refine"] else tg.TG_PREC_F64)
    else:
        s = {"solve": _solve_state, "host": _host_state, "routine": _routine_state,
             "dynamics": _dynamics_state}[what](case, seed)
    s["case"] = dict(case)
    return s


# ---- one pass ---------------------------------------------------------------
def run(state):
    case = state["case"]
    what, st = case["what"], torch.cuda.current_stream()
    if what == "solve":
        nk, ncol, B, s = case["nk"], _ncol(case), case["block"], state
        layout = tg.TG_LAYOUT_COLUMN if case["column"] else tg.TG_LAYOUT_LEVEL
        prec = tg.TG_PREC_F32_REFINE if case["refine"] else tg.TG_PREC_F64
        ld = s["f"].shape[-1] if not case["column"] else ncol
        if B:
            tg.blksolve_dev(B, s["a"], s["b"], s["c"], s["f"], s["x"], nk, nk - 1 if B == 3 else nk, ncol, s["ratio"],
                            s["add"], layout, ld, prec, stream=st)
        else:
            tg.trsolv_dev(s["a"], s["b"], s["c"], s["f"], s["x"], nk, nk, ncol, layout, ld, prec, stream=st)
        return s["x"] if case["column"] else s["x"][..., :ncol]
    if what == "plan":
        state["plan"].execute(st)
        return state["outs"]
    if what == "host":
        tg.solve_host(state["systems"])
        return [q["x"] for q in state["systems"]]
    if what == "dynamics":
        state["step"].replay(st)
        return {k: v[:, :state["ncol"]] for k, v in state["step"].outputs().items()}
    s, nk, ncol, ld, r = state, case["nk"], _ncol(case), state["ld"], case["routine"]
    if r == "dt":
        tg.dt_ng_post_dev(s["F"], s["C"], s["x"], nk, ncol, ld, s["post"], stream=st)
    elif r == "minor":
        tg.minor_ng_post_dev(s["F"], s["C"], s["x"], nk, ncol, ld, s["post"], stream=st)
    elif r == "comp":
        tg.comp_ng_dev(s["F"], s["C"], s["x"], nk, ncol, ld, stream=st)
        return s["x"][..., :ncol]
    elif r == "settei":
        s["qtotal"].copy_(s["F"]["qtotal0"])      # the heating that this step's settei_ng adds to
        tg.settei_ng_dev(s["F"], s["C"], s["x"], s["ti"], s["qtotal"], nk, ncol, ld, stream=st)
        return [v[:, :ncol] for v in (s["x"], s["ti"], s["qtotal"])]
    else:
        tg.oplus_ng_post_dev(s["F"], s["C"], s["x"], s["xiop2p"], s["xiop2d"], nk, ncol, ld, s["post"], Fe=s["Fe"],
                             Fn=s["Fn"], stream=st)
        return [s[k][:, :ncol] for k in ("x", "nm", "xiop2p", "xiop2d", "Fe", "Fn")]
    return [s["x"][:, :ncol], s["nm"][:, :ncol]]


# ---- what one pass cannot do without ----------------------------------------
# per level and column: fields read, fields written, operations (a power or an exponential counts as one)
ROUTINES = {"dt": (22, 2, 130), "minor": (14, 2, 260), "comp": (27, 3, 700), "settei": (28, 3, 300),
            "oplus": (28, 6, 220)}
FLOPS = {0: 8, 2: 70, 3: 210}     # per row of a system: the elimination and the back sweep


def _row_bytes(B):
    return 40 if not B else 8 * (3 * B * B + 2 * B)


def work(case):
    what = case["what"]
    if what == "plan":
        rows = [(nk * (nlon + 2 * g) * (nlat + 2 * g) * nsub) for nlon, nlat, g, nk, nsub in _grids(case)]
        per = [(0, 1 if case["grid"] == "global5" else 7)] + ([(case["block"], 1)] if case["block"] else [])
        return dict(bytes=sum(rows) * sum(n * _row_bytes(B) for B, n in per),
                    flops=sum(rows) * sum(n * FLOPS[B] for B, n in per))
    n = case["nk"] * _ncol(case)
    if what == "solve":
        return dict(bytes=n * _row_bytes(case["block"]), flops=n * FLOPS[case["block"]])
    if what == "host":
        per = [(0, 7)] + ([(case["block"], 1)] if case["block"] else [])
        return dict(bytes=n * sum(m * _row_bytes(B) for B, m in per), flops=n * sum(m * FLOPS[B] for B, m in per))
    if what == "routine":
        i, o, fl = ROUTINES[case["routine"]]
        return dict(bytes=8 * n * (i + o), flops=n * fl)
    # the step's own inputs (dt 18, settei 28, minor 4 x 12, oplus 27, comp 25) and results (2, 3, 8, 4, 6)
    return dict(bytes=8 * n * (146 + 23), flops=n * (130 + 300 + 4 * 260 + 220 + 10 * 30 + 700 + 19 * 20))


# ---- the same in 64 bits, from the formulas alone ---------------------------
def _thomas(a, b, c, f, k2):
    x = torch.zeros_like(f)
    w2, w3 = [c[0] / b[0]], [f[0] / b[0]]
    for k in range(1, k2):
        w1 = b[k] - a[k] * w2[-1]
        w2.append(c[k] / w1)
        w3.append((f[k] - a[k] * w3[-1]) / w1)
    x[k2 - 1] = w3[-1]
    for k in range(k2 - 2, -1, -1):
        x[k] = w3[k] - w2[k] * x[k + 1]
    return x


def _inverse(m):
    """Inverse of a 2x2 or 3x3 matrix of columns, [i][j] lists: adjugate over determinant."""
    if len(m) == 2:
        d = m[0][0] * m[1][1] - m[0][1] * m[1][0]
        return [[m[1][1] / d, -m[0][1] / d], [-m[1][0] / d, m[0][0] / d]]
    cof = [[m[(i + 1) % 3][(j + 1) % 3] * m[(i + 2) % 3][(j + 2) % 3] -
            m[(i + 1) % 3][(j + 2) % 3] * m[(i + 2) % 3][(j + 1) % 3] for j in range(3)] for i in range(3)]
    d = sum(m[0][j] * cof[0][j] for j in range(3))
    return [[cof[j][i] / d for j in range(3)] for i in range(3)]


def _block_thomas(P, Q, R, f, k2, ratio=None, add=None):
    """P, Q, R as [k, j, i, col], f as [k, i, col]."""
    B = f.shape[1]
    N = range(B)
    G = Z = None
    gs, zs = [], []
    for k in range(k2):
        q = [[Q[k, j, i] - (sum(P[k, n, i] * G[n][j] for n in N) if G else 0.0) for j in N] for i in N]
        v = [f[k, i] - (sum(P[k, n, i] * Z[n] for n in N) if Z else 0.0) for i in N]
        q = _inverse(q)
        G = [[sum(q[i][n] * R[k, j, n] for n in N) for j in N] for i in N]
        Z = [sum(q[i][n] * v[n] for n in N) for i in N]
        gs.append(G)
        zs.append(Z)
    u = torch.zeros_like(f)
    up = zs[-1]
    for k in range(k2 - 1, -1, -1):
        if k < k2 - 1:
            up = [zs[k][i] - sum(gs[k][i][n] * up[n] for n in N) for i in N]
        u[k] = torch.stack(up)
    if ratio is not None:
        u[k2] = ratio * u[k2 - 1] + add
    return u


def _mid_up(a):
    return torch.cat([.5 * (a[:-1] + a[1:]), 1.5 * a[-1:] - .5 * a[-2:-1]])


def _below(first, a):
    """Interface means with a given lowest value."""
    return torch.cat([first[None], .5 * (a[:-1] + a[1:])])


def _dt(F, C):
    tn, w, qt, dz, tx = F["tn"], F["w"], F["qtotal"], C["dz"], C["dtx2inv"]
    ez, dift, nk = F["expz"][:, None], F["dift"][:, None], F["tn"].shape[0]
    v = torch.cat([((tn[0] - F["t_lbc"]) * w[0] * 2.)[None], (tn[1:-1] - tn[:-2]) * w[1:-1], torch.zeros_like(tn[:1])])
    adv = F["horadv"] + torch.cat([.5 * (v[:-1] + v[1:]), v[-1:]]) / dz
    cpi, kmi, wi, qs = (_mid_up(F[k]) for k in ("cp", "km", "w", "qtotal"))
    rhs = cpi * (adv - tx * F["tnsmooth"]) * ez
    shear = []
    for u, lbc in ((F["un"], F["ulbc"]), (F["vn"], F["vlbc"])):
        d = torch.empty_like(tn)
        d[1:nk - 2] = (u[2:nk - 1] - u[:nk - 3]) / (2. * dz)
        d[0] = (u[0] + u[1] / 3. - 4. / 3. * lbc) / dz
        d[nk - 2] = d[nk - 3] / 3.
        d[nk - 1] = d[nk - 2] / 3.
        shear.append(d)
    rec = C["tsurplus"] * F["rkm12"] * (F["xnmbar"] * F["o1"] * C["rmassinv_o1"]) ** 2 * C["avo"] / F["mbar"]
    qm = C["grav"] * kmi / (C["p0"] * F["scht"]) * (shear[0] ** 2 + shear[1] ** 2) / ez
    rhs = rhs - (qs + F["hdt"] + rec + F["qji_tn"] + qm) * ez + F["cool_exp"]
    tni = torch.cat([F["tlbc"][None], .5 * (tn[:-2] + tn[1:-1]), tn[-2:-1]])
    h = F["schti"]
    rho = C["p0"] * C["expzmid_inv"] / (h * C["grav"]) * ez
    g = C["grav"] * (F["kt"] + h ** 2 * rho * F["cp"] * dift) / (C["p0"] * h * dz ** 2)
    f = C["grav"] ** 2 * h ** 2 * rho / (tni * C["p0"] * 2. * dz) * dift
    p = g[:-1] - f[:-1]
    q = -(g[1:] - f[1:] + g[:-1] + f[:-1])
    r = g[1:] + f[1:]
    q[-1], r[-1] = -g[nk - 2] - f[nk - 2], 0.
    q = q - ((cpi * (tx + F["cool_imp"]) + wi * C["gask"] / F["mbar"]) * ez)[:-1]
    rhs = rhs[:-1].clone()
    q[0] -= p[0]
    rhs[0] -= 2. * p[0] * F["t_lbc"]
    x = _thomas(p, q, r, rhs, nk - 1)
    return torch.cat([x, (x[-1] ** 2 / x[-2])[None]])


TAU, T00, SS = 1.86e3, 273., (1.710, 1.749, 1.718)
PHI = ((0., 1.35, 2.16, 1.11), (.673, 0., 1.616, .769), (.270, .404, 0., .322))


def _alpha(o2, o1, he, tni):
    """The 3x3 mutual-diffusion matrix of O2, O, He in N2."""
    d = [(tni / T00) ** (1.75 - s) for s in SS]
    (_, p12, p13, p14), (p21, _, p23, p24), (p31, p32, _, p34) = PHI    # species pairs of O2, O, He, N2
    c13, c23, c31, c32 = d[0] * p13 - p14, d[1] * p23 - p24, d[0] * p31 - d[2] * p34, d[1] * p32 - d[2] * p34
    return [[-(p14 + (p12 - p14) * o1 + c13 * he), (p12 - p14) * o2, c13 * o2],
            [(p21 - p24) * o1, -(p24 + (p21 - p24) * o2 + c23 * he), c23 * o1],
            [c31 * he, c32 * he, -(d[2] * p34 + c31 * o2 + c32 * o1)]]


def _lower(F, C):
    """O2, O, He at the lower boundary."""
    return [C["b"][i][0] * F["o2"][0] + C["b"][i][1] * F["o1"][0] + C["b"][i][2] * F["he"][0] + C["fb"][i]
            for i in range(3)]


def _rise(first, a, dz):
    return torch.cat([first[None], a[1:] - a[:-1]]) / dz


def _minor(F, C):
    tn, mbar, barm, dz, rmx, nk = F["tn"], F["mbar"], F["barm"], C["dzp"], C["rmx"], F["tn"].shape[0]
    phix = C["phix"]
    sal = [phix[i] - phix[3] for i in range(3)]
    lo = _lower(F, C)
    mb = 1. / (lo[0] * C["rmassinv_o2"] + lo[1] * C["rmassinv_o1"] + (1. - sum(lo)) * C["rmassinv_n2"] +
               lo[2] * C["rmassinv_he"])
    sp = [F[k] for k in ("o2", "o1", "he")]
    ps = [_below(.5 * (lo[i] + sp[i][0]), sp[i]) for i in range(3)]
    dps = [_rise(sp[i][0] - lo[i], sp[i], dz) for i in range(3)]
    dm = _rise(mbar[0] - mb, mbar, dz)
    tni = torch.cat([F["tlbc"][None], .5 * (tn[1:-1] + tn[:-2]), tn[-2:-1]])
    inv = _inverse(_alpha(ps[0], ps[1], ps[2], tni))
    mass = [C["rmass_o2"], C["rmass_o1"], C["rmass_he"]]
    ex = 1. - (rmx + dm) / barm
    for n in range(3):
        sa = sum(sal[i] * inv[i][n] for i in range(3))
        ex = ex + sa * (dps[n] - (1. - (mass[n] + dm) / barm) * ps[n])
    dm = dm / barm
    ax = -(barm / (TAU * C["rmass_n2"]) * (T00 / tni) ** 0.25 /
           (phix[2] + sal[0] * ps[0] + sal[1] * ps[1] + sal[2] * ps[2]))
    dt = torch.cat([(tni[1] - tni[0])[None], (tni[2:] - tni[:-2]) / 2., (tni[-1] - tni[-2])[None]])
    th = ex - C["alfax"] * dt / (dz * tni)
    wi, difk, ez, df = _mid_up(F["w"]), F["difk"][:, None], F["expz"][:, None], F["dfactor"]
    lo_, hi_ = C["expzmid_inv"] * difk[:-1], C["expzmid"] * difk[1:]
    ep, er = lo_ * (1. / dz - .5 * dm[:-1]), hi_ * (1. / dz + .5 * dm[1:])
    eq = lo_ * (1. / dz + .5 * dm[:-1]) + hi_ * (1. / dz - .5 * dm[1:])
    p, q, r = (torch.zeros_like(tn) for _ in range(3))
    e = ez[:-1]
    p[:-1] = ax[:-1] * (1. / dz + .5 * th[:-1]) / dz - e * (ep * df + .5 * wi[:-1]) / dz
    r[:-1] = ax[1:] * (1. / dz - .5 * th[1:]) / dz - e * (er * df - .5 * wi[:-1]) / dz
    q[:-1] = (-(ax[:-1] * (1. / dz - .5 * th[:-1]) + ax[1:] * (1. / dz + .5 * th[1:])) / dz +
              e * (eq * df / dz + C["dtx2inv"] - F["sloss"][:-1]))
    f = (F["ftm1_smooth"] * C["dtx2inv"] - F["hadvec"] + F["sprod"] * rmx / F["xnmbar"]) * ez
    l1, l2, l3 = F["flbc1"], F["flbc2"], F["flbc3"]
    q[0] += p[0] * (l1 + .5 * l2 * dz) / (l1 - .5 * l2 * dz)
    f[0] -= p[0] * l3 * dz / (l1 - .5 * l2 * dz)
    p[0] = 0.
    p[-1] = 1. + .5 * dz * th[-1]
    q[-1] = p[-1] - 2.
    f[-1] = -C["grav"] * rmx * F["fubc"] * dz / (C["p0"] * ax[-1] * C["avo"])
    return _thomas(p, q, r, f, nk)


def _comp(F, C):
    tn, dz, nk = F["tn"], C["dz"], F["tn"].shape[0]
    fs = F["fs"].reshape(4, 3, nk, -1)
    lo = _lower(F, C)
    mb = 1. / (lo[0] * C["rmassinv_o2"] + lo[1] * C["rmassinv_o1"] + lo[2] * C["rmassinv_he"] +
               (1. - sum(lo)) * C["rmassinv_n2"])
    names = ("o2", "o1", "he")
    sp = [_below(.5 * (lo[i] + F[n][0]), F[n]) for i, n in enumerate(names)]
    em, tni = _below(.5 * (mb + F["mbar"][0]), F["mbar"]), _below(F["tlbc"], tn)
    dm = _rise(F["mbar"][0] - mb, F["mbar"], dz)
    dt = _rise((tn[0] - F["tlbc"]) * 2, tn, dz)
    wi, df, ez = _mid_up(F["w"]), F["dfactor"], F["expz"]
    mass = (C["rmass_o2"], C["rmass_o1"], C["rmass_he"])
    ep = [1. - (mass[i] + dm) / em for i in range(3)]
    ep[2] = ep[2] - torch.cat([(-0.38 * dt / tni)[:-1], torch.zeros_like(tn[:1])])
    al = _alpha(*sp, tni)
    s = em * C["rmassinv_n2"] * (T00 / tni) ** 0.25 / TAU
    ak = [[v * s for v in row] for row in _inverse(al)]
    wk = dm / (em * 2.)
    n1 = nk - 1
    e, d0, d1 = ez[:-1, None], C["expzmid_inv"] * F["difk"][:-1, None], C["expzmid"] * F["difk"][1:, None]
    edp, edr = d0 * (1. / dz - wk[:-1]), d1 * (1. / dz + wk[1:])
    edq = d0 * (1. / dz + wk[:-1]) + d1 * (1. / dz - wk[1:])
    P, Q, R = (torch.zeros((n1, 3, 3, tn.shape[1]), dtype=tn.dtype, device=tn.device) for _ in range(3))  # [k,j,i]
    f = torch.zeros((n1, 3, tn.shape[1]), dtype=tn.dtype, device=tn.device)
    for i in range(3):
        for m in range(3):
            one = 1. if i == m else 0.
            lo_, hi_ = ak[i][m][:-1], ak[i][m][1:]
            P[:, m, i] = lo_ * (1. / dz + ep[m][:-1] / 2.) / dz - one * e / dz * (edp * df + .5 * wi[:-1])
            R[:, m, i] = hi_ * (1. / dz - ep[m][1:] / 2.) / dz - one * e / dz * (edr * df - .5 * wi[:-1])
            Q[:, m, i] = (-(lo_ * (1. / dz - ep[m][:-1] / 2.) + hi_ * (1. / dz + ep[m][1:] / 2.)) / dz +
                          one * e * (edq * df / dz + C["dtx2inv"]) - e * fs[m + 1, i, :-1])
        n = names[i]
        f[:, i] = e * (F[n + "nm_smooth"] * C["dtx2inv"] - (F[n + "_advec"] - fs[0, i]) + F["hd" + n])[:-1]
    p0 = P[0].clone()
    for m in range(3):
        for n in range(3):
            Q[0, m] += p0[n] * C["b"][n][m]
        f[0] -= p0[m] * C["fb"][m]
    P[0] = 0.
    up = [(1. + .5 * ep[m][-1] * dz) / (1. - .5 * ep[m][-1] * dz) for m in range(3)]
    flx = F["flx_he"] if C["calc_helium"] else torch.zeros_like(F["flx_he"])
    f00 = em[nk - 2] * C["rmassinv_n2"] * C["p0"] * (T00 / tn[nk - 2]) ** 0.25 / (TAU * C["grav"])
    t1 = (al[1][2][-1] - al[1][1][-1]) * flx / (f00 * (1. / dz - .5 * ep[1][-1]))
    t2 = (al[2][2][-1] - al[2][1][-1]) * flx / (f00 * (1. / dz - .5 * ep[2][-1]))
    for m in range(3):
        Q[-1, m] += up[m] * R[-1, m]
    f[-1] -= R[-1, 1] * t1 + R[-1, 2] * t2
    R[-1] = 0.
    u = _block_thomas(P, Q, R, f, n1).movedim(1, 0)
    top = torch.stack([up[0] * u[0, -1], up[1] * u[1, -1] + t1, up[2] * u[2, -1] + t2])
    u = torch.cat([u, top[:, None]], 1)
    if not C["calc_helium"]:
        u[2] = C["pshelb"]
    return u


def _solar(F, day, night):
    """Day and night values joined over the terminator; also |magnetic latitude|."""
    chi = F["chi"] * (180. / math.pi)
    x = torch.where(F["chi"] >= .5 * math.pi, night, day)
    dusk = .5 * (day + night) + .5 * (day - night) * torch.cos(math.pi * (chi - 80.) / 20.)
    return torch.where((chi - 80.) * (chi - 100.) < 0., dusk, x)


def _latitude(F):
    a = F["rlatm"].abs()
    mid = .5 * (1. + torch.cos(a * 6. - math.pi * 4. / 3.))
    return a, torch.where(a >= math.pi / 4.5, 1., torch.where(a <= math.pi / 18, 0., mid))


def _settei(F, C, qtotal):
    ev, dz, b, fb, nk = C["evergs"], C["dz"], C["b"], C["fb"], F["tn"].shape[0]
    tn, o2, o1, he, n2, ne, te, ti = (F[k] for k in ("tn", "o2", "o1", "he", "n2", "ne", "te", "ti"))
    arl, a = _latitude(F)
    day = -9.0e7 * min(C["f107"], 235.) * a
    fe = _solar(F, day + F["qteaur"], day / 2. + F["qteaur"]) * ev
    fe = torch.where(arl >= math.pi / 3., fe - 3.0e9 * ev, fe)
    mid = lambda first, x, last: torch.cat([first[None], .5 * (x[1:-1] + x[:-2]), last[None]])  # noqa: E731
    tei = mid(torch.maximum(1.5 * te[0] - .5 * te[1], F["t_lbc"]), te, 1.5 * te[-2] - .5 * te[-3])
    low = [.5 * (fb[0] + sum((b[0][j] + (1. if i == j else 0.)) * s[0] for j, s in enumerate((o2, o1, he))))
           for i in range(3)]
    oi = [mid(low[i], s, .5 * (s[-1] + s[-2])) for i, s in enumerate((o2, o1, he))]
    n2i = mid((1. - sum(low)).clamp(min=0.), n2, .5 * (n2[-1] + n2[-2])).clamp(min=0.)
    inv = [C["rmassinv_" + k] for k in ("o2", "o1", "he", "n2")]
    dens = [F["xnmbari"] * s * m for s, m in zip((*oi, n2i), inv)]
    rt = tei.sqrt()
    tek = 7.5e5 / (1. + 3.22e4 * tei ** 2 / ne * ((2.20e-16 + 7.92e-18 * rt) * dens[0] +
                                                  1.10e-16 * (1. + 5.7e-4 * tei) * dens[1] + 5.60e-16 * dens[2] +
                                                  (2.82e-17 - 3.41e-21 * tei) * rt * dens[3])) * ev
    sd = (torch.sin(F["dipmag"].abs().clamp(min=C["dipmin"])) ** 2).clamp(min=.10)
    p = 2. / 7. / (F["scht"] * dz ** 2) * sd
    th = tek / F["schti"]
    r = p * torch.cat([th[1:], 2. * th[-1:] - th[-2:-1]])
    p = p * th
    q = -(p + r)
    rhs = torch.zeros_like(tn)
    q[0] -= p[0]
    rhs[0] -= 2. * p[0] * F["t_lbc"] ** 3.5
    p[0] = 0.
    q[nk - 2] += r[nk - 2]
    rhs[nk - 2] += r[nk - 2] * dz * 3.5 * F["schti"][-1] * fe / tek[-1]
    r[nk - 2] = 0.
    qt = sum(F[k] for k in ("qo2p", "qop", "qn2p", "qnop", "qnp", "qop2d", "qop2p")).clamp(min=1e-20)
    qt = torch.cat([(qt[:-1] * qt[1:]).sqrt(), torch.zeros_like(qt[:1])])
    rne = torch.cat([ne[:-1] * ne[1:], (ne[-1] ** 3 / ne[-2])[None]]).clamp(min=1e4).sqrt()
    o2n, o1n, hen, n2n = (F["xnmbar"] * s * m for s, m in zip((o2, o1, he, n2), inv))
    if C["electron_heating"] == 6:
        y = torch.log(rne / (o2n + n2n + o1n))
        y = torch.exp(((((((-1.249e-5 * y - 5.755e-4) * y - 9.346e-3) * y - 5.9e-2) * y - 4.392e-2) * y + 1.056) * y +
                       5.342))
    else:
        y = torch.log(rne / (o2n + n2n + 0.1 * o1n))
        y = torch.exp(-((((0.001996 * y + 0.08034) * y + 1.166) * y + 6.941) * y + 12.75))
    rhs = rhs - y * qt * ev
    if C["et"]:
        rhs = rhs - (F["Q1"] + F["Q2"]) * 10.
    rt = te.sqrt()
    coll = torch.where(te >= 1000., 2.e-7 * torch.exp(-4605.2 / te), 5.71e-8 * torch.exp(-3352.6 / te))
    coll = torch.where(te > 2000., 2.53e-6 * rt * torch.exp(-17620. / te), coll)
    same = (te - tn).abs() < 1e-6
    dif = torch.where(same, 1., te - tn)
    l2v = 1.3e-4 * torch.where(same, 3200. / tn ** 2, (1. - torch.exp(-3200. * dif / (te * tn))) / dif) * coll
    ln = (o2n * (1.21e-18 * (1. + 3.6e-2 * rt) * rt + 6.9e-14 / rt + 3.125e-21 * te ** 2) +
          o1n * (7.9e-19 * (1. + 5.7e-4 * te) * rt + 3.4e-12 * (1. - 7.e-5 * te) / tn * (150. / te + 0.4)) +
          hen * 2.46e-17 * rt + n2n * (1.77e-19 * (1. - 1.21e-4 * te) * te + 2.9e-14 / rt + l2v))
    if C["et"]:
        ln = torch.where((te > 500.) & (F["Q2"] > 0.), ln * torch.exp(-7.54e-4 * (te - 500.)), ln)
    ln = ln * rne * ev
    op, o2p, npl, n2p, nop = (F[k] for k in ("op", "o2p", "nplus", "n2p", "nop"))
    ion = (op * inv[1] + o2p * inv[0] + npl * C["rmassinv_n4s"] + n2p * inv[3] + nop * C["rmassinv_no"])
    lei = 3.2e-8 * rne / (rt * te) * 15. * ev * C["rmass_o1"] * ion
    rtn = (2. * tn).sqrt()
    lin = 1e-14 * ev * (op * (5.8 * o2n + .21 * o1n * rtn + 2.8 * hen + 6.6 * n2n) +
                        o2p * (.14 * o2n * rtn + 4.36 * o1n + 1.63 * hen + 5.81 * n2n) +
                        npl * (5.84 * o2n + 5.84 * o1n + 3.05 * hen + 6.56 * n2n) +
                        n2p * (5.54 * o2n + 4.65 * o1n + 1.82 * hen + .27 * n2n * rtn) +
                        nop * (5.45 * o2n + 4.5 * o1n + 1.72 * hen + 5.92 * n2n))
    q = q - (ln + lei) / te ** 2.5
    rhs = rhs - ln * tn - lei * ti
    qe = (ln * (te - tn) + lei * (te - ti).clamp(min=0.)) * C["avo"] / F["xnmbar"]
    qi = torch.cat([(1.5 * qe[0] - .5 * qe[1])[None], .5 * (qe[:-2] + qe[1:-1]), (1.5 * qe[-2] - .5 * qe[-3])[None]])
    x = _thomas(p, q, r, rhs, nk - 1)[:nk - 1] ** (2. / 7.)
    te_out = torch.maximum(torch.cat([x, (x[-1] ** 2 / x[-2])[None]]), tn)
    ti_out = torch.maximum((F["qji_ti"] * F["xnmbar"] / C["avo"] + lei * te_out + lin * tn) / (lei + lin), tn)
    return te_out, ti_out, qtotal + qi


def _edge_mean(a):
    """Interface means, extrapolated at both ends from the levels below the top."""
    return torch.cat([(1.5 * a[0] - .5 * a[1])[None], .5 * (a[:-2] + a[1:-1]), (1.5 * a[-2] - .5 * a[-3])[None]])


def _oplus(F, C):
    tn, te, ti, o2, o1, n2, he, ne = (F[k] for k in ("tn", "te", "ti", "o2", "o1", "n2", "he", "ne"))
    xn, op, bz, nk, tx = F["xnmbar"], F["op"], F["bz"], F["tn"].shape[0], C["dtx2inv"] * C["nstep_sub"]
    _, a = _latitude(F)
    flux = _solar(F, 2.0e8 * a, -2.0e8 * a)
    tr = .5 * (tn + ti)
    wni, wii, q2p, q2d, qop = (_mid_up(F[k]) for k in ("w", "wi", "qop2p", "qop2d", "qop"))
    m2, m1, mn, mh = (C["rmassinv_" + k] for k in ("o2", "o1", "n2", "he"))
    vni = (18.1 * o2 * m2 + o1 * m1 * tr.sqrt() * (1. - .064 * torch.log10(tr)) ** 2 * C["colfac"] +
           3.6 * he * mh + 18.6 * n2 * mn)
    dj = 1.42e17 / (xn * vni)
    vni = 16 * 3.53e-11 * vni
    if abs(C["opdiffcap"]) >= 1e-9:
        dj = torch.minimum(dj, (C["opdiffcap"] / (1 + 2. ** (F["zpint"] - 6)))[:, None])
    h, bu = F["scht"], F["bx"] * F["u"] + F["by"] * F["v"] + F["scht"] * bz * wni
    t = (te + ti) * op
    d = torch.cat([(t[1] - t[0])[None], (t[2:] - t[:-2]) / 2., (t[-1] - t[-2])[None]])
    d[nk - 2] = t[nk - 2] - t[nk - 3]
    wd = vni * (d / (h * C["dlev"]) + C["rmass_op"] * C["grav"] / C["gask"] * op) * dj
    sc = torch.sin(F["dipmag"]) * torch.cos(F["dipmag"])
    dvb, hdz, tp = F["dvb"] / bz, 1. / (h * C["dz"]), .5 * (ti + te)
    hi = _edge_mean(hdz)
    gm = C["grav"] * C["rmass_op"] / (2. * C["gask"])
    t1 = 2. * torch.cat([tp[:-1], (2. * tp[-2] - tp[-3])[None]]) * hi + gm
    t0 = 2. * torch.cat([(2. * tp[0] - tp[1])[None], tp[:-1]]) * hi - gm
    di = _edge_mean(dj)
    div = dvb + F["bdotdh_djbz"] / (dj * bz ** 2)
    hm, hp = (hdz - .5 * div) * bz ** 2, (hdz + .5 * div) * bz ** 2
    ex = F["explicit_h"] - F["optm1_smooth2"] * tx
    below = torch.cat([(2. * bu[0] - bu[1])[None], bu[:-2]])
    p = (hm * di * t0)[:-1] + (wii * .5 * hdz)[:-1] + bz * below * .5 * hdz[:-1]
    q = (-(hp[:-1] * di[1:] * t0[1:] + hm[:-1] * di[:-1] * t1[:-1]) - wii[:-1] * 6. / C["re"] -
         bu[:-1] * dvb * bz - tx)
    up = torch.cat([-bu[1:-1], (2. * bu[-2] - bu[-3])[None]])
    r = hp[:-1] * di[1:] * t1[1:] - (wii * .5 * hdz)[:-1] + bz * up * .5 * hdz[:-1]
    ub, ua = -bz ** 2 * di[-1] * t0[-1], -bz ** 2 * di[-1] * t1[-1]
    ex = ex.clone()
    q[-1] += ub / ua * r[-1]
    ex[nk - 2] -= flux * r[-1] / ua
    r[-1] = 0.
    x2p = q2p / (xn * ((C["rk16"] + C["rk17"]) * n2 * mn + C["rk18"] * o1 * m1) + (F["rk19"] + F["rk20"]) * ne +
                 C["rk21"] + C["rk22"])
    x2d = (q2d + (F["rk20"] * ne + C["rk22"]) * x2p) / (
        xn * (C["rk23"] * n2 * mn + C["rk24"] * o1 * m1 + C["rk26"] * o2 * m2) + F["rk25"] * ne + C["rk27"])
    loss = xn * (F["rk1"] * o2 * m2 + F["rk2"] * n2 * mn + C["rk10"] * F["n2d"] * C["rmassinv_n2d"])
    q = q - loss[:-1]
    ex = ex - (qop + (F["rk19"] * ne + C["rk21"]) * x2p + (F["rk25"] * ne + C["rk27"]) * x2d +
               (C["rk18"] * x2p + C["rk24"] * x2d) * o1 * m1 * xn)
    q[0] -= p[0]
    ex[0] -= 2. * p[0] * F["qop"][0] / (1.5 * loss[0] - .5 * loss[1])
    x = _thomas(p, q, r, ex[:-1], nk - 1)
    return torch.cat([x, (x[-1] ** 2 / x[-2])[None]]), x2p, x2d, wd * sc * F["sndec"], wd * sc * F["csdec"]


def _filtered(x, cur, prev, mask, bnd, floor, both=True):
    """The lateral overwrite, the time filter and the floors of the scalar routines."""
    x = torch.where(mask, bnd, x)
    nm = DS * cur + DS2 * (prev + x)
    return x.clamp(min=floor), nm.clamp(min=floor) if both else nm


def _span(f, order, axis, mean):
    """Centred mean or difference over `order` points, narrower at the edges."""
    n = f.shape[axis]
    at = lambda d: f.index_select(axis, (torch.arange(n, device=f.device) + d).clamp(0, n - 1))  # noqa: E731
    sides = lambda o: (at(o) + at(-o)) / 2. if mean else (at(o) - at(-o)) / (2. * o)  # noqa: E731
    i = torch.arange(n, device=f.device).reshape([-1 if k == axis else 1 for k in range(3)])
    out = torch.where((i == 1) | (i == n - 2), sides(1), sides(order)) if order == 2 else sides(order)
    return torch.where((i == 0) | (i == n - 1), f if mean else 2. * sides(1), out)


def _advec(f, un, vn, racs, dlam, dphi, rei):
    """Horizontal advection of (level, lat, lon) fields, fourth order inside."""
    out = []
    for axis, v in ((2, un), (1, vn)):
        d1, m1 = _span(f, 1, axis, False), _span(v, 1, axis, True)
        i, n = torch.arange(f.shape[axis], device=f.device), f.shape[axis]
        edge = ((i < 2) | (i > n - 3)).reshape([-1 if k == axis else 1 for k in range(3)])
        wide = d1 * 4. / 3. * m1 - _span(f, 2, axis, False) / 3. * _span(v, 2, axis, True)
        out.append(torch.where(edge, d1 * m1, wide))
    return out[0] * racs[None, :, None] / dlam + out[1] * rei / dphi


def _smooth(f, sh):
    """Shapiro filter along latitude, then longitude."""
    for axis in (1, 2):
        i, n = torch.arange(f.shape[axis], device=f.device), f.shape[axis]
        i = i.reshape([-1 if k == axis else 1 for k in range(3)])
        m1, m2 = _span(f, 1, axis, True), _span(f, 2, axis, True)
        y = torch.where((i == 1) | (i == n - 2), f - sh * 8. * (f - m1), f - sh * (2. * m2 - 8. * m1 + 6. * f))
        f = torch.where((i == 0) | (i == n - 1), f, y)
    return f


def _ring(f, chunks, nlat):
    """Order-1 polar ring filter of (level, lat, lon) rows 2 .. nlat+1."""
    nlon = f.shape[2] - 4
    ang = torch.arange(1, nlon + 1, dtype=f.dtype, device=f.device) * (2. * math.pi / nlon)
    f = f.clone()
    for j in range(nlat):
        n = chunks[j] if j < len(chunks) else chunks[nlat - 1 - j] if nlat - 1 - j < len(chunks) else 0
        if not n:
            continue
        w, L = f[:, j + 2, 2:nlon + 2], nlon // n
        wave = w.mean(1, keepdim=True) + sum(2. / nlon * (w * t).sum(1, keepdim=True) * t
                                             for t in (torch.cos(ang), torch.sin(ang)))
        a = (w - wave).reshape(-1, n, L).mean(2)
        s = lambda d: torch.roll(a, d, 1)  # noqa: E731
        left = (-s(2) + 7. * s(1) + 7. * a - s(-1)) / 12.
        right = (-s(1) + 7. * a + 7. * s(-1) - s(-2)) / 12.
        m = torch.arange(1, L + 1, dtype=f.dtype, device=f.device)
        w = ((left[..., None] * (L - m) + right[..., None] * m) / L).reshape(-1, nlon) + wave
        f[:, j + 2] = torch.cat([w[:, -2:], w, w[:, :2]], 1)
    return f


def _comp_post(u, cur, prev, xn, zp, dz):
    """comp_ng's filter, N2 extrapolation above its 1% level and normalisation."""
    nm = [DS2 * (p + x) + DS * c for x, c, p in zip(u, cur, prev)]
    n2, nk = 1. - sum(u), u[0].shape[0]
    low = n2 < 0.01
    top = torch.where(low.any(0), low.int().argmax(0), nk)
    on = (top > 0) & (top < nk - 1)
    t = top.clamp(1, nk - 2)[None]
    at = lambda k: torch.log((n2 * xn).gather(0, k).clamp(min=1e-300))  # noqa: E731
    zk = zp[:, None]
    grown = torch.exp(at(t) + (at(t) - at(t - 1)) / dz * (zk - zp[t])) / xn
    n2x = torch.where(on & (torch.arange(nk, device=zp.device)[:, None] > t), grown, n2)
    out = []
    for v, d in ((u, n2x), (nm, 1. - sum(nm))):
        v = [x.clamp(min=1e-9) for x in v]
        s = sum(v) + d.clamp(min=1e-9)
        out += [x / s for x in v]
    return out


def _exact_dynamics(case, seed):
    grid, ring = _dyn_grid(case)
    h = dynamics.synthetic_inputs(grid, seed)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    up = lambda F: {k: t(np.moveaxis(v, 1, 2) if k == "fs" else v) for k, v in F.items()}  # noqa: E731
    shape = (grid.nk, grid.nlat + 4, grid.nlon + 4)
    un, vn, racs = t(h["winds"]["un"]).view(shape), t(h["winds"]["vn"]).view(shape), t(grid.racs)
    adv = lambda f: _advec(f.view(shape), un, vn, racs, grid.dlamda, grid.dphi, grid.re_inv).view(grid.nk, -1)  # noqa: E731
    smo = lambda f, sh=grid.shapiro: _smooth(f.view(shape), sh).view(grid.nk, -1)  # noqa: E731
    mask = t(grid.boundary_mask()).bool()
    out = {}
    F, C, bnd, n = up(h["oplus"]["F"]), h["oplus"]["C"], t(h["oplus"]["bnd"]), h["oplus"]["C"]["nstep_sub"]
    F0, op, tm1 = dict(F), F["op"], t(h["oplus"]["optm1"])
    for _ in range(n):
        x, out["xiop2p"], out["xiop2d"] = _oplus(dict(F0, op=op, optm1_smooth2=smo(tm1, grid.shapiro / n)), C)[:3]
        op, tm1 = _filtered(x, op, tm1, mask, bnd, 0.)
    out["op"], out["optm1"] = op, tm1
    for m in h["minor"]:
        cur, prev = t(m["fcomp"]), t(m["fcomp_tm1"])
        x = _minor(dict(up(m["F"]), ftm1_smooth=smo(prev), hadvec=adv(cur)), m["C"])
        out[m["name"] + "_upd"], out[m["name"] + "_nm_upd"] = _filtered(x, cur, prev, mask, t(m["bnd"]), 1e-12)
    out["te"], out["ti"], out["qtotal"] = _settei(up(h["settei"]["F"]), h["settei"]["C"], t(h["settei"]["qtotal"]))
    F, prev = up(h["dt"]["F"]), t(h["dt"]["tn_nm"])
    x = _dt(dict(F, horadv=adv(F["tn"]), tnsmooth=smo(prev), qtotal=out["qtotal"]), h["dt"]["C"])
    out["tn_upd"], out["tn_nm_upd"] = _filtered(x, F["tn"], prev, mask, t(h["dt"]["bnd"]), 100., both=False)
    c, names = h["comp"], ("o2", "o1", "he")
    F, prev = up(c["F"]), [t(c[s + "_nm"]) for s in names]
    for s, p in zip(names, prev):
        F[s + "_advec"], F[s + "nm_smooth"] = adv(F[s]), smo(p)
    u = [x.contiguous() for x in _comp(F, c["C"])]
    if ring:
        u = [_ring(x.view(shape), ring, grid.nlat).reshape(grid.nk, -1) for x in u]
    u = [torch.where(mask, t(c[s + "_bnd"]), x) for s, x in zip(names, u)]
    done = _comp_post(u, [F[s] for s in names], prev, t(c["xnmbar"]), t(c["zpmid"]), c["post_consts"]["dz"])
    out.update(zip(("o2_upd", "o1_upd", "he_upd", "o2nm_upd", "o1nm_upd", "henm_upd"), done))
    return out


def _exact_routine(case, seed):
    s, r, ncol = _routine_state(case, seed), case["routine"], _ncol(case)
    F, C = {k: v[..., :ncol] if v.shape[-1] == s["ld"] else v for k, v in s["F"].items()}, s["C"]
    if r == "comp":
        return _comp(F, C)
    if r == "settei":
        return list(_settei(F, C, F["qtotal0"]))
    got = _oplus(F, C) if r == "oplus" else ((_dt if r == "dt" else _minor)(F, C),)
    p = {k: v[..., :ncol] for k, v in s["post"].items() if torch.is_tensor(v)}
    floor = {"dt": 100., "minor": 1e-12, "oplus": 0.}[r]
    x, nm = _filtered(got[0], p["cur"], p["prev"], p["bnd_mask"].bool(), p["bnd"], floor, both=r != "dt")
    return [x, nm, *got[1:]]


def exact(case, seed):
    what, nk = case["what"], case.get("nk")
    if what == "dynamics":
        return _exact_dynamics(case, seed)
    if what == "routine":
        return _exact_routine(case, seed)
    if what == "host":
        out = []
        for q in _host_state(case, seed)["systems"]:
            a, b, c, f = (torch.from_numpy(np.ascontiguousarray(q[k])).cuda() for k in "abcf")
            if q["kind"]:
                u = _block_thomas(*(m.permute(2, 1, 0, 3) for m in (a, b, c)), f.movedim(0, 1), nk).movedim(0, 1)
            else:
                u = _thomas(a, b, c, f, nk)
            out.append(u.cpu().numpy())
        return out
    if what == "solve":
        s = _solve_state(case, seed)
        back = lambda v: v if v is None or not case["column"] else v.movedim(0, -1)  # noqa: E731
        a, b, c, f, ratio, add = (back(s[k]) for k in ("a", "b", "c", "f", "ratio", "add"))
        if case["block"]:
            x = _block_thomas(a, b, c, f, nk - 1 if case["block"] == 3 else nk, ratio, add)
        else:
            x = _thomas(a, b, c, f, nk)
        return x.movedim(-1, 0).contiguous() if case["column"] else x[..., :_ncol(case)]
    s = _plan_state(case, seed)
    for q in s["segs"]:
        solve = _block_thomas if q["kind"] else _thomas
        q["x"].copy_(solve(q["a"], q["b"], q["c"], q["f"], q["nk"]))
    return s["outs"]
