"""Performance cases of the fluid and radiation hot path.

Each case is one pass through the public host API (FluidContext,
RadiationContext) on a state that a run of that kind has in hand: flux
evaluations, conserved-to-primitive inversions, and whole Runge-Kutta stages
of one block, of many blocks, of a tiled mesh and of the radiation moments.
Sizes are the benchmark configurations' or smaller blocks of the same runs;
`draw` spreads them over the ranges in between.

`exact` restates the flux evaluation (reconstruction, Riemann solver), the
constrained-transport update and the inversion's known answer in plain torch
FP64.  Stages with floors, fixups and physical boundaries (blocks, torus,
bondi) and the radiation stage have no such value.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from phoebus_gb300 import abi, learned, radiation, states, torus
from phoebus_gb300.block import FIELDS, Block, GeomTables
from phoebus_gb300.fluid import FluidContext, MeshRK2

DEV = "cuda"
F64 = torch.float64
SPIN = 0.9375
HSLOPE = 0.3
TOL = 1e-10  # con2prim tolerance of the benchmark runs
TOL_ZONES = 1e-13  # of isolated zones, whose primitives amplify an error of the root up to 1e6 times


# ------------------------------------------------------------------ cases
def listed():
    return [
        # one flux evaluation of the shear-layer benchmark: 256^3, WENO5-Z + HLL
        dict(name="flux_shear_256", kind="flux", geom="mink", n1=256, n2=256, n3=256, recon="weno5z", riemann="hll"),
        # the blast-wave configuration's block: 64^3, PLM + LLF
        dict(name="flux_blast_64", kind="flux", geom="mink", n1=64, n2=64, n3=64, recon="linear", riemann="llf"),
        # a block of a Kerr-Schild (FMKS) mesh with odd extents
        dict(name="flux_kerr_97x66x35", kind="flux", geom="fmks", n1=97, n2=66, n3=35, recon="weno5z", riemann="hll"),
        # a handful of Kerr-Schild zones inverted without a previous solution:
        # the call's latency
        dict(name="c2p_kerr_1000", kind="c2p", n=1000, learned=False),
        # the inversion configuration: millions of cold Kerr-Schild zones
        dict(name="c2p_kerr_12m", kind="c2p", n=12_000_001, learned=False),
        # the same with the learned start
        dict(name="c2p_learned_4m", kind="c2p", n=4_194_305, learned=True),
        # the inversion inside a running simulation: a whole block, each zone
        # starting from the previous step's solution
        dict(name="c2p_warm_128", kind="warm", n1=128, n2=128, n3=128),
        # one Runge-Kutta stage of a shear-layer block
        dict(name="stage_shear_128", kind="stage", n1=128, n2=128, n3=128, recon="weno5z", riemann="hll"),
        # one stage over many independent blocks of uneven sizes, MP5 + HLL
        dict(name="blocks_mp5_48", kind="blocks", nblocks=48),
        # one stage of the FMKS torus on a tiled mesh
        dict(name="torus_96", kind="torus", n=96),
        # one stage of the radiation M1 moments
        dict(name="rad_stage_96", kind="rad", n=96),
        # one stage of the 1D Bondi regression run: launches and latency
        dict(name="bondi_128", kind="bondi", n=128),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["flux", "flux", "c2p", "warm", "stage", "blocks", "torus", "rad", "bondi"])
    if kind == "flux":
        return dict(kind="flux", geom=rng.choice(["mink", "fmks"]), n1=_logint(rng, 12, 256), n2=_logint(rng, 12, 128),
                    n3=_logint(rng, 8, 128), recon=rng.choice(["weno5z", "weno5z", "linear", "mp5"]),
                    riemann=rng.choice(["hll", "llf"]))
    if kind == "c2p":
        return dict(kind="c2p", n=_logint(rng, 500, 10_000_000), learned=rng.random() < 0.3)
    if kind == "warm":
        return dict(kind="warm", n1=_logint(rng, 16, 200), n2=_logint(rng, 16, 128), n3=_logint(rng, 8, 128))
    if kind == "stage":
        return dict(kind="stage", n1=_logint(rng, 16, 160), n2=_logint(rng, 16, 128), n3=_logint(rng, 8, 128),
                    recon=rng.choice(["weno5z", "linear", "mp5"]), riemann=rng.choice(["hll", "llf"]))
    if kind == "blocks":
        return dict(kind="blocks", nblocks=_logint(rng, 4, 60))
    if kind == "torus":
        return dict(kind="torus", n=2 * rng.randint(24, 56))
    if kind == "rad":
        return dict(kind="rad", n=rng.randint(16, 100))
    return dict(kind="bondi", n=_logint(rng, 32, 1024))


# ----------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(1_000_003 + int(seed))


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=F64)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=F64)


def _ideal_prims(rho, wv, P, B, gm1, mu=None):
    """The 12 primitives of the ideal gas with Cv = 1."""
    u = P / gm1
    T = u / rho
    out = torch.empty((abi.NPRIM,) + tuple(rho.shape), dtype=F64, device=rho.device)
    out[abi.PRHO] = rho
    for d in range(3):
        out[abi.PVEL + d] = wv[d]
        out[abi.PB + d] = B[d]
    out[abi.PENG] = u
    out[abi.PPRS] = P
    out[abi.PGM1] = gm1 + 1.0
    out[abi.PTMP] = T
    out[abi.PMU] = 0.0 if mu is None else mu
    return out


def _axes(b):
    """Cell-centre coordinates of the entire block, shaped for (k, j, i)."""
    x = [b.xmin[d] + (torch.arange(n, device=DEV, dtype=F64) + 0.5 - (g if d < b.ndim else 0)) * b.dx[d]
         for d, (n, g) in enumerate(zip((b.n1t, b.n2t, b.n3t), (b.ng,) * 3))]
    return x[0][None, None, :], x[1][None, :, None], x[2][:, None, None]


def _periodic(b, a):
    """The field with its ghost zones replaced by their periodic images."""
    for ax, n in ((-1, b.nx[0]), (-2, b.nx[1]), (-3, b.nx[2])):
        t = a.shape[ax]
        idx = (torch.arange(t, device=a.device) - b.ng) % n + b.ng
        a = a.index_select(a.dim() + ax, idx)
    return a.contiguous()


def _unit_block(case, ndim=3):
    nx = (case["n1"], case["n2"], case["n3"])
    return Block(nx, 4, ndim, (0.0, 0.0, 0.0), tuple(1.0 / n for n in nx), backend="torch", device=DEV)


def _shear_prims(b, g, Gamma):
    """The shear layer: v_x and rho follow a tanh profile across y = 1/2, with
    transverse velocity noise of 1e-3 drawn per zone."""
    X, Y, Z = _axes(b)
    shp = (b.n3t, b.n2t, b.n1t)
    t = torch.tanh((Y - 0.5) / 0.01).expand(shp)
    vx, vy, vz = 0.5 * t, 1e-3 * _randn(g, *shp), 1e-3 * _randn(g, *shp)
    W = 1.0 / torch.sqrt(1.0 - (vx * vx + vy * vy + vz * vz))
    one = torch.ones(shp, device=DEV, dtype=F64)
    zero = torch.zeros(shp, device=DEV, dtype=F64)
    return _periodic(b, _ideal_prims(1.5 + 0.5 * t, (W * vx, W * vy, W * vz), one, (0.01 * one, zero, zero),
                                     Gamma - 1.0))


def _blast_prims(b, g, Gamma):
    """The magnetised blast wave: P = 1 inside r < 0.1 of the box centre, 1e-3
    outside, at rest, B along X1, density noise of 1e-6."""
    X, Y, Z = _axes(b)
    shp = (b.n3t, b.n2t, b.n1t)
    r = torch.sqrt((X - 0.5) ** 2 + (Y - 0.5) ** 2 + (Z - 0.5) ** 2)
    rho = 1e-2 * (1.0 + 1e-6 * (2.0 * _rand(g, *shp) - 1.0))
    P = torch.where(r < 0.05, 1.0, 1e-3).to(F64)
    zero = torch.zeros(shp, device=DEV, dtype=F64)
    return _periodic(b, _ideal_prims(rho, (zero, zero, zero), P, (zero + 0.1, zero, zero), Gamma - 1.0))


def _wedge_block(case):
    """A block of an FMKS mesh: X1 = ln r over [2, 20], X2 off the axis."""
    n1, n2, n3 = case["n1"], case["n2"], case["n3"]
    x1 = (math.log(2.0), math.log(20.0))
    dx = ((x1[1] - x1[0]) / n1, 0.7 / n2, 2.0 * math.pi / n3)
    return Block((n1, n2, n3), 4, 3, (x1[0], 0.15, 0.0), dx, backend="torch", device=DEV)


def _wedge_prims(b, g, Gamma):
    """A smooth rotating flow with a poloidal and toroidal field and 4%
    pressure noise per zone."""
    X, Y, Z = _axes(b)
    shp = (b.n3t, b.n2t, b.n1t)
    e = torch.exp(-0.8 * X) * (1.0 + 0.3 * torch.sin(6.0 * Y) * torch.cos(2.0 * Z))
    rho = 0.2 * e.expand(shp).contiguous()
    P = (0.02 * rho ** Gamma + 1e-4) * (1.0 + 0.04 * (_rand(g, *shp) - 0.5))
    iX = torch.exp(-X)
    wv = [(-0.05 * iX * (1.0 + 0.5 * torch.sin(3.0 * Y + Z))).expand(shp),
          (0.03 * iX * torch.cos(4.0 * Y + 2.0 * Z)).expand(shp), (0.3 * iX ** 1.5 * torch.sin(3.0 * Y)).expand(shp)]
    B = [(0.02 * iX * torch.cos(3.0 * Y + Z)).expand(shp), (0.01 * iX * torch.sin(3.0 * Y + Z)).expand(shp),
         (0.02 * iX * torch.sin(2.0 * Y)).expand(shp)]
    return _ideal_prims(rho, wv, P, B, Gamma - 1.0)


GAMMA = {"weno5z": 5.0 / 3.0, "linear": 4.0 / 3.0, "mp5": 5.0 / 3.0}


def _fluid_params(case, **over):
    return abi.default_params(Gamma=GAMMA[case["recon"]], recon=case["recon"], riemann=case["riemann"], cfl=0.4,
                              c2p_tol=TOL, c2p_max_iter=100, **over)


def _flux_inputs(case, seed):
    g, G = _gen(seed), GAMMA[case["recon"]]
    if case["geom"] == "fmks":
        b = _wedge_block(case)
        return b, _wedge_prims(b, g, G)
    b = _unit_block(case)
    return b, (_blast_prims if case["recon"] == "linear" else _shear_prims)(b, g, G)


def _kerr_inputs(n, seed):
    """Independent zones in Kerr-Schild (FMKS) geometry: r in [1.5, 50], any
    angle, log rho in [-6, 0], log u/rho in [-4, 1], W in [1, 10],
    magnetisation b^2/rho in [1e-4, 1e2], isotropic directions."""
    g = _gen(seed)
    gm1 = 1.0 / 3.0
    U = _rand(g, 11, n)
    r, th = 1.5 + 48.5 * U[0], math.pi * (1e-6 + (1.0 - 2e-6) * U[1])
    x2 = states.theta_to_x2(th)
    met = _fmks(torch.log(r), x2)
    gam = met["gam"]

    def iso(a, c):
        cz = 2.0 * a - 1.0
        s = torch.sqrt((1.0 - cz * cz).clamp(min=0.0))
        return [s * torch.cos(2.0 * math.pi * c), s * torch.sin(2.0 * math.pi * c), cz]

    def dot(a, c):
        return sum(gam[m][k] * a[m] * c[k] for m in range(3) for k in range(3))

    rho, sie, W = 10.0 ** (-6.0 + 6.0 * U[2]), 10.0 ** (-4.0 + 5.0 * U[3]), 1.0 + 9.0 * U[4]
    nv, nb = iso(U[5], U[6]), iso(U[8], U[9])
    f = torch.sqrt(W * W - 1.0) / W / torch.sqrt(dot(nv, nv))
    v = [f * x for x in nv]
    ib = 1.0 / torch.sqrt(dot(nb, nb))
    bh = [ib * x for x in nb]
    Bm = torch.sqrt(10.0 ** (-4.0 + 6.0 * U[7]) * rho / (1.0 / (W * W) + dot(bh, v) ** 2))
    P = gm1 * rho * sie
    mu = 1.0 / ((1.0 + sie + P / rho) * W)
    prim = _ideal_prims(rho, [W * x for x in v], P, [Bm * x for x in bh], gm1, mu)
    return torch.log(r), x2, prim, met


def _turbulent_prims(b, g, gm1):
    """Minkowski zones of a turbulent box: smooth structure of order one with
    noise per zone, v up to 0.9, plasma beta of a few; mu of the zone."""
    shp = (b.n3t, b.n2t, b.n1t)
    X, Y, Z = _axes(b)
    t = torch.sin(2 * math.pi * X) * torch.cos(2 * math.pi * Y) + 0.5 * torch.sin(4 * math.pi * Z)
    rho = torch.exp(0.8 * t + 0.02 * _randn(g, *shp))
    P = 0.3 * rho * torch.exp(0.3 * _randn(g, *shp))
    v = [0.3 * torch.cos(2 * math.pi * (Y + 0.1 * d)) + 0.05 * _randn(g, *shp) for d in range(3)]
    vsq = sum(x * x for x in v)
    f = torch.sqrt(vsq.clamp(max=0.81) / vsq)
    W = 1.0 / torch.sqrt(1.0 - vsq.clamp(max=0.81))
    B = [0.2 + 0.05 * _randn(g, *shp) for _ in range(3)]
    mu = 1.0 / ((1.0 + (P / gm1 + P) / rho) * W)
    return _periodic(b, _ideal_prims(rho, [W * f * x for x in v], P, B, gm1, mu))


def _warm_inputs(case, seed):
    """A turbulent block and the previous step's mu, stale by up to 1%."""
    g, b = _gen(seed), _unit_block(case)
    prim = _turbulent_prims(b, g, 2.0 / 3.0)
    stale = prim[abi.PMU] * (1.0 + 0.01 * (2.0 * _rand(g, *b.shape) - 1.0))
    return b, prim, stale.clamp(max=1.0)


_WEIGHTS = {}


def _learned_weights(ctx, p):
    """One network for the Kerr-Schild zones, trained once per process."""
    if not _WEIGHTS:
        x, y = learned.training_pairs(ctx, p, 1_000_000, device=DEV)
        ctx.mlp_set_weights(learned.init_weights(7))
        ctx.MLPTrain(x, y, abi.default_train_opts(epochs=5))
        _WEIGHTS["theta"], _WEIGHTS["box"] = ctx.mlp_get_weights(), ctx.mlp_input_box()
    ctx.mlp_set_weights(_WEIGHTS["theta"])
    ctx.mlp_set_input_box(*_WEIGHTS["box"])


def _flat_blocks(blocks, names):
    """The blocks' fields as views of one array per field (how a host that
    packs its blocks holds them); returns those arrays."""
    flat = {}
    for name in names:
        nv = FIELDS[name]
        flat[name] = torch.zeros(sum(nv * b.N for b in blocks), dtype=F64, device=DEV)
        o = 0
        for b in blocks:
            v = flat[name][o:o + nv * b.N].view((nv,) + b.shape)
            if name in b.arrays:
                v.copy_(b.arrays[name])
            b.set(name, v)
            o += nv * b.N
    return flat


def _block_views(blocks, flat):
    out, o = [], 0
    for b in blocks:
        out.append(flat[o:o + abi.NCONS * b.N].view((abi.NCONS,) + b.shape))
        o += abi.NCONS * b.N
    return out


# ---------------------------------------------------------------- prepare
def prepare(case, seed):
    ctx = FluidContext(0)
    s = dict(case=case, ctx=ctx)
    kind = case["kind"]
    if kind == "flux":
        b, prim = _flux_inputs(case, seed)
        b.alloc(["flux", "face_sig", "cons"])
        b.set("prim", prim)
        if case["geom"] == "fmks":
            geo = abi.default_geometry(abi.GEOM_FMKS, a=SPIN, derefine_poles=0)
            b.geom = GeomTables(geo, b.n1t, b.n2t, "torch", DEV).alloc()
            ctx.GeometryFillFMKS(b)
        s.update(b=b, p=_fluid_params(case))
    elif kind == "c2p":
        n = case["n"]
        p = abi.default_params(gm1=1.0 / 3.0, c2p_tol=TOL_ZONES, c2p_max_iter=100)
        if case["learned"]:
            _learned_weights(ctx, p)
        x1, x2, prim, met = _kerr_inputs(n, seed)
        s["cons"] = _p2c(prim, met)
        s["geom"] = ctx.GeometryFMKSPoints(learned.kerr_geometry(), x1.contiguous(), x2.contiguous())
        s["prim"] = torch.zeros_like(prim)
        s["fail"], s["sig"] = torch.zeros(n, dtype=F64, device=DEV), torch.zeros((3, n), dtype=F64, device=DEV)
        s["p"] = p
    elif kind == "warm":
        b, prim, stale = _warm_inputs(case, seed)
        b.alloc(["cell_sig", "fail"])
        b.set("cons", _p2c(prim, _flat_metric()))
        prim[:abi.PMU] = 0.0
        b.set("prim", prim)
        s.update(b=b, stale=stale, p=abi.default_params(Gamma=5.0 / 3.0, c2p_tol=TOL, c2p_max_iter=100))
    elif kind == "stage":
        b = _unit_block(case).alloc()
        b.set("prim", _shear_prims(b, _gen(seed), GAMMA[case["recon"]]))
        b.set("cons", _p2c(b["prim"], _flat_metric()))
        s.update(b=b, out=b["cons"].clone(), p=_fluid_params(case), dt=_stage_dt(case))
    elif kind == "blocks":
        p = abi.default_params(Gamma=4.0 / 3.0, recon="mp5", riemann="hll", c2p_tol=TOL, c2p_max_iter=100)
        p.enable_floors, p.enable_c2p_fixup, p.enable_ceilings = 1, 1, 1
        p.rho0_floor, p.sie0_floor = 1e-8, 1e-8
        g, blocks = _gen(seed), []
        for n in states.uneven_block_sizes(case["nblocks"]):
            b = _unit_block(dict(n1=n, n2=n, n3=n)).alloc()
            b.set("prim", _turbulent_prims(b, g, 1.0 / 3.0))
            blocks.append(b)
        flat = _flat_blocks(blocks, ["prim", "cons", "fail"])
        for b in blocks:
            ctx.Initialize(p, b)
        out = flat["cons"].clone()
        s.update(p=p, blocks=blocks, flat=flat, out=out, outs=_block_views(blocks, out),
                 bases=[b["cons"] for b in blocks],
                 dt=0.1 * min(ctx.EstimateTimestepBlock(p, b, False).item() for b in blocks))
    elif kind == "torus":
        p, n = torus.torus_params(), case["n"]
        mesh = torus.torus_mesh(n=n, lo=16, hi=48)
        blocks = mesh.make_blocks(DEV, torus.torus_geometry())
        flat = _flat_blocks(blocks, ["prim", "cons", "fail"])
        torus.fill_torus(ctx, p, mesh, blocks, torus.torus_problem(seed=seed))
        out = flat["cons"].clone()
        s.update(p=p, mesh=mesh, blocks=blocks, flat=flat, out=out, outs=_block_views(blocks, out),
                 bases=[b["cons"] for b in blocks],
                 dt=0.4 * min(ctx.EstimateTimestepBlock(p, b, False).item() for b in blocks))
    elif kind == "rad":
        g = _gen(seed)
        hb, par, rpar = radiation.radiation_pulse_3d(n=case["n"])
        b = hb.to_device(DEV)
        rad = radiation.RadiationContext(ctx)
        p, rp = abi.default_params(**par), abi.default_rad_params(**rpar)
        b["rprim"][abi.RJ] *= 1.0 + 0.2 * _rand(g, *b.shape)
        b["prim"][abi.PVEL:abi.PVEL + 3] += 0.05 * (_rand(g, 3, *b.shape) - 0.5)
        e = b.entire()
        rad.MomentPrim2Con(rp, p, b, *e)
        rad.Initialize(rp, p, b)
        s.update(b=b, rad=rad, p=p, rp=rp, out=b["rcons"].clone(), dt=rad.EstimateTimestepBlock(rp, p, b))
    else:
        g = np.random.default_rng(seed)
        hb, par, _ = states.bondi_1d(case["n"])
        b = hb.to_device(DEV)
        ctx.GeometryFillFMKS(b)
        hb.geom = b.geom.to_host()
        states.bondi_fill(hb)
        hb["prim"][abi.PRHO] *= 1.0 + 1e-3 * g.uniform(-1, 1, hb.shape)
        b["prim"].copy_(torch.from_numpy(hb["prim"]))
        p = abi.default_params(**par)
        mesh = states.bondi_mesh(case["n"])
        rk = MeshRK2(ctx, p, mesh, [b])
        rk.initialize()
        s.update(p=p, mesh=mesh, blocks=[b], out=b["cons"].clone(), dt=0.5 * rk.estimate_dt(False))
        s.update(bases=[b["cons"]], outs=[s["out"]], flat=b.arrays)
    return s


# -------------------------------------------------------------------- run
def run(s):
    case, ctx, p = s["case"], s["ctx"], s["p"]
    kind = case["kind"]
    if kind == "flux":
        ctx.CalculateFluxes(p, s["b"])
        return {"flux": s["b"]["flux"], "face_sig": s["b"]["face_sig"]}
    if kind == "c2p":
        s["prim"][abi.PMU].zero_()  # no previous solution
        ctx.ConservedToPrimitiveZones(p, s["cons"], s["prim"], s["geom"], fail=s["fail"], cell_sig=s["sig"],
                                      learned=case["learned"])
        return {**_prim_groups(s["prim"]), "cell_sig": s["sig"], "fail": s["fail"]}
    if kind == "warm":
        b = s["b"]
        b["prim"][abi.PMU].copy_(s["stale"])  # the previous step's solution
        ctx.ConservedToPrimitive(p, b)
        return {**_prim_groups(b["prim"]), "cell_sig": b["cell_sig"], "fail": b["fail"]}
    if kind == "stage":
        b = s["b"]
        ctx.Stage(p, b, b["cons"], s["out"], 1.0, s["dt"])
        return {"cons": s["out"], "prim": b["prim"], "fail": b["fail"], "cell_sig": b["cell_sig"]}
    if kind == "blocks":
        ctx.StageBatched(p, s["blocks"], s["bases"], s["outs"], 1.0, s["dt"])
        return {"cons": s["out"], "prim": s["flat"]["prim"], "fail": s["flat"]["fail"]}
    if kind == "rad":
        b = s["b"]
        s["rad"].Stage(s["rp"], p, b, b["rcons"], s["out"], 1.0, s["dt"])
        return {"cons": s["out"], "prim": b["rprim"]}
    ctx.StageMesh(p, s["mesh"], s["blocks"], s["bases"], s["outs"], 1.0, s["dt"])
    return {"cons": s["out"], "prim": s["flat"]["prim"], "fail": s["flat"]["fail"]}


def _prim_groups(prim):
    return {"rho": prim[abi.PRHO], "wv": prim[abi.PVEL:abi.PVEL + 3], "u": prim[abi.PENG],
            "B": prim[abi.PB:abi.PB + 3], "P": prim[abi.PPRS], "T": prim[abi.PTMP], "mu": prim[abi.PMU]}


# ------------------------------------------------------------------- work
# FP64 operations of one cell and direction: both face states of one variable
# (reconstruction), and one face (two flux evaluations and their combination).
_RECON_FLOPS = {"weno5z": 90, "mp5": 60, "linear": 10}
_FACE_FLOPS = {"mink": 250, "fmks": 400}
# one inversion: setup and unwrapping, and a residual evaluation
_C2P_FLOPS, _RES_FLOPS = 200, 45


def work(case):
    kind = case["kind"]
    if kind == "c2p":
        n = case["n"]
        return {"bytes": 8.0 * n * (abi.NCONS + abi.GEOM_NLOC + abi.NPRIM + 4), "flops": n * (_C2P_FLOPS + 3.0 * _RES_FLOPS)}
    if kind == "warm":
        n = (case["n1"] + 8) * (case["n2"] + 8) * (case["n3"] + 8)
        return {"bytes": 8.0 * n * (abi.NCONS + 2 + abi.NPRIM + 4), "flops": n * (_C2P_FLOPS + 2.0 * _RES_FLOPS)}
    if kind == "bondi":
        n = case["n"]
        return {"bytes": 8.0 * n * 2 * (abi.NPRIM + abi.NCONS), "flops": n * 1000.0}
    if kind == "rad":
        n = float(case["n"]) ** 3
        return {"bytes": 8.0 * n * (8 + 2 * abi.RNPRIM + 2 * abi.RNCONS), "flops": n * (3 * 700.0 + 2000.0)}
    if kind == "blocks":
        n, recon, geom = float(sum(e ** 3 for e in states.uneven_block_sizes(case["nblocks"]))), "mp5", "mink"
    elif kind == "torus":
        n, recon, geom = float(case["n"]) ** 3, "weno5z", "fmks"
    else:
        n, recon, geom = float(case["n1"] * case["n2"] * case["n3"]), case["recon"], case.get("geom", "mink")
    flux = n * 3 * (9 * _RECON_FLOPS[recon] + _FACE_FLOPS[geom])
    if kind == "flux":
        return {"bytes": 8.0 * n * (9 + 3 * (abi.NCONS + 1)), "flops": flux}
    return {"bytes": 8.0 * n * (2 * abi.NPRIM + 2 * abi.NCONS + 4), "flops": flux + n * (_C2P_FLOPS + 2.0 * _RES_FLOPS)}


# ------------------------------------------------------------------ exact
def exact(case, seed):
    kind = case["kind"]
    if kind == "flux":
        b, prim = _flux_inputs(case, seed)
        flux = torch.zeros((3 * abi.NCONS,) + b.shape, dtype=F64, device=DEV)
        sig = torch.zeros((3,) + b.shape, dtype=F64, device=DEV)
        for d in range(3):
            _fluxes(case, b, prim, d, flux[abi.NCONS * d:abi.NCONS * (d + 1)], sig[d])
        return {"flux": flux, "face_sig": sig}
    if kind in ("c2p", "warm"):
        prim = _kerr_inputs(case["n"], seed)[2] if kind == "c2p" else _warm_inputs(case, seed)[1]
        return {**_prim_groups(prim), "cell_sig": None, "fail": None}
    if kind == "stage":
        b = _unit_block(case)
        prim = _shear_prims(b, _gen(seed), GAMMA[case["recon"]])
        U = _p2c(prim, _flat_metric())
        F = [torch.zeros((abi.NCONS,) + b.shape, dtype=F64, device=DEV) for _ in range(3)]
        for d in range(3):
            _fluxes(case, b, prim, d, F[d], None)
        _constrained_transport(F)
        du = sum((torch.roll(F[d], -1, 3 - d) - F[d]) / b.dx[d] for d in range(3))
        return {"cons": _periodic(b, U - _stage_dt(case) * du), "prim": None, "fail": None, "cell_sig": None}
    return None


def _stage_dt(case):
    return 0.15 / max(case["n1"], case["n2"], case["n3"])


def _flat_metric():
    one = [[1.0 if m == k else 0.0 for k in range(3)] for m in range(3)]
    return {"gam": one, "gamup": one, "alpha": 1.0, "beta": [0.0, 0.0, 0.0], "detgam": 1.0}


def _fmks(x1, x2):
    """The FMKS metric without derefined poles: Kerr-Schild in r = exp(X1) and
    theta = pi X2 + (1 - h)/2 sin(2 pi X2)."""
    r, th = torch.exp(x1), math.pi * x2 + 0.5 * (1.0 - HSLOPE) * torch.sin(2.0 * math.pi * x2)
    jt = math.pi * (1.0 + (1.0 - HSLOPE) * torch.cos(2.0 * math.pi * x2))
    a, s2, c2 = SPIN, torch.sin(th) ** 2, torch.cos(th) ** 2
    q = r * r + a * a * c2
    z = 2.0 * r / q
    zero = torch.zeros_like(q)
    g13 = -a * (1.0 + z) * s2 * r
    gam = [[(1.0 + z) * r * r, zero, g13], [zero, q * jt * jt, zero], [g13, zero, (q + a * a * (1.0 + z) * s2) * s2]]
    up11 = (1.0 / (1.0 + z) + a * a * s2 / q) / (r * r)
    gamup = [[up11, zero, a / (q * r)], [zero, 1.0 / (q * jt * jt), zero], [a / (q * r), zero, 1.0 / (q * s2)]]
    beta = [z / (1.0 + z) / r, zero, zero]
    return {"gam": gam, "gamup": gamup, "alpha": 1.0 / torch.sqrt(1.0 + z), "beta": beta,
            "detgam": torch.sqrt(q * q * (1.0 + z) * s2) * r * jt.abs()}


def _lower(met, v):
    g = met["gam"]
    if isinstance(g[0][0], float):
        return list(v)
    return [g[m][0] * v[0] + g[m][1] * v[1] + g[m][2] * v[2] for m in range(3)]


def _mhd(prim, met):
    """Conserved variables (without sqrt(gamma)) and what the fluxes share."""
    rho, wv, u, B, P = prim[0], prim[1:4], prim[4], prim[5:8], prim[8]
    wl = _lower(met, wv)
    Wsq = 1.0 + sum(wv[m] * wl[m] for m in range(3))
    W = torch.sqrt(Wsq)
    v, vl, Bl = [x / W for x in wv], [x / W for x in wl], _lower(met, B)
    vsq = sum(v[m] * vl[m] for m in range(3))
    Bv, BB = sum(B[m] * vl[m] for m in range(3)), sum(B[m] * Bl[m] for m in range(3))
    bsq = BB / Wsq + Bv * Bv
    rhoh = (rho + u + P) * Wsq
    bl = [Bl[m] / W + W * Bv * vl[m] for m in range(3)]
    D = rho * W
    S = [(rhoh + BB + (W * Bv) ** 2) * vl[m] - W * Bv * bl[m] for m in range(3)]
    tau = rhoh + BB - (P + 0.5 * bsq) - D
    return dict(W=W, v=v, vsq=vsq, Bv=Bv, bsq=bsq, rhoh=rhoh, bl=bl, U=[D, *S, tau, *B])


def _p2c(prim, met):
    U = _mhd(prim, met)["U"]
    return torch.stack([met["detgam"] * x for x in U])


def _minmod(a, b):
    return torch.where(a * b > 0.0, torch.where(a.abs() < b.abs(), a, b), torch.zeros_like(a))


def _mp5(m2, m1, c, p1, p2):
    f = (2.0 * m2 - 13.0 * m1 + 47.0 * c + 27.0 * p1 - 3.0 * p2) / 60.0
    mp = c + _minmod(p1 - c, 4.0 * (c - m1))
    dm, d0, dp = m2 + c - 2.0 * m1, m1 + p1 - 2.0 * c, c + p2 - 2.0 * p1
    m4p = _minmod(_minmod(4.0 * d0 - dp, 4.0 * dp - d0), _minmod(d0, dp))
    m4m = _minmod(_minmod(4.0 * dm - d0, 4.0 * d0 - dm), _minmod(d0, dm))
    ul, md = c + 4.0 * (c - m1), 0.5 * (c + p1) - 0.5 * m4p
    lc = 0.5 * (3.0 * c - m1) + 4.0 / 3.0 * m4m
    lo = torch.maximum(torch.minimum(torch.minimum(c, p1), md), torch.minimum(torch.minimum(c, ul), lc))
    hi = torch.minimum(torch.maximum(torch.maximum(c, p1), md), torch.maximum(torch.maximum(c, ul), lc))
    return torch.where((f - c) * (f - mp) <= 1e-12, f, f + _minmod(lo - f, hi - f))


def _limited(dm, dp, alpha):
    dc = torch.where(dm * dp > 0.0, 0.5 * (dm + dp), torch.zeros_like(dm))
    return torch.copysign(torch.minimum(dc.abs(), alpha * torch.minimum(dm.abs(), dp.abs())), dc)


def _reconstruct(recon, q):
    """(upper-face, lower-face) values of the cell from its five-point stencil."""
    q0, q1, q2, q3, q4 = q
    if recon == "mp5":
        return _mp5(q0, q1, q2, q3, q4), _mp5(q4, q3, q2, q1, q0)
    if recon == "linear":
        dq = _limited(q2 - q1, q3 - q2, 1.5)
        return q2 + 0.5 * dq, q2 - 0.5 * dq
    eps = 1e-100
    ind = [(q0 - 2 * q1 + q2, q0 - 4 * q1 + 3 * q2), (q1 - 2 * q2 + q3, q3 - q1), (q2 - 2 * q3 + q4, q4 - 4 * q3 + 3 * q2)]
    beta = [13.0 / 3.0 * a * a + c * c + eps for a, c in ind]
    tau = (beta[2] - beta[0]).abs()
    nl = [(x + tau) / x for x in beta]
    up = [(2 * q0 - 7 * q1 + 11 * q2) / 6, (-q1 + 5 * q2 + 2 * q3) / 6, (2 * q2 + 5 * q3 - q4) / 6]
    lo = [(2 * q4 - 7 * q3 + 11 * q2) / 6, (-q3 + 5 * q2 + 2 * q1) / 6, (2 * q2 + 5 * q1 - q0) / 6]
    out = []
    for n, c in ((nl, up), (nl[::-1], lo)):
        w = [0.1 * n[0] + eps, 0.6 * n[1] + eps, 0.3 * n[2] + eps]
        s = w[0] + w[1] + w[2]
        al = 3.0 * w[0] * w[1] * w[2] / s / (0.3 * w[0] * w[1] + 0.6 * w[0] * w[2] + 0.1 * w[1] * w[2]) + eps
        out.append(((w[0] * c[0] + w[1] * c[1] + w[2] * c[2]) / s, al))
    (l, al), (r, ar) = out
    a = 2.0 * al * ar / (al + ar)
    dq = _limited(q2 - q1, q3 - q2, 2.0)
    return a * l + (1 - a) * (q2 + 0.5 * dq), a * r + (1 - a) * (q2 - 0.5 * dq)


def _face_state(prim, met, d, Gamma):
    m = _mhd(prim, met)
    v, W, P, bl, B, U = m["v"], m["W"], prim[8], m["bl"], prim[5:8], m["U"]
    vt = v[d] - met["beta"][d] / met["alpha"]
    pt = P + 0.5 * m["bsq"]
    F = [U[0] * vt]
    F += [U[1 + k] * vt - bl[k] * B[d] / W + (pt if k == d else 0.0) for k in range(3)]
    F.append(U[4] * vt + pt * v[d] - m["Bv"] * B[d])
    F += [torch.zeros_like(vt) if k == d else B[k] * vt - B[d] * (v[k] - met["beta"][k] / met["alpha"]) for k in range(3)]
    Wsq = W * W
    va = m["bsq"] * Wsq / (m["rhoh"] + m["bsq"] * Wsq)
    cs = Gamma * P * Wsq / m["rhoh"]
    cm = cs + va * (1.0 - cs)
    v0, q = v[d] * (1.0 - cm), 1.0 - m["vsq"] * cm
    e = torch.sqrt((cm * (1.0 - m["vsq"]) * (met["gamup"][d][d] * q - v[d] * v0)).clamp(min=10 * 2.220446049250313e-16))
    c = met["alpha"] / q
    return U, F, c * (v0 - e) - met["beta"][d], c * (v0 + e) - met["beta"][d]


def _fluxes(case, b, prim, d, flux, sig):
    """Fluxes [8][...] and face speed of direction d at the faces a stage
    reads: faces s .. e+1 along d, s-1 .. e+1 across it."""
    ng, n, Gamma = b.ng, b.nx, GAMMA[case["recon"]]
    ax = 3 - d  # dimension of (variable, k, j, i) along d
    cells = [slice(None)] + [slice(ng - 1, ng + n[x] + 1) for x in (2, 1, 0)]

    def at(o):
        s = list(cells)
        s[ax] = slice(ng - 1 + o, ng + n[d] + 1 + o)
        return prim[:9][tuple(s)]

    up, lo = _reconstruct(case["recon"], [at(o) for o in range(-2, 3)])
    m = n[d] + 2
    left, right = up.narrow(ax, 0, m - 1), lo.narrow(ax, 1, m - 1)
    if case.get("geom", "mink") == "fmks":
        i, j = [b.xmin[x] + (torch.arange(-1, n[x] + 1, device=DEV, dtype=F64) + 0.5) * b.dx[x] for x in (0, 1)]
        if d == 0:
            i = b.xmin[0] + torch.arange(0, n[0] + 1, device=DEV, dtype=F64) * b.dx[0]
        elif d == 1:
            j = b.xmin[1] + torch.arange(0, n[1] + 1, device=DEV, dtype=F64) * b.dx[1]
        met = _fmks(*[x.contiguous() for x in torch.broadcast_tensors(i[None, None, :], j[None, :, None])])
    else:
        met = _flat_metric()
    Ul, Fl, ml, pl = _face_state(left, met, d, Gamma)
    Ur, Fr, mr, pr = _face_state(right, met, d, Gamma)
    gd, gg = met["detgam"], met["alpha"] * met["detgam"]
    faces = list(cells)
    faces[ax] = slice(ng, ng + n[d] + 1)
    faces = tuple(faces[1:])
    if case["riemann"] == "llf":
        c = torch.maximum(torch.maximum(-ml, pl), torch.maximum(-mr, pr))
        for k in range(abi.NCONS):
            flux[k][faces] = 0.5 * ((Fl[k] + Fr[k]) * gg - c * (Ur[k] - Ul[k]) * gd)
    else:
        cl, cr = torch.minimum(ml, mr).clamp(max=0.0), torch.maximum(pl, pr).clamp(min=0.0)
        for k in range(abi.NCONS):
            flux[k][faces] = ((cr * Fl[k] - cl * Fr[k]) * gg + cr * cl * (Ur[k] - Ul[k]) * gd) / (cr - cl)
        c = torch.maximum(-cl, cr)
    if sig is not None:
        sig[faces] = c


def _constrained_transport(F):
    """The induction fluxes from edge-averaged EMFs."""
    def lo(a, d):
        return torch.roll(a, 1, 2 - d)

    def hi(a, d):
        return torch.roll(a, -1, 2 - d)

    B = [[F[d][5 + k] for k in range(3)] for d in range(3)]
    e0 = 0.25 * (B[1][2] + lo(B[1][2], 2) - B[2][1] - lo(B[2][1], 1))
    e1 = -0.25 * (B[0][2] + lo(B[0][2], 2) - B[2][0] - lo(B[2][0], 0))
    e2 = 0.25 * (B[0][1] + lo(B[0][1], 1) - B[1][0] - lo(B[1][0], 0))
    zero = torch.zeros_like(e0)
    new = [[zero, 0.5 * (e2 + hi(e2, 1)), -0.5 * (e1 + hi(e1, 2))], [-0.5 * (e2 + hi(e2, 0)), zero, 0.5 * (e0 + hi(e0, 2))],
           [0.5 * (e1 + hi(e1, 0)), -0.5 * (e0 + hi(e0, 1)), zero]]
    for d in range(3):
        for k in range(3):
            F[d][5 + k] = new[d][k]
