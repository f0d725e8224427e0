"""The work a program using rfdem has it do, as timed cases.

Each case is a dict of plain values; ``prepare`` makes what the program holds before the
call, ``run`` is one pass through the public entry points. The families:

  explicit   blocks of explicit steps of one packed extended-model specimen and the frame
             (positions) read back after each block, as a loading program does
  batch      the same for several discs in one engine
  fire       one quasi-static load increment (single specimen, batch, or warm-started by
             the MLP) under a fixed iteration budget, so that a pass is a fixed amount of work
  create     a whole call: engine from host arrays, pre-strain, steps, positions back
  reference  explicit steps of the FP32 reference-model lattice specimen
  driver     md_Calculation*: a whole reference-model test from host buffers
  md         the drop-in md_* kernels called in the reference driver's order
  train      Adam steps of the warm-start MLP, weights read back
  forward    inference of the warm-start MLP
  pack       specimen packing

Specimens come out of a library packed once per size in a process (a program keeps its
packings too); the seed turns each drum about its axis by its own angle and draws the
bond strengths, so another seed is another specimen.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rockfit-dem_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import rfdem                          # noqa: E402
from rfdem.warm import WarmStart      # noqa: E402

R0 = 0.25                             # mean particle radius of the packed specimens, mm
PHI = 0.58                            # packing fraction
K = 32                                # slots per row
RADII = {"uniform": (0.8, 1.2), "log-uniform": (0.5, 1.5)}


def listed():
    return [
        # the headline workload: 4M particles in the damage regime, stepped in blocks
        dict(name="uniaxial-4m-damaged", family="explicit", n=1000000, drums=4, radii="log-uniform", gap=0.25,
             pre_lat=0.2, pre_ax=-0.03, steps=200),
        # an ordinary specimen (odd size) under load before failure: bonds intact, contacts in
        # parallel, the reference's one-cutoff list rule
        dict(name="uniaxial-26k", family="explicit", n=26113, drums=1, radii="uniform", gap=0.0, pre_lat=-0.004,
             pre_ax=-0.004, steps=400),
        # a strength statistics run: many small Brazilian discs of different sizes at once
        dict(name="brazil-batch-24", family="batch", nmin=2500, nmax=20000, specimens=24, steps=300),
        # the quasi-static configuration at its size
        dict(name="fire-1m", family="fire", mode="single", n=250000, drums=4, specimens=1, iters=120),
        # small quasi-static studies: several cylinders of a few thousand particles
        dict(name="fire-batch-6", family="fire", mode="batch", n=2600, drums=1, specimens=6, iters=300),
        # one specimen from host arrays to positions after a short run: setup counts
        dict(name="create-200k", family="create", n=199999, drums=1, radii="uniform", gap=0.25, pre_lat=0.1,
             pre_ax=-0.02, steps=100),
        # the reference model at the size of its test specimens: FP32 lattice, 198k particles
        dict(name="reference-198k", family="reference", diameter=52.0, height=104.0, steps=400),
        # a material fitter's simulation: a small Brazilian test from host buffers; launches
        # and latency are what it waits for
        dict(name="driver-brazil-885", family="driver", kind="brazil", diameter=16.0, height=6.0, steps=4000),
        # a migrating program that keeps its own step loop and calls the md_* kernels
        dict(name="md-198k", family="md", diameter=52.0, height=104.0, steps=8),
        # training the warm start on the pairs of two 1M-particle increments
        dict(name="train-2m", family="train", rows=2000000, steps=2),
        # the prediction of one load step of a 300k-particle specimen (ragged row count)
        dict(name="forward-300k", family="forward", rows=300007),
        # packing a specimen
        dict(name="pack-20k", family="pack", n=20011, radii="uniform", aspect=2.0),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    f = rng.choice(["explicit", "explicit", "batch", "fire", "create", "reference", "driver", "md", "train", "forward",
                    "pack"])
    if f in ("explicit", "create"):
        damaged = rng.random() < 0.5
        return dict(family=f, n=_log(rng, 1500, 250000), drums=rng.randint(1, 4) if f == "explicit" else 1,
                    radii=rng.choice(["uniform", "log-uniform"]) if damaged else "uniform",
                    gap=0.25 if damaged else rng.choice([0.0, 0.25]), pre_lat=0.2 if damaged else -0.004,
                    pre_ax=-0.03 if damaged else -0.004,
                    steps=rng.randint(100, 300) if f == "explicit" else rng.randint(50, 100))
    if f == "batch":
        lo = _log(rng, 1200, 8000)
        return dict(family=f, nmin=lo, nmax=lo * rng.randint(1, 6), specimens=rng.randint(2, 16),
                    steps=rng.randint(100, 300))
    if f == "fire":
        mode = rng.choice(["single", "batch", "warm"])
        return dict(family=f, mode=mode, n=_log(rng, 1500, 150000 if mode != "batch" else 20000), drums=1,
                    specimens=rng.randint(2, 8) if mode == "batch" else 1, iters=rng.randint(60, 120))
    if f in ("reference", "md"):
        d = math.exp(rng.uniform(math.log(9.0), math.log(50.0)))
        return dict(family=f, diameter=d, height=d * rng.uniform(1.0, 2.0),
                    steps=rng.randint(100, 400) if f == "reference" else rng.randint(2, 8))
    if f == "driver":
        kind = rng.choice(["uniaxial", "brazil"])
        d = rng.uniform(9.0, 25.0)
        return dict(family=f, kind=kind, diameter=d, height=d * (rng.uniform(1.0, 2.0) if kind == "uniaxial" else 0.4),
                    steps=rng.randint(500, 4000))
    if f == "train":
        return dict(family=f, rows=_log(rng, 3000, 1500000), steps=rng.randint(2, 4))
    if f == "forward":
        return dict(family=f, rows=_log(rng, 200, 2000000))
    return dict(family=f, n=_log(rng, 1500, 20000), radii=rng.choice(["uniform", "log-uniform"]),
                aspect=rng.choice([0.5, 1.0, 2.0]))


# --- packed specimens -----------------------------------------------------------
_LIBRARY = {}


def _packing(n, radii, aspect):
    key = (n, radii, aspect)
    if key not in _LIBRARY:
        lo, hi = RADII[radii]
        P, rad, _, H, _ = rfdem.pack_cylinder(n, R0, rmin=lo, rmax=hi, aspect=aspect, phi=PHI, seed=0xB2000000 + n,
                                              dist=radii)
        _LIBRARY[key] = (P.reshape(3, n), rad, H)
    return _LIBRARY[key]


def _column(n, drums, radii, aspect, rng):
    """`drums` packings on top of one another, each turned about the axis by its own angle;
    the column's aspect is `aspect`."""
    P, rad, H = _packing(n, radii, aspect / drums)
    parts = []
    for d in range(drums):
        a = rng.uniform(0.0, 2.0 * math.pi)
        c, s = math.cos(a), math.sin(a)
        parts.append(np.stack([c * P[0] - s * P[1], s * P[0] + c * P[1], P[2] + d * H]))
    return np.concatenate(parts, 1).reshape(-1), np.tile(rad, drums), H * drums


def _uniaxial(case, seed):
    rng = np.random.default_rng(seed)
    P, rad, H = _column(case["n"], case["drums"], case.get("radii", "uniform"), 2.0, rng)
    # strain rate 0.1/s, dt 1e-8 s; the fracture stop is out of reach of a block of steps
    t, R = rfdem.make_test_ext(rfdem.RF_TEST_UNIAXIAL, P, rad, R0, K=K, dt=0.01, v_load=-0.1 * H * 1e-6, max_strain=1.0,
                               min_stress=1e30)
    x = rfdem.ext_params_si(seed=0xB2000000 + seed)
    x.list_gap = case.get("gap", 0.25) * R0
    return t, R, rad, x


def _discs(case, seed):
    rng = np.random.default_rng(seed)
    tasks, params, Rs, rads = [], [], [], []
    m = case["specimens"]
    for q in range(m):
        n = int(round(math.exp(math.log(case["nmin"]) + (q + 0.5) / m * math.log(case["nmax"] / case["nmin"]))))
        P, rad, _ = _column(n, 1, "uniform", 0.5, rng)
        t, R = rfdem.make_test_ext(rfdem.RF_TEST_BRAZIL, P, rad, R0, K=K, dt=0.01, v_load=-5e-5, max_strain=1.0)
        tasks.append(t)
        params.append(rfdem.ext_params_si(weibull_m=rng.uniform(3.0, 10.0), seed=0xB2000000 + 1000 * seed + q))
        Rs.append(R)
        rads.append(rad)
    return tasks, params, Rs, rads


# --- the reference model's lattice specimens -------------------------------------
def _lattice(case, seed):
    kind = rfdem.RF_TEST_BRAZIL if case.get("kind") == "brazil" else rfdem.RF_TEST_UNIAXIAL
    return rfdem.make_test(kind, case["diameter"], case["height"], seed=0xB2000000 + seed, K=K)


def _clone(t):
    return type(t).from_buffer_copy(t)


def _md_state(case, seed):
    """Device buffers of a program with its own step loop: the lattice specimen squeezed by
    1.5 % before its bonds are made (overlapping pairs), a tenth of the slots broken (they
    go on as contacts), small random velocities and spins."""
    t, R = _lattice(case, seed)
    N, CN = int(t.N), int(t.C.N)
    g = torch.Generator(device="cuda").manual_seed(seed)
    dev = dict(device="cuda")
    c = torch.tensor([t.S.center.x, t.S.center.y, t.S.center.z], **dev)[:, None]
    x = (c + 0.985 * (torch.from_numpy(R).cuda().reshape(3, N) - c)).reshape(-1)
    s = dict(t=t, N=N, CN=CN, steps=case["steps"], R=x.contiguous(),
             V=1e-5 * torch.randn(3 * N, generator=g, **dev), W=1e-5 * torch.randn(3 * N, generator=g, **dev),
             F=torch.zeros(3 * N, **dev), M=torch.zeros(3 * N, **dev),
             CI=torch.zeros(N, dtype=torch.int64, **dev), CIs=torch.zeros(2 * N, dtype=torch.int64, **dev),
             pnC=torch.zeros(2 * CN, dtype=torch.int64, **dev), IL=torch.zeros(N * K, dtype=torch.int64, **dev),
             ty=torch.zeros(N * K, dtype=torch.uint8, **dev), iL=torch.zeros(N * K, **dev),
             FL=torch.zeros(2 * int(t.bloks), **dev), FLh=torch.zeros(2 * int(t.bloks)).pin_memory())
    s["sb"] = int(rfdem.lib.md_CellDistributionScratchBytes(N, CN))
    s["scratch"] = torch.zeros(s["sb"], dtype=torch.uint8, **dev)
    for k in ("Rij", "Oijt", "Fijn", "Fijt", "Mijn", "Mijt", "Mijadd"):
        s[k] = torch.zeros(3 * N * K, **dev)
    torch.cuda.synchronize()
    p = {k: v.data_ptr() for k, v in s.items() if isinstance(v, torch.Tensor)}
    s["p"] = p
    L, C = rfdem.lib, t.C
    rfdem.check(L.md_CellDistribution(p["R"], N, p["CI"], p["CIs"], p["pnC"], CN, C._1d_a, C.Nr, p["scratch"], s["sb"],
                                      None))
    rfdem.check(L.md_InteractionListConstruct(p["R"], N, p["CIs"], p["pnC"], p["IL"], K, C.a, C._1d_a, t.aacut, C.Nr, CN,
                                              None))
    rfdem.check(L.md_ConstructBoundInteractions(p["R"], p["V"], p["W"], p["IL"], p["ty"], p["iL"], p["Rij"], p["Oijt"],
                                                p["Fijn"], p["Fijt"], p["Mijn"], p["Mijt"], p["Mijadd"], N, K,
                                                t.Po.b_dd, t.Po.b_r, None))
    s["ty"] *= (torch.rand(N * K, generator=g, **dev) >= 0.1).to(torch.uint8)
    torch.cuda.synchronize()
    return s


def _md_run(s):
    L, t, p, N, CN = rfdem.lib, s["t"], s["p"], s["N"], s["CN"]
    P, C, S, Q = t.Po, t.C, t.S, t.Compress
    for _ in range(s["steps"]):
        rfdem.check(L.md_CellDistribution(p["R"], N, p["CI"], p["CIs"], p["pnC"], CN, C._1d_a, C.Nr, p["scratch"],
                                          s["sb"], None))
        rfdem.check(L.md_InteractionListReConstructBPM(p["R"], N, p["CIs"], p["pnC"], p["IL"], p["ty"], K, C.a, C._1d_a,
                                                       t.aacut, C.Nr, CN, None))
        s["F"].zero_()
        s["M"].zero_()
        rfdem.check(L.md_CalculateForcesDEM_22(p["R"], p["V"], p["W"], p["IL"], p["ty"], p["iL"], p["Rij"], p["Oijt"],
                                               p["Mijn"], p["Mijt"], p["F"], p["M"], N, K, P.dt, P.m_E, P.m_G, P.b_r,
                                               P.m_Ec, P.m_Gc, None))
        rfdem.check(L.md_CalculateForcesDEM_21(p["R"], p["V"], p["W"], p["IL"], p["ty"], p["iL"], p["Rij"], p["Oijt"],
                                               p["F"], p["M"], N, K, P.dt, P.hm_E, P.hm_G, P.p_A, P.p_mu, P.p_mur,
                                               P.p_m, P.p_r, None))
        rfdem.check(L.md_UniaxialCompression3_simple(p["R"], p["V"], p["F"], p["FL"], N, Q.center, Q.RR, Q.Top,
                                                     Q.Bottom, Q.TopR, Q.BottomR, Q.V, S.center.z + S.spacesized2.z,
                                                     t.bloks, None))
        s["FLh"].copy_(s["FL"])
        rfdem.check(L.md_SumForcesULoading(ctypes.byref(t), s["FLh"].data_ptr(), t.bloks, 0, 1, t.sz0, None, None))
        rfdem.check(L.md_CalculateIncrementsDEM(p["F"], p["V"], p["R"], p["M"], p["W"], N, P.dt_d_m, P.dt, P.dt_d_I,
                                                None))
        rfdem.check(L.md_ParallelepipedCutRestriction(p["R"], p["V"], p["F"], N, S.center, S.spacesized2, S.hidenpoint,
                                                      None))
        rfdem.check(L.md_DeleteFarLinks(p["R"], N, p["IL"], p["ty"], p["iL"], p["Rij"], p["Oijt"], p["Fijn"], p["Fijt"],
                                        p["Mijn"], p["Mijt"], p["Mijadd"], K, P.aa_farcut, None))
        rfdem.check(L.md_CompressU(ctypes.byref(t), Q.Stress))
    return {k: s[k] for k in ("R", "V", "W", "IL", "ty", "Rij", "Oijt", "Mijn", "Mijt")}


# --- the warm-start MLP ------------------------------------------------------------
def _mlp_inputs(rows, seed):
    """Features in the ranges a specimen gives (last motion of order 1, neighbours' relative
    motion smaller, constant and empty columns), corrections to learn, He-uniform weights."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    X = torch.randn(rows, 64, generator=g, device="cuda")
    X[:, 8:56] *= 0.2
    X[:, 58] = 1.0
    X[:, 59:] = 0.0
    X = X.bfloat16()
    T = 0.3 * torch.tanh(X[:, :6].float() + X[:, 6:12].float()) + 0.05 * torch.randn(rows, 6, generator=g, device="cuda")
    rng = np.random.default_rng(seed)
    W = []
    for l, (i, o) in enumerate(zip(rfdem.MLP_DIN, rfdem.MLP_DOUT)):
        w = rng.uniform(-1.0, 1.0, (o, i)) * math.sqrt(6.0 / i)
        b = rng.uniform(-0.1, 0.1, o)
        if l == 3:
            w[6:] = 0.0
            b[6:] = 0.0
        W.append((w.astype(np.float32), b.astype(np.float32)))
    return X, T.contiguous(), W


LR = 1e-3


# --- prepare / run ------------------------------------------------------------------
def prepare(case, seed):
    f = case["family"]
    if f == "explicit":
        t, R, rad, x = _uniaxial(case, seed)
        e = rfdem.Engine(t, R, ext=x, radius=rad)
        e.affine_strain(case["pre_lat"], case["pre_lat"], case["pre_ax"])
        return dict(f=f, e=e, steps=case["steps"], out=torch.empty(3 * e.N).pin_memory())
    if f == "batch":
        e = rfdem.BatchEngine(*_discs(case, seed))
        return dict(f=f, e=e, steps=case["steps"])
    if f == "fire":
        if case["mode"] == "batch":
            parts = [_uniaxial(dict(case, n=case["n"] + 211 * q), 64 * seed + q) for q in range(case["specimens"])]
            e = rfdem.BatchEngine([a[0] for a in parts], [a[3] for a in parts], [a[1] for a in parts],
                                  [a[2] for a in parts])
        else:
            t, R, rad, x = _uniaxial(case, seed)
            e = rfdem.Engine(t, R, ext=x, radius=rad)
        p = e.relax_params(max_iter=case["iters"], tol=1e-12)
        e.load_increment(p)                      # the run is under way: its buffers exist, a motion to predict from
        s = dict(f=f, e=e, p=p)
        if case["mode"] == "warm":
            s["ws"] = WarmStart(e.N, p.strain_inc, seed=seed)
            s["ws"].mlp.set_weights(_mlp_inputs(128, seed)[2])
            s["ws"].cmax = torch.full((6,), 0.01, device="cuda")
        return s
    if f == "create":
        t, R, rad, x = _uniaxial(case, seed)
        return dict(f=f, t=t, R=R, rad=rad, x=x, pre=(case["pre_lat"], case["pre_lat"], case["pre_ax"]),
                    steps=case["steps"])
    if f == "reference":
        t, R = _lattice(case, seed)
        e = rfdem.Engine(t, R)
        return dict(f=f, e=e, steps=case["steps"], out=torch.empty(3 * e.N).pin_memory())
    if f == "driver":
        t, R = _lattice(case, seed)
        return dict(f=f, t=t, R=R, steps=case["steps"])
    if f == "md":
        return dict(_md_state(case, seed), f=f)
    if f in ("train", "forward"):
        X, T, W = _mlp_inputs(case["rows"], seed)
        m = rfdem.MLP(seed)
        m.set_weights(W)
        rows = case["rows"]
        return dict(f=f, m=m, X=X, T=T, rows=rows, steps=case.get("steps", 1),
                    Y=torch.zeros((rows + 127) // 128 * 128, 16, device="cuda"))
    lo, hi = RADII[case["radii"]]
    return dict(f=f, n=case["n"], seed=0xB2000000 + seed,
                kw=dict(rmin=lo, rmax=hi, aspect=case["aspect"], phi=PHI, dist=case["radii"]))


def run(s):
    f = s["f"]
    if f in ("explicit", "reference"):
        s["e"].step_host(None, s["steps"], s["out"])
        _, r = s["e"].sync()
        return {"R": s["out"], "stress": r.Stress, "strain": r.Strain, "broken": int(r.broken_bonds)}
    if f == "batch":
        s["e"].step(s["steps"])
        rs = [s["e"].sync_spec(q)[1] for q in range(s["e"].nspec)]
        return {"R": s["e"].positions_f64(), "stress": np.array([r.Stress for r in rs]),
                "broken": int(rs[0].broken_bonds)}
    if f == "fire":
        if "ws" in s:
            r = [s["e"].load_increment_pred(s["p"], s["ws"].predict(s["e"]))]
        else:
            r = s["e"].load_increment(s["p"])
            r = r if isinstance(r, list) else [r]
        return {"R": s["e"].positions_f64(), "iterations": np.array([int(a.iterations) for a in r])}
    if f == "create":
        e = rfdem.Engine(_clone(s["t"]), s["R"], ext=s["x"], radius=s["rad"])
        e.affine_strain(*s["pre"])
        e.step(s["steps"])
        R = e.positions_f64()
        _, r = e.sync()
        e.close()
        return {"R": R, "broken": int(r.broken_bonds), "bonds": int(r.bonds_initial)}
    if f == "driver":
        res, curve, R = rfdem.run_test(_clone(s["t"]), s["R"], max_steps=s["steps"], curve_cap=s["steps"],
                                       want_positions=True)
        return {"R": R, "strain": np.ascontiguousarray(curve[:, 0]), "steps": int(res.steps),
                "broken": int(res.broken_bonds)}
    if f == "md":
        return _md_run(s)
    if f == "train":
        loss = [s["m"].train_step(s["X"], s["T"], s["rows"], LR) for _ in range(s["steps"])]
        return {"loss": np.array(loss), "weights": s["m"].weights()}
    if f == "forward":
        s["m"].forward(s["X"], s["rows"], s["Y"])
        torch.cuda.synchronize()                 # the pass runs on the MLP's own stream
        return s["Y"][:s["rows"], :6]
    R, rad, D, H, mo = rfdem.pack_cylinder(s["n"], R0, seed=s["seed"], **s["kw"])
    return {"R": R, "radius": rad, "diameter": D, "height": H}


# --- what a pass cannot do without ----------------------------------------------------
# Per particle and explicit step of the extended model: FP64 position, velocity and spin
# read and written, per bond record (b a particle) its partner, rest length, strengths
# and its state read and written, per contact (c) its overlap read and written. Where the
# state of a specimen stays in the L2 cache this is its traffic there, not in memory.
_FLOP_BOND, _FLOP_CONTACT, _FLOP_PARTICLE = 260, 150, 60


def _ext_step(b, c):
    return 128 + 117 * b + 24 * c, _FLOP_BOND * b + _FLOP_CONTACT * c + _FLOP_PARTICLE


def _lattice_n(case):
    return max(1, int(math.pi / 4 * case["diameter"] ** 2 * case["height"] / 1.02 ** 3 * 0.94))


def work(case):
    f = case["family"]
    if f in ("explicit", "create", "batch", "fire"):
        damaged = case.get("pre_lat", 0.0) > 0.05
        b, c = (2.6, 0.3) if damaged else (5.0, 1.0) if f == "explicit" else (5.0, 0.0)
        B, F = _ext_step(b, c)
        if f == "batch":
            m = case["specimens"]
            n = sum(math.exp(math.log(case["nmin"]) + (q + 0.5) / m * math.log(case["nmax"] / case["nmin"]))
                    for q in range(m))
        else:
            n = case["n"] * case["drums"] * case.get("specimens", 1)
        if f == "fire":                          # start positions and rotations, force and moment besides
            return {"bytes": n * case["iters"] * (B + 160 + 48), "flops": n * case["iters"] * (F + 60)}
        return {"bytes": n * (case["steps"] * B + (24 if f == "create" else 12)), "flops": n * case["steps"] * F}
    if f in ("reference", "driver"):             # FP32 positions
        n = _lattice_n(case)
        return {"bytes": n * case["steps"] * (96 + 105 * 5.9), "flops": n * case["steps"] * (200 * 5.9 + 40)}
    if f == "md":                                # rows of ids and types, bond state, particle vectors
        n = _lattice_n(case)
        return {"bytes": n * case["steps"] * (K * 9 + 5.3 * (100 + 4) + 0.6 * 24 + 144),
                "flops": n * case["steps"] * (200 * 5.3 + 120 * 0.6 + 40)}
    macs = sum(i * o for i, o in zip(rfdem.MLP_DIN[:3], rfdem.MLP_DOUT[:3])) + 128 * 6
    if f == "forward":
        return {"bytes": case["rows"] * (128 + 64) + 4 * macs, "flops": 2.0 * case["rows"] * macs}
    if f == "train":                             # forward, input gradients of three layers, weight gradients
        return {"bytes": case["steps"] * (case["rows"] * (128 + 24) + 28.0 * macs),
                "flops": 2.0 * case["steps"] * case["rows"] * (3 * macs - 64 * 128)}
    return {"bytes": case["n"] * 2000 * 200.0, "flops": case["n"] * 2000 * 500.0}


# --- 64-bit values ----------------------------------------------------------------------
# The reference model and the MLP have them. A specimen of the extended model in its
# damage regime, a relaxation stopped after a number of iterations and a packing follow
# trajectories in which rounding grows until another bond breaks or another step is
# rejected: what 64 bits gives is another run, not the value of this one.
def _pairs(x, cut):
    """Directed pairs (i, j) nearer than cut; x [N, 3]."""
    c = torch.floor((x - x.min(0).values) / cut).long() + 1
    n = c.max(0).values + 2
    key = (c[:, 2] * n[1] + c[:, 1]) * n[0] + c[:, 0]
    sk, order = torch.sort(key)
    got = []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                k = key + (dz * n[1] + dy) * n[0] + dx
                lo, hi = torch.searchsorted(sk, k), torch.searchsorted(sk, k, right=True)
                for m in range(int((hi - lo).max())):
                    i = torch.nonzero(lo + m < hi)[:, 0]
                    j = order[lo[i] + m]
                    near = (j != i) & ((x[j] - x[i]).square().sum(1) < cut * cut)
                    got.append(torch.stack([i[near], j[near]]))
    return torch.cat(got, 1)


def _cross(a, b):
    return torch.linalg.cross(a, b)


def _dot(a, b):
    return (a * b).sum(1, keepdim=True)


def _f32(v):
    return float(np.float32(v))


def _march64(t, x, v, w, i, j, il, bond, steps):
    """`steps` explicit steps of the reference model in 64 bits. i, j: directed pairs; il
    [P, 1] and bond [P]: 1 / rest length and intact bonds; particle arrays [N, 3]."""
    P, C = t.Po, t.Compress
    dt, E, G, br, Ec, Gc = (_f32(a) for a in (P.dt, P.m_E, P.m_G, P.b_r, P.m_Ec, P.m_Gc))
    hE, hG, pA, mu, mur, mP, rP = (_f32(a) for a in (P.hm_E, P.hm_G, P.p_A, P.p_mu, P.p_mur, P.p_m, P.p_r))
    dtm, dtI = _f32(P.dt_d_m), _f32(P.dt_d_I)
    brazil = t.kind == rfdem.RF_TEST_BRAZIL
    ax, lat = (1, 2) if brazil else (2, 1)
    cen = [C.center.x, C.center.y, C.center.z]
    zcut = t.S.center.y + t.S.spacesized2.y if brazil else t.S.center.z + t.S.spacesized2.z
    top, bot, topr, botr, vel = C.Top, C.Bottom, C.TopR, C.BottomR, C.V
    A, J = math.pi * br * br, math.pi * br ** 4
    zero = torch.zeros(len(i), 3, dtype=torch.float64, device=x.device)
    rij, ot, mn, mt = zero, zero.clone(), zero.clone(), zero.clone()
    bond = bond.clone()
    strain = []
    for _ in range(steps):
        strain.append((C.size_d.z - t.sz0) / t.sz0 if brazil else (C.size_d.z + (top - C.Top) - t.sz0) / t.sz0)
        F, M, Mc = torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(x)
        b = torch.nonzero(bond)[:, 0]
        if len(b):
            ib, jb, l = i[b], j[b], il[b]
            r = x[jb] - x[ib]
            d = r.norm(dim=1, keepdim=True)
            n = r / d
            ten = E * (d - 1 / l) * l
            tv = _cross(rij[b], n)
            ws, dw = w[jb] + w[ib], w[jb] - w[ib]
            ph = n * _dot(ws, n) * dt * 0.5
            turn = lambda q: q + _cross(tv - ph, q) + _dot(tv, ph) * q - ph * _dot(tv, q)  # noqa: E731
            c1 = _dot(n, dw)
            mn_, mt_ = turn(mn[b]) + n * c1 * (dt * 0.5 * G * l), turn(mt[b]) + (dw - n * c1) * (dt * 0.25 * E * l)
            u = v[jb] - v[ib] - _cross(0.5 * ws, r)
            ot_ = turn(ot[b]) + (u - n * _dot(n, u)) * dt
            k = G * l * A
            F.index_add_(0, ib, n * ten * A + ot_ * k)
            M.index_add_(0, ib, mn_ * J + mt_ * (dt * 0.25 * E * l) * J + 0.5 * _cross(r, ot_) * k)
            broke = ((ten + mt_.norm(dim=1, keepdim=True) * 4 * br > Ec) |
                     (G * l * ot_.norm(dim=1, keepdim=True) + mn_.norm(dim=1, keepdim=True) * 2 * br > Gc))
            keep = (~broke).double()
            rij[b], ot[b], mn[b], mt[b] = n, ot_ * keep, mn_ * keep, mt_ * keep
            bond[b] = ~broke[:, 0]
        a = torch.nonzero(~bond)[:, 0]
        a = a[(x[j[a]] - x[i[a]]).norm(dim=1) < 2 * rP] if len(a) else a
        if len(a):
            ia, ja = i[a], j[a]
            r = x[ja] - x[ia]
            d = r.norm(dim=1, keepdim=True)
            n = r / d
            c0 = torch.sqrt(rP * (rP - 0.5 * d).abs())
            Kn, Kt = 2 * hE * c0, 8 * hG * c0
            u = v[ja] - v[ia] + rP * _cross(n, w[ja] + w[ia])
            vn = _dot(n, u)
            fn = (d - 2 * rP) * Kn * (2.0 / 3.0)
            ut = u - n * vn
            o = ot[a]
            q = o - n * _dot(n, o)
            q2 = _dot(q, q)
            q = torch.where(q2 > 1e-18, q * torch.sqrt(_dot(o, o) / q2.clamp(min=1e-300)), q) + ut * dt
            ft = q * Kt
            fm = ft.norm(dim=1, keepdim=True)
            slip = fm > mu * fn.abs()
            cap = ft * (mu * fn.abs() / fm.clamp(min=1e-300))
            ot[a] = torch.where(slip, cap / Kt, q)
            ft = torch.where(slip, cap, ft - 1.8257 * pA * torch.sqrt(Kt * 0.5 * mP) * ut)
            F.index_add_(0, ia, n * (fn - 1.8257 * pA * vn * torch.sqrt(Kn * 0.5 * mP)) + ft)
            wi = w[ia]
            wn = wi.norm(dim=1, keepdim=True)
            Mc.index_add_(0, ia, _cross(n, ft) * rP - wi * (mur * fn.abs() / wn.clamp(min=1e-300)))
            Mc = Mc * (w.square().sum(1, keepdim=True) > 1e-18)
        M = M + Mc
        zone = ((x[:, 0] - cen[0]).square() + (x[:, lat] - cen[lat]).square() < C.RR) & (x[:, 2] < zcut)
        f0 = F[:, ax].clone()
        at, ab = zone & (x[:, ax] - topr > -1e-9), zone & (x[:, ax] - botr < 1e-9)
        stress = 0.5 * float((f0 * (at & (f0 > 0))).sum().abs() + (f0 * (ab & (f0 < 0))).sum().abs()) * C._1d_Area
        if brazil:                                # friction along the platens
            vl = torch.sqrt(v[:, 0] ** 2 + v[:, 2] ** 2)
            on = ((at & (f0 > 0)) | (ab & (f0 < 0))) & (vl * vl > 1e-9)
            s = on * 0.45 * f0.abs() / vl.clamp(min=1e-300)
            F[:, 0] -= s * v[:, 0]
            F[:, 2] -= s * v[:, 2]
        for on, at_x, at_v in ((zone & (x[:, ax] - top > -1e-9), top, vel), (zone & (x[:, ax] - bot < 1e-9), bot, 0.0)):
            x[:, ax] = torch.where(on, torch.full_like(f0, at_x), x[:, ax])
            v[:, ax] = torch.where(on, torch.full_like(f0, at_v), v[:, ax])
            F[:, ax] = F[:, ax] * ~on
        v = v + F * dtm
        x = x + v * dt
        w = w + M * dtI
        vel = 10.0 * C.VLoad if stress < 1e-9 else C.VLoad
        top += vel * P.dt
        topr = top - 2.0 * P.p_r
    return x, v, w, strain


def _mlp64(case, seed, train):
    X, T, W = _mlp_inputs(case["rows"], seed)
    W = [[torch.from_numpy(a).cuda().double().requires_grad_(train) for a in wb] for wb in W]

    def net(x):
        for l, (w, b) in enumerate(W):
            x = x @ w.T + b
            x = torch.relu(x) if l < 3 else x
        return x[:, :6]
    if not train:
        return net(X.double())
    flat = [a for wb in W for a in wb]
    m, v = [torch.zeros_like(a) for a in flat], [torch.zeros_like(a) for a in flat]
    losses = []
    for k in range(1, case["steps"] + 1):
        grads, loss = [torch.zeros_like(a) for a in flat], 0.0
        for q in range(0, case["rows"], 250000):
            e = (net(X[q:q + 250000].double()) - T[q:q + 250000].double()).square().sum() / (case["rows"] * 6)
            loss += float(e)
            grads = [a + b for a, b in zip(grads, torch.autograd.grad(e, flat))]
        losses.append(loss)
        with torch.no_grad():
            for a, g, p, q in zip(flat, grads, m, v):
                p.mul_(0.9).add_(0.1 * g)
                q.mul_(0.999).add_(0.001 * g * g)
                a -= LR * (p / (1 - 0.9 ** k)) / (torch.sqrt(q / (1 - 0.999 ** k)) + 1e-8)
    return {"loss": np.array(losses), "weights": [tuple(a.detach() for a in wb) for wb in W]}


def exact(case, seed):
    f = case["family"]
    if f == "forward":
        return _mlp64(case, seed, False)
    if f == "train":
        return _mlp64(case, seed, True)
    if f in ("reference", "driver"):
        t, R = _lattice(case, seed)
        x = torch.from_numpy(R).cuda().double().reshape(3, -1).T.contiguous()
        i, j = _pairs(x, t.Po.a_farcut)
        d = (x[j] - x[i]).norm(dim=1)
        x, v, w, strain = _march64(t, x, torch.zeros_like(x), torch.zeros_like(x), i, j, 1 / d[:, None], d < t.Po.b_d,
                                   case["steps"])
        R = x.T.reshape(-1)
        if f == "driver":
            # (the platen starts at ten times its speed until the first reaction is felt: in a
            # cylinder's first steps that reaction is of the order of float rounding)
            return {"R": R, "strain": np.array(strain) if case["kind"] == "brazil" else None, "steps": None,
                    "broken": None}
        return {"R": R, "stress": None, "strain": None, "broken": None}
    if f == "md":
        s = _md_state(case, seed)
        N = s["N"]
        k = torch.nonzero((s["IL"] >= 0) & (s["IL"] < N))[:, 0]
        i, j = k // K, s["IL"][k]
        x, v, w = (s[a].double().reshape(3, N).T.contiguous() for a in ("R", "V", "W"))
        d = (x[j] - x[i]).norm(dim=1)
        x, v, w, _ = _march64(s["t"], x, v, w, i, j, 1 / d[:, None], s["ty"][k] == 1, case["steps"])
        out = {a: None for a in ("IL", "ty", "Rij", "Oijt", "Mijn", "Mijt")}
        return dict(out, R=x.T.reshape(-1), V=v.T.reshape(-1), W=w.T.reshape(-1))
    return None
