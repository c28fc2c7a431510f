"""Measured cases: the work a program gives this library, through its public entry points.

A case names a kind of program and its sizes:

  steps     a beam resident on the GPU (Solver), advanced a chunk of time steps, then its state read back
  batch     several beams advanced together (Batch), as the serving form does between two looks at the loads
  static    load steps of the static solver (StaticSolver)
  routines  one time step through the per-routine device entry points, as a program that keeps the
            reference's own loop and its arrays on the GPU
  inputs    the input module on the device: horizons, volume correction, bond data, masses
  solve     a whole job from host arrays: create, step, read everything back

Beams are the synthetic ones of bb_pd_b200.beam. The seed draws what differs from one realisation of a
beam to the next: Young's modulus, the loading rate, and the lognormal critical stretch where a case has one.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import bb_pd_b200 as bb
from bb_pd_b200 import _native as N

LAWKW = {
    "linear": dict(law="linear", sc=2e-3),
    "bilinear": dict(law="bilinear", s0=1e-4, sc=2e-3),
    "trilinear": dict(law="trilinear", s0=1e-4, s1=3e-4, sc=2e-3),
    "exponential": dict(law="exponential", s0=1e-4, sc=2e-3),
}
LAWS = ("linear", "bilinear", "trilinear", "exponential")
RATE = -1e-11       # metres per step at the loaded nodes: quasi-static, elastic over a run of these cases
RATE32 = -5e-9      # the FP32 form's, at 2.5 mm spacing: its force rounding is absolute, it is used at larger displacements
BREAK_RATE = -1e-7  # the rate that takes a beam of 20 nodes depth at 5 mm past its peak in about 1 200 steps


def listed():
    return [
        # a test-sized beam under the reference's default scheme and law: latency of launch, barrier and one wave
        _steps("small_ec_exp", 24, 5, 6, 5e-3, "exponential", "eulercromer", steps=200),
        # the 20 000-node beam, one chunk of a serving loop
        _steps("beam20k_adr_tri", 100, 10, 20, 5e-3, "trilinear", "adr", steps=100),
        # the same beam past its peak load, held there: most of the work in bonds that have softened or broken
        _steps("beam20k_postpeak", 100, 10, 20, 5e-3, "trilinear", "adr", state="postpeak", steps=100),
        # notched beam, exponential law, a critical stretch per bond
        _steps("notched128k_adr_exp", 160, 20, 40, 2.5e-3, "exponential", "adr", sc="lognormal", notch=True, steps=100),
        # the benchmark's beam, 1.28M nodes
        _steps("beam1280k_adr_tri", 400, 40, 80, 1.25e-3, "trilinear", "adr", steps=500),
        # the FP32 form on a beam whose sides are no multiple of anything
        _steps("beam253k_fp32", 161, 39, 41, 2.5e-3, "trilinear", "adr", prec="fp32", steps=200),
        # eight beams of a size-effect series, depths 50 to 150 mm, two laws
        dict(name="batch8_series", kind="batch", members=8, depth=0.15, dx=5e-3, prec="fp64", steps=100),
        # one load step of the static solver on the 20 000-node beam
        dict(name="static20k_bilinear", kind="static", nx=100, ny=10, nz=20, dx=5e-3, law="bilinear"),
        # the reference's Euler-Cromer loop body on device arrays, 7.1M bonds
        dict(name="routines7M_ec_exp", kind="routines", nx=160, ny=20, nz=40, dx=2.5e-3, scheme="eulercromer"),
        # its ADR body on a small, odd-sized beam: many short launches
        dict(name="routines50k_adr_tri", kind="routines", nx=31, ny=7, nz=9, dx=5e-3, scheme="adr"),
        # the input module on a slightly irregular cloud of 20 000 points
        dict(name="inputs20k", kind="inputs", nx=100, ny=10, nz=20, dx=5e-3),
        # a whole job from host arrays, odd sizes, every field read back
        dict(name="solve29k_exp", kind="solve", nx=103, ny=13, nz=22, dx=5e-3, law="exponential", steps=100),
    ]


def _steps(name, nx, ny, nz, dx, law, scheme, prec="fp64", sc="scalar", notch=False, state="elastic", steps=100):
    c = dict(kind="steps", nx=nx, ny=ny, nz=nz, dx=dx, law=law, scheme=scheme, prec=prec, sc=sc, notch=notch,
             state=state, steps=steps)
    if name:
        c["name"] = name
    return c


def _sides(rng, lo, hi):
    """Sides of a beam of lo .. hi nodes (log-uniform), about 5 : 0.5 to 1 : 1, any parity."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    w = rng.uniform(0.5, 1.0)
    a = (n / (5.0 * w)) ** (1.0 / 3.0)
    nz = max(4, round(a))
    ny = max(3, round(w * a))
    nx = max(12, round(n / (ny * nz)))
    return nx, ny, nz


def draw(rng):
    kind = rng.choice(("steps", "steps", "steps", "steps", "batch", "static", "routines", "routines", "inputs", "solve"))
    dx = rng.choice((1.25e-3, 2.5e-3, 5e-3))
    if kind == "steps":
        state = rng.choice(("elastic", "elastic", "elastic", "postpeak"))
        if state == "postpeak":
            nx, ny, nz = _sides(rng, 1e4, 4e4)
            return _steps("", nx, ny, nz, 5e-3, rng.choice(LAWS), "adr", state=state, steps=100)
        prec = rng.choice(("fp64", "fp64", "fp32"))
        nx, ny, nz = _sides(rng, 1e5 if prec == "fp32" else 700, 1e6)   # the FP32 form is for large beams
        big = nx * ny * nz > 100000
        scheme = rng.choice(("adr", "adr", "eulercromer"))
        sc = rng.choice(("scalar", "lognormal"))
        return _steps("", nx, ny, nz, dx, rng.choice(LAWS), scheme, prec=prec, sc=sc, notch=rng.random() < 0.3,
                      steps=rng.randint(100, 200) if big else rng.randint(50, 300))
    if kind == "batch":
        return dict(kind="batch", members=rng.randint(2, 12), depth=rng.uniform(0.06, 0.15), dx=5e-3,
                    prec=rng.choice(("fp64", "fp64", "fp32")), steps=rng.randint(30, 100))
    if kind == "static":
        nx, ny, nz = _sides(rng, 2e3, 6e4)
        return dict(kind="static", nx=nx, ny=ny, nz=nz, dx=dx, law=rng.choice(LAWS))
    if kind == "routines":
        nx, ny, nz = _sides(rng, 700, 1.5e5)
        return dict(kind="routines", nx=nx, ny=ny, nz=nz, dx=dx, scheme=rng.choice(("adr", "eulercromer")))
    if kind == "inputs":
        nx, ny, nz = _sides(rng, 1e3, 2e5)
        return dict(kind="inputs", nx=nx, ny=ny, nz=nz, dx=dx)
    nx, ny, nz = _sides(rng, 2e3, 1.2e5)
    return dict(kind="solve", nx=nx, ny=ny, nz=nz, dx=dx, law=rng.choice(LAWS), steps=rng.randint(50, 200))


# ---- what a program has in hand before the call ----

def _rate(case):
    return RATE32 * case["dx"] / 2.5e-3 if case.get("prec") == "fp32" else RATE


def _beam(case, seed):
    """Host arrays of the case's beam for this seed, and the loading rate."""
    rng = np.random.default_rng(seed)
    E = 37e9 * (1 + 0.05 * rng.standard_normal())
    rate = _rate(case) * (1 + 0.05 * rng.standard_normal())
    nx, dx = case["nx"], case["dx"]
    kw = {}
    if case.get("notch"):   # between two node planes, right of midspan, 0.4 of the depth
        kw.update(notch_x=dx * (int(0.72 * nx) + 1.5), notch_depth=0.4 * case["nz"] * dx)
    if case.get("sc") == "lognormal":
        kw.update(sc_lognormal=(2e-3, 0.1))
    s = bb.beam.spec(nx, case["ny"], case["nz"], dx, E=E, supports=(2.25 * dx, (nx - 1.75) * dx),
                     seed=int(rng.integers(1 << 30)), **kw)
    return bb.beam.build(s), rate


def _solver(case, inp, rate, **kw):
    return bb.Solver(inp, scheme=case.get("scheme", "adr"), precision=case.get("prec", "fp64"), rate=rate,
                     **{**LAWKW[case["law"]], **kw})


def prepare(case, seed):
    kind = case["kind"]
    if kind == "steps":
        inp, rate = _beam(case, seed)
        if case["state"] == "postpeak":
            # load past the peak, then go on from the checkpoint with the load held
            n = round(1500 * (case["dx"] / 5e-3) * (case["nz"] / 20))
            s = _solver(case, inp, BREAK_RATE * (rate / RATE))
            s.step(n)
            ck = s.checkpoint()
            s.close()
            hold = -1e-13
            ck["step"] = round(BREAK_RATE * (rate / RATE) * n / hold)
            s = _solver(case, inp, hold)
            s.restore(ck)
        else:
            s = _solver(case, inp, rate)
        return dict(case=case, s=s)
    if kind == "batch":
        rng = np.random.default_rng(seed)
        rate = _rate(case) * (1 + 0.05 * rng.standard_normal())
        members = []
        for sp, law in bb.beam.size_effect_series(case["members"], depth_range=(0.05, case["depth"]), dx=case["dx"]):
            sp.seed = int(rng.integers(1 << 30))   # the depths stay, the material is drawn anew
            members.append(bb.Solver(bb.beam.build(sp), scheme="adr", precision=case["prec"], rate=rate, **LAWKW[law]))
        b = bb.Batch(case["prec"])
        for m in members:
            b.add(m)
        return dict(case=case, batch=b, members=members)
    if kind == "static":
        inp, rate = _beam(case, seed)
        return dict(case=case, s=bb.static.StaticSolver(inp, **LAWKW[case["law"]]), inc=-2e-7 * (case["dx"] / 5e-3) * (rate / RATE))
    if kind == "solve":
        inp, rate = _beam(case, seed)
        return dict(case=case, inp=inp, rate=rate)
    if kind == "inputs":
        X, g = _cloud(case, seed)
        return dict(case=case, X=X, **g)
    return _routine_arrays(case, seed)


def _cloud(case, seed):
    """Points of a lattice of spacing dx, each moved by up to 0.4 % of dx an axis (no family changes), and the
    scalars of the input module."""
    nx, ny, nz, dx = case["nx"], case["ny"], case["nz"], case["dx"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    f = lambda m: torch.arange(1, m + 1, device="cuda", dtype=torch.float64) * dx
    z, y, x = torch.meshgrid(f(nz), f(ny), f(nx), indexing="ij")
    X = torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)])
    X += 0.008 * dx * (torch.rand(X.shape, generator=g, device="cuda", dtype=torch.float64) - 0.5)
    h = 3.015 * dx
    return X.contiguous(), dict(horizon=h, radij=dx / 2, V=dx ** 3, bsc=18 * 37e9 / (math.pi * h ** 4),
                                nvol=4.0 / 3.0 * math.pi * h ** 3, dx=dx, dt=1.0)


def _routine_arrays(case, seed):
    inp, rate = _beam(case, seed)
    g = torch.Generator(device="cuda").manual_seed(seed)
    nN, nB, dx = inp["nNodes"], inp["nBonds"], case["dx"]
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a.T if a.ndim == 2 else a)).cuda()
    zb = lambda: torch.zeros(nB, dtype=torch.float64, device="cuda")
    zn = lambda: torch.zeros((3, nN), dtype=torch.float64, device="cuda")
    t = dict(X=dev(inp["undeformedCoordinates"]), bl=dev(inp["BONDLIST"]), L0=dev(inp["UNDEFORMEDLENGTH"]),
             BS=dev(inp["BONDSTIFFNESS"]), VCF=dev(inp["VOLUMECORRECTIONFACTORS"]), rho=dev(inp["DENSITY"]),
             mass=dev(inp["massVector"]), CF=dev(inp["CONSTRAINTFLAG"]))
    # a bent beam with a little noise: stretches on both sides of the softening limit
    x = t["X"][0]
    u = zn()
    u[2] = 4e-6 * (dx / 2.5e-3) * torch.sin(math.pi * x / x.max())
    u += 4e-8 * (dx / 2.5e-3) * torch.randn(u.shape, generator=g, device="cuda", dtype=torch.float64)
    u *= 1 - t["CF"]
    t.update(u=u, x=t["X"] + u, v=zn(), a=zn(), F=zn(), Fp=zn(), L=zb(), dX=zb(), dY=zb(), dZ=zb(), s=zb(), bsf=zb(),
             BSF=zb(), flag=zb(), fX=zb(), fY=zb(), fZ=zb(), sp=zb(), BT=zb(), fail=zb() + 1, s0=zb() + 1e-4)
    t["sc"] = 2e-3 * torch.exp(0.1 * torch.randn(nB, generator=g, device="cuda", dtype=torch.float64))
    t["v"] += 1e-9 * torch.randn(u.shape, generator=g, device="cuda", dtype=torch.float64)
    plan = C.c_void_p()
    st = torch.cuda.current_stream().cuda_stream
    N.check(N.lib().bbpd_nodal_plan_create(_p(t["bl"]), _i(nB), _i(nN), 8, C.c_void_p(st), C.byref(plan)))
    return dict(case=case, t=t, nN=nN, nB=nB, V=inp["cellVolume"], dt=inp["DT"], plan=_Plan(plan), step=2)


class _Plan:
    def __init__(self, h):
        self.h = h

    def __del__(self):
        N.lib().bbpd_nodal_plan_destroy(self.h)


def _p(t):
    return C.c_void_p(t.data_ptr())


def _i(n):
    return C.c_int64(n)


def _d(x):
    return C.c_double(x)


# ---- one pass ----

def _state(s):
    return {f: s.get(f) for f in ("displacement", "velocity", "force", "bsf", "flag", "fail")}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "steps":
        s, adr, n = state["s"], case["scheme"] == "adr", case["steps"]
        s.step(n)
        if adr:
            # between two snapshots a driver looks at the load, the shape and the damage
            return dict(reaction=s.reaction(n), displacement=s.get("displacement"), velocity=s.get("velocity"),
                        bsf=s.get("bsf"))
        return dict(displacement=s.get("displacement"), velocity=s.get("velocity"), bsf=s.get("bsf"))
    if kind == "batch":
        n = case["steps"]
        state["batch"].step(n)
        return [dict(reaction=m.reaction(n), displacement=m.get("displacement")) for m in state["members"]]
    if kind == "static":
        s = state["s"]
        st = s.step(state["inc"], tol=5e-3, cg_tol=1e-13)
        return dict(converged=int(st.converged), displacement=s.get("displacement"), force=s.get("force"),
                    bsf=s.get("bsf"), fail=s.get("fail"))
    if kind == "solve":
        with _solver(case, state["inp"], state["rate"]) as s:
            s.step(case["steps"])
            return dict(reaction=s.reaction(case["steps"]), **_state(s))
    if kind == "inputs":
        return _run_inputs(state)
    return _run_routines(state)


def _run_inputs(q):
    L, X = N.lib(), q["X"]
    n = X.shape[1]
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    nb = C.c_int64()
    new = lambda *s: torch.empty(s, dtype=torch.float64, device="cuda")
    nfam, fptr, mass = new(n), new(n), new(n)
    N.check(L.bbpd_dev_buildhorizons(_p(X), _i(n), _d(q["horizon"]), _i(0), C.byref(nb), _p(nfam), _p(fptr), None, None,
                                     None, st))
    m = nb.value
    fam, bl, L0, vcf, bs, bt, bfm, sf = new(2 * m), new(2, m), new(m), new(m), new(m), new(m), new(m), new(m)
    N.check(L.bbpd_dev_buildhorizons(_p(X), _i(n), _d(q["horizon"]), _i(m), C.byref(nb), None, None, _p(fam), _p(bl),
                                     _p(L0), st))
    N.check(L.bbpd_dev_calculatevolumecorrectionfactors(_p(L0), _i(m), _d(q["horizon"]), _d(q["radij"]), _p(vcf), st))
    N.check(L.bbpd_dev_buildbonddata(_p(bl), _i(m), _i(n), _p(nfam), None, _d(q["bsc"]), _d(q["bsc"]), _d(q["V"]),
                                     _d(q["nvol"]), _p(bs), _p(bt), _p(bfm), _p(sf), st))
    N.check(L.bbpd_dev_buildmassmatrix(_i(n), _d(q["dx"]), _d(q["bsc"]), _d(q["dt"]), _p(nfam), _p(mass), st))
    return dict(nfam=nfam, pointers=fptr, family=fam, bondlist=bl, L0=L0, vcf=vcf, stiffness=bs, mass=mass)


def _run_routines(q):
    L, t, nN, nB, V, dt = N.lib(), q["t"], _i(q["nN"]), _i(q["nB"]), _d(q["V"]), _d(q["dt"])
    adr = q["case"]["scheme"] == "adr"
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    P = {k: _p(v) for k, v in t.items()}
    N.check(L.bbpd_dev_calculatedeformedlength(P["x"], P["bl"], P["L0"], nB, nN, P["L"], P["dX"], P["dY"], P["dZ"],
                                               P["s"], st))
    if adr:
        N.check(L.bbpd_dev_calculatebsftrilinear(P["s"], _d(1e-4), _d(3e-4), _d(2e-3), P["BSF"], P["BT"], P["flag"],
                                                 nB, st))
    else:
        t["bsf"].zero_()
        N.check(L.bbpd_dev_calculatebsfexponential(P["s"], P["s0"], P["sc"], _d(25.0), _d(0.25), P["bsf"], P["BSF"],
                                                   P["BT"], P["flag"], nB, st))
    N.check(L.bbpd_dev_calculatebondforces(P["fX"], P["fY"], P["fZ"], P["fail"], P["dX"], P["dY"], P["dZ"], P["L"],
                                           P["s"], P["sp"], P["BS"], V, P["VCF"], P["BSF"], nB, st))
    t["F"].zero_()
    N.check(L.bbpd_dev_calculatenodalforces(q["plan"].h, P["F"], P["fX"], P["fY"], P["fZ"], st))
    names = ["u", "v", "x", "F", "L", "s", "BSF", "flag", "fX", "fY", "fZ"]
    if adr:
        cn = C.c_double()
        N.check(L.bbpd_dev_calculatedampingcoefficient(P["F"], P["mass"], P["Fp"], _d(1.0), P["v"], P["u"], nN,
                                                       C.byref(cn), st))
        N.check(L.bbpd_dev_timeintegrationADR(_i(q["step"]), _d(1.0), P["v"], P["F"], P["mass"], cn, P["v"], P["u"],
                                              P["CF"], nN, st))
        torch.add(t["X"], t["u"], out=t["x"])
        t["Fp"].copy_(t["F"])
        q["step"] += 1
        return dict({k: t[k] for k in names}, cn=cn.value)
    N.check(L.bbpd_dev_timeintegrationeulercromer(P["a"], P["F"], _d(0.0), P["v"], P["rho"], P["CF"], dt, P["u"],
                                                  P["x"], P["X"], nN, 3, st))
    return {k: t[k] for k in names + ["a", "bsf"]}


# ---- what a pass cannot do without ----

def _bonds(nx, ny, nz):
    """Bonds of a full lattice within 3.015 spacings (61 forward offsets, fewer at the faces)."""
    n = 0
    for dz in range(0, 4):
        for dy in range(-3, 4):
            for dx in range(-3, 4):
                if (dz, dy, dx) > (0, 0, 0) and dx * dx + dy * dy + dz * dz <= 9:
                    n += max(0, nx - abs(dx)) * max(0, ny - abs(dy)) * max(0, nz - dz)
    return n


def work(case):
    kind = case["kind"]
    if kind == "batch":
        nN = nB = 0
        for sp, _ in bb.beam.size_effect_series(case["members"], depth_range=(0.05, case["depth"]), dx=case["dx"]):
            nN += sp.nx * sp.ny * sp.nz
            nB += _bonds(sp.nx, sp.ny, sp.nz)
    else:
        nN, nB = case["nx"] * case["ny"] * case["nz"], _bonds(case["nx"], case["ny"], case["nz"])
    # 38 double operations a directed bond: vector, length, stretch, force and three sums
    bond_flops = 2 * 38 * nB
    if kind == "steps" or kind == "batch":
        per = 8 if (kind == "batch" or case.get("sc") == "lognormal") else 0
        step = 2 * nB * (12 + per) + nN * 181
        return {"bytes": case["steps"] * step + nN * 48 + nB * 8, "flops": case["steps"] * (bond_flops + 60 * nN)}
    if kind == "solve":
        step = 2 * nB * 12 + nN * 181
        return {"bytes": case["steps"] * step + nB * (40 + 24) + nN * (80 + 72),
                "flops": case["steps"] * (bond_flops + 60 * nN)}
    if kind == "static":
        # two Newton solves of about 280 conjugate-gradient iterations, each reading every bond's
        # scale, vector and ends once
        it = 2 * 280
        return {"bytes": it * (nB * 40 + nN * 3 * 8 * 7), "flops": it * (2 * nB * 14 + nN * 50)}
    if kind == "inputs":
        return {"bytes": nN * (24 + 24) + nB * 8 * (2 + 2 + 1 + 5), "flops": nN * 123 * 9 + nB * 10}
    per = 8 * (2 + 4 + 4 + 2 + 4 + 3)   # ends, constants, law arrays; length, vector, stretch; state; force
    return {"bytes": nB * per + nN * 8 * 3 * 9, "flops": 40 * nB + 60 * nN}


# ---- the same in plain torch, 64 bits ----

def exact(case, seed):
    kind = case["kind"]
    if kind == "steps" and case["state"] == "elastic":
        inp, rate = _beam(case, seed)
        if inp["nBonds"] > 2e7 or inp["nBonds"] * case["steps"] > 5e9:
            return None
        r = _loop(inp, case["law"], case["scheme"] == "adr", rate, case["steps"])
        out = dict(displacement=r["u"], velocity=r["v"], bsf=r["BSF"])
        return dict(out, reaction=r["reaction"]) if case["scheme"] == "adr" else out
    if kind == "solve":
        inp, rate = _beam(case, seed)
        if inp["nBonds"] * case["steps"] > 2e9:
            return None
        r = _loop(inp, case["law"], True, rate, case["steps"])
        return dict(reaction=r["reaction"], displacement=r["u"], velocity=r["v"], force=r["F"], bsf=r["BSF"],
                    flag=r["flag"], fail=r["fail"])
    if kind == "routines":
        return _exact_routines(case, seed)
    if kind == "inputs" and case["nx"] * case["ny"] * case["nz"] <= 40000:
        return _exact_inputs(case, seed)
    return None


def _law(law, s, st, k=25.0, alpha=0.25, s0=1e-4, s1=3e-4, sc=2e-3):
    """BSF, flag and fail after one evaluation of the law at stretch s (all bonds concrete)."""
    one = torch.ones_like(s)
    if law == "linear":
        st["fail"] = torch.where((st["fail"] == 1) & (s > sc), 0 * one, st["fail"])
        return
    soft = s > s0
    if law == "trilinear":
        beta, eta = 0.25, s1 / s0
        b = torch.where(soft & (s <= s1), 1 - (eta - beta) / (eta - 1) * (s0 / s) + (1 - beta) / (eta - 1),
                        torch.where(s > sc, one, 1 - (s0 * beta / s) * ((sc - s) / (sc - s1))))
        b = torch.where(soft, b, 0 * one)
        st["flag"] = torch.where(soft & (s <= s1), one, st["flag"])
    elif law == "bilinear":
        st["flag"] = torch.where(soft, one, st["flag"])
        b = torch.nan_to_num((s - s0) / s * (sc / (sc - s0)), nan=0.0) * st["flag"]
    else:
        mid = soft & (s <= sc)
        y = (s - s0) / (sc - s0)
        b = 1 - (s0 / s) * ((1 - (1 - torch.exp(-k * y)) / (1 - math.exp(-k))) + alpha * (1 - y)) / (1 + alpha)
        b = torch.where(mid, b, torch.where(s > sc, one, 0 * one))
        st["flag"] = torch.where(mid, one, st["flag"])
    st["BSF"] = torch.clamp(torch.maximum(st["BSF"], b), max=1.0)


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _gather_sum(i, j, f, nN):
    F = torch.zeros((3, nN), dtype=torch.float64, device=f.device)
    return F.index_add_(1, i, f).index_add_(1, j, -f)


def _loop(inp, law, adr, rate, steps):
    dev = _dev()
    g = lambda k: torch.from_numpy(np.ascontiguousarray(inp[k].T)).to(dev)
    X, bl, L0, BS, VCF = (g(k) for k in ("undeformedCoordinates", "BONDLIST", "UNDEFORMEDLENGTH", "BONDSTIFFNESS",
                                         "VOLUMECORRECTIONFACTORS"))
    CF, PF = g("CONSTRAINTFLAG") == 1, g("BODYFORCEFLAG") == 1
    i, j = bl[0].long() - 1, bl[1].long() - 1
    del bl
    V, dt, nN = inp["cellVolume"], inp["DT"], inp["nNodes"]
    kw = dict(sc=g("sc")) if "sc" in inp else {}
    m = g("massVector") if adr else g("DENSITY")
    z = lambda: torch.zeros_like(X)
    u, v, Fp = z(), z(), z()
    st = dict(BSF=torch.zeros_like(L0), flag=torch.zeros_like(L0), fail=torch.ones_like(L0))
    u[PF] = rate
    react = []
    for n in range(1, steps + 1):
        d = (X + u)[:, j] - (X + u)[:, i]
        L = torch.sqrt((d * d).sum(0))
        s = (L - L0) / L0
        _law(law, s, st, **kw)
        F = _gather_sum(i, j, (st["fail"] * BS * (1 - st["BSF"]) * s * V * VCF) * (d / L), nN)
        react.append(F[PF].sum())
        if adr:
            ok = v != 0
            c1 = -(u * u * torch.where(ok, (F - Fp) / m / torch.where(ok, dt * v, torch.ones_like(v)), 0 * v)).sum()
            c2 = (u * u).sum()
            r = (c1 / c2).item() if c2 != 0 else 0.0
            cn = 2 * math.sqrt(r) if r > 0 else 0.0
            cn = 1.9 if cn > 2 else cn
            v = 0.5 * dt * F / m if n == 1 else ((2 - cn * dt) * v + 2 * dt * F / m) / (2 + cn * dt)
            u = u + dt * v
            u[CF], v[CF], v[PF] = 0.0, 0.0, 0.0
            Fp = F
        else:
            a = F / m
            a[CF | PF] = 0.0
            v = v + a * dt
            u = u + v * dt
        u[PF] = rate * (n + 1)
    t = lambda a: a.t().cpu() if a.ndim == 2 else a.cpu()
    return dict(u=t(u), v=t(v), F=t(F), reaction=torch.stack(react).cpu(), **{k: t(x) for k, x in st.items()})


def _exact_routines(case, seed):
    q = _routine_arrays(case, seed)
    t, nN, dt = q["t"], q["nN"], q["dt"]
    i, j = t["bl"][0].long() - 1, t["bl"][1].long() - 1
    d = t["x"][:, j] - t["x"][:, i]
    L = torch.sqrt((d * d).sum(0))
    s = (L - t["L0"]) / t["L0"]
    st = dict(BSF=t["BSF"].clone(), flag=t["flag"].clone(), fail=t["fail"])
    adr = case["scheme"] == "adr"
    _law("trilinear" if adr else "exponential", s, st, **({} if adr else dict(sc=t["sc"])))
    f = (t["BS"] * (1 - st["BSF"]) * s * q["V"] * t["VCF"]) * (d / L)
    F = _gather_sum(i, j, f, nN)
    out = dict(L=L, s=s, BSF=st["BSF"], flag=st["flag"], fX=f[0], fY=f[1], fZ=f[2], F=F)
    u, v, held = t["u"], t["v"], t["CF"] == 1
    if not adr:
        a = torch.where(held, 0 * F, F / t["rho"])
        v = v + a * dt
        u = u + v * dt
        return dict(out, u=u, v=v, x=t["X"] + u, a=a, bsf=None)
    m = t["mass"]
    c1, c2 = -(u * u * (F / m / v)).sum(), (u * u).sum()
    r = (c1 / c2).item()
    cn = 2 * math.sqrt(r) if r > 0 else 0.0
    cn = 1.9 if cn > 2 else cn
    v = torch.where(held, 0 * v, ((2 - cn) * v + 2 * F / m) / (2 + cn))
    u = torch.where(held, 0 * u, u + v)
    return dict(out, u=u, v=v, x=t["X"] + u, cn=cn)


def _exact_inputs(case, seed):
    X, g = _cloud(case, seed)
    n, h, r = X.shape[1], g["horizon"], g["radij"]
    I, J, D = [], [], []
    for a in range(0, n, 2000):
        d = torch.sqrt((X[0, a:a + 2000, None] - X[0]) ** 2 + (X[1, a:a + 2000, None] - X[1]) ** 2
                       + (X[2, a:a + 2000, None] - X[2]) ** 2)
        i, j = torch.nonzero(d <= h, as_tuple=True)
        keep = i + a != j
        I.append(i[keep] + a), J.append(j[keep]), D.append(d[i[keep], j[keep]])
    i, j, d = torch.cat(I), torch.cat(J), torch.cat(D)
    nfam = torch.bincount(i, minlength=n).double()
    half = i < j
    a, b, L0 = i[half], j[half], d[half]
    vcf = torch.where(L0 <= h - r, torch.ones_like(L0), (h + r - L0) / (2 * r))
    bs = 2 * g["nvol"] / ((nfam[a] + nfam[b]) * g["V"]) * g["bsc"]
    mass = 0.25 * g["dt"] ** 2 * (nfam * g["dx"] ** 2) * (g["bsc"] / g["dx"])
    return dict(nfam=nfam, pointers=torch.cumsum(nfam, 0) - nfam + 1, family=(j + 1).double(),
                bondlist=torch.stack([a, b]).double() + 1, L0=L0, vcf=vcf, stiffness=bs, mass=mass)
