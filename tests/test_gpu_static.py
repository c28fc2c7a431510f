"""GPU static (implicit) solver against the oracle's restatement of the
reference's displacement-controlled Newton-Raphson (oracle/static_oracle.py,
direct sparse solves). The GPU solves each linear system by a preconditioned
conjugate gradient to a relative residual of 1e-13, so displacements agree to a
tolerance: 1e-8 of the largest displacement while the beam is elastic, 1e-6
through softening, with identical softening and broken-bond sets."""
import ctypes as C

import numpy as np
import pytest

import bb_pd_b200 as bb
from bb_pd_b200.static import StaticSolver
from oracle.static_oracle import StaticOracle

pytestmark = pytest.mark.gpu
CG = dict(cg_tol=1e-13, max_cg=200000)


def test_static_elastic_vs_oracle():
    inp = bb.beam.build(bb.beam.small(nx=20, ny=4, nz=6))
    g = StaticSolver(inp, law="linear", sc=1.0)
    o = StaticOracle(inp, law="linear", sc=1.0)
    for step in range(3):
        sg = g.step(-1e-6, tol=1e-9, **CG)
        so = o.step(-1e-6, tol=1e-9)
        assert sg.converged and so["converged"], (step, sg.residual, sg.reaction)
        ug, uo = g.get("displacement"), o.get("displacement")
        scale = np.abs(uo).max()
        assert np.abs(ug - uo).max() <= 1e-8 * scale, step
        np.testing.assert_allclose(sg.reaction, so["reaction"], rtol=1e-6)
    # equilibrium: no net force on the free DOFs, the held DOFs carry the load
    F = g.get("force")
    assert abs(F[:, 2].sum()) <= 1e-9 * np.abs(F).max()
    assert same_flags(g.get("fail"), np.ones(inp["nBonds"]))
    g.close()


def same_flags(a, b):
    return np.array_equal(np.asarray(a), np.asarray(b))


def test_static_softening_vs_oracle():
    """Notched beam, bilinear law (the reference's static driver uses
    calculatebondsofteningfactor with sc = 25 s0): five load steps take it into
    softening and the first bond failures."""
    dx = 5e-3
    inp = bb.beam.build(bb.beam.small(nx=24, ny=4, nz=8, notch_x=12.5 * dx, notch_depth=3.2 * dx))
    kw = dict(law="bilinear", s0=1e-4, sc=2.5e-3)
    g = StaticSolver(inp, **kw)
    o = StaticOracle(inp, **kw)
    for step in range(6):
        sg = g.step(-1e-5, tol=1e-6, max_newton=60, **CG)
        so = o.step(-1e-5, tol=1e-6, max_newton=60)
        assert sg.converged and so["converged"], step
        ug, uo = g.get("displacement"), o.get("displacement")
        assert np.abs(ug - uo).max() <= 1e-6 * np.abs(uo).max(), step
        assert same_flags(g.get("flag"), o.get("flag")), step
        assert same_flags(g.get("fail"), o.get("fail")), step
        np.testing.assert_allclose(g.get("bsf"), o.get("bsf"), rtol=0, atol=1e-6)
    assert g.get("flag").sum() > 100 and (g.get("fail") == 0).any()
    g.close()


def test_static_linearity_and_validation():
    inp = bb.beam.build(bb.beam.small(nx=16, ny=4, nz=5))
    a = StaticSolver(inp, law="linear", sc=1.0)
    b = StaticSolver(inp, law="linear", sc=1.0)
    a.step(-1e-7, tol=1e-10, **CG)
    b.step(-2e-7, tol=1e-10, **CG)
    ua, ub = a.get("displacement"), b.get("displacement")
    assert np.abs(ub - 2 * ua).max() <= 1e-5 * np.abs(ub).max()
    with pytest.raises(bb.BBPDError):
        a.step(-1e-7, tol=0.0)
    with pytest.raises(bb.BBPDError):
        a.get("velocity")
    bad_inp = dict(inp)
    bad_inp["BONDTYPE"] = np.full(inp["nBonds"], 4.0)
    with pytest.raises(bb.BBPDError):
        StaticSolver(bad_inp, law="linear", sc=1.0)
    a.close()
    b.close()


@pytest.mark.parametrize("nod", [3, 2])
def test_stiffness_triplets_vs_oracle(nod):
    """buildstiffnessmatrixCSCformat.m on the GPU: triplets (find order, failed
    bonds skipped, exact zeros dropped) and massVector bit-identical to the
    oracle's literal restatement, on deformed coordinates with damaged,
    interface and broken bonds."""
    from oracle import pyoracle as po
    P = po.P
    inp = bb.beam.build(bb.beam.small(nx=18, ny=4, nz=5))
    rng = np.random.default_rng(4)
    n, nB = inp["nNodes"], inp["nBonds"]
    X = np.asfortranarray(inp["undeformedCoordinates"][:, :nod] + rng.normal(0, 1e-5, (n, nod)))
    bl = inp["BONDLIST"]
    fail = (rng.random(nB) > 0.1).astype(np.float64)
    bsf = np.where(rng.random(nB) < 0.3, rng.random(nB), 0.0)
    bfm = np.where(rng.random(nB) < 0.2, 3.0, 1.0)
    vcf, bs, V = inp["VOLUMECORRECTIONFACTORS"], inp["BONDSTIFFNESS"], inp["cellVolume"]
    from bb_pd_b200.static import buildstiffnessmatrixCSCformat
    r, c, v, m = buildstiffnessmatrixCSCformat(X, bl, vcf, V, bs, bfm, fail, bsf, inp["UNDEFORMEDLENGTH"])
    L = po.lib()
    tot = L.orc_stiffness_coo(P(X), n, nod, P(bl), P(vcf), V, P(bs), P(bfm), P(fail), P(bsf), nB, 0, None, None,
                              None, None)
    orr, occ, ov, om = np.zeros(tot), np.zeros(tot), np.zeros(tot), np.zeros(n)
    L.orc_stiffness_coo(P(X), n, nod, P(bl), P(vcf), V, P(bs), P(bfm), P(fail), P(bsf), nB, tot, P(orr), P(occ),
                        P(ov), P(om))
    assert r.size == tot > 0
    for a, b in ((r, orr), (c, occ), (v, ov), (m, om)):
        assert np.array_equal(a, b)
    assert r.size <= (2 * nod) ** 2 * int(fail.sum())


@pytest.mark.parametrize("law,steps", [("trilinear", 4), ("exponential", 3)])
def test_static_other_laws_vs_oracle(law, steps):
    """The static solver with the trilinear and exponential laws against the
    oracle (its C law routines inside the restated Newton loop)."""
    dx = 5e-3
    inp = bb.beam.build(bb.beam.small(nx=24, ny=4, nz=8, notch_x=12.5 * dx, notch_depth=3.2 * dx))
    kw = dict(law=law, s0=1e-4, sc=2e-3)
    g = StaticSolver(inp, **kw)
    o = StaticOracle(inp, **kw)
    for step in range(steps):
        sg = g.step(-1e-5, tol=1e-6, max_newton=60, **CG)
        so = o.step(-1e-5, tol=1e-6, max_newton=60)
        assert sg.converged and so["converged"], step
        ug, uo = g.get("displacement"), o.get("displacement")
        assert np.abs(ug - uo).max() <= 1e-6 * np.abs(uo).max(), step
        assert same_flags(g.get("flag"), o.get("flag")), step
        assert same_flags(g.get("fail"), o.get("fail")), step
    assert g.get("flag").sum() > 100
    g.close()


# half a slice, a ragged last slice, more rows than warps, and a beam whose last
# 70 nodes have lost their bonds (slices without a row)
@pytest.mark.parametrize("nx,ny,nz,cut", [(6, 2, 2, 0), (13, 3, 5, 0), (40, 6, 8, 0), (30, 4, 6, 70)])
def test_static_solve_sizes_vs_oracle(nx, ny, nz, cut):
    """The linear solve where its rows and slices meet differently."""
    inp = dict(bb.beam.build(bb.beam.small(nx=nx, ny=ny, nz=nz)))
    if cut:   # the top layer's end, away from the loaded nodes
        keep = (inp["BONDLIST"] <= inp["nNodes"] - cut).all(axis=1)
        moved = np.nonzero(inp["BODYFORCEFLAG"].any(axis=1))[0]
        inp["BODYFORCEFLAG"] = inp["BODYFORCEFLAG"].copy(order="F")
        inp["BODYFORCEFLAG"][moved] = 0
        inp["BODYFORCEFLAG"][moved - cut, 2] = 1   # load nodes that keep their bonds
        for k in ("UNDEFORMEDLENGTH", "BONDSTIFFNESS", "VOLUMECORRECTIONFACTORS"):
            inp[k] = inp[k][keep].copy()
        inp["BONDLIST"] = np.asfortranarray(inp["BONDLIST"][keep])
        inp["nBonds"] = int(keep.sum())
    g = StaticSolver(inp, law="linear", sc=1.0)
    o = StaticOracle(inp, law="linear", sc=1.0)
    for step in range(2):
        sg = g.step(-1e-6, tol=1e-9, **CG)
        so = o.step(-1e-6, tol=1e-9)
        assert sg.converged and so["converged"], (step, sg.residual, sg.reaction)
        ug, uo = g.get("displacement"), o.get("displacement")
        assert np.abs(ug - uo).max() <= 1e-8 * np.abs(uo).max(), step
    g.close()


@pytest.mark.parametrize("nx,ny,nz,copies", [(20, 4, 6, 2), (12, 4, 4, 3)])
def test_static_solve_long_lists_vs_oracle(nx, ny, nz, copies):
    """Lists of more than 128 entries: every bond several times, its stiffness
    shared out."""
    inp = dict(bb.beam.build(bb.beam.small(nx=nx, ny=ny, nz=nz)))
    inp["BONDSTIFFNESS"] = inp["BONDSTIFFNESS"] / copies
    for k in ("UNDEFORMEDLENGTH", "BONDSTIFFNESS", "VOLUMECORRECTIONFACTORS"):
        inp[k] = np.tile(inp[k], copies)
    inp["BONDLIST"] = np.asfortranarray(np.tile(inp["BONDLIST"], (copies, 1)))
    inp["nBonds"] *= copies
    g = StaticSolver(inp, law="linear", sc=1.0)
    o = StaticOracle(inp, law="linear", sc=1.0)
    sg = g.step(-1e-6, tol=1e-9, **CG)
    so = o.step(-1e-6, tol=1e-9)
    assert sg.converged and so["converged"], (sg.residual, sg.reaction)
    ug, uo = g.get("displacement"), o.get("displacement")
    assert np.abs(ug - uo).max() <= 1e-8 * np.abs(uo).max()
    g.close()


@pytest.mark.parametrize("nx,ny,nz", [(50, 8, 12), (100, 12, 22)])
def test_static_solve_many_slices(nx, ny, nz):
    """More slices than the 148 that have a block of their own, and more than a
    block multiplies at a time: the nodal forces, summed by another kernel, are in
    equilibrium to 1e-6 of the reaction, which only a solved system gives (the
    rounding of the positions alone leaves about 1e-9)."""
    inp = bb.beam.build(bb.beam.small(nx=nx, ny=ny, nz=nz))
    g = StaticSolver(inp, law="linear", sc=1.0)
    st = g.step(-1e-6, tol=1e-6, **CG)
    assert st.converged and st.newton_iterations >= 1 and st.residual <= 1e-6 * st.reaction
    g.close()


def with_hubs(inp, hubs):
    """The input with a weak bond from each node of `hubs` to every other node."""
    inp = dict(inp)
    n, X = inp["nNodes"], inp["undeformedCoordinates"]
    i = np.repeat(hubs, n - 1)
    j = np.concatenate([np.delete(np.arange(n), h) for h in hubs])
    inp["BONDLIST"] = np.asfortranarray(np.concatenate([inp["BONDLIST"], np.stack([i, j], 1) + 1.0]))
    inp["UNDEFORMEDLENGTH"] = np.concatenate([inp["UNDEFORMEDLENGTH"], np.sqrt(((X[i] - X[j]) ** 2).sum(1))])
    inp["BONDSTIFFNESS"] = np.concatenate([inp["BONDSTIFFNESS"], np.full(i.size, 1e-6 * inp["BONDSTIFFNESS"][0])])
    inp["VOLUMECORRECTIONFACTORS"] = np.concatenate([inp["VOLUMECORRECTIONFACTORS"], np.ones(i.size)])
    inp["nBonds"] += i.size
    return inp


def test_static_solve_ignores_barrier_timeout():
    """barrier_timeout_s limits the waits of the time stepping alone: a linear solve
    whose blocks wait for the one with a list of 20 000 entries finishes whatever it is."""
    inp = with_hubs(bb.beam.build(bb.beam.small(nx=100, ny=10, nz=20)), [5000])
    g = StaticSolver(inp, law="linear", sc=1.0, barrier_timeout_s=1e-9)
    st = g.step(-1e-6, tol=1e-30, cg_tol=1e-30, max_cg=8, max_newton=1)
    assert st.cg_iterations == 8 and st.newton_iterations == 1
    g.close()


def set_launch(g, iterations, limit_s=0.0):
    L = bb._native.lib()
    L.bbpd_selftest_static_launch.argtypes = [C.c_void_p, C.c_int, C.c_double]
    bb._native.check(L.bbpd_selftest_static_launch(g._h, iterations, limit_s))


# one launch; launches that end between, at and just past the looks at the residual
# (every 8 iterations); max_cg on a launch's last iteration, before and after it
@pytest.mark.parametrize("launch,max_cg", [(1, 200000), (5, 200000), (8, 200000), (17, 200000), (16, 48), (16, 47),
                                           (16, 49)])
def test_static_solve_cut_into_launches(launch, max_cg):
    """A linear solve that goes over several launches carries all of its state from
    one to the next: the same iterates bit for bit and the same count."""
    inp = bb.beam.build(bb.beam.small(nx=20, ny=4, nz=6))
    out = []
    for n in (1024, launch):
        g = StaticSolver(inp, law="linear", sc=1.0)
        set_launch(g, n)
        st = [g.step(-1e-6, tol=1e-9, cg_tol=1e-13, max_cg=max_cg, max_newton=3) for _ in range(2)]
        out.append(([(s.cg_iterations, s.newton_iterations, s.residual, s.reaction) for s in st],
                    g.get("displacement"), g.get("force")))
        g.close()
    (a, ua, fa), (b, ub, fb) = out
    assert a == b and a[0][0] > launch
    assert np.array_equal(ua, ub) and np.array_equal(fa, fb)


def test_static_solve_wait_runs_out():
    """A barrier wait of the linear solve that runs out is reported, moves nothing
    and leaves the solver usable."""
    inp = with_hubs(bb.beam.build(bb.beam.small(nx=100, ny=10, nz=20)), [5000])
    kw = dict(tol=1e-30, cg_tol=1e-30, max_cg=8, max_newton=1)
    a, b = (StaticSolver(inp, law="linear", sc=1.0) for _ in range(2))
    a.step(-1e-6, **kw)
    set_launch(b, 1024, 1e-9)
    with pytest.raises(bb.BBPDError) as e:
        b.step(-1e-6, **kw)
    assert e.value.status == bb._native.ERR_TIMEOUT
    moved = (inp["BODYFORCEFLAG"] == 1) & (inp["CONSTRAINTFLAG"] != 1)
    assert np.array_equal(b.get("displacement") != 0, moved)
    set_launch(b, 1024, 10.0)
    b.step(0.0, **kw)
    assert np.array_equal(a.get("displacement"), b.get("displacement"))
    a.close()
    b.close()


# 4 lists of 480 among lists of 18, padding more than three quarters of the slices
# (lists stay lists); 4 among lists of 122 (slices); every node bonded to all others
@pytest.mark.parametrize("hf,hubs", [(1.5, 4), (3.015, 4), (1.5, 480)])
def test_static_solve_uneven_lists_vs_oracle(hf, hubs):
    inp = with_hubs(bb.beam.build(bb.beam.small(nx=20, ny=4, nz=6, horizon_factor=hf)),
                    list(range(0, 480, 480 // hubs)))
    g = StaticSolver(inp, law="linear", sc=1.0)
    o = StaticOracle(inp, law="linear", sc=1.0)
    for step in range(2):
        sg = g.step(-1e-6, tol=1e-9, **CG)
        so = o.step(-1e-6, tol=1e-9)
        assert sg.converged and so["converged"], (step, sg.residual, sg.reaction)
        ug, uo = g.get("displacement"), o.get("displacement")
        assert np.abs(ug - uo).max() <= 1e-8 * np.abs(uo).max(), step
    g.close()


def test_static_uneven_lists_memory():
    """A few nodes with very long lists do not make every list as long: some 130
    bytes a bond and 300 a node, not 16 bytes for 32 times the longest lists."""
    import torch
    inp = with_hubs(bb.beam.build(bb.beam.small(nx=100, ny=10, nz=20)), list(range(16, 20000, 313)))
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    g = StaticSolver(inp, law="linear", sc=1.0)
    used = free - torch.cuda.mem_get_info()[0]
    g.close()
    assert used <= 200 * inp["nBonds"] + 500 * inp["nNodes"], used
