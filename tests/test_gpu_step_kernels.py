"""The two forms of the time step, a block per slice (small beams) and a warp per
slice (step_kernel, above 6 slices per SM), beyond what the small beams of the other
tests reach."""
import numpy as np
import pytest

import bb_pd_b200 as bb
from oracle import pyoracle as po
from test_gpu_solver import BOND, LAWKW, NODAL, _contact_setup, compare, orun, same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(24, 5, 6), (60, 9, 13), (31, 30, 31)])
@pytest.mark.parametrize("law,scheme", [("trilinear", "adr"), ("linear", "eulercromer"), ("exponential", "eulercromer")])
def test_coordinates_leave_the_fast_range_within_a_launch(nx, ny, nz, law, scheme):
    """The loaded nodes lie at z = 0 and move by less than 2^-100 in the first step,
    where the division by shared reciprocals no longer holds: the launch goes over to
    IEEE operations from its second step on. Lengths off by up to 4 s0 keep the laws busy."""
    inp = dict(bb.beam.build(bb.beam.small(nx=nx, ny=ny, nz=nz)))
    X = inp["undeformedCoordinates"].copy(order="F")
    X[:, 2] -= X[:, 2].max()
    rng = np.random.default_rng(nx)
    inp["undeformedCoordinates"] = X
    inp["UNDEFORMEDLENGTH"] = inp["UNDEFORMEDLENGTH"] * (1 + 1e-4 * rng.integers(-4, 5, inp["nBonds"]))
    kw = dict(LAWKW[law], scheme=scheme, amplitude="smoothstep", applied_final=-1e-4, n_time_steps=2_000_000_000)
    s = bb.Solver(inp, **kw)
    r = orun(inp, **kw)
    s.step(12)
    r.step(1)
    z = r.get("deformed")[X[:, 2] == 0, 2]
    assert ((z != 0) & (np.abs(z) < 2.0 ** -100)).any()
    r.step(11)
    compare(s, r, law)
    s.step(3)
    r.step(3)
    compare(s, r, law)
    s.close()


# ---- step_kernel: 28 830 nodes, 901 slices, just above the 888 of 148 SMs

PAIRS = [("trilinear", "adr"), ("exponential", "eulercromer"), ("linear", "adr"), ("bilinear", "eulercromer")]
RATE = {"adr": -4e-6, "eulercromer": -8e-6}


@pytest.fixture(scope="module")
def big():
    return bb.beam.build(bb.beam.small(nx=31, ny=30, nz=31))


def solver(inp, **kw):
    s = bb.Solver(inp, **kw)
    i = s.info()
    # a slice per warp of blocks of 8; split_kernel would have two blocks on every SM
    assert i["block_threads"] == 256 and i["grid_blocks"] == (i["n_slices"] + 7) // 8
    return s


def lognormal_sc(inp, median=2e-3):
    return median * np.exp(0.1 * np.random.default_rng(2).standard_normal(inp["nBonds"]))


@pytest.mark.parametrize("law,scheme", PAIRS)
def test_per_bond_sc(big, law, scheme):
    """The instances with a critical stretch per bond, some bonds broken and of every
    type from the start."""
    rng = np.random.default_rng(3)
    inp = dict(big, sc=lognormal_sc(big, 2e-4 if law == "linear" else 2e-3),
               BONDTYPE=rng.integers(0, 3, big["nBonds"]).astype(np.float64))
    kw = dict(LAWKW[law], scheme=scheme, rate=RATE[scheme])
    s, r = solver(inp, **kw), orun(inp, **kw)
    for n in (1, 24):
        s.step(n)
        r.step(n)
        compare(s, r, law)
    assert (r.get("fail") == 0).any() if law == "linear" else (r.get("bsf") > 0).any()
    s.close()


@pytest.mark.parametrize("size", [(60, 9, 13), (31, 30, 31)])
@pytest.mark.parametrize("law", ["trilinear", "exponential"])
def test_per_bond_s0_s1(size, law):
    inp = dict(bb.beam.build(bb.beam.small(*size)))
    rng = np.random.default_rng(4)
    inp["s0"] = 1e-4 * (1 + 0.5 * rng.random(inp["nBonds"]))
    if law == "trilinear":
        inp["s1"] = 3 * inp["s0"]
    kw = dict(LAWKW[law], scheme="adr", rate=-4e-6)
    s, r = bb.Solver(inp, **kw), orun(inp, **kw)
    r.p.s0 = po.P(inp["s0"])
    if law == "trilinear":
        r.p.s1 = po.P(inp["s1"])
    s.step(25)
    r.step(25)
    compare(s, r, law)
    assert (r.get("bsf") > 0).any()
    s.close()


@pytest.mark.parametrize("size", [(60, 9, 13), (31, 30, 31)])
@pytest.mark.parametrize("law,scheme", [("trilinear", "adr"), ("linear", "eulercromer")])
def test_wide_dictionary(size, law, scheme):
    """A length of its own for every bond: more than 65 535 dictionary entries, so
    32-bit ids."""
    inp = dict(bb.beam.build(bb.beam.small(*size)))
    inp["UNDEFORMEDLENGTH"] = inp["UNDEFORMEDLENGTH"] * (1 + 5e-5 * np.random.default_rng(5).standard_normal(inp["nBonds"]))
    kw = dict(LAWKW[law], scheme=scheme, rate=-2e-5 if law == "linear" else -4e-6)
    s, r = bb.Solver(inp, **kw), orun(inp, **kw)
    assert s.info()["layout"] == 2
    s.step(25)
    r.step(25)
    compare(s, r, law)
    assert (r.get("fail") == 0).any() if law == "linear" else (r.get("bsf") > 0).any()
    s.close()


@pytest.mark.parametrize("size", [(60, 9, 13), (31, 30, 31)])
@pytest.mark.parametrize("law,scheme", [("trilinear", "adr"), ("linear", "eulercromer")])
def test_irregular_entries(size, law, scheme):
    """Bonds outside the fast division's conditions take IEEE operations: NaN
    stiffness (the force's NaN guard gives 0), zero and 2^-110 length (broken at once)."""
    inp = dict(bb.beam.build(bb.beam.small(*size)))
    pick = np.random.default_rng(6).permutation(inp["nBonds"])[:300]
    inp["BONDSTIFFNESS"], inp["UNDEFORMEDLENGTH"] = inp["BONDSTIFFNESS"].copy(), inp["UNDEFORMEDLENGTH"].copy()
    inp["BONDSTIFFNESS"][pick[:100]] = np.nan
    inp["UNDEFORMEDLENGTH"][pick[100:200]] = 0.0
    inp["UNDEFORMEDLENGTH"][pick[200:]] = 2.0 ** -110
    kw = dict(LAWKW[law], scheme=scheme, rate=-4e-6)
    s, r = bb.Solver(inp, **kw), orun(inp, **kw)
    s.step(20)
    r.step(20)
    compare(s, r, law)
    assert np.isfinite(r.get("force")).all()
    s.close()


@pytest.mark.parametrize("scheme", ["adr", "eulercromer"])
def test_contact_and_probes(big, scheme):
    inp, pens = _contact_setup(big, RATE[scheme])
    kw = dict(LAWKW["trilinear"], scheme=scheme)
    s, r = solver(inp, **kw), orun(inp, penetrators=pens, **kw)
    s.set_contact(pens)
    top = int(pens[0]["family"][0])
    s.set_probes([top, 7], [2, 0])
    for n in (1, 24):
        s.step(n)
        r.step(n)
        compare(s, r, "trilinear")
        assert s.reaction(n)[-1] == r.reaction
        u = r.get("displacement")
        assert np.array_equal(s.probes(n)[-1], [u[top - 1, 2], u[6, 0]])
    assert r.reaction != 0.0
    s.close()


@pytest.mark.parametrize("T", [1, 64])
def test_chunk_counts(big, T):
    kw = dict(LAWKW["trilinear"], scheme="adr", rate=-4e-6, n_chunks=T)
    s, r = solver(big, **kw), orun(big, **kw)
    s.step(20)
    r.step(20)
    compare(s, r, "trilinear")
    s.close()


@pytest.mark.parametrize("law", ["trilinear", "exponential"])
def test_damage_energy(big, law):
    kw = dict(LAWKW[law], scheme="adr", rate=-8e-6)
    s, r = solver(big, **kw), orun(big, **kw)
    s.track_damage_energy()
    nB, E = big["nBonds"], np.zeros(big["nBonds"])
    s0, sc = np.full(nB, kw["s0"]), np.full(nB, kw["sc"])
    for _ in range(15):
        r.step(1)
        po.lib().orc_damageenergy(po.P(big["BONDSTIFFNESS"]), po.P(s0), po.P(sc), po.P(big["UNDEFORMEDLENGTH"]),
                                  po.P(r.get("stretch")), 25.0, 0.25, big["cellVolume"], po.P(E), nB)
    s.step(6)
    s.step(9)
    assert (E > 0).any() and same(s.get("damage_energy"), E)
    s.close()


@pytest.mark.parametrize("scheme", ["adr", "eulercromer"])
def test_checkpoint_smoothstep_and_nonfinite(big, scheme):
    kw = dict(LAWKW["bilinear"], scheme=scheme, amplitude="smoothstep", applied_final=-4e-4, n_time_steps=40)
    s, r = solver(big, **kw), orun(big, **kw)
    s.step(11)
    ck = s.checkpoint()
    s.step(14)
    r.step(25)
    compare(s, r, "bilinear")
    assert (r.get("bsf") > 0).any()
    t = solver(big, **kw)
    t.step(2)
    t.restore(ck)
    t.step(14)
    for f in NODAL + BOND:
        assert same(s.get(f), t.get(f)), f
    u = t.get("displacement")
    u[5, 0] = np.nan
    t.set("displacement", u)
    with pytest.raises(bb.BBPDError) as e:
        t.step(1)
    assert e.value.status == bb._native.ERR_NONFINITE
    s.close()
    t.close()


@pytest.mark.parametrize("size", [(60, 9, 13), (31, 30, 31)])
@pytest.mark.parametrize("law,scheme", PAIRS)
@pytest.mark.parametrize("per_bond", [False, True])
def test_fp32_identical_to_tiled(size, law, scheme, per_bond):
    """The FP32 form of both kernels against the tiled kernel's: the same arithmetic
    from data staged elsewhere, so the same bits."""
    inp = dict(bb.beam.build(bb.beam.small(*size)))
    if per_bond:
        inp["sc"] = lognormal_sc(inp, 2e-4 if law == "linear" else 2e-3)
    kw = dict(LAWKW[law], scheme=scheme, rate=-2e-5 if law == "linear" else -8e-6, precision="fp32")
    a, b = bb.Solver(inp, **kw), bb.Solver(inp, node_order="tiled", **kw)
    assert a.info()["layout"] == 3 and b.info()["layout"] == 3 + 16
    for n in (1, 29):
        a.step(n)
        b.step(n)
        for f in NODAL + BOND:
            assert same(a.get(f), b.get(f)), (n, f)
    assert (a.get("fail") == 0).any() if law == "linear" else (a.get("bsf") > 0).any()
    a.close()
    b.close()


def test_fp32_identical_to_batch(big):
    kw = dict(LAWKW["trilinear"], scheme="adr", rate=-8e-6, precision="fp32")
    a, b = solver(big, **kw), solver(big, **kw)
    batch = bb.Batch("fp32")
    batch.add(b)
    a.step(30)
    batch.step(30)
    for f in NODAL + BOND:
        assert same(a.get(f), b.get(f)), f
    batch.close()
    a.close()
    b.close()
