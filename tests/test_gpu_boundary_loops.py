"""FluxMassDolfynBoundaryLoop1-5 and FluxMassDolfynRegionLoop on the GPU.

The host-buffer calls run the chain a solver step runs (inflow, area rate,
outlet fluxes, outflow per region, region factors, scaled outlet fluxes and
their su update) and every output is compared, bit for bit, with the
oracle, which is itself bit-identical to the reference's templates
(tests/test_oracle_vs_reference.py). The device-resident calls run the same
chain in the mesh's internal numbering, with every scalar left on the
device, and must give the same bits. Meshes: structured and jittered with
permuted numbering, six boundary regions (inlet, two outlets, symmetry,
wall, default) assigned at random, so that cells with several outlet faces
exercise the ordered su update; the large jittered mesh (112 x 104 x 96,
64,768 boundaries) takes the id-ordered sums through many staged passes.
"""
import numpy as np
import pytest

import oracle as O
from test_oracle_vs_reference import _with_regions

pytestmark = pytest.mark.gpu


def _setup(cg, kind, order):
    base = {"struct": lambda: O.structgen(20, 18, 16),
            "jitter": lambda: O.jitter(17, 15, 13, 0.25, seed=8, permute=True),
            "large": lambda: O.jitter(112, 104, 96, 0.25, seed=8, permute=True)}[kind]()
    m, splvl, rng = _with_regions(base, 41 if kind == "struct" else 42)
    mesh = cg.Mesh.from_arrays(m, order=order)
    assert mesh.set_regions(m["regionType"], m["regionUVW"], m["regionDen"], m["bndRegion"]) == cg.E_SUCCESS
    assert mesh.set_region_split(splvl) == cg.E_SUCCESS
    nF, nB, nC, nR = m["nFaces"], m["nBnd"], m["nCells"], m["nRegions"]
    d = dict(mf=rng.uniform(1e-6, 1e-2, nF) * rng.choice([-1.0, 1.0], nF),
             u=rng.uniform(1e-6, 1e-2, nB), v=rng.uniform(1e-6, 1e-2, nB), w=rng.uniform(1e-6, 1e-2, nB),
             den=rng.uniform(0.9, 1.1, nB), fr=rng.uniform(1e-6, 1e-2, nR), su=rng.standard_normal(nC))
    return m, splvl, mesh, d


def _oracle_chain(m, splvl, d, solve):
    flowin = O.boundary_loop1(m, d["mf"])
    ratearea = O.boundary_loop3(m, flowin)
    mf4, u4, v4, w4, flowout4 = O.boundary_loop4(m, splvl, d["mf"], d["u"], d["v"], d["w"], d["den"], ratearea)
    fr2, flowout2 = O.boundary_loop2(m, mf4, d["fr"])
    ff = O.region_loop(m, splvl, fr2, flowin)
    mf5, su5, u5, v5, w5, fo2 = O.boundary_loop5(m, mf4, d["su"], u4, v4, w4, 1.3, solve, ff, 0.25)
    return dict(flowin=flowin, ratearea=ratearea, mf4=mf4, u4=u4, v4=v4, w4=w4, flowout4=flowout4, fr2=fr2,
                flowout2=flowout2, ff=ff, mf5=mf5, su5=su5, u5=u5, v5=v5, w5=w5, fo2=fo2)


def _host_chain(cg, mesh, d, solve, f32=False):
    """The chain through the host-buffer calls; f32: float32 arrays (the
    reference's T = float instantiation)."""
    r = {}
    E = cg.E_SUCCESS
    rc, r["flowin"] = cg.FluxMassDolfynBoundaryLoop1(mesh, d["mf"].copy())
    assert rc == E
    rc, r["ratearea"] = cg.FluxMassDolfynBoundaryLoop3(mesh, r["flowin"], f32=f32)
    assert rc == E
    mf, u, v, w = d["mf"].copy(), d["u"].copy(), d["v"].copy(), d["w"].copy()
    rc, r["flowout4"] = cg.FluxMassDolfynBoundaryLoop4(mesh, mf, u, v, w, d["den"].copy(), r["ratearea"])
    assert rc == E
    r.update(mf4=mf.copy(), u4=u.copy(), v4=v.copy(), w4=w.copy())
    fr = d["fr"].copy()
    rc, r["flowout2"] = cg.FluxMassDolfynBoundaryLoop2(mesh, mf, fr)
    assert rc == E
    r["fr2"] = fr
    ff = np.full(len(fr), np.nan, fr.dtype)
    assert cg.FluxMassDolfynRegionLoop(mesh, ff, fr, r["flowin"]) == E
    r["ff"] = ff
    su = d["su"].copy()
    rc, r["fo2"] = cg.FluxMassDolfynBoundaryLoop5(mesh, mf, su, u, v, w, 1.3, solve, ff, 0.25)
    assert rc == E
    r.update(mf5=mf, su5=su, u5=u, v5=v, w5=w)
    return r


def test_many_regions_bit_exact(cg, gpu):
    """2,500 regions (more than one block of region sums: the region sums
    run in groups of 992): loops 1-5 and the region loop, and the momentum
    loop's boundary loop (wall shear onto each region's force tangent), bit
    for bit against the oracle."""
    base = O.jitter(30, 28, 26, 0.25, seed=12, permute=True)
    rng = np.random.Generator(np.random.Philox(key=43))
    nR = 2500
    m = dict(base)
    m["nRegions"] = nR
    m["regionType"] = rng.integers(0, 5, nR).astype(np.int32)
    m["regionUVW"] = rng.standard_normal(3 * nR)
    m["regionDen"] = rng.uniform(0.9, 1.1, nR)
    m["bndRegion"] = rng.integers(0, nR, m["nBnd"]).astype(np.int32)
    splvl = rng.uniform(0.2, 0.8, nR)
    mesh = cg.Mesh.from_arrays(m, order=3)
    assert mesh.set_regions(m["regionType"], m["regionUVW"], m["regionDen"], m["bndRegion"]) == cg.E_SUCCESS
    assert mesh.set_region_split(splvl) == cg.E_SUCCESS
    nF, nB, nC = m["nFaces"], m["nBnd"], m["nCells"]
    d = dict(mf=rng.uniform(1e-6, 1e-2, nF) * rng.choice([-1.0, 1.0], nF),
             u=rng.uniform(1e-6, 1e-2, nB), v=rng.uniform(1e-6, 1e-2, nB), w=rng.uniform(1e-6, 1e-2, nB),
             den=rng.uniform(0.9, 1.1, nB), fr=rng.uniform(1e-6, 1e-2, nR), su=rng.standard_normal(nC))
    want = _oracle_chain(m, splvl, d, (1, 1, 1))
    got = _host_chain(cg, mesh, d, (1, 1, 1))
    for k, v in want.items():
        assert np.array_equal(np.asarray(got[k]), np.asarray(v)), k
    # momentum loop's boundary loop on a shear the test sets
    shear = rng.standard_normal((nB, 3))
    ft0 = rng.standard_normal((nR, 3))
    mesh.boundary_shear(shear)
    mesh.region_force_tangent(nR, ft0)
    assert cg.FluxUVWDolfynBndsLoop1(mesh) == cg.E_SUCCESS
    assert np.array_equal(mesh.region_force_tangent(nR), O.uvw_bnds_loop1(m, shear, ft0))


@pytest.mark.parametrize("kind,order", [("struct", 2), ("jitter", 3), ("jitter", 0), ("large", 3)])
@pytest.mark.parametrize("solve", [(1, 1, 1), (0, 1, 0)])
def test_boundary_loops_bit_exact(cg, gpu, kind, order, solve):
    m, splvl, mesh, d = _setup(cg, kind, order)
    want = _oracle_chain(m, splvl, d, solve)
    got = _host_chain(cg, mesh, d, solve)
    for k, v in want.items():
        assert np.array_equal(np.asarray(got[k]), np.asarray(v)), k


@pytest.mark.parametrize("kind,order", [("struct", 2), ("jitter", 3)])
def test_device_loops_equal_host_loops(cg, gpu, kind, order):
    import torch
    dev = torch.device("cuda:0")
    m, splvl, mesh, d = _setup(cg, kind, order)
    solve = (1, 0, 1)
    host = _host_chain(cg, mesh, d, solve)
    c2o, f2o = mesh.numbering()

    def T(a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(dev)

    mf, su = T(d["mf"][f2o]), T(d["su"][c2o])
    u, v, w, den, fr = T(d["u"]), T(d["v"]), T(d["w"]), T(d["den"]), T(d["fr"])
    sc = torch.full((5,), np.nan, dtype=torch.float64, device=dev)      # flowin, ratearea, flowout4, flowout2, fo2
    ff = torch.full((m["nRegions"],), np.nan, dtype=torch.float64, device=dev)
    s = torch.cuda.current_stream()
    cg.dev_boundary_loop1(mesh, mf, sc[0:1], stream=s)
    cg.dev_boundary_loop3(mesh, sc[0:1], sc[1:2], stream=s)
    cg.dev_boundary_loop4(mesh, mf, u, v, w, den, sc[1:2], sc[2:3], stream=s)
    mf4, u4 = mf.clone(), u.clone()
    cg.dev_boundary_loop2(mesh, mf, fr, sc[3:4], stream=s)
    cg.dev_region_loop(mesh, ff, fr, sc[0:1], stream=s)
    sc[4] = 0.25
    cg.dev_boundary_loop5(mesh, mf, su, u, v, w, 1.3, solve, ff, sc[4:5], stream=s)
    torch.cuda.synchronize()

    def H(t):
        return t.cpu().numpy()

    def to_ref(t, n2o):
        """internal -> reference numbering (internal i is reference n2o[i])"""
        a = H(t)
        out = np.empty_like(a)
        out[n2o] = a
        return out

    scal = H(sc)
    for k, x in (("flowin", scal[0]), ("ratearea", scal[1]), ("flowout4", scal[2]), ("flowout2", scal[3]),
                 ("fo2", scal[4])):
        assert x == host[k], k
    assert np.array_equal(to_ref(mf4, f2o), host["mf4"]) and np.array_equal(H(u4), host["u4"])
    assert np.array_equal(H(fr), host["fr2"]) and np.array_equal(H(ff), host["ff"])
    assert np.array_equal(to_ref(mf, f2o), host["mf5"]) and np.array_equal(to_ref(su, c2o), host["su5"])
    for k, t in (("u5", u), ("v5", v), ("w5", w)):
        assert np.array_equal(H(t), host[k]), k


@pytest.mark.parametrize("kind,order", [("struct", 2), ("jitter", 3), ("large", 0)])
def test_float_instantiation_bit_exact(cg, gpu, kind, order):
    """The _f32 calls (float32 host arrays) on a mesh made from float arrays
    against the reference's own T = float instantiation (compiled
    unchanged) on the same float arrays: the whole chain, every array and
    scalar bit for bit."""
    if O.load_ref() is None:
        pytest.skip("reference build absent")
    m, splvl, _, d = _setup(cg, kind, order)
    m32 = dict(m)
    for k in ("faceLambda", "faceArea", "faceNorm", "faceCenter", "faceXpac", "faceXnac", "cellCenter", "cellVolume",
              "regionUVW", "regionDen"):
        if m.get(k) is not None:
            m32[k] = np.ascontiguousarray(np.asarray(m[k]), np.float32)
    sp32 = splvl.astype(np.float32)
    mesh = cg.Mesh.from_arrays(m32, order=order)
    assert mesh.set_regions(m["regionType"], m32["regionUVW"].astype(np.float64),
                            m32["regionDen"].astype(np.float64), m["bndRegion"]) == cg.E_SUCCESS
    assert mesh.set_region_split(sp32.astype(np.float64)) == cg.E_SUCCESS
    d32 = {k: np.ascontiguousarray(v, np.float32) for k, v in d.items()}
    solve = (1, 0, 1)
    want = O.ref_boundary_chain_f32(m32, sp32, d32, 1.3, solve, 0.25)
    got = _host_chain(cg, mesh, d32, solve, f32=True)
    for k in ("flowin", "ratearea", "flowout4", "flowout2", "fo2"):
        assert np.float32(got[k]).view(np.int32) == np.float32(want[k]).view(np.int32), (k, got[k], want[k])
    for k in ("mf5", "su5", "u5", "v5", "w5", "fr2", "ff"):
        assert got[k].dtype == np.float32
        assert np.array_equal(got[k].view(np.int32), want[k].view(np.int32)), k
    assert want["flowin"] != 0 and want["fo2"] != 0.25


def test_boundary_loop_errors(cg, gpu):
    m, splvl, mesh, d = _setup(cg, "struct", 2)
    short = d["mf"][:-1].copy()
    assert cg.FluxMassDolfynBoundaryLoop1(mesh, short)[0] == cg.E_INVALID_INDEX
    assert cg.FluxMassDolfynBoundaryLoop2(mesh, d["mf"].copy(), d["fr"][:-1].copy())[0] == cg.E_INVALID_INDEX
    assert mesh.set_region_split(splvl[:-1]) == cg.E_ARRAY_SIZE_MISMATCH
    rc = cg.lib().cupcfd_gpu_flux_mass_dolfyn_boundary_loop3(mesh.h, 1.0, None)
    assert rc == cg.E_NULL_PTR


def _values(kind, n, rng):
    u, sign = rng.uniform(1e-6, 1e-2, n), rng.choice([-1.0, 1.0], n)
    return {"one sign": -u, "both signs": u * sign,
            "ties": rng.integers(-500, 500, n) * 2.0 ** -rng.integers(0, 40, n),   # few bits: halves of a unit
            "powers": sign * 2.0 ** rng.integers(-30, 30, n),
            "zeros": np.where(rng.uniform(size=n) < 0.9, 0.0 * sign, u),
            "tiny": u * 2.0 ** -1060,                                               # subnormal, also as float
            "huge": np.where(np.arange(n) % 1000 == 700, 1e35, u) * sign,
            "infinite": np.where(np.arange(n) == n // 2, np.inf, u),
            "nan": np.where(np.arange(n) == n // 3, np.nan, u)}[kind]


@pytest.mark.parametrize("n", [0, 1, 33, 4095, 4096, 4097, 8200])   # a block holds 4,096 additions at a time
@pytest.mark.parametrize("kind", ["one sign", "both signs", "ties", "powers", "zeros", "tiny", "huge", "infinite", "nan"])
def test_ordered_sum_rounds_as_the_chain(cg, gpu, kind, n):
    """Loop 1's and loop 2's sums against the chain of additions itself, in
    double and in float: values of one sign, values that keep the sum crossing
    powers of two, ties, zeros of both signs, subnormals, infinities, NaN."""
    rng = np.random.default_rng(100 + n)
    mesh = cg.Mesh.structgen(40, 41, 42, order=cg.ORDER_OWNER)
    nB, nF = mesh.nBoundaries, mesh.nFaces
    face = np.empty(nB, np.int64)
    bnd = mesh.geometry()["faceBnd"]
    face[bnd[bnd >= 0]] = np.nonzero(bnd >= 0)[0]
    chosen = np.sort(rng.choice(nB, n, replace=False))
    region = np.zeros(nB, np.int32)
    vals = _values(kind, n, rng)
    for rtype in (1, 2):
        # three regions of the type, interleaved in boundary order
        region[chosen] = 1 + np.arange(n) % 3
        assert mesh.set_regions([0, rtype, rtype, rtype], np.zeros((4, 3)), np.ones(4), region) == cg.E_SUCCESS
        for t in (np.float64, np.float32):
            mf = np.zeros(nF, t)
            with np.errstate(over="ignore", invalid="ignore", under="ignore"):
                v = vals.astype(t)
                mf[face[chosen]] = v
                total, acc = t(0), np.array([0.5, 0.25, -3.0, 0.0], t)
                want_acc = acc.copy()
                for k in range(n):
                    total = total + v[k]
                    want_acc[1 + k % 3] += v[k]
            if rtype == 1:
                rc, got = cg.FluxMassDolfynBoundaryLoop1(mesh, mf)
            else:
                rc, got = cg.FluxMassDolfynBoundaryLoop2(mesh, mf, acc)
            assert rc == cg.E_SUCCESS, cg.last_error()
            same = lambda a, b: np.array_equal(np.asarray(a, np.float64), np.asarray(b, np.float64), equal_nan=True)
            assert same(got, total), (t, got, total)
            if rtype == 2:
                assert same(acc, want_acc), (t, acc, want_acc)


def _swings(group, n, rng, unit):
    """Values whose running sum rises through `group` of them and falls through the next, inside (1, 2);
    multiples of unit (0: any; those of an amplitude far above the sum's last place often tie)."""
    v = np.empty(n)
    v[0] = at = 1.05
    for i in range(1, n, group):
        w = rng.uniform(0.5, 1.5, min(group, n - i))
        to = (1.05 if at > 1.5 else 1.85) + rng.uniform(0, 0.1)
        w *= (to - at) / w.sum()
        v[i:i + group] = np.round(w / unit) * unit if unit else w
        at += v[i:i + group].sum()
    return v


@pytest.mark.parametrize("n", [4096, 4097, 8200])
@pytest.mark.parametrize("group", [8, 16, 32, 64, 256, 512, 1024])   # 8: one thread's additions, 256: one warp's
def test_ordered_sum_of_swinging_values(cg, gpu, group, n):
    """Totals and region sums of values that swing between two powers of two
    in step with the threads or warps of the sum, against the chain."""
    rng = np.random.default_rng(group + n)
    mesh = cg.Mesh.structgen(40, 41, 42, order=cg.ORDER_OWNER)
    nB, nF = mesh.nBoundaries, mesh.nFaces
    face = np.empty(nB, np.int64)
    bnd = mesh.geometry()["faceBnd"]
    face[bnd[bnd >= 0]] = np.nonzero(bnd >= 0)[0]
    chosen = np.sort(rng.choice(nB, n, replace=False))
    region = np.zeros(nB, np.int32)
    region[chosen] = 1
    assert mesh.set_regions([0, 2], np.zeros((2, 3)), np.ones(2), region) == cg.E_SUCCESS
    for seed in range(40):
        for t in (np.float64, np.float32):
            unit = np.finfo(t).eps if seed % 4 < 2 else 0
            v = ((-1) ** seed * _swings(group, n, np.random.default_rng(seed), unit)).astype(t)
            mf, acc = np.zeros(nF, t), np.zeros(2, t)
            mf[face[chosen]] = v
            rc, got = cg.FluxMassDolfynBoundaryLoop2(mesh, mf, acc)
            assert rc == cg.E_SUCCESS, cg.last_error()
            want = np.add.accumulate(v)[-1]   # one addition after another
            assert got == want and acc[1] == want, (seed, t, got, acc[1], want)


@pytest.mark.parametrize("more", [0, 3])
@pytest.mark.parametrize("wrong", [-1, "nR"])
def test_refused_regions_leave_the_mesh_as_it_was(cg, gpu, wrong, more):
    """set_regions with a region id out of range changes nothing: the chain
    then gives what it gave before (other types, ids and region counts in the
    refused call)."""
    m, splvl, mesh, d = _setup(cg, "struct", 2)
    solve = (1, 0, 1)
    want = _host_chain(cg, mesh, d, solve)
    nR = m["nRegions"] + more
    types = np.resize(np.roll(m["regionType"], 1), nR)
    ids = np.random.default_rng(5).integers(0, nR, m["nBnd"]).astype(np.int32)
    ids[m["nBnd"] // 2] = nR if wrong == "nR" else wrong
    assert mesh.set_regions(types, np.ones((nR, 3)), np.ones(nR), ids) == cg.E_INVALID_INDEX
    got = _host_chain(cg, mesh, d, solve)
    for k, x in want.items():
        assert np.array_equal(got[k], x), k


def test_regions_set_again(cg, gpu):
    """Loop 2's sums after regions of other counts and types replaced the ones before."""
    mesh = cg.Mesh.structgen(23, 19, 17, order=cg.ORDER_OWNER)
    nB, nF = mesh.nBoundaries, mesh.nFaces
    bnd = mesh.geometry()["faceBnd"]
    face = np.empty(nB, np.int64)
    face[bnd[bnd >= 0]] = np.nonzero(bnd >= 0)[0]
    rng = np.random.default_rng(9)
    mf = rng.standard_normal(nF)
    for nR in (2, 7, 3, 300, 1, 5000, 2):
        types = rng.integers(0, 5, nR).astype(np.int32)
        types[nR // 2] = 2
        region = rng.integers(0, nR, nB).astype(np.int32)
        assert mesh.set_regions(types, np.zeros((nR, 3)), np.ones(nR), region) == cg.E_SUCCESS
        acc = rng.standard_normal(nR)
        total, want = 0.0, acc.copy()
        for b in np.nonzero(types[region] == 2)[0]:
            total += mf[face[b]]
            want[region[b]] += mf[face[b]]
        rc, got = cg.FluxMassDolfynBoundaryLoop2(mesh, mf, acc)
        assert rc == cg.E_SUCCESS and got == total and np.array_equal(acc, want), nR
