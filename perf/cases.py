"""The framework's work at the sizes users run it, for timing and for comparing results.

A case names a kind of call, a mesh and the call's options:

  kind      dropin      GradientPhiGaussDolfyn and FluxMassDolfynFaceLoop on host arrays (the reference's calls)
            host_step   forward_adjoint on host arrays
            forward     dev_forward: gradient, mass flux and loss
            step        dev_forward_adjoint: the same and the adjoint
            gradient    dev_gradient with nGradient iterations (non-orthogonal correction)
            vjp         dev_gradient_adjoint and dev_mass_plain_adjoint (the backward of each loop by itself)
            momentum    dev_uvw_face_loop1
            boundaries  the boundary / region loops of the mass-flux step, as a solver step chains them
  mesh      struct (generated hexahedra) or jitter (vertices displaced by a quarter cell, numbering permuted)
  nx ny nz  cells per axis
  order     the cells' internal numbering: owner, morton (the constructors' default), rcm or native
  prec      f64 or f32 (FP32 storage with compensated sums)

The meshes, numbering and geometry come from the library's mesh handle, as a
user's program has them; exact() computes the outputs from those in FP64 with
plain torch.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch


def _package():
    """The package (its folder's name is not an identifier, so it is loaded by path)."""
    name = "cupcfd_b200"
    if name not in sys.modules:
        folder = os.path.join(os.getcwd(), "cup-cfd_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(folder, "__init__.py"),
                                                      submodule_search_locations=[folder])
        sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[name])
    return sys.modules[name]


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _case(kind, mesh, dims, order, prec, **more):
    nx, ny, nz = dims
    return dict(kind=kind, mesh=mesh, nx=nx, ny=ny, nz=nz, order=order, prec=prec, **more)


def listed():
    return [
        # the reference's two calls as an unchanged solver makes them, on its kernel benchmark's small mesh
        dict(name="dropin_f64_16", **_case("dropin", "struct", (16, 16, 16), "morton", "f64")),
        # one design step on a small mesh: latency and launches
        dict(name="step_f32_16", **_case("step", "struct", (16, 16, 16), "owner", "f32")),
        # plain FP64 forward at the middle size
        dict(name="forward_f64_128", **_case("forward", "struct", (128, 128, 128), "owner", "f64")),
        # the benchmark's step
        dict(name="step_f32_256", **_case("step", "struct", (256, 256, 256), "owner", "f32")),
        # irregular mesh, permuted numbering, renumbered along the Z curve
        dict(name="step_f32_jitter_192", **_case("step", "jitter", (192, 192, 192), "morton", "f32")),
        # FP64 sensitivities on an irregular mesh, reverse Cuthill-McKee numbering
        dict(name="step_f64_jitter_96", **_case("step", "jitter", (96, 96, 96), "rcm", "f64")),
        # a mesh whose rows, planes and cell count are no multiples of anything
        dict(name="step_f32_ragged", **_case("step", "struct", (149, 131, 137), "owner", "f32")),
        # gradient with two non-orthogonal corrections, which only an irregular mesh needs
        dict(name="gradient_f64_jitter_112", **_case("gradient", "jitter", (112, 112, 112), "morton", "f64", iters=3)),
        # the backward of the two loops on sensitivities that come from another program's loss
        dict(name="vjp_f64_128", **_case("vjp", "struct", (128, 128, 128), "morton", "f64")),
        # the momentum equation's face loop with inlets, outlets, walls and symmetry planes
        dict(name="momentum_f64_160", **_case("momentum", "struct", (160, 160, 160), "owner", "f64")),
        # flow in / out, rescaled outlets: the ordered sums over 221,184 boundary faces
        dict(name="boundaries_f64_192", **_case("boundaries", "struct", (192, 192, 192), "owner", "f64")),
        # sensitivities from and to (pinned) host arrays
        dict(name="host_step_f32_128", **_case("host_step", "struct", (128, 128, 128), "owner", "f32")),
    ]


# per kind: relative weight, fewest and most cells, precisions, orders
_RANGES = {
    "dropin": (1, 16 ** 3, 48 ** 3, ("f64",), ("morton", "owner", "native")),
    "step": (4, 16 ** 3, 224 ** 3, ("f32", "f32", "f64"), ("owner", "morton", "rcm")),
    "forward": (2, 16 ** 3, 192 ** 3, ("f64", "f32"), ("owner", "morton")),
    "gradient": (1, 16 ** 3, 128 ** 3, ("f64", "f32"), ("owner", "morton")),
    "vjp": (1, 16 ** 3, 128 ** 3, ("f64", "f32"), ("owner", "morton")),
    "momentum": (1, 16 ** 3, 160 ** 3, ("f64",), ("owner", "morton")),
    "boundaries": (1, 16 ** 3, 192 ** 3, ("f64",), ("owner", "morton")),
    "host_step": (1, 16 ** 3, 128 ** 3, ("f32", "f64"), ("owner", "morton")),
}


def draw(rng):
    kinds = sorted(_RANGES)
    kind = rng.choices(kinds, [_RANGES[k][0] for k in kinds])[0]
    _, least, most, precs, orders = _RANGES[kind]
    prec, order = rng.choice(precs), rng.choice(orders)
    if prec == "f64" and kind == "step":
        most = 128 ** 3
    if order == "rcm":
        most = min(most, 96 ** 3)  # that numbering is made on the host
    cells = math.exp(rng.uniform(math.log(least), math.log(most)))
    side = cells ** (1 / 3)
    nx = max(8, round(side * rng.uniform(0.75, 1.3)))
    ny = max(8, round(side * rng.uniform(0.75, 1.3)))
    nz = max(8, min(round(cells / (nx * ny)), most // (nx * ny)))
    # regions go by the sides of a generated mesh; corrections are for irregular ones
    mesh = "struct" if kind in ("dropin", "momentum", "boundaries") else "jitter" if kind == "gradient" else \
        rng.choice(("struct", "struct", "jitter"))
    more = {"iters": rng.randint(1, 3)} if kind == "gradient" else {}
    return _case(kind, mesh, (nx, ny, nz), order, prec, **more)


def _counts(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    nB = 2 * (ny * nz + nx * nz + nx * ny)
    nFi = (nx - 1) * ny * nz + nx * (ny - 1) * nz + nx * ny * (nz - 1)
    return nx * ny * nz, nFi + nB, nFi, nB


def work(case):
    """Each distinct input read once, each output written once; int32 ids, FP64 volumes; r: bytes of a real."""
    nC, nF, nFi, nB = _counts(case)
    r = 8 if case["prec"] == "f64" else 4
    ids = 4 * nF + 4 * nFi                       # the two cells of a face (a boundary face has one)
    geom = 4 * r * nF + 8 * nC + ids             # S, lambda; volumes
    fwd = geom + 5 * r * nC + r * nB + 3 * r * nC + r * nFi     # phi, rho, u, v, w; phi_b; gradient; mass flux
    kind = case["kind"]
    # operations: about 60 per cell side of an interior face in a forward, twice that with its adjoint
    flops = 60 * 2 * nFi
    if kind == "dropin":
        # gradient: phi in, two gradients out; mass loop: 12 gradient and 6 cell fields in, fluxes and rface in/out
        nbytes = geom + 7 * r * nC + (12 + 6 + 2) * r * nC + 4 * r * nC + 5 * r * nF + 6 * r * nF
    elif kind == "forward":
        nbytes = fwd + r * nFi
    elif kind in ("step", "host_step"):
        nbytes, flops = fwd + r * nFi + 5 * r * nC + r * nB, 2 * flops
    elif kind == "gradient":
        nbytes = geom + 4 * r * nC + r * nB
        if case["iters"] > 1:                    # centres of cells and faces, and the previous iterate, each time
            nbytes += (case["iters"] - 1) * (geom + 10 * r * nC + r * nB + 3 * r * nF)
        flops *= case["iters"]
    elif kind == "vjp":
        nbytes = geom + 4 * r * nC + r * nB + 4 * r * nF + ids + 8 * r * nC + r * nFi
    elif kind == "momentum":
        nbytes, flops = 224 * nC + 64 * nFi + 4 * nB, 2 * flops
    else:  # boundaries: per boundary its face, region, normal and area, flux and velocities in and out, its cell's su
        nbytes, flops = (4 + 4 + 32 + 16 + 7 * 8 + 16) * nB, 20 * nB
    return {"bytes": float(nbytes), "flops": float(flops)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
SMALL = 1e-18
BLEND = 0.9
DEFAULT, INLET, OUTLET, SYMP, WALL = range(5)
# regions: the default one, the inlet, two outlets, a symmetry plane, the walls
REGION_TYPE = np.array([DEFAULT, INLET, OUTLET, SYMP, WALL, OUTLET], np.int32)


def _mesh(case, seed):
    cg = _package()
    order = {"native": cg.ORDER_NATIVE, "morton": cg.ORDER_MORTON, "owner": cg.ORDER_OWNER,
             "rcm": cg.ORDER_RCM}[case["order"]]
    dims = (case["nx"], case["ny"], case["nz"])
    if case["mesh"] == "jitter":
        return cg.Mesh.jittered(*dims, jitter=0.25, seed=1 + seed % 1000, permute=True, order=order)
    return cg.Mesh.structgen(*dims, order=order)


def _regions(case, seed):
    """Region data of a generated mesh: flow in through the low x side and out through the high one (two outlets,
    the lower and the upper half), walls on the y sides, symmetry on the low z side, nothing on the high one. The
    generator numbers the x sides' boundaries first (low and high in turn), then the y and the z sides'."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    r = np.random.default_rng(seed)
    x = np.empty(2 * ny * nz, np.int32)
    x[0::2] = 1
    x[1::2] = np.where(np.arange(ny * nz) < ny * nz // 2, 2, 5)
    z = np.repeat(np.array([3, 0], np.int32), nx * ny)
    bnd = np.concatenate([x, np.full(2 * nx * nz, 4, np.int32), z])
    uvw = np.zeros((6, 3))
    uvw[1] = r.uniform(0.5, 1.5), 0.1, 0.0
    uvw[4] = 0.0, 0.0, r.uniform(-0.1, 0.1)
    return bnd, uvw, r.uniform(0.9, 1.1, 6), r.uniform(0.3, 0.7, 6)


def _set_regions(mesh, regions):
    cg = _package()
    bnd, uvw, den, split = regions
    if mesh.set_regions(REGION_TYPE, uvw, den, bnd) != cg.E_SUCCESS or mesh.set_region_split(split) != cg.E_SUCCESS:
        raise RuntimeError(cg.last_error())


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _fields(case, seed):
    """phi, phi_b ~ U[-1,1], rho ~ U[0.9,1.1], u, v, w ~ N(0,1), face weights ~ N(0,1), in the internal numbering."""
    nC, nF, _, nB = _counts(case)
    g = _generator(seed)
    d = dict(dtype=torch.float64 if case["prec"] == "f64" else torch.float32, device="cuda")
    phi = torch.rand(nC, generator=g, **d) * 2 - 1
    phiB = torch.rand(nB, generator=g, **d) * 2 - 1
    rho = torch.rand(nC, generator=g, **d) * 0.2 + 0.9
    vel = torch.randn(3, nC, generator=g, **d)
    gface = torch.randn(nF, generator=g, **d)
    gbar = torch.randn(3, nC, generator=g, **d) if case["kind"] == "vjp" else None
    # FP64 keeps the state as four blocks, FP32 as one record per cell
    state = torch.cat([rho[None], vel]) if case["prec"] == "f64" else torch.stack([rho, *vel], 1).contiguous()
    return dict(phi=phi, phiB=phiB, state=state, gface=gface, gbar=gbar)


def _momentum_fields(case, seed):
    """U[1e-6,1e-2] as the reference's kernel benchmark draws them; signed mass fluxes, random gradients."""
    nC, nF, _, nB = _counts(case)
    g = _generator(seed)
    d = dict(dtype=torch.float64, device="cuda")
    f = {k: torch.rand(nC, generator=g, **d) * (1e-2 - 1e-6) + 1e-6
         for k in ("u", "v", "w", "visC", "su", "sv", "sw", "au", "av", "aw")}
    f |= {k: torch.rand(nB, generator=g, **d) * (1e-2 - 1e-6) + 1e-6 for k in ("uB", "vB", "wB", "visB")}
    f["grads"] = torch.randn(9, nC, generator=g, **d) * 1e-2
    f["massFlux"] = torch.randn(nF, generator=g, **d) * 1e-2
    f["rFace"] = torch.zeros(2 * nF, **d)
    r = np.random.default_rng(seed + 1)
    return f, r.uniform(0.1, 2.0, nF), r.uniform(0.01, 0.2, nB)


def _boundary_fields(case, seed, bnd_face):
    """Mass fluxes that enter at the inlet and leave at the outlets (a tenth of them back), random elsewhere."""
    nC, nF, _, nB = _counts(case)
    g = _generator(seed)
    d = dict(dtype=torch.float64, device="cuda")
    region = torch.from_numpy(_regions(case, seed)[0]).cuda().long()
    rtype = torch.from_numpy(REGION_TYPE).cuda().long()[region]
    size = torch.rand(nB, generator=g, **d) * (1e-2 - 1e-6) + 1e-6
    back = torch.where(torch.rand(nB, generator=g, **d) < 0.1, -1.0, 1.0)
    mf = torch.randn(nF, generator=g, **d) * 1e-2
    mf[bnd_face] = torch.where(rtype == INLET, -size, size * back)
    f = dict(mf=mf, su=torch.randn(nC, generator=g, **d))
    f |= {k: torch.rand(nB, generator=g, **d) * (1e-2 - 1e-6) + 1e-6 for k in ("u", "v", "w")}
    f["den"] = torch.rand(nB, generator=g, **d) * 0.2 + 0.9
    f |= dict(fr=torch.zeros(6, **d), ff=torch.zeros(6, **d), sc=torch.zeros(5, **d))
    return f


def _host_fields(case, seed):
    """The inputs of the host calls, reference numbering."""
    nC, nF, _, nB = _counts(case)
    r = np.random.default_rng(seed)
    t = np.float64 if case["prec"] == "f64" else np.float32
    f = dict(phi=r.uniform(-1, 1, nC), phiB=r.uniform(-1, 1, nB), den=r.uniform(0.9, 1.1, nC),
             u=r.standard_normal(nC), v=r.standard_normal(nC), w=r.standard_normal(nC))
    if case["kind"] == "host_step":
        f["gface"] = r.standard_normal(nF)
    else:
        # vector arrays as the reference lays its records out: 8 bytes of the object, then the components
        f |= {k: np.ascontiguousarray(np.pad(r.standard_normal((nC, 3)), ((0, 0), (1, 0))))
              for k in ("dudx", "dvdx", "dwdx", "dpdx")}
        f |= dict(p=r.uniform(-1, 1, nC), ar=r.uniform(0.9, 1.1, nC), su=r.uniform(-1, 1, nC),
                  vis=r.uniform(0, 1, nC), massFlux=np.zeros(nF), rface=np.zeros(2 * nF), denB=np.zeros(nB),
                  visB=np.zeros(nB))
    return {k: v.astype(t) for k, v in f.items()}


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.from_numpy(a).dtype, pin_memory=True).numpy()
    t[...] = a
    return t


def prepare(case, seed):
    cg = _package()
    kind = case["kind"]
    nC, nF, _, nB = _counts(case)
    s = dict(kind=kind, case=dict(case), mesh=_mesh(case, seed), stream=torch.cuda.current_stream(),
             prec=cg.PREC_F64 if case["prec"] == "f64" else cg.PREC_F32C)
    if kind == "host_step":
        # pinned, inputs and outputs
        f = {k: _pinned(v) for k, v in _host_fields(case, seed).items()}
        t = f["phi"].dtype
        out = dict(grad=(nC, 3), massFlux=(nF,), phiBar=(nC,), phiBBar=(nB,), denBar=(nC,), uBar=(nC,), vBar=(nC,),
                   wBar=(nC,))
        return s | dict(f=f, out={k: _pinned(np.zeros(v, t)) for k, v in out.items()} | dict(loss=np.zeros(1)))
    if kind == "dropin":
        _set_regions(s["mesh"], _regions(case, seed))
        return s | dict(f=_host_fields(case, seed), g=np.zeros((nC, 4)), go=np.zeros((nC, 4)),
                        counts=np.zeros(4, np.int32))
    if kind == "momentum":
        _set_regions(s["mesh"], _regions(case, seed))
        f, rlencos, distance = _momentum_fields(case, seed)
        if s["mesh"].set_face_rlencos(rlencos) != cg.E_SUCCESS or \
                s["mesh"].set_boundary_distance(distance) != cg.E_SUCCESS:
            raise RuntimeError(cg.last_error())
        return s | dict(f=f)
    if kind == "boundaries":
        _set_regions(s["mesh"], _regions(case, seed))
        return s | dict(f=_boundary_fields(case, seed, _boundary_faces(s["mesh"], case)))
    f = _fields(case, seed)
    e = lambda *n: torch.zeros(n, dtype=f["phi"].dtype, device="cuda")  # noqa: E731
    s |= dict(f=f, grad=e(3, nC), grad_o=e(3, nC), mflux=e(nF), phiBar=e(nC), phiBBar=e(nB),
              stateBar=torch.zeros_like(f["state"]), loss=torch.zeros(1, dtype=torch.float64, device="cuda"))
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    cg = _package()
    kind, mesh, st, f = s["kind"], s["mesh"], s["stream"], s["f"]
    if kind == "step":
        cg.dev_forward_adjoint(mesh, s["prec"], f["phi"], f["phiB"], f["state"], f["gface"], s["grad"], s["mflux"],
                               s["phiBar"], s["phiBBar"], s["stateBar"], s["loss"], stream=st)
        return {k: s[k] for k in ("grad", "mflux", "phiBar", "phiBBar", "stateBar", "loss")}
    if kind == "forward":
        cg.dev_forward(mesh, s["prec"], f["phi"], f["phiB"], f["state"], s["grad"], s["mflux"], f["gface"], s["loss"],
                       stream=st)
        return {k: s[k] for k in ("grad", "mflux", "loss")}
    if kind == "gradient":
        cg.dev_gradient(mesh, s["prec"], f["phi"], f["phiB"], s["grad"], s["grad_o"], nGradient=s["case"]["iters"],
                        stream=st)
        return {k: s[k] for k in ("grad", "grad_o")}
    if kind == "vjp":
        cg.dev_gradient_adjoint(mesh, s["prec"], f["gbar"], s["phiBar"], s["phiBBar"], stream=st)
        cg.dev_mass_plain_adjoint(mesh, s["prec"], f["state"], f["gface"], s["stateBar"], stream=st)
        return {k: s[k] for k in ("phiBar", "phiBBar", "stateBar")}
    if kind == "momentum":
        cg.dev_uvw_face_loop1(mesh, BLEND, SMALL, f["u"], f["v"], f["w"], f["uB"], f["vB"], f["wB"], f["visC"],
                              f["visB"], f["massFlux"], f["grads"], f["rFace"], f["su"], f["sv"], f["sw"], f["au"],
                              f["av"], f["aw"], stream=st)
        return {k: f[k] for k in ("massFlux", "rFace", "su", "sv", "sw", "au", "av", "aw", "uB", "vB", "wB")}
    if kind == "boundaries":
        sc = f["sc"]
        f["fr"].zero_()
        sc[4:5].zero_()
        cg.dev_boundary_loop1(mesh, f["mf"], sc[0:1], stream=st)
        cg.dev_boundary_loop3(mesh, sc[0:1], sc[1:2], stream=st)
        cg.dev_boundary_loop4(mesh, f["mf"], f["u"], f["v"], f["w"], f["den"], sc[1:2], sc[2:3], stream=st)
        cg.dev_boundary_loop2(mesh, f["mf"], f["fr"], sc[3:4], stream=st)
        cg.dev_region_loop(mesh, f["ff"], f["fr"], sc[0:1], stream=st)
        cg.dev_boundary_loop5(mesh, f["mf"], f["su"], f["u"], f["v"], f["w"], 1.3, (1, 1, 1), f["ff"], sc[4:5],
                              stream=st)
        return {k: f[k] for k in ("mf", "su", "u", "v", "w", "fr", "ff", "sc")}
    if kind == "host_step":
        return dict(cg.forward_adjoint(mesh, s["prec"], *[f[k] for k in ("phi", "phiB", "den", "u", "v", "w",
                                                                         "gface")], out=s["out"]))
    # dropin
    s["counts"][:] = 0
    cg.check(cg.GradientPhiGaussDolfyn(mesh, 1, f["phi"], f["phiB"], s["g"], s["go"]))
    cg.check(cg.FluxMassDolfynFaceLoop(
        mesh, f["dudx"], f["dvdx"], f["dwdx"], f["dpdx"], f["den"], f["denB"], f["u"], f["v"], f["w"], f["massFlux"],
        f["p"], f["ar"], f["su"], f["rface"], SMALL, s["counts"], False, False, True, False, None, None, None, None,
        f["vis"], f["visB"], None, None))
    return dict(g=s["g"], go=s["go"], counts=s["counts"], **{k: f[k] for k in ("massFlux", "rface", "su", "denB",
                                                                              "visB")})


# ---------------------------------------------------------------------------
# the outputs in FP64, plain torch
# ---------------------------------------------------------------------------
def _inverse(p):
    q = torch.empty_like(p)
    q[p] = torch.arange(len(p), device=p.device)
    return q


def _connectivity(mesh, internal):
    """Faces and geometry on the GPU, internal (or reference) numbering: P, N (-1 on a boundary), b (-1 inside)."""
    geo = mesh.geometry()
    f2o = c2o = None
    if internal:
        cells, faces = mesh.numbering()
        c2o, f2o = torch.from_numpy(cells).cuda().long(), torch.from_numpy(faces).cuda().long()

    def faces_of(a):
        t = torch.from_numpy(a).cuda()
        return t[f2o] if internal else t

    def cells_of(a):
        t = torch.from_numpy(a).cuda()
        return t[c2o] if internal else t

    m = {k: faces_of(geo[v]).long() for k, v in (("P", "faceCell1"), ("N", "faceCell2"), ("b", "faceBnd"))}
    if internal:
        o2c = _inverse(c2o)
        m["P"], m["N"] = o2c[m["P"]], torch.where(m["N"] < 0, -1, o2c[m["N"].clamp(min=0)])
    m |= {k: faces_of(geo[v]) for k, v in (("S", "faceNorm"), ("lam", "faceLambda"), ("area", "faceArea"),
                                           ("xf", "faceCenter"))}
    m |= {k: cells_of(geo[v]) for k, v in (("V", "cellVolume"), ("xc", "cellCenter"))}
    m["inner"] = (m["N"] >= 0).nonzero()[:, 0]
    m["outer"] = (m["N"] < 0).nonzero()[:, 0]
    m["f2o"] = f2o
    return m


def _boundary_faces(mesh, case):
    """The internal face of each boundary id: a generated mesh's faces in label order are its x, y and z ones, and
    its boundary labels follow them (x sides by z, y and side; y sides by z, side and x; z sides by side, y and x)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    r = lambda n: torch.arange(n, device="cuda")  # noqa: E731
    row = r(nz * ny)[:, None] * (nx + 1)
    x = torch.cat([row, row + nx], 1).reshape(-1)
    first = ny * nz * (nx + 1)
    y = first + r(nz)[:, None, None] * nx * (ny + 1) + torch.tensor([0, ny * nx], device="cuda")[None, :, None] + r(nx)
    first += nx * nz * (ny + 1)
    z = first + torch.tensor([0, nx * ny * nz], device="cuda")[:, None] + r(nx * ny)
    faces = _inverse(torch.from_numpy(mesh.numbering()[1]).cuda().long())
    return faces[torch.cat([x, y.reshape(-1), z.reshape(-1)])]


def _gradient(m, phi, phiB, iters):
    i, o, nC = m["inner"], m["outer"], len(m["V"])
    P, N, S, lam = m["P"][i], m["N"][i], m["S"][i], m["lam"][i][:, None]
    grad = torch.zeros(nC, 3, dtype=torch.float64, device="cuda")
    for k in range(iters):
        pf = phi[N] * lam[:, 0] + phi[P] * (1 - lam[:, 0])
        if k:
            d = m["xf"][i] - (m["xc"][N] * lam + m["xc"][P] * (1 - lam))
            pf = pf + ((grad[N] * lam + grad[P] * (1 - lam)) * d).sum(1)
        new = torch.zeros_like(grad)
        t = pf[:, None] * S  # the reference adds a face's term into both of its cells with the same sign
        new.index_add_(0, P, t)
        new.index_add_(0, N, t)
        new.index_add_(0, m["P"][o], phiB[m["b"][o]][:, None] * m["S"][o])
        grad = new / m["V"][:, None]
    return grad


def _mass_plain(m, rho, vel):
    i = m["inner"]
    P, N, lam = m["P"][i], m["N"][i], m["lam"][i]
    rf = rho[N] * lam + rho[P] * (1 - lam)
    uf = vel[N] * lam[:, None] + vel[P] * (1 - lam[:, None])
    return rf, uf, rf * (uf * m["S"][i]).sum(1)


def _gradient_adjoint(m, h, nB):
    i, o = m["inner"], m["outer"]
    P, N, lam = m["P"][i], m["N"][i], m["lam"][i]
    t = ((h[P] + h[N]) * m["S"][i]).sum(1)
    phiBar = torch.zeros(len(m["V"]), dtype=torch.float64, device="cuda")
    phiBar.index_add_(0, P, (1 - lam) * t)
    phiBar.index_add_(0, N, lam * t)
    phiBBar = torch.zeros(nB, dtype=torch.float64, device="cuda")
    phiBBar[m["b"][o]] = (h[m["P"][o]] * m["S"][o]).sum(1)
    return phiBar, phiBBar


def _mass_adjoint(m, rf, uf, weight):
    i, nC = m["inner"], len(m["V"])
    P, N, lam, w = m["P"][i], m["N"][i], m["lam"][i], weight[m["inner"]]
    a = w * (uf * m["S"][i]).sum(1)
    b = (w * rf)[:, None] * m["S"][i]
    out = torch.zeros(nC, 4, dtype=torch.float64, device="cuda")
    both = torch.cat([a[:, None], b], 1)
    out.index_add_(0, P, both * (1 - lam[:, None]))
    out.index_add_(0, N, both * lam[:, None])
    return out


def _states(case, state):
    state = state.double()
    return (state[0], state[1:].T) if case["prec"] == "f64" else (state[:, 0], state[:, 1:])


def _exact_loops(case, m, f):
    """forward, step, gradient and vjp (internal numbering)."""
    kind, f64 = case["kind"], case["prec"] == "f64"
    nC, nF, _, nB = _counts(case)
    phi, phiB = f["phi"].double(), f["phiB"].double()
    if kind == "gradient":
        g = _gradient(m, phi, phiB, case["iters"]).T.contiguous()
        return dict(grad=g, grad_o=g.clone())
    rho, vel = _states(case, f["state"])
    rf, uf, mass = _mass_plain(m, rho, vel)
    weight = f["gface"].double()
    if kind == "vjp":
        phiBar, phiBBar = _gradient_adjoint(m, f["gbar"].double().T / m["V"][:, None], nB)
        sb = _mass_adjoint(m, rf, uf, weight)
        return dict(phiBar=phiBar, phiBBar=phiBBar, stateBar=sb.T.contiguous() if f64 else sb)
    g = _gradient(m, phi, phiB, 1)
    mflux = torch.zeros(nF, dtype=torch.float64, device="cuda")
    mflux[m["inner"]] = mass
    loss = ((m["V"] * (g * g).sum(1)).sum() + (weight[m["inner"]] * mass).sum())[None]
    out = dict(grad=g.T.contiguous(), mflux=mflux, loss=loss)
    if kind == "step":
        out["phiBar"], out["phiBBar"] = _gradient_adjoint(m, 2 * g, nB)
        sb = _mass_adjoint(m, rf, uf, weight)
        out["stateBar"] = sb.T.contiguous() if f64 else sb
    return out


def _exact_host_step(case, m, f):
    nB = _counts(case)[3]
    t = {k: torch.from_numpy(v).cuda().double() for k, v in f.items()}
    vel = torch.stack([t["u"], t["v"], t["w"]], 1)
    rf, uf, mass = _mass_plain(m, t["den"], vel)
    g = _gradient(m, t["phi"], t["phiB"], 1)
    mflux = torch.zeros_like(t["gface"])
    mflux[m["inner"]] = mass
    phiBar, phiBBar = _gradient_adjoint(m, 2 * g, nB)
    sb = _mass_adjoint(m, rf, uf, t["gface"])
    loss = ((m["V"] * (g * g).sum(1)).sum() + (t["gface"][m["inner"]] * mass).sum())[None]
    return dict(grad=g, massFlux=mflux, phiBar=phiBar, phiBBar=phiBBar, denBar=sb[:, 0].clone(),
                uBar=sb[:, 1].clone(), vBar=sb[:, 2].clone(), wBar=sb[:, 3].clone(), loss=loss)


def _exact_dropin(case, m, f, regions):
    bnd, uvw, den_r, _ = regions
    t = {k: torch.from_numpy(v).cuda() for k, v in f.items()}
    nC, nF, _, nB = _counts(case)
    g = _gradient(m, t["phi"], t["phiB"], 1)
    pad = lambda a: torch.cat([torch.zeros(len(a), 1, dtype=a.dtype, device="cuda"), a], 1)  # noqa: E731
    i, o = m["inner"], m["outer"]
    P, N, S, lam = m["P"][i], m["N"][i], m["S"][i], m["lam"][i]
    mean = lambda a: a[N] * (lam if a.dim() == 1 else lam[:, None]) + a[P] * (1 - (lam if a.dim() == 1 else lam[:, None]))  # noqa: E731,E501
    d = m["xf"][i] - mean(m["xc"])
    u = torch.stack([mean(t[a]) + (mean(t[b][:, 1:]) * d).sum(1) for a, b in (("u", "dudx"), ("v", "dvdx"),
                                                                              ("w", "dwdx"))], 1)
    mass = mean(t["den"]) * (u * S).sum(1)
    n = S / S.norm(dim=1, keepdim=True)
    dp = t["dpdx"][:, 1:][P]
    # a generated mesh has no auxiliary points: both are the origin, and the last three terms vanish
    pip, pin = t["p"][P] - (dp * m["xc"][P]).sum(1), t["p"][N] - (dp * m["xc"][N]).sum(1)
    apv = mean(t["den"] * t["ar"]) * (m["area"][i] * mean(m["V"])) / ((m["xc"][N] - m["xc"][P]) * n).sum(1)
    flux, rface, su, denB, visB = (t[k].clone() for k in ("massFlux", "rface", "su", "denB", "visB"))
    flux[i] = mass - apv * (pin - pip)
    rface.view(-1, 2)[i] = -apv[:, None].expand(-1, 2)
    reg = torch.from_numpy(bnd).cuda().long()[m["b"][o]]
    rt = torch.from_numpy(REGION_TYPE).cuda().long()[reg]
    uvw, den_r = torch.from_numpy(uvw).cuda(), torch.from_numpy(den_r).cuda()
    Po, So, bo = m["P"][o], m["S"][o], m["b"][o]
    vel = torch.stack([t["u"], t["v"], t["w"]], 1)
    q = den_r[reg] * (uvw[reg] * So).sum(1)
    out = t["den"][Po] * (vel[Po] * So).sum(1)
    back = (rt == OUTLET) & (out < 0)
    fl = torch.where(rt == INLET, q, torch.where(back, torch.full_like(out, SMALL), out))
    flux[o] = torch.where((rt == INLET) | (rt == OUTLET), fl, torch.where(rt == DEFAULT, flux[o], 0.0))
    su.index_add_(0, Po[rt == INLET], -q[rt == INLET])
    denB[bo[rt == OUTLET]] = t["den"][Po[rt == OUTLET]]
    visB[bo[back]] = t["vis"][Po[back]]
    return dict(g=pad(g), go=pad(g), counts=None, massFlux=flux, rface=rface, su=su, denB=denB, visB=visB)


def _exact_momentum(case, m, f, rlencos, distance, regions):
    """FluxUVWDolfynFaceLoop1 (UVWKernels.ipp:38-512), internal numbering."""
    bnd, uvw, _, _ = regions
    rl = torch.from_numpy(rlencos).cuda()[m["f2o"]]
    dist = torch.from_numpy(distance).cuda()
    i, o = m["inner"], m["outer"]
    rtype = torch.from_numpy(REGION_TYPE).cuda().long()
    reg = torch.from_numpy(bnd).cuda().long()[m["b"][o]]
    rt, uvw = rtype[reg], torch.from_numpy(uvw).cuda()
    bo, Po, So, xo = m["b"][o], m["P"][o], m["S"][o], m["xf"][o] - m["xc"][m["P"][o]]
    vel = torch.stack([f["u"], f["v"], f["w"]], 1)
    grad = f["grads"].T.reshape(-1, 3, 3)                     # [cell][component][axis]
    nF = len(m["P"])
    mf, rface = f["massFlux"].clone(), f["rFace"].clone()
    # values that the reference's loop carries from face to face, in label order
    label = m["f2o"]
    place = _inverse(label)
    setter = torch.full((nF,), -1, device="cuda")             # last inlet / outlet face up to each label
    inout = (rt == INLET) | (rt == OUTLET)
    setter[label[o[inout]]] = label[o[inout]]
    last = torch.cummax(setter, 0).values
    setsvis = setter.clone()
    setsvis[label[i]] = label[i]
    lastvis = torch.cummax(setsvis, 0).values
    slot = torch.full((nF,), -1, device="cuda")
    slot[o] = torch.arange(len(o), device="cuda")
    carried = last[label[i]]
    k = slot[place[carried.clamp(min=0)]].clamp(min=0)
    uF = torch.where((rt[k] == INLET)[:, None], uvw[reg[k]], vel[Po[k]])
    uF = torch.where((carried >= 0)[:, None], uF, 0.0)
    P, N, S, lam = m["P"][i], m["N"][i], m["S"][i], m["lam"][i]
    g = grad[N] * lam[:, None, None] + grad[P] * (1 - lam[:, None, None])
    vis = f["visC"][N] * lam + f["visC"][P] * (1 - lam)
    visface = vis * rl[i]
    x = m["xc"][N] - m["xc"][P]
    q = mf[i]
    conv = torch.clamp(q, max=0)[:, None] * vel[N] + torch.clamp(q, min=0)[:, None] * vel[P]
    blend = BLEND * (q[:, None] * uF - conv)
    term = -blend + vis[:, None] * ((g + g.transpose(1, 2)) * S[:, None, :]).sum(2) \
        - visface[:, None] * (g * x[:, None, :]).sum(2)
    s = torch.stack([f["su"], f["sv"], f["sw"]], 1)
    a = torch.stack([f["au"], f["av"], f["aw"]], 1)
    s.index_add_(0, P, term)
    s.index_add_(0, N, -term)
    pairs = rface.view(-1, 2)
    pairs[i, 0] = -visface - torch.clamp(q, min=0)
    pairs[i, 1] = -visface + torch.clamp(q, max=0)
    # inlets and outlets
    qo = mf[o]
    qo = torch.where((rt == OUTLET) & (qo < 0), torch.full_like(qo, SMALL), qo)
    mf[o] = torch.where(rt == OUTLET, qo, mf[o])
    uin = torch.where((rt == INLET)[:, None], uvw[reg], vel[Po])
    viso = torch.where(rt == INLET, f["visB"][bo], f["visC"][Po])
    vf = viso * rl[o]
    fl = -vf + torch.clamp(qo, max=0)
    go = grad[Po]
    t = -fl[:, None] * uin + viso[:, None] * ((go + go.transpose(1, 2)) * So[:, None, :]).sum(2) \
        - vf[:, None] * (go * xo[:, None, :]).sum(2)
    s.index_add_(0, Po[inout], t[inout])
    a.index_add_(0, Po[inout], -fl[inout][:, None].expand(-1, 3))
    new = {n: f[n].clone() for n in ("uB", "vB", "wB")}
    ub = torch.stack([new["uB"], new["vB"], new["wB"]], 1)
    ub[bo[inout]] = uin[inout]
    # symmetry planes
    y = rt == SYMP
    visfaces = torch.zeros(nF, dtype=torch.float64, device="cuda")
    visfaces[i], visfaces[o] = visface, vf
    lv = lastvis[label[o]]
    X = torch.where(lv >= 0, visfaces[place[lv.clamp(min=0)]], 0.0)
    us = vel[Po] + (go * xo[:, None, :]).sum(2)
    n = So / So.norm(dim=1, keepdim=True)
    force = 2 * f["visC"][Po][:, None] * ((us * n).sum(1)[:, None] * n) / dist[bo][:, None] * m["area"][o][:, None]
    s.index_add_(0, Po[y], (X[:, None] * vel[Po] - force)[y])
    a.index_add_(0, Po[y], X[y][:, None].expand(-1, 3))
    ub[bo[y]] = us[y]
    # walls
    y = rt == WALL
    X = f["visB"][bo] * m["area"][o] / xo.norm(dim=1)
    up = vel[Po] - uvw[reg]
    ut = up - (up * n).sum(1)[:, None] * n
    force = f["visB"][bo][:, None] * ut / dist[bo][:, None] * m["area"][o][:, None]
    force = torch.where((ut.abs().sum(1) > SMALL)[:, None], force, 0.0)
    s.index_add_(0, Po[y], (X[:, None] * vel[Po] - force)[y])
    a.index_add_(0, Po[y], X[y][:, None].expand(-1, 3))
    ub[bo[y]] = uvw[reg][y]
    cols = lambda t, names: {k: t[:, j].clone() for j, k in enumerate(names)}  # noqa: E731
    return dict(massFlux=mf, rFace=rface, **cols(s, ("su", "sv", "sw")), **cols(a, ("au", "av", "aw")),
                **cols(ub, ("uB", "vB", "wB")))


def _exact_boundaries(m, f, regions):
    """FluxMassDolfynBoundaryLoop1, 3, 4, 2, the region loop and 5 (MassKernels.ipp:311-554)."""
    bnd, _, _, split = regions
    reg, split = torch.from_numpy(bnd).cuda().long(), torch.from_numpy(split).cuda()
    rtype = torch.from_numpy(REGION_TYPE).cuda().long()
    face = torch.empty(len(reg), dtype=torch.int64, device="cuda")
    face[m["b"][m["outer"]]] = m["outer"]
    rt, cell = rtype[reg], m["P"][face]
    i, o = rt == INLET, rt == OUTLET
    mf, su, fr = f["mf"].clone(), f["su"].clone(), f["fr"].clone()
    u = torch.stack([f["u"], f["v"], f["w"]], 1)
    flowin = mf[face[i]].sum()
    rate = -flowin / m["area"][face[o]].sum()
    area, n = m["area"][face[o]], m["S"][face[o]] / m["S"][face[o]].norm(dim=1, keepdim=True)
    q = rate * area * split[reg[o]]
    out4 = q.sum()
    u[o] = (q / f["den"][o] / area)[:, None] * n
    fr.index_add_(0, reg[o], q)
    ff = torch.where(rtype == OUTLET, -split * flowin / fr, 0.0)
    mf[face[o]] = q * ff[reg[o]]
    u[o] *= 1.3
    su.index_add_(0, cell[o], -mf[face[o]])
    sc = torch.stack([flowin, rate, out4, q.sum(), mf[face[o]].sum()])
    return dict(mf=mf, su=su, u=u[:, 0].clone(), v=u[:, 1].clone(), w=u[:, 2].clone(), fr=fr, ff=ff, sc=sc)


def exact(case, seed):
    kind = case["kind"]
    with _mesh(case, seed) as mesh:
        m = _connectivity(mesh, internal=kind not in ("dropin", "host_step"))
        if kind == "boundaries":
            return _exact_boundaries(m, _boundary_fields(case, seed, _boundary_faces(mesh, case)),
                                     _regions(case, seed))
    if kind == "dropin":
        return _exact_dropin(case, m, _host_fields(case, seed), _regions(case, seed))
    if kind == "host_step":
        return _exact_host_step(case, m, _host_fields(case, seed))
    if kind == "momentum":
        return _exact_momentum(case, m, *_momentum_fields(case, seed), _regions(case, seed))
    return _exact_loops(case, m, _fields(case, seed))
