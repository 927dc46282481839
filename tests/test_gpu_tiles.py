"""The L2-prefetch tile kernels against the plain ones.

Every variant runs the same per-cell arithmetic in the same face order, so
results must be bit-identical:
  - the L2-prefetch kernels (the default when the user arrays start on
    16-byte boundaries) against the plain kernels, which the same call runs
    when phi, gface and the gradient are passed as views offset by one float;
  - the two-launch forward+adjoint (forward with the mass-flux adjoint, then
    the gradient adjoint) against dev_forward + dev_adjoint.
The device timers name the kernels each call ran, so every test checks that
the variant it means to test is the one that ran.

Cases: the Morton, owner and RCM numberings (the native one keeps the
reference's face order, which is not by owner, and has no tile ranges), a
ragged last tile, an odd cell count (the adjoint's gradient blocks are then
not 16-byte aligned, so only the forward takes the tile path), a jittered
mesh.
"""
import os

import pytest

pytestmark = pytest.mark.gpu


def _fields(torch, mesh, seed):
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    nC, nF, nB = mesh.nCells, mesh.nFaces, mesh.nBoundaries
    phi = (torch.rand(nC, generator=g, device=dev, dtype=torch.float64) * 2 - 1).float()
    phiB = (torch.rand(max(nB, 1), generator=g, device=dev, dtype=torch.float64) * 2 - 1).float()
    st = torch.randn(nC, 4, generator=g, device=dev, dtype=torch.float64).float()
    st[:, 0] = 0.9 + 0.2 * torch.rand(nC, generator=g, device=dev, dtype=torch.float64).float()
    gface = torch.randn(nF, generator=g, device=dev, dtype=torch.float64).float()
    return phi, phiB, st.contiguous(), gface


def _offset_copy(torch, t):
    """Same values in a buffer that starts 4 bytes past a 16-byte boundary."""
    buf = torch.empty(t.numel() + 4, dtype=t.dtype, device=t.device)
    v = buf[1:1 + t.numel()].view(t.shape)
    v.copy_(t)
    assert v.data_ptr() % 16 == 4
    return v


def _run(cg, torch, mesh, phi, phiB, st, gface, offset):
    dev = torch.device("cuda:0")
    nC, nF, nB = mesh.nCells, mesh.nFaces, mesh.nBoundaries
    if offset:
        phi, gface = _offset_copy(torch, phi), _offset_copy(torch, gface)
        grad = _offset_copy(torch, torch.full((3, nC), float("nan"), device=dev))
    else:
        grad = torch.full((3, nC), float("nan"), device=dev)
    mf = torch.full((nF,), -7.0, device=dev)
    loss = torch.full((1,), float("nan"), dtype=torch.float64, device=dev)
    pb = torch.full((nC,), float("nan"), device=dev)
    pbb = torch.full((max(nB, 1),), float("nan"), device=dev)
    sb = torch.full((nC, 4), float("nan"), device=dev)
    s = torch.cuda.current_stream()
    cg.timing_read()
    cg.timing_enable(True)
    try:
        cg.dev_forward(mesh, cg.PREC_F32C, phi, phiB, st, grad, mf, gface=gface, loss=loss, stream=s)
        cg.dev_adjoint(mesh, cg.PREC_F32C, grad, st, gface, pb, pbb, sb, stream=s)
        ran = set(cg.timing_read())
    finally:
        cg.timing_enable(False)
    mesh.check_status()
    torch.cuda.synchronize()
    _run.kernels = ran
    return [grad.clone(), mf, loss, pb, pbb, sb]


def _assert_same(a, b):
    import torch
    names = ["grad", "massFlux", "loss", "phiBar", "phiBBar", "stateBar"]
    for n, x, y in zip(names, a, b):
        assert torch.equal(x, y), n
        assert torch.isfinite(x).all(), n


CASES = [
    ("structgen", (12, 10, 8), "ORDER_OWNER"),     # 960 cells: ragged last tile
    ("structgen", (33, 17, 9), "ORDER_MORTON"),    # 5049 cells: odd count
    ("structgen", (40, 32, 24), "ORDER_RCM"),
    ("structgen", (64, 64, 64), "ORDER_OWNER"),    # whole tiles only
    ("jittered", (20, 18, 16), "ORDER_OWNER"),
]


def _mesh(cg, kind, dims, order):
    make = cg.Mesh.structgen if kind == "structgen" else cg.Mesh.jittered
    return make(*dims, order=getattr(cg, order))


@pytest.mark.parametrize("kind,dims,order", CASES)
def test_prefetch_equals_plain(cg, gpu, kind, dims, order):
    import torch
    mesh = _mesh(cg, kind, dims, order)
    fields = _fields(torch, mesh, 5)
    a = _run(cg, torch, mesh, *fields, offset=False)
    ka = _run.kernels
    b = _run(cg, torch, mesh, *fields, offset=True)
    assert "k_fwd_f32_pf" in ka and "k_fwd_f32" in _run.kernels
    if mesh.nCells % 4 == 0:
        assert "k_adj_f32_pf" in ka
    _assert_same(a, b)


def test_native_numbering_runs_plain_kernels(cg, gpu):
    """ORDER_NATIVE keeps the reference's face numbering, which is not sorted
    by owner, so there are no tile ranges and the mesh runs the plain
    kernels."""
    import torch
    mesh = cg.Mesh.structgen(16, 12, 8, order=cg.ORDER_NATIVE)
    assert not mesh.tiles
    _run(cg, torch, mesh, *_fields(torch, mesh, 1), offset=False)
    assert _run.kernels == {"k_fwd_f32", "k_reduce_partials", "k_adj_f32"}


def test_tile_path_can_be_disabled(cg, gpu, monkeypatch):
    import torch
    monkeypatch.setenv("CUPCFD_TILE_MODE", "0")
    off = cg.Mesh.structgen(16, 16, 16, order=cg.ORDER_OWNER)
    monkeypatch.delenv("CUPCFD_TILE_MODE")
    on = cg.Mesh.structgen(16, 16, 16, order=cg.ORDER_OWNER)
    assert not off.tiles and on.tiles
    fields = _fields(torch, on, 3)
    a = _run(cg, torch, off, *fields, offset=False)
    assert _run.kernels == {"k_fwd_f32", "k_reduce_partials", "k_adj_f32"}
    _assert_same(a, _run(cg, torch, on, *fields, offset=False))
    assert "k_fwd_f32_pf" in _run.kernels


def test_misaligned_state_is_rejected(cg, gpu):
    """float4 state records must start on 16-byte boundaries; a misaligned
    pointer is refused before anything is launched."""
    import torch
    mesh = cg.Mesh.structgen(8, 8, 8, order=cg.ORDER_OWNER)
    phi, phiB, st, gface = _fields(torch, mesh, 1)
    bad = _offset_copy(torch, st)
    grad = torch.zeros(3, mesh.nCells, device="cuda:0")
    mf = torch.zeros(mesh.nFaces, device="cuda:0")
    before = cg.launch_count()
    rc = cg.lib().cupcfd_gpu_dev_forward(mesh.h, cg.PREC_F32C, cg._p(phi), cg._p(phiB), cg._p(bad), None,
                                         cg._p(grad), cg._p(mf), None, None)
    assert rc == cg.E_CONFIG_INVALID_VALUE
    assert "16-byte" in cg.last_error()
    assert cg.launch_count() == before


def _run_pipeline(cg, torch, mesh, phi, phiB, st, gface, offset):
    """dev_forward_adjoint; offset views of phi/gface/grad force the plain kernels."""
    dev = torch.device("cuda:0")
    nC, nF, nB = mesh.nCells, mesh.nFaces, mesh.nBoundaries
    if offset:
        phi, gface = _offset_copy(torch, phi), _offset_copy(torch, gface)
        grad = _offset_copy(torch, torch.full((3, nC), float("nan"), device=dev))
    else:
        grad = torch.full((3, nC), float("nan"), device=dev)
    mf = torch.full((nF,), -7.0, device=dev)
    loss = torch.full((1,), float("nan"), dtype=torch.float64, device=dev)
    pb = torch.full((nC,), float("nan"), device=dev)
    pbb = torch.full((max(nB, 1),), float("nan"), device=dev)
    sb = torch.full((nC, 4), float("nan"), device=dev)
    s = torch.cuda.current_stream()
    cg.dev_forward_adjoint(mesh, cg.PREC_F32C, phi, phiB, st, gface, grad, mf, pb, pbb, sb, loss, stream=s)
    mesh.check_status()
    torch.cuda.synchronize()
    return [grad.clone(), mf, loss, pb, pbb, sb]


@pytest.mark.parametrize("kind,dims,order", CASES)
def test_forward_adjoint_pipeline_equals_separate_calls(cg, gpu, kind, dims, order):
    """The two-launch forward+adjoint (mass-flux adjoint moved into the
    forward) equals dev_forward followed by dev_adjoint, bit for bit, and
    so does the same call on offset pointers (plain kernels)."""
    import torch
    make = cg.Mesh.structgen if kind == "structgen" else cg.Mesh.jittered
    mesh = make(*dims, order=getattr(cg, order))
    fields = _fields(torch, mesh, 7)
    ref = _run(cg, torch, mesh, *fields, offset=False)
    _assert_same(_run_pipeline(cg, torch, mesh, *fields, offset=False), ref)
    _assert_same(_run_pipeline(cg, torch, mesh, *fields, offset=True), ref)


@pytest.mark.parametrize("kind,dims,order", [("structgen", (40, 32, 24), "ORDER_RCM"),
                                             ("structgen", (33, 17, 9), "ORDER_MORTON"),
                                             ("jittered", (20, 18, 16), "ORDER_OWNER")])
def test_six_incidence_kernels_equal_general_kernels(cg, gpu, kind, dims, order, monkeypatch):
    """On hexahedral meshes the L2-prefetch kernels run a specialisation for
    cells of exactly six incidences (compile-time trip count, no padding
    checks): the same arithmetic in the same order, so the forward+adjoint
    pipeline, the separate FP32 calls and the FP64 forward give the same bits
    as the general kernels (CUPCFD_FULL_WIDTH=0 at mesh creation)."""
    import torch
    monkeypatch.setenv("CUPCFD_FULL_WIDTH", "0")
    general = _mesh(cg, kind, dims, order)
    monkeypatch.delenv("CUPCFD_FULL_WIDTH")
    six = _mesh(cg, kind, dims, order)
    assert six.tiles and general.tiles and six.full_width == 6 and general.full_width == 0
    fields = _fields(torch, six, 13)
    _assert_same(_run_pipeline(cg, torch, six, *fields, offset=False),
                 _run_pipeline(cg, torch, general, *fields, offset=False))
    _assert_same(_run(cg, torch, six, *fields, offset=False), _run(cg, torch, general, *fields, offset=False))
    phi = fields[0].double()
    phiB = fields[1].double()
    st = fields[2].double().t().contiguous()
    gface = fields[3].double()
    outs = []
    for mesh in (six, general):
        grad = torch.full((3, mesh.nCells), float("nan"), dtype=torch.float64, device="cuda:0")
        mf = torch.zeros(mesh.nFaces, dtype=torch.float64, device="cuda:0")
        loss = torch.zeros(1, dtype=torch.float64, device="cuda:0")
        cg.dev_forward(mesh, cg.PREC_F64, phi, phiB, st, grad, mf, gface=gface, loss=loss,
                       stream=torch.cuda.current_stream())
        mesh.check_status()
        torch.cuda.synchronize()
        outs.append((grad, mf, loss))
    for x, y in zip(*outs):
        assert torch.equal(x, y)


def test_polyhedral_mesh_runs_general_kernels(cg, gpu):
    """Cells of other face counts keep the general kernels."""
    import oracle as O
    m = O.merge_cells(O.jitter(9, 8, 7, 0.25, seed=5, permute=True), 0.4, 11, max_cells=6)
    mesh = cg.Mesh.from_arrays(m, order=cg.ORDER_OWNER)
    assert mesh.tiles and mesh.full_width == 0


def test_device_timers_name_the_pipeline_kernels(cg, gpu):
    """cupcfd_gpu_timing_*: the forward+adjoint call's three launches, each
    timed on its stream, counted per kernel, and cleared by the read."""
    import torch
    mesh = cg.Mesh.structgen(32, 32, 32, order=cg.ORDER_OWNER)
    fields = _fields(torch, mesh, 2)
    cg.timing_read()
    cg.timing_enable(True)
    try:
        for _ in range(3):
            _run_pipeline(cg, torch, mesh, *fields, offset=False)
        t = cg.timing_read()
    finally:
        cg.timing_enable(False)
    assert {k: v[0] for k, v in t.items()} == {"k_fwd_madj_f32_pf": 3, "k_reduce_partials": 3, "k_gadj_f32_pf": 3}
    assert all(v[1] > 0 for v in t.values())
    assert cg.timing_read() == {}


def test_fp64_forward_prefetch_equals_plain(cg, gpu):
    """The FP64 forward and adjoint with the L2 prefetch (16-byte-aligned
    arrays) and the plain ones (phi and the gradient offset by one double)
    give bit-identical results."""
    import torch
    mesh = cg.Mesh.structgen(24, 20, 18, order=cg.ORDER_OWNER)
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev)
    g.manual_seed(4)
    nC, nF, nB = mesh.nCells, mesh.nFaces, mesh.nBoundaries
    phi = torch.rand(nC, generator=g, device=dev, dtype=torch.float64) * 2 - 1
    phiB = torch.rand(nB, generator=g, device=dev, dtype=torch.float64) * 2 - 1
    st = torch.randn(4, nC, generator=g, device=dev, dtype=torch.float64)
    gface = torch.randn(nF, generator=g, device=dev, dtype=torch.float64)
    buf = torch.empty(nC + 2, dtype=torch.float64, device=dev)
    phi_off = buf[1:1 + nC]
    phi_off.copy_(phi)
    assert phi_off.data_ptr() % 16 == 8
    gbuf = torch.empty(3 * nC + 2, dtype=torch.float64, device=dev)
    out = []
    for p, gr in ((phi, torch.empty(3, nC, dtype=torch.float64, device=dev)), (phi_off, gbuf[1:1 + 3 * nC].view(3, nC))):
        gr.fill_(float("nan"))
        mf = torch.zeros(nF, dtype=torch.float64, device=dev)
        loss = torch.zeros(1, dtype=torch.float64, device=dev)
        pb = torch.empty(nC, dtype=torch.float64, device=dev)
        pbb = torch.empty(nB, dtype=torch.float64, device=dev)
        sb = torch.empty(4, nC, dtype=torch.float64, device=dev)
        cg.timing_enable(True)
        try:
            s = torch.cuda.current_stream()
            cg.dev_forward(mesh, cg.PREC_F64, p, phiB, st, gr, mf, gface=gface, loss=loss, stream=s)
            cg.dev_adjoint(mesh, cg.PREC_F64, gr, st, gface, pb, pbb, sb, stream=s)
            names = set(cg.timing_read())
        finally:
            cg.timing_enable(False)
        out.append((gr.clone(), mf, loss, pb, pbb, sb, names))
    assert {"k_fwd_f64_pf", "k_adj_f64_pf"} <= out[0][-1] and {"k_fwd_f64", "k_adj_f64"} <= out[1][-1]
    for a, b in zip(out[0][:-1], out[1][:-1]):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dims", [(32, 6, 5),     # one slice per row: low and high x boundary in every slice
                                  (64, 8, 6),     # slices at one end of a row, interior rows
                                  (33, 12, 7),    # rows break inside slices, odd cell count, ragged last slice
                                  (100, 7, 8),    # several breaks per slice
                                  (257, 3, 4)])   # one cell past a tile
def test_run_form_equals_lists(cg, gpu, dims, monkeypatch):
    """Rows of cells numbered one after the other store their incidence lists
    in run form (one entry set per stretch of lanes); the kernels that read it
    give the bits of those that read the full lists (CUPCFD_RUNS=0 at mesh
    creation), FP32 and FP64."""
    import torch
    monkeypatch.setenv("CUPCFD_RUNS", "0")
    lists = cg.Mesh.structgen(*dims, order=cg.ORDER_OWNER)
    monkeypatch.delenv("CUPCFD_RUNS")
    runs = cg.Mesh.structgen(*dims, order=cg.ORDER_OWNER)
    assert lists.full_width == 6 and runs.full_width == 6
    assert runs.deviceBytes > lists.deviceBytes, "the run form was not built"
    fields = _fields(torch, runs, 17)
    _assert_same(_run_pipeline(cg, torch, runs, *fields, offset=False),
                 _run_pipeline(cg, torch, lists, *fields, offset=False))
    _assert_same(_run(cg, torch, runs, *fields, offset=False), _run(cg, torch, lists, *fields, offset=False))
    phi, phiB, st, gface = (t.double() for t in fields)
    st = st.t().contiguous()
    outs = []
    for mesh in (runs, lists):
        e = lambda *n: torch.full(n, float("nan"), dtype=torch.float64, device="cuda:0")
        o = [e(3, mesh.nCells), torch.zeros_like(gface), e(1), e(mesh.nCells), e(mesh.nBoundaries), e(4, mesh.nCells)]
        s = torch.cuda.current_stream()
        cg.dev_forward(mesh, cg.PREC_F64, phi, phiB, st, o[0], o[1], gface=gface, loss=o[2], stream=s)
        cg.dev_adjoint(mesh, cg.PREC_F64, o[0], st, gface, o[3], o[4], o[5], stream=s)
        mesh.check_status()
        torch.cuda.synchronize()
        outs.append(o)
    _assert_same(*outs)


def test_irregular_numbering_has_no_run_form(cg, gpu, monkeypatch):
    """A permuted mesh has no stretches worth storing and keeps the lists."""
    monkeypatch.setenv("CUPCFD_RUNS", "0")
    lists = cg.Mesh.jittered(20, 18, 16, order=cg.ORDER_OWNER)
    monkeypatch.delenv("CUPCFD_RUNS")
    assert cg.Mesh.jittered(20, 18, 16, order=cg.ORDER_OWNER).deviceBytes == lists.deviceBytes


@pytest.mark.parametrize("kind,dims,order", [("structgen", (33, 17, 9), "ORDER_OWNER"),     # 5,049 cells: 1 past a multiple of 4
                                             ("structgen", (37, 7, 10), "ORDER_MORTON"),    # 2,590: 2 past
                                             ("jittered", (15, 13, 11), "ORDER_RCM"),       # 2,145: 1 past
                                             ("structgen", (5, 5, 11), "ORDER_OWNER")])     # 275: 3 past, one whole tile
def test_any_cell_count_takes_the_prefetch_kernels(cg, gpu, kind, dims, order):
    """Component blocks of a cell count that is no multiple of four start off
    16-byte boundaries; the L2-prefetch kernels run all the same, with the
    plain kernels' bits, and the pipeline as two launches."""
    import torch
    mesh = _mesh(cg, kind, dims, order)
    assert mesh.nCells % 4
    fields = _fields(torch, mesh, 23)
    a = _run(cg, torch, mesh, *fields, offset=False)
    assert {"k_fwd_f32_pf", "k_adj_f32_pf"} <= _run.kernels
    b = _run(cg, torch, mesh, *fields, offset=True)
    assert {"k_fwd_f32", "k_adj_f32"} <= _run.kernels
    _assert_same(a, b)
    cg.timing_read()
    cg.timing_enable(True)
    try:
        _assert_same(_run_pipeline(cg, torch, mesh, *fields, offset=False), b)
        assert {"k_fwd_madj_f32_pf", "k_gadj_f32_pf"} <= set(cg.timing_read())
    finally:
        cg.timing_enable(False)


@pytest.mark.parametrize("kind,dims,order", CASES + [("structgen", (33, 12, 7), "ORDER_OWNER"), ("poly", (9, 8, 7), "ORDER_OWNER")])
@pytest.mark.parametrize("prec", ["PREC_F64", "PREC_F32C"])
def test_gradient_and_general_adjoints_prefetch_equals_plain(cg, gpu, kind, dims, order, prec):
    """dev_gradient (one to three iterations), dev_gradient_adjoint and
    dev_mass_plain_adjoint on arrays at 16-byte boundaries (L2-prefetch
    kernels) and off them (plain kernels): the same bits."""
    import torch
    if kind == "poly":
        import oracle as O
        mesh = cg.Mesh.from_arrays(O.merge_cells(O.jitter(*dims, 0.25, seed=5, permute=True), 0.4, 11, max_cells=6),
                                   order=getattr(cg, order))
    else:
        mesh = _mesh(cg, kind, dims, order)
    p = getattr(cg, prec)
    f64 = p == cg.PREC_F64
    t = torch.float64 if f64 else torch.float32
    nC, nF, nB = mesh.nCells, mesh.nFaces, mesh.nBoundaries
    phi, phiB, st, gface = (x.to(t) for x in _fields(torch, mesh, 29))
    st = st.t().contiguous() if f64 else st
    gbar = torch.randn(3, nC, generator=torch.Generator(device="cuda").manual_seed(3), device="cuda", dtype=t)

    def off(x):   # one element past a 16-byte boundary
        buf = torch.empty(x.numel() + 4, dtype=x.dtype, device=x.device)
        v = buf[1:1 + x.numel()].view(x.shape)
        v.copy_(x)
        return v

    e = lambda *n: torch.full(n, float("nan"), dtype=t, device="cuda")  # noqa: E731
    s = torch.cuda.current_stream()
    outs = []
    for at in (lambda x: x, off):
        o = []
        for n in (1, 2, 3):
            g, go = e(3, nC), e(3, nC)
            cg.dev_gradient(mesh, p, at(phi), phiB, g, go, nGradient=n, stream=s)
            assert torch.equal(g, go)
            o.append(g)
        pb, pbb, sb = e(nC), e(nB), torch.full_like(st, float("nan"))
        cg.dev_gradient_adjoint(mesh, p, at(gbar), pb, pbb, stream=s)
        cg.dev_mass_plain_adjoint(mesh, p, st, at(gface), sb, stream=s)
        mesh.check_status()
        torch.cuda.synchronize()
        outs.append(o + [pb, pbb, sb])
    for a, b in zip(*outs):
        assert torch.isfinite(a).all() and torch.equal(a, b)


@pytest.mark.parametrize("dims", [(128, 128, 64),    # 4,096 tiles: the last summed by one pass
                                  (129, 128, 64)])   # 4,128: folded by many blocks first
def test_forward_loss_is_the_pipelines(cg, gpu, dims):
    """The forward's loss adds the tiles' partials in one order whether one
    pass or two take them: the bits of the forward+adjoint call's loss, which
    takes one at every size."""
    import torch
    mesh = cg.Mesh.structgen(*dims, order=cg.ORDER_OWNER)
    fields = _fields(torch, mesh, 31)
    _assert_same(_run(cg, torch, mesh, *fields, offset=False), _run_pipeline(cg, torch, mesh, *fields, offset=False))


@pytest.mark.parametrize("kind,dims,order", [("structgen", (20, 18, 17), "ORDER_MORTON"),   # gathers from few lines
                                             ("jittered", (20, 18, 17), "ORDER_MORTON"),    # from many: values in flight
                                             ("jittered", (45, 45, 45), "ORDER_RCM"),       # 356 tiles: one wave of four an SM
                                             ("jittered", (56, 54, 53), "ORDER_MORTON"),    # 627: more
                                             ("poly", (20, 18, 17), "ORDER_MORTON"),
                                             ("poly", (62, 60, 61), "ORDER_MORTON")])       # over 296 tiles
def test_fp64_adjoint_forms_equal_the_plain_kernel(cg, gpu, kind, dims, order):
    """Each form of the FP64 adjoint's L2-prefetch kernel, as the mesh's lists
    and size choose it, with the plain kernel's bits."""
    import torch
    if kind == "poly":
        import oracle as O
        mesh = cg.Mesh.from_arrays(O.merge_cells(O.jitter(*dims, 0.25, seed=5, permute=True), 0.3, 11, max_cells=6),
                                   order=getattr(cg, order))
        assert mesh.full_width == 0
    else:
        mesh = _mesh(cg, kind, dims, order)
    nC, nB = mesh.nCells, mesh.nBoundaries
    st, gface = (x.double() for x in _fields(torch, mesh, 37)[2:])
    st = st.t().contiguous()
    grad = torch.randn(3 * nC + 1, generator=torch.Generator(device="cuda").manual_seed(4), device="cuda", dtype=torch.float64)
    outs = []
    for name, g in (("k_adj_f64_pf", grad[:-1].clone()), ("k_adj_f64", grad[1:])):
        if name == "k_adj_f64":
            g.copy_(grad[:-1].clone())   # the same values, 8 bytes past a 16-byte boundary
        o = [torch.full(n, float("nan"), dtype=torch.float64, device="cuda") for n in ((nC,), (nB,), (4, nC))]
        cg.timing_read()
        cg.timing_enable(True)
        try:
            cg.dev_adjoint(mesh, cg.PREC_F64, g, st, gface, *o, stream=torch.cuda.current_stream())
            assert set(cg.timing_read()) == {name}
        finally:
            cg.timing_enable(False)
        outs.append(o)
    for a, b in zip(*outs):
        assert torch.isfinite(a).all() and torch.equal(a, b)


def test_fp64_gradient_forms_on_mixed_cells(cg, gpu):
    """536 tiles of merged hexahedra take the gradient form with more warps
    (smaller meshes take the other, tests above): the plain kernel's bits."""
    import oracle as O
    import torch
    mesh = cg.Mesh.from_arrays(O.merge_cells(O.jitter(72, 72, 72, 0.25, seed=5, permute=True), 0.3, 11, max_cells=6),
                               order=cg.ORDER_MORTON)
    assert mesh.full_width == 0 and 444 * 256 < mesh.nCells <= 592 * 256
    phi, phiB = (x.double() for x in _fields(torch, mesh, 41)[:2])
    off = torch.empty(mesh.nCells + 1, dtype=torch.float64, device="cuda")[1:]
    off.copy_(phi)
    out = [torch.full((3, mesh.nCells), float("nan"), dtype=torch.float64, device="cuda") for _ in range(2)]
    for p, g in zip((phi, off), out):
        cg.dev_gradient(mesh, cg.PREC_F64, p, phiB, g, stream=torch.cuda.current_stream())
    torch.cuda.synchronize()
    assert torch.isfinite(out[0]).all() and torch.equal(*out)


@pytest.mark.parametrize("order,prefetch", [("ORDER_OWNER", False), ("ORDER_RCM", True)])
def test_random_numbering_takes_the_plain_kernels(cg, gpu, order, prefetch):
    """A permuted mesh of over 2^17 cells: kernels that gather more than the
    L2 prefetch saves run without it where the cells are numbered at random,
    and with it in an order that keeps neighbours together."""
    import torch
    mesh = cg.Mesh.jittered(53, 51, 50, order=getattr(cg, order))
    assert mesh.nCells > 1 << 17
    phi, phiB, st, gface = _fields(torch, mesh, 43)
    _run(cg, torch, mesh, phi, phiB, st, gface, offset=False)
    assert ("k_adj_f32_pf" in _run.kernels) == prefetch and ("k_adj_f32" in _run.kernels) != prefetch
    cg.timing_read()
    cg.timing_enable(True)
    try:
        e = lambda *n: torch.zeros(n, dtype=torch.float64, device="cuda")  # noqa: E731
        cg.dev_forward(mesh, cg.PREC_F64, phi.double(), phiB.double(), st.double().t().contiguous(), e(3, mesh.nCells),
                       e(mesh.nFaces), gface=gface.double(), loss=e(1), stream=torch.cuda.current_stream())
        ran = set(cg.timing_read())
    finally:
        cg.timing_enable(False)
    assert ("k_fwd_f64_pf" in ran) == prefetch and ("k_fwd_f64" in ran) != prefetch
