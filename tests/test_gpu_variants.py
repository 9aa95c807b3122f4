"""Kernel variants at the sizes where their splits can go wrong (tile edges, lane
remainders, the smallest and largest supports), against the complex128 oracle."""

import numpy
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    import torch
    from crocodile_gb300 import _lib, engine, synthesis
    from oracle import crocodile_oracle
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    return torch, _lib, engine, synthesis, crocodile_oracle


def _case(seed, n, S, Q, sep, G=1, rmax=0.3):
    rng = numpy.random.default_rng(seed)
    uvw = numpy.column_stack([rng.uniform(-rmax, rmax, n), rng.uniform(-rmax, rmax, n),
                              numpy.zeros(n)])
    shape = (G, Q, S) if sep else (G, Q, Q, S, S)
    gcf = rng.normal(size=shape) + 1j * rng.normal(size=shape)
    src = rng.integers(0, G, n)[:, None]
    return rng, uvw, gcf, src


@pytest.mark.parametrize("sep", [True, False])
@pytest.mark.parametrize("S,n", [(1, 1), (2, 33), (7, 5), (8, 100), (9, 257), (16, 31), (32, 3)])
def test_plain_fp64_degrid(env, S, n, sep):
    """Eight threads per visibility: supports below, at and above eight, a last block
    with idle threads.  Tolerance: S^2 products of unit-variance terms, each with a few
    roundings of 2^-53, against a sum that random signs leave S times smaller than its
    terms' total."""
    _, _, E, S_, O = env
    rng, uvw, gcf, src = _case(S + n, n, S, 4, sep, G=3)
    N = 96
    a = rng.normal(size=(N, N)) + 1j * rng.normal(size=(N, N))
    got = S_.convdegrid(gcf, a, uvw[:, :2], src, precision="fp64")
    want = O.convdegrid(gcf, a, uvw[:, :2], src)
    tol = 4 * (S * S + 8) * S * 2.0 ** -53
    assert numpy.abs(got - want).max() <= tol * max(numpy.abs(want).max(), 1.0)


@pytest.mark.parametrize("H,W,h,w,oh,ow", [(64, 64, 64, 64, 1, 1), (64, 128, 5, 37, 7, 9),
                                           (512, 64, 384, 33, 384, 64), (128, 512, 1, 512, 128, 31),
                                           (2048, 64, 2047, 2, 3, 64), (256, 256, 256, 256, 256, 255)])
@pytest.mark.parametrize("inverse", [False, True])
def test_fft_df_window(env, H, W, h, w, oh, ow, inverse):
    """Blocks of odd sizes and places in padded planes, three planes (an odd number of
    rows in pairs), read through strides; tolerance as for whole planes: 5e-14 of the
    peak (about 2^-44 per stage of double-float rounding)."""
    torch, _, E, S, O = env
    rng = numpy.random.default_rng(H + w)
    big = rng.normal(size=(3, h + 2, w + 3)) + 1j * rng.normal(size=(3, h + 2, w + 3))
    src = torch.from_numpy(big).cuda()[:, 1:h + 1, 2:w + 2]
    out = torch.full((3, H, W), 7.0, dtype=torch.complex128, device="cuda")
    E.fft_df_window(out, inverse, src, (oh, ow))
    r, c = H // 2 - h // 2, W // 2 - w // 2
    R, C = H // 2 - oh // 2, W // 2 - ow // 2
    for p in range(3):
        full = numpy.zeros((H, W), dtype=complex)
        full[r:r + h, c:c + w] = big[p, 1:h + 1, 2:w + 2]
        want = (O.ifft if inverse else O.fft)(full)
        got = out[p].cpu().numpy()[R:R + oh, C:C + ow]
        assert numpy.abs(got - want[R:R + oh, C:C + ow]).max() <= 5e-14 * numpy.abs(want).max()


def _grids(torch, rng, N, layers=1):
    g = rng.normal(size=(layers, N, N)) + 1j * rng.normal(size=(layers, N, N))
    return g.astype(numpy.complex64)


@pytest.mark.parametrize("sep", [True, False])
@pytest.mark.parametrize("S", list(range(1, 18)))
def test_degrid_direct_bits(env, S, sep):
    """The direct degridder adds in the tiled degridder's order: equal bits for every
    support (17: both tiled), visibility counts that leave lanes and batches partly
    filled, and stacked grids."""
    torch, L, E, _, _ = env
    from crocodile_gb300 import autotune
    for n, layers in ((1, 1), (37, 1), (1000, 3)):
        rng, uvw, gcf, src = _case(S, n, S, 4, sep, G=3)
        N = 80
        kt = E.KernelTable.from_gcf(gcf, 1, E.CF)
        lay = rng.integers(0, layers, n).astype(numpy.int32)
        plan = E.Plan(uvw, 1.0, (N, N), kt, src[:, 0].astype(numpy.int32),
                      layers=None if layers == 1 else (layers, lay))
        g = torch.from_numpy(_grids(torch, rng, N, layers)).cuda()
        got = {}
        for dvis in (0, 2, 4):
            autotune.set_tuning(dvis=dvis)
            try:
                got[dvis] = plan.degrid(kt, g)
            finally:
                autotune.set_tuning()
        plan.check()
        assert torch.equal(torch.view_as_real(got[0]), torch.view_as_real(got[2]))
        assert torch.equal(torch.view_as_real(got[4]), torch.view_as_real(got[2]))


@pytest.mark.parametrize("sep", [True, False])
@pytest.mark.parametrize("S", [1, 2, 4, 5, 8, 9, 11, 12, 16, 17])
def test_grid_direct(env, S, sep):
    """The direct gridder (cg_grid_sparse) over stacked grids and one grid against the
    oracle.  Tolerance 2e-6: complex64 products (2^-24 each) summed over at most a few
    hundred visibilities per cell."""
    torch, L, E, _, O = env
    for n, layers in ((3, 1), (500, 1), (700, 3)):
        rng, uvw, gcf, src = _case(S + n, n, S, 4, sep, G=3)
        N = 80
        kt = E.KernelTable.from_gcf(gcf, 1, E.CF)
        vis = rng.normal(size=n) + 1j * rng.normal(size=n)
        lay = rng.integers(0, layers, n).astype(numpy.int32)
        plan = E.Plan(uvw, 1.0, (N, N), kt, src[:, 0].astype(numpy.int32),
                      layers=None if layers == 1 else (layers, lay))
        g = torch.zeros((layers, N, N), dtype=E.CF, device="cuda")
        plan.grid_sparse(kt, E.cuda_tensor(vis, E.CF), g)
        model = E.cuda_tensor(_grids(torch, rng, N, layers), E.CF)  # and the fused pass by it
        res = torch.zeros_like(g)
        d = plan.degrid_grid(kt, model, E.cuda_tensor(vis, E.CF), res, residual=True)
        ref = plan.grid_sparse(kt, E.cuda_tensor(vis, E.CF) - d, torch.zeros_like(g))
        assert torch.equal(d, plan.degrid(kt, model))
        assert torch.linalg.norm(res - ref) <= 2e-6 * torch.linalg.norm(ref)
        plan.check()
        want = numpy.zeros((layers, N, N), dtype=complex)
        for p in range(layers):
            s = lay == p
            if s.any():
                O.convgrid(gcf, want[p], uvw[s, :2], src[s], vis[s])
        assert numpy.linalg.norm(g.cpu().numpy() - want) <= 2e-6 * numpy.linalg.norm(want)


@pytest.mark.parametrize("S", [1, 4, 5, 6, 7, 8, 9, 10, 13, 14, 16])
@pytest.mark.parametrize("N,per", [(64, 3.5), (81, 2.5), (100, 2.5), (450, 0.2)])
def test_grid_separable_dense(env, N, per, S):
    """Separable tables on dense visibilities (the register-window gridder): every
    window and tile edge, grids that end inside a tile, footprints that touch the
    grid's edges, items cut in short batches, weights, and the fused pass, against the
    oracle.  Tolerance 3e-6: a few hundred complex64 products summed per cell."""
    torch, L, E, _, O = env
    n = int(per * N * N)
    rng, uvw, gcf, src = _case(S + N, n, S, 4, True, G=2, rmax=0.5 - (S // 2 + 1) / N)
    x = O.frac_coords((N, N), 4, uvw[:, :2])
    ok = ((x[0] - S // 2 >= 0) & (x[0] - S // 2 + S <= N) & (x[2] - S // 2 >= 0) &
          (x[2] - S // 2 + S <= N))
    uvw, src = uvw[ok], src[ok]
    n = len(uvw)
    vis = (rng.normal(size=n) + 1j * rng.normal(size=n)).astype(numpy.complex64)
    wt = rng.uniform(0.5, 2, n).astype(numpy.float32)
    kt = E.KernelTable.from_gcf(gcf, 1, E.CF)
    plan = E.Plan(uvw, 1.0, (N, N), kt, src[:, 0].astype(numpy.int32))
    if per > 1 or S > 4:
        assert plan.info()["tile"] == (12 if per < 1 and (S == 5 or 10 <= S <= 13) else 8)
    v, w = E.cuda_tensor(vis, E.CF), E.cuda_tensor(wt, torch.float32)
    for got, val in ((plan.grid(kt, v, torch.zeros((N, N), dtype=E.CF, device="cuda")), vis),
                     (plan.grid_weighted(kt, v, w, torch.zeros((N, N), dtype=E.CF,
                                                               device="cuda")), vis * wt),
                     (plan.grid_weighted(kt, None, w, torch.zeros((N, N), dtype=E.CF,
                                                                  device="cuda")), wt)):
        want = numpy.zeros((N, N), dtype=complex)
        O.convgrid(gcf, want, uvw[:, :2], src, val)
        assert numpy.linalg.norm(got.cpu().numpy() - want) <= 3e-6 * numpy.linalg.norm(want)
    model = E.cuda_tensor(_grids(torch, rng, N)[0], E.CF)
    out = torch.zeros((N, N), dtype=E.CF, device="cuda")
    d = plan.degrid_grid(kt, model, v, out, residual=True)
    place = v.clone()  # in place: one traversal
    out2 = torch.zeros((N, N), dtype=E.CF, device="cuda")
    plan.degrid_grid(kt, model, place, out2, residual=True, vis_out=place)
    plan.check()
    dw = O.convdegrid(gcf, model.cpu().numpy().astype(complex), uvw[:, :2], src)
    want = numpy.zeros((N, N), dtype=complex)
    O.convgrid(gcf, want, uvw[:, :2], src, vis - dw)
    for got, ref in ((d, dw), (place, dw), (out, want), (out2, want)):
        assert numpy.linalg.norm(got.cpu().numpy() - ref) <= 3e-6 * numpy.linalg.norm(ref)


@pytest.mark.parametrize("n", [1, 31, 257, 100000])
def test_uvw_ranges(env, n):
    """Extremes and w bins in one pass: equal to numpy's, bins half to even, negative
    and NaN coordinates."""
    torch, L, E, S, _ = env
    rng = numpy.random.default_rng(n)
    uvw = rng.normal(size=(n, 3)) * 10.0 ** rng.integers(-3, 5, (n, 1))
    uvw[: n // 2, 2] = 2.5 * rng.integers(-9, 9, n // 2) + 1.25  # halves of the bin width
    st = E.Status()
    k = numpy.round(uvw[:, 2] / 2.5)
    assert E.uvw_ranges(uvw, 2.5, st) == (k.min(), k.max(), (uvw[:, :2].min(), uvw[:, :2].max()))
    st.check()
    assert E.uvw_ranges(-numpy.abs(uvw), 0.0, st)[2] == (-numpy.abs(uvw[:, :2]).max(),
                                                         -numpy.abs(uvw[:, :2]).min())
    uvw[n - 1, 1] = numpy.nan
    assert E.uvw_ranges(uvw, 0.0, st)[2][0] == -numpy.inf
    uvw[n - 1, 2] = 1e12
    E.uvw_ranges(uvw, 2.5, st)
    with pytest.raises(AssertionError):
        st.check()
    with pytest.raises(ValueError):
        S.w_cache_imaging(0.1, 1000.0, uvw, None, numpy.zeros(n), wstep=0, NpixFF=32, NpixKern=7,
                          Qpx=4)


@pytest.mark.parametrize("S,G", [(13, 1), (15, 5)])
def test_pad_even(env, S, G):
    torch, L, E, _, _ = env
    t = torch.randn((G, 4, 4, S, S), dtype=E.CF, device="cuda")
    uvw = torch.zeros((1, 3), dtype=torch.float64, device="cuda")
    p = E.KernelTable(t.reshape(-1), False, 4, S).padded_even(uvw, 1.0, (128, 128))
    want = torch.nn.functional.pad(torch.view_as_real(t), (0, 0, 1, 0, 1, 0))
    assert p.S == S + 1
    assert torch.equal(torch.view_as_real(p.table).reshape(want.shape), want)


@pytest.mark.parametrize("S", [2, 4, 6, 8, 9, 10, 11, 12, 13, 14, 15, 16])
def test_grid_lane_loads(env, S):
    """4-D tables on dense visibilities (the lane kernel with taps by loads, odd
    supports on its tiles too), grids that end inside a tile and a stack, gridding and
    the fused pass against the oracle.  Tolerance 3e-6: a few hundred complex64
    products summed per cell."""
    torch, L, E, _, O = env
    for N, layers in ((81, 1), (48, 2)):
        n = 3 * N * N
        rng, uvw, gcf, src = _case(S + N, n, S, 2, False, G=2)
        vis = (rng.normal(size=n) + 1j * rng.normal(size=n)).astype(numpy.complex64)
        lay = rng.integers(0, layers, n).astype(numpy.int32)
        kt = E.KernelTable.from_gcf(gcf, 1, E.CF)
        plan = E.Plan(uvw, 1.0, (N, N), kt, src[:, 0].astype(numpy.int32),
                      layers=None if layers == 1 else (layers, lay))
        assert plan.info()["tile"] == 16
        v = E.cuda_tensor(vis, E.CF)
        got = plan.grid(kt, v, torch.zeros((layers, N, N), dtype=E.CF, device="cuda"))
        model = E.cuda_tensor(_grids(torch, rng, N, layers), E.CF)
        out = torch.zeros_like(got)
        d = plan.degrid_grid(kt, model, v, out, residual=True).cpu().numpy()
        plan.check()
        mh = model.cpu().numpy().astype(complex)
        for p in range(layers):
            s = lay == p
            dw = O.convdegrid(gcf, mh[p], uvw[s, :2], src[s])
            want, res = (numpy.zeros((N, N), dtype=complex) for _ in range(2))
            O.convgrid(gcf, want, uvw[s, :2], src[s], vis[s])
            O.convgrid(gcf, res, uvw[s, :2], src[s], vis[s] - dw)
            for a, b in ((got[p].cpu().numpy(), want), (d[s], dw), (out[p].cpu().numpy(), res)):
                assert numpy.linalg.norm(a - b) <= 3e-6 * numpy.linalg.norm(b)


@pytest.mark.parametrize("S", [1, 9, 16])
@pytest.mark.parametrize("bad", [complex("nan"), complex("inf")])
def test_grid_separable_not_finite(env, S, bad):
    """A visibility that is not finite: only its footprint's cells are lost, also where
    the gridder keeps its window in registers (dense visibilities); the others as
    ever, 3e-6 as for test_grid_separable_dense."""
    torch, L, E, _, O = env
    N, n = 96, 60000
    rng, uvw, gcf, src = _case(S, n, S, 2, True, G=2)
    vis = (rng.normal(size=n) + 1j * rng.normal(size=n)).astype(numpy.complex64)
    vis[777] = bad
    kt = E.KernelTable.from_gcf(gcf, 1, E.CF)
    plan = E.Plan(uvw, 1.0, (N, N), kt, src[:, 0].astype(numpy.int32))
    got = plan.grid(kt, E.cuda_tensor(vis, E.CF),
                    torch.zeros((N, N), dtype=E.CF, device="cuda")).cpu().numpy()
    plan.check()
    want = numpy.zeros((N, N), dtype=complex)
    with numpy.errstate(invalid="ignore"):
        O.convgrid(gcf, want, uvw[:, :2], src, vis)
    ok = numpy.isfinite(want)
    assert ok.sum() == N * N - S * S
    numpy.testing.assert_array_equal(numpy.isfinite(got), ok)
    assert numpy.linalg.norm(got[ok] - want[ok]) <= 3e-6 * numpy.linalg.norm(want[ok])


@pytest.mark.parametrize("layers,n", [(1, 1), (1, 500), (4, 3), (4, 500)])
def test_plain_fp64_stack(env, layers, n):
    """The plain form's launches, one to each grid of a stack (some grids without a
    visibility, kernels without one, a last block with idle threads).  Tolerance as
    for test_plain_fp64_degrid, n terms to a cell at most."""
    torch, L, E, _, O = env
    N, S, G = 64, 5, 3
    rng, uvw, gcf, src = _case(n, n, S, 2, True, G=G)
    vis = rng.normal(size=n) + 1j * rng.normal(size=n)
    lay = rng.integers(0, layers, n).astype(numpy.int32)
    lay[lay == 2] = 0
    src[src == 1] = 0
    kt = E.KernelTable.from_gcf(gcf, 1, E.CD)
    plan = E.Plan(uvw, 1.0, (N, N), kt, src[:, 0].astype(numpy.int32), mode=L.CG_PLAN_GROUPS,
                  layers=None if layers == 1 else (layers, lay))
    v = E.cuda_tensor(vis, E.CD)
    grid = plan.grid_fp64(kt, v, torch.zeros((layers, N, N), dtype=E.CD, device="cuda"))
    model = E.cuda_tensor(rng.normal(size=(layers, N, N)) * (1 + 2j), E.CD)
    d = plan.degrid_fp64(kt, model).cpu().numpy()
    plan.check()
    tol = 4 * (max(n, S * S) + 8) * S * 2.0 ** -53
    for p in range(layers):
        s = lay == p
        want = numpy.zeros((N, N), dtype=complex)
        O.convgrid(gcf, want, uvw[s, :2], src[s], vis[s])
        dw = O.convdegrid(gcf, model[p].cpu().numpy(), uvw[s, :2], src[s])
        for a, b in ((grid[p].cpu().numpy(), want), (d[s], dw)):
            if b.size:
                assert numpy.abs(a - b).max() <= tol * max(numpy.abs(b).max(), 1.0)


@pytest.mark.parametrize("N,S,sep,layers,n", [
    (24, 7, True, 1, 1), (256, 8, True, 1, 1000), (1531, 9, False, 1, 4000),
    (2047, 8, True, 1, 3), (2100, 8, False, 1, 300000), (129, 17, True, 1, 5000),
    (1500, 17, False, 1, 9000), (640, 8, False, 12, 20000)])
def test_plan_lists(env, N, S, sep, layers, n):
    """The plan's offsets and items in one block (up to 16384 buckets), in two launches
    (tiles as buckets) and in separate passes (sub-tiles): every visibility sorted
    once, its record as assigned, the buckets' counts in order; then gridded ones,
    which need every item once: small whole numbers, exact in complex64."""
    torch, L, E, _, O = env
    rng, uvw, gcf, src = _case(N + n, n, S, 2, sep, G=2)
    gcf = numpy.ones_like(gcf)
    lay = rng.integers(0, layers, n).astype(numpy.int32)
    kt = E.KernelTable.from_gcf(gcf, 1, E.CF)
    plan = E.Plan(uvw, 1.0, (N, N), kt, src[:, 0].astype(numpy.int32),
                  layers=None if layers == 1 else (layers, lay))
    vis = rng.integers(-4, 5, n).astype(numpy.complex64)
    got = plan.grid(kt, E.cuda_tensor(vis, E.CF),
                    torch.zeros((layers, N, N), dtype=E.CF, device="cuda")).cpu().numpy()
    plan.check()
    recs, perm, counts = (t.cpu().numpy() for t in plan.export())
    x, _, y, _ = O.frac_coords((N, N), 2, uvw[:, :2])
    numpy.testing.assert_array_equal(numpy.sort(perm), numpy.arange(n))
    numpy.testing.assert_array_equal(recs[:, 0], (x - S // 2)[perm])
    numpy.testing.assert_array_equal(recs[:, 1], (y - S // 2)[perm])
    assert counts.sum() == n
    want = numpy.zeros((layers, N + S, N + S))
    numpy.add.at(want, (lay, y - S // 2, x - S // 2), vis.real)
    for axis in (1, 2):  # the footprints: S cells on from the corner
        want = sum(numpy.roll(want, t, axis) for t in range(S))
    numpy.testing.assert_array_equal(got.real, want[:, :N, :N])


def _near(a, b, tol=1e-6):
    """Within tol of b's norm: the same products summed in the same order, with a
    few roundings of 2^-24 to each."""
    a, b = a.cpu().numpy(), b.cpu().numpy()
    assert numpy.linalg.norm(a - b) <= tol * numpy.linalg.norm(b)


@pytest.mark.parametrize("N,held", [(64, [1, 0, 2]), (96, [3]), (2048, [0, 0]), (2048, [5]),
                                    (2048, [0, 7, 1, 0, 2]), (4096, [1, 1, 0, 9]), (8192, [0, 4, 1])])
def test_wstack_image(env, N, held):
    """Planes summed in the transform's last pass (from 2048), some or all of them
    without visibilities, against the transform and the sum by themselves."""
    torch, L, E, _, O = env
    g = torch.Generator(device="cuda").manual_seed(N + len(held))
    planes = torch.randn((len(held), N, N), dtype=E.CF, device="cuda", generator=g)
    w = torch.linspace(-700.0, 900.0, len(held), dtype=torch.float64, device="cuda")
    counts = torch.tensor(held, dtype=torch.int32, device="cuda")
    st = E.Status()
    want = E.wstack_combine(E.fft_(planes.clone(), True), 0.3, w, counts, st)
    got = E.wstack_image(planes.clone(), 0.3, w, counts, st)
    st.check()
    _near(got, want)
    assert E.fft_timeouts() == 0
    E.wstack_image(planes, 1.5, w, counts, st)  # l^2 + m^2 >= 1 in the corners
    with pytest.raises(Exception):
        st.check()


@pytest.mark.parametrize("S", [64, 96, 128, 256, 512])
def test_towers_stack(env, S):
    """Layers summed by chunk in the transform's last pass (sides 64 to 256), and the
    reverse in its first (to 512), chunks of one layer, of many and of none, against
    the transforms and sums by themselves."""
    torch, L, E, _, O = env
    first = numpy.array([0, 1, 1, 4, 4 + 3 * 1024 // S, 4 + 3 * 1024 // S + 2], numpy.int32)
    n = int(first[-1])
    g = torch.Generator(device="cuda").manual_seed(S)
    stack = torch.randn((n, S, S), dtype=E.CF, device="cuda", generator=g)
    w = numpy.random.default_rng(S).uniform(-3000, 3000, n)
    st = E.Status()
    want = E.towers_combine(E.fft_raw(stack.clone(), True), 0.2, w, first, st)
    _near(E.towers_image(stack.clone(), 0.2, w, first, st), want)
    images = torch.randn((len(first) - 1, S, S), dtype=E.CF, device="cuda", generator=g)
    want = E.fft_raw(E.towers_expand(images, 0.2, w, first, st), False)
    _near(E.towers_layers(images, 0.2, w, first, st), want)
    st.check()
    assert E.fft_timeouts() == 0
    for call, x in ((E.towers_image, stack), (E.towers_layers, images)):
        st = E.Status()
        call(x, 1.5, w, first, st)
        with pytest.raises(Exception):
            st.check()


@pytest.mark.parametrize("nk", [1, 3, 4, 6])
def test_aw_akern_blocks(env, nk):
    """A1 * A2 by four kernels to a block: part-filled last blocks, and one bad index
    that loses its own kernel's call only.  Tolerance 2e-6 of the norm against the
    complex128 form: sums of 256 products, twice."""
    torch, L, E, _, O = env
    rng = numpy.random.default_rng(nk)
    A = rng.normal(size=(5, 16, 16)) + 1j * rng.normal(size=(5, 16, 16))
    W = rng.normal(size=(2, 2, 2, 16, 16)) + 1j * rng.normal(size=(2, 2, 2, 16, 16))
    a1, a2 = rng.integers(0, 5, (2, nk)).astype(numpy.int32)
    wi = rng.integers(0, 2, nk).astype(numpy.int32)
    _near(E.aw_kernels(A, W, a1, a2, wi, dtype=E.CF).to(E.CD),
          E.aw_kernels(A, W, a1, a2, wi, dtype=E.CD), 2e-6)
    a1[-1] = 5
    with pytest.raises(Exception):
        E.aw_kernels(A, W, a1, a2, wi, dtype=E.CF)
        torch.cuda.synchronize()
