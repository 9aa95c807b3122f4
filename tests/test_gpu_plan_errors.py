"""Plans of which some visibilities were refused, used after the caller has reset the
status block: what was sorted is gridded and degridded, and nothing beyond it."""

import numpy
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    import torch
    from crocodile_gb300 import _lib, engine
    from oracle import crocodile_oracle
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    return torch, _lib, engine, crocodile_oracle


@pytest.mark.parametrize("sep", [True, False])
@pytest.mark.parametrize("layers", [1, 3])
@pytest.mark.parametrize("n,nbad", [(1, 1), (40, 40), (300, 1), (300, 77)])
def test_refused_rows_are_left_out(env, n, nbad, layers, sep):
    """Coordinates off the grid, footprints over its edge and kernel indices beyond the
    table, at the start, middle and end of the input.  Tolerance 2e-6 of the norm: a few
    hundred complex64 products to a cell; 1e-13 for the complex128 form."""
    torch, L, E, O = env
    N, S, Q, G = 64, 8, 4, 3
    rng = numpy.random.default_rng(n + nbad)
    uvw = numpy.column_stack([rng.uniform(-0.3, 0.3, (n, 2)), numpy.zeros(n)])
    shape = (G, Q, S) if sep else (G, Q, Q, S, S)
    gcf = rng.normal(size=shape) + 1j * rng.normal(size=shape)
    kidx = rng.integers(0, G, n).astype(numpy.int32)
    lay = rng.integers(0, layers, n).astype(numpy.int32)
    vis = rng.normal(size=n) + 1j * rng.normal(size=n)
    bad = rng.permutation(n)[:nbad]
    good = numpy.setdiff1d(numpy.arange(n), bad)
    uvw[bad[0::3], 0] = 0.7
    uvw[bad[1::3], 1] = 0.499
    kidx[bad[2::3]] = G
    model = rng.normal(size=(layers, N, N)) + 1j * rng.normal(size=(layers, N, N))
    want = numpy.zeros((layers, N, N), dtype=complex)
    wantd = numpy.zeros(n, dtype=complex)
    for p in range(layers):
        s = good[lay[good] == p]
        if len(s):
            O.convgrid(gcf, want[p], uvw[s, :2], kidx[s][:, None], vis[s])
            wantd[s] = O.convdegrid(gcf, model[p], uvw[s, :2], kidx[s][:, None])
    for mode, dt, tol in ((L.CG_PLAN_TILED, E.CF, 2e-6), (L.CG_PLAN_GROUPS, E.CD, 1e-13)):
        kt = E.KernelTable.from_gcf(gcf, 1, dt)
        plan = E.Plan(uvw, 1.0, (N, N), kt, kidx, mode,
                      layers=None if layers == 1 else (layers, lay))
        with pytest.raises(Exception):
            plan.check()
        plan.status.reset()
        m, v = E.cuda_tensor(model, dt), E.cuda_tensor(vis, dt)
        zero = lambda: torch.zeros((layers, N, N), dtype=dt, device="cuda")  # noqa: E731
        out = lambda: torch.zeros(n, dtype=dt, device="cuda")  # noqa: E731
        if mode == L.CG_PLAN_TILED:
            wt = torch.ones(n, dtype=torch.float32, device="cuda")
            fused = zero()
            got = [(plan.grid(kt, v, zero()), want), (plan.grid_sparse(kt, v, zero()), want),
                   (plan.grid_weighted(kt, v, wt, zero()), want),
                   (plan.degrid(kt, m, out()), wantd),
                   (plan.degrid_grid(kt, m, v, fused, vis_out=out()), wantd), (fused, want)]
        else:
            got = [(plan.grid_fp64(kt, v, zero()), want), (plan.degrid_fp64(kt, m, out()), wantd)]
        plan.check()
        for a, b in got:
            assert numpy.linalg.norm(a.cpu().numpy() - b) <= tol * numpy.linalg.norm(b)


def test_aw_kernels_bad_index(env):
    """An antenna index beyond the A-kernels is an IndexError of its call; the next call
    gives the kernels that it gave before, bit for bit."""
    torch, L, E, O = env
    rng = numpy.random.default_rng(2)
    A = rng.normal(size=(5, 16, 16)) + 1j * rng.normal(size=(5, 16, 16))
    W = rng.normal(size=(2, 2, 2, 16, 16)) + 1j * rng.normal(size=(2, 2, 2, 16, 16))
    a1, a2 = rng.integers(0, 5, (2, 6)).astype(numpy.int32)
    wi = rng.integers(0, 2, 6).astype(numpy.int32)
    want = E.aw_kernels(A, W, a1, a2, wi, dtype=E.CF)
    for i, bad in ((5, 5), (0, -1), (2, 100)):
        b = a1.copy()
        b[i] = bad
        with pytest.raises(IndexError):
            E.aw_kernels(A, W, b, a2, wi, dtype=E.CF)
    got = E.aw_kernels(A, W, a1, a2, wi, dtype=E.CF)
    assert torch.equal(torch.view_as_real(got), torch.view_as_real(want))


def test_arrays_that_are_too_short(env):
    """Fewer visibilities, weights, indices, results or cells than the plan has are
    refused before anything runs; more than it has are taken as before."""
    torch, L, E, O = env
    n, N, S, G = 40, 64, 8, 3
    rng = numpy.random.default_rng(4)
    uvw = numpy.column_stack([rng.uniform(-0.3, 0.3, (n, 2)), numpy.zeros(n)])
    gcf = rng.normal(size=(G, 4, S)) + 0j
    idx = rng.integers(0, 2, n).astype(numpy.int32)
    short, more = idx[:-1], numpy.append(idx, 0).astype(numpy.int32)
    kt, kd = E.KernelTable.from_gcf(gcf, 1, E.CF), E.KernelTable.from_gcf(gcf, 1, E.CD)
    groups = L.CG_PLAN_GROUPS
    for kw in (dict(kidx=short), dict(kidx=idx, layers=(2, short)),
               dict(kidx=idx, mode=groups, groups=(2, short))):
        with pytest.raises(ValueError):
            E.Plan(uvw, 1.0, (N, N), kt, **kw)
    E.Plan(uvw, 1.0, (N, N), kt, more, layers=(2, more)).check()
    plan = E.Plan(uvw, 1.0, (N, N), kt, idx, layers=(2, idx))
    plain = E.Plan(uvw, 1.0, (N, N), kd, idx, mode=groups)
    v, v1 = (torch.zeros(k, dtype=E.CF, device="cuda") for k in (n, n - 1))
    g, g1 = (torch.zeros((k, N, N), dtype=E.CF, device="cuda") for k in (2, 1))
    w1 = torch.zeros(n - 1, dtype=torch.float32, device="cuda")
    for call in (lambda: plan.grid(kt, v1, g), lambda: plan.grid(kt, v, g1),
                 lambda: plan.grid_sparse(kt, v1, g), lambda: plan.grid_sparse(kt, v, g1),
                 lambda: plan.grid_weighted(kt, None, w1, g), lambda: plan.degrid(kt, g1),
                 lambda: plan.degrid(kt, g, v1), lambda: plan.degrid_grid(kt, g1, v, g.clone()),
                 lambda: plan.degrid_grid(kt, g, v1, g.clone()),
                 lambda: plan.degrid_grid(kt, g, v, g1),
                 lambda: plan.degrid_grid(kt, g, v, g.clone(), vis_out=v1),
                 lambda: plain.grid_fp64(kd, v, g.to(E.CD)),  # complex64: half the bytes
                 lambda: plain.degrid_fp64(kd, g1)):
        with pytest.raises(ValueError):
            call()
    plan.check()
    plain.check()
