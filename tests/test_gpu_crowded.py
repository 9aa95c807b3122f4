"""Visibilities that meet in few cells: the gridders' sums against 64 bits.

Equal positive terms (natural weighting, a PSF) are the worst case of sums in 32 bits:
each addition rounds the same way while the sum stays in one binade.  In sequence, 512
of them are off by 3.7e-6 of the sum (rms over terms), 25,600 by 1.9e-4.  The windowed
gridders sum up to 512 at a time and then the windows, 5.3e-6 at 204,800: within 1e-5.
"""

import numpy
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-5


@pytest.fixture(scope="module")
def env():
    import torch
    from crocodile_gb300 import _lib, engine
    from oracle import crocodile_oracle
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    return torch, _lib, engine, crocodile_oracle


def _places(N, n, S, where, rng):
    """uvw of n visibilities whose footprints start in one cell, in the 3 x 3 cells
    around the middle of the grid (a corner of tiles), or in 16 x 16 from there on."""
    cells = {"cell": 1, "patch": 3, "tile": 16}[where]
    at = rng.integers(0, cells, (n, 2)) + S // 2 - (0 if where == "tile" else 2)
    return numpy.column_stack([at / N, numpy.zeros(n)])


def _exact(N, S, gcf, uvw, sep, value):
    """n equal visibilities in 64 bits: the kernel at each distinct place, times how many
    stand there."""
    out = numpy.zeros((N, N), dtype=complex)
    uv, count = numpy.unique(uvw[:, :2], axis=0, return_counts=True)
    k = numpy.outer(gcf[0], gcf[0]) if sep else gcf[0, 0]
    for (u, v), c in zip(uv, count):
        x, y = (int(round(p * N)) + N // 2 - S // 2 for p in (u, v))
        out[y:y + S, x:x + S] += c * value * k
    return out


def _check(env, N, n, S, sep, where, tile=0):
    torch, L, E, O = env
    Q = 4
    rng = numpy.random.default_rng(N + S)
    uvw = _places(N, n, S, where, rng)
    gcf = rng.uniform(0.2, 1, (Q, S) if sep else (Q, Q, S, S)).astype(numpy.float32).astype(complex)
    kt = E.KernelTable.from_gcf(gcf, 0, E.CF)
    plan = E.Plan(uvw, 1.0, (N, N), kt, tile=tile)
    value = numpy.float32(0.7391)
    v = torch.full((n,), float(value), dtype=E.CF, device="cuda")
    w = torch.full((n,), float(value), dtype=torch.float32, device="cuda")
    zero = lambda: torch.zeros((N, N), dtype=E.CF, device="cuda")  # noqa: E731
    want = _exact(N, S, gcf, uvw, sep, float(value))
    fused = zero()
    d = plan.degrid_grid(kt, zero(), v, fused, residual=True)
    got = [plan.grid(kt, v, zero()), plan.grid_weighted(kt, None, w, zero()), fused]
    plan.check()
    assert not d.any()
    box = slice(N // 2 - 32, N // 2 + 64)
    for g in got:
        err = g[box, box].cpu().numpy().astype(complex) - want[box, box]
        assert numpy.linalg.norm(err) <= TOL * numpy.linalg.norm(want)
        assert torch.count_nonzero(g) == numpy.count_nonzero(want)


@pytest.mark.parametrize("where", ["cell", "patch", "tile"])
@pytest.mark.parametrize("S,sep", [(3, True), (8, True), (16, True), (9, False), (16, False)])
@pytest.mark.parametrize("N,n", [(256, 204800), (2048, 204800), (300, 60000)])
def test_windowed(env, N, n, S, sep, where):
    """Calls of the windowed gridders (n S > 200 N): plans of one block and of two
    launches, their items short where n is small."""
    _check(env, N, n, S, sep, where)


@pytest.mark.parametrize("where", ["cell", "patch", "tile"])
@pytest.mark.parametrize("S,sep", [(3, True), (8, True), (16, True), (1, False), (7, False), (8, False),
                                   (9, False), (16, False)])
@pytest.mark.parametrize("N,per", [(1024, 200), (1024, 30), (300, 200)])
def test_few_visibilities(env, N, per, S, sep, where):
    """n S = per N: calls whose number of visibilities alone would send their taps
    one by one to the grid."""
    _check(env, N, per * N // S, S, sep, where)


@pytest.mark.parametrize("S,sep", [(8, True), (8, False)])
def test_few_on_a_large_grid(env, S, sep):
    _check(env, 8192, 204800, S, sep, "cell")


@pytest.mark.parametrize("where", ["cell", "tile"])
@pytest.mark.parametrize("S,sep", [(1, True), (8, True), (13, True), (9, False), (16, False)])
@pytest.mark.parametrize("tile", [4, 8, 16, 32])
@pytest.mark.parametrize("n", [1, 57, 512, 513, 3000])
def test_requested_tiles(env, n, tile, S, sep, where):
    """Tiles as requested, so small that a cell's taps come from many; and calls too
    small for any cell to be crowded."""
    _check(env, 512, n, S, sep, where, tile)


@pytest.mark.parametrize("layers,N,n,S,sep", [(1, 1024, 100000, 8, True), (1, 1024, 100000, 8, False),
                                              (1, 2048, 60000, 3, True), (2, 256, 6500, 9, False)])
def test_wstack_planes(env, layers, N, n, S, sep):
    """w-stacking of crowded planes that are not sparse by the edge of the windowed
    gridders' tiles, whatever tiles the plan has: the image (w 0: the sum of the planes'
    inverse transforms) against 64 bits."""
    torch, L, E, O = env
    from crocodile_gb300 import synthesis
    rng = numpy.random.default_rng(N + S)
    uvw = _places(N, n, S, "cell", rng)
    gcf = rng.uniform(0.2, 1, (4, S) if sep else (4, 4, S, S)).astype(numpy.float32).astype(complex)
    value = numpy.float32(0.7391)
    image = synthesis.w_stack_imaging(1.0, N, N * uvw, None, numpy.full(n, value + 0j), gcf,
                                      numpy.arange(n) % layers)
    want = O.ifft(_exact(N, S, gcf, uvw, sep, float(value)))
    assert numpy.linalg.norm(image - want) <= TOL * numpy.linalg.norm(want)


@pytest.mark.parametrize("N,n,S,tile", [(777, 13593, 2, 32), (777, 13593, 4, 64), (256, 60000, 2, 32),
                                        (256, 60000, 4, 64), (256, 60000, 1, 16)])
def test_narrow_supports_on_wide_tiles(env, N, n, S, tile):
    """Lane items of few taps beside their window's cells: those of full length are
    summed in the window all the same."""
    _check(env, N, n, S, False, "cell", tile)


@pytest.mark.parametrize("S", [1, 2, 4, 5])
@pytest.mark.parametrize("n", [65535, 65536])
def test_narrow_supports_dense(env, n, S):
    """Narrow separable supports on either side of the line between the gridders, on
    dense visibilities of one tile."""
    _check(env, 96, n, S, True, "tile")
