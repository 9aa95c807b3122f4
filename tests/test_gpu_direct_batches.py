"""The direct kernels' batches, 1 to 32 visibilities to a warp by the call's number."""

import numpy
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sep", [True, False])
@pytest.mark.parametrize("S", [3, 8, 9, 11, 12, 16])
@pytest.mark.parametrize("n", [3, 4863, 4865, 19457, 60001, 200003])
def test_batches(n, S, sep):
    """Degridding: the tiled degridder's bits, whatever batch a visibility stands in.
    Gridding tap by tap against the complex128 form, 2e-6 of the norm: products of 2^-24,
    and at most a hundred to a cell."""
    import torch
    from crocodile_gb300 import _lib as L, autotune, engine as E
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    rng = numpy.random.default_rng(n + S)
    N, Q, G = 1024, 2, 2
    uvw = numpy.column_stack([rng.uniform(-0.45, 0.45, (n, 2)), numpy.zeros(n)])
    shape = (G, Q, S) if sep else (G, Q, Q, S, S)
    gcf = rng.normal(size=shape) + 1j * rng.normal(size=shape)
    kidx = rng.integers(0, G, n).astype(numpy.int32)
    kt, kd = E.KernelTable.from_gcf(gcf, 1, E.CF), E.KernelTable.from_gcf(gcf, 1, E.CD)
    plan = E.Plan(uvw, 1.0, (N, N), kt, kidx)
    plain = E.Plan(uvw, 1.0, (N, N), kd, kidx, mode=L.CG_PLAN_GROUPS)
    model = torch.randn((N, N), dtype=E.CF, device="cuda")
    got = plan.degrid(kt, model)
    autotune.set_tuning(dvis=2)
    try:
        want = plan.degrid(kt, model)
    finally:
        autotune.set_tuning()
    assert torch.equal(torch.view_as_real(got), torch.view_as_real(want))
    vis = E.cuda_tensor(rng.normal(size=n) + 1j * rng.normal(size=n), E.CF)
    grid = plan.grid_sparse(kt, vis, torch.zeros((N, N), dtype=E.CF, device="cuda"))
    ref = plain.grid_fp64(kd, vis.to(E.CD), torch.zeros((N, N), dtype=E.CD, device="cuda"))
    plan.check()
    plain.check()
    assert torch.linalg.norm(grid.to(E.CD) - ref) <= 2e-6 * torch.linalg.norm(ref)
