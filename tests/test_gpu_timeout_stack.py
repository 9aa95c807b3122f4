"""Waits of w-stacking's transforms that run out are errors of the call."""

import pytest

pytestmark = pytest.mark.gpu


def test_wstack_wait_runs_out_and_next_call_is_right():
    """At a wait limit of 0 the column passes of w-stacking give up at the first poll
    of a copy that has not landed; each counts in the caller's status block as in the
    transforms' own counter, and check raises.  The next call at the default limit
    agrees with the transform and the sum by themselves to 1e-6 of the norm (the same
    products in the same order, a few roundings of 2^-24 to each)."""
    import torch
    from crocodile_gb300 import _lib as L, engine as E
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    lib = L.lib()
    N, layers = 2048, 3
    g = torch.Generator(device="cuda").manual_seed(3)
    planes = torch.randn((layers, N, N), dtype=E.CF, device="cuda", generator=g)
    w = torch.tensor([-300.0, 10.0, 500.0], dtype=torch.float64, device="cuda")
    counts = torch.ones(layers, dtype=torch.int32, device="cuda")
    st = E.Status()
    E.fft_timeouts(reset=True)
    default = lib.cg_get_wait_limit()
    try:
        assert lib.cg_set_wait_limit(0) == L.CG_OK
        E.wstack_image(planes.clone(), 0.3, w, counts, st)
        torch.cuda.synchronize()
    finally:
        lib.cg_set_wait_limit(default)
    given_up = E.fft_timeouts(reset=True)
    assert given_up > 0 and st.counts()[3] == given_up
    with pytest.raises(RuntimeError, match="code -7"):
        st.check()
    st.reset()
    want = E.wstack_combine(E.fft_(planes.clone(), True), 0.3, w, counts, st)
    got = E.wstack_image(planes, 0.3, w, counts, st)
    st.check()
    assert E.fft_timeouts() == 0
    assert torch.linalg.norm(got - want) <= 1e-6 * torch.linalg.norm(want)


def test_limit_of_zero_leaves_other_calls_as_they_are():
    """Calls whose kernels wait for nothing, or for the default limit at least, give the
    same results under a wait limit of 0: the direct gridder on a table of the lane
    layout (one visibility to a cell: sums in any order are the same), and w-towers'
    sums in the transforms' own pass."""
    import numpy
    import torch
    from crocodile_gb300 import _lib as L, engine as E
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    lib = L.lib()
    rng = numpy.random.default_rng(5)
    N, S, n = 256, 16, 25
    uv = (numpy.stack(numpy.meshgrid(numpy.arange(5), numpy.arange(5)), -1).reshape(-1, 2) - 2) * 32
    uvw = numpy.column_stack([uv / N, numpy.zeros(n)])
    kt = E.KernelTable.from_gcf(rng.normal(size=(2, 2, S, S)) + 0j, 0, E.CF)
    v = E.cuda_tensor(rng.normal(size=n) + 0j, E.CF)
    stack = E.cuda_tensor(rng.normal(size=(5, 128, 128)) + 0j, E.CF)
    w, first = numpy.linspace(-100, 100, 5), numpy.array([0, 2, 5], numpy.int32)

    def calls():
        st = E.Status()
        plan = E.Plan(uvw, 1.0, (N, N), kt, status=st)
        grid = plan.grid(kt, v, torch.zeros((N, N), dtype=E.CF, device="cuda"))
        image = E.towers_image(stack.clone(), 0.2, w, first, st)
        st.check()
        return torch.view_as_real(grid), torch.view_as_real(image)

    want = calls()
    default = lib.cg_get_wait_limit()
    try:
        assert lib.cg_set_wait_limit(0) == L.CG_OK
        got = calls()
    finally:
        lib.cg_set_wait_limit(default)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
