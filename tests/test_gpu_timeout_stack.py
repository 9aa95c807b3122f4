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
