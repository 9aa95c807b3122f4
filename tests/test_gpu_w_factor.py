"""The w-plane factors of the transforms' own passes, bit for bit those of the passes
that form the sums by themselves."""

import numpy
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    import torch
    from crocodile_gb300 import engine
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    return torch, engine


def _same(torch, a, b):
    assert torch.equal(torch.view_as_real(a) + 0.0, torch.view_as_real(b) + 0.0)  # -0 == 0


@pytest.mark.parametrize("w", [-700.37, 0.0, 1.5, 12345.678])
@pytest.mark.parametrize("N", [2048, 4096])
def test_wstack_factor(env, N, w):
    """One plane with a 1 in its corner: its transform is 1 / N^2 everywhere but for
    signs, exactly, so the image is the factor itself."""
    torch, E = env
    plane = torch.zeros((1, N, N), dtype=E.CF, device="cuda")
    plane[0, 0, 0] = 1.0
    mean_w = torch.tensor([w], dtype=torch.float64, device="cuda")
    counts = torch.ones(1, dtype=torch.int32, device="cuda")
    st = E.Status()
    want = E.wstack_combine(E.fft_(plane.clone(), True), 0.4, mean_w, counts, st)
    got = E.wstack_image(plane, 0.4, mean_w, counts, st)
    st.check()
    _same(torch, got, want)


@pytest.mark.parametrize("S", [64, 128, 256])
def test_towers_factor(env, S):
    """The same by sub-grids, one layer to a sum."""
    torch, E = env
    w = numpy.array([-3000.7, -1.25, 0.0, 17.0, 2999.1])
    first = numpy.arange(len(w) + 1, dtype=numpy.int32)
    stack = torch.zeros((len(w), S, S), dtype=E.CF, device="cuda")
    stack[:, 0, 0] = 1.0
    st = E.Status()
    want = E.towers_combine(E.fft_raw(stack.clone(), True), 0.3, w, first, st)
    got = E.towers_image(stack, 0.3, w, first, st)
    st.check()
    _same(torch, got, want)
