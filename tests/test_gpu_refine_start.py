"""The one-pass start of a refined solve against the operators it replaces."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def L():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mojo_poissonrecon_b200 import _native

    return _native.lib()


def stream():
    return torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("copying", [True, False])
@pytest.mark.parametrize("n", (9, 17, 33, 65, 129))
def test_start_matches_its_operators(L, n, copying):
    from padded import geometry

    rng = np.random.default_rng(n)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    rhs = dev(np.where(rng.random((n, n, n)) < 0.08, rng.normal(size=(n, n, n)) * 100.0, 0.0))
    screen = dev(np.where(rng.random((n, n, n)) < 0.04, rng.random((n, n, n)) * 2.0, 0.0))
    nan = lambda: torch.full((n, n, n), float("nan"), dtype=torch.float64, device="cuda")
    copies, x0 = (nan(), nan()), nan()
    D, invD, weights, r32 = (torch.zeros(geometry(L, n)[1], dtype=torch.float32, device="cuda") for _ in range(4))
    norms = torch.empty(2, dtype=torch.float64, device="cuda")
    ws = torch.empty(L.pb_refine_start_workspace_size(n), dtype=torch.uint8, device="cuda")
    status = L.pb_refine_start_f64(rhs.data_ptr(), screen.data_ptr(), n, 4.0,
                                   *(c.data_ptr() if copying else None for c in copies), x0.data_ptr(), D.data_ptr(),
                                   invD.data_ptr(), weights.data_ptr(), r32.data_ptr(), norms.data_ptr(),
                                   norms.data_ptr() + 8, ws.data_ptr(), ws.numel(), stream())
    assert status == 0, L.pb_last_error().decode()
    if copying:
        assert torch.equal(copies[0], rhs) and torch.equal(copies[1], screen)
    assert bool((x0 == 0.5).all())
    want = [torch.zeros_like(D) for _ in range(4)]
    assert L.pb_level_setup_f32(screen.data_ptr(), n, 4.0, *(t.data_ptr() for t in want[:3]), stream()) == 0
    for got, expected in zip((D, invD, weights), want):
        assert torch.equal(got, expected)
    norm2 = torch.empty(1, dtype=torch.float64, device="cuda")
    ws = torch.empty(L.pb_defect_workspace_size(n), dtype=torch.uint8, device="cuda")
    assert L.pb_defect_f64(x0.data_ptr(), None, None, rhs.data_ptr(), screen.data_ptr(), n, 4.0, want[3].data_ptr(),
                           None, norm2.data_ptr(), ws.data_ptr(), ws.numel(), stream()) == 0
    # the two may round a product's sum in one step or two: an ulp of the terms, at most 6 h^2 + pw screen
    scale = 2.0 ** -52 * (6.0 * (n - 1) ** 2 * (1 + 4.0 * float(screen.max())) + 100.0)
    assert float((r32 - want[3]).abs().max()) <= scale + 2.0 ** -23 * float(want[3].abs().max())
    assert abs(float(norms[0]) - float(norm2)) <= 1e-12 * float(norm2)
    exact = float(rhs.norm())
    assert abs(float(norms[1]) - exact) <= 1e-13 * exact
