"""A refined engine's solve takes a right-hand side and screen of any strides and
real type, as Tensor.copy_ does, and refuses other shapes before any launch."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("lean", [False, True])
@pytest.mark.parametrize("n", [17, 33])
def test_any_strides_and_types(n, lean):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mojo_poissonrecon_b200 import solver32

    rng = np.random.default_rng(n)
    # values that FP32 holds, so that the FP32 copy is the same system
    rhs = torch.from_numpy((rng.normal(size=(n, n, n)) * 100).astype(np.float32)).cuda().double()
    screen = torch.from_numpy(np.where(rng.random((n, n, n)) < 0.1, rng.random((n, n, n)), 0).astype(np.float32)).cuda()
    screen = screen.double()
    eng = solver32.RefinedEngine(n, 4.0, rhs.device, lean=lean)
    want, stats = eng.solve(rhs, screen, 1e-9, 50)
    want = want.clone()
    assert stats.cycles > 0
    wide = torch.zeros((n, n, 2 * n), dtype=torch.float64, device="cuda")
    wide[:, :, ::2] = rhs
    turned = screen.permute(2, 0, 1).contiguous().permute(1, 2, 0)
    assert not turned.is_contiguous() and torch.equal(turned, screen)
    for b, s in ((wide[:, :, ::2], turned), (rhs.float(), screen), (rhs, screen.float()), (rhs, screen)):
        got, _ = eng.solve(b, s, 1e-9, 50)
        assert torch.equal(got, want)
    for bad in ((rhs[1:], screen), (rhs, screen[:, : n - 1]), (rhs, screen[:, :, :2])):
        with pytest.raises(RuntimeError):
            eng.solve(*bad, 1e-9, 50)
    got, _ = eng.solve(rhs, screen, 1e-9, 50)
    assert torch.equal(got, want)
