"""The word-parallel extraction at the sides where its rows of 32 begin, end and
leave a remainder, against the reference-shaped entry points; and its finite
checks."""

import numpy as np
import pytest

from test_gpu_extract import bit_array, reference_shaped

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def L():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mojo_poissonrecon_b200 import _native

    return _native.lib()


@pytest.mark.parametrize("n", [2, 3, 31, 32, 33, 34, 63, 64, 65, 66, 97])
@pytest.mark.parametrize("kind", ["noise", "full", "none"])
def test_sides_match(L, n, kind):
    rng = np.random.default_rng(n)
    field = rng.normal(size=(n, n, n))  # every cell and edge at random: all words busy
    if kind == "full":
        field = np.where((np.indices((n, n, n)).sum(0) & 1) == 0, 1.0, -1.0) * (1.0 + rng.random((n, n, n)))
    elif kind == "none":
        field = 1.0 + rng.random((n, n, n))
    f = torch.from_numpy(field).cuda()
    d = torch.from_numpy(rng.random((n, n, n))).cuda()
    for got, want in zip(bit_array(L, f, d, 0.1), reference_shaped(L, f, d, 0.1)):
        assert np.array_equal(got, want)


@pytest.mark.parametrize("n", [5, 33, 70])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
@pytest.mark.parametrize("which", ["field", "density"])
def test_values_that_are_not_finite_are_refused(n, bad, which):
    import mojo_poissonrecon_b200 as mpr

    grids = dict(field=torch.rand(n, n, n, dtype=torch.float64, device="cuda") - 0.5,
                 density=torch.rand(n, n, n, dtype=torch.float64, device="cuda"))
    for place in ((0, 0, 0), (n - 1, n - 1, n - 1), (n // 2, 1, n - 1)):
        broken = {k: v.clone() for k, v in grids.items()}
        broken[which][place] = bad
        with pytest.raises(ValueError, match="field and iso_value" if which == "field" else "^density must be finite"):
            mpr.extract_isosurface(broken["field"], density=broken["density"])
    assert mpr.extract_isosurface(grids["field"], density=grids["density"]).faces.shape[0] > 0
    with pytest.raises(ValueError, match="same shape"):
        mpr.extract_isosurface(grids["field"], density=grids["density"][:-1])
