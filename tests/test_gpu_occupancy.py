"""The passes that read b, the screen and what depends on it only where they are not zero, against the dense ones.

A skipped read stands for a positive zero, so every result is the same to the last bit."""

import numpy as np
import pytest

from padded import geometry

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def L():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mojo_poissonrecon_b200 import _native

    return _native.lib()


def system(n, seed, kind):
    """A shell of screened nodes within a thicker shell of right-hand side; all, none, or single corners."""
    rng = np.random.default_rng(seed)
    c = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij")) / (n - 1) - 0.5
    r = np.sqrt((c ** 2).sum(0))
    near = {"shell": np.abs(r - 0.3) < 2.0 / n, "all": r >= 0, "none": r < 0, "corners": r > 0.866 * (1 - 1.5 / n)}[kind]
    wide = np.abs(r - 0.3) < 4.0 / n if kind == "shell" else near
    screen = np.where(near, rng.random((n, n, n)), 0.0)
    b = np.where(wide, rng.normal(size=(n, n, n)), 0.0)
    return b, screen


@pytest.mark.parametrize("kind", ("shell", "all", "none", "corners"))
@pytest.mark.parametrize("n", (5, 9, 31, 33, 65, 129, 161))
def test_sparse_passes_match_dense(L, n, kind):
    s = torch.cuda.current_stream().cuda_stream
    rng = np.random.default_rng(n)
    dev = lambda a, t=torch.float64: torch.from_numpy(np.ascontiguousarray(a)).to(t).cuda()
    b, screen = (dev(a) for a in system(n, n, kind))
    pitch, count = geometry(L, n)
    zeros = lambda: torch.zeros(count, dtype=torch.float32, device="cuda")
    D, invD, weights, r32 = (zeros() for _ in range(4))
    x0 = torch.empty_like(b)
    norms = torch.empty(2, dtype=torch.float64, device="cuda")
    ws = torch.empty(max(L.pb_refine_start_workspace_size(n), L.pb_fcg_workspace_size(n)), dtype=torch.uint8,
                     device="cuda")
    occupancy = torch.full((L.pb_occupancy_size(n) // 4,), -1, dtype=torch.int32, device="cuda")
    assert L.pb_refine_start_sparse_f64(b.data_ptr(), screen.data_ptr(), n, 4.0, None, None, x0.data_ptr(),
                                        D.data_ptr(), invD.data_ptr(), weights.data_ptr(), r32.data_ptr(),
                                        occupancy.data_ptr(), norms.data_ptr(), norms.data_ptr() + 8, ws.data_ptr(),
                                        ws.numel(), s) == 0, L.pb_last_error().decode()
    # the bits that must be set, and no others
    some = lambda a: (a != 0).cpu().numpy()
    tiles = (n + 31) // 32
    want = np.zeros((2, tiles, n, tiles), dtype=np.uint32)
    for m, set_ in enumerate((some(screen), some(screen) | some(b))):
        z, y, x = np.nonzero(set_)
        np.bitwise_or.at(want[m], (z // 32, y, x // 32), np.uint32(1) << (z % 32).astype(np.uint32))
    assert np.array_equal(occupancy.cpu().numpy().view(np.uint32), want.ravel())

    zp = zeros()
    inside = zp.view(n + 2, n + 2, pitch)[1:-1, 1:-1, 4:4 + n]
    inside.copy_(dev(rng.normal(size=(n, n, n)), torch.float32))
    ps = [dev(rng.normal(size=(n, n, n)), torch.float32) for _ in range(2)]
    xs = [dev(rng.normal(size=(n, n, n))) for _ in range(2)]
    for first, it, skew in ((1, 0, 0), (0, 1, 0), (0, 2, 0), (0, 2, 1)):
        got = []
        for sparse in (False, True):
            p, xx, r = [t.clone() for t in ps], [t.clone() for t in xs], r32.clone()
            if sparse and skew:  # padded arrays off the 16-byte boundaries: element loads
                r = torch.cat([r[:1], r])[1:]
            scal = torch.full((8,), 3.0, dtype=torch.float64, device="cuda")
            flags = torch.tensor([first, it, 0, 0], dtype=torch.int32, device="cuda")
            where = (occupancy.data_ptr(),) if sparse else ()
            direction = L.pb_fcg_direction_sparse_f64 if sparse else L.pb_fcg_direction_f64
            update = L.pb_fcg_update_sparse_f64 if sparse else L.pb_fcg_update_f64
            assert direction(zp.data_ptr(), p[0].data_ptr(), p[1].data_ptr(), r.data_ptr(), screen.data_ptr(), *where,
                             n, 4.0, scal.data_ptr(), flags.data_ptr(), ws.data_ptr(), ws.numel(), s) == 0
            assert update(zp.data_ptr(), p[0].data_ptr(), p[1].data_ptr(), xx[0].data_ptr(), xx[1].data_ptr(),
                          b.data_ptr(), screen.data_ptr(), *where, r.data_ptr(), n, 4.0, scal.data_ptr(),
                          flags.data_ptr(), ws.data_ptr(), ws.numel(), s) == 0
            got.append([*p, *xx, r, scal])
        for dense, sparse in zip(*got):
            bits = torch.int32 if dense.dtype == torch.float32 else torch.int64
            assert torch.equal(dense.view(bits), sparse.view(bits))
    if n % 2 == 0:
        return
    cn = (n + 1) // 2
    cpitch, ccount = geometry(L, cn)
    coarse = torch.zeros(ccount, dtype=torch.float32, device="cuda")
    coarse.view(cn + 2, cn + 2, cpitch)[1:-1, 1:-1, 4:4 + cn] = dev(rng.normal(size=(cn, cn, cn)), torch.float32)
    got = []
    for sparse in (False, True):
        up = zp.clone()
        if sparse:
            status = L.pb_prolong_fac_sparse_f32(coarse.data_ptr(), up.data_ptr(), weights.data_ptr(),
                                                 occupancy.data_ptr(), n, s)
        else:
            status = L.pb_prolong_fac_f32(coarse.data_ptr(), up.data_ptr(), weights.data_ptr(), n, s)
        assert status == 0
        got.append(up.view(torch.int32))
    assert torch.equal(*got)
    if n < 33 or (n - 1) & (n - 2):
        return
    got = []
    for sparse in (False, True):
        coef = torch.zeros(14, ccount, dtype=torch.float32, device="cuda")
        if sparse:
            status = L.pb_galerkin_sparse_f32(D.data_ptr(), n, 1, weights.data_ptr(), occupancy.data_ptr(),
                                              coef.data_ptr(), None, 0, s)
        else:
            status = L.pb_galerkin_f32(D.data_ptr(), n, 1, weights.data_ptr(), coef.data_ptr(), None, 0, s)
        assert status == 0
        got.append(coef.view(torch.int32))
    assert torch.equal(*got)


@pytest.mark.parametrize("kind", ("shell", "all"))
def test_planes_beyond_a_word(L, kind):
    """Blocks deeper than the 32 planes of a word read everything: pass 2 per node as ever, pass 1's sums to rounding."""
    from mojo_poissonrecon_b200 import tune

    n, s = 129, torch.cuda.current_stream().cuda_stream
    rng = np.random.default_rng(3)
    dev = lambda a, t=torch.float64: torch.from_numpy(np.ascontiguousarray(a)).to(t).cuda()
    b, screen = (dev(a) for a in system(n, 5, kind))
    pitch, count = geometry(L, n)
    D, invD, weights, r32, zp = (torch.zeros(count, dtype=torch.float32, device="cuda") for _ in range(5))
    zp.view(n + 2, n + 2, pitch)[1:-1, 1:-1, 4:4 + n].copy_(dev(rng.normal(size=(n, n, n)), torch.float32))
    norms = torch.empty(2, dtype=torch.float64, device="cuda")
    ws = torch.empty(max(L.pb_refine_start_workspace_size(n), L.pb_fcg_workspace_size(n)), dtype=torch.uint8,
                     device="cuda")
    occupancy = torch.empty(L.pb_occupancy_size(n) // 4, dtype=torch.int32, device="cuda")
    x0 = torch.empty_like(b)
    assert L.pb_refine_start_sparse_f64(b.data_ptr(), screen.data_ptr(), n, 4.0, None, None, x0.data_ptr(),
                                        D.data_ptr(), invD.data_ptr(), weights.data_ptr(), r32.data_ptr(),
                                        occupancy.data_ptr(), norms.data_ptr(), norms.data_ptr() + 8, ws.data_ptr(),
                                        ws.numel(), s) == 0
    ps = [dev(rng.normal(size=(n, n, n)), torch.float32) for _ in range(2)]
    xs = [dev(rng.normal(size=(n, n, n))) for _ in range(2)]
    flags = torch.tensor([0, 1, 0, 0], dtype=torch.int32, device="cuda")
    got = []
    for planes in (0, 48):
        if planes:
            L.pb_tune_set(tune.FCG_DIRECTION_PLANES, n, planes)
            L.pb_tune_set(tune.FCG_UPDATE_PLANES, n, planes)
        try:
            p, xx, r = [t.clone() for t in ps], [t.clone() for t in xs], r32.clone()
            sums, scal = (torch.full((8,), 3.0, dtype=torch.float64, device="cuda") for _ in range(2))
            assert L.pb_fcg_direction_sparse_f64(zp.data_ptr(), p[0].data_ptr(), p[1].data_ptr(), r.data_ptr(),
                                                 screen.data_ptr(), occupancy.data_ptr(), n, 4.0, sums.data_ptr(),
                                                 flags.data_ptr(), ws.data_ptr(), ws.numel(), s) == 0
            assert L.pb_fcg_update_sparse_f64(zp.data_ptr(), p[0].data_ptr(), p[1].data_ptr(), xx[0].data_ptr(),
                                              xx[1].data_ptr(), b.data_ptr(), screen.data_ptr(), occupancy.data_ptr(),
                                              r.data_ptr(), n, 4.0, scal.data_ptr(), flags.data_ptr(), ws.data_ptr(),
                                              ws.numel(), s) == 0
            got.append(([*p, *xx, r], sums[:4].cpu().numpy()))
        finally:
            L.pb_tune_set(tune.FCG_DIRECTION_PLANES, n, 0)
            L.pb_tune_set(tune.FCG_UPDATE_PLANES, n, 0)
    for a, c in zip(got[0][0], got[1][0]):
        assert torch.equal(a, c)
    # sums of 2.1M products in another order: relative 2.1e6 eps of their magnitudes at the very most
    assert np.allclose(got[0][1], got[1][1], rtol=1e-9, atol=0)
