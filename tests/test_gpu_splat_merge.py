"""The splat by merged cell lists: crowded cells, points on cell faces and at the
cube's corners, rejected samples, few and many points per cell, against the
oracle bit for bit; pb_splat_assemble_f64 and pb_interpolate_attributes_f64
against the separate entry points."""

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


def cloud(kind, count, n, rng):
    pts = rng.random((count, 3))
    if kind == "crowded":  # most points in eight cells around one node, many of them equal
        pts = 0.5 + (pts - 0.5) * (1.9 / (n - 1))
        pts[::3] = pts[0]
    elif kind == "faces":  # on nodes, edges and faces of the grid, the cube's corners among them
        pts = np.round(pts * (n - 1)) / (n - 1)
        pts[: count // 2, 0] = rng.random(count // 2)
        pts[:8] = [[a & 1, a >> 1 & 1, a >> 2] for a in range(8)][:count]
    nrm = rng.normal(size=(count, 3))
    nrm[rng.random(count) < 0.1] = 0.0  # rejected samples
    return np.ascontiguousarray(pts), nrm


@pytest.mark.parametrize("kind", ["spread", "crowded", "faces"])
@pytest.mark.parametrize("count,n,conf", [(1, 2, 0), (9, 2, 1), (40, 3, 0), (33, 5, 1), (3000, 9, 0), (700, 17, 1),
                                          (20000, 33, 1), (50, 65, 0)])
def test_grids_match(L, oracle, kind, count, n, conf):
    pts, nrm = cloud(kind, max(count, 8) if kind == "faces" else count, n, np.random.default_rng(count + n))
    count = len(pts)
    p, m = torch.from_numpy(pts).cuda(), torch.from_numpy(nrm).cuda()
    want = [np.zeros((n, n, n)) for _ in range(5)]
    a = lambda v: int(v.ctypes.data)
    accepted = oracle.lib().mpr_splat_f64(a(pts), a(nrm), count, n, conf, *(a(w) for w in want), 1.5)
    grids = [torch.zeros((n, n, n), dtype=torch.float64, device="cuda") for _ in range(5)]
    got = torch.full((2,), -1, dtype=torch.int64, device="cuda")
    ws = torch.empty(L.pb_splat_workspace_size(count, n), dtype=torch.uint8, device="cuda")
    assert L.pb_splat_f64(p.data_ptr(), m.data_ptr(), count, n, conf, *(g.data_ptr() for g in grids), 1.5,
                          got.data_ptr(), ws.data_ptr(), ws.numel(), stream()) == 0, L.pb_last_error()
    for g, w in zip(grids, want):
        assert np.array_equal(g.cpu().numpy(), w)

    density, vx, vy, vz, screen = grids
    rhs = torch.empty_like(density)
    assert L.pb_divide_f64(density.data_ptr(), n ** 3, 1.5, stream()) == 0
    assert L.pb_assemble_f64(vx.data_ptr(), vy.data_ptr(), vz.data_ptr(), screen.data_ptr(), rhs.data_ptr(), n, 4.0, 0.5,
                             stream()) == 0
    out = [torch.full_like(density, float("nan")) for _ in range(3)]
    ws = torch.empty(L.pb_splat_assemble_workspace_size(count, n), dtype=torch.uint8, device="cuda")
    assert L.pb_splat_assemble_f64(p.data_ptr(), m.data_ptr(), count, n, conf, 1.5, 4.0, 0.5,
                                   *(g.data_ptr() for g in out), got.data_ptr() + 8, ws.data_ptr(), ws.numel(),
                                   stream()) == 0, L.pb_last_error()
    for g, w in zip(out, (density, screen, rhs)):
        assert torch.equal(g.view(torch.int64), w.view(torch.int64))
    assert got.tolist() == [accepted, accepted]


@pytest.mark.parametrize("channels", [1, 3, 64])
@pytest.mark.parametrize("count,n,kind", [(5, 5, "spread"), (4000, 17, "crowded"), (900, 33, "faces")])
def test_attributes_match(L, channels, count, n, kind):
    pts, nrm = cloud(kind, count, n, np.random.default_rng(count))
    p, m = torch.from_numpy(pts).cuda(), torch.from_numpy(nrm).cuda()
    values = torch.rand(count, channels, dtype=torch.float64, device="cuda")
    vertices = torch.rand(257, 3, dtype=torch.float64, device="cuda") * 1.2 - 0.1
    fmap = torch.tensor([0.01, -0.02, 0.03, 0.97], dtype=torch.float64, device="cuda")
    grids = torch.full((channels + 1, n, n, n), float("nan"), dtype=torch.float64, device="cuda")
    want, got = (torch.full((257, channels), float("nan"), dtype=torch.float64, device="cuda") for _ in range(2))
    ws = torch.empty(L.pb_splat_attributes_workspace_size(count), dtype=torch.uint8, device="cuda")
    assert L.pb_splat_attributes_f64(p.data_ptr(), m.data_ptr(), count, n, 1, values.data_ptr(), channels,
                                     grids.data_ptr(), ws.data_ptr(), ws.numel(), stream()) == 0
    assert L.pb_sample_attributes_f64(vertices.data_ptr(), 257, fmap.data_ptr(), n, grids.data_ptr(), channels,
                                      want.data_ptr(), stream()) == 0
    ws = torch.empty(L.pb_interpolate_attributes_workspace_size(count, n, channels), dtype=torch.uint8, device="cuda")
    assert L.pb_interpolate_attributes_f64(p.data_ptr(), m.data_ptr(), count, n, 1, values.data_ptr(), channels,
                                           vertices.data_ptr(), 257, fmap.data_ptr(), got.data_ptr(), ws.data_ptr(),
                                           ws.numel(), stream()) == 0
    assert torch.equal(got, want) and bool(torch.isfinite(got).all())
