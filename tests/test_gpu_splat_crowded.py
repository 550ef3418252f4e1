"""Long lists of the splat (many points around one grid node): bit for bit with the
oracle at the edges of the rule, of a part and of a tile, and not far slower than
the same points spread out."""

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


def crowd(count, n, rng, cells):
    """Points of the eight cells around one node (of one cell where cells is 1)."""
    h = 1.0 / (n - 1)
    node = ((n - 1) // 2) * h
    pts = node + (rng.random((count, 3)) * (2.0 if cells == 8 and n > 2 else 1.0) - (1.0 if cells == 8 and n > 2 else 0.0)) * h
    nrm = rng.normal(size=(count, 3))
    nrm[rng.random(count) < 0.05] = 0.0  # rejected samples go to the last cell's lists
    return np.ascontiguousarray(np.clip(pts, 0.0, 1.0)), nrm


# the lists are long beyond 64 contributions to side 33, 128 to 65, 512 above; parts of 256, tiles of 224
@pytest.mark.parametrize("cells", [1, 8])
@pytest.mark.parametrize("n,count", [(2, 64), (2, 65), (3, 66), (3, 223), (3, 224), (3, 225), (5, 256), (5, 257),
                                     (5, 448), (5, 449), (9, 513), (33, 70), (65, 128), (65, 140), (129, 512),
                                     (129, 560), (9, 30000)])
def test_long_lists_match(L, oracle, n, count, cells):
    pts, nrm = crowd(count, n, np.random.default_rng(n * 7 + count), cells)
    p, m = torch.from_numpy(pts).cuda(), torch.from_numpy(nrm).cuda()
    rng = np.random.default_rng(5)
    want = [rng.normal(size=(n, n, n)) if n <= 9 else np.zeros((n, n, n)) for _ in range(5)]  # sums go on from these
    want[0] = np.abs(want[0])
    grids = [torch.from_numpy(w).cuda() for w in want]
    a = lambda v: int(v.ctypes.data)
    accepted = oracle.lib().mpr_splat_f64(a(pts), a(nrm), count, n, 1, *(a(w) for w in want), 1.5)
    got = torch.zeros(1, dtype=torch.int64, device="cuda")
    ws = torch.empty(L.pb_splat_workspace_size(count, n), dtype=torch.uint8, device="cuda")
    assert L.pb_splat_f64(p.data_ptr(), m.data_ptr(), count, n, 1, *(g.data_ptr() for g in grids), 1.5, got.data_ptr(),
                          ws.data_ptr(), ws.numel(), stream()) == 0, L.pb_last_error()
    assert int(got) == accepted
    for g, w in zip(grids, want):
        assert np.array_equal(g.cpu().numpy(), w)


def test_crowded_cloud_is_not_far_slower(L):
    """A million points at depth 3 within twenty times the same points' time at depth 8 (a thread per
    list took 140 times as long; the chain of additions of the longest list alone is two to three times)."""
    from mojo_poissonrecon_b200 import workloads

    pts, nrm = workloads.torus(1_000_000, seed=1)
    pts = np.ascontiguousarray((pts + 0.95) / 1.9)
    p, m = torch.from_numpy(pts).cuda(), torch.from_numpy(nrm).cuda()
    times = {}
    for depth in (8, 3):
        n = (1 << depth) + 1
        grids = [torch.empty((n, n, n), dtype=torch.float64, device="cuda") for _ in range(3)]
        got = torch.zeros(1, dtype=torch.int64, device="cuda")
        ws = torch.empty(L.pb_splat_assemble_workspace_size(len(pts), n), dtype=torch.uint8, device="cuda")
        taken = []
        for _ in range(5):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            assert L.pb_splat_assemble_f64(p.data_ptr(), m.data_ptr(), len(pts), n, 1, 1.5, 4.0, 0.5,
                                           *(g.data_ptr() for g in grids), got.data_ptr(), ws.data_ptr(), ws.numel(),
                                           stream()) == 0, L.pb_last_error()
            end.record()
            end.synchronize()
            taken.append(start.elapsed_time(end))
        times[depth] = min(taken)
    assert times[3] < 20.0 * times[8], times
