"""The fused FP64 V-cycle against the operators it is made of (relax, residual,
restrict, prolong: themselves bit-exact with the oracle in test_gpu_kernels.py),
bit for bit."""

import ctypes

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


def sides_of(n):
    out = [n]
    while out[-1] > 3:
        out.append((out[-1] + 1) // 2)
    return out


def problem(n, seed, kind):
    """Iterate, right-hand side and screens of every level."""
    rng = np.random.default_rng(seed)
    x, b = rng.normal(size=(n, n, n)), rng.normal(size=(n, n, n)) * (n - 1) ** 2
    screen = np.where(rng.random((n, n, n)) < 0.1, rng.random((n, n, n)) * 30.0, 0.0)
    if kind == "zero":  # nothing anywhere but one source: exact zeros, then values down to 1e-300
        x[:], b[:], screen[:] = 0.0, 0.0, 0.0
        b[n // 2, n // 3, n // 2] = 1e-290
    elif kind == "dense":  # every diagonal differs; magnitudes over many decades
        screen = rng.random((n, n, n)) * 10.0 ** rng.integers(-12, 12, (n, n, n))
        b *= 10.0 ** rng.integers(-30, 30, (n, n, n))
    screens = [screen]
    for m in sides_of(n)[1:]:
        screens.append(np.ascontiguousarray(screens[-1][::2, ::2, ::2]) * 4.0)
    return x, b, screens


def on_device(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def reference(L, x, b, screens, pw, pre, post, cycles):
    s = torch.cuda.current_stream().cuda_stream
    ws = torch.empty(1 << 16, dtype=torch.uint8, device="cuda")
    norm = torch.empty(1, dtype=torch.float64, device="cuda")
    ok = lambda status: (_ for _ in ()).throw(AssertionError(L.pb_last_error().decode())) if status else None

    def cycle(sol, rhs, level):
        n, scr = sol.shape[0], screens[level]
        if n <= 3:
            ok(L.pb_relax_f64(sol.data_ptr(), rhs.data_ptr(), scr.data_ptr(), n, pw, 40, s))
            return
        ok(L.pb_relax_f64(sol.data_ptr(), rhs.data_ptr(), scr.data_ptr(), n, pw, pre, s))
        res = torch.empty_like(sol)
        ok(L.pb_residual_f64(sol.data_ptr(), rhs.data_ptr(), scr.data_ptr(), res.data_ptr(), n, pw, norm.data_ptr(),
                             ws.data_ptr(), ws.numel(), s))
        coarse = torch.empty_like(screens[level + 1])
        ok(L.pb_restrict_f64(res.data_ptr(), coarse.data_ptr(), n, s))
        e = torch.zeros_like(coarse)
        cycle(e, coarse, level + 1)
        ok(L.pb_prolong_add_f64(e.data_ptr(), sol.data_ptr(), n, s))
        ok(L.pb_relax_f64(sol.data_ptr(), rhs.data_ptr(), scr.data_ptr(), n, pw, post, s))

    for _ in range(cycles):
        cycle(x, b, 0)
    return x


def fused(L, x, b, screens, pw, pre, post, cycles):
    n = x.shape[0]
    sides = sides_of(n)
    grids, keep = [], []
    for l, m in enumerate(sides):
        # scratch and coarse iterates hold NaN: a value read before it is written shows
        nan = [torch.full((m, m, m), float("nan"), dtype=torch.float64, device="cuda") for _ in range(3)]
        keep.append(nan)
        grids += [x if l == 0 else nan[0], nan[1], b if l == 0 else nan[2], screens[l]]
    k = len(sides)
    ws = torch.empty(L.pb_residual_workspace_size(n) + 256, dtype=torch.uint8, device="cuda")
    status = L.pb_vcycles_f64(k, (ctypes.c_int64 * k)(*sides), (ctypes.c_void_p * (4 * k))(*[g.data_ptr() for g in grids]),
                              pw, pre, post, cycles, ws.data_ptr(), ws.numel(),
                              torch.cuda.current_stream().cuda_stream)
    assert status == 0, L.pb_last_error().decode()
    return x


@pytest.mark.parametrize("kind", ["shell", "dense", "zero"])
@pytest.mark.parametrize("n", [3, 5, 9, 17, 33, 65, 129])
def test_cycles_match_their_operators(L, n, kind):
    x, b, screens = problem(n, n, kind)
    b, screens = on_device(b), [on_device(v) for v in screens]
    want = reference(L, on_device(x), b, screens, 4.0, 3, 3, 2)
    got = fused(L, on_device(x), b, screens, 4.0, 3, 3, 2)
    assert torch.equal(got.view(torch.int64), want.view(torch.int64))
