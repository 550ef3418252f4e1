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
    """Right-hand side and screens of every level."""
    rng = np.random.default_rng(seed)
    b = rng.normal(size=(n, n, n)) * (n - 1) ** 2
    screen = np.where(rng.random((n, n, n)) < 0.1, rng.random((n, n, n)) * 30.0, 0.0)
    if kind == "zero":  # nothing anywhere but one source: exact zeros, then values down to 1e-300
        b[:], screen[:] = 0.0, 0.0
        b[n // 2, n // 3, n // 2] = 1e-290
    elif kind == "dense":  # every diagonal differs; magnitudes over many decades
        screen = rng.random((n, n, n)) * 10.0 ** rng.integers(-12, 12, (n, n, n))
        b *= 10.0 ** rng.integers(-30, 30, (n, n, n))
    screens = [screen]
    for m in sides_of(n)[1:]:
        screens.append(np.ascontiguousarray(screens[-1][::2, ::2, ::2]) * 4.0)
    return b, screens


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


def fused(L, x, b, screens, pw, pre, post, cycles, norm=None):
    """The same cycles in one call; x: the constant that the iterate starts at."""
    n = b.shape[0]
    sides = sides_of(n)
    grids, keep = [], []
    for m, scr in zip(sides, screens):
        doubles, flags = ctypes.c_int64(), ctypes.c_int64()
        assert L.pb_vcycle_level_size(m, ctypes.byref(doubles), ctypes.byref(flags)) == 0
        # NaN everywhere: a value read before it is written shows
        level = [torch.full((doubles.value,), float("nan"), dtype=torch.float64, device="cuda") for _ in range(2)]
        level += [torch.full((max(flags.value, 1),), 255, dtype=torch.uint8, device="cuda"), scr]
        keep.append(level)
        grids += [t.data_ptr() for t in level]
    k = len(sides)
    args = (k, (ctypes.c_int64 * k)(*sides), (ctypes.c_void_p * (4 * k))(*grids))
    s = torch.cuda.current_stream().cuda_stream
    ws = torch.empty(L.pb_vcycle_workspace_size(n), dtype=torch.uint8, device="cuda")
    out = torch.empty_like(b)
    for status in (L.pb_vcycle_setup_f64(*args, b.data_ptr(), x, s),
                   L.pb_vcycles_f64(*args, pw, pre, post, cycles, norm.data_ptr() if norm is not None else None,
                                    ws.data_ptr(), ws.numel(), s),
                   L.pb_vcycle_field_f64(n, keep[0][0].data_ptr(), out.data_ptr(), s)):
        assert status == 0, L.pb_last_error().decode()
    return out


@pytest.mark.parametrize("kind", ["shell", "dense", "zero"])
@pytest.mark.parametrize("n", [3, 5, 9, 17, 33, 65, 129])
def test_cycles_match_their_operators(L, n, kind):
    b, screens = problem(n, n, kind)
    b, screens = on_device(b), [on_device(v) for v in screens]
    start = 0.0 if kind == "zero" else 0.5
    pre, post = (1, 2) if kind == "dense" else (3, 3)
    want = reference(L, torch.full_like(b, start), b, screens, 4.0, pre, post, 2)
    norm = torch.empty(2, dtype=torch.float64, device="cuda")
    got = fused(L, start, b, screens, 4.0, pre, post, 2, norm)
    assert torch.equal(got.view(torch.int64), want.view(torch.int64))
    ws = torch.empty(1 << 16, dtype=torch.uint8, device="cuda")
    assert L.pb_residual_f64(want.data_ptr(), b.data_ptr(), screens[0].data_ptr(), torch.empty_like(b).data_ptr(), n, 4.0,
                             norm.data_ptr() + 8, ws.data_ptr(), ws.numel(),
                             torch.cuda.current_stream().cuda_stream) == 0
    ours, theirs = norm.tolist()
    assert abs(ours - theirs) <= 1e-13 * theirs  # two trees of the same squares: n^3 2^-53 / 2 at the very most
