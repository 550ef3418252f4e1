"""The single-block cycle from each side it may start at, with unequal, single and no sweeps.

Tolerance as for the other FP32 cycles: 1e-4 of the largest value (each pass rounds its 27
products to 2^-24 of values of that size, and the operators' condition on at most 729
nodes magnifies them by less than 1e3)."""

import ctypes

import numpy as np
import pytest

import mg_reference as mg
from padded import from_padded, to_padded
from test_gpu_mg27 import gpu_hierarchy, gpu_ops, shell_screen

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def L():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mojo_poissonrecon_b200 import _native

    return _native.lib()


@pytest.fixture(scope="module")
def hierarchy(L):
    h = gpu_hierarchy(33, shell_screen(33, 3))
    return h, gpu_ops(L, h)


def restated(ops, ws, sizes, level, rhs, pre, post, inner):
    n = sizes[level]
    if n == 3:
        return np.linalg.solve(ops[level].toarray(), rhs.ravel()).reshape(n, n, n)
    e = np.zeros((n, n, n))
    for k in range(pre):
        e = mg.relax(ops[level], e, rhs, n)
    coarse, _ = mg.residual_restrict(ops[level], ws[level], e, rhs, n)
    e = mg.prolong(e, restated(ops, ws, sizes, level + 1, coarse, inner, inner, inner), ws[level], n)
    for k in range(post):
        e = mg.relax(ops[level], e, rhs, n)
    return e


@pytest.mark.parametrize("sweeps", [(1, 1, 1), (1, 2, 1), (0, 1, 2), (2, 0, 0), (3, 3, 2)])
@pytest.mark.parametrize("side", [9, 5, 3])
def test_cycle_from_each_side(L, hierarchy, side, sweeps):
    h, (ops, ws, sizes) = hierarchy
    s = torch.cuda.current_stream().cuda_stream
    k = sizes.index(side)
    tail = h.levels[k:]
    count, sides = len(tail), (ctypes.c_int64 * len(tail))(*(lv.n for lv in tail))
    ptrs = lambda ts: (ctypes.c_void_p * count)(*(t.data_ptr() for t in ts))
    image = torch.zeros(L.pb_coarse27_image_size(count, sides) // 4, dtype=torch.float32, device="cuda")
    assert L.pb_coarse27_image_f32(count, sides, ptrs([lv.coef for lv in tail]), ptrs([lv.invD for lv in tail]),
                                   ptrs([lv.weights for lv in tail]), h.inverse.data_ptr(), image.data_ptr(),
                                   image.numel() * 4, s) == 0, L.pb_last_error().decode()
    rhs = np.random.default_rng(side).normal(size=(side,) * 3).astype(np.float32).astype(np.float64)
    e = torch.zeros_like(tail[0].ea)
    assert L.pb_coarse27_cycle_f32(count, sides, image.data_ptr(), to_padded(L, rhs).data_ptr(), e.data_ptr(), *sweeps,
                                   s) == 0, L.pb_last_error().decode()
    got, want = from_padded(L, e, side), restated(ops, ws, sizes, k, rhs, *sweeps)
    assert np.abs(got - want).max() <= 1e-4 * np.abs(want).max()
