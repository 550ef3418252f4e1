"""Device-resident screened-Poisson multigrid.

Reference: python/mojo_poissonrecon/core.py:141-193 (_v_cycle) and :267-296
(hierarchy, cycle loop, final residual).  The reference keeps one NumPy grid
per level and drives the native kernels level by level; here the hierarchy
lives in HBM as torch tensors, by colour from side 33 up, and all cycles of a solve
are queued on one CUDA stream by one library call (pb_vcycles_f64).

Two solve modes:

* ``precision="fp64"`` — the reference algorithm: V(3,3) cycles with
  red-black Gauss-Seidel, boundary-normalised full weighting, trilinear
  prolongation and 40 sweeps on the 3^3 grid, all in FP64, from the initial
  guess 0.5.  With ``tol=None`` it runs exactly ``cycles`` cycles and is
  bit-identical to the reference.  With ``tol`` it repeats cycles until the
  relative residual ||b - A x||_2 / ||b||_2 <= tol.
* ``precision="fp32_refined"`` — defect correction: the FP64 residual of the
  FP64 iterate drives one FP32 V-cycle on A e = r from e = 0, and x += e in
  FP64, until the FP64 relative residual reaches ``tol``.  (Implemented in
  solver32.py.)
"""

from __future__ import annotations

import ctypes
from dataclasses import dataclass, field

import torch

from . import _native as nat


def level_sizes(n: int) -> list[int]:
    """Grid sides of the hierarchy: n, (n+1)/2, ... down to 3 (core.py:267-269)."""
    sizes = [n]
    while sizes[-1] > 3:
        sizes.append((sizes[-1] + 1) // 2)
    return sizes


@dataclass
class SolveStats:
    cycles: int = 0
    residual_norm: float = float("nan")
    rhs_norm: float = float("nan")
    history: list = field(default_factory=list)

    @property
    def relative_residual(self) -> float:
        if not self.rhs_norm > 0:
            return 0.0 if self.residual_norm == 0 else float("inf")
        return self.residual_norm / self.rhs_norm


class Hierarchy64:
    """FP64 levels of one solve: the iterate and right-hand side of each, in the
    library's layout (pb_vcycle_level_size), and its dense screen."""

    def __init__(self, screen: torch.Tensor, rhs: torch.Tensor, point_weight: float, workspace: nat.Workspace,
                 init: float = 0.5):  # core.py:270
        self.device = screen.device
        self.pw = float(point_weight)
        self.sizes = level_sizes(screen.shape[0])
        self.ws = workspace
        self.lib = nat.lib()
        self.stream = nat.stream_handle()
        L, s = self.lib, self.stream
        self.screens = [screen]
        for n in self.sizes[1:]:
            coarse = torch.empty((n, n, n), dtype=torch.float64, device=self.device)
            fine = self.screens[-1]
            nat.check(L.pb_restrict_f64(fine.data_ptr(), coarse.data_ptr(), fine.shape[0], s), "restrict")
            nat.check(L.pb_scale_f64(coarse.data_ptr(), coarse.numel(), 4.0, s), "scale")
            self.screens.append(coarse)
        self.levels = []
        for n in self.sizes:
            doubles, flags = ctypes.c_int64(), ctypes.c_int64()
            nat.check(L.pb_vcycle_level_size(n, ctypes.byref(doubles), ctypes.byref(flags)), "level size")
            self.levels.append((torch.empty(doubles.value, dtype=torch.float64, device=self.device),
                                torch.empty(doubles.value, dtype=torch.float64, device=self.device),
                                torch.empty(max(flags.value, 1), dtype=torch.uint8, device=self.device)))
        self.norm = torch.empty(1, dtype=torch.float64, device=self.device)
        k = len(self.sizes)
        self._sides = (ctypes.c_int64 * k)(*self.sizes)
        self._grids = (ctypes.c_void_p * (4 * k))(*[t.data_ptr() for level, scr in zip(self.levels, self.screens)
                                                    for t in (*level, scr)])
        nat.check(L.pb_vcycle_setup_f64(k, self._sides, self._grids, rhs.data_ptr(), init, s), "V-cycle set-up")

    def v_cycles(self, count: int, pre: int = 3, post: int = 3) -> None:
        """core.py:141-193, `count` times in one library call; the finest
        ||b - A x||_2 after them into `norm`."""
        ptr, size = self.ws.get(self.lib.pb_vcycle_workspace_size(self.sizes[0]))
        nat.check(self.lib.pb_vcycles_f64(len(self.sizes), self._sides, self._grids, self.pw, pre, post, count,
                                          self.norm.data_ptr(), ptr, size, self.stream), "V-cycles")

    def field(self) -> torch.Tensor:
        """The finest iterate as a dense grid; the levels' other arrays are released."""
        n = self.sizes[0]
        iterate = self.levels[0][0]
        self.levels = self._grids = None  # the right-hand side's memory holds the grid where it is large
        out = torch.empty((n, n, n), dtype=torch.float64, device=self.device)
        nat.check(self.lib.pb_vcycle_field_f64(n, iterate.data_ptr(), out.data_ptr(), self.stream), "V-cycle field")
        return out


def norm(values: torch.Tensor, workspace: nat.Workspace, out: torch.Tensor) -> torch.Tensor:
    L = nat.lib()
    ptr, size = workspace.get(1 << 16)  # per-block partial sums: at most 148*16 doubles
    nat.check(L.pb_norm_f64(values.data_ptr(), values.numel(), out.data_ptr(), ptr, size, nat.stream_handle()),
              "norm")
    return out


def solve_fp64(rhs: torch.Tensor, screen: torch.Tensor, point_weight: float, workspace: nat.Workspace, *,
               cycles: int = 4, tol: float | None = None, max_cycles: int = 200,
               has_points: bool = True) -> tuple[torch.Tensor, SolveStats]:
    """The reference's FP64 solve (core.py:267-296) on device grids.

    Returns the level-0 solution and stats; stats.residual_norm is the absolute
    final ||rhs - A x||_2 as the reference reports it."""
    stats = SolveStats()
    h = Hierarchy64(screen, rhs, point_weight, workspace, 0.5 if has_points else 0.0)
    if not has_points:
        h.v_cycles(0)
    elif tol is None:
        h.v_cycles(cycles)
        stats.cycles = cycles
    else:
        rhs_norm = norm(rhs, workspace, torch.empty(1, dtype=torch.float64, device=rhs.device))
        stats.rhs_norm = float(rhs_norm.item())
        target = tol * stats.rhs_norm
        if max_cycles < 1:
            h.v_cycles(0)
        while stats.cycles < max_cycles:
            h.v_cycles(1)
            stats.cycles += 1
            r = float(h.norm.item())
            stats.history.append(r)
            if r <= target:
                break
    stats.residual_norm = float(h.norm.item())  # core.py:289-296: absolute final residual norm
    if stats.rhs_norm != stats.rhs_norm:  # nan: not computed yet
        rhs_norm = norm(rhs, workspace, torch.empty(1, dtype=torch.float64, device=rhs.device))
        stats.rhs_norm = float(rhs_norm.item())
    return h.field(), stats
