"""The autotuner times the passes that the solver runs, with the occupancy words of a
sampled surface (prolongation and both FCG passes)."""

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

PASSES = {"pb_prolong_fac": 3, "pb_fcg_direction": 5, "pb_fcg_update": 7}  # the occupancy words' argument


class Recorder:
    """The library, its calls of the passes noted by name with their occupancy argument."""

    def __init__(self, library):
        self.library, self.calls = library, {}

    def __getattr__(self, name):
        fn = getattr(self.library, name)
        at = next((k for start, k in PASSES.items() if name.startswith(start)), None)
        if at is None:
            return fn

        def call(*args):
            self.calls.setdefault(name, set()).add(args[at])
            return fn(*args)

        return call


@pytest.mark.parametrize("n", [33, 65])
def test_solver_passes_are_timed(n, monkeypatch):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mojo_poissonrecon_b200 import _native, solver32, tune

    lib = _native.lib()
    rhs, screen = tune.shell_system(n, torch.device("cuda"))
    assert rhs.dtype == screen.dtype == torch.float64 and bool((rhs[screen != 0] != 0).all())
    assert 0 < int((screen != 0).sum()) < 0.15 * n ** 3
    solved, tuned = Recorder(lib), Recorder(lib)
    lib.pb_tune_clear()
    try:
        with monkeypatch.context() as m:
            m.setattr(_native, "lib", lambda: solved)
            m.setattr(solver32, "EAGER_LOOP", True)
            solver32.RefinedEngine(n, 4.0, rhs.device).solve(rhs, screen, 1e-8, 5)
        with monkeypatch.context() as m:
            m.setattr(_native, "lib", lambda: tuned)
            tune.autotune(n, params=(tune.PROLONG_PLANES, tune.FCG_DIRECTION_VARIANT, tune.FCG_UPDATE_VARIANT),
                          repeats=1, write=False)
    finally:
        lib.pb_tune_clear()
    assert set(solved.calls) == set(tuned.calls) and len(tuned.calls) == 3
    for name, words in tuned.calls.items():
        assert words and None not in words, name
