"""The tuning cache's entries belong to one set of kernels: those of another are not applied (no GPU)."""

from mojo_poissonrecon_b200 import tune


def test_choices_for_other_kernels_are_not_applied(tmp_path, monkeypatch):
    from mojo_poissonrecon_b200 import _native

    lib = _native.lib()
    path = str(tmp_path / "tune.json")
    entry = {"fcg_direction_variant": {"best": 1}, "prolong_planes": {"best": 4}}
    # keys without a kernel count (1: 6 resident blocks then, 4 now), of earlier and of later kernels
    stale = {"GPU X|n=257": entry}
    for kernels in (tune.KERNELS - 1, tune.KERNELS + 1):
        with monkeypatch.context() as m:
            m.setattr(tune, "KERNELS", kernels)
            stale[tune.cache_key("GPU X", 257)] = entry
    assert len(stale) == 3
    tune.store_cache(stale, path)
    lib.pb_tune_clear()
    try:
        assert tune.apply(lib, "GPU X", 257, path) == {}
        assert lib.pb_tune_get(tune.FCG_DIRECTION_VARIANT, 257) == 0
        tune.store_cache({**stale, tune.cache_key("GPU X", 257): entry}, path)
        assert tune.apply(lib, "GPU X", 257, path) == {"fcg_direction_variant": 1, "prolong_planes": 4}
    finally:
        lib.pb_tune_clear()
