"""The tuner's search and its cache, without a GPU."""
import json

import pytest

from nbo_correlatedgaussians_b200 import autotune


@pytest.mark.parametrize("n,nst", [(2, 2), (3, 4), (5, 24), (5, 1)])
@pytest.mark.parametrize("K", [5, 96, 301, 2048])
def test_no_kernel_is_timed_under_two_names(n, nst, K):
    """Energy kernels are told apart by (chunk, warps per tile, registers if one warp has
    the tile), gradient kernels by (chunk, registers)."""
    energy, grad = [], []
    for minb, lc_e, lc_g, e, g in autotune.separate_candidates(n, nst, K, 148):
        warps = autotune.energy_warps(nst, autotune.fused_tiles(K, lc_e), 148)
        if e:
            energy.append((lc_e, warps, minb if warps == 1 else None))
        if g:
            grad.append((lc_g, minb))
    assert len(set(energy)) == len(energy) and {x[0] for x in energy} == set(autotune.LC_E)
    assert sorted(grad) == sorted((lc, m) for lc in autotune.LC_G for m in ((8, 12, 16) if n <= 3 else (8, 12)))


def test_splits_are_bounded():
    for K in (1, 12, 96, 300, 1000):
        for lc in autotune.LC_S:
            s = autotune.splits(K, lc, 24)
            assert s[0] == 1 and max(s) * autotune.fused_tiles(K, lc) <= max(autotune.SPLIT_SLOTS, autotune.fused_tiles(K, lc))
    assert autotune.splits(12, 1, 24)[-1] == 24 and autotune.splits(12, 1, 4)[-1] == 4


def test_cache_entries_of_other_kernels_are_not_used(tmp_path, monkeypatch):
    monkeypatch.setattr(autotune, "CACHE", str(tmp_path / "cache.json"))
    tuned = {"lc_e": 2, "minb_e": 8, "lc_g": 4, "minb_g": 8, "sym": 2, "lc_s": 2, "minw_s": 248}
    applied = []
    monkeypatch.setattr(autotune, "apply", lambda eng, cfg: applied.append(cfg))
    monkeypatch.setattr(autotune, "tune", lambda eng, x, K: dict(tuned, table=[1]))

    class Eng:
        n, nst = 5, 24

    key = autotune._key(5, 24, 100)
    assert key.endswith(autotune.kernels())
    old = {key.rsplit("|", 1)[0]: dict(tuned, minw_s=268), key.rsplit("|", 1)[0] + "|0123456789ab": dict(tuned, minw_s=268)}
    (tmp_path / "cache.json").write_text(json.dumps(old))
    assert autotune.tuned(Eng(), None, 100) == tuned and not applied
    assert list(json.loads((tmp_path / "cache.json").read_text())) == [key]
    assert autotune.tuned(Eng(), None, 100) == tuned and applied == [tuned]
