"""Autotuner of the tile kernels.

For one (n, nst, K) it times, with the library's phase events, the energy
tiles over (ket-chunk width LC_e, register variant minb_e) and the gradient
tiles over (LC_g, minb_g) -- the two are independent -- and keeps the fastest
of each.  Results are cached in a JSON file keyed by GPU name, n, nst, a K bucket
(powers of two) and the kernels' sources, so a run pays for tuning once and not with
choices timed on other kernels.

The search space:
  LC_e   ket chunk of an energy tile (kets per warp per tile)
  LC_g   ket chunk of a gradient tile (also sets the partial-buffer depth)
  minw   minimum resident warps per SM the kernel is compiled for (one warp
         per block): 8 -> up to 255 registers per thread, 12 -> 168, 16 -> 128,
         20 -> 96 (the register file is split between the four schedulers, so
         these are the only distinct budgets).  Energy tiles that several warps
         share (few tiles, energy_warps) have one kernel whatever minb_e says, and the
         ordered gradient is compiled for 8 and 12 warps, and 16 for n <= 3: only
         these are tried
  sym    gradient pass over unordered pairs (bra and ket gradient per term,
         when the symmetry set is closed under inverse) instead of ordered
         pairs, with its own ket chunk lc_s and variant minw_s; sym = 2 fuses
         it with the energy pass (one pass for H, S and both gradients), kept
         when its total beats the best separate energy + gradient passes
  npc    splits of the symmetry terms per tile of the fused pass (one-warp
         variants): tried when the basis has few tiles (SPLIT_TILES), where each
         tile's chain of LC x nst terms, not the GPU's width, sets the time
"""
from __future__ import annotations

import ctypes
import functools
import glob
import hashlib
import json
import os

import numpy as np
import torch

from . import _lib
from .engine import Engine

CACHE = os.environ.get("NECG_TUNE_CACHE", os.path.join(os.path.dirname(os.path.abspath(__file__)), "tune_cache.json"))

LC_E = (1, 2, 4, 8, 16)
LC_G = (4, 8, 16, 32, 64)
MINB = (8, 12, 16, 20)
LC_S = (1, 2, 4, 8, 16)       # kets per tile of the symmetric gradient pass
MINW_SYM = (8, 12)
MINW_FUSED = (8, 12, 16, 108, 112, 118, 122, 248, 232, 216)
SPLITS = (1, 2, 3, 4, 6, 8, 12, 24)
SPLIT_TILES = 2048  # try splits below this many fused tiles
SPLIT_SLOTS = 8192  # and at most this many (tile, split) slots: 3 and more rounds of 16 warps on each of 148 SMs
# 100 + w: ket records re-read at each use (118 / 122: staged in shared memory,
# 8 / 12 warps); 248 / 232 / 216: blocks of 8 / 12 / 16 warps with bras and ket
# records in shared memory (the library also takes the codes 208 .. 268 of earlier block
# variants and runs the one with the same number of warps); a variant whose
# shared memory does not fit for n is refused by necg_set_symmetric and skipped


def fused_tiles(K: int, lc: int) -> int:
    """Tiles (32-row block, chunk of lc kets) over the lower triangle of K."""
    return sum((K - 1 - 32 * b) // lc + 1 for b in range((K + 31) // 32))


def splits(K: int, lc: int, nst: int) -> list[int]:
    """The numbers of splits tried for one-warp tiles of chunk lc."""
    tiles = fused_tiles(K, lc)
    return [s for s in SPLITS if s == 1 or (s <= nst and tiles < SPLIT_TILES and s * tiles <= SPLIT_SLOTS)]


def energy_warps(nst: int, tiles: int, sms: int) -> int:
    """Warps that share an energy tile (csrc/necg_tiles.h)."""
    w = 1
    while 2 * w <= nst and w < 8 and tiles * w < 12 * sms:
        w *= 2
    return w


def separate_candidates(n: int, nst: int, K: int, sms: int) -> list[tuple]:
    """(minb, lc_e, lc_g, energy, grad) of the separate passes' search: whether the energy
    and the gradient kernel of this setting are ones that no earlier setting ran."""
    out = []
    for minb in MINB:
        for lc_e, lc_g in zip(LC_E, LC_G):
            energy = minb == MINB[0] or energy_warps(nst, fused_tiles(K, lc_e), sms) == 1
            grad = minb in ((8, 12, 16) if n <= 3 else (8, 12))
            if energy or grad:
                out.append((minb, lc_e, lc_g, energy, grad))
    return out


@functools.cache
def kernels() -> str:
    """A digest of the kernels' sources."""
    h = hashlib.sha256()
    for f in sorted(glob.glob(os.path.join(os.path.dirname(os.path.abspath(__file__)), "csrc", "*"))):
        with open(f, "rb") as fh:
            h.update(os.path.basename(f).encode() + b"\0" + fh.read())
    return h.hexdigest()[:12]


def _bucket(K: int) -> int:
    b = 16
    while b < K:
        b *= 2
    return b


def _key(n: int, nst: int, K: int) -> str:
    name = torch.cuda.get_device_name() if torch.cuda.is_available() else "cpu"
    return f"{name}|n{n}|nst{nst}|K{_bucket(K)}|{kernels()}"


def load_cache() -> dict:
    try:
        with open(CACHE) as fh:
            return json.load(fh)
    except (OSError, ValueError):
        return {}


def save_cache(cache: dict) -> None:
    tmp = f"{CACHE}.{os.getpid()}.tmp"  # ranks of one node may save at the same time
    with open(tmp, "w") as fh:
        json.dump(cache, fh, indent=1, sort_keys=True)
    os.replace(tmp, CACHE)


def _phase_times(eng: Engine, x: torch.Tensor, K: int, reps: int) -> np.ndarray:
    L = eng.L
    g = torch.empty_like(x)
    f = torch.empty(1, dtype=torch.float64, device=x.device)
    buf = (ctypes.c_double * 5)()
    out = []
    for _ in range(reps):
        _lib.check(L.necg_outprod(eng.h, K, x.data_ptr(), f.data_ptr(), g.data_ptr(), None, None,
                                  torch.cuda.current_stream().cuda_stream), "necg_outprod")
        _lib.check(L.necg_phase_ms(eng.h, buf), "necg_phase_ms")
        out.append(list(buf))
    return np.array(out)


def tune(eng: Engine, x, K: int, reps: int = 3, report: bool = False) -> dict:
    """Time every candidate on this engine and input; returns the best setting."""
    L = eng.L
    x = eng._tensor(x)
    _lib.check(L.necg_profile(eng.h, 1), "necg_profile")
    L.necg_set_symmetric(eng.h, 0, 4, 8)
    rows = []
    best_e = (float("inf"), None)
    best_g = (float("inf"), None)
    sms = torch.cuda.get_device_properties(eng.device).multi_processor_count
    for minb, lc_e, lc_g, energy, grad in separate_candidates(eng.n, eng.nst, K, sms):
        _lib.check(L.necg_set_tiles(eng.h, lc_e, lc_g), "necg_set_tiles")
        _lib.check(L.necg_set_variant(eng.h, minb, minb), "necg_set_variant")
        _phase_times(eng, x, K, 1)  # warm-up (also builds the energy tile list)
        t = _phase_times(eng, x, K, reps).min(axis=0)
        e_ms, g_ms = float(t[1]), float(t[3] + t[4])
        rows.append({"minb": minb, "lc_e": lc_e, "lc_g": lc_g, "energy_ms": e_ms, "grad_ms": g_ms})
        if energy and e_ms < best_e[0]:
            best_e = (e_ms, (lc_e, minb))
        if grad and g_ms < best_g[0]:
            best_g = (g_ms, (lc_g, minb))
    res = {"lc_e": best_e[1][0], "minb_e": best_e[1][1], "lc_g": best_g[1][0], "minb_g": best_g[1][1],
           "energy_ms": best_e[0], "grad_ms": best_g[0], "sym": 0, "lc_s": 4, "minw_s": 8}
    # the symmetric gradient pass (unordered pairs), when the symmetry set allows it
    if L.necg_set_symmetric(eng.h, 1, 4, 8) == _lib.NECG_OK:
        _lib.check(L.necg_set_tiles(eng.h, res["lc_e"], res["lc_g"]), "necg_set_tiles")
        _lib.check(L.necg_set_variant(eng.h, res["minb_e"], res["minb_g"]), "necg_set_variant")
        for minw in MINW_SYM:
            for lc in LC_S:
                _lib.check(L.necg_set_symmetric(eng.h, 1, lc, minw), "necg_set_symmetric")
                _phase_times(eng, x, K, 1)
                t = _phase_times(eng, x, K, reps).min(axis=0)
                g_ms = float(t[3] + t[4])
                rows.append({"sym": 1, "minw": minw, "lc_s": lc, "grad_ms": g_ms})
                if g_ms < res["grad_ms"]:
                    res.update(grad_ms=g_ms, sym=1, lc_s=lc, minw_s=minw)
        # fused energy + symmetric gradient pass: phase 1 is the whole pair pass
        best_sep = res["energy_ms"] + res["grad_ms"]
        fused = None
        for minw in MINW_FUSED:
            for lc in LC_S:
                if L.necg_set_symmetric(eng.h, 2, lc, minw) != _lib.NECG_OK:
                    continue
                for npc in splits(K, lc, eng.nst) if minw < 200 else [1]:
                    _lib.check(L.necg_set_splits(eng.h, npc), "necg_set_splits")
                    _phase_times(eng, x, K, 1)
                    t = _phase_times(eng, x, K, reps).min(axis=0)
                    tot = float(t[1] + t[3] + t[4])
                    rows.append({"sym": 2, "minw": minw, "lc_s": lc, "npc": npc, "total_ms": tot})
                    if tot < best_sep and (fused is None or tot < fused[0]):
                        fused = (tot, lc, minw, npc)
                L.necg_set_splits(eng.h, 1)
        if fused is not None:
            res.update(sym=2, lc_s=fused[1], minw_s=fused[2], npc=fused[3], fused_ms=fused[0])
    if report:
        res["table"] = rows
    apply(eng, res)
    return res


def apply(eng: Engine, cfg: dict) -> None:
    _lib.check(eng.L.necg_set_tiles(eng.h, int(cfg["lc_e"]), int(cfg["lc_g"])), "necg_set_tiles")
    _lib.check(eng.L.necg_set_variant(eng.h, int(cfg["minb_e"]), int(cfg["minb_g"])), "necg_set_variant")
    sym = int(cfg.get("sym", 0))
    rc = eng.L.necg_set_symmetric(eng.h, sym, int(cfg.get("lc_s", 4)), int(cfg.get("minw_s", 8)))
    if rc != _lib.NECG_OK and sym:
        _lib.check(rc, "necg_set_symmetric")
    _lib.check(eng.L.necg_set_splits(eng.h, min(int(cfg.get("npc", 1)), eng.nst)), "necg_set_splits")


def tuned(eng: Engine, x, K: int, retune: bool = False) -> dict:
    """Apply the cached setting for (GPU, n, nst, K bucket) of these kernels, tuning on a
    miss; settings of other kernels leave the cache with the next one that is kept."""
    cache = load_cache()
    key = _key(eng.n, eng.nst, K)
    if key in cache and not retune:
        apply(eng, cache[key])
        return cache[key]
    res = tune(eng, x, K)
    cache = {k: v for k, v in cache.items() if k.endswith("|" + kernels())}
    cache[key] = {k: v for k, v in res.items() if k != "table"}
    try:
        save_cache(cache)
    except OSError:
        pass
    return cache[key]
