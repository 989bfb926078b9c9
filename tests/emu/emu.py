"""TEST INFRASTRUCTURE: ctypes wrappers of the host emulators of the kernels:
libnecg_emu.so runs the per-thread bodies of necg_lanes.cuh tile by tile and lane by
lane, libnecg_simt.so the warps and blocks of necg_device.cuh thread by thread."""
from __future__ import annotations

import ctypes
import os
import shutil
import subprocess

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "necg_emu.cu")
LIB = os.path.join(HERE, "libnecg_emu.so")
CSRC = os.path.join(os.path.dirname(os.path.dirname(HERE)), "nbo_correlatedgaussians_b200", "csrc")
_lib = None


def build() -> str:
    deps = [SRC] + [os.path.join(CSRC, f) for f in ("necg_lanes.cuh", "necg_math.cuh", "necg_tiles.h", "necg_hostscalar.cuh")]
    if os.path.exists(LIB) and all(os.path.getmtime(LIB) >= os.path.getmtime(d) for d in deps):
        return LIB
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    tmp = f"{LIB}.{os.getpid()}.tmp"  # processes started together may build at the same time
    subprocess.check_call([nvcc, "-O1", "-std=c++17", "-Xcompiler", "-fPIC", "--shared",
                           "-Wno-deprecated-gpu-targets", "-o", tmp, SRC])
    os.replace(tmp, LIB)
    return LIB


SIMT_LIB = os.path.join(HERE, "libnecg_simt.so")
_simt = None


def simt():
    """The emulation of the passes over unordered pairs (simt_emu.cpp)."""
    global _simt
    if _simt is None:
        deps = [os.path.join(HERE, f) for f in ("simt_emu.cpp", "simt.h", os.path.join("stub", "cuda_runtime.h"))]
        deps += [os.path.join(CSRC, f) for f in ("necg_device.cuh", "necg_lanes.cuh", "necg_math.cuh", "necg_tiles.h", "necg_maps.h")]
        if not os.path.exists(SIMT_LIB) or any(os.path.getmtime(SIMT_LIB) < os.path.getmtime(d) for d in deps):
            tmp = f"{SIMT_LIB}.{os.getpid()}.tmp"
            subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-U_FORTIFY_SOURCE", "-Wno-unknown-pragmas",
                                   "-I", os.path.join(HERE, "stub"), "-o", tmp, deps[0]])
            os.replace(tmp, SIMT_LIB)
        _simt = ctypes.CDLL(SIMT_LIB)
    return _simt


def _problem(p):
    """The arguments every entry of the emulation starts with (and the arrays behind them)."""
    c = _consts(p)
    return [ctypes.c_int(p.n), ctypes.c_int(p.nst), ctypes.c_int(p.K), ctypes.c_double(p.efs),
            *[ctypes.c_void_p(_p(a)) for a in c]], c


def lib():
    global _lib
    if _lib is None:
        _lib = ctypes.CDLL(build())
    return _lib


def _p(a):
    return a.ctypes.data


def _consts(p):
    arrs = [np.ascontiguousarray(a, dtype=np.float64) for a in (p.mass, p.ncv, p.scvv, p.sml, p.sms)]
    return arrs


def outprod(p, lc_e=4, lc_g=4):
    L = lib()
    c = _consts(p)
    x = np.ascontiguousarray(p.x)
    f = np.zeros(1)
    g = np.zeros(x.size)
    H = np.zeros((p.K, p.K))
    S = np.zeros((p.K, p.K))
    fn = L.emu_outprod
    fn.restype = ctypes.c_int
    rc = fn(ctypes.c_int(p.n), ctypes.c_int(p.nst), ctypes.c_int(p.K), ctypes.c_double(p.efs),
            *[ctypes.c_void_p(_p(a)) for a in c], ctypes.c_void_p(_p(x)), ctypes.c_int(lc_e), ctypes.c_int(lc_g),
            ctypes.c_void_p(_p(f)), ctypes.c_void_p(_p(g)), ctypes.c_void_p(_p(H)), ctypes.c_void_p(_p(S)))
    return rc, float(f[0]), g, H, S


def _pass(p, mode, variant, lc, npc, sms):
    args, keep = _problem(p)
    x = np.ascontiguousarray(p.x)
    f, g = np.zeros(1), np.full(x.size, np.nan)
    H, S = np.zeros((p.K, p.K)), np.zeros((p.K, p.K))
    rc = simt().simt_outprod(*args, ctypes.c_void_p(_p(x)), *[ctypes.c_int(v) for v in (mode, variant, lc, npc, sms)],
                             *[ctypes.c_void_p(_p(a)) for a in (f, g, H, S)])
    return rc, float(f[0]), g, H, S


def outprod_sym(p, lc_e=4, lc_s=4, variant=2, sms=148):
    """The symmetric gradient pass (unordered pairs, E known) emulated on the host.
    variant: 0 one-warp tiles, 1 with ket records re-read, 2 staged, 8 / 12 / 16 blocks of
    that many warps on a GPU of `sms` SMs."""
    return _pass(p, 1, variant, lc_s, 1, sms)


def outprod_fused(p, lc_s=4, variant=2, npc=1, sms=148):
    """The fused energy + symmetric gradient pass emulated on the host; npc: splits of
    the symmetry terms of one-warp tiles."""
    return _pass(p, 2, variant, lc_s, npc, sms)


def rrms(p, terms):
    L = lib()
    c = _consts(p)
    t = np.ascontiguousarray(terms, dtype=np.int32).reshape(-1, 5)
    out = np.zeros((len(t), 2))
    fn = L.emu_rrms
    fn.restype = ctypes.c_int
    rc = fn(ctypes.c_int(p.n), ctypes.c_int(p.nst), ctypes.c_int(p.K), ctypes.c_double(p.efs),
            *[ctypes.c_void_p(_p(a)) for a in c], ctypes.c_void_p(_p(np.ascontiguousarray(p.iv))),
            ctypes.c_int(len(t)), ctypes.c_void_p(_p(t)), ctypes.c_void_p(_p(out)))
    return rc, out


def dipole(p, lc=2):
    L = lib()
    c = _consts(p)
    comps = np.zeros(3 * p.n)
    dip = np.zeros(3)
    fn = L.emu_dipole
    fn.restype = ctypes.c_int
    rc = fn(ctypes.c_int(p.n), ctypes.c_int(p.nst), ctypes.c_int(p.K), ctypes.c_double(p.efs),
            *[ctypes.c_void_p(_p(a)) for a in c], ctypes.c_void_p(_p(np.ascontiguousarray(p.iv))),
            ctypes.c_void_p(_p(np.ascontiguousarray(p.C))), ctypes.c_int(lc), ctypes.c_void_p(_p(comps)),
            ctypes.c_void_p(_p(dip)))
    return rc, comps, dip


def elements(p, terms):
    L = lib()
    c = _consts(p)
    t = np.ascontiguousarray(terms, dtype=np.int32).reshape(-1, 3)
    mat = np.zeros((len(t), 4))
    tg = np.zeros((len(t), p.blk))
    tgs = np.zeros((len(t), p.blk))
    fn = L.emu_elements
    fn.restype = ctypes.c_int
    rc = fn(ctypes.c_int(p.n), ctypes.c_int(p.nst), ctypes.c_int(p.K), ctypes.c_double(p.efs),
            *[ctypes.c_void_p(_p(a)) for a in c], ctypes.c_void_p(_p(np.ascontiguousarray(p.iv))),
            ctypes.c_int(len(t)), ctypes.c_void_p(_p(t)), ctypes.c_void_p(_p(mat)), ctypes.c_void_p(_p(tg)),
            ctypes.c_void_p(_p(tgs)))
    return rc, mat, tg, tgs


def mass_records(p):
    """-8 A M A (packed lower) and tr(M A): of the bras (K, tri + 1) and kets (K, nst, tri + 1)."""
    args, keep = _problem(p)
    ob, ok = np.zeros((p.K, p.svh + 1)), np.zeros((p.K, p.nst, p.svh + 1))
    iv = np.ascontiguousarray(p.iv)
    assert lib().emu_mass_records(*args, *[ctypes.c_void_p(_p(a)) for a in (iv, ob, ok)]) == 0
    return ob, ok


def sym_lists(K, lc, w, nst, sms, nj=7):
    """The tile lists of the symmetric passes: dict of counts and arrays."""
    L = lib()
    head = np.zeros(6, np.int32)
    none = [None] * 7
    L.emu_sym_lists(K, lc, w, nst, sms, nj, ctypes.c_void_p(_p(head)), *none)
    out = dict(zip(("ntiles", "units", "nb", "tail0", "ntail", "parts"), head.tolist()))
    nkb = (K + 31) // 32
    out.update(tiles=np.full((out["ntiles"], 2), -9, np.int32), start=np.full(nkb + 1, -9, np.int32),
               groups=np.full((out["units"], 2), -9, np.int32), urange=np.full((nkb, 2), -9, np.int32),
               tslot=np.full(out["ntiles"], -9, np.int32), bgroups=np.full((out["nb"], 2), -9, np.int32),
               burange=np.full((nkb, 2), -9, np.int32))
    L.emu_sym_lists(K, lc, w, nst, sms, nj, ctypes.c_void_p(_p(head)),
                    *[ctypes.c_void_p(_p(out[k])) for k in ("tiles", "start", "groups", "urange", "tslot", "bgroups", "burange")])
    return out


class EmuShardOps:
    """The shard steps of ``nbo_correlatedgaussians_b200.shard.DeviceShardOps``
    run by the host emulation of the kernels, on CPU tensors, so that the
    sharded orchestration (tile ranges, the two all-reduces, E and GRADC from
    the summed rows) can be tested on CPU ranks with the gloo backend."""

    def __init__(self, p, lc_s=2):
        import torch
        self.torch = torch
        self.p = p
        self.lc = int(lc_s)
        self.n, self.blk = p.n, p.blk
        self.ps = p.n * (p.n + 1) // 2 + 1 + 3 * p.n
        self.device = torch.device("cpu")
        self._sums = None
        self._status = 0

    def _call_pairs(self, x, K, t0, t1):
        args, keep = _problem(self.p)
        rows, nt = np.zeros(2 * K), ctypes.c_int(0)
        sums = np.zeros(4 * (self.ps + 1) * K)
        rc = simt().simt_shard_pairs(*args, ctypes.c_void_p(_p(x)), ctypes.c_int(self.lc), ctypes.c_int(t0), ctypes.c_int(t1),
                                     ctypes.c_void_p(_p(rows)), ctypes.c_void_p(_p(sums)), ctypes.byref(nt))
        return rc, rows, sums, nt.value

    def tiles(self, K):
        x = np.ascontiguousarray(self.p.x)
        rc, _, _, nt = self._call_pairs(x, K, 0, 0)
        assert rc >= 0
        return nt

    def pairs(self, x, K, t0, t1):
        xn = np.ascontiguousarray(x.numpy())
        rc, rows, self._sums, _ = self._call_pairs(xn, K, t0, t1)
        assert rc >= 0
        self._status = 2 if rc & 1 else (3 if rc & 2 else 0)
        return self.torch.from_numpy(rows)

    def grad(self, x, K, rows, t0, t1):
        # the finalize kernel: E, norm and GRADC from the summed rows
        xn = np.ascontiguousarray(x.numpy())
        C = xn[K * self.blk:]
        r = rows.numpy()
        cHc, cSc = float(C @ r[:K]), float(C @ r[K:])
        E, norm = cHc / cSc, 1.0 / cSc
        g = np.zeros(K * self.blk + K)
        g[K * self.blk:] = 2.0 * norm * (r[:K] - E * r[K:])
        self._norm = norm
        args, keep = _problem(self.p)
        fields = np.zeros(self.ps * K)
        rc = simt().simt_shard_fields(*args, ctypes.c_void_p(_p(xn)), ctypes.c_void_p(_p(self._sums)), ctypes.c_double(E),
                                      ctypes.c_double(norm), ctypes.c_void_p(_p(fields)))
        assert rc == 0
        return (self.torch.tensor([E], dtype=self.torch.float64), self.torch.from_numpy(g),
                self.torch.from_numpy(fields))

    def finish(self, x, K, sums, g):
        args, keep = _problem(self.p)
        gn = np.ascontiguousarray(g.numpy()).copy()
        xn, sn = np.ascontiguousarray(x.numpy()), np.ascontiguousarray(sums.numpy())
        simt().simt_shard_finish(*args, ctypes.c_void_p(_p(xn)), ctypes.c_void_p(_p(sn)), ctypes.c_double(self._norm),
                                 ctypes.c_void_p(_p(gn)))
        return self.torch.from_numpy(gn)

    def status(self):
        return self._status
