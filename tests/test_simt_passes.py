"""The device code of the passes over unordered pairs, run thread by thread on the host
(tests/emu/simt_emu.cpp): one-warp tiles and their variants, split symmetry terms,
blocks of warps with their queue's split tail, the gradient with E given, and shards,
at sizes around the edges of row blocks and chunks; against the oracle, and where a
set's shift maps are not those of its coordinate maps against extended precision."""
import numpy as np
import pytest

from _util import TOL_E, TOL_ELEM, TOL_G, normwise
from emu import emu
from extended import Extended
from nbo_correlatedgaussians_b200 import synth
from oracle.oracle import Oracle
from test_gpu_raw_pass import _odd_shift_maps, make


def problem(system, K, seed):
    p = synth.make_problem(system, K, seed) if isinstance(system, str) else make(system, K, seed)
    p.C = np.random.default_rng(seed + K).normal(size=K)
    return p


def check(p, out, H=True):
    rc, f, g, Hm, Sm = out
    fo, go, Ho, So = Oracle.from_problem(p).outprod(p.x, nthreads=8, return_hs=True)
    assert rc == 0 and abs(f - fo) < TOL_E and normwise(g, go) < TOL_G
    for M, Mo in ((Hm, Ho), (Sm, So)):
        assert np.array_equal(M, M.T) and np.max(np.abs(M - Mo)) <= TOL_ELEM * max(1.0, np.max(np.abs(Mo)))


@pytest.mark.parametrize("system,K,lc,variant,npc", [
    ("He", 1, 1, 0, 1), ("He", 33, 3, 1, 2), ("He", 64, 7, 2, 1), ("He", 65, 1, 0, 1), ("H2", 31, 2, 2, 4), ("H2", 32, 5, 1, 1),
    ("H2", 45, 64, 0, 3), ("LiH", 5, 2, 2, 24), ("LiH", 33, 4, 1, 7), (1, 34, 2, 0, 1), (4, 35, 3, 2, 2)])
def test_one_warp_tiles(system, K, lc, variant, npc):
    p = problem(system, K, 3 * K)
    check(p, emu.outprod_fused(p, lc, variant, min(npc, p.nst)))
    check(p, emu.outprod_sym(p, 4, lc, variant))


@pytest.mark.parametrize("system,K,lc,warps,sms", [
    ("He", 1, 1, 8, 148), ("He", 70, 2, 16, 5), ("He", 97, 1, 12, 7), ("H2", 33, 1, 16, 3), ("H2", 64, 1, 8, 6), ("H2", 70, 3, 12, 4),
    ("LiH", 20, 1, 8, 148), ("LiH", 40, 1, 8, 5), ("LiH", 40, 2, 8, 2), (1, 40, 1, 8, 9), (4, 33, 1, 8, 11)])
def test_blocks_of_warps(system, K, lc, warps, sms):
    """Queue lengths that leave a partial round on a GPU of few SMs, so that its tail is split."""
    p = problem(system, K, 5 * K)
    check(p, emu.outprod_fused(p, lc, warps, 1, sms))
    check(p, emu.outprod_sym(p, 4, lc, warps, sms))


def test_the_tails_above_are_split():
    """The cases of test_blocks_of_warps cover unsplit queues and 2 to 8 parts."""
    cases = next(m for m in test_blocks_of_warps.pytestmark if m.name == "parametrize").args[1]
    nst = {"He": 2, "H2": 4, "LiH": 24}
    parts = {emu.sym_lists(K, lc, w, nst.get(s, 2), sms)["parts"] for s, K, lc, w, sms in cases}
    assert 1 in parts and 2 in parts and max(parts) >= 4


@pytest.mark.parametrize("K", [5, 37])
@pytest.mark.parametrize("variant,npc,sms", [(0, 1, 148), (1, 3, 148), (2, 1, 148), (8, 1, 3), (16, 1, 5)])
def test_shift_maps_of_their_own(K, variant, npc, sms):
    p = _odd_shift_maps(K)
    ref = Extended(p).evaluate()
    for rc, f, g, _, _ in (emu.outprod_fused(p, 2, variant, npc, sms), emu.outprod_sym(p, 4, 2, variant, sms)):
        assert rc == 0 and abs(f - float(ref["E"])) < TOL_E
        assert normwise(g[:p.siv].reshape(K, -1), ref["g"]) < 1e-11 and normwise(g[p.siv:], ref["gC"]) < 1e-11


def test_not_positive_definite_and_non_finite_flags():
    p = problem("He", 5, 3)
    p.iv[2 * p.blk:2 * p.blk + p.svh] = 0.0
    for variant in (0, 8):
        assert emu.outprod_fused(p, 2, variant)[0] & 1
    p = problem("He", 5, 3)
    p.iv[2 * p.blk] = np.nan
    for variant in (0, 8):
        assert emu.outprod_fused(p, 2, variant)[0] & 3
