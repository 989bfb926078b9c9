"""The pair passes' raw sums (derivatives with respect to B and e, folded into
gradients once per basis function): every particle count the symmetric passes
take, at sizes around the tile edges, against the oracle; and symmetry sets whose
shift maps are not those of their coordinate maps (kets folded in each term's
frame) against the host emulation, which folds every term by itself.  Tolerances
are those of the other parity tests (E 1e-10, gradient 1e-9 norm-wise; both
sides are FP64 sums of the same terms in another order)."""
import itertools

import numpy as np
import pytest

from _util import TOL_E, TOL_G, normwise
from oracle.oracle import Oracle

PASSES = [(0, 4, 8, 1), (1, 3, 8, 1), (1, 1, 12, 1), (2, 2, 118, 1), (2, 1, 122, 2), (2, 2, 12, 1), (2, 3, 228, 1),
          (2, 2, 248, 1), (2, 1, 268, 1)]
BLOCKS16 = (2, 3, 216, 1)  # 16-warp blocks fit for n <= 3


def make(n, K, seed, perms=None):
    """n equal particles around a heavier reference, some of their permutations."""
    from nbo_correlatedgaussians_b200.problem import Problem
    from nbo_correlatedgaussians_b200.symmetry import mass_matrix
    rng = np.random.default_rng(seed)
    perms = list(itertools.permutations(range(n)))[:2 if n > 1 else 1] if perms is None else perms
    sml = np.zeros((len(perms), n, n))
    for s, p in enumerate(perms):
        for i, j in enumerate(p):
            sml[s, i, j] = 1.0
    sms = np.stack([np.kron(np.linalg.inv(m), np.eye(3)) for m in sml])
    blk = n * (n + 1) // 2 + 3 * n
    iv = np.empty((K, blk))
    for k in range(K):
        L = np.tril(rng.normal(0.0, 0.3, (n, n)))
        L[np.diag_indices(n)] = rng.uniform(0.2, 3.0, n)
        iv[k, :blk - 3 * n] = np.concatenate([L[j:, j] for j in range(n)])
        iv[k, blk - 3 * n:] = rng.normal(0.0, 0.2, 3 * n)
    return Problem(n, K, 3e-3, mass_matrix(1836.15, [1.0] * n), np.array([float(n)] + [-1.0] * n),
                   np.full(len(perms), 1.0 / len(perms)), sml, sms, iv.reshape(-1), rng.normal(size=K))


def engine(p):
    from nbo_correlatedgaussians_b200.engine import Engine
    return Engine(p)


@pytest.mark.gpu
@pytest.mark.parametrize("n,K", [(1, 1), (1, 33), (2, 31), (3, 40), (4, 1), (4, 32), (4, 67), (5, 35)])
def test_every_particle_count(n, K):
    p = make(n, K, 100 * n + K)
    fo, go = Oracle.from_problem(p).outprod(p.x, nthreads=8)
    eng = engine(p)
    for mode, lc, minw, npc in PASSES + ([BLOCKS16] if n <= 3 else []):
        assert eng.L.necg_set_symmetric(eng.h, mode, lc, minw) == 0
        assert eng.L.necg_set_splits(eng.h, min(npc, p.nst)) == 0
        f, g = eng.outprod(p.x)
        assert abs(f - fo) < TOL_E and normwise(g, go) < TOL_G, (mode, lc, minw)
    # the gradient with E given (symmetric pass), one-warp tiles and lockstep blocks
    for lc, minw in ((2, 118), (3, 12), (2, 248)):
        assert eng.L.necg_set_symmetric(eng.h, 2, lc, minw) == 0
        H, S, _, _, en = eng.build_matrices(p.iv, p.C, parts=False)
        g = eng.make_grad_dev(p.iv, p.C, H, S, en).cpu().numpy()
        assert abs(float(en[0]) - fo) < TOL_E and normwise(g, go) < TOL_G, (lc, minw)


@pytest.mark.gpu
def test_make_grad_lockstep_with_split_tail():
    """A size whose lockstep queue ends in a partial round (its groups split over
    the symmetry terms), through the gradient with E given."""
    from nbo_correlatedgaussians_b200 import synth
    p = synth.make_problem("LiH", 200, 3)
    p.C = np.random.default_rng(3).normal(size=p.K)
    fo, go = Oracle.from_problem(p).outprod(p.x, nthreads=8)
    eng = engine(p)
    for lc in (1, 2, 5):
        assert eng.L.necg_set_symmetric(eng.h, 2, lc, 248) == 0
        H, S, _, _, en = eng.build_matrices(p.iv, p.C, parts=False)
        g = eng.make_grad_dev(p.iv, p.C, H, S, en).cpu().numpy()
        assert normwise(g, go) < TOL_G, lc


def _odd_shift_maps(K):
    """The H2 set with shift maps kron(sml^T, I3): closed under inverse, but not
    the maps of its coordinate maps (the proton swap is not orthogonal)."""
    from nbo_correlatedgaussians_b200 import synth
    p = synth.make_problem("H2", K, 50 + K)
    p.C = np.random.default_rng(K).normal(size=K)
    p.sms = np.stack([np.kron(m.T, np.eye(3)) for m in p.sml])
    return p


@pytest.mark.gpu
@pytest.mark.parametrize("K", [5, 37, 70])
def test_shift_maps_of_their_own(K):
    from emu import emu
    from nbo_correlatedgaussians_b200.batch import BatchEngine
    p = _odd_shift_maps(K)
    rc, fe, ge, He, Se = emu.outprod_fused(p, 2)
    assert rc == 0
    eng = engine(p)
    for mode, lc, minw, npc in PASSES[1:]:
        assert eng.L.necg_set_symmetric(eng.h, mode, lc, minw) == 0
        assert eng.L.necg_set_splits(eng.h, npc) == 0
        f, g = eng.outprod(p.x)
        assert abs(f - fe) < TOL_E and normwise(g, ge) < TOL_G, (mode, lc, minw)
    be = BatchEngine([p, make(2, 20, 9)], tune=False)
    be.plan()
    be.step()
    be.check()
    f, g = be.results(0)
    assert abs(f - fe) < TOL_E and normwise(g, ge) < TOL_G


@pytest.mark.parametrize("n,K", [(1, 3), (4, 34), (5, 9)])
def test_folded_terms_on_the_host(n, K):
    """The same terms folded one by one on the host, against the oracle."""
    from emu import emu
    p = make(n, K, 7 * n + K)
    fo, go = Oracle.from_problem(p).outprod(p.x, nthreads=8)
    for rc, f, g, _, _ in (emu.outprod(p), emu.outprod_sym(p, 4, 3), emu.outprod_fused(p, 2)):
        assert rc == 0 and abs(f - fo) < TOL_E and normwise(g, go) < TOL_G


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5])
def test_executed_counts_below_the_direct_formulation(n):
    from nbo_correlatedgaussians_b200.engine import term_flops
    t = term_flops(n)
    assert t["energy_executed"] < t["grad_executed"] < t["sym_executed"] < t["fused_executed"] < t["fused"]


def _subset(system, K, keep, shift=None):
    from nbo_correlatedgaussians_b200 import synth
    p = synth.make_problem(system, K, 31 * K)
    p.C = np.random.default_rng(K).normal(size=K)
    p.sml, p.sms, p.scvv = p.sml[keep], p.sms[keep], np.random.default_rng(1).uniform(0.5, 1.5, len(keep))
    if shift:
        p.sms = np.stack([np.kron(m.T, np.eye(3)) for m in p.sml])
    return p


@pytest.mark.gpu
@pytest.mark.parametrize("system,K,keep,shift", [
    ("LiH", 1, range(24), None), ("LiH", 33, range(24), None), ("LiH", 40, [0, 1, 2, 3, 4, 5], None),  # groups
    ("LiH", 20, [0, 3, 4], None),              # three-cycles: a group without involutions
    ("LiH", 20, [0, 1, 2], None),              # not closed under products: every (Pe, P)
    ("H2", 45, [0, 1, 2, 3], None), ("H2", 45, [0, 3], None), ("H2", 30, [2], None),
    ("H2", 30, [0, 1, 2, 3], "sml^T"),         # shift maps of their own: every (Pe, P)
    ("He", 70, [0, 1], None)])
def test_dipole_classes(system, K, keep, shift):
    """The dipole by classes of a group and by every pair of terms otherwise, unequal
    weights, against the oracle (the tolerance of the emulation's dipole test)."""
    p = _subset(system, K, list(keep), shift)
    comps_o, dip_o = Oracle.from_problem(p).dipole(p.iv, p.C, nthreads=8)
    eng = engine(p)
    for lc in (1, 2, 7):
        eng.set_tiles(lc, 4)
        comps, dip = eng.dipole(p.iv, p.C)
        scale = max(np.max(np.abs(comps_o)), 1e-300)
        assert np.max(np.abs(comps - comps_o)) <= 1e-11 * scale
        assert np.max(np.abs(dip - dip_o)) <= 1e-11 * max(np.max(np.abs(dip_o)), scale)


@pytest.mark.gpu
@pytest.mark.parametrize("n,K,lc,minw,npc", [(5, 70, 1, 248, 1), (5, 200, 2, 248, 1), (3, 130, 2, 216, 1), (3, 130, 1, 232, 1),
                                             (2, 90, 3, 118, 2), (4, 33, 2, 12, 1)])
def test_matrices_and_row_sums_agree(n, K, lc, minw, npc):
    """H and S written on request (block variants: with their queue's split tail;
    split symmetry terms) against the oracle, and the same E and gradient, bit for
    bit, whether they are asked for or not."""
    import torch
    from nbo_correlatedgaussians_b200 import _lib, synth
    system = {2: "He", 3: "H2", 5: "LiH"}.get(n)
    p = synth.make_problem(system, K, K) if system else make(n, K, K)
    p.C = np.random.default_rng(K).normal(size=K)
    fo, go, Ho, So = Oracle.from_problem(p).outprod(p.x, nthreads=8, return_hs=True)
    eng = engine(p)
    assert eng.L.necg_set_symmetric(eng.h, 2, lc, minw) == _lib.NECG_OK
    assert eng.L.necg_set_splits(eng.h, min(npc, p.nst)) == _lib.NECG_OK
    x = torch.from_numpy(p.x).to(eng.device)
    H = torch.full((K, K), np.nan, dtype=torch.float64, device=eng.device)
    S = torch.full_like(H, np.nan)
    f, g = eng.outprod_device(x, K, H=H, S=S)
    f2, g2 = eng.outprod_device(x, K)
    torch.cuda.synchronize()
    assert float(f) == float(f2) and torch.equal(g, g2)
    assert abs(float(f) - fo) < TOL_E and normwise(g.cpu().numpy(), go) < TOL_G
    for M, Mo in ((H, Ho), (S, So)):
        M = M.cpu().numpy()
        assert np.array_equal(M, M.T) and np.max(np.abs(M - Mo)) <= 1e-12 * max(1.0, np.max(np.abs(Mo)))


@pytest.mark.gpu
@pytest.mark.parametrize("K", [1, 7, 31, 32, 33, 63, 65, 96, 101])
@pytest.mark.parametrize("lc", [1, 3, 8])
def test_row_blocks_of_ragged_sizes(K, lc):
    """Every remainder class of K against 32 and chunks that do not divide the row
    blocks' ends: passes, matrices and dipole against the oracle."""
    from nbo_correlatedgaussians_b200 import synth
    p = synth.make_problem("H2", K, 9 * K + lc)
    p.C = np.random.default_rng(K).normal(size=K)
    o = Oracle.from_problem(p)
    fo, go, Ho, So = o.outprod(p.x, nthreads=8, return_hs=True)
    comps_o, _ = o.dipole(p.iv, p.C, nthreads=8)
    eng = engine(p)
    for mode, minw, npc in ((0, 8, 1), (1, 8, 1), (2, 12, 1), (2, 122, 3), (2, 248, 1), (2, 216, 1)):
        assert eng.L.necg_set_symmetric(eng.h, mode, lc, minw) == 0
        assert eng.L.necg_set_splits(eng.h, npc) == 0
        f, g = eng.outprod(p.x)
        assert abs(f - fo) < TOL_E and normwise(g, go) < TOL_G, (mode, minw)
    eng.set_tiles(lc, 4)
    H, S, _, _, en = eng.build_matrices(p.iv, p.C)
    assert abs(float(en[0]) - fo) < TOL_E
    assert np.max(np.abs(H.cpu().numpy() - Ho)) <= 1e-12 * max(1.0, np.max(np.abs(Ho)))
    assert np.max(np.abs(S.cpu().numpy() - So)) <= 1e-12 * max(1.0, np.max(np.abs(So)))
    comps, _ = eng.dipole(p.iv, p.C)
    assert np.max(np.abs(comps - comps_o)) <= 1e-11 * max(np.max(np.abs(comps_o)), 1e-300)


@pytest.mark.gpu
@pytest.mark.parametrize("n,K,lc", [(2, 290, 1), (3, 290, 1), (3, 290, 5), (1, 290, 1)])
@pytest.mark.parametrize("minw", [248, 232, 216])
def test_gradient_with_e_given_of_block_handles(n, K, lc, minw):
    """n <= 3 handles set to a block variant: one-warp tiles, on both sides of the
    count where more of them share an SM (chunk 1: 1500 tiles, chunk 5: 300)."""
    p = make(n, K, 11 * n + lc)
    fo, go = Oracle.from_problem(p).outprod(p.x, nthreads=8)
    eng = engine(p)
    assert eng.L.necg_set_symmetric(eng.h, 2, lc, minw) == 0
    H, S, _, _, en = eng.build_matrices(p.iv, p.C, parts=False)
    g = eng.make_grad_dev(p.iv, p.C, H, S, en).cpu().numpy()
    assert abs(float(en[0]) - fo) < TOL_E and normwise(g, go) < TOL_G
