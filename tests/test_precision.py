"""Accuracy where functions of very different widths meet, element by element,
against extended precision (tests/extended.py)."""
import numpy as np
import pytest

from _util import TOL_ELEM, TOL_G
from extended import Extended
from nbo_correlatedgaussians_b200 import synth

SYSTEMS = {"He": (2, 1), "H2": (3, 1), "LiH": (5, 1)}


def two_widths(system, K, r, seed=0):
    """Functions whose L is r times as large for every other one (tight and diffuse in
    both orders), shifts of about 0.3 widths, so that exp(-s A s) is harmless."""
    p = synth.make_problem(system, K, 900 + seed)
    rng = np.random.default_rng([seed, K])
    n, tri = p.n, p.n * (p.n + 1) // 2
    b = p.iv.reshape(K, -1)
    for k in range(K):
        scale = r if k % 4 in (1, 2) else 1.0
        L = np.tril(rng.normal(0.0, 0.1, (n, n)))
        L[np.diag_indices(n)] = rng.uniform(0.7, 1.4, n)
        b[k, :tri] = scale * np.concatenate([L[j:, j] for j in range(n)])
        b[k, tri:] = rng.normal(0.0, 0.3 / scale, 3 * n)
    p.iv, p.C = b.reshape(-1), rng.normal(size=K)
    return p


def check_elements(got, ref, scale, what):
    """Every element within the suite's bound for elements, against the sum of its terms."""
    got = np.asarray(got, dtype=np.float64)
    rel = np.abs(got.astype(np.longdouble) - ref) / np.maximum(scale, np.finfo(np.float64).tiny)
    assert rel.max() <= TOL_ELEM, (what, float(rel.max()), np.unravel_index(int(rel.argmax()), rel.shape))


RATIOS = [1.0, 10.0, 100.0, 1000.0, 1e4]


@pytest.mark.parametrize("system", list(SYSTEMS))
@pytest.mark.parametrize("r", RATIOS)
def test_elements_between_tight_and_diffuse_functions(system, r):
    """H of the separate and of the fused pass, and matel, on the host emulation."""
    from emu import emu
    p = two_widths(system, 8, r)
    ref = Extended(p).evaluate()
    rc, _, _, H, _ = emu.outprod(p)
    assert rc == 0
    check_elements(H, ref["H"], ref["aH"], "separate passes")
    rc, _, _, H, S = emu.outprod_fused(p, 2)
    assert rc == 0
    check_elements(H, ref["H"], ref["aH"], "fused pass")
    terms = [(1 + (i + j) % p.nst, i, j) for i in range(1, 9) for j in range(1, 9)]
    rc, mat, _, _ = emu.elements(p, terms)
    m = Extended(p).terms(terms)[0]
    assert rc == 0
    check_elements(mat[:, 1], m[:, 1], np.abs(m[:, 1]), "matel kinetic")


@pytest.mark.gpu
@pytest.mark.parametrize("system", list(SYSTEMS))
@pytest.mark.parametrize("r", RATIOS)
@pytest.mark.parametrize("K", [8, 40])
def test_matrices_between_tight_and_diffuse_functions(system, r, K):
    """Kinetic and H of build_matrices and of necg_matel, and H of the fused pass."""
    import torch
    from nbo_correlatedgaussians_b200.engine import Engine
    p = two_widths(system, K, r)
    ref = Extended(p).evaluate()
    eng = Engine(p)
    for lc in (1, 16):
        eng.set_tiles(lc, 4)
        H, S, Kin, Pot, _ = eng.build_matrices(p.iv, p.C)
        check_elements(Kin.cpu().numpy(), ref["T"], ref["aT"], "kinetic")
        check_elements(H.cpu().numpy(), ref["H"], ref["aH"], "H")
    x = torch.from_numpy(p.x).to(eng.device)
    H, S = (torch.zeros((K, K), dtype=torch.float64, device=eng.device) for _ in range(2))
    for mode, lc, minw in ((0, 4, 8), (2, 2, 118), (2, 2, 12), (2, 2, 248)):
        assert eng.L.necg_set_symmetric(eng.h, mode, lc, minw) == 0
        eng.outprod_device(x, K, H=H, S=S)
        check_elements(H.cpu().numpy(), ref["H"], ref["aH"], ("outprod", mode, minw))
    terms = [(1 + (i + j) % p.nst, i, j) for i in range(1, 9) for j in range(1, 9)]
    m = Extended(p).terms(terms)[0]
    check_elements(eng.matel(p.iv, terms)[:, 1], m[:, 1], np.abs(m[:, 1]), "matel")


def check_gradel(p, tg, terms):
    """The L block of every term's dh against its own largest component."""
    ref = Extended(p).terms(terms)[1][:, :p.svh]
    err = np.abs(np.asarray(tg)[:, :p.svh] - ref).max(1) / np.abs(ref).max(1)
    assert err.max() <= TOL_ELEM, (float(err.max()), terms[int(err.argmax())])


def all_terms(p, K):
    return [(1 + (i + j) % p.nst, i, j) for i in range(1, K + 1) for j in range(1, K + 1)]


@pytest.mark.parametrize("system", list(SYSTEMS))
@pytest.mark.parametrize("r", RATIOS)
def test_gradel_between_tight_and_diffuse_functions(system, r):
    from emu import emu
    p = two_widths(system, 8, r)
    rc, _, tg, _ = emu.elements(p, all_terms(p, 8))
    assert rc == 0
    check_gradel(p, tg, all_terms(p, 8))


@pytest.mark.gpu
@pytest.mark.parametrize("system", list(SYSTEMS))
@pytest.mark.parametrize("r", RATIOS)
def test_device_gradel_between_tight_and_diffuse_functions(system, r):
    from nbo_correlatedgaussians_b200.engine import Engine
    p = two_widths(system, 8, r)
    check_gradel(p, Engine(p).gradel(p.iv, all_terms(p, 8))[0], all_terms(p, 8))


def away_from_origin(system, K, lo, hi, shift, seed=0):
    """Tight functions (L diagonal lo .. hi) whose centres are spread by `shift`."""
    p = synth.make_problem(system, K, 70 + seed)
    rng = np.random.default_rng([seed, K])
    n, b = p.n, p.iv.reshape(K, -1)
    diagonal = [sum(n - q for q in range(j)) for j in range(n)]
    b[:, diagonal] = rng.uniform(lo, hi, (K, n))
    b[:, p.svh:] = rng.normal(0.0, shift, (K, 3 * n))
    p.iv, p.C = b.reshape(-1), rng.normal(size=K)
    return p


def check_components(p, g, ref, hi, shift, what):
    """The median relative error of GRADA's components: the suite's bound for gradients
    at 180 widths from the origin, where the differences of positions that the gradient is
    made of have lost that many digits, and by the square of that distance less nearer."""
    g = np.asarray(g)[:p.siv].reshape(p.K, -1)
    err = float(np.median(np.abs(g - ref) / np.abs(ref)))
    assert err <= TOL_G * (hi * shift / 180.0) ** 2, (what, err)


FAR = [("He", 40), ("H2", 40), ("LiH", 12)]


@pytest.mark.parametrize("system,K", FAR)
@pytest.mark.parametrize("lo,hi,shift", [(5.0, 60.0, 3.0), (2.0, 30.0, 1.0)])
def test_gradient_components_away_from_the_origin(system, K, lo, hi, shift):
    from emu import emu
    p = away_from_origin(system, K, lo, hi, shift)
    ref = Extended(p).evaluate()["g"]
    for what, out in (("ordered", emu.outprod(p)), ("fused", emu.outprod_fused(p, 2)), ("symmetric", emu.outprod_sym(p, 4, 2)),
                      ("blocks", emu.outprod_fused(p, 1, 8, 1, 3))):
        assert out[0] == 0
        check_components(p, out[2], ref, hi, shift, what)


@pytest.mark.gpu
@pytest.mark.parametrize("system,K", FAR)
@pytest.mark.parametrize("lo,hi,shift", [(5.0, 60.0, 3.0), (2.0, 30.0, 1.0)])
def test_device_gradient_components_away_from_the_origin(system, K, lo, hi, shift):
    from nbo_correlatedgaussians_b200.batch import BatchEngine
    from nbo_correlatedgaussians_b200.engine import Engine
    p = away_from_origin(system, K, lo, hi, shift)
    ref = Extended(p).evaluate()["g"]
    eng = Engine(p)
    for mode, lc, minw in ((0, 4, 8), (1, 2, 8), (2, 2, 118), (2, 2, 12), (2, 1, 248)):
        assert eng.L.necg_set_symmetric(eng.h, mode, lc, minw) == 0
        check_components(p, eng.outprod(p.x)[1], ref, hi, shift, (mode, minw))
    be = BatchEngine([p, p], tune=False)
    be.plan()
    be.step()
    be.check()
    check_components(p, be.results(0)[1], ref, hi, shift, "batch")


@pytest.mark.parametrize("system", ["He", "LiH"])
def test_permuted_kets_hold_the_permuted_values_of_the_bra(system):
    """A M A and tr(M A) of a function in the frame of a permutation that leaves M as it is
    are its own, bit for bit, so that their rounding cancels in an antisymmetric sum."""
    from emu import emu
    p = synth.make_problem(system, 9, 4)
    bra, ket = emu.mass_records(p)
    low = [(i, j) for i in range(p.n) for j in range(i + 1)]
    for P in range(p.nst):
        m = p.sml[P]
        assert np.array_equal(m @ p.mass @ m.T, p.mass)
        for k in range(p.K):
            full = np.zeros((p.n, p.n))
            for t, (i, j) in enumerate(low):
                full[i, j] = full[j, i] = bra[k, t]
            moved = m.T @ full @ m
            assert np.array_equal(ket[k, P, :-1], [moved[i, j] for i, j in low]) and ket[k, P, -1] == bra[k, -1]


@pytest.mark.gpu
@pytest.mark.parametrize("mode,lc,minw", [(0, 4, 8), (2, 2, 118), (2, 2, 248)])
def test_energy_of_antisymmetric_sums(mode, lc, minw):
    """E of LiH bases of K = 512 (the synthetic workloads' seeds 1 to 3), against 80-bit sums
    of the same terms: 30 roundings of E."""
    from nbo_correlatedgaussians_b200.engine import Engine
    for seed, E in ((1, "4.6758029388500884573"), (2, "7.1651162402481331"), (3, "3.8932810772307178317")):
        p = synth.make_problem("LiH", 512, seed)
        eng = Engine(p)
        assert eng.L.necg_set_symmetric(eng.h, mode, lc, minw) == 0
        f, _ = eng.outprod(p.x)
        assert abs(np.longdouble(f) - np.longdouble(E)) <= 30 * np.finfo(np.float64).eps / 2 * np.longdouble(E), seed
