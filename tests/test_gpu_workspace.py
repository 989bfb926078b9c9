"""What an engine holds on the device: the serving budget's estimate bounds it under
every setting that the tuner can choose, the K x K buffers of split symmetry terms are
there only for callers that want H and S, and settings that need less give memory back."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _engine(system, K):
    import torch
    from nbo_correlatedgaussians_b200 import synth
    from nbo_correlatedgaussians_b200.engine import Engine
    p = synth.make_problem(system, K, 7 * K)
    p.C = np.random.default_rng(K).normal(size=K)
    eng = Engine(p)
    return p, eng, torch.from_numpy(p.x).to(eng.device)


@pytest.mark.parametrize("system,K", [("He", 1), ("He", 16), ("He", 300), ("He", 2032), ("H2", 12), ("H2", 157), ("H2", 2048),
                                      ("LiH", 12), ("LiH", 96), ("LiH", 300), ("LiH", 1000)])
def test_the_estimate_bounds_the_workspace(system, K):
    from nbo_correlatedgaussians_b200 import autotune
    from nbo_correlatedgaussians_b200.serve import workspace_estimate
    p, eng, x = _engine(system, K)
    bound = workspace_estimate(p)
    for mode, variants in ((0, (8,)), (1, autotune.MINW_SYM), (2, autotune.MINW_FUSED)):
        for lc in autotune.LC_S:
            for minw in variants:
                if eng.L.necg_set_symmetric(eng.h, mode, lc, minw) != 0:
                    continue
                for npc in autotune.splits(K, lc, eng.nst) if mode == 2 and minw < 200 else [1]:
                    assert eng.L.necg_set_splits(eng.h, npc) == 0
                    eng.set_tiles(lc, 4)
                    eng.outprod_device(x, K)
                    eng.build_matrices(p.iv, p.C)
                    assert eng.workspace_bytes() <= bound, (mode, lc, minw, npc)
    eng.dipole(p.iv, p.C)
    autotune.tune(eng, x, K, reps=1)
    eng.outprod_device(x, K)
    assert eng.workspace_bytes() <= bound


def test_matrices_of_split_terms_only_on_request():
    import torch
    from nbo_correlatedgaussians_b200.batch import BatchEngine
    p, eng, x = _engine("LiH", 256)
    assert eng.L.necg_set_symmetric(eng.h, 2, 4, 12) == 0 and eng.L.necg_set_splits(eng.h, 12) == 0
    f, g = (t.clone() for t in eng.outprod_device(x, p.K))
    without = eng.workspace_bytes()
    H, S = (torch.zeros((p.K, p.K), dtype=torch.float64, device=eng.device) for _ in range(2))
    f2, g2 = eng.outprod_device(x, p.K, H=H, S=S)
    assert torch.equal(f, f2) and torch.equal(g, g2)
    assert eng.workspace_bytes() - without == 2 * 12 * p.K * p.K * 8
    be = BatchEngine([p], tune=False)
    h = be.engines[0]
    assert h.L.necg_set_symmetric(h.h, 2, 4, 12) == 0 and h.L.necg_set_splits(h.h, 12) == 0
    be.plan()
    be.step()
    be.check()
    assert h.workspace_bytes() < without + p.K * p.K * 8


def test_settings_that_need_less_give_memory_back():
    p, eng, x = _engine("LiH", 96)
    sizes, energies = [], []
    for lc, minw, npc in ((2, 12, 1), (1, 12, 24), (2, 12, 1)):
        assert eng.L.necg_set_symmetric(eng.h, 2, lc, minw) == 0 and eng.L.necg_set_splits(eng.h, npc) == 0
        energies.append(float(eng.outprod_device(x, p.K)[0]))
        sizes.append(eng.workspace_bytes())
    assert sizes[2] == sizes[0] < sizes[1] and energies[2] == energies[0]


def test_capture_after_a_change_that_needs_less():
    """A capture takes the buffers as they are."""
    import torch
    p, eng, x = _engine("H2", 40)
    f, g = torch.empty(1, dtype=torch.float64, device=eng.device), torch.empty_like(x)
    assert eng.L.necg_set_symmetric(eng.h, 2, 2, 12) == 0 and eng.L.necg_set_splits(eng.h, 4) == 0
    eng.outprod_device(x, p.K, f=f, g=g)
    ref = f.clone(), g.clone()
    assert eng.L.necg_set_splits(eng.h, 2) == 0
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        eng.outprod_device(x, p.K, f=f, g=g)
    f.zero_()
    g.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert abs(float(f) - float(ref[0])) < 1e-12 and float((g - ref[1]).abs().max()) <= 1e-12 * float(ref[1].abs().max())


def test_prepared_engines_allocate_nothing_in_their_first_step():
    p, eng, x = _engine("H2", 70)
    assert eng.L.necg_set_symmetric(eng.h, 2, 2, 248) == 0
    before = eng.workspace_bytes()
    assert eng.prepare_fused(p.K) > 0
    ready = eng.workspace_bytes()
    eng.outprod_device(x, p.K)
    assert before < ready == eng.workspace_bytes()


def test_captures_after_a_plain_evaluation():
    """A fused evaluation without H and S makes what a capture of the other calls at its
    size needs: the matrices, and the evaluation with H and S of split terms."""
    import torch
    p, eng, x = _engine("H2", 40)
    assert eng.L.necg_set_symmetric(eng.h, 2, 2, 12) == 0 and eng.L.necg_set_splits(eng.h, 4) == 0
    f, g = eng.outprod_device(x, p.K)
    iv, C = x[:p.siv].clone(), x[p.siv:].clone()
    H, S = (torch.zeros((p.K, p.K), dtype=torch.float64, device=eng.device) for _ in range(2))
    f1, g1 = torch.zeros_like(f), torch.zeros_like(g)
    torch.cuda.synchronize()
    graphs = [torch.cuda.CUDAGraph() for _ in range(2)]
    with torch.cuda.graph(graphs[0]):
        Hm, Sm, _, _, en = eng.build_matrices(iv, C, K=p.K, check=False)
    with torch.cuda.graph(graphs[1]):
        eng.outprod_device(x, p.K, f=f1, g=g1, H=H, S=S)
    for graph in graphs:
        graph.replay()
    torch.cuda.synchronize()
    for a, b in ((f1, f), (g1, g), (H, Hm), (S, Sm), (en[:1], f)):
        assert float((a - b).abs().max()) <= 1e-12 * float(b.abs().max())


def test_a_callers_graph_outlives_a_change_of_splits():
    """Fewer splits with the same lists leave the buffers that a captured graph holds."""
    import torch
    p, eng, x = _engine("H2", 40)
    f, g = torch.empty(1, dtype=torch.float64, device=eng.device), torch.empty_like(x)
    assert eng.L.necg_set_symmetric(eng.h, 2, 2, 12) == 0 and eng.L.necg_set_splits(eng.h, 4) == 0
    eng.outprod_device(x, p.K, f=f, g=g)
    ref = f.clone(), g.clone()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        eng.outprod_device(x, p.K, f=f, g=g)
    held = eng.workspace_bytes()
    assert eng.L.necg_set_splits(eng.h, 1) == 0
    eng.outprod_device(x, p.K)
    assert eng.workspace_bytes() == held
    f.zero_()
    g.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(f, ref[0]) and torch.equal(g, ref[1])
