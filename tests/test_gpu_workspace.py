"""What an engine holds on the device."""
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


def test_prepared_engines_allocate_nothing_in_their_first_step():
    p, eng, x = _engine("H2", 70)
    assert eng.L.necg_set_symmetric(eng.h, 2, 2, 248) == 0
    before = eng.workspace_bytes()
    assert eng.prepare_fused(p.K) > 0
    ready = eng.workspace_bytes()
    eng.outprod_device(x, p.K)
    assert before < ready == eng.workspace_bytes()
