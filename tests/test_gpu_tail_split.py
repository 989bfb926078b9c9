"""Block variants on the device at sizes whose queue's tail is split in different
ways, the number of parts taken from the library's own rule (csrc/necg_tiles.h): E, g, H
and S, and the gradient with E given, against one-warp tiles, which have no queue.  A
lost or doubled part would be an O(1) error."""
import numpy as np
import pytest

from _util import normwise

pytestmark = pytest.mark.gpu


def _parts(K, lc, w, nst, sms):
    from emu import emu
    return emu.sym_lists(K, lc, w, nst, sms)["parts"]


def _sizes(system, lc, w, nst, sms):
    """For each number of parts that sizes up to 560 give, the smallest such K."""
    first = {}
    for K in range(33, 560, 7):
        first.setdefault(_parts(K, lc, w, nst, sms), K)
    return first


@pytest.mark.parametrize("system,nst,lc,minw", [("LiH", 24, 1, 248), ("LiH", 24, 2, 248), ("H2", 4, 1, 232), ("H2", 4, 2, 216), ("He", 2, 1, 216)])
def test_split_tails(system, nst, lc, minw):
    import torch
    from nbo_correlatedgaussians_b200 import synth
    from nbo_correlatedgaussians_b200.engine import Engine
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    w = {248: 8, 232: 12, 216: 16}[minw]
    sizes = _sizes(system, lc, w, nst, sms)
    assert 1 in sizes and 2 in sizes and (nst < 8 or 8 in sizes)
    for parts, K in sizes.items():
        p = synth.make_problem(system, K, 60 + K)
        p.C = np.random.default_rng(K).normal(size=K)
        eng = Engine(p)
        x = torch.from_numpy(p.x).to(eng.device)
        res = []
        for variant in (118, minw):
            assert eng.L.necg_set_symmetric(eng.h, 2, lc, variant) == 0
            assert eng.L.necg_set_splits(eng.h, 1) == 0
            H, S = (torch.full((K, K), np.nan, dtype=torch.float64, device=eng.device) for _ in range(2))
            f, g = eng.outprod_device(x, K, H=H, S=S)
            eng.raise_status("outprod")
            Hm, Sm, _, _, en = eng.build_matrices(p.iv, p.C, parts=False)
            gm = eng.make_grad_dev(p.iv, p.C, Hm, Sm, en)
            res.append([float(f)] + [t.cpu().numpy() for t in (g, H, S, gm)])
        eng.close()
        one, blocks = res
        assert abs(blocks[0] - one[0]) <= 1e-12 * abs(one[0]), (parts, K)
        assert normwise(blocks[1], one[1]) < 1e-11 and normwise(blocks[4], one[1]) < 1e-11, (parts, K)
        for a, b in zip(blocks[2:4], one[2:4]):
            assert np.array_equal(a, a.T) and np.max(np.abs(a - b)) <= 1e-13 * np.max(np.abs(b)), (parts, K)
