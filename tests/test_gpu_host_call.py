"""necg_outprod_host with every kind of memory as its output."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_output_memory_of_every_kind():
    """Pageable and pinned memory get the same gradient, bit for bit; an address of
    device memory is the runtime's to take or refuse, not the process's end."""
    import torch
    from nbo_correlatedgaussians_b200 import _lib, synth
    from nbo_correlatedgaussians_b200.engine import Engine
    p = synth.make_problem("H2", 37, 5)
    eng = Engine(p)
    x = np.ascontiguousarray(p.x)
    f = ctypes.c_double()

    def call(ptr):
        return eng.L.necg_outprod_host(eng.h, p.K, x.ctypes.data, ctypes.addressof(f), ptr, None)

    g = np.full(x.size, np.nan)
    assert call(g.ctypes.data) == _lib.NECG_OK
    pinned = torch.full((x.size,), np.nan, dtype=torch.float64).pin_memory()
    assert call(pinned.data_ptr()) == _lib.NECG_OK
    assert np.array_equal(pinned.numpy(), g) and np.isfinite(g).all()
    device = torch.zeros(x.size, dtype=torch.float64, device="cuda")
    rc = call(device.data_ptr())
    torch.cuda.synchronize()
    assert rc != _lib.NECG_OK or np.array_equal(device.cpu().numpy(), g)
    call(g.ctypes.data)  # takes up an error that the runtime may have kept
    g2 = np.full(x.size, np.nan)
    assert call(g2.ctypes.data) == _lib.NECG_OK and np.array_equal(g2, g)
