"""The operation counts that bench.py's roofline is formed from: what the kernels execute
per term (counted from their own templates) and the fixed measure beside it."""
import pytest

from nbo_correlatedgaussians_b200.engine import term_flops

# energy, ordered gradient, symmetric, fused: operations executed per (k, l, P) term
EXECUTED = {2: (218, 524, 601, 642), 3: (432, 1061, 1195, 1266), 5: (1085, 2797, 3084, 3238)}


@pytest.mark.parametrize("n", sorted(EXECUTED))
def test_executed_counts(n):
    t = term_flops(n)
    assert tuple(t[k + "_executed"] for k in ("energy", "grad", "sym", "fused")) == EXECUTED[n]

