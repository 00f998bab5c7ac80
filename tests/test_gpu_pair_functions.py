"""The double-float reciprocal, quotient and roots of the plain step on the
device, over 2^20 pairs: no further from the exact values than two Newton
steps in pairs, which the split step takes, in the mean and at worst.

Why at worst too: one correction of an FP32 value whose residual is carried
in two words rounds its low word twice (2^-48 each, 2^-49 where the exponent
favours it), a Newton step the residual and its product as well."""
from __future__ import annotations

import math

import pytest

pytestmark = pytest.mark.gpu


def test_no_less_accurate_than_newton(pkg):
    e = pkg.probe_pairs()
    bits = {k: tuple(round(math.log2(x), 2) for x in v) for k, v in e.items()}
    for f in ("rcp", "div", "rsqrt", "sqrt"):
        assert e[f][0] <= e["newton_" + f][0], (f, bits)
        assert e[f][1] <= e["newton_" + f][1], (f, bits)
        assert e[f][1] < 2.0 ** -45 and e["newton_" + f][1] < 2.0 ** -45, bits
