"""NTT passes where their plans change: single-pass sizes, the last small-domain size and the first of
the register-blocked passes with even and odd stage counts (2^15 .. 2^17, and three passes at 2^21),
every mode against the inverse mode and, where plain Python is quick enough, against the oracle; all
words of the field's edges (0, 1, r - 1) among the inputs."""
import numpy as np
import pytest

import bendg
import bn254_ref as o
from gpu_helpers import fr_from_wire_mont, fr_wire_mont

pytestmark = pytest.mark.gpu


def inputs(n, seed):
    rng = np.random.default_rng(seed)
    w = rng.integers(0, 1 << 16, size=(n, 16), dtype=np.uint32)
    w[:, 15] = rng.integers(0, 0x3064, size=n, dtype=np.uint32)
    edge = bendg.ints_to_wire([0, 1, o.P_FR - 1, o.P_FR - 2])
    k = min(n, 4)
    w[:k] = edge[:k]
    if n > 8:
        w[n // 2: n // 2 + 4] = edge[::-1]
    return w


@pytest.mark.parametrize("log2n", [1, 2, 6, 7, 8, 14, 15, 16, 17, 21])
@pytest.mark.parametrize("pair", [(bendg.NTT_FORWARD, bendg.NTT_INVERSE),
                                  (bendg.NTT_COSET_FORWARD, bendg.NTT_COSET_INVERSE)])
def test_there_and_back(ctx, log2n, pair):
    x = inputs(1 << log2n, 40 + log2n).reshape(-1)
    assert np.array_equal(ctx.ntt(ctx.ntt(x, log2n, pair[0]), log2n, pair[1]), x)
    assert np.array_equal(ctx.ntt(ctx.ntt(x, log2n, pair[1]), log2n, pair[0]), x)


@pytest.mark.parametrize("log2n", [1, 7, 8, 15])
def test_against_the_oracle(ctx, log2n):
    x = inputs(1 << log2n, 90 + log2n)
    vals = fr_from_wire_mont(x)
    for mode, f in ((bendg.NTT_FORWARD, o.ntt), (bendg.NTT_INVERSE, o.intt), (bendg.NTT_COSET_FORWARD, o.coset_ntt)):
        assert np.array_equal(ctx.ntt(x.reshape(-1), log2n, mode), fr_wire_mont(f(vals)).reshape(-1)), mode
