"""Pair rounds over padded buckets (msm_pairs.cuh) where positions, CTAs and padding meet: sizes around
the CTA's 128 threads, and points drawn from a handful of multiples of the generator, so that buckets
hold equal points (tangents on several levels), opposite ones (sums at infinity between rounds) and
inputs at infinity.  Exact: checked through the discrete logarithms."""
import numpy as np
import pytest

import bendg
import bn254_ref as o
from gpu_helpers import g1_from_jac_wire, g1_wire, g2_from_jac_wire, g2_wire, scalars_wire

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rounds", [1, 2, 3])
@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 1031])
@pytest.mark.parametrize("curve", [bendg.CURVE_G1, bendg.CURVE_G2])
def test_repeated_points(ctx, curve, n, rounds):
    rng = np.random.default_rng(9000 + 10 * n + rounds)
    c = o.G1 if curve == bendg.CURVE_G1 else o.G2
    few = [0, 1, 2, 3, o.P_FR - 1, o.P_FR - 2]  # 0: infinity
    base = [c.mul(c.gen, k) for k in few]
    pick = rng.integers(0, len(few), size=n)
    values = [1, 2, 3, 5, 1 << 200, o.P_FR - 1, o.P_FR - 5]
    sc = [values[i] for i in rng.integers(0, len(values), size=n)]
    pts = [base[i] for i in pick]
    want = c.mul(c.gen, sum(few[i] * s for i, s in zip(pick, sc)) % o.P_FR)
    try:
        ctx.pair_rounds_override(rounds)
        if curve == bendg.CURVE_G1:
            got = g1_from_jac_wire(ctx.msm_g1(g1_wire(pts), scalars_wire(sc), n))
        else:
            got = g2_from_jac_wire(ctx.msm_g2(g2_wire(pts), scalars_wire(sc), n))
    finally:
        ctx.pair_rounds_override(-1)
    assert got == want
