"""The window reduction's tree (sums by the bits of a thread's index), its join over several parts and
the suffix scan of small sets: window widths from bucket sets smaller than a warp to many parts per
window, on threads and on cooperative groups, with digits at a set's first and last buckets and at the
powers of two where a bit's sum changes.  Exact: checked through the discrete logarithms."""
import numpy as np
import pytest

import bendg
import bn254_ref as o
from gpu_helpers import g1_from_jac_wire, g1_wire, g2_from_jac_wire, g2_wire, scalars_wire

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("coop", [0, 1])
@pytest.mark.parametrize("c", [3, 4, 5, 6, 7, 8, 10, 13, 16, 19])
@pytest.mark.parametrize("curve", [bendg.CURVE_G1, bendg.CURVE_G2])
def test_widths(ctx, curve, c, coop):
    rng = np.random.default_rng(7000 + 10 * c + coop)
    g = o.G1 if curve == bendg.CURVE_G1 else o.G2
    ends = sorted({d for b in range(c) for d in ((1 << b) - 1, 1 << b, (1 << b) + 1)})
    sc = [d << (c * (i % (250 // c))) for i, d in enumerate(ends)]
    sc += [int.from_bytes(rng.bytes(32), "little") % o.P_FR for _ in range(8)] + [0, o.P_FR - 1]
    n = len(sc)
    ks = [int(k) for k in rng.integers(1, 6, size=n)]  # few points: equal sums meet in the tree
    base = {k: g.mul(g.gen, k) for k in set(ks)}
    pts = [base[k] for k in ks]
    want = g.mul(g.gen, sum(k * s for k, s in zip(ks, sc)) % o.P_FR)
    try:
        ctx.window_override(0, 0 if curve == bendg.CURVE_G1 else 1, c)
        ctx.coop_reduce_override(coop)
        if curve == bendg.CURVE_G1:
            got = g1_from_jac_wire(ctx.msm_g1(g1_wire(pts), scalars_wire(sc), n))
        else:
            got = g2_from_jac_wire(ctx.msm_g2(g2_wire(pts), scalars_wire(sc), n))
    finally:
        ctx.coop_reduce_override(-1)
        ctx.window_override(0, 0 if curve == bendg.CURVE_G1 else 1, 0)
    assert got == want
