"""Device memory that a proof takes on a lane against what its key reserves, for circuits whose domain is
much smaller or larger than their assignment."""
import ctypes

import numpy as np
import pytest

import bendg
import bn254_ref as o
from test_gpu_batch import rs_words
from test_gpu_msm import gpu_points

pytestmark = pytest.mark.gpu


class Circuit:
    """the contents of the .bin files of a circuit of one constraint, with points drawn from a few hundred"""

    def __init__(self, ctx, ni, nw, lg, nh, nl):
        nz = ni + nw
        rng = np.random.default_rng(90 + lg + nl)
        ks = [int.from_bytes(rng.bytes(32), "little") % o.P_FR for _ in range(400)]
        g1 = np.asarray(gpu_points(ctx, bendg.CURVE_G1, ks)).reshape(400, -1)
        g2 = np.asarray(gpu_points(ctx, bendg.CURVE_G2, ks)).reshape(400, -1)
        some = lambda g, n: g[rng.integers(0, 400, size=n)]
        one = np.asarray(bendg.ints_to_wire([o.to_mont(1, o.P_FR)])).reshape(-1)
        row = np.concatenate([np.array([1, 0, 1, 0], dtype=np.uint32), one])  # nnz, two offsets, column, one
        self.witness = bendg.ints_to_wire([int.from_bytes(rng.bytes(31), "little") for _ in range(nz)]).reshape(-1)
        self.rs = rs_words(3, 5)
        bufs = {"header": np.array([1, ni, nw, lg, nz, nz, nh, nl], dtype=np.uint32), "witness": self.witness,
                "r1cs_a": row, "r1cs_b": row, "r1cs_c": row, "pk_g1": some(g1, 3), "pk_g2": some(g2, 2),
                "pk_a": some(g1, nz), "pk_b1": some(g1, nz), "pk_b2": some(g2, nz), "pk_h": some(g1, nh),
                "pk_l": some(g1, nl), "rs": self.rs}
        self.bufs = {k: np.ascontiguousarray(v, dtype=np.uint32) for k, v in bufs.items()}
        self.inputs = bendg.Inputs()
        for name, a in self.bufs.items():
            setattr(self.inputs, name, a.ctypes.data_as(ctypes.c_void_p).value if a.size else None)
            setattr(self.inputs, name + "_bytes", a.nbytes)


@pytest.mark.parametrize("ni,nw,lg,nh,nl", [(1, 393215, 18, 1 << 18, 0), (1, 3, 18, 1 << 18, 2),
                                            (1, (1 << 18) - 1, 14, 1 << 14, 1000)])
def test_scratch_stays_within_the_footprint(built_lib, ni, nw, lg, nh, nl):
    torch = pytest.importorskip("torch")
    with bendg.Context(0) as ctx:
        small = Circuit(ctx, 1, 7, 4, 15, 7)
        wide = Circuit(ctx, ni, nw, lg, nh, nl)
        ks, kw = ctx.pk_upload(small), ctx.pk_upload(wide)
        ctx.prove_batch([ks], [small.witness.ctypes.data], [small.rs.ctypes.data], lanes=1)  # the lane itself
        before, _ = torch.cuda.mem_get_info()
        proofs, _, status = ctx.prove_batch([kw], [wide.witness.ctypes.data], [wide.rs.ctypes.data], lanes=1)
        after, _ = torch.cuda.mem_get_info()
        assert status[0] == bendg.BG_OK
        assert before - after <= kw.footprint(), (before - after, kw.footprint())
        # fewer rounds, the same proof
        for rounds in (0, 2):
            ctx.pair_rounds_override(rounds)
            again, _ = kw.prove(wide.witness, wide.rs)
            assert ctx.proof_text(again) == ctx.proof_text(proofs[0])
        ks.release()
        kw.release()
