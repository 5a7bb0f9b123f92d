"""A proof that fails between its launches (an allocation that does not fit) leaves its context fit for
the next call: an MSM queued at once takes over the sorts' rank buffer, then proofs again."""
import os

import numpy as np
import pytest

import bendg
import bn254_ref as o
from conftest import GOLDEN
from gpu_helpers import g1_from_jac_wire, scalars_wire
from test_gpu_msm import gpu_points

pytestmark = pytest.mark.gpu


def test_calls_after_a_proof_out_of_memory(built_lib):
    torch = pytest.importorskip("torch")
    d = os.path.join(GOLDEN, "k10")
    want = open(os.path.join(d, "proof_ref.txt")).read()
    files = bendg.HostFiles(d)
    n = 9000
    rng = np.random.default_rng(77)
    ks = [int.from_bytes(rng.bytes(32), "little") % o.P_FR for _ in range(n)]
    sc = [int.from_bytes(rng.bytes(32), "little") % o.P_FR for _ in range(n)]
    total = o.G1.mul(o.G1.gen, sum(a * b for a, b in zip(ks, sc)) % o.P_FR)
    with bendg.Context(0) as ctx:
        pts, words = gpu_points(ctx, bendg.CURVE_G1, ks), scalars_wire(sc)
        ctx.prove_host(files)  # everything but the buckets below is allocated by now
        ctx.msm_g1(pts, words, n)
        free, _ = torch.cuda.mem_get_info()
        hog = torch.empty(free - (3 << 30), dtype=torch.uint8, device="cuda")
        try:
            for _ in range(3):
                # G2 bucket sets of 22-bit windows: 6.4 GB, asked for after msm_a and msm_b1 are queued
                ctx.window_override(0, bendg.CURVE_G2, 22)
                with pytest.raises(bendg.BgError) as e:
                    ctx.prove_host(files)
                assert e.value.status == bendg.BG_E_OOM
                ctx.window_override(0, bendg.CURVE_G2, 0)
                assert g1_from_jac_wire(ctx.msm_g1(pts, words, n)) == total
                proof, _ = ctx.prove_host(files)
                assert ctx.proof_text(proof) == want
        finally:
            del hog
            torch.cuda.empty_cache()
