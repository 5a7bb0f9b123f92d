"""Proof inputs whose words lie at or above their modulus stand for the residue: the proof is the one
that the reduced words give."""
import os

import numpy as np
import pytest

import bendg
import bn254_ref as o
from conftest import GOLDEN

pytestmark = pytest.mark.gpu


def lifted(words, p):
    """the largest 256-bit representative of each 16-word element"""
    vals = bendg.wire_to_ints(words)
    return bendg.ints_to_wire([v + (2**256 - 1 - v) // p * p if v else 0 for v in vals]).reshape(words.shape)


def test_blinding_words_and_key_points(ctx, tmp_path):
    import shutil
    d = os.path.join(GOLDEN, "k4")
    want = open(os.path.join(d, "proof_ref.txt")).read()
    for f in os.listdir(d):
        shutil.copy(os.path.join(d, f), tmp_path / f)
    for f, p in (("rs.bin", o.P_FR), ("pk_g1.bin", o.P_FQ), ("pk_g2.bin", o.P_FQ)):
        w = np.fromfile(tmp_path / f, dtype="<u4")
        lifted(w, p).astype("<u4").tofile(tmp_path / f)
    files = bendg.HostFiles(str(tmp_path))
    proof, _ = ctx.prove_host(files)
    assert ctx.proof_text(proof) == want
    key = ctx.pk_upload(files)
    proof, _ = key.prove(files.words("witness"), files.words("rs"))
    key.release()
    assert ctx.proof_text(proof) == want
