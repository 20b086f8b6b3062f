"""Iterates of the batch kernel with NT and float64 up to order 95, where the
FP32 basis of the scaling is orthonormal to FP32 only: a different rounding
anywhere before it can move the basis, and the iterates with it by 1e-6.  The
diagonals of X after three iterations are held to recorded ones
(golden/batch_nt_iterates.json) within 1e-11 of the largest entry: the same
basis with other roundings after it stays within 1e-13, another basis moves
them by 1e-7 or more.  Two problems of the record have an entry of the scaled
matrix close to the middle between two FP32 numbers; the others are at the
orders where the kernel's loops change."""
import json
import os

import numpy as np
import pytest

import madsdp_gpu as M
from madsdp_gpu import generators as g

pytestmark = pytest.mark.gpu

with open(os.path.join(os.path.dirname(__file__), "golden", "batch_nt_iterates.json")) as f:
    RECORD = json.load(f)


def _model(case):
    if case["model"] == "sos":
        return g.sos_hankel(case["d"], seed=case["seed"])
    return g.maxcut(case["n"], case["p"], seed=case["seed"])


def test_iterates_match_record(gpu_ctx):
    b = M.Batch([_model(c) for c in RECORD])
    b.initialize()
    b.iterate(3)
    for c, s in zip(RECORD, b.all_solutions()):
        want = np.array(c["diag"])
        assert np.abs(np.diag(s[0][0]) - want).max() <= 1e-11 * np.abs(want).max(), {k: c[k] for k in c if k != "diag"}
    b.close()
