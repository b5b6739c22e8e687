"""The prover's host conversion of Jacobian results to affine points: the
points of a call share one inversion, so identities and other points are mixed
in every position."""
import importlib
import random

import numpy as np
import pytest


@pytest.mark.parametrize("identities", [(), (0,), (2,), (0, 1, 4), tuple(range(5))])
def test_jac_to_affine(zkp, identities):
    P = importlib.import_module("zkwasm-prover_b200.prover")
    q, rng = P.Q_MOD, random.Random(3 + len(identities))
    mont = (1 << 256) % q
    rows, exp = [], []
    for i in range(5):
        x, y, z = (rng.randrange(1, q) for _ in range(3))
        if i in identities:
            x, y, z = 0, 1, 0
        rows.append([(v * mont % q >> (64 * j)) & (2 ** 64 - 1) for v in (x, y, z) for j in range(4)])
        exp.append((0, 0) if z == 0 else (x * pow(z, -2, q) % q, y * pow(z, -3, q) % q))
    assert P.jac_to_affine(np.array(rows, dtype=np.uint64)) == exp
    assert P.jac_to_affine(np.zeros((0, 12), dtype=np.uint64)) == []
