"""The MSM's bucket reduction by one tree per set, at the widths where it can go
wrong, against the known-discrete-log identity."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# 1 .. 2^21 buckets a set: one segment, one group, several groups (planes), the
# longest segments
@pytest.mark.parametrize("c", [5, 6, 9, 10, 14, 15, 18, 20, 22])
def test_msm_reduction_widths(O, gpu, c):
    H = gpu.host
    n = 2000
    d = O.rand_fr(n, 61)
    bases = H.to_device(O.g1_gen_bases(d))
    s = O.rand_fr(n, 62 + c)
    exp = O.msm_known_dlog(d, s)
    out = H.msm(bases, H.to_device(s), n=n, window_bits=c)
    torch.cuda.synchronize()
    assert (O.g1_jac_to_aff(H.to_host(out).reshape(1, 12)) == exp).all()
    table, c = H.msm_table_build(bases, n, c)
    out = H.msm_table(table, n, c, H.to_device(s), n=n)
    torch.cuda.synchronize()
    assert (O.g1_jac_to_aff(H.to_host(out).reshape(1, 12)) == exp).all()


def test_msm_batch_mixed_widths(O, gpu):
    """MSMs of widths 4..17 in one pipeline: sets of one and of many groups
    side by side, and an empty MSM."""
    H = gpu.host
    nmax = 1500
    d = O.rand_fr(nmax, 71)
    bases = H.to_device(O.g1_gen_bases(d))
    ns = [nmax, 0, 1, 700, 33, 1499, 64]
    ws = [4, 8, 13, 17, 5, 9, 15]
    cols = [O.rand_fr(max(n, 1), 80 + i) for i, n in enumerate(ns)]
    out = H.msm_batch(bases, [H.to_device(x) for x in cols], ns, ws)
    torch.cuda.synchronize()
    got = H.to_host(out)
    for i, n in enumerate(ns):
        exp = O.msm_known_dlog(d[:n], cols[i][:n]) if n else np.zeros((1, 8), np.uint64)
        assert (O.g1_jac_to_aff(got[i].reshape(1, 12)) == exp).all(), i
