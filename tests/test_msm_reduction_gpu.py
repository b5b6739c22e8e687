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


# the drop-in msm() lays its plan out in the caller's two buffers: scalars split
# by the endomorphism where the images fit too, whole scalars where not, and a
# refusal where neither does
@pytest.mark.parametrize("windows", [20, 30, 44, 54, 64])
@pytest.mark.parametrize("bits", [3, 5, 7, 10])
def test_dropin_msm_region_sizes(O, gpu, windows, bits):
    H, L = gpu.host, gpu.load_library()
    n, guard = 1000, 4096
    d = O.rand_fr(n, 91)
    bases, s = H.to_device(O.g1_gen_bases(d)), O.rand_fr(n, 92)
    exp = O.msm_known_dlog(d, s)
    sd = H.to_device(s)
    for workers in (0, 64, 1024):
        region = ((windows << bits) + 2 * workers) * 96
        words = 3 * n * windows * 4
        res = torch.full((region + guard,), 7, dtype=torch.uint8, device="cuda")
        srt = torch.full((words + guard,), 7, dtype=torch.uint8, device="cuda")
        dummy = torch.zeros(64, dtype=torch.int32, device="cuda")
        p = dummy.data_ptr()
        st = H.stream_handle()
        err = L.msm(res.data_ptr(), bases.data_ptr(), sd.data_ptr(), p, p, p, p, srt.data_ptr(), p, n, windows, bits,
                    64, workers, words, 1, st)
        assert err in (0, 1)
        if err == 0:
            regions = H.ptr_array([res])
            assert L.batch_msm_collect(p, p, p, p, regions.data_ptr(), workers, windows, bits, 1, st) == 0
            torch.cuda.synchronize()
            got = res[:96].cpu().numpy().view(np.uint64)
            assert (O.g1_jac_to_aff(got.reshape(1, 12)) == exp).all(), workers
        assert (res[region:] == 7).all() and (srt[words:] == 7).all()


# sets and windows without a point: no scalar but zero, and scalars whose one
# digit lies in the lowest, a middle or the topmost window
@pytest.mark.parametrize("n", [1, 3, 40])
@pytest.mark.parametrize("value", [0, 1, 1 << 19, 1 << 64, 1 << 126, (1 << 253) + 1])
@pytest.mark.parametrize("dense", [False, True])
def test_msm_empty_windows(O, gpu, n, value, dense):
    H = gpu.host
    d = O.rand_fr(n, 171)
    bases = H.to_device(O.g1_gen_bases(d))
    s = O.fr_vec([value if dense or i == n // 2 else 0 for i in range(n)])
    exp = O.msm_known_dlog(d, s)
    sd = H.to_device(s)
    table, c = H.msm_table_build(bases, n, 0)
    outs = [H.msm(bases, sd, n=n), H.msm(bases, sd, n=n, window_bits=13), H.msm_table(table, n, c, sd, n=n)]
    outs += [H.msm_batch(bases, [sd, sd], [n, n], [4, 11])]
    torch.cuda.synchronize()
    for out in outs:
        for got in H.to_host(out).reshape(-1, 12):
            assert (O.g1_jac_to_aff(got.reshape(1, 12)) == exp).all()


# batches whose buckets take segments of 16, of 32 on either side of four blocks
# an SM, and of 64 (the scratch's limit)
@pytest.mark.parametrize("count", [12, 24, 48, 60])
def test_msm_batch_segment_lengths(O, gpu, count):
    H = gpu.host
    n, c = 64, 14
    d = O.rand_fr(n, 151)
    bases = H.to_device(O.g1_gen_bases(d))
    cols = [O.rand_fr(n, 160 + i) for i in range(4)]
    dev = [H.to_device(x) for x in cols]
    out = H.msm_batch(bases, [dev[i % 4] for i in range(count)], [n] * count, [c] * count)
    torch.cuda.synchronize()
    got = O.g1_jac_to_aff(H.to_host(out).reshape(-1, 12))
    exp = [O.msm_known_dlog(d, x) for x in cols]
    for i in range(count):
        assert (got[i] == exp[i % 4][0]).all(), i
