"""The MSM's bucket reduction by one tree per set, at the widths where it can go
wrong, and the plans of the drop-in msm(), against the known-discrete-log
identity."""
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


def _plan(n, c, glv):
    """Windows, buckets and buffer sizes (bytes) of a drop-in plan."""
    W = -(-(128 if glv else 254) // c)
    B, NB = 1 << (c - 1), W << (c - 1)
    entries = n * W * (2 if glv else 1)
    L = max(8, -(-entries // (148 * 4 * 128)))
    nacc = max(1, -(-entries // L))
    s = 1
    while s < B and (NB // s > 32768 or B // s > 128 * 128 or NB // (2 * s) >= (2 if s < 32 else 4) * 148 * 128):
        s *= 2
    parts, m = 2 * nacc, nacc
    while m > 32:
        m = 2 * (-(-m // 32))
        parts += m
    sizes = [NB * 4, (NB + 1) * 4, (-(-NB // 4096) + 1) * 4, entries * 4, parts * 4, parts * 128, NB * 128,
             W * (B // s) * 128, W * 128, n * 64 if glv else 0]
    return W, NB, sizes


def _default_window(n, glv):
    cost = lambda c: (10 * n * (2 if glv else 1) * _plan(1, c, glv)[0] + 28 * _plan(1, c, glv)[1]  # noqa: E731
                      + 9 * 150 * (_plan(1, c, glv)[0] - 1) * c)
    return min(range(4, 21), key=cost)


def _fits(sizes, arenas):
    used = [0, 0]
    for k in sorted(range(10), key=lambda i: -sizes[i]):
        for a in ((1,) if k == 8 else (0, 1)):  # the window sums stay in the region
            start = -(-used[a] // 256) * 256
            if start + sizes[k] <= arenas[a]:
                used[a] = start + sizes[k]
                break
        else:
            return False
    return True


def _dropin_choice(n, windows, bits, workers):
    """(split or whole, W, c) that msm() takes in the caller's two buffers, or
    None where it refuses."""
    arenas = [3 * n * windows * 4, ((windows << bits) + 2 * workers) * 96 - 256]
    c0, c = _default_window(n, False), _default_window(n, True)
    most = _plan(n, c0, False)[1]
    if _plan(n, c, True)[1] > most:
        ok = [x for x in range(4, c) if _plan(n, x, True)[1] <= most]
        c = min(ok, key=lambda x: (_plan(n, x, True)[0], x))
    if _fits(_plan(n, c, True)[2], arenas):
        return "split", _plan(n, c, True)[0], c
    order = [c0] + [x for d in range(1, 20) for x in (c0 + d, c0 - d) if 4 <= x <= 22]
    for x in order:
        if _fits(_plan(n, x, False)[2], arenas):
            return "whole", _plan(n, x, False)[0], x
    return None


# windows, window bits and workers of the caller's buffers at 100003 points, and
# what msm() makes of them
REGIONS_100K = {(48, 3, 1953): ("split", 10, 13), (32, 3, 22737): ("whole", 20, 13), (26, 12, 2441): ("whole", 22, 12),
                (28, 10, 3051): ("whole", 24, 11), (26, 10, 11641): ("whole", 26, 10),
                (12, 14, 5960): ("whole", 29, 9), (14, 12, 22737): None}


def test_dropin_region_outcomes():
    for r, choice in REGIONS_100K.items():
        assert _dropin_choice(100003, *r) == choice, r


def _dropin_check(O, gpu, bases, d, s, windows, bits, workers, choice):
    """One msm() and its collect in buffers of exactly the stated sizes."""
    H, L = gpu.host, gpu.load_library()
    n, guard = s.shape[0], 4096
    region = ((windows << bits) + 2 * workers) * 96
    words = 3 * n * windows * 4
    res = torch.full((region + guard,), 7, dtype=torch.uint8, device="cuda")
    srt = torch.full((words + guard,), 7, dtype=torch.uint8, device="cuda")
    dummy = torch.zeros(64, dtype=torch.int32, device="cuda")
    p, st = dummy.data_ptr(), H.stream_handle()
    sd = H.to_device(s)
    err = L.msm(res.data_ptr(), bases.data_ptr(), sd.data_ptr(), p, p, p, p, srt.data_ptr(), p, n, windows, bits,
                64, workers, words, 1, st)
    assert err == (0 if choice else 1), (workers, choice)
    if choice:
        torch.cuda.synchronize()
        note = res[128:144].cpu().numpy().view(np.uint32)  # the parked window sums: W and c
        assert (note[1], note[2]) == choice[1:], (workers, choice)
        regions = H.ptr_array([res])
        assert L.batch_msm_collect(p, p, p, p, regions.data_ptr(), workers, windows, bits, 1, st) == 0
        torch.cuda.synchronize()
        got = res[:96].cpu().numpy().view(np.uint64)
        assert (O.g1_jac_to_aff(got.reshape(1, 12)) == O.msm_known_dlog(d, s)).all(), workers
    assert (res[region:] == 7).all() and (srt[words:] == 7).all()


# the drop-in msm() lays its plan out in the caller's two buffers: scalars split
# by the endomorphism where the images fit too, whole scalars where not, and a
# refusal where neither does
@pytest.mark.parametrize("windows", [20, 30, 44, 54, 64])
@pytest.mark.parametrize("bits", [3, 5, 7, 10])
def test_dropin_msm_region_sizes(O, gpu, windows, bits):
    n = 1000
    d = O.rand_fr(n, 91)
    bases, s = gpu.host.to_device(O.g1_gen_bases(d)), O.rand_fr(n, 92)
    for workers in (0, 64, 1024):
        _dropin_check(O, gpu, bases, d, s, windows, bits, workers, _dropin_choice(n, windows, bits, workers))


@pytest.fixture(scope="module")
def bases_100k(O, gpu):
    bases, k = gpu.schedule.bases_with_known_logs(100003, 5)
    return bases, _logs(O, k)


def _logs(O, k):
    d = np.zeros((k.shape[0], 4), np.uint64)
    d[:, 0] = k.cpu().numpy()
    return O.to_mont(d)


@pytest.mark.parametrize("region", REGIONS_100K)
def test_dropin_msm_region_choice(O, gpu, bases_100k, region):
    bases, d = bases_100k
    _dropin_check(O, gpu, bases, d, O.rand_fr(100003, 93), *region, REGIONS_100K[region])


# split scalars keep to the buckets of whole ones: 2.5 million points take 8
# windows of 16 bits, not 7 of 19
@pytest.mark.parametrize("n,W,window", [(1 << 17, 10, 13), (2_500_000, 8, 16)])
def test_dropin_msm_split_window(O, gpu, n, W, window):
    H, S = gpu.host, gpu.schedule
    bases, k = S.bases_with_known_logs(n, 5)
    cols = [S.scalars(n, m, 6 + i) for i, m in enumerate(("uniform", "small"))]
    b = H.ReferenceMsmBatch(bases, cols, n)
    b.enqueue()
    torch.cuda.synchronize()
    assert _dropin_choice(n, b.windows, b.c, b.worker) == ("split", W, window)
    for i in range(2):
        note = b.curve_buf[i * b.region:i * b.region + 2].reshape(-1).cpu().numpy().view(np.uint32)[32:36]
        assert (note[1], note[2]) == (W, window)
    got = O.g1_jac_to_aff(b.results())
    d = _logs(O, k)
    for i, c in enumerate(cols):
        assert (got[i] == O.msm_known_dlog(d, H.to_host(c))[0]).all(), i


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
