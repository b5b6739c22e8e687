"""The per-coset quotient and multi-open entry points against the oracle, bit
for bit: zkp_eval_h_fused (every constraint family, rotations of both signs),
zkp_ntt_batch_twisted + zkp_coset_combine (against the reference host's
field_mul_zip -> iNTT of 2^(k+e) -> extended_prepare(to_coset) sequence,
restated by the oracle), zkp_poly_divide_linear (against the reference's own
host recurrence, src/multiopen.rs:145-159) and zkp_poly_eval_batch."""
import ctypes
import importlib

import numpy as np
import pytest
import torch

import ref_cases as RC

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def P(gpu):
    return importlib.import_module("zkwasm-prover_b200.prover")


def _h(t):
    torch.cuda.synchronize()
    return t.detach().cpu().contiguous().numpy().view(np.uint64).reshape(-1, 4)


@pytest.mark.parametrize("log_n", [4, 12, 20])
def test_poly_divide_linear(O, gpu, P, log_n):
    L = gpu.load_library()
    n = 1 << log_n
    a = O.rand_fr(n, 70 + log_n)
    ad = RC.Dev().put(a)
    for z in (O.fr_ints(O.rand_fr(1, 71))[0], 0, 1, O.R_MOD - 1):
        q = torch.empty_like(ad)
        scratch = torch.empty((L.zkp_poly_divide_scratch_elems(n), 4), dtype=torch.int64, device="cuda")
        zh = np.array(P.limbs(z), dtype=np.uint64)
        assert L.zkp_poly_divide_linear(q.data_ptr(), ad.data_ptr(), zh.ctypes.data, n, scratch.data_ptr(), 0) == 0
        assert (_h(q) == O.poly_divide_linear(a, z)).all(), f"z={z}"


def test_poly_eval_batch(O, gpu, P):
    L = gpu.load_library()
    for log_n in (1, 10, 16):
        n = 1 << log_n
        polys = [O.rand_fr(n, 80 + i) for i in range(5)]
        x = O.fr_ints(O.rand_fr(1, 81))[0]
        d = RC.Dev()
        dp = d.ptrs([d.put(p) for p in polys])
        pw = P.powers(1, x, n)
        out = torch.empty((5, 4), dtype=torch.int64, device="cuda")
        scratch = torch.empty((L.zkp_poly_eval_batch_scratch_elems(5), 4), dtype=torch.int64, device="cuda")
        assert L.zkp_poly_eval_batch(out.data_ptr(), dp.data_ptr(), 5, pw.data_ptr(), n, scratch.data_ptr(), 0) == 0
        assert O.fr_ints(_h(out)) == [O.poly_eval(p, x) for p in polys]


@pytest.mark.parametrize("ext_bits", [1, 2, 3])
@pytest.mark.parametrize("pairs", [False, True])
def test_cosets_and_combine(O, gpu, P, ext_bits, pairs):
    """Coset values from coefficients (zkp_ntt_batch_twisted) and back
    (zkp_coset_combine) against the oracle's whole-domain restatement."""
    L = gpu.load_library()
    k = 12
    n, E = 1 << k, 1 << ext_bits
    N = n * E
    coeff = O.rand_fr(n, 90 + ext_bits)
    # forward: coset j of the zeta-coset extension of the coefficients
    ext = O.coset_ntt(coeff, k, k + ext_bits, RC.ZETA)
    tab = P.Tables(k)
    wN = O.omega(k + ext_bits)
    src = RC.Dev().put(coeff)
    tmp = torch.empty((n, 4), dtype=torch.int64, device="cuda")
    if pairs:
        twp = torch.empty((2 * n, 4), dtype=torch.int64, device="cuda")
        assert L.zkp_shoup_pairs(twp.data_ptr(), tab.tw.data_ptr(), n, 0) == 0
    for j in range(E):
        sj = RC.ZETA * pow(wN, j, O.R_MOD) % O.R_MOD
        twist = P.powers(1, sj, n)
        out = torch.empty((n, 4), dtype=torch.int64, device="cuda")
        if pairs:
            tp = torch.empty((2 * n, 4), dtype=torch.int64, device="cuda")
            assert L.zkp_shoup_pairs(tp.data_ptr(), twist.data_ptr(), n, 0) == 0
            assert L.zkp_ntt_batch_twisted(out.data_ptr(), src.data_ptr(), tmp.data_ptr(), twp.data_ptr(),
                                           tp.data_ptr(), 0, k, 1, n, n, 1, 0) == 0
        else:
            assert L.zkp_ntt_batch_twisted(out.data_ptr(), src.data_ptr(), tmp.data_ptr(), tab.tw.data_ptr(),
                                           twist.data_ptr(), 0, k, 1, n, n, 0, 0) == 0
        assert (_h(out) == ext[j::E]).all(), f"coset {j}"
    # backward: arbitrary values h on the extended domain, divided by Z_H per
    # coset, to coefficients with the coset undone
    hv = O.rand_fr(N, 95)
    t = [pow((pow(RC.ZETA * pow(wN, j, O.R_MOD), n, O.R_MOD) - 1) % O.R_MOD, -1, O.R_MOD) for j in range(E)]
    exp = O.field_mul_zip(hv, O.fr_vec(t))
    exp = O.intt(exp, k + ext_bits)
    exp = O.extended_prepare(exp, O.fr_vec([pow(RC.ZETA, -1, O.R_MOD), RC.ZETA]), 3, n, N, True)
    hc = RC.Dev().put(np.concatenate([O.mul(hv[j::E], O.fr_vec([t[j]])) for j in range(E)]))
    g = torch.empty_like(hc)
    tmpE = torch.empty_like(hc)
    assert L.zkp_ntt_batch_twisted(g.data_ptr(), hc.data_ptr(), tmpE.data_ptr(), tab.tw_inv.data_ptr(), 0,
                                   tab.n_inv.data_ptr(), k, E, n, n, 0, 0) == 0
    winv = P.powers(1, pow(wN, -1, O.R_MOD), n)
    wE = pow(wN, n, O.R_MOD)
    consts = P.fr_tensor([1] * E + [pow(wE, -kk, O.R_MOD) for kk in range(E)] +
                         [pow(RC.ZETA, -kk, O.R_MOD) * pow(E, -1, O.R_MOD) % O.R_MOD for kk in range(3)])
    out = torch.empty((N, 4), dtype=torch.int64, device="cuda")
    assert L.zkp_coset_combine(out.data_ptr(), g.data_ptr(), n, winv.data_ptr(), consts.data_ptr(), k, ext_bits,
                               0) == 0
    assert (_h(out) == exp).all()


# the factors of zkp_ntt_batch_twisted are any, not only the powers of a shift:
# short and radix-8 passes (7+6, 9+9, 11+6+6), both table layouts
@pytest.mark.parametrize("log_n,cols", [(12, 2), (13, 2), (13, 64), (18, 2), (23, 1)])
@pytest.mark.parametrize("pairs", [False, True])
@pytest.mark.parametrize("factors", ["random", "scaled"])
def test_twisted_transform_takes_any_factors(O, gpu, P, log_n, cols, pairs, factors):
    L = gpu.load_library()
    n = 1 << log_n
    tab = P.Tables(log_n)
    if factors == "random":
        mul = O.rand_fr(n, 230 + log_n)
    else:  # c s^k, whose first entry is not one
        c, s = O.fr_ints(O.rand_fr(2, 231))
        mul = O.mul(_h(P.powers(1, s, n)), O.fr_vec([c]))
    tw, tm = tab.tw, RC.Dev().put(mul)
    if pairs:
        tw, tp = (torch.empty((2 * n, 4), dtype=torch.int64, device="cuda") for _ in range(2))
        assert L.zkp_shoup_pairs(tw.data_ptr(), tab.tw.data_ptr(), n, 0) == 0
        assert L.zkp_shoup_pairs(tp.data_ptr(), tm.data_ptr(), n, 0) == 0
        tm = tp
    x = O.rand_fr(cols * n, 232)
    src = RC.Dev().put(x)
    tmp, out = (torch.empty((cols * n, 4), dtype=torch.int64, device="cuda") for _ in range(2))
    assert L.zkp_ntt_batch_twisted(out.data_ptr(), src.data_ptr(), tmp.data_ptr(), tw.data_ptr(), tm.data_ptr(), 0,
                                   log_n, cols, n, n, int(pairs), 0) == 0
    got = _h(out)
    for c in {0, cols // 2, cols - 1}:
        exp = O.ntt(O.mul(x[c * n:(c + 1) * n], mul), log_n)
        assert (got[c * n:(c + 1) * n] == exp).all(), c


# powers of a shift in two passes with every remainder of the in-block radix
# (7+6, 6+8, 9+9, 11+10) and three (11+6+6), strides wider than a column
@pytest.mark.parametrize("log_n", [13, 14, 16, 18, 21, 23])
@pytest.mark.parametrize("pairs", [False, True])
def test_coset_transform_of_several_passes(O, gpu, P, log_n, pairs):
    L = gpu.load_library()
    n, cols, stride = 1 << log_n, 2, (1 << log_n) + 24
    tab = P.Tables(log_n)
    w2 = O.omega(log_n + 1)
    shift = RC.ZETA * w2 % O.R_MOD
    twist = P.powers(1, shift, n)
    tw = tab.tw
    if pairs:
        tw, tp = (torch.empty((2 * n, 4), dtype=torch.int64, device="cuda") for _ in range(2))
        assert L.zkp_shoup_pairs(tw.data_ptr(), tab.tw.data_ptr(), n, 0) == 0
        assert L.zkp_shoup_pairs(tp.data_ptr(), twist.data_ptr(), n, 0) == 0
        twist = tp
    coeff = O.rand_fr(cols * stride, 190 + log_n)
    src = RC.Dev().put(coeff)
    tmp = torch.empty((cols * n, 4), dtype=torch.int64, device="cuda")
    out = torch.empty((cols * stride, 4), dtype=torch.int64, device="cuda")
    assert L.zkp_ntt_batch_twisted(out.data_ptr(), src.data_ptr(), tmp.data_ptr(), tw.data_ptr(), twist.data_ptr(), 0,
                                   log_n, cols, stride, stride, int(pairs), 0) == 0
    got = _h(out)
    for c in range(cols if log_n < 20 else 1):
        exp = O.coset_ntt(coeff[c * stride:c * stride + n], log_n, log_n + 1, RC.ZETA)[1::2]
        assert (got[c * stride:c * stride + n] == exp).all(), c


def test_eval_h_fused_matches_restatement(O, gpu, P):
    """Every family of zkp_eval_h_fused on random columns (rotation scale 2,
    as on a whole extended domain of E = 2) against the oracle's restatement of
    the reference's kernels in their chain order."""
    L = gpu.load_library()
    n, rs = 1 << 10, 2
    R = O.R_MOD
    rnd = iter(range(300, 10_000))
    col = lambda: O.rand_fr(n, next(rnd))  # noqa: E731
    y, beta, gamma = [O.fr_ints(O.rand_fr(1, s))[0] for s in (1, 2, 3)]
    yv, bv, gv = O.fr_vec([y]), O.fr_vec([beta]), O.fr_vec([gamma])
    l0, ll, la, X = col(), col(), col(), col()
    d = RC.Dev()
    # gates: two terms with rotations of both signs
    gcols = [col() for _ in range(4)]
    gco = O.rand_fr(2, 9)
    terms = [(gco[0:1], [(gcols[0], 0), (gcols[1], 1)]), (gco[1:2], [(gcols[2], -1), (gcols[3], 2)])]
    v, rots = [], []
    for c_, fs in terms:
        v.append(d.put(c_))
        for cc, r in fs:
            v.append(d.put(cc))
            rots.append(r)
        v.append(None)
    # permutation: 5 columns in chunks of 2
    pc = [col() for _ in range(5)]
    ps = [col() for _ in range(5)]
    pz = [col() for _ in range(3)]
    db = [beta * pow(P.DELTA, c, R) % R for c in range(5)]
    last = -3
    # lookups and shuffles
    lk = [[col() for _ in range(4)] for _ in range(2)]
    sh = [[col() for _ in range(5)]]  # z, (in, tab) x 2
    sbetas = [pow(beta, i + 1, R) for i in range(2)]
    scale = O.rand_fr(1, 11)
    a = P._EvalHArgs()
    a.n, a.rot_scale = n, rs
    keep = [d.put(yv), d.ptrs(v), d.i32(rots), d.put(l0), d.put(ll), d.put(la), d.put(X), d.put(bv), d.put(gv),
            d.ptrs([d.put(z) for z in pz]), d.ptrs([d.put(c_) for c_ in pc]), d.ptrs([d.put(c_) for c_ in ps]),
            d.put(O.fr_vec(db)), d.ptrs([d.put(c_) for q in lk for c_ in q]),
            d.ptrs([d.put(c_) for q in sh for c_ in q]), d.i32([2]), d.put(O.fr_vec(sbetas)), d.put(scale)]
    (a.y, a.gate_terms, a.gate_rots, a.l0, a.l_last, a.l_active, a.x, a.beta, a.gamma, a.perm_z, a.perm_cols,
     a.perm_sigmas, a.perm_dbeta, a.lookup_cols, a.shuffle_cols, a.shuffle_group_len, a.shuffle_betas,
     a.scale) = [t.data_ptr() for t in keep]
    a.gate_terms_n = len(v)
    a.perm_chunks, a.perm_chunk_len, a.perm_cols_n, a.perm_last_rot = 3, 2, 5, last
    a.lookups, a.shuffles = 2, 1
    h = torch.empty((n, 4), dtype=torch.int64, device="cuda")
    assert L.zkp_eval_h_fused(h.data_ptr(), ctypes.byref(a), 0) == 0
    # restatement in the chain order of src/eval_h.rs (rotations scaled by rs)
    sc_terms = [(c_, [(cc, r * rs) for cc, r in fs]) for c_, fs in terms]
    t = O.field_op_batch_mul_sum(O.zeros(n), sc_terms, n)
    t = O.permutation_eval_h_p1(t, pz[0], pz[-1], l0, ll, yv)
    t = O.permutation_eval_h_p2(t, pz, l0, ll, yv, last * rs)
    for j in range(3):
        Lp, Rp = O._rot(pz[j], rs), pz[j]
        for c in range(2 * j, min(5, 2 * j + 2)):
            Lp = O.mul(Lp, O.add(O.add(pc[c], O.mul(ps[c], bv)), gv))
            Rp = O.mul(Rp, O.add(O.add(pc[c], O.mul(X, O.fr_vec([db[c]]))), gv))
        t = O.add(O.mul(t, yv), O.mul(la, O.sub(Lp, Rp)))
    for q in lk:
        fb, tb = O.add(q[0], bv), O.add(q[1], bv)
        t = O.logup_eval_h(t, fb, O.one(n), tb, q[2], q[3], q[3], l0, ll, la, yv, rs)
    for q in sh:
        t = O.shuffle_eval_h_v2(t, [q[1], q[3]], [q[2], q[4]], O.fr_vec(sbetas), q[0], l0, ll, la, yv, rs)
    t = O.mul(t, scale)
    assert (_h(h) == t).all()


def _eval_h_both(O, gpu, P, n, rs, terms, chunks, chunk_len, lookups, groups, scaled=True):
    """zkp_eval_h_fused and the oracle's chain over random columns: gate terms
    as lists of rotations, `chunks` permutation chunks, `lookups`, and one
    shuffle for each of `groups` (input, table) pair counts."""
    L, R = gpu.load_library(), O.R_MOD
    rnd = iter(range(5000, 100_000))
    pool = [O.rand_fr(n, next(rnd)) for _ in range(24)]  # columns, reused in turn
    at = iter(range(10 ** 6))
    col = lambda: pool[next(at) % len(pool)]  # noqa: E731
    y, beta, gamma = [O.fr_ints(O.rand_fr(1, s))[0] for s in (21, 22, 23)]
    yv, bv, gv = O.fr_vec([y]), O.fr_vec([beta]), O.fr_vec([gamma])
    d = RC.Dev()
    dev = [d.put(c) for c in pool]
    at_dev = lambda c: next(t for p, t in zip(pool, dev) if p is c)  # noqa: E731
    l0, ll, la, X = pool[20], pool[21], pool[22], pool[23]
    gates = [(O.rand_fr(1, next(rnd)), [(col(), r) for r in rots]) for rots in terms]
    v, rots = [], []
    for c_, fs in gates:
        v.append(d.put(c_))
        v += [at_dev(cc) for cc, _ in fs]
        rots += [r for _, r in fs]
        v.append(None)
    m = max(0, chunks * chunk_len - 1)  # the last chunk is a column short
    pc, ps, pz = [col() for _ in range(m)], [col() for _ in range(m)], [col() for _ in range(chunks)]
    db = [beta * pow(P.DELTA, c, R) % R for c in range(m)]
    lk = [[col() for _ in range(4)] for _ in range(lookups)]
    sh = [[col() for _ in range(1 + 2 * g)] for g in groups]
    sbetas = [pow(beta, i + 1, R) for i in range(max(groups, default=1))]
    last = -3
    a = P._EvalHArgs()
    a.n, a.rot_scale = n, rs
    keep = [d.put(yv), d.put(bv), d.put(gv)]
    a.y, a.beta, a.gamma = [t.data_ptr() for t in keep]
    a.l0, a.l_last, a.l_active, a.x = [at_dev(c).data_ptr() for c in (l0, ll, la, X)]

    def put(name, t):
        keep.append(t)
        setattr(a, name, t.data_ptr())

    if gates:
        put("gate_terms", d.ptrs(v))
        put("gate_rots", d.i32(rots or [0]))
    if chunks:
        put("perm_z", d.ptrs([at_dev(c) for c in pz]))
        put("perm_cols", d.ptrs([at_dev(c) for c in pc]))
        put("perm_sigmas", d.ptrs([at_dev(c) for c in ps]))
        put("perm_dbeta", d.put(O.fr_vec(db)))
    if lookups:
        put("lookup_cols", d.ptrs([at_dev(c) for q in lk for c in q]))
    if groups:
        put("shuffle_cols", d.ptrs([at_dev(c) for q in sh for c in q]))
        put("shuffle_group_len", d.i32(list(groups)))
        put("shuffle_betas", d.put(O.fr_vec(sbetas)))
    scale = O.rand_fr(1, 24)
    if scaled:
        put("scale", d.put(scale))
    a.gate_terms_n = len(v)
    a.perm_chunks, a.perm_chunk_len, a.perm_cols_n, a.perm_last_rot = chunks, chunk_len, m, last
    a.lookups, a.shuffles = lookups, len(groups)
    h = torch.empty((n, 4), dtype=torch.int64, device="cuda")
    assert L.zkp_eval_h_fused(h.data_ptr(), ctypes.byref(a), 0) == 0
    t = O.field_op_batch_mul_sum(O.zeros(n), [(c_, [(cc, r * rs) for cc, r in fs]) for c_, fs in gates], n)
    if chunks:
        t = O.permutation_eval_h_p1(t, pz[0], pz[-1], l0, ll, yv)
        t = O.permutation_eval_h_p2(t, pz, l0, ll, yv, last * rs)
    for j in range(chunks):
        Lp, Rp = O._rot(pz[j], rs), pz[j]
        for c in range(chunk_len * j, min(m, chunk_len * (j + 1))):
            Lp = O.mul(Lp, O.add(O.add(pc[c], O.mul(ps[c], bv)), gv))
            Rp = O.mul(Rp, O.add(O.add(pc[c], O.mul(X, O.fr_vec([db[c]]))), gv))
        t = O.add(O.mul(t, yv), O.mul(la, O.sub(Lp, Rp)))
    for q in lk:
        t = O.logup_eval_h(t, O.add(q[0], bv), O.one(n), O.add(q[1], bv), q[2], q[3], q[3], l0, ll, la, yv, rs)
    for q in sh:
        t = O.shuffle_eval_h_v2(t, q[1::2], q[2::2], O.fr_vec(sbetas), q[0], l0, ll, la, yv, rs)
    if scaled:
        t = O.mul(t, scale)
    return _h(h), t


# every combination of absent families, one and several shuffles, and both block
# sizes (128 threads up to 151552 rows, 256 above)
@pytest.mark.parametrize("n", [1, 64, 1 << 10, 1 << 18])
@pytest.mark.parametrize("gates,chunks,lookups,groups", [
    (3, 0, 0, ()), (0, 3, 0, ()), (0, 0, 2, ()), (0, 0, 0, (2,)), (2, 1, 0, ()), (2, 2, 0, (1, 3)),
    (2, 0, 3, (2, 1)), (1, 3, 2, (1, 2, 3))])
def test_eval_h_fused_families(O, gpu, P, n, gates, chunks, lookups, groups):
    terms = [[0], [1, -1, 2], [-2, 0]][:gates]
    got, exp = _eval_h_both(O, gpu, P, n, 1 if n < 1 << 10 else 2, terms, chunks, 2, lookups, groups, n != 64)
    assert (got == exp).all()


# gate lists longer than the coefficients staged per block (entries below 256):
# terms that start on either side of the line, coefficients without a column
@pytest.mark.parametrize("tail", [[0, 0, 0, 2, 1], [0, 2, 1, 0, 3], [1, 1, 1, 0]])
def test_eval_h_fused_long_gate_lists(O, gpu, P, tail):
    terms = [[t % 3 - 1] for t in range(84)] + [[i - 1 for i in range(k)] for k in tail]  # the tail starts at 252
    got, exp = _eval_h_both(O, gpu, P, 1 << 10, 1, terms, 2, 3, 1, (1,))
    assert (got == exp).all()
