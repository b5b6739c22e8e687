"""Performance cases: the calls a prover makes of this library, with their sizes.

A case is a dict of plain values whose "kind" names the call:

  msm        one multi-scalar multiplication (zkp_msm through host.msm)
  commit     a pipeline of column commitments over the SRS table
             (host.msm_batch_table), the prover's commitment phases
  uneven     a pipeline of MSMs of different sizes over prefixes of the SRS
             (host.msm_batch)
  dropin     the reference host's calls: one msm() per column, then
             batch_msm_collect (host.ReferenceMsmBatch)
  ntt        drop-in ntt() of one column (host.ntt_raw)
  ntt_batch  batched transforms of whole columns in place (host.ntt_batch)
  coset      the quotient's coset transform, out of place (prover.ntt_into)
  extend     Lagrange columns to coefficients and the extended domain
             (host.extend_batch_tables)
  products   the grand products and sums of one argument each: a permutation
             chunk (zkp_permutation_z), a shuffle (zkp_shuffle_z) and a logup
             lookup (logup_sum_input_inv, eval_logup_z_compose)
  quotient   every constraint over one coset's rows (zkp_eval_h_fused)
  proof      one whole proof of a synthetic circuit (prover.HotPath.prove)

Every result is exact: field elements in canonical Montgomery form, and the
points of the MSM kinds as affine coordinates (the Jacobian representative is
not part of the contract; a host converts it, as the transcript needs).
"""
import ctypes
import importlib
import math

import numpy as np
import torch

PKG = "zkwasm-prover_b200"
Z = importlib.import_module(PKG)
P = importlib.import_module(PKG + ".prover")
H = Z.host

SCALARS = ("uniform", "small", "sparse", "mixed")


# ---------------------------------------------------------------- the cases


def listed():
    return [
        # a commitment to a short column (an instance column, a test circuit):
        # launches and latency
        {"name": "msm_1k", "kind": "msm", "n": 1 << 10, "scalars": "uniform"},
        # a witness column that is no power of two long, small values
        {"name": "msm_100k_small", "kind": "msm", "n": 100003, "scalars": "small"},
        # the commitment phases of a k = 20 proof: eight columns a pipeline
        {"name": "commit_8x1m", "kind": "commit", "n": 1 << 20, "count": 8, "scalars": "uniform"},
        # columns of many lengths and distributions over one SRS
        {"name": "uneven_24", "kind": "uneven", "n_min": 3001, "n_max": 1 << 18, "count": 24, "scalars": "mixed"},
        # an unchanged reference host: one msm() a column, then the collect
        {"name": "dropin_4x64k", "kind": "dropin", "n": 1 << 16, "count": 4, "scalars": "uniform"},
        # one short column through the drop-in transform: latency
        {"name": "ntt_8k", "kind": "ntt", "log_n": 13, "inverse": False},
        # advice columns to coefficients, k = 18
        {"name": "intt_16x256k", "kind": "ntt_batch", "log_n": 18, "cols": 16, "inverse": True},
        # one coset of eight quotient columns, k = 21
        {"name": "coset_8x2m", "kind": "coset", "log_n": 21, "cols": 8},
        # eight columns to the extended domain, k = 18, e = 3
        {"name": "extend_8x256k", "kind": "extend", "log_n": 18, "ext_bits": 3, "cols": 8},
        # the running products and sums of k = 20
        {"name": "products_1m", "kind": "products", "n": 1 << 20, "perm": 7},
        # the constraints of one coset, k = 17, at the column counts of the
        # SHPLONK shape (120 advice, 60 permutation columns, 24 lookups)
        {"name": "quotient_128k", "kind": "quotient", "log_n": 17, "gates": 17, "perm": 60, "chunk": 7, "lookups": 24,
         "shuffles": 4},
        # a whole proof of a small circuit: every phase, its launches and the
        # host's work between them
        {"name": "proof_k15", "kind": "proof", "k": 15, "advice": 40, "fixed": 10, "lookups": 6, "shuffles": 2,
         "perm": 20, "degree": 9, "multiopen": "shplonk"},
    ]


def _spread(rng, lo, hi):
    """A whole number from lo to hi, its logarithm uniform; often odd."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("msm", "msm", "commit", "uneven", "dropin", "ntt", "ntt_batch", "coset", "extend", "products",
                       "quotient", "proof"))
    if kind == "msm":
        return {"kind": kind, "n": _spread(rng, 1000, 1 << 21), "scalars": rng.choice(SCALARS[:3])}
    if kind == "commit":
        count = rng.randint(1, 8)
        return {"kind": kind, "n": _spread(rng, 1 << 14, (8 << 20) // count if count > 4 else 1 << 21),
                "count": count, "scalars": rng.choice(SCALARS)}
    if kind == "uneven":
        lo = _spread(rng, 500, 1 << 14)
        return {"kind": kind, "n_min": lo, "n_max": _spread(rng, 2 * lo, 1 << 18), "count": rng.randint(2, 32),
                "scalars": rng.choice(SCALARS)}
    if kind == "dropin":
        return {"kind": kind, "n": _spread(rng, 5000, 1 << 19), "count": rng.randint(1, 8),
                "scalars": rng.choice(SCALARS)}
    if kind == "ntt":
        return {"kind": kind, "log_n": rng.randint(10, 24), "inverse": rng.random() < 0.5}
    if kind == "ntt_batch":
        log_n = rng.randint(11, 21)
        return {"kind": kind, "log_n": log_n, "cols": rng.randint(1, min(33, 1 << (24 - log_n))),
                "inverse": rng.random() < 0.5}
    if kind == "coset":
        log_n = rng.randint(12, 22)
        return {"kind": kind, "log_n": log_n, "cols": rng.randint(1, min(33, 1 << (24 - log_n)))}
    if kind == "extend":
        log_n, e = rng.randint(13, 20), rng.randint(1, 3)
        return {"kind": kind, "log_n": log_n, "ext_bits": e, "cols": rng.randint(1, min(16, 1 << (24 - log_n - e)))}
    if kind == "products":
        return {"kind": kind, "n": _spread(rng, 4000, 1 << 21), "perm": rng.randint(1, 8)}
    if kind == "quotient":
        return {"kind": kind, "log_n": rng.randint(13, 17), "gates": rng.randint(1, 17), "perm": rng.randint(4, 60),
                "chunk": rng.randint(2, 7), "lookups": rng.randint(1, 24), "shuffles": rng.randint(1, 4)}
    advice = rng.randint(16, 40)
    return {"kind": "proof", "k": rng.randint(12, 15), "advice": advice, "fixed": 10, "lookups": rng.randint(1, 4),
            "shuffles": rng.randint(1, 2), "perm": rng.randint(6, 10), "degree": rng.choice((4, 5, 9)),
            "multiopen": rng.choice(("shplonk", "gwc"))}


# ---------------------------------------------------------------- inputs


def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + salt) & (2 ** 62 - 1))
    return g


def _column(n, g):
    """n seeded uniform field elements (canonical Montgomery form)."""
    t = torch.randint(-(2 ** 63), 2 ** 63 - 1, (n, 4), dtype=torch.int64, device="cuda", generator=g)
    t[:, 3] &= (1 << 61) - 1
    return t


def _scalars(n, kind, g):
    """Scalars as columns hold them: uniform values, small values (range-checked
    cells, below 2^20), or columns that are zero in nine rows of ten."""
    if kind == "uniform":
        return _column(n, g)
    if kind == "small":
        return P.small_fr(torch.randint(0, 1 << 20, (n,), device="cuda", generator=g))
    t = _column(n, g)
    return torch.where((torch.randint(0, 10, (n, 1), device="cuda", generator=g) == 0), t, torch.zeros_like(t))


def _scalar_kind(case, i):
    return SCALARS[i % 3] if case["scalars"] == "mixed" else case["scalars"]


def _sizes(case):
    """The uneven kind's lengths: from n_min to n_max in even steps of their
    logarithm, long and short ones alternating."""
    c = case["count"]
    a = [int(round(case["n_min"] * (case["n_max"] / case["n_min"]) ** (i / max(1, c - 1)))) for i in range(c)]
    return a[0::2] + a[1::2][::-1]


def _multiples(n, seed):
    return torch.randint(1, 2 ** 62, (n,), dtype=torch.int64, device="cuda", generator=_gen(seed, 1))


def _bases(n, seed):
    """n SRS-style points [k_i] G."""
    k = _multiples(n, seed)
    out = torch.empty((n, 8), dtype=torch.int64, device="cuda")
    Z.abi.check(H.lib().zkp_g1_multiples(out.data_ptr(), k.data_ptr(), n, H.stream_handle()), "zkp_g1_multiples")
    return out


def _msm_lengths(case):
    if case["kind"] == "uneven":
        return _sizes(case)
    return [case["n"]] * case.get("count", 1)


def _msm_scalars(case, seed):
    return [_scalars(n, _scalar_kind(case, i), _gen(seed, 2 + i)) for i, n in enumerate(_msm_lengths(case))]


def _powers(w, n):
    return P.powers(1, w, n)


class _EvalHArgs(ctypes.Structure):
    """zkp_eval_h_args of include/zkwasm_prover_kernel.h."""
    _fields_ = [("n", ctypes.c_uint32), ("rot_scale", ctypes.c_int), ("y", ctypes.c_void_p),
                ("gate_terms", ctypes.c_void_p), ("gate_rots", ctypes.c_void_p), ("gate_terms_n", ctypes.c_int),
                ("l0", ctypes.c_void_p), ("l_last", ctypes.c_void_p), ("l_active", ctypes.c_void_p),
                ("x", ctypes.c_void_p), ("beta", ctypes.c_void_p), ("gamma", ctypes.c_void_p),
                ("perm_chunks", ctypes.c_int), ("perm_chunk_len", ctypes.c_int), ("perm_cols_n", ctypes.c_int),
                ("perm_last_rot", ctypes.c_int), ("perm_z", ctypes.c_void_p), ("perm_cols", ctypes.c_void_p),
                ("perm_sigmas", ctypes.c_void_p), ("perm_dbeta", ctypes.c_void_p), ("lookups", ctypes.c_int),
                ("lookup_cols", ctypes.c_void_p), ("shuffles", ctypes.c_int), ("shuffle_cols", ctypes.c_void_p),
                ("shuffle_group_len", ctypes.c_void_p), ("shuffle_betas", ctypes.c_void_p),
                ("scale", ctypes.c_void_p)]


def _quotient_state(case, g):
    n = 1 << case["log_n"]
    keep = []

    def cols(m):
        t = torch.stack([_column(n, g) for _ in range(m)])
        keep.append(t)
        return [t[i].data_ptr() for i in range(m)]

    def ptrs(xs):
        t = H.to_device(np.array(xs, dtype=np.uint64))
        keep.append(t)
        return t.data_ptr()

    def consts(m):
        t = _column(m, g)
        keep.append(t)
        return [t[i:i + 1].data_ptr() for i in range(m)]

    terms, G = [], case["gates"]
    for cf in [consts(3) for _ in range(G)]:  # q (a b c + d) - e
        q, a, b, c, d, e = cols(6)
        terms += [cf[0], q, a, b, c, 0, cf[1], q, d, 0, cf[2], q, e, 0]
    rots = torch.zeros(8 * G, dtype=torch.int32, device="cuda")
    group = torch.ones(case["shuffles"], dtype=torch.int32, device="cuda")
    keep += [rots, group]
    a = _EvalHArgs()
    a.n, a.rot_scale = n, 1
    a.y, a.beta, a.gamma, a.scale = consts(4)
    a.gate_terms, a.gate_rots, a.gate_terms_n = ptrs(terms), rots.data_ptr(), len(terms)
    a.l0, a.l_last, a.l_active, a.x = cols(4)
    a.perm_chunks = -(-case["perm"] // case["chunk"])
    a.perm_chunk_len, a.perm_cols_n, a.perm_last_rot = case["chunk"], case["perm"], -5
    a.perm_z, a.perm_cols, a.perm_sigmas = (ptrs(cols(a.perm_chunks)), ptrs(cols(case["perm"])),
                                            ptrs(cols(case["perm"])))
    a.perm_dbeta = consts(case["perm"])[0]
    table = cols(1)[0]
    lk = []
    for _ in range(case["lookups"]):
        f, m, z = cols(3)
        lk += [f, table, m, z]
    a.lookups, a.lookup_cols = case["lookups"], ptrs(lk)
    a.shuffles, a.shuffle_cols = case["shuffles"], ptrs(sum((cols(3) for _ in range(case["shuffles"])), []))
    a.shuffle_group_len, a.shuffle_betas = group.data_ptr(), consts(4)[0]
    return {"args": a, "keep": keep, "h": H.empty_fr(n)}


def _products_state(case, g):
    n, m = case["n"], case["perm"]
    log_n = (n - 1).bit_length()
    st = {"n": n, "cols": [_column(n, g) for _ in range(m)], "sigmas": [_column(n, g) for _ in range(m)],
          "beta": _column(1, g), "gamma": _column(1, g), "dbeta": _column(m, g), "init": _column(1, g),
          "omegas": _powers(P.omega(log_n), n), "a": _column(n, g), "b": _column(n, g),
          "input": P.small_fr(torch.randint(0, 1 << 16, (n,), device="cuda", generator=g)),
          "table": P.small_fr(torch.arange(n, device="cuda") % (1 << 16)),
          "mult": P.small_fr(torch.randint(0, 50, (n,), device="cuda", generator=g)),
          "scratch": H.empty_fr(n + H.lib().zkp_scan_scratch_elems(n))}
    st["pc"], st["ps"] = H.ptr_array(st["cols"]), H.ptr_array(st["sigmas"])
    st["pi"], st["pt"] = H.ptr_array([st["a"]]), H.ptr_array([st["b"]])
    for k in ("z", "sz", "sum", "lz", "tmp", "tcopy"):
        st[k] = H.empty_fr(n)
    st["last"] = H.zeros_fr(1)
    return st


def prepare(case, seed):
    kind = case["kind"]
    g = _gen(seed)
    if kind in ("msm", "commit", "uneven", "dropin"):
        lens = _msm_lengths(case)
        top = max(lens)
        bases, cols = _bases(top, seed), _msm_scalars(case, seed)
        st = {"case": case, "bases": bases, "cols": cols, "lens": lens, "ptrs": H.ptr_array(cols)}
        n_arr = (ctypes.c_uint32 * len(lens))(*lens)
        if kind == "msm":
            st["scratch"] = H.msm_scratch(top)
        elif kind == "commit":
            # the table of the SRS is part of the proving key
            c = H.lib().zkp_msm_batch_table_default_window(ctypes.addressof(n_arr), len(lens))
            st["table"], st["c"] = H.msm_table_build(bases, top, c)
            nbytes = H.lib().zkp_msm_batch_table_scratch_bytes(ctypes.addressof(n_arr), len(lens), top, c)
            st["scratch"] = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        elif kind == "uneven":
            nbytes = H.lib().zkp_msm_batch_scratch_bytes(ctypes.addressof(n_arr), None, len(lens))
            st["scratch"] = torch.empty(max(1, nbytes), dtype=torch.uint8, device="cuda")
        else:
            st["batch"] = H.ReferenceMsmBatch(bases, cols, top)
        return st
    if kind in ("ntt", "ntt_batch", "coset"):
        log_n, cols = case["log_n"], case.get("cols", 1)
        st = {"case": case, "tables": P.Tables(log_n), "buf": _column(cols << log_n, g),
              "tmp": H.empty_fr(cols << log_n)}
        if kind == "coset":
            st["twist"] = _powers(P.ZETA * P.omega(log_n + 2) % P.R_MOD, 1 << log_n)
            st["out"] = H.empty_fr(cols << log_n)
        return st
    if kind == "extend":
        log_n, e, cols = case["log_n"], case["ext_bits"], case["cols"]
        t = P.Tables(log_n)
        mont = lambda x: np.array(P.limbs(x), dtype=np.uint64)  # noqa: E731
        tables = H.extend_tables(t.tw, t.tw_inv, t.n_inv, mont(P.ZETA), mont(P.omega(log_n + e)), log_n, e)
        return {"case": case, "tables": tables, "lagrange": _column(cols << log_n, g),
                "coeff": H.empty_fr(cols << log_n), "ext": H.empty_fr(cols << (log_n + e)),
                "scratch": H.empty_fr(cols << (log_n + e))}
    if kind == "products":
        return {"case": case, **_products_state(case, g)}
    if kind == "quotient":
        return {"case": case, **_quotient_state(case, g)}
    shape = P.Shape(**{k: v for k, v in case.items() if k not in ("name", "kind")})
    return {"case": case, "prover": P.HotPath(P.Circuit(shape, seed=int(seed) % (1 << 31)), "batched",
                                              seed=int(seed) % (1 << 31), pk_cache_gib=1.0)}


# ---------------------------------------------------------------- one pass


def _points(points):
    """Affine points as the transcript takes them: (count, 8) words."""
    words = [[(v >> (64 * j)) & 0xFFFFFFFFFFFFFFFF for v in pt for j in range(4)] for pt in points]
    return np.array(words, dtype=np.uint64).reshape(-1, 8).view(np.int64)


def _affine(jac):
    return _points(P.jac_to_affine(jac))


def _run_products(s):
    L, n, st = H.lib(), s["n"], H.stream_handle()
    p = lambda k: s[k].data_ptr()  # noqa: E731
    Z.abi.check(L.zkp_permutation_z(p("z"), p("pc"), p("ps"), s["case"]["perm"], p("beta"), p("gamma"), p("dbeta"),
                                    p("omegas"), p("init"), n, p("scratch"), st), "zkp_permutation_z")
    Z.abi.check(L.zkp_shuffle_z(p("sz"), p("pi"), p("pt"), p("beta"), 1, n, p("scratch"), st), "zkp_shuffle_z")
    Z.abi.check(L.logup_sum_input_inv(p("sum"), p("input"), p("tmp"), p("beta"), 0, n, st), "logup_sum_input_inv")
    s["tcopy"].copy_(s["table"])  # the call uses the table as scratch
    s["last"].zero_()
    Z.abi.check(L.eval_logup_z_compose(p("lz"), p("sum"), p("tcopy"), p("mult"), p("beta"), p("last"), n - 6, n, st),
                "eval_logup_z_compose")
    return [s["z"], s["sz"], s["lz"], s["last"]]


def run(s):
    kind = s["case"]["kind"] if "case" in s else None
    if kind == "msm":
        return _affine(H.to_host(H.msm(s["bases"], s["cols"][0], scratch=s["scratch"])))
    if kind == "commit":
        return _affine(H.to_host(H.msm_batch_table(s["table"], max(s["lens"]), s["c"], s["cols"], s["lens"],
                                                   scratch=s["scratch"], ptrs=s["ptrs"])))
    if kind == "uneven":
        return _affine(H.to_host(H.msm_batch(s["bases"], s["cols"], s["lens"], scratch=s["scratch"],
                                             ptrs=s["ptrs"])))
    if kind == "dropin":
        s["batch"].enqueue()
        return _affine(s["batch"].results())
    if kind == "ntt":
        t, c = s["tables"], s["case"]
        inv = c["inverse"]
        s["buf"], s["tmp"] = H.ntt_raw(s["buf"], s["tmp"], t.pq_inv if inv else t.pq, t.tw_inv if inv else t.tw,
                                       c["log_n"], t.n_inv if inv else None)
        return s["buf"]
    if kind == "ntt_batch":
        t, c = s["tables"], s["case"]
        inv = c["inverse"]
        r = H.ntt_batch(s["buf"], s["tmp"], t.tw_inv if inv else t.tw, c["log_n"], c["cols"],
                        t.n_inv if inv else None)
        if r is s["tmp"]:
            s["buf"], s["tmp"] = s["tmp"], s["buf"]
        return r
    if kind == "coset":
        P.ntt_into(s["out"], s["buf"], s["tables"], s["case"]["cols"], False, in_mul=s["twist"], tmp=s["tmp"])
        return s["out"]
    if kind == "extend":
        c = s["case"]
        H.extend_batch_tables(s["ext"], s["coeff"], s["lagrange"], c["cols"], c["log_n"], c["ext_bits"], s["tables"],
                              s["scratch"])
        return [s["ext"], s["coeff"]]
    if kind == "products":
        return _run_products(s)
    if kind == "quotient":
        Z.abi.check(H.lib().zkp_eval_h_fused(s["h"].data_ptr(), ctypes.byref(s["args"]), H.stream_handle()),
                    "zkp_eval_h_fused")
        return s["h"]
    proof = s["prover"].prove()
    evals = np.array([P.limbs(e, mont=False) for e in proof["evals"]], dtype=np.uint64).view(np.int64)
    return [_points([pt for _, pts in proof["commitments"] for pt in pts]), evals]


# ---------------------------------------------------------------- work and tolerance


# 32-bit multiply-adds (two operations each) of one 254-bit modular product:
# 64 for the product of eight-word factors, 64 for the reduction
_PRODUCT = 2 * 128


def _msm_products(n):
    """A bucket method with windows of about log2 n bits: one point addition
    (six products at least) a point and window of the 254-bit scalar."""
    return 6 * n * math.ceil(254 / max(4, math.log2(max(2, n))))


def work(case):
    kind = case["kind"]
    if kind in ("msm", "commit", "uneven", "dropin"):
        lens = _msm_lengths(case)
        share = {"uniform": 1.0, "small": 20 / 254, "sparse": 0.1}
        prod = sum(_msm_products(n) * share[_scalar_kind(case, i)] for i, n in enumerate(lens))
        return {"bytes": 64 * max(lens) + 32 * sum(lens) + 96 * len(lens), "flops": _PRODUCT * prod}
    if kind in ("ntt", "ntt_batch", "coset"):
        n, cols = 1 << case["log_n"], case.get("cols", 1)
        extra = n if kind == "coset" or case["inverse"] else 0
        return {"bytes": 64 * n * cols + 32 * n, "flops": _PRODUCT * cols * (n // 2 * case["log_n"] + extra)}
    if kind == "extend":
        n, e, cols = 1 << case["log_n"], 1 << case["ext_bits"], case["cols"]
        one = n // 2 * case["log_n"] + n
        return {"bytes": 32 * n * cols * (2 + e), "flops": _PRODUCT * cols * one * (1 + e)}
    if kind == "products":
        n, m = case["n"], case["perm"]
        # a column read twice less the second time; 3 products an inverse
        return {"bytes": 32 * n * (2 * m + 1 + 1 + 2 + 1 + 3 + 1), "flops": _PRODUCT * n * (4 * m + 5 + 5 + 7)}
    if kind == "quotient":
        n = 1 << case["log_n"]
        cols = 6 * case["gates"] + 4 + -(-case["perm"] // case["chunk"]) + 2 * case["perm"] + 1 + \
            3 * case["lookups"] + 3 * case["shuffles"]
        prod = 8 * case["gates"] + 4 * case["perm"] + 2 * -(-case["perm"] // case["chunk"]) + 8 * case["lookups"] + \
            11 * case["shuffles"]
        return {"bytes": 32 * n * (cols + 1), "flops": _PRODUCT * n * prod}
    n, e = 1 << case["k"], 1 << max(1, math.ceil(math.log2(case["degree"] - 1)))
    chunks = -(-case["perm"] // (case["degree"] - 2))
    msm = case["advice"] + 1 + 2 * case["lookups"] + chunks + case["shuffles"] + case["degree"] + 2
    cols = case["advice"] + 1 + chunks + 2 * case["lookups"] + case["shuffles"]
    ntt = n // 2 * case["k"] + n
    return {"bytes": 32 * n * (cols + case["fixed"] + case["perm"] + 4 + msm),
            "flops": _PRODUCT * (msm * _msm_products(n) + cols * (1 + e) * ntt + e * n * 6 * cols)}


def tolerance(case):
    return "exact"


# ---------------------------------------------------------------- the same in plain integers


_R = 0x30644E72E131A029B85045B68181585D2833E84879B9709143E1F593F0000001
_Q = 0x30644E72E131A029B85045B68181585D97816A916871CA8D3C208C16D87CFD47


def _ints(t):
    a = t.cpu().numpy().view(np.uint64)
    return [int.from_bytes(row.tobytes(), "little") for row in a]


def _g1_mul(k):
    """[k] (1, 2) in affine coordinates, (0, 0) for k = 0."""
    r, p = None, (1, 2)

    def add(a, b):
        if a is None:
            return b
        if b is None:
            return a
        if a[0] == b[0]:
            if (a[1] + b[1]) % _Q == 0:
                return None
            lam = 3 * a[0] * a[0] * pow(2 * a[1], -1, _Q) % _Q
        else:
            lam = (b[1] - a[1]) * pow(b[0] - a[0], -1, _Q) % _Q
        x = (lam * lam - a[0] - b[0]) % _Q
        return x, (lam * (a[0] - x) - a[1]) % _Q

    while k:
        if k & 1:
            r = add(r, p)
        p = add(p, p)
        k >>= 1
    return r or (0, 0)


def exact(case, seed):
    """The MSM kinds by the discrete logarithms of their bases, short
    transforms by their definition's recursion, in Python integers."""
    kind = case["kind"]
    rinv = pow(1 << 256, -1, _R)
    if kind in ("msm", "commit", "uneven", "dropin"):
        lens = _msm_lengths(case)
        if sum(lens) > 2_000_000:
            return None
        ks = [int(x) for x in _multiples(max(lens), seed).cpu().numpy()]
        pts = []
        for col in _msm_scalars(case, seed):
            pts.append(_g1_mul(sum(a * b for a, b in zip(_ints(col), ks)) * rinv % _R))
        return _points(pts)
    if kind in ("ntt", "ntt_batch", "coset"):
        n, cols = 1 << case["log_n"], case.get("cols", 1)
        if n * cols > 1 << 17:
            return None
        x = _ints(_column(cols * n, _gen(seed)))
        w = pow(7, (_R - 1) >> case["log_n"], _R)
        inv = case.get("inverse", False)
        if inv:
            w = pow(w, -1, _R)

        def dft(v, w):
            if len(v) == 1:
                return v
            a, b = dft(v[0::2], w * w % _R), dft(v[1::2], w * w % _R)
            t, u = [], 1
            for y in b:
                t.append(y * u % _R)
                u = u * w % _R
            return [(p + q) % _R for p, q in zip(a, t)] + [(p - q) % _R for p, q in zip(a, t)]

        out = []
        for c in range(cols):
            v = x[c * n:(c + 1) * n]
            if kind == "coset":
                s, t = P.ZETA * P.omega(case["log_n"] + 2) % _R, 1
                for i in range(n):
                    v[i], t = v[i] * t % _R, t * s % _R
            v = dft(v, w)
            if inv:
                ninv = pow(n, -1, _R)
                v = [y * ninv % _R for y in v]
            out += v
        return np.array([[(y >> (64 * j)) & 0xFFFFFFFFFFFFFFFF for j in range(4)] for y in out],
                        dtype=np.uint64).view(np.int64)
    return None
