"""Timed cases of the framework: single contractions, chains, grouped block
products, leg permutations and the block eigen / singular value steps, each
through the entry point that a program calls.

A case is a dict of plain values with a "kind":

rdm      contractQS of an MPS site tensor with itself on host QSpaces (the
         drop-in call of an interactive or scripted user): small, so the
         latency of one whole call counts.
overlap  contract_dev over both bonds of a device-resident site tensor (the
         reduced density matrix of the site): a few tiny output blocks, each
         a very deep sum.
hpsi     the four contract_dev calls of a two-site DMRG H*psi, the inner step
         of every Davidson / Lanczos solver.
batch    contract_batch of independent reduced density matrices (the serving
         loop's batches).
grouped  lists of block products with CG factors, as the per-output-block
         seam of contractQS hands them down: one-shot or through a reusable
         plan, real or complex, one or several products per output block,
         operands stored transposed or conjugated.
permute  permute_dev of a two-site wave function.
eig      eigQS_dev of the sectors of an NRG Hamiltonian, with truncation.
svd      svd_blocks of the sector matrices of a two-site wave function, the
         split of a DMRG sweep.
"""
import ctypes as C
import math

import numpy as np
import torch

from qspace_gb300 import Context, QSpace, contractQS, contract_batch, contract_dev, permute_dev, upload
from qspace_gb300 import workloads
from qspace_gb300._capi import Stats, check
from qspace_gb300.grouped import GroupedPlan, Packed
from qspace_gb300.linalg import eigQS_dev, svd_blocks
from qspace_gb300.qspace import make_opts


def listed():
    return [
        # the smallest call: the reduced density matrix of the U(1)xU(1) site
        # tensor, D = 512, host buffers in and out
        {"name": "rdm_host_fp64_d512", "kind": "rdm", "D": 512, "cplx": False, "prec": "fp64"},
        # one serving batch: 16 reduced density matrices of mid-size tensors
        {"name": "batch_fp64_16_d512", "kind": "batch", "jobs": 16, "D": 512, "cplx": True, "prec": "fp64"},
        # site density matrix of a large tensor: deep sums, tiny outputs
        {"name": "overlap_split_d8192", "kind": "overlap", "D": 8192, "cplx": True, "prec": "split"},
        # one Davidson step at a moderate bond, plain precision
        {"name": "hpsi_fp64_d2048", "kind": "hpsi", "D": 2048, "prec": "fp64"},
        # the same at the bond dimension of a production run, split precision
        {"name": "hpsi_split_d4096", "kind": "hpsi", "D": 4096, "prec": "split"},
        # the headline batch: 2000 complex products, planned once and replayed
        {"name": "grouped_split_plan_2000", "kind": "grouped", "blocks": 2000, "per_block": 1, "lo": 8, "hi": 1024,
         "cplx": True, "prec": "split", "plan": True, "flags": False},
        # a plain-precision list of the same sizes, planned on every call
        {"name": "grouped_fp64_300", "kind": "grouped", "blocks": 300, "per_block": 1, "lo": 8, "hi": 1024,
         "cplx": True, "prec": "fp64", "plan": False, "flags": False},
        # real blocks, several products summed into each, operands transposed
        # and sizes odd, planned on every call
        {"name": "grouped_split_real_480", "kind": "grouped", "blocks": 120, "per_block": 4, "lo": 17, "hi": 400,
         "cplx": False, "prec": "split", "plan": False, "flags": True},
        # small real blocks replayed from a plan: launches and latency
        {"name": "grouped_fp64_plan_small", "kind": "grouped", "blocks": 64, "per_block": 2, "lo": 4, "hi": 96,
         "cplx": False, "prec": "fp64", "plan": True, "flags": True},
        # a leg permutation of a large wave function (the fastest leg moves)
        {"name": "permute_psi_d8192", "kind": "permute", "D": 8192, "cplx": True, "perm": "4123"},
        # an NRG step's block eigendecomposition with truncation
        {"name": "eig_nrg_256", "kind": "eig", "dmax": 256, "nkeep": 1024},
        # the split of a two-site tensor in a DMRG sweep
        {"name": "svd_two_site_d128", "kind": "svd", "D": 128, "cplx": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rdm", "batch", "overlap", "hpsi", "hpsi", "grouped", "grouped", "grouped", "permute", "eig",
                       "svd"])
    prec, cplx = rng.choice(["fp64", "split"]), rng.random() < 0.5
    if kind == "rdm":
        return {"kind": kind, "D": _log(rng, 64, 1024), "cplx": cplx, "prec": prec}
    if kind == "batch":
        return {"kind": kind, "jobs": rng.randint(2, 32), "D": _log(rng, 64, 1024), "cplx": cplx, "prec": prec}
    if kind == "overlap":
        return {"kind": kind, "D": _log(rng, 1024, 8192), "cplx": cplx, "prec": prec}
    if kind == "hpsi":
        return {"kind": kind, "D": _log(rng, 256, 4096), "prec": prec}
    if kind == "grouped":
        hi = _log(rng, 64, 1024)
        lo = min(_log(rng, 4, 64), hi // 2)
        per = rng.choice([1, 1, 2, 4, 8])
        # at most the arithmetic of about 400 plain-precision products of
        # [8, 1024] each, or 2000 split ones
        most = (400 if prec == "fp64" else 1600) * (1024 / hi) ** 2
        blocks = _log(rng, 4, max(8, min(2000, most / per)))
        return {"kind": kind, "blocks": blocks, "per_block": per, "lo": lo, "hi": hi, "cplx": cplx, "prec": prec,
                "plan": rng.random() < 0.5, "flags": rng.random() < 0.5}
    if kind == "permute":
        p = list("1234")
        while p == list("1234"):
            rng.shuffle(p)
        return {"kind": kind, "D": _log(rng, 512, 8192), "cplx": cplx, "perm": "".join(p)}
    if kind == "eig":
        return {"kind": kind, "dmax": _log(rng, 24, 300), "nkeep": _log(rng, 64, 2048)}
    return {"kind": "svd", "D": _log(rng, 16, 160), "cplx": cplx}


# ------------------------------------------------------------------ inputs
_ctx = None


def _context():
    global _ctx
    if _ctx is None:
        _ctx = Context(0)
    return _ctx


class _View:
    """A device tensor's data as a torch tensor without a copy."""

    def __init__(self, t):
        self.t = t
        n = t.meta()[3] * (2 if t.meta()[4] else 1)
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (t.data_ptr, False), "version": 3,
                                         "stream": None}


def _data(t):
    return torch.as_tensor(_View(t), device="cuda")


def _pairs(case, seed):
    """Sizes and flags (the case's own) and factors (the seed's) of a list of
    block products; output blocks one after the other, operands in pair
    order."""
    rng = np.random.default_rng(0)
    nb, per = case["blocks"], case["per_block"]
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    size = lambda n: np.rint(np.exp(rng.uniform(lo, hi, n))).astype(np.int32)  # noqa: E731
    M, N, K = np.repeat(size(nb), per), np.repeat(size(nb), per), size(nb * per)
    n = nb * per
    trans = rng.integers(0, 16 if case["cplx"] else 4, n).astype(np.int32) if case["flags"] else np.zeros(n, np.int32)
    afac = np.random.default_rng(seed).uniform(-1.0, 1.0, n)
    return M, N, K, trans, afac, np.repeat(np.arange(nb, dtype=np.int32), per)


class _List(Packed):
    """A pair list over operands that already lie in device memory."""

    def __init__(self, case, seed):
        self.M, self.N, self.K, self.trans, self.afac, self.blk = _pairs(case, seed)
        self.n, self.cplx = len(self.M), bool(case["cplx"])
        a, b = self.M.astype(np.int64) * self.K, self.K.astype(np.int64) * self.N
        start = lambda s: np.concatenate([[0], np.cumsum(s)[:-1]]).astype(np.int64)  # noqa: E731
        self.a_off, self.b_off, self.a_elems, self.b_elems = start(a), start(b), int(a.sum()), int(b.sum())
        first = np.concatenate([[True], self.blk[1:] != self.blk[:-1]])
        c = (self.M.astype(np.int64) * self.N)[first]
        self.c_off = np.repeat(start(c), np.diff(np.append(np.flatnonzero(first), self.n)))
        self.c_elems = int(c.sum())
        self.lda = np.where(self.trans & 1, self.K, self.M).astype(np.int32)
        self.ldb = np.where(self.trans & 2, self.N, self.K).astype(np.int32)
        self.ldc = self.M.copy()


def _refill(qs, seed):
    """The tensor's sectors with new N(0,1) entries from the seed."""
    rng = np.random.default_rng(seed)
    qs.data = [rng.standard_normal(d.shape) + 1j * rng.standard_normal(d.shape) if np.iscomplexobj(d)
               else rng.standard_normal(d.shape) for d in qs.data]
    return qs


def _site(case, seed):
    return _refill(workloads.mps_site_tensor(0, case["D"], complex_data=case["cplx"]), seed)


def _psi4(case, seed):
    return _refill(workloads.rank4_psi(0, case["D"], complex_data=case["cplx"]), seed)


def _eig_blocks(case, seed):
    return workloads.nrg_eig_blocks(seed, dmax=case["dmax"])


def _svd_matrices(case, seed):
    """The sector matrices (L s1) x (s2 R) of a two-site wave function."""
    psi = workloads.two_site_state(seed, case["D"], complex_data=case["cplx"])
    lab = [tuple(int(q[b, 0]) for q in psi.Q) for b in range(psi.nblk)]
    out = []
    for s in sorted({a + b for a, b, _, _ in lab}):
        rows = sorted({(a, b) for a, b, _, _ in lab if a + b == s})
        cols = sorted({(c, d) for a, b, c, d in lab if a + b == s})
        at = {(x[:2], x[2:]): psi.data[i] for i, x in enumerate(lab) if x[0] + x[1] == s}
        hs = [next(at[r, c].shape[0] for c in cols if (r, c) in at) for r in rows]
        ws = [next(at[r, c].shape[3] for r in rows if (r, c) in at) for c in cols]
        out.append(np.block([[at[r, c].reshape(h, w) if (r, c) in at else np.zeros((h, w)) for c, w in zip(cols, ws)]
                             for r, h in zip(rows, hs)]))
    return out


def prepare(case, seed):
    kind, ctx = case["kind"], _context()
    if kind == "rdm":
        return {"case": case, "ctx": ctx, "A": _site(case, seed)}
    if kind == "batch":
        sites = [upload(_site(case, 1000 * seed + j), ctx) for j in range(case["jobs"])]
        return {"case": case, "jobs": [(a, "12*", a, "12") for a in sites]}
    if kind == "overlap":
        return {"case": case, "A": upload(_site(case, seed), ctx)}
    if kind == "hpsi":
        return {"case": case, "T": [upload(x, ctx) for x in workloads.hpsi_chain(seed, case["D"])]}
    if kind == "grouped":
        pk = _List(case, seed)
        es = 2 if case["cplx"] else 1
        gen = torch.Generator(device="cuda").manual_seed(seed)
        A = torch.randn(pk.a_elems * es, dtype=torch.float64, device="cuda", generator=gen)
        B = torch.randn(pk.b_elems * es, dtype=torch.float64, device="cuda", generator=gen)
        Cm = torch.zeros(pk.c_elems * es, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        state = {"case": case, "ctx": ctx, "pk": pk, "A": A, "B": B, "C": Cm}
        if case["plan"]:
            state["plan"] = GroupedPlan(pk, case["prec"], autotune=case["prec"] == "split", ctx=ctx)
        else:
            state["list"], state["opts"] = pk.pair_list(), make_opts(case["prec"])
        return state
    if kind == "permute":
        return {"case": case, "A": upload(_psi4(case, seed), ctx)}
    if kind == "eig":
        blocks = _eig_blocks(case, seed)
        q = np.arange(len(blocks), dtype=np.int32).reshape(-1, 1)
        return {"case": case, "H": upload(QSpace([q, q.copy()], blocks), ctx)}
    return {"case": case, "ctx": ctx, "blocks": _svd_matrices(case, seed)}


# --------------------------------------------------------------------- run
def run(state):
    case = state["case"]
    kind, prec = case["kind"], case.get("prec")
    if kind == "rdm":
        c = contractQS(state["A"], "12*", state["A"], "12", prec=prec, ctx=state["ctx"])
        return {"Q": c.Q, "data": c.data}
    if kind == "batch":
        return [_data(c) for c in contract_batch(state["jobs"], prec=prec)]
    if kind == "overlap":
        return _data(contract_dev(state["A"], "13*", state["A"], "13", prec=prec))
    if kind == "hpsi":
        L, psi, W, R = state["T"]
        x = contract_dev(L, "3", psi, "1", prec=prec)
        x = contract_dev(x, [2, 3], W, [1, 3], prec=prec)
        x = contract_dev(x, [2, 5], W, [3, 1], prec=prec)
        return _data(contract_dev(x, [2, 5], R, [3, 2], prec=prec))
    if kind == "grouped":
        if case["plan"]:
            state["plan"].run(state["A"].data_ptr(), state["B"].data_ptr(), state["C"].data_ptr())
        else:
            ctx, st = state["ctx"], Stats()
            check(ctx.lib.qs_grouped_gemm(ctx.h, C.byref(state["list"]), state["A"].data_ptr(),
                                          state["B"].data_ptr(), state["C"].data_ptr(), C.byref(state["opts"]),
                                          C.byref(st)))
        return state["C"]
    if kind == "permute":
        return _data(permute_dev(state["A"], case["perm"]))
    if kind == "eig":
        E, parts = eigQS_dev(state["H"], Nkeep=case["nkeep"])
        with torch.cuda.stream(torch.cuda.ExternalStream(state["H"].ctx.stream_ptr)):
            # kept and discarded vectors together: their sum of sizes is the blocks'
            vectors = torch.cat([_data(parts["AK"]), _data(parts["AD"])])
        return {"E": E, "keep": parts["keep"].astype(np.int64), "vectors": vectors}
    U, S, V = svd_blocks(state["blocks"], state["ctx"])
    return {"U": U, "S": S, "V": V}


# ------------------------------------------------------------------- exact
def _dense(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def _blocks(qs):
    """A QSpace as (labels per leg, block) with the blocks on the device."""
    return [([tuple(int(v) for v in np.atleast_1d(q[i])) for q in qs.Q],
             _dense(np.asarray(d).reshape(qs.block_dims(i)))) for i, d in enumerate(qs.data)]


def _contract(A, ia, B, ib, conj=False):
    """Sum over label-matching blocks, output blocks in label order."""
    ia, ib = [i - 1 for i in ia], [i - 1 for i in ib]
    right = {}
    for q, x in B:
        right.setdefault(tuple(q[i] for i in ib), []).append(([v for i, v in enumerate(q) if i not in ib], x))
    out = {}
    for q, x in A:
        keep = [v for i, v in enumerate(q) if i not in ia]
        for rest, y in right.get(tuple(q[i] for i in ia), []):
            z = torch.tensordot(x.conj() if conj else x, y, dims=(ia, ib))
            key = tuple(keep + rest)
            out[key] = out[key] + z if key in out else z
    return [(list(k), out[k]) for k in sorted(out)]


def _flat(x):
    """Column-major values, complex as (re, im) pairs."""
    x = x.permute(*reversed(range(x.ndim))).reshape(-1)
    return torch.view_as_real(x).reshape(-1) if x.is_complex() else x


def _cat(blocks):
    return torch.cat([_flat(x) for _, x in blocks])


def exact(case, seed):
    kind = case["kind"]
    if kind == "rdm":
        a = _blocks(_site(case, seed))
        return {"Q": [None, None], "data": [x.cpu().numpy() for _, x in _contract(a, [1, 2], a, [1, 2], True)]}
    if kind == "batch":
        out = []
        for j in range(case["jobs"]):
            a = _blocks(_site(case, 1000 * seed + j))
            out.append(_cat(_contract(a, [1, 2], a, [1, 2], True)))
        return out
    if kind == "overlap":
        a = _blocks(_site(case, seed))
        return _cat(_contract(a, [1, 3], a, [1, 3], True))
    if kind == "hpsi":
        L, psi, W, R = (_blocks(x) for x in workloads.hpsi_chain(seed, case["D"]))
        x = _contract(L, [3], psi, [1])
        x = _contract(x, [2, 3], W, [1, 3])
        x = _contract(x, [2, 5], W, [3, 1])
        return _cat(_contract(x, [2, 5], R, [3, 2]))
    if kind == "grouped":
        pk = _List(case, seed)
        es = 2 if case["cplx"] else 1
        gen = torch.Generator(device="cuda").manual_seed(seed)
        A = torch.randn(pk.a_elems * es, dtype=torch.float64, device="cuda", generator=gen)
        B = torch.randn(pk.b_elems * es, dtype=torch.float64, device="cuda", generator=gen)
        if case["cplx"]:
            A, B = (torch.view_as_complex(x.reshape(-1, 2)) for x in (A, B))
        out = torch.zeros(pk.c_elems, dtype=A.dtype, device="cuda")
        for p in range(pk.n):
            m, n, k, t = int(pk.M[p]), int(pk.N[p]), int(pk.K[p]), int(pk.trans[p])
            a = A[int(pk.a_off[p]):int(pk.a_off[p]) + m * k]
            b = B[int(pk.b_off[p]):int(pk.b_off[p]) + k * n]
            # column-major storage; the products are formed transposed
            at = a.reshape(m, k).T if t & 1 else a.reshape(k, m)
            bt = b.reshape(k, n).T if t & 2 else b.reshape(n, k)
            at, bt = at.conj() if t & 4 else at, bt.conj() if t & 8 else bt
            c = out[int(pk.c_off[p]):int(pk.c_off[p]) + m * n].reshape(n, m)
            c += float(pk.afac[p]) * (bt @ at)
        return torch.view_as_real(out).reshape(-1) if case["cplx"] else out
    if kind == "permute":
        p = [int(c) - 1 for c in case["perm"]]
        return torch.cat([_flat(_dense(x).permute(*p)) for x in _psi4(case, seed).data])
    if kind == "eig":
        return {"E": np.sort(np.concatenate([np.linalg.eigvalsh(b) for b in _eig_blocks(case, seed)])), "keep": None,
                "vectors": None}
    mats = _svd_matrices(case, seed)
    none = [None] * len(mats)
    return {"U": none, "S": [np.linalg.svd(m, compute_uv=False) for m in mats], "V": none}


# -------------------------------------------------------------------- work
def _sum_products(A, ia, B, ib):
    """(output element count, multiply-adds) of a contraction, from shapes."""
    ia, ib = [i - 1 for i in ia], [i - 1 for i in ib]
    right = {}
    for q, s in B:
        right.setdefault(tuple(q[i] for i in ib), []).append(
            ([v for i, v in enumerate(q) if i not in ib], [d for i, d in enumerate(s) if i not in ib]))
    out, macs = {}, 0
    for q, s in A:
        k = math.prod(s[i] for i in ia)
        m = [d for i, d in enumerate(s) if i not in ia]
        for rest, n in right.get(tuple(q[i] for i in ia), []):
            key = tuple([v for i, v in enumerate(q) if i not in ia] + rest)
            out[key] = m + n
            macs += math.prod(m) * math.prod(n) * k
    return [(list(k), out[k]) for k in sorted(out)], macs


def _shapes(qs):
    return [([tuple(int(v) for v in np.atleast_1d(q[i])) for q in qs.Q], list(qs.block_dims(i)))
            for i in range(qs.nblk)]


def _elems(blocks):
    return sum(math.prod(s) for _, s in blocks)


def work(case):
    kind = case["kind"]
    es = 16 if case.get("cplx") else 8
    fl = 8 if case.get("cplx") else 2
    if kind in ("rdm", "batch", "overlap"):
        a = _shapes(_site(case, 0))
        ctr = [1, 3] if kind == "overlap" else [1, 2]
        out, macs = _sum_products(a, ctr, a, ctr)
        n = case.get("jobs", 1)
        return {"bytes": n * es * (_elems(a) + _elems(out)), "flops": n * fl * macs}
    if kind == "hpsi":
        L, psi, W, R = (_shapes(x) for x in workloads.hpsi_chain(0, case["D"]))
        x, total = L, 0
        for ia, b, ib in (([3], psi, [1]), ([2, 3], W, [1, 3]), ([2, 5], W, [3, 1]), ([2, 5], R, [3, 2])):
            x, macs = _sum_products(x, ia, b, ib)
            total += macs
        return {"bytes": es * sum(map(_elems, (L, psi, W, R, x))), "flops": fl * total}
    if kind == "grouped":
        pk = _List(case, 0)
        flops = fl * float(np.sum(pk.M.astype(float) * pk.N * pk.K))
        return {"bytes": es * (pk.a_elems + pk.b_elems + pk.c_elems), "flops": flops}
    if kind == "permute":
        return {"bytes": 2 * es * _elems(_shapes(workloads.rank4_psi(0, case["D"]))), "flops": 0}
    if kind == "eig":
        n = [b.shape[0] for b in _eig_blocks(case, 0)]
        return {"bytes": 16 * sum(k * k for k in n), "flops": sum(10 / 3 * k ** 3 for k in n)}
    mn = [sorted(m.shape) for m in _svd_matrices(case, 0)]
    return {"bytes": es * sum(a * b + a * a + a * b for a, b in mn), "flops": fl / 2 * sum(12 * a * a * b for a, b in mn)}
