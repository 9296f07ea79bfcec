"""What the engine is timed on: calls of its public entry points over the sizes, options and data types that
programs use it with.

Kinds of cases (the "kind" of a case):

  step      one Golub-Kahan step written by a caller against the plug-in API (multiply, dot, add_scaled, norm,
            scale): the way code written for MatrixInterface / VectorInterface uses the adapters
  spmv      multiply and multiply_transpose of one matrix
  normals   the factory's random vectors (start blocks, Hutchinson samples)
  create    a host CSR matrix becomes a device matrix with its stored transpose, and is applied once
  products  the block solver's dense products: Gram pair, combination, projection
  cyclic    one null space by cyclic Lanczos
  lobpcg    one null space by block LOBPCG
  batch     many uneven null spaces in one persistent launch

Operators: "shift" (the quickstart's (Ax)_i = x_{i+N} - c x_i), "incidence" (edges x vertices of a random multigraph
whose components are a spanning path plus random edges; the null space holds the component indicators) and "planted"
([B | B W] with 8 random entries per row of B).

The solvers return a null space as some basis of it, and which basis depends on the last bits of every sum. What a
program does with it does not: it takes the null-space part out of its fields. The solver cases do that for k random
fields, which fixes the whole k-dimensional space, and return the parts taken out.
"""
import math

import numpy as np
import torch

import krans_b200 as kb
from krans_b200.serving import SolveRequest, solve_batch

DEV = "cuda:0"
_FP64, _MIXED = int(kb.Precision.FP64), int(kb.Precision.MIXED)


# ---- cases -----------------------------------------------------------------
def listed():
    return [
        # a caller's own Krylov step on the quickstart operator: calls, launches and read-backs, hardly any data
        dict(name="step_quickstart", kind="step", op="shift", n=1000, comps=3, c=0.5),
        # A x and A^T y of the largest graph (64 components x 2^16 vertices, 16.8M edges), plain FP64
        dict(name="spmv_incidence_4m", kind="spmv", op="incidence", n=4194304, comps=64, degree=8.0, fp32=False),
        # A x and A^T y with FP32 values, as the mixed-precision recurrence multiplies; rows of 8 and more entries
        dict(name="spmv_planted_500k_f32", kind="spmv", op="planted", n=500032, m=750001, comps=32, fp32=True),
        # a start block of 24 vectors in the reference's own random sequence
        dict(name="normals_mt_24x262144", kind="normals", n=262144, count=24, mode="mt19937"),
        # a new request's matrix: upload, device transpose, FP32 copy, first products
        dict(name="create_incidence_200k", kind="create", op="incidence", n=200003, comps=12, degree=6.0),
        # [X W P] of block size 96 on 2^18 rows: the dense half of a LOBPCG iteration
        dict(name="products_288x262144", kind="products", n=262144, p=288),
        # the same of a small served request: block size 12 on an odd number of rows
        dict(name="products_36x20011", kind="products", n=20011, p=36),
        # the quickstart: one small solve, one thread block, latency of every step counts
        dict(name="cyclic_quickstart", kind="cyclic", op="shift", n=1000, comps=3, c=0.5, mixed=False),
        # one larger solve on the whole GPU, mixed precision
        dict(name="cyclic_incidence_60k_mixed", kind="cyclic", op="incidence", n=60013, comps=6, degree=6.0, mixed=True),
        # block LOBPCG for the components of a small graph, one thread block
        dict(name="lobpcg_incidence_6k", kind="lobpcg", op="incidence", n=6000, comps=8, degree=8.0),
        # and of a larger one, on the whole GPU
        dict(name="lobpcg_incidence_50k", kind="lobpcg", op="incidence", n=50021, comps=8, degree=8.0),
        # the headline use: uneven requests, shift and incidence in turn, mixed precision, one launch
        dict(name="batch_64_mixed", kind="batch", count=64, n_lo=1000, n_hi=16000, mixed=True, pick=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _op(rng, lo, hi, ops=("shift", "incidence"), most=16):
    op = rng.choice(ops)
    n = _log(rng, lo, hi)
    if op == "shift":
        return dict(op=op, n=n, comps=rng.randint(1, most), c=round(rng.uniform(0.3, 0.9), 3))
    if op == "planted":
        return dict(op=op, n=max(n, 2000), m=int(max(n, 2000) * 1.5) + rng.randint(0, 31), comps=rng.randint(8, 32))
    comps = rng.randint(1, most)
    return dict(op=op, n=max(n, 8 * comps), comps=comps, degree=rng.choice([6.0, 8.0]))


def draw(rng):
    kind = rng.choice(["step", "spmv", "normals", "create", "products", "cyclic", "lobpcg", "batch"])
    if kind == "step":
        return dict(kind=kind, **_op(rng, 1000, 1000000))
    if kind == "spmv":
        return dict(kind=kind, fp32=rng.random() < 0.5, **_op(rng, 1000, 2000000, ("shift", "incidence", "planted")))
    if kind == "normals":
        return dict(kind=kind, n=_log(rng, 1000, 262144), count=rng.randint(1, 24), mode=rng.choice(["mt19937", "mt19937", "philox"]))
    if kind == "create":
        return dict(kind=kind, **_op(rng, 1000, 200000, ("shift", "incidence", "planted")))
    if kind == "products":
        return dict(kind=kind, n=_log(rng, 1000, 262144), p=3 * _log(rng, 2, 96))
    if kind == "cyclic":
        return dict(kind=kind, mixed=rng.random() < 0.5, **_op(rng, 1000, 40000, most=6))
    if kind == "lobpcg":
        return dict(kind=kind, op="incidence", n=_log(rng, 1000, 50000), comps=rng.randint(2, 8), degree=8.0)
    # plain FP64 takes several times as long for the same requests
    mixed = rng.random() < 0.75
    return dict(kind=kind, count=rng.randint(16, 64 if mixed else 24), n_lo=1000,
                n_hi=_log(rng, 4000, 12000) if mixed else _log(rng, 2000, 4000), mixed=mixed, pick=rng.randint(2, 1 << 30))


# ---- operators ---------------------------------------------------------------
class Csr:
    """Host CSR arrays of one operator and what is known of its null space."""

    def __init__(self, m, n, indptr, indices, data):
        self.m, self.n, self.indptr, self.indices, self.data = m, n, indptr, indices, data
        self.nnz = int(data.shape[0])

    def norm_bound(self):
        """Largest row or column norm: at most the spectral norm."""
        sq = self.data * self.data
        rows = np.add.reduceat(sq, self.indptr[:-1].astype(np.int64)) if self.nnz else np.zeros(1)
        cols = np.bincount(self.indices, weights=sq, minlength=self.n)
        return float(np.sqrt(max(rows.max(), cols.max())))


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _shift(case):
    n, N, c = case["n"], case["comps"], case["c"]
    m = n - N
    i = np.arange(m, dtype=np.int32)
    A = Csr(m, n, np.arange(0, 2 * m + 1, 2, dtype=np.int32), np.stack([i, i + N], 1).ravel(),
            np.tile(np.array([-c, 1.0]), m))
    return A


def _incidence(case, seed):
    """(matrix, component of each vertex): rows are edges, +1 at the tail and -1 at the head."""
    n, comps = case["n"], case["comps"]
    g = _gen(seed)
    border = torch.tensor([(n * i) // comps for i in range(comps + 1)], device=DEV)
    perm = torch.randperm(n, generator=g, device=DEV)
    inner = torch.ones(n, dtype=torch.bool, device=DEV)  # position i has a successor in its component
    inner[border[1:] - 1] = False
    a, b = perm[inner.nonzero().ravel()], perm[inner.nonzero().ravel() + 1]
    more = max(0, int(round(n * case["degree"] / 2)) - int(a.shape[0]))
    u = torch.randint(0, n, (more,), generator=g, device=DEV)
    comp = torch.bucketize(u, border, right=True) - 1
    lo, size = border[comp], border[comp + 1] - border[comp]
    off = 1 + (torch.rand(more, generator=g, device=DEV, dtype=torch.float64) * (size - 1)).long().clamp(max=size - 2)
    v = lo + (u - lo + off) % size  # another vertex of u's component
    a, b = torch.cat([a, perm[u]]), torch.cat([b, perm[v]])
    order = torch.randperm(a.shape[0], generator=g, device=DEV)
    a, b = a[order], b[order]
    flip = torch.rand(a.shape[0], generator=g, device=DEV) < 0.5
    sign = torch.where(flip, -1.0, 1.0).double()
    first = a < b
    cols = torch.stack([torch.where(first, a, b), torch.where(first, b, a)], 1).ravel().int()
    s = torch.where(first, sign, -sign)
    vals = torch.stack([s, -s], 1).ravel()
    m = int(a.shape[0])
    label = torch.empty(n, dtype=torch.int64, device=DEV)
    label[perm] = torch.bucketize(torch.arange(n, device=DEV), border, right=True) - 1
    A = Csr(m, n, np.arange(0, 2 * m + 1, 2, dtype=np.int32), cols.cpu().numpy(), vals.cpu().numpy())
    return A, label.cpu().numpy()


def _planted(case, seed):
    """[B | B W]: 8 random columns per row of B, 4 entries per column of W."""
    n, m, k = case["n"], case["m"], case["comps"]
    nk = n - k
    g = _gen(seed)
    cols = torch.randint(0, nk, (m, 8), generator=g, device=DEV)
    vals = torch.randn(m, 8, generator=g, device=DEV, dtype=torch.float64)
    wrow = torch.randperm(nk, generator=g, device=DEV)[:4 * k]
    wcol = torch.full((nk,), -1, dtype=torch.int64, device=DEV)
    wcol[wrow] = torch.arange(4 * k, device=DEV) // 4
    wval = torch.zeros(nk, dtype=torch.float64, device=DEV)
    wval[wrow] = torch.randn(4 * k, generator=g, device=DEV, dtype=torch.float64)
    rows = torch.arange(m, device=DEV)[:, None].expand(m, 8)
    hit = wcol[cols] >= 0
    key = torch.cat([(rows * n + cols).ravel(), (rows[hit] * n + nk + wcol[cols[hit]])])
    val = torch.cat([vals.ravel(), vals[hit] * wval[cols[hit]]])
    key, at = torch.unique(key, return_inverse=True)
    # duplicates are rare; their values are summed on the host in one order
    data = np.bincount(at.cpu().numpy(), weights=val.cpu().numpy(), minlength=int(key.shape[0]))
    indptr = torch.zeros(m + 1, dtype=torch.int64, device=DEV)
    indptr[1:] = torch.cumsum(torch.bincount(key // n, minlength=m), 0)
    return Csr(m, n, indptr.int().cpu().numpy(), (key % n).int().cpu().numpy(), data)


def _operator(case, seed):
    """(matrix, labels): labels of the components for an incidence matrix, else None."""
    if case["op"] == "shift":
        return _shift(case), None
    if case["op"] == "incidence":
        return _incidence(case, seed)
    return _planted(case, seed), None


def _device(A, fp32=False):
    return kb.CudaCsrMatrixAdapter(kb.default_context(), A.m, A.n, A.indptr, A.indices, A.data, fp32=fp32)


def _null_part(case, labels, F):
    """The null-space part of the rows of F, from the known null space."""
    if case["op"] == "incidence":
        cnt = np.bincount(labels, minlength=case["comps"]).astype(np.float64)
        return np.stack([(np.bincount(labels, weights=f, minlength=case["comps"]) / cnt)[labels] for f in F])
    n, N, c = case["n"], case["comps"], case["c"]
    out = np.zeros_like(F)
    for j in range(N):
        at = np.arange(j, n, N)
        v = c ** np.arange(len(at), dtype=np.float64)
        out[:, at] = np.outer(F[:, at] @ v / (v @ v), v)
    return out


def _fields(k, n, seed):
    return np.random.default_rng(int(seed) + 977).standard_normal((k, n))


class _View:
    """A device vector of the engine as torch sees it (the vector stays alive with the view)."""

    def __init__(self, v):
        self.v = v
        self.__cuda_array_interface__ = {"shape": (v.size(),), "typestr": "<f8", "data": (v.device_ptr(), False),
                                         "version": 3, "strides": None}


def _tensor(v):
    return torch.as_tensor(_View(v), device=DEV)


def _sizes(case):
    """The operators of a batch (sizes go with the case, entries with the seed): half shift, half incidence."""
    r = np.random.default_rng(int(case["pick"]))
    out = []
    for i in range(case["count"]):
        n = int(round(math.exp(r.uniform(math.log(case["n_lo"]), math.log(case["n_hi"])))))
        comps, c = int(r.integers(1, 17)), float(r.uniform(0.3, 0.9))
        out.append(dict(op="incidence", n=n, comps=comps, degree=6.0) if i % 2 else dict(op="shift", n=n, comps=comps, c=c))
    return out


def _batch(case, seed):
    """The instances of a batch: (case of one operator, matrix, labels)."""
    return [(one, *_operator(one, 1000003 * int(seed) + i)) for i, one in enumerate(_sizes(case))]


# ---- preparation -------------------------------------------------------------
def prepare(case, seed):
    ctx = kb.default_context()
    kind = case["kind"]
    if kind == "products":
        n, p = case["n"], case["p"]
        g = _gen(seed)
        Z = torch.randn(p, n, dtype=torch.float64, device=DEV, generator=g) / math.sqrt(n)
        W = Z * (0.5 + torch.rand(n, dtype=torch.float64, device=DEV, generator=g))  # N Z for a diagonal N
        q = p // 3
        Y = torch.randn(q, p, dtype=torch.float64, device=DEV, generator=g) / math.sqrt(p)
        new = lambda *s: torch.empty(*s, dtype=torch.float64, device=DEV)  # noqa: E731
        torch.cuda.synchronize()
        return dict(case=case, Z=Z, W=W, Y=Y, q=q, S=new(p, p), G=new(p, p), X=new(q, n), C=new(q, q))
    if kind == "normals":
        return dict(case=case, seed=int(seed) + 1)
    if kind == "batch":
        reqs, fields = [], []
        for i, (one, A, _) in enumerate(_batch(case, seed)):
            o = kb.CyclicLanczosOptions(k=one["comps"], tol_abs=1e-12 * A.norm_bound(), tol_rel=0.0, cg_maxit=1000,
                                        precision=kb.Precision(_MIXED if case["mixed"] else _FP64))
            reqs.append(SolveRequest(_device(A, fp32=case["mixed"]), o, seed=1 + int(seed) % 65536 + 100003 * i))
            fields.append(_fields(one["comps"], one["n"], int(seed) + i))
        return dict(case=case, reqs=reqs, fields=fields)
    A, labels = _operator(case, seed)
    r = np.random.default_rng([int(seed), 3])
    vec = lambda n: kb.CudaVectorAdapter.from_numpy(ctx, r.standard_normal(n))  # noqa: E731
    if kind == "create":
        return dict(case=case, A=A, x=vec(A.n), y=vec(A.m))
    if kind == "step":
        return dict(case=case, M=_device(A), x=vec(A.n), w=kb.CudaVectorAdapter(ctx, A.m), old=[vec(A.m) for _ in range(3)])
    if kind == "spmv":
        M, x, y = _device(A, fp32=case["fp32"]), vec(A.n), vec(A.m)
        Ax, ATy = kb.CudaVectorAdapter(ctx, A.m), kb.CudaVectorAdapter(ctx, A.n)
        return dict(case=case, M=M, x=x, y=y, Ax=Ax, ATy=ATy, prec=_MIXED if case["fp32"] else _FP64,
                    out=(_tensor(Ax), _tensor(ATy)))
    k, L = case["comps"], A.norm_bound()
    if kind == "cyclic":
        M = _device(A, fp32=case["mixed"])
        o = kb.CyclicLanczosOptions(k=k, tol_abs=1e-12 * L, tol_rel=0.0, cg_maxit=1000,
                                    precision=kb.Precision(_MIXED if case["mixed"] else _FP64))
    else:
        M = _device(A)
        o = kb.LOBPCGOptions(nev=k, block_size=k + k // 2, tol_abs=1e-12 * L, tol_rel=0.0)
    return dict(case=case, M=M, opt=o, seed=42 + int(seed) % 65536, fields=_fields(k, A.n, seed))


# ---- one pass ----------------------------------------------------------------
def _taken_out(U, F):
    return (F @ U.T) @ U


def run(state):
    ctx = kb.default_context()
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        M, x, w = state["M"], state["x"], state["w"]
        M.multiply(x, w)
        h = []
        for v in state["old"]:
            h.append(w.dot(v) / v.dot(v))
            w.add_scaled(v, -h[-1])
        beta = w.norm()
        w.scale(1.0 / beta)
        return dict(w=_tensor(w), h=np.array(h), beta=beta)
    if kind == "spmv":
        state["M"].multiply(state["x"], state["Ax"], state["prec"])
        state["M"].multiply_transpose(state["y"], state["ATy"], state["prec"])
        return state["out"]
    if kind == "normals":
        vf = kb.CudaVectorFactory(ctx, case["n"], seed=state["seed"], mode=case["mode"])
        return [_tensor(vf.create_random()) for _ in range(case["count"])]
    if kind == "create":
        A = state["A"]
        M = _device(A, fp32=True)
        Ax, ATy = kb.CudaVectorAdapter(ctx, A.m), kb.CudaVectorAdapter(ctx, A.n)
        M.multiply(state["x"], Ax)
        M.multiply_transpose(state["y"], ATy)
        return _tensor(Ax), _tensor(ATy)
    if kind == "products":
        n, p, q = case["n"], case["p"], state["q"]
        Z, W, Y, S, G, X, C = (state[i].data_ptr() for i in ("Z", "W", "Y", "S", "G", "X", "C"))
        kb.block_gram(ctx, n, p, Z, n, S, W, G)
        kb.block_combine(ctx, n, p, q, Z, n, Y, p, X)
        kb.block_gemm_tn(ctx, n, q, Z, q, X, n, C)
        return state["S"], state["G"], state["X"], state["C"]
    if kind == "batch":
        solve_batch(ctx, state["reqs"])
        return np.concatenate([_taken_out(r.basis(), F).ravel() for r, F in zip(state["reqs"], state["fields"])])
    vf = kb.CudaVectorFactory(ctx, state["M"].n, seed=state["seed"])
    if kind == "cyclic":
        U = kb.find_nullspace_cyclic_lanczos(state["M"], vf, state["opt"])
    else:
        U = kb.find_nullspace_lobpcg(state["M"], vf, state["opt"])
    return _taken_out(kb.basis_to_numpy(U), state["fields"])


# ---- what a pass cannot do without ---------------------------------------------
def _size(case):
    """(rows, columns, entries) of a case's operator, to within a few."""
    n = case["n"]
    if case["op"] == "shift":
        return n - case["comps"], n, 2 * (n - case["comps"])
    if case["op"] == "planted":
        return case["m"], n, 8 * case["m"] + 32 * case["comps"] * case["m"] // n
    m = int(round(n * case["degree"] / 2))
    return m, n, 2 * m


def work(case):
    kind = case["kind"]
    if kind == "normals":
        return dict(bytes=8.0 * case["n"] * case["count"], flops=0.0)
    if kind == "products":
        n, p = float(case["n"]), case["p"]
        q = p // 3
        # upper triangles of S and G, the combination, the projection
        return dict(bytes=8.0 * (n * (2 * p + q) + 2 * p * p + p * q + q * q),
                    flops=2.0 * n * (p * (p + 1) + p * q + q * q))
    if kind == "batch":
        total = 0.0
        for one in _sizes(case):
            m, n, z = _size(one)
            total += 4.0 * (m + 1) + 12.0 * z + 8.0 * n * one["comps"]
        return dict(bytes=total, flops=0.0)
    m, n, z = _size(case)
    if kind == "step":
        return dict(bytes=4.0 * (m + 1) + 12.0 * z + 8.0 * (n + 4 * m), flops=2.0 * z + 20.0 * m)
    if kind == "spmv":
        w = 8 if case["fp32"] else 12
        return dict(bytes=4.0 * (m + n + 2) + 2.0 * w * z + 16.0 * (m + n), flops=4.0 * z)
    if kind == "create":
        return dict(bytes=4.0 * (m + n + 2) + 2.0 * 16.0 * z + 16.0 * (m + n), flops=4.0 * z)
    return dict(bytes=4.0 * (m + 1) + 12.0 * z + 8.0 * n * case["comps"], flops=2.0 * z * case["comps"])


# ---- the same in 64 bits -------------------------------------------------------
def _times(A, x, dtype=np.float64):
    v = A.data.astype(dtype).astype(np.float64)
    p = torch.from_numpy(v * x.astype(dtype).astype(np.float64)[A.indices])
    return torch.segment_reduce(p, "sum", lengths=torch.from_numpy(np.diff(A.indptr).astype(np.int64))).numpy()


def _times_t(A, y, dtype=np.float64):
    v = A.data.astype(dtype).astype(np.float64)
    rows = np.repeat(np.arange(A.m), np.diff(A.indptr))
    return np.bincount(A.indices, weights=v * y.astype(dtype).astype(np.float64)[rows], minlength=A.n)


def exact(case, seed):
    kind = case["kind"]
    if kind == "normals":
        return None  # a sequence, not a value
    if kind == "products":
        s = prepare(case, seed)
        Z, W, Y, q = s["Z"], s["W"], s["Y"], s["q"]
        G = torch.triu((Z @ W.T))
        X = Y @ Z
        # column-major results: row j of each tensor is column j
        return Z @ Z.T, (G + torch.triu(G, 1).T), X, X @ Z[:q].T
    if kind == "batch":
        return np.concatenate([_null_part(one, labels, _fields(one["comps"], one["n"], int(seed) + i)).ravel()
                               for i, (one, _, labels) in enumerate(_batch(case, seed))])
    A, labels = _operator(case, seed)
    r = np.random.default_rng([int(seed), 3])
    if kind in ("create", "spmv"):
        x, y = r.standard_normal(A.n), r.standard_normal(A.m)
        dtype = np.float32 if case.get("fp32") else np.float64
        return _times(A, x, dtype), _times_t(A, y, dtype)
    if kind == "step":
        x = r.standard_normal(A.n)
        old = [r.standard_normal(A.m) for _ in range(3)]
        w, h = _times(A, x), []
        for v in old:
            h.append(float(w @ v) / float(v @ v))
            w = w - h[-1] * v
        beta = float(np.linalg.norm(w))
        return dict(w=w / beta, h=np.array(h), beta=beta)
    return _null_part(case, labels, _fields(case["comps"], A.n, seed))
