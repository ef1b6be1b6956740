"""Timed cases of the variational HCI hot path, each through the public Python API.

A case is a plain dict.  `kind` says which call it makes:

  sigma    GpuHam.sigma_device: y = H x on device vectors over a built matrix, what a
           caller's own eigensolver (and this library's Davidson) repeats
  product  GpuHam.matrix_matrix_prod: host vectors in and out (the reference's
           MatrixOperations interface)
  build    GpuHam.set_dets + build: a new determinant list becomes a stored matrix; one
           product with it is returned, which every stored element enters
  solve    GpuHam.set_dets + sparse_optimize: determinants in, energy and coefficients out,
           once per HCI iteration
  select   GpuHam.find_new_dets: the heat-bath selection step

Sizes are those of this repository's tests and benchmark (norb / electrons per spin:
10/4, 12/6, 20/8, 24/10; 6,943 to 551,147 determinants) and odd ones between them.  The
integrals are the seeded synthetic ones of risq_b200.fcidump.  The determinant sets are
made here from the seed: the pairs of spin strings of lowest orbital energy, with some
noise, closed under spin flip and listed by that energy.  Such sets have the alpha-group
sizes and the connections per determinant of the HCI sets of the same integrals (12/6,
131,611 determinants: 878 connections per row against 865; 10/4, 6,943: 347 against 345).
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from risq_b200 import GpuHam, _capi
from risq_b200.fcidump import synthetic_integrals

STORAGE = {"fp64": _capi.FP64, "mixed": _capi.MIXED, "fp64_upper": _capi.FP64_UPPER,
           "mixed_upper": _capi.MIXED_UPPER}
SELECT_MOST = 1 << 19  # more than any selection here returns
DAV_MAX_ITER = 2000  # the reference's 50 does not converge on these integrals
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def listed():
    return [
        # The smallest host call: a short vector through the reference's interface, where
        # copies, allocations and launches are the cost.
        dict(name="product_n10_1201x2", kind="product", norb=10, nel=4, n=1201, storage="fp64", nvec=2),
        # One sigma of a small space (the smoke test's size): launch latency.
        dict(name="sigma_n10_6943_fp64", kind="sigma", norb=10, nel=4, n=6943, storage="fp64", fp32=False),
        # The benchmark's config 0 space, FP64 rows: the plain path's sigma.
        dict(name="sigma_n12_131611_fp64", kind="sigma", norb=12, nel=6, n=131611, storage="fp64", fp32=False),
        # FP32 sigma of the mixed path where both triangles are stored.
        dict(name="sigma_n20_200003_fp32", kind="sigma", norb=20, nel=8, n=200003, storage="mixed", fp32=True),
        # FP32 sigma of the product path over the tiled upper triangle.
        dict(name="sigma_n20_551147_fp32_tiles", kind="sigma", norb=20, nel=8, n=551147, storage="mixed_upper",
             fp32=True),
        # FP64 sigma of the plain path over the tiled upper triangle, another orbital count.
        dict(name="sigma_n24_400009_fp64_tiles", kind="sigma", norb=24, nel=10, n=400009, storage="fp64_upper",
             fp32=False),
        # Build of an HCI iteration's matrix, FP64 rows.
        dict(name="build_n12_131611_fp64", kind="build", norb=12, nel=6, n=131611, storage="fp64"),
        # Build of the product path: FP32 + remainder, tiled upper triangle.
        dict(name="build_n20_551147_mixed_tiles", kind="build", norb=20, nel=8, n=551147, storage="mixed_upper"),
        # A whole small solve (early HCI iterations): latency of every stage.
        dict(name="solve_n10_6943_fp64", kind="solve", norb=10, nel=4, n=6943, storage="fp64", space=0, keep=0),
        # The benchmark's config 0 solve, reference search space.
        dict(name="solve_n12_131611_fp64", kind="solve", norb=12, nel=6, n=131611, storage="fp64", space=0, keep=0),
        # A large solve with the thick-restart space over tiles.
        dict(name="solve_n20_300007_fp64_tiles", kind="solve", norb=20, nel=8, n=300007, storage="fp64_upper",
             space=32, keep=8),
        # Selection from a mid-run variational space.
        dict(name="select_n20_30011", kind="select", norb=20, nel=8, n=30011, eps=1e-3, singles=True),
    ]


# (norb, electrons per spin, largest set drawn)
SYSTEMS = [(10, 4, 9001), (12, 6, 131611), (14, 6, 150001), (16, 7, 200003), (20, 8, 400009), (24, 10, 300007)]
# solves stay with systems whose lowest state has the start vectors' spin-flip parity
SOLVE_SYSTEMS = [(10, 4, 9001), (12, 6, 131611), (20, 8, 200003)]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) | 1


def draw(rng):
    kind = rng.choice(["sigma", "sigma", "sigma", "product", "build", "build", "solve", "solve", "select"])
    norb, nel, most = rng.choice(SOLVE_SYSTEMS if kind == "solve" else SYSTEMS)
    if kind == "sigma":
        storage = rng.choice(["fp64", "mixed", "fp64_upper", "mixed_upper"])
        return dict(kind=kind, norb=norb, nel=nel, n=_size(rng, 1000, most), storage=storage,
                    fp32=storage.startswith("mixed") and rng.random() < 0.7)
    if kind == "product":
        return dict(kind=kind, norb=norb, nel=nel, n=_size(rng, 300, min(most, 60000)),
                    storage=rng.choice(["fp64", "fp64_upper"]), nvec=rng.choice([1, 2, 4]))
    if kind == "build":
        return dict(kind=kind, norb=norb, nel=nel, n=_size(rng, 1000, most),
                    storage=rng.choice(["fp64", "mixed", "fp64_upper", "mixed_upper"]))
    if kind == "solve":
        space, keep = rng.choice([(0, 0), (0, 0), (32, 8)])
        return dict(kind=kind, norb=norb, nel=nel, n=_size(rng, 2000, most),
                    storage=rng.choice(["fp64", "fp64_upper"]), space=space, keep=keep)
    return dict(kind=kind, norb=norb, nel=nel, n=_size(rng, 1000, min(most, 30011)),
                eps=rng.choice([2e-3, 1e-3]), singles=rng.random() < 0.5)


# ---- inputs ---------------------------------------------------------------------------


def _strings(norb, nel, cap=60000):
    """Spin strings (int64 bit masks) by excitation rank from the lowest one, every rank whole."""
    hf = (1 << nel) - 1
    out, total = [torch.tensor([hf])], 1
    for r in range(1, nel + 1):
        holes = torch.combinations(torch.arange(nel), r)
        parts = torch.combinations(torch.arange(nel, norb), r)
        total += len(holes) * len(parts)
        if len(parts) == 0 or total > cap:
            break
        out.append((hf - (1 << holes).sum(1)[:, None] + (1 << parts).sum(1)[None, :]).reshape(-1))
    return torch.cat(out)


def _determinants(norb, nel, n, seed):
    """n determinants (up, dn int64 masks) in increasing order of noisy orbital energy, spin
    flips side by side, and that energy above the first one's."""
    gen = torch.Generator().manual_seed(seed)
    s = _strings(norb, nel)
    occ = ((s[:, None] >> torch.arange(norb)) & 1).double()
    e = occ @ (-3.0 + 4.0 * torch.arange(norb).double() / (norb - 1))
    e = e - e[0].clone() + 0.05 * torch.randn(len(e), generator=gen, dtype=torch.double)
    e[0] = -1.0  # the lowest determinant leads
    e, order = e.sort()
    s = s[order]
    lo, hi = float(2 * e[0]), float(2 * e[-1])
    for _ in range(50):  # the energy below which there are about 2 n pairs
        mid = (lo + hi) / 2
        lo, hi = (mid, hi) if int(torch.searchsorted(e, mid - e).sum()) < 2 * n + 100 else (lo, mid)
    k = torch.searchsorted(e, hi - e)
    a = torch.repeat_interleave(torch.arange(len(e)), k)
    b = torch.arange(len(a)) - torch.repeat_interleave(k.cumsum(0) - k, k)
    a, b = a[a <= b], b[a <= b]
    w = e[a] + e[b] + 0.3 * torch.randn(len(a), generator=gen, dtype=torch.double)
    w[(a == 0) & (b == 0)] = 2 * e[0] - 2.0
    w, order = w.sort()
    a, b = a[order], b[order]
    count = (1 + (a != b).long()).cumsum(0)
    m = int((count <= n).sum())
    if m and int(count[m - 1]) < n:  # one short: a closed-shell determinant fills the place
        j = m + int((a[m:] == b[m:]).nonzero()[0, 0])
        pick = torch.cat([torch.arange(m), torch.tensor([j])])
    else:
        pick = torch.arange(m)
    a, b, w = a[pick], b[pick], w[pick]
    keep = torch.stack([torch.ones_like(a, dtype=torch.bool), a != b], 1).reshape(-1)
    up = s[torch.stack([a, b], 1).reshape(-1)[keep]]
    dn = s[torch.stack([b, a], 1).reshape(-1)[keep]]
    w = torch.stack([w, w], 1).reshape(-1)[keep]
    return up, dn, w - w[0]


def _vector(w, seed, flip_even=False):
    """A unit vector of the shape of Davidson's: large on the low determinants, a long tail."""
    gen = torch.Generator().manual_seed(seed + 7)
    v = torch.randn(len(w), generator=gen, dtype=torch.double)
    if flip_even:  # equal weight on a determinant and its spin flip, as in a converged state
        head = torch.cat([torch.ones(1, dtype=torch.bool), w[1:] != w[:-1]])
        v = v[head][head.long().cumsum(0) - 1]
    v = v * torch.exp(-0.35 * w)
    v[0] = 1.0
    return v / v.norm()


def _rows(up, dn):
    d = np.zeros((len(up), 4), dtype=np.uint64)
    d[:, 0] = up.numpy().view(np.uint64)
    d[:, 2] = dn.numpy().view(np.uint64)
    return d


def _inputs(case, seed):
    ints = synthetic_integrals(case["norb"], seed)
    up, dn, w = _determinants(case["norb"], case["nel"], case["n"], seed)
    return ints, up, dn, w


def _block(case, seed, w):
    return torch.stack([_vector(w, seed + 100 * k) for k in range(case["nvec"])], 1)


def prepare(case, seed):
    ints, up, dn, w = _inputs(case, seed)
    g = GpuHam(ints)
    s = dict(case=case, g=g, dets=_rows(up, dn))
    kind = case["kind"]
    if kind in ("sigma", "product"):
        g.set_dets(s["dets"])
        g.build(STORAGE[case["storage"]])
    if kind in ("sigma", "build"):
        x = _vector(w, seed).to(DEV)  # read as a vector in the library's sorted order
        s["x"] = x.float() if case.get("fp32") else x
        s["y"] = torch.empty_like(s["x"])
    elif kind == "product":
        s["x"] = _block(case, seed, w).numpy()
    elif kind == "solve":
        g.set_subspace(case["space"], case["keep"])
    elif kind == "select":
        g.set_dets(s["dets"])
        s["c"] = _vector(w, seed, flip_even=True).numpy()
        # where the program collects what it selects
        s["list"] = np.zeros((SELECT_MOST, 4), dtype=np.int64)
        s["list_diag"] = np.zeros(SELECT_MOST)
    return s


def run(s):
    case, g = s["case"], s["g"]
    kind = case["kind"]
    if kind == "sigma":
        g.sigma_device(s["x"].data_ptr(), s["y"].data_ptr(), 1 if case["fp32"] else 0)
        return s["y"]
    if kind == "product":
        return g.matrix_matrix_prod(s["x"])
    if kind == "build":
        g.set_dets(s["dets"])
        st = g.build(STORAGE[case["storage"]])
        g.sigma_device(s["x"].data_ptr(), s["y"].data_ptr(), 0)
        return {"nnz": int(st["nnz_upper"]), "y": s["y"]}
    if kind == "solve":
        g.set_dets(s["dets"])
        e, c, _, _ = g.sparse_optimize(max_iter=DAV_MAX_ITER, precision=STORAGE[case["storage"]])
        return {"energy": e, "coeffs": c}
    d, diag = g.find_new_dets(s["c"], case["eps"], case["singles"])
    s["list"][:len(d)] = d.view(np.int64)
    s["list_diag"][:len(d)] = diag
    return {"count": len(d), "dets": s["list"], "diag": s["list_diag"]}


# ---- what a pass cannot do without ----------------------------------------------------


@functools.lru_cache(maxsize=None)
def _pairs(norb, nel, n):
    """Stored pairs (upper triangle) of such a set, from a sample of its rows."""
    up, dn, _ = _determinants(norb, nel, n, 0)
    occ = _occupations(up, dn, norb).float()
    rows = torch.arange(0, n, max(1, n // 512))
    excited = 2 * nel - (occ[rows.to(DEV)] @ occ.T)
    return int(((excited == 1) | (excited == 2)).sum().item() / len(rows) * n / 2)


def work(case):
    n, kind = case["n"], case["kind"]
    z = _pairs(case["norb"], case["nel"], n)
    if kind == "select":  # the lists of every determinant above eps, about its connections
        return {"bytes": n * (32 + 16), "flops": 2 * z}
    value = 4 if case.get("fp32") else 8
    vec = 4 if case.get("fp32") else 8
    matrix = z * (4 + value)  # each pair once: an index and a value
    if kind == "sigma":
        return {"bytes": matrix + n * (8 + 2 * vec), "flops": 4 * z}
    if kind == "product":  # the matrix once for all vectors
        return {"bytes": matrix + n * (8 + 16 * case["nvec"]), "flops": 4 * z * case["nvec"]}
    if kind == "build":  # the strings in, the matrix out, and the product's read of it
        return {"bytes": 2 * matrix + n * (32 + 8 + 16), "flops": 6 * z}
    # solve: the matrix written once, and read by as many products as these solves take at least
    products = 40
    return {"bytes": (1 + products) * matrix + n * (32 + 16 * products), "flops": 4 * z * products}


# ---- plain torch in 64 bits -----------------------------------------------------------


def _occupations(up, dn, norb):
    k = torch.arange(norb, device=DEV)
    up, dn = up.to(DEV), dn.to(DEV)
    return torch.cat([(up[:, None] >> k) & 1, (dn[:, None] >> k) & 1], 1)


def _popcount(x):
    x = x - ((x >> 1) & 0x5555555555555555)
    x = (x & 0x3333333333333333) + ((x >> 2) & 0x3333333333333333)
    x = (x + (x >> 4)) & 0x0F0F0F0F0F0F0F0F
    x = x + (x >> 8)
    x = x + (x >> 16)
    return (x + (x >> 32)) & 0x7F


def _lowest(x):
    return _popcount((x & -x) - 1)


class _Hamiltonian:
    """Slater-Condon elements over int64 strings, vectorised."""

    def __init__(self, ints):
        n = ints.norb
        p = torch.arange(n)
        hi, lo = torch.maximum(p[:, None], p[None, :]), torch.minimum(p[:, None], p[None, :])
        pair = hi * (hi + 1) // 2 + lo + 1  # 1-based packed index of (p, q)
        a, b = pair[:, :, None, None], pair[None, None, :, :]
        four = torch.maximum(a, b) * (torch.maximum(a, b) - 1) // 2 + torch.minimum(a, b)
        self.h = torch.from_numpy(ints.one_body)[pair].to(DEV)
        self.g = torch.from_numpy(ints.two_body)[four].to(DEV)  # (pq|rs)
        self.coul = torch.einsum("ijkk->ijk", self.g).contiguous()
        self.exch = torch.einsum("ikkj->ijk", self.g).contiguous()
        self.nuc = ints.nuc
        self.norb = n

    def diag(self, occ):
        a, b = occ[:, :self.norb].double(), occ[:, self.norb:].double()
        j = torch.einsum("ppqq->pq", self.g)
        k = torch.einsum("pqqp->pq", self.g)
        t = a + b
        return (self.nuc + t @ self.h.diagonal() + 0.5 * ((t @ j) * t).sum(1)
                - 0.5 * ((a @ k) * a).sum(1) - 0.5 * ((b @ k) * b).sum(1))

    @staticmethod
    def _move(s, i, j):
        """Sign of moving an electron of string s from orbital i to j."""
        lo, hi = torch.minimum(i, j), torch.maximum(i, j)
        between = ((1 << hi) - 1) & ~((1 << (lo + 1)) - 1)
        return 1 - 2 * (_popcount(s & between) & 1)

    def single(self, s1, s2, occ_same, occ_opp):
        i, j = _lowest(s1 & ~s2), _lowest(s2 & ~s1)
        v = self.h[i, j] + ((occ_same + occ_opp) * self.coul[i, j]).sum(1) - (occ_same * self.exch[i, j]).sum(1)
        return self._move(s1, i, j) * v

    def same(self, s1, s2):
        r, a = s1 & ~s2, s2 & ~s1
        i, j = _lowest(r), _lowest(a)
        k, l = _lowest(r & (r - 1)), _lowest(a & (a - 1))
        mid = s1 ^ (1 << i) ^ (1 << j)
        return self._move(s1, i, j) * self._move(mid, k, l) * (self.g[i, j, k, l] - self.g[i, l, k, j])

    def opposite(self, a1, b1, a2, b2):
        i, j = _lowest(a1 & ~a2), _lowest(a2 & ~a1)
        k, l = _lowest(b1 & ~b2), _lowest(b2 & ~b1)
        return self._move(a1, i, j) * self._move(b1, k, l) * self.g[i, j, k, l]


def _products(ints, up, dn, nel, xs):
    """H times the columns of xs (double, on DEV), by blocks of rows against every determinant."""
    H = _Hamiltonian(ints)
    up, dn = up.to(DEV), dn.to(DEV)
    occ = _occupations(up, dn, ints.norb)
    half = occ.half() if DEV == "cuda" else occ.float()
    occ = occ.double()
    n = len(up)
    ys = H.diag(occ)[:, None] * xs
    step = max(64, min(n, (1 << 30) // n))
    for r0 in range(0, n, step):
        r1 = min(n, r0 + step)
        common = half[r0:r1] @ half[r0:].T
        i, j = (common >= 2 * nel - 2).nonzero(as_tuple=True)
        i, j = i + r0, j + r0
        i, j = i[j > i], j[j > i]
        da, db = _popcount(up[i] ^ up[j]) // 2, _popcount(dn[i] ^ dn[j]) // 2
        v = torch.zeros(len(i), dtype=torch.double, device=DEV)
        for mask, value in (
                ((da == 1) & (db == 0), lambda p, q: H.single(up[p], up[q], occ[p, :H.norb], occ[p, H.norb:])),
                ((da == 0) & (db == 1), lambda p, q: H.single(dn[p], dn[q], occ[p, H.norb:], occ[p, :H.norb])),
                ((da == 2) & (db == 0), lambda p, q: H.same(up[p], up[q])),
                ((da == 0) & (db == 2), lambda p, q: H.same(dn[p], dn[q])),
                ((da == 1) & (db == 1), lambda p, q: H.opposite(up[p], dn[p], up[q], dn[q]))):
            at = mask.nonzero(as_tuple=True)[0]
            v[at] = value(i[at], j[at])
        ys.index_add_(0, i, v[:, None] * xs[j])
        ys.index_add_(0, j, v[:, None] * xs[i])
    return ys


def exact(case, seed):
    kind = case["kind"]
    if kind == "select":
        return None  # a list of determinants in visiting order, with the diagonal each was given
    ints, up, dn, w = _inputs(case, seed)
    if kind == "product":
        return _products(ints, up, dn, case["nel"], _block(case, seed, w).to(DEV))
    if kind in ("sigma", "build"):
        x = _vector(w, seed).to(DEV)
        if case.get("fp32"):
            x = x.float().double()
        order = np.lexsort((dn.numpy(), up.numpy()))  # the library's order: by (up, dn)
        y = _products(ints, up[order], dn[order], case["nel"], x[:, None])[:, 0]
        return y if kind == "sigma" else {"nnz": None, "y": y}
    if case["n"] > 7000:
        return None  # the dense matrix and its eigenvalues take too long
    H = _products(ints, up, dn, case["nel"], torch.eye(case["n"], dtype=torch.double, device=DEV))
    return {"energy": float(torch.linalg.eigvalsh(H)[0]), "coeffs": None}
