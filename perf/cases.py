"""Performance cases of the polar / SVD path: what a user's program has it do, by public entry point.

The path's work is one dense solve per call (QDWH-PD, Zolo-PD, the batched QDWH-PD, the symmetric
eigensolver, the SVD), so a case is one whole call on one matrix or one batch, from the smallest sizes
(where the chain of launches is the time) to the largest, square and tall, even and odd, in the forms a
handle offers (reference stopping rule, fast form, mixed form) and through the host-array boundary.

Matrices are A = U diag(s) V^T with seeded random orthogonal factors and the spectra of the benchmark
configurations (s log-uniform over the condition number, its ends pinned).  The polar factor of A is
determined to about eps * kappa, so the cases that return Q keep kappa <= 1e6; the ill-conditioned
headline case (kappa = 1e12) returns H, which is determined to eps whatever kappa is.  The eigen and
singular vectors are compared as they come, so those spectra are evenly spread.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
F64 = torch.float64


def _pkg():
    if "zolo_svd_b200" not in sys.modules:
        d = os.path.join(ROOT, "zolo-svd_b200")
        spec = importlib.util.spec_from_file_location("zolo_svd_b200", os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["zolo_svd_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["zolo_svd_b200"]


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one small matrix: a call in a loop of a larger program (a rotation fit, a local basis)
        {"name": "qdwh_96", "kind": "qdwh", "m": 96, "n": 96, "kappa": 1e6},
        # the QDWH-PD configuration's size
        {"name": "qdwh_1024", "kind": "qdwh", "m": 1024, "n": 1024, "kappa": 1e6},
        # a tall matrix of odd sizes: orthogonalising a set of vectors
        {"name": "qdwh_1537x771", "kind": "qdwh", "m": 1537, "n": 771, "kappa": 1e4},
        # the reference driver's own two calls (bounds, then PZOLOPD1) with its stopping rule
        {"name": "zolo_driver_2048", "kind": "zolo_driver", "m": 2048, "n": 2048, "kappa": 1e6, "rk": 8},
        # Zolo-PD in one call, fast form, odd and tall
        {"name": "zolo_fast_2501x1203", "kind": "zolo", "form": "fast", "m": 2501, "n": 1203, "kappa": 1e5, "rk": 8},
        # the Zolo-PD configuration's size, fast form in FP64
        {"name": "zolo_fast_4096", "kind": "zolo", "form": "fast", "m": 4096, "n": 4096, "kappa": 1e6, "rk": 8},
        # the headline: n = 8192, kappa = 1e12, mixed form
        {"name": "zolo_mixed_8192", "kind": "zolo", "form": "mixed", "m": 8192, "n": 8192, "kappa": 1e12, "rk": 8},
        # the batch configuration: 512 matrices, n log-uniform in [64, 1024], m in [n, 2n]
        {"name": "batch_512", "kind": "batch", "count": 512, "nmin": 64, "nmax": 1024, "sizes": 1004, "kappa": 1e6},
        # a batch of small matrices
        {"name": "batch_64_small", "kind": "batch", "count": 64, "nmin": 16, "nmax": 160, "sizes": 7, "kappa": 1e4},
        # singular value decomposition of a tall matrix, fast form
        {"name": "svd_2048x1024", "kind": "svd", "form": "fast", "m": 2048, "n": 1024, "rk": 8},
        # symmetric eigendecomposition, odd size
        {"name": "eig_701", "kind": "eig", "n": 701},
        # the reference-named host-array entry on a symmetric matrix with a shift (a spectral split)
        {"name": "host_split_512", "kind": "host", "n": 512},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["qdwh", "qdwh", "zolo_driver", "zolo", "zolo", "batch", "svd", "eig", "host"])
    kappa = 10.0 ** rng.uniform(1.0, 6.0)
    if kind == "qdwh":
        n = _log(rng, 32, 1600)
        return {"kind": kind, "m": int(n * rng.uniform(1.0, 2.0)), "n": n, "kappa": kappa}
    if kind == "zolo_driver":
        n = _log(rng, 128, 2200)
        return {"kind": kind, "m": int(n * rng.uniform(1.0, 1.4)), "n": n, "kappa": kappa, "rk": rng.randint(2, 8)}
    if kind == "zolo":
        n = _log(rng, 128, 4096)
        return {"kind": kind, "form": rng.choice(["fast", "mixed"]), "m": int(n * rng.uniform(1.0, 1.6)), "n": n,
                "kappa": kappa, "rk": rng.randint(4, 8)}
    if kind == "batch":
        nmax = _log(rng, 96, 900)
        return {"kind": kind, "count": _log(rng, 8, 256), "nmin": max(8, nmax // rng.randint(2, 16)), "nmax": nmax,
                "sizes": rng.randrange(1 << 20), "kappa": kappa}
    if kind == "svd":
        n = _log(rng, 100, 1200)
        return {"kind": kind, "form": rng.choice(["fast", "mixed"]), "m": int(n * rng.uniform(1.0, 2.0)), "n": n,
                "rk": 8}
    if kind == "eig":
        return {"kind": kind, "n": _log(rng, 70, 1000)}
    return {"kind": "host", "n": _log(rng, 32, 800)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _signs(n, g):
    return torch.randint(0, 2, (n,), generator=g, device="cuda", dtype=torch.int64).to(F64) * 2 - 1


def _cosine(n, cols=None):
    """The first `cols` columns of the orthogonal, symmetric cosine matrix sqrt(2/n) cos(pi (2i+1)(2j+1) / 4n)."""
    t = torch.cos(torch.arange(8 * n, dtype=F64, device="cuda") * (math.pi / (4 * n))) * math.sqrt(2.0 / n)
    i = 2 * torch.arange(n, device="cuda") + 1
    j = i if cols is None else i[:cols]
    return t[(i[:, None] * j[None, :]) % (8 * n)]


def _orthogonal(m, n, g):
    """m x n with orthonormal columns: two cosine transforms between random signs, the rows in random order (without
    that the columns keep a Toeplitz structure, on which unpivoted QR is less accurate than on a Haar matrix)."""
    left = _signs(m, g)[:, None] * _cosine(m)
    right = _signs(m, g)[:, None] * _cosine(m, n) * _signs(n, g)[None, :]
    return (left @ right)[torch.randperm(m, generator=g, device="cuda")]


def _spectrum(n, kappa, g):
    """Log-uniform in [1/kappa, 1], both ends pinned, descending."""
    e = torch.rand(n, generator=g, device="cuda", dtype=F64) * -math.log10(kappa)
    e[0] = 0.0
    if n > 1:
        e[-1] = -math.log10(kappa)
    return torch.sort(10.0 ** e, descending=True).values


def _even_spectrum(n, lo, hi, g):
    """Ascending, evenly spread in [lo, hi] with a quarter of a step of jitter."""
    i = torch.arange(n, device="cuda", dtype=F64)
    u = torch.rand(n, generator=g, device="cuda", dtype=F64) - 0.5
    return lo + (hi - lo) * (i + 0.5 + 0.5 * u) / n


def _general(m, n, kappa, g):
    u, v = _orthogonal(m, n, g), _orthogonal(n, n, g)
    s = _spectrum(n, kappa, g)
    return u, s, v


def _batch_sizes(case):
    r = np.random.default_rng(case["sizes"])
    out = []
    for _ in range(case["count"]):
        n = int(round(math.exp(r.uniform(math.log(case["nmin"]), math.log(case["nmax"])))))
        out.append((int(round(n * (1 + r.uniform(0, 1)))), n, 10.0 ** r.uniform(1.0, math.log10(case["kappa"]))))
    return out


def _symmetric(case, seed):
    g = _gen(seed)
    n = case["n"]
    z = _orthogonal(n, n, g)
    if case["kind"] == "host":
        w = _even_spectrum(n, -1.0, 1.0, g)
        k = n // 3
        sigma = 0.5 * float(w[k - 1] + w[k])  # between two eigenvalues: the split's shift
    else:
        w, sigma = _even_spectrum(n, -1.0, 2.0, g), 0.0
    a = (z * w[None, :]) @ z.T
    return 0.5 * (a + a.T), z, w, sigma


_HANDLES = {}


def _handle(form):
    """The library handle that the program keeps for one form of the algorithm."""
    if form not in _HANDLES:
        zb = _pkg()
        h = zb.Handle(0)
        if form in ("fast", "mixed"):
            for o in (zb.OPT_NS_FINISH, zb.OPT_CHOL_INVERSE, zb.OPT_BETA_FROB, zb.OPT_TERM_PLAN):
                h.set_option(o, 1)
        if form == "mixed":
            h.set_option(zb.OPT_MIXED, 1)
        _HANDLES[form] = h
    return _HANDLES[form]


def prepare(case, seed):
    """Column-major device arrays (tensor[j, i] = A[i, j]), output buffers and the handle."""
    kind = case["kind"]
    st = {"case": case, "zb": _pkg()}
    if kind == "host":
        a, _, _, sigma = _symmetric(case, seed)
        st.update(a=np.asfortranarray(a.cpu().numpy()), sigma=sigma)
        return st
    st["h"] = _handle(case.get("form", "default"))
    if kind == "eig":
        n = case["n"]
        a = _symmetric(case, seed)[0]
        st.update(a=a.contiguous(), w=torch.empty(n, dtype=F64, device="cuda"), z=torch.empty_like(a))
        return st
    g = _gen(seed)
    if kind == "batch":
        sizes = _batch_sizes(case)
        qs, hs = sum(m * n for m, n, _ in sizes), sum(n * n for _, n, _ in sizes)
        st.update(a=torch.empty(qs, dtype=F64, device="cuda"), q=torch.empty(qs, dtype=F64, device="cuda"),
                  hh=torch.empty(hs, dtype=F64, device="cuda"), members=[])
        oq = oh = 0
        for m, n, kappa in sizes:
            u, s, v = _general(m, n, kappa, g)
            st["a"][oq:oq + m * n].view(n, m).copy_((v * s[None, :]) @ u.T)
            st["members"].append((m, n, st["a"].data_ptr() + 8 * oq, m, st["q"].data_ptr() + 8 * oq, m,
                                  st["hh"].data_ptr() + 8 * oh, n))
            oq, oh = oq + m * n, oh + n * n
        return st
    m, n = case["m"], case["n"]
    if kind == "svd":
        u, v = _orthogonal(m, n, g), _orthogonal(n, n, g)
        s = _even_spectrum(n, 0.1, 1.0, g)
    else:
        u, s, v = _general(m, n, case["kappa"], g)
    st["a"] = ((v * s[None, :]) @ u.T).contiguous()
    st["q"] = torch.empty_like(st["a"])
    st["hh"] = torch.empty((n, n), dtype=F64, device="cuda")
    if kind == "svd":
        st["s"] = torch.empty(n, dtype=F64, device="cuda")
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(st):
    case, zb = st["case"], st["zb"]
    kind = case["kind"]
    if kind == "host":
        q, h, info = zb.pqdwhfacs("S", st["a"], sigma=st["sigma"], polar="T")
        return {"q": q, "h": h, "info": info}
    lib = st["h"]
    if kind == "eig":
        n = case["n"]
        zb.syev_dev(lib, n, st["a"].data_ptr(), n, st["w"].data_ptr(), st["z"].data_ptr(), n)
        return {"w": st["w"], "z": st["z"]}
    if kind == "batch":
        info, _ = zb.qdwh_batch_dev(lib, st["members"])
        return {"q": st["q"], "h": st["hh"], "info": sum(1 for v in info if v)}
    m, n = case["m"], case["n"]
    pa, pq, ph = st["a"].data_ptr(), st["q"].data_ptr(), st["hh"].data_ptr()
    if kind == "qdwh":
        zb.qdwh_dev(lib, "N", m, n, 0.0, pa, m, pq, m, ph, n, 0, 12, 0)
    elif kind == "zolo_driver":
        alpha, beta, _ = zb.bounds_dev(lib, m, n, pa, m, mode=1)
        zb.pzolopd1_dev(lib, "N", case["rk"], m, n, alpha, beta, pa, m, pq, m, ph, n)
    elif kind == "zolo":
        zb.polar_dev(lib, case["rk"], m, n, pa, m, pq, m, ph, n)
        if case["kappa"] > 1e6:
            return {"h": st["hh"]}
    else:
        zb.svd_dev(lib, m, n, pa, m, pq, m, st["s"].data_ptr(), ph, n, algo=1, rk=case["rk"])
        return {"u": st["q"], "s": st["s"], "v": st["hh"]}
    return {"q": st["q"], "h": st["hh"]}


# ---------------------------------------------------------------------------
# what a pass cannot do without, and its result in 64 bits
# ---------------------------------------------------------------------------
def _polar_flops(m, n, kappa):
    """QDWH's own steps (pqdwhfacs.f90:359-457) from L = 1/kappa: QR form 4mn^2 + n^3, Cholesky form
    3mn^2 + n^3/3, and the bounds' QR 2mn^2 - 2n^3/3 and H 2mn^2."""
    l, f = 1.0 / kappa, 4.0 * m * n * n - 2.0 * n ** 3 / 3.0
    while abs(1.0 - l) > 1e-15:
        d = (4.0 * (1.0 - l * l) / l ** 4) ** (1.0 / 3.0)
        a = math.sqrt(1.0 + d) + 0.5 * math.sqrt(8.0 - 4.0 * d + 8.0 * (2.0 - l * l) / (l * l * math.sqrt(1.0 + d)))
        b = (a - 1.0) ** 2 / 4.0
        c = a + b - 1.0
        f += 4.0 * m * n * n + n ** 3 if c > 100.0 else 3.0 * m * n * n + n ** 3 / 3.0
        l = min(1.0, l * (a + b * l * l) / (1.0 + c * l * l))
    return f


def work(case):
    kind = case["kind"]
    if kind == "batch":
        sizes = _batch_sizes(case)
        return {"bytes": 8.0 * sum(2 * m * n + n * n for m, n, _ in sizes),
                "flops": sum(_polar_flops(m, n, k) for m, n, k in sizes)}
    n = case["n"]
    if kind == "eig":  # reduction to tridiagonal form 4n^3/3, its eigenvectors 4n^3/3, back-transformation 2n^3
        return {"bytes": 8.0 * (2 * n * n + n), "flops": (8.0 / 3.0 + 2.0) * n ** 3}
    if kind == "host":
        return {"bytes": 8.0 * 3 * n * n, "flops": _polar_flops(n, n, 2.0 * n)}
    m = case["m"]
    if kind == "svd":
        return {"bytes": 8.0 * (2 * m * n + n * n + n),
                "flops": _polar_flops(m, n, 10.0) + (8.0 / 3.0 + 2.0) * n ** 3 + 2.0 * m * n * n}
    return {"bytes": 8.0 * (2 * m * n + n * n), "flops": _polar_flops(m, n, case["kappa"])}


def exact(case, seed):
    """Q = U V^T and H = V diag(s) V^T of the constructed factors (of a symmetric matrix with a shift Q = Z sign(w - sigma)
    Z^T and H = sym(Q^T A) = Z w sign(w - sigma) Z^T), s and w themselves; singular and eigenvectors only up to sign,
    so None."""
    kind = case["kind"]
    if kind == "host":
        _, z, w, sigma = _symmetric(case, seed)
        q = (z * torch.sign(w - sigma)[None, :]) @ z.T
        h = (z * (w * torch.sign(w - sigma))[None, :]) @ z.T
        return {"q": q.cpu().numpy(), "h": h.cpu().numpy(), "info": 0}
    if kind == "eig":
        return {"w": _symmetric(case, seed)[2], "z": None}
    g = _gen(seed)
    if kind == "batch":
        q, h = [], []
        for m, n, kappa in _batch_sizes(case):
            u, s, v = _general(m, n, kappa, g)
            q.append((v @ u.T).reshape(-1))
            h.append(((v * s[None, :]) @ v.T).reshape(-1))
        return {"q": torch.cat(q), "h": torch.cat(h), "info": 0}
    m, n = case["m"], case["n"]
    if kind == "svd":
        _orthogonal(m, n, g), _orthogonal(n, n, g)
        return {"u": None, "s": _even_spectrum(n, 0.1, 1.0, g), "v": None}
    u, s, v = _general(m, n, case["kappa"], g)
    h = (v * s[None, :]) @ v.T
    if kind == "zolo" and case["kappa"] > 1e6:
        return {"h": h}
    return {"q": v @ u.T, "h": h}
