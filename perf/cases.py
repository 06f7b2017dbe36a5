"""Timed cases of the library, each through the entry points its users call.

A program that uses the library builds a problem from its points once (the
cluster and the kernel handle are kept), then

  approximate   compresses the kernel matrix and multiplies the result with a
                block of vectors: starsh_b200_approximate (either engine, with
                device-resident factors) and starsh_b200_blrm_dmml_device;
  dropin        the same through the calls of the host interface:
                starsh_blrm__drsdd_b200[_mp] with every factor copied back to
                host memory, and starsh_blrm__dmml on host arrays;
  batch         many small problems of mixed kernels, sizes and tolerances in
                one starsh_b200_approximate_batch, then each one's product
                (what a server does with the requests of one group);
  product       products on a matrix that was compressed before, for the
                general and the symmetric format, with stored or regenerated
                dense blocks;
  cg            a solve by conjugate gradients on such a matrix;
  error         the relative Frobenius error of such a matrix.

Sizes are those of the repository's benchmark workloads and tests: 2-D and
3-D point sets of 2,000 to 102,400 points, block sizes 128 to 1024 (1500 for
a draw), tolerances 1e-3 to 1e-7.
"""
import ctypes
import math
import os
import random
import sys
from ctypes import POINTER, byref, c_double, c_int, c_void_p

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(
    os.path.abspath(__file__))), "stars-h_b200"))
import starsh_b200 as sb  # noqa: E402

DEV = "cuda"


def listed():
    return [
        # The reference's own example size (81 blocks of 400): a call whose
        # time is launches, host turnarounds and short serial kernels.
        dict(name="small_exp2d", op="approximate", kernel="exp", ndim=2,
             n=3600, nb=400, maxrank=100, oversample=10, tol=1e-5, nrhs=1,
             engine="mixed", symm=False, onfly=False),
        # The median request of the serving mix, with its 32 products; a
        # ragged last block.
        dict(name="request_matern2d", op="approximate", kernel="matern32",
             ndim=2, n=8281, nb=512, maxrank=256, oversample=10, tol=1e-4,
             nrhs=32, engine="mixed", symm=False, onfly=False),
        # A 3-D oscillating kernel of the same mix at its tighter tolerance,
        # symmetric format, dense blocks regenerated in the product.
        dict(name="request_sin3d_symm", op="approximate", kernel="sin",
             ndim=3, n=15625, nb=512, maxrank=200, oversample=10, tol=1e-6,
             nrhs=32, engine="mixed", symm=True, onfly=True),
        # Matern with a general smoothness (Bessel function per entry).
        dict(name="matern_general2d", op="approximate", kernel="matern",
             ndim=2, n=16384, nb=1024, maxrank=256, oversample=16, tol=1e-7,
             nrhs=8, engine="mixed", symm=False, onfly=False),
        # The benchmark's default workload: 10,000 blocks of 1024, the
        # largest 2-D problem.
        dict(name="large_sqexp2d", op="approximate", kernel="sqexp", ndim=2,
             n=102400, nb=1024, maxrank=256, oversample=16, tol=1e-7,
             nrhs=32, engine="mixed", symm=False, onfly=False),
        # The benchmark's electrostatics workload with its 64 products:
        # 16,384 blocks of 512 on random 3-D points.
        dict(name="large_coulomb3d", op="approximate", kernel="coulomb",
             ndim=3, n=65536, nb=512, maxrank=200, oversample=10, tol=1e-5,
             nrhs=64, engine="mixed", symm=False, onfly=False),
        # A host program that replaces the reference's library: FP64 engine
        # (the backend's default), factors and products in host memory.
        dict(name="dropin_fp64_sqexp2d", op="dropin", kernel="sqexp", ndim=2,
             n=16384, nb=512, maxrank=100, oversample=10, tol=1e-5, nrhs=16,
             engine="fp64", symm=False, onfly=False),
        # One group of the many-problem workload.
        dict(name="batch_mixed", op="batch", problems=24, nmin=1024,
             nmax=12000, mix=3, oversample=10, nrhs=32),
        # The product that the electrostatics workload reports, 64 columns.
        dict(name="product_64", op="product", kernel="coulomb", ndim=3,
             n=32768, nb=512, maxrank=200, oversample=10, tol=1e-5, nrhs=64,
             symm=False, onfly=False),
        # One vector at a time, as an iterative solver or a time stepper
        # calls it, on a symmetric matrix.
        dict(name="product_1_symm", op="product", kernel="exp", ndim=2,
             n=25600, nb=512, maxrank=200, oversample=10, tol=1e-5, nrhs=1,
             symm=True, onfly=False),
        # A covariance solve: exponential kernel with a nugget, one
        # right-hand side.
        dict(name="cg_exp2d", op="cg", kernel="exp", ndim=2, n=10000, nb=500,
             maxrank=200, oversample=10, tol=1e-6, nrhs=1, cg_tol=1e-8,
             noise=0.5, symm=False, onfly=False),
        # The accuracy check that follows an approximation.
        dict(name="error_sqexp2d", op="error", kernel="sqexp", ndim=2,
             n=25600, nb=1024, maxrank=256, oversample=16, tol=1e-7,
             symm=False, onfly=False),
    ]


KERNELS = {"exp": (2, 3), "sqexp": (2, 3), "matern32": (2, 3),
           "matern": (2,), "coulomb": (3,), "sin": (3,), "rbf": (3,)}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["approximate"] * 5 + ["dropin", "batch", "product",
                                           "product", "cg", "error"])
    if op == "batch":
        return dict(op=op, problems=rng.randint(6, 28), nmin=1024,
                    nmax=_log(rng, 3000, 12000), mix=rng.randint(10, 10 ** 6),
                    oversample=10, nrhs=rng.choice([1, 8, 32]))
    kernel = rng.choice(sorted(KERNELS))
    ndim = rng.choice(KERNELS[kernel])
    tol = rng.choice([1e-3, 1e-4, 1e-5, 1e-6, 1e-7])
    # the smooth kernels are used at the largest sizes
    hi = 70000 if kernel in ("sqexp", "coulomb") and tol >= 1e-5 else 30000
    n = _log(rng, 2000, hi if op == "approximate" else 24000)
    nb = _log(rng, 128, 1024) if n < 12000 else _log(rng, 400, 1024)
    if n >= 12000 and rng.random() < 0.1:
        nb = 1500
    nb = min(nb, n // 4)
    c = dict(op=op, kernel=kernel, ndim=ndim, n=n, nb=nb,
             maxrank=rng.choice([min(nb // 2, 256), min(nb // 2, 200), 100]),
             oversample=rng.choice([10, 16]), tol=tol,
             symm=rng.random() < 0.3, onfly=rng.random() < 0.3)
    if op in ("approximate", "dropin"):
        c["engine"] = "fp64" if rng.random() < 0.25 else "mixed"
    if op == "cg":
        c.update(kernel="exp", ndim=2, n=_log(rng, 2000, 12000), noise=0.5,
                 tol=1e-6, cg_tol=rng.choice([1e-6, 1e-8]))
        c["nb"] = min(_log(rng, 128, 800), c["n"] // 4)
        c["maxrank"] = min(c["nb"] // 2, 200)
    if op != "error":
        c["nrhs"] = rng.choice([1, 3, 8]) if op == "cg" else \
            rng.choice([1, 5, 8, 16, 32, 50, 64])
    return c


# ------------------------------------------------------------- point sets

def _points(kernel, ndim, n, rng):
    """(ndim, n) coordinates in Z-order: a jittered grid (spatial kernels),
    uniform points (electro-*), or the surfaces of 1-8 spheres (RBF)."""
    if kernel == "rbf":
        ns = int(rng.integers(1, 9))
        centre = rng.uniform(0.0, 1.0, (ns, 3))
        radius = rng.uniform(0.05, 0.2, ns)
        which = rng.integers(0, ns, n)
        v = rng.standard_normal((n, 3))
        v /= np.linalg.norm(v, axis=1)[:, None]
        x = (centre[which] + radius[which, None] * v).T
    elif kernel in ("coulomb", "sin"):
        x = rng.uniform(0.0, 1.0, (ndim, n))
    else:
        # the n points of the smallest grid that holds them, each moved by
        # less than half a cell
        side = int(math.ceil(round(n ** (1.0 / ndim), 6)))
        while side ** ndim < n:
            side += 1
        cell = np.sort(rng.choice(side ** ndim, n, replace=False))
        idx = np.stack([(cell // side ** d) % side for d in range(ndim)])
        x = (idx + 0.5 + 0.8 * (rng.random((ndim, n)) - 0.5)) / side
    lo, hi = x.min(axis=1, keepdims=True), x.max(axis=1, keepdims=True)
    q = ((x - lo) / (hi - lo) * 65535.0).astype(np.uint64)
    code = np.zeros(x.shape[1], dtype=np.uint64)
    for bit in range(16):
        for d in range(x.shape[0]):
            code |= ((q[d] >> np.uint64(bit)) & np.uint64(1)) << np.uint64(
                x.shape[0] * bit + d)
    return np.ascontiguousarray(x[:, np.argsort(code, kind="stable")])


BETA, WAVE_K, RBF_RAD, MATERN_NU, MATERN_BETA = 0.1, 20.0, 0.1, 0.7, 0.05


def _spec(case, seed):
    """The problem's description and its points, from the seed alone."""
    kernel = case["kernel"]
    rng = np.random.default_rng([int(seed), case["n"], case["ndim"]])
    return dict(case, noise=case.get("noise", 0.0),
                x=_points(kernel, case["ndim"], case["n"], rng))


def _batch_specs(case, seed):
    """The batch's problems: sizes, kernels and tolerances from the case,
    points from the seed."""
    r = random.Random(case["mix"])
    out = []
    for p in range(case["problems"]):
        kernel = r.choice(["exp", "sqexp", "matern32", "coulomb", "rbf"])
        n = _log(r, case["nmin"], case["nmax"])
        nb = 256 if n <= 2048 else 512 if n <= 8192 else 1024
        ndim = 3 if kernel in ("coulomb", "rbf") else 2
        out.append(_spec(dict(kernel=kernel, ndim=ndim, n=n, nb=nb,
                              maxrank=min(nb // 2, 256),
                              tol=r.choice([1e-3, 1e-5, 1e-7]), symm=False,
                              onfly=False), seed * 1000 + p))
    return out


# --------------------------------------------------------- library objects

def _lib():
    lib = sb.load()
    assert lib.starsh_b200_set_device(torch.cuda.current_device()) == 0
    if not hasattr(lib, "_cases_proto"):
        for name in ("starsh_esdata_free", "starsh_eddata_free",
                     "starsh_mddata_free"):
            f = getattr(lib, name)
            f.restype, f.argtypes = None, [c_void_p]
        lib._cases_proto = True
    return lib


def _malloc(values):
    """A malloc'd copy (the library owns and frees its point arrays)."""
    libc = ctypes.CDLL("libc.so.6")
    libc.malloc.restype = c_void_p
    a = np.ascontiguousarray(values, dtype=np.float64).ravel()
    p = libc.malloc(ctypes.c_size_t(a.nbytes))
    ctypes.memmove(p, a.ctypes.data, a.nbytes)
    return ctypes.cast(p, POINTER(c_double))


class Problem:
    """A STARSH_problem with its data and cluster, kept by the program."""

    def __init__(self, spec):
        lib = self.lib = _lib()
        k, n, x = spec["kernel"], spec["n"], spec["x"]
        self.spec, self.n = spec, n
        self.symm = b"S" if spec["symm"] else b"N"
        kern = c_void_p()
        if k in ("exp", "sqexp", "matern32", "matern"):
            self.data = POINTER(sb.SSData)()
            beta = MATERN_BETA if k == "matern" else BETA
            nu = MATERN_NU if k == "matern" else 1.5
            assert lib.starsh_ssdata_init(byref(self.data), n, spec["ndim"],
                                          _malloc(x), beta, nu,
                                          spec["noise"], 1.0) == 0
            kt = {"exp": sb.EXP, "sqexp": sb.SQREXP}.get(k, sb.MATERN)
            assert lib.starsh_ssdata_get_kernel(byref(kern), self.data, kt) == 0
            self.free_data = lib.starsh_ssdata_free
        elif k == "coulomb":
            self.data = POINTER(sb.Particles)()
            assert lib.starsh_esdata_init(byref(self.data), n, 3,
                                          _malloc(x)) == 0
            assert lib.starsh_esdata_get_kernel(byref(kern), self.data,
                                                sb.COULOMB) == 0
            self.free_data = lib.starsh_esdata_free
        elif k == "sin":
            self.data = POINTER(sb.EDData)()
            assert lib.starsh_eddata_init(byref(self.data), n, 3, _malloc(x),
                                          WAVE_K, 1.0) == 0
            assert lib.starsh_eddata_get_kernel(byref(kern), self.data,
                                                sb.SIN) == 0
            self.free_data = lib.starsh_eddata_free
        else:
            self.data = POINTER(sb.MDData)()
            assert lib.starsh_mddata_init(byref(self.data), n, _malloc(x.T),
                                          0, 1, 0, 0.0, RBF_RAD, 0.0) == 0
            kern = c_void_p(sb.kernel_symbol(lib, "starsh_generate_3d_virus"))
            self.free_data = lib.starsh_mddata_free
        shape = (sb.STARSH_int * 2)(n, n)
        self.P = POINTER(sb.Problem)()
        assert lib.starsh_problem_new(byref(self.P), 2, shape, self.symm,
                                      b"d", self.data, self.data, kern,
                                      b"case") == 0
        self.C = POINTER(sb.Cluster)()
        assert lib.starsh_cluster_new_plain(byref(self.C), self.data, n,
                                            spec["nb"]) == 0

    def format(self):
        F = POINTER(sb.Blrf)()
        assert self.lib.starsh_blrf_new_tlr(byref(F), self.P, self.symm,
                                            self.C, self.C) == 0
        return F

    def __del__(self):
        if getattr(self, "C", None):
            self.lib.starsh_cluster_free(self.C)
            self.lib.starsh_problem_free(self.P)
            self.free_data(self.data)


class Matrix:
    """A compressed matrix and its format."""

    def __init__(self, lib, M, F):
        self.lib, self.M, self.F = lib, M, F

    def ranks(self):
        """The rank of every block, -1 where it is stored dense."""
        F = self.F.contents
        out = np.full((F.nbrows, F.nbcols), -1, dtype=np.int32)
        if F.nblocks_far > 0:
            ij = np.ctypeslib.as_array(F.block_far, (F.nblocks_far, 2))
            out[ij[:, 0], ij[:, 1]] = np.ctypeslib.as_array(
                self.M.contents.far_rank, (F.nblocks_far,))
        return out

    def free(self):
        if self.M is not None:
            self.lib.starsh_blrm_free(self.M)
            self.lib.starsh_blrf_free(self.F)
            self.M = self.F = None

    def __del__(self):
        self.free()


ENGINE = {"fp64": sb.ENGINE_FP64, "mixed": sb.ENGINE_MIXED}


def _approximate(pr, engine, oversample):
    lib, sp = pr.lib, pr.spec
    lib.starsh_set_oversample(str(oversample).encode())
    F, M = pr.format(), POINTER(sb.Blrm)()
    info = lib.starsh_b200_approximate(byref(M), F, sp["maxrank"], sp["tol"],
                                       1 if sp["onfly"] else 0,
                                       ENGINE[engine], 0)
    assert info == 0, (info, lib.starsh_b200_last_error())
    return Matrix(lib, M, F)


def _product(mat, n, X, B, stream):
    """B = M X on the device; row j of X and B is column j of the operand."""
    info = mat.lib.starsh_b200_blrm_dmml_device(
        mat.M, X.shape[0], 1.0, X.data_ptr(), n, 0.0, B.data_ptr(), n,
        stream.cuda_stream)
    assert info == 0, (info, mat.lib.starsh_b200_last_error())


def _vectors(n, nrhs, seed):
    g = torch.Generator(device="cpu").manual_seed(int(seed) * 7919 + n)
    return torch.randn(nrhs, n, dtype=torch.float64, generator=g)


# ------------------------------------------------------------------- cases

def prepare(case, seed):
    s = dict(case=case, stream=torch.cuda.Stream())
    op = case["op"]
    if op == "batch":
        specs = _batch_specs(case, seed)
        s["problems"] = [Problem(sp) for sp in specs]
        s["X"] = [_vectors(sp["n"], case["nrhs"], seed * 1000 + p).to(DEV)
                  for p, sp in enumerate(specs)]
        s["B"] = [torch.empty_like(x) for x in s["X"]]
        torch.cuda.synchronize()
        return s
    pr = s["problem"] = Problem(_spec(case, seed))
    if op == "dropin":
        s["X"] = _vectors(case["n"], case["nrhs"], seed).numpy()
        s["B"] = np.empty_like(s["X"])
        return s
    if op != "error":
        s["X"] = _vectors(case["n"], case["nrhs"], seed).to(DEV)
        s["B"] = torch.empty_like(s["X"])
    if op in ("product", "cg", "error"):
        s["matrix"] = _approximate(pr, "mixed", case["oversample"])
    torch.cuda.synchronize()
    return s


def run(state):
    case, stream = state["case"], state["stream"]
    return {"approximate": _run_approximate, "dropin": _run_dropin,
            "batch": _run_batch, "product": _run_product, "cg": _run_cg,
            "error": _run_error}[case["op"]](case, state, stream)


def _run_approximate(case, s, stream):
    mat = _approximate(s["problem"], case["engine"], case["oversample"])
    _product(mat, case["n"], s["X"], s["B"], stream)
    ranks = mat.ranks()
    mat.free()
    return {"B": s["B"], "ranks": ranks}


def _run_dropin(case, s, stream):
    pr, n = s["problem"], case["n"]
    lib = pr.lib
    lib.starsh_set_oversample(str(case["oversample"]).encode())
    F, M = pr.format(), POINTER(sb.Blrm)()
    call = (lib.starsh_blrm__drsdd_b200 if case["engine"] == "fp64"
            else lib.starsh_blrm__drsdd_b200_mp)
    info = call(byref(M), F, case["maxrank"], case["tol"],
                1 if case["onfly"] else 0)
    assert info == 0, (info, lib.starsh_b200_last_error())
    mat = Matrix(lib, M, F)
    pd = POINTER(c_double)
    info = lib.starsh_blrm__dmml(M, case["nrhs"], 1.0,
                                 s["X"].ctypes.data_as(pd), n, 0.0,
                                 s["B"].ctypes.data_as(pd), n)
    assert info == 0, (info, lib.starsh_b200_last_error())
    ranks = mat.ranks()
    mat.free()
    return {"B": s["B"], "ranks": ranks}


def _run_batch(case, s, stream):
    prs = s["problems"]
    lib, np_ = prs[0].lib, len(prs)
    lib.starsh_set_oversample(str(case["oversample"]).encode())
    Fs = [pr.format() for pr in prs]
    Ms = (POINTER(sb.Blrm) * np_)()
    info = lib.starsh_b200_approximate_batch(
        np_, Ms, (POINTER(sb.Blrf) * np_)(*Fs),
        (c_int * np_)(*[pr.spec["maxrank"] for pr in prs]),
        (c_double * np_)(*[pr.spec["tol"] for pr in prs]), None,
        sb.ENGINE_MIXED, 0)
    assert info == 0, (info, lib.starsh_b200_last_error())
    mats = [Matrix(lib, Ms[p], Fs[p]) for p in range(np_)]
    for p, mat in enumerate(mats):
        _product(mat, prs[p].n, s["X"][p], s["B"][p], stream)
    ranks = [mat.ranks() for mat in mats]
    for mat in mats:
        mat.free()
    return {"B": s["B"], "ranks": ranks}


def _run_product(case, s, stream):
    _product(s["matrix"], case["n"], s["X"], s["B"], stream)
    return s["B"]


def _run_cg(case, s, stream):
    n, X = case["n"], s["B"]
    with torch.cuda.stream(stream):
        X.zero_()
    its = c_int()
    lib = s["problem"].lib
    info = lib.starsh_b200_dcg_device(s["matrix"].M, case["nrhs"],
                                      s["X"].data_ptr(), n, X.data_ptr(), n,
                                      case["cg_tol"], 0, stream.cuda_stream,
                                      byref(its))
    assert info == 0 and its.value >= 0, (info, its.value)
    return {"X": X, "iterations": its.value}


def _run_error(case, s, stream):
    return np.array([s["problem"].lib.starsh_blrm__dfe_b200(s["matrix"].M)])


# ------------------------------------------------- exact values, 64 bits

def _bessel_k(nu, x):
    """K_nu(x) = int_0^inf exp(-x cosh t) cosh(nu t) dt by the trapezoidal
    rule (the integrand is analytic and decays double-exponentially)."""
    h, s = 0.125, torch.zeros_like(x)
    for k in range(0, 110):
        t = k * h
        s += (0.5 if k == 0 else 1.0) * math.cosh(nu * t) * torch.exp(
            -x * math.cosh(t))
    return h * s


def _rows(spec, x, r0, r1):
    """Rows r0 .. r1 - 1 of the kernel matrix."""
    k = spec["kernel"]
    d2 = torch.zeros(r1 - r0, x.shape[1], dtype=torch.float64, device=DEV)
    for d in range(x.shape[0]):
        t = x[d, r0:r1, None] - x[d, None, :]
        d2 += t * t
    zero = d2 == 0.0
    if k == "exp":
        a = torch.exp(-torch.sqrt(d2) / BETA)
    elif k == "sqexp":
        a = torch.exp(-d2 / (2.0 * BETA * BETA))
    elif k == "matern32":
        r = torch.sqrt(d2) * math.sqrt(3.0) / BETA
        a = (1.0 + r) * torch.exp(-r)
    elif k == "matern":
        r = torch.sqrt(d2) * math.sqrt(2.0 * MATERN_NU) / MATERN_BETA
        r[zero] = 1.0
        a = (2.0 ** (1.0 - MATERN_NU) / math.gamma(MATERN_NU)
             * r ** MATERN_NU * _bessel_k(MATERN_NU, r))
    elif k == "rbf":
        return torch.exp(-d2 / (RBF_RAD * RBF_RAD))
    else:
        r = torch.sqrt(d2)
        r[zero] = 1.0
        a = (1.0 if k == "coulomb" else torch.sin(WAVE_K * r)) / r
        a[zero] = 0.0 if k == "coulomb" else 1.0
        return a
    a[zero] = 1.0 + spec["noise"]
    return a


def _exact_product(spec, X):
    x = torch.from_numpy(spec["x"]).to(DEV)
    n = spec["n"]
    B = torch.empty(X.shape[0], n, dtype=torch.float64, device=DEV)
    step = max(1, min(n, (1 << 26) // n))
    for r0 in range(0, n, step):
        r1 = min(n, r0 + step)
        B[:, r0:r1] = X @ _rows(spec, x, r0, r1).T
    return B


def exact(case, seed):
    op = case["op"]
    if op == "error":
        return None     # the error of one particular approximation
    if op == "batch":
        return {"B": [_exact_product(sp, _vectors(
            sp["n"], case["nrhs"], seed * 1000 + p).to(DEV))
            for p, sp in enumerate(_batch_specs(case, seed))]}
    spec = _spec(case, seed)
    X = _vectors(case["n"], case["nrhs"], seed).to(DEV)
    if op == "cg":
        A = _rows(spec, torch.from_numpy(spec["x"]).to(DEV), 0, case["n"])
        return {"X": torch.linalg.solve(A, X.T).T.contiguous()}
    B = _exact_product(spec, X)
    if op == "product":
        return B
    return {"B": B.cpu().numpy() if op == "dropin" else B}


def work(case):
    """One evaluation of every entry (about 25 operations), a rank-16
    sketch and projection of every block, each product's multiplications;
    points, vectors and products read or written once, the compressed
    matrix written by an approximation and read by a product."""
    op, rank = case["op"], 16.0
    if op == "batch":
        r = random.Random(case["mix"])
        total = {"bytes": 0.0, "flops": 0.0}
        for _ in range(case["problems"]):
            r.choice("abcde")
            n = _log(r, case["nmin"], case["nmax"])
            r.choice("abc")
            nb = 256 if n <= 2048 else 512 if n <= 8192 else 1024
            w = work(dict(op="approximate", n=n, nb=nb, ndim=3,
                          nrhs=case["nrhs"], symm=False))
            total = {k: total[k] + w[k] for k in total}
        return total
    n, nb, nrhs = float(case["n"]), float(case["nb"]), case.get("nrhs", 0)
    half = 0.5 if case["symm"] else 1.0
    nblk = n / nb
    matrix = 8.0 * half * n * (nb + 2.0 * rank * nblk)
    product = 2.0 * n * nrhs * (nb + 2.0 * rank * nblk)
    vectors = 16.0 * n * nrhs
    entries = half * n * n
    if op == "product":
        return {"bytes": matrix + vectors, "flops": product}
    if op == "cg":
        its = 300
        return {"bytes": its * matrix + vectors, "flops": its * product}
    points = 8.0 * n * case["ndim"]
    if op == "error":
        return {"bytes": matrix + points, "flops": entries * (25 + 2 * rank)}
    return {"bytes": points + matrix + vectors,
            "flops": entries * (25 + 4 * rank) + product}
