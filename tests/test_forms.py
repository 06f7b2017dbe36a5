"""Forms of the error check and of the product that the square, two-dimensional
exponential problems do not reach: every kernel family, dimensions beyond the
staged ones, point-major coordinates, formats with an empty block row, calls
from several host threads.  The oracle is numpy on the same points."""
import ctypes
import threading
from ctypes import POINTER, byref, c_double, c_void_p

import numpy as np
import pytest

import oracle
import starsh_b200 as sb
from harness import approximate_b200
from test_gpu_edges import CASES, ExpProblem, factors, product

pytestmark = pytest.mark.gpu


def _malloc(values):
    """A libc copy (the library frees the coordinates and lists it owns)."""
    values = np.ascontiguousarray(values)
    libc = ctypes.CDLL("libc.so.6")
    libc.malloc.restype = c_void_p
    p = libc.malloc(ctypes.c_size_t(max(1, values.nbytes)))
    ctypes.memmove(p, values.ctypes.data, values.nbytes)
    return ctypes.cast(p, POINTER(c_double if values.dtype == np.float64 else sb.STARSH_int))


# entries from the distances; each with the library's constructor
def _spatial(ktype, nu=0.5):
    def make(lib, x):
        d, k = POINTER(sb.SSData)(), c_void_p()
        assert lib.starsh_ssdata_init(byref(d), x.shape[1], x.shape[0], _malloc(x), 0.4, nu,
                                      0.0, 1.0) == 0
        assert lib.starsh_ssdata_get_kernel(byref(k), d, ktype) == 0
        return d, k
    return make


def _coulomb(lib, x):
    d, k = POINTER(sb.Particles)(), c_void_p()
    assert lib.starsh_esdata_init(byref(d), x.shape[1], x.shape[0], _malloc(x)) == 0
    assert lib.starsh_esdata_get_kernel(byref(k), d, 1) == 0
    return d, k


def _wave(ktype):
    def make(lib, x):
        d, k = POINTER(sb.EDData)(), c_void_p()
        assert lib.starsh_eddata_init(byref(d), x.shape[1], x.shape[0], _malloc(x), 5.0,
                                      1.0) == 0
        assert lib.starsh_eddata_get_kernel(byref(k), d, ktype) == 0
        return d, k
    return make


def _rbf(lib, x):
    d = POINTER(sb.MDData)()
    assert lib.starsh_mddata_init(byref(d), x.shape[1], _malloc(x.T), 3, 1, 0, 0.0, 0.7,
                                  1.0) == 0
    return d, c_void_p(sb.kernel_symbol(lib, "starsh_generate_3d_cube"))


def _inverse(r, zero):
    with np.errstate(divide="ignore", invalid="ignore"):
        return np.where(r == 0.0, zero, 1.0 / r)


FAMILIES = {
    "exp-1d": (1, _spatial(1), lambda r: np.exp(-r / 0.4)),
    "exp-5d": (5, _spatial(1), lambda r: np.exp(-r / 0.4)),
    "sqexp-3d": (3, _spatial(2), lambda r: np.exp(-r * r / (2 * 0.4 ** 2))),
    "sqexp-4d": (4, _spatial(2), lambda r: np.exp(-r * r / (2 * 0.4 ** 2))),
    "matern-half-2d": (2, _spatial(3, 1.5), lambda r: oracle.matern(r, 1.0, 0.4, 1.5)),
    "matern-2d": (2, _spatial(3, 0.7), lambda r: oracle.matern(r, 1.0, 0.4, 0.7)),
    "matern2-3d": (3, _spatial(4, 0.7),
                   lambda r: oracle.matern(r, 1.0, 0.4, 0.7, sqrt2nu=False)),
    "coulomb-3d": (3, _coulomb, lambda r: _inverse(r, 0.0)),
    "sin-3d": (3, _wave(1), lambda r: np.where(r == 0.0, 1.0, np.sin(5 * r) * _inverse(r, 0.0))),
    "cos-3d": (3, _wave(2), lambda r: np.where(r == 0.0, 1.0, np.cos(5 * r) * _inverse(r, 0.0))),
    "rbf-3d": (3, _rbf, lambda r: 1.0 / np.sqrt(1.0 + (r / 0.7) ** 2)),
}


class Problem:
    """Points along a line of boxes (the blocks differ in rank), TLR blocks of
    nb, or the far and near blocks given."""

    def __init__(self, lib, family, n, nb, symm=b"N", far=None, near=None):
        ndim, make, self.entries = FAMILIES[family]
        rng = np.random.default_rng(n)
        self.x = rng.uniform(0.0, 1.0, (ndim, n))
        self.x[0] = np.sort(3.0 * self.x[0])
        self.data, kern = make(lib, self.x)
        self.P, self.C, self.F = POINTER(sb.Problem)(), POINTER(sb.Cluster)(), POINTER(sb.Blrf)()
        assert lib.starsh_problem_new(byref(self.P), 2, (sb.STARSH_int * 2)(n, n), symm, b"d",
                                      self.data, self.data, kern, b"forms") == 0
        assert lib.starsh_cluster_new_plain(byref(self.C), self.data, n, nb) == 0
        if far is None:
            assert lib.starsh_blrf_new_tlr(byref(self.F), self.P, symm, self.C, self.C) == 0
        else:
            lists = [_malloc(np.array(b, np.int64).reshape(-1, 2)) for b in (far, near)]
            assert lib.starsh_blrf_new_from_coo(byref(self.F), self.P, symm, self.C, self.C,
                                                len(far), lists[0], len(near), lists[1],
                                                1) == 0

    def block(self, i, j):
        R = self.C.contents
        a = self.x[:, R.start[i]:R.start[i] + R.size[i]]
        b = self.x[:, R.start[j]:R.start[j] + R.size[j]]
        r2 = np.zeros((a.shape[1], b.shape[1]))
        for d in range(a.shape[0]):
            r2 += (a[d][:, None] - b[d]) ** 2
        return self.entries(np.sqrt(r2))


@pytest.mark.parametrize("family", sorted(FAMILIES))
def test_error_of_every_family(lib, family):
    """Entries agree with numpy's to 1e-13, so the relative error, whose change
    is at most ||change of D|| / ||D||, does to 2e-13 with its own rounding."""
    pr = Problem(lib, family, 1033, 129)
    M = approximate_b200(lib, pr.F, 60, 1e-2)
    c, _ = factors(M)
    assert len(c["far"]) > 0
    want = oracle.dfe(c, pr.block)
    assert 0.0 < want <= 1e-2
    assert abs(lib.starsh_blrm__dfe_b200(M) - want) <= 2e-13
    lib.starsh_blrm_free(M)


@pytest.mark.parametrize("n,nb", [(520, 65), (2113, 264)])
@pytest.mark.parametrize("nonear", [False, True])
def test_products_with_an_empty_block_row(lib, n, nb, nonear):
    """A block row without blocks gives beta B there, whichever kernels form
    the others; a column's bits do not depend on how many there are."""
    q = (n + nb - 1) // nb
    far = [(i, j) for i in range(q) for j in range(q)
           if i not in (2, q - 1) and abs(i - j) > 1]
    near = [] if nonear else [(i, i) for i in range(q) if i not in (2, q - 1)]
    pr = Problem(lib, "exp-1d", n, nb, far=far, near=near)
    M = approximate_b200(lib, pr.F, nb // 2, 1e-3)
    c, _ = factors(M)
    rng = np.random.default_rng(n)
    A, B0 = rng.standard_normal((n, 20)), rng.standard_normal((n, 20))
    for alpha, beta in ((1.0, 0.0), (-0.5, 2.0)):
        full = product(lib, M, A, alpha, beta, B0)
        want = oracle.dmml(c, pr.block, A, alpha, beta, B0)
        assert np.max(np.abs(full - want)) <= 1e-12 * max(1.0, np.max(np.abs(want)))
        np.testing.assert_array_equal(full[2 * nb:3 * nb], beta * B0[2 * nb:3 * nb])
        for nrhs in (1, 2, 3, 4, 5, 17):
            got = product(lib, M, A[:, :nrhs], alpha, beta, B0[:, :nrhs])
            np.testing.assert_array_equal(got, full[:, :nrhs])
    lib.starsh_blrm_free(M)


@pytest.mark.parametrize("n,nb,beta,tol,maxrank", CASES)
def test_fixed_width_blocks_against_the_svd(lib, n, nb, beta, tol, maxrank):
    """The fixed-width sketch of w = min(maxrank + 10, nb) columns against each
    block's own singular values: the error outside the sketched basis is, for
    every split w = k + p, at most (1 + e sqrt(3 k / (p + 1))) tail(k) + 5 e^2
    sqrt(w) / (p + 1) s_k+1 but for 2 exp(-p) + exp(-12) of the draws (Halko,
    Martinsson, Tropp 2011, theorem 10.7 with t = e, u = 5; p >= 10), the error
    inside at most tol."""
    pr = ExpProblem(lib, n, nb, beta)
    M = approximate_b200(lib, pr.F, maxrank, tol, engine=sb.ENGINE_FP64)
    c, _ = factors(M)
    for b, (i, j) in enumerate(c["far"]):
        D = pr.block(i, j)
        s = np.linalg.svd(D, compute_uv=False)
        tail = np.sqrt(np.append(np.cumsum(s[::-1] ** 2)[::-1], 0.0))
        nrm, w = tail[0], min(maxrank + 10, *D.shape)
        outside = 0.0
        if w < min(D.shape):
            outside = min((1 + np.e * np.sqrt(3 * k / (w - k + 1))) * tail[k] +
                          5 * np.e ** 2 * np.sqrt(w) / (w - k + 1) * s[k]
                          for k in range(0, w - 9))
        err = np.linalg.norm(D - c["U"][b] @ c["V"][b].T)
        assert err <= np.hypot(tol * nrm, outside) * (1 + 1e-9) + 1e-12 * nrm
    lib.starsh_blrm_free(M)


def test_calls_from_several_threads(lib):
    """Approximations, products and error checks called from four threads at
    once give what they give one after another."""
    probs = [ExpProblem(lib, 1300 + 65 * t, 130 + 13 * t, 0.5, seed=t) for t in range(4)]

    def work(t, out):
        pr = probs[t]
        for rep in range(5):
            F = POINTER(sb.Blrf)()
            assert lib.starsh_blrf_new_tlr(byref(F), pr.P, b"N", pr.C, pr.C) == 0
            M = approximate_b200(lib, F, 60 + 10 * t, 2e-2)
            x = np.random.default_rng(t).standard_normal((pr.x.shape[1], 1 + t))
            out.append((factors(M)[0]["ranks"].copy(), product(lib, M, x),
                        lib.starsh_blrm__dfe_b200(M)))
            lib.starsh_blrm_free(M)

    alone, together = [[] for _ in probs], [[] for _ in probs]
    for t in range(4):
        work(t, alone[t])
    threads = [threading.Thread(target=work, args=(t, together[t])) for t in range(4)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    for t in range(4):
        assert len(together[t]) == 5
        for a, b in zip(alone[t], together[t]):
            np.testing.assert_array_equal(a[0], b[0])
            np.testing.assert_array_equal(a[1], b[1])
            assert a[2] == b[2]
