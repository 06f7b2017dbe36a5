"""Kernels and dispatch rules at the sizes where they change: basis sizes of
the small SVD's ranges, few and many tiles (thread-block clusters or one CTA
per tile), one or two lanes, few and many right-hand sides.  The matrices come
from the library's own constructors; the checks are against numpy on the same
blocks or factors, and bit for bit between two routes that keep one summation
order."""
import ctypes
from ctypes import POINTER, byref, c_double, c_int, c_void_p

import numpy as np
import pytest

import oracle
import starsh_b200 as sb
from harness import approximate_b200, as_ref_blrm

pytestmark = pytest.mark.gpu


class ExpProblem:
    """exp(-r / beta) (plus a nugget) on uniform points of the unit square, in
    the order they were drawn: every block has about the same rank."""

    def __init__(self, lib, n, nb, beta, symm=b"N", noise=0.0, seed=0):
        self.lib, self.beta, self.noise = lib, beta, noise
        self.x = np.random.default_rng(seed).uniform(0.0, 1.0, (2, n))
        libc = ctypes.CDLL("libc.so.6")
        libc.malloc.restype = c_void_p
        p = libc.malloc(ctypes.c_size_t(self.x.nbytes))
        ctypes.memmove(p, self.x.ctypes.data, self.x.nbytes)
        self.data, kern = POINTER(sb.SSData)(), c_void_p()
        assert lib.starsh_ssdata_init(byref(self.data), n, 2,
                                      ctypes.cast(p, POINTER(c_double)), beta,
                                      0.5, noise, 1.0) == 0
        assert lib.starsh_ssdata_get_kernel(byref(kern), self.data, sb.EXP) == 0
        self.P, self.C, self.F = POINTER(sb.Problem)(), POINTER(sb.Cluster)(), POINTER(sb.Blrf)()
        assert lib.starsh_problem_new(byref(self.P), 2, (sb.STARSH_int * 2)(n, n),
                                      symm, b"d", self.data, self.data, kern,
                                      b"edges") == 0
        assert lib.starsh_cluster_new_plain(byref(self.C), self.data, n, nb) == 0
        assert lib.starsh_blrf_new_tlr(byref(self.F), self.P, symm, self.C, self.C) == 0

    def block(self, i, j):
        R = self.C.contents
        a = self.x[:, R.start[i]:R.start[i] + R.size[i]]
        b = self.x[:, R.start[j]:R.start[j] + R.size[j]]
        r = np.hypot(a[0][:, None] - b[0], a[1][:, None] - b[1])
        return np.exp(-r / self.beta) + (self.noise * (r == 0.0))


def factors(M):
    c = oracle.blrm_contents(as_ref_blrm(M))
    return c, [c["far"], c["near"], c["ranks"]] + c["U"] + c["V"]


def product(lib, M, A, alpha=1.0, beta=0.0, B=None):
    A = np.asfortranarray(A)
    B = np.zeros_like(A) if B is None else np.asfortranarray(B).copy(order="F")
    n, nrhs = A.shape
    pd = POINTER(c_double)
    assert lib.starsh_blrm__dmml_b200(M, nrhs, alpha, A.ctypes.data_as(pd), n, beta,
                                      B.ctypes.data_as(pd), n) == 0
    return B


# (n, nb, beta, tol, maxrank): ranks from about 6 to 280, odd block sizes; 100
# blocks (more than the 74 up to which the large pivoted Cholesky takes a
# cluster per tile) or 9
CASES = [(1010, 101, 0.5, 1e-1, 50), (1300, 130, 0.5, 3e-2, 64),
         (1985, 199, 0.5, 1e-2, 99), (2570, 257, 0.5, 3e-3, 128),
         (3000, 300, 0.5, 2e-3, 150), (3100, 310, 0.5, 1e-3, 290),
         (1560, 520, 0.5, 4e-4, 500)]


@pytest.mark.parametrize("engine", [sb.ENGINE_MIXED, sb.ENGINE_FP64])
@pytest.mark.parametrize("n,nb,beta,tol,maxrank", CASES)
def test_blocks_within_tol_and_independent_of_batches(lib, monkeypatch, engine, n, nb,
                                                      beta, tol, maxrank):
    """Every far block is within tol (the adaptive engine counts all of the
    energy it leaves out; the fixed-width sketch of k + 10 columns can miss a
    part, in expectation at most sqrt(1 + k / 9) of the cut, below 6), and
    batches of a few tiles, on one lane or two, give the same bits as one
    batch of all."""
    pr = ExpProblem(lib, n, nb, beta)
    M = approximate_b200(lib, pr.F, maxrank, tol, engine=engine)
    c, want = factors(M)
    slack = 1.0 if engine == sb.ENGINE_MIXED else 6.0
    for b, (i, j) in enumerate(c["far"]):
        D = pr.block(i, j)
        err = np.linalg.norm(D - c["U"][b] @ c["V"][b].T)
        assert err <= (slack * tol * (1 + 1e-9) + 1e-12) * np.linalg.norm(D)
    for b, (i, j) in enumerate(c["near"]):
        D = pr.block(i, j)
        assert np.max(np.abs(c["D"][b] - D)) <= 1e-13
    lib.starsh_blrm_free(M)
    for lanes, mb in (("1", "40"), ("2", "80")):
        monkeypatch.setenv("STARSH_B200_LANES", lanes)
        monkeypatch.setenv("STARSH_B200_WORKSPACE_MB", mb)
        M = approximate_b200(lib, pr.F, maxrank, tol, engine=engine)
        assert sb.stats(lib).batches > 1
        got = factors(M)[1]
        assert len(got) == len(want)
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b)
        lib.starsh_blrm_free(M)


@pytest.mark.parametrize("symm,onfly", [(b"N", 0), (b"S", 0), (b"N", 1), (b"S", 1)])
@pytest.mark.parametrize("n,nb", [(520, 65), (1033, 129), (2113, 264)])
def test_products_of_any_number_of_columns(lib, n, nb, symm, onfly):
    """A column's bits do not depend on how many are multiplied together (the
    one-thread chains of up to four, the tensor tiles of more), and agree
    with numpy on the same factors (sums of n terms in another order)."""
    pr = ExpProblem(lib, n, nb, 0.5, symm=symm)
    M = approximate_b200(lib, pr.F, nb // 2, 1e-2, onfly=onfly)
    c, _ = factors(M)
    rng = np.random.default_rng(n)
    A, B0 = rng.standard_normal((n, 70)), rng.standard_normal((n, 70))
    for alpha, beta in ((1.0, 0.0), (-0.5, 2.0)):
        full = product(lib, M, A, alpha, beta, B0)
        want = oracle.dmml(c, pr.block, A, alpha, beta, B0)
        assert np.max(np.abs(full - want)) <= 1e-12 * np.max(np.abs(want))
        for nrhs in (1, 2, 3, 4, 5, 16, 17, 33, 64):
            got = product(lib, M, A[:, :nrhs], alpha, beta, B0[:, :nrhs])
            np.testing.assert_array_equal(got, full[:, :nrhs])
    lib.starsh_blrm_free(M)


@pytest.mark.parametrize("symm,onfly", [(b"N", 0), (b"S", 1)])
@pytest.mark.parametrize("n,nb", [(520, 65), (1033, 129), (2113, 264)])
def test_error_of_ragged_blocks(lib, n, nb, symm, onfly):
    """The error's terms are differences of about 1e-2 of entries rounded at
    1e-16: 1e-11 relative."""
    pr = ExpProblem(lib, n, nb, 0.5, symm=symm)
    M = approximate_b200(lib, pr.F, nb // 2, 1e-2, onfly=onfly)
    want = oracle.dfe(factors(M)[0], pr.block)
    assert want > 1e-4
    assert abs(lib.starsh_blrm__dfe_b200(M) - want) <= 1e-11 * want
    lib.starsh_blrm_free(M)


@pytest.mark.parametrize("n,nb,nrhs", [(517, 65, 1), (1033, 129, 3), (1985, 199, 5)])
def test_cg_of_ragged_sizes(lib, n, nb, nrhs):
    """Solutions meet the tolerance in the same TLR system (numpy's product;
    1.5: the recurrence's residual and the true one part by rounding)."""
    pr = ExpProblem(lib, n, nb, 0.5, symm=b"S", noise=float(n) / 20)
    M = approximate_b200(lib, pr.F, nb // 2, 1e-2)
    c, _ = factors(M)
    B = np.asfortranarray(np.random.default_rng(n).standard_normal((n, nrhs)))
    X = np.zeros_like(B)
    tol = 1e-9
    it = lib.starsh_itersolvers__dcg_b200(M, nrhs, B.ctypes.data, n, X.ctypes.data, n,
                                          tol, None)
    assert 0 < it < n, lib.starsh_b200_last_error()
    R = B - oracle.dmml(c, pr.block, X)
    for j in range(nrhs):
        assert np.linalg.norm(R[:, j]) <= 1.5 * tol * np.linalg.norm(B[:, j])
    lib.starsh_blrm_free(M)
