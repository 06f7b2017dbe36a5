"""What several host threads share when they launch kernels: the lanes of one
call, the serving workers."""
import ctypes
import json
import os
import re
import subprocess
import sys
from ctypes import POINTER, c_double, c_int

import numpy as np
import pytest

import starsh_b200 as sb
from test_gpu_edges import ExpProblem

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "stars-h_b200", "csrc")


def source(name):
    """A source file without its comments."""
    with open(os.path.join(CSRC, name)) as f:
        text = re.sub(r"/\*.*?\*/", "", f.read(), flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


# A stand-in for the CUDA runtime's three calls: `limit` is the device-wide
# limit of each function, `sets` counts the calls that set it.
LIMIT_CHECK = r"""
#include <cstdio>
#include <map>
#include <mutex>
#include <thread>
#include <vector>
#include "smem_limit.cuh"
static thread_local int current = 0;
static std::mutex mu;
static std::map<std::pair<int, const void *>, int> limit;
static int sets = 0, refuse = 0;
extern "C" cudaError_t cudaGetDevice(int *d) { *d = current; return cudaSuccess; }
extern "C" cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 7; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute, int v)
{
    std::lock_guard<std::mutex> g(mu);
    ++sets;
    if (refuse) { --refuse; return cudaErrorInvalidValue; }
    limit[{current, f}] = v;
    return cudaSuccess;
}
static void a(int) {}
static void b(int) {}
#define CHECK(x) if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; }
int main()
{
    refuse = 1;                         // a refused setting is tried again
    CHECK((b200::allow_smem<a, 1000>() == cudaErrorInvalidValue));
    CHECK((b200::allow_smem<a, 1000>() == cudaSuccess));
    CHECK(sets == 2);
    std::vector<std::thread> th;        // threads on three devices
    for (int t = 0; t < 12; ++t)
        th.emplace_back([t] {
            current = t % 3;
            for (int q = 0; q < 1000; ++q) {
                b200::allow_smem<a, 1000>();
                b200::allow_smem<b, 2000>();
            }
        });
    for (auto &x : th) x.join();
    CHECK(limit.size() == 6);
    for (auto &x : limit) CHECK(x.second == (x.first.second == (const void *)a ? 1000 : 2000));
    CHECK(sets <= 2 + 2 * 12);          // not once a call
    current = 70;                       // beyond the devices remembered
    const int before = sets;
    b200::allow_smem<a, 1000>();
    b200::allow_smem<a, 1000>();
    CHECK(sets == before + 2);
    CHECK(b200::sm_count() == 7);
    return 0;
}
"""


def test_limit_is_one_number_per_kernel_and_device(tmp_path):
    src, exe = tmp_path / "limit.cpp", tmp_path / "limit"
    src.write_text(LIMIT_CHECK)
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", CSRC, "-I",
                    "/usr/local/cuda/include", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.parametrize("name", ["rsvd_kernels.cu", "sketch_i8.cu", "gen_sketch_i8.cu",
                                  "proj_i8.cu"])
def test_engine_kernels_take_their_limit_once(name):
    """No launch of the kernels that lanes and workers share sets a limit of
    its own, and no plain static is filled in by whichever thread is first."""
    text = source(name)
    assert "allow_smem<" in text
    assert "cudaFuncSetAttribute" not in text
    assert not re.search(r"static int sms = 0|static PFN\w+ encode", text)


@pytest.mark.parametrize("name", ["gemm_f64.cu", "dmml_dfe.cu"])
def test_limits_hold_on_every_device(name):
    """A limit is a device's: set once a process, a kernel that asks for more
    than 48 KB could run on the first device alone (the entry without
    allocations runs on whichever device is current)."""
    text = source(name)
    assert "allow_smem<" in text
    assert "cudaFuncSetAttribute" not in text and "once_flag" not in text


@pytest.mark.parametrize("name", ["engine.cu", "noalloc.cu"])
def test_a_refused_launch_is_reported_as_what_it_was(name):
    """gemm_f64_batched returns the launch error and thereby clears it: asked
    for once more, the runtime knows of none ("no error").  The small SVD's
    launches are looked at before the next product's."""
    text = source(name)
    calls = re.findall(r"gemm_f64_batched\(ta.*?;\s*return[^;]*;", text, flags=re.S)
    assert calls and all("cudaGetLastError" not in c and "cuda_fail(e," in c for c in calls)
    for m in re.finditer(r"launch_small_svd\(", text):
        after = text[m.end():m.end() + 500]
        assert 0 <= after.find("cudaGetLastError()") < after.find("gemm(STEP_ROTATE")


def test_roles_of_a_cta_meet_at_a_named_barrier():
    """k_gemv_b's copying and summing warps each run their own loop: they meet
    at a barrier that counts arrivals (both sides, all of the CTA's threads),
    not at two different __syncthreads()."""
    text = source("dmml_dfe.cu")
    body = text[text.index("k_gemv_b("):]
    body = body[:body.index("static void launch_gemv")]
    assert "__syncthreads" not in body and body.count("gvb_sync();") == 2
    assert re.search(r'"barrier\.sync\.aligned 1, %0;" ::"n"\(kGvThreadsB\) : "memory"', text)
    assert re.search(r"__launch_bounds__\(kGvThreadsB\)\s*k_gemv_b\(", text)
    assert re.search(r"k_gemv_b<NR><<<dim3\([^;]*?\), kGvThreadsB,", text)


@pytest.mark.gpu
def test_phase_times_of_the_benchmark_do_not_overlap(lib):
    """The benchmark's phases, and the kernels' rates that follow from them,
    are of a call whose phases run one after another: together they take no
    longer than the call."""
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--workload",
                        "c1-exp", "--steps", "2", "--warmup", "1", "--no-cpu"],
                       capture_output=True, text=True, cwd=ROOT,
                       env=dict(os.environ, STARSH_B200_WORKSPACE_MB="40"))
    assert r.returncode == 0, r.stderr[-2000:]
    line = [json.loads(x) for x in r.stdout.splitlines() if x.startswith("{")][0]
    ph = line["phases_ms"]
    together = sum(ph[k] for k in ("generation", "basis", "project", "svd", "output"))
    assert 0 < together <= ph["total_host"], ph


# The device memory a process holds after a one-lane call that fills the
# workspace and a two-lane call after it.
HELD = r"""
import ctypes, sys
sys.path[:0] = %r
import starsh_b200 as sb
import test_concurrency as tc
from harness import approximate_b200
from test_gpu_edges import ExpProblem
lib = sb.load()
assert lib.starsh_b200_set_device(0) == 0
cu = ctypes.CDLL("libcuda.so.1")
def used():
    pool, v = ctypes.c_void_p(), ctypes.c_uint64()
    assert cu.cuDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    assert cu.cuMemPoolGetAttribute(pool, 7, ctypes.byref(v)) == 0   # used now
    return v.value / 2.0**20
pr = ExpProblem(lib, 4000, 500, 0.5)
lib.starsh_blrm_free(approximate_b200(lib, pr.F, 180, 1e-1, engine=sb.ENGINE_FP64, flags=0))
assert sb.stats(lib).batches > 1
one = used()
for M in tc.batch(lib, [ExpProblem(lib, 4000, 500, 0.5, seed=1)], [1e-1], 180):
    lib.starsh_blrm_free(M)
assert sb.stats(lib).batches > 1
print("held", one, used())
"""


@pytest.mark.gpu
def test_lanes_share_the_workspace(lib):
    """400 MB for a call's batches in flight are 400 MB whichever lanes the
    calls took (and a few MB of sketch matrices and tile records)."""
    code = HELD % [os.path.join(ROOT, d) for d in ("stars-h_b200", "oracle", "tests")]
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True,
                       env=dict(os.environ, STARSH_B200_WORKSPACE_MB="400"))
    assert r.returncode == 0, r.stderr[-2000:]
    line = [x for x in r.stdout.splitlines() if x.startswith("held")][0].split()
    one, two = float(line[1]), float(line[2])
    assert 350 < one < 440 and two < 440, line


# Two lanes, then the same call where the system refuses every new thread (a
# default stack larger than the address space).
NO_THREAD = r"""
import ctypes, sys
sys.path[:0] = %r
import numpy as np
import starsh_b200 as sb
import test_concurrency as tc
from test_gpu_edges import ExpProblem
lib = sb.load()
assert lib.starsh_b200_set_device(0) == 0
probs = [ExpProblem(lib, 2000, 200, 0.5, seed=s) for s in range(2)]
def call():
    M = tc.batch(lib, probs, [5e-2, 1.1e-2], 180)
    assert sb.stats(lib).batches > 4
    return np.concatenate(tc.ranks(M))
want = call()
libc = ctypes.CDLL(None)
attr = ctypes.create_string_buffer(256)
assert libc.pthread_attr_init(attr) == 0
assert libc.pthread_attr_setstacksize(attr, ctypes.c_size_t(1 << 47)) == 0
assert libc.pthread_setattr_default_np(attr) == 0
np.testing.assert_array_equal(call(), want)
print("done")
"""


@pytest.mark.gpu
def test_one_lane_where_no_thread_can_be_had(lib):
    code = NO_THREAD % [os.path.join(ROOT, d) for d in ("stars-h_b200", "oracle", "tests")]
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True,
                       env=dict(os.environ, STARSH_B200_WORKSPACE_MB="80"))
    assert r.returncode == 0 and "done" in r.stdout, r.stderr[-2000:]


def batch(lib, probs, tols, maxrank):
    k = len(probs)
    lib.starsh_set_oversample(b"10")
    formats = (POINTER(sb.Blrf) * k)()
    for p, pr in enumerate(probs):
        F = POINTER(sb.Blrf)()
        assert lib.starsh_blrf_new_tlr(ctypes.byref(F), pr.P, b"N", pr.C, pr.C) == 0
        formats[p] = F
    M = (POINTER(sb.Blrm) * k)()
    info = lib.starsh_b200_approximate_batch(k, M, formats, (c_int * k)(*[maxrank] * k),
                                             (c_double * k)(*tols), None, sb.ENGINE_MIXED, 0)
    assert info == 0, (info, lib.starsh_b200_last_error())
    return M


def ranks(M):
    return [np.ctypeslib.as_array(m.contents.far_rank,
                                  shape=(m.contents.format.contents.nblocks_far,)).copy()
            for m in M]


@pytest.mark.gpu
def test_lanes_with_different_basis_sizes(lib, monkeypatch):
    """Two lanes whose batches hold bases of every range of 65 .. 160 rows
    (kernels that share a function and differ in their shared memory) succeed
    call after call, with the same ranks."""
    tols = [7e-2, 5e-2, 3e-2, 1.8e-2, 1.1e-2]     # bases of about 75 to 135
    probs = [ExpProblem(lib, 2000, 200, 0.5, seed=s) for s in range(len(tols))]
    monkeypatch.setenv("STARSH_B200_WORKSPACE_MB", "80")
    want = None
    for _ in range(40):
        M = batch(lib, probs, tols, 180)
        assert sb.stats(lib).batches > 10
        got = ranks(M)
        want = want or got
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b)
        for m in M:
            lib.starsh_blrm_free(m)
