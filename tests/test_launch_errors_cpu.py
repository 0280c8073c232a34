"""The host side without a GPU: the library's own object files against a stand-in for the CUDA runtime that
counts launches, fails the one it is told to, and writes down what reaches which stream. Work that was forked to the
handle's second stream is joined again whatever fails after it; a failed tuning run changes nothing; only chunks whose
matrices share the L2 cache are solved in turn."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "tokura_zgeev_batched_gb300")

# The host side that nvcc generates calls the functions with two underscores.
RUNTIME = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>
#include <cuda_runtime.h>
int launches = 0, fail_at = -1;
cudaError_t last = cudaSuccess;
std::string events;
static void note(const char* what, cudaStream_t s) {
  events += what;
  events += s == (cudaStream_t)2 ? "2 " : "1 ";
}
static std::vector<std::pair<dim3, std::pair<dim3, std::pair<size_t, cudaStream_t>>>> pushed;
extern "C" {
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) { *k = (cudaKernel_t)f; return cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, cudaStream_t s) {
  pushed.push_back({g, {b, {m, s}}});
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* m, void* s) {
  *g = pushed.back().first;
  *b = pushed.back().second.first;
  *m = pushed.back().second.second.first;
  *(cudaStream_t*)s = pushed.back().second.second.second;
  pushed.pop_back();
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t s) {
  if (launches++ == fail_at) {
    note("failed", s);
    return last = cudaErrorInvalidValue;
  }
  note("launch", s);
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  note(e == (cudaEvent_t)11 ? "fork" : "join", s);
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  note(e == (cudaEvent_t)11 ? "afterfork" : "afterjoin", s);
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* b, const void*, int, size_t, unsigned) {
  *b = 4;
  return cudaSuccess;
}
}
"""

VECTORS = RUNTIME + r"""
#include <mutex>
#include "zgeev_internal.h"
namespace tzg {
size_t backward_workspace_bytes(int n, int batch) { return 64ull * n * n * batch; }
}
int main(int argc, char** argv) {
  fail_at = std::atoi(argv[1]);
  std::mutex mu;
  tzg::ForkJoin fj;
  fj.aux = (cudaStream_t)2;
  fj.fork = (cudaEvent_t)11;
  fj.join = (cudaEvent_t)12;
  fj.mu = &mu;
  double2* p = (double2*)4096;  // never read
  const cudaError_t e = tzg::launch_vectors(4, std::atoi(argv[2]), 100, p, p, p, p, p, (char*)p, 300, (cudaStream_t)1,
                                            true, &fj, 65, true);
  std::printf("%d %s\n", (int)e, events.c_str());
}
"""

TUNER = RUNTIME + r"""
#include "tokura_handle.h"
#include "tokura_blas_ext.h"
static int calls = 0;
static cudaError_t timed() { return calls++ == fail_at ? cudaErrorUnknown : cudaSuccess; }
namespace tzg {
cudaError_t launch_plain(const PlainConfig&, int, int, const double2*, double2*, double2*, char*, int, cudaStream_t, int,
                         bool, const ForkJoin*) {
  return timed();
}
cudaError_t launch_ragged(int, int, int, const int*, const long long*, const long long*, long long, const double2*,
                          double2*, void*, char*, int, cudaStream_t, int, int, const ForkJoin*, int, bool) {
  return timed();
}
size_t ragged_workspace_bytes(int, long long) { return 256; }
}
extern "C" {
cudaError_t cudaMalloc(void** p, size_t) { *p = (void*)4096; return cudaSuccess; }
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)12; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 100.0f - calls; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp*, int) { return cudaErrorUnknown; }
}
int main(int argc, char** argv) {
  fail_at = std::atoi(argv[1]);
  tokurablas_t h;
  h.sm_count = 152;
  h.plain[20] = tzg::PlainConfig{4, 64};
  h.ragged_lanes = 2;
  const int st = argv[2][0] == 'p' ? tokuraAutotune(&h, 20, 20, 100, 0) : tokuraAutotuneRagged(&h, 100, 2, 20, 0);
  std::printf("%d %d %d %d %d\n", st, calls, h.plain[20].lanes, h.plain[20].threads, h.ragged_lanes);
}
"""

HOST = RUNTIME + r"""
#include "tokura_handle.h"
#include "tokura_blas_ext.h"
static long waits = 0, solves = 0;
namespace tzg {
cudaError_t launch_plain(const PlainConfig&, int, int, const double2*, double2*, double2*, char*, int, cudaStream_t, int,
                         bool, const ForkJoin*) {
  ++solves;
  return cudaSuccess;
}
}
extern "C" {
static size_t next = 1000;
cudaError_t cudaMalloc(void** p, size_t) { *p = (void*)4096; return cudaSuccess; }
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)next++; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)next++; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
}
int main(int argc, char** argv) {
  static tokurablas_t h;
  h.sm_count = 152;
  cuDoubleComplex* p = (cuDoubleComplex*)4096;
  const int st = tokura_zgeev_batched_host(&h, std::atoi(argv[1]), std::atoi(argv[2]), p, p, (char*)p, std::atoi(argv[3]));
  for (size_t at = 0; (at = events.find("afterjoin", at)) != std::string::npos; ++at) ++waits;
  std::printf("%d %ld %ld\n", st, solves, waits);
}
"""


def linked(source, name, directory):
    """`source` with the library's object file of that translation unit."""
    sys.path.insert(0, ROOT)
    from tokura_zgeev_batched_gb300 import build

    build.build()
    obj = os.path.join(PKG, "_build", name + ".o")
    if not os.path.exists(obj):
        build.build(force=True)
    (directory / "main.cpp").write_text(source)
    include = os.path.join(os.path.dirname(os.path.dirname(build._nvcc())), "include")
    exe = str(directory / "main")
    subprocess.check_call(["g++", "-std=c++17", "-I", include, "-I", os.path.join(PKG, "csrc"), "-I",
                           os.path.join(ROOT, "include"), str(directory / "main.cpp"), obj, "-o", exe, "-pthread"])
    return exe


@pytest.fixture(scope="module")
def vectors(tmp_path_factory):
    exe = linked(VECTORS, "zgeev_vectors.cu", tmp_path_factory.mktemp("vectors"))

    def run(fail_at, n):
        out = subprocess.run([exe, str(fail_at), str(n)], capture_output=True, text=True, timeout=60, check=True).stdout
        err, *events = out.split()
        return int(err), events
    return run


@pytest.mark.parametrize("n", [12, 24, 40])
def test_vectors_join_the_second_stream_after_a_failed_launch(vectors, n):
    err, events = vectors(-1, n)
    assert err == 0 and events.count("afterjoin1") == 1
    launches = sum(e.startswith("launch") for e in events)
    assert launches >= 4
    for k in range(launches):
        err, events = vectors(k, n)
        assert err == 1, (k, events)
        assert sum(e.startswith("failed") for e in events) == 1
        fork, join, wait = (events.index(e) if e in events else -1 for e in ("afterfork2", "join2", "afterjoin1"))
        assert fork >= 0 and fork < join < wait, (k, events)
        assert not any(e.endswith("2") for e in events[join + 1:]), (k, events)


@pytest.fixture(scope="module")
def tuner(tmp_path_factory):
    exe = linked(TUNER, "tokura_tuner.cu", tmp_path_factory.mktemp("tuner"))

    def run(fail_at, kind):
        out = subprocess.run([exe, str(fail_at), kind], capture_output=True, text=True, timeout=60, check=True).stdout
        return [int(v) for v in out.split()]
    return run


@pytest.mark.parametrize("kind", ["plain", "ragged"])
def test_a_failed_tuning_run_leaves_the_handle_as_it_was(tuner, kind):
    st, calls, *_ = tuner(-1, kind)
    assert st == 0 and calls > 10
    for k in range(calls):
        st, _, lanes, threads, ragged = tuner(k, kind)
        assert st == 1 and (lanes, threads, ragged) == (4, 64, 2), k


@pytest.mark.parametrize("n,batch,chunk,in_turn", [(4, 1048576, 4096, False), (4, 30000, 0, False), (32, 65536, 8192, False),
                                                   (33, 65536, 8192, True), (64, 65536, 0, True), (64, 30000, 2000, False)])
def test_chunks_solved_in_turn(tmp_path, n, batch, chunk, in_turn):
    exe = linked(HOST, "tokura_host_pipeline.cpp", tmp_path)
    out = subprocess.run([exe, str(n), str(batch), str(chunk)], capture_output=True, text=True, timeout=60, check=True)
    st, solves, waits = (int(v) for v in out.stdout.split())
    assert st == 0 and solves >= 5
    # each chunk's copy waits for the one before; in turn, its solve does too
    assert waits == (2 if in_turn else 1) * (solves - 1)
