"""The host path of an explicit handle against a stand-in for the CUDA runtime (host memory for
device memory, kernels that do nothing, a log of the calls): what a call has waited for when it
returns, which graphs are made when, and what the handle says after a launch that failed."""
import json
import os
import shutil
import subprocess
import sys

import pytest

from conftest import PKG

RUNTIME = r'''
#include <cuda_runtime_api.h>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>
static std::string calls;
static int fail_launch = -1, fail_make = 0, launched_kernels = 0, capturing = 0;
struct Graph { int kernels; };
static Graph* cap;
extern "C" {
const char* fake_log() { return calls.c_str(); }
void fake_clear() { calls.clear(); launched_kernels = 0; }
void fake_fail_launch(int k) { fail_launch = k; }      // the k-th graph launch from now on returns an error
void fake_fail_instantiate(int on) { fail_make = on; }
int fake_launched() { return launched_kernels; }       // kernels of the graphs launched
#define OK return cudaSuccess
void** __cudaRegisterFatBinary(void*) { static void* p; return &p; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* q) { *g = *b = dim3(1, 1, 1); *s = 0; *(void**)q = nullptr; OK; }
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void*) { *k = (cudaKernel_t)8; OK; }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t) {
    if (capturing) { cap->kernels++; OK; }
    calls += "kernel ";
    OK;
}
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; OK; }
cudaError_t cudaGetDevice(int* n) { *n = 0; OK; }
cudaError_t cudaSetDevice(int) { OK; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) { *v = a == cudaDevAttrMultiProcessorCount ? 152 : 0; OK; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) { std::memset(p, 0, sizeof *p); OK; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { OK; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { *n = 1; OK; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { static double b[64]; *p = b; OK; }
cudaError_t cudaGetLastError() { OK; }
cudaError_t cudaPeekAtLastError() { OK; }
const char* cudaGetErrorString(cudaError_t) { return "stand-in"; }
cudaError_t cudaMalloc(void** p, size_t n) { *p = std::calloc(n + 1, 1); OK; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = std::calloc(n + 1, 1); OK; }
cudaError_t cudaFree(void* p) { std::free(p); OK; }
cudaError_t cudaFreeHost(void* p) { std::free(p); OK; }
cudaError_t cudaMemGetInfo(size_t* a, size_t* b) { *a = *b = (size_t)1 << 36; OK; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); OK; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { if (!capturing) std::memcpy(d, s, n); OK; }
cudaError_t cudaMemset(void* d, int v, size_t n) { std::memset(d, v, n); OK; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { if (!capturing) std::memset(d, v, n); OK; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { std::memset(a, 0, sizeof *a); OK; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)16; OK; }
cudaError_t cudaStreamDestroy(cudaStream_t) { OK; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { calls += "wait-stream "; OK; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { capturing = 1; cap = new Graph{0}; OK; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { capturing = 0; *g = (cudaGraph_t)cap; OK; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete (Graph*)g; OK; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
    if (fail_make) { *e = nullptr; return cudaErrorMemoryAllocation; }
    *e = (cudaGraphExec_t) new Graph(*(Graph*)g);
    calls += "make" + std::to_string(((Graph*)g)->kernels) + " ";
    OK;
}
cudaError_t cudaGraphUpload(cudaGraphExec_t, cudaStream_t) { OK; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { delete (Graph*)e; OK; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
    if (fail_launch >= 0 && fail_launch-- == 0) return cudaErrorUnknown;
    launched_kernels += ((Graph*)e)->kernels;
    calls += "graph" + std::to_string(((Graph*)e)->kernels) + " ";
    OK;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)24; OK; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)24; OK; }
cudaError_t cudaEventDestroy(cudaEvent_t) { OK; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { calls += "event "; OK; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { calls += "wait-event "; OK; }
cudaError_t cudaEventElapsedTime(float* t, cudaEvent_t, cudaEvent_t) { *t = 1.0f; OK; }
}
'''

PROGRAM = r'''
import ctypes as C, json, os, sys, tempfile
sys.path.insert(0, sys.argv[1])
fake = C.CDLL(sys.argv[2])
fake.fake_log.restype = C.c_char_p
from cfd2d import capi, cases
capi.set_verbosity(0)
t, m, U0 = cases.vortex(4, flux="HLLC", recon="MINMOD", scheme="SSPRK3")
t.tau = 0.125
out = {}
def log():
    s = fake.fake_log().decode().split()
    fake.fake_clear()
    return s
with tempfile.TemporaryDirectory() as d:
    path = cases.write_task(t, m, d)
    h = capi.Solver(path, mesh=m)
    out["create"] = log()
    for reset in (0, 1):
        h.set_state(U0, reset_time_step=bool(reset))
        out["set_state%d" % reset] = log()
    def step(n):
        try:
            h.step(n)
            ok = True
        except capi.CfdError:
            ok = False
        i = h.get_info()
        r = dict(ok=ok, steps=i.step, time=i.time, kernels=fake.fake_launched())
        r["log"] = log()
        return r
    out["step7"] = step(7)
    other = capi.Solver(path, mesh=m)
    log()
    h, mine = other, h
    out["step9"] = [step(9), step(9)]
    h.close()
    log()
    h = mine
    out["step16"] = [step(16), step(16)]
    out["fail"] = []
    for k in (0, 1, 2, 3):
        fake.fake_fail_launch(k)
        out["fail"].append(step(21))
        fake.fake_fail_launch(-1)
    h.close()
    h = capi.Solver(path, mesh=m)
    log()
    fake.fake_fail_instantiate(1)
    out["no_graph"] = [step(16), step(16)]
print(json.dumps(out))
'''


@pytest.fixture(scope="module")
def seen(capi, tmp_path_factory):
    inc = next((p for p in ("/usr/local/cuda/include", os.path.join(os.environ.get("CUDA_HOME", ""), "include"))
                if os.path.exists(os.path.join(p, "cuda_runtime_api.h"))), None)
    if inc is None or shutil.which("g++") is None:
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("runtime")
    (d / "runtime.cpp").write_text(RUNTIME)
    (d / "program.py").write_text(PROGRAM)
    so = str(d / "runtime.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", inc, str(d / "runtime.cpp"), "-o", so], check=True)
    r = subprocess.run([sys.executable, str(d / "program.py"), PKG, so], capture_output=True, text=True,
                       env=dict(os.environ, LD_PRELOAD=so), timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    return json.loads(r.stdout.splitlines()[-1])


@pytest.mark.parametrize("call", ["set_state0", "set_state1"])
def test_set_state_returns_with_its_work_done(seen, call):
    log = seen[call]
    assert "kernel" in log
    last = len(log) - 1 - log[::-1].index("kernel")
    assert "wait-stream" in log[last:], log


def test_steps_and_time_are_those_launched_when_a_launch_fails(seen):
    per_step = seen["step7"]["kernels"] // 7
    before = seen["step16"][1]
    for r in seen["fail"]:
        assert not r["ok"]
        assert (r["steps"] - before["steps"]) * per_step == r["kernels"]
        assert r["time"] == 0.125 * r["steps"]
        before = r


def test_graph_of_many_steps_is_made_by_the_first_call_that_takes_them(seen):
    per_step = seen["step7"]["kernels"] // 7
    one, many = ["make%d" % per_step], ["make%d" % (8 * per_step)]

    def makes(log):
        return [c for c in log if c.startswith("make")]

    assert makes(seen["create"]) == one
    assert makes(seen["step7"]["log"]) == []
    alone, eight = ["graph%d" % per_step], ["graph%d" % (8 * per_step)]
    for calls, expect in (("step16", (alone * 8 + many + eight, eight * 2)),  # behind eight steps, for the others
                          ("step9", (alone * 9 + many, eight + alone))):      # behind all of them, for the next call
        for r, e in zip(seen[calls], expect):
            assert [c for c in r["log"] if c != "kernel"] == e + ["wait-stream"]


def test_steps_go_on_where_the_graph_of_many_cannot_be_made(seen):
    for k, r in enumerate(seen["no_graph"]):
        assert r["ok"] and r["steps"] == 16 * (k + 1) and r["kernels"] == 16 * (seen["step7"]["kernels"] // 7)
