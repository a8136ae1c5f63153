"""A stand-in for the CUDA runtime under the built objects of libcudapcg_b200, for checks of the host
side that need no GPU: device memory is host memory, kernels do nothing, and the stand-in keeps
account of what the real runtime leaves to the caller:

- large dynamic shared memory is granted per (device, kernel);
- a solve ends with the first scalar record that is read back after a graph launch (fake_finish);
- copies and fills on the legacy stream are not ordered with the solver's non-blocking stream: work
  there that may read or overwrite them before the legacy stream was waited for, and the reverse,
  is recorded (fake_report).
"""
import os
import shutil
import subprocess

from tests import helpers as H

OBJ = os.path.join(H.ROOT, "chfem_b200", "lib", "obj")
OBJECTS = [os.path.join(OBJ, o + ".o") for o in ("cudapcg_b200", "modal_apply", "asm_apply", "pore_maps", "batch_thermal", "learned")] + [
    os.path.join(OBJ, f"modal_{n}_{t}_{p}.o") for n in (1, 3) for t in ("float", "double") for p in ("PASS", "DENSITY", "BLOCK", "POINT")]

SOURCE = r'''
#include <cstddef>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <utility>
#include <vector>
typedef void* stream_t;
struct dim3_ { unsigned x, y, z; };
struct range { const char* p; size_t n; };
static int device = 0, asked = 0;
static std::map<std::pair<int, const void*>, int> granted;  // (device, kernel) -> bytes
static std::vector<range> legacy, queued;  // written, not waited for: on the legacy stream; by copies and fills elsewhere
static int n_legacy = 0, live = 0;
static std::vector<range> pinned;
static size_t rec_size = 0, rec_done = 0;
static int graphs = 0, launched = 0, launches = 0;
static thread_local int capturing = 0;
static std::recursive_mutex mu;
#define LOCK std::lock_guard<std::recursive_mutex> lock(mu);
static std::string bad;
static void violation(const char* what) { bad += std::string(what) + "\n"; }
static bool meets(const std::vector<range>& v, const void* p, size_t n) {
  for (const range& r : v)
    if (r.p < (const char*)p + n && (const char*)p < r.p + r.n) return true;
  return false;
}
static void on_legacy(const char* what, void* p, size_t n) {
  if (meets(queued, p, n)) violation((std::string(what) + " over memory that the solver's stream still writes").c_str());
  legacy.push_back({(const char*)p, n});
  n_legacy++;
}
static void on_stream(const char* what, stream_t s, void* p, size_t n, const void* src, size_t ns) {
  if (!s) { on_legacy(what, p, n); return; }
  if (meets(legacy, p, n) || (src && meets(legacy, src, ns))) violation((std::string(what) + " on memory that the legacy stream still writes").c_str());
  queued.push_back({(const char*)p, n});
}
extern "C" {
void fake_finish(size_t size, size_t done) { rec_size = size; rec_done = done; }  // a record's bytes, its flag's offset
int fake_graphs() { return graphs; }      // captures so far
int fake_launches() { return launches; }  // kernels launched so far, not counting captured ones
const char* fake_report() { return bad.c_str(); }
int fake_asked() { return asked; }
int fake_live() { return live; }  // streams, events and pinned blocks that were not destroyed
void fake_set_device(int d) { device = d; }

int cudaGetDevice(int* d) { *d = device; return 0; }
int cudaDeviceGetAttribute(int* v, int, int d) { *v = 100 + d; return 0; }
int cudaDeviceSynchronize() { LOCK legacy.clear(); queued.clear(); return 0; }
int cudaDeviceGetDefaultMemPool(void** p, int) { *p = nullptr; return 0; }
int cudaMemPoolSetAttribute(void*, int, void*) { return 0; }
int cudaMemPoolTrimTo(void*, size_t) { return 0; }
int cudaMemGetInfo(size_t* f, size_t* t) { *f = *t = (size_t)1 << 40; return 0; }
const char* cudaGetErrorString(int) { return "error of the stand-in"; }
int cudaGetLastError() { return 0; }
int cudaPeekAtLastError() { return 0; }
int cudaFuncSetAttribute(const void* f, int, int bytes) { LOCK asked++; granted[{device, f}] = bytes; return 0; }
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int, size_t smem, unsigned) { LOCK
  auto g = granted.find({device, f});
  if (smem > 48 * 1024 && (g == granted.end() || (size_t)g->second < smem)) { violation("occupancy of a kernel without its shared memory"); return 1; }
  *n = 1 + device;
  return 0;
}
int cudaMallocAsync(void** p, size_t n, stream_t) { LOCK if (capturing) violation("allocation during a capture"); *p = calloc(1, n ? n : 1); return *p ? 0 : 2; }
int cudaFreeAsync(void*, stream_t) { return 0; }  // kept: addresses stay distinct
int cudaHostAlloc(void** p, size_t n, unsigned) { LOCK live++; *p = calloc(1, n); pinned.push_back({(const char*)*p, n}); return 0; }
int cudaFreeHost(void* p) { LOCK live--; free(p); return 0; }
int cudaMemcpy(void* d, const void* s, size_t n, int kind) { LOCK memcpy(d, s, n); if (kind != 2) on_legacy("copy", d, n); return 0; }
int cudaMemset(void* d, int v, size_t n) { LOCK memset(d, v, n); on_legacy("fill", d, n); return 0; }
int cudaMemcpyToSymbol(const void*, const void*, size_t, size_t, int) { LOCK n_legacy++; return 0; }
int cudaGetSymbolAddress(void** p, const void*) { static char scratch[1 << 20]; *p = scratch; return 0; }
int cudaMemcpyAsync(void* d, const void* s, size_t n, int kind, stream_t st) { LOCK
  memcpy(d, s, n);
  if (kind != 2) on_stream("copy", st, d, n, kind == 3 ? s : nullptr, n);
  else if (launched && rec_size && n % rec_size == 0 && meets(pinned, d, n))
    for (size_t k = 0; k < n; k += rec_size) { const int one = 1; memcpy((char*)d + k + rec_done, &one, sizeof(int)); }
  return 0;
}
int cudaMemsetAsync(void* d, int v, size_t n, stream_t st) { LOCK memset(d, v, n); on_stream("fill", st, d, n, nullptr, 0); return 0; }
int cudaStreamCreateWithFlags(stream_t* s, unsigned) { LOCK static size_t next = 0x1000; live++; *s = (void*)next++; return 0; }
int cudaStreamDestroy(stream_t) { LOCK live--; return 0; }
int cudaStreamSynchronize(stream_t s) { LOCK if (s) queued.clear(); else { legacy.clear(); n_legacy = 0; } return 0; }
int cudaStreamIsCapturing(stream_t, int* c) { *c = 0; return 0; }
int cudaStreamBeginCapture(stream_t, int) { LOCK graphs++; capturing = 1; return 0; }
int cudaStreamEndCapture(stream_t, void** g) { capturing = 0; *g = (void*)1; return 0; }
int cudaGraphInstantiate(void** x, void*, unsigned long long) { *x = (void*)1; return 0; }
int cudaGraphDestroy(void*) { return 0; }
int cudaGraphExecDestroy(void*) { return 0; }
int cudaGraphLaunch(void*, stream_t s) { LOCK
  if (s && n_legacy) violation("launch before the legacy stream was waited for");
  launched = 1;
  return 0;
}
int cudaEventCreate(void** e) { LOCK live++; *e = (void*)1; return 0; }
int cudaEventDestroy(void*) { LOCK live--; return 0; }
int cudaEventRecord(void*, stream_t) { return 0; }
int cudaEventSynchronize(void*) { LOCK queued.clear(); return 0; }
int cudaEventElapsedTime(float* t, void*, void*) { *t = 1.f; return 0; }
int cudaLaunchKernel(const void* f, dim3_, dim3_, void**, size_t smem, stream_t s) { LOCK
  auto g = granted.find({device, f});
  if (smem > 48 * 1024 && (g == granted.end() || (size_t)g->second < smem)) { violation("launch of a kernel without its shared memory"); return 1; }
  if (s && n_legacy) violation("launch before the legacy stream was waited for");
  launches += !capturing;
  return 0;
}
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
static thread_local dim3_ cfg_g, cfg_b; static thread_local size_t cfg_s; static thread_local stream_t cfg_t;
unsigned __cudaPushCallConfiguration(dim3_ g, dim3_ b, size_t s, stream_t t) { cfg_g = g; cfg_b = b; cfg_s = s; cfg_t = t; return 0; }
int __cudaPopCallConfiguration(dim3_* g, dim3_* b, size_t* s, stream_t* t) { *g = cfg_g; *b = cfg_b; *s = cfg_s; *t = cfg_t; return 0; }
}
'''


def available():
    return bool(shutil.which("g++")) and all(os.path.exists(o) for o in OBJECTS)


def build(workdir):
    """libcudapcg_b200 over the stand-in, as a shared library; its path."""
    src, lib = os.path.join(str(workdir), "fake_cuda.cpp"), os.path.join(str(workdir), "libfake_cudapcg.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-o", lib, src, *OBJECTS], check=True,
                   capture_output=True, text=True)
    return lib
