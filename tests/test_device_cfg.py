"""Launch settings are asked per device: the objects of the operator passes, linked against a
stand-in for the CUDA runtime that grants large shared memory per device, opt in on each device
they are used on (a process may solve on one device after another)."""
import os
import shutil
import subprocess

import pytest

from tests import helpers as H

OBJ = os.path.join(H.ROOT, "chfem_b200", "lib", "obj")

RUNTIME = r'''
#include <cstddef>
#include <cstdio>
#include <map>
#include <utility>
static int device = 0, failed = 0;
static std::map<std::pair<int, const void*>, int> granted;  // (device, kernel) -> bytes
static int asked = 0;
struct dim3_ { unsigned x, y, z; };
extern "C" {
int cudaGetDevice(int* d) { *d = device; return 0; }
int cudaDeviceGetAttribute(int* v, int, int d) { *v = 100 + d; return 0; }
int cudaFuncSetAttribute(const void* f, int, int bytes) { asked++; granted[{device, f}] = bytes; return 0; }
// one CTA fits once its bytes are granted on the current device
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int, size_t smem, unsigned) {
  auto g = granted.find({device, f});
  if (smem > 48 * 1024 && (g == granted.end() || (size_t)g->second < smem)) { failed = 1; return 1; }
  *n = 1 + device;
  return 0;
}
int cudaGetLastError() { return 0; }
int cudaLaunchKernel(const void*, dim3_, dim3_, void**, size_t, void*) { return 0; }
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
unsigned __cudaPushCallConfiguration(dim3_, dim3_, size_t, void*) { return 0; }
int __cudaPopCallConfiguration(dim3_*, dim3_*, size_t*, void*) { return 0; }
}
namespace chfem {
template <int ND, typename T, int MODE> int md_ctas(bool, int, int, int, int);
template <int ND, typename T> int md_block_ctas(int, int, int, int, int);
template <int ND, typename T, int NR> int asm_block_ctas(int, int, int, int);
template <int ND, typename T, int MODE> int asm_te_ctas(int, int, int, int);
}
int main() {
  using namespace chfem;
  for (int round = 0; round < 2; round++)
    for (device = 0; device < 70; device += 23) {
      const int before = asked;
      const int n[] = {md_ctas<3, double, 1>(false, 640, 640, 640, 100), md_block_ctas<3, float>(6, 640, 640, 640, 100),
                       asm_block_ctas<3, float, 6>(640, 640, 640, 100), asm_te_ctas<3, double, 1>(640, 640, 640, 100)};
      for (int v : n)
        if (v != 100 * (1 + device)) { printf("device %d: %d CTAs\n", device, v); failed = 1; }
      const int want = round && device < 64 ? 0 : 4;  // kept per device; a device past the table is asked again
      if (asked - before != want) { printf("device %d, round %d: asked %d times\n", device, round, asked - before); failed = 1; }
    }
  return failed;
}
'''


@pytest.mark.skipif(not shutil.which("g++") or not os.path.exists(os.path.join(OBJ, "modal_apply.o")),
                    reason="needs g++ and the built objects")
def test_operator_passes_opt_in_on_every_device(tmp_path):
    src, exe = tmp_path / "runtime.cpp", tmp_path / "check"
    src.write_text(RUNTIME)
    subprocess.run(["g++", "-std=c++17", "-o", str(exe), str(src), os.path.join(OBJ, "modal_apply.o"), os.path.join(OBJ, "asm_apply.o")],
                   check=True, capture_output=True, text=True)
    p = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert p.returncode == 0, p.stdout
