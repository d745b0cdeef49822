"""The library's host code on a machine with two devices, whose runtime is a stand-in that keeps each
device's kernel attributes and refuses the launches that the real one refuses: the LU's panels after
a first factorisation on another device."""
from __future__ import annotations

import shutil
import subprocess
import sys
from pathlib import Path

import pytest

from flapjax_b200 import _lib
from flapjax_b200.build import nvcc

RUNTIME = r"""
#include <cuda_runtime_api.h>
#include <map>
#include <set>
#include <utility>
static int device = 0;
static cudaError_t last = cudaSuccess;
static std::map<std::pair<int, const void*>, size_t> smem;
static std::set<std::pair<int, const void*>> any_cluster;
struct Config { dim3 g, b; size_t smem; void* stream; };
static Config pushed;
static cudaError_t result(bool ok) { if (!ok) last = cudaErrorInvalidValue; return ok ? cudaSuccess : cudaErrorInvalidValue; }
static bool runs(const void* f, size_t bytes, unsigned cluster) {
    const auto it = smem.find({device, f});
    return bytes <= (it != smem.end() ? it->second : 48 * 1024) && (cluster <= 8 || any_cluster.count({device, f}));
}
static unsigned cluster_of(const cudaLaunchConfig_t* c) {
    for (unsigned i = 0; i < c->numAttrs; ++i)
        if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) return c->attrs[i].val.clusterDim.x;
    return 1;
}
extern "C" {
void stand_in_device(int d) { device = d; }
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "refused"; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
        if (v > 232448) return result(false);
        smem[{device, f}] = v;
    } else if (a == cudaFuncAttributeNonPortableClusterSizeAllowed) any_cluster.insert({device, f});
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void* f, const cudaLaunchConfig_t* c) {
    *n = runs(f, c->dynamicSmemBytes, cluster_of(c));
    return result(*n > 0);
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t bytes, cudaStream_t) { return result(runs(f, bytes, 1)); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    return result(runs(f, c->dynamicSmemBytes, cluster_of(c)));
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, void* st) { pushed = {g, b, s, st}; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* st) {
    *g = pushed.g; *b = pushed.b; *s = pushed.smem; *(void**)st = pushed.stream;
    return cudaSuccess;
}
}
"""

CALLS = r"""
import ctypes as C, sys
runtime, lib = C.CDLL(sys.argv[1], mode=C.RTLD_GLOBAL), C.CDLL(sys.argv[2])
lib.fj_last_error_string.restype = C.c_char_p
p = C.c_void_p(1 << 20)  # (nothing is read)
for device in (0, 1, 0):
    runtime.stand_in_device(device)
    for n in (64, 200, 384, 768, 2048, 3000):
        st = lib.fj_lu_factor(p, n, p, p, C.c_size_t(256 + 8 * n), None)
        assert st == 0, (device, n, lib.fj_last_error_string())
"""


def test_panels_on_a_second_device(tmp_path):
    if not _lib.LIB_PATH.exists():
        pytest.skip("libfj_uvlm.so not built (run __graft_entry__.build())")
    names = subprocess.run(["nm", "-D", "-u", str(_lib.LIB_PATH)], capture_output=True, text=True, check=True).stdout
    used = {w.split("@")[0] for w in names.split() if w.lstrip("_").startswith("cuda")}
    others = sorted(u for u in used if f" {u}(" not in RUNTIME)
    (tmp_path / "runtime.cc").write_text(RUNTIME)
    (tmp_path / "others.c").write_text("".join(f"static long w_{n}[8]; long {n}() {{ return 0; }}\n" for n in others)
                                       .replace("long __cudaRegisterFatBinary() { return 0; }",
                                                "long* __cudaRegisterFatBinary() { return w___cudaRegisterFatBinary; }"))
    (tmp_path / "map").write_text("libcudart.so.12 { global: *; };")
    inc, so, cc = Path(nvcc()).parents[1] / "include", tmp_path / "libcudart.so.12", shutil.which("gcc")
    subprocess.run([cc, "-shared", "-fPIC", "-w", "-I", str(inc), str(tmp_path / "runtime.cc"), str(tmp_path / "others.c"),
                    "-lstdc++", "-Wl,-soname,libcudart.so.12", f"-Wl,--version-script={tmp_path / 'map'}", "-o", str(so)],
                   check=True)
    r = subprocess.run([sys.executable, "-c", CALLS, str(so), str(_lib.LIB_PATH)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
