"""The launch of csrc/gemm_gated_tc.cu in a process that uses two devices, against a stand-in for the CUDA runtime: no GPU is needed.
How much shared memory a kernel may have is set per device; a device on which it was not set refuses the launch."""
import os
import subprocess
import sys

from lmsf_b200.csrc import build

FAKE = r"""
#include <stddef.h>
#include <string.h>
static int device, allowed[2], sms[2] = {148, 20};
static unsigned grid;
void set_device(int d) { device = d; }
unsigned last_grid() { return grid; }
int cudaGetDevice(int* d) { *d = device; return 0; }
int cudaDeviceGetAttribute(int* v, int attr, int d) { *v = sms[d]; return 0; }
int cudaFuncSetAttribute(const void* f, int attr, int v) { allowed[device] = v; return 0; }
struct Config { unsigned gx, gy, gz, bx, by, bz; size_t smem; void* stream; void* attrs; unsigned n; };
int cudaLaunchKernelExC(const struct Config* c, const void* f, void** args) { grid = c->gx; return (int)c->smem > allowed[device] ? 1 : 0; }
static int encode() { return 0; }
int cudaGetDriverEntryPoint(const char* name, void** p, unsigned long long flags, int* q) { *p = (void*)encode; *q = 0; return 0; }
int cudaGetDriverEntryPointByVersion(const char* n, void** p, unsigned v, unsigned long long f, int* q) { return cudaGetDriverEntryPoint(n, p, f, q); }
int cudaGetLastError() { return 0; }
int cudaLaunchKernel() { return 0; }
int __cudaLaunchKernel() { return 0; }
const char* cudaGetErrorString(int e) { return ""; }
static void* handle;
void** __cudaRegisterFatBinary(void* b) { return &handle; }
void __cudaRegisterFatBinaryEnd(void** h) {}
void __cudaUnregisterFatBinary(void** h) {}
void __cudaRegisterFunction() {}
int __cudaPushCallConfiguration() { return 0; }
int __cudaPopCallConfiguration() { return 0; }
int __cudaGetKernel() { return 0; }
char __cudaInitModule(void** h) { return 0; }
void __cudaRegisterVar() {}
"""

USE = """
import ctypes, sys
fake = ctypes.CDLL(sys.argv[1], mode=ctypes.RTLD_GLOBAL)
f = ctypes.CDLL(sys.argv[2]).lmsf_gemm_gated_tc
f.argtypes = [ctypes.c_void_p, ctypes.c_longlong, ctypes.c_void_p, ctypes.c_longlong, ctypes.c_void_p] + [ctypes.c_int] * 4 + [ctypes.c_void_p] * 2
for d in (0, 1, 0, 1):
    fake.set_device(d)
    print(d, f(4096, 8192, 4096, 64, 4096, 2048, 8192, 64, 0, None, None), fake.last_grid())
"""


def test_every_device_is_asked_and_set_up(tmp_path):
    (tmp_path / "fake.c").write_text(FAKE)
    (tmp_path / "use.py").write_text(USE)
    fake, lib = str(tmp_path / "libfake.so"), str(tmp_path / "libgated.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-w", str(tmp_path / "fake.c"), "-o", fake], check=True)
    subprocess.run([build._nvcc(), *build.ARCH_FLAGS, *build.BASE_FLAGS, "--cudart", "none", "-I", build.CSRC_DIR,
                    os.path.join(build.CSRC_DIR, "gemm_gated_tc.cu"), "-o", lib], check=True, capture_output=True)
    out = subprocess.run([sys.executable, str(tmp_path / "use.py"), fake, lib], capture_output=True, text=True)
    # (device, answer, blocks): one pair of blocks per two SMs of the device that is current
    assert out.stdout.split("\n")[:4] == ["0 0 148", "1 0 20", "0 0 148", "1 0 20"], out
