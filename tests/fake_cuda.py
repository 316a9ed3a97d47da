"""abi.cu, the host side of the library, linked against a fake of the CUDA runtime and of the kernel
launchers, for CPU tests of what it does when a call fails or an argument is refused."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np

from speedycolibri_b200 import _lib

# What a case needs from the runtime: handles and memory that look real, a log of the calls that put work on
# a stream, and the n-th of them refused.
SHIM = r"""
#include <cuda.h>
#include <driver_types.h>
#include <stdlib.h>
#include <string.h>
static int log_n, fail_at;
static char last, launched[1 << 16];
void fake_reset(int fail) { log_n = 0; fail_at = fail; last = 0; launched[0] = 0; }
int fake_queued(void) { return log_n; }
int fake_waited(void) { return last == 'w'; }
const char *fake_launches(void) { return launched; }  /* the launchers called since the reset, by their linker names */
static void note(const char *name) {
  if (strlen(launched) + strlen(name) + 2 < sizeof launched) strcat(strcat(launched, name), " ");
}
static int queue(void) { if (++log_n == fail_at) return 1; last = 'q'; return 0; }
int cudaMalloc(void **p, size_t n) { *p = malloc(n ? n : 1); return 0; }
int cudaFree(void *p) { free(p); return 0; }
int cudaHostAlloc(void **p, size_t n) { return cudaMalloc(p, n); }
int cudaFreeHost(void *p) { return cudaFree(p); }
static char *pinned;  /* the one page-locked allocation: where, how long, what the device may do with it */
static size_t pinned_n;
static unsigned long long pinned_access;
void fake_pin(char *at, size_t n, int access) { pinned = at; pinned_n = n; pinned_access = access; }
int cudaPointerGetAttributes(struct cudaPointerAttributes *a, char *p) {
  memset(a, 0, sizeof(*a));
  if (p >= pinned && p < pinned + pinned_n) a->type = cudaMemoryTypeHost, a->hostPointer = a->devicePointer = p;
  return 0;
}
static int pointer_attribute(void *value, int which, char *p) {
  if (p < pinned || p >= pinned + pinned_n) return 1;
  if (which == CU_POINTER_ATTRIBUTE_RANGE_START_ADDR) *(char **)value = pinned;
  else if (which == CU_POINTER_ATTRIBUTE_RANGE_SIZE) *(size_t *)value = pinned_n;
  else if (which == CU_POINTER_ATTRIBUTE_ACCESS_FLAGS) *(unsigned long long *)value = pinned_access;
  else return 1;
  return 0;
}
int cudaGetDriverEntryPoint(const char *name, void **fn, unsigned long long flags, int *found) {
  *fn = strcmp(name, "cuPointerGetAttribute") ? 0 : (void *)pointer_attribute;
  *found = 0;
  return 0;
}
int cudaGetDeviceCount(int *n) { *n = 1; return 0; }
int cudaDeviceGetAttribute(int *v) { *v = 148; return 0; }
int cudaGetDeviceProperties_v2(struct cudaDeviceProp *p) {
  memset(p, 0, sizeof(*p));
  p->major = 10;
  p->multiProcessorCount = 148;
  return 0;
}
int cudaStreamCreateWithFlags(void **s) { *s = malloc(1); return 0; }
int cudaEventCreate(void **e) { *e = malloc(1); return 0; }
const char *cudaGetErrorString(int e) { (void)e; return "refused by the test"; }
int cudaMemcpyAsync(void) { return queue(); }
int cudaMemsetAsync(void) { return queue(); }
int cudaEventRecord(void) { return queue(); }
int cudaStreamSynchronize(void) { last = 'w'; return 0; }
"""


def load(d):
    """libcoli_b200's host side over the fake, built in folder `d`; device 0 is initialised."""
    obj, shim, lib = str(d / "abi.o"), str(d / "shim.c"), str(d / "libfake.so")
    flags = [f for f in _lib.NVCC_FLAGS if f != "-shared"]
    subprocess.run(["nvcc", *flags, "-c", "-o", obj, "abi.cu"], cwd=_lib._CSRC, check=True, capture_output=True)
    undefined = [line.split()[-1] for line in subprocess.run(["nm", "-u", obj], check=True, capture_output=True, text=True).stdout.splitlines()]
    src = SHIM
    for s in undefined:
        if s.startswith("_ZN5colib"):
            src += f'int {s}(void) {{ note("{s}"); return !queue(); }}\n'  # a launcher answers 1 on success
        elif (s.startswith(("cuda", "__cuda")) or "coli_ep_" in s) and f" {s}(" not in src and f"*{s}(" not in src:
            src += f"int {s}(void) {{ return 0; }}\n"
    cuda_include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(shutil.which("nvcc")))), "include")
    open(shim, "w").write(src)
    subprocess.run(["gcc", "-w", "-fPIC", "-I", cuda_include, "-c", "-o", shim + ".o", shim], check=True)
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-Wl,-z,defs", "-o", lib, obj, shim + ".o", "-lpthread"], check=True)
    fake = C.CDLL(lib, mode=os.RTLD_LOCAL)
    fake.fake_launches.restype = C.c_char_p
    assert fake.coli_cuda_init((C.c_int * 1)(0), 1)
    return fake


def wrap_nvfp4(fake, O, I):
    """A handle of an [O,I] matrix of zeros."""
    h = C.c_void_p()
    q, s = np.zeros((O, (I + 1) // 2), np.uint8), np.zeros((O, (I + 15) // 16), np.uint8)
    fake.fake_reset(0)
    assert fake.coli_cuda_tensor_wrap_nvfp4(C.byref(h), q.ctypes.data_as(C.c_void_p), s.ctypes.data_as(C.c_void_p), C.c_float(1.0), I, O, 0)
    return h
