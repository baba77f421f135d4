"""A CUDA runtime without a device, for tests of the library's host side: allocations come
from the host heap and can be made to fail, launches are logged with their stream instead of
being run, and stream and event calls are logged in order.  It takes the real runtime's
place (same soname) in a child process that loads nothing else of CUDA."""
import json
import os
import subprocess
import sys

from aok_b200 import _lib

SOURCE = r"""
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <map>
#include <string>
#include <vector>
typedef int err_t;
typedef void* stream_t;
struct dim3_ { unsigned x, y, z; };
struct config_t { dim3_ grid, block; size_t smem; stream_t stream; void* attrs; unsigned nattrs; };
enum { OOM = 2 };
static std::map<void*, size_t> live;
static std::map<const void*, std::string> names;
static std::string ops;
static long nmalloc = 0, fail_at = -1, bad_frees = 0;
static size_t fail_size = ~(size_t)0;
static std::string fail_kernel;
static err_t last = 0;
static uintptr_t next_handle = 1;
static config_t pushed;
static err_t note(err_t e) { if (e) last = e; return e; }
static void op(const char* what, const void* a, const void* b) {
    char t[400];
    snprintf(t, sizeof(t), "%s %lx %lx\n", what, (unsigned long)(uintptr_t)a, (unsigned long)(uintptr_t)b);
    ops += t;
}
static err_t launch(const void* f, stream_t s, void** args) {
    const std::string name = names.count(f) ? names[f] : "?";
    // the coefficient table that the kernel writes (first argument) or reads (fourth)
    const int coef = name.find("k_compile_coefI") != std::string::npos ? 0
                     : name.find("k_prep_pbI") != std::string::npos    ? 3 : -1;
    if (!fail_kernel.empty() && name.find(fail_kernel) != std::string::npos) return note(OOM);
    op(("launch:" + name).c_str(), s, coef < 0 ? 0 : *(void**)args[coef]);
    return 0;
}
extern "C" {
// the test's side
void fake_fail(long at, size_t size) { nmalloc = 0; fail_at = at; fail_size = size; }
void fake_fail_kernel(const char* name) { fail_kernel = name; }
long fake_live() { return (long)live.size(); }
long fake_bad_frees() { return bad_frees; }
const char* fake_ops() { return ops.c_str(); }
void fake_clear() { ops.clear(); }
// the library's side
err_t cudaMalloc(void** p, size_t n) {
    if (nmalloc++ == fail_at || n >= fail_size) return note(OOM);
    *p = calloc(n ? n : 1, 1);
    live[*p] = n;
    return 0;
}
err_t cudaFree(void* p) {
    if (p && !live.erase(p)) ++bad_frees; else free(p);
    return 0;
}
err_t cudaMemcpy(void* d, const void* s, size_t n, int) { memcpy(d, s, n); return 0; }
err_t cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return 0; }
err_t cudaMemcpyAsync(void*, const void*, size_t, int, stream_t s) { op("copy", s, 0); return 0; }
err_t cudaMemsetAsync(void*, int, size_t, stream_t s) { op("set", s, 0); return 0; }
err_t cudaGetLastError() { err_t e = last; last = 0; return e; }
const char* cudaGetErrorString(err_t) { return "fake error"; }
err_t cudaGetDevice(int* d) { *d = 0; return 0; }
err_t cudaDeviceGetAttribute(int* v, int, int) { *v = 148; return 0; }
err_t cudaFuncGetAttributes(void* a, const void*) { memset(a, 0, 64); return 0; }
err_t cudaFuncSetAttribute(const void*, int, int) { return 0; }
err_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { *n = 1; return 0; }
err_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { *n = 1; return 0; }
err_t cudaGetSymbolAddress(void** p, const void*) { *p = 0; return note(1); }
err_t cudaStreamCreateWithFlags(stream_t* s, unsigned) { *s = (stream_t)(0x1000 + next_handle++); return 0; }
err_t cudaStreamDestroy(stream_t) { return 0; }
err_t cudaStreamSynchronize(stream_t) { return 0; }
err_t cudaStreamWaitEvent(stream_t s, void* e, unsigned) { op("wait", s, e); return 0; }
err_t cudaEventCreate(void** e) { *e = (void*)(0x2000 + next_handle++); return 0; }
err_t cudaEventCreateWithFlags(void** e, unsigned) { return cudaEventCreate(e); }
err_t cudaEventDestroy(void*) { return 0; }
err_t cudaEventRecord(void* e, stream_t s) { op("record", s, e); return 0; }
err_t cudaEventSynchronize(void*) { return 0; }
err_t cudaEventElapsedTime(float* t, void*, void*) { *t = 1.f; return 0; }
err_t cudaLaunchKernel(const void* f, dim3_, dim3_, void** args, size_t, stream_t s) { return launch(f, s, args); }
err_t cudaLaunchKernelExC(const config_t* c, const void* f, void** args) { return launch(f, c->stream, args); }
unsigned __cudaPushCallConfiguration(dim3_ g, dim3_ b, size_t m, stream_t s) { pushed = {g, b, m, s, 0, 0}; return 0; }
err_t __cudaPopCallConfiguration(dim3_* g, dim3_* b, size_t* m, stream_t* s) {
    *g = pushed.grid; *b = pushed.block; *m = pushed.smem; *s = pushed.stream;
    return 0;
}
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* f, char*, const char* name, int, void*, void*, void*, void*, int*) {
    names[f] = name;
}
// graphs and what else the library binds: not used here
#define REFUSE(f) err_t f() { return note(801); }
REFUSE(cudaGraphDestroy) REFUSE(cudaGraphExecDestroy) REFUSE(cudaGraphExecUpdate) REFUSE(cudaGraphInstantiate)
REFUSE(cudaGraphLaunch) REFUSE(cudaStreamBeginCapture) REFUSE(cudaStreamEndCapture)
}
"""

PRELUDE = """
import ctypes, json, sys
fake = ctypes.CDLL(sys.argv[1], mode=ctypes.RTLD_GLOBAL)
fake.fake_fail.argtypes = [ctypes.c_long, ctypes.c_size_t]
fake.fake_ops.restype = ctypes.c_char_p
for f in ("fake_live", "fake_bad_frees"):
    getattr(fake, f).restype = ctypes.c_long
NEVER = (-1, 2**64 - 1)
L = ctypes.CDLL(sys.argv[2])
L.aok_last_error.restype = ctypes.c_char_p
P, I64, F64 = ctypes.c_void_p, ctypes.c_int64, ctypes.c_double
buf = ctypes.create_string_buffer(4096)          # stands for every device array of a call
A = ctypes.addressof(buf)
def ops():
    t = [x.split() for x in fake.fake_ops().decode().splitlines()]
    fake.fake_clear()
    return t
def plan(ls, K, NZ, prec, max_batch):
    h = P()
    arr = (I64 * len(ls))(*ls)
    assert L.aok_plan_create(ctypes.byref(h), I64(len(ls)), arr, I64(K), I64(NZ), prec, I64(max_batch)) == 0
    return h
"""


def run(body, tmp_path):
    """Runs `body` after PRELUDE in a child process; returns what it prints last, as JSON."""
    if not os.path.exists(_lib.SO_PATH):
        _lib.build()
    src, so, ver = (str(tmp_path / n) for n in ("fake.cpp", "libcudart.so.12", "fake.map"))
    with open(src, "w") as f:
        f.write(SOURCE)
    with open(ver, "w") as f:
        f.write("libcudart.so.12 { global: *; };\n")
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-Wl,-soname,libcudart.so.12", f"-Wl,--version-script={ver}",
                    src, "-o", so], check=True)
    r = subprocess.run([sys.executable, "-c", PRELUDE + body, so, _lib.SO_PATH], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return json.loads(r.stdout.splitlines()[-1])


def ordered(log, first, second):
    """Whether the launch number `first` of the log is complete before launch number `second`
    starts, by stream order and events."""
    clock, events, seen, n = {}, {}, [], 0
    for what, s, e in log:
        c = clock.setdefault(s, {s: 0})
        if what == "record":
            events[e] = dict(c)
        elif what == "wait":
            for k, v in events.get(e, {}).items():
                c[k] = max(c.get(k, 0), v)
        else:
            before = dict(c)
            c[s] += 1
            if what.startswith("launch:"):
                seen.append((s, c[s], before))
    s, at, _ = seen[first]
    return seen[second][2].get(s, 0) >= at
