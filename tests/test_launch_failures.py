"""A launch that fails ends its call: the error comes back and nothing is launched behind it, since the kernels behind would take what
the scratch holds for their work list.  The host code runs against a CUDA runtime of stubs (no GPU, no kernel): memory is host
memory, and the n-th launch of a call reports cudaErrorLaunchOutOfResources."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

STUBS = r"""
#include <stdint.h>
#include <stdlib.h>
#include <string.h>
static int launches, fail_at, last;
void stub_arm(int n) { launches = 0; fail_at = n; last = 0; }
int stub_launches(void) { return launches; }
static int launch(void) { return ++launches == fail_at ? (last = 701) : 0; }
int cudaLaunchKernelExC(const void* c, const void* f, void** a) { return launch(); }
int cudaLaunchKernel(const void* f, ...) { return launch(); }
int cudaGetLastError(void) { int e = last; last = 0; return e; }
const char* cudaGetErrorString(int e) { return "stub"; }
unsigned __cudaPushCallConfiguration() { return 0; }
int __cudaPopCallConfiguration() { return 0; }
static void* fat[1];
void** __cudaRegisterFatBinary(void* p) { return fat; }
void __cudaRegisterFatBinaryEnd(void** h) {}
void __cudaUnregisterFatBinary(void** h) {}
void __cudaRegisterFunction() {}
void __cudaRegisterVar() {}
int cudaMalloc(void** p, size_t n) { *p = aligned_alloc(256, (n + 255) / 256 * 256); return *p ? 0 : 2; }
int cudaFree(void* p) { free(p); return 0; }
int cudaMemset(void* p, int v, size_t n) { memset(p, v, n); return 0; }
int cudaMemsetAsync(void* p, int v, size_t n, void* s) { return 0; }
int cudaMemcpy(void* d, const void* s, size_t n, int k) { memcpy(d, s, n); return 0; }
int cudaMemcpyAsync(void* d, const void* s, size_t n, int k, void* st) { memcpy(d, s, n); return 0; }
int cudaFuncSetAttribute(const void* f, int a, int v) { return 0; }
int cudaGetDevice(int* d) { *d = 0; return 0; }
int cudaGetDeviceCount(int* n) { *n = 1; return 0; }
int cudaDeviceGetAttribute(int* v, int a, int d) { *v = 148; return 0; }
int cudaStreamSynchronize(void* s) { return 0; }
static char symbol[4096];
int cudaGetSymbolAddress(void** p, const void* s) { *p = symbol; return 0; }
static int encode() { return 0; }
int cudaGetDriverEntryPoint(const char* n, void** p, unsigned long long f, int* r) { *p = (void*)encode; if (r) *r = 0; return 0; }
"""

CHILD = r"""
import ctypes as C, sys
stub = C.CDLL(sys.argv[1], mode=C.RTLD_GLOBAL)
from mference_b200 import _lib as L
lib = L.load()
call, d, f, bits, gate, tokens = sys.argv[2], *map(int, sys.argv[3:8])
cfg = L.MoEConfig(d=d, f=f, num_experts=16, top_k=4, bits=bits, shared_bits=4, group_size=64, scale_dtype=L.DT_F16, x_dtype=L.DT_BF16, route_scale=1.0,
                  max_tokens=tokens, flags=L.FLAG_PREFILL_TENSOR_CORE)
moe = C.c_void_p()
L.check(lib.mfb_moe_create(C.byref(cfg), C.byref(moe)))
base = (C.addressof(C.create_string_buffer(1 << 20)) + 4095) & ~4095      # never read: there are no kernels
w = L.LayerWeightsC(router_w=base, norm_w=base, pool=base, shared_blob=base, slot_stride=1 << 20, gate_group_size=gate)
layers = (L.LayerWeightsC * 3)(w, w, w)
run = {"layer": lambda: lib.mfb_moe_layer(moe, None, C.byref(w), base, base, tokens),
       "prefill": lambda: lib.mfb_moe_layer_prefill(moe, None, C.byref(w), base, base, tokens),
       "stack": lambda: lib.mfb_moe_stack(moe, None, layers, 3, base, tokens),
       "decode": lambda: lib.mfb_moe_decode(moe, None, C.byref(w), base, d, tokens, base, base, base, base)}[call]
stub.stub_arm(0)
assert run() == L.OK, lib.mfb_last_error()
total = stub.stub_launches()
for n in range(1, total + 1):
    stub.stub_arm(n)
    rc = run()
    assert rc == L.ERR_CUDA and stub.stub_launches() == n, (n, total, rc, stub.stub_launches())
print("launches", total)
"""


@pytest.fixture(scope="module")
def stubs(tmp_path_factory):
    folder = tmp_path_factory.mktemp("stubs")
    (folder / "stubs.c").write_text(STUBS)
    subprocess.run(["gcc", "-shared", "-fPIC", "-w", "-o", str(folder / "stubs.so"), str(folder / "stubs.c")], check=True)
    return str(folder / "stubs.so")


@pytest.mark.parametrize("call,d,f,bits,gate,tokens,least", [
    ("prefill", 512, 512, 2, 32, 90, 8),      # blocks of rows in fp32
    ("prefill", 512, 512, 2, 32, 66, 6),
    ("prefill", 1280, 256, 4, 64, 90, 8),
    ("prefill", 512, 512, 4, 64, 90, 6),      # tensor cores
    ("prefill", 512, 512, 4, 64, 5000, 6),
    ("layer", 512, 512, 4, 64, 1, 5),         # streaming kernels
    ("layer", 512, 512, 2, 32, 13, 5),
    ("layer", 512, 512, 4, 64, 90, 5),        # fp32 kernels
    ("stack", 512, 512, 4, 64, 1, 13),
    ("stack", 512, 512, 4, 64, 8, 16),
    ("decode", 512, 512, 4, 64, 8, 5),
    ("decode", 512, 512, 4, 64, 90, 4),
])
def test_a_launch_that_fails_ends_the_call(stubs, call, d, f, bits, gate, tokens, least):
    env = dict(os.environ, LD_PRELOAD=stubs, PYTHONPATH=ROOT)
    done = subprocess.run([sys.executable, "-c", CHILD, stubs, call, *map(str, (d, f, bits, gate, tokens))], env=env, cwd=ROOT, capture_output=True, text=True,
                          timeout=120)
    assert done.returncode == 0, done.stderr
    assert int(done.stdout.split()[-1]) >= least
