"""A process that works on a second GPU: the kernels that need more shared memory than the default ask for it on every device.
The library's host code runs here against a fake of the few runtime calls involved, launches of both kinds among them, and sees no
device, so no GPU takes part; the fake refuses a launch, as the real calls do, when the current device has not been asked."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

from open_transformers_b200 import build_native

FAKE = r"""
#include <stddef.h>
typedef struct { unsigned x, y, z; } dim3_;
typedef struct { dim3_ grid, block; size_t smem; void* stream; void* attrs; unsigned n_attrs; } config_;  /* cudaLaunchConfig_t */
static int device, last;
static struct { const void* f; int dev, bytes; } asked[256];
static int n_asked;
static int fake_launches, fake_early;
int fake_refuse_next;
void fake_set_device(int d) { device = d; }
int fake_asked(void) { return n_asked; }
int fake_launched(void) { return fake_launches; }
int fake_launched_early(void) { return fake_early; }
void fake_refuse(void) { fake_refuse_next = 1; }
int cudaGetDevice(int* d) { *d = device; return 0; }
int cudaGetLastError(void) { int e = last; last = 0; return e; }
int cudaDeviceGetAttribute(int* v, int attr, int d) { *v = 148; return 0; }
int cudaFuncSetAttribute(const void* f, int attr, int value) {
  if (fake_refuse_next) { fake_refuse_next = 0; return 999; }
  asked[n_asked].f = f; asked[n_asked].dev = device; asked[n_asked++].bytes = value;
  return 0;
}
static int launch(const void* f, dim3_ g, size_t smem) {
  int most = 48 << 10, i;
  for (i = 0; i < n_asked; ++i)
    if (asked[i].f == f && asked[i].dev == device && asked[i].bytes > most) most = asked[i].bytes;
  if (smem > (size_t)most || !g.x || !g.y || !g.z) return last = 1;
  ++fake_launches;
  return 0;
}
int cudaLaunchKernel(const void* f, dim3_ g, dim3_ b, void** args, size_t smem, void* stream) { return launch(f, g, smem); }
int cudaLaunchKernelExC(const config_* c, const void* f, void** args) {
  int rc = launch(f, c->grid, c->smem);
  if (!rc) ++fake_early;
  return rc;
}
"""

CHILD = r"""
import ctypes, sys
fake, lib = ctypes.CDLL(sys.argv[1]), ctypes.CDLL(sys.argv[2])
N, q = ctypes.c_void_p(0), ctypes.c_long(256)
i = [ctypes.c_int(v) for v in (1, 128, 2, 1)]

def calls(D):
    d, w, s = ctypes.c_int(D), ctypes.c_int(0), ctypes.c_float(1.0)
    fwd = lib.otb_attn_f32_fwd(N, q, N, q, N, q, N, *i, d, w, s, N)
    bwd = lib.otb_attn_f32_bwd(N, q, N, q, N, q, N, q, N, N, N, q, N, q, *i, d, w, s, N)
    norm = lib.otb_rmsnorm_bwd(N, N, N, N, N, ctypes.c_void_p(16), ctypes.c_long(8), ctypes.c_int(4096), s, ctypes.c_int(0), N)
    return fwd, bwd, norm

fake.fake_refuse()
assert lib.otb_attn_f32_fwd(N, q, N, q, N, q, N, *i, ctypes.c_int(64), ctypes.c_int(0), ctypes.c_float(1.0), N) == 999
counts = []
for dev in (0, 1, 0, 1):
    fake.fake_set_device(dev)
    for D in (64, 128):
        assert calls(D) == (0, 0, 0), (dev, D, calls(D))
    counts.append(fake.fake_asked())
assert fake.fake_launched() == 4 * 2 * (1 + 3 + 1)
assert fake.fake_launched_early() == 4 * 2 * 1  # the norm's: a small grid in a chain
assert counts[1] == 2 * counts[0] and counts[3] == counts[1], counts  # once per kernel and device
print("ok")
"""


def test_shared_memory_is_asked_for_on_every_device(tmp_path):
    lib = build_native.EXT / "libotb_cuda.so"
    if not lib.exists():
        pytest.skip("the CUDA library is not built here")
    (tmp_path / "fake.c").write_text(FAKE)
    fake = tmp_path / "libfake.so"
    cc = "/usr/bin/gcc" if Path("/usr/bin/gcc").exists() else "gcc"
    subprocess.run([cc, "-shared", "-fPIC", "-o", str(fake), str(tmp_path / "fake.c")], check=True)
    r = subprocess.run([sys.executable, "-c", CHILD, str(fake), str(lib)], env=dict(os.environ, LD_PRELOAD=str(fake), CUDA_VISIBLE_DEVICES=""), capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
