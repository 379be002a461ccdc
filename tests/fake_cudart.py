"""A stand-in for the few CUDA runtime calls that the native library's host code makes, to run that code without a GPU: it keeps
count of the launches, refuses those that need more shared memory than the current device was asked for and those of no threads or
too many, and refuses others on request. Preloaded into a child process, which sees no device."""
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
static const void* fake_f;
int fake_refuse_next;
static int code[2], skip[2], times[2];  /* launches that are refused: [0] ordinary, [1] early */
void fake_set_device(int d) { device = d; }
int fake_asked(void) { return n_asked; }
int fake_launched(void) { return fake_launches; }
const void* fake_last(void) { return fake_f; }
int fake_launched_early(void) { return fake_early; }
void fake_refuse(void) { fake_refuse_next = 1; }
void fake_refuse_launch(int early, int after, int n, int rc) { code[early] = rc; skip[early] = after; times[early] = n; }
void fake_reset(void) { fake_launches = fake_early = last = 0; times[0] = times[1] = 0; }
int fake_pending(void) { return last; }
int cudaGetDevice(int* d) { *d = device; return 0; }
int cudaGetLastError(void) { int e = last; last = 0; return e; }
int cudaDeviceGetAttribute(int* v, int attr, int d) { *v = 148; return 0; }
int cudaFuncSetAttribute(const void* f, int attr, int value) {
  if (fake_refuse_next) { fake_refuse_next = 0; return 999; }
  asked[n_asked].f = f; asked[n_asked].dev = device; asked[n_asked++].bytes = value;
  return 0;
}
static int encode(void) { return 0; }
int cudaGetDriverEntryPoint(const char* name, void** f, unsigned long long flags, int* found) { *f = (void*)encode; *found = 0; return 0; }
static int launch(int early, const void* f, dim3_ g, dim3_ b, size_t smem) {
  int most = 48 << 10, i;
  if (times[early] && skip[early]-- <= 0) { --times[early]; return last = code[early]; }
  for (i = 0; i < n_asked; ++i)
    if (asked[i].f == f && asked[i].dev == device && asked[i].bytes > most) most = asked[i].bytes;
  if (smem > (size_t)most || !g.x || !g.y || !g.z) return last = 1;
  if (!b.x || !b.y || !b.z || b.x * b.y * b.z > 1024) return last = 9;
  ++fake_launches;
  fake_f = f;
  return 0;
}
int cudaLaunchKernel(const void* f, dim3_ g, dim3_ b, void** args, size_t smem, void* stream) { return launch(0, f, g, b, smem); }
int cudaLaunchKernelExC(const config_* c, const void* f, void** args) {
  int rc = launch(1, f, c->grid, c->block, c->smem);
  if (!rc) ++fake_early;
  return rc;
}
"""


def run_with_fake(child: str, tmp_path) -> None:
    """Runs the source ``child`` with the fake's and the library's paths as its arguments; it prints "ok"."""
    lib = build_native.EXT / "libotb_cuda.so"
    if not lib.exists():
        pytest.skip("the CUDA library is not built here")
    (tmp_path / "fake.c").write_text(FAKE)
    fake = tmp_path / "libfake.so"
    cc = "/usr/bin/gcc" if Path("/usr/bin/gcc").exists() else "gcc"
    subprocess.run([cc, "-shared", "-fPIC", "-o", str(fake), str(tmp_path / "fake.c")], check=True)
    r = subprocess.run([sys.executable, "-c", child, str(fake), str(lib)], env=dict(os.environ, LD_PRELOAD=str(fake), CUDA_VISIBLE_DEVICES=""),
                       capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
