"""A process that works on a second GPU: the kernels that need more shared memory than the default ask for it on every device.
The library's host code runs here against a fake of the few runtime calls involved, launches of both kinds among them, and sees no
device, so no GPU takes part; the fake refuses a launch, as the real calls do, when the current device has not been asked."""
from fake_cudart import run_with_fake

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
assert counts[1] == 2 * counts[0] and counts[3] == counts[1], counts  # once per kernel and device
print("ok")
"""


def test_shared_memory_is_asked_for_on_every_device(tmp_path):
    run_with_fake(CHILD, tmp_path)
