"""The scratch memory of sfg_spread_forces: kept between calls up to a bound, given
back by sfg_release_scratch, shared by threads and streams, left alone while a
stream is being captured, and not carried over a device reset."""
import ctypes as C
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MIB = 1 << 20


class Rings:
    """Marker rings with forces, and the field they are spread onto."""

    def __init__(self, nx, ny, rings, nodes, seed):
        import torch
        rng = np.random.default_rng(seed)
        c = np.stack([rng.uniform(0, nx, rings), rng.uniform(8, ny - 9, rings)], -1)
        th = 2 * np.pi * np.arange(nodes) / nodes
        pos = c[:, None] + 5.0 * np.stack([np.cos(th), np.sin(th)], -1)[None]
        pos[..., 0] %= nx
        self.nx, self.ny, self.rings, self.m = nx, ny, rings, rings * nodes
        dev = dict(device="cuda")
        self.off = torch.arange(rings + 1, dtype=torch.int32, **dev) * nodes
        self.pos = torch.tensor(pos.reshape(-1, 2), **dev)
        self.frc = torch.tensor(rng.normal(0, 1e-3, (self.m, 2)), **dev)
        self.F = torch.zeros((2, ny, nx), dtype=torch.float64, **dev)

    def spread(self, lib, stream):
        p = lambda a: C.c_void_p(a.data_ptr())
        rc = lib.sfg_spread_forces(self.nx, self.ny, self.rings, p(self.off), p(self.pos),
                                   p(self.frc), p(self.F[0]), p(self.F[1]), self.m,
                                   C.c_void_p(stream.cuda_stream))
        assert rc == 0, lib.sfg_last_error()


def test_release_returns_what_a_call_keeps(sfg):
    import torch
    lib, st = sfg.load_library(), torch.cuda.current_stream()
    free = lambda: torch.cuda.mem_get_info()[0]
    small, big = Rings(256, 128, 40, 32, 1), Rings(4096, 4096, 40000, 32, 2)   # 0.1 and 60 MB
    small.spread(lib, st)
    want = small.F.clone()
    assert torch.equal(small.F, want)             # (torch's own memory is in place now)
    torch.cuda.synchronize()
    assert lib.sfg_release_scratch() == 0
    before = free()
    for r in (small, big, small):
        r.F.zero_()
        r.spread(lib, st)
        torch.cuda.synchronize()
        assert before - free() <= 32 * MIB        # the bound, also after a larger call
    assert before - free() > 0                    # (kept: what the pool is for)
    assert lib.sfg_release_scratch() == 0
    assert free() == before
    small.F.zero_()
    small.spread(lib, st)                         # and spreads may follow
    assert torch.equal(small.F, want)
    torch.cuda.synchronize()
    assert lib.sfg_release_scratch() == 0 and lib.sfg_release_scratch() == 0


def test_threads_and_streams_share_it(sfg):
    import torch
    lib = sfg.load_library()
    rings = [Rings(300 + 64 * k, 200, 60 + 20 * k, 40, k) for k in range(4)]
    want = []
    for r in rings:
        r.spread(lib, torch.cuda.current_stream())
        torch.cuda.synchronize()
        want.append(r.F.clone())
    torch.cuda.synchronize()
    fails = []

    def work(r, w):
        try:
            st = torch.cuda.Stream()
            with torch.cuda.stream(st):
                for k in range(30):
                    r.F.zero_()
                    r.spread(lib, st)
                    if k % 7 == 0:
                        assert lib.sfg_release_scratch() == 0
                    assert torch.equal(r.F, w)
        except BaseException as e:
            fails.append(e)

    ts = [threading.Thread(target=work, args=a) for a in zip(rings, want)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not fails, fails


def test_captured_calls_keep_nothing(sfg):
    import torch
    lib = sfg.load_library()
    r = Rings(256, 128, 40, 32, 3)
    r.spread(lib, torch.cuda.current_stream())
    torch.cuda.synchronize()
    want = r.F.clone()
    st, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.stream(st):
        r.F.zero_()
        g.capture_begin(capture_error_mode="thread_local")
        r.spread(lib, st)
        g.capture_end()
    for _ in range(3):
        r.F.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(r.F, want)


# A process of its own: the reset ends this process's context only, with nothing in
# flight.  (The first spread makes the pool, which the reset destroys.)
RESET = """
import sys
sys.path[:0] = [%r, %r]
import ctypes as C, os
import numpy as np, torch
import softflow_b200
from test_gpu_scratch_pool import Rings
lib = softflow_b200.load_library()
cuda = C.CDLL([l.split()[-1] for l in open("/proc/self/maps") if "libcudart" in l][0])
r = Rings(256, 128, 40, 32, 5)
r.spread(lib, torch.cuda.current_stream())
torch.cuda.synchronize()
want = r.F.cpu().numpy()
assert np.abs(want).max() > 0
assert cuda.cudaDeviceReset() == 0
cuda.cudaMalloc.argtypes = [C.POINTER(C.c_void_p), C.c_size_t]
cuda.cudaMemcpy.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_int]
rng = np.random.default_rng(5)
def put(a):
    p = C.c_void_p()
    assert cuda.cudaMalloc(C.byref(p), a.nbytes) == 0
    assert cuda.cudaMemcpy(p, C.c_void_p(a.ctypes.data), a.nbytes, 1) == 0
    return p
c = np.stack([rng.uniform(0, 256, 40), rng.uniform(8, 119, 40)], -1)
th = 2 * np.pi * np.arange(32) / 32
pos = c[:, None] + 5.0 * np.stack([np.cos(th), np.sin(th)], -1)[None]
pos[..., 0] %%= 256
pos = np.ascontiguousarray(pos.reshape(-1, 2))
frc = rng.normal(0, 1e-3, (1280, 2))
F = np.zeros((2, 128, 256))
d = [put(a) for a in (np.arange(41, dtype=np.int32) * 32, pos, frc, F[0], F[1])]
rc = lib.sfg_spread_forces(256, 128, 40, *d, 1280, None)
print("rc", rc, lib.sfg_last_error())
assert rc == 0
for k in (0, 1):
    assert cuda.cudaMemcpy(C.c_void_p(F[k].ctypes.data), d[3 + k], F[k].nbytes, 2) == 0
assert np.array_equal(F, want)
print("same after the reset", flush=True)
os._exit(0)     # (torch's own state belongs to the context that is gone)
"""


def test_device_reset_between_spreads(sfg):
    code = RESET % (ROOT, os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same after the reset" in r.stdout, r.stdout + r.stderr
