"""The standalone MLP calls, which hold no object of the library: after a device reset
by the program (in a child process, which ends with it) and from more threads than the
library has status words, each on a stream of its own.  32 rows: one warp adds to the
loss and to each gradient, so the results are the same bits every time."""
import ctypes as C
import glob
import os
import subprocess
import sys
import threading

import pytest

from pmdas_gb300 import _native as N
from pmdas_gb300 import kdgrid as K

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RESET = """
import ctypes as C, sys
import numpy as np
sys.path.insert(0, sys.argv[2])
from pmdas_gb300 import _native as N
lib, rt = N.load(), C.CDLL(sys.argv[1])
rt.cudaMalloc.argtypes = [C.POINTER(C.c_void_p), C.c_size_t]
rt.cudaMemcpy.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_int]

def up(a):
    p = C.c_void_p()
    assert rt.cudaMalloc(C.byref(p), a.nbytes) == 0
    assert rt.cudaMemcpy(p, a.ctypes.data, a.nbytes, 1) == 0
    return p

def down(p, a):
    b = np.empty_like(a)
    assert rt.cudaMemcpy(b.ctypes.data, p, b.nbytes, 2) == 0
    return b

rng = np.random.default_rng(1)
params = (rng.random(N.MLP_PARAMS, dtype=np.float32) - 0.5) * 0.4
x = rng.standard_normal((32, 16)).astype(np.float32)
y = (rng.standard_normal(32) * 0.1).astype(np.float32)
got = []
for again in range(3):
    # small blocks, where allocations of a few bytes made before the reset lay
    marks = [(m, up(m)) for m in (np.full(64, 7 + k, np.uint32) for k in range(200))]
    zeros, pred = np.zeros(N.MLP_PARAMS, np.float32), np.zeros(32, np.float32)
    p, f, t, g, o, m1, m2, loss = up(params), up(x), up(y), up(zeros), up(pred), up(zeros), up(zeros), C.c_float()
    assert lib.mdas_mlp_forward(p, f, 32, o, None) == 0
    assert lib.mdas_mlp_gradients(p, f, t, 32, g, C.byref(loss), None) == 0
    got.append((down(o, pred), loss.value, down(g, zeros)))
    assert lib.mdas_mlp_adam(p, m1, m2, g, 1, 1e-3, None) == 0
    assert all(np.array_equal(down(q, m), m) for m, q in marks)
    assert rt.cudaDeviceReset() == 0
for o, l, g in got[1:]:
    assert np.array_equal(o, got[0][0]) and l == got[0][1] and np.array_equal(g, got[0][2])
print("reset ok")
"""


def test_mlp_calls_after_a_device_reset(cuda):
    found = [p for d in (os.environ.get("CUDA_HOME", "/usr/local/cuda"),)
             for p in glob.glob(os.path.join(d, "lib64", "libcudart.so"))]
    if not found:
        pytest.skip("no shared CUDA runtime to reset the device with")
    r = subprocess.run([sys.executable, "-c", RESET, found[0], ROOT], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "reset ok" in r.stdout, r.stdout + r.stderr


def test_mlp_calls_from_more_threads_than_words(cuda):
    torch = cuda
    gen = torch.Generator().manual_seed(3)
    p = ((torch.rand(N.MLP_PARAMS, generator=gen) * 2 - 1) * 0.2).cuda()
    x = torch.randn(80, 32, 16, generator=gen).cuda()
    y = (torch.randn(80, 32, generator=gen) * 0.1).cuda()
    want = [K.mlp_gradients(p, x[k], y[k]) + (K.mlp_forward(p, x[k]),) for k in range(80)]
    grads, preds = torch.empty(80, N.MLP_PARAMS, device="cuda"), torch.empty(80, 32, device="cuda")
    losses = [[] for _ in range(80)]
    streams = [torch.cuda.Stream() for _ in range(80)]
    torch.cuda.synchronize()
    lib, start = N.load(), threading.Barrier(80)

    def work(k):
        start.wait()
        for _ in range(5):
            loss, s = C.c_float(), streams[k].cuda_stream
            rc = lib.mdas_mlp_gradients(p.data_ptr(), x[k].data_ptr(), y[k].data_ptr(), 32, grads[k].data_ptr(),
                                        C.byref(loss), s)
            rc |= lib.mdas_mlp_forward(p.data_ptr(), x[k].data_ptr(), 32, preds[k].data_ptr(), s)
            losses[k].append((rc, loss.value))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(80)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k, (g, loss, pred) in enumerate(want):
        assert losses[k] == [(0, loss)] * 5
        assert torch.equal(grads[k], g) and torch.equal(preds[k], pred)
