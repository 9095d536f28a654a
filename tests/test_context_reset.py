"""The library after the process's CUDA context has been replaced (cudaDeviceReset): what it sets per context and
kernel (shared memory limits, cluster sizes) is set again. Runs in a process of its own, without torch's allocator."""
import glob
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - collected on CPU boxes, skipped
    pytest.skip("CUDA device required", allow_module_level=True)

ROOT = Path(__file__).resolve().parents[1]

CHILD = r"""
import ctypes as C, sys
import numpy as np
lib, rt = C.CDLL(sys.argv[1]), C.CDLL(sys.argv[2])

def device(a):
    p = C.c_void_p()
    assert rt.cudaMalloc(C.byref(p), C.c_size_t(a.nbytes)) == 0
    assert rt.cudaMemcpy(p, a.ctypes.data_as(C.c_void_p), C.c_size_t(a.nbytes), 1) == 0
    return p

def host(p, shape):
    a = np.empty(shape)
    assert rt.cudaMemcpy(a.ctypes.data_as(C.c_void_p), p, C.c_size_t(a.nbytes), 2) == 0
    return a

def calls():
    rng, n, out = np.random.default_rng(0), 16, []
    off = np.array([[x, y, z] for z in (-2, 0, 2) for y in (-1, 0, 1) for x in (-3, 0, 1)], np.int32)
    x, y = device(rng.uniform(0.1, 0.9, n ** 3)), device(np.zeros(n ** 3))
    assert lib.pgj_cone_filter(n, device(off), device(np.ones(len(off))), len(off), x, y, None) == 0
    out.append(host(y, n ** 3))
    f = [device(rng.uniform(0.1, 0.9, n ** 3)) for _ in range(3)]
    m, change, d = 64, C.c_double(), C.c_double
    big = [device(rng.uniform(0.1, 0.9, m ** 3)) for _ in range(4)]
    w = np.exp(-np.linspace(-2, 2, 121) ** 2)
    new, scratch = device(np.zeros(m ** 3)), device(np.zeros(4 * m ** 3 + 512))
    assert lib.pgj_study1_oc(m, device(w / w.sum()), 60, *big, d(2.0), d(0.3), d(0.1), new, scratch, C.byref(change), None) == 0
    out.append(host(new, m ** 3))
    for n, prec in ((16, 0), (24, 1), (64, 0), (64, 1)):
        size, ctx = C.c_size_t(), C.c_void_p()
        assert lib.pgj_workspace_bytes(n, 1, prec, C.byref(size)) == 0
        ws = C.c_void_p()
        assert rt.cudaMalloc(C.byref(ws), size) == 0
        assert lib.pgj_ctx_create(n, 1, prec, d(0.5), d(0.5), ws, size, None, C.byref(ctx)) == 0
        assert lib.pgj_set_material(ctx, device(rng.uniform(0.5, 1.0, n ** 3)), None) == 0
        assert lib.pgj_set_alpha(ctx, d(0.5), None) == 0
        u, macro, info = device(np.zeros(3 * n ** 3)), np.eye(6)[0].copy(), (C.c_char * 64)()
        assert lib.pgj_solve(ctx, 1, macro.ctypes.data_as(C.c_void_p), d(1e-8), u, info, None) == 0
        out.append(host(u, 3 * n ** 3))
        assert lib.pgj_ctx_destroy(ctx) == 0
    return out

first = calls()
assert rt.cudaDeviceReset() == 0
assert all(np.array_equal(a, b) for a, b in zip(first, calls()))
print("same")
"""


def test_calls_after_a_device_reset(pkg):
    places = [os.path.join(os.path.dirname(torch.__file__), "..", "nvidia", "cuda_runtime", "lib", "libcudart.so.*"),
              "/usr/local/cuda/lib64/libcudart.so.*"]
    found = [f for p in places for f in sorted(glob.glob(p))]
    if not found:
        pytest.skip("no CUDA runtime library")
    lib = ROOT / "partial-green-jacobi_b200" / "libpgj.so"
    res = subprocess.run([sys.executable, "-c", CHILD, str(lib), found[0]], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0 and res.stdout.strip() == "same", res.stderr[-2000:]
