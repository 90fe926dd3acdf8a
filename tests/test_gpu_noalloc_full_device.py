"""After the first uw12c_dgemm_noalloc call of a process on a device, no later one takes
device memory, whatever its layout, tile or split: the first (one tile, no split) is made on
an empty device, the rest with the device filled up, in a process of its own, because kernels
and the fixed array stay loaded.  Products of small integers are exact."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]

SCRIPT = r'''
import ctypes
import torch
import libuw12_b200 as L

LL = ctypes.c_longlong
lib = ctypes.CDLL(str(L.library_path()))
P = ctypes.c_void_p
lib.uw12c_dgemm_noalloc.argtypes = [LL, LL, LL, ctypes.c_double, P, LL, ctypes.c_int, P, LL,
                                    ctypes.c_int, ctypes.c_double, P, LL, LL, LL,
                                    ctypes.POINTER(LL), LL, LL, ctypes.POINTER(LL), ctypes.c_int]
dev = torch.device("cuda")
shapes = [(24, 24, 16, 1), (24, 24, 4096, 0), (200, 200, 64, 0), (320, 320, 320, 0), (130, 16, 50, 0),
          (256, 8, 700, 0), (1024, 1024, 64, 0), (96, 40, 3000, 7), (64, 64, 0, 0)]
A = torch.randint(-3, 4, (1 << 20,), device=dev).double()
B = torch.randint(-3, 4, (1 << 20,), device=dev).double()
C = torch.empty(1 << 20, dtype=torch.float64, device=dev)


def call(m, n, k, split, ak, bn, off):
    lda, ldb = max(1, k if ak else m), max(1, n if bn else k)
    return lib.uw12c_dgemm_noalloc(
        m, n, k, 1.0, P(A.data_ptr() + 8 * off), lda, ak, P(B.data_ptr() + 8 * off), ldb, bn,
        0.0, P(C.data_ptr()), m, 1, 1, (LL * 6)(*[0] * 6), 1, 1, (LL * 4)(*[0] * 4), split)


variants = [(s, ak, bn, off) for s in shapes for ak in (0, 1) for bn in (0, 1) for off in (0, 1)]
want = []
for (m, n, k, s), ak, bn, off in variants:  # and the kernels of torch that the checks need
    a, b = A[off:off + m * k].cpu(), B[off:off + n * k].cpu()
    a = a.view(m, k) if ak else a.view(k, m).T
    b = b.view(k, n) if bn else b.view(n, k).T
    want.append((a @ b).T.contiguous().view(-1))
assert call(*shapes[0], 0, 0, 0) == 0
torch.cuda.synchronize()
fill = []
size = 8 << 30
while size >= 1 << 20 and torch.cuda.mem_get_info()[0] > 8 << 20:  # half of the array's size
    try:
        fill.append(torch.empty(size, dtype=torch.uint8, device=dev))
    except torch.OutOfMemoryError:
        size >>= 1
free0, _ = torch.cuda.mem_get_info()
for ((m, n, k, s), ak, bn, off), w in zip(variants, want):
    st = call(m, n, k, s, ak, bn, off)
    assert st == 0, (m, n, k, s, ak, bn, off, st)
    torch.cuda.synchronize()
    assert torch.equal(C[:m * n].cpu(), w), (m, n, k, s, ak, bn, off)
free1, _ = torch.cuda.mem_get_info()
print("free", free0 >> 20, free1 >> 20)
assert free1 >= free0
print("ok")
'''


def test_later_calls_take_no_device_memory(uw12lib, cuda_device):
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr[-2000:]
