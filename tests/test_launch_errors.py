"""CUDA errors come out of the entry points as errors, whatever their number: the library runs on stand-ins for the runtime's launches.

cudaErrorInvalidValue is 1, a number that is easily taken for an answer of one's own."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# what the entry points below call of the runtime; cudaLaunchKernelExC answers what it was told to
FAKE = r"""
static int made, answer, last;
static int encode(void) { return 0; }
int cudaFuncSetAttribute(const void* f, int a, int v) { return 0; }
int cudaOccupancyMaxActiveClusters(int* n, const void* f, const void* c) { *n = 74; return 0; }
int cudaGetDriverEntryPointByVersion(const char* s, void** p, unsigned v, unsigned long long f, int* q) { *p = (void*)encode; if (q) *q = 0; return 0; }
int cudaGetDriverEntryPoint(const char* s, void** p, unsigned long long f, int* q) { *p = (void*)encode; if (q) *q = 0; return 0; }
int cudaLaunchKernel(const void* f, ...) { return 0; }
int cudaGetLastError(void) { int e = last; last = 0; return e; }
int cudaLaunchKernelExC(const void* c, const void* f, void** a) { made++; return last = answer; }
void fake_answer(int e) { answer = e; made = 0; }
int fake_launches(void) { return made; }
"""

CALLS = """
import ctypes
from jittor_b200 import _capi as C
lib = C.lib

def tensor(dtype, *shape):
    d = C.Tensor()
    d.ptr, d.dtype, d.ndim = 1 << 20, C.DTYPE_CODES[dtype], len(shape)
    for i, s in enumerate(shape):
        d.shape[i] = s
    return d

x, y, w = tensor("bfloat16", 8, 64, 14, 14), tensor("bfloat16", 8, 14, 14, 64), tensor("bfloat16", 64, 64, 3, 3)
scratch, geo = (1 << 20, 1 << 40, None), (1, 1, 1, 1, 1, 1)
calls = {
    "bn_backward": lambda: lib.b200jt_bn_backward(x, x, 4096, 1568.0, 4096, 4096, 1e-5, 0, 4096, x, None),
    "conv2d": lambda: lib.b200jt_conv2d(x, w, x, *geo, 1, 4096, *scratch),
    "conv2d_formats": lambda: lib.b200jt_conv2d_formats(y, w, y, *geo, b"acdb", b"oihw", b"acdb", 4096, *scratch),
    "conv2d_backward_x": lambda: lib.b200jt_conv2d_backward_x(x, w, x, *geo, *scratch),
}
fake = ctypes.CDLL(None)
for name, call in calls.items():
    for error in (0, 1, 9):
        fake.fake_answer(error)
        print(name, error, call(), fake.fake_launches(), fake.cudaGetLastError())
"""


def test_a_failed_launch_is_reported(tmp_path):
    src, so = tmp_path / "fake.c", tmp_path / "fake.so"
    src.write_text(FAKE)
    subprocess.check_call(["gcc", "-shared", "-fPIC", "-w", "-o", str(so), str(src)])
    env = dict(os.environ, LD_PRELOAD=str(so), CUDA_VISIBLE_DEVICES="")
    out = subprocess.run([sys.executable, "-c", CALLS], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    want = [f"{name} {error} {error} 1 0" for name in ("bn_backward", "conv2d", "conv2d_formats", "conv2d_backward_x") for error in (0, 1, 9)]
    assert out.stdout.splitlines() == want               # the error itself, after the one launch that failed; none is left for the next call
