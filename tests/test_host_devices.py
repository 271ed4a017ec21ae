"""Per-device setup on the CPU, against a fake of the CUDA runtime with two
devices: kernel attributes hold for the device that is current when they are
set, so a context on the second device has to set all that the first one did."""
import os
import subprocess
import sys
import textwrap

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIB = os.path.join(ROOT, "linearsolve.jl_gb300", "libgblu.so")

FAKE = r"""
#include <stddef.h>
static int cur = 0, count[2] = {0, 0};
static unsigned long long rec[2][1024][3];
int cudaGetDeviceCount(int *n) { *n = 2; return 0; }
int cudaGetDevice(int *d) { *d = cur; return 0; }
int cudaSetDevice(int d) { cur = d; return 0; }
int cudaGetLastError(void) { return 0; }
int cudaDeviceGetAttribute(int *v, int attr, int device) { (void)device; *v = attr == 16 ? 152 : attr == 97 ? 232448 : 10; return 0; }
int cudaStreamCreateWithFlags(void **s, unsigned f) { (void)f; *s = NULL; return 0; }
int cudaOccupancyMaxActiveClusters(int *n, const void *f, const void *cfg) { (void)f; (void)cfg; *n = 1; return 0; }
int cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *f, int t, size_t b) { (void)f; (void)t; (void)b; *n = 1; return 0; }
int cudaFuncSetAttribute(const void *f, int attr, int value) {
  if (count[cur] < 1024) {
    unsigned long long *r = rec[cur][count[cur]++];
    r[0] = (unsigned long long)f; r[1] = (unsigned long long)attr; r[2] = (unsigned long long)value;
  }
  return 0;
}
int fake_count(int d) { return count[d]; }
unsigned long long fake_rec(int d, int i, int k) { return rec[d][i][k]; }
"""

CHILD = """
import ctypes, sys
fake, lib = ctypes.CDLL(sys.argv[1]), ctypes.CDLL(sys.argv[2])
fake.fake_rec.restype = ctypes.c_uint64
lib.gblu_create.argtypes = [ctypes.c_void_p, ctypes.c_int32, ctypes.c_uint64]
for d in (0, 1):
    h = ctypes.c_void_p()
    assert lib.gblu_create(ctypes.byref(h), d, 0) == 0, d
got = [{tuple(fake.fake_rec(d, i, k) for k in range(3)) for i in range(fake.fake_count(d))} for d in (0, 1)]
assert len(got[0]) > 20, len(got[0])
print(len(got[0]), len(got[1]), len(got[0] ^ got[1]))
"""


def test_second_device_gets_every_kernel_attribute(pkg, tmp_path):
    src, fake = tmp_path / "fake.c", tmp_path / "libfake.so"
    src.write_text(FAKE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(fake), str(src)], check=True)
    r = subprocess.run([sys.executable, "-c", textwrap.dedent(CHILD), str(fake), LIB], capture_output=True, text=True,
                       env=dict(os.environ, LD_PRELOAD=str(fake)))
    assert r.returncode == 0, r.stderr
    first, second, different = map(int, r.stdout.split())
    assert first == second and different == 0, (first, second, different)
