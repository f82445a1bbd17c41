"""What a library on one healthy device does not meet, on the host against a
stand-in for the CUDA runtime (fake_cudart.cpp).

Matrices, problems and densities destroyed while another device is current:
their memory goes back to its own device's pool, after a wait for that device,
and the caller's device stays current.  Blocks of 512 MiB and more are plain
allocations, given back as such.  And a device that refuses a cluster
launch: the plain march is launched in its place."""
import os
import shutil
import subprocess
import sys

import pytest

from fastdose_b200 import _lib

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

CHILD = """
import ctypes as C, sys
fake, kind, own, now = C.CDLL(sys.argv[1]), sys.argv[2], int(sys.argv[3]), int(sys.argv[4])
from fastdose_b200 import _lib
from fastdose_b200.types import make_volume
lib = _lib.get()
ok = lambda rc: _lib.check(rc, "call")

def report():
    v = [C.c_int() for _ in range(4)]
    fake.fake_report(*[C.byref(i) for i in v])
    return [i.value for i in v]

def context(device):
    h = C.c_void_p()
    ok(lib.fd2_context_create(device, C.byref(h)))
    return h

ctx = context(own)
before = report()[0]
zero = (C.c_int64 * 1)(0)

def matrix(cols, vt=0):
    h = C.c_void_p()
    ok(lib.fd2_matrix_create(ctx, 0, cols, 0, zero, None, None, vt, 0, C.byref(h)))
    return h

handles = []
if kind == "density":
    vol = make_volume((2, 2, 2), (0.25,) * 3)
    h = C.c_void_p()
    host = (C.c_float * 8)(*[1.0] * 8)
    ok(lib.fd2_density_create(ctx, host, vol.ctypes.data, C.byref(h)))
    handles.append((lib.fd2_density_destroy, h))
else:
    ms = [matrix(5), matrix(7, 1)]
    if kind == "large":  # its column scales and what finds them are blocks of 560 MB
        ms.append(matrix(140_000_000, 1))
        assert fake.fake_plain_blocks() >= 1, "a large block came from the pool"
    if kind == "problem":
        A, AT = matrix(0), matrix(0)
        f = (C.c_float * 1)()
        h = C.c_void_p()
        ok(lib.fd2_opt_problem_create(ctx, A, AT, A, AT, 0, 0, f, f, f, f, f, 1.0, 1.0, C.byref(h)))
        handles.append((lib.fd2_opt_problem_destroy, h))
        ms += [A, AT]
    handles += [(lib.fd2_matrix_destroy, m) for m in ms]
assert report()[0] > before
other = context(now)
for destroy, h in handles:
    destroy(h)
live, wrong, early, cur = report()
assert wrong == 0, f"{wrong} frees of another device's memory"
assert early == 0, f"{early} frees before the device was waited for"
assert live == before, f"{live - before} allocations left"
assert cur == now, f"device {cur} is current, not {now}"
print("HANDLES OK")
"""

CLUSTER = """
import ctypes as C, sys
import numpy as np
fake, refuse = C.CDLL(sys.argv[1]), int(sys.argv[2])
from fastdose_b200 import _lib, phantoms
from fastdose_b200.types import BEAM_DTYPE
lib = _lib.get()
ok = lambda rc: _lib.check(rc, "call")
ctx, kern = C.c_void_p(), C.c_void_p()
ok(lib.fd2_context_create(0, C.byref(ctx)))
k = phantoms.synthetic_kernel(n_phi=8)
p = lambda a: a.ctypes.data
f = [np.ascontiguousarray(a, np.float32) for a in (k.theta, k.A, k.a, k.B, k.b, k.phi)]
ok(lib.fd2_kernel_create(ctx, len(f[0]), *map(p, f[:5]), len(f[5]), p(f[5]), C.byref(kern)))
b = np.zeros(1, BEAM_DTYPE)
b["beamlet_size"] = 0.3
b["fmap_size"] = int(sys.argv[3])
b["sad"], b["long_spacing"], b["long_dim"] = 100.0, 0.25, 20
b["TermaBEV_pitch"] = b["DensityBEV_pitch"] = 4 * int(sys.argv[3]) ** 2
table = np.zeros(1, np.uint64)

def launches():
    v = [C.c_int(), C.c_int()]
    fake.fake_launches(C.byref(v[0]), C.byref(v[1]))
    return [i.value for i in v]

was = launches()
fake.fake_refuse(refuse)
ok(lib.fd2_dose_compute(ctx, int(sys.argv[3]) ** 2, 1, p(b), p(table), p(table), p(table), kern, None))
plain, cluster = (n - w for n, w in zip(launches(), was))
# the direction table, the march, and the reduction of the zenith bins' planes
assert (plain, cluster) == ((3, 0) if refuse else (2, 1)), (plain, cluster)
print("CLUSTER OK")
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    out = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-I", include, "-o", out, os.path.join(HERE, "fake_cudart.cpp")],
                   check=True)
    return out


@pytest.mark.parametrize("own,now", [(0, 0), (0, 1), (1, 0)])
@pytest.mark.parametrize("kind", ["matrix", "large", "problem", "density"])
def test_handles_return_memory_to_their_own_device(fake, kind, own, now):
    env = dict(os.environ, LD_PRELOAD=fake, PYTHONPATH=ROOT)
    p = subprocess.run([sys.executable, "-c", CHILD, fake, kind, str(own), str(now)], env=env, cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and "HANDLES OK" in p.stdout, p.stdout + p.stderr


@pytest.mark.parametrize("side", [20, 32])
@pytest.mark.parametrize("refuse", [0, 1])
def test_a_refused_cluster_launch_becomes_a_plain_one(fake, refuse, side):
    env = dict(os.environ, LD_PRELOAD=fake, PYTHONPATH=ROOT)
    p = subprocess.run([sys.executable, "-c", CLUSTER, fake, str(refuse), str(side)], env=env, cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and "CLUSTER OK" in p.stdout, p.stdout + p.stderr


def test_the_library_uses_the_shared_runtime():
    """The stand-in replaces the runtime only where it is linked dynamically."""
    out = subprocess.run(["ldd", _lib.LIB_PATH], capture_output=True, text=True, check=True).stdout
    assert "libcudart" in out
