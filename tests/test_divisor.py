"""The library's own host_divisor: its reciprocal against exact integers (on
the CPU), and quotients by its divisors against the hardware's division (on the
GPU), powers of two among them, as a run with DX = 2, 4 or 8 uses."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


class Divisor(C.Structure):
    _fields_ = [("mb", C.c_uint64), ("V", C.c_uint64), ("b", C.c_double), ("eb", C.c_int),
                ("ok", C.c_int)]


def host_divisor(lib):
    f = lib._Z12host_divisord
    f.argtypes = [C.c_double]
    f.restype = Divisor
    return f


def divisors():
    """Powers of two of the whole normal range, their neighbours, grid
    spacings, and significands of every size."""
    b = [2.0 ** e for e in range(-1022, 1024)]
    b += [np.nextafter(x, s) for x in b[::7] for s in (0.0, np.inf)]
    b += [5.0, 1.414, 9.81, 10.0, 20.0, 50.0, 3.0, 60.0, -4.0, -10.0]
    rng = np.random.default_rng(2)
    m = rng.integers(0, 1 << 52, 2000, dtype=np.uint64) >> rng.integers(0, 52, 2000).astype(np.uint64)
    e = rng.integers(1, 2047, 2000).astype(np.uint64)
    b += ((e << np.uint64(52)) | m).view(np.float64).tolist()
    return [float(x) for x in b if np.isfinite(x) and abs(x) >= 2.0 ** -1022]


def test_reciprocal_is_exact(gpu_lib):
    f = host_divisor(gpu_lib)
    for b in divisors():
        d = f(b)
        bits = int(np.float64(b).view(np.uint64))
        mb = (bits & ((1 << 52) - 1)) | (1 << 52)
        assert (d.mb, d.b, d.eb, d.ok) == (mb, b, (bits >> 52) & 0x7ff, 1), b
        assert d.V == min((1 << 116) // mb, (1 << 64) - 1), b
    for b in (0.0, -0.0, 5e-324, float("inf"), float("nan")):
        assert f(b).ok == 0, b


@pytest.mark.gpu
@pytest.mark.parametrize("only_powers", [True, False])
def test_quotients_match_hardware(gpu_lib, tmp_path, only_powers):
    import build as hcbuild
    so = str(tmp_path / "divisor_check.so")
    subprocess.run([hcbuild.nvcc()] + hcbuild.ARCH + hcbuild.NVFLAGS +
                   ["-shared", "-o", so, os.path.join(HERE, "divisor_check.cu")], check=True,
                   capture_output=True)
    f = host_divisor(gpu_lib)
    tab = [f(b) for b in divisors() if not only_powers or np.frexp(b)[0] == 0.5]
    assert len(tab) > 2000
    bad = C.c_uint64(0)
    first = (C.c_double * 4)()
    lib = C.CDLL(so)
    assert lib.divisor_check(C.c_uint64(1 << 28), C.c_uint64(17), (Divisor * len(tab))(*tab),
                             len(tab), C.byref(bad), first) == 0
    assert bad.value == 0, "%d mismatches; first a=%r b=%r got %r want %r" % (
        bad.value, first[0], first[1], first[2], first[3])
