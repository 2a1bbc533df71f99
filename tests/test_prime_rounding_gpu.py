"""Rounding of the direct-product transforms (csrc/prime_pass.cu) against
double precision, for primes over their whole range (both sides of the length
above which the sums run in two halves) and for q p with small and large q: no
larger than that of Bluestein's transforms of the same data, which such axes
take otherwise (odt_fft2c)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _Plan(C.Structure):   # PrimePlan (csrc/prime_pass.cuh)
    _fields_ = [("n", C.c_int), ("q", C.c_int), ("p", C.c_int), ("h", C.c_int), ("kp", C.c_int), ("w", C.c_int),
                ("tw", C.c_void_p), ("tab", C.c_void_p)]


def _direct(x, inverse):
    """Centred 2D transform of x [batch, n, n] on the device by direct products."""
    import torch

    from inverse_solver_b200 import _lib

    lib = _lib.load()
    plan_of = lib["_ZN3odt10prime_planEim"]
    plan_of.restype, plan_of.argtypes = _Plan, [C.c_int, C.c_size_t]
    table = lib["_ZN3odt11prime_tableERKNS_9PrimePlanEPf"]
    table.restype, table.argtypes = None, [C.POINTER(_Plan), C.c_void_p]
    axis = lib["_ZN3odt17launch_prime_axisEP6float2ixbifRKNS_9PrimePlanEP11CUstream_st"]
    axis.restype = C.c_int
    axis.argtypes = [C.c_void_p, C.c_int, C.c_longlong, C.c_bool, C.c_int, C.c_float, C.POINTER(_Plan), C.c_void_p]
    nb, n = x.shape[:2]
    plan = plan_of(n, 227 * 1024)
    assert plan.q * plan.p == n
    tab = np.zeros((2 * plan.h + 1) * plan.kp, np.float32)
    table(C.byref(plan), tab.ctypes.data)
    d_tab = torch.from_numpy(tab).cuda()
    d_tw = torch.from_numpy(np.exp(-2j * np.pi * np.arange(n) / n).astype(np.complex64)).cuda()
    plan.tab, plan.tw = d_tab.data_ptr(), d_tw.data_ptr()
    y = torch.from_numpy(x).cuda()
    sc = 1.0 / n if inverse else 1.0
    torch.cuda.synchronize()
    assert axis(y.data_ptr(), 1, n * nb, inverse, n // 2, sc, C.byref(plan), None) == 0
    assert axis(y.data_ptr(), n, nb, inverse, n // 2, sc, C.byref(plan), None) == 0
    torch.cuda.synchronize()
    return y.cpu().numpy()


def _bluestein(x, inverse):
    from inverse_solver_b200 import _lib

    a, out = _lib.Fft2cArgs(), x.copy()
    a.size[:] = [x.shape[2], x.shape[1], x.shape[0]]
    a.data, a.inverse, a.memory = out.ctypes.data, int(inverse), _lib.ODT_MEM_HOST
    _lib.check(_lib.load().odt_fft2c(C.byref(a)))
    return out


@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("n", [37, 61, 89, 103, 127, 131, 137, 139, 149, 151, 163, 181, 191, 199, 211, 223, 239, 241,
                               251, 2 * 101, 2 * 127, 2 * 151, 3 * 67, 227, 229, 233, 2 * 251, 10 * 37])
def test_direct_products_round_no_worse_than_bluestein(n, inverse):
    rng = np.random.default_rng(n)
    x = (rng.standard_normal((4, n, n)) + 1j * rng.standard_normal((4, n, n))).astype(np.complex64)
    f = np.fft.ifft2 if inverse else np.fft.fft2
    ref = np.fft.fftshift(f(np.fft.ifftshift(x.astype(complex), axes=(1, 2)), axes=(1, 2)), axes=(1, 2))
    e = [np.linalg.norm(y - ref) / np.linalg.norm(ref) for y in (_direct(x, inverse), _bluestein(x, inverse))]
    print("n = %d: direct %.2e, Bluestein %.2e" % (n, *e))
    assert e[0] <= e[1]
