"""momms_dgemm_noalloc where the plan steps its tiles by 16 or 8 and splits k: the partial tiles lie
in the fixed scratch (tests/test_f64_plan.py checks their room), the bits are momms_dgemm's."""
import ctypes

import numpy as np
import pytest

import momms_gb300 as mg
from tests import gpu_util as gu
from tests import oracle_util as ou

pytestmark = pytest.mark.gpu


def _call(fn, A_t, B_t, C_t, m, n, k):
    import torch
    one = ctypes.c_double(1.0)
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    return fn(m, n, k, ctypes.byref(one), ctypes.c_void_p(A_t.data_ptr()), A_t.stride(0), A_t.stride(1),
              ctypes.c_void_p(B_t.data_ptr()), B_t.stride(0), B_t.stride(1), ctypes.byref(one),
              ctypes.c_void_p(C_t.data_ptr()), C_t.stride(0), C_t.stride(1), s)


@pytest.mark.parametrize("shape", [(512, 512, 1024), (384, 384, 2048), (256, 256, 4096), (112, 736, 512),
                                   (256, 768, 1600), (250, 252, 4095), (20, 12, 5000), (40, 24, 9001), (8, 8, 30000)])
def test_small_steps_with_splits(gpu, shape):
    import torch
    m, n, k = shape
    rng = np.random.default_rng(m * 7 + n * 3 + k)
    A = np.asfortranarray(rng.uniform(-1, 1, (m, k)))  # m is even: columns start 16-byte aligned
    B = np.asfortranarray(rng.uniform(-1, 1, (k + k % 2, n)))[:k]
    C0 = np.asfortranarray(rng.uniform(-1, 1, (m, n)))
    A_t, B_t, want_t = (gu.to_device(x)[0] for x in (A, B, C0))
    mg.check(_call(gpu.momms_dgemm, A_t, B_t, want_t, m, n, k), gpu)
    torch.cuda.synchronize()
    want = want_t.cpu().numpy()
    exact, mag = ou.dd_gemm(A, B, C0)
    assert ou.bound_ratio(want, exact, mag, k, 2.0**-53) <= 1.0
    for _ in range(2):
        C_t, _, _ = gu.to_device(C0)
        mg.check(_call(gpu.momms_dgemm_noalloc, A_t, B_t, C_t, m, n, k), gpu)
        torch.cuda.synchronize()
        assert np.array_equal(C_t.cpu().numpy(), want)
    bits = ctypes.c_uint32(0)
    assert gpu.momms_noalloc_status(ctypes.byref(bits)) == mg.OK and bits.value == 0
