"""Row strides of the operand planes (whole 32-byte sectors, or 16 bytes under a scratch limit) and
the tile roles of split TF32 change no result."""
import ctypes

import numpy as np
import pytest

import momms_gb300 as mg
from tests import gpu_util as gu
from tests import oracle_util as ou

pytestmark = pytest.mark.gpu


def _operands(rng, m, n, k, dt):
    A = np.asfortranarray(rng.uniform(-1, 1, (m, k)).astype(dt))
    B = np.ascontiguousarray(rng.uniform(-1, 1, (k, n)).astype(dt))
    C0 = rng.uniform(-1, 1, (m, n)).astype(dt)
    return A, B, C0


# k: every remainder of a sector (16 halves, 8 floats) on both sides of a k-block
@pytest.mark.parametrize("mode", [(np.float32, mg.PREC_SPLIT_TF32, 0), (np.float64, mg.PREC_OZAKI, 4),
                                  (np.float64, mg.PREC_OZAKI, 8)], ids=["tf32", "s4", "s8"])
@pytest.mark.parametrize("k", [1, 7, 12, 57, 65, 72, 500, 1020, 1025])
def test_row_strides_give_the_same_bits(gpu, mode, k):
    dt, prec, s = mode
    m, n = 270, 1300
    A, B, C0 = _operands(np.random.default_rng(k), m, n, k, dt)
    C0 = np.asfortranarray(C0)
    want = gu.gemm_device(gpu, A, B, C0, -1.0, 0.5, precision=prec, slices=s)
    ref, mag = ou.dd_gemm(A.astype(np.float64), B.astype(np.float64), C0.astype(np.float64), -1.0, 0.5)
    if dt == np.float64:
        # 4 slices: operands rounded at 2^-33 of a row's or column's maximum
        assert np.all(np.abs(want - ref) <= 2 * (k + 2) * 2.0**-53 * mag + k * 2.0 ** (1 - 8 * s))
    # host operands under a budget that leaves the call no free scratch: 16-byte rows
    gpu.momms_set_staging_budget(300 << 20)
    try:
        got = gu.gemm_host(gpu, A, B, C0.copy(order="F"), -1.0, 0.5, precision=prec, slices=s)
    finally:
        gpu.momms_set_staging_budget(0)
    assert np.array_equal(got, want)
    # one operand packed (its rows are the pack's), the other not
    t, rs, cs = gu.to_device(B)
    pack = ctypes.c_void_p()
    src = mg.Operand(t.data_ptr(), rs, cs, mg.MEM_DEVICE, 0)
    code = mg.DTYPE_F32 if dt == np.float32 else mg.DTYPE_F64
    mg.check(gpu.momms_pack(code, prec, mg.ROLE_B, k, n, ctypes.byref(src), s, None, ctypes.byref(pack)), gpu)
    try:
        ta, ars, acs = gu.to_device(A)
        tc, crs, ccs = gu.to_device(C0)
        d = gu.make_desc(code, m, n, k, -1.0, 0.5, (ta.data_ptr(), ars, acs), (0, 0, 0), (tc.data_ptr(), crs, ccs),
                         precision=prec, slices=s)
        d.b = mg.Operand(pack.value, 0, 0, mg.MEM_PACKED, 0)
        mg.check(gpu.momms_gemm(ctypes.byref(d), None), gpu)
        assert np.array_equal(tc.cpu().numpy(), want)
    finally:
        gpu.momms_packed_destroy(pack)


@pytest.mark.parametrize("shape", [(1, 1, 3), (64, 1000, 40), (1000, 64, 40), (129, 257, 300), (513, 300, 1025)])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_tf32_bits_do_not_depend_on_the_order_of_c(gpu, shape, beta):
    """C by rows runs as C^T = B^T A^T: the same products and sums, whatever C's strides."""
    m, n, k = shape
    A, B, C0 = _operands(np.random.default_rng(m + n + k), m, n, k, np.float32)
    outs = []
    for view in (np.zeros((n, m), np.float32).T, np.zeros((m, n + 3), np.float32)[:, :n],
                 np.zeros((2 * m, 3 * n), np.float32)[::2, ::3], np.zeros((3 * n, 2 * m), np.float32).T[::2, ::3]):
        view[...] = C0
        outs.append(np.array(gu.gemm_device(gpu, A, B, view, 1.5, beta, precision=mg.PREC_SPLIT_TF32)))
    ref, mag = ou.dd_gemm(A.astype(np.float64), B.astype(np.float64), C0.astype(np.float64), 1.5, beta)
    # both operands' splits and the dropped lo*lo term: 3 * 2^-22 of each product
    assert np.all(np.abs(outs[0] - ref) <= (2 * (k + 2) * 2.0**-24 + 3 * 2.0**-22) * mag)
    for o in outs[1:]:
        assert np.array_equal(o, outs[0])


# one and several CTAs per tile (k-blocks of 32 dealt unevenly), tiles of a few rows and columns
@pytest.mark.parametrize("shape", [(1, 1, 33), (3, 5, 300), (130, 258, 4099), (513, 511, 257), (700, 700, 333),
                                   (1500, 1400, 700), (2300, 2100, 100)])
@pytest.mark.parametrize("order", ["F", "C"])
def test_tf32_split_over_a_cluster(gpu, shape, order):
    m, n, k = shape
    A, B, C0 = _operands(np.random.default_rng(m + k), m, n, k, np.float32)
    C = gu.gemm_device(gpu, A, B, np.array(C0, order=order), -1.0, 1.0, precision=mg.PREC_SPLIT_TF32)
    rows = np.unique(np.linspace(0, m - 1, 40).astype(int))
    ref, mag = ou.dd_gemm(A[rows].astype(np.float64), B.astype(np.float64), C0[rows].astype(np.float64), -1.0, 1.0)
    assert np.all(np.abs(C[rows] - ref) <= (2 * (k + 2) * 2.0**-24 + 3 * 2.0**-22) * mag)
