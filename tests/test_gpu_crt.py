"""The residue form of the emulated product on the GPU: the result is the exact integer product
rounded once, so it is within half an ulp (and alpha, beta) of the double-double oracle, over tile
and chunk edges, layouts, slice counts, passes under a scratch limit, and packed operands."""
import ctypes

import numpy as np
import pytest

import momms_gb300 as mg
from tests import gpu_util as gu
from tests import oracle_util as ou

pytestmark = pytest.mark.gpu


def _call(gpu, A, B, C0, s, alpha=1.0, beta=0.0):
    C = gu.gemm_device(gpu, A, B, C0, alpha, beta, precision=mg.PREC_OZAKI, slices=s)
    info = mg.CallInfo()
    gpu.momms_last_info(ctypes.byref(info))
    return C, info


# one and several TMEM chunks (16 k-blocks of 64), tile remainders in m and n, row and column quads
@pytest.mark.parametrize("shape", [(2049, 2050, 1024), (1300, 1027, 1025), (1153, 1281, 4001), (2049, 770, 1700)])
@pytest.mark.parametrize("s", [10, 12, 15])
def test_within_an_ulp_of_the_exact_product(gpu, shape, s):
    m, n, k = shape
    rng = np.random.default_rng(m + n + k + s)
    A = np.asfortranarray(rng.uniform(-1, 1, (m, k)))
    B = rng.uniform(-1, 1, (k, n))
    C, info = _call(gpu, A, B, np.zeros((m, n), order="F"), s)
    assert info.pairs < s * (s + 1) // 2  # the residue form ran
    rows = rng.choice(m, 24, replace=False)
    ref, mag = ou.dd_gemm(np.asfortranarray(A[rows]), np.asfortranarray(B), np.zeros((24, n), order="F"), 1.0, 0.0)
    # operands rounded at 2^-(8s+1) of their row or column maximum, one rounding of the product
    tol = 2.0**-53 * np.abs(ref) * 1.01 + k * 2.0 ** (-8 * s) * 1.01 + 2.0**-100 * mag
    assert np.all(np.abs(C[rows] - ref) <= tol)


def test_passes_and_packs_give_the_same_bits(gpu):
    """Streamed blocks (which hold their scratch to the digit form's by passes over the moduli)
    and packed operands (residues taken from their digits) against the plain call."""
    m, n, k, s = 2100, 1900, 2300, 8
    rng = np.random.default_rng(11)
    A = np.asfortranarray(rng.uniform(-1, 1, (m, k)))
    B = np.asfortranarray(rng.uniform(-1, 1, (k, n)))
    C0 = np.asfortranarray(rng.uniform(-1, 1, (m, n)))
    want, info = _call(gpu, A, B, C0, s, -1.0, 1.0)
    assert info.pairs < 36
    gpu.momms_set_staging_budget(300 << 20)  # 1280 x 1024 blocks of the whole k
    try:
        got = gu.gemm_host(gpu, A, B, C0.copy(order="F"), -1.0, 1.0, precision=mg.PREC_OZAKI, slices=s)
    finally:
        gpu.momms_set_staging_budget(0)
    assert np.array_equal(got, want)
    packs = []
    for role, x in ((mg.ROLE_A, A), (mg.ROLE_B, B)):
        t, rs, cs = gu.to_device(x)
        h = ctypes.c_void_p()
        src = mg.Operand(t.data_ptr(), rs, cs, mg.MEM_DEVICE, 0)
        mg.check(gpu.momms_pack(mg.DTYPE_F64, mg.PREC_OZAKI, role, *x.shape, ctypes.byref(src), s, None, ctypes.byref(h)), gpu)
        packs.append(h)
    tc, rs, cs = gu.to_device(C0)
    d = gu.make_desc(mg.DTYPE_F64, m, n, k, -1.0, 1.0, (0, 0, 0), (0, 0, 0), (tc.data_ptr(), rs, cs),
                     precision=mg.PREC_OZAKI, mem=mg.MEM_DEVICE, slices=s)
    d.a, d.b = (mg.Operand(h.value, 0, 0, mg.MEM_PACKED, 0) for h in packs)
    mg.check(gpu.momms_gemm(ctypes.byref(d), None), gpu)
    import torch
    torch.cuda.synchronize()
    assert np.array_equal(tc.cpu().numpy(), want)
    for h in packs:
        mg.check(gpu.momms_packed_destroy(h), gpu)
    bits = ctypes.c_uint32(0)
    assert gpu.momms_device_status(ctypes.byref(bits)) == mg.OK and bits.value == 0


@pytest.mark.parametrize("s", [5, 7, 9, 10, 11, 15])
def test_residues_of_packed_digits(gpu, s):
    """Digits are combined in pairs before they meet the moduli: the bits of the plain call, with
    entries whose digits are all at either end of their range among them."""
    m, n, k = 520, 700, 333
    rng = np.random.default_rng(s)
    ends = np.array([sum(d * 256.0 ** -(i + 1) for i in range(6)) for d in (127, 128, -127, -128)])
    ops = []
    for shape in ((m, k), (k, n)):
        x = rng.uniform(-1, 1, shape) * 0.49
        x[rng.uniform(size=shape) < 0.3] = rng.choice(ends)
        ops.append(np.asfortranarray(x))
    A, B = ops
    want, info = _call(gpu, A, B, np.zeros((m, n), order="F"), s)
    assert info.pairs < s * (s + 1) // 2 or s == 5
    packs = []
    for role, x in ((mg.ROLE_A, A), (mg.ROLE_B, B)):
        t, rs, cs = gu.to_device(x)
        h = ctypes.c_void_p()
        mg.check(gpu.momms_pack(mg.DTYPE_F64, mg.PREC_OZAKI, role, x.shape[0], x.shape[1],
                                ctypes.byref(mg.Operand(t.data_ptr(), rs, cs, mg.MEM_DEVICE, 0)), s, None,
                                ctypes.byref(h)), gpu)
        packs.append(h)
    try:
        for use in ((True, True), (True, False), (False, True)):
            tc, crs, ccs = gu.to_device(np.zeros((m, n), order="F"))
            dev = [gu.to_device(x) for x in (A, B)]
            d = gu.make_desc(mg.DTYPE_F64, m, n, k, 1.0, 0.0, (dev[0][0].data_ptr(),) + dev[0][1:],
                             (dev[1][0].data_ptr(),) + dev[1][1:], (tc.data_ptr(), crs, ccs),
                             precision=mg.PREC_OZAKI, slices=s)
            if use[0]:
                d.a = mg.Operand(packs[0].value, 0, 0, mg.MEM_PACKED, 0)
            if use[1]:
                d.b = mg.Operand(packs[1].value, 0, 0, mg.MEM_PACKED, 0)
            mg.check(gpu.momms_gemm(ctypes.byref(d), None), gpu)
            assert np.array_equal(tc.cpu().numpy(), want)
    finally:
        for h in packs:
            gpu.momms_packed_destroy(h)


def _pack(gpu, role, x, s):
    t, rs, cs = gu.to_device(x)
    h = ctypes.c_void_p()
    mg.check(gpu.momms_pack(mg.DTYPE_F64, mg.PREC_OZAKI, role, x.shape[0], x.shape[1],
                            ctypes.byref(mg.Operand(t.data_ptr(), rs, cs, mg.MEM_DEVICE, 0)), s, None, ctypes.byref(h)), gpu)
    return h


def _packed_call(gpu, packs, A, B, C0, s):
    """C0 + A B with the operands of `packs` (None: unpacked)."""
    import torch
    m, n, k = A.shape[0], B.shape[1], A.shape[1]
    (ta, *sa), (tb, *sb), (tc, *sc) = (gu.to_device(x) for x in (A, B, C0))
    d = gu.make_desc(mg.DTYPE_F64, m, n, k, 1.0, 1.0, (ta.data_ptr(), *sa), (tb.data_ptr(), *sb), (tc.data_ptr(), *sc),
                     precision=mg.PREC_OZAKI, mem=mg.MEM_DEVICE, slices=s)
    if packs[0]:
        d.a = mg.Operand(packs[0].value, 0, 0, mg.MEM_PACKED, 0)
    if packs[1]:
        d.b = mg.Operand(packs[1].value, 0, 0, mg.MEM_PACKED, 0)
    mg.check(gpu.momms_gemm(ctypes.byref(d), None), gpu)
    info = mg.CallInfo()
    gpu.momms_last_info(ctypes.byref(info))
    torch.cuda.synchronize()
    return tc.cpu().numpy(), info


@pytest.mark.parametrize("which", ["none", "a", "b", "ab"])
def test_without_room_for_more_scratch(gpu, monkeypatch, which):
    """Where the device has no room beyond the digit form's scratch: the same bits in more passes;
    from packs, whose digits are there, the digit form."""
    m, n, k, s = 1300, 1027, 1025, 7
    rng = np.random.default_rng(77)
    A = np.asfortranarray(rng.uniform(-1, 1, (m, k)))
    B = np.asfortranarray(rng.uniform(-1, 1, (k, n)))
    C0 = np.zeros((m, n), order="F")
    packs = [_pack(gpu, mg.ROLE_A, A, s) if "a" in which.replace("none", "") else None,
             _pack(gpu, mg.ROLE_B, B, s) if "b" in which else None]
    try:
        want, info = _packed_call(gpu, packs, A, B, C0, s)
        assert info.pairs < s * (s + 1) // 2
        monkeypatch.setenv("MOMMS_FREE_SCRATCH", "0")
        got, info = _packed_call(gpu, packs, A, B, C0, s)
    finally:
        for h in packs:
            if h:
                mg.check(gpu.momms_packed_destroy(h), gpu)
    if which == "none":
        assert info.pairs < s * (s + 1) // 2 and np.array_equal(got, want)
        return
    assert info.pairs == s * (s + 1) // 2
    # digits rounded at 2^-(8s+1), the diagonals past s + 1 left out, one rounding
    ref, _ = ou.dd_gemm(A, B, C0)
    assert np.all(np.abs(got - ref) <= 1.01 * (2.0**-53 * np.abs(ref) + 2.0 ** (-8 * s - 1) * k * (2 + (s - 1) / 2)))
