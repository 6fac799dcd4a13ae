"""The f64 kernel at the edges of its 32 x 32 (or 16-stepped) tiles, k-blocks of 16 and k steps
of 4, with operands staged by TMA (16-byte aligned) and by cp.async (any other strides)."""
import ctypes

import numpy as np
import pytest

import momms_gb300 as mg
from tests import gpu_util as gu
from tests import oracle_util as ou

pytestmark = pytest.mark.gpu

U64 = 2.0**-53
SHAPES = [(1, 1, 1), (8, 8, 4), (9, 7, 5), (16, 16, 16), (31, 33, 15), (32, 32, 17), (33, 65, 3), (47, 16, 100),
          (93, 110, 77), (160, 96, 1000), (20, 12, 5000), (513, 290, 67)]


def _operand(rng, rows, cols, layout):
    if layout == "col":
        return np.asfortranarray(rng.uniform(-1, 1, (rows, cols)))
    if layout == "row":
        return rng.uniform(-1, 1, (rows, cols))
    if layout == "odd":  # row-major, rows an odd number of elements apart, odd offset
        return rng.uniform(-1, 1, (rows, (cols + 1) // 2 * 2 + 3))[:, 1:1 + cols]
    return rng.uniform(-1, 1, (2 * rows, 3 * cols))[::2, ::3]  # neither index contiguous


@pytest.mark.parametrize("layouts", ["col col", "odd col", "col odd", "strided odd", "row strided"])
@pytest.mark.parametrize("shape", SHAPES)
def test_tile_edges(gpu, shape, layouts):
    m, n, k = shape
    la, lb = layouts.split()
    rng = np.random.default_rng(m * 1009 + n * 31 + k)
    A, B = _operand(rng, m, k, la), _operand(rng, k, n, lb)
    C0 = np.asfortranarray(rng.uniform(-1, 1, (m, n)))
    C = gu.gemm_device(gpu, A, B, C0, -0.75, 0.5)
    ref, mag = ou.dd_gemm(np.asfortranarray(A), np.asfortranarray(B), C0, alpha=-0.75, beta=0.5)
    assert ou.bound_ratio(C, ref, mag, k, U64) <= 1.0


def test_grouped_mixed_staging_equals_single(gpu):
    """TMA-staged and cp.async-staged problems through the same CTAs' pipelines."""
    import torch
    rng = np.random.default_rng(8)
    count = 40
    descs = (mg.GemmDesc * count)()
    keep, expected = [], []
    for i in range(count):
        m, n, k = (int(x) for x in rng.integers(5, 200, 3))
        la, lb = [("col", "col"), ("odd", "col"), ("col", "odd"), ("strided", "row")][i % 4]
        A, B = _operand(rng, m, k, la), _operand(rng, k, n, lb)
        C0 = np.asfortranarray(rng.uniform(-1, 1, (m, n)))
        expected.append(gu.gemm_device(gpu, A, B, C0))
        ta, tb, tc = (gu.to_device(x) for x in (A, B, C0))
        descs[i] = gu.make_desc(mg.DTYPE_F64, m, n, k, 1.0, 1.0, *((t[0].data_ptr(), t[1], t[2]) for t in (ta, tb, tc)),
                                mem=mg.MEM_DEVICE)
        keep.append((ta, tb, tc))
    mg.check(gpu.momms_gemm_grouped(descs, count, None), gpu)
    torch.cuda.synchronize()
    for i in range(count):
        assert np.array_equal(keep[i][2][0].cpu().numpy(), expected[i]), i
    bits = ctypes.c_uint32(0)
    assert gpu.momms_device_status(ctypes.byref(bits)) == mg.OK and bits.value == 0


@pytest.mark.parametrize("layouts", ["odd odd", "col odd", "odd col", "strided strided"])
@pytest.mark.parametrize("shape", [(1601, 1503, 23), (2003, 997, 49), (407, 3001, 16)])
def test_many_short_units_by_either_staging(gpu, shape, layouts):
    """Several units of one to four k-blocks per CTA: every unit's index travels with its first
    stage, whichever way the stage is filled. The bits are those of 16-byte aligned copies."""
    m, n, k = shape
    la, lb = layouts.split()
    rng = np.random.default_rng(m + n + k)
    A, B = _operand(rng, m, k, la), _operand(rng, k, n, lb)
    C0 = np.asfortranarray(rng.uniform(-1, 1, (m, n)))

    def aligned(x):  # column-major, columns an even number of elements apart
        y = np.zeros((x.shape[0] + x.shape[0] % 2, x.shape[1]), order="F")
        y[:x.shape[0]] = x
        return y[:x.shape[0]]

    want = gu.gemm_device(gpu, aligned(A), aligned(B), C0)
    for _ in range(3):
        assert np.array_equal(gu.gemm_device(gpu, A, B, C0), want)
    ref, mag = ou.dd_gemm(np.asfortranarray(A), np.asfortranarray(B), C0)
    assert ou.bound_ratio(want, ref, mag, k, U64) <= 1.0
