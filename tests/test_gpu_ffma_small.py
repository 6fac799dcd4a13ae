"""The f32 kernel of small products (32 x 32 tiles): the same bits as the 128 x 128 tile, which a
grouped launch of the same problem runs, over tile and stage edges, layouts, alignments, splits."""
import ctypes

import numpy as np
import pytest

import momms_gb300 as mg
from tests import gpu_util as gu
from tests import oracle_util as ou

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (32, 32, 32), (33, 31, 33), (64, 40, 127), (100, 257, 16), (250, 300, 200), (31, 64, 5000)]


def _operand(rng, rows, cols, layout):
    if layout == "col":
        return np.asfortranarray(rng.uniform(-1, 1, (rows, cols)).astype(np.float32))
    if layout == "row":
        return rng.uniform(-1, 1, (rows, cols)).astype(np.float32)
    return rng.uniform(-1, 1, (rows, cols + 6)).astype(np.float32)[:, 1:1 + cols]  # unaligned rows


@pytest.mark.parametrize("layouts", ["col col", "row col", "col row", "row row", "odd odd"])
@pytest.mark.parametrize("shape", SHAPES)
def test_same_bits_as_the_large_tile(gpu, shape, layouts):
    import torch
    m, n, k = shape
    la, lb = layouts.split()
    rng = np.random.default_rng(m * 7 + n * 131 + k)
    A, B = _operand(rng, m, k, la), _operand(rng, k, n, lb)
    C0 = np.asfortranarray(rng.uniform(-1, 1, (m, n)).astype(np.float32))
    C = gu.gemm_device(gpu, A, B, C0, -0.75, 0.5)
    ref, mag = ou.dd_gemm(np.asfortranarray(A), np.asfortranarray(B), C0, alpha=-0.75, beta=0.5)
    assert ou.bound_ratio(C, ref, mag, k, 2.0**-24) <= 1.0
    ops = [gu.to_device(x) for x in (A, B, C0)]
    d = (mg.GemmDesc * 1)(gu.make_desc(mg.DTYPE_F32, m, n, k, -0.75, 0.5, *((t.data_ptr(), rs, cs) for t, rs, cs in ops),
                                       mem=mg.MEM_DEVICE))
    mg.check(gpu.momms_gemm_grouped(d, 1, None), gpu)
    torch.cuda.synchronize()
    assert np.array_equal(ops[2][0].cpu().numpy(), C)
    bits = ctypes.c_uint32(0)
    assert gpu.momms_device_status(ctypes.byref(bits)) == mg.OK and bits.value == 0
