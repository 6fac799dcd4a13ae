"""The measured cases: C := beta*C + alpha*A*B through the library's public entry points.

A case names a path ("f64" and "f32": the plain modes, "emu": emulated FP64, "tf32": split TF32),
the sizes, the operands' storage order, where the operands live and the scalars; "batch" is a
captured plan of many uneven problems. Sizes come from the shape sweep, the tests and the benchmark
of this repository: single calls from a few dozen to 8192, batches of problems of 32 to 1024.
"""
import ctypes
import math

import numpy as np
import torch

import momms_gb300 as mg

PRECISION = {"f64": mg.PREC_PLAIN, "f32": mg.PREC_PLAIN, "emu": mg.PREC_OZAKI, "tf32": mg.PREC_SPLIT_TF32}
# batch mixes: probabilities of (plain f64, emulated f64, plain f32)
MIXES = {"half": (0.5, 0.0, 0.5), "served": (0.4, 0.4, 0.2)}


def _single(name, path, m, n, k, **more):
    case = {"name": name, "path": path, "m": m, "n": n, "k": k, "order": "col", "pad": 0, "alpha": 1.0, "beta": 1.0,
            "phi": 0.0, "target": 0.0, "slices": 0, "where": "device"}
    case.update(more)
    return case


def listed():
    return [
        # one small product in a caller's loop: launches and the k chain's latency
        _single("f64_small", "f64", 93, 110, 77),
        # the ordinary square update, column-major
        _single("f64_1024", "f64", 1024, 1024, 1024),
        # odd sizes, row-major operands whose rows are not 16-byte aligned, a subtracting update
        _single("f64_ragged", "f64", 1999, 1501, 2753, order="row", alpha=-1.0),
        # emulated FP64 at the sizes a mixed request stream has
        _single("emu_512", "emu", 512, 512, 512),
        # emulated FP64 on operands with spread exponents, a stated error target, C overwritten
        _single("emu_spread_2048", "emu", 2048, 2048, 2048, phi=2.0, target=1e-14, beta=0.0),
        # the largest square product
        _single("emu_8192", "emu", 8192, 8192, 8192),
        # the trailing update of a blocked factorisation
        _single("emu_rank_256", "emu", 8192, 8192, 256, alpha=-1.0),
        # host-resident operands: copies in, product, copy back
        _single("emu_host_4096", "emu", 4096, 4096, 4096, where="host"),
        # f32: one small product, and a large one
        _single("f32_small", "f32", 256, 300, 200),
        _single("f32_4096", "f32", 4096, 4096, 4096),
        # split TF32 on large odd sizes, row-major, C overwritten
        _single("tf32_ragged", "tf32", 6000, 3001, 4099, order="row", beta=0.0),
        # 512 uneven problems, half f64 and half f32, one captured plan
        {"name": "batch_512", "path": "batch", "count": 512, "mix": "half", "low": 32, "high": 1024, "sizes": 512},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _size(rng, low, high):
    """Log-uniform; half of them rounded to a multiple of 64, the others as they fall."""
    x = _log_int(rng, low, high)
    return max(low, x // 64 * 64) if rng.random() < 0.5 and x >= 128 else x


def draw(rng):
    path = rng.choice(["f64", "f64", "emu", "emu", "emu", "f32", "f32", "tf32", "tf32", "batch"])
    if path == "batch":
        return {"path": "batch", "count": _log_int(rng, 16, 512), "mix": rng.choice(sorted(MIXES)), "low": 32,
                "high": _log_int(rng, 256, 1024), "sizes": rng.randrange(1 << 20)}
    low, high, most = {"f64": (32, 4096, 8.0e9), "emu": (64, 8192, 8192.0**3), "f32": (32, 8192, 6.0e10),
                       "tf32": (64, 8192, 2.0e11)}[path]
    while True:
        m, n, k = (_size(rng, low, high) for _ in range(3))
        if 1.0 * m * n * k <= most:
            break
    case = _single("", path, m, n, k, order=rng.choice(["col", "row", "mixed"]), pad=rng.choice([0, 0, 1, 8]),
                   alpha=rng.choice([1.0, -1.0, 0.5]), beta=rng.choice([1.0, 0.0]))
    del case["name"]
    if path == "emu":
        case["phi"] = rng.choice([0.0, 0.0, 0.5, 2.0, 8.0])
        case["target"] = rng.choice([0.0, 1e-14])
        case["where"] = rng.choice(["device", "device", "packed", "host"])
        if case["where"] == "packed":
            case["phi"], case["slices"] = 0.0, rng.choice([7, 8])
        if case["where"] == "host":
            case["m"], case["n"], case["k"] = (min(x, 4096) for x in (m, n, k))
    return case


def _matrix(rows, cols, by_rows, pad, dtype, gen, phi=0.0):
    """A rows x cols view, one order contiguous, the other's stride `pad` above its least."""
    outer, inner = (rows, cols) if by_rows else (cols, rows)
    x = torch.rand((outer, inner + pad), dtype=dtype, device="cuda", generator=gen)
    if phi:
        x = (x - 0.5) * torch.exp(phi * torch.randn((outer, inner + pad), dtype=dtype, device="cuda", generator=gen))
    else:
        x = x * 2 - 1
    x = x[:, :inner]
    return x if by_rows else x.t()


def _operands(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = torch.float64 if case["path"] in ("f64", "emu") else torch.float32
    by_rows = {"col": (False, False, False), "row": (True, True, True), "mixed": (True, False, False)}[case["order"]]
    m, n, k = case["m"], case["n"], case["k"]
    a = _matrix(m, k, by_rows[0], case["pad"], dtype, gen, case["phi"])
    b = _matrix(k, n, by_rows[1], case["pad"], dtype, gen, case["phi"])
    c = _matrix(m, n, by_rows[2], case["pad"], dtype, gen)
    return a, b, c


def _batch_sizes(case):
    rng = np.random.default_rng(case["sizes"])
    kinds = rng.choice(3, case["count"], p=MIXES[case["mix"]])
    dims = np.exp(rng.uniform(np.log(case["low"]), np.log(case["high"]), (case["count"], 3))).astype(np.int64)
    return [(int(q), *(int(x) for x in d)) for q, d in zip(kinds, dims)]


def _batch_operands(case, seed):
    """Column-major operands of every problem, cut from one f64 and one f32 buffer of each role."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    sizes = _batch_sizes(case)
    buffers, used = {}, {}
    for single in (False, True):
        for role, extent in (("a", lambda m, n, k: m * k), ("b", lambda m, n, k: k * n), ("c", lambda m, n, k: m * n)):
            # every problem starts on a 256-byte boundary
            total = sum(-(-extent(m, n, k) // 64) * 64 for q, m, n, k in sizes if (q == 2) == single)
            dtype = torch.float32 if single else torch.float64
            buffers[role, single] = torch.rand(total, dtype=dtype, device="cuda", generator=gen) * 2 - 1
            used[role, single] = 0
    problems = []
    for q, m, n, k in sizes:
        ops = []
        for role, rows, cols in (("a", m, k), ("b", k, n), ("c", m, n)):
            at = used[role, q == 2]
            ops.append(buffers[role, q == 2][at:at + rows * cols].view(cols, rows).t())
            used[role, q == 2] = at + -(-rows * cols // 64) * 64
        problems.append((q, *ops))
    return problems, buffers


def _operand(x, mem):
    return mg.Operand(x.data_ptr(), x.stride(0), x.stride(1), mem, 0)


def _descriptor(single, precision, a, b, c, alpha, beta, mem, target=0.0, slices=0):
    d = mg.GemmDesc()
    d.dtype = mg.DTYPE_F32 if single else mg.DTYPE_F64
    d.precision = precision
    d.m, d.k = a.shape
    d.n = b.shape[1]
    d.alpha, d.beta = alpha, beta
    d.a, d.b, d.c = _operand(a, mem), _operand(b, mem), _operand(c, mem)
    d.target_rel_err, d.slices = target, slices
    return d


class _Handle:
    """A plan or packed operand of the library, released with the program's last reference to it."""

    def __init__(self, destroy):
        self.value, self.destroy = ctypes.c_void_p(), destroy

    def __del__(self):
        if self.value:
            self.destroy(self.value)


def _pinned(x):
    """A copy in pinned host memory, in the same order."""
    if x.stride(1) == 1:
        return x.contiguous().cpu().pin_memory()
    return x.t().contiguous().cpu().pin_memory().t()


def _prepare_batch(lib, case, seed):
    problems, buffers = _batch_operands(case, seed)
    descs = (mg.GemmDesc * len(problems))()
    for i, (q, a, b, c) in enumerate(problems):
        descs[i] = _descriptor(q == 2, mg.PREC_OZAKI if q == 1 else mg.PREC_PLAIN, a, b, c, 1.0, 1.0, mg.MEM_DEVICE,
                               1e-14 if q == 1 else 0.0)
    plan = _Handle(lib.momms_plan_destroy)
    mg.check(lib.momms_plan_create(descs, len(problems), ctypes.byref(plan.value)), lib)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    mg.check(lib.momms_plan_capture(plan.value, stream), lib)
    return {"lib": lib, "plan": plan, "stream": stream, "keep": buffers,
            "out": {"c64": buffers["c", False], "c32": buffers["c", True]}}


def prepare(case, seed):
    lib = mg.load_library()
    if case["path"] == "batch":
        return _prepare_batch(lib, case, seed)
    a, b, c = _operands(case, seed)
    mem = mg.MEM_DEVICE
    if case["where"] == "host":
        a, b, c = (_pinned(x) for x in (a, b, c))
        mem = mg.MEM_HOST
    d = _descriptor(case["path"] in ("f32", "tf32"), PRECISION[case["path"]], a, b, c, case["alpha"], case["beta"], mem,
                    case["target"], case["slices"])
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    packs = []
    if case["where"] == "packed":
        for role, x in ((mg.ROLE_A, a), (mg.ROLE_B, b)):
            pack = _Handle(lib.momms_packed_destroy)
            mg.check(lib.momms_pack(d.dtype, d.precision, role, x.shape[0], x.shape[1],
                                    ctypes.byref(_operand(x, mg.MEM_DEVICE)), case["slices"], stream,
                                    ctypes.byref(pack.value)), lib)
            packs.append(pack)
        d.a, d.b = (mg.Operand(p.value.value, 0, 0, mg.MEM_PACKED, 0) for p in packs)
    return {"lib": lib, "desc": d, "stream": stream, "keep": (a, b, packs), "out": c}


def run(state):
    lib = state["lib"]
    if "plan" in state:
        mg.check(lib.momms_plan_launch(state["plan"].value, state["stream"]), lib)
    else:
        status = lib.momms_gemm(ctypes.byref(state["desc"]), state["stream"])
        # a target that no slice count reaches still leaves the most exact result in C
        if status != mg.ERR_TARGET_UNREACHABLE:
            mg.check(status, lib)
    return state["out"]


def work(case):
    if case["path"] == "batch":
        sizes = _batch_sizes(case)
        return {"bytes": sum((4 if q == 2 else 8) * (m * k + k * n + 2 * m * n) for q, m, n, k in sizes),
                "flops": sum(2 * m * n * k for _, m, n, k in sizes)}
    m, n, k = case["m"], case["n"], case["k"]
    width = 8 if case["path"] in ("f64", "emu") else 4
    return {"bytes": width * (m * k + k * n + m * n * (2 if case["beta"] else 1)), "flops": 2 * m * n * k}


def _pieces(x, dim):
    """x = x1 + x2 + x3 with x1 and x2 of 19 bits under the largest entry along `dim`: sums of up to
    8192 products of two such pieces have no rounding in 64 bits."""
    top = torch.frexp(x.abs().amax(dim, keepdim=True)).exponent.double()
    out = []
    for bits in (19, 38):
        shift = 1.5 * torch.exp2(top + 52 - bits)
        out.append((x + shift) - shift)
        x = x - out[-1]
    return out + [x]


def _product(a, b):
    """a @ b, rounded about once."""
    if a.dtype == torch.float32:
        return a.double() @ b.double()
    a1, a2, a3 = _pieces(a, 1)
    b1, b2, b3 = _pieces(b, 0)
    r = a2 @ b3 + a3 @ b2
    r += a1 @ b3 + a3 @ b1 + a2 @ b2
    r += a1 @ b2 + a2 @ b1
    return r + a1 @ b1


def exact(case, seed):
    if case["path"] == "batch":
        problems, buffers = _batch_operands(case, seed)
        out = {False: buffers["c", False].clone(), True: buffers["c", True].double()}
        at = {False: 0, True: 0}
        for q, a, b, c in problems:
            part = out[q == 2][at[q == 2]:at[q == 2] + c.numel()]
            part += _product(a, b).t().reshape(-1)
            at[q == 2] += -(-c.numel() // 64) * 64
        return {"c64": out[False], "c32": out[True]}
    a, b, c = _operands(case, seed)
    r = case["alpha"] * _product(a, b)
    return r + case["beta"] * c.double() if case["beta"] else r
