"""Timed cases of the kami_b200 library, each one call (or one training step)
through its public Python entry points.

Kinds of work, and what each stands for:

* ``gemm``   -- ``api.gemm_batched`` once over a batch that is read from HBM:
  the batched GEMM of many small independent blocks (element matrices, block
  preconditioners, batched 16-bit blocks), FP64 or 16-bit inputs;
* ``repeat`` -- ``api.gemm_batched`` with NUM_ITER: every block multiplied many
  times from on-chip storage (the block-GEMM benchmark method);
* ``bmm``    -- forward and backward of the differentiable batched product;
* ``uneven`` -- ``api.GroupedPlan``: thousands of problems of different sizes
  in one launch, the plan kept by the program;
* ``split``  -- ``api.split_f64_gemm``: FP64-accurate products on the tensor
  cores, inputs spread over six decades;
* ``spgemm`` -- ``api.spgemm`` of two block-sparse matrices (16 x 16 tiles),
  structure and values;
* ``spmm``   -- ``api.spmm`` of a block-sparse matrix with a dense one.
"""
import numpy as np
import torch

from kami_b200 import api
from kami_b200.autograd import bmm

DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32, "f64": torch.float64,
          "s8": torch.int8}
SIZE = {"f16": 2, "bf16": 2, "f32": 4, "f64": 8}


def listed():
    return [
        # the smallest batch of the batched FP64 programs: launch latency counts
        {"name": "f64-32-b1024", "kind": "gemm", "dtype": "f64", "out": "f64", "M": 32, "N": 32, "K": 32,
         "batch": 1024},
        # their ordinary large batch, bound by memory and the FP64 pipe
        {"name": "f64-64-b8192", "kind": "gemm", "dtype": "f64", "out": "f64", "M": 64, "N": 64, "K": 64,
         "batch": 8192},
        # large FP64 blocks of ragged size (no compiled block shape covers them)
        {"name": "f64-ragged-b1500", "kind": "gemm", "dtype": "f64", "out": "f64", "M": 121, "N": 91, "K": 110,
         "batch": 1500},
        # 16-bit blocks with FP32 results, one pass over the batch
        {"name": "f16-128-b592", "kind": "gemm", "dtype": "f16", "out": "f32", "M": 128, "N": 128, "K": 128,
         "batch": 592},
        # the library's headline: 128^3 blocks multiplied 1000 times each
        {"name": "f16-128-repeat1000", "kind": "repeat", "dtype": "f16", "out": "f32", "M": 128, "N": 128, "K": 128,
         "batch": 592, "iters": 1000},
        # one training step's batched product: attention-like 64^3 heads
        {"name": "bmm-bf16-64-b4096", "kind": "bmm", "dtype": "bf16", "M": 64, "N": 64, "K": 64, "batch": 4096},
        # the same with sizes that are no power of two
        {"name": "bmm-f16-ragged-b1000", "kind": "bmm", "dtype": "f16", "M": 104, "N": 80, "K": 72, "batch": 1000},
        # uneven batches, sizes log-uniform in 8..128
        {"name": "uneven-f16-20000", "kind": "uneven", "dtype": "f16", "out": "f32", "count": 20000, "lo": 8,
         "hi": 128, "shapes": 0},
        {"name": "uneven-f64-20000", "kind": "uneven", "dtype": "f64", "out": "f64", "count": 20000, "lo": 8,
         "hi": 128, "shapes": 0},
        # FP64-accurate products by digit splitting, seven int8 digits
        {"name": "split-s8x7-64-b8192", "kind": "split", "digits": "s8", "slices": 7, "M": 64, "N": 64, "K": 64,
         "batch": 8192},
        # block SpGEMM of n = 16384 at 1 % of the tiles, from patterns to values
        {"name": "spgemm-16384", "kind": "spgemm", "dtype": "f16", "out": "f32", "blocks": 1024, "per_row": 10.24,
         "pattern": 1},
        # the same A times 256 dense columns
        {"name": "spmm-16384-n256", "kind": "spmm", "dtype": "f16", "out": "f32", "blocks": 1024, "per_row": 10.24,
         "pattern": 1, "N": 256, "layout": "row_kn"},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["gemm", "gemm", "repeat", "bmm", "uneven", "split", "spgemm", "spmm"])
    if kind == "gemm":
        dt = rng.choice(["f64", "f16", "bf16"])
        step = 2 if dt == "f64" else 8
        M, N, K = _log(rng, 8, 128), _log(rng, 8, 128), max(step, _log(rng, 8, 128) // step * step)
        out = "f64" if dt == "f64" else rng.choice(["f32", dt])
        per = (M + N) * K * SIZE[dt] + M * N * SIZE[out]
        return {"kind": kind, "dtype": dt, "out": out, "M": M, "N": N, "K": K,
                "batch": max(16, _log(rng, 1_000_000, 500_000_000) // per)}
    if kind == "repeat":
        n = rng.choice([16, 32, 64, 128])
        K = rng.choice([16, 32, 64, 128]) if n == 128 else n
        return {"kind": kind, "dtype": "f16", "out": "f32", "M": n, "N": n, "K": K, "batch": rng.choice([148, 296, 592]),
                "iters": _log(rng, 50, 1000)}
    if kind == "bmm":
        dt = rng.choice(["bf16", "f16"])
        M, N, K = (8 * _log(rng, 2, 16) for _ in range(3))
        per = 2 * (M * K + K * N + M * N) * SIZE[dt]
        return {"kind": kind, "dtype": dt, "M": M, "N": N, "K": K,
                "batch": max(16, _log(rng, 1_000_000, 300_000_000) // per)}
    if kind == "uneven":
        dt = rng.choice(["f16", "bf16", "f64"])
        return {"kind": kind, "dtype": dt, "out": "f64" if dt == "f64" else "f32", "count": _log(rng, 200, 20000),
                "lo": 8, "hi": rng.choice([48, 64, 96, 128]), "shapes": rng.randrange(1000)}
    if kind == "split":
        digits, slices = rng.choice([("s8", 7), ("s8", 8), ("f16", 6), ("f16", 7)])
        return {"kind": kind, "digits": digits, "slices": slices, "M": _log(rng, 16, 64), "N": _log(rng, 16, 64),
                "K": 2 * _log(rng, 8, 32), "batch": _log(rng, 256, 8192)}
    c = {"kind": kind, "dtype": rng.choice(["f16", "bf16"]), "out": "f32", "blocks": _log(rng, 64, 1024),
         "per_row": round(rng.uniform(2.0, 10.0), 2), "pattern": rng.randrange(1000)}
    if kind == "spmm":
        c["N"] = 8 * _log(rng, 2, 32)
        c["layout"] = rng.choice(["row_kn", "ref_nk"])
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(g, shape, dtype):
    return (torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) * 2 - 1).to(dtype)


def _decades(g, shape):
    """sign * 10^u, u uniform in [-3, 3]"""
    u = torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)
    s = torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)
    return torch.where(s < 0.5, -1.0, 1.0) * 10.0 ** (6 * u - 3)


def _pattern(case, which):
    """Bernoulli block pattern with about per_row entries per block-row:
    row pointers and ascending columns."""
    rng = np.random.default_rng([case["pattern"], which])
    nb = case["blocks"]
    rows, cols = np.nonzero(rng.random((nb, nb)) < case["per_row"] / nb)
    rp = np.zeros(nb + 1, dtype=np.int32)
    np.cumsum(np.bincount(rows, minlength=nb), out=rp[1:])
    return rp, cols.astype(np.int32)


def _shapes(case):
    rng = np.random.default_rng(case["shapes"])
    x = np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"]), (case["count"], 3)))
    return np.clip(8 * np.round(x / 8), 8, case["hi"]).astype(np.int64)


def _operands(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind in ("gemm", "repeat"):
        dt = DTYPES[case["dtype"]]
        return (_uniform(g, (case["batch"], case["M"], case["K"]), dt),
                _uniform(g, (case["batch"], case["N"], case["K"]), dt))
    if kind == "bmm":
        dt = DTYPES[case["dtype"]]
        b, M, N, K = case["batch"], case["M"], case["N"], case["K"]
        return _uniform(g, (b, M, K), dt), _uniform(g, (b, K, N), dt), _uniform(g, (b, M, N), dt)
    if kind == "uneven":
        sh = _shapes(case)
        dt = DTYPES[case["dtype"]]
        return (_uniform(g, (int((sh[:, 0] * sh[:, 2]).sum()),), dt),
                _uniform(g, (int((sh[:, 1] * sh[:, 2]).sum()),), dt))
    if kind == "split":
        return (_decades(g, (case["batch"], case["M"], case["K"])),
                _decades(g, (case["batch"], case["N"], case["K"])))
    dt = DTYPES[case["dtype"]]
    rp, ci = _pattern(case, 0)
    va = _uniform(g, (len(ci), 16, 16), dt)
    n = 16 * case["blocks"]
    if kind == "spmm":
        return rp, ci, va, _uniform(g, (n, case["N"]) if case["layout"] == "row_kn" else (case["N"], n), dt)
    rpb, cib = _pattern(case, 1)
    return rp, ci, va, rpb, cib, _uniform(g, (len(cib), 16, 16), dt)


def _bsr(rp, ci, values, blocks):
    return api.BSR(torch.from_numpy(rp).cuda(), torch.from_numpy(ci).cuda(), values, blocks)


def prepare(case, seed):
    ops = _operands(case, seed)
    kind = case["kind"]
    s = {"case": case}
    if kind in ("gemm", "repeat", "split"):
        s["A"], s["B"] = ops
        s["C"] = torch.empty((case["batch"], case["M"], case["N"]), dtype=DTYPES[case.get("out", "f64")], device="cuda")
    elif kind == "bmm":
        s["A"], s["B"], s["G"] = ops[0].requires_grad_(), ops[1].requires_grad_(), ops[2]
    elif kind == "uneven":
        s["A"], s["B"] = ops
        s["plan"] = api.GroupedPlan(_shapes(case), DTYPES[case["dtype"]], DTYPES[case["out"]])
        s["C"] = torch.empty(s["plan"].sizes[2], dtype=DTYPES[case["out"]], device="cuda")
    elif kind == "spmm":
        s["A"] = _bsr(ops[0], ops[1], ops[2], case["blocks"])
        s["B"] = ops[3]
    else:
        s["A"] = _bsr(ops[0], ops[1], ops[2], case["blocks"])
        s["B"] = _bsr(ops[3], ops[4], ops[5], case["blocks"])
    return s


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "gemm":
        return api.gemm_batched(s["A"], s["B"], s["C"])
    if kind == "repeat":
        return api.gemm_batched(s["A"], s["B"], s["C"], num_iter=c["iters"])
    if kind == "bmm":
        out = bmm(s["A"], s["B"])
        dA, dB = torch.autograd.grad(out, (s["A"], s["B"]), s["G"])
        return out, dA, dB
    if kind == "uneven":
        return s["plan"].run(s["A"], s["B"], s["C"])
    if kind == "split":
        return api.split_f64_gemm(s["A"], s["B"], s["C"], nslices=c["slices"], slice_dtype=DTYPES[c["digits"]])
    if kind == "spmm":
        return api.spmm(s["A"], s["B"], b_layout=c["layout"], out_dtype=DTYPES[c["out"]])
    r = api.spgemm(s["A"], s["B"], DTYPES[c["out"]])
    return r.row_ptr, r.col_idx, r.values


# ---------------------------------------------------------------------------
# least work of one pass
# ---------------------------------------------------------------------------
def _dense_pattern(case, which):
    rp, ci = _pattern(case, which)
    m = np.zeros((case["blocks"], case["blocks"]), dtype=np.float32)
    m[np.repeat(np.arange(case["blocks"]), np.diff(rp)), ci] = 1
    return m


def work(case):
    kind = case["kind"]
    if kind in ("gemm", "repeat", "bmm", "split"):
        b, M, N, K = case["batch"], case["M"], case["N"], case["K"]
        fl = 2 * b * M * N * K
        if kind == "bmm":
            # forward: A, B read, C written; backward: A, B, dC read, dA, dB written
            return {"bytes": b * SIZE[case["dtype"]] * (3 * (M * K + K * N) + 2 * M * N), "flops": 3 * fl}
        dt = case.get("dtype", "f64")
        return {"bytes": b * ((M + N) * K * SIZE[dt] + M * N * SIZE[case.get("out", "f64")]),
                "flops": fl * case.get("iters", 1)}
    if kind == "uneven":
        M, N, K = _shapes(case).T
        return {"bytes": int(((M + N) * K).sum()) * SIZE[case["dtype"]] + int((M * N).sum()) * SIZE[case["out"]],
                "flops": 2 * int((M * N * K).sum())}
    a = _dense_pattern(case, 0)
    nb, nnz = case["blocks"], int(a.sum())
    if kind == "spmm":
        return {"bytes": nnz * (512 + 4) + 16 * nb * case["N"] * (2 + SIZE[case["out"]]),
                "flops": 2 * 256 * nnz * case["N"]}
    b = _dense_pattern(case, 1)
    p = a @ b
    return {"bytes": (nnz + int(b.sum())) * (512 + 4) + 3 * 4 * (nb + 1)
            + int((p > 0).sum()) * (256 * SIZE[case["out"]] + 4), "flops": 2 * 16 ** 3 * int(p.sum())}


# ---------------------------------------------------------------------------
# the same outputs in 64 bits
# ---------------------------------------------------------------------------
def _dense(rp, ci, values, blocks):
    d = torch.zeros((blocks, blocks, 16, 16), dtype=torch.float64, device="cuda")
    rows = torch.from_numpy(np.repeat(np.arange(blocks), np.diff(rp))).cuda()
    d[rows, torch.from_numpy(ci.astype(np.int64)).cuda()] = values.double()
    return d.permute(0, 2, 1, 3).reshape(16 * blocks, 16 * blocks)


def exact(case, seed):
    ops = _operands(case, seed)
    kind = case["kind"]
    if kind in ("gemm", "repeat", "split"):
        A, B = ops
        return torch.bmm(A.double(), B.double().transpose(1, 2)) * case.get("iters", 1)
    if kind == "bmm":
        A, B, G = (x.double() for x in ops)
        return torch.bmm(A, B), torch.bmm(G, B.transpose(1, 2)), torch.bmm(A.transpose(1, 2), G)
    if kind == "uneven":
        A, B = (x.double() for x in ops)
        parts, a, b = [], 0, 0
        for M, N, K in _shapes(case).tolist():
            parts.append((A[a:a + M * K].view(M, K) @ B[b:b + N * K].view(N, K).T).reshape(-1))
            a += M * K
            b += N * K
        return torch.cat(parts)
    nb = case["blocks"]
    A = _dense(*ops[:3], nb)
    if kind == "spmm":
        B = ops[3].double()
        return A @ (B if case["layout"] == "row_kn" else B.T)
    C = (A @ _dense(*ops[3:], nb)).reshape(nb, 16, nb, 16).permute(0, 2, 1, 3)
    rows, cols = np.nonzero(_dense_pattern(case, 0) @ _dense_pattern(case, 1))
    return None, None, C[torch.from_numpy(rows).cuda(), torch.from_numpy(cols).cuda()]
