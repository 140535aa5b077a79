"""The work that users of this library have it do, as timed cases: products C = A B of block-sparse FP32 matrices through the
public entry points, from one activation row block to a 16384-deep column shard.

Every case names
  entry      "joint"     esmm_sgemm_joint: B's patterns in hand, A packed and scanned per call
             "row_major" esmm_preprocess_a + esmm_gemm_ab: patterns from the caller, A as it lies, no scratch memory
             "tf32x3"    esmm_sgemm_joint_tf32x3: the tensor-core variant, B split beforehand
             "host"      esmm_plan_run: A comes from and C goes to pinned host memory, B resident
  zeros      "uniform"   the same `pattern` in every 8-wide slice of K, in A's columns and B's rows
             "tiles"     each (gran rows of A x 8-slice) has each of its 8 k live with probability pa; B: gran columns, pb
             "mlp"       A = ReLU activations, the weakest 60 % of (32-row x 8-column) groups zeroed; B = weights pruned to
                         50 % in (8-row x 64-column) groups, by magnitude
  m, n, k    sizes
"""
from __future__ import annotations

import ctypes
import math

import torch

from __graft_entry__ import load_package

UNIFORM = {"11111111": 0xFF, "11110000": 0x0F, "11000000": 0x03, "10000000": 0x01}
MLP_A_LIVE, MLP_B_LIVE = 0.4, 0.5


def _uniform(name, entry, m, n, k, pattern):
    return {"name": name, "entry": entry, "zeros": "uniform", "m": m, "n": n, "k": k, "pattern": pattern}


def _tiles(name, entry, m, n, k, gran, pa, pb):
    return {"name": name, "entry": entry, "zeros": "tiles", "m": m, "n": n, "k": k, "gran": gran, "pa": pa, "pb": pb}


def _mlp(name, entry, m, n, k):
    return {"name": name, "entry": entry, "zeros": "mlp", "m": m, "n": n, "k": k}


def listed():
    return [
        # a small layer: launches, the packing pass and a partly filled GPU count as much as the multiply-adds
        _uniform("square_1024_half", "joint", 1024, 1024, 1024, "11110000"),
        # decoding: 16 token rows through the up-projection of a pruned MLP; latency and the live rows of B
        _mlp("decode_16", "joint", 16, 11008, 4096),
        # the same layer on a prompt of 2048 tokens
        _mlp("prefill_2048", "joint", 2048, 11008, 4096),
        # the density sweep's two ends: no zeros at all, and one k of eight
        _uniform("dense_4096", "joint", 4096, 4096, 4096, "11111111"),
        _uniform("eighth_4096", "joint", 4096, 4096, 4096, "10000000"),
        # A and B pruned independently of one another, in 64-wide tiles and (the pattern's own granularity) in 32-wide ones
        _tiles("tiles_4096_half", "joint", 4096, 4096, 4096, 64, 0.5, 0.5),
        _tiles("blocks_4096_fifth", "joint", 4096, 4096, 4096, 32, 0.2, 0.2),
        # ragged everywhere: no size a multiple of the tile, K not a multiple of the 8-wide slice
        _tiles("ragged_1000", "joint", 1000, 1508, 2012, 32, 0.5, 0.5),
        # one of eight column shards of a 16384^3 product at quarter density: the longest K and the most bytes
        _uniform("shard_16384", "joint", 16384, 2048, 16384, "11000000"),
        # the interface that takes everything from the caller
        _tiles("row_major_2048", "row_major", 2048, 2048, 2048, 64, 0.5, 0.5),
        # the tensor-core variant on the sweep's half-density inputs
        _uniform("tensor_4096_half", "tf32x3", 4096, 4096, 4096, "11110000"),
        # host memory to host memory at quarter density
        _uniform("host_4096_quarter", "host", 4096, 4096, 4096, "11000000"),
    ]


def _log_int(rng, lo, hi, step):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, v // step * step))


def draw(rng):
    entry = rng.choice(["joint"] * 6 + ["row_major", "tf32x3", "tf32x3", "host"])
    while True:
        case = {
            "entry": entry,
            "zeros": rng.choice(["uniform", "tiles", "tiles", "mlp"]),
            "m": _log_int(rng, 1, 4096, 1),
            "n": _log_int(rng, 256, 11008, 4),
            "k": _log_int(rng, 128, 8192, 8 if entry == "tf32x3" else 4),
        }
        if case["zeros"] == "uniform":
            case["pattern"] = rng.choice(sorted(UNIFORM))
        elif case["zeros"] == "tiles":
            case["gran"] = rng.choice([32, 64])
            case["pa"] = round(rng.uniform(0.15, 1.0), 2)
            case["pb"] = round(rng.uniform(0.15, 1.0), 2)
        # at most the work of the dense 4096^3 product
        if case["m"] * case["n"] * case["k"] <= 4096 ** 3:
            return case


# ---- inputs ---------------------------------------------------------------------------------------------------------
def _normal(gen, rows, cols, std=1.0):
    return torch.randn((rows, cols), generator=gen, device="cuda", dtype=torch.float32).mul_(std)


def _up(x, step):
    return -(-x // step) * step


def _matrices(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    m, n, k = case["m"], case["n"], case["k"]
    kp = _up(k, 8)
    if case["zeros"] == "uniform":
        byte = UNIFORM[case["pattern"]]
        live = torch.tensor([(byte >> (i & 7)) & 1 for i in range(k)], dtype=torch.float32, device="cuda")
        a = _normal(gen, m, k).mul_(live[None, :])
        b = _normal(gen, k, n).mul_(live[:, None])
        return a, b
    if case["zeros"] == "tiles":
        g = case["gran"]
        mp, np_ = _up(m, g), _up(n, g)
        a, b = _normal(gen, mp, kp), _normal(gen, kp, np_)
        la = torch.rand((mp // g, 1, kp), generator=gen, device="cuda") < case["pa"]
        lb = torch.rand((kp, np_ // g, 1), generator=gen, device="cuda") < case["pb"]
        a.view(mp // g, g, kp).mul_(la)
        b.view(kp, np_ // g, g).mul_(lb)
        return a[:m, :k].contiguous(), b[:k, :n].contiguous()
    mp, np_ = _up(m, 32), _up(n, 64)
    a = _normal(gen, mp, kp).relu_()
    a[m:].zero_()
    b = _normal(gen, kp, np_, 0.02)
    b[k:].zero_()
    norm_a = a.view(mp // 32, 32, kp // 8, 8).sum(dim=(1, 3))
    norm_b = b.view(kp // 8, 8, np_ // 64, 64).abs().sum(dim=(1, 3))
    keep_a = norm_a >= norm_a.flatten().kthvalue(max(1, round((1 - MLP_A_LIVE) * norm_a.numel()))).values
    keep_b = norm_b >= norm_b.flatten().kthvalue(max(1, round((1 - MLP_B_LIVE) * norm_b.numel()))).values
    a.view(mp // 32, 32, kp // 8, 8).mul_(keep_a[:, None, :, None])
    b.view(kp // 8, 8, np_ // 64, 64).mul_(keep_b[:, None, :, None])
    return a[:m, :k].contiguous(), b[:k, :n].contiguous()


class _HostPlan:
    """A host-buffer plan (B and its patterns on the GPU) and the pinned matrices of its caller."""

    def __init__(self, pkg, a, b):
        self.pkg, self.handle = pkg, ctypes.c_void_p()
        m, k = a.shape
        n = b.shape[1]
        h_b = b.cpu()
        self.a = torch.empty((m, k), dtype=torch.float32, pin_memory=True)
        self.a.copy_(a)
        self.c = torch.empty((m, n), dtype=torch.float32, pin_memory=True)
        pkg.check(pkg.lib().esmm_plan_create(m, n, k, h_b.data_ptr(), 8, ctypes.byref(self.handle)), "esmm_plan_create")

    def __del__(self):
        if self.handle:
            self.pkg.lib().esmm_plan_destroy(self.handle)


def prepare(case, seed):
    pkg = load_package()
    m, n, k = case["m"], case["n"], case["k"]
    a, b = _matrices(case, seed)
    s = {"pkg": pkg, "entry": case["entry"], "m": m, "n": n, "k": k}
    if case["entry"] == "host":
        torch.cuda.current_stream().synchronize()
        s["plan"] = _HostPlan(pkg, a, b)
        return s
    s["a"], s["b"] = a, b
    s["c"] = torch.empty((m, n), dtype=torch.float32, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    if case["entry"] == "tf32x3":
        torch.cuda.current_stream().synchronize()
        s["b_handle"] = pkg.Tf32x3B(b.data_ptr(), k, n)
        s["ws"] = torch.empty(pkg.tf32x3_workspace_bytes(m, k), dtype=torch.uint8, device="cuda")
        return s
    s["b_pat"] = torch.empty((-(-n // 32), -(-k // 8)), dtype=torch.uint8, device="cuda")
    pkg.preprocess_b(b.data_ptr(), k, n, s["b_pat"].data_ptr(), stream)
    if case["entry"] == "row_major":
        s["a_pat"] = torch.empty((-(-m // 32), -(-k // 8)), dtype=torch.uint8, device="cuda")
    else:
        s["ws"] = torch.empty(pkg.sgemm_joint_workspace_bytes(m, k), dtype=torch.uint8, device="cuda")
    return s


def run(s):
    pkg, m, n, k = s["pkg"], s["m"], s["n"], s["k"]
    if s["entry"] == "host":
        plan = s["plan"]
        pkg.check(pkg.lib().esmm_plan_run(plan.handle, plan.a.data_ptr(), plan.c.data_ptr()), "esmm_plan_run")
        return plan.c
    stream = torch.cuda.current_stream().cuda_stream
    a, b, c = s["a"].data_ptr(), s["b"].data_ptr(), s["c"].data_ptr()
    if s["entry"] == "joint":
        pkg.sgemm_joint(m, n, k, a, b, c, s["b_pat"].data_ptr(), s["ws"].data_ptr(), stream)
        return s["c"]
    if s["entry"] == "tf32x3":
        pkg.sgemm_joint_tf32x3(m, a, s["b_handle"], c, s["ws"].data_ptr(), stream)
        return s["c"]
    pkg.preprocess_a(a, m, k, s["a_pat"].data_ptr(), 32, stream)
    pkg.gemm_ab(m, n, k, a, b, c, s["a_pat"].data_ptr(), s["b_pat"].data_ptr(), 32, stream)
    return s["c"], s["a_pat"]


# ---- what a pass cannot do without --------------------------------------------------------------------------------------
def _densities(case):
    if case["zeros"] == "uniform":
        d = case["pattern"].count("1") / 8
        return d, d, d
    if case["zeros"] == "tiles":
        return case["pa"], case["pb"], case["pa"] * case["pb"]
    return MLP_A_LIVE, MLP_B_LIVE, MLP_A_LIVE * MLP_B_LIVE


def work(case):
    m, n, k = case["m"], case["n"], case["k"]
    da, db, joint = _densities(case)
    # A is read whole (where it is zero is found out in the pass), C written whole; of B the 32-column pieces of rows that
    # some row block of A has a live k for
    if case["zeros"] == "uniform":
        b_used = db
    else:
        gran = case.get("gran", 32)
        b_used = db * (1.0 - (1.0 - da) ** -(-m // gran))
    return {"bytes": 4.0 * (m * k + b_used * k * n + m * n), "flops": 2.0 * m * n * k * joint}


def tolerance(case):
    # 2-norm errors against the product in 64 bits, times about four.  One FP32 multiply-add chain over L live k: 4.1e-7
    # (L = 512), 1.1e-6 (4096), 1.6e-6 (8192), that is about 1.8e-8 sqrt(L).  The tensor-core variant adds the rounding
    # of its operands' low parts and of its accumulation runs: up to 1.8e-6 at every K.
    if case["entry"] == "tf32x3":
        return {"rel": 7e-6}
    live = case["k"] * _densities(case)[2]
    return {"rel": max(4e-7, 8e-8 * math.sqrt(live))}
