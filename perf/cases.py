"""Measured workloads of the BN254 G1 MSM library, through its C ABI binding.

Every pass goes from scalars to finished commitments: the MSM call a program
makes, then msm_b200_final_sum_async on its 254 partial results, which gives
one canonical affine point per MSM (standard form, fully reduced).  The
partial results themselves are Jacobian points whose coordinates depend on the
order of the additions, so the canonical point is what two correct builds have
in common, bit for bit.

A case is one call path:
  plain    msm_execute_async (2^k points) or msm_b200_execute_async (any
           count); scalars on the device or in page-locked host memory
  noalloc  msm_b200_execute_no_alloc_async (device buffers, up to 65,536 points)
  batch    msm_b200_batch_execute_async: a fixed list of MSMs over prefixes of
           one resident base table, then one final sum per MSM on side streams
  serve    msm_b200_server_submit for a burst of requests, wait for all, final
           sums on side streams; a request/response program, so a pass ends
           when its points are there
Scalars are uniform below r, or "skewed" as a prover's witness columns are:
40 % zeros, 20 % ones, 20 % below 2^16, the rest uniform, shuffled.
"""
import functools
import math
import os
import random
import sys

import numpy as np
import torch

PACKAGE = os.path.abspath("era-bellman-cuda_b200")
if PACKAGE not in sys.path:
    sys.path.insert(0, PACKAGE)

P = 0x30644E72E131A029B85045B68181585D97816A916871CA8D3C208C16D87CFD47
R = 0x30644E72E131A029B85045B68181585D2833E84879B9709143E1F593F0000001
TOP_LIMB = 0x30644E72  # of r: a smaller top limb makes any eight limbs a value below r
RESULT_BYTES = 254 * 96
POINT_WORDS = 20  # msm_b200_affine_point: x[8], y[8], infinity, reserved[3]
TABLE_POINTS = 1 << 18
SERVER_BUDGET = 2 << 30
SIDE_STREAMS = 8


def listed():
    return [
        # the smallest calls: a verifier's or a lookup argument's few hundred points; launches and dependent chains
        {"name": "plain_2e8", "path": "plain", "n": 1 << 8, "scalars": "uniform", "memory": "device"},
        # the small end of a prover's commitments (the benchmark's 2^12 config)
        {"name": "plain_2e12", "path": "plain", "n": 1 << 12, "scalars": "uniform", "memory": "device"},
        # a caller that may not allocate, a ragged count below its limit
        {"name": "noalloc_30000", "path": "noalloc", "n": 30000, "scalars": "uniform", "memory": "device"},
        # a witness column straight from the host
        {"name": "host_2e16_skewed", "path": "plain", "n": 1 << 16, "scalars": "skewed", "memory": "pinned"},
        # a ragged witness column on the device
        {"name": "ragged_200003_skewed", "path": "plain", "n": 200003, "scalars": "skewed", "memory": "device"},
        # a mid-size quotient or opening polynomial
        {"name": "plain_2e18", "path": "plain", "n": 1 << 18, "scalars": "uniform", "memory": "device"},
        # the same at 2^20, scalars streamed from the host while the first chunk computes
        {"name": "host_2e20", "path": "plain", "n": 1 << 20, "scalars": "uniform", "memory": "pinned"},
        # a ragged large MSM from the host
        {"name": "host_3000017", "path": "plain", "n": 3000017, "scalars": "uniform", "memory": "pinned"},
        # the headline: 2^22 resident uniform scalars
        {"name": "plain_2e22", "path": "plain", "n": 1 << 22, "scalars": "uniform", "memory": "device"},
        # a witness of 2^22: most digits zero, one bucket holding a fifth of all points
        {"name": "plain_2e22_skewed", "path": "plain", "n": 1 << 22, "scalars": "skewed", "memory": "device"},
        # a proof's commitments over one resident table
        {"name": "batch_24", "path": "batch", "count": 24, "lo_log": 10, "hi_log": 18, "lengths": 3, "scalars": "mixed"},
        # a burst of requests at the serving loop
        {"name": "serve_24", "path": "serve", "count": 24, "lo_log": 8, "hi_log": 18, "lengths": 4, "scalars": "mixed"},
    ]


def draw(rng):
    path = rng.choice(["plain", "plain", "plain", "plain", "noalloc", "batch", "serve"])
    if path in ("batch", "serve"):
        return {"path": path, "count": rng.randint(4, 32), "lo_log": rng.randint(8, 10), "hi_log": rng.randint(13, 18),
                "lengths": rng.randrange(1 << 20), "scalars": "mixed"}
    n = int(round(2 ** rng.uniform(8, 16 if path == "noalloc" else 22)))
    if rng.random() < 0.3:
        n = 1 << int(round(math.log2(n)))
    case = {"path": path, "n": n, "scalars": rng.choice(["uniform", "skewed"]), "memory": "device"}
    if path == "plain":
        case["memory"] = rng.choice(["device", "pinned"])
    return case


def lengths(case):
    """The MSM lengths of a case: log-uniform for a batch or a burst."""
    if "n" in case:
        return [case["n"]]
    rng = random.Random(case["lengths"])
    return [int(round(2 ** rng.uniform(case["lo_log"], case["hi_log"]))) for _ in range(case["count"])]


# -- inputs --------------------------------------------------------------------
def limbs(x):
    return [(x >> (32 * i)) & 0xFFFFFFFF for i in range(8)]


def below_r(gen, n):
    """n values uniform over the eight-limb values whose top limb is below r's (n x 8 int32, device)."""
    v = torch.randint(-(1 << 31), 1 << 31, (n, 8), dtype=torch.int32, device="cuda", generator=gen)
    v[:, 7] = torch.randint(0, TOP_LIMB, (n,), dtype=torch.int32, device="cuda", generator=gen)
    return v


@functools.lru_cache(maxsize=None)
def small_scalars():
    """Montgomery images of 0 .. 2^16 - 1 (65536 x 8 int32, device)."""
    mont = (1 << 256) % R
    raw = b"".join((v * mont % R).to_bytes(32, "little") for v in range(1 << 16))
    return torch.from_numpy(np.frombuffer(raw, dtype=np.int32).reshape(-1, 8).copy()).cuda()


def make_scalars(gen, n, kind):
    """Montgomery-form scalars (n x 8 int32, device)."""
    s = below_r(gen, n)  # a uniform Montgomery image is a uniform scalar
    if kind == "skewed":
        small = small_scalars()
        where = torch.randperm(n, generator=gen, device="cuda")
        zeros, ones, low = (4 * n) // 10, (2 * n) // 10, (2 * n) // 10
        s[where[:zeros]] = 0
        s[where[zeros:zeros + ones]] = small[1]
        picks = torch.randint(0, 1 << 16, (low,), device="cuda", generator=gen)
        s[where[zeros + ones:zeros + ones + low]] = small[picks]
    return s


def make_inputs(case, seed):
    """(multipliers k of the bases k G, the scalars of every MSM), made from the seed alone."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    sizes = lengths(case)
    k = below_r(gen, max(sizes) if "n" in case else TABLE_POINTS)
    k[:, 0] |= 1  # never zero
    kinds = [case["scalars"] if case["scalars"] != "mixed" else ("uniform", "skewed")[j % 2] for j in range(len(sizes))]
    return k, [make_scalars(gen, n, kind) for n, kind in zip(sizes, kinds)]


# -- the program ---------------------------------------------------------------
class Program:
    """What a program holds for its whole life: the library, a memory pool and its streams."""

    def __init__(self):
        import bellman_cuda
        self.bc = bc = bellman_cuda.BellmanCuda()
        bc.set_device(0)
        bc.msm_set_up()
        self.pool = bc.mem_pool_create(0)
        self.stream = bc.stream_create(False)
        self.side = [bc.stream_create(False) for _ in range(SIDE_STREAMS)]
        self.ready = bc.event_create(False, True)
        self.done = [bc.event_create(False, True) for _ in self.side]

    def bases(self, k):
        out = torch.empty((len(k), 16), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        self.bc.generator_multiples(k.data_ptr(), out.data_ptr(), len(k), self.stream)
        self.bc.stream_synchronize(self.stream)
        return out

    def final_sum(self, results, point, stream):
        self.bc.check(self.bc.final_sum_async(results, point, stream), "msm_b200_final_sum_async")

    def final_sums(self, results, points):
        """One final sum per MSM, spread over the side streams between the work before and after on the main one."""
        bc = self.bc
        used = min(len(self.side), len(results))
        bc.event_record(self.ready, self.stream)
        for s in self.side[:used]:
            bc.check(bc.lib.bc_stream_wait_event(s, self.ready), "bc_stream_wait_event")
        for j, (r, p) in enumerate(zip(results, points)):
            self.final_sum(r, p, self.side[j % used])
        for s, e in zip(self.side[:used], self.done):
            bc.event_record(e, s)
            bc.check(bc.lib.bc_stream_wait_event(self.stream, e), "bc_stream_wait_event")


@functools.lru_cache(maxsize=None)
def program():
    return Program()


class State:
    """A case's inputs, buffers and handles; the handles go when the state does."""

    def __init__(self, case, seed):
        self.case = case
        self.prog = program()
        bc = self.prog.bc
        k, scalars = make_inputs(case, seed)
        self.bases = self.prog.bases(k)
        if case.get("memory") == "pinned":
            scalars = [s.cpu().pin_memory() for s in scalars]
        self.scalars = scalars
        self.results = torch.zeros((len(scalars), RESULT_BYTES // 4), dtype=torch.int32, device="cuda")
        self.points = torch.zeros((len(scalars), POINT_WORDS), dtype=torch.int32, device="cuda")
        self.counts = [len(s) for s in scalars]
        self.scalar_ptrs = [s.data_ptr() for s in scalars]
        self.result_ptrs = [r.data_ptr() for r in self.results]
        self.point_ptrs = [p.data_ptr() for p in self.points]
        self.table = self.batch = self.server = None
        torch.cuda.synchronize()
        if case["path"] in ("batch", "serve"):
            self.table = bc.base_table_create(self.bases.data_ptr(), TABLE_POINTS, self.prog.stream)
        if case["path"] == "batch":
            self.batch = bc.batch_create(self.table, self.counts)
        if case["path"] == "serve":
            self.server = bc.server_create(self.table, SERVER_BUDGET)

    def __del__(self):
        bc = self.prog.bc
        torch.cuda.synchronize()
        if self.server is not None:
            bc.server_destroy(self.server)
        if self.batch is not None:
            bc.batch_destroy(self.batch)
        if self.table is not None:
            bc.base_table_destroy(self.table)


def prepare(case, seed):
    return State(case, seed)


def run(state):
    prog, bc, case = state.prog, state.prog.bc, state.case
    path = case["path"]
    if path == "batch":
        bc.batch_execute(state.batch, state.scalar_ptrs, state.result_ptrs, prog.stream)
        prog.final_sums(state.result_ptrs, state.point_ptrs)
        return state.points
    if path == "serve":
        tickets = [bc.server_submit(state.server, s, n, r) for s, n, r in zip(state.scalar_ptrs, state.counts, state.result_ptrs)]
        for t in tickets:
            bc.check(bc.server_wait(state.server, t)[0], "msm_b200_server_wait")
        prog.final_sums(state.result_ptrs, state.point_ptrs)
        bc.stream_synchronize(prog.stream)
        return state.points
    n, bases, scalars, results = case["n"], state.bases.data_ptr(), state.scalar_ptrs[0], state.result_ptrs[0]
    if path == "noalloc":
        bc.check(bc.msm_no_alloc(prog.stream, bases, scalars, results, n), "msm_b200_execute_no_alloc_async")
    elif n & (n - 1) == 0:
        bc.msm(prog.pool, prog.stream, bases, scalars, results, n.bit_length() - 1)
    else:
        bc.check(bc.msm_any(prog.pool, prog.stream, bases, scalars, results, n), "msm_b200_execute_async")
    prog.final_sum(results, state.point_ptrs[0], prog.stream)
    return state.points


def work(case):
    # each scalar (32 B) and base (64 B) read once, each point written; the
    # arithmetic is 256-bit modular integer work, no floating-point operations
    sizes = lengths(case)
    read = 32 * sum(sizes) + 64 * max(sizes)
    return {"bytes": read + 4 * POINT_WORDS * len(sizes), "flops": 0}


def tolerance(case):
    return "exact"  # canonical points of exact arithmetic


# -- the same points from plain integer arithmetic -----------------------------
def dot_mod_r(a, b):
    """sum a_i b_i mod r of two n x 8 limb tensors: 16-bit limbs, products summed exactly in float64."""
    a16 = a.cpu().numpy().view(np.uint16)
    b16 = b.cpu().numpy().view(np.uint16)
    total = 0
    for at in range(0, len(a16), 1 << 20):  # 2^20 products below 2^32: sums below 2^52
        m = a16[at:at + (1 << 20)].astype(np.float64).T @ b16[at:at + (1 << 20)].astype(np.float64)
        total += sum(int(m[i, j]) << (16 * (i + j)) for i in range(16) for j in range(16))
    return total % R


def generator_multiple(s):
    """s G on y^2 = x^3 + 3, G = (1, 2), as (x, y), or None for infinity."""
    acc, add = None, (1, 2)
    while s:
        if s & 1:
            acc = point_add(acc, add)
        add = point_add(add, add)
        s >>= 1
    return acc


def point_add(p, q):
    if p is None or q is None:
        return q if p is None else p
    if p[0] == q[0]:
        if (p[1] + q[1]) % P == 0:
            return None
        slope = 3 * p[0] * p[0] * pow(2 * p[1], -1, P) % P
    else:
        slope = (q[1] - p[1]) * pow(q[0] - p[0], -1, P) % P
    x = (slope * slope - p[0] - q[0]) % P
    return x, (slope * (p[0] - x) - p[1]) % P


def exact(case, seed):
    k, scalars = make_inputs(case, seed)
    unmont = pow(1 << 256, -1, R)
    rows = []
    for s in scalars:
        point = generator_multiple(dot_mod_r(k[:len(s)].contiguous(), s) * unmont % R)
        rows.append(limbs(point[0]) + limbs(point[1]) + [0] * 4 if point else [0] * 16 + [1, 0, 0, 0])
    return np.array(rows, dtype=np.uint32).view(np.int32)
