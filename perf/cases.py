"""The products this library is used for, as cases that can be timed.

The matrices are the kinds that `tilespgemm_gb300/matrices.py` and the
benchmark name: 2D 5-point and 3D 27-point stencils, R-MAT graphs, uniform
random rectangular matrices, and batches of small mixed ones.  They are made
on the GPU: a case's sizes (its entries and C's among them) are its own, the
values, and where a random pattern's rows and columns lie, come from the seed.
The calls are the package's public ones:
`Context.spgemm_raw` (operands and C on the device, or both in host memory),
`Context.spgemm_batched_raw` and `Plan.execute_raw`.
"""
from __future__ import annotations

import functools
import math
import random

import numpy as np
import torch

from tilespgemm_gb300 import Context
from tilespgemm_gb300.api import CSR

_CHUNK = 1 << 27   # products expanded at a time by the plain restatement


def listed():
    return [
        # a request of the serving loop at its smallest grid: launches and the
        # host's part of the call are all there is
        dict(name="laplacian-32", call="spgemm", matrix="laplacian", nx=32, ny=32, op="AA", where="device"),
        # the plain 2D product the library quotes first (65,536 rows)
        dict(name="laplacian-256", call="spgemm", matrix="laplacian", nx=256, ny=256, op="AA", where="device"),
        # a 3D grid of ordinary size whose rows do not fill the last tile-row
        dict(name="stencil-31", call="spgemm", matrix="stencil", side=31, op="AA", where="device"),
        # the headline product: 23 M entries squared to 106 M, FP64-bound
        dict(name="stencil-96", call="spgemm", matrix="stencil", side=96, op="AA", where="device"),
        # a caller with host arrays: copies both ways beside the kernels
        dict(name="stencil-64-host", call="spgemm", matrix="stencil", side=64, op="AA", where="host"),
        # graphs of the serving loop's range, A*A^T: the smallest, an
        # ordinary one, and the largest, whose hub rows are millions long
        dict(name="rmat-12-aat", call="spgemm", matrix="rmat", scale=12, edges=8, graph=1, op="AAT", where="device"),
        dict(name="rmat-15-aat", call="spgemm", matrix="rmat", scale=15, edges=16, graph=1, op="AAT", where="device"),
        dict(name="rmat-18-aat", call="spgemm", matrix="rmat", scale=18, edges=16, graph=1, op="AAT", where="device"),
        # two-step paths of a graph, A*A (the other half of the requests)
        dict(name="rmat-16-aa", call="spgemm", matrix="rmat", scale=16, edges=12, graph=2, op="AA", where="device"),
        # a general rectangular A*B without structure, int64 row pointers,
        # no size a multiple of the tile: about one entry per tile of C
        dict(name="uniform-ab", call="spgemm", matrix="uniform", m=120007, k=80021, n=100003, per_a=16, per_b=12,
             graph=3, op="AB", where="device"),
        # one wave of the batched workload: 512 products of 64 to 16,384 rows
        dict(name="batch-512", call="batched", matrix="mixed", count=512, graph=4, op="AA", where="device"),
        # a solver that squares the same pattern again with new values
        dict(name="stencil-48-plan", call="plan", matrix="stencil", side=48, op="AA", where="device"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("laplacian", "stencil", "rmat", "rmat", "uniform", "mixed", "plan"))
    if kind == "laplacian":
        return dict(call="spgemm", matrix="laplacian", nx=_log_int(rng, 32, 512), ny=_log_int(rng, 32, 512), op="AA",
                    where=rng.choice(("device", "device", "host")))
    if kind == "stencil":
        return dict(call="spgemm", matrix="stencil", side=_log_int(rng, 8, 88), op=rng.choice(("AA", "AA", "AAT")),
                    where=rng.choice(("device", "device", "host")))
    if kind == "rmat":
        scale = rng.randint(12, 17)
        return dict(call="spgemm", matrix="rmat", scale=scale, edges=_log_int(rng, 8, 16 if scale > 16 else 32),
                    graph=rng.randint(5, 1 << 20), op=rng.choice(("AA", "AAT")), where="device")
    if kind == "uniform":
        return dict(call="spgemm", matrix="uniform", m=_log_int(rng, 1000, 200000), k=_log_int(rng, 1000, 200000),
                    n=_log_int(rng, 1000, 200000), per_a=_log_int(rng, 2, 24), per_b=_log_int(rng, 2, 24),
                    graph=rng.randint(5, 1 << 20), op="AB", where="device")
    if kind == "mixed":
        return dict(call="batched", matrix="mixed", count=_log_int(rng, 8, 256), graph=rng.randint(5, 1 << 20), op="AA",
                    where="device")
    if rng.random() < 0.5:
        return dict(call="plan", matrix="stencil", side=_log_int(rng, 8, 72), op="AA", where="device")
    return dict(call="plan", matrix="rmat", scale=rng.randint(12, 16), edges=_log_int(rng, 8, 24),
                graph=rng.randint(5, 1 << 20), op=rng.choice(("AA", "AAT")), where="device")


# ---- matrices: (m, n, row pointer, columns, values) on the GPU ----------------


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uniform(g, n, lo, hi):
    return torch.empty(n, dtype=torch.float64, device="cuda").uniform_(lo, hi, generator=g)


def _rowptr(rows, m):
    rp = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(torch.bincount(rows, minlength=m), 0)
    return rp


def _stencil(dims, offsets, g):
    """Grid stencil with neighbour couplings in [0.5, 1.5] and their sum on the
    diagonal; `offsets` ascend in the grid's numbering (first dimension fastest)."""
    n = math.prod(dims)
    idx = torch.arange(n, device="cuda")
    at, step, steps = [], 1, []
    for d in dims:
        at.append(idx // step % d)
        steps.append(step)
        step *= d
    ok = torch.ones((n, len(offsets)), dtype=torch.bool, device="cuda")
    shift = []
    for q, off in enumerate(offsets):
        for a, d, o in zip(at, dims, off):
            if o:
                ok[:, q] &= (a + o >= 0) & (a + o < d)
        shift.append(sum(o * s for o, s in zip(off, steps)))
    cols = idx[:, None] + torch.tensor(shift, device="cuda")[None, :]
    v = _uniform(g, n * len(offsets), 0.5, 1.5).view(n, len(offsets)) * ok
    centre = offsets.index((0,) * len(dims))
    v[:, centre] = 0
    if len(dims) == 2:
        v = -v
    v[:, centre] = v.sum(1).abs()
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(ok.sum(1), 0)
    return n, n, rp, cols[ok].to(torch.int32), v[ok]


def _merged(m, n, rows, cols, g):
    key = torch.unique(rows * n + cols)
    return m, n, _rowptr(key // n, m), (key % n).to(torch.int32), _uniform(g, key.numel(), -1.0, 1.0)


def _rmat(scale, edges, graph, seed, g):
    """The graph's vertices renumbered by an exclusive or, which keeps the
    quadrants' shares at every level and moves its hubs."""
    n, ne = 1 << scale, edges << scale
    rows = torch.zeros(ne, dtype=torch.int64, device="cuda")
    cols = torch.zeros_like(rows)
    for _ in range(scale):
        u = torch.rand(ne, device="cuda", generator=graph)
        rows = rows * 2 + (u >= 0.76)
        cols = cols * 2 + (((u >= 0.57) & (u < 0.76)) | (u >= 0.95))
    at = random.Random(seed).randrange(n)
    return _merged(n, n, rows ^ at, cols ^ at, g)


def _random(m, n, per, graph, row0, col0, g):
    """Uniform columns; rows and columns counted from row0 and col0 on."""
    rows = torch.arange(m, device="cuda").repeat_interleave(per)
    cols = torch.randint(n, rows.shape, device="cuda", generator=graph)
    return _merged(m, n, (rows + row0) % m, (cols + col0) % n, g)


def _banded(n, per, graph, turned, g):
    """|i - j| <= n/16; turned: both numberings run backwards."""
    rows = torch.arange(n, device="cuda").repeat_interleave(per)
    half = max(1, n // 16)
    cols = (rows + torch.randint(-half, half + 1, rows.shape, device="cuda", generator=graph)).clamp_(0, n - 1)
    return _merged(n, n, n - 1 - rows, n - 1 - cols, g) if turned else _merged(n, n, rows, cols, g)


def _operands(case, seed):
    """([A, ...], [B, ...] or None) of the case."""
    g, graph, at = _gen(seed), _gen(case.get("graph", 0)), random.Random(seed)
    if case["matrix"] == "laplacian":
        return [_stencil((case["nx"], case["ny"]), [(0, -1), (-1, 0), (0, 0), (1, 0), (0, 1)], g)], None
    if case["matrix"] == "stencil":
        offsets = [(x, y, z) for z in (-1, 0, 1) for y in (-1, 0, 1) for x in (-1, 0, 1)]
        return [_stencil((case["side"],) * 3, offsets, g)], None
    if case["matrix"] == "rmat":
        return [_rmat(case["scale"], case["edges"], graph, seed, g)], None
    if case["matrix"] == "uniform":
        m, k, n = case["m"], case["k"], case["n"]
        row0, mid0, col0 = at.randrange(m), at.randrange(k), at.randrange(n)
        return [_random(m, k, case["per_a"], graph, row0, mid0, g)], [_random(k, n, case["per_b"], graph, mid0, col0, g)]
    sizes, As = random.Random(case["graph"]), []
    for i in range(case["count"]):   # even instances banded, odd ones uniform
        n = _log_int(sizes, 64, 16384)
        per, first = sizes.randint(2, min(64, n)), at.randrange(n)
        As.append(_random(n, n, per, graph, first, first, g) if i % 2 else _banded(n, per, graph, first % 2, g))
    return As, None


# ---- the calls ----------------------------------------------------------------


@functools.lru_cache(maxsize=None)
def _context():
    """One context for the program's life, as a program keeps it."""
    return Context(0)


def _matrix(t, where, bits):
    m, n, rp, col, val = t
    rp = rp.to(torch.int64 if bits == 64 else torch.int32)
    if where == "host":
        rp, col, val = (x.cpu().pin_memory() for x in (rp, col, val))
    return CSR(m, n, rp, col, val)


def prepare(case, seed):
    As, Bs = _operands(case, seed)
    bits = 64 if case["op"] == "AB" else 32
    state = dict(case=case, ctx=_context(), A=[_matrix(t, case["where"], bits) for t in As],
                 B=None if Bs is None else [_matrix(t, case["where"], bits) for t in Bs])
    if case["call"] == "plan":
        state["plan"] = state["ctx"].plan(state["A"][0], op=case["op"])
    return state


class _Span:
    """An array of C where the library left it; it keeps C alive."""

    def __init__(self, owner, ptr, n, typestr, device):
        self.owner = owner
        setattr(self, "__cuda_array_interface__" if device else "__array_interface__",
                dict(shape=(n,), typestr=typestr, data=(ptr, False), strides=None, version=3))


def _arrays(outs):
    """C's row pointer, columns and values; a batch's, which lie in one
    allocation, from the first instance's start to the last one's end."""
    a, b = outs[0].s, outs[-1].s
    device = outs[0].where == "device"
    view = functools.partial(torch.as_tensor, device="cuda") if device else np.asarray
    rp = a.rowptr_bits // 8

    def span(first, last, n, size, typestr):
        return view(_Span(outs, first, (last - first) // size + n, typestr, device))
    return dict(rowptr=span(a.row_ptr, b.row_ptr, b.m + 1, rp, "<i%d" % rp),
                col=span(a.col, b.col, b.nnz, 4, "<i4"),
                val=span(a.val, b.val, b.nnz, 8, "<f8"))


def run(state):
    case, ctx, A, B = state["case"], state["ctx"], state["A"], state["B"]
    if case["call"] == "batched":
        return _arrays(ctx.spgemm_batched_raw(A, B, op=case["op"], out=case["where"])[0])
    if case["call"] == "plan":
        return _arrays([state["plan"].execute_raw(A[0].val, out=case["where"])[0]])
    return _arrays([ctx.spgemm_raw(A[0], B[0] if B else None, op=case["op"], out=case["where"])[0]])


# ---- the same products in plain torch -----------------------------------------


def _rows_of(rp):
    return torch.repeat_interleave(torch.arange(rp.numel() - 1, device="cuda"), rp.diff())


def _transpose(t):
    m, n, rp, col, val = t
    order = torch.argsort(col.long(), stable=True)
    return n, m, _rowptr(col.long(), n), _rows_of(rp)[order].to(torch.int32), val[order]


def _product(A, B, values=True):
    """C = A*B by expanding, sorting and adding up the products of a block of
    rows at a time: (products, row pointer, columns, values)."""
    (m, _, rp, col, val), (_, n, brp, bcol, bval) = A, B
    per_entry = brp.diff()[col.long()]
    done = torch.zeros(col.numel() + 1, dtype=torch.int64, device="cuda")
    done[1:] = torch.cumsum(per_entry, 0)
    by_row = done[rp]
    rows = _rows_of(rp)
    counts, cols, vals, r0 = [], [], [], 0
    while r0 < m:
        r1 = int(torch.searchsorted(by_row, by_row[r0] + _CHUNK, right=True).item()) - 1
        r1 = min(m, max(r0 + 1, r1))
        e0, e1 = int(rp[r0].item()), int(rp[r1].item())
        src = torch.repeat_interleave(torch.arange(e0, e1, device="cuda"), per_entry[e0:e1])
        q = brp[col[src].long()] + torch.arange(src.numel(), device="cuda") - (done[src] - done[e0])
        key, order = torch.sort((rows[src] - r0) * n + bcol[q].long())
        if values:
            p = (val[src] * bval[q])[order]
            key, inv, cnt = torch.unique_consecutive(key, return_inverse=True, return_counts=True)
            vals.append(torch.zeros(key.numel(), dtype=torch.float64, device="cuda").index_add_(0, inv, p))
            cols.append((key % n).to(torch.int32))
        else:
            key = torch.unique_consecutive(key)
        counts.append(torch.bincount(key // n, minlength=r1 - r0))
        r0 = r1
    rpc = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    rpc[1:] = torch.cumsum(torch.cat(counts), 0)
    return int(done[-1].item()), rpc, torch.cat(cols) if values else None, torch.cat(vals) if values else None


def _pairs(case, seed):
    As, Bs = _operands(case, seed)
    return list(zip(As, Bs or (As if case["op"] == "AA" else [_transpose(t) for t in As])))


def exact(case, seed):
    got = [_product(a, b) for a, b in _pairs(case, seed)]
    if len(got) > 1:   # a batch: the instances' entries one behind the other
        return dict(rowptr=None, col=torch.cat([x[2] for x in got]), val=torch.cat([x[3] for x in got]))
    return dict(rowptr=got[0][1], col=got[0][2], val=got[0][3])


def work(case):
    size = 8 if case["op"] == "AB" else 4
    bytes_, flops = 0, 0
    for a, b in _pairs(case, 0):
        products, rpc, _, _ = _product(a, b, values=False)
        flops += 2 * products
        for t in (a, b)[:2 if case["op"] == "AB" else 1]:
            if case["call"] == "plan":
                bytes_ += 8 * t[3].numel()   # the values; the pattern is the plan's
            else:
                bytes_ += size * (t[0] + 1) + 12 * t[3].numel()
        bytes_ += 4 * (a[0] + 1) + 12 * int(rpc[-1].item())
    return dict(bytes=bytes_, flops=flops)
