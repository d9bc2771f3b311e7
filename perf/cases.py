"""The work a user of this framework has it do, as measurable cases.

One Newton step of an implicit elastodynamics simulation generates the block
system of the current state (``generate``), reduces its raw 3x3 triplets to a
block-upper matrix (``assemble``), builds and applies the MAS or block-Jacobi
preconditioner (``build``), multiplies by the matrix (``spmv``), predicts a
start from earlier solutions (``warm``) and runs the PCG (``pcg``); ``solve``
is the whole step through ``GlobalLinearSystem``. The listed cases take each of
them at sizes from a toy cube to the 1.65 M-DoF stack of eight 40^3-cell cubes,
in FP64 and in mixed precision, on three scenes:

* ``stack``: ``cubes`` tetrahedral cubes of ``cells``^3 cells on the ground,
  neighbours coupled by point-triangle barrier blocks;
* ``bar``: a bar of ``cells`` x ``across`` x ``across`` cells with both end
  layers fixed (identity rows), nearly incompressible: many PCG iterations;
* ``cloth``: a cloth of ``cells``^2 vertices over ``bodies`` affine bodies of
  four block rows each: 16 triplets per body, 12x3 couplings, a few very long
  rows.

The systems are built here from the seed with torch (linear elasticity on
jittered Kuhn-split cells, rank-1 barrier blocks), in the triplet order the
framework's producers write: one kinetic block per vertex, ten blocks per tet,
then the contacts; unwritten contact slots keep row -1.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from libuipc_b200 import _abi
from libuipc_b200.gpu_scene import GpuTetMesh
from libuipc_b200.linear_system import (B200MAS, B200PCG, B200Jacobi, GlobalLinearSystem, Solver, partition_graph,
                                        partition_maps, partition_rcb)

DEV = torch.device("cuda", 0)
H = 0.01  # cell size [m]
DT = 0.01  # time step [s]
RHO = 1e3
MATERIAL = {"stack": (1e5, 0.45), "bar": (1e6, 0.49), "cloth": (1e4, 0.3)}  # Young's modulus [Pa], Poisson's ratio


def listed() -> list[dict]:
    return [
        # the default scene settings (FP64, block Jacobi, |r.z| rule) on a toy scene: launches and latency
        {"name": "solve_cube10_default", "op": "solve", "scene": "stack", "cubes": 1, "cells": 10,
         "precision": "fp64", "precond": "diag", "rule": "rz", "tol": 1e-3},
        # an interactive cloth over bodies: MAS on the cloth, 12x12 block Jacobi on the bodies, mixed precision
        {"name": "solve_cloth128_mixed", "op": "solve", "scene": "cloth", "cells": 128, "bodies": 25,
         "precision": "mixed", "precond": "mas", "rule": "relres", "tol": 1e-4},
        # the headline: the whole mixed solve of the 1.65 M-DoF stack
        {"name": "solve_stack8x40_mixed", "op": "solve", "scene": "stack", "cubes": 8, "cells": 40,
         "precision": "mixed", "precond": "mas", "rule": "relres", "tol": 1e-4},
        # FP64 PCG with MAS on the stiff bar, parts from the connectivity-only partitioner (padded parts)
        {"name": "pcg_bar200_fp64", "op": "pcg", "scene": "bar", "cells": 200, "across": 20, "partition": "graph",
         "precision": "fp64", "precond": "mas", "rule": "relres", "tol": 1e-4},
        # triplets to block-upper BSR, read back on the device: a small ragged cloth with very long body rows
        {"name": "assemble_cloth61", "op": "assemble", "scene": "cloth", "cells": 61, "bodies": 4},
        # the same at full size
        {"name": "assemble_stack8x40", "op": "assemble", "scene": "stack", "cubes": 8, "cells": 40},
        # y = A x with x.Ax as an external Krylov method calls it: FP64 on the bar, FP32 on the stack
        {"name": "spmv_bar200_fp64", "op": "spmv", "scene": "bar", "cells": 200, "across": 20, "precision": "fp64"},
        {"name": "spmv_stack8x40_mixed", "op": "spmv", "scene": "stack", "cubes": 8, "cells": 40,
         "precision": "mixed"},
        # MAS build and one apply: a mid-sized odd stack in FP64, the large one with the BF16 inverses
        {"name": "build_stack3x17_fp64", "op": "build", "scene": "stack", "cubes": 3, "cells": 17,
         "precision": "fp64"},
        {"name": "build_stack8x40_mixed", "op": "build", "scene": "stack", "cubes": 8, "cells": 40,
         "precision": "mixed"},
        # the Galerkin start from the eight latest solutions
        {"name": "warm_bar200_hist8", "op": "warm", "scene": "bar", "cells": 200, "across": 20, "history": 8},
        # the Newton system of the bar at a deformed state, generated on the device
        {"name": "generate_bar200", "op": "generate", "scene": "bar", "cells": 200, "across": 20},
    ]


def _logint(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    op = rng.choice(["solve", "solve", "pcg", "assemble", "spmv", "build", "warm", "generate"])
    scene = rng.choice(["stack", "stack", "bar", "cloth"])
    if op in ("generate", "warm"):
        scene = "bar"
    c: dict = {"op": op, "scene": scene}
    if scene == "stack":
        c["cubes"] = rng.randint(1, 8)
        c["cells"] = _logint(rng, 4, 36)
    elif scene == "bar":
        c["across"] = _logint(rng, 3, 20)
        c["cells"] = c["across"] * rng.randint(3, 10)
    else:
        c["cells"] = _logint(rng, 9, 256)
        c["bodies"] = rng.randint(1, 8) ** 2
    if op in ("solve", "pcg"):
        # block Jacobi takes hundreds of iterations, the bar many more: those at the looser tolerances only
        c["precond"] = "mas" if scene == "bar" else rng.choice(["diag", "mas", "mas"])
        tight = [] if scene == "bar" or c["precond"] == "diag" else [("relres", 1e-6)]
        c["rule"], c["tol"] = rng.choice([("rz", 1e-3), ("relres", 1e-4)] + tight)
    if op in ("solve", "pcg", "spmv", "build"):
        c["precision"] = rng.choice(["fp64", "mixed"])
    if op in ("solve", "pcg", "build") and c.get("precond") != "diag" and c["cells"] < 100:
        c["partition"] = rng.choice(["rcb", "graph"])
    if op == "warm":
        c["history"] = rng.randint(1, 8)
    return c


# ---------------------------------------------------------------------------
# the scenes
# ---------------------------------------------------------------------------
def _lattice(nx: int, ny: int, nz: int):
    """Vertices of an nx x ny x nz cell lattice (x fastest) and its 6 Kuhn tets per cell."""
    gx, gy, gz = nx + 1, ny + 1, nz + 1
    z, y, x = torch.meshgrid(*(torch.arange(n, device=DEV) for n in (gz, gy, gx)), indexing="ij")
    pos = torch.stack([x, y, z], -1).reshape(-1, 3).double() * H
    cz, cy, cx = torch.meshgrid(*(torch.arange(n, device=DEV) for n in (nz, ny, nx)), indexing="ij")
    corner = ((cz * gy + cy) * gx + cx).reshape(-1)
    step = (1, gx, gx * gy)
    tets = []
    for a, b in ((0, 1), (1, 2), (2, 0), (1, 0), (2, 1), (0, 2)):
        c = 3 - a - b
        even = (a, b) in ((0, 1), (1, 2), (2, 0))
        p = [torch.zeros_like(corner), torch.full_like(corner, step[a]), torch.full_like(corner, step[a] + step[b]),
             torch.full_like(corner, step[a] + step[b] + step[c])]
        q = [corner + o for o in p]
        if not even:
            q[1], q[2] = q[2], q[1]
        tets.append(torch.stack(q, -1))
    return pos, torch.stack(tets, 1).reshape(-1, 4)


def _gradients(pos: torch.Tensor, tets: torch.Tensor):
    """Shape gradients [nt, 4, 3] and volumes of tets."""
    e = pos[tets[:, 1:]] - pos[tets[:, :1]]
    inv = torch.linalg.inv(e)  # rows of e are the edges: gradients of 1..3 are the columns of its inverse
    g = torch.empty(tets.shape[0], 4, 3, dtype=torch.float64, device=DEV)
    g[:, 1:] = inv.transpose(1, 2)
    g[:, 0] = -g[:, 1:].sum(1)
    return g, torch.linalg.det(e).abs() / 6.0


def _upper(va, vb, blocks, at, rows, cols, vals):
    """Blocks [m, 3, 3] of the pairs (va, vb) into triplet slots `at`, upper orientation, column-major."""
    t = va > vb
    rows[at] = torch.where(t, vb, va).int()
    cols[at] = torch.where(t, va, vb).int()
    vals[at] = torch.where(t[:, None, None], blocks, blocks.transpose(1, 2)).reshape(-1, 9)


def _elastic(nodes, g, scale, lam, mu, at, rows, cols, vals):
    """scale * (lam ga gb^T + mu gb ga^T + mu (ga.gb) I) of every node pair a <= b into slots at + pair."""
    k = nodes.shape[1]
    eye = torch.eye(3, dtype=torch.float64, device=DEV)
    pair = 0
    for a in range(k):
        for b in range(a, k):
            ga, gb = g[:, a], g[:, b]
            blk = lam * ga[:, :, None] * gb[:, None, :] + mu * gb[:, :, None] * ga[:, None, :]
            blk += mu * (ga * gb).sum(1)[:, None, None] * eye
            _upper(nodes[:, a], nodes[:, b], blk * scale[:, None, None], at + pair, rows, cols, vals)
            pair += 1


def _rank1(nodes, w, n, k, at, rows, cols, vals):
    """k w_a w_b n n^T of every node pair a <= b into slots at + pair."""
    nn = n[:, :, None] * n[:, None, :] * k[:, None, None]
    pair = 0
    for a in range(nodes.shape[1]):
        for b in range(a, nodes.shape[1]):
            _upper(nodes[:, a], nodes[:, b], nn * (w[:, a] * w[:, b])[:, None, None], at + pair, rows, cols, vals)
            pair += 1


def _triplets(T: int):
    return (torch.full((T,), -1, dtype=torch.int32, device=DEV), torch.full((T,), -1, dtype=torch.int32, device=DEV),
            torch.zeros((T, 9), dtype=torch.float64, device=DEV))


class _System:
    """Raw triplets, gradient and what the MAS needs of one scene."""

    def __init__(self, case: dict, seed: int):
        self.gen = torch.Generator(device=DEV)
        self.gen.manual_seed(int(seed) % (1 << 62))
        {"stack": self._stack, "bar": self._bar, "cloth": self._cloth}[case["scene"]](case)

    def rand(self, *shape):
        return torch.rand(*shape, dtype=torch.float64, device=DEV, generator=self.gen)

    def randn(self, *shape):
        return torch.randn(*shape, dtype=torch.float64, device=DEV, generator=self.gen)

    def _solid(self, rest, tets, scene, extra: int):
        """Kinetic + elastic triplets of jittered tets; `extra` slots follow. Returns the element scale."""
        E, nu = MATERIAL[scene]
        mu, lam = E / (2 * (1 + nu)), E * nu / ((1 + nu) * (1 - 2 * nu))
        nv, nt = rest.shape[0], tets.shape[0]
        self.offset, self.bodies, self.nb = 0, 0, nv
        self.rest, self.cells = rest, tets
        pos = rest + 0.1 * H * (self.rand(nv, 3) - 0.5)
        g, vol = _gradients(pos, tets)
        self.rows, self.cols, self.vals = _triplets(nv + 10 * nt + extra)
        mass = torch.zeros(nv, dtype=torch.float64, device=DEV)
        mass.index_add_(0, tets.reshape(-1), (vol * RHO / 4).repeat_interleave(4))
        v = torch.arange(nv, device=DEV)
        eye = torch.eye(3, dtype=torch.float64, device=DEV)
        _upper(v, v, mass[:, None, None] * eye, v, self.rows, self.cols, self.vals)
        _elastic(tets, g, vol * DT * DT, lam, mu, nv + 10 * torch.arange(nt, device=DEV), self.rows, self.cols,
                 self.vals)
        # a smooth velocity change plus the jitter's internal forces
        phase = (pos @ (self.randn(3, 3) * 12.0)).sin()
        self.b = (mass[:, None] * (DT * DT * torch.tensor([0.0, 9.8, 0.0], dtype=torch.float64, device=DEV)
                                   + 1e-3 * phase + 2e-4 * self.randn(nv, 3))).reshape(-1)
        return DT * DT * E * H

    def _stack(self, case):
        n, m = case["cells"], case["cubes"]
        p, t = _lattice(n, n, n)
        per = p.shape[0]
        rest = torch.cat([p + torch.tensor([0.0, k * (n * H + 1e-3), 0.0], dtype=torch.float64, device=DEV)
                          for k in range(m)])
        tets = torch.cat([t + k * per for k in range(m)])
        nv, nt, g = rest.shape[0], tets.shape[0], n + 1
        ids = torch.arange(per, device=DEV).reshape(g, g, g)  # z, y, x
        bottom, top = ids[:, 0, :], ids[:, -1, :]
        nc = (m - 1) * g * g
        scale = self._solid(rest, tets, "stack", g * g + 10 * nc)
        # ground barrier under the lowest cube: one diagonal block per candidate, a tenth of them inactive
        at = nv + 10 * nt + torch.arange(g * g, device=DEV)
        ey = torch.tensor([0.0, 1.0, 0.0], dtype=torch.float64, device=DEV)
        one = torch.ones(g * g, 1, dtype=torch.float64, device=DEV)
        k = scale * (1.5 * self.randn(g * g)).exp() * (self.rand(g * g) > 0.1)
        _rank1(bottom.reshape(-1, 1), one, ey.expand(g * g, 3), k, at, self.rows, self.cols, self.vals)
        if nc == 0:
            return
        # each bottom vertex of the upper cube against a triangle of the lower one's top
        i = torch.arange(g, device=DEV).clamp(max=g - 2)
        tri = torch.stack([top[i][:, i], top[i + 1][:, i], top[i][:, i + 1]], -1).reshape(-1, 3)
        nodes = torch.cat([torch.cat([(bottom.reshape(-1, 1) + (q + 1) * per), tri + q * per], 1)
                           for q in range(m - 1)])
        w = self.rand(nc, 3) + 0.05
        w = torch.cat([torch.ones(nc, 1, dtype=torch.float64, device=DEV), -w / w.sum(1, keepdim=True)], 1)
        nrm = ey + 0.05 * self.randn(nc, 3)
        nrm = nrm / nrm.norm(dim=1, keepdim=True)
        k = scale * (1.5 * self.randn(nc)).exp()
        live = torch.arange(nc, device=DEV) % 10 < 7  # pairs that are not in contact leave their slots unwritten
        at = nv + 10 * nt + g * g + 10 * torch.arange(nc, device=DEV)
        _rank1(nodes[live], w[live], nrm[live], k[live], at[live], self.rows, self.cols, self.vals)

    def _bar(self, case):
        rest, tets = _lattice(case["cells"], case["across"], case["across"])
        self._solid(rest, tets, "bar", 0)
        x = rest[:, 0]
        self.fixed = (x < 0.5 * H) | (x > x.max() - 0.5 * H)
        fr, fc = self.fixed[self.rows.long()], self.fixed[self.cols.long()]
        self.vals[fr | fc] = 0.0
        eye = torch.eye(3, dtype=torch.float64, device=DEV).reshape(9)
        self.vals[(fr | fc) & (self.rows == self.cols)] = eye
        self.b.view(-1, 3)[self.fixed] = 0.0

    def _cloth(self, case):
        n, nbody = case["cells"], case["bodies"]
        off = 4 * nbody
        E, nu = MATERIAL["cloth"]
        lam, mu = E * nu / (1 - nu * nu), E / (2 * (1 + nu))
        gy, gx = torch.meshgrid(torch.arange(n, device=DEV), torch.arange(n, device=DEV), indexing="ij")
        rest = torch.stack([gx * H, torch.zeros_like(gx), gy * H], -1).reshape(-1, 3).double()
        pos = rest + 0.05 * H * self.randn(n * n, 3)
        ids = torch.arange(n * n, device=DEV).reshape(n, n)
        a, b, c, d = ids[:-1, :-1].reshape(-1), ids[:-1, 1:].reshape(-1), ids[1:, :-1].reshape(-1), \
            ids[1:, 1:].reshape(-1)
        tris = torch.stack([torch.stack([a, b, d], -1), torch.stack([a, d, c], -1)], 1).reshape(-1, 3)
        # hinges: across the cell diagonal, and across the edges between cells
        inner = torch.stack([ids[:-2, :-1].reshape(-1), ids[1:-1, :-1].reshape(-1), ids[1:-1, 1:].reshape(-1),
                             ids[2:, 1:].reshape(-1)], -1)
        hinges = torch.cat([torch.stack([b, a, d, c], -1), inner])
        nv, ntri, nh = n * n, tris.shape[0], hinges.shape[0]
        # every vertex inside a body's footprint touches it
        side = max(int(round(math.sqrt(nbody))), 1)
        cell = (rest[:, [0, 2]] / (n * H) * side).floor().clamp(0, side - 1).long()
        frac = rest[:, [0, 2]] / (n * H) * side - cell
        touch = ((frac - 0.5).abs() < 0.3).all(1).nonzero().reshape(-1)
        body = (cell[touch, 1] * side + cell[touch, 0]).clamp(max=nbody - 1)
        nt = touch.shape[0]
        self.rows, self.cols, self.vals = _triplets(nv + 6 * ntri + 10 * nh + 16 * nbody + 15 * nt)
        self.nb, self.offset, self.bodies, self.rest = nv + off, off, nbody, rest
        self.cells = torch.cat([tris, hinges[:, [0, 1, 3]], hinges[:, [0, 2, 3]]])
        eye = torch.eye(3, dtype=torch.float64, device=DEV)
        mass = RHO * 1e-3 * H * H
        v = torch.arange(nv, device=DEV)
        _upper(v + off, v + off, (mass * eye).expand(nv, 3, 3), v, self.rows, self.cols, self.vals)
        # membrane: in-plane gradients of each triangle
        e1, e2 = pos[tris[:, 1]] - pos[tris[:, 0]], pos[tris[:, 2]] - pos[tris[:, 0]]
        nrm = torch.linalg.cross(e1, e2)
        dbl = nrm.norm(dim=1, keepdim=True)
        nrm = nrm / dbl
        g1, g2 = torch.linalg.cross(e2, nrm) / dbl, torch.linalg.cross(nrm, e1) / dbl
        g = torch.stack([-g1 - g2, g1, g2], 1)
        area = 0.5 * dbl.reshape(-1)
        at = nv + 6 * torch.arange(ntri, device=DEV)
        _elastic(tris + off, g, area * 1e-3 * DT * DT, lam, mu, at, self.rows, self.cols, self.vals)
        # bending: rank-1 along the hinge normal
        w = torch.tensor([1.0, -1.0, -1.0, 1.0], dtype=torch.float64, device=DEV).expand(nh, 4)
        hn = torch.tensor([0.0, 1.0, 0.0], dtype=torch.float64, device=DEV) + 0.05 * self.randn(nh, 3)
        at = nv + 6 * ntri + 10 * torch.arange(nh, device=DEV)
        kb = torch.full((nh,), 0.02 * E * 1e-3 * DT * DT, dtype=torch.float64, device=DEV)
        _rank1(hinges + off, w, hn, kb, at, self.rows, self.cols, self.vals)
        # bodies: the 16 blocks of a 12x12 SPD matrix, zeros below the diagonal
        base = nv + 6 * ntri + 10 * nh
        L = torch.eye(12, dtype=torch.float64, device=DEV) + 0.2 * self.randn(nbody, 12, 12)
        M = L @ L.transpose(1, 2) * (0.1 * RHO * H**3)
        r4 = torch.arange(nbody, device=DEV) * 4
        for i in range(4):
            for j in range(4):
                s = base + 16 * torch.arange(nbody, device=DEV) + 4 * i + j
                self.rows[s], self.cols[s] = (r4 + i).int(), (r4 + j).int()
                blk = M[:, 3 * i:3 * i + 3, 3 * j:3 * j + 3]
                self.vals[s] = blk.transpose(1, 2).reshape(-1, 9) if i <= j else 0.0
        # cloth-body contacts: x_body = p + A xbar, so body row i carries c_i n n^T
        base += 16 * nbody
        xb = torch.cat([torch.ones(nt, 1, dtype=torch.float64, device=DEV), self.rand(nt, 3) - 0.5], 1)
        nodes = torch.cat([4 * body[:, None] + torch.arange(4, device=DEV), (touch + off)[:, None]], 1)
        wc = torch.cat([xb, -torch.ones(nt, 1, dtype=torch.float64, device=DEV)], 1)
        cn = torch.tensor([0.0, 1.0, 0.0], dtype=torch.float64, device=DEV) + 0.02 * self.randn(nt, 3)
        kc = 0.1 * E * 1e-3 * DT * DT * self.randn(nt).exp()
        _rank1(nodes, wc, cn, kc, base + 15 * torch.arange(nt, device=DEV), self.rows, self.cols, self.vals)
        phase = (pos @ (self.randn(3, 3) * 12.0)).sin()
        self.b = torch.cat([0.01 * self.randn(off, 3) * RHO * H**3 * 1e-2,
                            mass * (1e-3 * phase + 2e-4 * self.randn(nv, 3))]).reshape(-1)

    # -- what the MAS needs --------------------------------------------------
    def adjacency(self):
        n = self.rest.shape[0]
        k = self.cells.shape[1]
        pairs = torch.cat([self.cells[:, [a, b]] for a in range(k) for b in range(k) if a != b])
        key = torch.unique(pairs[:, 0] * n + pairs[:, 1])
        start = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
        start[1:] = torch.bincount(key // n, minlength=n).cumsum(0)
        return start.int().cpu().numpy(), (key % n).int().cpu().numpy()

    def mas_args(self, partition: str):
        start, lst = self.adjacency()
        if partition == "graph":
            parts = partition_graph(start, lst)
        else:
            parts = partition_rcb(self.rest.cpu().numpy())
        p2r, r2p = partition_maps(parts)
        return (self.offset, self.rest.shape[0], start, lst, p2r, r2p)

    def abd(self):
        return (0, self.bodies) if self.bodies else None

    # -- plain torch, FP64 -----------------------------------------------------
    def upper(self):
        """(rowptr, col, blocks [U, 9]) of the block-upper matrix: runs summed."""
        keep = ((self.rows >= 0) & (self.rows <= self.cols)).nonzero().reshape(-1)
        key = self.rows[keep].long() * self.nb + self.cols[keep].long()
        uniq, inv = torch.unique(key, return_inverse=True)
        vals = torch.zeros(uniq.shape[0], 9, dtype=torch.float64, device=DEV).index_add_(0, inv, self.vals[keep])
        rowptr = torch.zeros(self.nb + 1, dtype=torch.int64, device=DEV)
        rowptr[1:] = torch.bincount(uniq // self.nb, minlength=self.nb).cumsum(0)
        return rowptr.int(), (uniq % self.nb).int(), vals

    def matvec(self):
        rowptr, col, vals = self.upper()
        j = col.long()
        i = torch.repeat_interleave(torch.arange(self.nb, device=DEV), (rowptr[1:] - rowptr[:-1]).long())
        blk = vals.view(-1, 3, 3).transpose(1, 2)  # [p, q]
        off = (i != j).nonzero().reshape(-1)

        def mul(x):
            x = x.reshape(-1, 3)
            y = torch.zeros_like(x)
            y.index_add_(0, i, torch.einsum("kpq,kq->kp", blk, x[j]))
            y.index_add_(0, j[off], torch.einsum("kpq,kp->kq", blk[off], x[i[off]]))
            return y.reshape(-1)

        return mul

    def field(self):
        """A smooth displacement of the block rows, flat."""
        n = self.nb - self.rest.shape[0]
        p = torch.cat([self.rand(n, 3), self.rest]) if n else self.rest
        return ((p @ (self.randn(3, 3) * 8.0) + self.randn(3)).sin() * 1e-3 + 1e-5 * self.randn(self.nb, 3)).reshape(-1)


def _precision(case) -> int:
    return _abi.B2S_PRECISION_MIXED if case["precision"] == "mixed" else _abi.B2S_PRECISION_FP64


def _deformed_bar(case, seed):
    """The bar's mesh and a bent, twisted, jittered state with its kinetic target (numpy / device)."""
    rest, tets = _lattice(case["cells"], case["across"], case["across"])
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed) % (1 << 62))
    x = rest.clone()
    th = (rest[:, 0] / rest[:, 0].max() - 0.5) * float(torch.rand(1, generator=gen, device=DEV)) * 1.5
    mid = 0.5 * rest.max(0).values
    y, z = rest[:, 1] - mid[1], rest[:, 2] - mid[2]
    x[:, 1] = mid[1] + th.cos() * y - th.sin() * z
    x[:, 2] = mid[2] + th.sin() * y + th.cos() * z
    x += 0.08 * H * (torch.rand(x.shape, generator=gen, device=DEV, dtype=torch.float64) - 0.5)
    xt = x + 1e-3 * H * torch.randn(x.shape, generator=gen, device=DEV, dtype=torch.float64)
    fixed = (rest[:, 0] < 0.5 * H) | (rest[:, 0] > rest[:, 0].max() - 0.5 * H)
    return rest, tets, x.reshape(-1).contiguous(), xt.reshape(-1).contiguous(), fixed


def prepare(case: dict, seed: int) -> dict:
    op = case["op"]
    if op == "generate":
        rest, tets, x, xt, fixed = _deformed_bar(case, seed)
        E, nu = MATERIAL["bar"]
        cfg = {"E": E, "nu": nu, "rho": RHO, "dt": DT, "kappa": 1e9, "dhat": 1e-3}
        mesh = GpuTetMesh(rest.cpu().numpy(), tets.cpu().numpy(), cfg, DEV, fixed=fixed.cpu().numpy())
        torch.cuda.synchronize()
        return {"case": case, "mesh": mesh, "x": x, "xt": xt}
    sysm = _System(case, seed)
    solver = Solver(0)
    st = {"case": case, "solver": solver, "nb": sysm.nb, "rows": sysm.rows, "cols": sysm.cols, "vals": sysm.vals,
          "b": sysm.b}
    if op == "assemble":
        st.update(_bsr_room(sysm))
    if op == "solve":
        pcg = B200PCG(tol_rate=case["tol"],
                      stop_rule=_abi.B2S_STOP_RZ if case["rule"] == "rz" else _abi.B2S_STOP_RELRES,
                      precision=_precision(case))
        pre = (B200MAS(*sysm.mas_args(case.get("partition", "rcb")), abd=sysm.abd()) if case["precond"] == "mas"
               else B200Jacobi(abd=sysm.abd()))
        st["system"] = GlobalLinearSystem(solver, pcg, pre)
    if op in ("pcg", "build", "spmv", "warm"):
        solver.assemble(sysm.nb, sysm.rows, sysm.cols, sysm.vals)
        for k in ("rows", "cols", "vals"):
            del st[k]
    if op in ("pcg", "build", "warm"):
        if case.get("precond", "mas") == "mas":
            solver.mas_init(*sysm.mas_args(case.get("partition", "rcb")))
        if sysm.bodies:
            solver.abd_init(*sysm.abd())
    if op in ("pcg", "warm"):
        solver.precond_assemble(_abi.B2S_PRECOND_JACOBI if case.get("precond") == "diag" else _abi.B2S_PRECOND_MAS)
        st["x"] = torch.zeros_like(sysm.b)
    if op in ("spmv", "build"):
        f = torch.float32 if case["precision"] == "mixed" else torch.float64
        st["b"] = (sysm.field() if op == "spmv" else sysm.b).to(f)
        st["x"] = torch.empty_like(st["b"])
    if op == "warm":
        mul = sysm.matvec()
        true = sysm.field()
        st["b"] = mul(true)
        amp = 0.3
        st["history"] = []
        for _ in range(case["history"]):
            st["history"].append(true + amp * sysm.field())
            amp *= 1.4
    torch.cuda.synchronize()
    return st


def _bsr_room(sysm) -> dict:
    """Room for the assembled matrix, sized by its number of distinct blocks."""
    keep = (sysm.rows >= 0) & (sysm.rows <= sysm.cols)
    u = int(torch.unique(sysm.rows[keep].long() * sysm.nb + sysm.cols[keep].long()).shape[0])
    return {"rowptr": torch.empty(sysm.nb + 1, dtype=torch.int32, device=DEV),
            "col": torch.empty(u, dtype=torch.int32, device=DEV),
            "val": torch.empty(u, 9, dtype=torch.float64, device=DEV)}


def run(st: dict):
    case = st["case"]
    op = case["op"]
    if op == "generate":
        return st["mesh"].system(st["x"], st["xt"])
    s = st["solver"]
    if op == "solve":
        return st["system"].solve(st["nb"], st["rows"], st["cols"], st["vals"], st["b"])
    if op == "assemble":
        s.assemble(st["nb"], st["rows"], st["cols"], st["vals"])
        s._check(s.lib.b2s_get_upper_bsr(s.h, st["rowptr"].data_ptr(), st["col"].data_ptr(), st["val"].data_ptr()))
        return st["rowptr"], st["col"], st["val"]
    if op == "spmv":
        dot = (s.spmv_mixed if case["precision"] == "mixed" else s.spmv)(st["b"], st["x"], with_dot=True)
        return st["x"], dot
    if op == "build":
        s.precond_assemble(_abi.B2S_PRECOND_MAS)
        (s.precond_apply_mixed if case["precision"] == "mixed" else s.precond_apply)(st["b"], st["x"])
        return st["x"]
    if op == "warm":
        s.ws_predict(st["b"], st["x"], st["history"], _abi.B2S_WS_MODE_HISTORY)
        return st["x"]
    s.pcg(st["b"], st["x"], tol=case["tol"],
          stop_rule=_abi.B2S_STOP_RZ if case["rule"] == "rz" else _abi.B2S_STOP_RELRES, precision=_precision(case))
    return st["x"]


# ---------------------------------------------------------------------------
# the least work, and what correct results look like
# ---------------------------------------------------------------------------
def _sizes(case):
    """Block rows, raw triplets, unique upper blocks, MAS vertices (the blocks to a few per cent)."""
    n = case["cells"]
    if case["scene"] == "stack":
        m, g = case["cubes"], n + 1
        nv, nt, c = m * g**3, 6 * m * n**3, (m - 1) * g * g
        return nv, nv + 10 * nt + g * g + 10 * c, 8 * nv + 3 * c, nv
    if case["scene"] == "bar":
        a = case["across"]
        nv, nt = (n + 1) * (a + 1) ** 2, 6 * n * a * a
        return nv, nv + 10 * nt, 8 * nv, nv
    nv, nbody, tri = n * n, case["bodies"], 2 * (n - 1) ** 2
    touch = int(0.36 * nv)
    T = nv + 6 * tri + 10 * ((n - 1) ** 2 + (n - 2) * (n - 1)) + 16 * nbody + 15 * touch
    return nv + 4 * nbody, T, 8 * nv + 4 * touch, nv


def _iterations(case) -> int:
    """PCG iterations, roughly (fitted to the listed cases)."""
    n = case["cells"]
    base = {"stack": 20 + 2.5 * n, "bar": 4.0 * n, "cloth": 25.0}[case["scene"]]
    if case["precond"] == "diag":
        base *= 2.5
    return int(base * (1.5 if case["tol"] < 1e-5 else 1.0)) + 1


def work(case: dict) -> dict:
    nb, T, U, nv = _sizes(case)
    op = case["op"]
    n = 3 * nb
    clusters = nv / 16 * 16 / 15  # every level together
    word = 4 if case.get("precision") == "mixed" else 8
    assemble = {"bytes": 80.0 * T + 76.0 * U, "flops": 9.0 * T}
    spmv = {"bytes": U * (4 + 9.0 * word) + 2.0 * n * word, "flops": 36.0 * U}
    inverse = 2 * 1176 * (2 if word == 4 else 4)  # one triangle of a 48 x 48 inverse, BF16 or FP32
    build = {"bytes": 76.0 * U + clusters * inverse / 2, "flops": 9.0 * U + clusters * 48.0**3}
    apply = {"bytes": clusters * inverse / 2 + 2.0 * n * word, "flops": clusters * 2 * 48.0**2}
    if case.get("precond") == "diag":
        build, apply = {"bytes": 72.0 * nb, "flops": 60.0 * nb}, {"bytes": 72.0 * nb, "flops": 18.0 * nb}
    pcg = {k: _iterations(case) * (spmv[k] + apply[k]) for k in spmv} if op in ("solve", "pcg") else None
    if op == "solve":
        return {k: assemble[k] + build[k] + pcg[k] for k in spmv}
    if op == "assemble":
        return assemble
    if op == "spmv":
        return spmv
    if op == "build":
        return {k: build[k] + apply[k] for k in spmv}
    if op == "pcg":
        return pcg
    if op == "warm":
        k = case["history"]
        return {"bytes": 76.0 * U + 8.0 * n * (k + 2), "flops": k * 36.0 * U + k * k * 6.0 * U}
    nt = (T - nb) // 10
    return {"bytes": 80.0 * T + nt * 16.0 + 3 * 24.0 * nb, "flops": nt * 3000.0}


def tolerance(case: dict):
    op = case["op"]
    mixed = case.get("precision") == "mixed"
    if op in ("solve", "pcg"):
        # the PCG stops at the first iteration that meets its rule, so another order of the same sums may stop an
        # iteration earlier or later, and the answers then differ by part of the error that the rule leaves. Measured
        # against the same solve in the other precision: up to 2e-3 under |r.z| <= 1e-3 |r0.z0|, 4e-6 at a relative
        # residual of 1e-4, 2e-7 at 1e-6 (FP32 recursion); the error left is 2e-2, 3e-5 and 2e-7
        return {"rel": 1e-2 if case["rule"] == "rz" else max(0.2 * case["tol"], 1e-6)}
    if op == "assemble":
        return {"rel": 1e-15}  # a few FP64 additions per entry: 4e-16 from another order
    if op == "spmv":
        return {"rel": 8e-6 if mixed else 2e-14}  # 1.9e-6 and 6e-15 from the FP64 sums in another order
    if op == "build":
        # 5e-4 from the FP64 inverses with BF16 entries of the scaled inverses, 9e-7 with FP32 ones
        return {"rel": 2e-3 if mixed else 4e-6}
    if op == "warm":
        return {"rel": 1e-13}  # 1.5e-14 from another order, with the Gram matrix of nearly parallel vectors
    return {"rel": 2e-13}  # 6e-14 from torch's own derivatives and eigenvalues (the gradient's cancellation)


# ---------------------------------------------------------------------------
# 64-bit answers in plain torch
# ---------------------------------------------------------------------------
def exact(case: dict, seed: int):
    op = case["op"]
    if op in ("solve", "pcg"):
        return None  # an iterate that meets the stop rule, not the solution itself
    if op == "generate":
        return _exact_generate(case, seed)
    sysm = _System(case, seed)
    if op == "assemble":
        return sysm.upper()
    if op == "spmv":
        mul = sysm.matvec()
        x = sysm.field()
        x = x.float().double() if case["precision"] == "mixed" else x
        y = mul(x)
        return y, float(x @ y)
    if op == "build":
        b = sysm.b.float().double() if case["precision"] == "mixed" else sysm.b
        return _exact_apply(sysm, case, b)
    mul = sysm.matvec()
    true = sysm.field()
    b = mul(true)
    amp, hist = 0.3, []
    for _ in range(case["history"]):
        hist.append(true + amp * sysm.field())
        amp *= 1.4
    V = torch.stack(hist, 1)
    AV = torch.stack([mul(h) for h in hist], 1)
    return V @ torch.linalg.solve(V.T @ AV, V.T @ b)


def _exact_apply(sysm, case, r):
    """z = P r of the MAS (and the bodies' 12x12 block Jacobi) with FP64 inverses."""
    off, vn, start, lst, p2r, r2p = sysm.mas_args(case.get("partition", "rcb"))
    slot = torch.from_numpy(r2p.astype(np.int64)).to(DEV)
    src = torch.repeat_interleave(torch.arange(vn, device=DEV),
                                  torch.from_numpy(np.diff(start).astype(np.int64)).to(DEV))
    dst = torch.from_numpy(lst.astype(np.int64)).to(DEV)
    rowptr, col, vals = sysm.upper()
    i = torch.repeat_interleave(torch.arange(sysm.nb, device=DEV), (rowptr[1:] - rowptr[:-1]).long())
    j = col.long()
    blk = vals.view(-1, 3, 3).transpose(1, 2)
    z = torch.zeros(sysm.nb, 3, dtype=torch.float64, device=DEV)
    rv = r.view(-1, 3)
    if sysm.bodies:
        n = 4 * sysm.bodies
        m = ((i < n) & (j < n) & (i // 4 == j // 4)).nonzero().reshape(-1)
        B = torch.zeros(sysm.bodies, 4, 4, 3, 3, dtype=torch.float64, device=DEV)
        B[i[m] // 4, i[m] % 4, j[m] % 4] = blk[m]
        B[i[m] // 4, j[m] % 4, i[m] % 4] = blk[m].transpose(1, 2)
        B = B.permute(0, 1, 3, 2, 4).reshape(-1, 12, 12)
        z[:n] = torch.linalg.solve(B, rv[:n].reshape(-1, 12, 1)).reshape(n, 3)
    levels, sz = 1, -(-max(len(p2r), vn) // 16) * 16
    while sz > 16:
        sz = -(-(sz // 16) // 16) * 16
        levels += 1
    levels = min(levels + 1, 6)
    inr = ((i >= off) & (j >= off)).nonzero().reshape(-1)
    a, b, ab = i[inr] - off, j[inr] - off, blk[inr]
    node, count = slot, len(p2r)
    valid = torch.from_numpy(p2r >= 0).to(DEV)
    for _ in range(levels):
        banks = -(-count // 16)
        # Galerkin matrices of this level's banks, zero diagonal entries -> 1
        na, nb_ = node[a], node[b]
        m = (na // 16 == nb_ // 16).nonzero().reshape(-1)
        G = torch.zeros(banks * 256, 3, 3, dtype=torch.float64, device=DEV)
        G.index_add_(0, na[m] * 16 + nb_[m] % 16, ab[m])
        m = m[a[m] != b[m]]
        G.index_add_(0, nb_[m] * 16 + na[m] % 16, ab[m].transpose(1, 2))
        G = G.view(banks, 16, 16, 3, 3).permute(0, 1, 3, 2, 4).reshape(banks, 48, 48)
        dg = torch.diagonal(G, dim1=1, dim2=2)
        dg[dg == 0] = 1.0
        R = torch.zeros(banks * 16, 3, dtype=torch.float64, device=DEV).index_add_(0, node, rv[off:off + vn])
        Z = torch.linalg.solve(G, R.view(banks, 48, 1)).reshape(-1, 3)
        z[off:off + vn] += Z[node]
        # the next level: connected components inside each bank, by bank then lowest lane
        C = torch.eye(16, dtype=torch.bool, device=DEV).expand(banks, 16, 16).clone().view(-1)
        ns, nd = node[src], node[dst]
        m = ns // 16 == nd // 16
        C[ns[m] * 16 + nd[m] % 16] = True
        C = C.view(banks, 16, 16).float()
        for _ in range(4):
            C = ((C @ C) > 0).float()
        lowest = C.argmax(2)
        alive = torch.zeros(banks * 16, dtype=torch.bool, device=DEV)
        alive[:count] = valid
        elected = (lowest == torch.arange(16, device=DEV)) & alive.view(banks, 16)
        rank = elected.reshape(-1).long().cumsum(0) - 1
        head = torch.arange(banks, device=DEV)[:, None] * 16 + lowest
        node = rank[head.reshape(-1)][node]
        count = int(elected.sum())
        valid = torch.ones(count, dtype=torch.bool, device=DEV)
    return z.reshape(-1)


def _exact_generate(case, seed):
    """Kinetic + stable Neo-Hookean blocks (PSD-projected) and the gradient, by torch's own derivatives."""
    rest, tets, x, xt, fixed = _deformed_bar(case, seed)
    E, nu = MATERIAL["bar"]
    mu, lam = E / (2 * (1 + nu)), E * nu / ((1 + nu) * (1 - 2 * nu))
    g, vol = _gradients(rest, tets)
    nv, nt = rest.shape[0], tets.shape[0]

    def psi(f):  # f: F column by column
        c0, c1, c2 = f[0:3], f[3:6], f[6:9]
        J = torch.dot(torch.linalg.cross(c0, c1), c2)
        return 0.5 * mu * (torch.dot(f, f) - 3.0) - mu * (J - 1.0) + 0.5 * lam * (J - 1.0) ** 2

    xv = x.view(-1, 3)
    F = torch.einsum("tqa,tqb->tba", xv[tets], g).reshape(-1, 9)
    grad, hess = torch.func.vmap(torch.func.grad(psi)), torch.func.vmap(torch.func.hessian(psi))
    rows, cols, vals = _triplets(nv + 10 * nt)
    out = torch.zeros_like(xv)
    mass = torch.zeros(nv, dtype=torch.float64, device=DEV)
    mass.index_add_(0, tets.reshape(-1), (vol * RHO / 4).repeat_interleave(4))
    v = torch.arange(nv, device=DEV)
    _upper(v, v, mass[:, None, None] * torch.eye(3, dtype=torch.float64, device=DEV), v, rows, cols, vals)
    out += mass[:, None] * (xv - xt.view(-1, 3))
    for lo in range(0, nt, 16384):
        s = slice(lo, min(lo + 16384, nt))
        w, Q = torch.linalg.eigh(hess(F[s]))
        Hs = (Q * w.clamp(min=0.0)[:, None, :]) @ Q.transpose(1, 2)
        Hs = Hs.view(-1, 3, 3, 3, 3) * (vol[s] * DT * DT)[:, None, None, None, None]  # [b, a, d, c]
        P = grad(F[s]).view(-1, 3, 3) * (vol[s] * DT * DT)[:, None, None]  # [b, a]
        out.index_add_(0, tets[s].reshape(-1), torch.einsum("tba,tqb->tqa", P, g[s]).reshape(-1, 3))
        pair = 0
        for q in range(4):
            for r in range(q, 4):
                B = torch.einsum("tb,tbadc,td->tac", g[s, q], Hs, g[s, r])
                at = nv + 10 * torch.arange(s.start, s.stop, device=DEV) + pair
                _upper(tets[s, q], tets[s, r], B, at, rows, cols, vals)
                pair += 1
    fr, fc = fixed[rows.long()], fixed[cols.long()]
    vals[fr | fc] = 0.0
    vals[(fr | fc) & (rows == cols)] = torch.eye(3, dtype=torch.float64, device=DEV).reshape(9)
    out[fixed] = 0.0
    return rows, cols, vals, out.reshape(-1)
