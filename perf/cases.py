"""What this framework's users have it compute, as measurable cases.

A case names a kind of call and its sizes.  ``prepare`` builds what the program holds before the call (the
operator's plan, the cells, output buffers, a stepper or a ragged batch), ``run`` makes one call through the
package's public entry points, ``work`` counts what the call cannot do without, and ``exact`` gives the result
in plain torch float64.

The operator is the hard-sphere collision operator (gamma = 1): its reduced radial tensor up to L = 16 and
K = 12 is the repository's committed quadrature, and the operator of any smaller (L, K) is a part of it, since
a triplet's K x K x K block does not depend on where L and K are cut off.  Cells are Maxwellians with small
drifts and temperature changes plus a perturbation that falls off with degree, as in the benchmark.
"""
from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "collision-factorization_b200"))

import cf_b200  # noqa: E402
from cf_b200 import geometry, implicit, ragged, rtensor, stepping  # noqa: E402

R_FILE = os.path.join("tests", "golden", "R_hs_k11_l16_pad20.npy")
BUCKETS = ((4, 4), (6, 6), (8, 6), (10, 8))  # (L, K) of a mixed-resolution run, finest last
SHARES = (0.4, 0.3, 0.2, 0.1)
PAD = 20  # quadrature padding of the reference's precomputed operators


def listed():
    return [
        # one distribution function through the MEX signature, the reference's own way of calling it
        {"name": "mex_single_l4_k4", "kind": "mex", "L": 4, "K": 4, "B": 1},
        # a few tens of cells on the device with the default form, at the size of a shipped operator (K_max = 4)
        {"name": "q_l4_k5_b100", "kind": "q", "form": "af", "L": 4, "K": 5, "B": 100},
        # the largest shipped operator (K_max = 4, L = 12) over a field of cells
        {"name": "q_l12_k5_b2048", "kind": "q", "form": "af_sym", "L": 12, "K": 5, "B": 2048},
        # the benchmark's default workload
        {"name": "q_l10_k8_b4096", "kind": "q", "form": "af_sym", "L": 10, "K": 8, "B": 4096},
        # the finest resolution, in double and in single precision
        {"name": "q_l16_k12_b1024", "kind": "q", "form": "af_sym", "L": 16, "K": 12, "B": 1024},
        {"name": "q32_l16_k12_b1024", "kind": "q", "form": "af_sym_f32", "L": 16, "K": 12, "B": 1024},
        # Jacobian applies, as a Krylov solver or a linear stability study makes them
        {"name": "jv_l10_k8_b4096", "kind": "jv", "L": 10, "K": 8, "B": 4096},
        # a field of mixed resolutions, one graph replay per time step
        {"name": "ragged_b16384", "kind": "ragged", "B": 16384},
        # an implicit step's linear solve with the Maxwellian block preconditioner
        {"name": "gmres_l8_k8_b2048", "kind": "gmres", "L": 8, "K": 8, "B": 2048, "dt_nu": 10.0},
        # explicit stepping of an odd-sized field with the default form, four steps per graph replay
        {"name": "rk2_l8_k6_b1001", "kind": "rk2", "form": "af", "L": 8, "K": 6, "B": 1001, "steps": 4},
        # a batch in host memory through the batched MEX-style call
        {"name": "host_l10_k8_b1500", "kind": "host", "form": "af_sym", "L": 10, "K": 8, "B": 1500},
        # computing an operator: the reduced radial tensor at the shipped K_max = 4, L = 4
        {"name": "rtensor_l4_k5", "kind": "rtensor", "L": 4, "K": 5},
    ]


def draw(rng):
    kind = rng.choice(["mex", "q", "q", "q", "jv", "jv", "ragged", "gmres", "rk2", "host", "rtensor"])
    if kind == "mex":
        L, K = rng.randint(2, 6), rng.randint(3, 8)
        return {"kind": kind, "L": L, "K": K, "B": 1}
    if kind == "rtensor":
        return {"kind": kind, "L": rng.randint(2, 4), "K": rng.randint(3, 5)}
    if kind == "ragged":
        return {"kind": kind, "B": _log_int(rng, 512, 16384)}
    if kind == "gmres":
        L, K = rng.randint(3, 8), rng.choice([4, 5, 6, 8])
        return {"kind": kind, "L": L, "K": K, "B": _log_int(rng, 32, 2048), "dt_nu": rng.choice([1.0, 10.0, 100.0])}
    L, K = rng.randint(3, 12), rng.choice([3, 4, 5, 6, 7, 8, 8, 10, 12])
    if K <= 5 or K == 12:
        L = rng.randint(3, 16)
    case = {"kind": kind, "L": L, "K": K, "B": 0}
    passes = 4 if kind == "jv" else 1  # J.v does twice a Q's work per cell, and less of it per load
    if kind == "q":
        case["form"] = rng.choice(["af", "af_sym", "af_sym"] + (["af_sym_f32"] if K in (4, 6, 8, 12) else []))
    elif kind == "host":
        case["form"] = rng.choice(["af", "af_sym"])
    elif kind == "rk2":
        case["form"], case["steps"] = rng.choice(["af", "af_sym"]), rng.choice([1, 2, 4])
        passes = 2 * case["steps"]
    if case.get("form") == "af":
        passes *= 2
    # no more work than 1024 cells at L = 16, K = 12
    top = int(min(4096, 8.0e10 / (passes * _counts(L)["entries"] * K * K * 2)))
    case["B"] = _log_int(rng, min(16, top), top)
    return case


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# ------------------------------------------------------------------------------ operators and cells
@functools.lru_cache(maxsize=None)
def _geo(L):
    return geometry.generate_geometry(L)


@functools.lru_cache(maxsize=None)
def _triplets16():
    tri = [(a, b, c) for a in range(17) for b in range(17) for c in range(17)
           if abs(a - b) <= c <= a + b and (a + b + c) % 2 == 0]
    return {t: i for i, t in enumerate(tri)}


@functools.lru_cache(maxsize=None)
def _R_full():
    return np.load(R_FILE)


@functools.lru_cache(maxsize=None)
def _operator(L, K):
    """The operator's host arrays: labels, vals, ic_map, R (sorted for the contraction) and its triplets."""
    g = geometry.sort_for_contraction(_geo(L))
    at = [_triplets16()[tuple(int(x) for x in t)] for t in g.l_triplets]
    R = np.asfortranarray(_R_full()[:K, :K, :K][..., at])
    return np.asfortranarray(g.labels), g.vals, g.ic_map, R, g.l_triplets


@functools.lru_cache(maxsize=None)
def _counts(L):
    """Entries, (triplet, q1, q2) runs and (triplet, q1) slices of the list folded over q2 <-> q3."""
    g = _geo(L)
    q = g.labels.astype(np.int64) - 1
    l = np.floor(np.sqrt(q)).astype(np.int64)
    keep = (l[:, 1] < l[:, 2]) | ((l[:, 1] == l[:, 2]) & (q[:, 1] <= q[:, 2]))
    nq = (L + 1) ** 2
    sl = g.ic_map[keep].astype(np.int64) * nq + q[keep, 0]
    return {"entries": int(keep.sum()), "slices": int(np.unique(sl).size),
            "runs": int(np.unique(sl * nq + q[keep, 1]).size)}


def _plan(L, K):
    lab, val, ic, R, _ = _operator(L, K)
    return cf_b200.CollisionOperator(lab, val, ic, R, (L + 1) ** 2, K, device=torch.cuda.current_device())


def _cells(L, K, B, seed, decay=0.6):
    """[B, K, N_Q] float64 on the device."""
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed) * 1000003 + 17)
    l = torch.arange((L + 1) ** 2, device=dev).double().sqrt().floor()
    k = torch.arange(K, device=dev).double()
    w = 1e-2 * torch.exp(-decay * (k[:, None] + l[None, :]))
    f = torch.randn((B, K, l.numel()), dtype=torch.float64, device=dev, generator=gen) * w
    f[:, 0, 0] += 1.0
    if L >= 1:
        f[:, 0, 1:4] += 0.1 * torch.randn((B, 3), dtype=torch.float64, device=dev, generator=gen)
    if K >= 2:
        f[:, 1, 0] += 0.1 * torch.randn(B, dtype=torch.float64, device=dev, generator=gen)
    return f


def _directions(L, K, B, seed):
    v = _cells(L, K, B, int(seed) + 500, decay=0.3)
    v[:, 0, 0] -= 1.0
    return (v / v.flatten(1).norm(dim=1)[:, None, None]).contiguous()


def _bucket_counts(B):
    n = [int(B * s) for s in SHARES[:-1]]
    return n + [B - sum(n)]


def _nu(L, K):
    """The decay rate of the equilibrium's first stress mode, the time scale of the implicit steps."""
    _, _, _, R, tri = _operator(L, K)
    # dQ/df at f = e(k = 0, q = 0) couples a mode to itself through the triplets (2, 0, 2) and (2, 2, 0)
    y00 = 1.0 / math.sqrt(4.0 * math.pi)
    return abs(sum(float(R[0, 0, 0, i]) for i, t in enumerate(tri) if tuple(t) in ((2, 0, 2), (2, 2, 0))) * y00)


def _host(f):
    """A batch as the MEX-style calls take it: column-major [N_Q x K x B] in host memory."""
    return np.asfortranarray(f.cpu().numpy().transpose(2, 1, 0))


# ------------------------------------------------------------------------------ the cases
def prepare(case, seed):
    kind, L, K, B = case["kind"], case.get("L"), case.get("K"), case.get("B")
    if kind == "rtensor":
        gamma = float(np.random.default_rng(seed).uniform(0.0, 1.0))  # a variable-hard-sphere exponent
        return {"kind": kind, "args": rtensor.sumfac_inputs(_geo(L), K - 1, gamma, PAD, PAD)}
    if kind == "ragged":
        counts = _bucket_counts(B)
        ops = [_plan(*b) for b in BUCKETS]
        rb = ragged.RaggedBatch(ops, counts, ["af_sym"] * len(BUCKETS), tail_split=4, family="tile")
        fs = [_cells(*b, n, seed + i) for i, (b, n) in enumerate(zip(BUCKETS, counts))]
        return {"kind": kind, "batch": rb, "f": fs, "q": [torch.zeros_like(f) for f in fs]}
    if kind in ("mex", "host"):
        f = _host(_cells(L, K, B, seed))
        f = np.asfortranarray(f[:, :, 0]) if kind == "mex" else f
        return {"kind": kind, "f": f, "q": np.zeros_like(f, order="F"), "op": _operator(L, K)[:4], "L": L, "K": K,
                "form": case.get("form")}
    op, f = _plan(L, K), _cells(L, K, B, seed)
    if kind == "q":
        return {"kind": kind, "op": op, "f": f, "form": case["form"]}
    if kind == "jv":
        return {"kind": kind, "op": op, "f": f, "v": _directions(L, K, B, seed)}
    if kind == "rk2":
        st = stepping.RK2Stepper(op, f, form=case["form"])
        return {"kind": kind, "stepper": st, "start": st.state.clone(), "dt": 0.2 / _nu(L, K), "steps": case["steps"]}
    dt = case["dt_nu"] / _nu(L, K)
    return {"kind": kind, "op": op, "f": f, "b": _directions(L, K, B, seed), "dt": dt,
            "P": torch.from_numpy(implicit.block_preconditioner(op, dt)).to(f.device)}


def run(state):
    kind = state["kind"]
    if kind == "q":
        return state["op"].q(state["f"], form=state["form"])
    if kind == "jv":
        return state["op"].jv(state["f"], state["v"], folded=True)
    if kind == "ragged":
        for q in state["q"]:
            q.zero_()
        return state["batch"].q_graph(state["f"], state["q"])
    if kind == "gmres":
        # the solution alone: the iteration counts and the last residuals hang on rounding
        return implicit.gmres_solve(state["op"], state["f"], state["b"], state["dt"], precond=state["P"])[0]
    if kind == "rk2":
        st = state["stepper"]
        st.state.copy_(state["start"])
        st.step_graph(state["dt"], state["steps"])
        return st.cells()
    if kind == "rtensor":
        return rtensor.compute_R(state["args"], device=torch.cuda.current_device())
    state["q"][...] = 0.0
    args = (state["q"], state["f"], *state["op"], (state["L"] + 1) ** 2, state["K"])
    if kind == "mex":
        cf_b200.angular_first_collision_kernel_mex(*args)
    else:
        cf_b200.contract_batched(*args, form=state["form"])
    return state["q"]


# ------------------------------------------------------------------------------ what a pass needs
def _flops(L, K, jv=False):
    """Angular first over the folded list: the Gaunt sums, the outer products and the K^3 step, per cell."""
    c, n = _counts(L), 2 if jv else 1
    return 2.0 * (n * (c["entries"] * K + c["runs"] * K * K) + c["slices"] * K ** 3)


def _op_bytes(L, K):
    c = _counts(L)
    return 12.0 * c["entries"] + 8.0 * K ** 3 * len(_operator(L, K)[4]) / 2


def work(case):
    kind = case["kind"]
    if kind == "ragged":
        n = _bucket_counts(case["B"])
        return {"bytes": sum(16.0 * (l + 1) ** 2 * k * c + _op_bytes(l, k) for (l, k), c in zip(BUCKETS, n)),
                "flops": sum(_flops(l, k) * c for (l, k), c in zip(BUCKETS, n))}
    L, K = case["L"], case["K"]
    M = (L + 1) ** 2 * K
    if kind == "rtensor":
        s = rtensor.grid_sizes(K - 1, L, PAD, PAD)
        inner = s["N_chi"] * s["N_eps"]
        outer = s["N_x"] * (s["N_u1"] + s["N_y2"] * s["N_t2"])
        points = s["N_x"] * (s["N_u1"] * s["N_t1"] + s["N_y2"] * s["N_t2"]) * inner
        n_l = len(_operator(L, K)[4])
        # per point and per post-collision velocity, the angular x radial products; per item, a rank-2 update of R
        return {"bytes": 8.0 * (K ** 3 * n_l + s["N_t1"] * s["N_u1"] * (L + 1) ** 2 * n_l),
                "flops": 4.0 * points * M + 2.0 * outer * n_l * K * K * K}
    B = case["B"]
    if kind == "jv":
        return {"bytes": 24.0 * M * B + _op_bytes(L, K), "flops": _flops(L, K, True) * B}
    if kind == "gmres":  # at least six Arnoldi steps and a last residual: one J.v and the vector passes each
        return {"bytes": 6 * 40.0 * M * B + _op_bytes(L, K), "flops": 7 * _flops(L, K, True) * B}
    n = 2 * case["steps"] if kind == "rk2" else 1
    return {"bytes": 16.0 * M * B + _op_bytes(L, K), "flops": n * _flops(L, K) * B}


# ------------------------------------------------------------------------------ the same in plain torch
@functools.lru_cache(maxsize=2)
def _dense(L, K):
    """[(l1, l2, l3, G [d1, d2, d3], R [K, K, K])] on the device, one per triplet."""
    lab, val, ic, R, tri = _operator(L, K)
    q, t = lab.astype(np.int64) - 1, ic.astype(np.int64) - 1
    out = []
    for i, (a, b, c) in enumerate(tri):
        z = np.flatnonzero(t == i)
        G = np.zeros((2 * a + 1, 2 * b + 1, 2 * c + 1))
        G[q[z, 0] - a * a, q[z, 1] - b * b, q[z, 2] - c * c] = val[z]
        out.append((int(a), int(b), int(c), torch.from_numpy(G).cuda(),
                    torch.from_numpy(np.ascontiguousarray(R[..., i])).cuda()))
    return out


def _rows(l):
    return slice(l * l, (l + 1) ** 2)


def _bilinear(L, K, f, g):
    """sum G R f(q2, k2) g(q3, k3) for cells [B, K, N_Q]."""
    B = f.shape[0]
    out = torch.zeros_like(f)
    for b0 in range(0, B, 256):
        fb, gb = f[b0:b0 + 256], g[b0:b0 + 256]
        n = fb.shape[0]
        for a, b, c, G, R in _dense(L, K):
            d1 = 2 * a + 1
            h = torch.matmul(gb[:, :, _rows(c)], G.permute(2, 0, 1).reshape(2 * c + 1, -1))  # [n, k3, q1 q2]
            h = h.view(n, K, d1, 2 * b + 1).permute(0, 2, 3, 1)  # [n, q1, q2, k3]
            phi = torch.matmul(fb[:, :, _rows(b)].unsqueeze(1), h)  # [n, q1, k2, k3]
            out[b0:b0 + 256, :, _rows(a)] += torch.matmul(R.reshape(K, K * K), phi.reshape(n, d1, K * K).transpose(1, 2))
    return out


def _jacobian(L, K, f):
    """J(f) [B, M, M] with rows and columns k N_Q + q."""
    B, nq = f.shape[0], (L + 1) ** 2
    J = torch.zeros((B, K, nq, K, nq), dtype=f.dtype, device=f.device)
    for a, b, c, G, R in _dense(L, K):
        for other, mine, g, r in ((c, b, G, R), (b, c, G.transpose(1, 2), R.transpose(1, 2))):
            # g [q1, mine, other], r [k1, k_mine, k_other]
            y = torch.matmul(f[:, :, _rows(other)].transpose(1, 2), r.reshape(K * K, K).T)  # [B, other, k1 k_mine]
            x = torch.matmul(g.reshape(-1, 2 * other + 1), y)  # [B, q1 mine, k1 k_mine]
            x = x.view(B, 2 * a + 1, 2 * mine + 1, K, K).permute(0, 3, 1, 4, 2)
            J[:, :, _rows(a), :, _rows(mine)] += x
    return J.view(B, K * nq, K * nq)


def exact(case, seed):
    kind, L, K, B = case["kind"], case.get("L"), case.get("K"), case.get("B")
    if kind == "rtensor":
        return None
    if kind == "ragged":
        return [_bilinear(*b, f, f) for b, f in
                ((b, _cells(*b, n, seed + i)) for i, (b, n) in enumerate(zip(BUCKETS, _bucket_counts(B))))]
    f = _cells(L, K, B, seed)
    if kind in ("mex", "host"):
        q = _host(_bilinear(L, K, f, f))
        return np.asfortranarray(q[:, :, 0]) if kind == "mex" else q
    if kind == "q":
        return _bilinear(L, K, f, f)
    if kind == "jv":
        v = _directions(L, K, B, seed)
        return _bilinear(L, K, v, f) + _bilinear(L, K, f, v)
    if kind == "rk2":
        dt = 0.2 / _nu(L, K)
        for _ in range(case["steps"]):
            q = _bilinear(L, K, f, f)
            p = f + dt * q
            f = f + 0.5 * dt * (q + _bilinear(L, K, p, p))
        return f
    dt, b = case["dt_nu"] / _nu(L, K), _directions(L, K, B, seed)
    x = torch.empty_like(b)
    for b0 in range(0, B, 128):
        A = -dt * _jacobian(L, K, f[b0:b0 + 128])
        A.diagonal(dim1=1, dim2=2).add_(1.0)
        x[b0:b0 + 128] = torch.linalg.solve(A, b[b0:b0 + 128].flatten(1).unsqueeze(2)).view_as(x[b0:b0 + 128])
    return x
