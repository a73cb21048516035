"""The work that a user of this framework has it do, as cases to be timed.

The framework fits quantum circuits to unitaries, so the calls that carry a user's
program are: f, gradient and Hessian-vector product of a brickwall or a general
circuit (one inner step of the matrix-free trust region), the dense Hessian (one step
of the full-Hessian trust region), its sampled and block-encoding forms, many small
problems in one batch, gates on one large state, and the two optimisers of the Python
module.  Every case goes through the package's public functions with host gates, as a
program calls them; only the large states of `apply` live on the GPU.

`exact` restates the same sums with plain torch in complex128 (states as matrices,
one column per basis state, forward and adjoint sweeps gate by gate).
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from rqcopt_hpc_b200 import batch, gpu, real, rqcopt_hpc
from rqcopt_hpc_b200.abi import Statevector

PRECISION = {"c128": gpu.PRECISION_C128, "mixed": gpu.PRECISION_MIXED, "c64": gpu.PRECISION_C64}


# ------------------------------------------------------------------------------ cases

def listed():
    return [
        # the smallest call: one tCG step of a six-qubit fit, bound by latency and launches
        {"name": "hvp_L6", "kind": "hvp", "L": 6, "depth": 5, "tdepth": 3, "precision": "c128", "perms": "ring"},
        # the two optimisers of the Python module on their ordinary sizes (a five-qubit
        # circuit of 18 gates, a brickwall on eight qubits, both against a dense unitary)
        {"name": "module_circuit_L5", "kind": "module_circuit", "L": 5, "ngates": 18, "niter": 4},
        {"name": "module_brickwall_L8", "kind": "module_brickwall", "L": 8, "depth": 5, "niter": 4, "nsamples": 0},
        # one tCG step of an ordinary and of a large fit (forward and adjoint sweeps over all basis columns)
        {"name": "hvp_L12", "kind": "hvp", "L": 12, "depth": 9, "tdepth": 5, "precision": "c128", "perms": "ring"},
        {"name": "hvp_L14", "kind": "hvp", "L": 14, "depth": 9, "tdepth": 5, "precision": "c128", "perms": "ring"},
        # the same step with complex64 passes, as a mixed-precision run makes it
        {"name": "hvp_c64_L14", "kind": "hvp", "L": 14, "depth": 9, "tdepth": 5, "precision": "c64", "perms": "ring"},
        # f and gradient of a general circuit: gates on arbitrary pairs of an odd number of wires
        {"name": "circuit_gradient_L11", "kind": "circuit", "L": 11, "ngates": 61, "tgates": 20, "what": "gradient"},
        # one step of the full-Hessian trust region
        {"name": "hessian_L10", "kind": "hessian", "L": 10, "depth": 7, "tdepth": 3},
        # the same from Haar-random states, for registers too large for all columns
        {"name": "sampled_L14", "kind": "sampled", "L": 14, "depth": 8, "tdepth": 4, "nsamples": 32},
        # block encoding of a six-qubit operator
        {"name": "blockenc_L12", "kind": "blockenc", "L": 12, "depth": 9, "hdepth": 3},
        # many small fits at once, each at its own size (complex64, as the batched runs use it)
        {"name": "batch_c64", "kind": "batch", "count": 48, "precision": "c64", "mix": 0},
        # gates on one large state that stays on the GPU
        {"name": "apply_L27", "kind": "apply", "L": 27, "ngates": 64, "dtype": "c128"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: the kinds above over their sizes, with the variants that are used
    beside them (f or gradient alone, real-orthogonal circuits, arbitrary wire orders)."""
    kind = rng.choice(["hvp", "hvp", "gradient", "f", "circuit", "hessian", "sampled", "blockenc", "batch", "apply",
                       "real", "module_circuit", "module_brickwall"])
    if kind in ("hvp", "gradient", "f"):
        return {"kind": kind, "L": rng.choice([4, 6, 8, 10, 12, 14]), "depth": rng.randint(2, 9),
                "tdepth": rng.randint(1, 5), "precision": rng.choice(["c128", "c128", "c64"]),
                "perms": rng.choice(["ring", "ring", "ring", "any"])}
    if kind == "circuit":
        return {"kind": kind, "L": rng.randint(4, 12), "ngates": _log(rng, 8, 90), "tgates": _log(rng, 4, 40),
                "what": rng.choice(["f", "gradient", "hvp"])}
    if kind == "hessian":
        return {"kind": kind, "L": rng.choice([4, 6, 8, 10]), "depth": rng.randint(2, 9), "tdepth": rng.randint(1, 5)}
    if kind == "sampled":
        return {"kind": kind, "L": rng.choice([6, 8, 10, 12, 14]), "depth": rng.randint(3, 8), "tdepth": rng.randint(1, 5),
                "nsamples": _log(rng, 5, 64)}
    if kind == "blockenc":
        return {"kind": kind, "L": rng.choice([4, 8, 12]), "depth": rng.randint(3, 9), "hdepth": rng.randint(1, 4)}
    if kind == "batch":
        precision = rng.choice(["c64", "c64", "mixed", "c128"])
        return {"kind": kind, "count": _log(rng, 4, 64 if precision == "c64" else 24), "precision": precision,
                "mix": rng.randint(1, 1 << 20)}
    if kind == "apply":
        dtype = rng.choice(["c128", "c64"])
        return {"kind": kind, "L": rng.randint(10, 27 if dtype == "c128" else 28), "ngates": _log(rng, 5, 70), "dtype": dtype}
    if kind == "real":
        return {"kind": kind, "L": rng.choice([4, 6, 8, 10, 12]), "depth": rng.randint(2, 9), "tdepth": rng.randint(1, 5)}
    if kind == "module_circuit":
        return {"kind": kind, "L": rng.randint(3, 7), "ngates": _log(rng, 5, 30), "niter": rng.randint(2, 5)}
    return {"kind": kind, "L": rng.choice([4, 6, 8]), "depth": rng.randint(2, 5), "niter": rng.randint(2, 5),
            "nsamples": rng.choice([0, 0, 24])}


# ------------------------------------------------------------------------------ inputs

def _haar(rng, n=4):
    z = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(2)
    q, r = np.linalg.qr(z)
    d = np.diagonal(r)
    return q * (d / np.abs(d))


def _orth(rng):
    q, r = np.linalg.qr(rng.standard_normal((4, 4)))
    return q * np.sign(np.diagonal(r))


def _haar_stack(rng, n):
    return np.stack([_haar(rng) for _ in range(n)])


def _perms(rng, L, nlayers, kind):
    """Layers of neighbouring pairs, alternately shifted by one wire (ring), or an
    arbitrary order of the wires in every layer."""
    if kind == "ring":
        return np.stack([np.roll(np.arange(L), -(l % 2)) for l in range(nlayers)]).astype(np.int32)
    return np.stack([rng.permutation(L) for _ in range(nlayers)]).astype(np.int32)


def _antisymm(r):
    """16 reals as an anti-Hermitian matrix."""
    w = np.zeros((4, 4), np.complex128)
    for a in range(4):
        w[a, a] = 1j * r[5 * a]
        for c in range(a + 1, 4):
            p, q = r[4 * a + c], r[4 * c + a]
            w[a, c] = 0.5 * (p - q) + 0.5j * (p + q)
            w[c, a] = -np.conj(w[a, c])
    return w


def _tangents(rng, gates):
    return np.stack([g @ _antisymm(rng.standard_normal(16)) for g in gates])


def _wires(rng, L, n):
    return np.array([rng.choice(L, 2, replace=False) for _ in range(n)], np.int32)


def _batch_problems(case, rng):
    """Fits of four sizes in even shares, depths 3 to 9, each against a target of its own."""
    order = np.random.default_rng(case["mix"])
    out = []
    for _ in range(case["count"]):
        L, depth = int(order.choice([6, 8, 10, 12])), int(order.choice([3, 5, 7, 9]))
        out.append((L, _haar_stack(rng, depth), _perms(rng, L, depth, "ring"), _haar_stack(rng, 3),
                    _perms(rng, L, 3, "ring")))
    return out, [_tangents(rng, p[1]) for p in out]


def _inputs(case, seed):
    """The arrays of a case, from the seed alone."""
    rng = np.random.default_rng(seed)
    k, L = case["kind"], case.get("L")
    if k in ("hvp", "gradient", "f", "hessian", "sampled"):
        style = case.get("perms", "ring")
        v, p = _haar_stack(rng, case["depth"]), _perms(rng, L, case["depth"], style)
        tv, tp = _haar_stack(rng, case["tdepth"]), _perms(rng, L, case["tdepth"], style)
        return {"v": v, "p": p, "tv": tv, "tp": tp, "z": _tangents(rng, v), "seed": int(rng.integers(1 << 40))}
    if k == "real":
        v = np.stack([_orth(rng) for _ in range(case["depth"])])
        tv = np.stack([_orth(rng) for _ in range(case["tdepth"])])
        w = np.zeros((case["depth"], 4, 4))
        for l in range(case["depth"]):
            w[l][np.triu_indices(4, 1)] = rng.standard_normal(6)
        return {"v": v, "p": _perms(rng, L, case["depth"], "ring"), "tv": tv, "tp": _perms(rng, L, case["tdepth"], "ring"),
                "z": v @ (w - w.transpose(0, 2, 1))}
    if k == "circuit":
        g, w = _haar_stack(rng, case["ngates"]), _wires(rng, L, case["ngates"])
        return {"g": g, "w": w, "tg": _haar_stack(rng, case["tgates"]), "tw": _wires(rng, L, case["tgates"]),
                "z": _tangents(rng, g)}
    if k == "blockenc":
        return {"v": _haar_stack(rng, case["depth"]), "p": _perms(rng, L, case["depth"], "ring"),
                "tv": _haar_stack(rng, case["hdepth"]), "tp": _perms(rng, L // 2, case["hdepth"], "ring")}
    if k == "apply":
        return {"g": _haar_stack(rng, case["ngates"]), "w": _wires(rng, L, case["ngates"])}
    if k == "module_circuit":
        return {"u": np.ascontiguousarray(_haar(rng, 1 << L)), "g": _haar_stack(rng, case["ngates"]),
                "w": _wires(rng, L, case["ngates"])}
    if k == "module_brickwall":
        return {"u": np.ascontiguousarray(_haar(rng, 1 << L)), "v": _haar_stack(rng, case["depth"]),
                "p": _perms(rng, L, case["depth"], "ring")}
    problems, dirs = _batch_problems(case, rng)
    return {"problems": problems, "dirs": dirs}


def _state(case, seed, device):
    gen = torch.Generator(device=device).manual_seed(seed)
    psi = torch.randn(1 << case["L"], dtype=torch.complex128 if case["dtype"] == "c128" else torch.complex64,
                      device=device, generator=gen)
    return psi / torch.linalg.vector_norm(psi)


# ------------------------------------------------------------------------------ the calls

def prepare(case, seed):
    """What a program holds before the call: gates, layouts and targets (host arrays);
    for `apply` the state on the GPU and the one that is written."""
    s = {"case": case, **_inputs(case, seed)}
    k = case["kind"]
    if k in ("hvp", "gradient", "f", "hessian", "sampled", "blockenc"):
        s["target"] = gpu.Target(brickwall=(s["tv"], s["tp"]))
    elif k == "circuit":
        s["target"] = gpu.Target(circuit=(s["tg"], s["tw"]))
    elif k == "real":
        s["target"] = real.Target(brickwall=(s["tv"], s["tp"]))
    elif k == "apply":
        s["psi"] = _state(case, seed, "cuda")
        s["out"] = torch.empty_like(s["psi"])
    return s


def run(s):
    c = s["case"]
    k, L = c["kind"], c.get("L")
    if k != "batch":
        gpu.set_precision(PRECISION[c.get("precision", "c128")])
    if k == "hvp":
        return gpu.brickwall_unitary_target_projected_hessian_vector_product(s["target"], s["v"], s["z"], s["p"], L)
    if k == "gradient":
        return gpu.brickwall_unitary_target_and_projected_gradient(s["target"], s["v"], s["p"], L)
    if k == "f":
        return gpu.brickwall_unitary_target(s["target"], s["v"], s["p"], L)
    if k == "circuit":
        if c["what"] == "f":
            return gpu.circuit_unitary_target(s["target"], s["g"], s["w"], L)
        if c["what"] == "gradient":
            return gpu.circuit_unitary_target_and_projected_gradient(s["target"], s["g"], s["w"], L)
        return gpu.circuit_unitary_target_projected_hessian_vector_product(s["target"], s["g"], s["z"], s["w"], L)
    if k == "hessian":
        return gpu.brickwall_unitary_target_gradient_vector_hessian_matrix(s["target"], s["v"], s["p"], L)
    if k == "sampled":
        return gpu.brickwall_unitary_target_gradient_vector_hessian_matrix_sampling(
            s["target"], s["v"], s["p"], L, c["nsamples"], gpu.seed_rng_state(s["seed"]))
    if k == "blockenc":
        return gpu.brickwall_blockenc_target_gradient_vector_hessian_matrix(s["target"], s["v"], s["p"], L)
    if k == "batch":
        f, g, h = batch.evaluate(s["problems"], s["dirs"], batch.EVAL_HVP, PRECISION[c["precision"]])
        return f, np.concatenate(g), np.concatenate(h)
    if k == "real":
        return real.brickwall_unitary_target_projected_hessian_vector_product(s["target"], s["v"], s["z"], s["p"], L)
    if k == "module_circuit":
        return rqcopt_hpc.optimize_quantum_circuit(L, s["u"], s["g"], s["w"], c["niter"])
    if k == "module_brickwall":
        return rqcopt_hpc.optimize_brickwall_circuit(L, s["u"], s["v"], s["p"], c["niter"], c["nsamples"])
    g, w, a, b = s["g"], s["w"], s["psi"], s["out"]
    if c["dtype"] == "c128":
        ret = gpu.lib().apply_quantum_circuit(g.ctypes.data, len(g), w.ctypes.data,
                                              ctypes.byref(Statevector(a.data_ptr(), L)),
                                              ctypes.byref(Statevector(b.data_ptr(), L)))
    else:
        ret = gpu.lib().rqcopt_apply_quantum_circuit_c64(g.ctypes.data, len(g), w.ctypes.data, a.data_ptr(),
                                                         b.data_ptr(), L)
    if ret != 0:
        raise gpu.RqcError("apply_quantum_circuit", ret)
    return b


# ------------------------------------------------------------------------------ work

def _orbits(L, case):
    """Basis columns the sum over all 2^L needs at least: the layers of a ring repeat one
    gate on all its pairs, so circuit and target commute with a shift by two wires and the
    columns of an orbit of L/2 contribute alike."""
    return (1 << L) / (L // 2 if case.get("perms", "ring") == "ring" and L > 2 else 1)


def _sweep_flops(L, columns, G, Gt, what):
    """Two real operations per real multiply-add; a 4x4 complex product on a state is 32 per
    amplitude.  Target Gt products; forward one per gate (with tangent three); reverse one
    product and one outer sum per gate (with tangent three of each)."""
    per_gate = {"f": 1, "gradient": 3, "hvp": 9}[what]
    return 32.0 * columns * (1 << L) * (Gt + per_gate * G)


def _hessian_flops(L, columns, depth, Gt):
    """Forward chain, adjoint chain and one sweep that carries 16 tangents per layer begun:
    every active state is contracted with the adjoint state and taken through the gate."""
    active = sum(16 * a + 8 + 1 for a in range(depth))
    return 32.0 * columns * (1 << L) * (Gt + 2 * depth * (L // 2) + 2 * (L // 2) * active)


def work(case):
    """Bytes: inputs and results once.  Flops: the sums above."""
    k, L, n = case["kind"], case.get("L"), 0
    if k == "batch":
        order, flops, nbytes = np.random.default_rng(case["mix"]), 0.0, 0
        for _ in range(case["count"]):
            L, depth = int(order.choice([6, 8, 10, 12])), int(order.choice([3, 5, 7, 9]))
            flops += _sweep_flops(L, _orbits(L, {}), depth * L // 2, 3 * L // 2, "hvp")
            nbytes += 256 * (2 * depth + 3) + 256 * depth
        return {"bytes": nbytes, "flops": flops}
    if k in ("hvp", "gradient", "f", "real"):
        what = "hvp" if k == "real" else k
        flops = _sweep_flops(L, _orbits(L, case), case["depth"] * L // 2, case["tdepth"] * L // 2, what)
        if k == "real":   # real products
            flops /= 4
        n = 256 * (2 * case["depth"] + case["tdepth"]) + 256 * case["depth"]
    elif k == "circuit":
        flops = _sweep_flops(L, 1 << L, case["ngates"], case["tgates"], case["what"])
        n = 256 * (2 * case["ngates"] + case["tgates"])
    elif k in ("hessian", "sampled", "blockenc"):
        columns = {"hessian": _orbits(L, case), "sampled": case.get("nsamples", 0), "blockenc": (1 << (L // 2)) / max(1, L // 4)}[k]
        Gt = case.get("tdepth", 0) * (L // 2)
        flops = _hessian_flops(L, columns, case["depth"], Gt)
        n = 256 * (case["depth"] + case.get("tdepth", 0)) + 8 * (16 * case["depth"]) ** 2
    elif k == "apply":
        size = 16 if case["dtype"] == "c128" else 8
        flops = 32.0 * (1 << L) * case["ngates"]
        n = 2 * size * (1 << L)
    elif k == "module_circuit":   # at least f and gradient, one Hessian product and f of the candidate per iteration
        flops = case["niter"] * _sweep_flops(L, 1 << L, case["ngates"], 0, "hvp")
        n = 16 * (1 << (2 * L)) + 512 * case["ngates"]
    else:
        columns = case["nsamples"] or 1 << L
        flops = case["niter"] * _hessian_flops(L, columns, case["depth"], 0)
        n = 16 * (1 << (2 * L)) + 512 * case["depth"]
    return {"bytes": n, "flops": flops}


# ------------------------------------------------------------------------------ exact values

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.complex128, device=_device())


def _split(x, L, i, j):
    a, b = min(i, j), max(i, j)
    return x.view(1 << a, 2, 1 << (b - a - 1), 2, -1)


def _ordered(g, i, j):
    """The gate as a (2, 2, 2, 2) tensor whose first wire is the lower-numbered one."""
    g = g.view(2, 2, 2, 2)
    return g if i < j else g.permute(1, 0, 3, 2)


def _gate(g, i, j, x, L):
    return torch.einsum("xyij,aibjc->axbyc", _ordered(g, i, j), _split(x, L, i, j)).reshape(x.shape)


def _outer(phi, psi, i, j, L):
    """Sum over the rest of the register and all columns of phi_x psi_y, (4, 4)."""
    def rows(x):
        x = _split(x, L, i, j).permute(1, 3, 0, 2, 4) if i < j else _split(x, L, i, j).permute(3, 1, 0, 2, 4)
        x = x.reshape(4, -1)
        s = math.gcd(x.shape[1], 1024)
        return x.reshape(4, s, -1).transpose(0, 1)
    return torch.bmm(rows(phi), rows(psi).transpose(1, 2)).sum(0)


def _sweep(L, gates, dirs, wires, psi, end, want):
    """Forward and adjoint sweep of a block of columns (the columns of psi): the value, the
    gate gradients and the gate Hessian-vector products.  end(psi_n, dpsi_n) gives the value
    and the adjoint states that the sweep back begins with."""
    n, hvp = len(gates), want == "hvp"
    states, dpsi = [], torch.zeros_like(psi)
    for k in range(n):
        states.append((psi, dpsi))
        i, j = wires[k]
        if hvp:
            dpsi = _gate(gates[k], i, j, dpsi, L) + _gate(dirs[k], i, j, psi, L)
        psi = _gate(gates[k], i, j, psi, L)
        if want == "f":
            states.clear()
    value, phi, dphi = end(psi, dpsi)
    dg = torch.zeros((n, 4, 4), dtype=psi.dtype, device=psi.device)
    hg = torch.zeros_like(dg)
    if want == "f":
        return value, dg, hg
    for k in reversed(range(n)):
        i, j = wires[k]
        psi, dpsi = states.pop()
        dg[k] = _outer(phi, psi, i, j, L)
        gt = gates[k].T
        if hvp:
            hg[k] = _outer(dphi, psi, i, j, L) + _outer(phi, dpsi, i, j, L)
            dphi = _gate(gt, i, j, dphi, L) + _gate(dirs[k].T, i, j, phi, L)
        phi = _gate(gt, i, j, phi, L)
    return value, dg, hg


def _circuit_of(v, p, L):
    """Gates and wires of a brickwall, gate by gate."""
    per = L // 2
    wires = [(int(p[l][2 * q]), int(p[l][2 * q + 1])) for l in range(len(v)) for q in range(per)]
    return [v[l] for l in range(len(v)) for _ in range(per)], wires


def _columns(L, most=1 << 24):
    """Blocks of basis columns as matrices of at most `most` amplitudes."""
    n = 1 << L
    c = min(n, max(1, most >> L))
    for b in range(0, n, c):
        e = torch.zeros((n, c), dtype=torch.complex128, device=_device())
        e[torch.arange(b, b + c), torch.arange(c)] = 1
        yield e


def _target_sums(L, gates, dirs, wires, tgates, twires, want, blocks=None):
    total = None
    for e in blocks if blocks is not None else _columns(L, 1 << (24 if len(gates) < 70 else 23)):
        u = e
        for g, (i, j) in zip(tgates, twires):
            u = _gate(g, i, j, u, L)
        phi = -u.conj()
        got = _sweep(L, gates, dirs, wires, e, lambda x, dx: ((phi * x).sum(), phi, torch.zeros_like(phi)), want)
        total = got if total is None else [a + b for a, b in zip(total, got)]
    return total


def _project(v, z, dg, hg):
    """Riemannian gradient and Hessian-vector product of every gate, 16 reals each."""
    def reals(v, x):
        w = v.conj().T @ x
        a = 0.5 * (w - w.conj().T)
        return (a.real + a.imag).reshape(16)
    grad, hvp = [], []
    for l in range(len(v)):
        d, h = dg[l].conj(), hg[l].conj()
        grad.append(reals(v[l], d))
        if z is not None:
            dh = d.conj().T
            hvp.append(reals(v[l], h - 0.5 * (z[l] @ dh @ v[l] + v[l] @ dh @ z[l])))
    return torch.cat(grad), torch.cat(hvp) if z is not None else None


def _layers(x, nl):
    return x.reshape(nl, -1, 4, 4).sum(1)


def _np(*xs):
    return tuple(x.cpu().numpy() for x in xs)


def _brickwall_exact(L, v, z, p, tv, tp, want):
    v, z, tv = _t(v), _t(z), _t(tv)
    g, w = _circuit_of(v, p, L)
    d, _ = _circuit_of(z, p, L)
    tg, tw = _circuit_of(tv, tp, L)
    f, dg, hg = _target_sums(L, g, d, w, tg, tw, want)
    if want == "f":
        return np.complex128(f.item())
    grad, hvp = _project(v, z if want == "hvp" else None, _layers(dg, len(v)), _layers(hg, len(v)))
    return (np.complex128(f.item()),) + (_np(grad, hvp) if want == "hvp" else _np(grad))


def _hessian_exact(L, v, p, ends, starts, scale=1.0):
    """f, gradient and Hessian matrix, one column per tangent direction: starts() gives
    pairs (columns, end function)."""
    v = _t(v)
    nl = len(v)
    g, w = _circuit_of(v, p, L)
    f, grad, H = None, None, []
    for col in range(16 * nl):
        z = torch.zeros((nl, 4, 4), dtype=torch.complex128, device=v.device)
        z[col // 16] = v[col // 16] @ _t(_antisymm(np.eye(16)[col % 16]))
        d, _ = _circuit_of(z, p, L)
        total = None
        for e, end in zip(starts, ends):
            got = _sweep(L, g, d, w, e, end, "hvp")
            total = got if total is None else [a + b for a, b in zip(total, got)]
        f, dg, hg = (scale * x for x in total)
        grad, hvp = _project(v, z, _layers(dg, nl), _layers(hg, nl))
        H.append(hvp)
    return (f,) + _np(grad, torch.stack(H, 1))


def _pcg_normals(seed, n):
    """n complex normals of the PCG32 pair seeded with `seed` (O'Neill 2014, XSH-RR): 64-bit
    words of two 32-bit generators, two words per Box-Muller normal, two normals per amplitude."""
    A, M = 6364136223846793005, (1 << 64) - 1

    def out(s):
        x, r = (((s >> 18) ^ s) >> 27) & 0xFFFFFFFF, s >> 59
        return ((x >> r) | (x << ((32 - r) & 31))) & 0xFFFFFFFF

    def seeded(state, seq):
        inc = ((seq << 1) | 1) & M
        return ((inc + state) * A + inc) & M, inc

    def stream(gen, count):
        """`count` outputs: states by doubling jumps of the affine step, in wrapping uint64."""
        state, inc = gen
        s = np.empty(count, np.uint64)
        s[0], have, a, c = state, 1, A, inc
        while have < count:
            m = min(have, count - have)
            s[have:have + m] = s[:m] * np.uint64(a) + np.uint64(c)
            a, c, have = (a * a) & M, (a * c + c) & M, have + m
        x = (((s >> np.uint64(18)) ^ s) >> np.uint64(27)).astype(np.uint32)
        r = (s >> np.uint64(59)).astype(np.uint32)
        return (x >> r) | (x << ((np.uint32(32) - r) & np.uint32(31)))

    state, inc = seeded(seed, (A * seed + 1442695040888963407) & M)
    words = []
    for _ in range(4):
        hi = out(state)
        state = (state * A + inc) & M
        lo = out(state)
        state = (state * A + inc) & M
        words.append((hi << 32) | lo)
    if words[2] & (M >> 1) == words[3] & (M >> 1):
        words[3] ^= M
    first, second = seeded(words[0], words[2]), seeded(words[1], words[3])
    u = (stream(first, 4 * n).astype(np.uint64) << np.uint64(32)) | stream(second, 4 * n).astype(np.uint64)
    u = u.astype(np.float64) * 2.0 ** -64
    u1, u2 = u[0::2], u[1::2]
    u1 = np.where(u1 == 0, 1.0, u1)
    x = np.sqrt(-2 * np.log(u1)) * np.sin(2 * np.pi * u2)
    return (x[0::2] + 1j * x[1::2]) / np.sqrt(2)


def _exact_of(case, s):
    k, L = case["kind"], case.get("L")
    if k in ("hvp", "gradient", "f"):
        return _brickwall_exact(L, s["v"], s["z"], s["p"], s["tv"], s["tp"], k)
    if k == "real":
        f, grad, hvp = _brickwall_exact(L, s["v"], s["z"], s["p"], s["tv"], s["tp"], "hvp")
        upper = [4 * a + b for a in range(4) for b in range(a + 1, 4)]
        six = lambda x: (np.sqrt(2) * x.reshape(-1, 16)[:, upper]).reshape(-1)  # noqa: E731
        return float(f.real), six(grad), six(hvp)
    if k == "circuit":
        g, z, tg = _t(s["g"]), _t(s["z"]), _t(s["tg"])
        f, dg, hg = _target_sums(L, list(g), list(z), s["w"].tolist(), list(tg), s["tw"].tolist(), case["what"])
        if case["what"] == "f":
            return np.complex128(f.item())
        grad, hvp = _project(g, z if case["what"] == "hvp" else None, dg, hg)
        return (np.complex128(f.item()),) + (_np(grad, hvp) if case["what"] == "hvp" else _np(grad))
    if k == "batch":
        got = [_brickwall_exact(q[0], q[1], z, q[2], q[3], q[4], "hvp") for q, z in zip(s["problems"], s["dirs"])]
        return np.array([x[0] for x in got]), np.concatenate([x[1] for x in got]), np.concatenate([x[2] for x in got])
    if k == "apply":
        psi = _state(case, s["state_seed"], _device()).to(torch.complex128)
        for g, (i, j) in zip(_t(s["g"]), s["w"].tolist()):
            psi = _gate(g, i, j, psi, L)
        return psi
    if k in ("hessian", "sampled"):
        tg, tw = _circuit_of(_t(s["tv"]), s["tp"], L)
        scale = 1.0
        if k == "hessian":
            starts = list(_columns(L, 1 << 22))
        else:
            e = _t(_pcg_normals(s["seed"], case["nsamples"] << L).reshape(case["nsamples"], -1).T)
            starts, scale = [e / torch.linalg.vector_norm(e, dim=0)], (1 << L) / case["nsamples"]
        ends = []
        for e in starts:
            u = e
            for g, (i, j) in zip(tg, tw):
                u = _gate(g, i, j, u, L)
            phi = -u.conj()
            ends.append(lambda x, dx, phi=phi: ((phi * x).sum(), phi, torch.zeros_like(phi)))
        f, grad, H = _hessian_exact(L, s["v"], s["p"], ends, starts, scale)
        return np.complex128(f.item()), grad, H
    if k == "blockenc":
        half = L // 2
        at = torch.tensor([sum(((b >> i) & 1) << (2 * i + 1) for i in range(half)) for b in range(1 << half)],
                          device=_device())
        h = torch.eye(1 << half, dtype=torch.complex128, device=_device())
        for g, (i, j) in zip(*_circuit_of(_t(s["tv"]), s["tp"], half)):
            h = _gate(g, i, j, h, half)
        e = torch.zeros((1 << L, 1 << half), dtype=torch.complex128, device=_device())
        e[at, torch.arange(1 << half, device=_device())] = 1

        def end(x, dx):
            d, phi, dphi = x[at] - h, torch.zeros_like(x), torch.zeros_like(x)
            phi[at], dphi[at] = d.conj(), dx[at].conj()
            return 0.5 * d.abs().square().sum().to(x.dtype), phi, dphi

        f, grad, H = _hessian_exact(L, s["v"], s["p"], [end], [e])
        return np.float64(f.real.item()), grad, H
    return None


def exact(case, seed):
    """The optimisers' results have no closed form.  Nor are Hessians and sampled Hessians
    restated where the plain sweeps (16 per layer) would take too long."""
    k = case["kind"]
    if k.startswith("module"):
        return None
    if k in ("hessian", "sampled", "blockenc"):
        L, columns = case["L"], {"hessian": 1 << case["L"], "sampled": case.get("nsamples", 0), "blockenc": 1 << (case["L"] // 2)}[k]
        per_sweep = case["depth"] * (L // 2) * (1.2e-3 + 4e-10 * (columns << L))
        if 16 * case["depth"] * per_sweep > 18:
            return None
    return _exact_of(case, {**_inputs(case, seed), "state_seed": seed})
