"""What the encoder's users run, as cases that can be timed and compared.

A case is a dict of plain values; its ``kind`` names the entry point and its
other entries the sizes.  ``listed`` gives the standing cases, ``draw`` more
of the same ranges, ``prepare`` what a program holds before the call,
``run`` one pass, ``work`` what a pass cannot do without, ``exact`` the
64-bit values of its outputs in plain numpy and torch.

The fast precision works in complex64 and keeps its gates, environments and
fidelities in complex128 and float64 storage; a fast pass hands them on in
the precision they are computed in (complex64, float32), an exact pass as
they are.  Where a gate's environment is (nearly) rank deficient the sweep's
new gate is free there, so a fast sweep is judged by the state its gates
prepare, all 2^n amplitudes of it, which every caller builds next.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from qmprs_gb300 import engine as E
from qmprs_gb300 import warmstart as W
from qmprs_gb300.circuit import Circuit
from qmprs_gb300.synthesis.mps_encoding import Sequential


def listed() -> list:
    return [
        # one small state from host memory to a circuit: the reference's own
        # call, all latency
        dict(name="prepare_8q", kind="prepare", n=8, chi=64, layers=2, sweeps=1),
        # sweeps of the README configuration (10 qubits, 15 layers): one
        # state that fits a block's shared memory, both precisions
        dict(name="sweep_10q", kind="sweep", qubits="10", layers=15, sweeps=4, precision="fast"),
        dict(name="sweep_10q_exact", kind="sweep", qubits="10", layers=15, sweeps=2, precision="exact"),
        # sweeps of the 20-qubit configuration (10 layers): one large state,
        # a long chain of small launches
        dict(name="sweep_20q", kind="sweep", qubits="20", layers=10, sweeps=2, precision="fast"),
        # sweeps of a mixed batch as the benchmark has it (uneven sizes, 6
        # layers): throughput of the tile passes
        dict(name="sweep_batch", kind="sweep", qubits="12*9 13*7 14*7 15*7 16*7 17*7 18*7 19*7 20*6", layers=6,
             sweeps=2, precision="fast"),
        # disentangling layers of one large state, and of a mixed batch
        dict(name="layers_20q", kind="layers", qubits="20", bond=16, layers=3, precision="fast"),
        dict(name="layers_batch", kind="layers", qubits="11*5 12*5 13*5 14*5 15*5 16*5 17*5 18*5", bond=16, layers=2,
             precision="fast"),
        # a whole encode of a mixed batch in the exact precision
        dict(name="encode_batch_exact", kind="encode", qubits="8*3 9*2 11*2 12*2 13*2 14 15 16", bond=8, chi=64,
             layers=2, sweeps=1, precision="exact"),
        # statevector -> MPS -> statevector: the 20-qubit configuration with
        # bonds up to 256, and a mixed batch at bond 64
        dict(name="mps_20q_chi256", kind="mps", qubits="20", family="uniform", bond=0, chi=256),
        dict(name="mps_batch", kind="mps", qubits="12*8 13*8 14*8 15*8 16*8 17*8", family="mps", bond=32, chi=64),
        # gate environments of a training batch at fixed layers (the
        # backward pass of the warm start's circuit loss)
        dict(name="environments_batch", kind="env", qubits="13*8 14*8 15*8 16*8", layers=8),
        # the warm-start network's forward and backward on one minibatch
        dict(name="network_step", kind="network", rows=4096),
    ]


def draw(rng) -> dict:
    def log_int(lo, hi):
        return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))

    def mixed(lo, hi, count):
        return " ".join(str(rng.randint(lo, hi)) for _ in range(count))

    kind = rng.choice(["prepare", "sweep", "sweep", "sweep_batch", "layers", "layers", "encode", "mps", "mps_batch",
                       "env", "network"])
    if kind == "prepare":
        return dict(kind="prepare", n=rng.randint(3, 10), chi=rng.choice([4, 16, 64, 100]), layers=rng.randint(1, 2),
                    sweeps=rng.randint(0, 2))
    if kind == "sweep":
        precision = rng.choice(["fast", "fast", "exact"])
        n = rng.randint(4, 20 if precision == "fast" else 16)
        return dict(kind="sweep", qubits=str(n), layers=rng.randint(2, 15 if n <= 13 else 8),
                    sweeps=rng.randint(1, 2), precision=precision)
    if kind == "sweep_batch":
        return dict(kind="sweep", qubits=mixed(rng.choice([6, 12]), rng.choice([12, 15, 18]), log_int(2, 48)),
                    layers=rng.randint(2, 6), sweeps=rng.randint(1, 2), precision="fast")
    if kind == "layers":
        qubits = str(rng.randint(11, 20)) if rng.random() < 0.5 else mixed(11, rng.choice([13, 16, 18]), log_int(2, 48))
        return dict(kind="layers", qubits=qubits, bond=rng.choice([12, 16, 24]), layers=rng.randint(1, 3),
                    precision=rng.choice(["fast", "fast", "exact"]))
    if kind == "encode":
        return dict(kind="encode", qubits=mixed(6, rng.choice([11, 14, 16]), log_int(1, 16)), bond=rng.choice([6, 8, 12]),
                    chi=rng.choice([16, 64]), layers=rng.randint(1, 2), sweeps=1, precision="exact")
    if kind == "mps":
        return dict(kind="mps", qubits=str(rng.randint(9, 20)), family="uniform", bond=0,
                    chi=rng.choice([16, 48, 64, 100, 128, 256]))
    if kind == "mps_batch":
        return dict(kind="mps", qubits=mixed(8, rng.choice([13, 17]), log_int(2, 64)), family="mps",
                    bond=rng.choice([8, 16, 32]), chi=64)
    if kind == "env":
        return dict(kind="env", qubits=mixed(rng.choice([5, 12]), rng.choice([12, 13, 16]), log_int(1, 32)),
                    layers=rng.randint(2, 8))
    return dict(kind="network", rows=log_int(100, 8192))


# ---- sizes and inputs ------------------------------------------------------------

def _qubits(case) -> list:
    out = []
    for word in str(case["qubits"]).split():
        n, _, count = word.partition("*")
        out += [int(n)] * int(count or 1)
    return out


def _rng(seed: int) -> torch.Generator:
    return torch.Generator().manual_seed(seed)


def _normal(gen, *shape) -> torch.Tensor:
    return torch.view_as_complex(torch.randn(*shape, 2, generator=gen, dtype=torch.float64))


def _uniform_state(gen, n: int) -> torch.Tensor:
    """Real and imaginary parts i.i.d. uniform in [0, 1), normalised."""
    v = torch.view_as_complex(torch.rand(2 ** n, 2, generator=gen, dtype=torch.float64))
    return (v / v.norm()).cuda()


def _mps_state(gen, n: int, bond: int) -> torch.Tensor:
    """A random MPS of the given bond, contracted and normalised."""
    dims = [1] + [min(bond, 2 ** min(i, n - i)) for i in range(1, n)] + [1]
    v = torch.ones(1, 1, dtype=torch.complex128, device="cuda")
    for i in range(n):
        a = _normal(gen, dims[i], 2 * dims[i + 1]).cuda()
        v = (v @ a).reshape(-1, dims[i + 1])
        v = v / v.norm()
    return v.reshape(-1)


def _unitaries(gen, count: int, m: int, spread: float) -> torch.Tensor:
    """Unitaries around the identity: polar factors of I + spread * Gaussian."""
    u, _, vh = torch.linalg.svd(torch.eye(m, dtype=torch.complex128) + spread * _normal(gen, count, m, m))
    return u @ vh


def _apply(psi: torch.Tensor, g: torch.Tensor, q: int) -> torch.Tensor:
    m = g.shape[0]
    v = psi.reshape(2 ** q, m, -1)
    return torch.einsum("ab,ibj->iaj", g, v).reshape(-1)


def _layered(gen, n: int, L: int):
    """Gates of L layers (generation order, two-qubit gates on sites 0..n-2
    and a one-qubit gate on the last) and a target state near their circuit:
    the circuit of slightly different gates, with noise."""
    gates, near = [], []
    spread = 0.5 / math.sqrt(n * L)
    for _ in range(L):
        two, one = _unitaries(gen, n - 1, 4, 0.4), _unitaries(gen, 1, 2, 0.4)
        gates.append([*two, one[0]])
        near.append([*(two @ _unitaries(gen, n - 1, 4, spread)), (one @ _unitaries(gen, 1, 2, spread))[0]])
    psi = _circuit_state(near, n)
    noise = _normal(gen, 2 ** n).cuda()
    psi = psi + 0.2 * noise / noise.norm()
    return gates, psi / psi.norm()


def _circuit_state(gates, n: int) -> torch.Tensor:
    psi = torch.zeros(2 ** n, dtype=torch.complex128, device="cuda")
    psi[0] = 1.0
    for layer in reversed(gates):
        for q, g in enumerate(layer):
            psi = _apply(psi, g.cuda(), q)
    return psi


def _store(plan, gate_lists):
    """The plan's gate store and arity of every state's layers."""
    store = np.zeros(plan.gate_elems, dtype=np.complex128)
    arity = np.zeros(plan.gate_elems // 16, dtype=np.int8)
    for b, layers in enumerate(gate_lists):
        n, base = plan.nqubits[b], int(plan.gate_off[b])
        for l, layer in enumerate(layers):
            for s, g in enumerate(layer):
                off = base + (l * n + s) * 16
                store[off: off + g.numel()] = g.numpy().reshape(-1)
                arity[off // 16] = 1 if s == n - 1 else 2
    return torch.from_numpy(store.view(np.float64)).cuda(), torch.from_numpy(arity).cuda()


def _pack(states, precision: str) -> torch.Tensor:
    v = torch.cat(states).to(torch.complex128 if precision == "exact" else torch.complex64)
    return torch.view_as_real(v).reshape(-1).contiguous()


def _inputs(case, seed: int):
    """The case's states and gates in 64 bits, from the seed alone."""
    gen, kind = _rng(seed), case["kind"]
    if kind == "prepare":
        return _uniform_state(gen, case["n"]).cpu().numpy()
    if kind == "network":
        rows = case["rows"]
        x = torch.zeros(rows, W.DIMS[0])
        x[:, :W.FEAT] = 0.5 * torch.randn(rows, W.FEAT, generator=gen)
        y = torch.randn(rows, W.DIMS[-1], generator=gen)
        params = []
        for i in range(len(W.DIMS) - 1):
            w = torch.randn(W.DIMS[i + 1], W.DIMS[i], generator=gen) * math.sqrt(2.0 / W.DIMS[i])
            params.append((w.numpy(), 0.1 * torch.randn(W.DIMS[i + 1], generator=gen).numpy()))
        return x, y, params
    ns = _qubits(case)
    if kind in ("sweep", "env"):
        return [_layered(gen, n, case["layers"]) for n in ns]
    if case.get("family") == "uniform":
        return [_uniform_state(gen, n) for n in ns]
    return [_mps_state(gen, n, case["bond"]) for n in ns]


def prepare(case, seed):
    kind = case["kind"]
    got = _inputs(case, seed)
    if kind == "prepare":
        return dict(case=case, vector=got, encoder=Sequential(Circuit))
    if kind == "network":
        x, y, params = got
        model = W.WarmStartMLP()
        model.load_params(params)
        return dict(case=case, model=model, x=x.cuda(), y=y.cuda(), weight=torch.ones(len(x), device="cuda"))
    eng, ns = E.engine(), _qubits(case)
    precision = case.get("precision", "fast")
    state = dict(case=case, engine=eng)
    if kind in ("sweep", "env"):
        plan = eng.plan(ns, case["layers"], 4, precision)
        state["start"], state["arity"] = _store(plan, [g for g, _ in got])
        state["gates"] = torch.empty_like(state["start"])
        state["count"] = torch.full((plan.B,), case["layers"], dtype=torch.int32, device="cuda")
        state["target"] = _pack([t for _, t in got], precision)
    else:
        plan = eng.plan(ns, case.get("layers", 1), case.get("chi", 2), precision)
        state["vectors"] = _pack(got, precision)
    state["plan"] = plan
    return state


# ---- one pass --------------------------------------------------------------------

def _complex(x: torch.Tensor, precision: str) -> torch.Tensor:
    x = x if precision == "exact" else x.to(torch.float32)
    return torch.view_as_complex(x.view(-1, 2))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "prepare":
        enc = state["encoder"]
        circuit = enc.prepare_state(state["vector"], case["chi"], num_layers=case["layers"], num_sweeps=case["sweeps"])
        out = {"state": np.asarray(circuit.get_statevector()).astype(np.complex64),
               "layer_fidelities": enc.last_run["layer_fidelities"].astype(np.complex64)}
        if case["sweeps"]:
            out["sweep_fidelities"] = enc.last_run["sweep_fidelities"].astype(np.float32)
        return out
    if kind == "network":
        model = state["model"]
        y = model.forward(state["x"], train=True)
        loss, grads = model.backward(state["y"], state["weight"])
        return {"y": y, "loss": torch.tensor(loss, dtype=torch.float32), "dW": [g[0] for g in grads],
                "db": [g[1] for g in grads]}
    eng, plan, precision = state["engine"], state["plan"], case.get("precision", "fast")
    if kind == "sweep":
        state["gates"].copy_(state["start"])
        sf, done = eng.stage_sweeps(plan, state["target"], state["gates"], state["arity"], state["count"],
                                    case["sweeps"], reuse="sweep")
        if precision == "exact":
            return {"gates": _complex(state["gates"], precision), "done": done, "fidelities": sf}
        circuit = eng.stage_circuit(plan, state["gates"], state["arity"], state["count"], reuse="sweep")
        return {"state": _complex(circuit, precision), "done": done, "fidelities": sf.to(torch.float32)}
    if kind == "env":
        return {"environments": _complex(eng.environments(plan, state["target"], state["start"], state["arity"],
                                                          state["count"], env=state["gates"]), "fast")}
    if kind == "layers":
        gates, arity, nl, lf = eng.stage_layers(plan, state["vectors"], case["layers"], 1 - 1e-6, reuse=True)
        return {"gates": _complex(gates, precision), "arity": arity, "count": nl, "fidelities": _complex(lf, precision)}
    if kind == "encode":
        res = eng.encode(state["vectors"], case["chi"], case["layers"], case["sweeps"], nqubits=plan.nqubits,
                         precision=precision)
        return {"gates": res.gates, "arity": res.arity, "count": res.num_layers, "fidelity": res.fidelity,
                "layer_fidelities": res.layer_fidelities, "sweep_fidelities": res.sweep_fidelities}
    tensors, bonds, target = eng.stage_mps(plan, state["vectors"], case["chi"], reuse=True)
    # the site tensors' gauge is free within (nearly) equal singular values;
    # the state they contract to is not
    dense = eng.mps_to_statevector(plan, tensors, bonds)
    return {"bonds": bonds, "target": _complex(target, "fast"), "dense": _complex(dense, "fast")}


def work(case):
    """Bytes: the inputs and outputs once.  Flops: 32 per amplitude and
    applied two-qubit gate or environment (four complex multiply-adds)."""
    kind = case["kind"]
    if kind == "network":
        per_row = 2 * sum(a * b for a, b in zip(W.DIMS, W.DIMS[1:]))
        par = sum(a * b + b for a, b in zip(W.DIMS, W.DIMS[1:]))
        return {"bytes": 4.0 * case["rows"] * (W.DIMS[0] + 2 * W.DIMS[-1]) + 8.0 * par,
                "flops": float(case["rows"]) * (3 * per_row - 2 * W.DIMS[0] * W.DIMS[1])}
    ns = [case["n"]] if kind == "prepare" else _qubits(case)
    amp = 16.0 if case.get("precision", "fast") == "exact" else 8.0
    L, S = case.get("layers", 1), case.get("sweeps", 0)
    vec = sum(2.0 ** n for n in ns)
    gates = sum(float(L * n * 256) for n in ns)
    per_gate = sum(32.0 * L * n * 2 ** n for n in ns)
    if kind == "sweep" and case["precision"] == "exact":
        return {"bytes": amp * vec + 2 * gates, "flops": 4 * S * per_gate}
    if kind == "sweep":
        return {"bytes": 2 * amp * vec + 2 * gates, "flops": (4 * S + 1) * per_gate}
    if kind == "env":
        return {"bytes": amp * vec + 2 * gates, "flops": 4 * per_gate}
    # per layer: a Gram of width 4 and a projection over remainders that
    # halve (about 2 x 64 per amplitude), then the inverse layer
    layer = per_gate + L * 128.0 * vec
    if kind == "layers":
        return {"bytes": amp * vec + gates, "flops": layer}
    chi = case["chi"]
    mps = 0.0
    for n in ns:
        r = 1
        for c in range(n - 1, 0, -1):
            keep = min(chi, 2 ** c, 2 * r)
            mps += 2.0 ** c * (4.0 * (2 * r) ** 2 + 8.0 * 2 * r * keep) + 8.0 * 2.0 ** c * keep * 2 * r
            r = keep
    if kind == "mps":
        return {"bytes": 3 * amp * vec, "flops": mps}
    return {"bytes": amp * vec + gates, "flops": mps + layer + (4 * S + 1) * per_gate}


# ---- 64-bit values -----------------------------------------------------------------

def _pivot(x: np.ndarray, free: np.ndarray) -> int:
    mag = np.where(free, np.abs(x), -1.0)
    return int(np.nonzero(mag >= (1 - 1e-6) * mag.max())[0][0])


def _rows_phased(vh: np.ndarray) -> np.ndarray:
    out = vh.copy()
    for row in out:
        z = row[_pivot(row, np.ones(row.size, bool))]
        row *= np.conj(z) / abs(z)
    return out


def _truncated(v: np.ndarray, n: int, chi: int):
    """Right-to-left truncated SVD (tail weight 1e-10, at most chi): the
    sites (l, p, r) and the last remainder, not rescaled."""
    sites, r, m = [None] * n, 1, v
    for c in range(n - 1, 0, -1):
        m = m.reshape(2 ** c, 2 * r)
        tall = np.linalg.qr(m, mode="r") if m.shape[0] > 2 * m.shape[1] else m
        _, s, vh = np.linalg.svd(tall, full_matrices=False)
        tail = np.cumsum((s * s)[::-1])[::-1]
        keep = max(1, min(chi, int(np.sum(tail > 1e-10 * tail[0]))))
        sites[c] = _rows_phased(vh[:keep]).reshape(keep, 2, r)
        m = m @ sites[c].reshape(keep, -1).conj().T
        r = keep
    sites[0] = m.reshape(1, 2, r)
    return sites


def _contracted(sites) -> np.ndarray:
    v = sites[0].reshape(2, -1)
    for a in sites[1:]:
        v = (v @ a.reshape(a.shape[0], -1)).reshape(-1, a.shape[2])
    return v.reshape(-1)


def _target(v: np.ndarray, n: int, chi: int) -> np.ndarray:
    t = _contracted(_truncated(v, n, chi))
    return t * (np.linalg.norm(v) / np.linalg.norm(t))


def _complement(x: np.ndarray) -> np.ndarray:
    """Columns completing the orthonormal rows of x, by pivoted reflections."""
    k, n = x.shape
    free, ws = np.ones(n, bool), []

    def reflect(w, v):
        return v - w * (2 * np.vdot(w, v) / np.vdot(w, w).real)

    for a in range(k):
        v = x[a].copy()
        for w in ws:
            v = reflect(w, v)
        v[~free] = 0
        j = _pivot(v, free)
        w = np.conj(v[j] / abs(v[j])) * v
        w[j] += 1
        ws.append(w)
        free[j] = False
    cols = []
    for j in np.nonzero(free)[0]:
        v = np.eye(n, dtype=complex)[j]
        for w in reversed(ws):
            v = reflect(w, v)
        cols.append(v)
    return np.stack(cols, axis=1)


def _first_gate(m4: np.ndarray) -> np.ndarray:
    """(A x B) CX (Ry x I) with first column m4: the two-qubit state's Schmidt form."""
    m = m4.reshape(2, 2)
    lam, v = np.linalg.eigh(m.conj().T @ m)
    lam, v = np.maximum(lam[::-1], 0), _rows_phased(v[:, ::-1].T).T
    s = np.sqrt(lam / lam.sum())
    a = m @ v
    a[:, 0] /= np.linalg.norm(a[:, 0])
    a[:, 1] = a[:, 1] / np.linalg.norm(a[:, 1]) if s[1] > 1e-8 * s[0] else _complement(a[:, :1].T)[:, 0]
    ry = np.array([[s[0], -s[1]], [s[1], s[0]]])
    return np.kron(a, v.conj()) @ np.eye(4)[[0, 1, 3, 2]] @ np.kron(ry, np.eye(2))


def _layer(psi: np.ndarray, n: int) -> list:
    """The bond-2 layer of psi, one gate per site."""
    sites = _truncated(psi, n, 2)
    sites[0] = sites[0] / np.linalg.norm(sites[0])
    out = []
    for s, a in enumerate(sites):
        starts, ends = a.shape[0] == 1, a.shape[2] == 1
        if starts and ends:
            v = a.reshape(1, 2)
            out.append(np.concatenate([v.T, _complement(v)], axis=1))
        elif ends:
            out.append(a.reshape(2, 2).T)
        elif starts:
            out.append(_first_gate(a.reshape(-1)))
        else:
            b = _complement(a.reshape(2, 4))
            ph = np.where(np.abs(b[0]) > 1e-12, b[0] / np.maximum(np.abs(b[0]), 1e-300), 1.0)
            b = b / ph
            rows = a.reshape(2, 4)
            out.append(np.stack([rows[0], b[:, 0], rows[1], b[:, 1]], axis=1))
    return out


def _layers(target: torch.Tensor, n: int, L: int):
    """Layers in generation order and the zero-state overlap after each."""
    psi = target / target.norm()
    layers, fids = [], []
    for _ in range(L):
        layer = [torch.from_numpy(g) for g in _layer(psi.cpu().numpy(), n)]
        # a block's gates from its end to its start, and blocks are disjoint
        for q in range(n - 1, -1, -1):
            psi = _apply(psi, layer[q].conj().T.contiguous().cuda(), q)
        layers.append(layer)
        f = complex(psi[0].conj().cpu())
        fids.append(f)
        if abs(f - 1) <= 1e-6 + 1e-5:
            break
    return layers, fids


def _best_unitary(env: np.ndarray, prev: np.ndarray):
    """Maximiser of Re Tr(W^H E); on E's null space (singular values up to
    1e-6 of the largest) the unitary completion nearest to prev."""
    u, s, vh = np.linalg.svd(env)
    sig = s > 1e-6 * s[0]
    w = u[:, sig] @ vh[sig]
    if not sig.all():
        us, vn = u[:, sig], vh[~sig].conj().T
        x = prev @ vn
        x = x - us @ (us.conj().T @ x)
        a, _, b = np.linalg.svd(x, full_matrices=False)
        w = w + a @ b @ vn.conj().T
    return w, float(s.sum())


def _env(t: torch.Tensor, psi: torch.Tensor, n: int, q: int, m: int) -> torch.Tensor:
    tt, pp = t.reshape(2 ** q, m, -1), psi.reshape(2 ** q, m, -1)
    return torch.einsum("iaj,ibj->ab", tt.conj(), pp)


def _backward(target: torch.Tensor, gates: list, n: int, update: bool):
    """One pass over all gates from the circuit's end; gates changed in place
    with update.  Returns the environments and the last nuclear norm."""
    psi, t, nuc = _circuit_state(gates, n), target, 0.0
    envs = [[None] * n for _ in gates]
    for l, layer in enumerate(gates):
        for q in range(n - 1, -1, -1):
            g = layer[q]
            psi = _apply(psi, g.conj().T.contiguous().cuda(), q)
            e = _env(t, psi, n, q, g.shape[0]).cpu()
            envs[l][q] = e
            if update:
                w, nuc = _best_unitary(e.resolve_conj().numpy(), g.conj().resolve_conj().numpy())
                g = layer[q] = torch.from_numpy(w.conj())
            t = _apply(t, g.conj().T.contiguous().cuda(), q)
    return envs, nuc


def _flat(layer_lists, L: int) -> np.ndarray:
    """Per state, L * n slots of 16 entries."""
    parts = []
    for layers in layer_lists:
        n = len(layers[0])
        out = np.zeros((L * n, 16), complex)
        for l, layer in enumerate(layers):
            for s, g in enumerate(layer):
                out[l * n + s, : g.numel()] = g.numpy().reshape(-1)
        parts.append(out.reshape(-1))
    return np.concatenate(parts)


def exact(case, seed):
    kind, got = case["kind"], _inputs(case, seed)
    if kind == "network":
        return _exact_network(*got)
    if kind == "env":
        return {"environments": _flat([_backward(t, g, n, False)[0] for n, (g, t) in zip(_qubits(case), got)],
                                      case["layers"])}
    S = case.get("sweeps", 0)
    if kind == "sweep":
        fids = []
        for n, (gates, t) in zip(_qubits(case), got):
            fids += [_backward(t, gates, n, True)[1] / float(t.norm()) for _ in range(S)]
        out = {"done": None, "fidelities": np.array(fids)}
        if case["precision"] == "exact":
            return {**out, "gates": _flat([g for g, _ in got], case["layers"])}
        return {**out, "state": torch.cat([_circuit_state(g, n) for n, (g, _) in zip(_qubits(case), got)])}
    ns = [case["n"]] if kind == "prepare" else _qubits(case)
    states = [torch.from_numpy(got).cuda()] if kind == "prepare" else got
    if kind == "mps":
        t = np.concatenate([_target(v.cpu().numpy(), n, case["chi"]) for v, n in zip(states, ns)])
        return {"bonds": None, "target": t, "dense": t}
    L = case["layers"]
    all_layers, lf, sf, fid = [], np.zeros((len(ns), L), complex), np.zeros((len(ns), S)), []
    for b, (v, n) in enumerate(zip(states, ns)):
        t = v if kind == "layers" else torch.from_numpy(_target(v.cpu().numpy(), n, case["chi"])).cuda()
        layers, f = _layers(t, n, L)
        lf[b, : len(f)] = f
        for k in range(S):
            sf[b, k] = _backward(t, layers, n, True)[1] / float(t.norm())
        if kind == "encode":
            fid.append(float(torch.vdot(_circuit_state(layers, n), v).abs()))
        all_layers.append(layers)
    if kind == "prepare":
        out = {"state": _circuit_state(all_layers[0], ns[0]), "layer_fidelities": lf[0, : len(all_layers[0])]}
        return {**out, "sweep_fidelities": sf[0]} if S else out
    gates = _flat(all_layers, L)
    if kind == "layers":
        return {"gates": gates, "arity": None, "count": None, "fidelities": lf.reshape(-1)}
    return {"gates": gates, "arity": None, "count": None, "fidelity": np.array(fid), "layer_fidelities": lf,
            "sweep_fidelities": sf}


def _exact_network(x, y, params):
    x, y = x.double(), y.double()
    ps = [(torch.from_numpy(w).double().requires_grad_(), torch.from_numpy(b).double().requires_grad_())
          for w, b in params]
    h = x
    for w, b in ps[:-1]:
        h = torch.nn.functional.gelu(h @ w.T + b, approximate="tanh")
    out = h @ ps[-1][0].T + ps[-1][1] + x[:, :W.DIMS[-1]]
    a = torch.view_as_complex(out.reshape(-1, 16, 2))
    u = torch.view_as_complex(y.reshape(-1, 16, 2))
    # min over the phase of |Y - e^{i phi} U|^2
    per_row = a.abs().square().sum(1) + u.abs().square().sum(1) - 2 * (u.conj() * a).sum(1).abs()
    loss = per_row.mean()
    loss.backward()
    last = len(ps) - 1
    return {"y": out.detach(), "loss": float(loss.detach()),
            "dW": [w.grad.T.contiguous() if i == last else w.grad for i, (w, _) in enumerate(ps)],
            "db": [b.grad for _, b in ps]}
