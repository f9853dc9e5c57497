"""The work that users of this package have it do, as cases that can be timed.

``listed()`` names them, ``draw(rng)`` gives one more of the same ranges,
``prepare`` makes what a program holds before the call, ``run`` is one pass
through the public classes, ``work`` counts the bytes and operations the path
cannot do without, and ``exact`` computes the result in plain numpy where that
is quick.  Kinds:

  layer   SparseState.apply_gate on a loaded state: the calls of a program that
          drives the state itself (1-qubit, CZ and general 2-qubit gates, each
          with its top-k truncation), then the read of the entries
  bass    BASS.simulate on a whole circuit (the adaptive method): TFIM Trotter
          or brickwork circuits, complex128 or complex64, with or without
          2-qubit rotations
  fixed   FixedBasisSimulator.simulate (no basis adaptation, top-k)
  batch   BatchedBASS.simulate: circuits of uneven size advancing together
  dense   ExactSimulator.simulate_device: the dense state that sparse results
          are scored against
"""
import importlib.util
import os
import sys

import numpy as np


def _pkg():
    """The package (its folder's name is not an identifier), from the working folder."""
    if "bass_b200" not in sys.modules:
        d = os.path.join(os.getcwd(), "bass-basis-adapative-sparse-simulations-_b200")
        spec = importlib.util.spec_from_file_location("bass_b200", os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        m = importlib.util.module_from_spec(spec)
        sys.modules["bass_b200"] = m
        spec.loader.exec_module(m)
    import bass_b200.bass, bass_b200.batch, bass_b200.circuits, bass_b200.dense  # noqa: E401, F401
    import bass_b200.fixed, bass_b200.gates, bass_b200.state  # noqa: E401, F401
    return sys.modules["bass_b200"]


def listed():
    return [
        # a few gates on a small state, read back: launches and latency
        {"name": "layer_n12_k256", "kind": "layer", "n": 12, "k": 256, "ones": 2, "twos": 1, "dtype": "complex128"},
        # the same on an ordinary state whose size is no power of two
        {"name": "layer_n30_k150001", "kind": "layer", "n": 30, "k": 150001, "ones": 6, "twos": 2,
         "dtype": "complex64"},
        # and at the largest budget in use, where device memory counts
        {"name": "layer_n40_k4m", "kind": "layer", "n": 40, "k": 1 << 22, "ones": 6, "twos": 2,
         "dtype": "complex128"},
        # a laptop-size adaptive run (the smoke test's): host and launch bound
        {"name": "brick_n12_k64", "kind": "bass", "circuit": "brick", "n": 12, "k": 64, "depth": 10,
         "dtype": "complex128", "pairs": False},
        # ordinary brickwork run of the parity fixtures
        {"name": "brick_n40_k16k", "kind": "bass", "circuit": "brick", "n": 40, "k": 1 << 14, "depth": 10,
         "dtype": "complex128", "pairs": False},
        # the benchmark's brickwork run at its full budget, fewer layers
        {"name": "brick_n40_k4m", "kind": "bass", "circuit": "brick", "n": 40, "k": 1 << 22, "depth": 8,
         "dtype": "complex128", "pairs": False},
        # the TFIM Trotter workload (many small angles, diagonal 2-qubit gates)
        {"name": "tfim_n24_k64k", "kind": "bass", "circuit": "tfim", "n": 24, "k": 1 << 16, "depth": 20,
         "dtype": "complex128", "pairs": False},
        # its precision form, at a ragged budget
        {"name": "tfim_n31_k300003_c64", "kind": "bass", "circuit": "tfim", "n": 31, "k": 300003, "depth": 8,
         "dtype": "complex64", "pairs": False},
        # 2-qubit basis rotations switched on
        {"name": "pairs_n20_k4k", "kind": "bass", "circuit": "brick", "n": 20, "k": 4096, "depth": 4,
         "dtype": "complex128", "pairs": True},
        # fixed-basis run of general 2-qubit gates
        {"name": "fixed_n28_k200k", "kind": "fixed", "n": 28, "k": 200000, "depth": 4},
        # many circuits of uneven size at once (the batched workload's ranges)
        {"name": "batch_16", "kind": "batch", "count": 16, "layers": 10, "m_low": 10, "m_high": 17},
        # the dense state a sparse result is compared with
        {"name": "dense_n24", "kind": "dense", "n": 24, "depth": 2},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["layer", "layer", "layer", "bass", "bass", "bass", "bass", "fixed", "batch", "dense"])
    dtype = rng.choice(["complex128", "complex128", "complex64"])
    if kind == "layer":
        k = _log_int(rng, 200, 1 << 22)
        n = rng.randint(max(10, k.bit_length() + 2), 44)
        return {"kind": kind, "n": n, "k": k, "ones": rng.randint(1, 6), "twos": rng.randint(0, 2), "dtype": dtype}
    if kind == "bass":
        circuit = rng.choice(["brick", "tfim"])
        k = _log_int(rng, 64, 1 << 21)
        n = rng.randint(max(12, k.bit_length() + 3), 44)
        depth = rng.randint(4, 10) if k > 100000 else rng.randint(6, 14)
        return {"kind": kind, "circuit": circuit, "n": n, "k": k, "depth": depth, "dtype": dtype, "pairs": False}
    if kind == "fixed":
        k = _log_int(rng, 500, 1000000)
        return {"kind": kind, "n": rng.randint(max(12, k.bit_length() + 2), 36), "k": k, "depth": rng.randint(2, 5)}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(4, 16), "layers": rng.randint(4, 10), "m_low": rng.randint(8, 11),
                "m_high": rng.randint(12, 17)}
    n = rng.randint(12, 23)
    return {"kind": kind, "n": n, "depth": rng.randint(1, 24 if n < 18 else 24 - n + 1)}


# ---- inputs --------------------------------------------------------------------

def _haar(rng, d):
    z = (rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d))) / np.sqrt(2.0)
    q, r = np.linalg.qr(z)
    v = np.diag(r)
    return q * (v / np.abs(v))


def _entries(case, rng):
    """k distinct keys of n bits with Gaussian amplitudes of norm 1 (|a|^2
    exponentially distributed, as in a scrambled circuit)."""
    n, k = case["n"], case["k"]
    x = np.unique(rng.integers(0, 1 << n, size=k + k // 8 + 64, dtype=np.uint64))
    while len(x) < k:
        x = np.unique(np.concatenate([x, rng.integers(0, 1 << n, size=k, dtype=np.uint64)]))
    x = np.sort(rng.permutation(x)[:k])
    a = rng.standard_normal(k) + 1j * rng.standard_normal(k)
    a /= np.sqrt(np.sum(np.abs(a) ** 2))
    return x, a.astype(case["dtype"])


def _layer_gates(case, rng):
    """(qubits, matrix) of the layer: 1-qubit Haar gates, then per 2-qubit gate
    a CZ and a Haar gate on other pairs."""
    n = case["n"]
    out = [((int(q),), _haar(rng, 2)) for q in rng.permutation(n)[:case["ones"]]]
    for _ in range(case["twos"]):
        a, b = (int(v) for v in rng.permutation(n)[:2])
        out.append(((a, b), np.diag([1, 1, 1, -1]).astype(np.complex128)))
        a, b = (int(v) for v in rng.permutation(n)[:2])
        out.append(((a, b), _haar(rng, 4)))
    return out


def _pair_layers(case, rng):
    """Brickwork of general 2-qubit gates (the fixed-basis workload)."""
    n = case["n"]
    return [((i, i + 1), _haar(rng, 4)) for layer in range(case["depth"]) for i in range(layer % 2, n - 1, 2)]


def _dense_layers(case, rng):
    """A Haar 1-qubit gate on every qubit, then 2-qubit gates on neighbours."""
    n, out = case["n"], []
    for layer in range(case["depth"]):
        out += [((q,), _haar(rng, 2)) for q in range(n)]
        out += [((i, i + 1), _haar(rng, 4)) for i in range(layer % 2, n - 1, 2)]
    return out


def _gate_objects(gates):
    g = _pkg().gates
    return [g.SingleQubitGate(q[0], m) if len(q) == 1 else g.TwoQubitGate(q[0], q[1], m) for q, m in gates]


def _circuit(case, rng):
    c = _pkg().circuits
    if case["circuit"] == "tfim":
        return c.tfim_circuit(case["n"], case["depth"], J=1.0, h=1.0, dt=0.1, rng=rng, disorder_strength_h=0.5)
    return c.brickwork_circuit(case["n"], case["depth"], rng=rng)


def _batch_sizes(case):
    """(qubits, layers, K) of each circuit of a batch: uneven, the case's own."""
    rng = np.random.default_rng([case["count"], case["layers"], case["m_low"], case["m_high"]])
    lo = max(2, case["layers"] // 2)
    return [(int(rng.integers(22, 41)), int(rng.integers(lo, case["layers"] + 1)),
             1 << int(rng.integers(case["m_low"], case["m_high"] + 1))) for _ in range(case["count"])]


def prepare(case, seed):
    p = _pkg()
    rng = np.random.default_rng([int(seed), 17])
    kind = case["kind"]
    if kind == "layer":
        x, a = _entries(case, rng)
        st = p.state.SparseState(case["n"], case["k"], dtype=np.dtype(case["dtype"]))
        st.load(x, a)
        return {"kind": kind, "state": st, "gates": _gate_objects(_layer_gates(case, rng))}
    if kind == "bass":
        sim = p.bass.BASS(case["n"], case["k"], dtype=np.dtype(case["dtype"]), use_2qubit_rotations=case["pairs"])
        return {"kind": kind, "sim": sim, "circuit": _circuit(case, rng)}
    if kind == "fixed":
        sim = p.fixed.FixedBasisSimulator(case["n"], case["k"], verbose=False)
        return {"kind": kind, "sim": sim, "circuit": _gate_objects(_pair_layers(case, rng))}
    if kind == "batch":
        specs, circuits = [], []
        for n, layers, k in _batch_sizes(case):
            circuits.append(p.circuits.tfim_circuit(n, layers, J=1.0, h=float(rng.uniform(0.5, 1.8)), dt=0.05, rng=rng,
                                                    disorder_strength_h=0.2))
            specs.append((n, k))
        return {"kind": kind, "sim": p.batch.BatchedBASS(specs), "circuits": circuits}
    return {"kind": kind, "sim": p.dense.ExactSimulator(case["n"], verbose=False),
            "circuit": _gate_objects(_dense_layers(case, rng))}


# ---- one pass --------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "layer":
        st = state["state"]
        for g in state["gates"]:
            st.apply_gate(g)
        return {"x": st.x, "alpha": st.alpha, "gamma": st.gamma}
    if kind == "bass":
        st = state["sim"].simulate(state["circuit"])
        return {"x": st.x, "alpha": st.alpha, "gamma": st.gamma, "frames": np.stack(state["sim"].U)}
    if kind == "fixed":
        sim = state["sim"]
        st = sim.simulate(state["circuit"], seed=1)
        return {"x": st.x, "alpha": st.alpha, "gamma": sim.gamma_history, "nnz": sim.nnz_history}
    if kind == "batch":
        return [{"x": s.x, "alpha": s.alpha, "gamma": s.gamma} for s in state["sim"].simulate(state["circuits"])]
    return state["sim"].simulate_device(state["circuit"])


# ---- what the path cannot do without ---------------------------------------------

def _growth(sizes_in, per_gate, k, limit):
    """Entries read and written over a run of gates that each multiply the
    entry count by at most `per_gate`, kept at k (and at most `limit`)."""
    n, moved, seen = sizes_in, 0, 0
    for f in per_gate:
        m = min(n * f, k, limit)
        moved += n + m
        seen += n
        n = m
    return n, moved, seen


def work(case):
    kind = case["kind"]
    if kind == "dense":
        gates = case["depth"] * (case["n"] + (case["n"] - 1) // 2)
        return {"bytes": 2 * 16 * (1 << case["n"]) * gates, "flops": 14 * (1 << case["n"]) * gates}
    if kind == "batch":
        b = f = 0
        for n, layers, k in _batch_sizes(case):
            _, moved, seen = _growth(1, ([1] * (n - 1) + [2] * n) * layers, k, 1 << n)
            b += 16 * (moved + 2 * k)
            f += 28 * seen
        return {"bytes": b, "flops": f}
    entry = 16 if case.get("dtype") == "complex64" else 24
    if kind == "layer":
        _, moved, seen = _growth(case["k"], [2] * case["ones"] + [1, 4] * case["twos"], case["k"], 1 << case["n"])
    elif kind == "fixed":
        pairs = [4 for layer in range(case["depth"]) for _ in range(layer % 2, case["n"] - 1, 2)]
        _, moved, seen = _growth(1, pairs, case["k"], 1 << case["n"])
    elif case["circuit"] == "tfim":
        _, moved, seen = _growth(1, ([1] * (case["n"] - 1) + [2] * case["n"]) * case["depth"], case["k"], 1 << case["n"])
    else:
        # CZ on half of the pairs, general in a rotated frame
        _, moved, seen = _growth(1, ([2] * case["n"] + [1] * (case["n"] // 4)) * case["depth"], case["k"], 1 << case["n"])
    return {"bytes": entry * (moved + 2 * case["k"]), "flops": 28 * seen}


# ---- the result in plain numpy ------------------------------------------------------

def _np_gate(x, a, qubits, m):
    """A gate on the sorted entries (x, a): every entry's children, summed by
    key; children whose products are all zero are dropped."""
    one = np.uint64(1)
    bits = [np.uint64(q) for q in qubits]
    d = len(m)
    idx = np.zeros(len(x), np.int64)
    base = x.copy()
    for b in bits:
        idx = (idx << 1) | ((x >> b) & one).astype(np.int64)
        base &= ~(one << b)
    keys, vals = [], []
    for o in range(d):
        key = base.copy()
        for j, b in enumerate(bits):
            if (o >> (len(bits) - 1 - j)) & 1:
                key |= one << b
        v = m[o, idx] * a
        live = v != 0
        keys.append(key[live])
        vals.append(v[live])
    keys, vals = np.concatenate(keys), np.concatenate(vals)
    u, inv = np.unique(keys, return_inverse=True)
    out = np.zeros(len(u), np.complex128)
    np.add.at(out, inv, vals)
    return u, out


def _np_topk(x, a, k):
    """The k entries of largest |a|^2 (smaller key first among equals), and
    the kept and total mass."""
    p = a.real ** 2 + a.imag ** 2
    total = p.sum()
    if len(x) <= k:
        return x, a, total, total, False
    t = np.partition(p, len(p) - k)[len(p) - k]
    keep = p > t
    tied = np.nonzero(p == t)[0]
    keep[tied[:k - int(keep.sum())]] = True
    return x[keep], a[keep], p[keep].sum(), total, True


def exact(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng([int(seed), 17])
    if kind == "layer":
        if case["k"] > 400000:
            return None
        x, a = _entries(case, rng)
        a = a.astype(np.complex128)
        gamma = 1.0
        for qubits, m in _layer_gates(case, rng):
            x, a = _np_gate(x, a, qubits, m)
            x, a, kept, _, cut = _np_topk(x, a, case["k"])
            if cut:
                gamma *= np.sqrt(kept)
                a = a / np.sqrt(kept)
        return {"x": None, "alpha": a.astype(case["dtype"]), "gamma": float(gamma)}
    if kind == "fixed":
        if case["k"] * case["depth"] * case["n"] > 30000000:
            return None
        x, a = np.zeros(1, np.uint64), np.ones(1, np.complex128)
        gam, nnz = [1.0], [1.0]
        for qubits, m in _pair_layers(case, rng):
            x, a = _np_gate(x, a, qubits, m)
            x, a, kept, total, cut = _np_topk(x, a, case["k"])
            g = gam[-1]
            if cut:
                g *= np.sqrt(kept / total)
                a = a / np.sqrt(kept)
            gam.append(float(g))
            nnz.append(float(len(x)))
        return {"x": None, "alpha": a, "gamma": np.array(gam), "nnz": np.array(nnz)}
    if kind == "dense":
        if case["n"] > 22:
            return None
        n = case["n"]
        psi = np.zeros(1 << n, np.complex128)
        psi[0] = 1.0
        for qubits, m in _dense_layers(case, rng):
            if len(qubits) == 1:
                v = psi.reshape(-1, 2, 1 << qubits[0])
                psi = np.stack([m[o, 0] * v[:, 0] + m[o, 1] * v[:, 1] for o in (0, 1)], axis=1).reshape(-1)
            else:  # neighbours q, q + 1: index (bit_q << 1) | bit_(q + 1)
                v = psi.reshape(-1, 2, 2, 1 << qubits[0])  # axes: high, bit q + 1, bit q, low
                w = [v[:, 0, 0], v[:, 1, 0], v[:, 0, 1], v[:, 1, 1]]
                r = [sum(m[o, i] * w[i] for i in range(4)) for o in range(4)]
                psi = np.stack([np.stack([r[0], r[2]], axis=1), np.stack([r[1], r[3]], axis=1)], axis=1).reshape(-1)
        return psi
    return None
