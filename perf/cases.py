"""Performance cases: the work a user of this package has it do, through its
public entry points.

Each case is a dict of plain values; ``prepare`` builds what a program has in
hand before the call (a state, gates, a captured circuit), ``run`` is one pass
through the public API, ``work`` the bytes and operations the pass cannot do
without and ``exact`` the same outputs from 64-bit torch code.

Two-site updates determine the new site tensors only up to a unitary on the
bond, so their outputs are compared as the merged pairs A'B' (the two-site
tensor a program reads next, from ``ops.contract_gate`` with the identity
gate), whole circuits as statevectors.  The gates' spectra are the ones the
path meets with a decided rank: entangling layers that double the bond up to
the cap (rank exactly 2 chi_mid) and small-step evolution whose truncated
weight is well below the kept weight.

Kinds
  layer      one brickwork layer of two-site gates on an MPS (or its centre
             gate only): ``entangle`` = random local rotations around CZ, the
             bond doubles to the cap; ``trotter`` = RZZ of a small step at the
             cap, the bond is truncated back
  circuit    a whole seeded Haar brickwork circuit from |0...0>, device-resident,
             read out as a statevector
  graph      many instances of uneven size, their circuits captured as one CUDA
             graph, replayed and read out as statevectors
  canonical  a canonical sweep (QR of every site): left, right or mixed
  sample     batched conditional sampling of a right-canonical MPS
  local      nearest-neighbour <ZZ> and single-site <X> of every site
  mpo        <H> of a bond-5 Heisenberg MPO
  tdvp       the environment steps and the local operator of one TDVP site
"""
import math

import torch

import atlasq_gb300 as aq
from atlasq_gb300 import ops
from atlasq_gb300.circuits import CZ, haar_brickwork, haar_unitary, rzz
from atlasq_gb300.sampling import sample_tensors

DEV = "cuda:0"
C64, C128 = torch.complex64, torch.complex128


def _dt(case):
    return C128 if case.get("dtype") == "c128" else C64


def listed():
    return [
        # one gate between two reads of a small state: launch and host latency
        {"name": "gate_q10_chi16", "kind": "layer", "gate": "entangle", "bonds": "centre", "sites": 10, "chi": 16,
         "dtype": "c64"},
        # a whole small circuit (10 qubits, depth 10, nothing truncated), read as a statevector
        {"name": "circuit_q10_d10", "kind": "circuit", "sites": 10, "depth": 10},
        # the benchmark's layer: 40 qubits at chi 256, the bulk gates factor 512 x 512 and keep 256
        {"name": "layer_q40_chi256", "kind": "layer", "gate": "entangle", "bonds": "even", "sites": 40, "chi": 256,
         "dtype": "c64"},
        # time evolution at a cap that is no power of two; odd bonds
        {"name": "trotter_q32_chi100", "kind": "layer", "gate": "trotter", "bonds": "odd", "sites": 32, "chi": 100,
         "dtype": "c64"},
        # the largest bond the package takes: one CZ-ladder gate at chi 512 (1024 x 1024)
        {"name": "gate_q22_chi512", "kind": "layer", "gate": "entangle", "bonds": "centre", "sites": 22, "chi": 512,
         "dtype": "c64"},
        # double precision, the form that gates are promoted to
        {"name": "layer_q20_chi48_c128", "kind": "layer", "gate": "entangle", "bonds": "even", "sites": 20,
         "chi": 48, "dtype": "c128"},
        # many uneven instances advanced by one captured graph
        {"name": "graph_24x_q6to10", "kind": "graph", "instances": 24, "lo": 6, "hi": 10, "depth": 6},
        # canonicalisation around the centre: left sweep, then right sweep
        {"name": "mixed_q40_chi256", "kind": "canonical", "form": "mixed", "sites": 40, "chi": 256, "dtype": "c64"},
        # shots from a canonical state
        {"name": "sample_q50_chi256_16k", "kind": "sample", "sites": 50, "chi": 256, "shots": 16384},
        # all nearest-neighbour and single-site observables
        {"name": "local_q50_chi256", "kind": "local", "sites": 50, "chi": 256, "dtype": "c64"},
        # the energy of a Hamiltonian
        {"name": "mpo_q16_chi128", "kind": "mpo", "sites": 16, "chi": 128, "dtype": "c64"},
        # one TDVP site
        {"name": "tdvp_chi200_d5", "kind": "tdvp", "chi_l": 200, "chi_r": 200, "mpo": 5, "dtype": "c64"},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["layer", "layer", "layer", "layer", "circuit", "graph", "canonical", "canonical", "sample",
                       "local", "mpo", "tdvp"])
    dtype = "c128" if rng.random() < 0.2 else "c64"
    if kind == "layer":
        chi = _log_int(rng, 8, 256 if dtype == "c64" else 48)
        return {"kind": "layer", "gate": rng.choice(["entangle", "trotter"]),
                "bonds": rng.choice(["even", "odd", "centre"]), "sites": rng.randint(6, 40),
                "chi": chi + chi % 2, "dtype": dtype}
    if kind == "circuit":
        return {"kind": "circuit", "sites": rng.randint(5, 10), "depth": rng.randint(3, 12)}
    if kind == "graph":
        lo = rng.randint(5, 7)
        return {"kind": "graph", "instances": rng.randint(3, 24), "lo": lo, "hi": lo + rng.randint(1, 3),
                "depth": rng.randint(3, 6)}
    if kind == "canonical":
        return {"kind": "canonical", "form": rng.choice(["left", "right", "mixed"]), "sites": rng.randint(6, 40),
                "chi": _log_int(rng, 8, 256 if dtype == "c64" else 96), "dtype": dtype}
    if kind == "sample":
        return {"kind": "sample", "sites": rng.randint(8, 50), "chi": _log_int(rng, 8, 256),
                "shots": _log_int(rng, 50, 16384)}
    if kind == "tdvp":
        return {"kind": "tdvp", "chi_l": _log_int(rng, 8, 200 if dtype == "c64" else 80),
                "chi_r": _log_int(rng, 8, 200 if dtype == "c64" else 80), "mpo": rng.randint(1, 6), "dtype": dtype}
    return {"kind": kind, "sites": rng.randint(6, 50 if kind == "local" else 16),
            "chi": _log_int(rng, 8, (256 if kind == "local" else 128) if dtype == "c64" else 64), "dtype": dtype}


# ------------------------------------------------------------------ inputs
def _randn(shape, dtype, gen):
    r = torch.float64 if dtype == C128 else torch.float32
    return torch.complex(torch.randn(shape, generator=gen, dtype=r, device=DEV),
                         torch.randn(shape, generator=gen, dtype=r, device=DEV))


def _isometry(rows, cols, dtype, gen):
    """Orthonormal columns when rows >= cols, orthonormal rows otherwise."""
    if rows >= cols:
        return torch.linalg.qr(_randn((rows, cols), dtype, gen))[0]
    return torch.linalg.qr(_randn((cols, rows), dtype, gen))[0].transpose(0, 1).contiguous()


def _chain(sites, chi):
    return [min(chi, 1 << min(i + 1, 30), 1 << min(sites - 1 - i, 30)) for i in range(sites - 1)]


def _layer_bonds(case):
    n = case["sites"]
    if case["bonds"] == "centre":
        return [n // 2 - 1]
    return list(range(0 if case["bonds"] == "even" else 1, n - 1, 2))


def _layer_dims(case):
    dims = _chain(case["sites"], case["chi"])
    if case["gate"] == "entangle":  # the gate doubles the bond to the cap
        for b in _layer_bonds(case):
            dims[b] = min(dims[b], max(1, case["chi"] // 2))
    return dims


def _layer_state(case, seed):
    """Site tensors (mixed gauge around every gate bond, Schmidt values in
    [0.3, 1]) and the layer's gates (host matrices, as a circuit has them)."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    host = torch.Generator().manual_seed(seed + 1)
    dt, n = _dt(case), case["sites"]
    dims = [1] + _layer_dims(case) + [1]
    T = [None] * n
    gates = []
    for b in _layer_bonds(case):
        l, m, r = dims[b], dims[b + 1], dims[b + 2]
        S = 0.3 + 0.7 * torch.rand(m, generator=gen, dtype=torch.float64, device=DEV)
        T[b] = (_isometry(2 * l, m, dt, gen) * S.to(dt)).reshape(l, 2, m).contiguous()
        T[b + 1] = _isometry(m, 2 * r, dt, gen).reshape(m, 2, r).contiguous()
        if case["gate"] == "entangle":
            u = [haar_unitary(host, 2).to(C128) for _ in range(4)]
            U = torch.kron(u[0], u[1]) @ CZ.to(C128) @ torch.kron(u[2], u[3])
        else:
            U = rzz(0.08 + 0.04 * float(torch.rand(1, generator=host)))
        gates.append((b, U.to(dt)))
    for i in range(n):
        if T[i] is None:
            T[i] = _randn((dims[i], 2, dims[i + 1]), dt, gen) / math.sqrt(2.0 * dims[i])
    return T, dims[1:-1], gates


def _canonical_state(case, seed):
    """Site tensors that a few gates took out of canonical form: isometries
    (towards the centre) with their bonds rescaled by factors in [0.6, 1]."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    n, dt = case["sites"], _dt(case)
    dims = [1] + _chain(n, case["chi"]) + [1]
    T = []
    for i in range(n):
        l, r = dims[i], dims[i + 1]
        A = _isometry(2 * l, r, dt, gen) if i < n // 2 else _isometry(l, 2 * r, dt, gen)
        S = 0.6 + 0.4 * torch.rand(r, generator=gen, dtype=torch.float64, device=DEV)
        T.append((A.reshape(l, 2, r) * S.to(dt)).contiguous())
    return T


def _right_isometric(sites, chi, dtype, gen):
    dims = [1] + _chain(sites, chi) + [1]
    T = []
    for i in range(sites):
        l, r = dims[i], dims[i + 1]
        A = _isometry(l, 2 * r, dtype, gen).reshape(l, 2, r)
        T.append(A.contiguous())
    return T


def _polarised(case, seed):
    """A right-isometric MPS biased towards |0> and rotated about y: magnetised in
    z and in x, as the states whose observables are of interest."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    dt, dims = _dt(case), [1] + _chain(case["sites"], case["chi"]) + [1]
    c, s = math.cos(0.3), math.sin(0.3)
    T = []
    for i in range(case["sites"]):
        l, r = dims[i], dims[i + 1]
        A = _randn((l, 2, r), dt, gen)
        A[:, 1, :] *= 0.4
        A = torch.stack([c * A[:, 0] - s * A[:, 1], s * A[:, 0] + c * A[:, 1]], dim=1)
        T.append((A / math.sqrt(1.16 * 2 * r)).contiguous())
    return T


def _heisenberg(n, seed, dtype):
    """Bond-5 MPO of sum J (XX + YY + ZZ) + h Z with disordered fields."""
    gen = torch.Generator().manual_seed(seed)
    P = [torch.tensor(m, dtype=C128) for m in ([[0, 1], [1, 0]], [[0, -1j], [1j, 0]], [[1, 0], [0, -1]])]
    eye, sites = torch.eye(2, dtype=C128), []
    for i in range(n):
        J = 0.5 + torch.rand(3, generator=gen, dtype=torch.float64)
        h = 1.0 + float(torch.rand(1, generator=gen, dtype=torch.float64))
        W = torch.zeros(5, 2, 2, 5, dtype=C128)
        W[0, :, :, 0] = eye
        W[4, :, :, 4] = eye
        W[0, :, :, 4] = h * P[2]
        for k in range(3):
            W[0, :, :, 1 + k] = J[k] * P[k]
            W[1 + k, :, :, 4] = P[k]
        if i == 0:
            W = W[0:1]
        if i == n - 1:
            W = W[..., 4:5]
        sites.append(W.to(dtype=dtype, device=DEV).contiguous())
    return aq.MPO(sites)


def _observables(n):
    X = torch.tensor([[0, 1], [1, 0]], dtype=C64)
    Z = torch.tensor([[1, 0], [0, -1]], dtype=C64)
    return [{i: Z, i + 1: Z} for i in range(n - 1)] + [{i: X} for i in range(n)]


def _mps(n, dt, chi=256, tensors=None, resident=False):
    m = aq.AdaptiveMPS(n, bond_dim=1, eps_bond=1e-8, chi_max_per_bond=chi, device=DEV, dtype=dt,
                       dtype_policy=aq.DTypePolicy(default=dt), device_resident=resident)
    if tensors is not None:
        m.tensors = tensors
        m.bond_dims = [t.shape[2] for t in tensors[:-1]]
    return m


def _graph_circuits(case, seed):
    ns = [case["lo"] + b % (case["hi"] - case["lo"] + 1) for b in range(case["instances"])]
    return ns, [haar_brickwork(n, case["depth"], seed=seed * 1000 + b) for b, n in enumerate(ns)]


def prepare(case, seed):
    kind, dt = case["kind"], _dt(case)
    if kind == "layer":
        T, dims, gates = _layer_state(case, seed)
        return {"kind": kind, "mps": _mps(case["sites"], dt, case["chi"]), "T": T, "dims": dims, "gates": gates,
                "eye": torch.eye(4, dtype=dt, device=DEV)}
    if kind == "circuit":
        return {"kind": kind, "n": case["sites"], "ops": haar_brickwork(case["sites"], case["depth"], seed=seed)}
    if kind == "graph":
        ns, circuits = _graph_circuits(case, seed)
        batch = aq.MPSBatch([_mps(n, C64, 64, resident=True) for n in ns])
        return {"kind": kind, "captured": batch.capture(circuits)}
    if kind == "canonical":
        return {"kind": kind, "form": case["form"], "mps": _mps(case["sites"], dt), "T": _canonical_state(case, seed)}
    if kind == "sample":
        gen = torch.Generator(device=DEV).manual_seed(seed)
        return {"kind": kind, "T": _right_isometric(case["sites"], case["chi"], C64, gen), "shots": case["shots"],
                "seed": seed}
    if kind == "local":
        return {"kind": kind, "mps": _mps(case["sites"], dt, tensors=_polarised(case, seed)), "dt": dt,
                "obs": [{i: o.to(dt) for i, o in ob.items()} for ob in _observables(case["sites"])]}
    if kind == "mpo":
        return {"kind": kind, "mps": _mps(case["sites"], dt, tensors=_polarised(case, seed)), "dt": dt,
                "mpo": _heisenberg(case["sites"], seed, dt)}
    if kind == "tdvp":
        gen = torch.Generator(device=DEV).manual_seed(seed)
        l, r, D = case["chi_l"], case["chi_r"], case["mpo"]
        return {"kind": kind, "A": _randn((l, 2, r), dt, gen) / math.sqrt(2.0 * r),
                "W": _randn((D, 2, 2, D), dt, gen), "L": _randn((l, D, l), dt, gen) / l,
                "R": _randn((r, D, r), dt, gen) / r}
    raise ValueError(kind)


# ------------------------------------------------------------------ one pass
def run(s):
    kind = s["kind"]
    if kind == "layer":
        m = s["mps"]
        m.tensors = s["T"]
        m.bond_dims = s["dims"]
        m.reset_stats()
        for b, U in s["gates"]:
            m.apply_two_site_gate(b, U)
        T = m.tensors
        pairs = [ops.contract_gate(T[b], T[b + 1], s["eye"]) for b, _ in s["gates"]]
        return [pairs, torch.tensor(m.bond_dims)]
    if kind == "circuit":
        m = _mps(s["n"], C64, 64, resident=True)
        for _, q, U in s["ops"]:
            m.apply_two_site_gate(q, U)
        return m.to_statevector()
    if kind == "graph":
        batch = s["captured"].replay().finish()
        return [m.to_statevector() for m in batch.instances]
    if kind == "canonical":
        m = s["mps"]
        m.tensors = s["T"]
        m.bond_dims = [t.shape[2] for t in s["T"][:-1]]
        if s["form"] == "left":
            m.to_left_canonical()
        elif s["form"] == "right":
            m.canonicalize_right_to_left()
        else:
            m.to_mixed_canonical(m.num_qubits // 2)
        return list(m.tensors)
    if kind == "sample":
        return list(sample_tensors(s["T"], s["shots"], s["seed"], return_pz=True))
    if kind == "local":
        return torch.tensor(aq.local_expectations(s["mps"], s["obs"]), dtype=s["dt"])
    if kind == "mpo":
        return torch.tensor(aq.expectation_value(s["mpo"], s["mps"]), dtype=s["dt"])
    if kind == "tdvp":
        return [aq.tdvp_left_environment(s["L"], s["A"], s["W"]), aq.tdvp_right_environment(s["R"], s["A"], s["W"]),
                aq.tdvp_apply_local_H(s["L"], s["W"], s["A"], s["R"])]
    raise ValueError(kind)


# ------------------------------------------------------------------ work
def _brickwork_work(n, depth):
    by, fl = 0.0, 0.0
    dims = [1] * (n + 1)
    for layer in range(depth):
        for b in range(layer % 2, n - 1, 2):
            l, m, r = dims[b], dims[b + 1], dims[b + 2]
            k = min(4 * m, 2 * l, 2 * r)
            fl += _gate_flops(l, m, r, k)
            dims[b + 1] = k
            by += 16 * 8
    return by, fl


def _gate_flops(l, m, r, k):
    """Contraction and gate, the smaller Gram matrix, and the projection onto k vectors."""
    return 32.0 * l * m * r + 128.0 * l * r + 8.0 * (4.0 * l * r) * (2 * min(l, r)) + 8.0 * 4.0 * l * r * k


def work(case):
    kind, es = case["kind"], 16 if case.get("dtype") == "c128" else 8
    by = fl = 0.0
    if kind == "layer":
        dims = [1] + _layer_dims(case) + [1]
        for b in _layer_bonds(case):
            l, m, r = dims[b], dims[b + 1], dims[b + 2]
            k = min(case["chi"], 2 * l, 2 * r, 2 * m)
            by += es * (2.0 * l * m + 2.0 * m * r + 16 + 4.0 * l * r)
            fl += _gate_flops(l, m, r, k) + 32.0 * l * k * r  # the last term: the merged pair
    elif kind == "circuit":
        by, fl = _brickwork_work(case["sites"], case["depth"])
        by += 8.0 * 2 ** case["sites"]
    elif kind == "graph":
        mid = (case["lo"] + case["hi"]) / 2
        b, f = _brickwork_work(int(mid), case["depth"])
        by, fl = case["instances"] * (b + 8.0 * 2 ** int(mid)), case["instances"] * f
    elif kind == "canonical":
        dims = [1] + _chain(case["sites"], case["chi"]) + [1]
        for i in range(case["sites"]):
            l, r = dims[i], dims[i + 1]
            by += 2.0 * es * 2 * l * r
            fl += 16.0 * 2 * l * r * r + 8.0 * 2 * l * r * l  # QR with its thin Q, and R absorbed by the neighbour
    elif kind == "sample":
        dims = [1] + _chain(case["sites"], case["chi"]) + [1]
        for i in range(case["sites"]):
            by += 8.0 * 2 * dims[i] * dims[i + 1]
            fl += 16.0 * case["shots"] * dims[i] * dims[i + 1]
        by += case["shots"] * 8.0 * (1 + case["sites"])
    elif kind in ("local", "mpo"):
        dims = [1] + _chain(case["sites"], case["chi"]) + [1]
        D = 5 if kind == "mpo" else 1
        for i in range(case["sites"]):
            l, r = dims[i], dims[i + 1]
            by += es * 2.0 * l * r
            step = 16.0 * l * l * r + 16.0 * l * r * r
            # local: left and right environments and up to three operator steps per site; mpo: D channels and the norm
            fl += step * (5 if kind == "local" else D + 1)
    elif kind == "tdvp":
        l, r, D = case["chi_l"], case["chi_r"], case["mpo"]
        by = es * (2.0 * D * l * l + 2.0 * D * r * r + 4.0 * l * r)
        fl = 2 * D * (16.0 * l * l * r + 16.0 * l * r * r) + 64.0 * D * D * (l * r)
    return {"bytes": by, "flops": fl}


# ------------------------------------------------------------------ 64-bit values
def _statevector(n, circuit):
    psi = torch.zeros(2 ** n, dtype=C128)
    psi[0] = 1
    for _, q, U in circuit:
        psi = torch.einsum("ab,lbr->lar", U.to(C128), psi.reshape(2 ** q, 4, -1)).reshape(-1)
    return psi


def _sweep_qr(T, left, lo, hi):
    """Householder QR sweep over sites lo..hi in 64 bits (diagonal of R real, LAPACK's signs)."""
    for i in (range(lo, hi) if left else range(hi, lo, -1)):
        l, _, r = T[i].shape
        if left:
            Q, R = torch.linalg.qr(T[i].reshape(2 * l, r))
            T[i] = Q.reshape(l, 2, -1)
            T[i + 1] = torch.einsum("ab,bpr->apr", R, T[i + 1])
        else:
            Q, R = torch.linalg.qr(T[i].reshape(l, 2 * r).transpose(0, 1))
            T[i] = Q.transpose(0, 1).reshape(-1, 2, r)
            T[i - 1] = torch.einsum("apb,bc->apc", T[i - 1], R.transpose(0, 1))


def _environment_value(T, W):
    E = torch.ones(1, 1, 1, dtype=C128, device=DEV)
    for A, w in zip(T, W):
        M = torch.einsum("Lab,bsB->LasB", E, A)
        M = torch.einsum("LstR,LasB->RatB", w, M)
        E = torch.einsum("atr,RatB->RrB", A.conj(), M)
    return E[0, 0, 0]


def _local_values(T, n):
    """<Z_i Z_i+1> and <X_i> (symmetric operators) from 64-bit environments."""
    Z = torch.tensor([1.0, -1.0], dtype=C128, device=DEV)
    Le, Re = [torch.ones(1, 1, dtype=C128, device=DEV)], [None] * n + [torch.ones(1, 1, dtype=C128, device=DEV)]

    def step(E, A, B):
        return torch.einsum("asr,asB->rB", A.conj(), torch.einsum("ab,bsB->asB", E, B))

    for A in T:
        Le.append(step(Le[-1], A, A))
    for i in range(n - 1, -1, -1):
        Re[i] = torch.einsum("asr,bsr->ab", torch.einsum("asc,cr->asr", T[i].conj(), Re[i + 1]), T[i])
    norm = Le[n][0, 0]
    out = []
    for i in range(n - 1):
        E = step(Le[i], T[i], T[i] * Z[None, :, None])
        E = step(E, T[i + 1], T[i + 1] * Z[None, :, None])
        out.append((E * Re[i + 2]).sum() / norm)
    for i in range(n):
        out.append((step(Le[i], T[i], T[i].flip(1)) * Re[i + 1]).sum() / norm)
    return torch.stack(out)


def exact(case, seed):
    kind = case["kind"]
    if kind == "layer":
        T, dims, gates = _layer_state(case, seed)
        pairs = []
        for b, U in gates:
            A, B = T[b].to(C128), T[b + 1].to(C128)
            X = torch.einsum("apr,rqj->apqj", A, B)
            X = torch.einsum("pqst,astj->apqj", U.to(device=DEV, dtype=C128).reshape(2, 2, 2, 2), X)
            X = X.reshape(2 * A.shape[0], 2 * B.shape[2])
            if min(X.shape) > case["chi"] and case["gate"] == "trotter":  # truncated at the cap
                if X.shape[0] < X.shape[1]:
                    V = torch.linalg.eigh(X @ X.conj().transpose(0, 1))[1][:, -case["chi"]:]
                    X = V @ (V.conj().transpose(0, 1) @ X)
                else:
                    V = torch.linalg.eigh(X.conj().transpose(0, 1) @ X)[1][:, -case["chi"]:]
                    X = (X @ V) @ V.conj().transpose(0, 1)
            pairs.append(X)
        return [pairs, None]
    if kind == "circuit":
        return _statevector(case["sites"], haar_brickwork(case["sites"], case["depth"], seed=seed))
    if kind == "graph":
        ns, circuits = _graph_circuits(case, seed)
        return [_statevector(n, c) for n, c in zip(ns, circuits)]
    if kind == "canonical":
        T = [t.to(C128).cpu() for t in _canonical_state(case, seed)]
        n = len(T)
        if case["form"] == "left":
            _sweep_qr(T, True, 0, n - 1)
        elif case["form"] == "right":
            _sweep_qr(T, False, 0, n - 1)
        else:
            _sweep_qr(T, True, 0, n // 2)
            _sweep_qr(T, False, n // 2, n - 1)
        return T
    if kind == "local":
        return _local_values([t.to(C128) for t in _polarised(case, seed)], case["sites"])
    if kind == "mpo":
        T = [t.to(C128) for t in _polarised(case, seed)]
        W = _heisenberg(case["sites"], seed, C128).tensors
        eye = torch.eye(2, dtype=C128, device=DEV).reshape(1, 2, 2, 1)
        return (_environment_value(T, W) / _environment_value(T, [eye] * len(T))).reshape(())
    if kind == "tdvp":
        s = prepare(case, seed)
        A, W, L, R = (s[k].to(C128) for k in ("A", "W", "L", "R"))
        left = torch.einsum("qlsj,qtu,lstn->unj", torch.einsum("qli,isj->qlsj", L, A), A.conj(), W)
        right = torch.einsum("unj,qtu,lstn,isj->qli", R, A.conj(), W, A)
        local = torch.einsum("li,lstn,isj,nj->itj", L.sum(0), W, A, R.sum(0))
        return [left, right, local]
    return None  # sampling: its decisions are whole numbers
