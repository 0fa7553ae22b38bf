"""Timed cases of the engine: whole calls through the Python binding, as a
program that uses the engine makes them, with their inputs, their work, their
tolerances and an independent 64-bit evaluation of the same inputs.

A case is a dict of plain values.  ``kind`` says which call it is:

  circuit   reset, the gate calls of one seeded circuit, then what the program
            reads: DO MEASUREMENT (all spins) and / or the amplitudes (host
            copy of a small state, device view of a large one)
  gradient  energy and gradient of the hardware-efficient ansatz on a kept
            adjoint context (one step of an optimiser loop)
  batch     energies and gradients of many ansatz instances of uneven size
  observe   energy of the ansatz Hamiltonian and all spins of a given state
  events    GENERATE EVENTS: basis-state samples of a given state
  unitary   dense k-qubit unitaries on random targets of a given state

The circuits, the ansatz and its Hamiltonian are the generators of
riken-braket_b200/circuits.py; the sizes are those of its tests and benchmark.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
from __graft_entry__ import load_package  # noqa: E402

pkg = load_package()
C = pkg.circuits

PRECISION = {"c128": 0, "c64": 1}
AMP_BYTES = {"c128": 16, "c64": 8}


def listed():
    return [
        # The reference's sample programs (hadamards08, adder6x2, shor12) have 8 to 12
        # qubits: latency of one short program whose amplitudes and spins are printed.
        dict(name="brick_c128_8q", kind="circuit", circuit="brick", precision="c128", n=8, depth=6, fuse=0, mode=0, read="both_host"),
        # A program of mixed gates just above the smallest tile, in complex<float>.
        dict(name="random_c64_13q", kind="circuit", circuit="random", precision="c64", n=13, depth=200, fuse=0, mode=0, read="amps_host"),
        # The 20-qubit brick (the smallest of the benchmark family): 10 fused layers, all amplitudes and spins.
        dict(name="brick_c128_20q", kind="circuit", circuit="brick", precision="c128", n=20, depth=10, fuse=5, mode=0, read="both"),
        # The benchmark's own circuit: 30 qubits, 20 layers, fusion blocks of 5 qubits, DO MEASUREMENT.
        dict(name="brick_c128_30q", kind="circuit", circuit="brick", precision="c128", n=30, depth=20, fuse=5, mode=0, read="both"),
        # The QFT workload in complex<float>, gate by gate inside the fused passes (the default mode).
        dict(name="qft_c64_29q", kind="circuit", circuit="qft", precision="c64", n=29, depth=5, fuse=6, mode=0, read="amps"),
        # The same workload with each fusion block as one tensor-core unitary.
        dict(name="qft_tensor_c64_28q", kind="circuit", circuit="qft", precision="c64", n=28, depth=5, fuse=6, mode=1, read="amps"),
        # The benchmark's gradient: 20 qubits, 16 layers, 640 parameters, one optimiser step.
        dict(name="gradient_c128_20q", kind="gradient", precision="c128", n=20, depth=16),
        # A larger complex<float> gradient of few layers (the upper sizes of the batch workload).
        dict(name="gradient_c64_23q", kind="gradient", precision="c64", n=23, depth=5),
        # The batch workload at its lower sizes, where most of its instances lie.
        dict(name="batch_c128_10_15q", kind="batch", precision="c128", count=96, n_min=10, n_max=15, depth_min=4, depth_max=16),
        # The optimiser's and the benchmark's observables of a large given state.
        dict(name="observe_c128_27q", kind="observe", precision="c128", n=27),
        # Sampling from a large state (GENERATE EVENTS 1000).
        dict(name="events_c128_26q", kind="events", precision="c128", n=26, shots=1000),
        # Dense block unitaries (bra's fused 2^k x 2^k blocks given as matrices) in complex<double>.
        dict(name="unitary_c128_24q", kind="unitary", precision="c128", n=24, k=4, blocks=4),
    ]


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["circuit", "circuit", "circuit", "gradient", "batch", "observe", "events", "unitary"])
    precision = rng.choice(["c128", "c64"])
    c = dict(kind=kind, precision=precision)
    if kind == "circuit":
        circuit = rng.choice(["brick", "random", "qft"])
        n = rng.randint(5, 28)
        depth = rng.randint(2, 20) if circuit == "brick" else rng.randint(50, 400) if circuit == "random" else rng.randint(1, 5)
        mode = 1 if circuit == "qft" and precision == "c64" and n >= 13 and rng.random() < 0.4 else 0
        fuse = 6 if mode else rng.choice([0, 0, 3, 4, 5, 6])
        # Spins of a deep random state are sums that nearly cancel: only complex<double> states are read that way.
        read = rng.choice(["both", "amps"]) if precision == "c128" else "amps"
        c.update(circuit=circuit, n=n, depth=depth, fuse=0 if circuit == "random" else fuse, mode=mode,
                 read=read + ("_host" if n <= 13 else ""))
    elif kind == "gradient":
        c.update(n=rng.randint(6, 23), depth=rng.randint(2, 16))
    elif kind == "batch":
        lo = rng.randint(6, 12)
        c.update(count=log_int(rng, 12, 128), n_min=lo, n_max=rng.randint(lo + 1, 16), depth_min=4, depth_max=rng.randint(6, 16))
    elif kind == "observe":
        c.update(n=rng.randint(8, 28))
    elif kind == "events":
        c.update(n=rng.randint(6, 27), shots=log_int(rng, 1, 20000))
    else:
        c.update(n=rng.randint(14, 26), k=rng.randint(2, 6), blocks=rng.randint(1, 6))
    return c


# ---- inputs ---------------------------------------------------------------


def circuit_ops(case, seed):
    if case["circuit"] == "brick":
        return C.brick(case["n"], case["depth"], seed=seed, fuse_k=case["fuse"])
    if case["circuit"] == "qft":
        return C.qft_brick(case["n"], case["depth"], seed=seed, fuse_k=case["fuse"])
    return C.random_circuit(case["n"], case["depth"], seed=seed)


class DeviceAmplitudes:
    """The amplitudes of a state as a torch view of the engine's own memory (kept alive by the view)."""

    def __init__(self, state):
        self.state = state
        c128 = state.precision == PRECISION["c128"]
        self.dtype = torch.complex128 if c128 else torch.complex64
        self.__cuda_array_interface__ = {"shape": (1 << state.n,), "typestr": "<c16" if c128 else "<c8",
                                         "data": (state.device_pointer(), False), "version": 3, "strides": None}


def device_view(state):
    return torch.as_tensor(DeviceAmplitudes(state), device="cuda:0")


def random_amplitudes(n, precision, seed):
    """A normalised state: a random product state (magnetised, as prepared states are) plus Gaussian noise."""
    dtype = torch.complex128 if precision == "c128" else torch.complex64
    g = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)
    a = torch.ones(1, dtype=dtype, device="cuda")
    for _ in range(n):
        v = rng.standard_normal(2) + 1j * rng.standard_normal(2)
        v = torch.tensor(v / np.linalg.norm(v), dtype=dtype, device="cuda")
        a = (v[:, None] * a[None, :]).reshape(-1)
    a += torch.randn(1 << n, dtype=dtype, device="cuda", generator=g).mul_(0.7 * 2.0 ** (-n / 2))
    norm = math.sqrt(float(torch.view_as_real(a).square().sum(dtype=torch.float64)))
    return a.div_(norm)


def loaded_state(case, seed):
    s = pkg.State(case["n"], PRECISION[case["precision"]])
    device_view(s).copy_(random_amplitudes(case["n"], case["precision"], seed))
    torch.cuda.synchronize()
    return s


def block_unitaries(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(case["blocks"]):
        d = 1 << case["k"]
        q, r = np.linalg.qr(rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d)))
        out.append((q * (np.diag(r) / np.abs(np.diag(r))), [int(x) for x in rng.permutation(case["n"])[:case["k"]]]))
    return out


def batch_shapes(case):
    """(n, layers) of each instance: the uneven mix belongs to the case, the parameters to the seed."""
    return [(n, layers) for n, layers, _ in C.batch_instances(case["count"], case["n_min"], case["n_max"],
                                                               case["depth_min"], case["depth_max"], seed_base=1)]


def batch_thetas(case, seed):
    rng = np.random.default_rng(seed)
    return [rng.uniform(-math.pi, math.pi, 2 * n * layers) for n, layers in batch_shapes(case)]


def gradient_theta(case, seed):
    return np.random.default_rng(seed).uniform(-math.pi, math.pi, 2 * case["n"] * case["depth"])


def prepare(case, seed):
    kind, precision = case["kind"], PRECISION[case["precision"]]
    if kind == "circuit":
        s = pkg.State(case["n"], precision)
        if case["mode"]:
            s.set_fusion_mode(case["mode"])
        return dict(case=case, state=s, ops=circuit_ops(case, seed), view=device_view(s))
    if kind == "gradient":
        spec, _ = pkg.adjoint.ansatz_spec(case["n"], case["depth"])
        return dict(case=case, ctx=pkg.adjoint.AdjointContext(case["n"], precision), spec=spec,
                    theta=gradient_theta(case, seed), terms=C.ansatz_hamiltonian(case["n"]))
    if kind == "batch":
        instances = []
        for n, layers in batch_shapes(case):
            spec, params = pkg.adjoint.ansatz_spec(n, layers)
            instances.append((n, spec, params, C.ansatz_hamiltonian(n)))
        return dict(case=case, batch=pkg.adjoint.Batch(instances, precision), thetas=batch_thetas(case, seed))
    s = loaded_state(case, seed)
    if kind == "observe":
        return dict(case=case, state=s, terms=C.ansatz_hamiltonian(case["n"]))
    if kind == "events":
        return dict(case=case, state=s, seed=seed)
    return dict(case=case, state=s, blocks=block_unitaries(case, seed), view=device_view(s))


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "circuit":
        s = state["state"]
        s.reset()
        s.apply(state["ops"])
        out = {}
        if case["read"].startswith("both"):
            out["spins"] = s.spins()
        if case["read"].endswith("_host"):
            out["amps"] = s.amplitudes()
        else:
            s.canonicalize()
            out["amps"] = state["view"]
        return out
    if kind == "gradient":
        energy, grad = state["ctx"].gradient(state["spec"], state["theta"], state["terms"])
        return {"value_and_grad": np.concatenate(([energy], grad))}
    if kind == "batch":
        energies, grads = state["batch"].run(state["thetas"])
        return {"energies": energies, "grads": np.concatenate(grads)}
    s = state["state"]
    if kind == "observe":
        e = s.expectation(state["terms"])
        return {"energy": e.real, "spins": s.spins()}
    if kind == "events":
        return {"events": s.generate_events(case["shots"], seed=state["seed"])}
    for u, q in state["blocks"]:
        s.apply_unitary(u, q)
    s.canonicalize()
    return {"amps": state["view"]}


# ---- work -----------------------------------------------------------------

DENSE = ("H", "U2", "U3", "EX", "EY")  # a 2x2 matrix: 4 complex products and 2 sums per amplitude pair
PHASE = ("U1", "U", "EZ")              # a factor on half (two qubits: a quarter) of the amplitudes


def ops_flops(ops, n):
    dense = sum(1 for m, _, _ in ops if m in DENSE)
    phases = sum(0.25 if m == "U" else 0.5 for m, _, _ in ops if m in PHASE)
    return (14.0 * dense + 6.0 * phases) * (1 << n)


def ansatz_flops(n, layers):
    """Forward sweep, two inverse sweeps, lambda = H psi and one overlap per parameter."""
    rot = 2 * n * layers
    return (3 * 14.0 * rot / 2 + 3 * 6.0 * rot / 2 + 4.0 * rot + 2 * 8.0 * (n + 1)) * (1 << n)


def work(case):
    kind, amp = case["kind"], AMP_BYTES[case["precision"]]
    if kind == "circuit":
        size = amp << case["n"]
        return {"bytes": float(size), "flops": ops_flops(circuit_ops(case, 1), case["n"])}
    if kind == "gradient":
        return {"bytes": 8.0 * (4 * case["n"] * case["depth"] + 1), "flops": ansatz_flops(case["n"], case["depth"])}
    if kind == "batch":
        shapes = batch_shapes(case)
        return {"bytes": 8.0 * sum(4 * n * layers + 1 for n, layers in shapes),
                "flops": sum(ansatz_flops(n, layers) for n, layers in shapes)}
    size = amp << case["n"]
    if kind == "observe":  # |a|^2 and the pair products of every qubit
        return {"bytes": float(size), "flops": (4.0 + 8.0 * case["n"]) * (1 << case["n"])}
    if kind == "events":
        return {"bytes": float(size + 8 * case["shots"]), "flops": 4.0 * (1 << case["n"])}
    return {"bytes": 2.0 * size, "flops": 8.0 * (1 << case["k"]) * (1 << case["n"]) * case["blocks"]}


# ---- tolerances -------------------------------------------------------------


def tolerance(case):
    """Relative 2-norm errors, about four times those seen against exact().
    complex<double>: amplitudes, gradients and reductions were 5e-16 to 4e-15 off;
    a gate near X may lose up to three digits in its factored form.  The spins
    of a deep circuit are sums that cancel to about 2^(-n/2) and keep an
    absolute error of some 1e-16.  complex<float>: amplitudes 3e-7 (13 qubits, 200
    gates) to 1e-6, gradients with their energy to 1e-6 (one vector: an energy
    alone may cancel to nearly nothing); the tensor-core blocks
    add their norm drift of about 1e-6 per block pass."""
    kind, c128 = case["kind"], case["precision"] == "c128"
    if kind == "events":
        return {"rel": 0.0, "differ": 0.001}  # an event moves only where its draw lies within rounding of a bin edge
    if kind == "observe" or c128:  # reductions are summed in 64 bits for both precisions
        spins = kind == "circuit" and case["read"].startswith("both")
        return {"rel": max(1e-12, 4e-16 * 2.0 ** (case["n"] / 2)) if spins else 1e-12}
    return {"rel": 2e-5 if case.get("mode") else 5e-6}


# ---- the same in 64 bits, without the engine --------------------------------


def bit_view(a, n, qubits):
    """`a` as a tensor with one axis of 2 for each listed qubit (ascending), plain axes between."""
    shape, axis_of, last = [], {}, n
    for q in sorted(qubits, reverse=True):
        shape.append(1 << (last - q - 1))
        axis_of[q] = len(shape)
        shape.append(2)
        last = q
    shape.append(1 << last)
    return a.view(shape), axis_of


def part(a, n, bits):
    """View of the amplitudes whose qubits have the given values: {qubit: 0 or 1}."""
    v, axis = bit_view(a, n, bits)
    for q in sorted(bits):  # the lowest qubits have the last axes
        v = v.select(axis[q], bits[q])
    return v


def apply_matrix(a, n, m, t, controls=()):
    ones = {c: 1 for c in controls}
    x, y = part(a, n, {t: 0, **ones}), part(a, n, {t: 1, **ones})
    x0 = x.clone()
    x.copy_(m[0][0] * x0 + m[0][1] * y)
    y.copy_(m[1][0] * x0 + m[1][1] * y)


def scale(a, n, bits, f):
    part(a, n, bits).mul_(f)


def gate(a, n, op):
    """One instruction of circuits.py on the torch state `a`."""
    mnem, q, p = op
    r = math.sqrt(0.5)
    e = lambda x: complex(math.cos(x), math.sin(x))  # noqa: E731
    if mnem == "H":
        apply_matrix(a, n, [[r, r], [r, -r]], q[0])
    elif mnem in ("X", "CNOT"):
        ctl = {q[0]: 1} if mnem == "CNOT" else {}
        x, y = part(a, n, {q[-1]: 0, **ctl}), part(a, n, {q[-1]: 1, **ctl})
        x0 = x.clone()
        x.copy_(y)
        y.copy_(x0)
    elif mnem == "Y":
        apply_matrix(a, n, [[0, -1j], [1j, 0]], q[0])
    elif mnem in ("Z", "CZ"):
        scale(a, n, {x: 1 for x in q}, -1.0)
    elif mnem == "U1":
        scale(a, n, {q[0]: 1}, e(p[0]))
    elif mnem == "U":
        f = e(2.0 * math.pi / float(1 << abs(int(p[0]))))
        scale(a, n, {x: 1 for x in q}, f if p[0] >= 0 else f.conjugate())
    elif mnem == "U2":
        apply_matrix(a, n, [[r, -r * e(p[1])], [r * e(p[0]), r * e(p[0]) * e(p[1])]], q[0])
    elif mnem == "U3":
        s, c = math.sin(0.5 * p[0]), math.cos(0.5 * p[0])
        apply_matrix(a, n, [[c, -s * e(p[2])], [s * e(p[1]), c * e(p[1]) * e(p[2])]], q[0])
    elif mnem == "EX":
        apply_matrix(a, n, [[math.cos(p[0]), 1j * math.sin(p[0])], [1j * math.sin(p[0]), math.cos(p[0])]], q[0])
    elif mnem == "EY":
        apply_matrix(a, n, [[math.cos(p[0]), math.sin(p[0])], [-math.sin(p[0]), math.cos(p[0])]], q[0])
    elif mnem == "EZ":
        scale(a, n, {q[0]: 0}, e(p[0]))
        scale(a, n, {q[0]: 1}, e(-p[0]))
    elif mnem == "SWAP":
        x, y = part(a, n, {q[0]: 1, q[1]: 0}), part(a, n, {q[0]: 0, q[1]: 1})
        x0 = x.clone()
        x.copy_(y)
        y.copy_(x0)
    elif mnem not in ("BEGIN FUSION", "END FUSION"):
        raise ValueError(mnem)


def exact_spins(a, n):
    out = np.empty((n, 3))
    for q in range(n):
        x, y = part(a, n, {q: 0}), part(a, n, {q: 1})
        c = complex((x.conj() * y).sum())
        z = float(torch.view_as_real(x.contiguous()).square().sum() - torch.view_as_real(y.contiguous()).square().sum())
        out[q] = c.real, c.imag, 0.5 * z
    return out


def exact_energy(a, n, spins):
    """<H> of circuits.ansatz_hamiltonian: X terms from the spins, ZZ terms from the parities."""
    e = float(spins[:, 0].sum())  # 0.5 <X_i> = <S_x>
    p = torch.view_as_real(a).square().sum(-1)
    for i in range(n):
        j = (i + 1) % n
        v, axis = bit_view(p, n, {i, j})
        for x in (0, 1):
            for y in (0, 1):
                w = v.select(max(axis[i], axis[j]), x).select(min(axis[i], axis[j]), y)
                e += float(w.sum()) * (1.0 if x == y else -1.0)
    return e


def zero_state(n):
    a = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    a[0] = 1.0
    return a


def exact_gradient(n, layers, theta):
    ops, _ = C.ansatz(n, layers, thetas=theta)
    psi = zero_state(n)
    for op in ops:
        gate(psi, n, op)
    lam = torch.zeros_like(psi)
    idx = torch.arange(1 << n, device="cuda")
    diag = torch.zeros(1 << n, dtype=torch.float64, device="cuda")
    for i in range(n):
        diag += 1.0 - 2.0 * (((idx >> i) ^ (idx >> ((i + 1) % n))) & 1)
        x, y = part(lam, n, {i: 0}), part(lam, n, {i: 1})
        x += 0.5 * part(psi, n, {i: 1})
        y += 0.5 * part(psi, n, {i: 0})
    lam += diag * psi
    energy = float((psi.conj() * lam).sum().real)
    grad = torch.zeros(theta.size, dtype=torch.float64, device="cuda")
    k = theta.size
    for op in reversed(ops):
        if op[0] in ("EY", "EZ"):
            k -= 1
            q = op[1][0]
            l0, l1, p0, p1 = (part(s, n, {q: b}) for s in (lam, psi) for b in (0, 1))
            if op[0] == "EY":  # <lam| Y |psi> = sum -i conj(l0) p1 + i conj(l1) p0
                o = (l1.conj() * p0).sum().real - (l0.conj() * p1).sum().real
            else:
                o = (l0.conj() * p0).sum().imag - (l1.conj() * p1).sum().imag
            grad[k] = o  # -2 scale Im <lam|P|psi> with scale = -1/2
        for s in (psi, lam):
            gate(s, n, op if op[0] == "CZ" else (op[0], op[1], (-op[2][0],)))
    return energy, grad.cpu().numpy()


def exact(case, seed):
    kind, n = case["kind"], case.get("n", 0)
    if kind == "events":
        return None
    if kind == "circuit":
        ops = circuit_ops(case, seed)
        if len(ops) * (1 << n) > 3e10:
            return None
        a = zero_state(n)
        for op in ops:
            gate(a, n, op)
        out = {"spins": exact_spins(a, n)} if case["read"].startswith("both") else {}
        out["amps"] = a
        return out
    if kind == "gradient":
        if 6 * n * case["depth"] * (1 << n) > 3e10:
            return None
        energy, grad = exact_gradient(n, case["depth"], gradient_theta(case, seed))
        return {"value_and_grad": np.concatenate(([energy], grad))}
    if kind == "batch":
        shapes = batch_shapes(case)
        if sum(n * layers for n, layers in shapes) > 15000:
            return None
        got = [exact_gradient(n, layers, t) for (n, layers), t in zip(shapes, batch_thetas(case, seed))]
        return {"energies": np.array([e for e, _ in got]), "grads": np.concatenate([g for _, g in got])}
    a = random_amplitudes(n, case["precision"], seed).to(torch.complex128)
    if kind == "observe":
        spins = exact_spins(a, n)
        return {"energy": exact_energy(a, n, spins), "spins": spins}
    for u, q in block_unitaries(case, seed):
        axes = [n - 1 - x for x in reversed(q)]
        t = torch.movedim(a.view([2] * n), axes, list(range(len(q))))
        shape = t.shape
        t = torch.from_numpy(u).to("cuda") @ t.reshape(1 << len(q), -1)
        a = torch.movedim(t.reshape(shape), list(range(len(q))), axes).reshape(-1)
    return {"amps": a}
