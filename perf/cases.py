"""The work that programs built on this library have it do, as cases to time.

A case is one use of the public entry points (the C ABI through
``qcs_gb300.capi``, the qc_* API, the batch engine, the cost model's training)
at one size.  ``prepare`` makes what such a program holds before the call, from
a seed; ``run`` is the call; ``exact`` is the same result in 64 bits by plain
torch, without this library.

Kinds of case (``use``):

  api      the smallest programs: Bernstein-Vazirani gate by gate through the
           qc_* API, then every qubit measured -- latency and launches
  plain    a whole gate list, no fusion asked for (the default of the library
           and of qc_create), run again and again from |0...0>
  sweep    the same with new angles on every call (a variational loop) and
           <Z> of three qubits read back
  fused    a gate list fused into blocks of at most k qubits
  grover   QFT, then rounds of (Hadamard layer, phase flip, diffusion), fused
  readout  norm, P(0), <Z>, the most likely state and 1024 shots of one state
  batch    many small circuits at once, <Z_0> and 1024 shots each
  train    the fusion cost model trained on timing records
"""
import ctypes
import math

import numpy as np
import torch

from qcs_gb300 import capi
from qcs_gb300 import workloads as W

C64, C128 = "c64", "c128"


def listed():
    return [
        # the README's smallest programs: a handful of qubits, one gate a call
        {"name": "api_bv_10q", "use": "api", "n": 10},
        # a small circuit from the test range, an odd qubit count, one state
        {"name": "plain_c64_13q", "use": "plain", "n": 13, "prec": C64, "sem": "physical",
         "circuit": "random", "depth": 0},
        # a variational loop: every call has new angles, so no list repeats
        {"name": "sweep_c64_16q", "use": "sweep", "n": 16, "prec": C64, "depth": 8},
        # the 20-qubit complex128 configuration: QFT, then 200 random gates
        {"name": "plain_c128_20q", "use": "plain", "n": 20, "prec": C128, "sem": "physical",
         "circuit": "random", "depth": 0},
        # a program that depends on the reference's exact numbers
        {"name": "reference_c128_17q", "use": "plain", "n": 17, "prec": C128,
         "sem": "reference", "circuit": "random", "depth": 0},
        # a state in HBM, one gate at a time: the default settings at an odd size
        {"name": "plain_c64_27q", "use": "plain", "n": 27, "prec": C64, "sem": "physical",
         "circuit": "brick", "depth": 8},
        # the headline: 30 qubits, depth 40, 7-qubit blocks
        {"name": "fused7_c64_30q", "use": "fused", "n": 30, "k": 7, "circuit": "brick",
         "depth": 40},
        # the circuits of the cost model's evaluation, on a state that stays in L2
        {"name": "fused6_c64_20q", "use": "fused", "n": 20, "k": 6, "circuit": "mixed",
         "depth": 20},
        # the Grover configuration (QFT + rounds) with its fused diffusions
        {"name": "grover_c64_26q", "use": "grover", "n": 26, "k": 7, "rounds": 8},
        # what is read from a large state after a circuit
        {"name": "readout_c64_28q", "use": "readout", "n": 28, "prec": C64},
        # the batch configuration's ranges: 10-22 qubits, 4-16 layers
        {"name": "batch_384", "use": "batch", "count": 384, "n_min": 10, "n_max": 22},
        # fitting the planner's cost model on a machine's timing records
        {"name": "train_4096", "use": "train", "rows": 4096, "batch": 256, "epochs": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    use = rng.choice(("api", "plain", "plain", "sweep", "fused", "grover", "readout", "batch",
                      "train"))
    if use == "api":
        return {"use": use, "n": rng.randint(4, 16)}
    if use == "plain":
        prec = rng.choice((C64, C64, C128))
        n = rng.randint(10, 27 if prec == C64 else 22)
        circuit = rng.choice(("random", "brick", "mixed"))
        depth = 0 if circuit == "random" else rng.randint(3, 8 if n > 24 else 16)
        if n > 25:
            circuit, depth = "brick", rng.randint(3, 8)
        sem = "reference" if prec == C128 and rng.random() < 0.4 else "physical"
        return {"use": use, "n": n, "prec": prec, "sem": sem, "circuit": circuit, "depth": depth}
    if use == "sweep":
        return {"use": use, "n": rng.randint(8, 20), "prec": rng.choice((C64, C64, C128)),
                "depth": rng.randint(3, 12)}
    if use == "fused":
        return {"use": use, "n": rng.randint(14, 28), "k": rng.randint(4, 7),
                "circuit": rng.choice(("brick", "mixed", "random")), "depth": rng.randint(6, 32)}
    if use == "grover":
        return {"use": use, "n": rng.randint(14, 26), "k": rng.randint(5, 7),
                "rounds": rng.randint(3, 12)}
    if use == "readout":
        return {"use": use, "n": rng.randint(9, 28), "prec": rng.choice((C64, C64, C128))}
    if use == "batch":
        n_min = rng.randint(6, 12)
        return {"use": use, "count": _log_int(rng, 16, 384), "n_min": n_min,
                "n_max": rng.randint(n_min + 1, 22)}
    batch = _log_int(rng, 100, 1000)
    return {"use": use, "rows": _log_int(rng, 300, 4096), "batch": batch,
            "epochs": rng.randint(1, 6)}


# ---- inputs ----------------------------------------------------------------

def _circuit(case, seed):
    """The gate list of a plain, fused or grover case, from |0...0>."""
    n = case["n"]
    if case["use"] == "grover":
        w = W.grover_workload(n, seed, iterations=case["rounds"])
        g = W.basis_gates(n, w.basis)
        g.extend(w.qft)
        g.extend(w.rounds)
        return g
    if case["circuit"] == "brick":
        return W.brick_circuit(n, case["depth"], seed)
    if case["circuit"] == "mixed":
        return W.mixed_circuit(n, case["depth"], seed)
    basis, gates = W.random_circuit(n, seed, 200)
    g = W.basis_gates(n, basis)
    g.extend(gates)
    return g


SWEEP_STEPS = 8  # angle sets a variational case goes round


def _sweep_ops(case, seed):
    """`depth` layers of RY, RZ on every qubit and a CNOT ladder; one op array
    per angle set."""
    n, g = case["n"], W.GateList()
    for _ in range(case["depth"]):
        for q in range(n):
            g.add(W.RY, q)
            g.add(W.RZ, q)
        for q in range(n - 1):
            g.add(W.CNOT, q + 1, q)
    ops = g.ops()
    turn = np.random.RandomState(seed % (1 << 32)).uniform(0, 2 * math.pi, (SWEEP_STEPS, len(ops)))
    sets = []
    for a in turn:
        o = ops.copy()
        o["angle"] = np.where(ops["kind"] == W.CNOT, 0.0, a)
        sets.append(o)
    return sets


def _sweep_qubits(n):
    return (0, n // 2, n - 1)


def _instances(case, seed):
    return W.variational_batch(case["count"], seed, n_range=(case["n_min"], case["n_max"]))


def _amplitudes(case, seed):
    """A normalised random state: (2^n, 2) reals on the GPU, of the case's type."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    real = torch.float64 if case["prec"] == C128 else torch.float32
    a = torch.randn((1 << case["n"], 2), generator=gen, device="cuda", dtype=real)
    total = sum(float(p.double().square().sum()) for p in a.split(1 << 24))
    return a.mul_(1.0 / math.sqrt(total))


def _draws(seed, count):
    return np.random.RandomState(seed % (1 << 32)).uniform(0, 1, count)


def _records(case, seed):
    """Feature rows like those of the planner's items, and log2 ms to fit."""
    r = np.random.RandomState(seed % (1 << 32))
    rows = case["rows"]
    x = np.zeros((rows, capi.COSTMODEL_FEATURES), dtype=np.float32)
    x[np.arange(rows), r.randint(0, 7, rows)] = 1.0
    x[:, 7] = r.randint(24, 33, rows) / 32.0
    x[:, 8] = r.randint(1, 8, rows) / 8.0
    x[:, 9] = r.randint(1, 80, rows) / 64.0
    x[:, 10:18] = r.uniform(size=(rows, 8)) < 0.3
    x[:, 18:20] = r.uniform(size=(rows, 2))
    y = (8 * x[:, 7] - 6 + 2 * x[:, 6] * x[:, 8] + x[:, 18] + 0.1 * r.normal(size=rows))
    return x, y.astype(np.float32)


LEARNING_RATE = 1e-3


class _Amplitudes:
    """The state's live buffer for torch, without a copy; keeps the state."""

    def __init__(self, state, ptr):
        self.state = state
        kind = "<f8" if state.precision == capi.C128 else "<f4"
        self.__cuda_array_interface__ = {"shape": (state.size, 2), "typestr": kind,
                                         "data": (ptr, False), "version": 3, "strides": None}


def _view(s):
    """Amplitudes of s["state"] as a tensor (one view per buffer)."""
    ptr = s["state"].device_ptr()
    if ptr not in s["views"]:
        s["views"][ptr] = torch.as_tensor(_Amplitudes(s["state"], ptr), device="cuda")
    return s["views"][ptr]


def _state(case):
    return capi.State(case["n"], capi.C128 if case.get("prec") == C128 else capi.C64,
                      capi.REFERENCE if case.get("sem") == "reference" else capi.PHYSICAL)


def prepare(case, seed):
    use = case["use"]
    s = {"case": case, "use": use, "views": {}}
    if use == "api":
        s["circuit"] = _Circuit(case["n"])
        s["hidden"] = int(_draws(seed, 1)[0] * (1 << (case["n"] - 1)))
        s["seed"] = seed % (1 << 31)
    elif use == "sweep":
        s["state"] = _state(case)
        s["sets"] = _sweep_ops(case, seed)
        s["step"] = 0
    elif use in ("plain", "fused", "grover"):
        s["state"] = _state(case)
        s["ops"] = _circuit(case, seed).ops()
    elif use == "readout":
        s["state"] = _state(case)
        _view(s).copy_(_amplitudes(case, seed))
        torch.cuda.synchronize()
        s["draws"] = _draws(seed, 1024)
    elif use == "batch":
        s["batch"] = capi.Batch(_instances(case, seed), shots=1024, seed=seed)
    else:
        s["model"] = capi.CostModel(seed=seed)
        s["init"] = s["model"].params()
        s["records"] = _records(case, seed)
    return s


class _Circuit:
    """A t_q_circuit that is destroyed with this object."""

    def __init__(self, n):
        self.n = n
        self.api = capi.api()
        self.c = self.api.qc_create_ex(n, capi.C64, capi.PHYSICAL, 0)
        if not self.c:
            raise RuntimeError("qc_create_ex failed")

    def __del__(self):
        if getattr(self, "c", None):
            self.api.qc_destroy(self.c)


def run(s):
    use, case = s["use"], s["case"]
    if use == "api":
        c = s["circuit"]
        libc = capi.libc()
        libc.srand(s["seed"])
        c.api.qc_set_basis(c.c, 0)
        c.api.qc_bernstein_vazirani(c.c, s["hidden"])
        bits = (ctypes.c_int * c.n)()
        c.api.qc_measure_all(c.c, bits)
        bits = np.array(bits, dtype=np.int64)
        found = int((bits << np.arange(c.n)).sum())
        return {"bits": bits, "p": c.api.qc_get_probability64(c.c, found)}
    if use == "sweep":
        st = s["state"]
        ops = s["sets"][s["step"] % SWEEP_STEPS]
        s["step"] += 1
        st.set_basis(0)
        st.run(ops)
        z = [st.expect_z(q) for q in _sweep_qubits(case["n"])]
        return {"z": z, "amplitudes": _view(s)}
    if use == "plain":
        s["state"].set_basis(0)
        s["state"].run(s["ops"])
        return _view(s)
    if use in ("fused", "grover"):
        s["state"].set_basis(0)
        s["state"].run(s["ops"], fusion_k=case["k"])
        return _view(s)
    if use == "readout":
        st, q = s["state"], case["n"] // 2
        return {"norm": st.norm_sq(), "p0": st.prob_zero(0), "z": st.expect_z(q),
                "argmax": st.argmax(), "samples": st.sample(s["draws"])}
    if use == "batch":
        z, samples, _ = s["batch"].run()
        return {"z": z, "samples": samples}
    m, (x, y) = s["model"], s["records"]
    m.set_params(s["init"])
    loss = m.train(x, y, epochs=case["epochs"], batch=case["batch"], lr=LEARNING_RATE)
    return {"params": m.params(), "loss": loss}


# ---- what a pass cannot do without ---------------------------------------------

# Real operations per amplitude: a real or purely imaginary 2x2 takes two
# products and a sum per real of the output; a phase is one complex product on
# the amplitudes it touches; permutations and signs take none.
_FLOPS = {W.H: 6, W.RX: 6, W.RY: 6, W.RZ: 6, W.P: 3, W.CPHASE: 1.5, W.PHASE_FLIP: 0,
          W.DIFFUSION: 4}


def _gate_flops(kinds, n):
    return sum(_FLOPS.get(int(k), 0) for k in kinds) * float(1 << n)


def work(case):
    use = case["use"]
    if use in ("api", "sweep", "plain", "fused", "grover"):
        n = case["n"]
        amp = 16.0 if case.get("prec") == C128 else 8.0
        if use == "api":
            kinds = [W.H] * (2 * n)
        elif use == "sweep":
            kinds = _sweep_ops(case, 0)[0]["kind"]
        else:
            kinds = _circuit(case, 0).kinds
        return {"bytes": amp * (1 << n) + 32.0 * len(kinds), "flops": _gate_flops(kinds, n)}
    if use == "readout":
        amps = float(1 << case["n"])
        return {"bytes": (16.0 if case["prec"] == C128 else 8.0) * amps, "flops": 4 * amps}
    if use == "batch":
        flops = nbytes = 0.0
        for n, g in _instances(case, 0):
            flops += _gate_flops(g.kinds, n)
            nbytes += 32.0 * len(g) + 8.0 * (1 + 1024)
        return {"bytes": nbytes, "flops": flops}
    f, h = capi.COSTMODEL_FEATURES, 64
    weights = f * h + 2 * h * h + h
    steps = case["epochs"] * case["rows"]
    return {"bytes": 4.0 * (case["rows"] * (f + 1) + 2 * weights), "flops": 6.0 * weights * steps}


# ---- the same results in 64 bits -------------------------------------------------

def _matrix(kind, angle):
    c, s = math.cos(angle / 2), math.sin(angle / 2)
    r = 1.0 / math.sqrt(2.0)
    return {W.H: (r, r, r, -r), W.X: (0, 1, 1, 0), W.Y: (0, -1j, 1j, 0), W.Z: (1, 0, 0, -1),
            W.P: (1, 0, 0, complex(math.cos(angle), math.sin(angle))),
            W.RX: (c, -1j * s, -1j * s, c), W.RY: (c, -s, s, c),
            W.RZ: (complex(c, -s), 0, 0, complex(c, s)), W.CNOT: (0, 1, 1, 0),
            W.CPHASE: (1, 0, 0, complex(math.cos(angle), math.sin(angle)))}[kind]


def _apply(psi, m, target, control=-1, keep_high=False):
    """In place.  keep_high: the reference's controlled rule [[u00, u01], [0, 1]]."""
    n = psi.numel().bit_length() - 1
    if control < 0:
        v = psi.view(-1, 2, 1 << target)
        a, b = v[:, 0], v[:, 1]
    else:
        lo, hi = min(control, target), max(control, target)
        v = psi.view(1 << (n - 1 - hi), 2, 1 << (hi - lo - 1), 2, 1 << lo)
        if target > control:
            a, b = v[:, 0, :, 1], v[:, 1, :, 1]
        else:
            a, b = v[:, 1, :, 0], v[:, 1, :, 1]
    if m[1] == 0 and m[2] == 0:
        if m[0] != 1:
            a.mul_(m[0])
        if m[3] != 1 and not keep_high:
            b.mul_(m[3])
        return
    x = a * m[0] + b * m[1]
    if not keep_high:
        b.copy_(a * m[2] + b * m[3])
    a.copy_(x)


def _simulate(ops, n, reference=False):
    psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    psi[0] = 1
    for o in ops:
        kind = int(o["kind"])
        if kind == W.PHASE_FLIP:
            psi[int(o["index"])] *= -1
        elif kind == W.DIFFUSION:
            psi.neg_().add_(-2 * psi.mean())
        elif kind in (W.CNOT, W.CPHASE):
            _apply(psi, _matrix(kind, float(o["angle"])), int(o["target"]), int(o["control"]),
                   reference)
        else:
            _apply(psi, _matrix(kind, float(o["angle"])), int(o["target"]))
    return psi


def _exact_batch(case, seed):
    """<Z_0> of each instance: per layer one 2x2 on every qubit, then the CNOT
    ladder as one permutation."""
    out = []
    for n, g in _instances(case, seed):
        psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
        psi[0] = 1
        i = torch.arange(1 << n, device="cuda")
        src = i ^ ((i << 1) & ((1 << n) - 1))  # bit q + 1 ^= bit q, for every q upwards
        layer = 3 * n - 1
        for at in range(0, len(g), layer):
            for q in range(n):
                ry = np.array(_matrix(W.RY, g.angles[at + 2 * q])).reshape(2, 2)
                rz = np.array(_matrix(W.RZ, g.angles[at + 2 * q + 1])).reshape(2, 2)
                _apply(psi, [complex(v) for v in (rz @ ry).reshape(-1)], q)
            psi = psi[src]
        p = torch.view_as_real(psi).square().sum(1).view(-1, 2).sum(0)
        out.append(float(p[0] - p[1]))
    return np.array(out)


def _exact_train(case, seed):
    x, y = (torch.from_numpy(a).double().cuda() for a in _records(case, seed))
    p = torch.from_numpy(capi.CostModel(seed=seed).params()).double().cuda()
    f, h = x.shape[1], 64
    sizes = [f * h, h, h * h, h, h * h, h, h, 1]

    def loss_of(p, x, y):
        w1, b1, w2, b2, w3, b3, w4, b4 = p.split(sizes)
        a = torch.relu(x @ w1.view(f, h) + b1)
        a = torch.relu(a @ w2.view(h, h) + b2)
        a = torch.relu(a @ w3.view(h, h) + b3)
        return ((a @ w4 + b4) - y).square().mean()

    b1, b2, lr = (float(np.float32(v)) for v in (0.9, 0.999, LEARNING_RATE))
    m, v, step = torch.zeros_like(p), torch.zeros_like(p), 0
    batch = min(case["batch"], case["rows"])
    for _ in range(case["epochs"]):
        for r in range(0, case["rows"], batch):
            q = p.clone().requires_grad_(True)
            (grad,) = torch.autograd.grad(loss_of(q, x[r:r + batch], y[r:r + batch]), q)
            step += 1
            m = b1 * m + (1 - b1) * grad
            v = b2 * v + (1 - b2) * grad * grad
            p = p - lr * (m / (1 - b1 ** step)) / ((v / (1 - b2 ** step)).sqrt() + 1e-8)
    return {"params": p, "loss": float(loss_of(p, x, y))}


def exact(case, seed):
    use, n = case["use"], case.get("n", 0)
    if use == "api":
        # the input register reads the hidden string, the ancilla (|0> - |1>) /
        # sqrt(2) the draw; the state that is left has probability one
        return {"bits": None, "p": 1.0}
    if use == "sweep":
        psi = _simulate(_sweep_ops(case, seed)[0], n)
        pr = torch.view_as_real(psi).square().sum(1)
        z = []
        for q in _sweep_qubits(n):
            half = pr.view(-1, 2, 1 << q).sum((0, 2))
            z.append(float(half[0] - half[1]))
        return {"z": z, "amplitudes": torch.view_as_real(psi)}
    if use in ("plain", "fused", "grover"):
        g = _circuit(case, seed)
        if len(g) * float(1 << n) > 1.5e11:
            return None  # minutes in 64 bits
        psi = _simulate(g.ops(), n, case.get("sem") == "reference")
        return torch.view_as_real(psi)
    if use == "readout":
        norm = p0 = z = 0.0
        q = n // 2
        chunk = 1 << min(n, 24)
        for at, a in enumerate(_amplitudes(case, seed).split(chunk)):
            pr = a.double().square().sum(1)
            norm += float(pr.sum())
            p0 += float(pr[0::2].sum())
            half = pr.view(-1, 2, 1 << q).sum((0, 2))  # q < 24
            z += float(half[0] - half[1])
        return {"norm": norm, "p0": p0, "z": z, "argmax": None, "samples": None}
    if use == "batch":
        return {"z": _exact_batch(case, seed), "samples": None}
    return _exact_train(case, seed)
