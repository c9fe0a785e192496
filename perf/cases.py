"""The calls this library's users make, as timed cases.

A case is one pass through the public entry points (class ``ZXH``, the
``adjoint`` helpers, ``Batch``) on seeded inputs of the shapes the benchmark
configurations and the tests use. Kinds:

* ``plain``    -- the drop-in call: push a gate list, execute, draw shots, read the
  state on the device (H on all, layers of U3 + cp chain). complex128, the
  reference's type; 12 qubits is the latency of a small job, 20 the ordinary one.
* ``window``   -- one diagonal window (p / cp gates) applied to a live state; after
  a CX chain when ``chain`` is set, where every selector is a parity of several bits.
* ``layers``   -- execute of U3 on every qubit + cz on a random matching, the
  large-state circuit.
* ``hidden``   -- the hidden-string circuit and its shots: CX fan-in, so the last
  H layer acts on transported qubits.
* ``sample``   -- many shots from a large live state, read back to the host.
* ``state``    -- the amplitudes in the reference's get_state order, into a device buffer,
  after a circuit with CX (the affine map is not the identity).
* ``energy``   -- one objective evaluation of a variational loop: execute an ansatz,
  then the expectation of the transverse-field Ising observable.
* ``gradient`` -- the same with the adjoint gradient of every parameter.
* ``batch``    -- energies and gradients of many uneven circuits in one launch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from zxh_adae_b200 import ZXH, workloads
from zxh_adae_b200 import adjoint as ad
from zxh_adae_b200 import records as rc
from zxh_adae_b200.batch import Batch

DEVICE = "cuda:0"


def listed():
    return [
        # a small job through the backend: latency of planning, launches and reads
        {"name": "plain_12q_c128", "kind": "plain", "n": 12, "layers": 10, "shots": 1024, "dtype": "complex128"},
        # the ordinary job: 20 qubits, 10 layers, 1024 shots
        {"name": "plain_20q_c128", "kind": "plain", "n": 20, "layers": 10, "shots": 1024, "dtype": "complex128"},
        # a large diagonal batch on a large state, the headline microbenchmark
        {"name": "window_30q_c64", "kind": "window", "n": 30, "gates": 4096, "chain": False, "dtype": "complex64"},
        # the same after X / CX transport, in the reference's precision
        {"name": "window_cx_28q_c128", "kind": "window", "n": 28, "gates": 1024, "chain": True, "dtype": "complex128"},
        # large-state layers of single-qubit gates and cz matchings, both types
        {"name": "layers_30q_c64", "kind": "layers", "n": 30, "layers": 2, "dtype": "complex64"},
        {"name": "layers_27q_c128", "kind": "layers", "n": 27, "layers": 4, "dtype": "complex128"},
        # an oracle-type circuit at full width and its shots
        {"name": "hidden_28q_c64", "kind": "hidden", "n": 28, "shots": 100000, "dtype": "complex64"},
        # a million shots from a large state
        {"name": "sample_29q_c64", "kind": "sample", "n": 29, "shots": 1000000, "dtype": "complex64"},
        # the whole state vector in the reference's order
        {"name": "state_27q_c64", "kind": "state", "n": 27, "dtype": "complex64"},
        # one energy of a 24-qubit variational run
        {"name": "energy_24q_c64", "kind": "energy", "n": 24, "reps": 8, "dtype": "complex64"},
        # energy and 432 gradients of the same ansatz
        {"name": "gradient_24q_c64", "kind": "gradient", "n": 24, "reps": 8, "dtype": "complex64"},
        # a sweep over uneven circuits: energies and gradients in one launch
        {"name": "batch_64x10-20q_c64", "kind": "batch", "count": 64, "nmin": 10, "nmax": 20, "layers": 20,
         "dtype": "complex64"},
    ]


def draw(rng):
    kind = rng.choice(["plain", "window", "layers", "hidden", "sample", "state", "energy", "gradient", "batch"])
    dtype = rng.choice(["complex64", "complex128"])
    wide = dtype == "complex128"

    def spread(lo, hi):  # whole numbers spread over the logarithm
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if kind == "plain":
        return {"kind": kind, "n": rng.randint(4, 20), "layers": rng.randint(1, 10), "shots": spread(16, 4096),
                "dtype": "complex128"}
    if kind == "window":
        return {"kind": kind, "n": rng.randint(14, 28 if wide else 30), "gates": spread(16, 4096),
                "chain": rng.random() < 0.5, "dtype": dtype}
    if kind == "layers":
        return {"kind": kind, "n": rng.randint(12, 27 if wide else 29), "layers": rng.randint(1, 4), "dtype": dtype}
    if kind == "hidden":
        return {"kind": kind, "n": rng.randint(10, 26 if wide else 28), "shots": spread(100, 100000), "dtype": dtype}
    if kind == "sample":
        return {"kind": kind, "n": rng.randint(10, 27 if wide else 29), "shots": spread(1000, 1000000),
                "dtype": dtype}
    if kind == "state":
        return {"kind": kind, "n": rng.randint(10, 26 if wide else 27), "dtype": dtype}
    if kind == "energy":
        return {"kind": kind, "n": rng.randint(8, 22 if wide else 24), "reps": rng.randint(1, 8), "dtype": dtype}
    if kind == "gradient":
        return {"kind": kind, "n": rng.randint(8, 22 if wide else 24), "reps": rng.randint(1, 8), "dtype": dtype}
    nmin = rng.randint(6, 14)
    return {"kind": kind, "count": spread(4, 64), "nmin": nmin, "nmax": rng.randint(nmin, 17 if wide else 19),
            "layers": rng.randint(2, 20), "dtype": dtype}


# ---------------------------------------------------------------------------
# inputs


def _state_circuit(n, seed):
    """H on all, U3 on all, a CX chain and X on some qubits, U3 on all: a dense state
    whose affine map mixes neighbouring bits."""
    rng = np.random.default_rng(seed)
    flips = [(rc.X, 0, int(q)) for q in rng.permutation(n)[: max(1, n // 3)]]
    return np.concatenate([workloads.h_all(n), workloads.u3_layer(n, seed), workloads.cx_chain(n),
                           rc.as_records(flips), workloads.u3_layer(n, seed + 1)])


def _product_circuit(n, seed):
    """RY by a random angle on every qubit: a product state with uneven probabilities."""
    th = np.random.default_rng(seed).uniform(0.6, 2.4, n)
    return rc.as_records([(rc.U3, 0, q, th[q], 0.0, 0.0) for q in range(n)])


def _ansatz(case, seed):
    circ = ad.hardware_efficient_ansatz(case["n"], case["reps"])
    rng = np.random.default_rng(seed)
    # an energy is asked for near a variational run's start (angles around zero), a
    # gradient anywhere
    if case["kind"] == "energy":
        params = rng.normal(0.0, 0.1, circ.nparams)
    else:
        params = rng.uniform(-math.pi, math.pi, circ.nparams)
    return circ, params, ad.tfim_terms(case["n"])


def _batch_circuits(case, seed):
    span = case["nmax"] - case["nmin"] + 1
    out = []
    for i in range(case["count"]):
        n = case["nmin"] + (7 * i) % span
        m, recs, terms, _h = workloads.batch_tfim(1, 1000 * seed + i, n, n, case["layers"])[0]
        out.append((m, recs, terms))
    return out


def _hidden(case, seed):
    return workloads.hidden_string(case["n"] - 1, seed)


def _torch_dtype(case):
    return torch.complex64 if case["dtype"] == "complex64" else torch.complex128


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "seed": seed}
    if kind == "batch":
        st["batch"] = Batch(_batch_circuits(case, seed), dtype=case["dtype"])
        return st
    n = case["n"]
    sim = ZXH(n, dtype=case["dtype"], device=0)
    st["sim"] = sim
    if kind == "plain":
        st["gates"] = workloads.plain_layers(n, case["layers"], seed)
        st["out"] = torch.empty(1 << n, dtype=_torch_dtype(case), device=DEVICE)
    elif kind == "window":
        head = workloads.h_all(n)
        sim.push_gates(np.concatenate([head, workloads.cx_chain(n)]) if case["chain"] else head)
        sim.execute()
        st["gates"] = workloads.diag_batch(n, case["gates"], seed)
    elif kind == "layers":
        st["gates"] = workloads.u3_matching_layers(n, case["layers"], seed)
    elif kind == "hidden":
        st["gates"], _secret = _hidden(case, seed)
    elif kind == "sample":
        sim.push_gates(_product_circuit(n, seed))
        sim.execute()
    elif kind == "state":
        sim.push_gates(_state_circuit(n, seed))
        sim.execute()
        st["out"] = torch.empty(1 << n, dtype=_torch_dtype(case), device=DEVICE)
    else:
        st["circ"], st["params"], st["terms"] = _ansatz(case, seed)
    return st


# ---------------------------------------------------------------------------
# one pass


class _DeviceArray:
    """A simulator's live state for torch.as_tensor (the CUDA array interface). The
    tensor keeps this object, and so the simulator that owns the memory."""

    def __init__(self, sim, ptr, count, typestr):
        self.sim = sim
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr, False), "version": 2}


def _view(sim):
    """The live state as a tensor, without a copy."""
    ptr, m, eb, _phase = sim.state_view()
    return torch.as_tensor(_DeviceArray(sim, ptr, 1 << m, "<c8" if eb == 8 else "<c16"), device=DEVICE)


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "batch":
        energies, grads = st["batch"].run("persistent")
        return {"energies": energies, "gradients": grads}
    sim = st["sim"]
    if kind == "plain":
        sim.clear_gates()
        sim.set_seed(st["seed"])
        sim.push_gates(st["gates"])
        sim.execute()
        sim.measure(case["shots"])
        words = sim.results_words()
        sim.get_state_device(st["out"].data_ptr(), st["out"].numel())
        return {"words": words.view(np.int64), "state": st["out"]}
    if kind == "window":
        sim.apply(st["gates"])
        return {"state": _view(sim)}
    if kind == "layers":
        sim.clear_gates()
        sim.push_gates(st["gates"])
        sim.execute()
        return {"state": _view(sim)}
    if kind == "hidden":
        sim.clear_gates()
        sim.set_seed(st["seed"])
        sim.push_gates(st["gates"])
        sim.execute()
        sim.measure(case["shots"])
        return {"words": sim.results_words().view(np.int64)}
    if kind == "sample":
        sim.set_seed(st["seed"])
        sim.measure(case["shots"])
        return {"words": sim.results_words().view(np.int64)}
    if kind == "state":
        sim.get_state_device(st["out"].data_ptr(), st["out"].numel())
        return {"state": st["out"]}
    if kind == "energy":
        return {"energy": ad.energy(sim, st["circ"], st["params"], st["terms"])}
    energy, grads = ad.adjoint(sim, st["circ"], st["params"], st["terms"])
    return {"energy": energy, "gradients": grads}


# ---------------------------------------------------------------------------
# what a pass cannot do without

# floating-point operations per amplitude: a 2x2 complex gate, a real rotation, P, CP, RZ
_GATE, _ROT, _P, _CP, _RZ = 14.0, 6.0, 3.0, 1.5, 6.0


def work(case):
    kind = case["kind"]
    eb = 8 if case["dtype"] == "complex64" else 16
    if kind == "batch":
        flops = by = 0.0
        for i in range(case["count"]):
            n = case["nmin"] + (7 * i) % (case["nmax"] - case["nmin"] + 1)
            fwd = case["layers"] * (n * (_ROT + 2 * _P) + (n - 1) * _CP)
            grad = case["layers"] * (3 * n + n - 1) * 4.0
            flops += (3 * fwd + grad + 6.0 * n) * 2.0 ** n
            by += 8.0 * (4 * n * case["layers"] * 2)  # angles in, gradients out
        return {"bytes": by, "flops": flops}
    n = case["n"]
    size = 2.0 ** n
    if kind == "plain":
        fl = n * _GATE + case["layers"] * (n * _GATE + (n - 1) * _CP)
        return {"bytes": size * eb + 8.0 * case["shots"], "flops": fl * size}
    if kind == "window":
        # each amplitude is read and written once, whatever the window's size
        return {"bytes": 2 * size * eb, "flops": 6.0 * size}
    if kind == "layers":
        return {"bytes": size * eb, "flops": case["layers"] * (n * _GATE + n // 2 * _CP) * size}
    if kind == "hidden":
        return {"bytes": size * eb + 8.0 * case["shots"], "flops": 2 * n * 4.0 * size}
    if kind == "sample":
        return {"bytes": size * eb + 16.0 * case["shots"], "flops": 4.0 * size}
    if kind == "state":
        return {"bytes": 2 * size * eb, "flops": 6.0 * size}
    fwd = (case["reps"] + 1) * n * (_ROT + _RZ)
    if kind == "energy":
        return {"bytes": size * eb, "flops": (fwd + 6.0 * n) * size}
    grad = 2 * n * (case["reps"] + 1) * 4.0
    return {"bytes": size * eb, "flops": (3 * fwd + grad + 6.0 * n) * size}


def tolerance(case):
    wide = case["dtype"] == "complex128"
    # a draw at the edge of two outcomes may fall to either
    if case["kind"] in ("sample", "hidden"):
        return {"differ": 1e-4}
    if case["kind"] == "plain":
        return {"rel": 2e-14, "differ": 0.005}
    if case["kind"] in ("energy", "gradient", "batch"):
        return {"rel": 1e-12 if wide else 4e-6}
    if case["kind"] == "window":  # phases of thousands of radians: their sums' own rounding
        return {"rel": 5e-13 if wide else 1.5e-6}
    return {"rel": 2e-14 if wide else 1.5e-6}


# ---------------------------------------------------------------------------
# the same in 64 bits, densely


def _u3(th, la, ph):
    c, s = math.cos(th / 2), math.sin(th / 2)
    e = lambda x: complex(math.cos(x), math.sin(x))  # noqa: E731
    return c, -e(la) * s, e(ph) * s, e(ph + la) * c


def _apply(psi, n, g, inverse=False):
    """One record on a dense state (qubit q at bit q), in place."""
    t, cq, q = int(g["type"]), int(g["cq"]), int(g["q"])
    th, la, ph = float(g["theta"]), float(g["lam"]), float(g["phi"])
    sign = -1.0 if inverse else 1.0
    if t == rc.BARRIER:
        return
    if t in (rc.CP, rc.CX):
        hi, lo = max(cq, q), min(cq, q)
        v = psi.view(1 << (n - 1 - hi), 2, 1 << (hi - lo - 1), 2, 1 << lo)
        if t == rc.CP:
            v[:, 1, :, 1, :] *= complex(math.cos(sign * th), math.sin(sign * th))
        else:
            a, b = (v[:, 1, :, 0, :], v[:, 1, :, 1, :]) if cq == hi else (v[:, 0, :, 1, :], v[:, 1, :, 1, :])
            tmp = a.clone()
            a.copy_(b)
            b.copy_(tmp)
        return
    v = psi.view(1 << (n - 1 - q), 2, 1 << q)
    if t == rc.P:
        v[:, 1, :] *= complex(math.cos(sign * th), math.sin(sign * th))
        return
    if t == rc.RZ:
        v[:, 0, :] *= complex(math.cos(sign * th / 2), -math.sin(sign * th / 2))
        v[:, 1, :] *= complex(math.cos(sign * th / 2), math.sin(sign * th / 2))
        return
    a = v[:, 0, :].clone()
    b = v[:, 1, :]
    if t == rc.X:
        v[:, 0, :] = b
        v[:, 1, :] = a
        return
    if t == rc.H:
        r = math.sqrt(0.5)
        u = (r, r, r, -r)
    elif t == rc.U3:
        u = _u3(th, la, ph)
        if inverse:
            c = [complex(x).conjugate() for x in u]
            u = (c[0], c[2], c[1], c[3])
    else:
        raise ValueError(f"no dense form of gate {t}")
    v[:, 0, :] = torch.add(a * u[0], b, alpha=u[1])
    b.mul_(u[3]).add_(a, alpha=u[2])


def _dense(n, gates, psi=None):
    if psi is None:
        psi = torch.zeros(1 << n, dtype=torch.complex128, device=DEVICE)
        psi[0] = 1.0
    for g in gates:
        _apply(psi, n, g)
    return psi


def _bit(n, q):
    return (torch.arange(1 << n, device=DEVICE) >> q) & 1


def _h_psi(psi, n, terms):
    d = torch.zeros(1 << n, dtype=torch.float64, device=DEVICE)
    out = torch.zeros_like(psi)
    for t in terms:
        q0, q1, c = int(t["q0"]), int(t["q1"]), float(t["coef"])
        if int(t["kind"]) == rc.TERM_X:
            v = psi.view(1 << (n - 1 - q0), 2, 1 << q0)
            out.view(v.shape).add_(v.flip(1), alpha=c)
            continue
        z = 1.0 - 2.0 * _bit(n, q0)
        if int(t["kind"]) == rc.TERM_ZZ:
            z = z * (1.0 - 2.0 * _bit(n, q1))
        d.add_(z, alpha=c)
    return out.add_(psi * d)


def _dense_gradient(n, gates, terms):
    """<H> and d<H>/d theta of every record, walking back with inverse gates."""
    psi = _dense(n, gates)
    lam = _h_psi(psi, n, terms)
    e = torch.vdot(psi, lam).real
    grads = torch.zeros(len(gates), dtype=torch.float64, device=DEVICE)
    for k in range(len(gates) - 1, -1, -1):
        g = gates[k]
        t, cq, q = int(g["type"]), int(g["cq"]), int(g["q"])
        v, w = psi.view(1 << (n - 1 - q), 2, 1 << q), lam.view(1 << (n - 1 - q), 2, 1 << q)
        im = lambda a, b: (a.conj() * b).imag.sum()  # noqa: E731
        if t == rc.U3:  # RY: Im <lam|Y|psi>
            grads[k] = (w[:, 1, :].conj() * v[:, 0, :]).real.sum() - (w[:, 0, :].conj() * v[:, 1, :]).real.sum()
        elif t == rc.RZ:
            grads[k] = im(w[:, 0, :], v[:, 0, :]) - im(w[:, 1, :], v[:, 1, :])
        elif t == rc.P:
            grads[k] = -2.0 * im(w[:, 1, :], v[:, 1, :])
        elif t == rc.CP:
            hi, lo = max(cq, q), min(cq, q)
            shape = (1 << (n - 1 - hi), 2, 1 << (hi - lo - 1), 2, 1 << lo)
            grads[k] = -2.0 * im(lam.view(shape)[:, 1, :, 1, :], psi.view(shape)[:, 1, :, 1, :])
        _apply(psi, n, g, inverse=True)
        _apply(lam, n, g, inverse=True)
    return float(e), grads.cpu().numpy()


def _reversed_bits(psi, n):
    """The reference's get_state order: qubit 0 at the most significant bit."""
    return psi.view((2,) * n).permute(tuple(range(n - 1, -1, -1))).reshape(-1) if n <= 24 else psi[_bitrev(n)]


def _bitrev(n):
    i = torch.arange(1 << n, device=DEVICE)
    r = torch.zeros_like(i)
    for q in range(n):
        r |= ((i >> q) & 1) << (n - 1 - q)
    return r




def exact(case, seed):
    kind = case["kind"]
    if kind in ("sample", "hidden"):
        return None
    if kind == "batch":
        if case["count"] * 2.0 ** case["nmax"] > 64 * 2.0 ** 14:
            return None
        es, gs = [], []
        for n, recs, terms in _batch_circuits(case, seed):
            e, g = _dense_gradient(n, recs, terms)
            es.append(e)
            gs.append(g)
        return {"energies": np.array(es), "gradients": np.concatenate(gs)}
    n = case["n"]
    if kind == "plain":
        psi = _dense(n, workloads.plain_layers(n, case["layers"], seed))
        return {"words": None, "state": _reversed_bits(psi, n)}
    if kind == "window":
        # the real-address order of a state that X / CX have relabelled is the qubit
        # order before the relabelling: transport the gates instead
        psi = torch.full((1 << n,), 2.0 ** (-n / 2), dtype=torch.complex128, device=DEVICE)
        gates = workloads.diag_batch(n, case["gates"], seed)
        return {"state": psi * _window_phase(n, gates, case["chain"])}
    if kind == "layers":
        return {"state": _dense(n, workloads.u3_matching_layers(n, case["layers"], seed))}
    if kind == "state":
        return {"state": _reversed_bits(_dense(n, _state_circuit(n, seed)), n)}
    circ, params, terms = _ansatz(case, seed)
    recs = circ.records(params)
    if kind == "energy":
        psi = _dense(n, recs)
        return {"energy": float(torch.vdot(psi, _h_psi(psi, n, terms)).real)}
    e, g = _dense_gradient(n, recs, terms)
    return {"energy": e, "gradients": circ.gradient(g)}


def _window_phase(n, gates, chain):
    """exp(i sum theta) of a p / cp window over the real index: qubit q's bit is bit q,
    or, after the CX chain, the parity of bits 0..q. The coefficients of equal
    selectors are summed first; chunks keep the index arrays small."""
    lin = np.zeros(n)
    quad = np.zeros((n, n))
    for g in gates:
        if int(g["type"]) == rc.P:
            lin[int(g["q"])] += float(g["theta"])
        else:
            a, b = sorted((int(g["cq"]), int(g["q"])))
            quad[a, b] += float(g["theta"])
    lin_t = torch.from_numpy(lin).to(DEVICE)
    quad_t = torch.from_numpy(quad).to(DEVICE)
    out = torch.empty(1 << n, dtype=torch.complex128, device=DEVICE)
    step = 1 << min(n, 22)
    shifts = torch.arange(n, device=DEVICE)
    for at in range(0, 1 << n, step):
        i = torch.arange(at, at + step, device=DEVICE)
        bits = ((i[:, None] >> shifts) & 1).double()
        if chain:
            bits = torch.remainder(torch.cumsum(bits, 1), 2.0)
        th = bits @ lin_t + ((bits @ quad_t) * bits).sum(1)
        out[at:at + step] = torch.polar(torch.ones_like(th), th)
    return out
