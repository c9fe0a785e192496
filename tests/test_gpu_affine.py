"""Affine tile passes: gates with any pair deltas in tiles of 2^12 amplitudes, at the
smallest states that take them (12 qubits: one tile), and above; deltas inside the runs,
dependent modulo the runs and spread over all bits; real and complex matrices; windows of
single and paired selectors; the adjoint form with checkpoints. Against the oracle, its dense
adjoint and the general strided passes (knob affine = 0)."""
import math

import numpy as np
import pytest

from oracle import observables as ob
from oracle.bridge import Oracle
from zxh_adae_b200 import ZXH, workloads
from zxh_adae_b200 import adjoint as ad
from zxh_adae_b200.records import CP, CX, H, P, RX, RZ, U3, X, Z, as_records

pytestmark = pytest.mark.gpu

TOL = {"complex64": 1e-6, "complex128": 1e-12}  # the parity suite's bounds on amplitudes


def layer(n, rng, gates, window):
    qs = rng.permutation(n)[: int(rng.integers(1, n + 1))]
    if gates == "real":
        recs = [(U3, 0, int(q), rng.uniform(0, 6), 0.0, 0.0) for q in qs]
    elif gates == "h":
        recs = [(H, 0, int(q)) for q in qs]
    else:
        recs = [(U3, 0, int(q), *rng.uniform(0, 6, 3)) for q in qs]
    if window == "linear":
        recs += [(int(rng.choice([RZ, P, Z])), 0, int(q), rng.uniform(0, 6)) for q in rng.permutation(n)[: n // 2]]
    elif window == "chain":
        recs += [(CP, i, i + 1, rng.uniform(0, 6)) for i in range(n - 1)]
    elif window == "dense":  # pairs of every kind, a pair of a qubit with itself, repeats
        for _ in range(40):
            a, b = (int(v) for v in rng.integers(0, n, 2))
            recs.append((CP, a, b, rng.uniform(0, 6)))
    return recs


def circuit(n, links, gates, window, seed, layers=4):
    rng = np.random.default_rng(seed)
    recs = [(H, 0, q) for q in range(n)]
    for _ in range(layers):
        if links == "chain":
            recs += [(CX, i, i + 1) for i in range(n - 1)]
        elif links == "back":  # from the high qubits down: deltas inside the runs mix
            recs += [(CX, i + 1, i) for i in range(n - 1)]
        else:
            recs += [(CX, int(a), int(b)) for a, b in rng.integers(0, n, (3 * n, 2)) if a != b]
        recs += [(X, 0, int(q)) for q in rng.permutation(n)[:3]]
        recs += layer(n, rng, gates, window)
    return as_records(recs)


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("window", ["none", "linear", "chain", "dense"])
@pytest.mark.parametrize("n,links,gates", [(12, "chain", "complex"), (12, "random", "real"), (13, "back", "complex"),
                                           (14, "chain", "h"), (15, "random", "complex"), (16, "back", "real")])
def test_affine_passes_against_oracle(n, links, gates, window, dtype):
    g = circuit(n, links, gates, window, seed=n)
    o = Oracle(n)
    o.push(g)
    o.execute()
    for affine in (1, 0):
        s = ZXH(n, dtype=dtype)
        s.set_param("affine", affine)
        s.push_gates(g)
        s.execute()
        assert np.max(np.abs(s.get_state(0).astype(np.complex128) - o.get_state(0))) <= TOL[dtype], affine
        s.close()


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
def test_affine_layers_applied_one_by_one(dtype):
    # phases an apply leaves over meet a batch of affine passes as its first window
    n = 13
    rng = np.random.default_rng(4)
    parts = [workloads.h_all(n), workloads.u3_layer(n, 1), workloads.cx_chain(n),
             as_records(layer(n, rng, "complex", "chain")), workloads.u3_layer(n, 2), workloads.cx_chain(n),
             as_records(layer(n, rng, "real", "linear"))]
    s = ZXH(n, dtype=dtype)
    s.push_gates(parts[0])
    s.execute()
    for p in parts[1:]:
        s.apply(p)
    o = Oracle(n)
    o.push(np.concatenate(parts))
    o.execute()
    assert np.max(np.abs(s.get_state(0).astype(np.complex128) - o.get_state(0))) <= TOL[dtype]
    s.close()


def ansatz(n, links, window, seed, layers=3):
    rng = np.random.default_rng(seed)
    recs, par = [], []

    def add(rec, parameter):
        recs.append(rec)
        par.append(sum(p >= 0 for p in par) if parameter else -1)

    for _ in range(layers):
        for q in rng.permutation(n):
            add((U3, 0, int(q), 0.0, 0.0, 0.0) if rng.random() < 0.7 else (RX, 0, int(q), 0.0), True)
        add((H, 0, int(rng.integers(n))), False)
        if window == "dense":
            for a, b in rng.integers(0, n, (20, 2)):
                if a != b:
                    add((CP, int(a), int(b), 0.0), True)
            add((Z, 0, 2), False)
        for q in rng.permutation(n)[: n - 2]:
            add((RZ if rng.random() < 0.5 else P, 0, int(q), 0.0), True)
        if links == "chain":
            for i in range(n - 1):
                add((CX, i, i + 1), False)
        else:
            for a, b in rng.integers(0, n, (2 * n, 2)):
                if a != b:
                    add((CX, int(a), int(b)), False)
        add((X, 0, int(rng.integers(n))), False)
    return ad.Circuit(n, as_records(recs), par)


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("n,links,window", [(12, "chain", "linear"), (12, "random", "dense"), (13, "random", "linear"),
                                            (15, "chain", "dense")])
def test_affine_gradients_against_dense_adjoint(n, links, window, dtype):
    circ = ansatz(n, links, window, seed=n)
    terms = ad.tfim_terms(n, h=0.6)
    p = np.random.default_rng(n).uniform(-math.pi, math.pi, circ.nparams)
    e_ref, g_ref = ob.dense_adjoint(n, circ.records(p), terms)
    s = ZXH(n, dtype=dtype)
    s.push_gates(circ.records(p))
    # energies and gradients are sums of 2 n unit terms of the state's relative error
    tol = 2 * n * (1e-12 if dtype == "complex128" else 1e-6)
    for affine in (0, 1):
        s.set_param("affine", affine)
        for every in (0, 7):
            e, g = s.adjoint_gradient(terms, every)
            assert abs(e - e_ref) <= tol, affine
            assert np.max(np.abs(g - g_ref)) <= tol, affine
    want = ob.oracle_state(n, circ.records(p))
    assert np.max(np.abs(ob.qubit_order(s.get_state(), n) - want)) <= TOL[dtype]  # the forward output stays
    s.close()


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
def test_affine_rotations_at_the_ends_of_their_forms(dtype):
    # cosine or sine zero, equal, and sign changes: the coefficient factored out of a rotation
    n = 12
    edge = [math.pi, 3 * math.pi, math.pi / 2, -math.pi / 2, 2 * math.pi, 3.0, 1e-3, 0.3]
    recs = [(H, 0, q) for q in range(n)]
    for r in range(3):
        recs += [(CX, i, (i + 1 + r) % n) for i in range(n)]
        recs += [(U3, 0, q, edge[(q + r) % len(edge)], 0.0, 0.0) for q in range(n)]
        recs += [(RZ, 0, q, 0.1 * q + r) for q in range(n)]
    g = as_records(recs)
    terms = ad.tfim_terms(n)
    e_ref, g_ref = ob.dense_adjoint(n, g, terms)
    s = ZXH(n, dtype=dtype)
    s.push_gates(g)
    e, grad = s.adjoint_gradient(terms)
    tol = 2 * n * (1e-12 if dtype == "complex128" else 1e-6)
    assert abs(e - e_ref) <= tol and np.max(np.abs(grad - g_ref)) <= tol
    want = ob.oracle_state(n, g)
    assert np.max(np.abs(ob.qubit_order(s.get_state(), n) - want)) <= TOL[dtype]
    s.close()


@pytest.mark.parametrize("turn", [9e-16, 2e-16, 5e-17])
def test_affine_gates_next_to_a_rotation_keep_their_phase(turn):
    # complex128: real amplitudes, then U3 gates whose imaginary parts are a fraction of
    # an ulp of 1; the state's imaginary part is their sum and carries no other error than
    # its own rounding (a relative 2^-53 per gate and amplitude; 1e-12 is 4500 of them)
    n = 12
    g = as_records([(U3, 0, q, 0.4 + 0.1 * q, 0.0, 0.0) for q in range(n)] + [(CX, i, i + 1) for i in range(n - 1)] +
                   [(U3, 0, q, 1.1 + 0.1 * q, turn, 0.0) for q in range(n)])
    o = Oracle(n)
    o.push(g)
    o.execute()
    want = o.get_state(0).imag
    s = ZXH(n, dtype="complex128")
    s.push_gates(g)
    s.execute()
    assert np.linalg.norm(s.get_state(0).imag - want) <= 1e-12 * np.linalg.norm(want)
    s.close()


@pytest.mark.parametrize("mode", ["persistent", "graph", "sequential"])
@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
def test_batched_tiles_against_dense_adjoint(mode, dtype):
    # circuits below, at and above the tile size, real and complex gates, with CX
    from zxh_adae_b200.batch import Batch

    circs = []
    for n, links, window in [(11, "chain", "linear"), (12, "random", "dense"), (14, "chain", "linear"), (9, "random", "dense")]:
        c = ansatz(n, links, window, seed=n)
        p = np.random.default_rng(n).uniform(-math.pi, math.pi, c.nparams)
        circs.append((n, c.records(p), ad.tfim_terms(n, h=0.8)))
    for n in (12, 13):  # a real queue's circuits (rotations), in the same batch
        circs.append(workloads.batch_tfim(1, n, n, n, 3)[0][:3])
    ref = [ob.dense_adjoint(n, r, t) for n, r, t in circs]
    for which in (circs, circs[-2:]):
        want = ref if which is circs else ref[-2:]
        b = Batch(which, dtype=dtype)
        for threads in (256, 128, 256):
            b.set("threads", threads)
            b.set("task_items", 32 if threads == 128 else 512)
            e, g = b.run(mode)
            for k, (n, _r, _t) in enumerate(which):
                tol = 2 * n * (1e-12 if dtype == "complex128" else 1e-6)
                assert abs(e[k] - want[k][0]) <= tol, (threads, n)
                assert np.max(np.abs(b.gradients(g)[k] - want[k][1])) <= tol, (threads, n)
        b.close()


@pytest.mark.parametrize("n", [3, 7, 12, 14])
def test_first_layer_on_expanded_qubits(n):
    # every qubit expanded and |0>: the first gate of each is part of the product state
    g = np.concatenate([as_records([(X, 0, 1), (CX, 0, n - 1)]), workloads.u3_layer(n, n),
                        as_records([(P, 0, q, 0.3 + q) for q in range(n)]), workloads.u3_layer(n, n + 1),
                        workloads.cx_chain(n), workloads.u3_layer(n, n + 2)])
    for part in (g, g[: n + 2], g[2:]):
        o = Oracle(n)
        o.push(part)
        o.execute()
        for dtype in ("complex64", "complex128"):
            s = ZXH(n, eager_expand_all=True, dtype=dtype)
            s.push_gates(part)
            s.execute()
            assert np.max(np.abs(s.get_state(0).astype(np.complex128) - o.get_state(0))) <= TOL[dtype]
            s.close()


# 2^22 amplitudes are 1024 tiles, on two or three CTAs an SM (296 or 444 on 148 SMs, 148 for the
# complex128 adjoint): every CTA takes several. Against the strided passes, whose own error has
# the same bound.
SEVERAL = 22


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("links,window", [("random", "dense"), ("chain", "chain"), ("back", "linear")])
@pytest.mark.parametrize("gates", ["complex", "real", "h"])
def test_affine_ctas_with_several_tiles(gates, links, window, dtype):
    g = circuit(SEVERAL, links, gates, window, seed=3, layers=2)
    states = []
    for affine in (0, 1):
        s = ZXH(SEVERAL, dtype=dtype)
        s.set_param("affine", affine)
        s.push_gates(g)
        s.execute()
        states.append(s.get_state(0))
        s.close()
    assert np.max(np.abs(states[0].astype(np.complex128) - states[1])) <= 2 * TOL[dtype]


def formed(n, links, window, form):
    circ = ansatz(n, links, window, seed=5, layers=2)
    recs = circ.records(np.random.default_rng(n).uniform(-math.pi, math.pi, circ.nparams))
    rx = (recs["type"] == U3) & (recs["lam"] != 0.0)
    assert rx.any()
    if form == "real":
        recs["theta"][rx] = 0.0
    elif form == "rotations":
        recs["lam"][rx] = recs["phi"][rx] = 0.0
    return recs


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("links,window", [("random", "dense"), ("chain", "linear")])
@pytest.mark.parametrize("form", ["complex", "real", "rotations"])
def test_adjoint_ctas_with_several_tiles(form, links, window, dtype):
    # RX by an angle is complex, by zero real but not taken as a rotation (its generator is X)
    n = SEVERAL
    recs = formed(n, links, window, form)
    terms = ad.tfim_terms(n, h=0.6)
    tol = 2 * 2 * n * (1e-12 if dtype == "complex128" else 1e-6)
    s = ZXH(n, dtype=dtype)
    s.push_gates(recs)
    s.set_param("affine", 0)
    e_ref, g_ref = s.adjoint_gradient(terms)
    s.set_param("affine", 1)
    for every in (0, 20):
        e, g = s.adjoint_gradient(terms, every)
        assert abs(e - e_ref) <= tol and np.max(np.abs(g - g_ref)) <= tol, every
    s.close()


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
def test_batch_tasks_of_several_tiles(dtype):
    # a queue whose levels are one circuit's 1024 tiles, in tasks of 3 or 4: a real queue, and one with
    # complex gates and CX chains
    from zxh_adae_b200.batch import Batch

    n = SEVERAL
    real = workloads.batch_tfim(1, n, n, n, 2)[0][:3]
    c = ansatz(n, "chain", "dense", seed=7, layers=2)
    mixed = (n, c.records(np.random.default_rng(7).uniform(-math.pi, math.pi, c.nparams)), ad.tfim_terms(n))
    tol = 2 * 2 * n * (1e-12 if dtype == "complex128" else 1e-6)
    for which in (real, mixed):
        s = ZXH(n, dtype=dtype)
        s.set_param("affine", 0)
        s.push_gates(which[1])
        e_ref, g_ref = s.adjoint_gradient(which[2])
        s.close()
        b = Batch([which], dtype=dtype)
        for mode in ("persistent", "graph"):
            e, g = b.run(mode)
            assert abs(e[0] - e_ref) <= tol and np.max(np.abs(b.gradients(g)[0] - g_ref)) <= tol, mode
        b.close()


def few_gates(n, gates, before, after, seed):
    # a U3 layer, a window, CX, a few U3, their window, CX, a window in another map
    rng = np.random.default_rng(seed)

    def window(terms):
        recs = [(RZ, 0, int(q), rng.uniform(0, 6)) for q in rng.permutation(n)[:terms]]
        return as_records(recs + [(CP, int(a), int(b), rng.uniform(0, 6)) for a, b in rng.integers(0, n, (terms, 2))])

    u3 = [(U3, 0, int(q), *rng.uniform(0, 6, 3)) for q in rng.permutation(n)[:gates]]
    parts = [workloads.h_all(n), workloads.u3_layer(n, seed), window(before), workloads.cx_chain(n), as_records(u3),
             as_records([(RZ, 0, q, rng.uniform(0, 6)) for _, _, q, *_ in u3]), workloads.cx_chain(n), window(after)]
    return np.concatenate([p for p in parts if len(p)])


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("n", [12, 14, 15, 18])
def test_few_gates_beside_windows(n, dtype):
    # batches that fit one strided pass, beside windows that no tile pass takes: both sides of the
    # lines between one strided pass and a tile pass with a diagonal one
    for gates in (1, 2, 3, 5):
        for before, after in ((1, 0), (0, 1), (3, 2), (n, 0), (0, n)):
            g = few_gates(n, gates, before, after, seed=n + gates)
            o = Oracle(n)
            o.push(g)
            o.execute()
            s = ZXH(n, dtype=dtype)
            s.push_gates(g)
            s.execute()
            assert np.max(np.abs(s.get_state(0).astype(np.complex128) - o.get_state(0))) <= TOL[dtype], (gates, before, after)
            s.close()


@pytest.mark.parametrize("n", [22, 23, 24])
def test_few_complex128_gates_on_large_states(n):
    for gates in (1, 3, 4, 7):
        for before, after in ((0, 0), (2, 2)):
            g = few_gates(n, gates, before, after, seed=n + gates)
            states = []
            for affine in (0, 1):
                s = ZXH(n, dtype="complex128")
                s.set_param("affine", affine)
                s.push_gates(g)
                s.execute()
                states.append(s.get_state(0))
                s.close()
            assert np.max(np.abs(states[0] - states[1])) <= 2 * TOL["complex128"], (gates, before, after)
