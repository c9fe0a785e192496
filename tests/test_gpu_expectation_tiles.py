"""Expectation values around the tile size of their pass (2^12 amplitudes): below it, at
it and above, the identity map, CX chains, dense maps and unexpanded qubits, repeated and
many terms, against the oracle's state.

Bound: the state's own error (1e-12, 1e-6 per amplitude in the parity suite; the energies
of complex64 states are off by their amplitudes' relative error, about 1e-6 of the sum of
the coefficients) times the sum of |coefficients|."""
import numpy as np
import pytest

from oracle import observables as ob
from zxh_adae_b200 import ZXH, workloads
from zxh_adae_b200.records import CX, H, TERM_X, TERM_Z, TERM_ZZ, U3, X, as_records, as_terms

pytestmark = pytest.mark.gpu

TOL = {"complex64": 2e-6, "complex128": 1e-12}


def circuit(n, kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "lazy":  # two thirds of the qubits expanded
        touched = [int(q) for q in rng.permutation(n)[: 2 * n // 3]]
        recs = [(U3, 0, q, *rng.uniform(0, 6, 3)) for q in touched]
        return as_records(recs + [(CX, touched[0], touched[1])])
    recs = [workloads.h_all(n), workloads.u3_layer(n, seed)]
    if kind == "chain":
        recs.append(workloads.cx_chain(n))
    if kind == "dense":
        pairs = rng.integers(0, n, (5 * n, 2))
        recs.append(as_records([(CX, int(a), int(b)) for a, b in pairs if a != b] + [(X, 0, 3), (X, 0, n - 1)]))
    return np.concatenate(recs)


def observable(n, which, seed):
    rng = np.random.default_rng(seed)
    if which == "chain":
        return as_terms([(TERM_ZZ, i, i + 1, 1.0) for i in range(n - 1)] + [(TERM_X, i, 0, 0.7) for i in range(n)])
    if which == "repeated":  # the same flips and selectors several times, zero coefficients
        return as_terms([(TERM_X, q % 3, 0, 0.3 + q) for q in range(9)] + [(TERM_Z, 1, 0, 0.5)] * 3 +
                        [(TERM_ZZ, 2, 2, 0.25), (TERM_X, n - 1, 0, 0.0)])
    if which == "empty":
        return as_terms([])
    kinds = rng.integers(1, 4, 256)  # as many as a call takes
    qs = rng.integers(0, n, (256, 2))
    return as_terms([(int(k), int(a), int(b), float(c)) for k, (a, b), c in zip(kinds, qs, rng.uniform(-1, 1, 256))])


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("which", ["chain", "repeated", "many", "empty"])
@pytest.mark.parametrize("n,kind", [(11, "chain"), (12, "plain"), (12, "dense"), (13, "chain"), (16, "dense"),
                                    (17, "plain"), (18, "lazy"), (20, "lazy")])
def test_expectation_tiles(n, kind, which, dtype):
    gates, terms = circuit(n, kind, n), observable(n, which, n)
    s = ZXH(n, dtype=dtype)
    s.push_gates(gates)
    s.execute()
    scale = max(1.0, float(np.sum(np.abs(terms["coef"]))))
    assert abs(s.expectation(terms) - ob.oracle_energy(n, gates, terms)) <= TOL[dtype] * scale
    s.close()


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("n", [12, 18, 19])
def test_expectation_of_few_terms(n, dtype):
    # both sides of the lines between one gather per X term and tiles: Z terms alone, one, two
    # and three X terms, up to and above the counts that take the gathers
    gates = circuit(n, "chain", n)
    rng = np.random.default_rng(n)
    s = ZXH(n, dtype=dtype)
    s.push_gates(gates)
    s.execute()
    for nx, nd in [(0, 1), (0, 4), (0, 5), (0, 12), (0, 13), (0, 33), (1, 0), (1, 8), (1, 9), (1, 33), (2, 12), (2, 13), (3, 0)]:
        terms = as_terms([(TERM_X, int(q), 0, 0.4) for q in rng.permutation(n)[:nx]] +
                         [(TERM_ZZ, int(a), int(b), 0.3) for a, b in rng.integers(0, n, (nd, 2))])
        scale = max(1.0, float(np.sum(np.abs(terms["coef"]))))
        assert abs(s.expectation(terms) - ob.oracle_energy(n, gates, terms)) <= TOL[dtype] * scale, (nx, nd)
    s.close()
