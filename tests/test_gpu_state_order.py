"""The state in virtual order (zxh_get_state, zxh_get_state_device) around the tile sizes
of its pass: runs of 2^6 (complex64) / 2^5 (complex128) amplitudes, tiles of up to 2^12 /
2^11, the identity map, CX / X transport, unexpanded qubits and dependent columns."""
import numpy as np
import pytest

from oracle.bridge import Oracle
from zxh_adae_b200 import ZXH, workloads
from zxh_adae_b200.records import CX, H, U3, X, as_records

pytestmark = pytest.mark.gpu

TOL = {"complex64": 1e-6, "complex128": 1e-12}  # the parity suite's bounds on amplitudes


def circuit(n, kind, seed=3):
    rng = np.random.default_rng(seed + n)
    if kind == "lazy":  # a third of the qubits touched by H, CX onto untouched ones
        touched = [int(q) for q in rng.permutation(n)[: max(1, n // 3)]]
        recs = [(H, 0, q) for q in touched]
        recs += [(U3, 0, q, *rng.uniform(0, 6, 3)) for q in touched]
        recs += [(CX, q, int(t)) for q in touched for t in rng.permutation(n)[:3] if int(t) != q]
        return as_records(recs)
    recs = [workloads.h_all(n), workloads.u3_layer(n, seed)]
    if kind == "chain" and n > 1:
        recs.append(workloads.cx_chain(n))
    if kind == "dense" and n > 1:
        pairs = rng.integers(0, n, (6 * n, 2))
        recs.append(as_records([(CX, int(a), int(b)) for a, b in pairs if a != b] + [(X, 0, int(q)) for q in pairs[:5, 0]]))
    return np.concatenate(recs)


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("n", [1, 2, 5, 6, 7, 8, 10, 11, 12, 13, 17])
@pytest.mark.parametrize("kind", ["plain", "chain", "dense", "lazy"])
def test_state_order_against_oracle(n, kind, dtype):
    gates = circuit(n, kind)
    o = Oracle(n)
    o.push(gates)
    o.execute()
    s = ZXH(n, dtype=dtype)
    s.push_gates(gates)
    s.execute()
    for order in (0, 1):
        err = np.max(np.abs(s.get_state(order).astype(np.complex128) - o.get_state(order)))
        assert err <= TOL[dtype], (order, err)
    rev = np.array([int(format(i, f"0{n}b")[::-1], 2) for i in range(1 << n)])
    assert np.array_equal(s.get_state(0)[rev], s.get_state(1))  # the same bytes, moved
    s.close()


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
def test_state_order_dependent_columns(dtype):
    # CX with control = target clears the qubit's row: two real addresses share an output
    n = 7
    gates = np.concatenate([workloads.h_all(n), as_records([(CX, 2, 2)])])
    s = ZXH(n, dtype=dtype)
    s.push_gates(gates)
    s.execute()
    got = s.get_state(1)
    amp = 2.0 ** (-n / 2)
    want = np.where((np.arange(1 << n) >> 2) & 1, 0.0, amp)
    live = np.abs(got) > 0
    assert np.array_equal(live, want > 0)
    assert np.max(np.abs(got[live] - amp)) <= TOL[dtype]
    s.close()
