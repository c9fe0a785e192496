"""What the host side launches, without a GPU: the library's objects linked with a CUDA
runtime that only logs (fake_cuda.cpp), the package run on it in a child process."""
import os
import subprocess
import sys
import textwrap
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    objs = sorted((ROOT / "zxh_adae_b200" / "csrc" / "_build").glob("*.o"))
    if not objs:
        pytest.skip("no object files: the library was not built in this tree")
    out = tmp_path_factory.mktemp("fake") / "libfake.so"
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-std=c++17", f"-I{CUDA}/include", "-Wl,-Bsymbolic", "-Wl,--no-undefined",
                    "-o", str(out), str(ROOT / "tests" / "fake_cuda.cpp"), *map(str, objs)], check=True)
    return out


PRELUDE = """
import ctypes, sys
import numpy as np
from zxh_adae_b200 import ZXH, workloads as wl, records as rc
from zxh_adae_b200 import adjoint as ad
from zxh_adae_b200.batch import Batch
from zxh_adae_b200._core import _lib
_lib.fake_take_log.restype = ctypes.c_char_p
_lib.fake_fail_malloc.argtypes = [ctypes.c_long]
def launches():  # (chained, grid, kernel) since the last call
    out = [l.split(" ", 2) for l in _lib.fake_take_log().decode().splitlines()]
    short = lambda k: k.replace("(anonymous namespace)::", "").replace("zxh::", "").replace("void ", "").split("(")[0]
    return [(c == "1", int(g), short(k)) for c, g, k in out]
"""


def run(fake, body):
    env = dict(os.environ, ZXH_B200_LIB=str(fake), PYTHONPATH=str(ROOT))
    r = subprocess.run([sys.executable, "-c", PRELUDE + textwrap.dedent(body)], env=env, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout



def test_batch_tasks_hold_whole_shares_of_a_cta(fake):
    # 256 circuits of 11 qubits: 16 strided items an op (complex64) are one task of two
    # rounds of the CTA's 8 warps, not 13 items and 3
    run(fake, """
    b = Batch([c[:3] for c in wl.batch_tfim(256, 5, 11, 11, 10)])
    ops, tasks, _ = b.stats()
    assert tasks == ops, (ops, tasks)
    """)


def test_batch_kernel_without_tiles(fake):
    # circuits below 12 qubits have no tile passes: their queue runs the form of the kernel
    # that leaves room for two CTAs an SM, but where there is one task an SM in complex128
    run(fake, """
    def form(cnt, n, dtype, threads=256):
        b = Batch([c[:3] for c in wl.batch_tfim(cnt, 5, n, n, 4)], dtype=dtype)
        b.set("threads", threads)
        launches(); b.run("persistent")
        (k,) = [k for _, _, k in launches() if "batch_kernel" in k]
        return k
    for dtype, e in (("complex64", "float2"), ("complex128", "double2")):
        assert form(512, 7, dtype) == f"batch_kernel<{e}, true, 256, false>"
        assert form(4, 7, dtype) == f"batch_kernel<{e}, true, 256, {'true' if e == 'double2' else 'false'}>"
        assert form(2, 12, dtype) == f"batch_kernel<{e}, true, 256, true>"
        for t in (64, 128):
            assert form(2, 12, dtype, t) == f"batch_kernel<{e}, true, {t}, false>"
    """)


def test_batch_after_a_failed_rebuild(fake):
    # another thread count is another pass set: where it cannot be placed, the handle goes
    # back to the one it had, or, where that fails too, refuses to run
    run(fake, """
    b = Batch([c[:3] for c in wl.batch_tfim(2, 5, 12, 12, 4)])
    before = b.stats()[:2]
    for failures in (1, 100):
        _lib.fake_fail_malloc(failures)
        try:
            b.set("threads", 64)
            raise SystemExit("the rebuild did not fail")
        except MemoryError:
            pass
        assert b.get("threads") == 256
        launches()
        try:
            b.run("persistent")
            ran = True
        except RuntimeError:
            ran = False
        assert ran == (failures == 1) and ran == any("batch_kernel" in k for _, _, k in launches())
        assert not ran or b.stats()[:2] == before
    _lib.fake_fail_malloc(0)
    b.set("threads", 256)  # a later setting builds the program again
    b.run("persistent")
    """)


def test_chained_kernels_take_states_without_restrict():
    # a kernel that may start before its predecessor has ended must not promise that nobody
    # else writes its state: loads through such a pointer may move above the wait. Tables that
    # were uploaded before the run, the state a draw only reads, and outputs may be __restrict__
    import re

    seen = 0
    for src in sorted((ROOT / "zxh_adae_b200" / "csrc").glob("*.cu")):
        for m in re.finditer(r"__global__[^;{]*?(\w+)\(((?:const uint8_t|const E|const uint64_t|const double|E )[^{;]*)\)\s*\{", src.read_text()):
            name, params, body = m[1], m[2], src.read_text()[m.end():]
            body = body[: body.index("\n}\n")]
            if "chain_wait()" not in body and "affine_body" not in body:
                continue
            seen += 1
            held = set(re.findall(r"__restrict__ (\w+)", params))
            assert held <= {"blob", "terms", "counts", "offsets", "real_out", "words"} | (
                {"state"} if src.name == "sampler.cu" else set()), (src.name, name, held)
    assert seen >= 8


@pytest.mark.parametrize("n,chained", [(20, True), (21, False), (28, False)])
def test_passes_behind_a_span_pass(fake, n, chained):
    # CX from every other qubit to the last: the RY layer is span passes, then affine tile passes
    # (strided ones with affine = 0); the first of these starts before the span pass has ended
    # on small states only, the others always
    run(fake, f"""
    n = {n}
    g = np.concatenate([wl.h_all(n), rc.as_records([(rc.CX, q, n - 1) for q in range(0, n - 1, 2)]),
                        rc.as_records([(rc.U3, 0, q, 0.3 + q, 0.0, 0.0) for q in range(n)])])
    for affine, kind in ((1, "affine_kernel"), (0, "grow_kernel")):
        s = ZXH(n)
        s.set_param("affine", affine)
        s.push_gates(g)
        launches(); s.execute()
        ks = launches()
        behind = [i for i in range(1, len(ks)) if ks[i][2].startswith(kind) and "span_land" in ks[i - 1][2]]
        assert len(behind) == 1, ks
        assert [c for c, _, _ in ks[1:]] == [i not in behind or {chained} for i in range(1, len(ks))], ks
    """)


def test_few_terms_take_the_gathers(fake):
    # expectations of a few terms: one kernel that gathers; tiles where these are the faster
    run(fake, """
    def kernels(n, dtype, nx, nd):
        s = ZXH(n, dtype=dtype)
        s.push_gates(wl.h_all(n)); s.execute(); launches()
        s.expectation(rc.as_terms([(rc.TERM_X, q, 0, 1.0) for q in range(nx)] + [(rc.TERM_ZZ, i % n, (i + 3) % n, 1.0) for i in range(nd)]))
        return {k.split("<")[0] for _, _, k in launches()}
    gather, tile = {"lambda_kernel"}, {"lambda_tile_kernel"}
    for dtype, most in (("complex64", 4), ("complex128", 12)):
        assert kernels(24, dtype, 0, 1) == kernels(28, dtype, 0, most) == gather
        assert kernels(24, dtype, 0, most + 1) == kernels(24, dtype, 1, 0) == tile
        assert kernels(16, dtype, 2, 12) == kernels(18, dtype, 0, 32) == gather
        assert kernels(16, dtype, 16, 15) == kernels(18, dtype, 3, 0) == tile
    assert kernels(22, "complex128", 1, 4) == gather and kernels(22, "complex64", 1, 4) == tile
    """)


def test_batches_of_few_gates(fake):
    # complex128 batches after CX transport that one strided pass serves faster, and windows
    # that only a strided pass can take (one pass, not a tile pass and a diagonal one)
    run(fake, """
    def kernels(n, dtype, gates, window):
        s = ZXH(n, dtype=dtype)
        g = [wl.h_all(n), wl.cx_chain(n), rc.as_records([(rc.U3, 0, 2 * q + 5, 0.3, 0.2, 0.1) for q in range(gates)])]
        if window: g.append(rc.as_records([(rc.RZ, 0, 2 * q + 5, 0.3, 0.0, 0.0) for q in range(gates)]))
        s.push_gates(np.concatenate(g)); launches(); s.execute()
        return [k.split("<")[0] for _, _, k in launches()][1:]
    tile, strided = ["affine_kernel"], ["grow_kernel"]
    for n, gates, window, want in ((21, 4, 1, tile), (22, 1, 1, strided), (22, 4, 0, tile), (23, 2, 1, tile), (23, 3, 1, strided),
                                   (24, 3, 0, tile), (24, 4, 0, strided), (28, 4, 0, strided), (28, 8, 0, tile)):
        assert kernels(n, "complex128", gates, window) == want, (n, gates, window)
        assert kernels(n, "complex64", gates, window) == tile, (n, gates, window)
    # windows whose selectors flip with several coordinates of the batch's tiles, before and after
    # it: one strided pass on small states, a diagonal pass of their own beside tiles on large ones
    def ks(n, dtype, before, after):
        g = [wl.h_all(n), wl.u3_layer(n, 1)]
        if before: g.append(rc.as_records([(rc.RZ, 0, q, 0.3, 0.0, 0.0) for q in range(n)]))
        g += [wl.cx_chain(n), rc.as_records([(rc.U3, 0, 5, 0.3, 0.2, 0.1)])]
        if after: g += [wl.cx_chain(n), rc.as_records([(rc.RZ, 0, q, 0.3, 0.0, 0.0) for q in range(n)])]
        s = ZXH(n, dtype=dtype); s.push_gates(np.concatenate(g)); launches(); s.execute()
        return [k.split("<")[0] for _, _, k in launches()]
    for dtype in ("complex64", "complex128"):
        for before, after in ((0, 1), (1, 0), (1, 1)):
            small, large = ks(16, dtype, before, after), ks(24, dtype, before, after)
            assert small[-1] == "grow_kernel" and not {"affine_kernel", "diag_kernel", "walsh_kernel"} & set(small), small
            assert "grow_kernel" not in large and "affine_kernel" in large, large
    """)


def test_gradients_on_a_map_that_is_not_onto(fake):
    # CX of a qubit on itself leaves 11 pair deltas of 12 qubits, fewer than a tile needs: the
    # sweep's gates run as strided passes, which the batch kernel has too
    run(fake, """
    n = 12
    rest = [q for q in range(n) if q != 7]
    g = rc.as_records([(rc.H, 0, q) for q in rest] + [(rc.CX, 7, 7)] + [(rc.U3, 0, q, 0.3, 0.0, 0.0) for q in rest])
    t = rc.as_terms([(rc.TERM_Z, 0, 0, 1.0)])
    for dtype in ("complex64", "complex128"):
        Batch([(n, g, t)], dtype=dtype).run("persistent")
        s = ZXH(n, dtype=dtype); s.push_gates(g); launches(); s.adjoint_gradient(t)
        ks = {k.split("<")[0] for _, _, k in launches()}
        assert "grow_kernel" in ks and "adj_pair_kernel" not in ks, ks
    """)


def test_the_affine_tests_run_affine_passes(fake):
    # the circuits of test_gpu_affine.py: tile passes forward and in the sweep, none with affine = 0
    run(fake, """
    from tests.test_gpu_affine import ansatz, circuit, formed, SEVERAL
    def kinds(n, g, affine, grad=False):
        s = ZXH(n); s.set_param("affine", affine); s.push_gates(g); launches()
        s.adjoint_gradient(ad.tfim_terms(n)) if grad else s.execute()
        ks = launches()
        tiles = [grid for _, grid, k in ks if k.startswith("affine_kernel")]
        return tiles, sum(k.startswith("grow_kernel") for _, _, k in ks)
    for n, links, gates in [(12, "chain", "complex"), (12, "random", "real"), (13, "back", "complex"), (14, "chain", "h"),
                            (15, "random", "complex"), (16, "back", "real"), (SEVERAL, "random", "h")]:
        for window in ("none", "linear", "chain", "dense"):
            g = circuit(n, links, gates, window, seed=n)
            tiles, strided = kinds(n, g, 1)
            assert tiles and max(tiles) <= 1 << (n - 12), (n, links, gates, window)
            assert n < SEVERAL or 2 * max(tiles) < 1 << (n - 12)  # several tiles a CTA
            assert kinds(n, g, 0)[0] == [] and kinds(n, g, 0)[1] > 0
    for n, links, window in [(12, "chain", "linear"), (15, "chain", "dense")]:
        g = ansatz(n, links, window, n).records(np.zeros(ansatz(n, links, window, n).nparams))
        assert len(kinds(n, g, 1, True)[0]) > 3 and kinds(n, g, 0, True)[0] == []
    for form, want in (("complex", "0"), ("real", "1"), ("rotations", "2")):
        for dtype in ("complex64", "complex128"):
            s = ZXH(SEVERAL, dtype=dtype); s.push_gates(formed(SEVERAL, "chain", "linear", form)); launches()
            s.adjoint_gradient(ad.tfim_terms(SEVERAL))
            sweep = {k.split(", ")[2][0] for _, _, k in launches() if k.startswith("affine_kernel") and ", true, " in k}
            assert want in sweep and min(sweep) == want, (form, dtype, sweep)
    """)


def test_forms_of_real_gates(fake):
    # after CX transport: rotations, H and their products run with a factored coefficient in both
    # types; a phase of 1e-16 makes a complex128 gate complex
    run(fake, """
    def form(dtype, *gates):
        g = np.concatenate([wl.h_all(13), wl.cx_chain(13)] + [rc.as_records([(*x[:1], 0, q, *x[1:]) for q in range(13)]) for x in gates])
        s = ZXH(13, dtype=dtype); s.push_gates(g); launches(); s.execute()
        return {k.split(", ")[2][0] for _, _, k in launches() if k.startswith("affine")}
    ry, h = (rc.U3, 0.3, 0.0, 0.0), (rc.H,)
    for dtype in ("complex64", "complex128"):
        for gates in ((ry,), (h,), (ry, ry), (h, ry), (ry, h, ry, h, ry), ((rc.U3, np.pi / 2, np.pi, 0.0), ry)):
            assert form(dtype, *gates) == {"2"}, (dtype, gates)
        assert form(dtype, ry, (rc.U3, 0.3, 0.2, 0.1)) == {"0"}
    assert form("complex128", (rc.U3, 0.3, 1e-16, 0.0)) == {"0"} and form("complex64", (rc.U3, 0.3, 1e-16, 0.0)) == {"2"}
    """)


def test_windows_on_a_single_amplitude(fake):
    # no qubit expanded: 8 bytes of complex64 state, below the 16 of a bulk copy
    run(fake, """
    for dtype, n in (("complex64", 0), ("complex64", 1), ("complex128", 0)):
        s = ZXH(4, dtype=dtype)
        s.push_gates(rc.as_records([(rc.X, 0, 1)] + [(rc.H, 0, 2)] * n)); s.execute(); launches()
        assert s.state_view()[1] == n
        s.apply(rc.as_records([(rc.P, 0, 1, 0.3, 0.0, 0.0), (rc.CP, 1, 0, 0.3, 0.0, 0.0)])); s.flush()
        (k,) = [k for _, _, k in launches() if k.startswith("diag_kernel")]
        staged = k.split(", ")[2] == "true"
        assert staged == (dtype == "complex64" and n == 1), k
    """)
