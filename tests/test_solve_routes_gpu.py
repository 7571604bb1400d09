"""Which form a demag solve takes (one launch, separate kernels in a loop graph, host polling) and what it may not
change: the potential, the calls that are taken, and what a handle keeps from one call for the next."""

import ctypes as C
import json
import os
import subprocess
import sys
import threading
from pathlib import Path

import numpy as np
import pytest
import torch

from mumag_matrixfree2_gb300 import _abi, fem_utils
from mumag_matrixfree2_gb300 import synthetic as syn
from mumag_matrixfree2_gb300.cuda_backend import MinimizerParams

pytestmark = pytest.mark.gpu


def _problem(workload="cube8_h2_air24", precision="fp64"):
    knt, ijk = syn.box_mesh(syn.WORKLOADS[workload])
    A, K1, Js, k, _ = syn.reduced_materials([syn.Material(), syn.AIR])
    s = fem_utils.prepare(knt, ijk, A, K1, Js, k)
    prob = fem_utils.make_problem(s)
    if precision != "fp64":
        prob.set_precision(precision)
    prob.build_poisson(1e-12, "amgcl")
    return s, prob


@pytest.mark.parametrize("precision", ["fp64", "fp32_precond", "mixed"])
@pytest.mark.parametrize("offset", [0, 1, 4, 8])
def test_potential_at_any_address(cuda_ok, precision, offset):
    """A potential that no kernel can read as doubles where it lies is copied, as a copy takes any address."""
    s, prob = _problem(precision=precision)
    m = torch.from_numpy(syn.initial_state(s.N, seed=3, amplitude=0.3)).cuda()
    x0 = torch.from_numpy(0.01 * np.random.default_rng(4).standard_normal(s.N) * s.boundary_mask).cuda()
    ref, it0, rr0, _ = prob.solve_u(m, x0.clone(), 1e-10)
    buf = torch.zeros(8 * s.N + 16, dtype=torch.uint8, device="cuda")
    buf[offset:offset + 8 * s.N].copy_(x0.view(torch.uint8))
    torch.cuda.synchronize()
    it, rr = C.c_int(), C.c_double()
    rc = _abi.lib().mm_solve_u_dev(prob.h, C.c_void_p(m.data_ptr()), C.c_void_p(buf.data_ptr() + offset), 1e-10, 2000,
                                   C.byref(it), C.byref(rr))
    assert (rc, it.value, rr.value) == (0, it0, rr0)
    U = np.frombuffer(buf[offset:offset + 8 * s.N].cpu().numpy().tobytes(), np.float64)
    assert np.array_equal(U, ref.cpu().numpy())
    assert not buf[:offset].any() and not buf[offset + 8 * s.N:].any()


def _launches(prob, *args):
    n = prob.launch_count()
    out = prob.solve_u(*args)
    return out, prob.launch_count() - n


@pytest.mark.parametrize("precision", ["fp64", "fp32_precond", "mixed"])
@pytest.mark.parametrize("workload", ["cube8_h2_air24", "cube16_h2_air48", "cube40_h2_air200"])
def test_every_route_of_a_solve_gives_the_same_bits(cuda_ok, workload, precision):
    """One launch on every SM, on a third of them, on one cluster's number, on fewer blocks than a cluster has; the loop
    graph of separate kernels; and the host's polling."""
    s, prob = _problem(workload, precision)
    m = syn.initial_state(s.N, seed=12, amplitude=0.3)
    x0 = 0.01 * np.random.default_rng(13).standard_normal(s.N) * s.boundary_mask
    prob.set_option("graph", 0)
    ref, polled = _launches(prob, m, x0, 1e-10)
    prob.set_option("graph", 1)
    for blocks in (-1, 10**6, 50, 17, 16, 15, 8, 0):
        prob.set_option("one_launch", blocks)
        assert prob.get_option("one_launch") == blocks
        out, n = _launches(prob, m, x0, 1e-10)
        assert out[1:] == ref[1:] and np.array_equal(out[0], ref[0]), blocks
        assert (n < polled // 2) == (blocks != 0), (blocks, n, polled)
    with pytest.raises(_abi.MMError):
        prob.set_option("one_launch", -2)


@pytest.mark.parametrize("precision", ["fp64", "fp32_precond", "mixed"])
def test_loop_graph_holds_the_coarse_cycle(cuda_ok, precision):
    """The separate kernels' loop graph with levels 1 .. 3 in one cooperative launch, against the one launch: the same
    bits, fewer launches than with five, and the graph did hold it."""
    s, prob = _problem("cube80_h1.6_air200", precision)
    m = syn.initial_state(s.N, seed=14, amplitude=0.1)
    ref, one = _launches(prob, m, np.zeros(s.N), 1e-10)
    prob.set_option("one_launch", 0)
    out, n = [], []
    for cc in (0, 3):
        prob.set_option("coarse_cycle", cc)
        r, k = _launches(prob, m, np.zeros(s.N), 1e-10)
        assert prob.get_option("coarse_cycle") == cc
        assert r[1:] == ref[1:] and np.array_equal(r[0], ref[0]), cc
        n.append(k)
    assert one < n[1] < n[0]


@pytest.mark.parametrize("method,precision,cpp", [("pcohen_hs", "fp64", False), ("pcohen", "fp64", True),
                                                  ("pcohen_hs", "fp32_precond", False)])
def test_minimizer_graph_with_every_form_of_its_demag_solve(cuda_ok, method, precision, cpp):
    """The minimizer's graph with its demag solve as one launch, on a third of the SMs and as a nested loop of separate
    kernels, against its host loop: the same state, counts and energies."""
    s, prob = _problem("cube16_h2_air48", precision)
    m0 = syn.initial_state(s.N, seed=15, amplitude=0.2)
    mp = MinimizerParams(method=method, max_iter=40, tau_f=1e-8, eps_a=1e-6, cg_tol=1e-10, cpp_semantics=cpp)
    runs = {}
    for blocks, graph in ((-1, 1), (50, 1), (0, 1), (-1, 1), (-1, 0), (0, 0)):
        prob.set_option("one_launch", blocks)
        prob.set_option("min_graph", graph)
        m, U, info = prob.minimize(np.array([0.0, 0.0, -0.3]), m0, np.zeros(s.N), mp)
        assert info["device_loop"] == bool(graph)
        runs[blocks, graph] = (m, U, [info[k] for k in ("iters", "evals", "preco_iters", "demag_iters", "E", "gnorm")])
    m, U, counts = runs.pop((0, 0))
    assert counts[0] > 2
    for route, r in runs.items():
        assert r[2] == counts and np.array_equal(r[0], m) and np.array_equal(r[1], U), route


def test_a_solve_beside_another_streams_work(cuda_ok):
    """Kernels of another stream before, beside and after solves of either form: both give what they give alone."""
    s, prob = _problem("cube40_h2_air200")
    m = syn.initial_state(s.N, seed=16, amplitude=0.3)
    ref = prob.solve_u(m, np.zeros(s.N), 1e-10)[0]
    a = torch.randn(1024, 1024, device="cuda", dtype=torch.float64)
    want = a
    for _ in range(8):
        want = torch.sin(want) + a
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    for blocks in (-1, 50, 0):
        prob.set_option("one_launch", blocks)
        with torch.cuda.stream(side):
            got = a
            for _ in range(8):
                got = torch.sin(got) + a
        U = prob.solve_u(m, np.zeros(s.N), 1e-10)[0]
        side.synchronize()
        assert np.array_equal(U, ref) and torch.equal(got, want)


def test_autotuner_does_not_depend_on_the_last_call(cuda_ok):
    """A solve beside three other problems' runs as separate kernels; the autotuner of that handle, called alone later, times
    the one launch all the same: about as many launches as on a handle that never had company."""
    s, prob = _problem("cube16_h2_air48")
    m = syn.initial_state(s.N, seed=17, amplitude=0.3)
    others = [_problem("cube8_h2_air24") for _ in range(3)]
    zero = np.zeros(s.N)
    alone = _launches(prob, m, zero, 1e-10)[1]
    stop = threading.Event()
    gate = threading.Barrier(4)

    def work(so, po):
        mo = syn.initial_state(so.N, seed=18, amplitude=0.3)
        gate.wait()
        while not stop.is_set():
            po.minimize(np.array([0.0, 0.0, -0.3]), mo, np.zeros(so.N), MinimizerParams(max_iter=40, tau_f=1e-12))

    threads = [threading.Thread(target=work, args=o) for o in others]
    for t in threads:
        t.start()
    gate.wait()
    beside = []
    for _ in range(2000):
        beside.append(_launches(prob, m, zero, 1e-10)[1])
        if beside[-1] > 4 * alone:
            break
    stop.set()
    for t in threads:
        t.join()
    assert beside[-1] > 4 * alone  # the handle's last solve ran as separate kernels
    counts = []
    for p in (prob, _problem("cube16_h2_air48")[1]):
        n = p.launch_count()
        p.autotune(reps=3)
        counts.append(p.launch_count() - n)
    assert counts[0] <= 1.25 * counts[1], counts


def _pool_bytes():
    """Bytes in use of the device's default memory pool, which holds every problem's buffers."""
    cu = C.CDLL("libcuda.so.1")
    pool, used = C.c_void_p(), C.c_uint64()
    torch.cuda.synchronize()
    assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), torch.cuda.current_device()) == 0
    assert cu.cuMemPoolGetAttribute(pool, 7, C.byref(used)) == 0  # CU_MEMPOOL_ATTR_USED_MEM_CURRENT
    return used.value


@pytest.mark.parametrize("precision", ["fp64", "fp32_precond", "mixed"])
def test_autotuner_keeps_one_layout_of_an_operator(cuda_ok, precision):
    """Neither autotuning nor setting the lanes leaves a copy of an operator for every number of lanes that was tried:
    at most a second one where the lanes that are kept need more padding."""
    s, prob = _problem("cube40_h2_air200", precision)
    m = syn.initial_state(s.N, seed=19, amplitude=0.3)
    ref = prob.solve_u(m, np.zeros(s.N), 1e-10)
    before = _pool_bytes()
    for lanes in (2, 4, 8, 16, 32, 8):
        prob.set_option("csr_lanes", lanes)
        prob.solve_u(m, np.zeros(s.N), 1e-10)
    entry = {"fp64": 12, "fp32": 8}
    rep = prob.autotune(reps=2)
    once = sum(o["nnz"] * entry[o["precision"]] for o in rep["operators"])
    assert _pool_bytes() - before <= 2 * once
    for _ in range(2):
        prob.autotune(reps=1)
    assert _pool_bytes() - before <= 2 * once
    for restrict, coarse in ((0, 0), (3, 3)):  # operators laid out anew where they come into use again
        prob.set_option("fuse_restrict", restrict)
        prob.set_option("coarse_fuse", coarse)
        out, n = _launches(prob, m, np.zeros(s.N), 1e-10)
        assert n < 8 * max(1, prob.last_refinements()) and abs(out[1] - ref[1]) <= (2 if precision == "mixed" else 1)
        assert np.abs(out[0] - ref[0]).max() <= 1e-7 * np.abs(ref[0]).max()


# a runtime whose occupancy queries say that the device holds no cluster of 16, or no block, of a kernel with 200 KB
NO_ROOM = """
#include <dlfcn.h>
#include <stddef.h>
#include <stdlib.h>
int cudaOccupancyMaxActiveClusters(int* n, const void* f, const void* cfg) { *n = 0; return 0; }
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int t, size_t smem, unsigned fl) {
  void* rt = dlopen("libcudart.so.13", RTLD_NOLOAD | RTLD_LAZY);
  int (*real)(int*, const void*, int, size_t, unsigned) =
      rt ? dlsym(rt, "cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags") : NULL;
  int rc = real ? real(n, f, t, smem, fl) : 1;
  if (getenv("NO_BLOCKS") && smem == 200 * 1024) *n = 0;
  return rc;
}
"""


def _solve_small(precision):
    s, prob = _problem(precision=precision)
    (U, it, rr, rc), n = _launches(prob, syn.initial_state(s.N, seed=20, amplitude=0.3), np.zeros(s.N), 1e-10)
    return {"U": [float(u).hex() for u in U], "it": it, "rr": rr.hex(), "rc": rc, "launches": n}


@pytest.mark.parametrize("precision", ["fp64", "fp32_precond", "mixed"])
def test_a_device_without_room_for_the_launch(cuda_ok, precision, tmp_path):
    """A device that cannot place the cluster runs a grid of blocks, one that cannot place a block separate kernels: the
    same potential, and no failed launch.  What the runtime says is faked in a process of its own."""
    (tmp_path / "fake.c").write_text(NO_ROOM)
    fake = tmp_path / "fake.so"
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(fake), str(tmp_path / "fake.c"), "-ldl"], check=True)
    ref = _solve_small(precision)
    root = Path(__file__).resolve().parents[1]
    code = f"import json; from tests.test_solve_routes_gpu import _solve_small; print(json.dumps(_solve_small({precision!r})))"
    for env in ({}, {"NO_BLOCKS": "1"}):
        r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300,
                           env={**os.environ, "LD_PRELOAD": str(fake), **env})
        assert r.returncode == 0, r.stderr[-2000:]
        got = json.loads(r.stdout.strip().splitlines()[-1])
        n, n0 = got.pop("launches"), ref["launches"]
        assert got == {k: v for k, v in ref.items() if k != "launches"}
        assert (n > 2 * n0) if env else (n == n0), (n, n0)


@pytest.mark.parametrize("precision", ["fp64", "fp32_precond"])
def test_few_blocks_for_many_rows(cuda_ok, precision):
    """357,911 rows: eight blocks hold their 88 partials of 2 KB each in shared memory; four cannot, and the solve takes the
    separate kernels."""
    s, prob = _problem("cube80_h1.6_air200", precision)
    m = syn.initial_state(s.N, seed=21, amplitude=0.3)
    ref, one = _launches(prob, m, np.zeros(s.N), 1e-10)
    for blocks in (8, 4):
        prob.set_option("one_launch", blocks)
        out, n = _launches(prob, m, np.zeros(s.N), 1e-10)
        assert out[1:] == ref[1:] and np.array_equal(out[0], ref[0]), blocks
        assert (n == one) == (blocks == 8)


@pytest.mark.parametrize("precision", ["fp64", "fp32_precond"])
def test_dealt_out_rows_against_compressed_rows(cuda_ok, precision):
    """The separate kernels read rows dealt out over their lanes; the coarse cycle reads the same operators' compressed rows
    (level 1, folded and not): for every number of lanes the same solve bit for bit, in the loop graph and polled."""
    s, prob = _problem("cube80_h1.6_air200", precision)
    m = syn.initial_state(s.N, seed=22, amplitude=0.3)
    prob.set_option("one_launch", 0)
    for lanes in (2, 4, 8, 16, 32):
        prob.set_option("csr_lanes", lanes)
        ref = None
        for graph, cycle in ((1, 0), (1, 3), (0, 3), (0, 0)):
            prob.set_option("graph", graph)
            prob.set_option("coarse_cycle", cycle)
            out = prob.solve_u(m, np.zeros(s.N), 1e-10)
            assert prob.get_option("coarse_cycle") == cycle and out[3] == 0
            ref = ref or out
            assert out[1:] == ref[1:] and np.array_equal(out[0], ref[0]), (lanes, graph, cycle)


@pytest.mark.parametrize("workload, shares", [("cube40_h2_air200", True), ("cube80_h1.6_air200", False)])
def test_a_solve_beside_another_problem(cuda_ok, workload, shares):
    """Beside one other problem in flight a solve of 59,319 rows takes its share of the SMs in one launch, and one of
    357,911 rows separate kernels, as it always did; the potential has the same bits."""
    s, prob = _problem(workload)
    m = syn.initial_state(s.N, seed=23, amplitude=0.3)
    ref, alone = _launches(prob, m, np.zeros(s.N), 1e-10)
    so, po = _problem("cube16_h2_air48")
    mo = syn.initial_state(so.N, seed=24, amplitude=0.3)
    stop, gate = threading.Event(), threading.Barrier(2)

    def work():
        gate.wait()
        while not stop.is_set():
            po.minimize(np.array([0.0, 0.0, -0.3]), mo, np.zeros(so.N), MinimizerParams(max_iter=200, tau_f=1e-14))

    t = threading.Thread(target=work)
    t.start()
    gate.wait()
    counts = set()
    for _ in range(40):
        out, n = _launches(prob, m, np.zeros(s.N), 1e-10)
        counts.add(n)
        assert out[1:] == ref[1:] and np.array_equal(out[0], ref[0])
    stop.set()
    t.join()
    assert (max(counts) == alone) == shares, (counts, alone)


@pytest.mark.parametrize("precision", ["fp64", "fp32_precond", "mixed"])
def test_threads_solve_and_minimize_with_the_bits_of_one(cuda_ok, precision):
    """Five threads at once, each solving and minimizing on a handle of its own: how many others are in flight changes the
    form of a solve and of the minimizer's graph, not what they return."""
    n = 5
    handles = [_problem("cube16_h2_air48", precision) for _ in range(n)]
    mp = MinimizerParams(max_iter=6, tau_f=1e-10, eps_a=1e-8, cg_tol=1e-10)

    def both(k):
        s, prob = handles[k]
        m = syn.initial_state(s.N, seed=30 + k, amplitude=0.2)
        U = prob.solve_u(m, np.zeros(s.N), 1e-10)
        return (U[0], *U[1:3], *prob.minimize(np.array([0.0, 0.0, -0.3]), m, np.zeros(s.N), mp)[:2])

    ref = [both(k) for k in range(n)]
    bad, gate = [], threading.Barrier(n)

    def work(k):
        gate.wait()
        for _ in range(4):
            if not all(np.array_equal(a, b) for a, b in zip(both(k), ref[k])):
                bad.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(n)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
