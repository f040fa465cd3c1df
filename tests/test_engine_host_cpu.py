"""The engine's host code on a recording stand-in for the device (cpp/engine_on_fake_device.cpp): what it does when a call
fails in the middle of a flush, and which plan a list of gates takes."""
from __future__ import annotations

import os
import subprocess

import numpy as np
import pytest

import build_ext
import llgpu
import oracle
import test_blockplan_cpu
from conftest import PKG, REPO
from llgpu import OP_CNOT, OP_H, OP_RX, OP_RY, OP_RZ, OP_U2, make_ops


@pytest.fixture(scope="module")
def exe(built):
    out = os.path.join(PKG, "_build", "cpp_tests")
    os.makedirs(out, exist_ok=True)
    inc = ["-I" + os.path.join(REPO, "include"), "-I" + build_ext.CSRC, "-I" + os.path.join(build_ext.CUDA_HOME, "include")]
    path = os.path.join(out, "engine_on_fake_device")
    objs = [os.path.join(build_ext.OBJ, s + ".o") for s in build_ext.CXX_SOURCES]
    # kernels that no scenario reaches stay undefined
    r = subprocess.run(["g++", "-O1", "-std=c++17", "-w", *inc, "-x", "c++", os.path.join(build_ext.CSRC, "llg_engine.cu"),
                        os.path.join(REPO, "tests", "cpp", "engine_on_fake_device.cpp"), "-x", "none", *objs, "-o", path,
                        "-no-pie", "-Wl,--unresolved-symbols=ignore-all"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return path


def run(exe, *args):
    r = subprocess.run([exe, *args], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr


@pytest.mark.parametrize("call", ["weights", "copy", "record", "wait", "block"])
def test_a_failing_call_leaves_nothing_in_flight(exe, call):
    run(exe, call)


def launches(exe, tmp_path, n, precision, ops):
    """(blocks, tile passes, single gates) of a flush."""
    path = str(tmp_path / "ops")
    np.ascontiguousarray(ops, dtype=llgpu.OP_DTYPE).tofile(path)
    r = subprocess.run([exe, "flush", str(n), str(llgpu.PRECISIONS[precision]), path], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
    return tuple(int(x) for x in r.stdout.split())


def random_list(n, count, share, gate, seed=3):
    """`count` gates, `share` of them CNOTs between random qubits, the others gate(rng, qubit)."""
    rng = np.random.default_rng(seed)
    recs = []
    for _ in range(count):
        if rng.random() < share:
            a, b = (int(x) for x in rng.choice(n, size=2, replace=False))
            recs.append((OP_CNOT, a, b))
        else:
            recs.append(gate(rng, int(rng.integers(n))))
    return make_ops(recs)


S = np.sqrt(0.5)
SAME = {
    "h": [lambda rng, q: (OP_H, q), lambda rng, q: (OP_U2, q, 0, 0.0, None, [[S, S], [S, -S]])],
    "ry": [lambda rng, q: (OP_RY, q, 0, 0.8), lambda rng, q: (OP_U2, q, 0, 0.0, None, [[np.cos(0.4), -np.sin(0.4)], [np.sin(0.4), np.cos(0.4)]])],
    "rx": [lambda rng, q: (OP_RX, q, 0, 0.8),
           lambda rng, q: (OP_U2, q, 0, 0.0, None, [[np.cos(0.4), -1j * np.sin(0.4)], [-1j * np.sin(0.4), np.cos(0.4)]])],
    "rz": [lambda rng, q: (OP_RZ, q, 0, 0.8), lambda rng, q: (OP_U2, q, 0, 0.0, None, np.diag([np.exp(-0.4j), np.exp(0.4j)]))],
}


@pytest.mark.parametrize("precision", ["complex128", "df64"])
@pytest.mark.parametrize("n", [6, 8, 9, 10, 11, 12, 14])
@pytest.mark.parametrize("gate", list(SAME))
def test_a_gate_by_name_or_by_its_matrix(exe, tmp_path, gate, n, precision):
    # the plan follows what the gates cost, not what they are called
    for count, share in ((1000, 0.5), (1000, 0.25), (200, 0.25)):
        named, matrix = (launches(exe, tmp_path, n, precision, random_list(n, count, share, g)) for g in SAME[gate])
        assert (named[0] > 0) == (matrix[0] > 0)


# where one form takes at most 0.8 of the other's time on the GPU, in both formats alike
@pytest.mark.parametrize("precision", ["complex128", "df64"])
@pytest.mark.parametrize("n", [6, 8, 10, 12, 16, 20])
def test_the_faster_form(exe, tmp_path, n, precision):
    layers = make_ops([r for layer in range(20) for r in
                       [(k, q, 0, 0.3 + 0.1 * q + layer) for q in range(n) for k in (OP_RX, OP_RY, OP_RZ)] +
                       [(OP_CNOT, q, q + 1) for q in range(layer % 2, n - 1, 2)]])
    assert launches(exe, tmp_path, n, precision, layers)[0] > 0
    short = make_ops([(OP_RY, q, 0, 0.4) for q in range(n)])
    if n <= 10:
        assert launches(exe, tmp_path, n, precision, short)[0] == 0
        cnots = random_list(n, 1000, 1.0, None)
        assert launches(exe, tmp_path, n, precision, cnots)[0] == 0


def changing(n, layers, cnots, seed=1):
    """Layers of rotations and CNOTs, then CNOTs between random qubits alone."""
    rng = np.random.default_rng(seed)
    recs = []
    for layer in range(layers):
        for q in range(n):
            recs += [(k, q, 0, float(rng.uniform(0.2, 3))) for k in (OP_RX, OP_RY, OP_RZ)]
        recs += [(OP_CNOT, q, q + 1) for q in range(layer % 2, n - 1, 2)]
    return make_ops(recs + [(OP_CNOT, *(int(x) for x in rng.choice(n, size=2, replace=False))) for _ in range(cnots)])


@pytest.mark.parametrize("n,precision", [(10, "complex128"), (14, "df64"), (24, "df64")])
def test_a_list_that_changes_on_its_way(exe, tmp_path, n, precision):
    # the rotations as blocks, the CNOTs (5 to a block) as tile passes
    layers, cnots = (120, 400) if n < 24 else (30, 300)
    alone = launches(exe, tmp_path, n, precision, changing(n, layers, 0))
    assert alone[0] > 16 and alone[1] == 0
    both = launches(exe, tmp_path, n, precision, changing(n, layers, cnots))
    assert alone[0] - 16 <= both[0] <= alone[0] + 16 and both[1] > 0


@pytest.mark.parametrize("blocks", [0, 1, 7, 10000])
@pytest.mark.parametrize("n", [6, 7, 9, 11, 13])
def test_a_plan_and_what_is_left_of_the_list(exe, tmp_path, n, blocks):
    # registers of few qubits, whose blocks hold most of them; the plan's gates first, then the others in their order
    for seed in range(4):
        ops = test_blockplan_cpu._random_ops(max(n, 9), 300, 100 * n + seed)
        ops = ops[(ops["q0"] < n) & (ops["q1"] < n) & (ops["mask"] >> np.uint64(n) == 0)][:150]
        np.ascontiguousarray(ops, dtype=llgpu.OP_DTYPE).tofile(tmp_path / "ops")
        run(exe, "plan", str(n), str(blocks), str(tmp_path / "ops"), str(tmp_path / "out"))
        raw = (tmp_path / "out").read_bytes()
        nsteps, ngates, nleft = np.frombuffer(raw, np.int64, 3)
        steps = np.frombuffer(raw, llgpu.BLOCK_STEP_DTYPE, nsteps, 24)
        at = 24 + steps.nbytes
        gates = np.frombuffer(raw, llgpu.BLOCK_GATE_DTYPE, ngates, at)
        left = np.frombuffer(raw, llgpu.OP_DTYPE, nleft, at + gates.nbytes)
        assert steps["is_block"].sum() <= blocks and (blocks < 10000 or nleft == 0)
        psi = np.zeros(1 << n, dtype=complex)
        psi[0] = 1.0
        for s in steps:
            qubits = list(s["q"]) if s["is_block"] else list(range(n))
            for g in gates[s["gate_begin"]:s["gate_begin"] + s["ngates"]]:
                psi = test_blockplan_cpu._apply(psi, n, g, qubits)
        assert np.max(np.abs(oracle.run_ops(n, left, psi) - oracle.run_ops(n, ops))) <= 1e-12


@pytest.mark.parametrize("more", [0, 1, 2, 3, 5, 8, 9, 40])
def test_little_device_memory(exe, more):
    run(exe, "room", str(more))


@pytest.mark.parametrize("n,precision", [(12, "complex128"), (16, "df64")])
def test_small_angles(exe, tmp_path, n, precision):
    # angles of 0.01 are in reach of a block, angles of 0.001 are not, beside qubits with strong ones they are again
    def layers(angle, strong=False):
        recs = []
        for layer in range(8):
            recs += [(OP_RY, q, 0, 1.1 if strong and q % 2 else angle) for q in range(n)] + [(OP_RZ, q, 0, 0.4) for q in range(n)]
            recs += [(OP_CNOT, q, (q + 1) % n) for q in range(n)]
        return make_ops(recs)
    assert launches(exe, tmp_path, n, precision, layers(0.01))[0] > 0
    assert launches(exe, tmp_path, n, precision, layers(0.001))[0] == 0
    assert launches(exe, tmp_path, n, precision, layers(0.001, True))[0] > 0
