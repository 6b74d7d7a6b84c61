"""The work that programs have this library do, as cases that can be timed and compared.

Every case goes through the public entry points (``CliffordState``,
``CompiledCircuit``, ``Batch``, ``Server``), on synthetic circuits of this
repository: rotated surface-code memories, random Clifford circuits, the
low-space S-state distillation protocol and gate teleportation.  Kinds:

steps     a program that drives the state op by op, as users of the
          reference's binding do: gates, channels, measurements, one call each,
          then the records read back (``what``: the distillation protocol, a
          random Clifford circuit, a noisy surface-code round)
sample    a compiled surface-code memory run from |0...0>; ``to`` says what the
          program takes from it: everything left on the device, the records in
          pinned host memory, or detectors and the observable on the host
feed      a compiled circuit with feed-forward, run from |0...0> (``what``: the
          distillation protocol, whose corrections are conditional H S S H;
          gate teleportation, whose corrections are conditional S gates)
slice     rounds of a memory run on from the state's present tableau (no
          reset), the records to pinned host memory: a long memory kept on the
          device and advanced slice by slice
batch     uneven surface-code jobs in one launch
serve     a burst of jobs through the request loop: submit, wait, records,
          release

All outputs are bits packed in 64-bit words: records, detectors and the state's
tableau (its own device buffers).  They are whole numbers and there is nothing
to say about them in floating point, so there is no ``exact``.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "plaquette-simulator_gb300", "python"))

from plaquette_simulator import CliffordState, _lib, circuits  # noqa: E402
from plaquette_simulator.batch import Batch, Job, Server  # noqa: E402
from plaquette_simulator.circuit import CompiledCircuit  # noqa: E402

NOISE = (1e-4, 1e-3, 5e-3)  # the physical error rates of the benchmark's job mixes


# ------------------------------------------------------------------- cases
def listed():
    return [
        # The smallest program: one five-qubit protocol of the reference's own
        # tests, about 200 calls on a tableau of a few KB.  Latency and launches.
        {"name": "steps_distill_n5_s1000", "kind": "steps", "what": "distill", "n": 5, "shots": 1000},
        # The plain benchmark circuit: 1000 gates on 64 qubits, then every qubit measured.
        {"name": "steps_random_n64_s1024", "kind": "steps", "what": "random", "n": 64, "gates": 1000, "shots": 1024},
        # Op by op with noise and feed-forward resets, where a call moves megabytes: one round at d = 7.
        {"name": "steps_noisy_d7_s20000", "kind": "steps", "what": "round", "d": 7, "p": 1e-3, "shots": 20000},
        # A decoder's smallest sampling call: a few hundred shots of the smallest code, records on the host.
        {"name": "sample_d3_s256", "kind": "sample", "d": 3, "rounds": 3, "p": 1e-3, "shots": 256, "to": "host"},
        # An ordinary one: detectors and the observable of the d = 5 benchmark circuit.
        {"name": "sample_d5_s4096", "kind": "sample", "d": 5, "rounds": 5, "p": 1e-3, "shots": 4096,
         "to": "detectors"},
        # The headline workload, left on the device.
        {"name": "sample_d15_s16384", "kind": "sample", "d": 15, "rounds": 15, "p": 1e-3, "shots": 16384,
         "to": "device"},
        # The largest tableau (19 GB), a ragged shot count.
        {"name": "sample_d21_s50001", "kind": "sample", "d": 21, "rounds": 21, "p": 5e-3, "shots": 50001,
         "to": "device"},
        # Feed-forward of the benchmark: 90 distillation blocks side by side.
        {"name": "feed_distill_b90_s16384", "kind": "feed", "what": "distill", "blocks": 90, "shots": 16384},
        # Feed-forward whose corrections are Clifford gates: teleported S gates, a ragged shot count.
        {"name": "feed_teleport_n60_s4097", "kind": "feed", "what": "teleport", "data": 60, "layers": 4,
         "p": 1e-3, "shots": 4097},
        # A memory advanced on its present tableau: 13 rounds at d = 13.
        {"name": "slice_d13_s10000", "kind": "slice", "d": 13, "rounds": 13, "p": 1e-3, "shots": 10000},
        # Uneven jobs in one launch (d in 3..21, shots log-uniform in 256..65536).
        {"name": "batch_16", "kind": "batch", "jobs": 16, "mix": 12345, "dmax": 21, "smax": 65536},
        # The request loop under a burst of the serving mix, its smaller and ordinary jobs.
        {"name": "serve_24", "kind": "serve", "jobs": 24, "mix": 777, "dmax": 15, "smax": 16384},
    ]


def _log_int(rng, lo, hi):
    """An integer spread over [lo, hi] by its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["steps", "steps", "sample", "sample", "sample", "feed", "feed", "slice", "batch", "serve"])
    if kind == "steps":
        what = rng.choice(["distill", "random", "round"])
        if what == "distill":
            return {"kind": kind, "what": what, "n": 5, "shots": _log_int(rng, 20, 60000)}
        if what == "random":
            return {"kind": kind, "what": what, "n": _log_int(rng, 2, 120), "gates": _log_int(rng, 30, 1000),
                    "shots": _log_int(rng, 20, 8000)}
        return {"kind": kind, "what": what, "d": rng.choice([3, 5, 7]), "p": rng.choice(NOISE),
                "shots": _log_int(rng, 60, 20000)}
    if kind == "sample":
        d = rng.choice(list(range(3, 26, 2)))
        n = 2 * d * d - 1
        most = min(65536, int(16e9 * 8 / (2 * n + 1) ** 2))
        return {"kind": kind, "d": d, "rounds": rng.choice([d, rng.randint(1, d)]), "p": rng.choice(NOISE),
                "shots": _log_int(rng, 64, most),
                "to": rng.choice(["device", "host", "detectors"]) if d <= 15 else "device"}
    if kind == "feed":
        if rng.random() < 0.5:
            return {"kind": kind, "what": "distill", "blocks": _log_int(rng, 1, 90), "shots": _log_int(rng, 64, 16384)}
        return {"kind": kind, "what": "teleport", "data": _log_int(rng, 4, 80), "layers": rng.randint(1, 5),
                "p": rng.choice((0.0,) + NOISE), "shots": _log_int(rng, 64, 6000)}
    if kind == "slice":
        d = rng.choice([3, 5, 7, 9, 11, 13])
        return {"kind": kind, "d": d, "rounds": rng.randint(1, d), "p": rng.choice(NOISE),
                "shots": _log_int(rng, 64, 10000)}
    if kind == "batch":
        return {"kind": kind, "jobs": rng.randint(4, 16), "mix": rng.randrange(1 << 30), "dmax": rng.choice([9, 15, 19]),
                "smax": rng.choice([4096, 16384, 32768])}
    return {"kind": kind, "jobs": rng.randint(4, 24), "mix": rng.randrange(1 << 30), "dmax": rng.choice([7, 11, 15]),
            "smax": rng.choice([1024, 4096, 16384])}


# ---------------------------------------------------------------- circuits
def _teleport(data, layers, p):
    """`layers` layers of H on every third data qubit, a CX brickwork over the
    data and teleported S gates on every second data qubit: the ancilla (H S
    from |0>) takes a CX from its data qubit and is measured, the data qubit
    gets a conditional S and a conditional Z (two conditional S gates) and the
    ancilla is reset.  Data qubits 0..data-1, ancillas after them."""
    half = (data + 1) // 2
    c = circuits.Circuit(data + half)
    rec = 0
    for layer in range(layers):
        for q in range(layer % 3, data, 3):
            c.h(q)
            if p > 0:
                c.depolarize1(q, p)
        for q in range(layer % 2, data - 1, 2):
            c.cx(q, q + 1)
            if p > 0:
                c.depolarize2(q, q + 1, p)
        for i in range(half):
            c.h(data + i)
            c.s(data + i)
            c.cx(2 * i, data + i)
        for i in range(half):
            c.m(data + i)
        for i in range(half):
            c.s_if(2 * i, rec + i)
            c.s_if(2 * i, rec + i)
            c.s_if(2 * i, rec + i)
        rec += half
        for i in range(half):
            c.r(data + i)
        rec += half
    for q in range(data):
        c.m(q)
    return c


def _slice_circuit(d, rounds, p):
    """The rounds of a memory, without its final data measurements."""
    c = circuits.surface_code_memory(d, rounds, p=p)
    return circuits.Circuit(c.num_qubits, c.ops[:-d * d], c.params)


def _feed_circuit(case):
    if case["what"] == "distill":
        return circuits.distillation_blocks(case["blocks"])
    return _teleport(case["data"], case["layers"], case["p"])


def _jobs(case, seed):
    """An uneven mix: d uniform over the odd distances up to dmax (d rounds),
    shots log-uniform, p uniform.  The shapes are the case's, the jobs' random
    draws the seed's."""
    rng = circuits.SplitMix64(case["mix"])
    kept, jobs = {}, []
    for j in range(case["jobs"]):
        d = 3 + 2 * rng.below((case["dmax"] - 1) // 2)
        p = NOISE[rng.below(len(NOISE))]
        lo, hi = math.log(256), math.log(case["smax"])
        shots = int(round(math.exp(lo + rng.uniform() * (hi - lo)) / 64)) * 64
        if (d, p) not in kept:
            kept[(d, p)] = circuits.surface_code_memory(d, d, p=p)
        jobs.append(Job(kept[(d, p)], shots, seed + j, d, p))
    return jobs


def _steps_ops(case, seed):
    """The calls of an op-by-op program: (op code, qubits, record) in order."""
    H, S, X, CX, M = circuits.OP_H, circuits.OP_S, circuits.OP_X, circuits.OP_CX, circuits.OP_M
    P1, P2 = circuits.OP_PAULI1, circuits.OP_PAULI2
    if case["what"] == "distill":
        src = circuits.distillation_blocks(1)
    elif case["what"] == "random":
        src = circuits.random_clifford(case["n"], case["gates"], seed)
    else:
        src = circuits.surface_code_memory(case["d"], 1, p=case["p"])
        src = circuits.Circuit(src.num_qubits, src.ops[:-case["d"] ** 2], src.params)
    out, rec, last = [], 0, {}
    for code, a, b, c in src.ops:
        if code == M:
            out.append((M, a, rec, None))
            last[a] = rec
            rec += 1
        elif code == circuits.OP_R:  # as the reference resets: H S S H where the measured bit is 1
            for g in (circuits.OP_H_IF, circuits.OP_S_IF, circuits.OP_S_IF, circuits.OP_H_IF):
                out.append((g, a, last[a], None))
        elif code in (circuits.OP_H_IF, circuits.OP_S_IF):
            out.append((code, a, c, None))
        elif code == P1:
            out.append((code, a, b, src.params[c:c + 3]))
        elif code == P2:
            out.append((code, a, b, src.params[c:c + 15]))
        else:
            assert code in (H, S, X, CX)
            out.append((code, a, b, None))
    return out, rec, src.num_qubits


# ------------------------------------------------------------------ states
class _Words:
    """Device words of the library as an array that torch can look at."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<i8", "data": (ptr, False), "version": 3}


def _device_words(ptr, shape, owner):
    return torch.as_tensor(_Words(ptr, shape, owner), device="cuda")


def _tableau(handle, n, owner):
    """x, z [2n+1, n, words] and r [2n+1, words] of a state, its own buffers."""
    x, z, r, w = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_uint64()
    _lib.check(_lib.load().ps_get_device_tableau(handle, ctypes.byref(x), ctypes.byref(z), ctypes.byref(r),
                                                 ctypes.byref(w)))
    rows, w = 2 * n + 1, w.value
    return {"x": _device_words(x.value, (rows, n, w), owner), "z": _device_words(z.value, (rows, n, w), owner),
            "r": _device_words(r.value, (rows, w), owner)}


def _device_records(handle, first, count, words, owner):
    """Results and determined flags of a circuit's records on the device."""
    res, det = ctypes.c_void_p(), ctypes.c_void_p()
    _lib.check(_lib.load().ps_get_record_device(handle, first, ctypes.byref(res), ctypes.byref(det)))
    return {"results": _device_words(res.value, (count, words), owner),
            "determined": _device_words(det.value, (count, words), owner)}


class _Compiled:
    """A compiled circuit on its state, as a sampling program keeps it."""

    def __init__(self, circuit, shots, seed, to, reset, first=None):
        self.to, self.reset = to, reset
        self.st = CliffordState(circuit.num_qubits, shots, seed, True)
        if first is not None:  # where the slices start: the tableau that another circuit left
            CompiledCircuit(first, self.st).run(reset=True)
        self.cc = CompiledCircuit(circuit, self.st)
        self.out = _tableau(self.st.handle, circuit.num_qubits, self.st)
        nm, w = circuit.num_measurements(), self.st.words()
        self.records = _device_records(self.st.handle, self.cc.first_record, nm, w, self.st)
        if to == "host":
            self.host = [torch.empty((nm, w), dtype=torch.int64, pin_memory=True) for _ in range(2)]
            self.words = [h.numpy().view(np.uint64) for h in self.host]

    def run(self):
        self.cc.run(reset=self.reset)
        if self.to == "host":
            self.cc.copy_records_words(self.words[0], self.words[1])
            return dict(self.out, results=self.host[0], determined=self.host[1])
        if self.to == "detectors":
            return dict(self.out, **self.records, detectors=self.cc.detectors(self.defs).view(np.int64))
        return dict(self.out, **self.records)


class _Steps:
    """A program that makes one call for each op and reads its records at the end."""

    def __init__(self, case, seed):
        self.ops, self.nrec, n = _steps_ops(case, seed)
        self.st = CliffordState(n, case["shots"], seed, True)
        for _ in range(self.nrec):  # the records that the program measures into
            self.st.measure_qubit(0)
        self.out = _tableau(self.st.handle, n, self.st)

    def run(self):
        st = self.st
        st.reset_clifford_state()
        for code, a, b, p in self.ops:
            if code == circuits.OP_H:
                st.apply_hadamard_gate(a)
            elif code == circuits.OP_S:
                st.apply_phase_gate(a)
            elif code == circuits.OP_CX:
                st.apply_control_not_gate(a, b)
            elif code == circuits.OP_M:
                st.measure_qubit(a, measurement_id=b)
            elif code == circuits.OP_H_IF:
                st.apply_hadamard_gate_with_apply_flag(a, b)
            elif code == circuits.OP_S_IF:
                st.apply_phase_gate_with_apply_flag(a, b)
            elif code == circuits.OP_PAULI1:
                st.pauli_channel_1(a, *p)
            elif code == circuits.OP_PAULI2:
                st.pauli_channel_2(a, b, p)
            else:
                st.apply_pauli_x_gate(a)
        bits = [st.record_bits(k) for k in range(self.nrec)]
        return dict(self.out, results=np.stack([b[0] for b in bits]), determined=np.stack([b[1] for b in bits]))


class _Batch:
    def __init__(self, case, seed):
        self.jobs = _jobs(case, seed)
        self.batch = Batch(self.jobs)
        L = _lib.load()
        self.out = []
        for j, job in enumerate(self.jobs):
            c, s = ctypes.c_void_p(), ctypes.c_void_p()
            _lib.check(L.ps_batch_job(self.batch._h, j, ctypes.byref(c), ctypes.byref(s)))
            t = _tableau(s, job.num_qubits, self.batch)
            nm, w = job.circuit.num_measurements(), t["r"].shape[1]
            rec = _device_records(s, 0, 2 * nm, w, self.batch)["results"]  # results, then determined: one block
            self.out.append(dict(t, records=rec))

    def run(self):
        self.batch.run()
        return self.out


class _Serve:
    def __init__(self, case, seed):
        self.jobs = _jobs(case, seed)
        self.server = Server(hbm_budget_bytes=8 << 30)

    def run(self):
        ids = [self.server.submit(j) for j in self.jobs]
        out = []
        for i in ids:
            res, det = self.server.records(i)
            self.server.release(i)
            out.append([res.view(np.int64), det.view(np.int64)])
        return out


def prepare(case, seed):
    kind = case["kind"]
    seed = seed % (1 << 30)
    if kind == "steps":
        return _Steps(case, seed)
    if kind == "sample":
        s = _Compiled(circuits.surface_code_memory(case["d"], case["rounds"], p=case["p"]), case["shots"], seed,
                      case["to"], True)
        if case["to"] == "detectors":
            dets, obs = circuits.surface_code_detectors(case["d"], case["rounds"])
            s.defs = dets + [obs]
        return s
    if kind == "feed":
        return _Compiled(_feed_circuit(case), case["shots"], seed, "device", True)
    if kind == "slice":
        d, p = case["d"], case["p"]
        return _Compiled(_slice_circuit(d, case["rounds"], p), case["shots"], seed, "host", False,
                         first=_slice_circuit(d, 1, p))
    if kind == "batch":
        return _Batch(case, seed)
    return _Serve(case, seed)


def run(state):
    return state.run()


# -------------------------------------------------------------------- work
def _words(shots):
    return -(-shots // 64)


def _tableau_bytes(n, shots):
    return (2 * n + 1) * (2 * n + 1) * _words(shots) * 8


def _record_bytes(circuit, shots):
    return 2 * circuit.num_measurements() * _words(shots) * 8


def work(case):
    """Bytes of one pass: each input read once, each output written once."""
    kind = case["kind"]
    if kind == "steps":
        # One call at a time: the columns and signs that a gate reads and
        # writes, a measurement's column and record.
        ops, _, n = _steps_ops(case, 1)
        row = _words(case["shots"]) * 8
        per = {circuits.OP_H: 6, circuits.OP_S: 5, circuits.OP_H_IF: 6, circuits.OP_S_IF: 5, circuits.OP_CX: 8,
               circuits.OP_X: 3, circuits.OP_PAULI1: 4, circuits.OP_PAULI2: 6, circuits.OP_M: 1}
        return {"bytes": row * (2 * n + 1) * (sum(per[o[0]] for o in ops) + 2 * n + 1), "flops": 0}
    if kind == "sample":
        c = circuits.surface_code_memory(case["d"], case["rounds"], p=case["p"])
        return {"bytes": _tableau_bytes(c.num_qubits, case["shots"]) + _record_bytes(c, case["shots"]), "flops": 0}
    if kind == "feed":
        c = _feed_circuit(case)
        return {"bytes": _tableau_bytes(c.num_qubits, case["shots"]) + _record_bytes(c, case["shots"]), "flops": 0}
    if kind == "slice":
        c = _slice_circuit(case["d"], case["rounds"], case["p"])
        return {"bytes": 2 * _tableau_bytes(c.num_qubits, case["shots"]) + _record_bytes(c, case["shots"]), "flops": 0}
    total = 0
    for j in _jobs(case, 0):
        total += _record_bytes(j.circuit, j.shots)
        if kind == "batch":
            total += _tableau_bytes(j.num_qubits, j.shots)
    return {"bytes": total, "flops": 0}
