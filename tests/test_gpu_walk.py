"""The walk (ps_walk.h): runs whose x / z are shared by all shots but not
known to the host -- runs without reset, and circuits with conditional
Paulis -- against the oracle and against the per-shot kernels, bit for bit.
Sizes at the edges of its words (rows 2n + 1 and qubits n around multiples
of 32 and 64, the largest register it takes and the first it does not), and
tableaux that it must leave to the per-shot kernels."""
import numpy as np
import pytest

from drivers import random_mixed_circuit
from test_gpu_conditional_paulis import conditional_circuit


def _same(st, o):
    gx, gz, gr = st.device_to_host_numpy()
    ox, oz, orr = o.tableau()
    assert np.array_equal(gx, ox) and np.array_equal(gz, oz) and np.array_equal(gr, orr)


def _records(st, cc, nm):
    return [st.record(cc.first_record + k) for k in range(nm)]


def _walked(cc, reset):
    """The plan holds the walk's sign launch (profiling runs the circuit)."""
    return cc.profile(reset=reset)["sign_program"]["launches"] == 1


@pytest.mark.gpu
@pytest.mark.parametrize("n,shots", [(1, 1), (2, 64), (5, 130), (31, 65), (32, 128), (33, 200), (63, 64), (64, 129),
                                     (65, 70), (96, 64)])
def test_runs_without_reset_match_oracle(ps, O, n, shots):
    from plaquette_simulator.circuit import CompiledCircuit
    for circ in (random_mixed_circuit(n, 60 + 4 * n, seed=7 * n, flags=False),
                 conditional_circuit(n, 3 * n, ops=60 + n, flags_only_pauli=True)):
        nm = circ.num_measurements()
        st = ps.CliffordState(n, shots, 3, True)
        cc = CompiledCircuit(circ, st)
        o = O.Oracle(n, shots, seed=3)
        for k in range(3):  # from |0...0> without reset, then twice from what that left
            cc.run()
            table = circ.op_array()
            table[table[:, 0] >= 11, 3] += k * nm  # the oracle numbers its records over the runs
            o.run(table, circ.param_array())
            _same(st, o)
            for m, (res, det) in enumerate(_records(st, cc, nm)):
                ores, odet = o.record(k * nm + m)
                assert np.array_equal(res, ores) and np.array_equal(det, odet), (k, m)
        assert _walked(cc, False)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [127, 128, 223, 449, 511, 512])
@pytest.mark.parametrize("reset", [False, True])
def test_large_registers_equal_per_shot_kernels(ps, n, reset):
    from plaquette_simulator.circuit import CompiledCircuit
    circ = conditional_circuit(n, n, ops=400, flags_only_pauli=True) if n < 400 else \
        random_mixed_circuit(n, 900, seed=n, flags=False)
    if reset and not any(o[0] >= 11 for o in circ.ops):  # keep it off the plan that the host compiles
        rec = next(i for i, o in enumerate(circ.ops) if o[0] in (7, 8))
        q = circ.ops[rec][1]
        circ.ops[rec + 1:rec + 1] = [(g, q, 0, 0) for g in (11, 12, 12, 11)]
    out = []
    for walk in (True, False):
        st = ps.CliffordState(n, 100, 11, True)
        cc = CompiledCircuit(circ, st, shared_xz=walk)
        for _ in range(2):
            cc.run(reset=reset)
        out.append((st.tableau_words(0, st.words()), _records(st, cc, circ.num_measurements()), st.event_counter()))
        assert cc.stats["shared_xz"] == 0 or not reset
        assert _walked(cc, reset) == (walk and n <= 511)
    (ta, ra, ea), (tb, rb, eb) = out
    assert ea == eb and all(np.array_equal(u, v) for u, v in zip(ta, tb))
    assert all(np.array_equal(u, v) for a, b in zip(ra, rb) for u, v in zip(a, b))


@pytest.mark.gpu
@pytest.mark.parametrize("d,rounds,shots", [(3, 4, 200), (5, 3, 4097), (9, 2, 64), (3, 3, 9728), (3, 3, 9729)])
def test_memory_slices_equal_per_shot_kernels(ps, d, rounds, shots):
    """Noisy rounds run on from a memory's tableau, resets ending the slice
    (applied in their phase) and resets before more gates (deferred)."""
    from plaquette_simulator import circuits as C
    from plaquette_simulator.circuit import CompiledCircuit
    full = C.surface_code_memory(d, rounds, p=5e-3)
    circ = C.Circuit(full.num_qubits, full.ops[:-d * d], full.params)
    out = []
    for walk in (True, False):
        st = ps.CliffordState(circ.num_qubits, shots, 21, True)
        cc = CompiledCircuit(circ, st, shared_xz=walk)
        cc.run(reset=True)
        for _ in range(3):
            cc.run(reset=False)
        out.append((st.tableau_words(0, st.words()), _records(st, cc, circ.num_measurements())))
    (ta, ra), (tb, rb) = out
    assert all(np.array_equal(u, v) for u, v in zip(ta, tb))
    assert all(np.array_equal(u, v) for a, b in zip(ra, rb) for u, v in zip(a, b))


@pytest.mark.gpu
@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("why", ["conditional_clifford", "one_shot_differs", "last_padded_word", "loaded", "shared"])
def test_tableaux_left_to_the_per_shot_kernels(ps, why, graph):
    """Shots whose x / z differ, and tableaux that came from the host (and
    one that the walk does take): the same run gives what the per-shot
    kernels give."""
    from plaquette_simulator.circuit import CompiledCircuit
    n, shots = 20, 64 * 5 + 3
    before, circ = random_mixed_circuit(n, 200, seed=5, flags=why == "conditional_clifford"), \
        random_mixed_circuit(n, 300, seed=6, flags=False)
    out = []
    for walk in (True, False):
        st = ps.CliffordState(n, shots, 17, True)
        if why in ("one_shot_differs", "last_padded_word"):
            # one shot's S gate differs: a record that is 1 in that shot alone
            forced = np.zeros(shots, np.uint8)
            forced[70 if why == "one_shot_differs" else shots - 1] = 1
            st.apply_hadamard_gate(3)
            st.measure_qubit(3, forced=forced)
            st.apply_hadamard_gate_with_apply_flag(7, 0)
        else:
            CompiledCircuit(before, st, shared_xz=False).run()
        if why == "loaded":
            st.load_tableau_words(0, *st.tableau_words(0, st.words()))
        cc = CompiledCircuit(circ, st, graph=graph, shared_xz=walk)
        for _ in range(2):
            cc.run()
        out.append((st.tableau_words(0, st.words()), _records(st, cc, circ.num_measurements())))
    (ta, ra), (tb, rb) = out
    assert all(np.array_equal(u, v) for u, v in zip(ta, tb))
    assert all(np.array_equal(u, v) for a, b in zip(ra, rb) for u, v in zip(a, b))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [17, 172, 256, 511])
def test_long_phases_equal_per_shot_kernels(ps, n):
    """Phases of more than 512 measurements after deep random layers (pivot
    rows with Paulis on every column): runs of random ones across the 512 that
    are held at a time, deterministic ones between them, resets among both."""
    from plaquette_simulator import circuits as C
    from plaquette_simulator.circuit import CompiledCircuit
    rng = np.random.default_rng(n)
    circ = C.Circuit(n)
    for _ in range(2):
        for _ in range(6):
            for q in range(n):
                (circ.h, circ.s)[int(rng.integers(2))](q)
            order = rng.permutation(n)
            for a, b in zip(order[0::2], order[1::2]):
                (circ.cx, circ.cz)[int(rng.integers(2))](int(a), int(b))
        for q in rng.integers(0, n, 2 * n + 600):
            (circ.r if rng.integers(4) == 0 else circ.m)(int(q))
    out = []
    for walk in (True, False):
        st = ps.CliffordState(n, 70, 5, True)
        cc = CompiledCircuit(circ, st, shared_xz=walk)
        cc.run()
        assert _walked(cc, False) == walk  # (runs it once more)
        out.append((st.tableau_words(0, st.words()), _records(st, cc, circ.num_measurements())))
    (ta, ra), (tb, rb) = out
    assert all(np.array_equal(u, v) for u, v in zip(ta, tb))
    assert all(np.array_equal(u, v) for a, b in zip(ra, rb) for u, v in zip(a, b))


@pytest.mark.gpu
@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("n,shots", [(20, 512), (20, 513), (20, 3267), (300, 512)])
@pytest.mark.parametrize("odd", [0, 70, -1, None])
def test_check_beside_the_walk(ps, n, shots, odd, graph):
    """Tableaux of more than eight shot-words or 16 MB (and of eight), whose
    one odd shot is in the first word, in another or the last: the walk beside
    the check is dropped for the per-shot kernels, or kept (no odd shot)."""
    from plaquette_simulator.circuit import CompiledCircuit
    circ = random_mixed_circuit(n, 300, seed=6, flags=False)
    out = []
    for walk in (True, False):
        st = ps.CliffordState(n, shots, 17, True)
        forced = np.zeros(shots, np.uint8)
        if odd is not None:
            forced[odd] = 1
        st.apply_hadamard_gate(3)
        st.measure_qubit(3, forced=forced)
        st.apply_hadamard_gate_with_apply_flag(7, 0)
        cc = CompiledCircuit(circ, st, graph=graph, shared_xz=walk)
        for _ in range(2):
            cc.run()
        out.append((st.tableau_words(0, st.words()), _records(st, cc, circ.num_measurements())))
    (ta, ra), (tb, rb) = out
    assert all(np.array_equal(u, v) for u, v in zip(ta, tb))
    assert all(np.array_equal(u, v) for a, b in zip(ra, rb) for u, v in zip(a, b))
