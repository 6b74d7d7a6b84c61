"""The op-by-op API's launches (set up while the op before still runs, tables
and measurements as kernel arguments): gates, channels, measurements, resets
and flag gates called back to back, at the edges of the channel kernel's
blocks (64 rows, 8 shot-words), bit for bit against the oracle."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 31, 32, 96])
@pytest.mark.parametrize("shots", [1, 65, 511, 513, 1100])
def test_ops_back_to_back_match_oracle(ps, O, n, shots):
    from plaquette_simulator import circuits as C
    rng = C.SplitMix64(1000 * n + shots)
    st = ps.CliffordState(n, shots, 9, True)
    o = O.Oracle(n, shots, seed=9)
    p1, p2 = (0.2, 0.0, 0.3), [0.002 * (j + 1) for j in range(15)]
    nrec = 0
    for k in range(120):
        a, b, kind = rng.below(n), rng.below(n), rng.below(12)
        if kind < 2:
            st.apply_hadamard_gate(a)
            op = (C.OP_H, a, 0, 0)
        elif kind == 2:
            st.apply_phase_gate(a)
            op = (C.OP_S, a, 0, 0)
        elif kind in (3, 4) and a != b:
            st.apply_control_not_gate(a, b)
            op = (C.OP_CX, a, b, 0)
        elif kind == 5 and a != b:
            st.apply_control_phase_gate(a, b)
            op = (C.OP_CZ, a, b, 0)
        elif kind in (6, 7):
            st.pauli_channel_1(a, *p1)
            op = (C.OP_PAULI1, a, 0, 0)
        elif kind == 8 and a != b:
            st.pauli_channel_2(a, b, p2)
            op = (C.OP_PAULI2, a, b, 3)
        elif kind == 9:
            st.measure_qubit(a)
            op = (C.OP_M, a, 0, -1)
            nrec += 1
        elif kind == 10:
            st.reset_qubit(a)
            op = (C.OP_R, a, 0, -1)
            nrec += 1
        elif nrec:
            r = rng.below(nrec)
            st.apply_hadamard_gate_with_apply_flag(a, r)
            op = (C.OP_H_IF, a, 0, r)
        else:
            continue
        o.run(np.array([op], np.int32), np.array(p1 + tuple(p2), np.float32))
    gx, gz, gr = st.device_to_host_numpy()
    ox, oz, orr = o.tableau()
    assert np.array_equal(gx, ox) and np.array_equal(gz, oz) and np.array_equal(gr, orr)
    for r in range(nrec):
        res, det = st.record(r)
        ores, odet = o.record(r)
        assert np.array_equal(res, ores) and np.array_equal(det, odet), r


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 100, 128, 129, 256, 300])
@pytest.mark.parametrize("words", [152, 154, 306, 612])
def test_measurements_of_wide_states_equal_narrow_ones(ps, n, words):
    """Wide states measure with fewer threads a shot-word: every shot-word
    ends as in a narrow state that holds only those shots."""
    from plaquette_simulator import circuits as C
    shots = 64 * words - 7
    rng = C.SplitMix64(n + words)
    ops = [(rng.below(6), rng.below(n), rng.below(n)) for _ in range(60)]

    def run(st):
        rec = []
        for kind, a, b in ops:
            if kind < 2:
                st.apply_hadamard_gate(a)
            elif kind == 2 and a != b:
                st.apply_control_not_gate(a, b)
            elif kind == 3:
                st.apply_phase_gate(a)
            elif kind == 4:
                rec.append(st.measure_qubit(a, 0.3))
            else:
                rec.append(st.reset_qubit(a))
        return [np.concatenate([st.record(r)[0], st.record(r)[1]]) for r in rec]

    wide = ps.CliffordState(n, shots, 13, True)
    recs = run(wide)
    for first, count in ((0, 2), (words // 2 & ~1, 2), (words - 2, 2)):
        k = min(64 * count, shots - 64 * first)
        narrow = ps.CliffordState(n, k, 13, True)
        narrow.set_shot_offset(64 * first)
        nrec = run(narrow)
        for u, v in zip(wide.tableau_words(first, count), narrow.tableau_words(0, count)):
            assert np.array_equal(u, v)
        for u, v in zip(recs, nrec):
            assert np.array_equal(u[:shots][64 * first:64 * first + k], v[:k])
            assert np.array_equal(u[shots:][64 * first:64 * first + k], v[k:])
