"""Runs of random measurements in the per-shot kernels, where shots differ in
their pivots: conditional Clifford gates make the shots' x / z differ, then
long runs of M / R follow in which a shot may be random or deterministic
beside others of its word, at several pivots, with resets, biased and forced
draws, and qubits measured again.  Every tile width, columns and rows at the
edges of a warp, against the oracle."""
import numpy as np
import pytest


def scattered_circuit(n, seed, rounds=4):
    from plaquette_simulator import circuits as C
    rng = C.SplitMix64(seed)
    c = C.Circuit(n)
    nrec = 0
    for _ in range(rounds):
        for q in range(n):
            if rng.below(2):
                c.h(q)
        for q in range(n - 1):
            if rng.below(3):
                c.cx(q, q + 1) if rng.below(2) else c.cx(q + 1, q)
        for q in range(n):
            if rng.below(3) == 0:
                c.s(q)
        if nrec:
            for _ in range(n):
                (c.h_if if rng.below(2) else c.s_if)(rng.below(n), rng.below(nrec))
        for _ in range(n + 3):  # a run of measurements, some qubits twice
            q = rng.below(n)
            if rng.below(4) == 0:
                c.r(q)
            else:
                c.m(q, bias=(0.5, 0.25, 0.9)[rng.below(3)])
            nrec += 1
    return c


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 7, 16, 31, 33, 65])
@pytest.mark.parametrize("meas_words", [1, 2, 4])
@pytest.mark.parametrize("forced", [False, True])
def test_scattered_pivots_match_oracle(ps, O, n, meas_words, forced):
    from plaquette_simulator.circuit import CompiledCircuit
    c = scattered_circuit(n, 31 * n + meas_words)
    shots, nm = 64 * 5 + 9, c.num_measurements()
    f = np.random.default_rng(n).integers(0, 256, size=(nm, (shots + 7) // 8), dtype=np.uint8) if forced else None
    st = ps.CliffordState(n, shots, 8, True)
    cc = CompiledCircuit(c, st, meas_words=meas_words)
    cc.set_forced(f)
    cc.run()
    o = O.Oracle(n, shots, seed=8)
    o.run(c.op_array(), c.param_array(), f)
    gx, gz, gr = st.device_to_host_numpy()
    ox, oz, orr = o.tableau()
    assert np.array_equal(gx, ox) and np.array_equal(gz, oz) and np.array_equal(gr, orr)
    for k in range(nm):
        res, det = st.record(cc.first_record + k)
        ores, odet = o.record(k)
        assert np.array_equal(res, ores) and np.array_equal(det, odet), k
