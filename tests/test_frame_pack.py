"""The sign program as the device reads it (FrameProgram::pack_noise): on the
CPU, each channel's four row lists hold exactly the rows that its entries
named, short ones in the channel's slot, longer ones from even places, and the measurement ops, moved to a table without the
channels' entries, give the same records and signs as before -- linearized or
not, over random circuits with channels on one and two qubits."""
import os
import shutil
import subprocess

import pytest

from test_frame_linear import CSRC, PROGRAM, ROOT

MAIN = r"""
int main() {
    int lists = 0, longer = 0, launches = 0;
    const int64_t sizes[] = {1, 2, 5, 17, 40};
    for (int64_t n : sizes)
        for (uint64_t seed = 1; seed <= 6; ++seed)
            for (int lin = 0; lin < 2; ++lin) {
                FrameBuilder a = build(n, seed * 100 + n, 12);
                if (lin) a.linearize(1u << 20);
                FrameProgram b = a.prog;
                b.pack_noise();
                std::vector<uint32_t> bases;
                for (const auto &L : a.prog.launches)
                    if (L.seg >= 0) bases.push_back((uint32_t)a.prog.ops[L.op0].arg);
                bases.push_back((uint32_t)a.prog.slot_off.size());
                for (size_t k = 0; k + 1 < bases.size(); ++k)
                    for (uint32_t q = bases[k]; q + 1 < bases[k + 1]; ++q) {
                        uint32_t at = b.slot_rows[q].t0;
                        for (uint32_t c = 0; c < 4; ++c) {
                            std::vector<uint16_t> want;
                            for (uint32_t t = a.prog.slot_off[q]; t < a.prog.slot_off[q + 1]; ++t)
                                if ((a.prog.tab[t] >> (28 + c)) & 1u) want.push_back((uint16_t)(a.prog.tab[t] & kFrameRowMask));
                            const uint32_t len = b.slot_rows[q].len[c];
                            ++lists;
                            if (len <= FrameProgram::kSlotShort) {
                                const uint16_t *r = b.slot_rows[q].rows[c];
                                if (want != std::vector<uint16_t>(r, r + len)) {
                                    std::printf("FAIL n=%lld short list\n", (long long)n);
                                    return 1;
                                }
                                continue;
                            }
                            ++longer;
                            if ((at & 1u) || at + len > b.nrows.size() ||
                                want != std::vector<uint16_t>(b.nrows.begin() + at, b.nrows.begin() + at + len)) {
                                std::printf("FAIL n=%lld list\n", (long long)n);
                                return 1;
                            }
                            at += (len + 1) & ~1u;
                        }
                    }
                for (const auto &L : b.launches) {
                    launches++;
                    if ((L.tab0 & 3u) || L.tab1 > b.tab.size()) {
                        std::printf("FAIL n=%lld range\n", (long long)n);
                        return 1;
                    }
                    for (uint32_t i = L.op0; i < L.op1; ++i)
                        if ((b.ops[i].kind & 0xFFu) != F_NOISE && (b.ops[i].off < L.tab0 || b.ops[i].off > L.tab1)) {
                            std::printf("FAIL n=%lld op outside its range\n", (long long)n);
                            return 1;
                        }
                }
                for (uint64_t key = 0; key < 3; ++key) {
                    const Result ra = run(a.prog, n, key * 77 + seed), rb = run(b, n, key * 77 + seed);
                    if (ra.rec != rb.rec || ra.R != rb.R) {
                        std::printf("FAIL n=%lld run\n", (long long)n);
                        return 1;
                    }
                }
            }
    std::printf("OK %d %d %d\n", lists, longer, launches);
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_packed_program_equals_the_builder_s(tmp_path):
    src = tmp_path / "pack.cpp"
    src.write_text(PROGRAM[:PROGRAM.index("int main() {")] + MAIN)
    exe = tmp_path / "pack"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, "-I", os.path.join(ROOT, "include"), "-o", str(exe),
                    str(src), os.path.join(CSRC, "ps_frame.cpp")], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
    words = out.stdout.split()
    assert words[0] == "OK" and all(int(v) > 0 for v in words[1:4])
