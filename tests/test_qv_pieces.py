"""The copies of the Coulomb kernel's q_ov rows, compiled for the host: every source lies on a 16-byte boundary, no copy reads
outside the matrix, and the staged window holds the row's columns at its phase."""
import os
import subprocess
import textwrap

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dftbaby_b200", "csrc")

PROGRAM = textwrap.dedent("""
    #include <stdio.h>
    #include <stdlib.h>
    #include <string.h>
    #include "qv_pieces.cuh"

    int main(int argc, char **argv) {
        const int M = atoi(argv[1]), K = atoi(argv[2]), off = atoi(argv[3]), kbeg = atoi(argv[4]), kend = atoi(argv[5]);
        double *base = (double *)aligned_alloc(64, (((size_t)M * K + 16) * 8 + 63) / 64 * 64);
        double *Q = base + off;
        for (long i = 0; i < (long)M * K; ++i) Q[i] = i + 1;
        int bad = 0;
        for (int row = 0; row < (M + 63) / 64 * 64; ++row)
            for (int k0 = 0; kbeg + k0 < kend; k0 += QV_K) {
                double win[2 * QV_PIECES];
                for (int i = 0; i < 2 * QV_PIECES; ++i) win[i] = -1.0;
                const int phase = row < M ? qv_phase(Q, K, row, kbeg) : 0;
                for (int pc = 0; pc < 16 + phase; ++pc) {
                    const QvPiece p = qv_piece(Q, M, K, row, kbeg, kend, pc);
                    const int most = pc < 16 ? 2 : 1, left = p.left - k0, n = left < 0 ? 0 : (left < most ? left : most);
                    const double *src = qv_source(p, Q, k0, n);
                    if (p.src + k0 < Q) {  // the kernel's copy of the first element alone
                        bad += p.src + k0 + 1 != Q || n == 0;
                        if (n > 1) win[1] = Q[0];
                        continue;
                    }
                    bad += ((uintptr_t)src & 15) != 0;
                    bad += n > 0 && (src < Q || src + n > Q + (long)M * K);
                    if (bad) break;
                    win[2 * pc] = win[2 * pc + 1] = 0.0;
                    memcpy(win + 2 * pc, src, 8 * n);
                }
                for (int i = 0; i < QV_K && !bad; ++i) {
                    const int k = kbeg + k0 + i;
                    bad += win[phase + i] != (row < M && k < kend ? Q[(long)row * K + k] : 0.0);
                }
                if (bad) {
                    printf("row %d stage at %d\\n", row, k0);
                    return 1;
                }
            }
        return 0;
    }
""")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("qv")
    src, exe = d / "check.cpp", d / "check"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    return str(exe)


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("M,K,kbeg,kend", [(1, 1, 0, 1), (1, 99, 0, 99), (1, 97, 32, 97), (37, 99, 0, 99), (64, 33, 0, 33), (65, 31, 0, 31), (3, 64, 32, 64),
                                           (5, 257, 64, 192), (5, 257, 192, 257), (63, 32, 0, 32), (2, 95, 64, 95)])
def test_copies(program, M, K, kbeg, kend, off):
    r = subprocess.run([program] + [str(x) for x in (M, K, off, kbeg, kend)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
