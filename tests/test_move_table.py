"""The move table of the specialised kernels against the general move.

A host program applies both to random sites, words and random bytes on every
specialised geometry: the general move (slots, transition table, walls, as
csrc/elp_device.cuh) and the table move of csrc/elp_sweep2.cu (one entry per
row and option, offsets per boundary class).  Acceptance, the three new words
and their sites must agree, and every index must stay inside the domain.
"""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "mc-polymer-simulation_b200", "csrc")

PROGRAM = r"""
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include "elp_internal.h"
typedef uint32_t u32;
static const u32 U = 1u << 16, WALL = U | 0x10 | 3;
static const int CODES[] = {1, 2, 4, 5, 6, 7, 8, 9, 10, 11, 13, 14, 15};
int main(int argc, char** argv)
{
    elp_geometry g;
    memset(&g, 0, sizeof g);
    g.tx = atoi(argv[1]); g.ty = atoi(argv[2]); g.tz = atoi(argv[3]); g.periodic = atoi(argv[4]);
    const int linear = atoi(argv[5]);
    g.L = g.periodic ? g.tx : 2 * g.tx * (g.ty == g.tx ? 1 : 2);
    g.ncol = elp_pick_ncol(g.tx);
    elp_smem_layout lay;
    elp_layout(&g, &lay);
    static uint8_t tab[4096];
    static u32 mv[ELP_MOVES_MAX];
    elp_build_table(tab);
    if (elp_move_table(&g, &lay, mv) > ELP_MOVES_MAX) return 2;
    const int per = g.periodic, sx = lay.sx, sxy = lay.sxy, W = lay.words;
    const bool soff = !per || (g.tx - 1) * (1 + sx + sxy) <= 32767;
    u32* S = (u32*)calloc(W, 4);
    long bad = 0, acc = 0;
    srand(7);
    for (long it = 0; it < 400000; it++) {
        int c[3], n[3] = {g.tx, g.ty, g.tz};
        for (int k = 0; k < 3; k++) c[k] = rand() % 3 ? rand() % n[k] : (rand() % 2 ? 0 : n[k] - 1);   // faces often
        const int sh = per ? 0 : rand() % 4, p = lay.ox + sh + c[0] + sx * c[1] + sxy * c[2];
        int nb[16];
        for (u32 b = 0; b < 16; b++) {
            nb[b] = -1;
            if (b && b != 15 && !elp_valid_bond(b)) continue;
            int q[3] = {c[0] + elp_bt(b), c[1] + elp_bu(b), c[2] + elp_bv(b)}, out = 0;
            for (int k = 0; k < 3; k++) {
                if (per) q[k] = (q[k] + g.L) % g.L;
                else out |= q[k] < 0 || q[k] >= n[k];
            }
            nb[b] = lay.ox + sh + q[0] + sx * q[1] + sxy * q[2];
            if (nb[b] < 0 || nb[b] >= W) return 3;
            if (b == 15) continue;
            S[nb[b]] = out ? WALL : rand() % 3 == 0 ? 0 : CODES[rand() % (12 + linear)] | (rand() % 2 ? 1u : 1u + rand() % 4) << 16;
        }
        const u32 wP = S[p], bo = wP & 15, s = rand() & 1, r4 = rand() & 15;
        if (s && wP && bo != 15 && S[nb[bo]] == 0) { for (int b = 0; b < 16; b++) if (nb[b] >= 0) S[nb[b]] = 0; continue; }
        // the general move
        int ok = 0, qB = -1, qY = -1;
        u32 rP = 0, rB = 0, rY = 0, s1 = 0, s2 = 0, wB = 0;
        int live = wP != 0;
        if (live && !s) { live = wP >= 2 * U; s2 = bo; }
        if (live && s) {
            live = bo != 15 && S[nb[bo]] != WALL;
            if (live) { qB = nb[bo]; wB = S[qB]; s1 = bo; s2 = wB >= 2 * U ? 0 : wB & 15; }
        }
        const u32 e = live ? tab[s1 << 8 | s2 << 4 | r4] : 0, d1 = e & 15, d2 = e >> 4;
        if (e) {
            qY = nb[d1];
            ok = d2 ? !(d1 && S[qY]) : S[qY] != WALL;
            rP = (wP & ~15u) + (s ? (d1 ? 0 : U) : 0u - U) + (d1 ? d1 : d2);
            rB = s2 ? 0 : wB - U;
            rY = d2 ? d2 | U : S[qY] + U;
        }
        // the table move
        const u32 R = (s ? 0xFF80u : 0) | r4 << 2;
        const int cls = (c[0] == 0 ? 0 : c[0] == g.L - 1 ? 2 : 1) + 3 * (c[1] == 0 ? 0 : c[1] == g.L - 1 ? 2 : 1) +
                        9 * (c[2] == 0 ? 0 : c[2] == g.L - 1 ? 2 : 1);
        const u32* of = mv + ELP_MOVE_ENTRIES + (per ? 16 * cls : 0);
        const u32 V = of[bo];
        const int pB = soff ? 4 * p + ((int)V >> 14) : (int)((4 * p + (V >> 14)) & 0x3FFFF);
        if (pB < 0 || pB >= 4 * W || pB & 3) return 4;
        const u32 X = s ? S[pB / 4] : wP;
        const bool c2 = X >= 2 * U;
        u32 ix = R & (V | 0x3C);
        if (c2 != (bool)s) ix += (X & 15) << 6;
        if (ix >= 4 * ELP_MOVE_ENTRIES || ix & 3) return 5;
        const u32 E = mv[ix / 4], V2 = of[E >> 28];
        const int pY = !per ? 4 * p + ((int)E >> 18) : soff ? 4 * p + ((int)V2 >> 14) : (int)((4 * p + (V2 >> 14)) & 0x3FFFF);
        if (pY < 0 || pY >= 4 * W || pY & 3) return 6;
        const u32 wY = S[pY / 4];
        const int ok2 = E && !(wY & E & (per ? 0xF : 0x1F));
        const u32 nP = ((wP & ~15u) | (E >> 5 & 15)) + (E & 0x30000u) - U, nB = c2 ? X - U : 0, nY = wY + U + (E >> 9 & 15);
        if (ok != ok2) bad++;
        else if (ok) {
            acc++;
            if (nP != rP || (s && (nB != rB || pB != 4 * qB)) || pY != 4 * qY || (d1 && nY != rY)) bad++;
        }
        for (int b = 0; b < 16; b++) if (nb[b] >= 0) S[nb[b]] = 0;
    }
    printf("%ld %ld\n", acc, bad);
    return 0;
}
"""

GEOMETRIES = [(16, 16, 16, 0), (32, 16, 16, 0), (32, 32, 16, 0), (32, 32, 32, 0), (48, 24, 24, 0), (24, 24, 24, 0),
              (20, 20, 20, 0), (40, 20, 20, 0), (16, 16, 16, 1), (18, 18, 18, 1), (20, 20, 20, 1), (22, 22, 22, 1),
              (24, 24, 24, 1), (26, 26, 26, 1), (28, 28, 28, 1), (30, 30, 30, 1), (32, 32, 32, 1)]


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("moves")
    src, exe = d / "moves.cpp", d / "moves"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, str(src), os.path.join(CSRC, "elp_host.cpp"), "-o", str(exe)],
                   check=True)
    return str(exe)


@pytest.mark.parametrize("linear", [0, 1])
@pytest.mark.parametrize("geom", GEOMETRIES)
def test_table_move_equals_general_move(program, geom, linear):
    out = subprocess.run([program, *map(str, geom), str(linear)], capture_output=True, text=True)
    assert out.returncode == 0, f"index out of range (code {out.returncode})"
    accepted, bad = map(int, out.stdout.split())
    assert bad == 0 and accepted > 20000
