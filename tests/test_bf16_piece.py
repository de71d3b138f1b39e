"""Pieces of four bf16 at any address (csrc/bf16_piece.h): the code that the exact-order GEMM loads its operands with, run
on the CPU over a memory that notes what is read: every load is aligned, no byte outside the elements asked for is
touched, and the elements come out in their places."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fe2o3_b200", "csrc")

SOURCE = r"""
#include <cstdio>
#include <cstring>
#include "bf16_piece.h"

alignas(16) static uint16_t memory[64];
static int from, to, bad;   // the bytes that may be read
struct Noted {
    static void see(const void *p, int bytes) {
        const int at = (int)((const char *)p - (const char *)memory);
        if (at % bytes != 0 || at < from || at + bytes > to) bad = 1;
    }
    static uint32_t half(const uint16_t *p) { see(p, 2); return *p; }
    static uint32_t word(const uint16_t *p) { see(p, 4); uint32_t w; memcpy(&w, p, 4); return w; }
    static void two_words(const uint16_t *p, uint32_t &a, uint32_t &b) { see(p, 8); memcpy(&a, p, 4); memcpy(&b, p + 2, 4); }
};

int main() {
    for (int i = 0; i < 64; ++i) memory[i] = (uint16_t)(0x4100 + 7 * i);
    int pieces = 0;
    for (int base = 0; base < 16; ++base)
        for (int end = 0; end <= 24; ++end)
            for (int first = 0; first < 28; first += 4)
                for (int ok = 0; ok < 2; ++ok)
                    for (int vec = 0; vec < (base % 4 == 0 ? 2 : 1); ++vec) {
                        const int last = first + 4 < end ? first + 4 : end;
                        from = 2 * (base + first);
                        to = ok && last > first ? 2 * (base + last) : from;
                        uint32_t w[3] = {0, 0, 0}, got[2];
                        const bool halves = load_piece<Noted>(w, memory + base, first, end, ok, vec);
                        join_piece(w, halves, got[0], got[1]);
                        for (int i = 0; i < 4; ++i) {
                            const uint32_t want = ok && first + i < end ? memory[base + first + i] : 0u;
                            if ((got[i / 2] >> (16 * (i % 2)) & 0xffffu) != want) bad = 1;
                        }
                        if (bad) { printf("base %d end %d first %d ok %d vec %d\n", base, end, first, ok, vec); return 1; }
                        ++pieces;
                    }
    printf("ok %d\n", pieces);
    return 0;
}
"""


def test_pieces_read_their_own_elements_only(tmp_path):
    (tmp_path / "pieces.cpp").write_text(SOURCE)
    exe = str(tmp_path / "pieces")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", CSRC, str(tmp_path / "pieces.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
