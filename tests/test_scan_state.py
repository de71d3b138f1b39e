"""The counters that the device-wide scan keeps between launches (csrc/scan_state.h): the same rules that its blocks
follow on the device, run on the CPU in random interleavings of blocks, with launches that overlap against the
contract, blocks that give up and launch numbers that wrap around."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fe2o3_b200", "csrc")

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
#include "scan_state.h"

struct Words {
    static scan_word add(scan_word *p, scan_word v) { const scan_word o = *p; *p += v; return o; }
    static void fetch_or(scan_word *p, scan_word v) { *p |= v; }
    static void store(scan_word *p, scan_word v) { *p = v; }
};

constexpr uint32_t kMax = 16, kExpired = 4, kState = 6;
std::mt19937 rng;
uint32_t below(uint32_t n) { return rng() % n; }

scan_word state;
scan_word desc[kMax];
uint32_t status;   // first one wins, as on the device
void report(uint32_t s) { if (!status) status = s; }
void take_status() { if (status == kState) { state = 0; for (scan_word &d : desc) d = 0; } status = 0; }

struct Launch {
    bool ring;
    uint32_t blocks, tiles, tickets;
    std::vector<uint32_t> value, out;
    Launch() {
        ring = below(2);
        tiles = 1 + below(kMax);
        blocks = ring ? 1 + below(6) : tiles;
        tickets = ring ? tiles + blocks : blocks;
        for (uint32_t i = 0; i < tiles; ++i) value.push_back(1 + below(1u << 20));
        out.assign(tiles, 0xdeadbeefu);
    }
    bool right() const {
        uint32_t run = 0;
        for (uint32_t i = 0; i < tiles; ++i) { if (out[i] != run) return false; run += value[i]; }
        return true;
    }
};

struct Block {
    Launch *l;
    int phase;   // 0 starts, 1 draws a ticket, 2 publishes its tile's sum, 3 adds up the tiles before, 4 finishes, 5 is gone
    uint32_t tag, tile, next, sum;
};

// false: waits
bool step(Block &b) {
    scan_word w;
    switch (b.phase) {
    case 0:
        b.tag = scan_tag(state);
        b.phase = 1;
        return true;
    case 1:
        if (scan_take<Words>(&state, b.l->tickets, w)) {
            b.tile = scan_tickets(w);
        } else {
            report(kState);
            b.tile = ~0u;
        }
        if (!b.l->ring) b.tag = scan_tag(w);
        b.phase = b.tile < b.l->tiles ? 2 : b.l->ring ? 4 : 5;
        return true;
    case 2:
        desc[b.tile] = ((scan_word)b.tag << 32) | b.l->value[b.tile];
        b.next = b.sum = 0;
        b.phase = 3;
        return true;
    case 3:
        if (b.next == b.tile) { b.l->out[b.tile] = b.sum; b.phase = b.l->ring ? 1 : 4; return true; }
        if ((uint32_t)(desc[b.next] >> 32) != b.tag) return false;
        b.sum += (uint32_t)desc[b.next++];
        return true;
    default:
        if (!scan_finish<Words>(&state, desc, kMax, b.tag, b.l->blocks, b.l->tickets)) report(kState);
        b.phase = 5;
        return true;
    }
}

void run(std::vector<Launch *> launches) {
    std::vector<Block> blocks;
    for (Launch *l : launches)
        for (uint32_t i = 0; i < l->blocks; ++i) blocks.push_back(Block{l, 0, 0, 0, 0, 0});
    // blocks that are resident when the launch begins draw before any is through
    if (launches.size() == 1)
        for (Block &b : blocks) step(b);
    uint32_t idle = 0;
    while (!blocks.empty()) {
        const uint32_t i = below(blocks.size());
        if (step(blocks[i])) idle = 0;
        else if (++idle > 200 * blocks.size()) { report(kExpired); blocks[i].phase = 4; }   // its wait runs out
        if (blocks[i].phase == 5) { blocks[i] = blocks.back(); blocks.pop_back(); }
    }
}

#define CHECK(c) do { if (!(c)) { printf("trial %d: %s, line %d\n", trial, #c, __LINE__); return 1; } } while (0)

int main(int argc, char **argv) {
    const int trials = atoi(argv[1]);
    int overlapped_reports = 0;
    for (int trial = 0; trial < trials; ++trial) {
        rng.seed(trial);
        state = 0;
        for (scan_word &d : desc) d = 0;
        status = 0;
        if (trial % 4 == 3) {   // launch numbers about to wrap around, descriptors of the last launches standing
            state = (scan_word)(0xfffffff8u + below(7)) << 32;
        }
        for (int i = 0; i < 8; ++i) { Launch l; run({&l}); CHECK(status == 0 && l.right()); }
        if (trial % 2) { Launch a, b; run({&a, &b}); }           // two at once
        else { Launch a; a.tickets += 1 + below(3); run({&a}); }    // one that ends before it has drawn all its tickets
        overlapped_reports += status != 0;
        const bool reads = below(2);
        if (reads) take_status();
        for (int i = 0; i < 4; ++i) {
            Launch l;
            status = 0;   // (this launch's own report)
            run({&l});
            CHECK(status != 0 || l.right());   // never wrong in silence
            if (reads) take_status();
        }
        if (status) take_status();
        Launch once; run({&once});
        take_status();
        for (int i = 0; i < 3; ++i) { Launch l; run({&l}); CHECK(status == 0 && l.right()); }   // put right for good
    }
    printf("ok %d\n", overlapped_reports);
    return 0;
}
"""


def test_scan_counters_recover(tmp_path):
    (tmp_path / "model.cpp").write_text(SOURCE)
    exe = str(tmp_path / "model")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, str(tmp_path / "model.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe, "20000"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
