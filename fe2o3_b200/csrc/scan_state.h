// What the device-wide scan (scan.cu) keeps on the device from one launch to the next, and the rules by which its
// blocks use it.  The rules are written over three operations on a 64-bit word, so that a test can run them on the
// CPU in any interleaving.
//
// One word holds the launch number, which also marks the launch's descriptors, so that nothing has to be cleared in
// between, the tickets drawn (which tile a block works on) and the blocks that have finished.  The last block to
// finish closes the launch.  That only works for one launch at a time: where two overlap on one context, or one of
// them ended early, the word is no longer that of one launch, some block notices and marks it.  From then on every
// launch draws nothing, does nothing and reports FE2O3_KSTATUS_SCAN_STATE, until the host, which clears everything
// when it takes that status, has seen it.
#ifndef FE2O3_SCAN_STATE_H
#define FE2O3_SCAN_STATE_H
#include <stdint.h>

#ifdef __CUDACC__
#define FE2O3_SCAN_FN __device__ __forceinline__
#else
#define FE2O3_SCAN_FN inline
#endif

typedef unsigned long long scan_word;

// {launch number: 32, marked: 1, blocks finished: 11, tickets drawn: 20}
constexpr uint32_t kScanTicketBits = 20, kScanBlockBits = 11;
constexpr scan_word kScanTicket = 1, kScanBlock = 1ull << kScanTicketBits, kScanMark = 1ull << (kScanTicketBits + kScanBlockBits);

FE2O3_SCAN_FN uint32_t scan_tickets(scan_word w) { return (uint32_t)w & ((1u << kScanTicketBits) - 1u); }
FE2O3_SCAN_FN uint32_t scan_blocks(scan_word w) { return ((uint32_t)w >> kScanTicketBits) & ((1u << kScanBlockBits) - 1u); }
// The launch number as descriptors carry it: never that of a cleared descriptor, which is 0.
FE2O3_SCAN_FN uint32_t scan_tag(scan_word w) { return (uint32_t)(w >> 32) + 1u; }

// One ticket of a launch that has `tickets` of them; false when there is none.
template <typename Words>
FE2O3_SCAN_FN bool scan_take(scan_word *state, uint32_t tickets, scan_word &drawn) {
    drawn = Words::add(state, kScanTicket);
    if (!(drawn & kScanMark) && scan_tickets(drawn) < tickets) return true;
    Words::fetch_or(state, kScanMark);
    return false;
}

// Last act of a block of the launch with this tag; false when the word is not that of one launch.
template <typename Words>
FE2O3_SCAN_FN bool scan_finish(scan_word *state, scan_word *desc, uint32_t max_tiles, uint32_t tag, uint32_t blocks, uint32_t tickets) {
    const scan_word before = Words::add(state, kScanBlock);
    if (!(before & kScanMark) && scan_tag(before) == tag) {
        const uint32_t finished = scan_blocks(before) + 1u;
        if (finished < blocks) return true;
        if (finished == blocks && scan_tickets(before) == tickets) {   // every ticket drawn and none too many
            uint32_t next = tag;
            if (next == 0xffffffffu) {   // its tag would be 0, and after it descriptors of long ago would match
                for (uint32_t i = 0; i < max_tiles; ++i) desc[i] = 0;
                next = 0;
            }
            Words::store(state, (scan_word)next << 32);
            return true;
        }
    }
    Words::fetch_or(state, kScanMark);
    return false;
}

#endif
