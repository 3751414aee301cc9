// The ring of weight pieces in the absorb kernel: which stage a piece takes and which barrier phase it is.  Plain C++, so that
// a host test can go through every wait of a schedule.
//
// A waiter on an mbarrier names a phase by one bit, its parity: the wait also passes while the phase TWO before the one it
// means is the last one complete.  So a waiter has to have seen the phase before itself.  TMA copies land in any order, and
// each of the kernel's MMA issuers waits for its own pieces alone; a stage therefore belongs to ONE issuer, for good, and every
// issuer walks its stages in the order of its own pieces.  (A ring shared by the issuers gives a stage to another issuer at
// every wrap: that one can find the barrier a phase behind and read weights that have not landed.)
#pragma once

#include <cstdint>

namespace mla {

struct AbsorbRing {
    uint32_t per_issuer;                            // stages of each issuer
    // piece `half` (0 or 1: the first or last 64 inputs) of issuer d's d-tile in the block's unit number `unit`
    static constexpr uint32_t count(uint32_t unit, uint32_t half) { return 2 * unit + half; }
    constexpr uint32_t stage(uint32_t d, uint32_t unit, uint32_t half) const { return d * per_issuer + count(unit, half) % per_issuer; }
    constexpr uint32_t parity(uint32_t unit, uint32_t half) const { return (count(unit, half) / per_issuer) & 1; }
};

}  // namespace mla
