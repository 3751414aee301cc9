// The ring of weight tiles in the projection kernel for few rows: which stage a k-block takes, which barrier phase it is, and which
// of the MMA issuers it belongs to.  Plain C++, so that a host test can go through every wait of a schedule.
//
// A stage belongs to ONE issuer, for good, as in the absorb's ring (mla_absorb_ring.h has the reason: a wait names its phase by
// one bit, copies land in any order, and an issuer that has not seen a stage's phase before can pass a wait a phase early).  With
// k-blocks dealt out in turn instead, nine stages and four issuers, a stage went to another issuer at every wrap: blocks of 10 and
// more k-blocks could read tiles that had not landed, release them early and leave copies in flight behind.
#pragma once

#include <cstdint>

namespace mla {

struct FewRing {
    static constexpr uint32_t stages = 9, issuers = 4;
    static constexpr uint32_t stage(uint32_t i) { return i % stages; }                    // of k-block i of the block
    static constexpr uint32_t parity(uint32_t i) { return (i / stages) & 1; }
    static constexpr uint32_t issuer(uint32_t i) { return stage(i) % issuers; }           // the first `issuers` k-blocks: one each
    // the issuer's k-block behind i: its next stage of this round, or its first one of the next
    static constexpr uint32_t next(uint32_t i) { return stage(i) + issuers < stages ? i + issuers : i - stage(i) + stages + issuer(i); }
};

}  // namespace mla
