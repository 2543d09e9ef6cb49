// rtc_claims.h - what the host knows of a job ring's work units (host side).
#pragma once

#include <algorithm>
#include <cstdint>

namespace rtc {

// Units are claimed on the device from one global sequence; the host reads the claim cursor one batch late.
// Claims that found nothing left move the cursor past the units there were, and an admission puts it back to
// where the new units begin: so a cursor counts only up to the units admitted when it was polled.
struct RingClaims {
    uint64_t limit = 0;                  // units admitted
    uint64_t claimed = 0;                // units claimed, as of the last observed poll
    uint32_t live = 0;                   // live slots, likewise
    uint64_t polled_limit[2] = {0, 0};   // `limit` when each poll was queued

    void polled(int slot) { polled_limit[slot] = limit; }
    void observe(int slot, uint64_t cursor, uint32_t live_slots) {
        claimed = std::min(cursor, polled_limit[slot]);
        live = live_slots;
    }
    // Whether every unit not yet claimed has an idle slot waiting for it: from here on the queue only runs
    // down.  Both counts are late, and a unit claimed meanwhile is still counted as unclaimed: the answer may
    // come a batch or two after the fact, never before it.
    bool runs_down(uint32_t slots) const { return limit - claimed + live <= slots; }
};

}  // namespace rtc
