// Device memory of a batch with row ids, and what the server charges a request
// for it.
//
// Two passes keep per item (query and tile) its hits and its first row-id slot
// or list entry, and, where that stays within a limit, the row ids of items
// with few hits.  The server sets the limit of the kept ids for each of its
// slots aside from its budget, and charges a request for its items (the
// look-back's record of a tile, more than the two passes take) and its ids.
#ifndef WAH_BUDGET_H
#define WAH_BUDGET_H
#include <stddef.h>
#include <stdint.h>
#include <algorithm>

namespace wah {

constexpr size_t ITEM_BYTES = 16;                  // two passes: hits and offset of an item
constexpr size_t KEPT_IDS = 32;                    // row ids kept per item
constexpr size_t KEPT_AT_MOST = (size_t)64 << 20;  // bytes of kept ids of a batch
constexpr size_t RECORD_BYTES = 48;                // look-back record of a tile

inline size_t kept_bytes(uint64_t nitems, size_t at_most) {
    const size_t b = nitems * KEPT_IDS * 4;
    return b <= at_most ? b : 0;
}
inline size_t batch_scratch(uint64_t nitems, size_t kept_at_most) {
    return nitems * ITEM_BYTES + kept_bytes(nitems, kept_at_most);
}
// A request over ntiles tiles with at most rid_cap row ids.
inline size_t request_charge(uint64_t ntiles, uint64_t rid_cap) { return ntiles * RECORD_BYTES + 16 + rid_cap * 4; }
// Kept ids of each of a server's slots: a quarter of the budget in all.
inline size_t slot_kept(size_t budget, uint32_t nslots) { return std::min(KEPT_AT_MOST, budget / 4 / nslots); }

}  // namespace wah
#endif
