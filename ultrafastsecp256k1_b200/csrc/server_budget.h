// What of a server's memory budget its key table takes.
#pragma once
#include <stdint.h>

namespace uf {

inline uint64_t key_table_bytes(uint32_t log2, uint64_t slot) { return log2 ? (slot << log2) + 256 : 0; }

// log2 of the table that the budget holds beside one launch slot: the one asked
// for, or half of it (none below 2^min_log2) where the budget holds only three
// quarters of that; -1, refused, where it does not hold that much.  A key's slot is
// 768 bytes; three quarters are the 576 bytes of a table of eight points, with
// which budgets were chosen that have to go on working.
inline int key_table_fit(uint32_t log2, uint32_t min_log2, uint64_t slot, uint64_t budget, uint64_t launch_slot) {
    if (budget < launch_slot || budget - launch_slot < key_table_bytes(log2, slot / 4 * 3)) return -1;
    if (budget - launch_slot >= key_table_bytes(log2, slot)) return (int)log2;
    return log2 > min_log2 ? (int)log2 - 1 : 0;
}

}  // namespace uf
