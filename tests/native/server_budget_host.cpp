// Test harness: what of a server's memory budget its key table takes (csrc/server_budget.h).
#include "../../ultrafastsecp256k1_b200/csrc/server_budget.h"

extern "C" int sb_fit(uint32_t log2, uint32_t min_log2, uint64_t slot, uint64_t budget, uint64_t launch_slot) {
    return uf::key_table_fit(log2, min_log2, slot, budget, launch_slot);
}
