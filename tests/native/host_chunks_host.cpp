// Test harness: how a host-buffer call is cut into chunks (csrc/host_chunks.h).
#include "../../ultrafastsecp256k1_b200/csrc/host_chunks.h"

// Sizes of the chunks of a call of `items`, | 1 << 40 where a chunk waits for the
// one before it; returns their number (at most cap).
extern "C" int hc_cut(size_t wave, size_t items, unsigned long long* out, int cap) {
    const uf::HostChunks c(wave);
    int k = 0;
    for (size_t off = 0; off < items && k < cap; ++k) {
        const size_t m = c.size(k, items - off);
        out[k] = m | (c.after_previous(k, m) ? 1ull << 40 : 0);
        off += m;
    }
    return k;
}

extern "C" int hc_count(size_t wave, size_t items, int limit) { return (int)uf::HostChunks(wave).count(items, limit); }
