// How a host-buffer call is cut into chunks that are packed, copied in and
// verified while one another's are (Backend::verify_host_strided).
#pragma once
#include <stddef.h>

#include <algorithm>

namespace uf {

// The FP64 kernel (wave != 0): chunks of one wave, 256 items per SM (37,888 on a
// 148-SM B200).  A smaller one would take the device as long as a full one once it
// holds more than 128 items per SM (0.68 ms; 0.54 below), and the CPU packs and
// copies in a wave in 0.2 ms.
//
// The integer kernels: chunks double from 16,384 items to 131,072.  They run four
// blocks per SM, so a launch of 37,888 is no whole wave of theirs and a small last
// chunk takes as long as a large one: in FP64 waves 37,889 items took 2.24 ms and
// 131,073 4.39, this way 1.75 and 4.11 (ECDSA, variant 4).
struct HostChunks {
    size_t first, most;
    bool waves;
    explicit HostChunks(size_t wave)
        : first(wave ? wave : size_t{1} << 14), most(wave ? wave : size_t{1} << 17), waves(wave != 0) {}
    // items of chunk k where `left` are left
    size_t size(size_t k, size_t left) const {
        return std::min(left, std::min(most, first << std::min<size_t>(k, 20)));
    }
    // chunks of a call, counted up to `limit`
    size_t count(size_t items, size_t limit) const {
        size_t k = 0;
        for (; items && k < limit; ++k) items -= size(k, items);
        return k;
    }
    // A last chunk of at most half a wave starts after the chunk before it: its
    // small blocks would fill the first SMs to finish, two by two.
    bool after_previous(size_t k, size_t m) const { return waves && k > 0 && m <= most / 2; }
};

}  // namespace uf
