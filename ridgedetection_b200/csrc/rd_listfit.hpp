// rd_listfit.hpp -- room for the neighbour lists of a decimation.
//
// A list's start is a 32-bit offset, but the lists of 46,342 points that all lie
// within 2 r2 of one another already hold 2^31 entries: lengths are added up in
// 64 bits, and lists that do not fit their buffer or the offsets are not built (the
// decimation then walks the hash buckets).
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define RD_HD __host__ __device__
#else
#define RD_HD
#endif

namespace rdb {

// longest list a warp's scan of 32 lengths takes without overflowing 32 bits
constexpr int LIST_LEN_MAX = (1 << 26) - 1;

// length as the scan adds it
RD_HD inline int list_len(int n) { return n > LIST_LEN_MAX ? LIST_LEN_MAX : n; }

// total: sum of list_len over all points.  A list of LIST_LEN_MAX entries needs as
// many points, whose lists together are far beyond any room.
RD_HD inline bool lists_fit(int64_t total, int64_t room)
{
    return total <= room && total <= INT32_MAX;
}

}  // namespace rdb
