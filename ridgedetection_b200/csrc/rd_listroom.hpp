// rd_listroom.hpp -- sizes of the lists kept across the evolve passes, for the host
// code that allocates them and the kernels that lay them out and fill them.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define RD_ROOM_HD __host__ __device__
#else
#define RD_ROOM_HD
#endif

namespace rdb {

// candidates of a block of points (k_assign_cull): the 1M helix has 17 blocks (of
// 7,812) with more than 32 (up to 119), over jumps of the spatial order that two boxes
// do not cover, and scanning 790 chosen points for each of them outlasted the rest of
// the pass
constexpr int CAND_MAX = 128;

// rows of the region of a key with n members when its cloud is regrouped: room for the
// list to grow before the next time
RD_ROOM_HD constexpr int list_room(const int n) { return n + (n >> 2) + 8; }

// rows that the regions of ns keys with n members in all can take
RD_ROOM_HD constexpr int64_t list_rows(const int64_t n, const int64_t ns) { return n + n / 4 + 8 * ns; }

// Whether a cloud's lists can be kept: their rows and the points' positions in them
// are 31-bit numbers.
RD_ROOM_HD constexpr bool lists_possible(const int64_t n, const int64_t ns)
{
    return n <= (int64_t(1) << 30) && list_rows(n, ns) <= INT32_MAX;
}

}  // namespace rdb
