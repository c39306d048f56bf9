// Running sums over the lanes of a warp whose bounds never go backwards.  No CUDA types: the same code runs over an array of
// 32 values in tests/test_lane_scan_host.py.
#pragma once

#ifdef __CUDACC__
#define TB_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define TB_HOST_DEVICE inline
#endif

namespace tb {

// Sum of the lanes up to and including this one, of non-negative values.  add_below(v, o) adds the value of lane - o, where
// there is one; max_below(v, o) is the larger of the two.  The sums are formed in a tree that differs from lane to lane, so
// where a lane's own share is around the last bit its sum can round below its left neighbour's; the running maximum behind
// them makes them monotone.
template <typename Value, typename AddBelow, typename MaxBelow>
TB_HOST_DEVICE Value monotone_lane_sums(Value v, AddBelow add_below, MaxBelow max_below) {
    for (int o = 1; o < 32; o <<= 1) v = add_below(v, o);
    for (int o = 1; o < 32; o <<= 1) v = max_below(v, o);
    return v;
}

}  // namespace tb
