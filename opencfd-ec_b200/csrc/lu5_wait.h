// Bounds of the waits of the version-5 sweep (lusgs5.cuh).  No CUDA in here: tested on the host.
//
// Warp E waits for words of other tiles, in rounds of polls (loads in L2 and votes, about half a
// microsecond); the other roles of its CTA wait for one another and so, in the end, for E, by tries of an
// mbarrier, which the hardware suspends for 3.95 us where the phase does not complete (B200, 2,000 tries).
// They get at least as many tries as E gets rounds: E's bound runs out first, and the terms it then
// delivers end their waits.
#pragma once
#ifdef __CUDACC__
#define LU5_HD __host__ __device__ __forceinline__
#else
#define LU5_HD inline
#endif

namespace ocfd {

constexpr int LU5_ROUND = 8;          // units of a wait's bound (polls of about 64 ns) in a round of E
constexpr int LU5_SPARE = 25000;      // 0.1 s of tries beyond E's bound

LU5_HD int lu5_rounds(long long limit) { return (int)(limit / LU5_ROUND < (1 << 30) ? limit / LU5_ROUND : (1 << 30)); }
LU5_HD int lu5_tries(long long limit) { return lu5_rounds(limit) + LU5_SPARE; }

}  // namespace ocfd
