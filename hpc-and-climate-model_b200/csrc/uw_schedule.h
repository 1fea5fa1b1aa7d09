// uw_schedule.h -- the rules that size the worklist launches, in one place for the host, the kernels and
// the tests (plain C++, no CUDA types).
#pragma once

#if defined(__CUDACC__)
#define UW_RULE __host__ __device__ __forceinline__
#else
#define UW_RULE static inline
#endif

// The worklist entry of thread tid, -1 for none: 32 per warp, or as few (a power of two) as spread the n
// entries over at most `spread` warps (0: full warps).  The fewer columns a warp holds, the fewer branches
// it runs for the others': with one warp per scheduler (592) against full warps, 64 columns take 6.5 and
// 6.9 ms, 256 columns 6.8 and 7.5, 1,024 columns 7.7 and 8.1.
UW_RULE int uw_spread(int n, int spread, int tid)
{
    int lanes = 32;
    while (lanes > 1 && (n + lanes / 2 - 1) / (lanes / 2) <= spread) lanes /= 2;
    const int t = (tid >> 5) * lanes + (tid & 31);
    return (tid & 31) < lanes && t < n ? t : -1;
}

// Threads of a worklist launch over at most n entries: one each, or a warp for each of `spread` warps.
UW_RULE int uw_list_threads(int n, int spread)
{
    return n >= 32 * spread ? n : 32 * (n < spread ? n : spread);
}

// Whether a stream whose latest call was number `last` counts among those that share the GPU with call
// number `tick`: a call of its own among the latest 32, one for each stream that the library keeps buffers
// for.  A program that uses its streams in turn shares the warps between them; one that has gone over to
// a single stream has them to itself from its 32nd call on.  (With every stream ever used counted, a process
// that once ran on 32 of them spread its later calls over 18 warps: 256 columns 7.5 instead of 6.8 ms.)
UW_RULE bool uw_stream_shares(unsigned long long last, unsigned long long tick) { return tick - last < 32; }
