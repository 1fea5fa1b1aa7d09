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
// it runs for the others', and the more warps wait for their instructions.  16 / 64 / 256 / 1,024 / 4,096 / 16,384
// columns, ms, with full warps 6.6 / 7.7 / 8.1 / 8.2 / 8.4 / 9.5, at two warps per multiprocessor 6.0 / 6.5 / 6.9 / 7.9 /
// 8.4 / 9.6, at one per scheduler (592 in all, as here) 6.0 / 6.5 / 6.9 / 7.7 / 8.7 / 9.5, at four per scheduler 6.0 /
// 6.5 / 6.9 / 7.7 / 10.4 / 11.9.
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

// Worklist entries up to which the FP64 worklist launches take 4 (UW_MODE_RESUME 6, in a batch 5) resident blocks
// of 128 threads per multiprocessor, and above which 7 (UW_LIST_MINB, `dense`): what 4 blocks hold.  A short
// worklist's time is its slowest columns' chain, which the spills of the smaller register cap lengthen by 4 to 7 %; a
// longer one at 4 blocks waits for a second wave.  Both caps, ms, at 148 multiprocessors (75,776 entries),
// entries / columns: 12 levels 74,392 / 254,439 6.3 and 6.6, 77,808 / 266,393 6.9 and 6.7; 30 levels 74,444 / 162,480
// 16.3 and 17.6, 77,922 / 170,113 19.7 and 18.0, of dry columns 74,726 / 395,925 18.9 and 19.7, 78,145 / 414,526 22.5
// and 20.2, of moist ones 74,665 / 111,410 16.0 and 17.1, 78,116 / 116,644 19.8 and 18.0; 63 levels 74,352 35.4 and
// 36.8, 77,871 40.7 and 37.6; 30 levels 458,106 101.9 and 98.8.  A plan with 64,197 and 65,410 entries in its two
// classes 46.2 and 51.6, with 85,469 and 87,106 61.1 and 59.4.  (At 137,000 to 151,000 entries, two waves at either
// cap, 4 blocks are 1 to 6 % faster from 30 levels on and up to 6 % slower below 20.)
UW_RULE int uw_short_list(int multiprocessors) { return 4 * 128 * multiprocessors; }
