// Which binaries a warp of a launch takes, and how many blocks that needs: plain
// integer arithmetic, written apart from the kernels so that it can be checked on
// the host at sizes no test can run.
#pragma once

#ifdef __CUDACC__
#define GBX_HD __host__ __device__ __forceinline__
#else
#define GBX_HD inline
#endif

namespace gbx {

// get_ll: a warp takes two binaries, a block of kLlBlock threads eight, and the
// grid covers any int num_bin in one round.  Counted in warps, of which there are
// at most 2^30, so that a binary and one more stride fit 32 unsigned bits; the
// threads, 16 num_bin, would leave them from 2^28 binaries on.
constexpr int kLlBlock = 128;

GBX_HD unsigned ll_first_binary(unsigned block, unsigned thread)
{
    return 2 * (block * (kLlBlock / 32) + (thread >> 5));
}

GBX_HD unsigned ll_stride(unsigned blocks) { return 2 * blocks * (kLlBlock / 32); }

GBX_HD unsigned ll_blocks(int num_bin)
{
    return (unsigned)(((long long)num_bin + 7) / 8);
}

// Row-major fill: kBulkWarps warps a block, each takes binaries first, first +
// stride, ...  64-bit: the step past the last binary of the largest batches leaves
// 32 bits.
constexpr int kBulkWarps = 2;

GBX_HD long long bulk_first_binary(unsigned block, unsigned warp) { return (long long)block * kBulkWarps + warp; }

GBX_HD long long bulk_stride(unsigned blocks) { return (long long)blocks * kBulkWarps; }

GBX_HD int bulk_blocks(int num_bin) { return num_bin / kBulkWarps + (num_bin % kBulkWarps != 0); }

// A few FP64 binaries: log2 of the blocks that work on each (0: tiles, one block or
// less), by the number of binaries, the window and the SMs; `fits(lc)` says whether a
// cluster of 2^lc blocks can be resident.  The measurements are at the dispatch.
template <typename Fits>
inline int cluster_log2(int num_bin, int N, int sms, Fits &&fits)
{
    if (N < 256) return 0;
    if (num_bin <= sms / 8 && fits(3)) return 3;
    if (num_bin <= 3 * sms / 8 && fits(2)) return 2;
    return 0;
}

}  // namespace gbx
