// What kernels whose CTAs walk over blocks and masked tiles share: the queue of blocks, and which pairs of a tile are visible.
#pragma once

#include "common.cuh"
#include "sm100_ptx.cuh"

namespace sntl {

// bit i: whether i < n
__device__ __forceinline__ uint32_t bits_below(int n) { return n <= 0 ? 0u : n >= 32 ? 0xffffffffu : (1u << n) - 1u; }

// Which of the 32 keys from key0 on the query at position pos sees (keys below `end` exist for it)
__device__ __forceinline__ uint32_t keys_seen(const AttnShape& s, int pos, int end, int key0)
{
    uint32_t seen = bits_below(end - key0);
    if (s.window > 0) seen &= ~bits_below(pos - s.window + 1 - key0) | bits_below(s.global_tokens - key0);
    return seen;
}
// Which of the 32 queries from position pos0 on see the key
__device__ __forceinline__ uint32_t queries_seeing(const AttnShape& s, int key, int pos0)
{
    uint32_t seen = key < s.Skv ? 0xffffffffu : 0u;
    if (s.causal) seen &= ~bits_below(key - pos0);
    if (s.window > 0 && key >= s.global_tokens) seen &= bits_below(key + s.window - pos0);
    return seen;
}

// The blocks that a CTA computes one after the other: its own, then blocks of the grid that have not started, which the block scheduler
// hands over on request (one is asked for when the last tile of a block is being staged).  Set-up, first loads and first products of
// a block so run under the end of the one before, and its code has been fetched.  Block number u of a CTA; each of kWarps warps
// reads the answer for it.
template <int kWarps> struct BlockQueue {
    alignas(16) uint4 answer[2];
    uint64_t full[2], empty[2];

    __device__ __forceinline__ void init()
    {
        for (int i = 0; i < 2; ++i) {
            ptx::mbar_init(&full[i], 1);
            ptx::mbar_init(&empty[i], kWarps);
        }
    }
    // by one thread; false: a wait gave up
    __device__ __forceinline__ bool ask(int u, volatile uint32_t* abort_flag)
    {
        if (u > 2 && !ptx::mbar_wait(&empty[u & 1], (((u - 1) >> 1) - 1) & 1, abort_flag, 20)) return false;
        ptx::mbar_arrive_expect_tx(&full[u & 1], 16);
        ptx::clc_try_cancel(&answer[u & 1], &full[u & 1]);
        return true;
    }
    // by a whole warp: block number u, or -1 where there is none
    __device__ __forceinline__ int get(int u, volatile uint32_t* abort_flag)
    {
        if (!ptx::mbar_wait_warp(&full[u & 1], ((u - 1) >> 1) & 1, abort_flag, 21)) return -1;
        const int block = ptx::warp_uniform(ptx::clc_first_block(&answer[u & 1]));
        ptx::fence_proxy_async_smem();
        __syncwarp();
        if ((threadIdx.x & 31) == 0) ptx::mbar_arrive(&empty[u & 1]);
        return block;
    }
};

}  // namespace sntl
