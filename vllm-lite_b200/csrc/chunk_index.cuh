// Portions of a step cut into chunks of a fixed number of tokens, counted from each portion's start: which chunk of the launch is
// whose.  Requests that bring fewer than `least` tokens have no chunks (a walk token by token serves them).
#pragma once

__device__ __forceinline__ int ci_chunks_of(const int* cu, int b, int B, int tokens, int least) {
    const int n = b < B ? cu[b + 1] - cu[b] : 0;
    return n >= least ? (n + tokens - 1) / tokens : 0;
}
// Chunk number `idx` of the launch: request b and its chunk c.  Called by whole warps; false beyond the last chunk.
__device__ __forceinline__ bool ci_find(const int* cu, int B, int tokens, int least, int idx, int* b, int* c) {
    const int lane = threadIdx.x & 31;
    int base = 0;
    for (int b0 = 0; b0 < B; b0 += 32) {
        const int k = ci_chunks_of(cu, b0 + lane, B, tokens, least);
        int x = k;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        const int total = __shfl_sync(0xffffffffu, x, 31);
        if (idx < base + total) {
            const int src = __ffs(__ballot_sync(0xffffffffu, base + x > idx)) - 1;
            *b = b0 + src;
            *c = idx - base - __shfl_sync(0xffffffffu, x - k, src);
            return true;
        }
        base += total;
    }
    return false;
}
__device__ __forceinline__ int ci_first(const int* cu, int b, int tokens, int least) {     // chunks of the requests before b; by whole warps
    int k = 0;
    for (int i = threadIdx.x & 31; i < b; i += 32) k += ci_chunks_of(cu, i, b, tokens, least);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) k += __shfl_xor_sync(0xffffffffu, k, o);
    return k;
}
// The request with the `rank`-th most tokens (ties: the lower index), so that a launch that walks every request from chunk to chunk begins
// the longest walks first and the short ones fill up what they leave (more than 32 requests: in their own order).  By whole warps.
__device__ __forceinline__ int ci_by_length(const int* cu, int B, int rank) {
    if (B > 32) return rank;
    const int lane = threadIdx.x & 31, n = lane < B ? cu[lane + 1] - cu[lane] : -1;
    int ahead = 0;
    for (int j = 0; j < B; ++j) {
        const int o = __shfl_sync(0xffffffffu, n, j);
        ahead += (o > n || (o == n && j < lane)) ? 1 : 0;
    }
    return __ffs(__ballot_sync(0xffffffffu, lane < B && ahead == rank)) - 1;
}
