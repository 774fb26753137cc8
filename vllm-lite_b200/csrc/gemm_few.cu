// bfloat16 products of up to 48 rows with float32 accumulation:  C[M, N] = A[M, K] * W[N, K]^T  (weights stored [out, in]), N up to 48 rows
// of W an SM.
//
// Such a product is over in three to twenty microseconds, and what takes the time is the way through it: the launch, the first bytes' way in, the
// K blocks one after another.  So a block owns 16, 32 or 48 rows of W (one tile an SM at most) and its eight warps take K's blocks of 64
// columns in turn, each with places of its own in shared memory that it fills itself by TMA, waits for and multiplies from (mma.sync,
// A's rows as the 16-row operand): no barrier, no empty places to hand back, and the copies' issue, 200 to 400 cycles each, runs in
// eight warps side by side (one warp issuing for all eight: 800 cycles a block of K, 12.5 us where this takes 3.6).  W's first blocks are
// asked for before the kernel in front has ended.  At the end the warps' sums are added in warp order in the ring's memory, and the
// activation of a gate/up product is applied there.
// Behind a small kernel, weights from memory (us; in brackets W's bytes alone), against the library's product: 32 rows: 512 x 2,048 3.0 / 4.3,
// 2,048 x 2,048 3.6 / 5.0 (1.3), 4,096 x 2,048 5.4 / 5.9 (2.6), 2,048 x 8,192 9.0 / 12.5 (5.1), 4,096 x 4,096 8.3 / 9.1 (5.1), 4,096 x 12,288
// 19.7 / 21.4 (15.4); 48 rows: 2,048 x 2,048 4.3 / 5.0, but 4,096 x 4,096 9.7 / 9.2; 64 rows: 2,048 x 2,048 5.2 / 5.4.  Against the weight-streaming
// kernel (gemm_bf16.cu), 16 rows: 2,048 x 2,048 2.9 / 4.8, 4,096 x 4,096 7.4 / 9.2, 6,144 x 4,096 10.2 / 10.9, 4,096 x 12,288 18.2 / 25.4, which
// reads A anew for every 16 rows of W; 8 rows: 3.7 / 3.2, 7.3 / 7.4, 10.0 / 9.2, 17.4 / 17.7.
#include "tc5.cuh"

namespace {
constexpr int BK = 64, WARPS = 8;
// NR rows of W (a tile), MT tiles of 16 rows of A; a warp has WS places for a block of W and AS for one of A.
template <int NR, int MT> struct Shape {
    static constexpr int ROWS = 16 * MT, WS = 3, AS = 2, W_BYTES = NR * 128, A_BYTES = ROWS * 128, RED_LD = NR + 1;
    static constexpr size_t RING = (size_t)WARPS * (WS * W_BYTES + AS * A_BYTES), RED = sizeof(float) * WARPS * ROWS * RED_LD;
    // More than half of an SM's memory: one block an SM.  Blocks that start while the kernel in front still holds most SMs would otherwise
    // gather on the first that are free (2,048 x 8,192 at 9 rows in a decode step: 37 us, 8 alone).
    static constexpr size_t USED = 1024 + (RING > RED ? RING : RED), SMEM = USED > 120 * 1024 ? USED : 120 * 1024;
    static_assert(SMEM <= 227 * 1024, "the ring does not fit");
};

__device__ __forceinline__ void ldsm4(unsigned (&r)[4], const void* smem) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(tc5::smem_u32(smem)));
}
__device__ __forceinline__ void mma(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <typename TO, int NR, int MT>
__global__ void __launch_bounds__(32 * WARPS)
gemm_few_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, TO* __restrict__ C, int M, int N, int K, int ldc,
                int swiglu, unsigned* err) {
    using S = Shape<NR, MT>;
    extern __shared__ unsigned char raw[];
    unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023);
    float* red = reinterpret_cast<float*>(ring);                  // [WARPS][ROWS][RED_LD], when the ring is done with
    __shared__ __align__(8) unsigned long long w_full[WARPS * S::WS], a_full[WARPS * S::AS];
    __shared__ int s_expired;
    pdl_launch_dependents();
    const int tid = threadIdx.x, warp = tc5::warp_number(), lane = tid & 31;
    unsigned long long* wf = w_full + warp * S::WS;               // a warp's own places, which it alone fills and reads
    unsigned long long* af = a_full + warp * S::AS;
    unsigned char* Ws = ring + warp * S::WS * S::W_BYTES;
    unsigned char* As = ring + WARPS * S::WS * S::W_BYTES + warp * S::AS * S::A_BYTES;
    if (lane == 0) {
        for (int i = 0; i < S::WS; ++i) tc5::mbar_init(&wf[i], 1);
        for (int i = 0; i < S::AS; ++i) tc5::mbar_init(&af[i], 1);
        tc5::mbar_fence_init();
    }
    if (tid == 0) s_expired = 0;
    __syncthreads();
    // K's blocks go to the warps in turn
    const int n0 = (int)blockIdx.x * NR, steps = ((K + BK - 1) / BK + WARPS - 1 - warp) / WARPS;
    const bool lead = tc5::elect_one();
    int iw = 0, sw = 0, ia = 0, sa = 0;                           // the next copies: number, place
    auto put_w = [&]() {
        if (iw < steps) {
            if (lead) {
                tc5::mbar_arrive_expect_tx(&wf[sw], S::W_BYTES);
                tc5::tma_load_2d(Ws + sw * S::W_BYTES, &map_w, (iw * WARPS + warp) * BK, n0, &wf[sw]);
            }
            ++iw;
            if (++sw == S::WS) sw = 0;
        }
    };
    auto put_a = [&]() {
        if (ia < steps) {
            if (lead) {
                tc5::mbar_arrive_expect_tx(&af[sa], S::A_BYTES);
                tc5::tma_load_2d(As + sa * S::A_BYTES, &map_a, (ia * WARPS + warp) * BK, 0, &af[sa]);
            }
            ++ia;
            if (++sa == S::AS) sa = 0;
        }
    };
#pragma unroll
    for (int i = 0; i < S::WS; ++i) put_w();                      // weights need not wait for the kernel before
    pdl_wait();
#pragma unroll
    for (int i = 0; i < S::AS; ++i) put_a();
    const int ar = lane & 15, ac = lane >> 4, br = (lane & 7) + ((lane >> 4) << 3), bc = (lane >> 3) & 1, g = lane >> 2, t2 = (lane & 3) * 2;
    float acc[MT][NR / 8][4];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NR / 8; ++j) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.f;
    bool ok = true;
    int done = 0, w = 0, wp = 0, a = 0, ap = 0;                   // the next block: number, places, parities
#pragma unroll 1
    for (; done < steps; ++done) {
        if (!tc5::warp_wait(&wf[w], wp) || !tc5::warp_wait(&af[a], ap)) { ok = false; break; }
        const unsigned char* wt = Ws + w * S::W_BYTES;
        const unsigned char* at = As + a * S::A_BYTES;
        unsigned x[4][MT][4], y[4][NR / 16][4];
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
#pragma unroll
            for (int i = 0; i < MT; ++i) ldsm4(x[kk][i], at + (16 * i + ar) * 128 + (((2 * kk + ac) ^ (ar & 7)) << 4));
#pragma unroll
            for (int j = 0; j < NR / 16; ++j) ldsm4(y[kk][j], wt + (16 * j + br) * 128 + (((2 * kk + bc) ^ (br & 7)) << 4));
        }
        __syncwarp();
        put_w();                                                  // (the fragments are in registers: the places are free)
        put_a();
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int i = 0; i < MT; ++i)
#pragma unroll
                for (int j = 0; j < NR / 16; ++j) {
                    mma(acc[i][2 * j], x[kk][i], y[kk][j][0], y[kk][j][1]);
                    mma(acc[i][2 * j + 1], x[kk][i], y[kk][j][2], y[kk][j][3]);
                }
        if (++w == S::WS) { w = 0; wp ^= 1; }
        if (++a == S::AS) { a = 0; ap ^= 1; }
    }
    if (!ok) {                                                    // copies that nobody waited for: waited for once more
        for (int i = done; i < iw; ++i) { tc5::warp_wait(&wf[w], wp); if (++w == S::WS) { w = 0; wp ^= 1; } }
        for (int i = done; i < ia; ++i) { tc5::warp_wait(&af[a], ap); if (++a == S::AS) { a = 0; ap ^= 1; } }
        if (lane == 0) s_expired = 1;
        if (lane == 0 && err) atomicOr(err, VL_DEV_WAIT_EXPIRED | VL_DEV_IN_GEMM_FEW);
    }
    __syncthreads();                                              // every warp's places are done with
    if (s_expired) return;
    float* r = red + warp * S::ROWS * S::RED_LD;
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NR / 8; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) r[(16 * i + g + 8 * (e >> 1)) * S::RED_LD + 8 * j + t2 + (e & 1)] = acc[i][j][e];
    __syncthreads();
    auto sum = [&](int m, int n) {                                // the warps' shares, in order
        float v = red[m * S::RED_LD + n];
#pragma unroll
        for (int q = 1; q < WARPS; ++q) v += red[(q * S::ROWS + m) * S::RED_LD + n];
        return v;
    };
    if (swiglu) {                                                 // blocks of 8 gate rows and their 8 up rows
        for (int i = tid; i < S::ROWS * NR / 2; i += 32 * WARPS) {
            const int m = i / (NR / 2), n = i % (NR / 2), at_g = n / 8 * 16 + n % 8;
            if (m < M && n0 + at_g + 8 < N) {
                const float gt = sum(m, at_g), up = sum(m, at_g + 8);
                C[(size_t)m * ldc + n0 / 2 + n] = from_f32<TO>(gt / (1.0f + expf(-gt)) * up);
            }
        }
    } else {
        for (int i = tid; i < S::ROWS * NR; i += 32 * WARPS) {
            const int m = i / NR, n = i % NR;
            if (m < M && n0 + n < N) C[(size_t)m * ldc + n0 + n] = from_f32<TO>(sum(m, n));
        }
    }
}

template <typename TO, int NR, int MT>
int launch(const bf16* A, const bf16* W, TO* C, int M, int N, int K, int lda, int ldw, int ldc, int swiglu, unsigned* err, cudaStream_t s) {
    using S = Shape<NR, MT>;
    static bool ready = false;                                    // per instantiation
    if (!ready) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_few_kernel<TO, NR, MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
        if (e != cudaSuccess) return (int)e;
        ready = true;
    }
    CUtensorMap map_a, map_w;
    int rc = tc5_make_map(&map_a, A, M, K, lda, S::ROWS);
    if (!rc) rc = tc5_make_map(&map_w, W, N, K, ldw, NR);
    if (rc) return rc;
    return vl_launch(gemm_few_kernel<TO, NR, MT>, dim3((N + NR - 1) / NR), dim3(32 * WARPS), S::SMEM, s, map_a, map_w, C, M, N, K, ldc, swiglu, err);
}
template <typename TO>
int pick(const bf16* A, const bf16* W, TO* C, int M, int N, int K, int lda, int ldw, int ldc, int swiglu, unsigned* err, int sms, cudaStream_t s) {
#define FEW(NR, MT) return launch<TO, NR, MT>(A, W, C, M, N, K, lda, ldw, ldc, swiglu, err, s)
    if (M > 32) FEW(16, 3);
    if (M > 16) {
        if (N <= 16 * sms) FEW(16, 2);
        if (N <= 32 * sms) FEW(32, 2);
        FEW(48, 2);
    }
    if (N <= 16 * sms) FEW(16, 1);
    if (N <= 32 * sms) FEW(32, 1);
    FEW(48, 1);
#undef FEW
}
}  // namespace

// swiglu: W holds blocks of 8 gate rows and their 8 up rows (N a multiple of 16), C is [M, N / 2].
extern "C" int vl_gemm_bf16_few(const void* A, const void* W, void* C, int out_dtype, int M, int N, int K, int lda, int ldw, int ldc, int swiglu,
                                int sms, unsigned* err, void* stream) {
    if (M <= 0 || N <= 0) return VL_OK;
    if (K <= 0 || lda < K || ldw < K || ldc < (swiglu ? N / 2 : N) || (swiglu && N % 16) || sms <= 0) return VL_ERR_ARGUMENT;
    if (M > 48 || K % 8 || lda % 8 || ldw % 8 || (((uintptr_t)A | (uintptr_t)W) & 15)) return VL_ERR_UNSUPPORTED;
    cudaStream_t s = (cudaStream_t)stream;
    if (out_dtype == VL_BF16) return pick((const bf16*)A, (const bf16*)W, (bf16*)C, M, N, K, lda, ldw, ldc, swiglu, err, sms, s);
    if (out_dtype == VL_F32) return pick((const bf16*)A, (const bf16*)W, (float*)C, M, N, K, lda, ldw, ldc, swiglu, err, sms, s);
    return VL_ERR_UNSUPPORTED;
}
