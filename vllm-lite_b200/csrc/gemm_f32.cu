// True float32 matrix product for the 32-bit path:  C[M,N] = A[M,K] * W[N,K]^T
// (a linear layer, y = x W^T with the weight stored [out, in]; no bias:
//  crates/model/src/components/attention/gqa/norm.rs:21-26 of the reference).
//
// Plain FFMA on CUDA cores: no tensor cores, no TF32, no split of K.  Every
// output element is the sum over k = 0..K-1 in that order, whatever M is and
// wherever the element lies in its tile, so a row's result is bit-for-bit the
// same whether it is computed alone or among thousands.
//
// What bounds it: for few rows the latency of the weights' way in, for many the multiply-adds.  Tiles of A and W come
// in by cp.async, a ring of STAGES steps of BK columns, so that a small product asks for everything at once and a large
// one never waits for memory between its steps; both stay k-fastest in shared memory, rows BK + 4 floats apart (a
// quarter warp's 16-byte reads then meet no bank twice), and a thread takes four values of k per read.  Measured, and beside it
// tiles of 64 x 64 without the ring, one step of 16 columns after another: 8 x 320 x 96 2.9 us and 8.0; 8 x 96 x 256 4.7 and 19.2; 1 x 4,096
// x 4,096 60 and 292; 64 x 6,144 x 4,096 178 and 453; 1,024 x 4,096 x 4,096 902 (38 TFLOP/s) and 1,508.
#include "common.cuh"

__device__ __forceinline__ void gf_copy(float* smem, const float* gmem, int bytes, bool wide) {   // the rest of 16 (4) bytes: zeros
    const unsigned dst = (unsigned)__cvta_generic_to_shared(smem);
    if (wide) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(gmem), "r"(bytes) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(gmem), "r"(bytes) : "memory");
}

// A block of (BM / TM) x (BN / TN) threads makes a BM x BN tile; thread (ty, tx) owns rows ty + i BM / TM and columns
// tx + j BN / TN.  VEC: 16-byte copies (rows on 16-byte boundaries), else 4-byte ones.
// SWIGLU: W's N rows are gates and ups (group = 0: N / 2 gates, then their ups; g > 0, a power of two: blocks of g gates, then their g ups) and C[M, N / 2]
// is silu(gate) * up: a tile takes BN / 2 gates and their ups, a thread both of a result, so that the pass over [M, N] and its launch,
// all there is to a small step's activation, go away (a tiny model's generation, 48 such launches fewer of 545: 3.01 -> 2.87 ms).
template <int BM, int BN, int TM, int TN, int BK, int STAGES, bool VEC, bool SWIGLU>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_f32_nt_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C,
                   int M, int N, int K, int lda, int ldw, int ldc, int group) {
    constexpr int TX = BN / TN, TY = BM / TM, NT = TX * TY, LD = BK + 4, STAGE = (BM + BN) * LD, STEP = VEC ? 4 : 1;
    extern __shared__ __align__(16) float sm[];
    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int steps = (K + BK - 1) / BK;
    auto w_row = [&](int r) {                                     // W's row of the tile's column r (N: none)
        if (!SWIGLU) return n0 + r;
        const int half = N / 2, up = r >= BN / 2, i = n0 / 2 + r - (up ? BN / 2 : 0);
        if (i >= half) return N;
        return i + (i & -group) + (up ? (group ? group : half) : 0);
    };
    auto fetch = [&](int step) {
        if (step < steps) {
            float* buf = sm + (step % STAGES) * STAGE;
            const int k0 = step * BK;
            for (int i = tid; i < (BM + BN) * (BK / STEP); i += NT) {
                const int r = i / (BK / STEP), kk = (i - r * (BK / STEP)) * STEP, k = k0 + kk;
                const bool of_a = r < BM;
                const int row = of_a ? m0 + r : w_row(r - BM);
                const bool in = row < (of_a ? M : N) && k < K;
                const float* src = of_a ? A : W;
                if (in) src += (size_t)row * (of_a ? lda : ldw) + k;
                gf_copy(buf + r * LD + kk, src, in ? 4 * min(STEP, K - k) : 0, VEC);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");      // (an empty group behind the end keeps the count)
    };
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) fetch(s);
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();                                          // this step has landed, and everyone is done with the one before
        fetch(step + STAGES - 1);
        const float* a = sm + (step % STAGES) * STAGE + ty * LD;
        const float* w = sm + (step % STAGES) * STAGE + (BM + tx) * LD;
#pragma unroll
        for (int k = 0; k < BK; k += 4) {
            float4 av[TM], wv[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) av[i] = *reinterpret_cast<const float4*>(a + i * TY * LD + k);
#pragma unroll
            for (int j = 0; j < TN; ++j) wv[j] = *reinterpret_cast<const float4*>(w + j * TX * LD + k);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    acc[i][j] = fmaf(av[i].x, wv[j].x, acc[i][j]);
                    acc[i][j] = fmaf(av[i].y, wv[j].y, acc[i][j]);
                    acc[i][j] = fmaf(av[i].z, wv[j].z, acc[i][j]);
                    acc[i][j] = fmaf(av[i].w, wv[j].w, acc[i][j]);
                }
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty + i * TY;
        if (m >= M) continue;
        if constexpr (SWIGLU) {
#pragma unroll
            for (int j = 0; j < TN / 2; ++j) {
                const int n = n0 / 2 + tx + j * TX;
                const float g = acc[i][j], u = acc[i][j + TN / 2];
                if (n < N / 2) C[(size_t)m * ldc + n] = g / (1.0f + expf(-g)) * u;
            }
        } else {
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const int n = n0 + tx + j * TX;
                if (n < N) C[(size_t)m * ldc + n] = acc[i][j];
            }
        }
    }
}

template <int BM, int BN, int TM, int TN, int BK, int STAGES>
static int launch_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, bool swiglu, int group,
                      cudaStream_t s) {
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM), block((BM / TM) * (BN / TN));
    const size_t smem = sizeof(float) * (size_t)STAGES * (BM + BN) * (BK + 4);
    const bool vec = lda % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
    if (grid.y > 65535) return VL_ERR_UNSUPPORTED;
    auto kernel = swiglu ? (vec ? gemm_f32_nt_kernel<BM, BN, TM, TN, BK, STAGES, true, true> : gemm_f32_nt_kernel<BM, BN, TM, TN, BK, STAGES, false, true>)
                         : (vec ? gemm_f32_nt_kernel<BM, BN, TM, TN, BK, STAGES, true, false> : gemm_f32_nt_kernel<BM, BN, TM, TN, BK, STAGES, false, false>);
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    return vl_launch(kernel, grid, block, smem, s, A, W, C, M, N, K, lda, ldw, ldc, group);
}

// The largest tile whose number fills the SMs, since a larger one reads its operands fewer times; else the smallest, which
// spreads a small product over the most SMs and has the shortest way through a step.
extern "C" int vl_gemm_f32_nt(const float* A, const float* W, float* C, int M, int N, int K,
                              int lda, int ldw, int ldc, int swiglu, int group, void* stream) {
    if (M <= 0 || N <= 0) return VL_OK;
    if (K <= 0 || lda < K || ldw < K || ldc < (swiglu ? N / 2 : N)) return VL_ERR_ARGUMENT;
    if (swiglu && (N % 2 || group < 0 || (group & (group - 1)) || (group > 0 && N / 2 % group))) return VL_ERR_ARGUMENT;
    cudaStream_t s = (cudaStream_t)stream;
    auto tiles = [&](int bm, int bn) { return (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn); };
    if (M > 64 && tiles(128, 128) >= 120) return launch_f32<128, 128, 8, 8, 32, 3>(A, W, C, M, N, K, lda, ldw, ldc, swiglu != 0, group, s);
    if (M > 16 && tiles(64, 64) >= 120) return launch_f32<64, 64, 4, 4, 32, 3>(A, W, C, M, N, K, lda, ldw, ldc, swiglu != 0, group, s);
    if (M > 16) return launch_f32<32, 32, 2, 2, 64, 3>(A, W, C, M, N, K, lda, ldw, ldc, swiglu != 0, group, s);
    return launch_f32<8, 32, 1, 2, 64, 4>(A, W, C, M, N, K, lda, ldw, ldc, swiglu != 0, group, s);
}
