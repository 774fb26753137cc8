// The grouped form of the tcgen05 matrix product, for routed feed-forwards with many rows:
//     C[m, :] = A[m, :] * W[g(m)]^T,   rows sorted by group (moe.cu: vl_moe_align), W [G, N, K] stacked.
// csrc/gemm_tc5.cu and csrc/gemm_tc5_pair.cu lay the rows of A along the tensor core's 128 or 256 rows and
// the rows of W along its columns.  A group brings a few hundred rows or fewer, so half a tile would be padding
// and W would be read once for every 128 rows.  Here the operands change places: 256 rows of W are the rows of a
// tile, which a pair of SMs computes (tcgen05 cta_group::2, as in csrc/gemm_tc5_pair.cu), and up to 256 rows of A its
// columns, as many as the group has (in steps of 32).  A K block of a tile costs an SM 16 KB of W and up to 16 KB of A, which 256
// columns want in 512 cycles (half of what an SM takes in); with fewer columns, and while an expert's rows are few, W's way out of
// memory bounds the kernel.
//
// Tiles are taken in turn by all pairs (pair p the tiles p, p + pairs, ..), those of a group's rows of A innermost, then its
// rows of W, so that what runs at the same time shares its rows of W and of A in L2.  (Equal shares of neighbouring tiles, cut
// anywhere along K, were built and measured: every pair is then in a group of its own, nothing is shared, and 148 SMs
// that leave float32 pieces take 10 us for it: 104 us where this order takes 71.)
// 32 groups of 256 rows, 2,048 x 2,048 a gate/up: 98 us with 128 rows of A as the tile's rows -> 68 (1,011 TFLOP/s),
// 2,048 x 1,024: 50 -> 40; groups of 384 rows 163 (of unequal sizes, in a model) -> 88 and 78 -> 50.
//
// The epilogue can do what a routed feed-forward needs around its first product: multiply the float32
// sums of row m by row_scale[row_index[m]] (the expert weight on the input: W (s a) = s (W a)), and
// apply the gated activation to blocks of 8 gate and 8 up columns (act 0..2: C is [M, N / 2]) or, act 16, the
// square of max(v, 0) to every column of a plain W.
//
// Roles: warp 0 copies (TMA, 128-byte swizzle; an elected lane), warp 1 of the pair's first block issues the products,
// warps 2..9 are the epilogue: two groups of four warps, each takes every second chunk of 32 columns of the accumulator,
// turns it round through shared memory (a thread holds one row of W there, a row of C wants them side by side) and
// stores 16 bytes a thread.  Two accumulators in tensor memory: a tile's epilogue runs beside the next tile's products.
// Every wait on an mbarrier is bounded.
#include "tc5.cuh"

using namespace tc5;

namespace {
constexpr int BK = 64, UMMA_K = 16, ROWS = 128;              // rows of W a block
constexpr int COLS = 256;                                    // most rows of A a tile
constexpr unsigned W_BYTES = ROWS * BK * 2, A_BYTES = COLS / 2 * BK * 2, STAGE_BYTES = W_BYTES + A_BYTES;
constexpr int STAGES = 6, ACCS = 2;
constexpr int GROUPS = 2, NUM_THREADS = 64 + GROUPS * 128;
constexpr int MAX_EXPERTS = 1024;
constexpr int TOKEN_BOXES = 8;               // boxes of 16, 32 .. 128 rows of A
constexpr unsigned CHUNK_BYTES = 32 * 272;    // a group's chunk on its way: 32 rows of C x 128 bfloat16, 16 bytes of padding a row

enum { PLAIN = 0, SILU = 1, OTHER = 2 };     // the epilogue: C as it is; silu(gate) * up; what Args::act says

struct TokenMaps { CUtensorMap m[TOKEN_BOXES]; };

struct Args {
    int N, ldc, kb, n_tiles;                 // kb: K blocks; n_tiles: tiles of a group's rows of W
    int wide;                                // rows of C begin on 16-byte boundaries
    int act;                                 // OTHER: 1 max(g, 0) u, 2 capped swish, 16 square of max(v, 0)
    float alpha, limit, shift;
    int fine;                                // the activation's exponential: expf, else __expf
    const int* starts;                       // first row of every group, [groups + 1]
    int groups;
    const int* row_index;
    const float* row_scale;
    unsigned* err;
};

struct Tables { int tile[MAX_EXPERTS + 1], row[MAX_EXPERTS + 1]; };       // tiles of the groups before; first row
struct Tile { int n0, wrow, t0, rows, T; };

__device__ __forceinline__ int tiles_of(int rows) { return (rows + COLS - 1) / COLS; }
__device__ __forceinline__ int columns_of(int rows) {        // of each of a group's tiles
    const int nt = tiles_of(rows);
    return nt ? ((rows + nt - 1) / nt + 31) & ~31 : 32;
}
__device__ __forceinline__ Tile tile_at(const Args& f, const Tables& tb, int tile, int& e) {
    while (tb.tile[e + 1] <= tile) ++e;                      // tiles come in order; groups without rows have none
    Tile t;
    const int local = tile - tb.tile[e], rows = tb.row[e + 1] - tb.row[e], nt = tiles_of(rows);
    t.T = columns_of(rows);
    const int n = local / nt;
    t.n0 = n * 2 * ROWS;
    t.wrow = e * f.N + t.n0;
    t.t0 = tb.row[e] + (local - n * nt) * t.T;
    t.rows = min(t.T, tb.row[e + 1] - t.t0);
    return t;
}

__device__ __forceinline__ void group_sync(int group) { asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory"); }
// the same, and whether any thread of the group says so
__device__ __forceinline__ bool group_any(int group, bool mine) {
    unsigned any;
    asm volatile("{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n bar.red.or.pred q, %2, 128, p;\n selp.u32 %0, 1, 0, q;\n}"
                 : "=r"(any) : "r"((unsigned)mine), "r"(1 + group) : "memory");
    return any != 0;
}

__device__ __forceinline__ float exp_of(float x, const Args& f) { return f.fine ? expf(x) : __expf(x); }
__device__ __forceinline__ float silu_gated(float g, float u, const Args& f) { return g / (1.0f + exp_of(-g, f)) * u; }
// the other gated activations of csrc/activation.cu: 1 max(g, 0) u, 2 capped swish
__device__ __forceinline__ float other_gated(float g, float u, const Args& f) {
    if (f.act == 1) return fmaxf(g, 0.f) * u;
    if (f.limit > 0.f) { g = fminf(g, f.limit); u = fminf(fmaxf(u, -f.limit), f.limit); }
    return g / (1.0f + exp_of(-f.alpha * g, f)) * (u + f.shift);
}

// Rows of `BYTES` bytes from shared memory to rows of C: a thread moves 16 bytes, neighbours side by side.
// `left` = columns of C from this block's first one to the end of the row.
template <int BYTES, int STRIDE>
__device__ __forceinline__ void copy_rows(const unsigned char* turn, bf16* dst, int ldc, int valid, int left, int wide, int tid) {
    constexpr int SEGS = BYTES / 16;
    const int seg = tid % SEGS;
#pragma unroll
    for (int i = 0; i < 32 * SEGS / 128; ++i) {
        const int row = tid / SEGS + i * (128 / SEGS);
        if (row >= valid) continue;
        const uint4 v = *reinterpret_cast<const uint4*>(turn + row * STRIDE + seg * 16);
        bf16* p = dst + (size_t)row * ldc + seg * 8;
        if (wide && seg * 8 + 8 <= left) {
            *reinterpret_cast<uint4*>(p) = v;
        } else {
            const bf16* s = reinterpret_cast<const bf16*>(turn + row * STRIDE + seg * 16);
            for (int j = 0; j < 8; ++j)
                if (seg * 8 + j < left) p[j] = s[j];
        }
    }
}

// One chunk: this thread's row of W (quarter * 32 + lane of the block's 128) against 32 rows of C, of which `valid` are
// real.  C's first row begins at crow; the block's first row of W is n0.
template <int ACT>
__device__ __forceinline__ void store_chunk(const unsigned (&v)[32], unsigned char* turn, bf16* crow, const Args& f, int valid, int n0,
                                            int quarter, int lane, int tid, int group) {
    group_sync(group);                                       // the chunk before has left shared memory
    if (ACT == SILU || (ACT == OTHER && f.act < 16)) {
        // rows of W in blocks of 8 gate and 8 up rows: lanes 8 apart exchange, each forms every second row of C
        const int up = (lane >> 3) & 1;
        bf16* dst = reinterpret_cast<bf16*>(turn + up * 144) + quarter * 16 + (lane >> 4) * 8 + (lane & 7);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const float a = __uint_as_float(v[2 * j]), b = __uint_as_float(v[2 * j + 1]);
            const float other = __shfl_xor_sync(0xffffffffu, up ? a : b, 8);
            const float g = up ? other : a, u = up ? b : other;
            dst[j * 144] = __float2bfloat16_rn(ACT == SILU ? silu_gated(g, u, f) : other_gated(g, u, f));
        }
        group_sync(group);
        copy_rows<128, 144>(turn, crow + n0 / 2, f.ldc, valid, (f.N - n0) / 2, f.wide, tid);
    } else {
        bf16* dst = reinterpret_cast<bf16*>(turn) + quarter * 32 + lane;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            float o = __uint_as_float(v[i]);
            if (ACT == OTHER) { o = fmaxf(o, 0.f); o *= o; }
            dst[i * 136] = __float2bfloat16_rn(o);
        }
        group_sync(group);
        copy_rows<256, 272>(turn, crow + n0, f.ldc, valid, f.N - n0, f.wide, tid);
    }
}
}  // namespace

template <int ACT>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_tc5_grouped_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ TokenMaps maps_a, bf16* __restrict__ C,
                        const __grid_constant__ Args f) {
    extern __shared__ unsigned char grouped_smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)grouped_smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) unsigned long long full_bar[STAGES], empty_bar[STAGES], acc_full_bar[ACCS], acc_empty_bar[ACCS];
    __shared__ __align__(16) unsigned char turn_all[GROUPS][CHUNK_BYTES];
    __shared__ unsigned tmem_base_slot;
    __shared__ int failed;
    __shared__ Tables tb;
    const int warp = warp_number(), lane = threadIdx.x & 31;
    const int rank = (int)cluster_rank(), pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;

    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) { mbar_init(&full_bar[i], 1); mbar_init(&empty_bar[i], 1); }
        for (int i = 0; i < ACCS; ++i) { mbar_init(&acc_full_bar[i], 1); mbar_init(&acc_empty_bar[i], 2 * GROUPS * 4); }
        mbar_fence_init();
        failed = 0;
    }
    // Never launched as a programmatic dependent (see the launcher); the order is kept all the same: nothing of the SM pair is
    // taken while earlier kernels run.
    pdl_wait();
    pdl_launch_dependents();
    if (warp == 1) alloc_pair(&tmem_base_slot, ACCS * COLS);
    if (warp == 2) {
        int tiles = 0;
        for (int e0 = 0; e0 < f.groups; e0 += 32) {
            const int e = e0 + lane;
            const int row = e < f.groups ? f.starts[e] : 0, mine = e < f.groups ? tiles_of(f.starts[e + 1] - row) * f.n_tiles : 0;
            int x = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (e < f.groups) { tb.tile[e] = tiles + x - mine; tb.row[e] = row; }
            tiles += __shfl_sync(0xffffffffu, x, 31);
        }
        if (lane == 0) { tb.tile[f.groups] = tiles; tb.row[f.groups] = f.starts[f.groups]; }
    }
    tc5_fence_before();
    __syncthreads();
    cluster_sync();                                          // the other block's mbarriers exist before anything arrives there
    tc5_fence_after();
    const unsigned tmem_base = tmem_base_slot;
    const int tiles = tb.tile[f.groups];

    if (warp == 0) {                                         // ---- TMA producer ----
        const bool lead = elect_one();
        int s = 0, e = 0;
        unsigned phase = 1;                                  // of the stage's next "free": the first round finds all free
        bool ok = true;
        for (int tile = pair; tile < tiles && ok; tile += pairs) {
            const Tile t = tile_at(f, tb, tile, e);
            const int own = t.T / 2;                         // rows of A that this block brings
            const CUtensorMap* map_a = &maps_a.m[own / 16 - 1];
            const unsigned bytes = W_BYTES + (unsigned)(own * BK * 2);
            for (int kb = 0; kb < f.kb; ++kb) {
                if (!warp_wait(&empty_bar[s], phase)) {
                    if (lead) atomicOr(&failed, 1);
                    ok = false;
                    break;
                }
                if (lead) {
                    if (rank == 0) mbar_arrive_expect_tx(&full_bar[s], 2 * bytes);       // the bytes of both blocks
                    const unsigned bar = map_to_rank(smem_u32(&full_bar[s]), 0);
                    unsigned char* st = smem + (size_t)s * STAGE_BYTES;
                    tma_load_2d_pair(st, &map_w, kb * BK, t.wrow + rank * ROWS, bar);
                    tma_load_2d_pair(st + W_BYTES, map_a, kb * BK, t.t0 + rank * own, bar);
                }
                if (++s == STAGES) { s = 0; phase ^= 1u; }
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {                                     // ---- MMA issuer of the pair ----
            const bool lead = elect_one();
            int s = 0, e = 0, i = 0;
            unsigned phase = 0;
            bool ok = true;
            for (int tile = pair; tile < tiles && ok; tile += pairs, ++i) {
                const unsigned idesc = make_idesc(2 * ROWS, tile_at(f, tb, tile, e).T);
                const int acc = i % ACCS;
                if (i >= ACCS && !warp_wait(&acc_empty_bar[acc], (unsigned)((i / ACCS - 1) & 1))) {
                    if (lead) atomicOr(&failed, 2);
                    break;
                }
                tc5_fence_after();
                const unsigned tmem_c = tmem_base + (unsigned)(acc * COLS);
                for (int kb = 0; kb < f.kb; ++kb) {
                    if (!warp_wait(&full_bar[s], phase)) {
                        if (lead) atomicOr(&failed, 4);
                        ok = false;
                        break;
                    }
                    tc5_fence_after();
                    const unsigned char* st = smem + (size_t)s * STAGE_BYTES;
                    const unsigned long long wdesc = make_smem_desc(st), adesc = make_smem_desc(st + W_BYTES);
                    if (lead) {
#pragma unroll
                        for (int k = 0; k < BK / UMMA_K; ++k)
                            mma_pair(tmem_c, wdesc + (unsigned long long)(k * 2), adesc + (unsigned long long)(k * 2), idesc,
                                     (kb > 0 || k > 0) ? 1u : 0u);
                        commit_pair(&empty_bar[s]);          // both blocks' stages are free once these have read them
                        if (kb + 1 == f.kb) commit_pair(&acc_full_bar[acc]);
                    }
                    if (++s == STAGES) { s = 0; phase ^= 1u; }
                }
            }
        }
    } else {                                                 // ---- epilogue: warps 2..9 ----
        const int quarter = warp & 3, group = (warp - 2) >> 2, tid = threadIdx.x - 64 - group * 128;
        unsigned char* turn = turn_all[group];
        int e = 0, i = 0;
        for (int tile = pair; tile < tiles; tile += pairs, ++i) {
            const Tile t = tile_at(f, tb, tile, e);
            const int acc = i % ACCS;
            if (group_any(group, !mbar_wait_bounded(&acc_full_bar[acc], (unsigned)((i / ACCS) & 1)))) {
                atomicOr(&failed, 8);                        // the whole group leaves
                break;
            }
            tc5_fence_after();
            for (int c0 = group * 32; c0 < t.T; c0 += GROUPS * 32) {
                unsigned v[32];
                tc5_ld32(tmem_base + ((unsigned)(quarter * 32) << 16) + (unsigned)(acc * COLS + c0), v);
                const int valid = min(32, t.rows - c0);
                if (f.row_scale) {
                    float scale = 0.f;
                    if (lane < valid) {
                        const int p = f.row_index ? f.row_index[t.t0 + c0 + lane] : t.t0 + c0 + lane;
                        scale = p >= 0 ? f.row_scale[p] : 0.f;
                    }
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        v[j] = __float_as_uint(__uint_as_float(v[j]) * __shfl_sync(0xffffffffu, scale, j));
                }
                store_chunk<ACT>(v, turn, C + (size_t)(t.t0 + c0) * f.ldc, f, valid, t.n0 + rank * ROWS, quarter, lane, tid, group);
            }
            tc5_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_remote(map_to_rank(smem_u32(&acc_empty_bar[acc]), 0));      // this warp has read the accumulator
        }
    }
    tc5_fence_before();
    __syncthreads();
    cluster_sync();                                          // neither block frees or leaves while the other may still read it
    tc5_fence_after();
    if (warp == 1) dealloc_pair(tmem_base, ACCS * COLS);
    if (threadIdx.x == 0 && failed && f.err)
        atomicOr(f.err, VL_DEV_WAIT_EXPIRED | VL_DEV_IN_GEMM_GROUPED | ((unsigned)failed << VL_DEV_ROLE_SHIFT));
}

// ---- host side -------------------------------------------------------------------------------
namespace {
int pair_count() {
    static int n = 0;
    if (!n) {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
        n = sms < 2 ? 1 : sms / 2;
    }
    return n;
}

template <int ACT>
int launch_grouped(const CUtensorMap& map_w, const TokenMaps& maps_a, bf16* C, const Args& f, cudaStream_t s) {
    auto kern = gemm_tc5_grouped_kernel<ACT>;
    const size_t smem = (size_t)STAGES * STAGE_BYTES + 1024;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * pair_count());
    cfg.blockDim = dim3(NUM_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    // The cluster attribute and no other: csrc/gemm_tc5_pair.cu says why a kernel of paired blocks is never
    // launched as a programmatic dependent.
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, kern, map_w, maps_a, C, f);
}
}  // namespace

// A [M, K] (the rows sorted by group; group e has the rows starts[e] .. starts[e + 1], starts[G] <= M), W [G, N, K],
// C [M, N] or, with a gated act, [M, N / 2]; bfloat16.  fine: the gated activations' exponential is the full one (2,048 tokens through 32 experts,
// eight layers: 4,800 us with either).  row_scale (optional) is indexed by row_index[m] (row_index null: by m).
extern "C" int vl_gemm_bf16_tc5_grouped(const void* A, const void* W, void* C, int M, int N, int K, int G,
                                        const int* starts, const int* row_index, const float* row_scale,
                                        int act, float alpha, float limit, float shift, int fine, unsigned* err, void* stream) {
    if (M <= 0 || N <= 0) return VL_OK;
    if (K <= 0 || K % 8 || G <= 0 || G > MAX_EXPERTS || !starts) return VL_ERR_UNSUPPORTED;
    const bool gated = act >= 0 && act < 16;                 // 16: a function of one argument on a plain W
    if (act < -1 || (act > 2 && act != 16) || (gated && N % 16)) return VL_ERR_ARGUMENT;
    if ((long long)G * N >= (1ll << 31) || ((long long)M / COLS + G) * ((N + 2 * ROWS - 1) / (2 * ROWS)) >= (1ll << 30)) return VL_ERR_UNSUPPORTED;
    if (((uintptr_t)A | (uintptr_t)W) & 15) return VL_ERR_UNSUPPORTED;
    Args f = {};
    f.N = N; f.ldc = gated ? N / 2 : N;
    f.kb = (K + BK - 1) / BK; f.n_tiles = (N + 2 * ROWS - 1) / (2 * ROWS);
    f.wide = ((uintptr_t)C & 15) == 0 && f.ldc % 8 == 0;
    f.act = act; f.alpha = alpha; f.limit = limit; f.shift = shift; f.fine = fine;
    f.starts = starts; f.groups = G; f.row_index = row_index; f.row_scale = row_scale;
    f.err = err;
    CUtensorMap map_w;
    TokenMaps maps_a;
    int rc = tc5_make_map(&map_w, W, G * N, K, K, ROWS);
    for (int i = 0; i < TOKEN_BOXES && !rc; ++i) rc = tc5_make_map(&maps_a.m[i], A, M, K, K, 16 * (i + 1));
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    if (act < 0) return launch_grouped<PLAIN>(map_w, maps_a, (bf16*)C, f, s);
    return act == 0 ? launch_grouped<SILU>(map_w, maps_a, (bf16*)C, f, s) : launch_grouped<OTHER>(map_w, maps_a, (bf16*)C, f, s);
}
