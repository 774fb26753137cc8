// bfloat16 decode attention over the paged cache as a persistent, warp-specialised stream:
// -DFA_HD=64 or 128.  The function and the partial-result layout are those of vl_flash_decode
// (csrc/flash_attn.cu): a token at position p reads the keys lo..p of its request,
//     s_j = (q . k_j) * scale;  p = softmax_j(s);  o = sum_j p_j v_j,
// on as many blocks as there are SMs.
//
// A decode step is bound by one read of the keys and values, so every block reads the same number of key tiles: the tiles of
// all (token, KV head) items, one item behind the other, are cut into equal runs, whatever lengths the requests have and
// whatever context the launch was sized for.  A block's run is a few pieces of items; an item that lies in one block's run is
// finished there, the others leave unnormalised partial results with their maximum and sum, which the block that arrives
// last at the item's counter adds up in the order of the pieces.  No run is shorter than an item's pieces in the scratch
// allow (S of them).  Where the cuts lie, and with them the last bits of a result, follows from the lengths of all requests, the number of
// blocks and S: the same request beside others, or in a step sized for another bound, may differ by rounding.
// (Dealing out (token, KV head, chunk of 1,024 keys) items in turn leaves half of the blocks without work where requests are shorter
// than the bound: 64 requests of 400 to 1,500 keys, bound 2,048, 8 KV heads of 128: 78.5 us with the merge's launch, 55.9 in equal runs.)
//   warp 4   producer: looks up the pages of a piece and copies its K and V rows, 64 keys a
//        stage, by TMA boxes (cp.async.bulk.tensor.3d, 128-byte swizzle, one box per page: its blocks
//        of 64 columns one after the other) into a ring of stages that runs on across work items; it also brings the item's
//        query rows (bulk copies) and its description into one of two slots.  The producer runs
//        ahead of the arithmetic by the depth of the ring, so the start-up of the next item is
//        hidden behind the stream of this one;
//   warps 0..3   consumers: per stage each warp takes 16 of the 64 keys (mma.sync m16n8k16, the query
//        heads of the KV head as rows), keeps its own running maximum, sum and output; at the end of
//        a piece the four are merged through shared memory in warp order and written as the item's
//        result or as a partial one.
// Keys outside the item's range are masked by position; pages outside it, or that the block table
// does not hold, are fetched from beyond the end of the tensor (zeros); the values of keys
// behind the request's last one are cleared as fragments (another request's leftovers may be anything).
// Every wait on an mbarrier is bounded; when one expires the block's consumers give up together, the block records
// VL_DEV_WAIT_EXPIRED and stops.  It has then not counted its pieces: whoever clears the error zeroes the counters too.
#include "tc5.cuh"

#ifndef FA_HD
#define FA_HD 128
#endif

using namespace tc5;

namespace {
constexpr int HD = FA_HD;
static_assert(HD == 64 || HD == 128, "this kernel is built for head sizes 64 and 128");
constexpr int BN = 64, CB = HD / 64, KSTEPS = HD / 16, DTILES = HD / 8;
constexpr int ROWS = 16;                               // query heads per work item (rows of the tensor-core tile)
constexpr int CONSUMERS = 4, NTHREADS = 32 * (CONSUMERS + 1);
constexpr unsigned ROW_BYTES = 128;
constexpr unsigned KV_BYTES = BN * HD * 2;             // K (or V) of a stage: CB blocks of [64 rows][128 bytes]
constexpr unsigned STAGE_BYTES = 2 * KV_BYTES;
constexpr int NST = HD == 128 ? 5 : 8;                 // stages in the ring
constexpr int QLD = HD + 8;                            // padded query row (elements)
constexpr unsigned Q_BYTES = ROWS * QLD * 2;
constexpr int OLD = HD + 4;                            // padded row of the merge buffer (floats)
constexpr unsigned MERGE_BYTES = CONSUMERS * ROWS * OLD * 4;
constexpr unsigned SMEM_BYTES = NST * STAGE_BYTES + MERGE_BYTES + 2 * Q_BYTES + 256;

struct ItemInfo {                                      // what the producer tells the consumers about a piece
    int tok, out_row, h0, nvalid, c0, c1, piece, pieces, counter;   // out_row: the token's number within the launch; nvalid 0: the end
};

__device__ __forceinline__ void ldmatrix_x4(unsigned (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(unsigned (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma16816(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float exp2_mufu(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<unsigned*>(&v);
}
__device__ __forceinline__ void bulk_copy_g2s(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void consumer_barrier() { asm volatile("bar.sync 1, 128;" ::: "memory"); }
// The same, and whether all four warps still have what they waited for: one whose wait ran out takes the others along, so that none
// stays at a barrier that it does not reach.
__device__ __forceinline__ bool consumers_agree(bool ok) {
    int all;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbar.red.and.pred q, 1, 128, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
                 : "=r"(all) : "r"((int)ok) : "memory");
    return all != 0;
}
}  // namespace

extern "C" __global__ void __launch_bounds__(NTHREADS, 1)
flash_decode_tma_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                        const bf16* __restrict__ q, int q_stride,
                        const int* __restrict__ block_table, int max_blocks,
                        const int* __restrict__ req_index, const int* __restrict__ positions,
                        int T, int nq, int nkv, int page_size, int num_pages, float scale_log2, int window,
                        int bound, int S, float* __restrict__ part_acc, float* __restrict__ part_ml, unsigned* err,
                        const int* __restrict__ token_index, bf16* __restrict__ out, int* arrivals, const float* __restrict__ sinks, int settled) {
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* ring = smem;                                            // [NST][K | V]
    float* sO = reinterpret_cast<float*>(smem + NST * STAGE_BYTES);        // [4][16][OLD]
    bf16* Qs = reinterpret_cast<bf16*>(smem + NST * STAGE_BYTES + MERGE_BYTES);   // [2][16][QLD]
    unsigned char* tail = smem + NST * STAGE_BYTES + MERGE_BYTES + 2 * Q_BYTES;
    unsigned long long* full = reinterpret_cast<unsigned long long*>(tail);       // [NST]
    unsigned long long* empty = full + NST;                                       // [NST]
    unsigned long long* q_full = empty + NST;                                     // [2]
    unsigned long long* q_empty = q_full + 2;                                     // [2]
    ItemInfo* info = reinterpret_cast<ItemInfo*>(q_empty + 2);                    // [2]
    __shared__ float s_m[CONSUMERS][ROWS], s_l[CONSUMERS][ROWS];
    __shared__ int failed, s_last[2], s_scan[NTHREADS / 32], s_most, s_z, s_before;
    __shared__ ItemInfo s_partial[2];                    // the pieces of items that other blocks share: the run's first and last
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_launch_dependents();
    if (smem_u32(smem) & 1023u) {                        // (uniform) never expected; the tiles would be misread
        if (tid == 0 && err) atomicOr(err, VL_DEV_WAIT_EXPIRED);
        return;
    }
    if (tid == 32 * CONSUMERS) {                         // both maps on their way before the first copy asks for them
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_k) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_v) : "memory");
    }
    if (tid == 0) {
        for (int i = 0; i < NST; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], CONSUMERS); }
        for (int i = 0; i < 2; ++i) { mbar_init(&q_full[i], 1); mbar_init(&q_empty[i], CONSUMERS); }
        mbar_fence_init();
        failed = 0;
        s_most = 0;
        s_z = T;
        s_before = 0;
        s_partial[0].nvalid = s_partial[1].nvalid = 0;
    }
    for (int i = tid; i < 2 * ROWS * QLD / 2; i += NTHREADS) reinterpret_cast<unsigned*>(Qs)[i] = 0u;   // rows no head uses stay zero
    fence_proxy_async_smem();
    __syncthreads();
    const int grp = nq / nkv;
    const int htiles = (grp + ROWS - 1) / ROWS;
    const int ny = nkv * htiles;
    if (!settled) pdl_wait();                            // a kernel before this one may be writing the step's description
    // the keys [lo, n) of token z (its number within the launch): none for a padded place or a position beyond the bound
    auto keys_of = [&](int z, int* tok, int* lo) -> int {
        const int k = token_index ? token_index[z] : z, pos = positions[k];
        if (tok) *tok = k;
        *lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
        return pos >= 0 && pos < bound ? pos + 1 : 0;
    };
    // Where this block's run lies, from the step's description alone (which, `settled`, may be read before the wait for the kernel before): the
    // number of tiles, the longest item, and the token in which the run begins.  A round is a token a thread; what the first rounds found is kept.
    constexpr int KEPT = 2;
    int total = 0, kept = 0, own[KEPT] = {0, 0}, upto[KEPT] = {0, 0};
    auto round = [&](int z0, int& n) -> int {            // tiles of token z0 + tid; tiles of the tokens up to it, in this round
        int lo = 0;
        const int z = z0 + tid, keys = z < T ? keys_of(z, nullptr, &lo) : 0, most = keys > 0 ? (keys - 1) / BN - lo / BN + 1 : 0;
        n = ny * most;
        int x = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int y = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x += y; }
        const int longest = __reduce_max_sync(0xffffffffu, most);
        if (lane == 0) atomicMax(&s_most, longest);
        if (lane == 31) s_scan[warp] = x;
        __syncthreads();
        int all = 0;
        for (int w = 0; w < NTHREADS / 32; ++w) { if (w == warp) x += all; all += s_scan[w]; }
        total += all;
        __syncthreads();
        return total - all + x;
    };
    for (int z0 = 0, r = 0; z0 < T; z0 += NTHREADS, ++r) {
        int n;
        const int u = round(z0, n);
        if (r == 0) { own[0] = n; upto[0] = u; kept = total; }
        if (r == 1) { own[1] = n; upto[1] = u; kept = total; }
    }
    // (a run as long as the longest item leaves no item in more than two runs; S > 1)
    const int grid = gridDim.x, all_tiles = total;
    const int per = max(max((all_tiles + grid - 1) / grid, 1), (s_most + S - 2) / (S - 1));
    const int first = (int)min((long long)blockIdx.x * per, (long long)all_tiles), last = (int)min((long long)first + per, (long long)all_tiles);
    total = kept;                                        // the rounds that were not kept, once more
    for (int z0 = 0, r = 0; z0 < T; z0 += NTHREADS, ++r) {
        int n = r == 0 ? own[0] : own[1], u = r == 0 ? upto[0] : upto[1];
        if (r >= KEPT) u = round(z0, n);
        if (u > first && u - n <= first) { s_z = z0 + tid; s_before = u - n; }
    }
    __syncthreads();

    if (warp == CONSUMERS) {                             // ---- producer (whole warp) ----
        const int box_rows = page_size < BN ? page_size : BN, nbox = BN / box_rows;
        const int beyond = num_pages * nkv * page_size;  // a row coordinate past the tensor: zeros
        int stage_it = 0;                                // stages issued so far, over all pieces
        int z = s_z, before = s_before;
        bool ok = true, bad_page = false;                // (flagged at the end: nothing is written before the wait)
        struct Piece { ItemInfo ii; const int* table; int stop, kvh, row; };
        // lane b < nbox owns box b of every key tile: the cache row of the box's first key, looked up one tile ahead of its use
        auto lookup = [&](const Piece& p, int st) -> int {
            if (lane >= nbox || st > (p.ii.c1 - 1) / BN) return beyond;
            const int key = st * BN + lane * box_rows;
            if (key >= p.ii.c1 || key + box_rows - 1 < p.ii.c0) return beyond;
            const int blk = key / page_size;
            const int page = blk < max_blocks ? p.table[blk] : -1;
            if (page < 0 || page >= num_pages) {
                bad_page = true;
                return beyond;
            }
            return (page * nkv + p.kvh) * page_size + (key - blk * page_size);
        };
        // the piece that begins with tile `at`: its item's share of this run (three reads one behind the other)
        auto piece_at = [&](int at) -> Piece {
            Piece p;
            int tok = 0, lo = 0, keys = 0, tz = 0;
            while (at < last && z < T) {
                keys = keys_of(z, &tok, &lo);
                tz = keys > 0 ? (keys - 1) / BN - lo / BN + 1 : 0;
                if (at < before + ny * tz) break;
                before += ny * tz;
                ++z;
            }
            p.ii.nvalid = 0;
            if (at >= last || z >= T) return p;          // the end of the run
            const int y = (at - before) / tz, start = before + y * tz;                // the item's first tile
            const int kvh = y / htiles, htile = y - kvh * htiles;
            p.stop = min(last, start + tz);
            p.kvh = kvh;
            p.table = block_table + (size_t)req_index[tok] * max_blocks;
            p.ii.tok = tok; p.ii.out_row = z;
            p.ii.h0 = kvh * grp + htile * ROWS;
            p.ii.nvalid = min(ROWS, grp - htile * ROWS);
            const int tile0 = lo / BN - start;           // + a tile's number in the launch = its number in the request
            p.ii.c0 = max((at + tile0) * BN, lo);
            p.ii.c1 = min((p.stop + tile0) * BN, keys);
            p.ii.piece = (int)blockIdx.x - start / per;
            p.ii.pieces = (start + tz - 1) / per - start / per + 1;
            p.ii.counter = z * ny + y;
            p.row = lookup(p, p.ii.c0 / BN);
            return p;
        };
        Piece cur = piece_at(first), nxt = cur;
        pdl_wait();                                      // q and the cache are written by the kernel before
        for (int n = 0;; ++n) {
            const int ib = n & 1, nvalid = cur.ii.nvalid;
            if (lane == 0 && n >= 2 && !mbar_wait_bounded(&q_empty[ib], (unsigned)((n / 2 - 1) & 1))) ok = false;
            ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
            if (!ok) break;
            if (lane == 0) {
                info[ib] = cur.ii;
                mbar_arrive_expect_tx(&q_full[ib], (unsigned)(nvalid * HD * 2));
            }
            __syncwarp();
            if (nvalid == 0) break;
            if (lane < nvalid)
                bulk_copy_g2s(Qs + (size_t)(ib * ROWS + lane) * QLD, q + (size_t)cur.ii.tok * q_stride + (size_t)(cur.ii.h0 + lane) * HD,
                              HD * 2, &q_full[ib]);
            const int st0 = cur.ii.c0 / BN, st1 = (cur.ii.c1 - 1) / BN, ask = min(st0 + NST - 1, st1);
            int row = cur.row;
            for (int st = st0; st <= st1 && ok; ++st, ++stage_it) {
                const int row_next = lookup(cur, st + 1);
                const int s = stage_it % NST;
                if (lane == 0) {
                    if (stage_it >= NST && !mbar_wait_bounded(&empty[s], (unsigned)((stage_it / NST - 1) & 1))) ok = false;
                    else mbar_arrive_expect_tx(&full[s], STAGE_BYTES);
                }
                ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
                if (ok && lane < nbox) {
                    // the box of page b: its blocks of 64 columns one after the other, box_rows rows of 128 bytes each
                    unsigned char* kt = ring + (unsigned)s * STAGE_BYTES + (unsigned)(lane * CB * box_rows) * ROW_BYTES;
                    tma_load_3d(kt, &map_k, 0, row, 0, &full[s]);
                    tma_load_3d(kt + KV_BYTES, &map_v, 0, row, 0, &full[s]);
                }
                row = row_next;
                if (st == ask) nxt = piece_at(cur.stop);  // the next piece is found while a ring of copies is on its way
            }
            cur = nxt;
        }
        if (bad_page && err) atomicOr(err, VL_DEV_BAD_PAGE);
        if (!ok && lane == 0) atomicExch(&failed, 1);
    } else {                                             // ---- consumers ----
        const int g = lane >> 2, t = lane & 3;
        // what head h's sums are multiplied by: one over L (maximum M, both in units of log2), a sink's term in it
        auto inverse = [&](float M, float L, int h) -> float {
            if (!sinks) return L > 0.f ? 1.0f / L : 0.f;
            const float sk = sinks[h], m = M * 0.6931471805599453f, x = fmaxf(m, sk), a = expf(m - x);
            return a / (L * a + expf(sk - x));
        };
        const unsigned ring_u32 = smem_u32(ring);
        const int kr0 = warp * 16;                       // this warp's 16 keys of every stage
        // byte offsets of this lane's ldmatrix rows inside a [64 rows][128 bytes] block and its swizzle
        // a stage holds, for K and for V, box after box (a page, or 64 rows of one), in a box the blocks of
        // 64 columns one after the other, in a block its rows of 128 bytes
        const int box_rows = page_size < BN ? page_size : BN;
        const unsigned blk_bytes = (unsigned)box_rows * ROW_BYTES;           // from one block of 64 columns to the next
        auto row_offset = [&](int r) { return (unsigned)(r / box_rows) * CB * blk_bytes + (unsigned)(r % box_rows) * ROW_BYTES; };
        const unsigned k_row = row_offset(kr0 + (lane & 7) + 8 * (lane >> 4));
        const unsigned v_row = row_offset(kr0 + (lane & 7) + 8 * ((lane >> 3) & 1));
        const unsigned sw = (unsigned)(lane & 7);
        int stage_it = 0, n = 0;
        bool ok = true;
        pdl_wait();
        // the places without keys: rows of zeros, and the ones beyond the bound are flagged
        for (int z = blockIdx.x; z < T; z += grid) {
            int tok, lo;
            if (keys_of(z, &tok, &lo) > 0) continue;
            if (tid == 0 && err && positions[tok] >= 0) atomicOr(err, VL_DEV_BEYOND_BOUND);
            bf16* row = out + (size_t)tok * nq * HD;
            if ((uintptr_t)out & 15) {                   // (uniform) the caller's rows may begin anywhere
                for (int i = tid; i < nq * HD; i += 32 * CONSUMERS) row[i] = __float2bfloat16(0.f);
                continue;
            }
            for (int i = tid; i < nq * HD / 8; i += 32 * CONSUMERS) reinterpret_cast<uint4*>(row)[i] = make_uint4(0u, 0u, 0u, 0u);
        }
        for (;; ++n) {
            const int ib = n & 1;
            if (!consumers_agree(__all_sync(0xffffffffu, mbar_wait_bounded(&q_full[ib], (unsigned)((n / 2) & 1))))) { ok = false; break; }
            const ItemInfo ii = info[ib];
            if (ii.nvalid == 0) break;
            unsigned qf[KSTEPS][4];
#pragma unroll
            for (int ks = 0; ks < KSTEPS; ++ks)
                ldmatrix_x4(qf[ks], smem_u32(Qs + (size_t)(ib * ROWS + (lane & 7) + 8 * ((lane >> 3) & 1)) * QLD + ks * 16 + 8 * (lane >> 4)));
            __syncwarp();
            if (lane == 0) mbar_arrive(&q_empty[ib]);    // the slot may be written again
            float o[DTILES][4], m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
#pragma unroll
            for (int d = 0; d < DTILES; ++d) { o[d][0] = o[d][1] = o[d][2] = o[d][3] = 0.f; }
            const int st0 = ii.c0 / BN, st1 = (ii.c1 - 1) / BN;
            for (int st = st0; st <= st1; ++st, ++stage_it) {
                const int s = stage_it % NST;
                if (!__all_sync(0xffffffffu, mbar_wait_bounded(&full[s], (unsigned)((stage_it / NST) & 1)))) { ok = false; break; }
                const unsigned kt = ring_u32 + (unsigned)s * STAGE_BYTES, vt = kt + KV_BYTES;
                // Slots behind the request's last key hold whatever the page's earlier owner left there.  Their probabilities are zero,
                // but 0 * NaN is NaN: those keys' values are cleared as fragments (zeroing them in shared memory and fencing it against the
                // TMA unit's next write cost 2 to 3 us at the end of every item).
                const int left = ii.c1 - (st * BN + kr0);        // keys of this warp's 16 that are read
                const bool tail = left < 16;
                unsigned keep0 = 0xffffffffu, keep1 = 0xffffffffu;
                if (tail) {
                    keep0 = (2 * t < left ? 0xffffu : 0u) | (2 * t + 1 < left ? 0xffff0000u : 0u);
                    keep1 = (2 * t + 8 < left ? 0xffffu : 0u) | (2 * t + 9 < left ? 0xffff0000u : 0u);
                }
                float sc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
                for (int ks = 0; ks < KSTEPS; ++ks) {
                    unsigned kb[4];
                    const unsigned chunk16 = (unsigned)(2 * ks + ((lane >> 3) & 1));      // 16-byte piece of the key row
                    ldmatrix_x4(kb, kt + (chunk16 >> 3) * blk_bytes + k_row + (((chunk16 & 7) ^ sw) << 4));
                    mma16816(sc[0], qf[ks], kb[0], kb[1]);
                    mma16816(sc[1], qf[ks], kb[2], kb[3]);
                }
                float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
                for (int nn = 0; nn < 2; ++nn)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int j = st * BN + kr0 + nn * 8 + 2 * t + (e & 1);
                        const float v = (j >= ii.c0 && j < ii.c1) ? sc[nn][e] * scale_log2 : -INFINITY;
                        sc[nn][e] = v;
                        mx[e >> 1] = fmaxf(mx[e >> 1], v);
                    }
                float corr[2], base[2];
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
                    mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
                    const float mn = fmaxf(m_run[r], mx[r]);
                    base[r] = (mn == -INFINITY) ? 0.f : mn;
                    corr[r] = exp2_mufu(m_run[r] - base[r]);
                    m_run[r] = mn;
                    l_run[r] *= corr[r];
                }
                unsigned pf[4];
                {
                    const float p00 = exp2_mufu(sc[0][0] - base[0]), p01 = exp2_mufu(sc[0][1] - base[0]);
                    const float p02 = exp2_mufu(sc[0][2] - base[1]), p03 = exp2_mufu(sc[0][3] - base[1]);
                    const float p10 = exp2_mufu(sc[1][0] - base[0]), p11 = exp2_mufu(sc[1][1] - base[0]);
                    const float p12 = exp2_mufu(sc[1][2] - base[1]), p13 = exp2_mufu(sc[1][3] - base[1]);
                    l_run[0] += p00 + p01 + p10 + p11;
                    l_run[1] += p02 + p03 + p12 + p13;
                    pf[0] = pack_bf16(p00, p01); pf[1] = pack_bf16(p02, p03);
                    pf[2] = pack_bf16(p10, p11); pf[3] = pack_bf16(p12, p13);
                }
#pragma unroll
                for (int dp = 0; dp < DTILES / 2; ++dp) {
                    unsigned vb[4];
                    const unsigned chunk16 = (unsigned)(2 * dp + (lane >> 4));            // 16-byte piece of the value row
                    ldmatrix_x4_trans(vb, vt + (chunk16 >> 3) * blk_bytes + v_row + (((chunk16 & 7) ^ sw) << 4));
                    if (tail) { vb[0] &= keep0; vb[1] &= keep1; vb[2] &= keep0; vb[3] &= keep1; }
                    o[2 * dp][0] *= corr[0]; o[2 * dp][1] *= corr[0]; o[2 * dp][2] *= corr[1]; o[2 * dp][3] *= corr[1];
                    o[2 * dp + 1][0] *= corr[0]; o[2 * dp + 1][1] *= corr[0]; o[2 * dp + 1][2] *= corr[1]; o[2 * dp + 1][3] *= corr[1];
                    mma16816(o[2 * dp], pf, vb[0], vb[1]);
                    mma16816(o[2 * dp + 1], pf, vb[2], vb[3]);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[s]);   // this warp has read the stage
            }
            // the four warps' partial results, merged in warp order
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 1);
                l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 2);
            }
#pragma unroll
            for (int d = 0; d < DTILES; ++d) {
                float* pa = sO + ((size_t)warp * ROWS + g) * OLD + d * 8 + 2 * t;
                pa[0] = o[d][0]; pa[1] = o[d][1];
                pa[8 * OLD] = o[d][2]; pa[8 * OLD + 1] = o[d][3];
            }
            if (t == 0) {
                s_m[warp][g] = m_run[0]; s_l[warp][g] = l_run[0];
                s_m[warp][g + 8] = m_run[1]; s_l[warp][g + 8] = l_run[1];
            }
            ok = consumers_agree(ok);
            if (!ok) break;
            for (int idx = tid; idx < ii.nvalid * HD; idx += 32 * CONSUMERS) {
                const int r = idx / HD, e = idx - r * HD;
                float M = -INFINITY;
#pragma unroll
                for (int w = 0; w < CONSUMERS; ++w) M = fmaxf(M, s_m[w][r]);
                float acc = 0.f, L = 0.f;
#pragma unroll
                for (int w = 0; w < CONSUMERS; ++w) {
                    const float wgt = (s_m[w][r] == -INFINITY) ? 0.f : exp2_mufu(s_m[w][r] - M);
                    acc += sO[((size_t)w * ROWS + r) * OLD + e] * wgt;
                    L += s_l[w][r] * wgt;
                }
                const int h = ii.h0 + r;
                if (ii.pieces == 1) {
                    out[((size_t)ii.tok * nq + h) * HD + e] = __float2bfloat16(acc * inverse(M, L, h));
                } else {
                    const size_t prow = ((size_t)ii.out_row * nq + h) * S + ii.piece;
                    __stcg(part_acc + prow * HD + e, acc);
                    if (e == 0) { __stcg(part_ml + 2 * prow, M); __stcg(part_ml + 2 * prow + 1, L); }
                }
            }
            if (ii.pieces > 1 && tid == 0) s_partial[n > 0] = ii;
        }                                                // (the agreement on the next piece also frees the merge buffer)
        // The items shared with other blocks, at the end of the run so that the stream does not wait for it: count this block's
        // pieces; whoever comes last adds up all of an item's, in their order.
        if (ok && (s_partial[0].nvalid || s_partial[1].nvalid)) {     // (the same in all four warps, which have just agreed)
            __threadfence();                             // this thread's parts, before the block's arrivals are counted
            consumer_barrier();
            if (tid < 2) s_last[tid] = s_partial[tid].nvalid && atomicAdd(&arrivals[s_partial[tid].counter], 1) == s_partial[tid].pieces - 1;
            consumer_barrier();
            if (s_last[0] || s_last[1]) __threadfence();
            for (int k = 0; k < 2; ++k) {
                if (!s_last[k]) continue;
                const ItemInfo ii = s_partial[k];
                for (int idx = tid; idx < ii.nvalid * HD; idx += 32 * CONSUMERS) {
                    const int r = idx / HD, e = idx - r * HD, h = ii.h0 + r;
                    const size_t prow = ((size_t)ii.out_row * nq + h) * S;
                    float M = -INFINITY, acc = 0.f, L = 0.f;
                    for (int p = 0; p < ii.pieces; ++p) {
                        const float2 ml = make_float2(__ldcg(part_ml + 2 * (prow + p)), __ldcg(part_ml + 2 * (prow + p) + 1));
                        const float a = __ldcg(part_acc + (prow + p) * HD + e), m = fmaxf(M, ml.x);
                        const float old = M == -INFINITY ? 0.f : exp2_mufu(M - m), now = ml.x == -INFINITY ? 0.f : exp2_mufu(ml.x - m);
                        acc = acc * old + a * now;
                        L = L * old + ml.y * now;
                        M = m;
                    }
                    out[((size_t)ii.tok * nq + h) * HD + e] = __float2bfloat16(acc * inverse(M, L, h));
                }
                if (tid == 0) arrivals[ii.counter] = 0;  // as the next launch finds it
            }
        }
        if (!ok && lane == 0) atomicExch(&failed, 1);
    }
    __syncthreads();
    if (tid == 0 && failed && err) atomicOr(err, VL_DEV_WAIT_EXPIRED | VL_DEV_IN_FLASH_DECODE_TMA);
}

extern "C" int vl_flash_decode_tma_head_dim() { return HD; }

// Arguments and scratch (S partial results a token and head, S > 1) as for vl_flash_decode; positions from `bound` on are
// flagged and get rows of zeros.  `arrivals`: a counter per (token, KV head, 16 query heads), zero before and after.  Page sizes
// that are a multiple of 8 and divide 64 or are a multiple of it.  `settled`: block_table, req_index, positions and token_index were
// complete before the kernel ahead of this one in the stream began (copies brought them), so a dependent launch may read them early.
extern "C" int vl_flash_decode_tma(const void* q, int q_stride, const void* kcache, const void* vcache,
                                   const int* block_table, int max_blocks, const int* req_index, const int* positions,
                                   int T, int nq, int nkv, int hd, int page_size, int num_pages, float scale, int window,
                                   int bound, int S, float* part_acc, float* part_ml, unsigned* err,
                                   const int* token_index, void* out, int* arrivals, const float* sinks, int settled, void* stream) {
    if (T <= 0) return VL_OK;
    if (hd != HD) return VL_ERR_UNSUPPORTED;
    if (nq <= 0 || nkv <= 0 || nq % nkv || page_size <= 0 || max_blocks <= 0 || num_pages <= 0 || q_stride % 8) return VL_ERR_ARGUMENT;
    if (bound <= 0 || S < 2 || !out || !arrivals) return VL_ERR_ARGUMENT;
    if (page_size % 8 || (page_size < BN ? BN % page_size : page_size % BN)) return VL_ERR_UNSUPPORTED;
    if ((((uintptr_t)q | (uintptr_t)kcache | (uintptr_t)vcache) & 15)) return VL_ERR_UNSUPPORTED;
    const long long rows = (long long)num_pages * nkv * page_size;
    const int grp = nq / nkv, htiles = (grp + ROWS - 1) / ROWS;
    const long long most = (long long)T * nkv * htiles * ((bound + BN - 1) / BN);       // key tiles, were every place full
    if (rows + BN >= (1ll << 31) || most >= (1ll << 31)) return VL_ERR_UNSUPPORTED;
    const int box_rows = page_size < BN ? page_size : BN;
    CUtensorMap map_k, map_v;
    int rc = tc5_make_map_blocks(&map_k, kcache, (int)rows, HD, HD, box_rows);
    if (rc) return rc;
    rc = tc5_make_map_blocks(&map_v, vcache, (int)rows, HD, HD, box_rows);
    if (rc) return rc;
    static int num_sms = 0;
    if (!num_sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || num_sms <= 0) num_sms = 148;
    }
    cudaError_t e = cudaFuncSetAttribute(flash_decode_tma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES);
    if (e != cudaSuccess) return (int)e;
    const int grid = (int)(most < num_sms ? most : num_sms);
    return vl_launch(flash_decode_tma_kernel, dim3(grid), dim3(NTHREADS), SMEM_BYTES, (cudaStream_t)stream,
                     map_k, map_v, (const bf16*)q, q_stride, block_table, max_blocks, req_index, positions, T, nq, nkv,
                     page_size, num_pages, scale * 1.4426950408889634f, window, bound, S, part_acc, part_ml, err, token_index,
                     (bf16*)out, arrivals, sinks, settled);
}
