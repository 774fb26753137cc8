// The recurrence of `vl_decay_scan` (csrc/recurrent.cu) over long portions, with the norm per head and the gate behind it:
//     o_t = (S + diag(u) k_t v_t^T)^T r_t,   S <- diag(w_t) S + k_t v_t^T,   out = rms_head(o) * norm * silu(gate)
// (S: D x P a head, D, P up to 128 and multiples of 4; w in (0, 1) per head and key channel), float32 throughout.
//
// Walked token by token one request keeps few warps busy with a chain of 2,048 steps.  Here a portion is cut into chunks of 64
// tokens that are worked off all at once, but for the state's way from chunk to chunk, which is one multiply-add an element:
//   (1) per chunk and head: the 64 x 64 matrix A_ts = sum_d r_td k_sd prod_{s<j<t} w_jd (t > s), A_tt = sum_d r_td u_d k_td; the part of
//       the outputs that stays inside the chunk, A V; what the chunk adds to the state, sum_s (k_s prod_{j>s} w_j) v_s^T; r_t times the
//       decays since the chunk's start;
//   (2) per head: S at every chunk's start, S <- diag(prod w) S + what the chunk added;
//   (3) per chunk and head: A V + (decayed r) S, normed and gated.
// No decay is ever divided by: for a pair of tokens in different halves of a run of 64, 32 or 16 tokens the product splits at
// the middle into one factor of r_t and one of k_s, both running products of numbers below 1, as the walk's own; pairs within 8 tokens
// multiply their few decays directly.  The products (2,016 pairs x D in a chunk, then 64 x 64 x P, 64 x D x P twice) are plain
// multiply-adds on tiles in shared memory.  One request of 2,048 tokens, 32 heads of 64 x 64, by the counters: (1) 79 us, shared memory's data path busy to 67
// %, the issue slots to 54 %, 12 % of DRAM's rate; (2) 16.5 us, waiting for its reads; (3) 34 us, 53 %, 51 % and 21 %.
// One request of 2,048 tokens, 32 heads of 64 x 64: 119 us with the norm and the gate, against 413 for the walk and the norm's kernel
// behind it; 128 x 128: 395 against 1,193; 512 tokens: 37 against 107; 64 tokens: 27 against 18.  A lone portion wins from 100 to 220 tokens on, by the
// heads' number and size (the caller decides; ops.decay_chunks_pay has the measurements).
#include "common.cuh"
#include "chunk_index.cuh"

#define CT 64                          // tokens of a chunk
#define DCH_MIN 96                     // portions of fewer tokens are walked
#define DCH_MAX 128                    // most rows and columns of a head's state

__device__ __forceinline__ float4 dc_ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void dc_st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void dc_fma(float4& a, float x, float4 v) { a.x += x * v.x; a.y += x * v.y; a.z += x * v.z; a.w += x * v.w; }
__device__ __forceinline__ float dc_at(const float4& v, int i) { return i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w)); }

struct DecayRows { const float* p; int ld, col; };                // rows [T, ld], the first column

// acc (rows 4 ty .., columns 4 tx ..) += a b over k in [0, n), a[row][k], b[k][column]
__device__ __forceinline__ void dc_product(float4 (&acc)[4], const float* a, int lda, const float* b, int ldb, int n) {
    for (int k = 0; k < n; k += 4) {
        float4 x[4], y[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            x[i] = dc_ld4(a + i * lda + k);
            y[i] = dc_ld4(b + (k + i) * ldb);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int i = 0; i < 4; ++i) dc_fma(acc[i], dc_at(x[i], e), y[e]);
    }
}

// The four tokens around the diagonal of A: a row takes the values up to its own token.  What lies behind is left out, not multiplied by
// A's zero, so that an infinity or a NaN in a token's value stays out of the tokens before it.
__device__ __forceinline__ void dc_triangle(float4 (&acc)[4], const float4 (&x)[4], const float4 (&y)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int e = 0; e <= i; ++e) dc_fma(acc[i], dc_at(x[i], e), y[e]);
}

// A running product of decays over `n` tokens (a multiple of 8), first to last (DOWN) or last to first, of one channel: put(t, x[t] times the decays of the tokens passed
// before t); returns the product of all.  Eight tokens' numbers are on their way from shared memory together.
template <bool DOWN, typename Put>
__device__ __forceinline__ float dc_chain(const float* x, const float* w, int ld, int t0, int n, Put put) {
    float f = 1.f;
    for (int i = 0; i < n; i += 8) {
        float a[8], g[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int t = DOWN ? t0 + i + e : t0 + n - 1 - i - e;
            a[e] = x[t * ld]; g[e] = w[t * ld];
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) { put(DOWN ? t0 + i + e : t0 + n - 1 - i - e, a[e] * f); f *= g[e]; }
    }
    return f;
}

// The i-th pair of tokens (s before t) in different halves of runs of 2 `half` tokens.
__device__ __forceinline__ void dc_pair(int i, int half, int& t, int& s) {
    const int seg = i / (half * half), e = i - seg * half * half;
    t = seg * 2 * half + half + e / half;
    s = seg * 2 * half + e % half;
}

#define DCH_LDA (CT + 4)
// Buffers of chunk and head number i = chunk * H + head: added [D][P], start [D][P] (S at the chunk's start), rdec [64][D], inner [64][P],
// keep [D].
__global__ void __launch_bounds__(256, 3)
decay_prep_kernel(DecayRows r, DecayRows k, DecayRows v, DecayRows w, const float* __restrict__ u, const int* __restrict__ cu, int B,
                  float* __restrict__ added, float* __restrict__ rdec, float* __restrict__ inner, float* __restrict__ keep, int H, int D, int P) {
    extern __shared__ __align__(16) float sm[];
    pdl_launch_dependents();
    pdl_wait();
    int b, c;
    if (!ci_find(cu, B, CT, DCH_MIN, blockIdx.x, &b, &c)) return;
    const int h = blockIdx.y, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int row0 = cu[b] + c * CT, m = min(CT, cu[b + 1] - row0);
    const int LD = D + 4, D4 = D >> 2;
    const size_t ch = (size_t)blockIdx.x * H + h;
    float* R = sm;                                                // [64][LD], later the values [64][68]
    float* K = R + CT * (LD > DCH_LDA ? LD : DCH_LDA);
    float* X = K + CT * LD;                                       // r or k times one level's decays
    float* W = X + CT * LD;                                       // the decays; when they are used up A [64][68]
    for (int i = tid; i < CT * D4; i += 256) {                    // (tokens behind the portion: nothing added, nothing decayed)
        const int t = i / D4, d = 4 * (i - t * D4);
        const size_t row = row0 + t, at = (size_t)h * D + d;
        const bool in = t < m;
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f), one = make_float4(1.f, 1.f, 1.f, 1.f);
        dc_st4(R + t * LD + d, in ? dc_ld4(r.p + row * r.ld + r.col + at) : z);
        dc_st4(K + t * LD + d, in ? dc_ld4(k.p + row * k.ld + k.col + at) : z);
        dc_st4(W + t * LD + d, in ? dc_ld4(w.p + row * w.ld + w.col + at) : one);
    }
    __syncthreads();
    // A's elements stay in registers until the decays' place is free: three blocks fit an SM instead of two (a third of (1)'s time)
    float far[4], mid[2], close = 0.f, near[8];
    // pairs in different halves of a run of 2 `half` tokens
#pragma unroll
    for (int half = 32; half >= 8; half >>= 1) {
        for (int i = tid; i < (CT / half) * D; i += 256) {        // a run of `half` tokens of one channel
            const int seg = i / D, d = i - seg * D, t0 = seg * half;
            auto put = [&](int t, float v) { X[t * LD + d] = v; };
            if (seg & 1) dc_chain<true>(R + d, W + d, LD, t0, half, put);      // behind the middle: r times the decays from there on
            else dc_chain<false>(K + d, W + d, LD, t0, half, put);             // before it: k times the decays behind the token
        }
        __syncthreads();
        // 32 half pairs: a thread takes `each` neighbouring s for one or two t
        if (half == 32) {
            const float* a = X + (32 + ty) * LD;
            const float* q = X + tx * LD;
            float s[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
            for (int d = 0; d < D; d += 4) {
                const float4 a0 = dc_ld4(a + d), a1 = dc_ld4(a + 16 * LD + d), b0 = dc_ld4(q + d), b1 = dc_ld4(q + 16 * LD + d);
                s[0][0] += a0.x * b0.x; s[0][0] += a0.y * b0.y; s[0][0] += a0.z * b0.z; s[0][0] += a0.w * b0.w;
                s[0][1] += a0.x * b1.x; s[0][1] += a0.y * b1.y; s[0][1] += a0.z * b1.z; s[0][1] += a0.w * b1.w;
                s[1][0] += a1.x * b0.x; s[1][0] += a1.y * b0.y; s[1][0] += a1.z * b0.z; s[1][0] += a1.w * b0.w;
                s[1][1] += a1.x * b1.x; s[1][1] += a1.y * b1.y; s[1][1] += a1.z * b1.z; s[1][1] += a1.w * b1.w;
            }
            far[0] = s[0][0]; far[1] = s[0][1]; far[2] = s[1][0]; far[3] = s[1][1];
        } else {
#pragma unroll
            for (int n = 0; n < half / 8; ++n) {
                int t, s;
                dc_pair(tid + 256 * n, half, t, s);
                float x = 0.f, y = 0.f;
                for (int d = 0; d < D; d += 4) {
                    const float4 a = dc_ld4(X + t * LD + d), q = dc_ld4(X + s * LD + d);
                    x += a.x * q.x; y += a.y * q.y; x += a.z * q.z; y += a.w * q.w;
                }
                if (half == 16) mid[n] = x + y; else close = x + y;
            }
        }
        __syncthreads();
    }
    // pairs within 8 tokens and the tokens themselves: a warp a run, four channels a lane, everything in registers
    {
        const int t0 = 8 * (tid >> 5), d = 4 * (tid & 31);
        const bool on = d < D;
        float4 rr[8], ww[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            rr[e] = on ? dc_ld4(R + (t0 + e) * LD + d) : make_float4(0.f, 0.f, 0.f, 0.f);
            ww[e] = on ? dc_ld4(W + (t0 + e) * LD + d) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        const float4 uu = on ? dc_ld4(u + (size_t)h * D + d) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            float4 q = on ? dc_ld4(K + (t0 + s) * LD + d) : make_float4(0.f, 0.f, 0.f, 0.f);
            float sum[8];
            sum[s] = (rr[s].x * (uu.x * q.x) + rr[s].y * (uu.y * q.y)) + (rr[s].z * (uu.z * q.z) + rr[s].w * (uu.w * q.w));
#pragma unroll
            for (int t = s + 1; t < 8; ++t) {
                sum[t] = (rr[t].x * q.x + rr[t].y * q.y) + (rr[t].z * q.z + rr[t].w * q.w);
                q.x *= ww[t].x; q.y *= ww[t].y; q.z *= ww[t].z; q.w *= ww[t].w;
            }
#pragma unroll
            for (int t = s; t < 8; ++t) {
                const float v = warp_sum(sum[t]);
                if ((tid & 31) == t) near[s] = v;
            }
        }
    }
    // r times the decays since the chunk's start (to memory); k times those up to its end (X); the chunk's own decay
    __syncthreads();
    for (int i = tid; i < 2 * D; i += 256) {
        const int d = i < D ? i : i - D;
        if (i < D) keep[ch * D + d] = dc_chain<true>(R + d, W + d, LD, 0, CT, [&](int t, float v) { rdec[(ch * CT + t) * D + d] = v; });
        else dc_chain<false>(K + d, W + d, LD, 0, CT, [&](int t, float v) { X[t * LD + d] = v; });
    }
    __syncthreads();
    float* A = W;
    for (int i = tid; i < CT * DCH_LDA / 4; i += 256) dc_st4(A + 4 * i, make_float4(0.f, 0.f, 0.f, 0.f));
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) A[(32 + ty + 16 * (i >> 1)) * DCH_LDA + tx + 16 * (i & 1)] = far[i];
#pragma unroll
    for (int n = 0; n < 3; ++n) {
        int t, s;
        dc_pair(n < 2 ? tid + 256 * n : tid, n < 2 ? 16 : 8, t, s);
        A[t * DCH_LDA + s] = n < 2 ? mid[n] : close;
    }
    if ((tid & 31) < 8) {
        const int t0 = 8 * (tid >> 5), t = tid & 31;
#pragma unroll
        for (int s = 0; s < 8; ++s)
            if (s <= t) A[(t0 + t) * DCH_LDA + t0 + s] = near[s];
    }
    for (int p0 = 0; p0 < P; p0 += 64) {                          // 64 columns of the values at a time, in the place of r
        __syncthreads();
        for (int i = tid; i < CT * 16; i += 256) {
            const int t = i >> 4, p = 4 * (i & 15);
            dc_st4(R + t * DCH_LDA + p, t < m && p0 + p < P ? dc_ld4(v.p + (size_t)(row0 + t) * v.ld + v.col + (size_t)h * P + p0 + p)
                                                             : make_float4(0.f, 0.f, 0.f, 0.f));
        }
        __syncthreads();
        const bool cols = p0 + 4 * tx < P;
        float4 acc[4] = {};
        for (int d0 = 4 * ty; d0 < D; d0 += 64) {                 // (the values of a step of four tokens serve both products)
            float4 sum[4] = {};
#pragma unroll 2
            for (int k = 0; k < CT; k += 4) {
                float4 y[4], x[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) { y[i] = dc_ld4(R + (k + i) * DCH_LDA + 4 * tx); x[i] = dc_ld4(X + (k + i) * LD + d0); }
#pragma unroll
                for (int e = 0; e < 4; ++e)
#pragma unroll
                    for (int i = 0; i < 4; ++i) dc_fma(sum[i], dc_at(x[e], i), y[e]);
                if (d0 < 64 && k <= 4 * ty) {                     // (A is zero above the diagonal)
#pragma unroll
                    for (int i = 0; i < 4; ++i) x[i] = dc_ld4(A + (4 * ty + i) * DCH_LDA + k);
                    if (k == 4 * ty) {
                        dc_triangle(acc, x, y);
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; ++e)
#pragma unroll
                            for (int i = 0; i < 4; ++i) dc_fma(acc[i], dc_at(x[i], e), y[e]);
                    }
                }
            }
            if (cols) {
#pragma unroll
                for (int i = 0; i < 4; ++i) dc_st4(added + (ch * D + d0 + i) * P + p0 + 4 * tx, sum[i]);
            }
        }
        if (4 * ty >= D) {                                        // (rows of the state there are none)
            const float* a = A + 4 * ty * DCH_LDA;
            dc_product(acc, a, DCH_LDA, R + 4 * tx, DCH_LDA, 4 * ty);
            float4 x[4], y[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) { x[i] = dc_ld4(a + i * DCH_LDA + 4 * ty); y[i] = dc_ld4(R + (4 * ty + i) * DCH_LDA + 4 * tx); }
            dc_triangle(acc, x, y);
        }
        if (cols) {
#pragma unroll
            for (int i = 0; i < 4; ++i) dc_st4(inner + (ch * CT + 4 * ty + i) * P + p0 + 4 * tx, acc[i]);
        }
    }
}

// The state of a request lies as vl_decay_scan keeps it: row d and column p of head h at scan_at(h, d, p).
struct ScanLayout { int rows, L, cols, tiles; };
__device__ __forceinline__ size_t scan_at(const ScanLayout& y, int h, int d, int p) {
    const int z = p / y.cols, col = p - z * y.cols, l = d / y.rows, i = d - l * y.rows;
    return (((size_t)h * y.tiles + z) * y.rows + i) * (y.cols * y.L) + col * y.L + l;
}
__global__ void __launch_bounds__(256)
decay_chain_kernel(const float* __restrict__ added, const float* __restrict__ keep, float* __restrict__ start, float* __restrict__ state,
                   long long state_stride, const int* __restrict__ cu, const int* __restrict__ slots, ScanLayout lay, int H, int D, int P) {
    pdl_launch_dependents();
    pdl_wait();
    const int b = blockIdx.y, n = cu[b + 1] - cu[b];
    if (n < DCH_MIN) return;
    const int first = ci_first(cu, b, CT, DCH_MIN), chunks = (n + CT - 1) / CT;
    const int idx = blockIdx.x * 256 + threadIdx.x, per = D * (P >> 2), h = idx / per;
    if (h >= H) return;
    const int e = idx - h * per, d = e / (P >> 2), p = 4 * (e - d * (P >> 2));
    float* S = state + (long long)slots[b] * state_stride;
    float4 s = make_float4(S[scan_at(lay, h, d, p)], S[scan_at(lay, h, d, p + 1)], S[scan_at(lay, h, d, p + 2)], S[scan_at(lay, h, d, p + 3)]);
    const size_t at = (size_t)(first * H + h) * D + d, step = (size_t)H * D;
#pragma unroll 8
    for (int c = 0; c < chunks; ++c) {                            // (the reads of eight chunks are on their way together)
        const float4 x = dc_ld4(added + (at + c * step) * P + p);
        const float g = keep[at + c * step];
        dc_st4(start + (at + c * step) * P + p, s);
        s.x = g * s.x + x.x; s.y = g * s.y + x.y; s.z = g * s.z + x.z; s.w = g * s.w + x.w;
    }
    S[scan_at(lay, h, d, p)] = s.x; S[scan_at(lay, h, d, p + 1)] = s.y;
    S[scan_at(lay, h, d, p + 2)] = s.z; S[scan_at(lay, h, d, p + 3)] = s.w;
}

template <typename TP, int NC>                                    // NC: 64 columns of the values a step
__global__ void __launch_bounds__(256, 2)
decay_out_kernel(const float* __restrict__ rdec, const float* __restrict__ start, const float* __restrict__ inner,
                 const TP* __restrict__ gate, int ld, int gate_col, const float* __restrict__ norm, float eps, const int* __restrict__ cu,
                 int B, TP* __restrict__ out, int H, int D, int P) {
    extern __shared__ __align__(16) float sm[];
    pdl_launch_dependents();
    pdl_wait();
    int b, c;
    if (!ci_find(cu, B, CT, DCH_MIN, blockIdx.x, &b, &c)) return;
    const int h = blockIdx.y, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int row0 = cu[b] + c * CT, m = min(CT, cu[b + 1] - row0);
    const size_t ch = (size_t)blockIdx.x * H + h;
    const int LD = D + 4, LDP = 64 * NC + 4, D4 = D >> 2;
    float* R = sm;                                                // [64][LD]
    float* S = R + CT * LD;                                       // [D][LDP]
    for (int i = tid; i < CT * D4; i += 256) {
        const int t = i / D4, d = 4 * (i - t * D4);
        dc_st4(R + t * LD + d, dc_ld4(rdec + ch * CT * D + 4 * i));
    }
    for (int i = tid; i < D * 16 * NC; i += 256) {
        const int d = i / (16 * NC), p = 4 * (i - d * 16 * NC);
        dc_st4(S + d * LDP + p, p < P ? dc_ld4(start + (ch * D + d) * P + p) : make_float4(0.f, 0.f, 0.f, 0.f));
    }
    float4 acc[NC][4];
#pragma unroll
    for (int e = 0; e < NC; ++e)
#pragma unroll
        for (int i = 0; i < 4; ++i)
            acc[e][i] = 64 * e + 4 * tx < P ? dc_ld4(inner + (ch * CT + 4 * ty + i) * P + 64 * e + 4 * tx) : make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
#pragma unroll
    for (int e = 0; e < NC; ++e) dc_product(acc[e], R + 4 * ty * LD, LD, S + 64 * e + 4 * tx, LDP, D);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int t = 4 * ty + i;
        float ss = 0.f;
#pragma unroll
        for (int e = 0; e < NC; ++e) ss += acc[e][i].x * acc[e][i].x + acc[e][i].y * acc[e][i].y + acc[e][i].z * acc[e][i].z + acc[e][i].w * acc[e][i].w;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);      // (columns behind P are zero)
        const float inv = 1.f / sqrtf(ss / (float)P + eps);
        if (t >= m) continue;
#pragma unroll
        for (int e = 0; e < NC; ++e) {
            const int p = 64 * e + 4 * tx;
            if (p >= P) continue;
            const float4 a = acc[e][i], w = dc_ld4(norm + (size_t)h * P + p), z = Quad<TP>::load(gate + (size_t)(row0 + t) * ld + gate_col + (size_t)h * P + p);
            Quad<TP>::store(out + (size_t)(row0 + t) * H * P + (size_t)h * P + p,
                            make_float4(a.x * inv * w.x * (z.x / (1.f + expf(-z.x))), a.y * inv * w.y * (z.y / (1.f + expf(-z.y))),
                                        a.z * inv * w.z * (z.z / (1.f + expf(-z.z))), a.w * inv * w.w * (z.w / (1.f + expf(-z.w)))));
        }
    }
}

// Steps whose requests bring one token each: a block per head and request.  What bounds it is the state, read and written once; the walk of
// vl_decay_scan gives 2 KB of it to a block that first clears and fills staging buffers for sixteen tokens.  Here a thread asks for eight of
// the state's tiles (of `cols` columns) at once, r, k, w and u lie in registers, and the head's norm and gate follow in the block.  The
// state is kept as that kernel keeps it, a lane's four rows of a tile 128 floats apart, and a column's sum runs in its order.
// 32 requests, 32 heads of 64 x 64: 10.2 us (the read and write of the state take 5.0) against 24.5 for the walk and the norm's kernel, 64: 15.8
// and 44.6 (10.1), 8: 3.9 and 9.1, 1: 3.3 and 5.1; 32 requests, heads of 128 x 128: 32 and 126 (20).
#define DS_TILES 8
template <typename TP, int L>
__global__ void __launch_bounds__(128)
decay_step_kernel(DecayRows r, DecayRows k, DecayRows v, DecayRows w, const float* __restrict__ u, float* __restrict__ state,
                  long long state_stride, const int* __restrict__ cu, const int* __restrict__ slots, const TP* __restrict__ gate, int ld,
                  int gate_col, const float* __restrict__ norm, float eps, TP* __restrict__ out, int T, int H, int D, int P, int Z) {
    constexpr int CT_ = 128 / L;                                  // columns of a tile
    __shared__ float s_o[DCH_MAX], s_part[4];
    pdl_launch_dependents();
    pdl_wait();
    const int h = blockIdx.x, b = blockIdx.y, row = cu[b], tid = threadIdx.x, col = tid / L, l = tid % L;
    if (cu[b + 1] - row != 1) {
        // the rows behind the last token (padding of a replayed step) hold zeros, not what the buffer held before
        if (b >= cu[gridDim.y] && b < T && tid < P) out[((size_t)b * H + h) * P + tid] = from_f32<TP>(0.f);
        return;
    }
    float* S = state + (long long)slots[b] * state_stride + (size_t)h * Z * 4 * 128 + tid;
    const bool on = 4 * l < D;
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    const size_t at = (size_t)h * D + 4 * l;
    const float4 rr = on ? dc_ld4(r.p + (size_t)row * r.ld + r.col + at) : z4, kk = on ? dc_ld4(k.p + (size_t)row * k.ld + k.col + at) : z4;
    const float4 ww = on ? dc_ld4(w.p + (size_t)row * w.ld + w.col + at) : z4, uu = on ? dc_ld4(u + at) : z4;
    const float* vrow = v.p + (size_t)row * v.ld + v.col + (size_t)h * P;
    float ss = 0.f;
    for (int z0 = 0; z0 < Z; z0 += DS_TILES) {
        float s[DS_TILES][4], vj[DS_TILES];
#pragma unroll
        for (int e = 0; e < DS_TILES; ++e) {
            const int z = z0 + e, p = z * CT_ + col;
            vj[e] = z < Z && p < P ? vrow[p] : 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) s[e][i] = z < Z ? S[((size_t)z * 4 + i) * 128] : 0.f;
        }
#pragma unroll
        for (int e = 0; e < DS_TILES; ++e) {
            const int z = z0 + e, p = z * CT_ + col;
            if (z >= Z) break;
            float acc0 = 0.f, acc1 = 0.f;
            const float kv0 = kk.x * vj[e], kv1 = kk.y * vj[e], kv2 = kk.z * vj[e], kv3 = kk.w * vj[e];
            acc0 += rr.x * (s[e][0] + uu.x * kv0);
            acc1 += rr.y * (s[e][1] + uu.y * kv1);
            acc0 += rr.z * (s[e][2] + uu.z * kv2);
            acc1 += rr.w * (s[e][3] + uu.w * kv3);
            S[((size_t)z * 4 + 0) * 128] = ww.x * s[e][0] + kv0;
            S[((size_t)z * 4 + 1) * 128] = ww.y * s[e][1] + kv1;
            S[((size_t)z * 4 + 2) * 128] = ww.z * s[e][2] + kv2;
            S[((size_t)z * 4 + 3) * 128] = ww.w * s[e][3] + kv3;
            float o = acc0 + acc1;
#pragma unroll
            for (int d = L >> 1; d > 0; d >>= 1) o += __shfl_xor_sync(0xffffffffu, o, d);
            if (l == 0 && p < P) { s_o[p] = o; ss += o * o; }
        }
    }
    ss = warp_sum(ss);
    if ((tid & 31) == 0) s_part[tid >> 5] = ss;
    __syncthreads();
    const float inv = 1.f / sqrtf(((s_part[0] + s_part[1]) + (s_part[2] + s_part[3])) / (float)P + eps);
    if (tid < P) {
        const float z = to_f32(gate[(size_t)row * ld + gate_col + (size_t)h * P + tid]);
        out[((size_t)row * H + h) * P + tid] = from_f32<TP>(s_o[tid] * inv * norm[(size_t)h * P + tid] * (z / (1.f + expf(-z))));
    }
}

// One token a request (others are left alone); T rows, of which those behind the last token become zeros; arguments as vl_decay_chunks'.
extern "C" int vl_decay_step(const float* rp, int ldr, int rc, const float* kp, int ldk, int kc, const float* vp, int ldv, int vc,
                             const float* wp, int ldw, int wc, const float* u, float* state, long long state_stride, int lay_rows,
                             int lay_lanes, int lay_cols, int lay_tiles, const int* cu, const int* slots, int B, const void* gate, int dtype,
                             int ldg, int gate_col, const float* norm, float eps, void* out, int T, int H, int D, int P, void* stream) {
    if (B <= 0) return VL_OK;
    if (H <= 0 || D <= 0 || P <= 0 || D > DCH_MAX || P > DCH_MAX || D % 4 || B > 65535) return VL_ERR_UNSUPPORTED;
    if (rc < 0 || kc < 0 || vc < 0 || wc < 0 || gate_col < 0 || rc + H * D > ldr || kc + H * D > ldk || vc + H * P > ldv || wc + H * D > ldw ||
        gate_col + H * P > ldg || !gate || !norm || lay_rows != 4 || lay_lanes * lay_cols != 128 || lay_lanes * 4 < D || lay_cols * lay_tiles < P)
        return VL_ERR_ARGUMENT;
    if (((ldr | rc | ldk | kc | ldw | wc) & 3) || (((uintptr_t)rp | (uintptr_t)kp | (uintptr_t)wp | (uintptr_t)u) & 15)) return VL_ERR_UNSUPPORTED;
    cudaStream_t s = (cudaStream_t)stream;
#define DC_STEP(TP, LL)                                                                                                          \
    case LL:                                                                                                                     \
        return vl_launch(decay_step_kernel<TP, LL>, dim3(H, B), dim3(128), 0, s, DecayRows{rp, ldr, rc}, DecayRows{kp, ldk, kc}, \
                         DecayRows{vp, ldv, vc}, DecayRows{wp, ldw, wc}, u, state, state_stride, cu, slots, (const TP*)gate, ldg, \
                         gate_col, norm, eps, (TP*)out, T, H, D, P, lay_tiles)
#define DC_STEPS(TP) switch (lay_lanes) { DC_STEP(TP, 1); DC_STEP(TP, 2); DC_STEP(TP, 4); DC_STEP(TP, 8); DC_STEP(TP, 16); DC_STEP(TP, 32); }
    if (dtype == VL_BF16) DC_STEPS(bf16)
    if (dtype == VL_F32) DC_STEPS(float)
#undef DC_STEPS
#undef DC_STEP
    return VL_ERR_UNSUPPORTED;
}

extern "C" int vl_decay_min_chunk() { return DCH_MIN; }
// Floats of scratch for a launch of up to `chunks` chunks.
extern "C" long long vl_decay_chunk_floats(int chunks, int H, int D, int P) {
    return (long long)chunks * H * (2ll * D * P + (long long)CT * (D + P) + D);
}

// r, k, v, w: columns rc .. of rows ldr wide and so on (float32).  `chunks`: at least the chunks of all portions of DCH_MIN tokens and
// more; requests that bring fewer are left alone.  state rows as vl_decay_scan's, described by lay_* (vl_decay_scan: rows a lane, lanes a
// column, columns a block, blocks a head); gate and out of `dtype`, norm float32 [H * P].
extern "C" int vl_decay_chunks(const float* rp, int ldr, int rc, const float* kp, int ldk, int kc, const float* vp, int ldv, int vc,
                               const float* wp, int ldw, int wc, const float* u, float* state, long long state_stride, int lay_rows,
                               int lay_lanes, int lay_cols, int lay_tiles, const int* cu, const int* slots, int B, int chunks, float* scratch,
                               const void* gate, int dtype, int ldg, int gate_col, const float* norm, float eps, void* out, int H, int D,
                               int P, void* stream) {
    if (B <= 0 || chunks <= 0) return VL_OK;
    if (H <= 0 || D <= 0 || P <= 0 || D > DCH_MAX || P > DCH_MAX || D % 4 || P % 4) return VL_ERR_UNSUPPORTED;
    if (rc < 0 || kc < 0 || vc < 0 || wc < 0 || gate_col < 0 || rc + H * D > ldr || kc + H * D > ldk || vc + H * P > ldv || wc + H * D > ldw ||
        gate_col + H * P > ldg || !gate || !norm || !scratch || lay_rows <= 0 || lay_lanes <= 0 || lay_cols <= 0 || lay_tiles <= 0 ||
        lay_rows * lay_lanes < D || lay_cols * lay_tiles < P || H > 65535 || B > 65535)
        return VL_ERR_ARGUMENT;
    if (((ldr | rc | ldk | kc | ldv | vc | ldw | wc | ldg | gate_col) & 3) ||
        (((uintptr_t)rp | (uintptr_t)kp | (uintptr_t)vp | (uintptr_t)wp | (uintptr_t)u | (uintptr_t)scratch | (uintptr_t)gate | (uintptr_t)norm |
          (uintptr_t)out) & 15))
        return VL_ERR_UNSUPPORTED;
    const size_t n = (size_t)chunks * H;
    float* added = scratch;
    float* start = added + n * D * P;
    float* rdec = start + n * D * P;
    float* inner = rdec + n * CT * D;
    float* keep = inner + n * CT * P;
    const int LD = D + 4;
    const ScanLayout lay = {lay_rows, lay_lanes, lay_cols, lay_tiles};
    cudaStream_t s = (cudaStream_t)stream;
    const size_t prep = sizeof(float) * CT * ((size_t)2 * LD + 2 * (LD > DCH_LDA ? LD : DCH_LDA));
    cudaError_t e = cudaFuncSetAttribute(decay_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)prep);
    if (e != cudaSuccess) return (int)e;
    int rcode = vl_launch(decay_prep_kernel, dim3(chunks, H), dim3(256), prep, s, DecayRows{rp, ldr, rc}, DecayRows{kp, ldk, kc}, DecayRows{vp, ldv, vc},
                          DecayRows{wp, ldw, wc}, u, cu, B, added, rdec, inner, keep, H, D, P);
    if (rcode) return rcode;
    rcode = vl_launch(decay_chain_kernel, dim3((H * D * (P / 4) + 255) / 256, B), dim3(256), 0, s, (const float*)added, (const float*)keep, start,
                      state, state_stride, cu, slots, lay, H, D, P);
    if (rcode) return rcode;
    auto outputs = [&](auto kernel, auto* g, auto* o, int nc) {
        const size_t smem = sizeof(float) * ((size_t)CT * LD + (size_t)D * (64 * nc + 4));
        const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (err != cudaSuccess) return (int)err;
        return vl_launch(kernel, dim3(chunks, H), dim3(256), smem, s, (const float*)rdec, (const float*)start, (const float*)inner, g, ldg, gate_col,
                         norm, eps, cu, B, o, H, D, P);
    };
    if (dtype == VL_BF16)
        return P <= 64 ? outputs(decay_out_kernel<bf16, 1>, (const bf16*)gate, (bf16*)out, 1) : outputs(decay_out_kernel<bf16, 2>, (const bf16*)gate, (bf16*)out, 2);
    if (dtype == VL_F32)
        return P <= 64 ? outputs(decay_out_kernel<float, 1>, (const float*)gate, (float*)out, 1) : outputs(decay_out_kernel<float, 2>, (const float*)gate, (float*)out, 2);
    return VL_ERR_UNSUPPORTED;
}
