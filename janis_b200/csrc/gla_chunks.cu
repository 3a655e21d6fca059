// Gated linear attention's recurrence in prompts, 16 tokens at a time on the tensor cores (bfloat16 inputs):
//
//   S_t = diag(a_t) S_(t-1) + k_t v_t^T,   o_t = S_t^T q_t,   a_t = sigmoid(z_t + b)^(1/tau) per key channel
//
// With b_t[i] the sum of log a[i] from the chunk's start up to t, the tokens of a chunk are three products:
//
//   o_t   = S_0^T (q_t e^(b_t))  +  sum_(s <= t) A[t, s] v_s,      A[t, s] = sum_i q_t[i] k_s[i] e^(b_t[i] - b_s[i])
//   S_end = diag(e^(b_end)) S_0 + sum_s (k_s e^(b_end - b_s)) v_s^T
//
// A first kernel forms, for all chunks at the same time, the weighted queries and keys, A and e^(b_end) - 1.  No exponent in
// them is positive, so nothing overflows however strong a decay is; b is summed in double and kept as two floats, so that a difference is
// as exact as one logarithm.  The second kernel is the chain over the chunks.  What the recurrence keeps as floats enters
// its products as sums of three bfloat16 numbers (both operands where both are floats: the six products that reach a float's
// last bits), the large and the small parts in accumulators of their own, and S takes a chunk's sum by one rounded addition.
// A chunk with an infinite or NaN value adds up A v one token after another: the zeros of A above the diagonal would
// carry it to the tokens before it (0 x inf).
//
// A CTA owns 32 value columns of a sequence's head, four warps to 16 of them: each keeps S for a quarter of the key channels in
// registers (as the accumulators of the last product, which are at the same time second operands of the first), and the
// four sums of a result meet in shared memory.  The chain bounds it: some 250 instructions a warp and two barriers a chunk.
//
// Few sequences leave SMs idle: their chains run in pieces at the same time, as many as give two CTAs an SM, once for the pieces' end
// states alone and once from the states that these give, where that takes less time (gla_pieces_pay; one sequence of 2,048 tokens: 151 us for
// the chain -> 29 + 62; a scratch without room for the states keeps whole chains).
//
// 8 heads of 128 x 256, against gla_scan_kernel (bound by shared memory: three 16-byte reads for 16 multiply-adds a lane) with its
// kernel for the decays: whole chains of one sequence of 2,048 tokens 374 -> 200 us (in pieces 140), 300 tokens 60 -> 43,
// eight of 512 666 -> 210.  Errors
// against 64 bits over 2,048 tokens: results 3.3e-7 -> 1.4e-7, states 3.2e-7 -> 0.7e-7; where the states remember a thousand tokens
// 5.3e-6 -> 1.9e-7 and 7.3e-6 -> 2.1e-7.
#include <math.h>

#include "mma_bf16.cuh"

namespace janis {

constexpr int GQ = 16;                       // tokens a chunk
constexpr int GC_COLS = 32;                  // value columns a CTA
constexpr int GC_STAGES = 3;

struct GlaChunkShape {
    int row_elems, q_off, k_off, v_off, H, d, dv, n_tok;
    float q_scale, inv_tau;
};

// What the first kernel leaves: weighted queries and keys [2][3][n_tok][H d], A [n_tok][H][3][16] (bfloat16 parts), and
// e^(b_end) - 1 [chunk][H d] floats, the sequences' chunks one after another.
struct GlaChunkScratch {
    bf16 *qk, *a;
    float* grow;
};
__host__ __device__ inline GlaChunkScratch gla_chunk_scratch(void* p, const GlaChunkShape& g) {
    GlaChunkScratch s;
    s.qk = reinterpret_cast<bf16*>(p);
    s.a = s.qk + (size_t)6 * g.n_tok * g.H * g.d;
    s.grow = reinterpret_cast<float*>(s.a + (size_t)g.n_tok * g.H * 48);
    return s;
}

__device__ __forceinline__ void split3_one(float x, bf16& hi, bf16& mid, bf16& lo) {
    hi = __float2bfloat16_rn(x);
    x -= __bfloat162float(hi);
    mid = __float2bfloat16_rn(x);
    lo = __float2bfloat16_rn(x - __bfloat162float(mid));
}

// A CTA per (chunk, head), the sequences' chunks counted through: first a thread per key channel, then a thread per pair of tokens.
// (The step's n_tok / 16 + n_seq bound the chunks' number; a place for every chunk of the step in every sequence would be
// 2 million CTAs for 256 prompts of 64 tokens.)
__global__ void __launch_bounds__(256)
gla_chunk_terms_kernel(const bf16* __restrict__ rows, const bf16* __restrict__ z_rows, const bf16* __restrict__ bias, GlaChunkShape g,
                       int n_seq, const int* __restrict__ seq_first_row, const int* __restrict__ seq_start, const int* __restrict__ seq_end,
                       GlaChunkScratch out) {
    extern __shared__ float gla_terms[];
    const int d = g.d, ld = d + 1, place = blockIdx.x, h = blockIdx.y;
    float *q_s = gla_terms, *k_s = q_s + GQ * ld, *hi_s = k_s + GQ * ld, *lo_s = hi_s + GQ * ld;      // [16][ld]
    grid_dependents_launch();
    int seq = 0, chunk = 0;
    if (!find_piece(place, seq_start, seq_end, n_seq, GQ, seq, chunk)) return;
    const int row0 = seq_first_row[seq] + chunk * GQ, n = min(GQ, seq_end[seq] - seq_start[seq] - chunk * GQ);
    grid_dependency_wait();
    const size_t plane = (size_t)g.n_tok * g.H * d;
    for (int i = threadIdx.x; i < d; i += 256) {
        const float bi = __bfloat162float(bias[h * d + i]);
        double b = 0.0;
        for (int t = 0; t < n; ++t) {
            const bf16* row = rows + (size_t)(row0 + t) * g.row_elems;
            const float z = __bfloat162float(z_rows[(size_t)(row0 + t) * g.H * d + h * d + i]) + bi;
            float la = (fminf(z, 0.f) - log1pf(expf(-fabsf(z)))) * g.inv_tau;
            la = la < -1e5f ? -1e5f : la;                               // (e^-1e5 is 0 already)
            b += (double)la;
            const float hi = (float)b, q = __bfloat162float(row[g.q_off + h * d + i]) * g.q_scale;
            q_s[t * ld + i] = q;
            k_s[t * ld + i] = __bfloat162float(row[g.k_off + h * d + i]);
            hi_s[t * ld + i] = hi;
            lo_s[t * ld + i] = (float)(b - (double)hi);
            const size_t at = (size_t)(row0 + t) * g.H * d + h * d + i;
            split3_one(q * expf(hi), out.qk[at], out.qk[plane + at], out.qk[2 * plane + at]);
        }
        for (int t = 0; t < n; ++t) {
            const size_t at = 3 * plane + (size_t)(row0 + t) * g.H * d + h * d + i;
            const float left = (float)(b - ((double)hi_s[t * ld + i] + (double)lo_s[t * ld + i]));
            split3_one(k_s[t * ld + i] * expf(left), out.qk[at], out.qk[plane + at], out.qk[2 * plane + at]);
        }
        out.grow[((size_t)place * g.H + h) * d + i] = expm1f((float)b);
    }
    __syncthreads();
    const int t = threadIdx.x >> 4, s = threadIdx.x & 15;
    if (t >= n) return;
    float acc[2] = {0.f, 0.f};
    if (s <= t) {
        for (int i = 0; i < d; i += 2)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float x = (hi_s[t * ld + i + e] - hi_s[s * ld + i + e]) + (lo_s[t * ld + i + e] - lo_s[s * ld + i + e]);
                acc[e] = fmaf(q_s[t * ld + i + e] * k_s[s * ld + i + e], expf(x), acc[e]);
            }
    }
    bf16* dst = out.a + ((size_t)(row0 + t) * g.H + h) * 48 + s;
    split3_one(acc[0] + acc[1], dst[0], dst[16], dst[32]);
}

__host__ __device__ constexpr int gla_stage_bytes(int d) {
    return (6 * GQ * (d + 8) + 3 * GQ * (GQ + 8) + GQ * (GC_COLS + 8)) * 2 + d * 4;
}
__host__ __device__ constexpr int gla_chain_bytes(int d) { return GC_STAGES * gla_stage_bytes(d) + 8 * GQ * 20 * 4; }

// Where few sequences leave SMs idle a chain runs in pieces of `length` chunks at the same time, in two launches: STATES takes every piece
// but a sequence's last from a state of zeros (its first from the stored state) to its end and leaves that, the piece's decay and a copy
// of the stored state; then the pieces run as WHOLE chains do, each from the states before it folded together.  The decay is kept as itself
// and as decay - 1: what a piece of hundreds of tokens leaves of a state may be its ten-thousandth part, which S + S (decay - 1) has at
// the precision of S, and of a state that hardly decays S decay rounds away what S + S (decay - 1) keeps.  The fold takes the one that does not cancel.
struct GlaPieces {
    int length, most;                        // chunks a piece; pieces a sequence at most (0: whole chains)
    float *ends, *grows;                     // [seq][most + 1][H][dv][d]: the stored state, then a piece's end; [seq][most][2][H][d]: decay - 1, decay
};
enum { GLA_WHOLE = 0, GLA_STATES = 1 };

template <int NK, int PHASE>                 // d = 64 NK key channels: 16 NK a warp
__global__ void __launch_bounds__(256)
gla_chain_kernel(const bf16* __restrict__ rows, GlaChunkShape g, GlaChunkScratch in, const int* __restrict__ seq_slot,
                 const int* __restrict__ seq_first_row, const int* __restrict__ seq_start, const int* __restrict__ seq_end,
                 float* __restrict__ state, float* __restrict__ o_out, GlaPieces pieces) {
    constexpr int D = 64 * NK, LDK = D + 8, LDA = GQ + 8, LDV = GC_COLS + 8, STAGE = gla_stage_bytes(D);
    constexpr int Q_AT = 0, K_AT = 3 * GQ * LDK * 2, A_AT = 2 * K_AT, V_AT = A_AT + 3 * GQ * LDA * 2, G_AT = V_AT + GQ * LDV * 2;
    extern __shared__ __align__(16) unsigned char gla_raw[];
    float* sum_s = reinterpret_cast<float*>(gla_raw + GC_STAGES * STAGE);            // [8 warps][16 tokens][20]
    const int seq = pieces.most ? blockIdx.x / pieces.most : blockIdx.x, piece = pieces.most ? blockIdx.x % pieces.most : 0;
    const int h = blockIdx.y, col0 = blockIdx.z * GC_COLS;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, pt = warp >> 2, quarter = warp & 3;
    const int gr = lane >> 2, gc = (lane & 3) * 2, lr = lane & 7, lm = lane >> 3;
    grid_dependents_launch();
    const int slot = seq_slot[seq], row0 = seq_first_row[seq], n_tok = seq_end[seq] - seq_start[seq];
    if (n_tok <= 0) return;
    grid_dependency_wait();
    const uint32_t raw = (uint32_t)__cvta_generic_to_shared(gla_raw);
    const size_t plane = (size_t)g.n_tok * g.H * D;
    const int chunks = (n_tok + GQ - 1) / GQ, c0 = piece * pieces.length, c1 = pieces.most ? min(chunks, c0 + pieces.length) : chunks;
    if (c0 >= chunks || (PHASE == GLA_STATES && c1 == chunks)) return;
    const size_t place0 = (size_t)pieces_before(seq_start, seq_end, seq, GQ);
    // this thread's pieces: column qi of rows qx, qx + STEP, ... of the weighted queries and keys; one piece of A, of the values
    // and of the decays (fewer threads bring those)
    constexpr int STEP = 256 / (D / 8);
    const int qi = tid % (D / 8) * 8, qx = tid / (D / 8), at_ = tid / 6, ai = tid % 6, vt = tid / (GC_COLS / 8), vi = tid % (GC_COLS / 8) * 8;
    const size_t hd = (size_t)g.H * D;
    const bf16* qk0 = in.qk + (size_t)row0 * hd + h * D + qi;
    const bf16* a0 = in.a + ((size_t)(row0 + at_) * g.H + h) * 48 + ai * 8;
    const bf16* v0 = rows + (size_t)(row0 + vt) * g.row_elems + g.v_off + h * g.dv + col0 + vi;
    const float* g0 = in.grow + (place0 * g.H + h) * D + tid * 4;
    auto fetch = [&](int c) {                                              // (a group for every chunk, an empty one past the last)
        if (c < c1) {
            const uint32_t to = raw + (c % GC_STAGES) * STAGE;
            const int n = n_tok - c * GQ;                                  // tokens from the chunk's first on
            const bf16* q = qk0 + (size_t)c * GQ * hd;
            const uint32_t q_to = to + Q_AT + (qx * LDK + qi) * 2;
#pragma unroll
            for (int it = PHASE == GLA_STATES ? 3 * GQ / STEP : 0; it < 6 * GQ / STEP; ++it) {      // (states: the keys alone)
                const int x = qx + it * STEP, t = x % GQ;
                const bool ok = t < n;
                copy16_or_zero(q_to + it * STEP * LDK * 2, q + (x / GQ) * plane + (ok ? t : 0) * hd, ok);
            }
            if (PHASE != GLA_STATES && tid < GQ * 6) copy16_or_zero(to + A_AT + (((ai >> 1) * GQ + at_) * LDA + (ai & 1) * 8) * 2, at_ < n ? a0 + (size_t)c * GQ * g.H * 48 : in.a, at_ < n);
            if (tid < GQ * (GC_COLS / 8)) copy16_or_zero(to + V_AT + (vt * LDV + vi) * 2, vt < n ? v0 + (size_t)c * GQ * g.row_elems : rows, vt < n);
            if (tid < D / 4) copy16_or_zero(to + G_AT + tid * 16, g0 + (size_t)c * hd, true);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    // S[col][channel]: tile j holds channels n0 + 8 j + gc, + 1 of columns col0 + 16 pt + gr (0, 1) and + 8 (2, 3)
    const int n0 = quarter * 16 * NK;
    float S[2 * NK][4];
    float* st = slot >= 0 ? state + (((size_t)slot * g.H + h) * g.dv + col0 + 16 * pt) * D + n0 : nullptr;
    // this thread's places in state number x of the sequence's pieces (0: the stored one, q + 1: the end of piece q)
    auto end_of = [&](int x) { return pieces.ends + ((((size_t)seq * (pieces.most + 1) + x) * g.H + h) * g.dv + col0 + 16 * pt) * D + n0; };
    auto load_state = [&](const float* from, float (&to)[2 * NK][4]) {
#pragma unroll
        for (int j = 0; j < 2 * NK; ++j) {
            float2 a = make_float2(0.f, 0.f), b = a;
            if (from != nullptr) {
                a = *reinterpret_cast<const float2*>(from + (size_t)gr * D + 8 * j + gc);
                b = *reinterpret_cast<const float2*>(from + (size_t)(gr + 8) * D + 8 * j + gc);
            }
            to[j][0] = a.x; to[j][1] = a.y; to[j][2] = b.x; to[j][3] = b.y;
        }
    };
    auto store_state = [&](float* to) {
#pragma unroll
        for (int j = 0; j < 2 * NK; ++j) {
            *reinterpret_cast<float2*>(to + (size_t)gr * D + 8 * j + gc) = make_float2(S[j][0], S[j][1]);
            *reinterpret_cast<float2*>(to + (size_t)(gr + 8) * D + 8 * j + gc) = make_float2(S[j][2], S[j][3]);
        }
    };
    if (PHASE == GLA_STATES) {
        load_state(piece == 0 ? st : nullptr, S);
        if (piece == 0) store_state(end_of(0));
    } else if (c1 - c0 == chunks) load_state(st, S);
    else {
        // (the stored state's copy: the last piece may have written the state by now)
        load_state(end_of(piece == 0 ? 0 : 1), S);
        for (int q = 1; q < piece; ++q) {
            const float* gq = pieces.grows + (((size_t)seq * pieces.most + q) * 2 * g.H + h) * D + n0;
            float e[2 * NK][4];
            load_state(end_of(q + 1), e);
#pragma unroll
            for (int j = 0; j < 2 * NK; ++j) {
                const float2 gw = *reinterpret_cast<const float2*>(gq + 8 * j + gc), keep = *reinterpret_cast<const float2*>(gq + hd + 8 * j + gc);
                auto fold = [](float s, float grow, float decay, float end) { return decay < 0.5f ? fmaf(s, decay, end) : s + fmaf(s, grow, end); };
                S[j][0] = fold(S[j][0], gw.x, keep.x, e[j][0]);
                S[j][1] = fold(S[j][1], gw.y, keep.y, e[j][1]);
                S[j][2] = fold(S[j][2], gw.x, keep.x, e[j][2]);
                S[j][3] = fold(S[j][3], gw.y, keep.y, e[j][3]);
            }
        }
    }
    float piece_grow = 0.f, piece_decay = 1.f;                             // of channel tid over the piece's chunks
    for (int c = 0; c < GC_STAGES - 1; ++c) fetch(c0 + c);
    for (int c = c0; c < c1; ++c) {
        asm volatile("cp.async.wait_group %0;" ::"n"(GC_STAGES - 2) : "memory");
        __syncthreads();                                                   // chunk c is there; chunk c - 1 and the sums have been read
        fetch(c + GC_STAGES - 1);
        const uint32_t at = raw + (c % GC_STAGES) * STAGE;
        const float* grow = reinterpret_cast<const float*>(gla_raw + (c % GC_STAGES) * STAGE + G_AT);
        if (PHASE == GLA_STATES && tid < D) {
            piece_grow += fmaf(piece_grow, grow[tid], grow[tid]);
            piece_decay *= 1.f + grow[tid];
        }
        // o: this quarter's channels of the state; the first quarter adds the chunk's own tokens
        if constexpr (PHASE != GLA_STATES) {
            float hi[2][4], rest[2][4];
#pragma unroll
            for (int p = 0; p < 2; ++p)
#pragma unroll
                for (int e = 0; e < 4; ++e) hi[p][e] = rest[p][e] = 0.f;
#pragma unroll
            for (int k = 0; k < NK; ++k) {
                uint32_t a[3][4], b[3][2][2];                                  // b: [part][columns 0..7, 8..15][channels 0..7, 8..15]
#pragma unroll
                for (int z = 0; z < 3; ++z)
                    ldmatrix4(a[z], at + Q_AT + ((z * GQ + lr + (lm & 1) * 8) * LDK + n0 + 16 * k + (lm >> 1) * 8) * 2);
#pragma unroll
                for (int p = 0; p < 2; ++p)
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        split3(S[2 * k + e][2 * p], S[2 * k + e][2 * p + 1], b[0][p][e], b[1][p][e], b[2][p][e]);
#pragma unroll
                for (int p = 0; p < 2; ++p) mma_16816(rest[p], a[2], b[0][p][0], b[0][p][1]);
#pragma unroll
                for (int p = 0; p < 2; ++p) mma_16816(hi[p], a[0], b[0][p][0], b[0][p][1]);
#pragma unroll
                for (int p = 0; p < 2; ++p) mma_16816(rest[p], a[1], b[1][p][0], b[1][p][1]);
#pragma unroll
                for (int p = 0; p < 2; ++p) mma_16816(rest[p], a[0], b[2][p][0], b[2][p][1]);
#pragma unroll
                for (int p = 0; p < 2; ++p) mma_16816(rest[p], a[1], b[0][p][0], b[0][p][1]);
#pragma unroll
                for (int p = 0; p < 2; ++p) mma_16816(rest[p], a[0], b[1][p][0], b[1][p][1]);
            }
            if (quarter == 0) {
                uint32_t b[4];
                ldmatrix4_trans(b, at + V_AT + ((lr + (lm & 1) * 8) * LDV + 16 * pt + (lm >> 1) * 8) * 2);
                float own[2][4];
#pragma unroll
                for (int p = 0; p < 2; ++p)
#pragma unroll
                    for (int e = 0; e < 4; ++e) own[p][e] = 0.f;
                if (__all_sync(0xffffffffu, all_finite(b[0], b[1], b[2], b[3]))) {
#pragma unroll
                    for (int z = 2; z >= 0; --z) {
                        uint32_t a[4];
                        ldmatrix4(a, at + A_AT + ((z * GQ + lr + (lm & 1) * 8) * LDA + (lm >> 1) * 8) * 2);
#pragma unroll
                        for (int p = 0; p < 2; ++p) mma_16816(z ? rest[p] : own[p], a, b[2 * p], b[2 * p + 1]);
                    }
                } else {
                    // an infinite or NaN value counts from its token on: the products' zeros would carry it to the tokens before
                    const bf16* stage = reinterpret_cast<const bf16*>(gla_raw + (c % GC_STAGES) * STAGE);
                    const bf16 *a_s = stage + A_AT / 2, *v_s = stage + V_AT / 2 + 16 * pt + gc;
#pragma unroll
                    for (int p = 0; p < 2; ++p)
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            for (int s = 0; s <= gr + 8 * (e >> 1); ++s) {
                                const bf16* as = a_s + (gr + 8 * (e >> 1)) * LDA + s;
                                const float w = __bfloat162float(as[0]) + (__bfloat162float(as[GQ * LDA]) + __bfloat162float(as[2 * GQ * LDA]));
                                own[p][e] = fmaf(w, __bfloat162float(v_s[s * LDV + 8 * p + (e & 1)]), own[p][e]);
                            }
                }
#pragma unroll
                for (int p = 0; p < 2; ++p)
#pragma unroll
                    for (int e = 0; e < 4; ++e) hi[p][e] += own[p][e];
            }
#pragma unroll
            for (int p = 0; p < 2; ++p)
#pragma unroll
                for (int e = 0; e < 2; ++e)
                    *reinterpret_cast<float2*>(sum_s + (warp * GQ + gr + 8 * e) * 20 + 8 * p + gc) =
                        make_float2(hi[p][2 * e] + rest[p][2 * e], hi[p][2 * e + 1] + rest[p][2 * e + 1]);
        }
        // the state at the chunk's end
        {
            uint32_t v[4];
            ldmatrix4_trans(v, at + V_AT + ((lr + (lm >> 1) * 8) * LDV + 16 * pt + (lm & 1) * 8) * 2);
#pragma unroll
            for (int j = 0; j < NK; ++j) {
                uint32_t b[3][4];
#pragma unroll
                for (int z = 0; z < 3; ++z)
                    ldmatrix4_trans(b[z], at + K_AT + ((z * GQ + lr + (lm & 1) * 8) * LDK + n0 + 16 * j + (lm >> 1) * 8) * 2);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float x[4] = {0.f, 0.f, 0.f, 0.f}, y[4] = {0.f, 0.f, 0.f, 0.f};
                    mma_16816(y, v, b[2][2 * e], b[2][2 * e + 1]);
                    mma_16816(x, v, b[0][2 * e], b[0][2 * e + 1]);
                    mma_16816(y, v, b[1][2 * e], b[1][2 * e + 1]);
                    const float2 gw = *reinterpret_cast<const float2*>(grow + n0 + 16 * j + 8 * e + gc);
                    float(&s)[4] = S[2 * j + e];
                    s[0] += fmaf(s[0], gw.x, x[0] + y[0]);
                    s[1] += fmaf(s[1], gw.y, x[1] + y[1]);
                    s[2] += fmaf(s[2], gw.x, x[2] + y[2]);
                    s[3] += fmaf(s[3], gw.y, x[3] + y[3]);
                }
            }
        }
        if constexpr (PHASE != GLA_STATES) {
            __syncthreads();                                               // the quarters' sums are there
            const int t = tid >> 4, col = (tid & 15) * 2, p = col >> 4;
            if (c * GQ + t < n_tok) {
                const float* src = sum_s + (p * 4 * GQ + t) * 20 + (col & 15);
                float2 y = *reinterpret_cast<const float2*>(src);
#pragma unroll
                for (int q = 1; q < 4; ++q) {
                    const float2 w = *reinterpret_cast<const float2*>(src + q * GQ * 20);
                    y.x += w.x;
                    y.y += w.y;
                }
                *reinterpret_cast<float2*>(o_out + ((size_t)(row0 + c * GQ + t) * g.H + h) * g.dv + col0 + col) = y;
            }
        }
    }
    if (PHASE == GLA_STATES) {
        store_state(end_of(piece + 1));
        if (blockIdx.z == 0 && tid < D) {
            float* to = pieces.grows + (((size_t)seq * pieces.most + piece) * 2 * g.H + h) * D + tid;
            to[0] = piece_grow;
            to[hd] = piece_decay;
        }
    } else if (st != nullptr && c1 == chunks) store_state(st);
}

// How a step's chains are cut: where the sequences' chains leave SMs idle, into pieces that fill two CTAs an SM, of 16 chunks or more.
// (`most` bounds a sequence's pieces by the step's tokens: the host does not know the lengths.)
static GlaPieces gla_pieces(int n_tok, int n_seq, int H, int d, int dv) {
    GlaPieces p = {0, 0, nullptr, nullptr};
    const long long ctas = (long long)n_seq * H * (dv / GC_COLS), chunks = n_tok / GQ + 1;
    if (d > 128 || ctas > 148) return p;                  // (256 channels: one CTA an SM)
    const long long want = 296 / ctas * n_seq;            // pieces in all
    long long length = (chunks + want - 1) / want;
    if (length < 16) length = 16;
    const long long most = (chunks + length - 1) / length;
    if (most < 2) return p;                               // (p.most is 0: no pieces)
    p.length = (int)length;
    p.most = (int)most;
    return p;
}
// Whether pieces take less time than whole chains, whose time is that of the longest sequence's.  In chunks of a CTA that has an SM to itself
// (1.18 us at 128 key channels): of two CTAs on an SM each takes 1.64 a chunk; for the states alone 0.42 and 0.76; a launch and the fold
// cost 8.5.  All of it, with the terms' kernel, 8 heads of 128 x 256, whole -> pieces: one sequence of 2,048 tokens 208 -> 153 us, of 1,024 112 -> 89,
// of 600 79 -> 81 (whole), of 300 54 -> 62 (whole); two of 1,024 138 -> 153 (whole), of 2,000 and 50 204 -> 157; 4 heads, one of 600 75 -> 62.
static bool gla_pieces_pay(const GlaPieces& p, int n_tok, int n_seq, int H, int dv, int longest) {
    const int per = H * (dv / GC_COLS);                   // CTAs a piece
    const int whole = (longest + GQ - 1) / GQ;
    const double pieces = ceil(n_tok / GQ / (double)p.length + 0.5 * (n_seq - 1)), states = pieces - n_seq;
    return p.length * ((pieces * per > 148 ? 1.64 : 1.0) + (states * per > 148 ? 0.76 : 0.42)) + 8.5 < whole;
}
static long long gla_piece_floats(const GlaPieces& p, int n_seq, int H, int d, int dv) {
    return p.most ? (long long)n_seq * H * d * ((long long)(p.most + 1) * dv + 2 * p.most) : 0;
}

template <int NK, int PHASE>
static int gla_chain_launch(const bf16* rows, const GlaChunkShape& g, const GlaChunkScratch& in, const int* seq_slot, const int* seq_first_row,
                            const int* seq_start, const int* seq_end, int n_seq, float* state, float* o_out, const GlaPieces& pieces,
                            cudaStream_t stream) {
    constexpr int bytes = gla_chain_bytes(64 * NK);
    const cudaError_t e = cudaFuncSetAttribute(gla_chain_kernel<NK, PHASE>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return fail("gla_chunks: shared memory of %d bytes refused: %s", bytes, cudaGetErrorString(e));
    // (launched once its predecessor is over: its few CTAs run long and have to lie on SMs of their own)
    return launch_kernel_after("gla_chain", gla_chain_kernel<NK, PHASE>, dim3(n_seq * (pieces.most ? pieces.most : 1), g.H, g.dv / GC_COLS), dim3(256),
                               bytes, stream, 1, rows, g, in, seq_slot, seq_first_row, seq_start, seq_end, state, o_out, pieces);
}

}  // namespace janis

using namespace janis;

static long long gla_chunk_floats(int n_tok, int n_seq, int H, int d) {
    return 3LL * n_tok * H * d + 24LL * n_tok * H + ((long long)n_tok / GQ + n_seq) * H * d;         // (d is a multiple of 64)
}

// Floats of scratch for a step of n_tok tokens in n_seq sequences: what lets its chains run in pieces too; 0 where the chunked form does not take the sizes.
JANIS_EXPORT long long janis_gla_chunks_floats(int n_tok, int n_seq, int H, int d, int dv) {
    if (n_tok <= 0 || n_seq <= 0 || H <= 0 || H > 65535 || !(d == 64 || d == 128 || d == 256) || dv <= 0 || dv % GC_COLS) return 0;
    return gla_chunk_floats(n_tok, n_seq, H, d) + gla_piece_floats(gla_pieces(n_tok, n_seq, H, d, dv), n_seq, H, d, dv);
}

// The same for whole chains, which is the least that janis_gla_chunks takes.
JANIS_EXPORT long long janis_gla_chunks_least(int n_tok, int n_seq, int H, int d, int dv) {
    return janis_gla_chunks_floats(n_tok, n_seq, H, d, dv) ? gla_chunk_floats(n_tok, n_seq, H, d) : 0;
}

// longest: tokens of the longest sequence, for the choice between pieces and whole chains (0: taken to be the mean)
JANIS_EXPORT int janis_gla_chunks(const void* rows, int row_elems, int q_off, int k_off, int v_off, const void* z, const void* bias, int n_tok,
                                  const int* seq_slot, const int* seq_first_row, const int* seq_start, const int* seq_end, float* state,
                                  float* o_out, int n_seq, int H, int d, int dv, float q_scale, float tau, int longest, void* scratch,
                                  long long scratch_floats, cudaStream_t stream) {
    if (n_seq <= 0 || n_tok <= 0) return 0;
    const long long all = janis_gla_chunks_floats(n_tok, n_seq, H, d, dv), need = janis_gla_chunks_least(n_tok, n_seq, H, d, dv);
    if (need == 0 || scratch == nullptr || scratch_floats < need)
        return fail("gla_chunks: %d heads of %d x %d (or a scratch of %lld floats) are not taken", H, d, dv, scratch_floats);
    if (!(tau > 0.f)) return fail("gla_chunks: tau must be positive");
    if (row_elems % 8 || v_off % 8 || (((uintptr_t)rows | (uintptr_t)scratch) & 15) || (((uintptr_t)state | (uintptr_t)o_out) & 7))
        return fail("gla_chunks: rows of %d elements, values at %d: not in whole pieces of 16 bytes", row_elems, v_off);
    GlaChunkShape g;
    g.row_elems = row_elems; g.q_off = q_off; g.k_off = k_off; g.v_off = v_off; g.H = H; g.d = d; g.dv = dv; g.n_tok = n_tok;
    g.q_scale = q_scale; g.inv_tau = 1.0f / tau;
    const GlaChunkScratch s = gla_chunk_scratch(scratch, g);
    const size_t bytes = (size_t)4 * GQ * (d + 1) * sizeof(float);
    const cudaError_t e = cudaFuncSetAttribute(gla_chunk_terms_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return fail("gla_chunks: shared memory of %zu bytes refused: %s", bytes, cudaGetErrorString(e));
    if (launch_kernel("gla_chunk_terms", gla_chunk_terms_kernel, dim3(n_tok / GQ + n_seq, H), dim3(256), bytes, stream, 1, (const bf16*)rows,
                      (const bf16*)z, (const bf16*)bias, g, n_seq, seq_first_row, seq_start, seq_end, s))
        return 1;
    GlaPieces pieces = gla_pieces(n_tok, n_seq, H, d, dv);
    if (longest <= 0) longest = (n_tok + n_seq - 1) / n_seq;
    if (scratch_floats < all || (pieces.most && !gla_pieces_pay(pieces, n_tok, n_seq, H, dv, longest))) pieces.most = 0;
    if (pieces.most) {
        pieces.ends = (float*)scratch + need;
        pieces.grows = pieces.ends + (long long)n_seq * (pieces.most + 1) * H * dv * d;
    }
#define JANIS_GLA_CHAIN(NK)                                                                                                       \
    if (pieces.most && gla_chain_launch<NK, GLA_STATES>((const bf16*)rows, g, s, seq_slot, seq_first_row, seq_start, seq_end, n_seq, state, o_out, pieces, stream)) \
        return 1;                                                                                                                  \
    return gla_chain_launch<NK, GLA_WHOLE>((const bf16*)rows, g, s, seq_slot, seq_first_row, seq_start, seq_end, n_seq, state, o_out, pieces, stream);
    if (d == 64) { JANIS_GLA_CHAIN(1) }
    if (d == 128) { JANIS_GLA_CHAIN(2) }
    JANIS_GLA_CHAIN(4)
#undef JANIS_GLA_CHAIN
}
