// The state-space-duality recurrence of a prompt, 64 tokens at a time on the tensor cores (bfloat16 inputs):
//
//   S_t[p, n] = e^(x_t) S_(t-1)[p, n] + delta_t u_t[p] B_t[n],   o_t[p] = sum_n S_t[p, n] C_t[n] + D u_t[p],
//   x_t = delta_t A, delta_t = softplus(dt_t + bias), one A, D and delta per head
//
// With c_t the sum of x from the chunk's start up to t, the tokens of a chunk are three products:
//
//   o_t   = e^(c_t) S_0 C_t  +  sum_(s <= t) M[t, s] u_s  + D u_t,     M[t, s] = (C_t . B_s) e^(c_t - c_s) delta_s
//   S_end = e^(c_end) S_0 + sum_s (e^(c_end - c_s) delta_s u_s) B_s^T
//
// What the recurrence keeps as floats stays float: S, M and the weighted inputs enter the products as sums of three
// bfloat16 numbers, so that every product is exact and the sums are float.  Each sum over hi parts and over the rest
// has an accumulator of its own, and S takes a chunk's sum by one rounded addition: the tensor cores cut their sums
// off instead of rounding them, which over hundreds of additions into one accumulator would add up.  c_t is summed in
// double and kept as two floats, so that the difference of two of them is as exact as one x; the decay of a whole chunk
// is applied as S + S (e^c - 1).
//
// Two things the products cannot take: an infinite or NaN input u_s, which the zeros of M above the diagonal would carry to the
// tokens before it (0 x inf), and an A above 0, whose e^(c_t) may overflow where S_0 is 0.  A chunk that meets either runs as
// the recurrence is written, one token after another, from the same registers.
//
// A CTA owns up to 64 channels of a sequence's head, two warps to 16 of them: each keeps S for half of the states in registers (as
// the accumulators of the last product, which are at the same time the second operands of the first one), adds up
// e^(c_t) S_0 C_t over its states, and gives its partner the sums of those 32 tokens of a chunk whose results the partner
// finishes.  Tokens come by cp.async a chunk ahead, and one warp forms a chunk's decays while the chunk before is
// computed.  What bounds it is the chain of a chunk: some 2,000 instructions a warp and three barriers.  Two warps a channel
// tile instead of one hide each other's waits (328 us -> 218); few sequences' chains are shared by two CTAs (220 -> 157).
//
// 72 heads of 64 channels, 128 states, with the scan of selective_scan_staged_kernel (an issue slot in two, 263 instructions
// a token and warp) and its kernel for the step sizes: one sequence of 2,048 tokens 954 -> 209 us (157 shared), 300 tokens 148 -> 39, eight
// of 512 1,400 -> 229, eight of 8 49 -> 29, one of 4 27 -> 23.  Errors against 64 bits over 2,048 tokens: results 1.1e-7 for
// 1.0e-7, states 0.8e-7 for 0.7e-7; where the states remember a thousand tokens 1.5e-7 for 5.5e-7 and 1.2e-7 for 6.6e-7.
#include "mma_bf16.cuh"

namespace janis {

constexpr int DQ = 64;                       // tokens a chunk
constexpr int DUP = 64 + 8;                  // padded row of u
constexpr int MTP = 16 + 8;                  // padded row of a 16 x 16 tile of M

struct DualityShape {
    int u_stride, u_off, dt_stride, dt_off, bc_stride, b_off, c_off;
    int C, cph, cpg;
};

__host__ __device__ constexpr int duality_stage_elems(int N) { return 2 * DQ * (N + 8) + DQ * DUP; }
constexpr int DXP = 64 + 8;                  // padded row of the exchanged sums
__host__ __device__ constexpr size_t duality_smem(int N) {
    return (size_t)2 * duality_stage_elems(N) * 2 + (size_t)10 * 3 * 16 * MTP * 2 + (size_t)DQ * DXP * 4 + 2 * (5 * DQ + 4) * 4;
}

__device__ __forceinline__ float duality_softplus(float v) { return v > 20.f ? v : log1pf(expf(v)); }

// Where few sequences leave half of the SMs idle, two CTAs (a cluster) share a chain: the first runs its first part; the second takes
// the state alone through that part, then runs the rest.  This is where the rest starts, in tokens: a chunk's state alone takes 0.58 of
// a chunk's time (the decays, which one warp forms, stay), so that at seven tenths both take as long (x = 0.58 x + 1 - x; at three
// fifths 166 us for 157).  n_tok for chains of less than four chunks, which one CTA runs.  The bits are those of one CTA: each chunk's
// state is formed by the same instructions.
__device__ __forceinline__ int duality_split(int n_tok) {
    const int chunks = (n_tok + DQ - 1) / DQ;
    return chunks < 4 ? n_tok : (7 * chunks + 5) / 10 * DQ;
}

template <int NK>                            // N = 16 NK states, NK even
__global__ void __launch_bounds__(256)
duality_scan_kernel(const bf16* __restrict__ u_rows, const bf16* __restrict__ dt_rows, const bf16* __restrict__ bc_rows,
                    const float* __restrict__ dt_bias, const float* __restrict__ A, const float* __restrict__ D,
                    DualityShape g, int parts, const int* __restrict__ seq_slot, const int* __restrict__ seq_first_row,
                    const int* __restrict__ seq_start, const int* __restrict__ seq_end, float* __restrict__ state,
                    float* __restrict__ out) {
    constexpr int N = 16 * NK, NH = NK / 2, LDN = N + 8, STAGE = duality_stage_elems(N), SCAL = 5 * DQ + 4;
    extern __shared__ __align__(16) unsigned char duality_raw[];
    bf16* stage_s = reinterpret_cast<bf16*>(duality_raw);                  // [2]: B [64][LDN], C [64][LDN], u [64][DUP]
    bf16* m_s = stage_s + 2 * STAGE;                                       // [10 tiles on and below the diagonal][3][16][MTP]
    float* swap_s = reinterpret_cast<float*>(m_s + 10 * 3 * 16 * MTP);     // [64 tokens][DXP]: sums for the partner
    float* scal_s = swap_s + DQ * DXP;                                     // [2] of the decays below
    const int seq = blockIdx.x / parts, part = blockIdx.x % parts, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5, npt = nwarp >> 1;
    const int half = warp >= npt, pt = warp - half * npt;                  // half of the states, tile of 16 channels
    const int c0 = blockIdx.y * npt * 16, cw = c0 + pt * 16, head = c0 / g.cph, group = c0 / g.cpg;
    const int gr = lane >> 2, gc = (lane & 3) * 2;                         // a lane's row and first column of an 8 x 8 tile
    const int lr = lane & 7, lm = lane >> 3;                               // row and matrix that the lane addresses in ldmatrix
    grid_dependents_launch();
    const int slot = seq_slot[seq], row0 = seq_first_row[seq], n_tok = seq_end[seq] - seq_start[seq];
    const int split = parts == 2 ? duality_split(n_tok) : n_tok;
    if (n_tok <= 0 || (part == 1 && split == n_tok)) return;
    const int stop = part == 0 ? split : n_tok;                            // (split < n_tok: whole chunks)
    const float Ah = A[head], Dh = D[head], bias = dt_bias[head];
    grid_dependency_wait();

    const uint32_t stage_a = (uint32_t)__cvta_generic_to_shared(stage_s);
    const uint32_t m_a = (uint32_t)__cvta_generic_to_shared(m_s);
    const bf16* bsrc = bc_rows + (size_t)row0 * g.bc_stride + g.b_off + (size_t)group * N;
    const int c_from_b = g.c_off - g.b_off;
    // this thread's pieces: one column of the rows of B and C side by side, one of the inputs'
    const int bq = tid % (4 * NK), bt = tid / (4 * NK), b_step = blockDim.x / (4 * NK), which = bq >= 2 * NK, bi = (bq - which * 2 * NK) * 8;
    const int ut = tid / (2 * npt), ui = tid % (2 * npt) * 8;              // (64 npt threads: 32 rows at a time)
    bsrc += (which ? c_from_b : 0) + bi;
    const bf16* usrc = u_rows + (size_t)row0 * g.u_stride + g.u_off + c0 + ui;
    auto fetch = [&](int t0, int buf) {
        const uint32_t to = stage_a + buf * STAGE * 2, b_to = to + (which * DQ * LDN + bi) * 2;
        const int n = n_tok - t0;
        const bf16* b0 = bsrc + (size_t)t0 * g.bc_stride;
#pragma unroll 4
        for (int t = which && part == 1 && t0 < split ? DQ : bt; t < DQ; t += b_step) {              // (the state alone: no C)
            const bool ok = t < n;
            copy16_or_zero(b_to + t * LDN * 2, b0 + (ok ? (size_t)t * g.bc_stride : 0), ok);
        }
        const bf16* u0 = usrc + (size_t)t0 * g.u_stride;
#pragma unroll
        for (int t = ut; t < DQ; t += 32) {
            const bool ok = t < n;
            copy16_or_zero(to + (2 * DQ * LDN + t * DUP + ui) * 2, u0 + (ok ? (size_t)t * g.u_stride : 0), ok);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // The decays of the chunk from t0 on, by one warp (a lane two tokens): c_t = hi + lo, delta_t, e^(c_t),
    // e^(c_end - c_t) delta_t, and e^(c_end) - 1
    const bf16* dsrc = dt_rows + (size_t)row0 * g.dt_stride + g.dt_off + head;
    auto decays = [&](int t0, float* s) {
        float dl[2];
        double c[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int t = t0 + 2 * lane + e;
            const bool in = t < n_tok;
            dl[e] = in ? duality_softplus(__bfloat162float(dsrc[(size_t)t * g.dt_stride]) + bias) : 0.f;
            c[e] = !in ? 0.0 : dl[e] * Ah < -1e5f ? -1e5 : (double)dl[e] * (double)Ah;      // (e^-1e5 is 0 already)
        }
        c[1] += c[0];
        double before = c[1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double v = __shfl_up_sync(0xffffffffu, before, o);
            if (lane >= o) before += v;
        }
        const double end = __shfl_sync(0xffffffffu, before, 31);
        before = __shfl_up_sync(0xffffffffu, before, 1);
        if (lane == 0) before = 0.0;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int t = 2 * lane + e;
            const double ct = before + c[e];
            const float h = (float)ct;
            s[t] = h;
            s[DQ + t] = (float)(ct - (double)h);
            s[2 * DQ + t] = dl[e];
            s[3 * DQ + t] = expf(h);
            s[4 * DQ + t] = expf((float)(end - ct)) * dl[e];
        }
        if (lane == 0) s[5 * DQ] = expm1f((float)end);
    };

    // S[p][n]: tile j holds n = n0 + 8 j + gc, + 1 of channels cw + gr (0, 1) and cw + gr + 8 (2, 3)
    const int n0 = half * 16 * NH;
    float S[2 * NH][4];
    float* st = slot >= 0 ? state + ((size_t)slot * g.C + cw) * N + n0 : nullptr;
#pragma unroll
    for (int j = 0; j < 2 * NH; ++j) {
        float2 a = make_float2(0.f, 0.f), b = a;
        if (st != nullptr) {
            a = *reinterpret_cast<const float2*>(st + (size_t)gr * N + 8 * j + gc);
            b = *reinterpret_cast<const float2*>(st + (size_t)(gr + 8) * N + 8 * j + gc);
        }
        S[j][0] = a.x; S[j][1] = a.y; S[j][2] = b.x; S[j][3] = b.y;
    }
    // (both CTAs have read the stored state before the second one writes it)
    if (split < n_tok) asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;\n" ::: "memory");

    // Tokens one after another: for the chunks that the products cannot take
    auto plain = [&](int t0, int n_here, int buf, bool results) {
        const bf16 *B_s = stage_s + (size_t)buf * STAGE + n0, *C_s = B_s + DQ * LDN, *u_s = stage_s + (size_t)buf * STAGE + 2 * DQ * LDN + pt * 16;
        const float* delta_s = scal_s + buf * SCAL + 2 * DQ;
        for (int t = 0; t < n_here; ++t) {
            const float dl = delta_s[t], grown = expm1f(dl * Ah), ua = __bfloat162float(u_s[t * DUP + gr]), ub = __bfloat162float(u_s[t * DUP + gr + 8]);
            float ya = 0.f, yb = 0.f;
#pragma unroll
            for (int j = 0; j < 2 * NH; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const float b = __bfloat162float(B_s[t * LDN + 8 * j + gc + e]), c = __bfloat162float(C_s[t * LDN + 8 * j + gc + e]);
                    S[j][e] += fmaf(S[j][e], grown, dl * ua * b);
                    S[j][2 + e] += fmaf(S[j][2 + e], grown, dl * ub * b);
                    ya = fmaf(S[j][e], c, ya);
                    yb = fmaf(S[j][2 + e], c, yb);
                }
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
                ya += __shfl_xor_sync(0xffffffffu, ya, o);
                yb += __shfl_xor_sync(0xffffffffu, yb, o);
            }
            if ((lane & 3) == 0 && half) swap_s[t * DXP + pt * 16 + gr] = ya, swap_s[t * DXP + pt * 16 + gr + 8] = yb;
            if ((lane & 3) == 0 && !half && results) {
                float* y = out + (size_t)(row0 + t0 + t) * g.C + cw + gr;
                y[0] = fmaf(Dh, ua, ya), y[8] = fmaf(Dh, ub, yb);
            }
        }
        __syncthreads();
        for (int i = lane; i < 16 * n_here && !half && results; i += 32) {
            // (a lane's own warp wrote what it adds to, before the barrier)
            const int t = i >> 4, ch = i & 15;
            out[(size_t)(row0 + t0 + t) * g.C + cw + ch] += swap_s[t * DXP + pt * 16 + ch];
        }
    };
    const bool shrinks = Ah <= 0.f;

    fetch(0, 0);
    if (warp == nwarp - 1) decays(0, scal_s);
    int buf = 0;
    for (int t0 = 0; t0 < stop; t0 += DQ, buf ^= 1) {
        const bool more = t0 + DQ < stop, results = part == 0 || t0 >= split;
        const int n_here = min(DQ, n_tok - t0), tiles = (n_here + 15) / 16;
        if (more) {
            fetch(t0 + DQ, buf ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        bool good = shrinks;                                               // the inputs that this thread brought are finite
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const uint4 v = *reinterpret_cast<const uint4*>(stage_s + (size_t)buf * STAGE + 2 * DQ * LDN + (ut + 32 * t) * DUP + ui);
            good = good && all_finite(v.x, v.y, v.z, v.w);
        }
        if (!__syncthreads_and(good)) {
            if (more && warp == nwarp - 1) decays(t0 + DQ, scal_s + (buf ^ 1) * SCAL);
            plain(t0, n_here, buf, results);
            __syncthreads();                                               // the buffers have been read
            continue;
        }
        const uint32_t b_a = stage_a + buf * STAGE * 2, c_a = b_a + DQ * LDN * 2, u_a = c_a + DQ * LDN * 2;
        const float* hi_s = scal_s + buf * SCAL;
        const float *lo_s = hi_s + DQ, *delta_s = lo_s + DQ, *grow_s = delta_s + DQ, *left_s = grow_s + DQ;

        // the chunk's start, over this warp's states; tiles of tokens 0 and 3 are the first warp's to finish, 1 and 2 the second's
        float mine[2][2][4];
        if (results) {
            float hi[4][2][4], rest[4][2][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int p = 0; p < 2; ++p)
#pragma unroll
                    for (int e = 0; e < 4; ++e) hi[i][p][e] = rest[i][p][e] = 0.f;
#pragma unroll
            for (int k = 0; k < NH; ++k) {
                uint32_t b[3][2][2];                                       // [part][channels 0..7, 8..15][k 0..7, 8..15]
#pragma unroll
                for (int p = 0; p < 2; ++p)
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        split3(S[2 * k + h][2 * p], S[2 * k + h][2 * p + 1], b[0][p][h], b[1][p][h], b[2][p][h]);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (i >= tiles) break;
                    uint32_t a[4];
                    ldmatrix4(a, c_a + ((16 * i + lr + (lm & 1) * 8) * LDN + n0 + 16 * k + (lm >> 1) * 8) * 2);
#pragma unroll
                    for (int p = 0; p < 2; ++p) mma_16816(rest[i][p], a, b[2][p][0], b[2][p][1]);
#pragma unroll
                    for (int p = 0; p < 2; ++p) mma_16816(hi[i][p], a, b[0][p][0], b[0][p][1]);
#pragma unroll
                    for (int p = 0; p < 2; ++p) mma_16816(rest[i][p], a, b[1][p][0], b[1][p][1]);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const bool own = (i == 1 || i == 2) == (half == 1);
#pragma unroll
                for (int p = 0; p < 2; ++p)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float v = hi[i][p][e] + rest[i][p][e];
                        if (own) mine[i >> 1][p][e] = v;
                        else swap_s[(16 * i + gr + (e >> 1) * 8) * DXP + pt * 16 + 8 * p + gc + (e & 1)] = v;
                    }
            }
        }

        // M, a tile of 16 x 16 at a time
        for (int m = results ? warp : 10; m < tiles * (tiles + 1) / 2; m += nwarp) {
            const int i = m >= 6 ? 3 : m >= 3 ? 2 : m >= 1 ? 1 : 0, j = m - i * (i + 1) / 2;
            float acc[2][2][4];                                            // [even and odd k][8 columns each]
#pragma unroll
            for (int q = 0; q < 2; ++q)
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[q][h][e] = 0.f;
#pragma unroll
            for (int k = 0; k < NK; ++k) {
                uint32_t a[4], b[4];
                ldmatrix4(a, c_a + ((16 * i + lr + (lm & 1) * 8) * LDN + 16 * k + (lm >> 1) * 8) * 2);
                ldmatrix4(b, b_a + ((16 * j + lr + (lm >> 1) * 8) * LDN + 16 * k + (lm & 1) * 8) * 2);
                mma_16816(acc[k & 1][0], a, b[0], b[1]);
                mma_16816(acc[k & 1][1], a, b[2], b[3]);
            }
            const int ta = 16 * i + gr, tb = ta + 8;
            const float ha = hi_s[ta], la = lo_s[ta], hb = hi_s[tb], lb = lo_s[tb];
            bf16* tile = m_s + (size_t)m * 3 * 16 * MTP;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int s = 16 * j + 8 * h + gc;
                const float2 hs = *reinterpret_cast<const float2*>(hi_s + s), ls = *reinterpret_cast<const float2*>(lo_s + s);
                const float2 ds = *reinterpret_cast<const float2*>(delta_s + s);
                float v[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] = acc[0][h][e] + acc[1][h][e];
                v[0] = s <= ta ? v[0] * (expf((ha - hs.x) + (la - ls.x)) * ds.x) : 0.f;
                v[1] = s + 1 <= ta ? v[1] * (expf((ha - hs.y) + (la - ls.y)) * ds.y) : 0.f;
                v[2] = s <= tb ? v[2] * (expf((hb - hs.x) + (lb - ls.x)) * ds.x) : 0.f;
                v[3] = s + 1 <= tb ? v[3] * (expf((hb - hs.y) + (lb - ls.y)) * ds.y) : 0.f;
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    uint32_t p[3];
                    split3(v[2 * r], v[2 * r + 1], p[0], p[1], p[2]);
#pragma unroll
                    for (int z = 0; z < 3; ++z)
                        *reinterpret_cast<uint32_t*>(tile + (z * 16 + gr + 8 * r) * MTP + 8 * h + gc) = p[z];
                }
            }
        }
        if (more && warp == nwarp - 1) decays(t0 + DQ, scal_s + (buf ^ 1) * SCAL);
        if (results) __syncthreads();

        // the chunk's own tokens, and the results of this warp's tiles of tokens
        const bf16* u_s = stage_s + (size_t)buf * STAGE + 2 * DQ * LDN;
        uint32_t ub[4][4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k < tiles && results) ldmatrix4_trans(ub[k], u_a + ((16 * k + lr + (lm & 1) * 8) * DUP + pt * 16 + (lm >> 1) * 8) * 2);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int i = half == 0 ? 3 * q : 1 + q;
            if (i >= tiles || !results) continue;
            float hi[2][2][4], rest[2][4];                                 // (hi: even and odd tiles)
#pragma unroll
            for (int p = 0; p < 2; ++p)
#pragma unroll
                for (int e = 0; e < 4; ++e) hi[0][p][e] = hi[1][p][e] = rest[p][e] = 0.f;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (k > i) break;
                const uint32_t at = m_a + ((i * (i + 1) / 2 + k) * 3 * 16 * MTP + (lr + (lm & 1) * 8) * MTP + (lm >> 1) * 8) * 2;
                uint32_t a[3][4];
#pragma unroll
                for (int z = 0; z < 3; ++z) ldmatrix4(a[z], at + z * 16 * MTP * 2);
#pragma unroll
                for (int p = 0; p < 2; ++p) mma_16816(rest[p], a[2], ub[k][2 * p], ub[k][2 * p + 1]);
#pragma unroll
                for (int p = 0; p < 2; ++p) mma_16816(hi[k & 1][p], a[0], ub[k][2 * p], ub[k][2 * p + 1]);
#pragma unroll
                for (int p = 0; p < 2; ++p) mma_16816(rest[p], a[1], ub[k][2 * p], ub[k][2 * p + 1]);
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int t = 16 * i + gr + 8 * e;
                if (t >= n_here) continue;
                const float grown = grow_s[t];
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    const int ch = pt * 16 + 8 * p + gc;
                    const float2 other = *reinterpret_cast<const float2*>(swap_s + t * DXP + ch);
                    const __nv_bfloat162 u2 = *reinterpret_cast<const __nv_bfloat162*>(u_s + t * DUP + ch);
                    float2 y;
                    y.x = fmaf(Dh, __low2float(u2), fmaf(mine[q][p][2 * e] + other.x, grown, (hi[0][p][2 * e] + hi[1][p][2 * e]) + rest[p][2 * e]));
                    y.y = fmaf(Dh, __high2float(u2), fmaf(mine[q][p][2 * e + 1] + other.y, grown, (hi[0][p][2 * e + 1] + hi[1][p][2 * e + 1]) + rest[p][2 * e + 1]));
                    *reinterpret_cast<float2*>(out + (size_t)(row0 + t0 + t) * g.C + c0 + ch) = y;
                }
            }
        }

        // the state at the chunk's end
        uint32_t w[4][3][4];                                               // the weighted inputs, transposed: [tile of tokens][part]
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (k >= tiles) break;
            uint32_t b[4];
            ldmatrix4_trans(b, u_a + ((16 * k + lr + (lm >> 1) * 8) * DUP + pt * 16 + (lm & 1) * 8) * 2);
#pragma unroll
            for (int h = 0; h < 2; ++h) {                                  // tokens 16 k + 8 h + gc, + 1
                const float2 l = *reinterpret_cast<const float2*>(left_s + 16 * k + 8 * h + gc);
#pragma unroll
                for (int e = 0; e < 2; ++e) {                              // channels gr, gr + 8
                    const uint32_t v = b[2 * h + e];
                    split3(__uint_as_float(v << 16) * l.x, __uint_as_float(v & 0xffff0000u) * l.y, w[k][0][2 * h + e],
                           w[k][1][2 * h + e], w[k][2][2 * h + e]);
                }
            }
        }
        const float grown = hi_s[5 * DQ];
#pragma unroll
        for (int j = 0; j < NH; ++j) {                                     // 16 states at a time
            float hi[2][2][4], lo[2][4];                                   // (hi: even and odd tiles)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int e = 0; e < 4; ++e) hi[0][h][e] = hi[1][h][e] = lo[h][e] = 0.f;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (k >= tiles) break;
                uint32_t b[4];
                ldmatrix4_trans(b, b_a + ((16 * k + lr + (lm & 1) * 8) * LDN + n0 + 16 * j + (lm >> 1) * 8) * 2);
#pragma unroll
                for (int h = 0; h < 2; ++h) mma_16816(lo[h], w[k][2], b[2 * h], b[2 * h + 1]);
#pragma unroll
                for (int h = 0; h < 2; ++h) mma_16816(hi[k & 1][h], w[k][0], b[2 * h], b[2 * h + 1]);
#pragma unroll
                for (int h = 0; h < 2; ++h) mma_16816(lo[h], w[k][1], b[2 * h], b[2 * h + 1]);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int e = 0; e < 4; ++e) S[2 * j + h][e] += fmaf(S[2 * j + h][e], grown, (hi[0][h][e] + hi[1][h][e]) + lo[h][e]);
        }
        __syncthreads();                                                   // the buffers have been read
    }
    if (st != nullptr && stop == n_tok) {
#pragma unroll
        for (int j = 0; j < 2 * NH; ++j) {
            *reinterpret_cast<float2*>(st + (size_t)gr * N + 8 * j + gc) = make_float2(S[j][0], S[j][1]);
            *reinterpret_cast<float2*>(st + (size_t)(gr + 8) * N + 8 * j + gc) = make_float2(S[j][2], S[j][3]);
        }
    }
}

template <int NK>
static int duality_launch(const bf16* u, const bf16* dt, const bf16* bc, const float* dt_bias, const float* A, const float* D,
                          const DualityShape& g, int tiles, const int* seq_slot, const int* seq_first_row, const int* seq_start,
                          const int* seq_end, int n_seq, float* state, float* out, cudaStream_t stream) {
    constexpr size_t bytes = duality_smem(16 * NK);
    const cudaError_t e = cudaFuncSetAttribute(duality_scan_kernel<NK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return fail("duality_scan: shared memory of %zu bytes refused: %s", bytes, cudaGetErrorString(e));
    // (launched once its predecessor is over: its few CTAs run long and have to lie on SMs of their own; 148 SMs)
    const int parts = 2LL * n_seq * (g.C / (16 * tiles)) <= 148 ? 2 : 1;
    return launch_kernel_after("duality_scan", duality_scan_kernel<NK>, dim3(n_seq * parts, g.C / (16 * tiles)), dim3(64 * tiles), bytes, stream, parts,
                               u, dt, bc, dt_bias, A, D, g, parts, seq_slot, seq_first_row, seq_start, seq_end, state, out);
}

}  // namespace janis

using namespace janis;

// Whether janis_duality_scan takes a call: rows and columns in whole 16-byte pieces, a head's channels in whole tiles (of 16
// channels) and CTAs (of four tiles, or of the head), a number of states that the kernel is compiled for.
JANIS_EXPORT int janis_duality_scan_takes(const void* u, int u_stride, int u_off, const void* bc, int bc_stride, int b_off, int c_off,
                                          const void* state, const void* out, int C, int N, int cph, int cpg) {
    if (cph <= 0 || cpg <= 0 || C % cph || C % cpg || cpg % cph) return 0;
    if (!(cph % 64 == 0 || cph == 16 || cph == 32 || cph == 48)) return 0;
    if (!(N == 32 || N == 64 || N == 128)) return 0;
    if (u_stride % 8 || u_off % 8 || bc_stride % 8 || b_off % 8 || c_off % 8) return 0;
    if (((uintptr_t)u | (uintptr_t)bc) & 15) return 0;
    return (((uintptr_t)state | (uintptr_t)out) & 7) == 0;
}

JANIS_EXPORT int janis_duality_scan(const void* u, int u_stride, int u_off, const void* dt, int dt_stride, int dt_off,
                                    const float* dt_bias, const float* A, const void* bc, int bc_stride, int b_off, int c_off,
                                    const float* D, const int* seq_slot, const int* seq_first_row, const int* seq_start,
                                    const int* seq_end, int n_seq, float* state, float* out, int C, int N, int cph, int cpg,
                                    cudaStream_t stream) {
    if (n_seq <= 0) return 0;
    if (!janis_duality_scan_takes(u, u_stride, u_off, bc, bc_stride, b_off, c_off, state, out, C, N, cph, cpg))
        return fail("duality_scan: %d channels, %d states, %d a head, %d a group (or their rows' alignment) are not taken", C, N, cph, cpg);
    DualityShape g;
    g.u_stride = u_stride; g.u_off = u_off; g.dt_stride = dt_stride; g.dt_off = dt_off; g.bc_stride = bc_stride;
    g.b_off = b_off; g.c_off = c_off; g.C = C; g.cph = cph; g.cpg = cpg;
    const int tiles = cph % 64 == 0 ? 4 : cph / 16;
    if (C / (16 * tiles) > 65535) return fail("duality_scan: too many channels (%d)", C);
#define JANIS_DUALITY(NK)                                                                                                  \
    return duality_launch<NK>((const bf16*)u, (const bf16*)dt, (const bf16*)bc, dt_bias, A, D, g, tiles, seq_slot, seq_first_row, \
                              seq_start, seq_end, n_seq, state, out, stream);
    if (N == 32) { JANIS_DUALITY(2) }
    if (N == 64) { JANIS_DUALITY(4) }
    JANIS_DUALITY(8)
#undef JANIS_DUALITY
}
