// out[M, N] = x[M, K] * W[N, K]^T of float operands at float precision, on the tensor cores.
//
// A float of 2^-110 and more is the sum of three bfloat16 numbers to its last bit (hi, mid, lo: 8 bits each of 24), products of bfloat16
// numbers are exact in float, and the tensor cores add them up in float: x w = (xh + xm + xl)(wh + wm + wl), of which
// xm wl, xl wm and xl wl (2^-25 of the product and less) are left out.  Where a block of W holds nothing but bfloat16 numbers
// (a bfloat16 checkpoint run in 32 bits) wm and wl are zero and three products are left; the kernel looks at every block it
// splits, so nothing is remembered about a matrix.
//
// The tensor cores cut the sum's last bits off each time they add to it, which would show after thousands of additions
// of the same sign; so they only add up CHUNK blocks of 32 k at a time, and registers add the chunks, rounding to nearest.  (An
// output of one product is within 3.1 2^-24, where a float product has half a unit; large sums come out some 1.8e-7 of their size too small.)
// Every output is formed from its own row of x and row of W in one order, whatever M, N and the tiling are.  An output
// that does not come out finite (an infinity or NaN among the operands, or beyond the range) is formed again as a plain sum of
// float products, so infinities and NaN go where they go in such a sum; and a smaller float whose last bits lo has no place for is split into NaN, so
// that the outputs it counts in are such plain sums too (683 x 18432 over 2304: one such row of x or W 276 -> 530 us; one number in every row 23 ms).  Any M, N, K.  Optional epilogue: cap * tanh(v / cap).
//
// x is split once, by a kernel of its own, into three planes of bfloat16.  A CTA owns 128 rows of W (the lanes of tensor memory)
// and up to 192 rows of x (its columns).  Some warps read a block of 32 k of W into registers, ahead, split it, and write it
// into a ring of three stages as the tensor cores read it (rows of 64 bytes, 64-byte swizzle); one thread brings x's planes by
// TMA; two warps issue the products into two accumulators in tensor memory, while others add the chunk before to their
// registers.
//
// Against pairs of multiply-adds on the CUDA cores (the form before, 74 TFLOP/s at best), one B200, W of bfloat16 numbers (of any floats), L2 flushed:
// 683 x 18432 over 2304 1,309 -> 180 (261) us, 683 x 2304 over 9216 831 -> 150 (189), over 2048 187 -> 42 (54), 3 x 256000 over 2304
// 1,650 -> 502 (587), 1 x 2304 over 9216 356 -> 212 (259); errors against 64 bits over 2,304 k 6.1e-7 -> 2.1e-7 (3.4e-7) of the result, of
// operands of one sign 3.3e-7 -> 2.5e-7.  What bounds it: many rows of x, the products and what a block costs besides (waits, commits, the
// splitting of W where it is any floats); few rows, W's way from memory.  Chunks of 32 x 2 k are as long as the cut-off
// bits allow: 32 x 4 has an error of 3.9e-7 (7.5e-7).
#include "common.cuh"
#include "mma_bf16.cuh"
#include "tcgen05.cuh"

namespace janis {

int* tc05_timeout_counter();          // gemm_tc05.cu
namespace tc { bool make_planes_map(CUtensorMap* map, const void* ptr, int rows, int K, int planes, int box_k, int box_rows); }

namespace f32 {

using namespace tc;

constexpr int BK = 32, STAGES = 3;
constexpr int CHUNK = 2;              // blocks of 32 k between additions in registers
// A wait by parity tells a barrier's phase only from the one beside it, so whoever waits for a phase has to have seen the one before.  A
// stage's blocks go to both issuers and both groups of splitting warps in turn, and the copies of x of two stages may land in any order; so
// a block's barriers are not its stage's but one of CYCLE pairs, which come back after whole rounds of stages, issuers and groups:
//   full[b % CYCLE]   is waited for by the issuer of block b, who was the issuer of b - CYCLE and has seen that phase;
//   empty[b % CYCLE]  by the group that splits block b + STAGES, which split b + STAGES - CYCLE, and by the thread that brings x (all blocks in turn).
// None of them comes round again under a waiter: block b + CYCLE is brought to its stage after block b has been consumed, by that issuer, and
// consumed after that group and that thread have passed their waits for block b's stage (tests run the waits in a model with random delays).
constexpr int CYCLE = 12;
__host__ __device__ constexpr int stage_of(int b) { return b % STAGES; }
__host__ __device__ constexpr int pair_of(int b) { return b % CYCLE; }
__host__ __device__ constexpr int parity_of(int b) { return (b / CYCLE) & 1; }
__host__ __device__ constexpr int issuer_of(int b) { return (b / CHUNK) & 1; }
__host__ __device__ constexpr int group_of(int b, int groups) { return b % groups; }
static_assert(CYCLE % STAGES == 0 && CYCLE % (2 * CHUNK) == 0 && CYCLE % 2 == 0, "whole rounds of stages, issuers and groups of splitting warps");
constexpr int W_ROWS = 128, W_PLANE = W_ROWS * 64;     // a plane: one of hi, mid, lo
__host__ __device__ constexpr int stage_bytes(int cols) { return 3 * (W_PLANE + cols * 64); }
__host__ __device__ constexpr int smem_bytes(int cols) { return STAGES * stage_bytes(cols) + 1024; }

// Four floats from k on; zeros past the row's end and where !ok.  The loads are volatile so that they stay where they stand: the
// compiler may move others down to the block that uses them.  CONSTANT: of a matrix that nobody writes while the kernel lives (W), through the
// read-only path; x is the kernel before's result, which may still be at it when this one starts.
template <bool VEC, bool CONSTANT>
__device__ __forceinline__ float4 load4(const float* row, int k, int K, bool ok) {
    float4 v;
    if (VEC) {
#define JANIS_LOAD4(KIND)                                                                                                            \
    asm volatile("{\n.reg .pred p;\nsetp.ne.s32 p, %5, 0;\nmov.b32 %0, 0;\nmov.b32 %1, 0;\nmov.b32 %2, 0;\nmov.b32 %3, 0;\n"         \
                 "@p ld.global" KIND ".v4.f32 {%0, %1, %2, %3}, [%4];\n}\n"                                                          \
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)                                                                       \
                 : "l"(row + k), "r"((int)(ok && k < K)))
        if (CONSTANT) JANIS_LOAD4(".nc");
        else JANIS_LOAD4("");
#undef JANIS_LOAD4
    } else {
        float e[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
#define JANIS_LOAD1(KIND)                                                                                                            \
    asm volatile("{\n.reg .pred p;\nsetp.ne.s32 p, %2, 0;\nmov.b32 %0, 0;\n@p ld.global" KIND ".f32 %0, [%1];\n}\n"                 \
                 : "=f"(e[j])                                                                                                       \
                 : "l"(row + k + j), "r"((int)(ok && k + j < K)))
            if (CONSTANT) JANIS_LOAD1(".nc");
            else JANIS_LOAD1("");
#undef JANIS_LOAD1
        }
        v = make_float4(e[0], e[1], e[2], e[3]);
    }
    return v;
}

// Whether x is one of those that the three parts do not add up to: below 2^-110, the last of its 24 bits is below 2^-133, the smallest
// bfloat16 number (one of bfloat16's own bits alone is hi itself).  A NaN takes its hi's place.
constexpr float SPLIT_FROM = 0x1p-110f;
__device__ __forceinline__ bool lost(float x) { return fabsf(x) < SPLIT_FROM && (__float_as_uint(x) & 0xffffu); }
__device__ __forceinline__ uint32_t nan_where_lost(float x, float y, uint32_t hi) { return hi | (lost(x) ? 0x7fffu : 0u) | (lost(y) ? 0x7fff0000u : 0u); }

__device__ __forceinline__ void store8(uint32_t shared, uint32_t a, uint32_t b) {
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(shared), "r"(a), "r"(b) : "memory");
}

// Whether `mine` holds for any thread of four warps that split W together (group `turn`)
__device__ __forceinline__ bool any_of_group(int turn, bool mine) {
    uint32_t any;
    asm volatile("{\n.reg .pred p, q;\nsetp.ne.s32 p, %1, 0;\nbarrier.cta.red.or.pred q, %2, 128, p;\nselp.u32 %0, 1, 0, q;\n}\n"
                 : "=r"(any) : "r"((int)mine), "r"(1 + turn) : "memory");
    return any != 0;
}

// x [M, K] as three planes [3][M][Kp] of bfloat16 numbers that add up to it; Kp: K rounded up to 8, zeros behind K
template <bool VEC>
__global__ void __launch_bounds__(256)
split_rows_kernel(const float* x, bf16* __restrict__ planes, int M, int K, int Kp) {
    grid_dependents_launch();
    grid_dependency_wait();
    const int per_row = Kp / 8;
    const size_t n = (size_t)M * per_row, plane = (size_t)M * Kp;
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (size_t)gridDim.x * 256) {
        const size_t m = i / per_row;
        const int k = (int)(i - m * per_row) * 8;
        const float4 a = load4<VEC, false>(x + m * K, k, K, true), b = load4<VEC, false>(x + m * K, k + 4, K, true);
        uint4 hi, mid, lo;
        split3(a.x, a.y, hi.x, mid.x, lo.x);
        split3(a.z, a.w, hi.y, mid.y, lo.y);
        split3(b.x, b.y, hi.z, mid.z, lo.z);
        split3(b.z, b.w, hi.w, mid.w, lo.w);
        hi.x = nan_where_lost(a.x, a.y, hi.x);
        hi.y = nan_where_lost(a.z, a.w, hi.y);
        hi.z = nan_where_lost(b.x, b.y, hi.z);
        hi.w = nan_where_lost(b.z, b.w, hi.w);
        bf16* to = planes + m * Kp + k;
        *reinterpret_cast<uint4*>(to) = hi;
        *reinterpret_cast<uint4*>(to + plane) = mid;
        *reinterpret_cast<uint4*>(to + 2 * plane) = lo;
    }
}

// SUMS warps that add up, SPLITS warps that split W (groups of four take blocks in turn), and four warps of which two issue the
// products and one brings x.  VEC: rows of W are 16-byte aligned, K a multiple of 4.
template <int SUMS, int SPLITS, int MOST_COLS, bool VEC>
__global__ void __launch_bounds__((SUMS + SPLITS + 4) * 32, SUMS == 8 ? 1 : 2)
gemm_f32_kernel(const __grid_constant__ CUtensorMap map_x, const float* x, const float* W, float* __restrict__ out,
                int M, int N, int K, int cols, float cap, int* __restrict__ timeouts) {
    constexpr int GROUPS = SUMS / 4, UNITS = MOST_COLS / 16 / GROUPS;       // units of 16 columns of sums in a thread
    constexpr int TURNS = SPLITS / 4, NW = W_ROWS / 16, AHEAD = 2;          // 16 rows of W a pass of four warps, 8 threads a row
    extern __shared__ unsigned char smem_raw[];
    static_assert(CYCLE % TURNS == 0, "whole rounds of groups");
    __shared__ __align__(8) unsigned long long bars[2 * CYCLE + 5];
    __shared__ uint32_t tmem_slot;
    __shared__ int low_bits[STAGES];                      // 1 + the last block whose W was not all bfloat16 numbers
    __shared__ int failed;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t stage0 = ((uint32_t)__cvta_generic_to_shared(smem_raw) + 1023) & ~1023u;
    const uint32_t full = (uint32_t)__cvta_generic_to_shared(bars), empty = full + 8 * CYCLE;
    const uint32_t sums_there = empty + 8 * CYCLE, sums_taken = sums_there + 16, all_done = sums_taken + 16;
    const int stage_size = stage_bytes(cols), x_plane = cols * 64;
    const int m_tiles = (M + cols - 1) / cols;            // neighbouring CTAs take the rows of x of one strip of W
    const int m0 = (int)(blockIdx.x % m_tiles) * cols, n0 = (int)(blockIdx.x / m_tiles) * W_ROWS;
    const int n_blocks = (K + BK - 1) / BK, n_chunks = (n_blocks + CHUNK - 1) / CHUNK;
    const int tmem_cols = 2 * cols <= 32 ? 32 : (2 * cols <= 64 ? 64 : (2 * cols <= 128 ? 128 : (2 * cols <= 256 ? 256 : 512)));

    if (threadIdx.x == 0) {
        for (int i = 0; i < CYCLE; ++i) {
            mbar_init(full + 8 * i, 5);          // four warps of W, the copies of x
            mbar_init(empty + 8 * i, 1);
        }
        for (int i = 0; i < STAGES; ++i) low_bits[i] = 0;
        for (int i = 0; i < 2; ++i) {
            mbar_init(sums_there + 8 * i, 1);
            mbar_init(sums_taken + 8 * i, SUMS);
        }
        mbar_init(all_done, 2);
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == SUMS + SPLITS) tmem_alloc((uint32_t)__cvta_generic_to_shared(&tmem_slot), tmem_cols);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = tmem_slot;
    grid_dependents_launch();
    grid_dependency_wait();                               // the planes are the kernel before's result

    // Registers go to the warps that hold sums: of 640 x 96 at launch 256 x 128 + 256 x 96 + 128 x 32 are in use, of 384 x 80 (two
    // CTAs an SM) 128 x 96 + 128 x 104 + 128 x 32.
    if (warp >= SUMS + SPLITS) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
        const int issuer = warp - SUMS - SPLITS;
        if (issuer < 2) {
            // Two warps issue products, a chunk each in turn and into an accumulator each: what a block costs an issuer besides (waits,
            // commits: 1,100 cycles in all) lies beside the other's.  The whole warp runs the loop, so that descriptors stay in the uniform
            // registers that the products take them from, and the elected lane issues (a thread of the programmer's choice under a branch
            // took twice as long).
            const uint32_t idesc = instr_desc(W_ROWS, cols);
            const uint32_t plane16 = (uint32_t)x_plane >> 4;                    // (an address in a descriptor counts 16 bytes)
            const uint32_t d = tmem + issuer * cols;
            bool ok = true;
            for (int c = issuer; c < n_chunks && ok; c += 2) {              // (issuer_of)
                if (c >= 2 && !__all_sync(0xffffffffu, mbar_wait(sums_taken + 8 * issuer, (c / 2 - 1) & 1))) { ok = false; break; }
                const int first = c * CHUNK, last = min(first + CHUNK, n_blocks) - 1;
                for (int b = first; b <= last; ++b) {
                    const int s = stage_of(b);
                    if (!__all_sync(0xffffffffu, mbar_wait(full + 8 * pair_of(b), parity_of(b)))) { ok = false; break; }
                    // The splitters' writes are fenced for the tensor cores here, behind the barrier that orders them.
                    fence_async_shared();
                    fence_after_sync();
                    const uint64_t w = smem_desc_64(stage0 + s * stage_size), xs = w + (3 * W_PLANE >> 4);
                    const bool whole = *(volatile int*)&low_bits[s] == b + 1;
                    uint32_t add = b != first;            // the chunk's first product replaces what the accumulator held
                    if (elect_one()) {
                        if (whole) {                      // small ones first
                            umma(d, w + (2 * W_PLANE >> 4), xs, idesc, add);
                            umma(d, w + (2 * W_PLANE >> 4) + 2, xs + 2, idesc, 1);
                            umma(d, w + (W_PLANE >> 4), xs + plane16, idesc, 1);
                            umma(d, w + (W_PLANE >> 4) + 2, xs + plane16 + 2, idesc, 1);
                            umma(d, w + (W_PLANE >> 4), xs, idesc, 1);
                            umma(d, w + (W_PLANE >> 4) + 2, xs + 2, idesc, 1);
                            add = 1;
                        }
                        umma(d, w, xs + 2 * plane16, idesc, add);
                        umma(d, w + 2, xs + 2 * plane16 + 2, idesc, 1);
                        umma(d, w, xs + plane16, idesc, 1);
                        umma(d, w + 2, xs + plane16 + 2, idesc, 1);
                        umma(d, w, xs, idesc, 1);
                        umma(d, w + 2, xs + 2, idesc, 1);
                        umma_commit(empty + 8 * pair_of(b));
                        if (b == last) umma_commit(sums_there + 8 * issuer);
                    }
                    __syncwarp();
                }
            }
            if (!ok) atomicExch(&failed, 1);
            if (elect_one()) umma_commit(all_done);
            __syncwarp();
            mbar_wait(all_done, 0);
        } else if (issuer == 2 && lane == 0) {            // brings the planes of x
            int b = 0;
            for (; b < n_blocks; ++b) {
                const int before = b - STAGES;            // what the stage held
                if (before >= 0 && !mbar_wait_parked(empty + 8 * pair_of(before), parity_of(before), &failed)) { atomicExch(&failed, 1); break; }
                mbar_expect_tx(full + 8 * pair_of(b), 3 * x_plane);
                tma_load_3d(stage0 + stage_of(b) * stage_size + 3 * W_PLANE, &map_x, b * BK, m0, 0, full + 8 * pair_of(b));
            }
            // no copy is on its way when the CTA leaves, also where a wait was given up (then for some seconds at most)
            for (int j = max(0, b - STAGES); j < b; ++j)
                if (!mbar_wait_parked(full + 8 * pair_of(j), parity_of(j), &failed)) mbar_wait(full + 8 * pair_of(j), parity_of(j));
        }
        __syncwarp();
        asm volatile("bar.sync 0;" ::: "memory");         // the last sums have been read
        if (warp == SUMS + SPLITS) {
            tmem_free(tmem, tmem_cols);
            if (failed && lane == 0) atomicAdd(timeouts, 1);
        }
    } else if (warp >= SUMS) {
        if (SUMS == 4) asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
        const int thread = threadIdx.x - SUMS * 32, turn = thread >> 7;
        const int quad = thread & 7, r = (thread & 127) >> 3;                    // 4 k of rows r, r + 16, ...
        const uint32_t place = r * 64 + (((quad >> 1) ^ ((r >> 1) & 3)) << 4) + (quad & 1) * 8;
        const float* wr = W + (size_t)min(n0 + r, N - 1) * K;
        const int rows = N - n0 - r;                      // a pass of this thread's is within W where 16 i < rows
        float4 wv[AHEAD][NW];
        auto fetch = [&](int b, int a) {
            const int k = b * BK + quad * 4;
#pragma unroll
            for (int i = 0; i < NW; ++i) wv[a][i] = load4<VEC, true>(wr + (size_t)(i * 16) * K, k, K, i * 16 < rows);
        };
#pragma unroll
        for (int a = 0; a < AHEAD; ++a) fetch(turn + a * TURNS, a);
        bool ok = true;
        for (int b0 = turn; b0 < n_blocks; b0 += AHEAD * TURNS) {
#pragma unroll
            for (int a = 0; a < AHEAD; ++a) {
                const int b = b0 + a * TURNS;
                if (b >= n_blocks) break;
                const int s = stage_of(b), before = b - STAGES;
                // (who gives up goes on without waiting, as the other warps of the group count on it at their barrier, and arrives nowhere)
                if (ok && before >= 0) ok = mbar_wait_parked(empty + 8 * pair_of(before), parity_of(before), &failed);
                const uint32_t to = stage0 + s * stage_size + place;
                uint32_t low = 0;
#pragma unroll
                for (int i = 0; i < NW; ++i)
                    low |= __float_as_uint(wv[a][i].x) | __float_as_uint(wv[a][i].y) | __float_as_uint(wv[a][i].z) | __float_as_uint(wv[a][i].w);
                // Whether mid and lo have to be written is asked of all four warps: the stage may hold what another group left there.
                if (any_of_group(turn, (low & 0xffffu) != 0)) {
                    float least[NW];
#pragma unroll
                    for (int i = 0; i < NW; ++i) {
                        uint32_t h0, h1, m0_, m1, l0, l1;
                        split3(wv[a][i].x, wv[a][i].y, h0, m0_, l0);
                        split3(wv[a][i].z, wv[a][i].w, h1, m1, l1);
                        const uint32_t at = to + i * 16 * 64;
                        least[i] = fminf(fminf(fabsf(wv[a][i].x), fabsf(wv[a][i].y)), fminf(fabsf(wv[a][i].z), fabsf(wv[a][i].w)));
                        store8(at, h0, h1);
                        store8(at + W_PLANE, m0_, m1);
                        store8(at + 2 * W_PLANE, l0, l1);
                    }
                    if ((thread & 127) == 0) *(volatile int*)&low_bits[s] = b + 1;
#pragma unroll
                    for (int i = NW / 2; i > 0; i >>= 1)
#pragma unroll
                        for (int j = 0; j < i; ++j) least[j] = fminf(least[j], least[j + i]);
                    // (numbers as small are hardly ever there, and asking for each one in the loop above costs a quarter)
                    if (least[0] < SPLIT_FROM) {
#pragma unroll
                        for (int i = 0; i < NW; ++i)
                            if (lost(wv[a][i].x) || lost(wv[a][i].y) || lost(wv[a][i].z) || lost(wv[a][i].w)) store8(to + i * 16 * 64, 0x7fff7fffu, 0x7fff7fffu);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < NW; ++i)
                        store8(to + i * 16 * 64, __byte_perm(__float_as_uint(wv[a][i].x), __float_as_uint(wv[a][i].y), 0x7632),
                               __byte_perm(__float_as_uint(wv[a][i].z), __float_as_uint(wv[a][i].w), 0x7632));
                }
                if (b + AHEAD * TURNS < n_blocks) fetch(b + AHEAD * TURNS, a);
                __syncwarp();
                if (lane == 0 && ok) mbar_arrive(full + 8 * pair_of(b));
            }
        }
        if (!ok) atomicExch(&failed, 1);
        asm volatile("bar.sync 0;" ::: "memory");
    } else {
        if (SUMS == 8) asm volatile("setmaxnreg.inc.sync.aligned.u32 128;");
        else asm volatile("setmaxnreg.inc.sync.aligned.u32 96;");
        float acc[UNITS][16];
        const int quarter = warp & 3, group = warp >> 2;
        const uint32_t mine = tmem + ((uint32_t)(quarter * 32) << 16);
#pragma unroll
        for (int u = 0; u < UNITS; ++u)
#pragma unroll
            for (int j = 0; j < 16; ++j) acc[u][j] = 0.f;
        bool ok = true;
        for (int c = 0; c < n_chunks; ++c) {              // add the chunk in tensor memory to the registers
            if (!mbar_wait_parked(sums_there + 8 * (c & 1), (c / 2) & 1, &failed)) { ok = false; break; }
            fence_after_sync();
#pragma unroll
            for (int u = 0; u < UNITS; ++u) {
                const int col = (group + u * GROUPS) * 16;
                if (col >= cols) break;
                uint32_t v[16];
                tmem_load16(v, mine + (c & 1) * cols + col);
                tmem_wait_load();
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[u][j] += __uint_as_float(v[j]);
            }
            fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(sums_taken + 8 * (c & 1));
        }
        if (!ok) atomicExch(&failed, 1);
        fence_before_sync();
        asm volatile("bar.sync 0;" ::: "memory");
        if (failed) return;

        const int n = n0 + quarter * 32 + lane;           // neighbouring lanes hold neighbouring columns of out
        bool finite = true;
#pragma unroll
        for (int u = 0; u < UNITS; ++u) {
            const int col = (group + u * GROUPS) * 16;
            if (col >= cols) break;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const int m = m0 + col + j;
                if (m >= M || n >= N) break;
                float v = acc[u][j];
                finite &= fabsf(v) <= 3.402823466e38f;
                if (cap > 0.f) v = cap * tanhf(v / cap);
                out[(size_t)m * N + n] = v;
            }
        }
        if (__all_sync(0xffffffffu, finite)) return;
        // Hardly ever: a sum that is not finite is formed again by the warp, of plain products.  (A loop of its own: beside the stores
        // above it cost every output, 683 x 18432 over 2304: 300 us with x read through the read-only path, 379 by plain loads, 180 apart.)
#pragma unroll
        for (int u = 0; u < UNITS; ++u) {
            const int col = (group + u * GROUPS) * 16;
            if (col >= cols) break;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const int m = m0 + col + j;
                if (m >= M) break;
                uint32_t odd = __ballot_sync(0xffffffffu, n < N && !(fabsf(acc[u][j]) <= 3.402823466e38f));
                while (odd) {
                    const int l = __ffs(odd) - 1;
                    odd &= odd - 1;
                    const float *xp = x + (size_t)m * K, *wp = W + (size_t)(n - lane + l) * K;
                    float plain = 0.f;
                    for (int k = lane; k < K; k += 32) plain = fmaf(__ldcg(xp + k), wp[k], plain);
                    plain = warp_sum(plain);
                    if (cap > 0.f) plain = cap * tanhf(plain / cap);
                    if (lane == l) out[(size_t)m * N + n] = plain;
                }
            }
        }
    }
}

template <int SUMS, int SPLITS, int MOST_COLS, bool VEC>
static int launch(const CUtensorMap& map_x, const float* x, const float* W, float* out, int M, int N, int K, int cols, float cap,
                  long long tiles, int* timeouts, cudaStream_t stream) {
    auto kernel = gemm_f32_kernel<SUMS, SPLITS, MOST_COLS, VEC>;
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes(MOST_COLS));
        if (e != cudaSuccess) return fail("gemm_f32: shared memory of %d bytes refused: %s", smem_bytes(MOST_COLS), cudaGetErrorString(e));
        configured = true;
    }
    return launch_kernel("gemm_f32", kernel, dim3((unsigned)tiles), dim3((SUMS + SPLITS + 4) * 32), smem_bytes(cols), stream, 1, map_x, x, W,
                         out, M, N, K, cols, cap, timeouts);
}

}  // namespace f32
}  // namespace janis

using namespace janis;

JANIS_EXPORT int janis_launches_made() { return launches_made(); }

// How the kernel orders block b of 32 k, with `groups` groups of splitting warps (for tests): its stage, the pair of barriers and the
// parity of their phase, its issuer, its group; then the numbers of stages and of pairs, blocks a chunk.
JANIS_EXPORT void janis_gemm_f32_order(int b, int groups, int* out) {
    const int v[8] = {f32::stage_of(b), f32::pair_of(b), f32::parity_of(b), f32::issuer_of(b), f32::group_of(b, groups), f32::STAGES, f32::CYCLE, f32::CHUNK};
    for (int i = 0; i < 8; ++i) out[i] = v[i];
}

// rows of x whose planes take no more than 64 MB (256 at least): a product of more rows is made in parts
static int f32_part_rows(int M, int K) {
    const long long rows = (64ll << 20) / (6ll * ((K + 7) / 8 * 8)) / 256 * 256;
    const long long most = rows < 256 ? 256 : rows;
    return (int)(M < most ? M : most);
}

// bfloat16 numbers of room for the planes of x that janis_gemm_f32 wants
JANIS_EXPORT long long janis_gemm_f32_room(int M, int K) {
    return M <= 0 || K <= 0 ? 0 : 3ll * f32_part_rows(M, K) * ((K + 7) / 8 * 8);
}

// planes: 16-byte aligned room of janis_gemm_f32_room(M, K) bfloat16 numbers
JANIS_EXPORT int janis_gemm_f32(const float* x, const float* W, float* out, int M, int N, int K, float cap, void* planes,
                                cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return fail("gemm_f32: K must be positive, found %d", K);
    if ((M + 63) / 64 > 65535) return fail("gemm_f32: too many rows (%d)", M);
    if (planes == nullptr || ((uintptr_t)planes & 15)) return fail("gemm_f32: the planes of x need 16-byte aligned room");
    static thread_local int sms = 0;
    if (sms == 0) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
            return fail("gemm_f32: the device does not say how many SMs it has");
    }
    int* timeouts = tc05_timeout_counter();
    if (timeouts == nullptr) return fail("gemm_f32: the counter of timeouts has no address");
    const long long strips = (N + f32::W_ROWS - 1) / f32::W_ROWS;
    const bool w_vec = K % 4 == 0 && (uintptr_t)W % 16 == 0;
    const int part = f32_part_rows(M, K), Kp = (K + 7) / 8 * 8;
    for (int first = 0; first < M; first += part, x += (size_t)part * K, out += (size_t)part * N) {
        const int rows = M - first < part ? M - first : part;
        // Up to 64 rows of x: two CTAs an SM.  More: as many rows a CTA as make the last round of CTAs full; a block costs its
        // products (in proportion to the rows) and the splitting of W.
        const bool small = rows <= 64;
        int cols = (rows + 15) / 16 * 16;
        if (!small) {
            long long best = -1;
            for (int c = 64; c <= 192; c += 16) {
                const long long cost = (strips * ((rows + c - 1) / c) + sms - 1) / sms * (c + 48);
                if (best < 0 || cost <= best) { best = cost; cols = c; }
            }
        }
        const long long tiles = strips * ((rows + cols - 1) / cols);
        if (tiles > 0x7fffffff) return fail("gemm_f32: %d x %d outputs are too many", rows, N);
        CUtensorMap map_x;
        if (!tc::make_planes_map(&map_x, planes, rows, Kp, 3, f32::BK, cols))
            return fail("gemm_f32: cuTensorMapEncodeTiled is not available or refused the operands");
        const long long pieces = (long long)rows * (Kp / 8);
        const dim3 grid((unsigned)(pieces > 256ll * 8 * sms ? 8 * sms : (pieces + 255) / 256));
        const bool x_vec = K % 4 == 0 && (uintptr_t)x % 16 == 0;
        if (launch_kernel("gemm_f32", x_vec ? f32::split_rows_kernel<true> : f32::split_rows_kernel<false>, grid, dim3(256), 0, stream, 1, x,
                          (bf16*)planes, rows, K, Kp))
            return 1;
        const int failed = small ? (w_vec ? f32::launch<4, 4, 64, true>(map_x, x, W, out, rows, N, K, cols, cap, tiles, timeouts, stream)
                                          : f32::launch<4, 4, 64, false>(map_x, x, W, out, rows, N, K, cols, cap, tiles, timeouts, stream))
                                 : (w_vec ? f32::launch<8, 8, 192, true>(map_x, x, W, out, rows, N, K, cols, cap, tiles, timeouts, stream)
                                          : f32::launch<8, 8, 192, false>(map_x, x, W, out, rows, N, K, cols, cap, tiles, timeouts, stream));
        if (failed) return 1;
    }
    return 0;
}
