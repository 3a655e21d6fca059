// out[M, N] = x[M, K] * W[N, K]^T in true 32-bit: float operands, fused
// multiply-adds on the CUDA cores, no tensor-core mode of any kind.  Each output
// element is accumulated by one thread, the even and the odd k each in ascending
// order and the two sums added at the end, so its value
// depends on its own row of x and row of W only: not on M, not on the tiling of
// other rows.  Any M, N, K.  Optional epilogue: cap * tanh(v / cap).
//
// The multiply-adds bound it (74 TFLOP/s of them), so everything else has to stay out of their issue slots.
// `fma.rn.f32x2` multiplies the pairs (k, k + 1) of a row of x and a row of W as they lie in memory, so nothing is
// transposed or duplicated: tiles of 16 k come by `cp.async` into a ring of shared memory and 16-byte reads take
// four k of a row.  A CTA owns 64 x 64 outputs, a thread 8 rows of them and TN = 8 or 4 columns.
// 683 x 18432 outputs over 2304 k: 1.32 ms, 44 TFLOP/s (1.92 ms with 4 x 4 outputs a thread, scalar multiply-adds and
// tiles stored transposed); 683 x 2304 over 9216: 0.84 ms against 1.09.  The error against 64 bits is 6.1e-7 of the
// result against 8.6e-7, as two sums of half the length round less.
#include "common.cuh"

namespace janis {

constexpr int BM = 64, BN = 64, BK = 16, LD = BK + 4, STAGES = 4;      // rows of 80 bytes: eight of them lie in different banks

typedef unsigned long long f32x2;

__device__ __forceinline__ void fma_pair(f32x2& c, f32x2 a, f32x2 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}

__device__ __forceinline__ void load_pairs(f32x2 (&v)[2], uint32_t shared) {
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(v[0]), "=l"(v[1]) : "r"(shared));
}

// Bytes [0, n) of BYTES from global memory, zeros behind them
template <int BYTES>
__device__ __forceinline__ void copy_async(uint32_t shared, const void* src, int n) {
    if (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(shared), "l"(src), "r"(n) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(shared), "l"(src), "r"(n) : "memory");
}

// TN = 8: 2 warps of 64 x 32 outputs; TN = 4: 4 warps of 64 x 16.  VEC: rows are 16-byte aligned, K a multiple of 4.
template <int TN, bool VEC>
__global__ void __launch_bounds__(512 / TN)
gemm_f32_kernel(const float* __restrict__ x, const float* __restrict__ W, float* __restrict__ out, int M, int N,
                int K, float cap) {
    constexpr int NT = 512 / TN, STAGE_BYTES = (BM + BN) * LD * 4;
    __shared__ __align__(16) float tile[STAGES][BM + BN][LD];          // rows of x, then rows of W
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // neighbouring CTAs take the rows of x above one strip of W, so that the strip is fetched from memory once
    const int m_tiles = (M + BM - 1) / BM;
    const int m0 = (int)(blockIdx.x % m_tiles) * BM, n0 = (int)(blockIdx.x / m_tiles) * BN;
    const int tm = lane & 7, tn = warp * 4 * TN + (lane >> 3);         // rows tm + 8 i, columns tn + 4 j
    const int n_tiles = (K + BK - 1) / BK;
    grid_dependents_launch();
    grid_dependency_wait();                                            // x is the kernel before's result

    // The pieces this thread brings: column kp of rows first, first + STEP, ...  Nobody stores the products of rows past the end;
    // in the place of such a row of x stands the tile's row of W, which comes anyway.  (The last row of x over and over is a few
    // lines of L2 for which all CTAs wait: one row against 18,432 x 2,304 took 375 us.  Reading nothing and writing zeros costs
    // instructions in every tile: 1,370 us for 1,332 at 683 rows.)
    constexpr int PER = BK / (VEC ? 4 : 1), STEP = NT / PER, PIECES = (BM + BN) / STEP;
    const int first = tid / PER, kp = tid % PER * (VEC ? 4 : 1);
    const float* src[PIECES];
#pragma unroll
    for (int e = 0; e < PIECES; ++e) {
        const int r = first + e * STEP;
        const bool of_x = e < PIECES / 2 && (!VEC || m0 + r < M);          // (without VEC the 32 addresses have no registers to spare)
        const int row = of_x ? min(m0 + r, M - 1) : min(n0 + r % BM, N - 1);
        src[e] = (of_x ? x : W) + (size_t)row * K + kp;
    }
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(&tile[0][0][0]);
    auto fetch = [&](int t) {                                          // (a group for every tile, an empty one past the last)
        if (t < n_tiles) {
            const uint32_t to = base + (t % STAGES) * STAGE_BYTES + (first * LD + kp) * 4;
            const int n = t * BK + kp < K ? (VEC ? 16 : 4) : 0;
#pragma unroll
            for (int e = 0; e < PIECES; ++e) copy_async<VEC ? 16 : 4>(to + e * STEP * LD * 4, n ? src[e] + t * BK : src[e] - kp, n);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    f32x2 acc[8][TN];                                                  // (sum over even k, sum over odd k)
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;

    for (int t = 0; t < STAGES - 1; ++t) fetch(t);
    for (int t = 0; t < n_tiles; ++t) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();                                               // tile t is there; tile t - 1 has been read by all
        fetch(t + STAGES - 1);
        const uint32_t xa = base + (t % STAGES) * STAGE_BYTES + tm * (LD * 4);
        const uint32_t wa = base + (t % STAGES) * STAGE_BYTES + (BM + tn) * (LD * 4);
#pragma unroll
        for (int kk = 0; kk < BK; kk += 4) {
            f32x2 a[8][2];
#pragma unroll
            for (int i = 0; i < 8; ++i) load_pairs(a[i], xa + (8 * i * LD + kk) * 4);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                f32x2 w[2];
                load_pairs(w, wa + (4 * j * LD + kk) * 4);
#pragma unroll
                for (int i = 0; i < 8; ++i) fma_pair(acc[i][j], a[i][0], w[0]);
#pragma unroll
                for (int i = 0; i < 8; ++i) fma_pair(acc[i][j], a[i][1], w[1]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = m0 + tm + 8 * i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tn + 4 * j;
            if (n >= N) continue;
            float even, odd;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(even), "=f"(odd) : "l"(acc[i][j]));
            float v = even + odd;
            if (cap > 0.f) v = cap * tanhf(v / cap);
            out[(size_t)m * N + n] = v;
        }
    }
}

}  // namespace janis

using namespace janis;

JANIS_EXPORT int janis_gemm_f32(const float* x, const float* W, float* out, int M, int N, int K, float cap,
                                cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return fail("gemm_f32: K must be positive, found %d", K);
    if ((M + BM - 1) / BM > 65535) return fail("gemm_f32: too many rows (%d)", M);
    const long long tiles = (long long)((M + BM - 1) / BM) * ((N + BN - 1) / BN);
    if (tiles > 0x7fffffff) return fail("gemm_f32: %d x %d outputs are too many", M, N);
    const dim3 grid((unsigned)tiles);
    static thread_local int sms = 0;
    if (sms == 0) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
            return fail("gemm_f32: the device does not say how many SMs it has");
    }
    // The time is what the busiest quarter of an SM has to do.  Warps of 64 x 32 outputs read less from shared memory an
    // instruction (44 TFLOP/s against 37 when the SMs are full); warps of half the size leave less undone in the last round.
    const long long quarters = 4ll * sms;
    const long long large = (2 * tiles + quarters - 1) / quarters * 20, small = (4 * tiles + quarters - 1) / quarters * 12;
    const bool vec = K % 4 == 0 && ((uintptr_t)x | (uintptr_t)W) % 16 == 0;
    if (large <= small)
        return vec ? launch_kernel("gemm_f32", gemm_f32_kernel<8, true>, grid, dim3(64), 0, stream, 1, x, W, out, M, N, K, cap)
                   : launch_kernel("gemm_f32", gemm_f32_kernel<8, false>, grid, dim3(64), 0, stream, 1, x, W, out, M, N, K, cap);
    return vec ? launch_kernel("gemm_f32", gemm_f32_kernel<4, true>, grid, dim3(128), 0, stream, 1, x, W, out, M, N, K, cap)
               : launch_kernel("gemm_f32", gemm_f32_kernel<4, false>, grid, dim3(128), 0, stream, 1, x, W, out, M, N, K, cap);
}
