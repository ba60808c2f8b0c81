// The 32-bit matrix product of the true float path: C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]), all
// float, plain FFMA (no tensor cores, hence no reduced-precision matrix mode). Every output element
// is one sequential chain of fused multiply-adds over k = 0..K-1, so its value depends on neither M,
// nor the tile it falls in, nor what else is in the batch. The reference has no device float path;
// its float arithmetic is the f64 `linear` of helios/crates/helios-hal/src/reference.rs:24-41.
//
// A thread owns TM x TN outputs, BM / TM and BN / TN apart, and reads four k of each of its rows and columns at a time from shared memory in 16-byte pieces; slices of BK k
// are copied ahead into a ring of STAGES, as they lie in memory. Bound by issue slots (70 % of an active SM's cycles issue, 60 % of them FFMA) and the last wave where a product has tiles enough,
// else by the waits of a chain; the FFMA pipes would allow 74 TFLOP/s.
// Two shapes: 64 x 128 with 8 x 8 outputs a thread for products that fill the GPU with such tiles; 32 x 32 with 4 x 4 (4 x 2 where the tiles are few) for the others, which spreads a narrow
// product over all SMs.  (Two multiply-adds to an instruction, fma.rn.f32x2, take as long as two: 58 TFLOP/s from registers against 64.) Measured on one B200 (before: one shape of 64 x 64 with 4 x 4 outputs a thread, copied when needed): 394 rows, K 896, 9,728 columns 340 -> 229 to 246 us, K 4,864, 896 columns
// 302 -> 161 to 166 us; 3 rows, 151,936 columns 625 -> 244 us; 1 row, K 4,864 265 -> 101 us; 2,048 rows, 9,728 columns 1,393 -> 819 us (44 TFLOP/s).
#include "common.cuh"

namespace {
__device__ __forceinline__ void copy16(float* to, const float* from, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from), "r"(live ? 16 : 0));
}
__device__ __forceinline__ void copy4(float* to, const float* from, bool live) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from), "r"(live ? 4 : 0));
}

template <int BM, int BN, int TM, int TN, int BK, int STAGES, bool WIDE>
__global__ void __launch_bounds__((BM / TM) * (BN / TN)) sgemm_kernel(const float* __restrict__ a, const float* __restrict__ w, const float* __restrict__ bias,
                                                                       float* __restrict__ c, int m, int n, int k, int lda, int ldc) {
    constexpr int DOWN = BM / TM, ACROSS = BN / TN, THREADS = DOWN * ACROSS, QUADS = BK / 4, LD = BK + 4, STAGE = (BM + BN) * LD;
    extern __shared__ __align__(16) float ring[];  // STAGES times [BM + BN][LD]: rows of A, then rows of W
    const int tid = threadIdx.x, ty = tid / ACROSS, tx = tid % ACROSS;
    const int row0 = blockIdx.y * BM, col0 = blockIdx.x * BN;
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    // a slice's rows as they lie in memory; zeros past the matrix (they add exact zeros to a chain's end)
    auto fetch = [&](int slice) {
        float* stage = ring + slice % STAGES * STAGE;
        const int k0 = slice * BK;
#pragma unroll
        for (int unit = tid; unit < (BM + BN) * QUADS; unit += THREADS) {
            const int r = unit / QUADS, kk = k0 + unit % QUADS * 4;
            const bool from_a = r < BM;
            const int at = from_a ? row0 + r : col0 + r - BM;
            const bool live = at < (from_a ? m : n);
            const float* p = from_a ? a + (size_t)(live ? at : 0) * lda : w + (size_t)(live ? at : 0) * k;
            float* to = stage + r * LD + unit % QUADS * 4;
            if (WIDE) {
                copy16(to, p + (kk < k ? kk : 0), live && kk < k);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) copy4(to + e, p + (kk + e < k ? kk + e : 0), live && kk + e < k);
            }
        }
    };
    const int slices = (k + BK - 1) / BK;
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < slices) fetch(s);
        asm volatile("cp.async.commit_group;");
    }
    for (int slice = 0; slice < slices; ++slice) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2));
        __syncthreads();  // this slice is there, and the one before it has been read
        if (slice + STAGES - 1 < slices) fetch(slice + STAGES - 1);
        asm volatile("cp.async.commit_group;");
        const float* as = ring + slice % STAGES * STAGE + ty * LD;
        const float* ws = ring + slice % STAGES * STAGE + (BM + tx) * LD;
#pragma unroll
        for (int kk = 0; kk < BK; kk += 4) {
            float av[TM][4], wv[TN][4];
#pragma unroll
            for (int i = 0; i < TM; ++i) load4(as + i * DOWN * LD + kk, av[i]);
#pragma unroll
            for (int j = 0; j < TN; ++j) load4(ws + j * ACROSS * LD + kk, wv[j]);
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(av[i][e], wv[j][e], acc[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int r = row0 + ty + i * DOWN;
        if (r >= m) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int col = col0 + tx + j * ACROSS;
            if (col < n) c[(size_t)r * ldc + col] = acc[i][j] + (bias ? bias[col] : 0.f);
        }
    }
}

template <int BM, int BN, int TM, int TN, int BK, int STAGES, bool WIDE>
int launch_kernel(dim3 grid, const float* a, const float* w, const float* bias, float* c, int m, int n, int k, int lda, int ldc, cudaStream_t stream) {
    constexpr int bytes = STAGES * (BM + BN) * (BK + 4) * 4;
    if (bytes > 48 * 1024) {
        const int status = (int)cudaFuncSetAttribute(sgemm_kernel<BM, BN, TM, TN, BK, STAGES, WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (status) return status;
    }
    sgemm_kernel<BM, BN, TM, TN, BK, STAGES, WIDE><<<grid, (BM / TM) * (BN / TN), bytes, stream>>>(a, w, bias, c, m, n, k, lda, ldc);
    return launch_status();
}

bool aligned(const float* a, const float* w, int k, int lda) { return ((lda | k) & 3) == 0 && (((uintptr_t)a | (uintptr_t)w) & 15) == 0; }

template <int BM, int BN, int TM, int TN, int BK, int STAGES>
int launch_tiles(const float* a, const float* w, const float* bias, float* c, int m, int n, int k, int lda, int ldc, cudaStream_t stream) {
    const dim3 grid((n + BN - 1) / BN, (m + BM - 1) / BM);
    if (grid.y > 65535) return HB_UNSUPPORTED_SIZE;
    return aligned(a, w, k, lda) ? launch_kernel<BM, BN, TM, TN, BK, STAGES, true>(grid, a, w, bias, c, m, n, k, lda, ldc, stream)
                : launch_kernel<BM, BN, TM, TN, BK, STAGES, false>(grid, a, w, bias, c, m, n, k, lda, ldc, stream);
}
}  // namespace

// A rows are `lda` floats apart, C rows `ldc`; W is dense [n, k]. Zero padding of the k tail adds
// exact zeros to the chain and does not change the result.  sms: the device's multiprocessors.
HB_EXPORT int hb_sgemm_f32(const float* a, const float* w, const float* bias, float* c, int m, int n, int k, int lda,
                           int ldc, int sms, cudaStream_t stream) {
    if (m <= 0 || n <= 0) return 0;
    if (k <= 0) return HB_BAD_ARGUMENT;
    // large tiles from two to an SM on (148 SMs, 394 rows, 9,728 columns: 532 of them 246 us; 896 columns: 49 of them would leave two SMs in three idle) and where rows do not leave half
    // of one empty.  Rows that are not on 16-byte boundaries are copied four bytes at a time, twice as many copies an output in small tiles: large ones from three to four SMs on (1,003 columns, K
    // 1,001: 88 large tiles 90 us, small ones 82; 128: 92 and 124; 288: 155 and 236)
    const long long large = (long long)((m + 63) / 64) * ((n + 127) / 128);
    if (m > 32 && large >= (aligned(a, w, k, lda) ? 2LL * sms : 3LL * sms / 4)) return launch_tiles<64, 128, 8, 8, 16, 4>(a, w, bias, c, m, n, k, lda, ldc, stream);
    // Up to three small tiles to an SM a product is the chains of a few warps: twice as many warps, half as many outputs each, and slices of 64 k between barriers (394 rows, K 4,864, 896
    // columns: 163 -> 138 us; K 896: 35 -> 30; 1 row, K 4,864: 100 -> 63).  With more tiles the loads per output count (3 rows, 151,936 columns: 244 and 278).
    const long long small = (long long)((m + 31) / 32) * ((n + 31) / 32);
    if (small <= 3LL * sms) return launch_tiles<32, 32, 4, 2, 64, 3>(a, w, bias, c, m, n, k, lda, ldc, stream);
    return launch_tiles<32, 32, 4, 4, 32, 4>(a, w, bias, c, m, n, k, lda, ldc, stream);
}
