// The grouped bfloat16 matrix product of a feed-forward made of experts, on the 5th-generation tensor cores, and its
// counterpart for a handful of rows.
//
// Rows arrive sorted by expert in runs padded to whole tiles of 128 rows (csrc/moe.cu); tile i of the rows multiplies the
// matrix of expert tile_expert[i], and tiles whose entry is -1 (beyond the last run) are skipped:
//     C[128 i .. 128 i + 127, :] = A[128 i .. 128 i + 127, :] W[tile_expert[i]]^T,    W stacked [experts * n, k].
//
// * The tile kernel (prompt-sized steps) is the tile shape of csrc/gemm_tcgen05.cu with the weight tile's row taken from the
//   tile list: one persistent block per SM walks 128 x BN tiles, warp 0 (one lane) fetches operand tiles with TMA into a ring,
//   one lane of warp 1 issues tcgen05.mma (kind::f16, M 128, N BN, K 16) into two accumulators in tensor memory that alternate,
//   warps 2-5 drain a finished accumulator while the next tile's products run.  All three roles read the tile list (written by
//   the plan kernel just before) and skip the same tiles, so their counters stay in step.  Every wait is bounded; when one runs
//   out the status word says so, all roles leave their loops, tensor memory is freed and the block returns.
// * The pair kernel (steps that bring an expert more than a tile of rows on average) is the shape of csrc/gemm_pair_tcgen05.cu: two SMs on two neighbouring
//   row tiles of one expert, each keeping its own rows and half of the weight tile, so that a weight tile is fetched once for 256 rows and a block moves 32 KB
//   per 64-deep step where the tile kernel moves 48.  Every block lists the pairs of tiles from the plan's tile list; a run's odd last tile has a pair of its own, whose
//   second half is not stored.
// * The rows kernel (steps of a few tokens) streams each used expert's matrix once: a block takes the real rows of one
//   tile (tile_rows[i] of them, eight at a time) into shared memory and its warps walk output columns two at a time, every lane reading
//   16 bytes of both matrix rows per step.  Such a step is bound by the bytes of the matrices it touches, not by arithmetic.
#include "gemm_pair_tcgen05.cuh"

namespace {
template <int BN>
struct GroupedLayout {
    static constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr int ROOM = 227 * 1024 - 1024 - 256;
    static constexpr int STAGES = ROOM / STAGE_BYTES > 6 ? 6 : ROOM / STAGE_BYTES;
    static constexpr int ACC_STRIDE = 256;  // columns between the two accumulators
    static constexpr int TMEM_COLS = 512;
    static constexpr size_t SMEM = 1024 + (size_t)STAGES * STAGE_BYTES + 256;
};

struct GroupedParams {
    bf16* c;                 // [rows, n]
    const int* tile_expert;  // [tiles_m]
    int rows, n, k, ldc;     // n: columns per expert
    int act;                 // what is applied to an accumulator before its one rounding (activated() in common.cuh)
    int* status;
};

template <int BN>
__device__ __forceinline__ void store_grouped_row(const GroupedParams& p, unsigned lane_addr, int r, int col0) {
#pragma unroll 1
    for (int c = 0; c < BN; c += 16) {
        float v[16];
        tmem_ld16(lane_addr + c, v);
        if (p.act != HB_ACT_NONE) {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = activated(v[j], p.act);
        }
        const int col = col0 + c;
        if (r < p.rows && col < p.n) {
            bf16* dst = p.c + (size_t)r * p.ldc + col;
            if (col + 16 <= p.n && (p.ldc & 7) == 0) {
                uint4 w[2];
                __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(w);
#pragma unroll
                for (int j = 0; j < 8; ++j) h[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
                reinterpret_cast<uint4*>(dst)[0] = w[0];
                reinterpret_cast<uint4*>(dst)[1] = w[1];
            } else {
                for (int j = 0; j < 16 && col + j < p.n; ++j) dst[j] = __float2bfloat16_rn(v[j]);
            }
        }
    }
}

template <int BN>
__global__ void __launch_bounds__(THREADS) gemm_grouped_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                                                               const GroupedParams p, int tiles_m, int tiles_n) {
    using L = GroupedLayout<BN>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned long long* full = reinterpret_cast<unsigned long long*>(tiles + (size_t)L::STAGES * L::STAGE_BYTES);
    unsigned long long* empty = full + L::STAGES;
    unsigned long long* acc_full = empty + L::STAGES;  // [2]
    unsigned long long* acc_empty = acc_full + 2;      // [2]
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(acc_empty + 2);
    volatile int* failed = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    let_next_kernel_start();
    const int total = tiles_m * tiles_n;
    const int k_blocks = (p.k + BK - 1) / BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < L::STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 4); }
        *failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(L::TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = *tmem_slot;
    // the tile list and the rows come from the kernels before: nothing is read ahead of them
    wait_for_previous_kernels();

    if (warp == 0) {
        if (lane == 0) {  // producer
            int s = 0;
            unsigned turn = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
                const int tile_m = t % tiles_m, tile_n = t / tiles_m;
                const int expert = p.tile_expert[tile_m];
                if (expert < 0) continue;
                const int row0 = tile_m * BM, w_row0 = expert * p.n + tile_n * BN;
                for (int kb = 0; kb < k_blocks; ++kb) {
                    if (!mbar_ready(smem_u32(&empty[s]), turn ^ 1u) && !mbar_wait(&empty[s], turn ^ 1u, failed)) { *failed = 1; ok = false; break; }
                    unsigned char* a_tile = tiles + (size_t)s * L::STAGE_BYTES;
                    mbar_expect_tx(&full[s], L::STAGE_BYTES);
                    tma_load_2d(a_tile, &map_x, &full[s], kb * BK, row0);
                    tma_load_2d(a_tile + L::A_BYTES, &map_w, &full[s], kb * BK, w_row0);
                    if (++s == L::STAGES) { s = 0; turn ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {  // tensor-core issuer
            const unsigned idesc = umma_idesc(BN);
            const unsigned a_low0 = desc_low(tiles), b_low0 = desc_low(tiles + L::A_BYTES), step = (unsigned)L::STAGE_BYTES >> 4;
            const unsigned full0 = smem_u32(&full[0]), empty0 = smem_u32(&empty[0]);
            int s = 0, i = 0;
            unsigned turn = 0, a_low = a_low0, b_low = b_low0;
            bool ok = true;
            for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
                if (p.tile_expert[t % tiles_m] < 0) continue;
                const int buf = i & 1;
                if (!mbar_wait(&acc_empty[buf], ((i >> 1) & 1) ^ 1, failed)) { *failed = 1; ok = false; break; }  // the epilogue has drained it
                tc_fence_after();
                const unsigned acc = tmem + buf * L::ACC_STRIDE;
                for (int kb = 0; kb < k_blocks; ++kb) {
                    if (!mbar_ready(full0 + 8u * (unsigned)s, turn) && !mbar_wait(&full[s], turn, failed)) { *failed = 1; ok = false; break; }
                    umma_stage(acc, a_low, b_low, idesc, kb > 0 ? 1u : 0u);
                    umma_commit_at(empty0 + 8u * (unsigned)s);  // the stage is free once these products have read it
                    a_low += step;
                    b_low += step;
                    if (++s == L::STAGES) { s = 0; turn ^= 1u; a_low = a_low0; b_low = b_low0; }
                }
                if (ok) umma_commit(&acc_full[buf]);
                ++i;
            }
        }
    } else {  // epilogue: warps 2..5 read TMEM lane quarters 2, 3, 0, 1
        const int quarter = warp & 3;
        bool ok = true;
        int i = 0;
        for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
            const int tile_m = t % tiles_m, tile_n = t / tiles_m;
            if (p.tile_expert[tile_m] < 0) continue;
            const int buf = i & 1;
            if (!mbar_wait(&acc_full[buf], (i >> 1) & 1, failed)) { *failed = 1; ok = false; break; }
            tc_fence_after();
            store_grouped_row<BN>(p, tmem + buf * L::ACC_STRIDE + ((unsigned)(quarter * 32) << 16), tile_m * BM + quarter * 32 + lane, tile_n * BN);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {  // this warp's quarter of the accumulator may be written again
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[buf])) : "memory");
            }
            ++i;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *failed) atomicOr(p.status, HB_STATUS_WAIT_EXPIRED | HB_STATUS_IN_GEMM_TILES);
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(L::TMEM_COLS) : "memory");
    }
}

template <int BN>
int launch_grouped(const CUtensorMap& map_x, const CUtensorMap& map_w, const GroupedParams& p, int tiles_m, int tiles_n, int blocks, cudaStream_t stream) {
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(gemm_grouped_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GroupedLayout<BN>::SMEM);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    return launch_after_previous(gemm_grouped_kernel<BN>, dim3(blocks), THREADS, GroupedLayout<BN>::SMEM, stream, map_x, map_w, p, tiles_m, tiles_n);
}

// ---------------------------------------------------------------- two row tiles of an expert on two SMs
constexpr int GP_STAGES = 6, GP_MOST_TILES = 4096;
constexpr unsigned GP_STAGE_BYTES = 32 * 1024;
__host__ __device__ constexpr size_t grouped_pair_smem(int tiles_m) { return 1024 + (size_t)GP_STAGES * GP_STAGE_BYTES + 256 + ((size_t)tiles_m * 2 + 15) / 16 * 16; }

// The first tiles of the pairs, in ascending order: bit 15 says that the next tile belongs to the pair too.  One warp; returns how many.
__device__ __forceinline__ int list_pairs(const int* __restrict__ tile_expert, int tiles_m, unsigned short* list) {
    const int lane = threadIdx.x & 31;
    int count = 0, run_start = 0, before = -1;
    for (int base = 0; base < tiles_m; base += 32) {
        const int i = base + lane, e = i < tiles_m ? tile_expert[i] : -1, next = i + 1 < tiles_m ? tile_expert[i + 1] : -1;
        int previous = __shfl_up_sync(0xffffffffu, e, 1);
        if (lane == 0) previous = before;
        const unsigned starts = __ballot_sync(0xffffffffu, e >= 0 && e != previous), upto = starts & (0xffffffffu >> (31 - lane));
        const int start = upto ? base + 31 - __clz(upto) : run_start;
        const bool begins = e >= 0 && ((i - start) & 1) == 0;
        const unsigned all = __ballot_sync(0xffffffffu, begins);
        if (begins) list[count + __popc(all & ((1u << lane) - 1))] = (unsigned short)(i | (next == e ? 0x8000 : 0));
        count += __popc(all);
        if (starts) run_start = base + 31 - __clz(starts);
        before = __shfl_sync(0xffffffffu, e, 31);
    }
    return count;
}

// 32 columns of one row from column c of the tile on; SwiGLU: columns c of the tile's first half (gate) and of its second (up).
__device__ __forceinline__ void store_grouped_pair_row(const GroupedParams& p, unsigned lane_addr, int r, int tile_n, int begin, int end) {
    const bool glu = p.act == HB_ACT_SWIGLU;
    const int width = glu ? p.n / 2 : p.n, out0 = tile_n * (glu ? 128 : 256);
#pragma unroll 1
    for (int c = begin; c < end; c += 32) {
        const int col = out0 + c;
        if (col >= width) break;
        float v[32];
        tmem_ld32(lane_addr + c, v);
        if (glu) {
            float u[32];
            tmem_ld32(lane_addr + 128 + c, u);
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = v[j] / (1.0f + expf(-v[j])) * u[j];
        } else if (p.act != HB_ACT_NONE) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = activated(v[j], p.act);
        }
        bf16* dst = p.c + (size_t)r * p.ldc + col;
        if (col + 32 <= width && (p.ldc & 7) == 0) {
            uint4 w[4];
            __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(w);
#pragma unroll
            for (int j = 0; j < 16; ++j) h[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
#pragma unroll
            for (int j = 0; j < 4; ++j) reinterpret_cast<uint4*>(dst)[j] = w[j];
        } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
                if (col + j < width) dst[j] = __float2bfloat16_rn(v[j]);
        }
    }
}

// Bound by the matrices where an expert has about a pair of tiles (16 of [2,048, 2,048], 3,640 rows: 58.7 us on single SMs, 39.1 on pairs; their bytes
// alone take 21), by the products beyond.  The activation is the epilogue's, under the next tile's products.
__global__ void __launch_bounds__(PAIR_THREADS) gemm_grouped_pair_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                                                                         const GroupedParams p, int tiles_m, int tiles_n) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned long long* full = reinterpret_cast<unsigned long long*>(tiles + (size_t)GP_STAGES * GP_STAGE_BYTES);  // used in the leader only
    unsigned long long* empty = full + GP_STAGES;
    unsigned long long* acc_full = empty + GP_STAGES;  // [2]
    unsigned long long* acc_empty = acc_full + 2;      // [2], used in the leader only: 16 warps arrive, 8 of each block
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(acc_empty + 2);
    volatile int* failed = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* listed = reinterpret_cast<int*>(tmem_slot + 2);
    unsigned short* list = reinterpret_cast<unsigned short*>(tiles + (size_t)GP_STAGES * GP_STAGE_BYTES + 256);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned rank = cluster_rank();
    const bool leader = rank == 0;
    const int me = blockIdx.x >> 1, all = gridDim.x >> 1;
    const int k_blocks = (p.k + BK - 1) / BK;
    let_next_kernel_start();

    if (threadIdx.x == 0) {
        for (int s = 0; s < GP_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 16); }
        *failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    wait_for_previous_kernels();  // the tile list and the rows come from the kernels before
    if (warp == 0) {
        const int count = list_pairs(p.tile_expert, tiles_m, list);
        if (lane == 0) *listed = count;
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // both blocks' barriers exist before either signals the other's
    tc_fence_after();
    const unsigned tmem = *tmem_slot;
    const int n_pairs = *listed, total = n_pairs * tiles_n;

    if (warp == 0) {
        if (lane == 0) {  // producer
            const unsigned full0 = in_leader(&full[0]);
            int s = 0;
            unsigned turn = 0;
            bool ok = true;
            for (int t = me; t < total && ok; t += all) {
                const int first = list[t % n_pairs] & 0x7fff, row0 = (first + (int)rank) * BM;
                const int w_row0 = p.tile_expert[first] * p.n + (t / n_pairs) * 256 + (int)rank * 128;
                for (int kb = 0; kb < k_blocks; ++kb) {
                    if (!mbar_ready(smem_u32(&empty[s]), turn ^ 1u) && !mbar_wait(&empty[s], turn ^ 1u, failed)) { *failed = 1; ok = false; break; }
                    unsigned char* a_tile = tiles + (size_t)s * GP_STAGE_BYTES;
                    const unsigned bar = full0 + 8u * (unsigned)s;
                    if (leader) mbar_expect_tx(&full[s], 2u * GP_STAGE_BYTES);
                    tma_load_2d_pair(a_tile, &map_x, bar, kb * BK, row0);
                    tma_load_2d_pair(a_tile + A_BYTES, &map_w, bar, kb * BK, w_row0);
                    if (++s == GP_STAGES) { s = 0; turn ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && leader) {  // tensor-core issuer of the pair
            const unsigned idesc = pair_idesc(256);
            const unsigned a_low0 = desc_low(tiles), b_low0 = desc_low(tiles + A_BYTES), step = GP_STAGE_BYTES >> 4;
            const unsigned full0 = smem_u32(&full[0]), empty0 = smem_u32(&empty[0]);
            int s = 0;
            unsigned turn = 0, a_low = a_low0, b_low = b_low0;
            bool ok = true;
            for (int t = me, i = 0; t < total && ok; t += all, ++i) {
                const int buf = i & 1;
                if (!mbar_wait(&acc_empty[buf], ((i >> 1) & 1) ^ 1, failed)) { *failed = 1; ok = false; break; }  // both epilogues have drained it
                tc_fence_after();
                const unsigned acc = tmem + buf * ACC_STRIDE;
                for (int kb = 0; kb < k_blocks; ++kb) {
                    if (!mbar_ready(full0 + 8u * (unsigned)s, turn) && !mbar_wait(&full[s], turn, failed)) { *failed = 1; ok = false; break; }
                    umma_pair_stage(acc, a_low, b_low, idesc, kb > 0 ? 1u : 0u);
                    umma_commit_both_at(empty0 + 8u * (unsigned)s);  // the stage is free in both blocks once these products have read it
                    a_low += step;
                    b_low += step;
                    if (++s == GP_STAGES) { s = 0; turn ^= 1u; a_low = a_low0; b_low = b_low0; }
                }
                if (ok) umma_commit_both(&acc_full[buf]);
            }
        }
    } else {  // epilogue: warps 2..9; warp w reads lane quarter w % 4 and the half (w - 2) / 4 of this block's columns
        const int quarter = warp & 3, half = (warp - 2) >> 2, cols = p.act == HB_ACT_SWIGLU ? 128 : 256;
        bool ok = true;
        for (int t = me, i = 0; t < total && ok; t += all, ++i) {
            const int buf = i & 1;
            if (!mbar_wait(&acc_full[buf], (i >> 1) & 1, failed)) { *failed = 1; ok = false; break; }
            tc_fence_after();
            const int entry = list[t % n_pairs];
            if (leader || (entry & 0x8000))  // a lone tile has no second half
                store_grouped_pair_row(p, tmem + buf * ACC_STRIDE + ((unsigned)(quarter * 32) << 16), ((entry & 0x7fff) + (int)rank) * BM + quarter * 32 + lane, t / n_pairs,
                                       half * cols / 2, (half + 1) * cols / 2);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) arrive_in_leader(in_leader(&acc_empty[buf]));  // this warp's share of the accumulator may be written again
        }
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *failed) atomicOr(p.status, HB_STATUS_WAIT_EXPIRED | HB_STATUS_IN_GEMM_TILES);
    cluster_sync();  // neither block leaves while the other may still read its shared memory or signal its barriers
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

cudaLaunchConfig_t grouped_pair_config(int pairs, int tiles_m, cudaStream_t stream, cudaLaunchAttribute (&attributes)[2]) {
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(2 * pairs);
    config.blockDim = dim3(PAIR_THREADS);
    config.dynamicSmemBytes = grouped_pair_smem(tiles_m);
    config.stream = stream;
    attributes[0].id = cudaLaunchAttributeClusterDimension;
    attributes[0].val.clusterDim.x = 2;
    attributes[0].val.clusterDim.y = 1;
    attributes[0].val.clusterDim.z = 1;
    attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[1].val.programmaticStreamSerializationAllowed = overlap_launches() ? 1 : 0;
    config.attrs = attributes;
    config.numAttrs = 2;
    return config;
}

// How many pairs of blocks the device runs at a time (a pair needs two SMs of one processing cluster); the kernel is allowed its most shared memory once.
int resident_grouped_pairs() {
    static const int pairs = [] {
        if (cudaFuncSetAttribute(gemm_grouped_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)grouped_pair_smem(GP_MOST_TILES)) != cudaSuccess) return -1;
        cudaLaunchAttribute attributes[2];
        cudaLaunchConfig_t config = grouped_pair_config(sm_count(), GP_MOST_TILES, nullptr, attributes);
        config.numAttrs = 1;
        int clusters = 0;
        return cudaOccupancyMaxActiveClusters(&clusters, gemm_grouped_pair_kernel, &config) == cudaSuccess && clusters > 0 ? clusters : sm_count() / 2;
    }();
    return pairs;
}

// ---------------------------------------------------------------- a few rows per expert: the matrices stream once
constexpr int ROWS_AT_ONCE = 8, COLUMNS_PER_BLOCK = 32, COLUMNS_AT_ONCE = 2, ROWS_THREADS = 256, ROWS_MOST_SHARED = 200 * 1024;

// Columns `col` and `col + 1` of ROWS rows in shared memory: a lane takes every 32nd 16-byte piece of the matrix rows, several of them asked for
// before the first is used (the step is bound by how many bytes are on their way), the lanes meet in a butterfly.  Every sum has the same
// shape whatever ROWS is.
template <int ROWS>
__device__ __forceinline__ void stream_columns(const bf16* __restrict__ first_row, int columns, const bf16* rows, int chunks, float (&sum)[COLUMNS_AT_ONCE][ROWS]) {
    const int lane = threadIdx.x & 31;
    const size_t k = (size_t)chunks * 8;
#pragma unroll
    for (int c = 0; c < COLUMNS_AT_ONCE; ++c)
#pragma unroll
        for (int r = 0; r < ROWS; ++r) sum[c][r] = 0.f;
    const bf16* second = first_row + (columns > 1 ? k : 0);  // an odd last column is read twice and stored once
#pragma unroll 4
    for (int piece = lane; piece < chunks; piece += 32) {
        const uint4 raw[COLUMNS_AT_ONCE] = {__ldg(reinterpret_cast<const uint4*>(first_row + piece * 8)), __ldg(reinterpret_cast<const uint4*>(second + piece * 8))};
        float w[COLUMNS_AT_ONCE][8];
#pragma unroll
        for (int c = 0; c < COLUMNS_AT_ONCE; ++c) {
            const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw[c]);
#pragma unroll
            for (int i = 0; i < 4; ++i) { const float2 f = __bfloat1622float2(p[i]); w[c][2 * i] = f.x; w[c][2 * i + 1] = f.y; }
        }
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            const uint4 xr = *reinterpret_cast<const uint4*>(rows + (size_t)r * k + piece * 8);
            const __nv_bfloat162* xp = reinterpret_cast<const __nv_bfloat162*>(&xr);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 f = __bfloat1622float2(xp[i]);
#pragma unroll
                for (int c = 0; c < COLUMNS_AT_ONCE; ++c) {
                    sum[c][r] = fmaf(f.x, w[c][2 * i], sum[c][r]);
                    sum[c][r] = fmaf(f.y, w[c][2 * i + 1], sum[c][r]);
                }
            }
        }
    }
#pragma unroll
    for (int c = 0; c < COLUMNS_AT_ONCE; ++c)
#pragma unroll
        for (int r = 0; r < ROWS; ++r) sum[c][r] = warp_sum(sum[c][r]);
}

template <int ROWS>
__device__ __forceinline__ void stream_tile(const bf16* __restrict__ we, const bf16* rows, bf16* __restrict__ c, int count, int n, int k, int act) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int j = warp * COLUMNS_AT_ONCE; j < COLUMNS_PER_BLOCK; j += ROWS_THREADS / 32 * COLUMNS_AT_ONCE) {
        const int col = blockIdx.x * COLUMNS_PER_BLOCK + j;
        if (col >= n) break;
        float sum[COLUMNS_AT_ONCE][ROWS];
        stream_columns<ROWS>(we + (size_t)col * k, n - col, rows, k / 8, sum);
        const int r = lane % ROWS, which = lane / ROWS;  // lane: row r of column col + which
        if (which < COLUMNS_AT_ONCE && r < count && col + which < n) {
            float mine = sum[0][0];
#pragma unroll
            for (int cc = 0; cc < COLUMNS_AT_ONCE; ++cc)
#pragma unroll
                for (int rr = 0; rr < ROWS; ++rr)
                    if (which == cc && r == rr) mine = sum[cc][rr];
            c[(size_t)r * n + col + which] = __float2bfloat16_rn(activated(mine, act));
        }
    }
}

// row_token: null, or the row of `a` that stands in a slot (the rows then need not be gathered first).
__global__ void __launch_bounds__(ROWS_THREADS) gemm_grouped_rows_kernel(const bf16* __restrict__ a, int a_stride, const int* __restrict__ row_token,
                                                                         const bf16* __restrict__ w, bf16* __restrict__ c, const int* __restrict__ tile_expert,
                                                                         const int* __restrict__ tile_rows, int pad, int n, int k, int act) {
    extern __shared__ __align__(16) unsigned char rows_raw[];
    bf16* rows = reinterpret_cast<bf16*>(rows_raw);  // [ROWS_AT_ONCE, k]
    let_next_kernel_start();
    wait_for_previous_kernels();  // the tile list and the rows come from the kernels before
    const int tile = blockIdx.y;
    const int expert = tile_expert[tile];
    if (expert < 0) return;
    const int real = tile_rows[tile];
    const bf16* we = w + (size_t)expert * n * k;
    const int chunks = k / 8;  // 16-byte pieces of a row
    for (int first = 0; first < real; first += ROWS_AT_ONCE) {
        const int count = min(ROWS_AT_ONCE, real - first), filled = count <= 2 ? count : (count <= 4 ? 4 : ROWS_AT_ONCE);
        __syncthreads();
        for (int e = threadIdx.x; e < filled * chunks; e += ROWS_THREADS) {
            const int r = e / chunks, piece = e - r * chunks;
            uint4 value = make_uint4(0, 0, 0, 0);
            if (r < count) {
                const int slot = tile * pad + first + r;
                value = *reinterpret_cast<const uint4*>(a + (size_t)(row_token ? row_token[slot] : slot) * a_stride + piece * 8);
            }
            *reinterpret_cast<uint4*>(rows + (size_t)r * k + piece * 8) = value;
        }
        __syncthreads();
        bf16* out = c + (size_t)(tile * pad + first) * n;
        if (count == 1) stream_tile<1>(we, rows, out, count, n, k, act);
        else if (count == 2) stream_tile<2>(we, rows, out, count, n, k, act);
        else if (count <= 4) stream_tile<4>(we, rows, out, count, n, k, act);
        else stream_tile<ROWS_AT_ONCE>(we, rows, out, count, n, k, act);
    }
}

// ---------------------------------------------------------------- some rows per expert: the matrices stream into the tensor cores
// Steps that bring each expert a few rows read the experts' matrices once for them, so they are bound by how many bytes are on their way; the kernel above also spends its float
// units on every row.  Here a warp owns 16 columns of the result and walks all of k in pieces of 32: a lane asks for 16 bytes of two matrix rows per piece, eight pieces ahead, and they
// go straight into the fragments of mma.m16n8k16 (a sum over k may take a piece's k in any order; the rows of `a`, in shared memory, are read in the same order).  Nothing but the rows'
// staging is shared between warps: eight of them, as every row in shared memory takes its bytes from the L1, which holds the loads in flight.  A row's sum has the same shape whatever
// other rows there are.  Measured over 16 experts of [7168, 4096], two per token, against the kernel above: 32 tokens 139 us (5.9 TB/s), 249 before; 64 tokens 180 us, 389 before;
// [4096, 3584] and 16 tokens 75 us (5.9 TB/s), 82 before.  (In one running sum of the tensor cores, which loses to the kernel above in precision: 133, 169 and 71 us; two warps to 16
// columns, each over half of k: 145, 195 and 79 us; pieces added up two by two: 143, 190 and 77 us.)
constexpr int STREAM_WARPS = 8, STREAM_COLUMNS = 16 * STREAM_WARPS, STREAM_THREADS = 32 * STREAM_WARPS, AHEAD = 8, PIECE = 32;

__host__ __device__ constexpr int padded_row(int k) {  // 64 bytes past a multiple of 128, so that two rows' 64-byte pieces fall on different banks
    const int whole = (k + PIECE - 1) / PIECE * PIECE;
    return whole % 64 == 0 ? whole + 32 : whole;
}
constexpr int STREAM_MOST_K = 200 * 1024 / 16, STREAM_MOST_SHARED = 8 * padded_row(STREAM_MOST_K) * 2;  // eight rows of the longest; sixteen are taken up to 100 KB
static_assert(STREAM_MOST_SHARED <= 227 * 1024, "an SM's shared memory");
__device__ __forceinline__ void multiply(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

// Columns col0 .. col0 + 15 of `count` (up to 8 TILES) rows in shared memory.
template <int TILES>
__device__ __forceinline__ void stream_columns(const bf16* __restrict__ we, const bf16* rows, bf16* __restrict__ c, int col0, int count, int n, int k, int act) {
    static_assert(TILES == 1 || TILES == 2, "eight or sixteen rows");
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, pieces = (k + PIECE - 1) / PIECE, ld = padded_row(k);
    const bf16* w0 = we + (size_t)min(col0 + g, n - 1) * k + t * 8;
    const bf16* w1 = we + (size_t)min(col0 + g + 8, n - 1) * k + t * 8;
    const bf16* mine[TILES];  // the row a lane reads (the last one for rows that are not there; their products go nowhere)
#pragma unroll
    for (int z = 0; z < TILES; ++z) mine[z] = rows + (size_t)min(z * 8 + g, count - 1) * ld + t * 8;
    float acc[TILES][4];
#pragma unroll
    for (int z = 0; z < TILES; ++z) acc[z][0] = acc[z][1] = acc[z][2] = acc[z][3] = 0.f;
    uint4 lo[AHEAD], hi[AHEAD];
    auto fetch = [&](int u, int piece) {
        const int at = piece * PIECE;
        lo[u] = hi[u] = make_uint4(0, 0, 0, 0);
        if (at + t * 8 < k) {
            asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(lo[u].x), "=r"(lo[u].y), "=r"(lo[u].z), "=r"(lo[u].w) : "l"(w0 + at));
            asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(hi[u].x), "=r"(hi[u].y), "=r"(hi[u].z), "=r"(hi[u].w) : "l"(w1 + at));
        }
    };
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) fetch(u, u);
    for (int first = 0; first < pieces; first += AHEAD) {
        // The tensor cores cut sums off towards zero, so they add up sixteen products and float the rest, in short sums: of four pieces each, then of these
        float run[2][TILES][4];
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
#pragma unroll
            for (int z = 0; z < TILES; ++z) {
                float one[4] = {}, other[4] = {};
                if (first + u < pieces) {
                    const uint4 b = *reinterpret_cast<const uint4*>(mine[z] + (first + u) * PIECE);
                    multiply(one, lo[u].x, hi[u].x, lo[u].y, hi[u].y, b.x, b.y);
                    multiply(other, lo[u].z, hi[u].z, lo[u].w, hi[u].w, b.z, b.w);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float& sum = run[u & 1][z][i];
                    sum = u < 2 ? one[i] + other[i] : sum + (one[i] + other[i]);
                    if (u == AHEAD - 1) acc[z][i] += run[0][z][i] + run[1][z][i];
                }
            }
            fetch(u, first + AHEAD + u);
        }
    }
#pragma unroll
    for (int z = 0; z < TILES; ++z)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = z * 8 + 2 * t + (i & 1), column = col0 + g + 8 * (i >> 1);
            if (row < count && column < n) c[(size_t)row * n + column] = __float2bfloat16_rn(activated(acc[z][i], act));
        }
}

// row_token: null, or the row of `a` that stands in a slot (the rows then need not be gathered first).  at_once: rows in shared memory, up to 16.
__global__ void __launch_bounds__(STREAM_THREADS, 2) gemm_grouped_stream_kernel(const bf16* __restrict__ a, int a_stride, const int* __restrict__ row_token,
                                                                           const bf16* __restrict__ w, bf16* __restrict__ c, const int* __restrict__ tile_expert,
                                                                           const int* __restrict__ tile_rows, int pad, int at_once, int n, int k, int act) {
    extern __shared__ __align__(16) unsigned char rows_raw[];
    bf16* rows = reinterpret_cast<bf16*>(rows_raw);  // [at_once, padded_row(k)]
    let_next_kernel_start();
    wait_for_previous_kernels();  // the tile list and the rows come from the kernels before
    const int tile = blockIdx.y;
    const int expert = tile_expert[tile];
    if (expert < 0) return;
    const int real = tile_rows[tile], ld = padded_row(k), chunks = (k + PIECE - 1) / PIECE * (PIECE / 8);  // 16-byte pieces of a row
    const bf16* we = w + (size_t)expert * n * k;
    const int col0 = (blockIdx.x * STREAM_WARPS + (threadIdx.x >> 5)) * 16;
    for (int first = 0; first < real; first += at_once) {
        const int count = min(at_once, real - first);
        if (first) __syncthreads();
        for (int e = threadIdx.x; e < count * chunks; e += STREAM_THREADS) {
            const int r = e / chunks, piece = e - r * chunks, slot = tile * pad + first + r;
            uint4 value = make_uint4(0, 0, 0, 0);
            if (piece * 8 < k) value = *reinterpret_cast<const uint4*>(a + (size_t)(row_token ? row_token[slot] : slot) * a_stride + piece * 8);
            *reinterpret_cast<uint4*>(rows + (size_t)r * ld + piece * 8) = value;
        }
        __syncthreads();
        if (col0 >= n) continue;
        bf16* out = c + (size_t)(tile * pad + first) * n;
        if (count <= 8) stream_columns<1>(we, rows, out, col0, count, n, k, act);
        else stream_columns<2>(we, rows, out, col0, count, n, k, act);
    }
}
}  // namespace

// a [rows, k] and c [rows, n] dense bfloat16 (rows a multiple of 128), w [experts, n, k] dense bfloat16, k a multiple of 8.
HB_EXPORT int hb_moe_gemm_tiles(const void* a, const void* w, void* c, const int* tile_expert, int rows, int experts, int n, int k, int act,
                                int* status, cudaStream_t stream) {
    if (rows <= 0 || n <= 0) return 0;
    if (k <= 0 || rows % BM || experts <= 0 || (k % 8) || !tile_expert) return HB_BAD_ARGUMENT;
    if ((long long)experts * n > 0x7fffffffLL) return HB_UNSUPPORTED_SIZE;
    const int bn = n % 256 == 0 || n >= 1024 ? 256 : 128;
    CUtensorMap map_x, map_w;
    if (int code = make_map(&map_x, a, rows, k, k, BM)) return code;
    if (int code = make_map(&map_w, w, experts * n, k, k, bn)) return code;
    const int tiles_m = rows / BM, tiles_n = (n + bn - 1) / bn;
    if ((long long)tiles_m * tiles_n > 0x7fffffffLL) return HB_UNSUPPORTED_SIZE;
    const int blocks = min(tiles_m * tiles_n, sm_count());
    const GroupedParams p{(bf16*)c, tile_expert, rows, n, k, n, act, status};
    return bn == 256 ? launch_grouped<256>(map_x, map_w, p, tiles_m, tiles_n, blocks, stream)
                     : launch_grouped<128>(map_x, map_w, p, tiles_m, tiles_n, blocks, stream);
}

// The same product on pairs of SMs; act HB_ACT_SWIGLU: every 256 rows of an expert's matrix are 128 gate rows followed by their 128 up rows (n a multiple of 256),
// c [rows, n / 2].
HB_EXPORT int hb_moe_gemm_pairs(const void* a, const void* w, void* c, const int* tile_expert, int rows, int experts, int n, int k, int act, int* status,
                                cudaStream_t stream) {
    if (rows <= 0 || n <= 0) return 0;
    if (k <= 0 || rows % BM || experts <= 0 || (k % 8) || !tile_expert || act < HB_ACT_NONE || act > HB_ACT_SWIGLU) return HB_BAD_ARGUMENT;
    if ((long long)experts * n > 0x7fffffffLL || rows / BM > GP_MOST_TILES || (act == HB_ACT_SWIGLU && n % 256)) return HB_UNSUPPORTED_SIZE;
    CUtensorMap map_x, map_w;
    if (int code = make_map(&map_x, a, rows, k, k, BM)) return code;
    if (int code = make_map(&map_w, w, experts * n, k, k, 128)) return code;
    const int tiles_m = rows / BM, tiles_n = (n + 255) / 256, resident = resident_grouped_pairs();
    if (resident < 1) return HB_UNSUPPORTED_SIZE;
    if ((long long)tiles_m * tiles_n > 0x7fffffffLL) return HB_UNSUPPORTED_SIZE;
    const GroupedParams p{(bf16*)c, tile_expert, rows, n, k, act == HB_ACT_SWIGLU ? n / 2 : n, act, status};
    cudaLaunchAttribute attributes[2];
    const int pairs = tiles_m * tiles_n < resident ? tiles_m * tiles_n : resident;
    const cudaLaunchConfig_t config = grouped_pair_config(pairs, tiles_m, stream, attributes);
    return (int)cudaLaunchKernelEx(&config, gemm_grouped_pair_kernel, map_x, map_w, p, tiles_m, tiles_n);
}

// The same product for steps of a few rows; tile_rows[i]: the real rows at the start of tile i.  row_token (or null): the row of `a` that stands in
// a slot, rows a_stride elements apart.
HB_EXPORT int hb_moe_gemm_rows(const void* a, int a_stride, const int* row_token, const void* w, void* c, const int* tile_expert, const int* tile_rows, int pad, int rows, int n, int k,
                               int act, cudaStream_t stream) {
    if (rows <= 0 || n <= 0) return 0;
    if (k <= 0 || pad <= 0 || rows % pad || (k % 8) || (a_stride % 8) || !tile_expert || !tile_rows) return HB_BAD_ARGUMENT;
    if ((((uintptr_t)a | (uintptr_t)w) & 15)) return HB_BAD_ARGUMENT;
    const size_t shared = (size_t)ROWS_AT_ONCE * k * sizeof(bf16);
    if (shared > ROWS_MOST_SHARED || rows / pad > 65535) return HB_UNSUPPORTED_SIZE;
    if (shared > 48 * 1024) {  // always the most that any call takes: another thread's call may come between this and the launch
        cudaError_t e = cudaFuncSetAttribute(gemm_grouped_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ROWS_MOST_SHARED);
        if (e != cudaSuccess) return (int)e;
    }
    const dim3 grid((n + COLUMNS_PER_BLOCK - 1) / COLUMNS_PER_BLOCK, rows / pad);
    return launch_after_previous(gemm_grouped_rows_kernel, grid, dim3(ROWS_THREADS), shared, stream, (const bf16*)a, a_stride, row_token, (const bf16*)w, (bf16*)c, tile_expert,
                                 tile_rows, pad, n, k, act);
}

// The same with some rows per expert: `most` real rows per tile at the most, any number of rows and columns.  row_token (or null): the row of `a` that stands in
// a slot, rows a_stride elements apart.
HB_EXPORT int hb_moe_gemm_stream(const void* a, int a_stride, const int* row_token, const void* w, void* c, const int* tile_expert, const int* tile_rows, int pad, int most, int rows, int n,
                               int k, int act, cudaStream_t stream) {
    if (rows <= 0 || n <= 0) return 0;
    if (k <= 0 || pad <= 0 || most <= 0 || rows % pad || (k % 8) || (a_stride % 8) || !tile_expert || !tile_rows) return HB_BAD_ARGUMENT;
    if ((((uintptr_t)a | (uintptr_t)w) & 15)) return HB_BAD_ARGUMENT;
    const size_t per_row = (size_t)padded_row(k) * sizeof(bf16);
    // shared memory for no more rows than a tile can have: what is left decides how many blocks, and bytes on their way, an SM holds
    const int limit = most < pad ? most : pad, at_once = limit > 8 && 16 * per_row <= 100 * 1024 ? (limit < 16 ? limit : 16) : (limit < 8 ? limit : 8);
    const size_t shared = at_once * per_row;
    if (k > STREAM_MOST_K || rows / pad > 65535) return HB_UNSUPPORTED_SIZE;
    if (shared > 48 * 1024) {  // always the most that any call takes: another thread's call may come between this and the launch
        cudaError_t e = cudaFuncSetAttribute(gemm_grouped_stream_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, STREAM_MOST_SHARED);
        if (e != cudaSuccess) return (int)e;
    }
    const dim3 grid((n + STREAM_COLUMNS - 1) / STREAM_COLUMNS, rows / pad);
    return launch_after_previous(gemm_grouped_stream_kernel, grid, dim3(STREAM_THREADS), shared, stream, (const bf16*)a, a_stride, row_token, (const bf16*)w, (bf16*)c, tile_expert,
                                 tile_rows, pad, at_once, n, k, act);
}
