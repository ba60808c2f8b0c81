// Products of a few rows with a matrix of a few megabytes, C[M, N] = A[M, K] W[N, K]^T, M up to 16, bfloat16: what a decoded token asks of a small model.
//
// Such a product is a chain of waits: the launch, the weights, the rows, the sums.  Here the weights do not wait for the kernel before: every warp has its first units
// of the matrix on their way into registers before it waits for that kernel, so that afterwards only the rows, which are in L2, and the
// sums remain.  That asks for a matrix that no kernel still in flight writes, a model's weights: where the caller does not say so (`settled`), the launch is an ordinary one,
// behind the kernel before (one row, in chains of such products: [896, 896] 4.2 us in the library, 2.2 here; [9,728, 896] with SwiGLU 8.1 in two launches, 5.0 here, 2.7 of them for
// the bytes).
//
// A unit is 16 rows of W by 64 of k.  A block takes whole tiles of 16 rows (or, for sums that are left in pieces, a part of k of one tile), its warps an even share of their
// units one after another.  A lane asks for 16 bytes of two matrix rows per 32 of k, which go straight into the fragments of mma.m16n8k16 with the step's rows
// as the eight columns (a sum over k may take k in any order; the rows are read in the same order).  A tile that several warps share meets in shared memory, in warp
// order.  A result depends on the shapes and the row alone, not on the other rows.
//   epilogue 0: C bfloat16 (+ bias), 1: C float (+ bias), 2: SwiGLU, C bfloat16 [M, N / 2], gate and up rows of W in turn in runs of gu_block,
//   3: float pieces [parts, M, N], each the sum over one of `parts` equal parts of k, to be added up in order by the reader.
#include "common.cuh"

namespace {
typedef __nv_bfloat16 bf16;
constexpr int WARPS = 8, THREADS = WARPS * 32, UNIT_K = 64;
enum : int { FEW_BF16 = 0, FEW_F32 = 1, FEW_SWIGLU = 2, FEW_PIECES = 3 };

struct FewArgs {
    const bf16* x;
    const bf16* w;
    const bf16* bias_h;
    const float* bias_f;
    void* c;
    int x_stride, c_stride, rows, n, k;
    int tiles_each, parts;   // tiles of a block; or parts of a tile (one tile and one part to a block)
    int gu_block, gu_shift;  // SwiGLU: runs of a power of two (or one run of all, and an exponent that leaves no run but the first)
};

__device__ __forceinline__ uint4 weights16(const bf16* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void multiply(float (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int NT, int RING, int EPI>
__global__ void __launch_bounds__(THREADS, 2) few_rows_kernel(const FewArgs a) {
    constexpr bool GLU = EPI == FEW_SWIGLU;
    constexpr int SUMS = 128 * NT;
    __shared__ float red[WARPS * 2 * SUMS];  // a warp's part of its first tile and of its last
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int k_units = a.k / UNIT_K, tiles = a.n / 16;
    const int tile0 = EPI == FEW_PIECES ? blockIdx.x / a.parts : blockIdx.x * a.tiles_each, piece = EPI == FEW_PIECES ? blockIdx.x - tile0 * a.parts : 0;
    const int ku0 = EPI == FEW_PIECES ? piece * k_units / a.parts : 0, each = EPI == FEW_PIECES ? (piece + 1) * k_units / a.parts - ku0 : k_units;  // units of a tile here
    const int n_tiles = EPI == FEW_PIECES ? 1 : min(a.tiles_each, tiles - tile0), units = n_tiles * each;
    auto begins = [&](int w) { return units * w / WARPS; };
    const int begin = begins(warp), count = begins(warp + 1) - begin, first_tile = begin / each;

    auto matrix_row = [&](int tile, int r) {
        if (!GLU) return tile * 16 + r;
        const int gate = tile * 8 + (r & 7);
        return gate + ((gate >> a.gu_shift) + (r >> 3)) * a.gu_block;
    };
    // the weights: rows g and g + 8 of a tile, 32 of k each: lo, lo + 32, hi, hi + 32
    uint4 ring[RING][4];
    const bf16 *lo, *hi;
    int ask_tile = first_tile, ask_ku = begin - first_tile * each, to_ask = count;
    auto enter = [&]() {
        lo = a.w + (size_t)matrix_row(tile0 + ask_tile, g) * a.k + (ku0 + ask_ku) * UNIT_K + t * 8;
        hi = a.w + (size_t)matrix_row(tile0 + ask_tile, g + 8) * a.k + (ku0 + ask_ku) * UNIT_K + t * 8;
    };
    auto ask = [&](int slot) {
        if (to_ask-- <= 0) return;
        ring[slot][0] = weights16(lo);
        ring[slot][1] = weights16(lo + 32);
        ring[slot][2] = weights16(hi);
        ring[slot][3] = weights16(hi + 32);
        lo += UNIT_K, hi += UNIT_K;
        if (++ask_ku == each) {
            ask_ku = 0, ++ask_tile;
            enter();
        }
    };
    enter();
#pragma unroll
    for (int u = 0; u < RING; ++u) ask(u);

    wait_for_previous_kernels();  // the rows come from them
    let_next_kernel_start();      // not before: kernels further down the stream would take the room that the next ones need
    uint4 rows[RING][NT][2];
    const bf16* mine = a.x + (size_t)g * a.x_stride + ku0 * UNIT_K + t * 8;
    int row_ku = begin - first_tile * each, rows_to_ask = count;
    auto ask_rows = [&](int slot) {
        if (rows_to_ask-- <= 0) return;
#pragma unroll
        for (int z = 0; z < NT; ++z)
#pragma unroll
            for (int half = 0; half < 2; ++half)
                rows[slot][z][half] = z * 8 + g < a.rows ? *reinterpret_cast<const uint4*>(mine + (size_t)z * 8 * a.x_stride + row_ku * UNIT_K + half * 32) : make_uint4(0, 0, 0, 0);
        if (++row_ku == each) row_ku = 0;
    };
#pragma unroll
    for (int u = 0; u < RING; ++u) ask_rows(u);

    auto emit = [&](int tile, int r, int token, float value, float other) {
        if (token >= a.rows) return;
        if (EPI == FEW_SWIGLU) {  // the projections are rounded before the activation, as separate kernels would store them
            const float gate = __bfloat162float(__float2bfloat16_rn(value)), up = __bfloat162float(__float2bfloat16_rn(other));
            reinterpret_cast<bf16*>(a.c)[(size_t)token * a.c_stride + (tile0 + tile) * 8 + r] = __float2bfloat16_rn(gate / (1.0f + expf(-gate)) * up);
            return;
        }
        const int col = (tile0 + tile) * 16 + r;
        if (EPI == FEW_PIECES) {
            reinterpret_cast<float*>(a.c)[((size_t)piece * a.rows + token) * a.n + col] = value;
            return;
        }
        if (a.bias_h) value += __bfloat162float(a.bias_h[col]);
        if (a.bias_f) value += a.bias_f[col];
        if (EPI == FEW_F32) reinterpret_cast<float*>(a.c)[(size_t)token * a.c_stride + col] = value;
        else reinterpret_cast<bf16*>(a.c)[(size_t)token * a.c_stride + col] = __float2bfloat16_rn(value);
    };

    float acc[NT][4];
#pragma unroll
    for (int z = 0; z < NT; ++z) acc[z][0] = acc[z][1] = acc[z][2] = acc[z][3] = 0.f;
    int tile = first_tile, ku = begin - first_tile * each, part = ku;
    for (int done = 0; done < count; done += RING) {
#pragma unroll
        for (int u = 0; u < RING; ++u) {
            if (done + u >= count) break;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const uint4 l = ring[u][half], h = ring[u][2 + half];
#pragma unroll
                for (int z = 0; z < NT; ++z) {
                    const uint4 b = rows[u][z][half];
                    multiply(acc[z], l.x, h.x, l.y, h.y, b.x, b.y);
                    multiply(acc[z], l.z, h.z, l.w, h.w, b.z, b.w);
                }
            }
            ask(u);
            ask_rows(u);
            if (++ku == each || done + u + 1 == count) {  // units part .. ku of the tile are summed up
                if (part == 0 && ku == each) {
#pragma unroll
                    for (int z = 0; z < NT; ++z)
#pragma unroll
                        for (int c = 0; c < (GLU ? 2 : 4); ++c) emit(tile, g + 8 * (c >> 1), z * 8 + 2 * t + (c & 1), acc[z][c], acc[z][c ^ 2]);
                } else {
                    float* to = red + (warp * 2 + (tile != first_tile)) * SUMS;
#pragma unroll
                    for (int z = 0; z < NT; ++z)
#pragma unroll
                        for (int c = 0; c < 4; ++c) to[z * 128 + c * 32 + lane] = acc[z][c];
                }
#pragma unroll
                for (int z = 0; z < NT; ++z) acc[z][0] = acc[z][1] = acc[z][2] = acc[z][3] = 0.f;
                if (ku == each) ku = 0, ++tile;
                part = ku;
            }
        }
    }
    __syncthreads();
    constexpr int EACH = GLU ? SUMS / 2 : SUMS;
    for (int e = threadIdx.x; e < n_tiles * EACH; e += THREADS) {  // tiles of several warps, in warp order
        const int of = e / EACH, i = e % EACH, index = GLU ? i / 64 * 128 + i % 64 : i, from = of * each, to = from + each;
        float sum = 0.f, other = 0.f;
        bool shared_tile = false;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            const int b = begins(w), next = begins(w + 1);
            if (b >= to || next <= from || b == next || (b <= from && next >= to)) continue;
            const float* part_of = red + (w * 2 + (b < from)) * SUMS + index;
            sum += part_of[0];
            if (GLU) other += part_of[64];
            shared_tile = true;
        }
        const int z = index / 128, c = index / 32 & 3, l = index & 31;
        if (shared_tile) emit(of, (l >> 2) + 8 * (c >> 1), z * 8 + 2 * (l & 3) + (c & 1), sum, other);
    }
}

template <int EPI>
int launch_few(const FewArgs& a, int blocks, bool settled, cudaStream_t stream) {
    if (a.rows <= 8) return launch_in_turn(settled, few_rows_kernel<1, 4, EPI>, dim3(blocks), dim3(THREADS), 0, stream, a);
    return launch_in_turn(settled, few_rows_kernel<2, 3, EPI>, dim3(blocks), dim3(THREADS), 0, stream, a);
}
}  // namespace

// x [rows, k] (row stride x_stride), w [n, k] dense, bfloat16; k a multiple of 64, n of 16.  epilogue as above; parts: of epilogue 3 (1 otherwise);
// blocks: how many the device should hold at a time; settled: no kernel still in flight writes w.
HB_EXPORT int hb_few_rows(const void* x, int x_stride, const void* w, const void* bias_h, const float* bias_f, void* c, int c_stride, int rows, int n, int k, int epilogue,
                          int gu_block, int parts, int blocks, int settled, cudaStream_t stream) {
    if (rows <= 0 || n <= 0) return 0;
    if (rows > 16 || k <= 0 || k % UNIT_K || n % 16 || (x_stride & 7) || ((((uintptr_t)x) | ((uintptr_t)w)) & 15)) return HB_UNSUPPORTED_SIZE;
    if (blocks < 1 || parts < 1 || parts > k / UNIT_K || epilogue < FEW_BF16 || epilogue > FEW_PIECES) return HB_BAD_ARGUMENT;
    FewArgs a{(const bf16*)x, (const bf16*)w, (const bf16*)bias_h, bias_f, c, x_stride, c_stride, rows, n, k, 1, 1, 0, 0};
    const int tiles = n / 16;
    a.tiles_each = (tiles + blocks - 1) / blocks;
    const int grid = (tiles + a.tiles_each - 1) / a.tiles_each;
    if (epilogue == FEW_SWIGLU) {
        const int inter = n / 2;
        if (bias_h || bias_f || n % 32 || gu_block < 8 || inter % gu_block || (gu_block != inter && (gu_block & (gu_block - 1)))) return HB_UNSUPPORTED_SIZE;
        a.gu_block = gu_block;
        a.gu_shift = gu_block == inter ? 31 : __builtin_ctz((unsigned)gu_block);
        return launch_few<FEW_SWIGLU>(a, grid, settled != 0, stream);
    }
    if (epilogue == FEW_PIECES) {
        if (bias_h || bias_f) return HB_BAD_ARGUMENT;
        a.parts = parts;
        return launch_few<FEW_PIECES>(a, tiles * parts, settled != 0, stream);
    }
    return epilogue == FEW_F32 ? launch_few<FEW_F32>(a, grid, settled != 0, stream) : launch_few<FEW_BF16>(a, grid, settled != 0, stream);
}
