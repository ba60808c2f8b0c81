// What the matrix-product kernels on pairs of SMs share: sizes of a pair's tile and ring, cluster and tcgen05.cta_group::2 helpers in inline PTX.
#pragma once
#include "gemm_tcgen05.cuh"

namespace {
constexpr int PAIR_THREADS = 320;  // producer warp, tensor-core warp, eight epilogue warps (two per quarter of the accumulator's lanes)
constexpr int PAIR_ROWS = 2 * BM;  // rows of a tile
constexpr int ACC_STRIDE = 256;    // tensor-memory columns between the two accumulators
constexpr int TMEM_COLS = 512;
constexpr int A_BYTES = BM * BK * 2;
constexpr int SMEM_ROOM = 227 * 1024 - 1024 - 512;

__host__ __device__ constexpr int b_bytes(int bn) { return (bn / 2) * BK * 2; }
__host__ __device__ constexpr int stage_bytes(int bn) { return A_BYTES + b_bytes(bn); }
__host__ __device__ constexpr int stages_for(int bn) { return SMEM_ROOM / stage_bytes(bn) > 8 ? 8 : SMEM_ROOM / stage_bytes(bn); }

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The address, in the cluster's shared window, of the leader's copy of a barrier of this block.
__device__ __forceinline__ unsigned in_leader(const void* local) {
    unsigned remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(remote) : "r"(smem_u32(local)));
    return remote;
}
__device__ __forceinline__ void arrive_in_leader(unsigned remote_bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote_bar) : "memory");
}
// This block's tile into its own shared memory; the bytes count on the leader's barrier.
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, unsigned leader_bar, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(smem_u32(dst)), "l"(map), "r"(leader_bar), "r"(x), "r"(y) : "memory");
}
// Arrives on the barrier at this offset in both blocks of the pair once the products issued so far have finished.
__device__ __forceinline__ void umma_commit_both(unsigned long long* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"((unsigned short)3) : "memory");
}
// Four products over one 64-deep stage: K advances by 16 elements = 32 bytes = 2 units of the descriptor's address field.
__device__ __forceinline__ void umma_pair_stage(unsigned tmem_d, unsigned a_low, unsigned b_low, unsigned idesc, unsigned accumulate_first) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\t.reg .b32 al, bl;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.eq.b32 q, 0, 0;\n\t"
        "mov.b64 da, {%1, %5};\n\t"
        "mov.b64 db, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, p;\n\t"
        "add.u32 al, %1, 2;\n\t"
        "add.u32 bl, %2, 2;\n\t"
        "mov.b64 da, {al, %5};\n\t"
        "mov.b64 db, {bl, %5};\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, q;\n\t"
        "add.u32 al, %1, 4;\n\t"
        "add.u32 bl, %2, 4;\n\t"
        "mov.b64 da, {al, %5};\n\t"
        "mov.b64 db, {bl, %5};\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, q;\n\t"
        "add.u32 al, %1, 6;\n\t"
        "add.u32 bl, %2, 6;\n\t"
        "mov.b64 da, {al, %5};\n\t"
        "mov.b64 db, {bl, %5};\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, q;\n\t}"
        ::"r"(tmem_d), "r"(a_low), "r"(b_low), "r"(idesc), "r"(accumulate_first), "r"(DESC_HIGH) : "memory");
}
__device__ __forceinline__ void umma_commit_both_at(unsigned bar_addr) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar_addr), "h"((unsigned short)3) : "memory");
}

// Instruction descriptor of kind::f16: float accumulator, bfloat16 operands, both K-major, M = 256 over the pair, N = bn.
__device__ __forceinline__ unsigned pair_idesc(int bn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(bn >> 3) << 17) | ((unsigned)(PAIR_ROWS >> 4) << 24);
}

// 32 consecutive float columns of this thread's accumulator lane.
__device__ __forceinline__ void tmem_ld32(unsigned taddr, float (&v)[32]) {
    unsigned r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
          "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
          "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
          "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
}  // namespace
