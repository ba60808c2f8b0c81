// Recurrences over a float matrix state, walked in chunks of 64 tokens at float precision:
//     delta rule:    S <- a S;  u = b (v - S^T k);  S <- S + k u^T;  o = S^T q     (a one number per head, or one per key entry)
//     retention:     S <- a S + k v^T;  o = S^T q                                  (a fixed per head)
//     wkv:           o = S^T q + (sum_i u_i k_i q_i) v;  S <- diag(w) S + k v^T
// With A_t the (diagonal) decay of token t, A(j, i] the product over the tokens behind j up to i, and S0 the state at the chunk's start,
//     u_i = b_i (v_i - (A(0, i] k_i)^T S0 - sum_(j < i) (k_i^T A(j, i] k_j) u_j),     o_i = (A(0, i] q_i)^T S0 + sum_(j <= i) (q_i^T A(j, i] k_j) u_j,
//     S_end = A(0, end] S0 + sum_j (A(j, end] k_j) u_j^T                              (no rule: u = v; wkv: the query's decay ends a token earlier).
// prepare_chunks works on all chunks side by side: it makes the small matrices and solves the triangular system for [b K | b V], so that a chunk's
// u = U0 - W S0.  walk_chunks carries the state through a row's chunks, a block per head and ETILE value columns: two products of 64 x n and n x 64 per
// chunk instead of 64 dependent tokens.  What a token holds reaches later tokens only: a value that is not finite leaves the tokens before it as they are (and those behind it,
// where an infinity counts, NaN; the scan may keep the infinity).
//
// Precision.  The scan that takes the tokens one after another (recurrent.cu: decoded tokens, other sizes, the float32 mode) is what these kernels must not fall behind.
//  * Products run on the tensor cores over floats cut into three bfloat16 values each, which together are the float; of the nine products the three below 2^-27 of a term are
//    left out.  The tensor cores cut sums off towards zero, so sixteen terms at a time are added up in float.  (Two tf32 halves, the lower one cut off after eleven bits, in running
//    sums: 1.3 to 2 times the scan's distance from 64 bits where decays are strong, and 1.25 times for retention and wkv over 128 tokens.)
//  * What weighs most under strong decays is done in float: a token's own block of sixteen, the last block for the state, and the ones on the diagonal of the inverses.
//  * Weights are products of the tokens' decays, never exponentials of sums of logarithms, made in double and rounded once: a decay per token and head as a table of all pairs, a decay
//    per key entry from the ends of blocks of 16 tokens.  Where such a block's decays are too strong to divide by, it is taken pair by pair.
// Distance from 64 bits, heads of 64, 96 and 128, rows of 128 to 2,048 tokens, decays from 0.999 to 1e-9 a token, several seeds: outputs 0.45 to 1.00 of the scan's (8e-8 to 6.7e-7),
// states 0.43 to 1.07 (few entries count under strong decays; 0.97 on average there).
//
// Measured on one B200, a prompt of 2,048 tokens, 16 heads of 128 x 128 (the token-by-token scan): delta rule 239 us (790), with a decay per key entry 273 (1,060),
// retention 147 (434; 290 in segments side by side), wkv with 32 heads of 64 146 (377); the delta rule with 32 heads 376 (942).  With two tf32 halves: 231, 247, 138, 126 and 386.
// What bounds it: the walk is a chain of chunks (4 us each with a delta rule, 3.6 without: products behind one another, six for each in float); the preparation waits for shared
// memory and for chains of products: 96 us (delta rule, two blocks to an SM), 130 (decay per entry, 169 KB and one block), 28 (retention).
#include "common.cuh"

namespace {
constexpr int CHUNK = 64, SUB = 16, SUBS = CHUNK / SUB;
constexpr float STEEP = 1e-25f;  // decays over a sub-block from here on may be divided out
enum : int { RULE_DELTA = 0, RULE_CHANNEL_DELTA = 1, RULE_RETENTION = 2, RULE_WKV = 3 };
__host__ __device__ constexpr bool is_delta(int rule) { return rule == RULE_DELTA || rule == RULE_CHANNEL_DELTA; }

struct Args {
    const float* k;      // [tokens, stride]: group g at g * n
    const float* q;
    const float* v;      // head h at h * e
    int k_stride, q_stride, v_stride;
    const float* x;      // the decay's pre-activations [tokens, x_stride]: head h at x_off + h, or its n entries at x_off + h * n
    int x_stride, x_off;
    const float* step;   // delta rules: b = sigmoid(step), head h at step_off + h
    int step_stride, step_off;
    const float* rate;   // delta rules: a_log [heads]; retention: the decay [heads]; wkv: w0 [heads * n]
    const float* bias;   // delta rule: dt_bias [heads], channel delta: [heads * n]; wkv: the bonus u [heads * n]
    float* scratch;      // per chunk of the span and head: see Pieces
    float* state;        // (slot, head): [e, n_padded] at state + slot * slot_stride + state_off
    size_t slot_stride;
    int state_off;
    const int* slots;
    const int* chunks;   // [chunks, 2]: the first token and the number of tokens of every chunk
    const int* walks;    // [walks, 3]: the chunks of a row that is walked, from and up to, and the row
    int chunk0, chunk1;  // the span of chunks this launch works on
    float* out;          // [tokens, heads * e]
    int heads, groups, n, n_padded, e;
    float q_scale;
    int by_four;         // keys, queries, decays and their strides allow 16-byte loads
    int v_by_four;       // values likewise
    int* status;
};

// What prepare_chunks leaves per chunk and head, in floats: rows as wide as they lie in the walk's shared memory, so that a matrix is one copy.
template <int RULE, int N>
struct Pieces {
    static constexpr int QLD = N + 4, KLD = N + 8, BLD = CHUNK + 4;
    static constexpr int Q = 0, K = CHUNK * QLD, B = K + CHUNK * KLD, FADE = B + CHUNK * BLD, W = FADE + N;
    __host__ __device__ static size_t u(int) { return W + (is_delta(RULE) ? CHUNK * QLD : 0); }
    __host__ __device__ static size_t size(int e) { return u(e) + (is_delta(RULE) ? (size_t)CHUNK * e : 0); }
};

__device__ __forceinline__ float softplus_of(float z) { return z > 20.f ? z : log1pf(expf(z)); }

// ---------------------------------------------------------------- products of floats on the tensor cores
// A float is exactly three bfloat16 values: the nearest one, the nearest one to the rest, and what is left (seven bits at the most).  Integer operations round; an infinity or a NaN
// gives a NaN in the last.  Two floats at a time, as a fragment wants them.
struct Thirds {
    uint32_t a, b, c;
};
__device__ __forceinline__ Thirds thirds(float x, float y) {
    const uint32_t xa = __float_as_uint(x) + 0x8000u, ya = __float_as_uint(y) + 0x8000u;
    x -= __uint_as_float(xa & 0xffff0000u), y -= __uint_as_float(ya & 0xffff0000u);
    const uint32_t xb = __float_as_uint(x) + 0x8000u, yb = __float_as_uint(y) + 0x8000u;
    x -= __uint_as_float(xb & 0xffff0000u), y -= __uint_as_float(yb & 0xffff0000u);
    return {__byte_perm(xa, ya, 0x7632), __byte_perm(xb, yb, 0x7632), __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632)};
}
__device__ __forceinline__ void multiply(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, const float (&c)[4]) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}
// sum + rest += a b.  The tensor cores cut sums off where float arithmetic rounds, always towards zero; so the products of the leading thirds, sixteen at a time, are added up in float,
// and only the small ones stay in a running sum of the tensor cores (what is cut off there is 2^-8 of that).  Left out: products below 2^-27 of a term.
__device__ __forceinline__ void multiply(float (&sum)[4], float (&rest)[4], const Thirds (&a)[4], const Thirds& b0, const Thirds& b1) {
    const float none[4] = {};
    float lead[4];
    multiply(lead, a[0].a, a[1].a, a[2].a, a[3].a, b0.a, b1.a, none);
    multiply(rest, a[0].a, a[1].a, a[2].a, a[3].a, b0.b, b1.b, rest);
    multiply(rest, a[0].b, a[1].b, a[2].b, a[3].b, b0.a, b1.a, rest);
    multiply(rest, a[0].a, a[1].a, a[2].a, a[3].a, b0.c, b1.c, rest);
    multiply(rest, a[0].b, a[1].b, a[2].b, a[3].b, b0.b, b1.b, rest);
    multiply(rest, a[0].c, a[1].c, a[2].c, a[3].c, b0.a, b1.a, rest);
#pragma unroll
    for (int i = 0; i < 4; ++i) sum[i] += lead[i];
}
// A lane's share of sixteen terms: terms t and t + 8 make a fragment's first pair, t + 4 and t + 12 its second one (a sum may take its terms in any order).
// `p`: its first term of row g; terms `step` apart, row g + 8 `down` away.
__device__ __forceinline__ void row_thirds(Thirds (&x)[4], const float* p, int step, int down) {
    x[0] = thirds(p[0], p[8 * step]), x[1] = thirds(p[down], p[down + 8 * step]);
    x[2] = thirds(p[4 * step], p[12 * step]), x[3] = thirds(p[down + 4 * step], p[down + 12 * step]);
}
__device__ __forceinline__ Thirds stored_thirds(const uint32_t* p, int plane) { return {p[0], p[plane], p[2 * plane]}; }
__device__ __forceinline__ void store_thirds(uint32_t* p, int plane, const Thirds& x, const Thirds& y) {  // of two neighbouring columns
    *reinterpret_cast<uint2*>(p) = make_uint2(x.a, y.a);
    *reinterpret_cast<uint2*>(p + plane) = make_uint2(x.b, y.b);
    *reinterpret_cast<uint2*>(p + 2 * plane) = make_uint2(x.c, y.c);
}
__device__ __forceinline__ void multiply(float (&sum)[4], float (&rest)[4], const Thirds (&a)[4], const float* p, int step) {
    multiply(sum, rest, a, thirds(p[0], p[8 * step]), thirds(p[4 * step], p[12 * step]));
}

// `count` consecutive values as `VL` floats, zeros (or `fill`) past the end
template <int VL>
__device__ __forceinline__ void load_some(const float* p, int live, bool wide, float fill, float (&x)[VL]) {
    if (wide && live >= VL) {
        if constexpr (VL == 4) {
            load4(p, x);
        } else {
            const float2 y = *reinterpret_cast<const float2*>(p);
            x[0] = y.x, x[1] = y.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < VL; ++i) x[i] = i < live ? p[i] : fill;
    }
}
template <int VL>
__device__ __forceinline__ void store_some(float* p, const float (&x)[VL]) {
    if constexpr (VL == 4) *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
    else *reinterpret_cast<float2*>(p) = make_float2(x[0], x[1]);
}
template <int VL>
__device__ __forceinline__ void read_some(const float* p, float (&x)[VL]) {
    if constexpr (VL == 4) load4(p, x);
    else {
        const float2 y = *reinterpret_cast<const float2*>(p);
        x[0] = y.x, x[1] = y.y;
    }
}

// ---------------------------------------------------------------- every chunk on its own: grid (chunks of the span, heads)
// A decay per token and head (SCALAR) is kept out of the products: they are plain ones of keys and queries, and the weight A(j, i] of a pair comes from a table of products in
// double, rounded once.  A decay per key entry goes into keys and queries, from the ends of their blocks of sixteen tokens.
constexpr bool has_scalar_decay(int rule) { return rule == RULE_DELTA || rule == RULE_RETENTION; }

template <int RULE, int N>
struct Layout {  // shared memory of a chunk's preparation, in floats
    static constexpr bool DELTA = is_delta(RULE), SCALAR = has_scalar_decay(RULE);
    static constexpr int BLOCKS = SCALAR || N <= 64 ? 2 : 1, THREADS = 512 / BLOCKS;  // sixteen warps to an SM, in as many blocks as its shared memory holds
    static constexpr int LD = N + 4, WLD = CHUNK + 4, TLD = CHUNK + 8, ILD = SUB + 4;
    static constexpr int XLD = SCALAR ? N + 8 : 2 * LD;         // the solution: columns at a time, over the queries (and the scaled keys)
    static constexpr int KS = 0, QS = CHUNK * LD;                               // keys; queries
    static constexpr int AS = QS + (SCALAR ? CHUNK * XLD : CHUNK * LD);         // decays, later keys times the decays behind them in their sub-block; SCALAR: the weights [i][j]
    static constexpr int CS = AS + (SCALAR ? CHUNK * WLD : CHUNK * LD);         // keys over the decays up to them in their sub-block
    static constexpr int AT = CS + (SCALAR ? 0 : CHUNK * LD);                   // (delta) [j][i]: b_i k_i^T A(j, i] k_j
    static constexpr int INVERSE = AT + (DELTA ? CHUNK * TLD : 0);              // (delta) [i][j % 16]: the sub-blocks of (I + at^T)^-1 on the diagonal, its ones included
    static constexpr int WHOLE = INVERSE + (DELTA ? CHUNK * ILD : 0);           // [sub-block][entry]: the product of its decays; SCALAR: the tokens' decays in double
    static constexpr int MIDDLE = WHOLE + (SCALAR ? 2 * CHUNK : SUBS * N);      // the two in the middle multiplied
    static constexpr int BETA = MIDDLE + (SCALAR ? 0 : N);
    static constexpr int OWN = BETA + CHUNK;                                    // (wkv) sum_i u_i k_i q_i; SCALAR: A(0, i]
    static constexpr int FLOATS = OWN + CHUNK;
};

template <int RULE, int N>
__global__ void __launch_bounds__(Layout<RULE, N>::THREADS, Layout<RULE, N>::BLOCKS) prepare_chunks_kernel(const Args a) {
    using P = Layout<RULE, N>;
    using Piece = Pieces<RULE, N>;
    constexpr bool DELTA = P::DELTA, SCALAR = P::SCALAR;
    constexpr int THREADS = P::THREADS, WARPS = THREADS / 32, LD = P::LD, WLD = P::WLD, TLD = P::TLD, ILD = P::ILD, VL = N / 32;
    extern __shared__ __align__(16) float memory[];
    float *ks = memory + P::KS, *qs = memory + P::QS, *as = memory + P::AS, *cs = memory + P::CS, *at = memory + P::AT, *inverse = memory + P::INVERSE, *whole = memory + P::WHOLE,
          *middle = memory + P::MIDDLE, *beta = memory + P::BETA, *own = memory + P::OWN;
    double* const decays = reinterpret_cast<double*>(whole);
    __shared__ int steep[SUBS];     // whether a sub-block's decays multiply up to less than STEEP somewhere
    const int chunk = a.chunk0 + blockIdx.x, head = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int first = a.chunks[2 * chunk], count = a.chunks[2 * chunk + 1];
    const int group = head / (a.heads / a.groups), c0 = lane * VL, live_c = a.n - c0;
    float* const piece = a.scratch + ((size_t)blockIdx.x * a.heads + head) * Piece::size(a.e);

    if (DELTA && threadIdx.x >= CHUNK) {
        for (int i = threadIdx.x - CHUNK; i < CHUNK * TLD; i += THREADS - CHUNK) at[i] = 0.f;
    } else if (threadIdx.x < CHUNK) {  // a token's gates by one thread
        const int j = threadIdx.x;
        const size_t t = first + (j < count ? j : 0);
        if (DELTA) beta[j] = j < count ? (float)(1.0 / (1.0 + exp(-(double)a.step[t * a.step_stride + a.step_off + head]))) : 0.f;
        if (RULE == RULE_DELTA) decays[j] = expf(-expf(a.rate[head]) * softplus_of(a.x[t * a.x_stride + a.x_off + head] + a.bias[head]));
        if (RULE == RULE_RETENTION) decays[j] = a.rate[head];
    }
    if (threadIdx.x < SUBS) steep[threadIdx.x] = 0;
    if (SCALAR) {
        __syncthreads();
        if (threadIdx.x <= CHUNK) {  // a column of the weights per thread; the last thread: those of the chunk's start
            const int j = (int)threadIdx.x < CHUNK ? (int)threadIdx.x : -1;
            double weight = 1.0;
            for (int i = j < 0 ? 0 : j; i < count; ++i) {
                if (i > j) weight *= decays[i];
                (j < 0 ? own[i] : as[i * WLD + j]) = (float)weight;
            }
        }
    }
    {
        const bool wide = a.by_four != 0;
        float fixed = 0.f, per_entry[VL], bonus[VL];
#pragma unroll
        for (int i = 0; i < VL; ++i) per_entry[i] = bonus[i] = 0.f;
        if (RULE == RULE_CHANNEL_DELTA) fixed = -expf(a.rate[head]);
        if (RULE == RULE_CHANNEL_DELTA) load_some<VL>(a.bias + (size_t)head * a.n + c0, live_c, false, 0.f, per_entry);
        if (RULE == RULE_WKV) {
            load_some<VL>(a.rate + (size_t)head * a.n + c0, live_c, false, 0.f, per_entry);
            load_some<VL>(a.bias + (size_t)head * a.n + c0, live_c, false, 0.f, bonus);
        }
        constexpr int AT_ONCE = 4;  // tokens a warp has on their way
#pragma unroll
        for (int base = 0; base < CHUNK / WARPS; base += AT_ONCE) {
            float k[AT_ONCE][VL], q[AT_ONCE][VL], x[AT_ONCE][VL];
#pragma unroll
            for (int u = 0; u < AT_ONCE; ++u) {
                const int j = warp + WARPS * (base + u), live = j < count ? live_c : 0;
                const size_t t = first + (j < count ? j : 0);
                load_some<VL>(a.k + t * a.k_stride + (size_t)group * a.n + c0, live, wide, 0.f, k[u]);
                load_some<VL>(a.q + t * a.q_stride + (size_t)group * a.n + c0, live, wide, 0.f, q[u]);
                if (!SCALAR) load_some<VL>(a.x + t * a.x_stride + a.x_off + (size_t)head * a.n + c0, live, wide, 0.f, x[u]);
            }
#pragma unroll
            for (int u = 0; u < AT_ONCE; ++u) {
                const int j = warp + WARPS * (base + u);
                const bool there = j < count;
                float ik = 1.f, iq = a.q_scale;
                if (DELTA) {  // keys and queries become unit vectors
                    float sum_k = 0.f, sum_q = 0.f;
#pragma unroll
                    for (int i = 0; i < VL; ++i) { sum_k = fmaf(k[u][i], k[u][i], sum_k); sum_q = fmaf(q[u][i], q[u][i], sum_q); }
                    ik = 1.0f / sqrtf(warp_sum(sum_k) + 1e-6f);
                    iq = a.q_scale / sqrtf(warp_sum(sum_q) + 1e-6f);
                }
                float decay[VL], bonus_dot = 0.f;
#pragma unroll
                for (int i = 0; i < VL; ++i) {
                    if (RULE == RULE_WKV) bonus_dot = fmaf(bonus[i] * k[u][i], q[u][i], bonus_dot);
                    k[u][i] *= ik;
                    q[u][i] *= iq;
                    float d = 1.f;
                    if (RULE == RULE_CHANNEL_DELTA) d = expf(fixed * softplus_of(x[u][i] + per_entry[i]));
                    if (RULE == RULE_WKV) d = expf(-expf(x[u][i] + per_entry[i]));
                    decay[i] = there && i < live_c ? d : 1.f;
                }
                store_some<VL>(ks + j * LD + c0, k[u]);
                store_some<VL>(qs + j * LD + c0, q[u]);
                if (!SCALAR) store_some<VL>(as + j * LD + c0, decay);
                if (RULE == RULE_WKV) {
                    bonus_dot = warp_sum(bonus_dot);
                    if (lane == 0) own[j] = bonus_dot;
                }
            }
        }
    }
    __syncthreads();

    if constexpr (!SCALAR) {
        for (int unit = threadIdx.x; unit < SUBS * N; unit += THREADS) {
            const int sub = unit / N, c = unit - sub * N;
            double product = 1.0;
#pragma unroll
            for (int i = 0; i < SUB; ++i) product *= as[(sub * SUB + i) * LD + c];
            if (!(product >= STEEP)) steep[sub] = 1;  // a NaN too: the pairs below reach forward only, whatever they hold
            whole[sub * N + c] = (float)product;
        }
        __syncthreads();
        for (int c = threadIdx.x; c < N; c += THREADS) middle[c] = whole[N + c] * whole[2 * N + c];

        // Pairs inside a steep sub-block, entry by entry in float: a key walks forward through the decays and meets every later row.  A sub-block's warps share its keys; with
        // a delta rule half of them take the keys' rows, the others the queries'.  (Taking every sub-block this way cost 17,000 of a block's 77,000 clocks.)
        {
            constexpr int SHARES = DELTA ? WARPS / 8 : WARPS / 4;
            const int sub = warp & 3, share = (warp >> 2) % SHARES;
            const bool of_keys = DELTA && (warp >> 2) < SHARES;
            const float* rows = of_keys ? ks : qs;
            if (sub * SUB < count && steep[sub]) {
#pragma unroll 1
                for (int j = share; j < SUB; j += SHARES) {
                    float w[VL], p[SUB];
                    read_some<VL>(ks + (sub * SUB + j) * LD + c0, w);
#pragma unroll
                    for (int i = 0; i < SUB; ++i) {
                        p[i] = 0.f;
                        if (i >= j) {
                            float x[VL], decay[VL];
                            read_some<VL>(rows + (sub * SUB + i) * LD + c0, x);
                            read_some<VL>(as + (sub * SUB + i) * LD + c0, decay);
                            if (RULE != RULE_WKV && i > j) {
#pragma unroll
                                for (int z = 0; z < VL; ++z) w[z] *= decay[z];
                            }
#pragma unroll
                            for (int z = 0; z < VL; ++z) p[i] = fmaf(w[z], x[z], p[i]);
                            if (RULE == RULE_WKV && i > j) {
#pragma unroll
                                for (int z = 0; z < VL; ++z) w[z] *= decay[z];
                            }
                        }
                    }
                    // sixteen sums over the warp's lanes: at every step a lane hands half of its sums to the lane across
#pragma unroll
                    for (int width = 8, offset = 16; width > 0; width >>= 1, offset >>= 1) {
                        const bool upper = lane & offset;
#pragma unroll
                        for (int m = 0; m < width; ++m) {
                            const float give = upper ? p[m] : p[m + width], keep = upper ? p[m + width] : p[m];
                            p[m] = keep + __shfl_xor_sync(0xffffffffu, give, offset);
                        }
                    }
                    const float sum = p[0] + __shfl_xor_sync(0xffffffffu, p[0], 1);
                    const int i = ((lane >> 4) & 1) * 8 + ((lane >> 3) & 1) * 4 + ((lane >> 2) & 1) * 2 + ((lane >> 1) & 1);
                    if ((lane & 1) == 0) {
                        const int row = sub * SUB + i, column = sub * SUB + j;
                        if (of_keys) {
                            at[column * TLD + row] = i > j ? beta[row] * sum : 0.f;
                        } else {
                            const float value = RULE == RULE_WKV && i == j ? own[row] : sum;
                            piece[Piece::B + row * Piece::BLD + column] = i >= j ? value : 0.f;
                        }
                    }
                }
            }
        }
        __syncthreads();

        // A thread takes an entry of a sub-block through its tokens: forward from the block's start for rows, backward from its end for columns.  In double: a float product's
        // sixteen roundings would be the largest error there is.
#pragma unroll
        for (int unit = threadIdx.x; unit < SUBS * N; unit += THREADS) {
            const int sub = unit / N, c = unit - sub * N;
            float decay[SUB], key[SUB];
            double passed = 1.0;
#pragma unroll
            for (int i = 0; i < SUB; ++i) {
                const int at_i = (sub * SUB + i) * LD + c;
                decay[i] = as[at_i];
                key[i] = ks[at_i];
                if (RULE != RULE_WKV) passed *= decay[i];
                qs[at_i] = (float)(qs[at_i] * passed);
                if (DELTA) ks[at_i] = (float)(key[i] * passed);
                if (RULE == RULE_WKV) passed *= decay[i];
            }
            const double back = 1.0 / passed;
            double left = 1.0;
#pragma unroll
            for (int i = SUB - 1; i >= 0; --i) {
                const double weighed = key[i] * left;
                as[(sub * SUB + i) * LD + c] = (float)weighed;
                cs[(sub * SUB + i) * LD + c] = (float)(weighed * back);
                left *= decay[i];
            }
        }
        __syncthreads();
    }

    // The pairs of two sub-blocks as a product: (row block, column block) times (keys' rows, queries' rows), a warp each.  SCALAR: weighed afterwards.  Otherwise columns carry the
    // decays behind them in their block, and those of blocks between come on top; inside one block, where a row's decays from the block's start on already hold the column's,
    // columns have them divided out.
    {
        const int g = lane >> 2, t = lane & 3;
        constexpr int PAIRS = SUBS * (SUBS + 1) / 2;
        for (int task = warp; task < (DELTA ? 2 * PAIRS : PAIRS); task += WARPS) {
            const int pair = task % PAIRS, r = pair < 1 ? 0 : (pair < 3 ? 1 : (pair < 6 ? 2 : 3)), b = pair - r * (r + 1) / 2;
            const bool keys = DELTA && task < PAIRS;
            if (r * SUB >= count || (!SCALAR && r == b && steep[r])) continue;
            const float* rows = (keys ? ks : qs) + (r * SUB + g) * LD + t;
            const float* columns = (SCALAR ? ks : (r == b ? cs : as)) + (b * SUB + g) * LD + t;
            const float* between = (r - b == 2 ? whole + (b + 1) * N : middle) + t;
            float acc[2][4] = {}, rest[2][4] = {};
            if (SCALAR || r - b < 2) {
#pragma unroll 2
                for (int kk = 0; kk < N; kk += 16) {
                    Thirds x[4];
                    row_thirds(x, rows + kk, 1, 8 * LD);
#pragma unroll
                    for (int z = 0; z < 2; ++z) multiply(acc[z], rest[z], x, columns + z * 8 * LD + kk, 1);
                }
            } else {
#pragma unroll 2
                for (int kk = 0; kk < N; kk += 16) {
                    Thirds x[4];
                    row_thirds(x, rows + kk, 1, 8 * LD);
                    const float f[4] = {between[kk], between[kk + 4], between[kk + 8], between[kk + 12]};
#pragma unroll
                    for (int z = 0; z < 2; ++z) {
                        const float* y = columns + z * 8 * LD + kk;
                        multiply(acc[z], rest[z], x, thirds(y[0] * f[0], y[8] * f[2]), thirds(y[4] * f[1], y[12] * f[3]));
                    }
                }
            }
#pragma unroll
            for (int z = 0; z < 2; ++z) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int row = r * SUB + g + 8 * (i >> 1), column = b * SUB + z * 8 + 2 * t + (i & 1);
                    float x = acc[z][i] + rest[z][i];
                    if (SCALAR && row < count && row >= column) x *= as[row * WLD + column];
                    if (keys) {
                        at[column * TLD + row] = row > column ? beta[row] * x : 0.f;
                    } else {
                        if (RULE == RULE_WKV && row == column) x = own[row];
                        piece[Piece::B + row * Piece::BLD + column] = row >= column ? x : 0.f;
                    }
                }
            }
        }
    }

    // What the walk takes from the chunk's keys and queries: queries with the decays from the chunk's start on, keys with those up to its end.
    const int live = min(CHUNK, (count + SUB - 1) & ~(SUB - 1));
    for (int unit = threadIdx.x; unit < live * (N / 4); unit += THREADS) {
        const int i = unit / (N / 4), c = (unit - i * (N / 4)) * 4, sub = i / SUB;
        float x[4], y[4];
        load4(qs + i * LD + c, x);
        load4((SCALAR ? ks : as) + i * LD + c, y);
        if (SCALAR) {
            const float since = i < count ? own[i] : 0.f, until = i < count ? as[(count - 1) * WLD + i] : 0.f;
#pragma unroll
            for (int z = 0; z < 4; ++z) x[z] *= since, y[z] *= until;
        } else {
            for (int m = 0; m < SUBS; ++m) {
                if (m == sub) continue;
                float f[4];
                load4(whole + m * N + c, f);
#pragma unroll
                for (int z = 0; z < 4; ++z) (m < sub ? x : y)[z] *= f[z];
            }
        }
        store4(piece + Piece::Q + i * Piece::QLD + c, x);
        store4(piece + Piece::K + i * Piece::KLD + c, y);
    }
    for (int c = threadIdx.x; c < N; c += THREADS)
        piece[Piece::FADE + c] = SCALAR ? (c < a.n ? own[count - 1] : 1.f) : whole[c] * whole[N + c] * whole[2 * N + c] * whole[3 * N + c];

    if constexpr (DELTA) {
        // (I + L) X = [b K | b V], L strictly lower, by sub-blocks of 16 rows: X_r = (I + L_rr)^-1 (rhs_r - sum_(m < r) L_rm X_m).  The inverses of the four diagonal blocks
        // are made in float by substitution, a column per lane, and taken to the rows in float too; the rest are products, in which a warp keeps to columns of its own.
        constexpr int XLD = P::XLD, WIDE = XLD - 8;
        float* xs = qs;  // [64][WIDE columns at a time], over what has been written out
        __syncthreads();  // a diagonal block of L may be another warp's pair
        if (warp < SUBS && lane < SUB) {
            const float* lower = at + warp * SUB * TLD + warp * SUB;
            float column[SUB];
#pragma unroll
            for (int i = 0; i < SUB; ++i) {
                float x = i == lane ? 1.f : 0.f;
#pragma unroll
                for (int m = 0; m < i; ++m) x = fmaf(-lower[m * TLD + i], column[m], x);
                column[i] = x;
                inverse[(warp * SUB + i) * ILD + lane] = x;
            }
        }
        const int g = lane >> 2, t = lane & 3;
        for (int col0 = 0; col0 < N + a.e; col0 += WIDE) {
            const int columns = min(WIDE, N + a.e - col0);
            __syncthreads();  // queries and keys, or the columns before, have been written out
            {  // a thread keeps to four columns and takes every few rows of them
                const int quads = columns / 4, quad = threadIdx.x % quads, stride = THREADS / quads, column = col0 + quad * 4;
                constexpr int AT_ONCE = 8;
                for (int base = threadIdx.x / quads; base < live; base += AT_ONCE * stride) {
                    if (threadIdx.x >= stride * quads) break;
                    float x[AT_ONCE][4];
#pragma unroll
                    for (int u = 0; u < AT_ONCE; ++u) {
                        const int i = base + u * stride;
                        x[u][0] = x[u][1] = x[u][2] = x[u][3] = 0.f;
                        if (i >= live) continue;
                        if (column < N) load4(ks + i * LD + column, x[u]);
                        else if (i < count) load_some<4>(a.v + (size_t)(first + i) * a.v_stride + (size_t)head * a.e + (column - N), 4, a.v_by_four != 0, 0.f, x[u]);
                    }
#pragma unroll
                    for (int u = 0; u < AT_ONCE; ++u) {
                        const int i = base + u * stride;
                        if (i >= live) continue;
                        const float b = beta[i];
#pragma unroll
                        for (int z = 0; z < 4; ++z) x[u][z] *= b;
                        if (column < N) {
                            if (SCALAR) {
                                const float since = i < count ? own[i] : 0.f;
#pragma unroll
                                for (int z = 0; z < 4; ++z) x[u][z] *= since;
                            } else {
                                for (int m = 0; m < i / SUB; ++m) {
                                    float f[4];
                                    load4(whole + m * N + column, f);
#pragma unroll
                                    for (int z = 0; z < 4; ++z) x[u][z] *= f[z];
                                }
                            }
                        }
                        store4(xs + i * XLD + quad * 4, x[u]);
                    }
                }
            }
            __syncthreads();
            constexpr int T = WIDE / 8 / WARPS;  // tiles of eight columns to a warp
            const int n0 = warp * (T * 8), tiles = min(T, (columns - n0) / 8);
            if (tiles > 0) {
#pragma unroll 1
                for (int r = 0; r * SUB < live; ++r) {
                    float acc[T][4] = {}, rest[T][4] = {};
#pragma unroll 1
                    for (int kk = 0; kk < r * SUB; kk += 16) {
                        Thirds x[4];
                        row_thirds(x, at + (kk + t) * TLD + r * SUB + g, TLD, 8);
#pragma unroll
                        for (int z = 0; z < T; ++z)
                            if (z < tiles) multiply(acc[z], rest[z], x, xs + (kk + t) * XLD + n0 + z * 8 + g, XLD);
                    }
                    float* mine = xs + (r * SUB + g) * XLD + n0 + 2 * t;
#pragma unroll
                    for (int z = 0; z < T; ++z) {
                        if (z >= tiles) continue;
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            float2* at_row = reinterpret_cast<float2*>(mine + 8 * h * XLD + z * 8);
                            const float2 x = *at_row;
                            *at_row = make_float2(x.x - (acc[z][2 * h] + rest[z][2 * h]), x.y - (acc[z][2 * h + 1] + rest[z][2 * h + 1]));
                            acc[z][2 * h] = acc[z][2 * h + 1] = 0.f;
                        }
                    }
                    __syncwarp();
#pragma unroll 5
                    for (int j = 0; j < SUB - 1; ++j) {
                        const float x0 = inverse[(r * SUB + g) * ILD + j], x1 = inverse[(r * SUB + g + 8) * ILD + j];
#pragma unroll
                        for (int z = 0; z < T; ++z) {
                            if (z >= tiles) continue;
                            const float2 y = *reinterpret_cast<const float2*>(xs + (r * SUB + j) * XLD + n0 + z * 8 + 2 * t);
                            if (j < g) acc[z][0] = fmaf(x0, y.x, acc[z][0]), acc[z][1] = fmaf(x0, y.y, acc[z][1]);  // a row takes nothing from later ones, whatever they hold
                            if (j < g + 8) acc[z][2] = fmaf(x1, y.x, acc[z][2]), acc[z][3] = fmaf(x1, y.y, acc[z][3]);
                        }
                    }
                    __syncwarp();
#pragma unroll
                    for (int z = 0; z < T; ++z) {
                        if (z >= tiles) continue;
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            float2* at_row = reinterpret_cast<float2*>(mine + 8 * h * XLD + z * 8);
                            const float2 x = *at_row;
                            *at_row = make_float2(x.x + acc[z][2 * h], x.y + acc[z][2 * h + 1]);
                        }
                    }
                    __syncwarp();
                }
            }
            __syncthreads();
            for (int unit = threadIdx.x; unit < live * (columns / 4); unit += THREADS) {
                const int i = unit / (columns / 4), c = (unit - i * (columns / 4)) * 4, column = col0 + c;
                float x[4];
                load4(xs + i * XLD + c, x);
                store4(column < N ? piece + Piece::W + i * Piece::QLD + column : piece + Piece::u(a.e) + (size_t)i * a.e + (column - N), x);
            }
        }
    }
}

// ---------------------------------------------------------------- the state through a row's chunks: grid (value column tiles, heads, rows that are walked)
// Warps 0 .. 3: u of sixteen tokens each; 0 .. 7: the state, sixteen entries each; 8 .. 11: outputs of sixteen tokens each, beside the state's.
constexpr int WALK_THREADS = 384;
constexpr unsigned WAIT_LIMIT = 1u << 24;
__device__ __forceinline__ uint32_t shared_address(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void expect_bytes(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(shared_address(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_ahead(float* to, const float* from, unsigned bytes, unsigned long long* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(shared_address(to)), "l"(from), "r"(bytes),
                 "r"(shared_address(bar))
                 : "memory");
}
__device__ __forceinline__ void wait_for(unsigned long long* bar, unsigned parity, volatile int* failed) {
    for (unsigned spin = 0; spin < WAIT_LIMIT; ++spin) {
        unsigned done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(shared_address(bar)), "r"(parity) : "memory");
        if (done) return;
        if ((spin & 1023) == 1023 && *failed) return;
    }
    *failed = 1;
}

template <int RULE, int N, int ETILE>
constexpr int walk_bytes() {
    return ((is_delta(RULE) ? 2 : 1) * CHUNK * (N + 4) + CHUNK * (N + 8) + CHUNK * (CHUNK + 4) + (3 * N / 2 + CHUNK + 3 * CHUNK / 2) * (ETILE + 8)) * 4;
}

template <int RULE, int N, int ETILE>
__global__ void __launch_bounds__(WALK_THREADS) walk_chunks_kernel(const Args a) {
    constexpr bool DELTA = is_delta(RULE);
    using Piece = Pieces<RULE, N>;
    constexpr int LD = Piece::QLD, KLD = Piece::KLD, BLD = Piece::BLD, SLD = ETILE + 8, TILES = ETILE / 8;
    constexpr int SPLANE = N / 2 * SLD, UPLANE = CHUNK / 2 * SLD;
    extern __shared__ __align__(16) float memory[];
    __shared__ __align__(8) unsigned long long rows_there, columns_there;
    __shared__ int failed;
    float* qs = memory;                             // [64][N]: queries
    float* ws = qs + CHUNK * LD;                    // (delta) [64][N]
    float* ks = ws + (DELTA ? CHUNK * LD : 0);      // [64][N]: keys
    float* bs = ks + CHUNK * KLD;                   // [64][64]
    // a state's and u's thirds are made once, by the warp that has them: entry c and c + 8 of sixteen in a word, as the fragments of all warps take them
    uint32_t* ss = reinterpret_cast<uint32_t*>(bs + CHUNK * BLD);  // three of [N / 2][ETILE]: the state at the chunk's start
    uint32_t* uts = ss + 3 * SPLANE;                // three of [32][ETILE]: u
    float* us = reinterpret_cast<float*>(uts + 3 * UPLANE);  // [64][ETILE]: u as it is
    const int head = blockIdx.y, e0 = blockIdx.x * ETILE;
    const int* walk = a.walks + 3 * blockIdx.z;
    const int from = max(walk[0], a.chunk0), to = min(walk[1], a.chunk1);
    if (from >= to) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const bool keeps = warp < 8 && warp * 16 < N;  // this warp owns the state's entries 16 warp .. + 15
    const int channel = warp * 16 + g;
    float* const kept = a.state + (size_t)a.slots[walk[2]] * a.slot_stride + a.state_off + ((size_t)head * a.e + e0) * a.n_padded;

    auto piece_of = [&](int chunk) { return a.scratch + ((size_t)(chunk - a.chunk0) * a.heads + head) * Piece::size(a.e); };
    auto live_of = [&](int chunk) { return min(CHUNK, (a.chunks[2 * chunk + 1] + SUB - 1) & ~(SUB - 1)); };
    // one thread asks for a chunk's matrices; every thread waits for them
    auto fetch_rows = [&](int chunk, int live) {
        if (threadIdx.x) return;
        const float* p = piece_of(chunk);
        const unsigned bytes = live * LD * 4;
        expect_bytes(&rows_there, (DELTA ? 2 : 1) * bytes);
        copy_ahead(qs, p + Piece::Q, bytes, &rows_there);
        if (DELTA) copy_ahead(ws, p + Piece::W, bytes, &rows_there);
    };
    auto fetch_columns = [&](int chunk, int live) {
        if (threadIdx.x) return;
        const float* p = piece_of(chunk);
        expect_bytes(&columns_there, live * (KLD + BLD) * 4);
        copy_ahead(ks, p + Piece::K, live * KLD * 4, &columns_there);
        copy_ahead(bs, p + Piece::B, live * BLD * 4, &columns_there);
    };

    if (threadIdx.x == 0) {
        failed = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(shared_address(&rows_there)));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(shared_address(&columns_there)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    int live = live_of(from);
    fetch_rows(from, live);
    fetch_columns(from, live);
    float s[TILES][4] = {};
    auto show_state = [&](int z) { store_thirds(ss + (warp * 8 + g) * SLD + z * 8 + 2 * t, SPLANE, thirds(s[z][0], s[z][2]), thirds(s[z][1], s[z][3])); };
    if (keeps) {
#pragma unroll
        for (int z = 0; z < TILES; ++z) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int c = channel + (i >> 1) * 8, column = z * 8 + 2 * t + (i & 1);
                s[z][i] = c < a.n ? kept[(size_t)column * a.n_padded + c] : 0.f;
            }
            show_state(z);
        }
    }
    __syncthreads();  // the state at the first chunk's start is there
    unsigned parity = 0;

    for (int chunk = from; chunk < to; ++chunk) {
        const int first = a.chunks[2 * chunk], count = a.chunks[2 * chunk + 1];
        const float* piece = piece_of(chunk);
        const int row0 = (warp & 3) * 16;
        const bool active = row0 < live;
        float given[TILES][4], fade[2] = {1.f, 1.f};  // asked for before anything is waited for
        if (warp < 4 && active) {
#pragma unroll
            for (int z = 0; z < TILES; ++z)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int i = row0 + g + 8 * h, column = e0 + z * 8 + 2 * t;
                    if (DELTA) {
                        const float2 y = *reinterpret_cast<const float2*>(piece + Piece::u(a.e) + (size_t)i * a.e + column);
                        given[z][2 * h] = y.x, given[z][2 * h + 1] = y.y;
                    } else {
                        const float* v = a.v + (size_t)(first + i) * a.v_stride + (size_t)head * a.e + column;
                        given[z][2 * h] = i < count ? v[0] : 0.f, given[z][2 * h + 1] = i < count ? v[1] : 0.f;
                    }
                }
        }
        if (keeps) {
            fade[0] = piece[Piece::FADE + channel];
            fade[1] = piece[Piece::FADE + channel + 8];
        }
        wait_for(&rows_there, parity, &failed);

        float o[TILES][4] = {}, rest[TILES][4] = {};
        if (active && (warp >= 8 || (DELTA && warp < 4))) {
            const float* rows = (warp < 4 ? ws : qs) + (row0 + g) * LD + t;
#pragma unroll 2
            for (int kk = 0; kk < N; kk += 16) {
                Thirds x[4];
                row_thirds(x, rows + kk, 1, 8 * LD);
#pragma unroll
                for (int z = 0; z < TILES; ++z) {
                    const uint32_t* y = ss + (kk / 2 + t) * SLD + z * 8 + g;
                    multiply(o[z], rest[z], x, stored_thirds(y, SPLANE), stored_thirds(y + 4 * SLD, SPLANE));
                }
            }
        }
        if (warp < 4 && active) {
#pragma unroll
            for (int z = 0; z < TILES; ++z) {
                float u[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) u[i] = DELTA ? given[z][i] - (o[z][i] + rest[z][i]) : given[z][i];
                float* at = us + (row0 + g) * SLD + z * 8 + 2 * t;
                *reinterpret_cast<float2*>(at) = make_float2(u[0], u[1]);
                *reinterpret_cast<float2*>(at + 8 * SLD) = make_float2(u[2], u[3]);
                store_thirds(uts + (row0 / 2 + g) * SLD + z * 8 + 2 * t, UPLANE, thirds(u[0], u[2]), thirds(u[1], u[3]));
            }
        }
        wait_for(&columns_there, parity, &failed);
        parity ^= 1;
        __syncthreads();  // u and this chunk's columns are there, its rows have been read
        const bool more = chunk + 1 < to;
        const int next_live = more ? live_of(chunk + 1) : 0;
        if (more) fetch_rows(chunk + 1, next_live);

        // Earlier blocks of sixteen tokens on the tensor cores; a row's own block, and the chunk's last one for the state, token by token in float: what weighs most is rounded as
        // a scan rounds it, and a token gets nothing from later ones, whatever they hold.
        if (keeps) {
            float sum[TILES][4] = {}, small[TILES][4] = {};
            const int before = live - SUB;
#pragma unroll 1
            for (int kk = 0; kk < before; kk += 16) {
                Thirds y[4];
                row_thirds(y, ks + (kk + t) * KLD + channel, KLD, 8);
#pragma unroll
                for (int z = 0; z < TILES; ++z) {
                    const uint32_t* u = uts + (kk / 2 + t) * SLD + z * 8 + g;
                    multiply(sum[z], small[z], y, stored_thirds(u, UPLANE), stored_thirds(u + 4 * SLD, UPLANE));
                }
            }
#pragma unroll
            for (int z = 0; z < TILES; ++z)
#pragma unroll
                for (int i = 0; i < 4; ++i) s[z][i] = fmaf(fade[i >> 1], s[z][i], sum[z][i] + small[z][i]);
#pragma unroll 4
            for (int j = before; j < count; ++j) {
                const float k0 = ks[j * KLD + channel], k1 = ks[j * KLD + channel + 8];
#pragma unroll
                for (int z = 0; z < TILES; ++z) {
                    const float2 u = *reinterpret_cast<const float2*>(us + j * SLD + z * 8 + 2 * t);
                    s[z][0] = fmaf(k0, u.x, s[z][0]), s[z][1] = fmaf(k0, u.y, s[z][1]);
                    s[z][2] = fmaf(k1, u.x, s[z][2]), s[z][3] = fmaf(k1, u.y, s[z][3]);
                }
            }
#pragma unroll
            for (int z = 0; z < TILES; ++z) show_state(z);
        }
        if (warp >= 8 && active) {
            const float* rows = bs + (row0 + g) * BLD + t;
#pragma unroll 1
            for (int kk = 0; kk < row0; kk += 16) {
                Thirds x[4];
                row_thirds(x, rows + kk, 1, 8 * BLD);
#pragma unroll
                for (int z = 0; z < TILES; ++z) {
                    const uint32_t* u = uts + (kk / 2 + t) * SLD + z * 8 + g;
                    multiply(o[z], rest[z], x, stored_thirds(u, UPLANE), stored_thirds(u + 4 * SLD, UPLANE));
                }
            }
#pragma unroll
            for (int z = 0; z < TILES; ++z)
#pragma unroll
                for (int i = 0; i < 4; ++i) o[z][i] += rest[z][i];
#pragma unroll 4
            for (int j = 0; j < SUB; ++j) {
                const float w0 = bs[(row0 + g) * BLD + row0 + j], w1 = bs[(row0 + g + 8) * BLD + row0 + j];
#pragma unroll
                for (int z = 0; z < TILES; ++z) {
                    const float2 u = *reinterpret_cast<const float2*>(us + (row0 + j) * SLD + z * 8 + 2 * t);
                    if (j <= g) o[z][0] = fmaf(w0, u.x, o[z][0]), o[z][1] = fmaf(w0, u.y, o[z][1]);
                    if (j <= g + 8) o[z][2] = fmaf(w1, u.x, o[z][2]), o[z][3] = fmaf(w1, u.y, o[z][3]);
                }
            }
#pragma unroll
            for (int z = 0; z < TILES; ++z)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int i = row0 + g + 8 * h;
                    if (i < count)
                        *reinterpret_cast<float2*>(a.out + ((size_t)(first + i) * a.heads + head) * a.e + e0 + z * 8 + 2 * t) = make_float2(o[z][2 * h], o[z][2 * h + 1]);
                }
        }
        __syncthreads();  // the columns and u have been read, the next state is there
        if (more) fetch_columns(chunk + 1, next_live);
        live = next_live;
    }
    if (threadIdx.x == 0 && failed) atomicOr(a.status, HB_STATUS_WAIT_EXPIRED | HB_STATUS_IN_CHUNKED_WALK);
    if (keeps) {
#pragma unroll
        for (int z = 0; z < TILES; ++z)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int c = channel + (i >> 1) * 8;
                if (c < a.n) kept[(size_t)(z * 8 + 2 * t + (i & 1)) * a.n_padded + c] = s[z][i];
            }
    }
}

template <typename Kernel>
int allow_shared(Kernel kernel, int bytes) {
    return bytes > 48 * 1024 ? (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) : 0;
}

template <int RULE, int N, int ETILE>
int launch_walk(const Args& a, int walks, cudaStream_t stream) {
    constexpr int bytes = walk_bytes<RULE, N, ETILE>();
    const int status = allow_shared(walk_chunks_kernel<RULE, N, ETILE>, bytes);
    if (status) return status;
    walk_chunks_kernel<RULE, N, ETILE><<<dim3(a.e / ETILE, a.heads, walks), WALK_THREADS, bytes, stream>>>(a);
    return launch_status();
}

template <int RULE, int N>
int launch_rule(const Args& given, int walks, int beside, int chunks, int span, int sms, cudaStream_t stream) {
    constexpr int bytes = Layout<RULE, N>::FLOATS * 4;
    int status = allow_shared(prepare_chunks_kernel<RULE, N>, bytes);
    if (status) return status;
    for (int at = 0; at < chunks; at += span) {  // the scratch of a span is used again by the next one
        Args a = given;
        a.chunk0 = at;
        a.chunk1 = at + span < chunks ? at + span : chunks;
        prepare_chunks_kernel<RULE, N><<<dim3(a.chunk1 - a.chunk0, a.heads), Layout<RULE, N>::THREADS, bytes, stream>>>(a);
        status = launch_status();
        if (status) return status;
        // 16 value columns to a block while those blocks, of all rows side by side, fit the SMs, else 32, which read the chunk's pieces half as often (16 heads of 128 x 128, four
        // rows of 2,048: delta rule 753 us, 882 with 16 columns; retention 473 and 559)
        const bool narrow = a.e % 32 != 0 || (long long)beside * a.heads * (a.e / 16) <= sms;
        status = narrow ? launch_walk<RULE, N, 16>(a, walks, stream) : launch_walk<RULE, N, 32>(a, walks, stream);
        if (status) return status;
    }
    return 0;
}

template <int RULE>
size_t piece_floats(int n, int e) {
    return n <= 64 ? Pieces<RULE, 64>::size(e) : Pieces<RULE, 128>::size(e);
}
}  // namespace

// Floats of scratch that one chunk of one head takes (0: sizes the chunks do not take).
HB_EXPORT long long hb_chunked_float_scratch(int rule, int n, int e) {
    if (n <= 0 || n > 128 || e <= 0 || e % 16) return 0;
    switch (rule) {
        case RULE_DELTA: return (long long)piece_floats<RULE_DELTA>(n, e);
        case RULE_CHANNEL_DELTA: return (long long)piece_floats<RULE_CHANNEL_DELTA>(n, e);
        case RULE_RETENTION: return (long long)piece_floats<RULE_RETENTION>(n, e);
        case RULE_WKV: return (long long)piece_floats<RULE_WKV>(n, e);
    }
    return 0;
}

// Rows through their chunks of at most 64 consecutive tokens (tables as in Args; a row's chunks follow one another), `span` chunks at a time: scratch holds span * heads times
// what hb_chunked_float_scratch says, on a 16-byte boundary.  beside: how many rows of the longest one's length the walks amount to.  out [tokens, heads * e] on an 8-byte boundary; tokens of no chunk keep theirs.
HB_EXPORT int hb_chunked_float(int rule, const float* k, int k_stride, const float* q, int q_stride, const float* v, int v_stride, const float* x, int x_stride, int x_off,
                               const float* step, int step_stride, int step_off, const float* rate, const float* bias, float* scratch, float* state, long long slot_stride,
                               int state_off, const int* slots, const int* table, int chunks, const int* walk_table, int walks, int beside, int span, float* out, int heads, int groups, int n,
                               int n_padded, int e, float q_scale, int sms, int* status, cudaStream_t stream) {
    if (chunks <= 0 || walks <= 0) return 0;
    if (n <= 0 || n > 128 || e <= 0 || e % 16 || heads <= 0 || heads > 65535 || walks > 65535 || groups <= 0 || heads % groups) return HB_UNSUPPORTED_SIZE;
    if (n_padded < n || span <= 0 || !k || !q || !v || !rate || !scratch || !state || !slots || !table || !walk_table || !out || !status) return HB_BAD_ARGUMENT;
    if ((((uintptr_t)scratch) & 15) || (((uintptr_t)out) & 7)) return HB_BAD_ARGUMENT;
    if (rule != RULE_RETENTION && (!x || !bias)) return HB_BAD_ARGUMENT;
    if ((rule == RULE_DELTA || rule == RULE_CHANNEL_DELTA) && !step) return HB_BAD_ARGUMENT;
    const bool vector = rule == RULE_CHANNEL_DELTA || rule == RULE_WKV;
    const int by_four = ((k_stride | q_stride | n | (vector ? x_stride | x_off : 0)) & 3) == 0 && (((uintptr_t)k | (uintptr_t)q | (vector ? (uintptr_t)x : 0)) & 15) == 0;
    const Args a{k, q, v, k_stride, q_stride, v_stride, x, x_stride, x_off, step, step_stride, step_off, rate, bias, scratch, state, (size_t)slot_stride, state_off, slots, table,
                 walk_table, 0, 0, out, heads, groups, n, n_padded, e, q_scale, by_four, (v_stride & 3) == 0 && ((uintptr_t)v & 15) == 0, status};
    const bool small = n <= 64;
    switch (rule) {
        case RULE_DELTA: return small ? launch_rule<RULE_DELTA, 64>(a, walks, beside, chunks, span, sms, stream) : launch_rule<RULE_DELTA, 128>(a, walks, beside, chunks, span, sms, stream);
        case RULE_CHANNEL_DELTA:
            return small ? launch_rule<RULE_CHANNEL_DELTA, 64>(a, walks, beside, chunks, span, sms, stream) : launch_rule<RULE_CHANNEL_DELTA, 128>(a, walks, beside, chunks, span, sms, stream);
        case RULE_RETENTION: return small ? launch_rule<RULE_RETENTION, 64>(a, walks, beside, chunks, span, sms, stream) : launch_rule<RULE_RETENTION, 128>(a, walks, beside, chunks, span, sms, stream);
        case RULE_WKV: return small ? launch_rule<RULE_WKV, 64>(a, walks, beside, chunks, span, sms, stream) : launch_rule<RULE_WKV, 128>(a, walks, beside, chunks, span, sms, stream);
    }
    return HB_BAD_ARGUMENT;
}
