// The attention of attention_chunk.cu (32-bit scores and weights, `Sight`) for prompt portions of
// bfloat16 rows of D = 64 or 128 features, on the 5th-generation tensor cores: tcgen05.mma with
// accumulators in tensor memory, keys and values by TMA.
//
// A block takes 128 rows (token, query head of the group) of one sequence and one kv head and walks
// the tiles of 64 keys that any of them sees; two blocks an SM, so that one's products run beside the
// other's exponentials.  Two threads share a row, each half of a tile's keys and half of the
// row's output features (warps w and w + 4 hold the same lanes of tensor memory).  Warp 3 fetches pages
// and warp 7 issues the products beside that: a warp more would leave a thread 96 registers instead of
// 128.  A tile: s = q k^T into 64 columns of tensor memory for
// either half of the features (added in float32: one sum over all of them is cut off at every
// product, 2.1e-7 from 64 bits in the results instead of 1.5e-7); scale, penalty, cap, mask and maximum
// in registers; the weights over the scores' columns as three bfloat16 terms (each the upper half of what
// the ones before it leave: their sum is the float32 weight), 32 columns each; three products with the
// values, the small terms first, into columns of the tile's own.  The sums over tiles are float32
// multiply-adds in registers (acc <- acc * correction + tile's share), so that what the tensor cores add
// up is a tile's share only.
//
// Nothing loses precision against the kernels on mma.sync: products of bfloat16 operands are exact,
// a weight has its 24 bits.  exp(score - maximum) is 2^(v U - M), one multiply-add and ex2.approx, with
// M the rounded product of the maximum with U: M is the same in all weights of a row, so its rounding
// leaves their ratios alone.  A row's tiles lie at absolute multiples of 64: its result does not
// depend on what shares its block or step.  Rows in which a product met an infinity or NaN are formed
// again on the CUDA cores once everything is stored.
//
// The pair of blocks: an item's tiles go by the parity of their place to two blocks of a cluster, which
// exchange half of the features each through distributed shared memory at the end.  A pair alone on the
// GPU takes 4.2 us a tile and block at 128 features (8,000 cycles: two products' latencies and some 800
// instructions a warp between them at two to four warps a scheduler) and 2.5 at 64, which is what bounds
// it: the longest rows' tiles one after the other.  On a full GPU an instruction is issued in 24 to 29 %
// of the cycles, the tensor cores are at work in 13 to 15 %.  Measured (us; mma.sync in tiles of 64 rows, one block a
// row tile, pairs): 2,048 tokens of 16 heads of 128 on 4 kv heads 213, 114, 88; under a window of
// 1,024 and a cap 156, 92, 96; prompts of 1,201 and 1,172 tokens 153, 100, 84; with distance slopes
// 158, 139, 98; heads of 64 135, 86, 65.  Four threads a row instead of two: 134 instead of 114.
//
// Every wait is bounded (status 3).  A thread whose wait ran out waits for nothing more but goes on to
// the end; the issuer then issues nothing more, so that no other wait for it succeeds either and the
// fetcher overwrites nothing.  The copies and products in flight are waited for, neither block of the
// pair stores a result, and the tensor memory is freed.

#include <cuda.h>

#include <atomic>

#include "attention_sight.cuh"
#include "tcgen05_common.cuh"
#include "tensor_maps.cuh"

DE_DEFINE_PDL_SWITCH

#ifndef ROLE_SPINS                     // how often a wait of the tiles' loop looks before it gives up
#define ROLE_SPINS tc5::SPIN_LIMIT
#endif

namespace {

using namespace tc5;

constexpr int UROWS = 128;             // rows of an item = lanes of tensor memory
constexpr int UKT = 64;                // keys of a tile
constexpr int UTHREADS = 256;
constexpr int FETCHER = 3, ISSUER = 7; // warps
constexpr int UCOLS = 256;             // columns of tensor memory of a block
constexpr int P_TERM = 32;             // columns of a term of the weights
constexpr int S_HALF = 64;             // columns of half a score, of one half of the features
constexpr int O_COL = 128;             // the tile's share of the results begins here

template <int D> struct Umma {
    static constexpr int KS = D / 64;                        // 64-feature sub-tiles of a row
    static constexpr int STAGES = D == 64 ? 3 : 2;
    static constexpr int SUB_Q = UROWS * 128, SUB_KV = UKT * 128;   // bytes of a sub-tile
    static constexpr int SMEM = KS * SUB_Q + STAGES * 2 * KS * SUB_KV + 2 * UROWS * 4 + 256;
};

__device__ __forceinline__ void umma_a_tmem(unsigned d, unsigned a, unsigned long long b_desc,
                                            unsigned idesc, bool accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.u32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
        "}\n"
        ::"r"(d), "r"(a), "l"(b_desc), "r"(idesc), "r"((unsigned)accumulate) : "memory");
}
__device__ __forceinline__ void tmem_load_16cols(unsigned taddr, unsigned (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15])
        : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_store_8cols(unsigned taddr, const unsigned (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]),
                   "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void before_sync() {
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
}
__device__ __forceinline__ void after_sync() {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
}
__device__ __forceinline__ float exp2_fast(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ unsigned upper_halves(float lo, float hi) {
    return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632);
}
// The pair of blocks (a cluster of two): the barrier that every thread of both reaches, the address of
// `mine`'s counterpart in block `rank`, and stores there.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ unsigned peer_address(const void* mine, int rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(smem_u32(mine)), "r"(rank));
    return r;
}
__device__ __forceinline__ void store_peer(unsigned at, unsigned v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;\n" ::"r"(at), "r"(v) : "memory");
}
__device__ __forceinline__ void store_peer(unsigned at, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;\n" ::"r"(at), "f"(v) : "memory");
}
__device__ __forceinline__ void store_peer(unsigned at, unsigned long long a, unsigned long long b) {
    asm volatile("st.shared::cluster.v2.b64 [%0], {%1, %2};\n" ::"r"(at), "l"(a), "l"(b) : "memory");
}

// two IEEE operations in one instruction
typedef unsigned long long Two;
__device__ __forceinline__ Two two(float a, float b) {
    Two r;
    asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void untwo(Two v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;\n" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ Two fma_two(Two a, Two b, Two c) {
    Two r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ Two mul_two(Two a, Two b) {
    Two r;
    asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ Two add_two(Two a, Two b) {
    Two r;
    asm("add.rn.f32x2 %0, %1, %2;\n" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// as tanh_near
__device__ __forceinline__ Two tanh_near_two(Two x) {
    const Two u = mul_two(x, x);
    Two p = fma_two(u, two(-0.00589515036f, -0.00589515036f), two(0.0207959637f, 0.0207959637f));
    p = fma_two(u, p, two(-0.0537838265f, -0.0537838265f));
    p = fma_two(u, p, two(0.133319244f, 0.133319244f));
    p = fma_two(u, p, two(-0.333332986f, -0.333332986f));
    return fma_two(mul_two(x, u), p, x);
}
// minus the upper half of x >= 0
__device__ __forceinline__ float minus_upper(float x) {
    return __uint_as_float((__float_as_uint(x) & 0xffff0000u) | 0x80000000u);
}
// kind::f16, bfloat16 operands, a K-major, b MN-major (the values as the cache holds them)
__host__ __device__ constexpr unsigned idesc_pv(int n) { return instr_desc(128, n) | (1u << 16); }

// FORM 0: no cap, no penalty, scale > 0: the weights follow from the products as they are.  1: a cap,
// no penalty.  2: everything `Sight` can say.
template <int D, int FORM>
__global__ void __launch_bounds__(UTHREADS, 2)
attn_chunk_tcgen05_kernel(const __nv_bfloat16* __restrict__ q, int q_stride, void* __restrict__ out,
                          int out_stride, const __grid_constant__ CUtensorMap map_k,
                          const __grid_constant__ CUtensorMap map_v,
                          const __nv_bfloat16* __restrict__ k_pages,
                          const __nv_bfloat16* __restrict__ v_pages,
                          const int* __restrict__ block_table, int table_stride, int num_pages,
                          const int* __restrict__ seq_slot, const int* __restrict__ seq_qstart,
                          const int* __restrict__ seq_qlen, const int* __restrict__ seq_pos0,
                          const WorkItem* __restrict__ items, const float* __restrict__ r1,
                          const float* __restrict__ r2, int heads, int kv_heads, int page, int box,
                          float scale, Sight sight, const float* __restrict__ fv, int out_f32,
                          int* __restrict__ status) {
    using U = Umma<D>;
    constexpr int KS = U::KS, STAGES = U::STAGES, HD = D / 2;   // HD: output features of a thread
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* q_s = smem_raw;                              // [KS] sub-tiles of 128 rows
    unsigned char* k_s = q_s + KS * U::SUB_Q;                   // [STAGES][KS] sub-tiles of 64 keys
    unsigned char* v_s = k_s + STAGES * KS * U::SUB_KV;
    float* share_s = reinterpret_cast<float*>(v_s + STAGES * KS * U::SUB_KV);   // [2][128]
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(share_s + 2 * UROWS);
    unsigned long long* kv_full = bars;                         // [STAGES] a tile's pages have landed
    unsigned long long* s_done = bars + STAGES;                 // a tile's scores are complete
    unsigned long long* p_ready = bars + STAGES + 1;            // its weights are written (every thread arrives)
    unsigned long long* o_done = bars + STAGES + 2;             // its share of the results is complete
    unsigned long long* drained = bars + STAGES + 3;            // the products of an issuer that gave up
    unsigned* gone_s = reinterpret_cast<unsigned*>(bars + STAGES + 4);   // [STAGES] boxes without a page
    unsigned* spoilt_s = gone_s + STAGES;                       // [8]
    unsigned* tmem_slot = spoilt_s + 8;
    volatile unsigned* gave_up_s = tmem_slot + 1;               // a wait of the pair ran out

    const int rank = blockIdx.x & 1;                            // in its pair of blocks
    const WorkItem it = items[(blockIdx.x >> 1) / kv_heads];
    if (it.kv_begin >= it.kv_end || (smem_u32(smem_raw) & 1023u) != 0) {
        if ((smem_u32(smem_raw) & 1023u) != 0 && threadIdx.x == 0) atomicExch(status, 4);
        pdl_wait();
        return;
    }
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int half = warp >> 2;
    const int rowi = (warp & 3) * 32 + lane;
    const int hk = (int)(blockIdx.x >> 1) % kv_heads;
    const int g = heads / kv_heads;
    const int qlen = seq_qlen[it.seq], pos0 = seq_pos0[it.seq];
    const int slot = seq_slot[it.seq], tok0 = seq_qstart[it.seq];
    const int rows_total = qlen * g;

    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < STAGES; ++i) mbar_init(&kv_full[i], 1);
        mbar_init(s_done, 1);
        mbar_init(p_ready, UTHREADS);
        mbar_init(o_done, 1);
        mbar_init(drained, 1);
        *gave_up_s = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == ISSUER) tmem_alloc(tmem_slot, UCOLS);

    // The keys that any row sees: [0, k_first) and [k_lo, k_hi).  Of the tiles that hold them the block
    // takes those whose place, key / 64, has its rank's parity: tile t of the block begins at key
    // tile_at(t).
    const int last_row = min(it.row0 + UROWS, rows_total) - 1;
    const int k_hi = min(it.kv_end, pos0 + last_row / g + 1);
    const int k_lo = max(it.kv_begin, sight_lo(sight, pos0 + it.row0 / g));
    const int k_first = it.kv_begin > 0 ? 0 : sight_first(sight, k_lo);
    const TileWalk walk(k_lo, k_first, UKT);
    const int jump = walk.jump_at > 0 ? walk.jump_at / UKT : 0;          // tiles before the jump
    const int near = (jump > 0 ? walk.jump_to : walk.start) / UKT, end = (k_hi + UKT - 1) / UKT;
    const int n_first = (jump - rank + 1) / 2, near_mine = near + ((near ^ rank) & 1);
    const int n_tiles = n_first + max(0, (end - near_mine + 1) / 2);
    auto tile_at = [&](int t) {
        return (t < n_first ? rank + 2 * t : near_mine + 2 * (t - n_first)) * UKT;
    };

    const int r = it.row0 + rowi;
    const bool live = r < rows_total;
    const int tok = live ? r / g : 0;
    const int hq = hk * g + (live ? r % g : 0);
    const int pos = pos0 + tok;

    pdl_wait();            // q, and the keys and values of this step's tokens, are just written

    // q's rows into shared memory, operand layout (16-byte piece index xor row % 8)
    {
        const __nv_bfloat16* src = q + (size_t)(tok0 + tok) * q_stride + hq * D;
        const bool whole = q_stride % 8 == 0 && (uintptr_t)q % 16 == 0;
#pragma unroll
        for (int i = 0; i < D / 16; ++i) {
            const int c = half * (D / 16) + i;
            uint4 u = make_uint4(0u, 0u, 0u, 0u);
            if (live && whole) {
                u = *reinterpret_cast<const uint4*>(src + c * 8);
            } else if (live) {
                const unsigned short* e = reinterpret_cast<const unsigned short*>(src + c * 8);
                u.x = e[0] | (unsigned)e[1] << 16; u.y = e[2] | (unsigned)e[3] << 16;
                u.z = e[4] | (unsigned)e[5] << 16; u.w = e[6] | (unsigned)e[7] << 16;
            }
            *reinterpret_cast<uint4*>(q_s + (c >> 3) * U::SUB_Q + rowi * 128 +
                                      (((c & 7) ^ (rowi & 7)) << 4)) = u;
        }
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");   // generic writes -> tensor core
    before_sync();
    __syncthreads();
    after_sync();
    const unsigned tmem = *tmem_slot;
    bool ok = true;
    auto wait = [&](void* bar, unsigned parity) { return mbar_wait(bar, parity, status, ROLE_SPINS); };

    // a tile's pages, a box a lane (at most 8)
    auto fetch = [&](int t) {
        const unsigned box_bytes = (unsigned)box * 128u;
        const int stage = t % STAGES, key = tile_at(t) + lane * box;
        const bool wanted = lane * box < UKT && key < k_hi && (key + box > k_lo || key < k_first);
        int id = -1;
        if (wanted) {
            id = block_table[(size_t)slot * table_stride + key / page];
            if (id >= num_pages) id = -1;
            if (id < 0) atomicExch(status, 2);                   // a seen key without a page
        }
        const unsigned got = __ballot_sync(0xffffffffu, id >= 0);
        const unsigned missing = __ballot_sync(0xffffffffu, wanted && id < 0);
        if (lane == 0) {
            gone_s[stage] = missing;
            mbar_expect_tx(&kv_full[stage], __popc(got) * 2 * KS * box_bytes);
        }
        __syncwarp();
        if (id >= 0) {
            const int y = (id * kv_heads + hk) * page + key % page;
#pragma unroll
            for (int sub = 0; sub < KS; ++sub) {
                const unsigned at = (stage * KS + sub) * U::SUB_KV + lane * box_bytes;
                tma_load_2d(k_s + at, &map_k, &kv_full[stage], 64 * sub, y);
                tma_load_2d(v_s + at, &map_v, &kv_full[stage], 64 * sub, y);
            }
        }
    };
    auto scores = [&](int t) {
        if (ok) ok = wait(&kv_full[t % STAGES], (t / STAGES) & 1);
        after_sync();
        if (lane == 0) {
#pragma unroll
            for (int k = 0; k < D / 16; ++k) {
                const int into = k / (D / 32), sub = k >> 2;
                const unsigned long long a = smem_desc(q_s + sub * U::SUB_Q) + 2 * (k & 3);
                const unsigned long long b =
                    smem_desc(k_s + ((t % STAGES) * KS + sub) * U::SUB_KV) + 2 * (k & 3);
                if (ok) umma_bf16(tmem + S_HALF * into, a, b, instr_desc(128, UKT),
                                  k % (D / 32) > 0);
            }
            if (ok) umma_commit(s_done);
        }
        __syncwarp();
    };
    // the products of tile t's weights, once they are written, and the next tile's scores behind them
    auto products = [&](int t) {
        if (ok) ok = wait(p_ready, t & 1);
        after_sync();
        if (lane == 0) {
            // 16 keys of a term are 8 columns; 16 keys of the values 2 groups of 8 rows.  The values are
            // MN-major, their leading offset from 64 features to the next 64
            unsigned long long b = smem_desc(v_s + (t % STAGES) * KS * U::SUB_KV);
            if (KS == 2) b += (unsigned long long)((U::SUB_KV >> 4) - 1) << 16;
#pragma unroll
            for (int term = 2; term >= 0; --term)
#pragma unroll
                for (int k = 0; k < UKT / 16; ++k)
                    if (ok) umma_a_tmem(tmem + O_COL, tmem + P_TERM * term + 8 * k,
                                        b + (unsigned long long)(k * 2048 >> 4), idesc_pv(D),
                                        term < 2 || k > 0);
            if (ok) umma_commit(o_done);
        }
        __syncwarp();
        if (t + 1 < n_tiles) scores(t + 1);
    };
    int fetched = 0;
    if (warp == FETCHER)
        for (; fetched < STAGES && fetched < n_tiles; ++fetched) fetch(fetched);
    if (warp == ISSUER && n_tiles > 0) scores(0);

    const bool penalty = FORM == 2 && r1 != nullptr;
    const float pen1 = penalty ? r1[hq] : 0.0f, pen2 = penalty ? r2[hq] : 0.0f;
    const int row_lo = max(it.kv_begin, sight_lo(sight, pos));
    const int row_first = it.kv_begin > 0 ? 0 : sight_first(sight, row_lo);
    const int row_hi = live ? min(it.kv_end, pos + 1) : 0;
    constexpr float LOG2E = 1.4426950408889634f, LOG2E_LOW = 1.9259629911266175e-8f;
    const bool capped = FORM != 0 && sight.softcap > 0.0f;
    // a weight is 2^(v U - M): v the product (FORM 0), tanh of the capped quotient, or the score
    // (in two terms, since a rounded factor would bend all of a row's weights the same way; the lower one
    // above 0, so that a hidden key's -inf stays that)
    const double unit64 = 1.4426950408889634 * (FORM == 0 ? (double)scale : capped ? (double)sight.softcap : 1.0);
    float unit = (float)unit64;
    if ((double)unit >= unit64) unit = __uint_as_float(__float_as_uint(unit) - 1);
    const float unit_low = (float)(unit64 - (double)unit);
    const float to_quotient = capped ? (FORM == 1 ? scale / sight.softcap : 1.0f / sight.softcap)
                                     : 1.0f;
    const unsigned lanes = (unsigned)((warp & 3) * 32) << 16;
    float M = -INFINITY, top = -INFINITY, l = 0.0f;
    // a thread's features: two runs, D / 2 apart, so that it holds both features of a turned pair
    constexpr int RUN = HD / 2;
    auto feature = [&](int i) { return (i < RUN ? 0 : D / 2 - RUN) + RUN * half + i; };
    Two acc[HD / 2];
#pragma unroll
    for (int i = 0; i < HD / 2; ++i) acc[i] = 0ull;

    for (int t = 0; t < n_tiles; ++t) {
        const int kt = tile_at(t), stage = t % STAGES, k0 = kt + 32 * half;
        if (ok) ok = wait(s_done, t & 1);
        after_sync();
        const unsigned gone = gone_s[stage];
        float v[32];
        {
#pragma unroll
            for (int c = 0; c < 32; c += 16) {
                unsigned one[16], other[16];
                tmem_load_16cols(tmem + lanes + 32 * half + c, one);
                tmem_load_16cols(tmem + lanes + S_HALF + 32 * half + c, other);
                tmem_wait_loads();
#pragma unroll
                for (int i = 0; i < 16; i += 2)
                    untwo(add_two(two(__uint_as_float(one[i]), __uint_as_float(one[i + 1])),
                                  two(__uint_as_float(other[i]), __uint_as_float(other[i + 1]))),
                          v[c + i], v[c + i + 1]);
            }
        }
        before_sync();
        if (FORM == 2) {
            const float far = (float)(pos - k0);                 // (whole numbers: exact)
            if (penalty && sight.linear) {
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    const Two dist = add_two(two(far, far), two((float)-i, (float)(-i - 1)));
                    untwo(fma_two(two(-pen1, -pen1), dist,
                                  mul_two(two(v[i], v[i + 1]), two(scale, scale))), v[i], v[i + 1]);
                }
            } else {
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    v[i] *= scale;
                    if (penalty) v[i] -= pen1 * log1pf(pen2 * (far - (float)i));
                }
            }
        }
        if (FORM != 0 && (FORM == 1 || capped)) {
            const Two by = two(to_quotient, to_quotient);
            float far = 0.0f;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                untwo(mul_two(two(v[2 * i], v[2 * i + 1]), by), v[2 * i], v[2 * i + 1]);
                far = fmaxf(far, fmaxf(fabsf(v[2 * i]), fabsf(v[2 * i + 1])));
            }
            if (__any_sync(0xffffffffu, far > TANH_NEAR)) {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    v[i] = fabsf(v[i]) > TANH_NEAR ? tanhf(v[i]) : tanh_near(v[i]);
            } else {
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    untwo(tanh_near_two(two(v[2 * i], v[2 * i + 1])), v[2 * i], v[2 * i + 1]);
            }
        }
        const bool inside = k0 + 32 <= row_hi && (k0 >= row_lo || k0 + 32 <= row_first) && gone == 0;
        if (!__all_sync(0xffffffffu, inside)) {
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                const int key = k0 + i;
                const bool seen = (key >= row_lo || key < row_first) && key < row_hi;
                if (!seen || (gone != 0 && ((gone >> ((32 * half + i) / box)) & 1u)))
                    v[i] = -INFINITY;
            }
        }
        float t4[4] = {v[0], v[1], v[2], v[3]};
#pragma unroll
        for (int i = 4; i < 32; ++i) t4[i & 3] = fmaxf(t4[i & 3], v[i]);
        const float mine = fmaxf(fmaxf(t4[0], t4[1]), fmaxf(t4[2], t4[3]));
        share_s[half * UROWS + rowi] = mine;
        asm volatile("bar.sync %0, 64;\n" ::"r"(1 + (warp & 3)) : "memory");
        after_sync();                    // (both halves have read the scores that the weights replace)
        top = fmaxf(top, fmaxf(mine, share_s[(half ^ 1) * UROWS + rowi]));
        // (a row that has seen nothing yet: every weight is 2^-inf = 0)
        const float ref = top == -INFINITY ? 0.0f : top * unit;
        const float corr = exp2_fast(M - ref);
        M = top == -INFINITY ? -INFINITY : ref;
        const Two unit2 = two(unit, unit), low2 = two(unit_low, unit_low), ref2 = two(-ref, -ref);
        Two sum2[2] = {0ull, 0ull};
#pragma unroll
        for (int c = 0; c < 32; c += 16) {
            unsigned hi[8], mid[8], lo[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const Two vv = two(v[c + 2 * i], v[c + 2 * i + 1]);
                float a, b;
                untwo(fma_two(vv, low2, fma_two(vv, unit2, ref2)), a, b);
                a = exp2_fast(a);
                b = exp2_fast(b);
                hi[i] = upper_halves(a, b);
                Two w = two(a, b);
                sum2[i & 1] = add_two(sum2[i & 1], w);
                w = add_two(w, two(minus_upper(a), minus_upper(b)));     // what is left: exact
                untwo(w, a, b);
                mid[i] = upper_halves(a, b);
                untwo(add_two(w, two(minus_upper(a), minus_upper(b))), a, b);
                lo[i] = upper_halves(a, b);
            }
            const unsigned at = tmem + lanes + 16 * half + (c >> 1);
            tmem_store_8cols(at, hi);
            tmem_store_8cols(at + P_TERM, mid);
            tmem_store_8cols(at + 2 * P_TERM, lo);
        }
        {
            float a, b;
            untwo(add_two(sum2[0], sum2[1]), a, b);
            l = fmaf(l, corr, a + b);
        }
        // Pages come whole: values that no row sees may hold anything, and 0 * NaN is NaN in
        // the product.  Four threads a key.
        if (kt + UKT > k_hi || (kt < k_lo && kt + UKT > k_first) || gone != 0) {
            const int j = tid >> 2, key = kt + j;
            if (key >= k_hi || (key < k_lo && key >= k_first) || ((gone >> (j / box)) & 1u)) {
                if (ok) ok = wait(&kv_full[stage], (t / STAGES) & 1);
                constexpr int PIECES = KS * 2;           // of 16 bytes, a thread
                const int c = (tid & 3) * PIECES;
                uint4* row = reinterpret_cast<uint4*>(
                    v_s + (stage * KS + (c >> 3)) * U::SUB_KV + j * 128 + (c & 7) * 16);
#pragma unroll
                for (int i = 0; i < PIECES; ++i) row[i] = make_uint4(0u, 0u, 0u, 0u);
            }
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        }
        asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
        before_sync();
        mbar_arrive(p_ready);
        if (warp == ISSUER) products(t);
        if (ok) ok = wait(o_done, t & 1);
        after_sync();
        if (warp == FETCHER && fetched < n_tiles && __all_sync(0xffffffffu, ok)) fetch(fetched++);
#pragma unroll
        for (int run = 0; run < 2; ++run) {          // (see feature)
            unsigned o[RUN];
            if constexpr (RUN == 32) tmem_load_32cols(tmem + lanes + O_COL + feature(run * RUN), o);
            else tmem_load_16cols(tmem + lanes + O_COL + feature(run * RUN), o);
            tmem_wait_loads();
#pragma unroll
            for (int i = 0; i < RUN / 2; ++i)
                acc[run * RUN / 2 + i] =
                    fma_two(acc[run * RUN / 2 + i], two(corr, corr),
                            two(__uint_as_float(o[2 * i]), __uint_as_float(o[2 * i + 1])));
        }
        before_sync();
    }
    // Copies and products in flight end before the block does (a fetcher whose waits all succeeded has
    // seen every tile's products complete, which began after the tile's copies).
    if (warp == FETCHER && !__all_sync(0xffffffffu, ok))
        for (int t = max(0, fetched - STAGES); t < fetched; ++t)
            mbar_wait(&kv_full[t % STAGES], (t / STAGES) & 1, status);
    if (warp == ISSUER && !__all_sync(0xffffffffu, ok)) {
        if (lane == 0) umma_commit(drained);
        __syncwarp();
        mbar_wait(drained, 0, status);
    }
    pdl_trigger();

    // back by position: cosines and sines of the block's tokens and this rank's pairs, where q was (all
    // products with it are over); pair p of token k at p xor k
    float2* turn_s = reinterpret_cast<float2*>(q_s);           // [128][RUN]
    if (fv != nullptr) {
        const int first = it.row0 / g, count = last_row / g - first + 1;
        for (int e = tid; e < count * RUN; e += UTHREADS) {
            const int k = e / RUN, p = e % RUN;
            float sn, cs;
            sincosf((float)(pos0 + first + k) * fv[RUN * rank + p], &sn, &cs);
            turn_s[k * RUN + (p ^ (k & (RUN - 1)))] = make_float2(cs, -sn);
        }
    }
    share_s[half * UROWS + rowi] = l;
    asm volatile("bar.sync %0, 64;\n" ::"r"(1 + (warp & 3)) : "memory");
    // (the same sum in both halves)
    l = share_s[rowi] + share_s[UROWS + rowi];
    // The pair's results: block `rank` finishes the rows' features of half `rank`, with what the other
    // block's threads of that half leave in its memory, where the key tiles were.
    float4* from_s = reinterpret_cast<float4*>(k_s);           // [HD / 4][128]
    float* from_ml = reinterpret_cast<float*>(from_s + HD / 4 * UROWS);   // [2][128]
    cluster_sync();                          // both blocks are through their tiles
    if (!ok)
        for (int b = 0; b < 2; ++b) store_peer(peer_address(const_cast<unsigned*>(gave_up_s), b), 1u);
    if (half != rank) {
        const unsigned to = peer_address(from_s + rowi, rank ^ 1);
        const unsigned to_ml = peer_address(from_ml + rowi, rank ^ 1);
#pragma unroll
        for (int i = 0; i < HD / 4; ++i) store_peer(to + i * UROWS * 16, acc[2 * i], acc[2 * i + 1]);
        store_peer(to_ml, M);
        store_peer(to_ml + UROWS * 4, l);
    }
    cluster_sync();
    const bool whole = *gave_up_s == 0u;
    if (half == rank) {
        const float M_peer = from_ml[rowi], both = fmaxf(M, M_peer);
        const float ref = both == -INFINITY ? 0.0f : both;
        const float f0 = exp2_fast((rank == 0 ? M : M_peer) - ref);      // block 0's part comes first
        const float f1 = exp2_fast((rank == 0 ? M_peer : M) - ref);
        const float l_peer = from_ml[UROWS + rowi];
        l = fmaf(rank == 0 ? l : l_peer, f0, (rank == 0 ? l_peer : l) * f1);
        M = both;
#pragma unroll
        for (int i = 0; i < HD / 4; ++i) {
            const float4 p = from_s[i * UROWS + rowi];
            const Two peer[2] = {two(p.x, p.y), two(p.z, p.w)};
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const Two a = acc[2 * i + e];
                acc[2 * i + e] = fma_two(rank == 0 ? a : peer[e], two(f0, f0),
                                         mul_two(rank == 0 ? peer[e] : a, two(f1, f1)));
            }
        }
    }
    if (sight.sink != nullptr)
        l += exp2_fast(fmaf(sight.sink[hq], LOG2E_LOW,
                            fmaf(sight.sink[hq], LOG2E, M == -INFINITY ? 0.0f : -M)));
    const float inv = l > 0.0f ? sight.out_scale / l : 0.0f;
    const size_t token = (size_t)(tok0 + tok);
    const size_t o = token * out_stride + hq * D;
    const bool pieces = out_f32 ? out_stride % 4 == 0 && (uintptr_t)out % 16 == 0
                                : out_stride % 8 == 0 && (uintptr_t)out % 16 == 0;
    const __nv_bfloat16* gate = (const __nv_bfloat16*)sight.gate;
    const bool per_feature = gate != nullptr && !sight.gate_per_head;
    const bool gate_pieces = sight.ld_gate % 8 == 0 && (uintptr_t)gate % 16 == 0;
    const float head_gate =
        per_feature ? 1.0f : sight_gate<__nv_bfloat16>(sight, live ? token : 0, hq, D, 0);
    float zero = 0.0f;
    if (live && whole && half == rank) {
#pragma unroll
        for (int i = 0; i < HD / 2; ++i) acc[i] = mul_two(acc[i], two(inv, inv));
        if (fv != nullptr) {
            const int k = tok - it.row0 / g;
            const float2* turn = turn_s + k * RUN;
#pragma unroll
            for (int p = 0; p < RUN; p += 2) {
                float a[2], b[2];
                untwo(acc[p / 2], a[0], a[1]);
                untwo(acc[(RUN + p) / 2], b[0], b[1]);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const float2 cs = turn[(p + e) ^ (k & (RUN - 1))];
                    rope_rotate(a[e], b[e], cs.x, cs.y, a[e], b[e]);
                }
                acc[p / 2] = two(a[0], a[1]);
                acc[(RUN + p) / 2] = two(b[0], b[1]);
            }
        }
#pragma unroll
        for (int c = 0; c < HD; c += 8) {
            float x[8];
            const int at = feature(c);
#pragma unroll
            for (int i = 0; i < 8; i += 2) untwo(acc[(c + i) / 2], x[i], x[i + 1]);
            if (per_feature) {
                const __nv_bfloat16* gp = gate + token * sight.ld_gate + hq * D + at;
                float f[8];
                if (gate_pieces) {
                    load_piece(gp, f);
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) f[i] = to_float(gp[i]);
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) x[i] *= 1.0f / (1.0f + expf(-f[i]));
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) x[i] *= head_gate;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) zero = fmaf(x[i], 0.0f, zero);
            if (pieces && out_f32) {
                store8((float*)out + o + at, x);
            } else if (pieces) {
                store8((__nv_bfloat16*)out + o + at, x);
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    store_out<__nv_bfloat16>(out, out_f32, o + at + i, x[i]);
            }
        }
    }
    const unsigned met = __ballot_sync(0xffffffffu, live && whole && half == rank && !(zero == 0.0f));
    if (lane == 0) spoilt_s[warp] = met;
    before_sync();
    __syncthreads();
    if (warp == ISSUER) tmem_dealloc(tmem, UCOLS);
    if (half != rank) return;
    // rows that met an infinity or NaN
    const unsigned spoilt = spoilt_s[warp];
    if (spoilt == 0) return;
    for (int b = 0; b < 32; ++b) {
        if (!((spoilt >> b) & 1u)) continue;
        const int row = it.row0 + (warp & 3) * 32 + b, tk = row / g, h = hk * g + row % g;
        const bool penalty = r1 != nullptr;
        float mr, lr, res[D / 32];
        row_again<D>(q + (size_t)(tok0 + tk) * q_stride + h * D, k_pages, v_pages,
                     block_table + (size_t)slot * table_stride, num_pages, hk, kv_heads, page,
                     pos0 + tk, it.kv_begin, it.kv_end, scale, penalty ? r1[h] : 0.0f,
                     penalty ? r2[h] : 0.0f, penalty, sight, mr, lr, res);
        const float inv = sight_inverse(sight, h, mr, lr);
        const size_t o = (size_t)(tok0 + tk) * out_stride + h * D;
#pragma unroll
        for (int i = 0; i < D / 32; ++i) res[i] *= inv;
#pragma unroll
        for (int i = 0; i < D / 64; ++i) {                     // pairs (i, i + D / 2)
            const int col = lane + 32 * i;
            if (fv != nullptr) {
                float sn, cs;
                sincosf((float)(pos0 + tk) * fv[col], &sn, &cs);
                rope_rotate(res[i], res[i + D / 64], cs, -sn, res[i], res[i + D / 64]);
            }
            if (col / RUN != rank) continue;                   // the other block's
#pragma unroll
            for (int e = 0; e < 2; ++e)
                store_out<__nv_bfloat16>(out, out_f32, o + col + e * (D / 2), res[i + e * (D / 64)] *
                    sight_gate<__nv_bfloat16>(sight, (size_t)(tok0 + tk), h, D, col + e * (D / 2)));
        }
    }
}

template <int D, int FORM>
int launch(const void* q, int q_stride, void* out, int out_stride, const void* k_pages,
           const void* v_pages, const int* block_table, int table_stride, int num_pages,
           const int* seq_slot, const int* seq_qstart, const int* seq_qlen, const int* seq_pos0,
           const int* items, int num_items, const float* r1, const float* r2, int heads, int kv_heads,
           int page, int box, float scale, const Sight& sight, const float* fv, int out_f32,
           int* status, cudaStream_t s) {
    CUtensorMap map_k, map_v;
    const long long rows = (long long)num_pages * kv_heads * page;
    int code = tensor_maps::get(&map_k, k_pages, rows, D, D, box, 64);
    if (!code) code = tensor_maps::get(&map_v, v_pages, rows, D, D, box, 64);
    if (code) return code;
    auto kernel = attn_chunk_tcgen05_kernel<D, FORM>;
    static std::atomic<unsigned long long> sized{0};         // a bit a device
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return (int)e;
    const unsigned long long bit = device < 64 ? 1ull << device : 0ull;
    if (!(sized.load() & bit)) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Umma<D>::SMEM);
        if (e == cudaSuccess)                                // (two blocks an SM)
            e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        if (e != cudaSuccess) return (int)e;
        sized |= bit;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)num_items * (unsigned)kv_heads * 2);
    cfg.blockDim = dim3(UTHREADS);
    cfg.dynamicSmemBytes = Umma<D>::SMEM;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_pdl ? 2 : 1;
    return de_check(cudaLaunchKernelEx(
        &cfg, kernel, (const __nv_bfloat16*)q, q_stride, out, out_stride, map_k, map_v,
        (const __nv_bfloat16*)k_pages, (const __nv_bfloat16*)v_pages, block_table, table_stride,
        num_pages, seq_slot, seq_qstart, seq_qlen, seq_pos0, (const WorkItem*)items, r1, r2, heads,
        kv_heads, page, box, scale, sight, fv, out_f32, status));
}

}  // namespace

DE_EXPORT int de_attn_chunk_tcgen05_rows() { return UROWS; }

// Whether the kernel takes such heads and pages (bfloat16): boxes of 8 to 64 keys a page.
DE_EXPORT int de_attn_chunk_tcgen05_ok(int dk, int dv, int page) {
    return dk == dv && (dk == 64 || dk == 128) && page > 0 && page % 8 == 0;
}

// As de_attn_chunk for bfloat16, with items of 128 rows; keys and values in pages of their own.  fv
// [dv / 2] or null: every result is turned back by its token's position, pairs (i, i + dv / 2), before the
// gate (as attn_finish turns them).
DE_EXPORT int de_attn_chunk_tcgen05(const void* q, int q_stride, void* out, int out_stride,
                                    const void* k_pages, const void* v_pages,
                                    const int* block_table, int table_stride, int num_pages,
                                    const int* seq_slot, const int* seq_qstart, const int* seq_qlen,
                                    const int* seq_pos0, const int* items, int num_items,
                                    const float* r1, const float* r2, int heads, int kv_heads,
                                    int dk, int dv, int page, float scale, int chunk, int window,
                                    int keep_first, float softcap, int out_f32, int linear,
                                    const float* sink, const void* out_gate, int ld_out_gate,
                                    int gate_per_head, float out_scale, const float* fv, int* status,
                                    void* stream) {
    if (num_items <= 0) return 0;
    if (!de_attn_chunk_tcgen05_ok(dk, dv, page) || kv_heads <= 0 || heads % kv_heads != 0) return -2;
    if ((uintptr_t)k_pages % 16 != 0 || (uintptr_t)v_pages % 16 != 0) return -5;
    const Sight sight = {chunk, window, keep_first, softcap, dv, linear, sink, out_gate, ld_out_gate,
                         gate_per_head, out_scale};
    int box = 8;                                             // keys of a box: a page's, or part of it
    while (box < UKT && page % (box * 2) == 0) box *= 2;
    const int form = r1 != nullptr ? 2 : (softcap > 0.0f ? 1 : (scale > 0.0f ? 0 : 2));
#define GO(D, FORM)                                                                             \
    return launch<D, FORM>(q, q_stride, out, out_stride, k_pages, v_pages, block_table,         \
                           table_stride, num_pages, seq_slot, seq_qstart, seq_qlen, seq_pos0,   \
                           items, num_items, r1, r2, heads, kv_heads, page, box, scale, sight,  \
                           fv, out_f32, status, (cudaStream_t)stream)
    if (dk == 64) {
        if (form == 0) GO(64, 0);
        if (form == 1) GO(64, 1);
        GO(64, 2);
    }
    if (form == 0) GO(128, 0);
    if (form == 1) GO(128, 1);
    GO(128, 2);
#undef GO
}
