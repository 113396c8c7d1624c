// Longer portions through the mixers that carry a matrix state per head, in chunks of 64 tokens
// instead of token by token (recurrent.cu has the rules and the token-by-token scan): what depends
// on a chunk's own tokens is formed for all chunks side by side, and only a short chain runs from
// chunk to chunk.  Float32 multiply-adds throughout.
//
// A fixed decay per head (retention, lightning attention), S <- d S + k v^T, o = S^T q, with t and s
// the places inside the chunk and S0 the state before it:
//   o_t = d^(t+1) S0^T q_t + sum over s <= t of d^(t-s) (q_t . k_s) v_s
//   S   = d^n S0 + sum over s of d^(n-1-s) k_s v_s^T
//
// The delta rule with a decay g_t per key channel, S <- diag(g_t) S; u_t = beta_t (v_t - S^T k_t);
// S <- S + k_t u_t^T; o_t = S^T q_t, with b_t the product of g_0 .. g_t (channel by channel) and
// w_ts = (b_t / b_s) k_s:
//   A_ts = k_t . w_ts (s < t),  P_ts = q_t . w_ts (s <= t)
//   u = X_v - X_k S0, where X solves (1 + diag(beta) A) X = diag(beta) [v | b k]
//   o = (b q) S0 + P u,   S = diag(b_n) S0 + sum over s of (b_n / b_s) k_s u_s^T
// No quotient is formed: b_t / b_s is the product of the decays between, walked channel by channel
// (w_ts from w_(t-1)s), so nothing overflows however fast the state decays.
//
// A cut of a portion changes the order of float32 sums only.
//
// Figures below: 2,048 tokens of 16 heads of 128 x 128 on B200.  The scan takes 0.37 us a
// token for the delta rule, 760 us in all, by chunks 205 us; under a decay per head a layer with its
// products took 1,861 us by the scan, 194 us by chunks (98 of them here).

#include "common.cuh"

DE_DEFINE_PDL_SWITCH

namespace {

constexpr int CH = 64;             // tokens of a chunk
constexpr int LD = CH + 4;         // a row of 64 in shared memory

struct Item {                      // a chunk
    int seq, token, count, portion;
};
struct Portion {
    int seq, first, chunks, pad;   // its first item and how many
};
// What of a portion lies among the items [begin, begin + m) of a launch: from which item of the launch
// on, and how many.
__device__ __forceinline__ Portion part_of(Portion p, int begin, int m) {
    const int lo = max(p.first, begin), hi = min(p.first + p.chunks, begin + m);
    p.first = lo - begin;
    p.chunks = max(hi - lo, 0);
    return p;
}

__device__ __forceinline__ void cp16(float* dst, const float* src, bool ok) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int bytes = ok ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void cp4(float* dst, const float* src, bool ok) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int bytes = ok ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(src), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
// two IEEE multiply-adds in one instruction
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a,
                                     unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;\n" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long pair(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpair(unsigned long long v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;\n" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ float4 four(const float* p) { return *reinterpret_cast<const float4*>(p); }

// A tile of 64 x 64 on 128 threads: a thread has rows row .. row + 3, row + 16 .. row + 19 and
// columns col .. col + 3.  Lanes l and l ^ 1 share rows, l and l ^ 2 columns, so that 16-byte reads
// of shared memory pass in two wavefronts.
struct Tile {
    unsigned long long acc[8][2];
    int row, col;
    __device__ __forceinline__ Tile() {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        row = (warp >> 1) * 32 + (((lane >> 1) & 1) | ((lane >> 3) & 2)) * 4;
        col = (warp & 1) * 32 + ((lane & 1) | ((lane >> 1) & 6)) * 4;
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = 0ull;
    }
    // rows of a [k][LD] against columns of b [k][LD], n values of k
    template <int N> __device__ __forceinline__ void add(const float* a, const float* b) {
#pragma unroll 16
        for (int k = 0; k < N; ++k) {
            const float4 a0 = four(a + k * LD + row), a1 = four(a + k * LD + row + 16);
            const float4 b0 = four(b + k * LD + col);
            const float v[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
            const unsigned long long p0 = pair(b0.x, b0.y), p1 = pair(b0.z, b0.w);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const unsigned long long aa = pair(v[i], v[i]);
                fma2(acc[i][0], aa, p0);
                fma2(acc[i][1], aa, p1);
            }
        }
    }
    __device__ __forceinline__ int row_of(int i) const { return row + (i & 3) + (i >> 2) * 16; }
    __device__ __forceinline__ float4 get(int i) const {
        float4 v;
        unpair(acc[i][0], v.x, v.y);
        unpair(acc[i][1], v.z, v.w);
        return v;
    }
};

// d^0 .. d^64, products formed in double precision
__device__ __forceinline__ void powers(float d, float* pw) {
    if (threadIdx.x <= CH) {
        double p = 1.0;
        for (int i = 0; i < (int)threadIdx.x; ++i) p *= (double)d;
        pw[threadIdx.x] = (float)p;
    }
}

// N rows of 64 columns (rows beyond `rows` are zeros) into tile [N][LD]; 128 threads
template <int N = 64>
__device__ __forceinline__ void load_tile(float* tile, const float* src, size_t ld, int rows) {
#pragma unroll
    for (int i = 0; i < N / 8; ++i) {
        const int e = threadIdx.x + 128 * i, r = e >> 4, c = (e & 15) * 4;
        cp16(tile + r * LD + c, r < rows ? src + (size_t)r * ld + c : src, r < rows);
    }
}
template <int N = 64>
__device__ __forceinline__ void load_tile(float* tile, const __nv_bfloat16* src, size_t ld,
                                          int rows) {
#pragma unroll
    for (int i = 0; i < N / 8; ++i) {
        const int e = threadIdx.x + 128 * i, r = e >> 4, c = (e & 15) * 4;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (r < rows) {
            const uint2 u = *reinterpret_cast<const uint2*>(src + (size_t)r * ld + c);
            v = make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u),
                            __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
        }
        *reinterpret_cast<float4*>(tile + r * LD + c) = v;
    }
}

// ------------------------------------------------------------------------------------------
// A decay per head.  products: pt[item][h][s][t] = d^(t-s) q_t . k_s (0 for s > t) and
// xt[item][h][c][t] = d^(t+1) q_t[c].  grid (items, H), 128 threads.  64 channels at a time, so that 512
// blocks are one round: 25 us, the way in of operands that are used once a block (all 128 at once, three
// blocks an SM: 28).
// ------------------------------------------------------------------------------------------
template <int DK>
__global__ void __launch_bounds__(128, 4)
decay_products_kernel(const float* __restrict__ q, int ldq, const float* __restrict__ k, int ldk,
                      const float* __restrict__ decay, const Item* __restrict__ items,
                      float* __restrict__ xt, float* __restrict__ pt, int H) {
    extern __shared__ __align__(16) float sh[];
    float* qs = sh;                                  // [64][LD]: 64 channels at a time
    float* ks = qs + 64 * LD;
    __shared__ float pw[CH + 1];
    const Item it = items[blockIdx.x];
    const int h = blockIdx.y;
    powers(decay[h], pw);
    pdl_wait();
    const size_t at = (size_t)blockIdx.x * H + h;
    float* x = xt + at * DK * CH;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Tile tile;
    for (int half = 0; half < DK; half += 64) {
        // turned on the way in: a warp copies 8 channels of 4 tokens at a time
        for (int c0 = 0; c0 < 64; c0 += 8)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int t = (i * 4 + warp) * 4 + (lane >> 3), c = c0 + (lane & 7);
                const bool ok = t < it.count;
                const size_t tok = (size_t)(it.token + (ok ? t : 0));
                cp4(qs + c * LD + t, q + tok * ldq + h * DK + half + c, ok);
                cp4(ks + c * LD + t, k + tok * ldk + h * DK + half + c, ok);
            }
        cp_commit();
        cp_wait<0>();
        __syncthreads();
        if (warp != 2) tile.add<64>(ks, qs);         // (its 32 s lie behind its 32 t: zeros)
        for (int e = threadIdx.x; e < 64 * CH / 4; e += 128) {
            const int c = e >> 4, t = (e & 15) * 4;
            const float4 v = four(qs + c * LD + t);
            *reinterpret_cast<float4*>(x + (half + c) * CH + t) = make_float4(
                v.x * pw[t + 1], v.y * pw[t + 2], v.z * pw[t + 3], v.w * pw[t + 4]);
        }
        __syncthreads();
    }
    pdl_trigger();
    float* p = pt + at * CH * CH;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int s = tile.row_of(i);
        float4 v = tile.get(i);
        const int d = tile.col - s;
        v.x = d >= 0 ? v.x * pw[d] : 0.0f;
        v.y = d >= -1 ? v.y * pw[d + 1] : 0.0f;
        v.z = d >= -2 ? v.z * pw[d + 2] : 0.0f;
        v.w = d >= -3 ? v.w * pw[d + 3] : 0.0f;
        *reinterpret_cast<float4*>(p + s * CH + tile.col) = v;
    }
}

// What a chunk adds to the state by itself: states[item][h][c][j] = sum_s d^(n-1-s) k_s[c] v_s[j].
// grid (items, H, DK / 64 * dv / 64), 128 threads.  33 us: 64 x 64 outputs a block
// over 64 tokens, too short a sum to hide the operands' way in.
template <typename VT>
__global__ void __launch_bounds__(128, 4)
decay_states_kernel(const float* __restrict__ k, int ldk, const VT* __restrict__ v, int ldv,
                    const float* __restrict__ decay, const Item* __restrict__ items,
                    float* __restrict__ states, int H, int dk, int dv) {
    __shared__ __align__(16) float ks[CH * LD], vs[CH * LD];
    __shared__ float pw[CH + 1];
    const Item it = items[blockIdx.x];
    const int h = blockIdx.y, cols = dv / 64;
    const int c0 = (int)blockIdx.z / cols * 64, j0 = (int)blockIdx.z % cols * 64;
    powers(decay[h], pw);
    pdl_wait();
    load_tile(ks, k + (size_t)it.token * ldk + h * dk + c0, ldk, it.count);
    load_tile(vs, v + (size_t)it.token * ldv + h * dv + j0, ldv, it.count);
    cp_commit();
    cp_wait<0>();
    __syncthreads();
    for (int e = threadIdx.x; e < it.count * 16; e += 128) {
        const int s = e >> 4;
        float4* p = reinterpret_cast<float4*>(ks + s * LD + (e & 15) * 4);
        const float f = pw[it.count - 1 - s];
        p->x *= f; p->y *= f; p->z *= f; p->w *= f;
    }
    __syncthreads();
    Tile tile;
    tile.add<CH>(ks, vs);
    pdl_trigger();
    float* o = states + (((size_t)blockIdx.x * H + h) * dk + c0) * dv + j0;
#pragma unroll
    for (int i = 0; i < 8; ++i)
        *reinterpret_cast<float4*>(o + (size_t)tile.row_of(i) * dv + tile.col) = tile.get(i);
}

// The states at the chunks' starts: states[item] becomes the state before the chunk, the slot keeps
// the one after the last.  grid (portions, elements / 1024), 256 threads with four elements each.
// Eight states are asked for before any is used: 9 us, memory's rate.
__global__ void __launch_bounds__(256)
decay_pass_kernel(float* __restrict__ states, const float* __restrict__ decay,
                  const Item* __restrict__ items, const Portion* __restrict__ portions, int begin,
                  int m, float* __restrict__ state, long long slot_stride,
                  const int* __restrict__ seq_slot, int H, int size) {
    const Portion p = part_of(portions[blockIdx.x], begin, m);
    const int e = ((int)blockIdx.y * 256 + (int)threadIdx.x) * 4;
    if (e >= H * size || p.chunks == 0) {
        pdl_wait();
        return;
    }
    const int last = items[p.first + p.chunks - 1].count;
    float* slot = state + (size_t)seq_slot[p.seq] * slot_stride;
    const double d = (double)decay[e / size];
    double f64 = 1.0, flast = 1.0;
    for (int i = 0; i < CH; ++i) f64 *= d;
    for (int i = 0; i < last; ++i) flast *= d;
    const float full = (float)f64, part = (float)flast;
    pdl_wait();
    float4 s = four(slot + e);
    float* base = states + (size_t)p.first * H * size + e;
    const size_t step = (size_t)H * size;
    for (int n0 = 0; n0 < p.chunks; n0 += 8) {       // eight chunks' elements asked for at once
        float4 add[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            add[i] = n0 + i < p.chunks ? four(base + (n0 + i) * step)
                                       : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int n = n0 + i;
            if (n >= p.chunks) break;
            const float f = n == p.chunks - 1 ? part : full;
            *reinterpret_cast<float4*>(base + n * step) = s;
            s.x = fmaf(f, s.x, add[i].x);
            s.y = fmaf(f, s.y, add[i].y);
            s.z = fmaf(f, s.z, add[i].z);
            s.w = fmaf(f, s.w, add[i].w);
        }
    }
    pdl_trigger();
    *reinterpret_cast<float4*>(slot + e) = s;
}

// ------------------------------------------------------------------------------------------
// The delta rule.  What a chunk's tokens give by themselves: at[item][h][s][t] = A_ts,
// pt[item][h][s][t] = P_ts (0 for s > t), xt[item][h][c][t] = b_t q_t, kd[item][h][t][c] = b_t k_t,
// kh[item][h][s][c] = (b_n / b_s) k_s and bn[item][h][c] = b_n.  grid (items, H), 256 threads.
// A thread walks w of two columns s over the tokens, an eighth of the channels each (lanes 4 apart
// share a column), as the scan walks the state; the eight sums of a column meet four tokens at a time,
// each lane left with two of the 16 results.  Two blocks an SM (a chunk's vectors are 99 KB): 55 us, an
// instruction issued in 40 % of the cycles; four warps with a quarter of the channels a lane took 76.
// ------------------------------------------------------------------------------------------
template <int DK>
__global__ void __launch_bounds__(256, 2)
delta_chunk_kernel(const float* __restrict__ q, int ldq, const float* __restrict__ k, int ldk,
                   const float* __restrict__ g, int ldg, const Item* __restrict__ items,
                   float* __restrict__ at, float* __restrict__ pt, float* __restrict__ xt,
                   float* __restrict__ kd, float* __restrict__ kh, float* __restrict__ bn, int H,
                   int rep) {
    constexpr int W = DK + 4, R = DK / 32;           // a row in shared memory; quads of a lane
    extern __shared__ __align__(16) float sh[];
    float* qs = sh;                                  // [CH][W]
    float* ks = qs + CH * W;
    float* gs = ks + CH * W;
    const Item it = items[blockIdx.x];
    const int h = blockIdx.y, hk = h / rep;
    const size_t where = (size_t)blockIdx.x * H + h;
    pdl_wait();
    for (int e = threadIdx.x; e < CH * DK / 4; e += 256) {
        const int t = e / (DK / 4), c = e % (DK / 4) * 4;
        const bool ok = t < it.count;
        const size_t tok = (size_t)(it.token + (ok ? t : 0));
        cp16(qs + t * W + c, q + tok * ldq + hk * DK + c, ok);
        cp16(ks + t * W + c, k + tok * ldk + hk * DK + c, ok);
        if (ok) cp16(gs + t * W + c, g + tok * ldg + h * DK + c, true);
        else *reinterpret_cast<float4*>(gs + t * W + c) = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
    }
    cp_commit();
    cp_wait<0>();
    __syncthreads();
    if (threadIdx.x < 2 * DK) {                      // (whole warps)
        const int c = threadIdx.x % DK;
        if (threadIdx.x < DK) {
            float b = 1.0f;
            float* x = xt + (where * DK + c) * CH;
            float* d = kd + where * CH * DK + c;
#pragma unroll 2
            for (int t = 0; t < CH; t += 4) {
                float v[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    b *= gs[(t + i) * W + c];
                    v[i] = b * qs[(t + i) * W + c];
                    d[(size_t)(t + i) * DK] = b * ks[(t + i) * W + c];
                }
                *reinterpret_cast<float4*>(x + t) = make_float4(v[0], v[1], v[2], v[3]);
            }
            bn[where * DK + c] = b;
        } else {
            float* o = kh + where * CH * DK + c;
            float r = 1.0f;
#pragma unroll 4
            for (int t = CH - 1; t >= 0; --t) {
                o[(size_t)t * DK] = r * ks[t * W + c];
                r *= gs[t * W + c];
            }
        }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int share = lane >> 2, s0 = warp * 8 + (lane & 3) * 2, s1 = s0 + 1;
    unsigned long long w0[2 * R], w1[2 * R];         // neighbouring channels in pairs
#pragma unroll
    for (int i = 0; i < 2 * R; ++i) w0[i] = w1[i] = 0ull;
    // what a lane writes: A or P, of column s0 or s1, two of four tokens
    const bool is_p = share & 4, second = share & 2, later = share & 1;
    float* rows = (is_p ? pt : at) + (where * CH + (second ? s1 : s0)) * CH;
    for (int t = later * 4; t < warp * 8; t += 8)
        *reinterpret_cast<float4*>(rows + t) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int t = warp * 8; t < CH; t += 4) {
        float va[2][4], vp[2][4];                    // by column and token
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int tt = t + i;
            unsigned long long sa0 = 0ull, sa1 = 0ull, sp0 = 0ull, sp1 = 0ull;
            const bool near = tt < warp * 8 + 8;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int o = tt * W + 32 * r + 4 * share;
                const float4 gg = four(gs + o), kk = four(ks + o), qq = four(qs + o);
                const unsigned long long gv[2] = {pair(gg.x, gg.y), pair(gg.z, gg.w)};
                const unsigned long long kv[2] = {pair(kk.x, kk.y), pair(kk.z, kk.w)};
                const unsigned long long qv[2] = {pair(qq.x, qq.y), pair(qq.z, qq.w)};
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    w0[2 * r + x] = mul2(w0[2 * r + x], gv[x]);
                    w1[2 * r + x] = mul2(w1[2 * r + x], gv[x]);
                }
                if (near) {                          // (a column begins inside its warp's 8 tokens)
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        if (tt == s0) w0[2 * r + x] = kv[x];
                        if (tt == s1) w1[2 * r + x] = kv[x];
                    }
                }
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    fma2(sa0, kv[x], w0[2 * r + x]);
                    fma2(sa1, kv[x], w1[2 * r + x]);
                    fma2(sp0, qv[x], w0[2 * r + x]);
                    fma2(sp1, qv[x], w1[2 * r + x]);
                }
            }
            float lo, hi;
            unpair(sa0, lo, hi);
            va[0][i] = tt <= s0 ? 0.0f : lo + hi;    // A is strictly below the diagonal
            unpair(sa1, lo, hi);
            va[1][i] = tt <= s1 ? 0.0f : lo + hi;
            unpair(sp0, lo, hi);
            vp[0][i] = lo + hi;
            unpair(sp1, lo, hi);
            vp[1][i] = lo + hi;
        }
        // the shares' sums: at each step a lane keeps half of what it has and gives the other half
        float one[2][4], two[4], out[2];
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int i = 0; i < 4; ++i)
                one[c][i] = (is_p ? vp[c][i] : va[c][i]) +
                            __shfl_xor_sync(0xffffffffu, is_p ? va[c][i] : vp[c][i], 16);
#pragma unroll
        for (int i = 0; i < 4; ++i)
            two[i] = (second ? one[1][i] : one[0][i]) +
                     __shfl_xor_sync(0xffffffffu, second ? one[0][i] : one[1][i], 8);
#pragma unroll
        for (int i = 0; i < 2; ++i)
            out[i] = (later ? two[2 + i] : two[i]) +
                     __shfl_xor_sync(0xffffffffu, later ? two[i] : two[2 + i], 4);
        *reinterpret_cast<float2*>(rows + t + 2 * later) = make_float2(out[0], out[1]);
    }
    pdl_trigger();
}

// X of (1 + diag(beta) A) X = diag(beta) [v | b k]: xv[item][h][t][j] and, turned, xkt[item][h][c][t].
// grid (items, H, ceil((dv + DK) / 128)), 64 threads with two columns each: forward substitution by
// blocks of 16 tokens, a thread's earlier rows in shared memory of its own.  35 us: a chain of 64
// rows, an instruction issued in a third of the cycles.  (A column a thread, twice the warps: 42, the
// reads of A, which all lanes share, are what fills shared memory's pipe.)
template <int DK>
__global__ void __launch_bounds__(64)
delta_solve_kernel(const float* __restrict__ at, const float* __restrict__ v, int ldv,
                   const float* __restrict__ kd, const float* __restrict__ beta, int ldb,
                   const Item* __restrict__ items, float* __restrict__ xv,
                   float* __restrict__ xkt, int H, int dv) {
    extern __shared__ __align__(16) float sh[];
    float* as = sh;                                  // [CH][LD]: [s][t]
    float* xs = as + CH * LD;                        // [CH][128]
    __shared__ float bs[CH];
    const Item it = items[blockIdx.x];
    const int h = blockIdx.y;
    const size_t where = (size_t)blockIdx.x * H + h;
    const int j = blockIdx.z * 128 + 2 * threadIdx.x;          // columns j, j + 1 of [v | k]
    const bool live = j < dv + DK, is_v = j < dv;
    pdl_wait();
    for (int e = threadIdx.x; e < CH * 16; e += 64)
        cp16(as + (e >> 4) * LD + (e & 15) * 4, at + where * CH * CH + e * 4, true);
    cp_commit();
    bs[threadIdx.x] = (int)threadIdx.x < it.count
                          ? beta[(size_t)(it.token + threadIdx.x) * ldb + h] : 0.0f;
    cp_wait<0>();
    __syncthreads();
    float* mine = xs + 2 * threadIdx.x;
    for (int t0 = 0; t0 < CH; t0 += 16) {
        float2 rhs[16];
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            const int t = t0 + r;
            rhs[r] = make_float2(0.0f, 0.0f);
            if (live && t < it.count)
                rhs[r] = is_v ? *reinterpret_cast<const float2*>(
                                    v + (size_t)(it.token + t) * ldv + h * dv + j)
                              : *reinterpret_cast<const float2*>(kd + (where * CH + t) * DK + j - dv);
        }
        unsigned long long acc[16];
#pragma unroll
        for (int r = 0; r < 16; ++r) acc[r] = 0ull;
#pragma unroll 4
        for (int s = 0; s < t0; ++s) {
            const unsigned long long x = *reinterpret_cast<const unsigned long long*>(mine + s * 128);
#pragma unroll
            for (int r = 0; r < 16; r += 4) {
                const float4 a = four(as + s * LD + t0 + r);
                fma2(acc[r], pair(a.x, a.x), x);
                fma2(acc[r + 1], pair(a.y, a.y), x);
                fma2(acc[r + 2], pair(a.z, a.z), x);
                fma2(acc[r + 3], pair(a.w, a.w), x);
            }
        }
        float o0[16], o1[16];
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            float s0, s1;
            unpair(acc[r], s0, s1);
            const float b = bs[t0 + r];
            o0[r] = b * (rhs[r].x - s0);
            o1[r] = b * (rhs[r].y - s1);
            const unsigned long long x = pair(o0[r], o1[r]);
#pragma unroll
            for (int i = (r + 1) & ~3; i < 16; i += 4) {       // (acc up to r has been used)
                const float4 a = four(as + (t0 + r) * LD + t0 + i);
                fma2(acc[i], pair(a.x, a.x), x);
                fma2(acc[i + 1], pair(a.y, a.y), x);
                fma2(acc[i + 2], pair(a.z, a.z), x);
                fma2(acc[i + 3], pair(a.w, a.w), x);
            }
        }
        // (not sooner: a store would hold back the reads of A after it)
#pragma unroll
        for (int r = 0; r < 16; ++r)
            *reinterpret_cast<float2*>(mine + (t0 + r) * 128) = make_float2(o0[r], o1[r]);
        if (!live) continue;
        if (is_v) {
#pragma unroll
            for (int r = 0; r < 16; ++r)
                *reinterpret_cast<float2*>(xv + (where * CH + t0 + r) * dv + j) =
                    make_float2(o0[r], o1[r]);
        } else {
            float* o = xkt + (where * DK + j - dv) * CH + t0;
#pragma unroll
            for (int r = 0; r < 16; r += 4) {
                *reinterpret_cast<float4*>(o + r) = make_float4(o0[r], o0[r + 1], o0[r + 2], o0[r + 3]);
                *reinterpret_cast<float4*>(o + CH + r) =
                    make_float4(o1[r], o1[r + 1], o1[r + 2], o1[r + 3]);
            }
        }
    }
    pdl_trigger();
}

// The chain from chunk to chunk: states[item] = the state before the chunk, u = X_v - X_k S0 in
// X_v's place, then the state after it.  grid (portions, H, dv / 16), 4 DK + 64 threads: a block has 16
// columns of a head's state in two sides of eight, and each side's 2 DK threads go through the chunks by
// themselves, a warp 16 rows of the state.  For u every warp sums over its own rows; the warps' parts
// meet in shared memory.  Two warps more bring the chunks' operands, which both sides read, through two
// stages, so that one side's multiply-adds fill the other's waits.  88 us, 2.8 us a chunk, shared
// memory's pipe at work in 62 % of the cycles (128 blocks, one an SM; columns in slices of 16 are what
// gives the chain a block on most SMs).  All 16 columns on eight warps that wait for one another three
// times a chunk took 105 us, on 16 warps 109; four warps to bring the operands instead of two, 4 us more.
constexpr int PC = 16, PS = PC / 2, BRING = 64;
template <int DK> struct Pass {
    static constexpr int W = DK + 4;
    static constexpr int STAGE = DK * LD + CH * W;             // xkt, kh
    static constexpr int WARPS = DK / 16, SIDE = 2 * DK;       // of a side
    static constexpr int THREADS = 2 * SIDE + BRING;
    static constexpr int OWN = DK * PS + CH * PS + WARPS * CH * PS;      // floats of a side: S0, u, parts
    static constexpr size_t SMEM = (size_t)(2 * STAGE + 2 * OWN) * sizeof(float);
};
__device__ __forceinline__ void bar_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int threads) {
    asm volatile("bar.arrive %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}

template <int DK>
__global__ void __launch_bounds__(4 * DK + BRING)
delta_pass_kernel(const float* __restrict__ xkt, const float* __restrict__ kh,
                  const float* __restrict__ bn, float* __restrict__ xv, float* __restrict__ states,
                  const Portion* __restrict__ portions, int begin, int m,
                  float* __restrict__ state, long long slot_stride,
                  const int* __restrict__ seq_slot, int H, int dv) {
    constexpr int W = Pass<DK>::W, STAGE = Pass<DK>::STAGE, WARPS = Pass<DK>::WARPS;
    constexpr int SIDE = Pass<DK>::SIDE;
    extern __shared__ __align__(16) float sh[];
    const Portion p = part_of(portions[blockIdx.x], begin, m);
    const int h = blockIdx.y;
    pdl_wait();
    if (p.chunks == 0) return;
    // named barriers: 1 + side within a side, 3 + 2 side + stage "landed", 7 + 2 side + stage "used"
    if (threadIdx.x >= 2 * SIDE) {
        const int tid = threadIdx.x - 2 * SIDE;
        for (int n = 0; n < p.chunks; ++n) {
            float* st = sh + (n & 1) * STAGE;
            if (n >= 2) {
                bar_sync(7 + (n & 1), SIDE + BRING);
                bar_sync(9 + (n & 1), SIDE + BRING);
            }
            const size_t where = (size_t)(p.first + n) * H + h;
            const float* a = xkt + where * DK * CH;
            const float* b = kh + where * CH * DK;
#pragma unroll 8
            for (int e = tid; e < DK * 16; e += BRING)
                cp16(st + (e >> 4) * LD + (e & 15) * 4, a + e * 4, true);
#pragma unroll 8
            for (int e = tid; e < CH * DK / 4; e += BRING)
                cp16(st + DK * LD + e / (DK / 4) * W + e % (DK / 4) * 4, b + e * 4, true);
            cp_commit();
            cp_wait<0>();
            __threadfence_block();
            bar_arrive(3 + (n & 1), SIDE + BRING);
            bar_arrive(5 + (n & 1), SIDE + BRING);
        }
        pdl_trigger();
        return;
    }
    const int side = threadIdx.x >= SIDE, tid = threadIdx.x - side * SIDE;
    const int warp = tid >> 5, lane = tid & 31, rows0 = warp * 16;
    // [DK][PS]: the state before the chunk, of each 16 rows row r at r % 4 * 4 + r / 4
    float* ss = sh + 2 * STAGE + side * Pass<DK>::OWN;
    float* us = ss + DK * PS;                                  // [CH][PS], token t at place(t)
    float* red = us + CH * PS;                                 // [WARPS][CH][PS], likewise
    // place(t) = t % 4 * 16 + t / 4: what lanes side by side write or read lies side by side
    const int j0 = blockIdx.z * PC + side * PS;
    // for u: 16 groups of four tokens by two of four columns
    const int tg = (lane & 1) | ((lane >> 1) & 14), j4 = ((lane >> 1) & 1) * 4;
    // for S: four groups of four rows by two of four columns, and of 16 tokens four; the sums over the
    // tokens meet, and a thread keeps four columns of one row
    const int c4 = rows0 + ((lane & 1) | ((lane >> 1) & 2)) * 4, part = lane >> 3;
    const int row = c4 + (lane >> 4) * 2 + ((lane >> 3) & 1);
    const int row_place = rows0 + ((row & 3) * 4 + ((row & 15) >> 2));
    // u's tokens: half of the warps' parts each on lanes 16 apart
    const int e = warp * 16 + (lane & 15), upper = lane >> 4;
    float* slot = state + (size_t)seq_slot[p.seq] * slot_stride + (size_t)h * DK * dv + j0;
    float4 S = four(slot + (size_t)row * dv + j4);
    for (int n = 0; n < p.chunks; ++n) {
        const size_t where = (size_t)(p.first + n) * H + h;
        const float b = bn[where * DK + row];
        float4 u[CH * PS / 4 / (WARPS * 16)];
#pragma unroll
        for (int i = 0; i < CH * PS / 4 / (WARPS * 16); ++i) {
            const int at = e + i * WARPS * 16, t = (at >> 1) % 16 * 4 + (at >> 5);
            u[i] = four(xv + (where * CH + t) * dv + j0 + (at & 1) * 4);
        }
        *reinterpret_cast<float4*>(states + (where * DK + row) * dv + j0 + j4) = S;
        *reinterpret_cast<float4*>(ss + row_place * PS + j4) = S;
        bar_sync(3 + 2 * side + (n & 1), SIDE + BRING);        // the chunk has landed, S0 is written
        const float* st = sh + (n & 1) * STAGE;
        {
            // X_k S0 over this warp's rows of the state
            unsigned long long acc[4][2];
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = 0ull;
            const float* xa = st + rows0 * LD + tg * 4;
            const float* sb = ss + rows0 * PS + j4;
#pragma unroll
            for (int c = 0; c < 16; ++c) {
                const float4 t = four(xa + c * LD), y = four(sb + (c % 4 * 4 + c / 4) * PS);
                const float v[4] = {t.x, t.y, t.z, t.w};
                const unsigned long long y0 = pair(y.x, y.y), y1 = pair(y.z, y.w);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const unsigned long long vv = pair(v[i], v[i]);
                    fma2(acc[i][0], vv, y0);
                    fma2(acc[i][1], vv, y1);
                }
            }
            float* rd = red + (warp * CH + tg) * PS + j4;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float4 r;
                unpair(acc[i][0], r.x, r.y);
                unpair(acc[i][1], r.z, r.w);
                *reinterpret_cast<float4*>(rd + i * 16 * PS) = r;
            }
        }
        bar_sync(1 + side, SIDE);
#pragma unroll
        for (int i = 0; i < CH * PS / 4 / (WARPS * 16); ++i) {
            const int at = e + i * WARPS * 16, t = (at >> 1) % 16 * 4 + (at >> 5);
            const float* from = red + upper * (WARPS / 2) * CH * PS + at * 4;
            float4 sum = four(from);
#pragma unroll
            for (int w = 1; w < WARPS / 2; ++w) {
                const float4 r = four(from + w * CH * PS);
                sum.x += r.x; sum.y += r.y; sum.z += r.z; sum.w += r.w;
            }
            sum.x += __shfl_xor_sync(0xffffffffu, sum.x, 16);
            sum.y += __shfl_xor_sync(0xffffffffu, sum.y, 16);
            sum.z += __shfl_xor_sync(0xffffffffu, sum.z, 16);
            sum.w += __shfl_xor_sync(0xffffffffu, sum.w, 16);
            const float4 out = make_float4(u[i].x - sum.x, u[i].y - sum.y, u[i].z - sum.z, u[i].w - sum.w);
            *reinterpret_cast<float4*>(upper ? xv + (where * CH + t) * dv + j0 + (at & 1) * 4
                                             : us + at * 4) = out;
        }
        bar_sync(1 + side, SIDE);
        {
            // S <- diag(b_n) S + sum over the tokens of kh u
            unsigned long long acc[4][2];
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = 0ull;
            const float* ka = st + DK * LD + part * 4 * W + c4;
            const float* ub = us + part * PS + j4;
#pragma unroll
            for (int s16 = 0; s16 < 4; ++s16)                  // tokens 16 s16 + 4 part + i
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 kk = four(ka + (s16 * 16 + i) * W);
                    const float4 y = four(ub + (i * 16 + s16 * 4) * PS);
                    const float v[4] = {kk.x, kk.y, kk.z, kk.w};
                    const unsigned long long y0 = pair(y.x, y.y), y1 = pair(y.z, y.w);
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const unsigned long long vv = pair(v[r], v[r]);
                        fma2(acc[r][0], vv, y0);
                        fma2(acc[r][1], vv, y1);
                    }
                }
            if (n + 2 < p.chunks) bar_arrive(7 + 2 * side + (n & 1), SIDE + BRING);
            float d[4][4], two[2][4], one[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                unpair(acc[r][0], d[r][0], d[r][1]);
                unpair(acc[r][1], d[r][2], d[r][3]);
            }
            const bool q = lane & 16, o = lane & 8;
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int x = 0; x < 4; ++x)
                    two[r][x] = (q ? d[2 + r][x] : d[r][x]) +
                                __shfl_xor_sync(0xffffffffu, q ? d[r][x] : d[2 + r][x], 16);
#pragma unroll
            for (int x = 0; x < 4; ++x)
                one[x] = (o ? two[1][x] : two[0][x]) +
                         __shfl_xor_sync(0xffffffffu, o ? two[0][x] : two[1][x], 8);
            S.x = fmaf(b, S.x, one[0]);
            S.y = fmaf(b, S.y, one[1]);
            S.z = fmaf(b, S.z, one[2]);
            S.w = fmaf(b, S.w, one[3]);
        }
    }
    pdl_trigger();
    *reinterpret_cast<float4*>(slot + (size_t)row * dv + j4) = S;
}

// ------------------------------------------------------------------------------------------
// The read-outs, both rules: out[t][j] = sum_c xt[c][t] S0[c][j] + sum_s pt[s][t] u_s[j].
// grid (items, H, dv / 64), 128 threads; steps of 32 through two stages.  u: rows of the step
// (u_by_item 0) or of the chunks' own rows [item][h][64][dv].  40 us on four blocks an SM, whose 1,024
// blocks are two rounds (steps of 64, three blocks: 43); the multiply-adds alone are 26.
// ------------------------------------------------------------------------------------------
template <typename VT>
__global__ void __launch_bounds__(128, 4)
chunk_out_kernel(const float* __restrict__ xt, const float* __restrict__ states,
                 const float* __restrict__ pt, const VT* __restrict__ u, int ldu, int u_by_item,
                 const Item* __restrict__ items, float* __restrict__ out, int H, int dk, int dv) {
    extern __shared__ __align__(16) float sh[];      // [2][2][32][LD]
    const Item it = items[blockIdx.x];
    const int h = blockIdx.y, j0 = blockIdx.z * 64;
    const size_t at = (size_t)blockIdx.x * H + h;
    const int of_state = dk / 32, steps = of_state + 2;
    pdl_wait();
    auto load = [&](int step) {
        float* a = sh + (step & 1) * 2 * 32 * LD;
        float* b = a + 32 * LD;
        if (step < of_state) {
            load_tile<32>(a, xt + (at * dk + step * 32) * CH, CH, 32);
            load_tile<32>(b, states + (at * dk + step * 32) * dv + j0, dv, 32);
        } else {
            const int s0 = (step - of_state) * 32;
            load_tile<32>(a, pt + (at * CH + s0) * CH, CH, 32);
            if (u_by_item) load_tile<32>(b, u + (at * CH + s0) * dv + j0, dv, it.count - s0);
            else load_tile<32>(b, u + (size_t)(it.token + s0) * ldu + h * dv + j0, ldu, it.count - s0);
        }
        cp_commit();
    };
    load(0);
    Tile tile;
    for (int step = 0; step < steps; ++step) {
        if (step + 1 < steps) load(step + 1);
        else cp_commit();
        cp_wait<1>();
        __syncthreads();
        const float* a = sh + (step & 1) * 2 * 32 * LD;
        // (the last 32 u say nothing to the first 32 tokens, which are the first two warps' rows)
        if (step + 1 < steps || threadIdx.x >= 64) tile.add<32>(a, a + 32 * LD);
        __syncthreads();
    }
    pdl_trigger();
    unsigned spoilt = 0;
    float* o = out + (size_t)it.token * (H * dv) + h * dv + j0 + tile.col;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int t = tile.row_of(i);
        const float4 v = tile.get(i);
        if (t >= it.count) continue;
        *reinterpret_cast<float4*>(o + (size_t)t * (H * dv)) = v;
        if (!(fmaf(v.x, 0.0f, fmaf(v.y, 0.0f, fmaf(v.z, 0.0f, v.w * 0.0f))) == 0.0f)) spoilt |= 1u << i;
    }
    // an infinity or NaN: a token's sums again, without the products of pt's zeros with the u of later
    // tokens, which would spoil this one too
    for (int i = 0; spoilt != 0; ++i, spoilt >>= 1) {
        if (!(spoilt & 1u)) continue;
        const int t = tile.row_of(i);
        for (int e = 0; e < 4; ++e) {
            const int j = j0 + tile.col + e;
            float r = 0.0f;
            for (int c = 0; c < dk; ++c)
                r = fmaf(xt[(at * dk + c) * CH + t], states[(at * dk + c) * dv + j], r);
            for (int s = 0; s <= t; ++s)
                r = fmaf(pt[(at * CH + s) * CH + t],
                         to_float(u_by_item ? u[(at * CH + s) * dv + j]
                                            : u[(size_t)(it.token + s) * ldu + h * dv + j]), r);
            o[(size_t)t * (H * dv) + e] = r;
        }
    }
}

}  // namespace

DE_EXPORT int de_chunk_tokens() { return CH; }

// Whether portions of these sizes go by chunks: the state's rows are 64 or 128 key channels and its
// columns whole tiles of 64.
DE_EXPORT int de_chunk_ok(int dk, int dv) { return (dk == 64 || dk == 128) && dv > 0 && dv % 64 == 0; }

static int need_smem(const void* kernel, size_t bytes) {
    return bytes > 48 * 1024
               ? (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)bytes)
               : 0;
}

// The read-outs and the new states of the portions in `items` / `portions` under a decay per head,
// `group` items at a time (a portion that is cut goes on from the state that the group before it left:
// the same bits).  work, for a group of m: m H (64 dk + 64 64 + dk dv) floats, xt [m, H, dk, 64], pt
// [m, H, 64, 64] and the states [m, H, dk, dv].
DE_EXPORT int de_decay_chunks(int v_dtype, const float* q, int ldq, const float* k, int ldk,
                              const void* v, int ldv, const float* decay, const int* items,
                              int n_items, const int* portions, int n_portions, float* work,
                              int group, float* state, long long slot_stride, const int* seq_slot,
                              float* out, int H, int dk, int dv, void* stream) {
    if (n_items <= 0 || n_portions <= 0) return 0;
    if (!de_chunk_ok(dk, dv) || ldk % 4 || ldv % 4 || (uintptr_t)k % 16 ||
        (uintptr_t)v % (v_dtype == DE_BF16 ? 8 : 16) || slot_stride % 4 || (uintptr_t)state % 16 ||
        (uintptr_t)work % 16 || group <= 0)
        return -2;
    cudaStream_t s = (cudaStream_t)stream;
    const Portion* po = (const Portion*)portions;
    const size_t psmem = (size_t)2 * 64 * LD * sizeof(float);
    const size_t osmem = (size_t)4 * 32 * LD * sizeof(float);
    const dim3 pgrid(n_portions, (H * dk * dv / 4 + 255) / 256);
    int e;
#define RUN(...)                                                                                \
    do {                                                                                        \
        if ((e = (__VA_ARGS__)) != 0) return e;                                                 \
    } while (0)
    for (int begin = 0; begin < n_items; begin += group) {
        const int m = n_items - begin < group ? n_items - begin : group;
        const Item* it = (const Item*)items + begin;
        const size_t mh = (size_t)m * H;
        float* xt = work;
        float* pt = xt + mh * dk * CH;
        float* states = pt + mh * CH * CH;
        if (dk == 64) {
            RUN(need_smem((const void*)decay_products_kernel<64>, psmem));
            RUN(de_launch(decay_products_kernel<64>, dim3(m, H), dim3(128), psmem, s, q, ldq, k, ldk,
                          decay, it, xt, pt, H));
        } else {
            RUN(need_smem((const void*)decay_products_kernel<128>, psmem));
            RUN(de_launch(decay_products_kernel<128>, dim3(m, H), dim3(128), psmem, s, q, ldq, k,
                          ldk, decay, it, xt, pt, H));
        }
        const dim3 grid(m, H, dk / 64 * (dv / 64)), ogrid(m, H, dv / 64);
        if (v_dtype == DE_BF16)
            RUN(de_launch(decay_states_kernel<__nv_bfloat16>, grid, dim3(128), 0, s, k, ldk,
                          (const __nv_bfloat16*)v, ldv, decay, it, states, H, dk, dv));
        else
            RUN(de_launch(decay_states_kernel<float>, grid, dim3(128), 0, s, k, ldk,
                          (const float*)v, ldv, decay, it, states, H, dk, dv));
        RUN(de_launch(decay_pass_kernel, pgrid, dim3(256), 0, s, states, decay, it, po, begin, m,
                      state, slot_stride, seq_slot, H, dk * dv));
        if (v_dtype == DE_BF16) {
            RUN(need_smem((const void*)chunk_out_kernel<__nv_bfloat16>, osmem));
            RUN(de_launch(chunk_out_kernel<__nv_bfloat16>, ogrid, dim3(128), osmem, s, xt, states, pt,
                          (const __nv_bfloat16*)v, ldv, 0, it, out, H, dk, dv));
        } else {
            RUN(need_smem((const void*)chunk_out_kernel<float>, osmem));
            RUN(de_launch(chunk_out_kernel<float>, ogrid, dim3(128), osmem, s, xt, states, pt,
                          (const float*)v, ldv, 0, it, out, H, dk, dv));
        }
    }
    return 0;
}

// The same for the delta rule: g [N, ldg] decays, beta [N, ldb], v float32.  work, for a group of m:
// m H (2 64 64 + 4 64 dk + dk + 64 dv + dk dv) floats, at and pt [m, H, 64, 64], xt, kd, kh, xkt
// [m, H, dk, 64], the states [m, H, dk, dv], xv [m, H, 64, dv] and bn [m, H, dk].
DE_EXPORT int de_delta_chunks(const float* q, int ldq, const float* k, int ldk, const float* v,
                              int ldv, const float* g, int ldg, const float* beta, int ldb,
                              const int* items, int n_items, const int* portions, int n_portions,
                              float* work, int group, float* state, long long slot_stride,
                              const int* seq_slot, float* out, int H, int rep, int dk, int dv,
                              void* stream) {
    if (n_items <= 0 || n_portions <= 0) return 0;
    if (!de_chunk_ok(dk, dv) || ldq % 4 || ldk % 4 || ldg % 4 || ldv % 2 || (uintptr_t)q % 16 ||
        (uintptr_t)k % 16 || (uintptr_t)g % 16 || (uintptr_t)v % 8 || slot_stride % 4 ||
        (uintptr_t)state % 16 || (uintptr_t)work % 16 || rep <= 0 || H % rep || group <= 0)
        return -2;
    cudaStream_t s = (cudaStream_t)stream;
    const Portion* po = (const Portion*)portions;
    const size_t csmem = (size_t)3 * CH * (dk + 4) * sizeof(float);
    const size_t ssmem = (size_t)(CH * LD + CH * 128) * sizeof(float);
    const size_t osmem = (size_t)4 * 32 * LD * sizeof(float);
    const dim3 pgrid(n_portions, H, dv / PC);
    int e;
#define DELTA(DK)                                                                               \
    do {                                                                                        \
        RUN(need_smem((const void*)delta_chunk_kernel<DK>, csmem));                     \
        RUN(de_launch(delta_chunk_kernel<DK>, dim3(m, H), dim3(256), csmem, s, q, ldq, k, ldk,  \
                      g, ldg, it, at, pt, xt, kd, kh, bn, H, rep));                             \
        RUN(need_smem((const void*)delta_solve_kernel<DK>, ssmem));                     \
        RUN(de_launch(delta_solve_kernel<DK>, sgrid, dim3(64), ssmem, s, (const float*)at, v,   \
                      ldv, (const float*)kd, beta, ldb, it, xv, xkt, H, dv));                   \
        RUN(need_smem((const void*)delta_pass_kernel<DK>, Pass<DK>::SMEM));             \
        RUN(de_launch(delta_pass_kernel<DK>, pgrid, dim3(Pass<DK>::THREADS), Pass<DK>::SMEM, s, \
                      (const float*)xkt, (const float*)kh, (const float*)bn, xv, states, po,    \
                      begin, m, state, slot_stride, seq_slot, H, dv));                          \
    } while (0)
    for (int begin = 0; begin < n_items; begin += group) {
        const int m = n_items - begin < group ? n_items - begin : group;
        const Item* it = (const Item*)items + begin;
        const size_t mh = (size_t)m * H, turned = mh * dk * CH;
        float* at = work;
        float* pt = at + mh * CH * CH;
        float* xt = pt + mh * CH * CH;
        float* kd = xt + turned;
        float* kh = kd + turned;
        float* xkt = kh + turned;
        float* states = xkt + turned;
        float* xv = states + mh * dk * dv;
        float* bn = xv + mh * CH * dv;
        const dim3 sgrid(m, H, (dv + dk + 127) / 128);
        if (dk == 64) DELTA(64);
        else DELTA(128);
        RUN(need_smem((const void*)chunk_out_kernel<float>, osmem));
        RUN(de_launch(chunk_out_kernel<float>, dim3(m, H, dv / 64), dim3(128), osmem, s,
                      (const float*)xt, (const float*)states, (const float*)pt, (const float*)xv, 0,
                      1, it, out, H, dk, dv));
    }
    return 0;
}
