// What the kernels of attention with 32-bit scores and weights share (attention_chunk.cu,
// attention_chunk_tcgen05.cu): which keys a row sees, its scores, the walk over tiles of keys, and a
// row formed again on the CUDA cores.
#pragma once

#include "common.cuh"

namespace {

constexpr int TILE = 32;          // keys of a tile of the kernels on the CUDA cores

struct WorkItem {
    int seq, row0, kv_begin, kv_end, partial, pad0, pad1, pad2;
};

// Which keys a row sees besides j <= i, and what happens to its scores.
struct Sight {
    int chunk;          // > 0: keys of the row's own chunk of positions only
    int window;         // > 0: the last `window` keys only ...
    int keep_first;     // ... and the first `keep_first` keys of the sequence
    float softcap;      // > 0: score <- softcap * tanh(score / softcap)
    int v_stride;       // elements from one key's values to the next in v_pages: dv, or the key
                        // size where the values are the first dv features of the key rows
    int linear;         // the distance penalty is r1[h] * (i - j) instead of the logarithmic one
    const float* sink;  // [heads] or null: the softmax's denominator also holds exp(sink[h]), a
                        // weight without a key or a value (not scaled, no penalty)
    const void* gate;   // or null: a row's result is multiplied by sigmoid(gate) before it is
    int ld_gate;        // stored; gate of the queries' type, rows ld_gate apart, one number a
    int gate_per_head;  // feature ([heads dv]) or, with gate_per_head, one a head ([heads])
    float out_scale;    // every row's result is multiplied by this before it is stored
};
template <typename T>
__device__ __forceinline__ float sight_gate(const Sight& s, size_t token, int head, int dv,
                                            int feature) {
    if (s.gate == nullptr) return 1.0f;
    const T* g = (const T*)s.gate + token * s.ld_gate + (s.gate_per_head ? head : head * dv + feature);
    return 1.0f / (1.0f + expf(-to_float(*g)));
}
// out_scale / (the row's sum of weights, with the sink's share): m is the row's reference maximum
__device__ __forceinline__ float sight_inverse(const Sight& s, int head, float m, float l) {
    if (s.sink != nullptr) l += expf(s.sink[head] - m);
    return l > 0.0f ? s.out_scale / l : 0.0f;
}

// first key of the near range of a row at `pos` (does not fall as pos grows)
__device__ __forceinline__ int sight_lo(const Sight& m, int pos) {
    int lo = 0;
    if (m.chunk > 0) lo = pos / m.chunk * m.chunk;
    if (m.window > 0) lo = max(lo, pos - m.window + 1);
    return lo;
}
// keys [0, this) are seen as well
__device__ __forceinline__ int sight_first(const Sight& m, int lo) {
    return (m.window > 0 && m.keep_first > 0) ? min(m.keep_first, lo) : 0;
}
__device__ __forceinline__ float sight_score(const Sight& m, float s, float scale, float pen1,
                                             float pen2, bool penalty, float dist) {
    s *= scale;
    if (penalty) s -= m.linear ? pen1 * dist : pen1 * log1pf(pen2 * dist);
    if (m.softcap > 0.0f) s = m.softcap * tanhf(s / m.softcap);
    return s;
}
// The tiles a block walks: those of the kept first keys [0, kf), then from the tile of `lo` on.
struct TileWalk {
    int start, jump_at, jump_to;
    __device__ __forceinline__ TileWalk(int lo, int kf, int tile) {
        const int near = (lo / tile) * tile, first_end = ((kf + tile - 1) / tile) * tile;
        start = kf > 0 ? 0 : near;
        jump_at = (kf > 0 && first_end < near) ? first_end : -1;
        jump_to = near;
    }
    __device__ __forceinline__ int next(int kt, int tile) const {
        const int n = kt + tile;
        return n == jump_at ? jump_to : n;
    }
};
template <typename T>
__device__ __forceinline__ void store_out(void* out, int out_f32, size_t at, float x) {
    if (out_f32) ((float*)out)[at] = x;
    else ((T*)out)[at] = from_float<T>(x);
}

// 16 bytes as floats
__device__ __forceinline__ void load_piece(const float* p, float* f) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
}
__device__ __forceinline__ void load_piece(const __nv_bfloat16* p, float* f) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f[2 * i] = __uint_as_float(w[i] << 16);
        f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}

// A row formed again, as attn_chunk_kernel forms it (features and keys in ascending order, keys of
// weight 0 skipped), by one warp straight from the pages: for rows in which the products on the
// tensor cores met an infinity or NaN.  A weight of 0 times such a value is NaN there, so that a
// value that the row does not see would spoil it, and an infinite value meets lower terms of a
// weight that are 0.  q: the row's D query features; a lane returns features lane, lane + 32, ...
// Rows without such values pay for the look at their results: 0 to 0.25 us a launch, up to 3 %.
template <int D, typename Q>
__device__ __forceinline__ void row_again(
    const Q* q, const __nv_bfloat16* k_pages, const __nv_bfloat16* v_pages, const int* table,
    int num_pages, int hk, int kv_heads, int page, int pos, int kv_begin, int kv_end, float scale,
    float pen1, float pen2, bool penalty, const Sight& sight, float& m_out, float& l_out,
    float (&acc)[D / 32]) {
    const int lane = threadIdx.x & 31;
    const int lo = max(kv_begin, sight_lo(sight, pos)), hi = min(kv_end, pos + 1);
    const int first = kv_begin > 0 ? 0 : sight_first(sight, lo);
    const TileWalk walk(lo, first, TILE);
    float m = -INFINITY, l = 0.0f;
#pragma unroll
    for (int i = 0; i < D / 32; ++i) acc[i] = 0.0f;
    for (int kt = walk.start; kt < hi; kt = walk.next(kt, TILE)) {
        const int kpos = kt + lane;
        bool valid = (kpos >= lo || kpos < first) && kpos < hi;
        long long at = 0;
        if (valid) {
            const int id = table[kpos / page];
            valid = id >= 0 && id < num_pages;
            if (valid) at = ((long long)id * kv_heads + hk) * page + kpos % page;
        }
        float s = 0.0f;
        if (valid) {
            for (int i = 0; i < D; i += 8) {
                float k[8];
                load_piece(k_pages + at * D + i, k);
#pragma unroll
                for (int e = 0; e < 8; ++e) s = fmaf(to_float(q[i + e]), k[e], s);
            }
            s = sight_score(sight, s, scale, pen1, pen2, penalty, (float)(pos - kpos));
        } else {
            s = -INFINITY;
        }
        const float m_new = fmaxf(m, warp_max(s));
        if (m_new == -INFINITY) continue;
        const float p = valid ? expf(s - m_new) : 0.0f;
        const float corr = expf(m - m_new);
        l = l * corr + warp_sum(p);
#pragma unroll
        for (int i = 0; i < D / 32; ++i) acc[i] *= corr;
        for (int j = 0; j < TILE; ++j) {
            const float pj = __shfl_sync(0xffffffffu, p, j);
            const long long row = __shfl_sync(0xffffffffu, at, j);
            if (pj == 0.0f) continue;
#pragma unroll
            for (int i = 0; i < D / 32; ++i)
                acc[i] = fmaf(pj, to_float(v_pages[row * sight.v_stride + lane + 32 * i]), acc[i]);
        }
        m = m_new;
    }
    m_out = m;
    l_out = l;
}

// tanh(x) for |x| <= TANH_NEAR to 7e-8 of its value (as good as tanhf and a third of its
// instructions): x + x^3 P(x^2), P of degree 4 fitted to tanh at Chebyshev nodes by reweighted
// least squares (3e-9 but for float32's rounding).  Scores under a cap mostly lie here; the others
// take tanhf of the quotient, as in the kernels above.
constexpr float TANH_NEAR = 0.6f;
__device__ __forceinline__ float tanh_near(float x) {
    const float u = x * x;
    float p = fmaf(u, -0.00589515036f, 0.0207959637f);
    p = fmaf(u, p, -0.0537838265f);
    p = fmaf(u, p, 0.133319244f);
    p = fmaf(u, p, -0.333332986f);
    return fmaf(x * u, p, x);
}

}  // namespace
