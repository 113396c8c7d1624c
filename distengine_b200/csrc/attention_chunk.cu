// Softmax attention inside chunks of positions, over the paged cache, with a penalty that grows
// with the logarithm of the distance, keys and values of different sizes, and values that are
// cached normalised.  Scores, the penalty, the softmax weights and the weighted sum of the values are
// all 32-bit, for float32 or bfloat16 storage: on the CUDA cores, or for bfloat16 rows of 64 and 128
// features on the tensor cores with the weights as three bfloat16 terms.
//
//   score(i, j) = (q_i . k_j) * scale - r1[h] * log(1 + r2[h] * (i - j))
//   token i sees key j when j <= i and floor(i / chunk) = floor(j / chunk)   (chunks of positions
//   counted from 0 of the sequence, whatever portion of it a step brings)
//
// A row is (token, query head within its kv head's group); a block takes a tile of 8 rows of one
// sequence and one kv head, a warp a row, a lane a key of the current tile of 32 keys.  Tiles of
// keys lie at absolute multiples of 32 and a row walks the tiles of its chunk in ascending order,
// so a row's result does not depend, bit for bit, on what shares its tile.  The kernels below for other
// sizes, longer portions, single tokens and the tensor cores each sum in an order of their own; which
// one takes a row depends on its step (on how many rows the step's portions have and, for bfloat16
// rows of 64 and 128 features, how many single tokens there are).
// The host's work items are those of the other attention kernels (kernels/attention_plan.py),
// unsplit: a chunk bounds every key range.
//
// The same kernels also serve attention whose keys are bounded by a sliding window that keeps the
// first tokens of the sequence, with a soft cap on the scores (`Sight`):
//
//   token i sees key j when j <= i and (i - j < window or j < keep_first)
//   score <- softcap * tanh(score / softcap)
//
// A block then walks the tiles of the kept first keys and jumps to the tile in which its rows'
// windows begin.  r1 / r2 null: no distance penalty.  `out_f32`: the rows' results are written as
// float32 (for a kernel that turns them by position or gates them before they are rounded).
//
// Three more parameters of `Sight` serve attention whose softmax has a sink: a distance penalty
// that is linear, r1[h] * (i - j); `sink` [heads], a learned score per head that joins the
// denominator as exp(sink[h]) without a key or a value (it is added once, when a row's sums are
// complete, whatever the tiles and the step's cut); and `gate`, sigmoid of which multiplies a
// row's result in float32 before it is stored (one number a feature or one a head); `out_scale` is
// one more factor of every result, for a mixer whose result joins another's.  qkv_prepare
// is what stands between such a mixer's projection and these kernels (bias, a short convolution
// over time with the slot's kept rows, norms, rotation, value mixing, the cache write), and
// conv_keep moves the kept rows on.

#include "attention_sight.cuh"

DE_DEFINE_PDL_SWITCH

namespace {

constexpr int ROWS = 8;
constexpr int MAX_D = 256;        // of a value: the weighted sums live in registers
constexpr int MAX_DK = 576;       // of a key: shared memory only

// k copied, v divided by its root mean square over the head (eps inside the root), both into the
// pages.  proj row = [... | k (G dk) | v (G dv)] from column k_col on.  grid (tokens, kv heads).
template <typename T>
__global__ void kv_write_normed_kernel(const T* __restrict__ proj, int ld, int k_col,
                                       const int* __restrict__ positions,
                                       const int* __restrict__ token_slot, int G, int dk, int dv,
                                       float eps, T* __restrict__ k_pages, T* __restrict__ v_pages,
                                       const int* __restrict__ block_table, int table_stride,
                                       int page, int num_pages, int* __restrict__ status) {
    __shared__ float scratch[33];
    const int n = blockIdx.x, hk = blockIdx.y;
    const int pos = positions[n], slot = token_slot[n];
    pdl_wait();
    const int page_id = block_table[(size_t)slot * table_stride + pos / page];
    const T* ks = proj + (size_t)n * ld + k_col + hk * dk;
    const T* vs = proj + (size_t)n * ld + k_col + G * dk + hk * dv;
    float ss = 0.0f;
    for (int i = threadIdx.x; i < dv; i += blockDim.x) {
        const float x = to_float(vs[i]);
        ss = fmaf(x, x, ss);
    }
    const float inv = 1.0f / sqrtf(block_sum(ss, scratch) / (float)dv + eps);
    pdl_trigger();
    if (page_id < 0 || page_id >= num_pages) {       // never written outside the pool
        if (threadIdx.x == 0) atomicExch(status, 1);
        return;
    }
    const size_t at = ((size_t)page_id * G + hk) * page + (size_t)(pos % page);
    for (int i = threadIdx.x; i < dk; i += blockDim.x) k_pages[at * dk + i] = ks[i];
    for (int i = threadIdx.x; i < dv; i += blockDim.x)
        v_pages[at * dv + i] = from_float<T>(to_float(vs[i]) * inv);
}

// four neighbouring features in one load
__device__ __forceinline__ float4 load_four(const float* p) {
    return *reinterpret_cast<const float4*>(p);
}
__device__ __forceinline__ float4 load_four(const __nv_bfloat16* p) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u),
                       __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
}
// two in one store
__device__ __forceinline__ void store_pair(float* p, float a, float b) {
    *reinterpret_cast<float2*>(p) = make_float2(a, b);
}
__device__ __forceinline__ void store_pair(__nv_bfloat16* p, float a, float b) {
    *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(a, b);
}
// and four
__device__ __forceinline__ void store_four(float* p, const float4& v) {
    *reinterpret_cast<float4*>(p) = v;
}
__device__ __forceinline__ void store_four(__nv_bfloat16* p, const float4& v) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const unsigned*>(&a),
                                              *reinterpret_cast<const unsigned*>(&b));
}

// Queries and keys turned by position, values turned by position over all their features, keys
// and values into the pages.  proj row = [q (H dk) | k (G dk) | v (G dv) | ...] (a run that reads
// another run's cache has q only: write_kv 0).  Pairs are (i, i + n/2) of the first n features:
// n = rot with the angles pos * fk[i] for q and k, n = dv with pos * fv[i] for v (fv null: values
// are stored as they are).  q is turned in place.  One block a token.
template <typename T>
__global__ void kv_write_rotated_kernel(T* __restrict__ proj, int ld, const int* __restrict__ positions,
                                        const int* __restrict__ token_slot,
                                        const float* __restrict__ fk, int rot,
                                        const float* __restrict__ fv, int H, int G, int dk, int dv,
                                        T* __restrict__ k_pages, T* __restrict__ v_pages,
                                        const int* __restrict__ block_table, int table_stride,
                                        int page, int num_pages, int write_kv,
                                        int* __restrict__ status) {
    const int n = blockIdx.x;
    const int pos = positions[n];
    const float fpos = (float)pos;
    T* row = proj + (size_t)n * ld;
    const int half = rot / 2, per = dk - half;       // work items a head: pairs, then plain features
    size_t at = 0;
    bool can_write = write_kv != 0;
    if (can_write) {
        const int page_id = block_table[(size_t)token_slot[n] * table_stride + pos / page];
        if (page_id < 0 || page_id >= num_pages) {   // never written outside the pool
            if (threadIdx.x == 0) atomicExch(status, 1);
            can_write = false;
        }
        at = ((size_t)page_id * G) * page + (size_t)(pos % page);
    }
    pdl_wait();
    const int qk_heads = H + (write_kv ? G : 0);
    for (int idx = threadIdx.x; idx < qk_heads * per; idx += blockDim.x) {
        const int h = idx / per, i = idx - h * per;
        T* src = row + h * dk;
        T* dst = src;                                // q in place
        if (h >= H) {
            if (!can_write) continue;
            dst = k_pages + (at + (size_t)(h - H) * page) * dk;
        }
        if (i < half) {
            float sn, cs, ra, rb;
            sincosf(fpos * fk[i], &sn, &cs);
            rope_rotate(to_float(src[i]), to_float(src[i + half]), cs, sn, ra, rb);
            dst[i] = from_float<T>(ra);
            dst[i + half] = from_float<T>(rb);
        } else if (h >= H) {
            dst[i + half] = src[i + half];
        }
    }
    if (can_write) {
        const T* vs = row + (H + G) * dk;
        if (fv != nullptr) {
            const int vhalf = dv / 2, vper = dv - vhalf;
            for (int idx = threadIdx.x; idx < G * vper; idx += blockDim.x) {
                const int h = idx / vper, i = idx - h * vper;
                const T* src = vs + h * dv;
                T* dst = v_pages + (at + (size_t)h * page) * dv;
                if (i < vhalf) {
                    float sn, cs, ra, rb;
                    sincosf(fpos * fv[i], &sn, &cs);
                    rope_rotate(to_float(src[i]), to_float(src[i + vhalf]), cs, sn, ra, rb);
                    dst[i] = from_float<T>(ra);
                    dst[i + vhalf] = from_float<T>(rb);
                } else {
                    dst[i + vhalf] = src[i + vhalf];
                }
            }
        } else {
            for (int idx = threadIdx.x; idx < G * dv; idx += blockDim.x) {
                const int h = idx / dv, i = idx - h * dv;
                v_pages[(at + (size_t)h * page) * dv + i] = vs[idx];
            }
        }
    }
    pdl_trigger();
}

// a token's cosines and sines of one list of frequencies, [half] each (as every head would form them)
__device__ __forceinline__ void angles(float* tab, const float* __restrict__ freq, int half, float pos) {
    for (int i = threadIdx.x; i < half; i += blockDim.x)
        sincosf(pos * freq[i], tab + half + i, tab + i);
}
// E (4 or 8) neighbouring features, in 16-byte pieces (four of bfloat16: 8 bytes)
template <int E, typename T> __device__ __forceinline__ void load_features(const T* p, float (&v)[E]) {
    if constexpr (E == 8 && sizeof(T) == 2) {
        const uint4 u = *reinterpret_cast<const uint4*>(p);
        const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int i = 0; i < E; ++i)
            v[i] = __uint_as_float(i & 1 ? w[i / 2] & 0xffff0000u : w[i / 2] << 16);
    } else {
#pragma unroll
        for (int i = 0; i < E; i += 4) {
            const float4 f = load_four(p + i);
            v[i] = f.x; v[i + 1] = f.y; v[i + 2] = f.z; v[i + 3] = f.w;
        }
    }
}
template <int E, typename T> __device__ __forceinline__ void store_features(T* p, const float (&v)[E]) {
    if constexpr (E == 8 && sizeof(T) == 2) {
        __nv_bfloat162 w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(w);
    } else {
#pragma unroll
        for (int i = 0; i < E; i += 4) store_four(p + i, make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]));
    }
}
// E neighbouring pairs (i, i + half) of src turned into dst
template <int E, typename T>
__device__ __forceinline__ void turn_features(const T* src, T* dst, const float* tab, int half, int i) {
    float a[E], b[E], c[E], s[E], x[E], y[E];
    load_features<E>(src + i, a);
    load_features<E>(src + i + half, b);
    load_features<E>(tab + i, c);
    load_features<E>(tab + half + i, s);
#pragma unroll
    for (int e = 0; e < E; ++e) rope_rotate(a[e], b[e], c[e], s[e], x[e], y[e]);
    store_features<E>(dst + i, x);
    store_features<E>(dst + i + half, y);
}

// The same in groups of E features, the token's angles formed once for all heads: where half the
// turned part, the plain part and the values' (half) rows are whole groups, and everything lies at
// such addresses.  2,048 tokens, 16 + 4 heads of 128, a product before it: 6.0 us in groups of eight, 7.4
// in groups of four (cold 13, and 23 with each head forming its angles).  In bfloat16 the values go with
// queries and keys in one pass over all groups, so that most threads have one (6.0 against 7.4 in two
// passes, in groups of four at rot 120 7.35 and 7.8); in float32, several a thread, two passes are the
// sooner ones (rot 64: 7.9 and 8.4).
template <typename T, int E>
__global__ void kv_write_rotated_vec_kernel(
    T* __restrict__ proj, int ld, const int* __restrict__ positions,
    const int* __restrict__ token_slot, const float* __restrict__ fk, int rot,
    const float* __restrict__ fv, int H, int G, int dk, int dv, T* __restrict__ k_pages,
    T* __restrict__ v_pages, const int* __restrict__ block_table, int table_stride, int page,
    int num_pages, int write_kv, int* __restrict__ status) {
    __shared__ __align__(16) float ktab[MAX_D], vtab[MAX_D];
    const int n = blockIdx.x;
    const int pos = positions[n];
    T* row = proj + (size_t)n * ld;
    const int half = rot / 2, vhalf = dv / 2;
    size_t at = 0;
    bool can_write = write_kv != 0;
    if (can_write) {
        const int page_id = block_table[(size_t)token_slot[n] * table_stride + pos / page];
        if (page_id < 0 || page_id >= num_pages) {   // never written outside the pool
            if (threadIdx.x == 0) atomicExch(status, 1);
            can_write = false;
        }
        at = ((size_t)page_id * G) * page + (size_t)(pos % page);
    }
    angles(ktab, fk, half, (float)pos);
    if (can_write && fv != nullptr) angles(vtab, fv, vhalf, (float)pos);
    __syncthreads();
    pdl_wait();
    // groups of pairs, then plain groups, of queries and keys; then the values'
    const int per = (dk - half) / E, vper = (fv != nullptr ? vhalf : dv) / E;
    const int of_qk = (H + (can_write ? G : 0)) * per, of_v = can_write ? G * vper : 0;
    auto query_or_key = [&](int idx) {
        const int h = idx / per, i = (idx - h * per) * E;
        T* src = row + h * dk;
        T* dst = h < H ? src : k_pages + (at + (size_t)(h - H) * page) * dk;   // q in place
        if (i < half) {
            turn_features<E>(src, dst, ktab, half, i);
        } else if (h >= H) {
            float plain[E];
            load_features<E>(src + i + half, plain);
            store_features<E>(dst + i + half, plain);
        }
    };
    auto value = [&](int idx) {
        const int h = idx / vper, i = (idx - h * vper) * E;
        const T* src = row + (H + G) * dk + h * dv;
        T* dst = v_pages + (at + (size_t)h * page) * dv;
        if (fv != nullptr) {
            turn_features<E>(src, dst, vtab, vhalf, i);
        } else {
            float plain[E];
            load_features<E>(src + i, plain);
            store_features<E>(dst + i, plain);
        }
    };
    if constexpr (sizeof(T) == 2) {
        for (int idx = threadIdx.x; idx < of_qk + of_v; idx += blockDim.x) {
            if (idx < of_qk) query_or_key(idx);
            else value(idx - of_qk);
        }
    } else {
        for (int idx = threadIdx.x; idx < of_qk; idx += blockDim.x) query_or_key(idx);
        for (int idx = threadIdx.x; idx < of_v; idx += blockDim.x) value(idx);
    }
    pdl_trigger();
}

// What lies between a mixer's stacked projection and its attention, for mixers that do more to
// q, k and v than turn them: proj row = [q (H dk) | k (G dk) | v (G dv) | ...], C = (H + G) dk +
// G dv channels.  In this order, each step optional:
//   bias      u = proj + bias[c]
//   taps      a short causal convolution over time on every channel, y_t = sum_j taps[c][j] *
//             u_(t - K + 1 + j), zeros before the sequence's start; inputs before the step's first
//             token of the sequence come from the slot's state, kept[i] = projection (without
//             bias) at position pos0 - (K - 1) + i, as conv_keep leaves them; with keep_here (a
//             step in which every sequence brings one token, so no other block reads the
//             slot) the block moves the kept rows on itself and conv_keep is not needed
//   norm      q and k divided by their root mean square (eps inside the root) and weighted: 1 over
//             every head with weights [dk] that all heads share (or without weights: a turn keeps
//             a head's root mean square, so this is also the norm that follows the turn), 2 over
//             the whole projection with weights [H dk] and [G dk]
//   freq      the first `rot` features of every head of q and k turned by position, angle = pos *
//             freq[i] (reduced in double precision), cosine and sine times `magnitude`; pairs are
//             (2i, 2i + 1) with `adjacent`, else (i, i + rot / 2)
//   temp      q times 1 + temp_coef * ln(floor((pos + 1) / temp_every) + 1)
//   mix       1: the values (as they are cached) are also left in v_first [N, G dv];
//             2: v <- (1 - lambda) v + lambda v_first, lambda one number on the device
// With v_from_k the projection has no v columns, C = (H + G) dk, and a head's values are its keys
// as they stand before the norm and the turn (dv = dk).
// q goes to q_out [N, H dk] in the activation type, k and v into the pages.  All arithmetic is
// float32.  One block a token; shared memory: C + rot + H + G floats.
struct Prepare {
    const float* bias;
    const float* taps;
    int by_tap;                      // taps lie [K][C] at 16-byte addresses, as does the bias; else [C][K]
    int K;
    float* state;
    long long slot_stride;
    int conv_offset;
    int norm;
    const float* q_weight;
    const float* k_weight;
    float eps;
    const float* freq;
    int rot;
    float magnitude;
    int adjacent;
    float temp_coef;
    int temp_every;
    int mix;
    const float* lambda;
    float* v_first;
    int keep_here;
    int v_from_k;
};

// Two sums over a block at once; every thread gets both.  The order of the additions depends on
// the block's size only.
__device__ __forceinline__ void block_sum2(float& a, float& b, float* scratch /* 66 floats */) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int warps = (blockDim.x + 31) >> 5;
    a = warp_sum(a);
    b = warp_sum(b);
    if (lane == 0) {
        scratch[warp] = a;
        scratch[32 + warp] = b;
    }
    __syncthreads();
    if (warp < 2) {
        float t = lane < warps ? scratch[32 * warp + lane] : 0.0f;
        t = warp_sum(t);
        if (lane == 0) scratch[64 + warp] = t;
    }
    __syncthreads();
    a = scratch[64];
    b = scratch[65];
}

template <int PN> __device__ __forceinline__ void load_run(const float* p, int wide, float* f) {
    if (wide) {
#pragma unroll
        for (int e = 0; e < PN; e += 4) load_piece(p + e, f + e);
    } else {
#pragma unroll
        for (int e = 0; e < PN; ++e) f[e] = p[e];
    }
}

// VEC: the rows of proj are whole 16-byte pieces at 16-byte addresses and C is a whole number of
// pieces; a thread then takes the convolution of a piece's channels at once.  The sums are the
// same chains of multiply-adds either way.
// The taps come tap by tap (a lane's channels side by side): 2,402 tokens of 3,072 channels with
// four taps 44 us, 60 where a channel's taps lay together (32 lines a request).
// CONV: there are taps, more than one.  (A kernel of its own: without the convolution it needs 48
// registers, five blocks an SM, with it 54; 2,048 tokens of 16 + 4 heads of 128 without taps 26 us in
// one kernel for both, 23 so.)
template <typename T, bool VEC, bool CONV>
__global__ void qkv_prepare_kernel(const T* __restrict__ proj, int ld, T* __restrict__ q_out,
                                   const int* __restrict__ positions,
                                   const int* __restrict__ token_seq,
                                   const int* __restrict__ token_slot,
                                   const int* __restrict__ seq_pos0, Prepare pp, int H, int G,
                                   int dk, int dv, T* __restrict__ k_pages, T* __restrict__ v_pages,
                                   const int* __restrict__ block_table, int table_stride, int page,
                                   int num_pages, int* __restrict__ status) {
    extern __shared__ __align__(16) float sh[];
    __shared__ float scratch[66];
    const int n = blockIdx.x;
    const int qk = (H + G) * dk, C = pp.v_from_k ? qk : qk + G * dv, half = pp.rot / 2;
    const int v_col = pp.v_from_k ? H * dk : qk;     // where the values stand in sh
    float* cs_tab = sh + C;                          // [half] cosines, then [half] sines
    float* inv_s = cs_tab + pp.rot;                  // [H + G]
    const int pos = positions[n], slot = token_slot[n];
    const int off = pos - seq_pos0[token_seq[n]];    // the token's place in its sequence's portion
    const int page_id = block_table[(size_t)slot * table_stride + pos / page];
    const bool can_write = page_id >= 0 && page_id < num_pages;
    if (!can_write && threadIdx.x == 0) atomicExch(status, 1);   // never written outside the pool
    for (int i = threadIdx.x; i < half; i += blockDim.x) {
        // the angle in turns, its whole turns taken off in double precision: what is left, of up to
        // half a turn, keeps float32's digits
        const double turns = (double)pos * ((double)pp.freq[i] * 0.15915494309189535);
        float sn, cs;
        sincospif((float)(2.0 * (turns - rint(turns))), &sn, &cs);
        cs_tab[i] = cs * pp.magnitude;
        cs_tab[half + i] = sn * pp.magnitude;
    }
    pdl_wait();
    const T* row = proj + (size_t)n * ld;
    if (VEC && CONV) {
        constexpr int PN = 16 / (int)sizeof(T);
        const int K = pp.K;
        const float* kept = pp.state + (size_t)slot * pp.slot_stride + pp.conv_offset;
        for (int c0 = threadIdx.x * PN; c0 < C; c0 += blockDim.x * PN) {
            float acc[PN], b[PN];
#pragma unroll
            for (int e = 0; e < PN; ++e) acc[e] = b[e] = 0.0f;
            if (pp.bias) load_run<PN>(pp.bias + c0, pp.by_tap, b);
            for (int j = 0; j < K; ++j) {
                const int rel = off - (K - 1) + j;
                if (pos - (K - 1) + j < 0) continue;             // before the sequence's start
                float x[PN];
                if (rel >= 0) {
                    load_piece(proj + (size_t)(n - (K - 1) + j) * ld + c0, x);
                } else {
#pragma unroll
                    for (int e = 0; e < PN; ++e) x[e] = kept[(size_t)(off + j) * C + c0 + e];
                }
                float w[PN];
                if (pp.by_tap) {
                    load_run<PN>(pp.taps + (size_t)j * C + c0, 1, w);
                } else {
#pragma unroll
                    for (int e = 0; e < PN; ++e) w[e] = pp.taps[(c0 + e) * K + j];
                }
#pragma unroll
                for (int e = 0; e < PN; ++e) acc[e] = fmaf(w[e], x[e] + b[e], acc[e]);
            }
#pragma unroll
            for (int e = 0; e < PN; e += 4)
                store_four(sh + c0 + e, make_float4(acc[e], acc[e + 1], acc[e + 2], acc[e + 3]));
        }
    } else if (CONV) {
        const int K = pp.K;
        const float* kept = pp.state + (size_t)slot * pp.slot_stride + pp.conv_offset;
        for (int c = threadIdx.x; c < C; c += blockDim.x) {
            const float b = pp.bias ? pp.bias[c] : 0.0f;
            float acc = 0.0f;
            for (int j = 0; j < K; ++j) {
                const int rel = off - (K - 1) + j;
                if (pos - (K - 1) + j < 0) continue;             // before the sequence's start
                const float x = rel >= 0 ? to_float(proj[(size_t)(n - (K - 1) + j) * ld + c])
                                         : kept[(size_t)(off + j) * C + c];
                acc = fmaf(pp.taps[pp.by_tap ? j * C + c : c * K + j], x + b, acc);
            }
            sh[c] = acc;
        }
    } else if (VEC) {
        constexpr int PN = 16 / (int)sizeof(T);
        for (int c0 = threadIdx.x * PN; c0 < C; c0 += blockDim.x * PN) {
            float x[PN];
            load_piece(row + c0, x);
            if (pp.bias == nullptr && pp.taps == nullptr) {      // (C is a number of pieces)
#pragma unroll
                for (int e = 0; e < PN; e += 4)
                    store_four(sh + c0 + e, make_float4(x[e], x[e + 1], x[e + 2], x[e + 3]));
                continue;
            }
#pragma unroll
            for (int e = 0; e < PN; ++e) {
                x[e] += pp.bias ? pp.bias[c0 + e] : 0.0f;
                sh[c0 + e] = pp.taps != nullptr ? pp.taps[c0 + e] * x[e] : x[e];   // one tap
            }
        }
    } else {
        const float tap = pp.taps != nullptr ? 1.0f : 0.0f;     // a convolution of one tap
        for (int c = threadIdx.x; c < C; c += blockDim.x) {
            const float x = to_float(row[c]) + (pp.bias ? pp.bias[c] : 0.0f);
            sh[c] = tap != 0.0f ? pp.taps[c] * x : x;
        }
    }
    __syncthreads();
    if (CONV && pp.keep_here) {
        // every thread has read what it needs of the kept rows; a thread moves its channels on
        float* kept = pp.state + (size_t)slot * pp.slot_stride + pp.conv_offset;
        for (int c = threadIdx.x; c < C; c += blockDim.x) {
            for (int i = 0; i + 2 < pp.K; ++i) kept[(size_t)i * C + c] = kept[(size_t)(i + 1) * C + c];
            kept[(size_t)(pp.K - 2) * C + c] = to_float(row[c]);
        }
    }
    if (pp.norm == 1) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
        for (int h = warp; h < H + G; h += warps) {
            float ss = 0.0f;
            if (dk % 4 == 0) {
                for (int i = 4 * lane; i < dk; i += 128) {
                    const float4 v = *reinterpret_cast<const float4*>(sh + h * dk + i);
                    ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss))));
                }
            } else {
                for (int i = lane; i < dk; i += 32) ss = fmaf(sh[h * dk + i], sh[h * dk + i], ss);
            }
            ss = warp_sum(ss);
            if (lane == 0) inv_s[h] = 1.0f / sqrtf(ss / (float)dk + pp.eps);
        }
    } else if (pp.norm == 2) {
        float sq = 0.0f, sk = 0.0f;
        for (int i = threadIdx.x; i < H * dk; i += blockDim.x) sq = fmaf(sh[i], sh[i], sq);
        for (int i = H * dk + threadIdx.x; i < qk; i += blockDim.x) sk = fmaf(sh[i], sh[i], sk);
        block_sum2(sq, sk, scratch);
        const float iq = 1.0f / sqrtf(sq / (float)(H * dk) + pp.eps);
        const float ik = 1.0f / sqrtf(sk / (float)(G * dk) + pp.eps);
        for (int h = threadIdx.x; h < H + G; h += blockDim.x) inv_s[h] = h < H ? iq : ik;
    }
    __syncthreads();
    pdl_trigger();
    float temp = 1.0f;
    if (pp.temp_every > 0) temp = 1.0f + pp.temp_coef * logf((float)((pos + 1) / pp.temp_every) + 1.0f);
    const size_t at = ((size_t)(can_write ? page_id : 0) * G) * page + (size_t)(pos % page);
    const bool split = !pp.adjacent && half > 0;     // partners half a turned part apart
    if (dk % 4 == 0 && dv % 4 == 0 && pp.rot % (split ? 8 : 4) == 0 && C % 4 == 0) {
        // a warp a head, four neighbouring features a lane (turned together, or all plain)
        const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
        auto four = [](const float* p) { return *reinterpret_cast<const float4*>(p); };
        for (int h = threadIdx.x >> 5; h < H + G; h += warps) {
            const bool is_q = h < H;
            if (!is_q && !can_write) continue;
            const float* x = sh + h * dk;
            const float* wt = pp.norm == 0 ? nullptr : is_q ? pp.q_weight : pp.k_weight;
            if (wt && pp.norm == 2) wt += (is_q ? h : h - H) * dk;
            const float inv = pp.norm != 0 ? inv_s[h] : 1.0f, mul = is_q ? temp : 1.0f;
            T* dst = is_q ? q_out + (size_t)n * (H * dk) + h * dk
                          : k_pages + (at + (size_t)(h - H) * page) * dk;
            auto normed = [&](int i) {
                float4 v = four(x + i);
                v.x *= inv; v.y *= inv; v.z *= inv; v.w *= inv;
                if (wt) {
                    const float w0 = wt[i], w1 = wt[i + 1], w2 = wt[i + 2], w3 = wt[i + 3];
                    v.x *= w0; v.y *= w1; v.z *= w2; v.w *= w3;
                }
                return v;
            };
            for (int i = 4 * lane; i < dk; i += 128) {
                float4 v = normed(i);
                float other;
                if (split && i < pp.rot) {
                    const bool first = i < half;
                    const int p = first ? i : i - half;
                    const float4 o = normed(first ? i + half : i - half);
                    const float4 c = four(cs_tab + p), s = four(cs_tab + half + p);
                    if (first) {
                        rope_rotate(v.x, o.x, c.x, s.x, v.x, other);
                        rope_rotate(v.y, o.y, c.y, s.y, v.y, other);
                        rope_rotate(v.z, o.z, c.z, s.z, v.z, other);
                        rope_rotate(v.w, o.w, c.w, s.w, v.w, other);
                    } else {
                        rope_rotate(o.x, v.x, c.x, s.x, other, v.x);
                        rope_rotate(o.y, v.y, c.y, s.y, other, v.y);
                        rope_rotate(o.z, v.z, c.z, s.z, other, v.z);
                        rope_rotate(o.w, v.w, c.w, s.w, other, v.w);
                    }
                } else if (!split && i < pp.rot) {
                    const float* c = cs_tab + i / 2;
                    rope_rotate(v.x, v.y, c[0], c[half], v.x, v.y);
                    rope_rotate(v.z, v.w, c[1], c[half + 1], v.z, v.w);
                }
                v.x *= mul; v.y *= mul; v.z *= mul; v.w *= mul;
                store_four(dst + i, v);
            }
        }
        if (pp.mix == 0) {
            for (int h = threadIdx.x >> 5; h < (can_write ? G : 0); h += warps)
                for (int i = 4 * lane; i < dv; i += 128)
                    store_four(v_pages + (at + (size_t)h * page) * dv + i, four(sh + v_col + h * dv + i));
            return;
        }
    } else {
        const bool paired = dk % 2 == 0 && (!split || half % 2 == 0);
        // neighbouring features two at a time (turned together, or both plain), one store for both
        for (int idx = threadIdx.x; idx < (paired ? (H + G) * (dk / 2) : 0); idx += blockDim.x) {
            const int h = idx / (dk / 2), i = idx - h * (dk / 2);
            const bool is_q = h < H;
            if (!is_q && !can_write) continue;
            const float* x = sh + h * dk;
            const float* wt = nullptr;
            float inv = 1.0f;
            if (pp.norm != 0) {
                inv = inv_s[h];
                wt = is_q ? pp.q_weight : pp.k_weight;
                if (pp.norm == 2) wt += (is_q ? h : h - H) * dk;
            }
            const float mul = is_q ? temp : 1.0f;
            T* dst = is_q ? q_out + (size_t)n * (H * dk) + h * dk
                          : k_pages + (at + (size_t)(h - H) * page) * dk;
            const int a = 2 * i, b = a + 1;
            float ra = x[a] * inv * (wt ? wt[a] : 1.0f), rb = x[b] * inv * (wt ? wt[b] : 1.0f);
            if (split && a < pp.rot) {                   // both features lie in one half of the turned part
                const bool first = a < half;
                const int p = first ? a : a - half, o = first ? a + half : a - half;
                const float oa = x[o] * inv * (wt ? wt[o] : 1.0f);
                const float ob = x[o + 1] * inv * (wt ? wt[o + 1] : 1.0f);
                float other;
                if (first) {
                    rope_rotate(ra, oa, cs_tab[p], cs_tab[half + p], ra, other);
                    rope_rotate(rb, ob, cs_tab[p + 1], cs_tab[half + p + 1], rb, other);
                } else {
                    rope_rotate(oa, ra, cs_tab[p], cs_tab[half + p], other, ra);
                    rope_rotate(ob, rb, cs_tab[p + 1], cs_tab[half + p + 1], other, rb);
                }
            } else if (!split && i < half) {
                rope_rotate(ra, rb, cs_tab[i], cs_tab[half + i], ra, rb);
            }
            store_pair(dst + a, ra * mul, rb * mul);
        }
        const int per = dk - half;                       // work items a head: pairs, then plain features
        for (int idx = threadIdx.x; idx < (paired ? 0 : (H + G) * per); idx += blockDim.x) {
            const int h = idx / per, i = idx - h * per;
            const bool is_q = h < H;
            if (!is_q && !can_write) continue;
            const float* x = sh + h * dk;
            const float* wt = nullptr;
            float inv = 1.0f;
            if (pp.norm != 0) {
                inv = inv_s[h];
                wt = is_q ? pp.q_weight : pp.k_weight;
                if (pp.norm == 2) wt += (is_q ? h : h - H) * dk;
            }
            const float mul = is_q ? temp : 1.0f;
            T* dst = is_q ? q_out + (size_t)n * (H * dk) + h * dk
                          : k_pages + (at + (size_t)(h - H) * page) * dk;
            if (i < half) {
                const int a = pp.adjacent ? 2 * i : i, b = pp.adjacent ? 2 * i + 1 : i + half;
                float ra, rb;
                rope_rotate(x[a] * inv * (wt ? wt[a] : 1.0f), x[b] * inv * (wt ? wt[b] : 1.0f),
                            cs_tab[i], cs_tab[half + i], ra, rb);
                dst[a] = from_float<T>(ra * mul);
                dst[b] = from_float<T>(rb * mul);
            } else {
                const int a = i + half;
                dst[a] = from_float<T>(x[a] * inv * (wt ? wt[a] : 1.0f) * mul);
            }
        }
    }
    if (pp.mix == 0 && dv % 2 == 0) {                // plain values, two at a time
        for (int idx = threadIdx.x; idx < (can_write ? G * (dv / 2) : 0); idx += blockDim.x) {
            const int h = idx / (dv / 2), i = 2 * (idx - h * (dv / 2));
            const float* v = sh + v_col + h * dv + i;
            store_pair(v_pages + (at + (size_t)h * page) * dv + i, v[0], v[1]);
        }
        return;
    }
    const float lam = pp.mix == 2 ? pp.lambda[0] : 0.0f;
    for (int idx = threadIdx.x; idx < G * dv; idx += blockDim.x) {
        float v = sh[v_col + idx];
        if (pp.mix == 2) v = (1.0f - lam) * v + lam * pp.v_first[(size_t)n * (G * dv) + idx];
        const T stored = from_float<T>(v);
        if (pp.mix == 1) pp.v_first[(size_t)n * (G * dv) + idx] = to_float(stored);
        if (can_write) {
            const int h = idx / dv, i = idx - h * dv;
            v_pages[(at + (size_t)h * page) * dv + i] = stored;
        }
    }
}

// The same for steps with portions, heads of D = 64 or 128 features (keys and values alike), norm over a
// head or none, values as they are: runs of RUN tokens, a lane four neighbouring channels of a head
// (32 or 16 lanes a head), which hold their taps, bias and weights for the run, read every row of
// proj once and keep the last K - 1 inputs in registers; a head's squares and the partners of a turn
// go from lane to lane.  The sums are those of the kernel above, bit for bit.  grid (runs, heads in
// blocks of 8 warps).  Bound by instructions and the latency of a token after the other (some 200 a head
// and token; the kernel above reads taps and bias, 48 KB, for every token).  Prompts of 1,201 and 1,172
// tokens of 16 + 4 + 4 heads of 128 with three taps 31 us against 45; runs of 8 tokens 29, of 16 27,
// but portions of 400 17 and 24 instead of 13.
constexpr int RUN = 4;            // at most 32: a lane a token

template <typename T, int D, int KK>              // KK: taps, 1 for none
__global__ void __launch_bounds__(256, 3)
qkv_prepare_runs_kernel(const T* __restrict__ proj, int ld, T* __restrict__ q_out,
                        const int* __restrict__ positions, const int* __restrict__ token_seq,
                        const int* __restrict__ token_slot, const int* __restrict__ seq_pos0,
                        Prepare pp, int H, int G, T* __restrict__ k_pages, T* __restrict__ v_pages,
                        const int* __restrict__ block_table, int table_stride, int page,
                        int num_pages, int n_tokens, int* __restrict__ status) {
    constexpr int LANES = D / 4, PER = 32 / LANES;   // lanes of a head, heads of a warp
    __shared__ __align__(16) float tab[RUN][D];      // a token's cosines, then its sines
    const int n0 = blockIdx.x * RUN, count = min(RUN, n_tokens - n0);
    const int heads = H + (pp.v_from_k ? G : 2 * G), C = heads * D, half = pp.rot / 2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int h = ((int)blockIdx.y * 8 + warp) * PER + lane / LANES;
    const int i0 = lane % LANES * 4, c = h * D + i0;
    const bool live = h < heads, is_q = h < H, is_k = !is_q && h < H + G;
    const int g = is_q ? 0 : is_k ? h - H : h - H - G;         // kv head
    // lane i < RUN: token i
    int pos = 0, off = 0, slot = 0, page_id = -1, in_page = 0;
    float temp = 1.0f;
    if (lane < count) {
        pos = positions[n0 + lane];
        slot = token_slot[n0 + lane];
        off = pos - seq_pos0[token_seq[n0 + lane]];
        page_id = block_table[(size_t)slot * table_stride + pos / page];
        in_page = pos % page;
        if (page_id < 0 || page_id >= num_pages) {   // never written outside the pool
            page_id = -1;
            if (warp == 0) atomicExch(status, 1);
        }
        if (pp.temp_every > 0)
            temp = 1.0f + pp.temp_coef * logf((float)((pos + 1) / pp.temp_every) + 1.0f);
    }
    for (int e = threadIdx.x; e < count * half; e += 256) {
        const int i = e / half, f = e - i * half;
        // the angle as in the kernel above
        const double turns = (double)positions[n0 + i] * ((double)pp.freq[f] * 0.15915494309189535);
        float sn, cs;
        sincospif((float)(2.0 * (turns - rint(turns))), &sn, &cs);
        tab[i][f] = cs * pp.magnitude;
        tab[i][half + f] = sn * pp.magnitude;
    }
    float w[KK][4], b[4] = {0.0f, 0.0f, 0.0f, 0.0f}, wt[4] = {1.0f, 1.0f, 1.0f, 1.0f};
    const float* weight = pp.norm == 0 ? nullptr : is_q ? pp.q_weight : is_k ? pp.k_weight : nullptr;
    if (live) {
        if (pp.bias) load_run<4>(pp.bias + c, pp.by_tap, b);
        if (KK > 1) {
#pragma unroll
            for (int j = 0; j < KK; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    w[j][e] = pp.taps[pp.by_tap ? (size_t)j * C + c + e : (size_t)(c + e) * KK + j];
        }
        if (weight)
#pragma unroll
            for (int e = 0; e < 4; ++e) wt[e] = weight[i0 + e];
    }
    __syncthreads();
    pdl_wait();
    auto fetch = [&](int i) {
        return live && i < count ? load_four(proj + (size_t)(n0 + i) * ld + c)
                                 : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    };
    auto take = [&](float (&to)[4], const float4& v) {           // an input, with its bias
        to[0] = v.x; to[1] = v.y; to[2] = v.z; to[3] = v.w;
        if (pp.bias)
#pragma unroll
            for (int e = 0; e < 4; ++e) to[e] += b[e];
    };
    float4 in = fetch(0), in_next = fetch(1);        // two tokens ahead
    float x[KK][4];                                  // the token's input last
#pragma unroll 1
    for (int i = 0; i < count; ++i) {
        const float4 now = in;
        in = in_next;
        in_next = fetch(i + 2);
        const int n = n0 + i, tpos = __shfl_sync(0xffffffffu, pos, i);
        const int toff = __shfl_sync(0xffffffffu, off, i), id = __shfl_sync(0xffffffffu, page_id, i);
        const int row = __shfl_sync(0xffffffffu, in_page, i);
        const float mul = __shfl_sync(0xffffffffu, temp, i);
        if (KK > 1 && (i == 0 || toff == 0)) {
            // the inputs before this token: of its portion, or what the slot keeps
            const int tslot = __shfl_sync(0xffffffffu, slot, i);
            const float* kept = pp.state + (size_t)tslot * pp.slot_stride + pp.conv_offset;
#pragma unroll
            for (int j = 0; j + 1 < KK; ++j) {
                const int rel = toff - (KK - 1) + j;
                float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (live && rel >= 0) {
                    v = load_four(proj + (size_t)(n - (KK - 1) + j) * ld + c);
                } else if (live && tpos - (KK - 1) + j >= 0) {
                    const float* k = kept + (size_t)(toff + j) * C + c;
                    v = make_float4(k[0], k[1], k[2], k[3]);
                }
                take(x[j], v);
            }
        } else {
#pragma unroll
            for (int j = 0; j + 1 < KK; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) x[j][e] = x[j + 1][e];
        }
        take(x[KK - 1], now);
        float y[4];
        if (KK == 1) {
#pragma unroll
            for (int e = 0; e < 4; ++e) y[e] = x[0][e];
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) y[e] = 0.0f;
#pragma unroll
            for (int j = 0; j < KK; ++j) {
                if (tpos - (KK - 1) + j < 0) continue;           // before the sequence's start
#pragma unroll
                for (int e = 0; e < 4; ++e) y[e] = fmaf(w[j][e], x[j][e], y[e]);
            }
        }
        const size_t at = ((size_t)max(id, 0) * G + g) * page + (size_t)row;
        const float4 plain = make_float4(y[0], y[1], y[2], y[3]);
        const bool has_v = live && id >= 0 && (pp.v_from_k ? is_k : !is_q && !is_k);
        if (has_v)
            store_four(v_pages + at * D + i0, plain);
        float4 v = plain;
        if (pp.norm == 1) {
            float ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, 0.0f))));
#pragma unroll
            for (int o = LANES / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            const float inv = 1.0f / sqrtf(ss / (float)D + pp.eps);
            v.x *= inv; v.y *= inv; v.z *= inv; v.w *= inv;
            if (weight) { v.x *= wt[0]; v.y *= wt[1]; v.z *= wt[2]; v.w *= wt[3]; }
        }
        if (!pp.adjacent && half > 0) {              // partners half a turned part apart
            const bool first = i0 < half;
            const int from = i0 < pp.rot ? lane + (first ? half / 4 : -(half / 4)) : lane;
            const float4 o = make_float4(
                __shfl_sync(0xffffffffu, v.x, from), __shfl_sync(0xffffffffu, v.y, from),
                __shfl_sync(0xffffffffu, v.z, from), __shfl_sync(0xffffffffu, v.w, from));
            if (i0 < pp.rot) {
                const int p = first ? i0 : i0 - half;
                const float4 cs = *reinterpret_cast<const float4*>(&tab[i][p]);
                const float4 sn = *reinterpret_cast<const float4*>(&tab[i][half + p]);
                float other;
                if (first) {
                    rope_rotate(v.x, o.x, cs.x, sn.x, v.x, other);
                    rope_rotate(v.y, o.y, cs.y, sn.y, v.y, other);
                    rope_rotate(v.z, o.z, cs.z, sn.z, v.z, other);
                    rope_rotate(v.w, o.w, cs.w, sn.w, v.w, other);
                } else {
                    rope_rotate(o.x, v.x, cs.x, sn.x, other, v.x);
                    rope_rotate(o.y, v.y, cs.y, sn.y, other, v.y);
                    rope_rotate(o.z, v.z, cs.z, sn.z, other, v.z);
                    rope_rotate(o.w, v.w, cs.w, sn.w, other, v.w);
                }
            }
        } else if (i0 < pp.rot) {
            const float* cs = &tab[i][i0 / 2];
            rope_rotate(v.x, v.y, cs[0], cs[half], v.x, v.y);
            rope_rotate(v.z, v.w, cs[1], cs[half + 1], v.z, v.w);
        }
        if (live && is_q) {
            v.x *= mul; v.y *= mul; v.z *= mul; v.w *= mul;
            store_four(q_out + (size_t)n * (H * D) + h * D + i0, v);
        } else if (live && is_k && id >= 0) {
            store_four(k_pages + at * D + i0, v);
        }
    }
    pdl_trigger();
}

// After qkv_prepare: every sequence's slot keeps the last K - 1 rows of the first C columns of
// proj (the convolution's inputs of the next step), kept[i] = the row at position
// pos0 + qlen - (K - 1) + i; a portion shorter than K - 1 moves the older rows up.  The layout is
// the one that the state mixers' convolution keeps (recurrent.cu); a model whose only
// convolution is this mixer's needs no other library for it.  grid (sequences, channels / 256): a
// thread a channel, 2.4 us in a layer of two sequences of 3,072 channels (6.5 with a block a sequence).
template <typename T>
__global__ void conv_keep_kernel(const T* __restrict__ proj, int ld, float* __restrict__ state,
                                 long long slot_stride, int conv_offset,
                                 const int* __restrict__ seq_slot,
                                 const int* __restrict__ seq_qstart,
                                 const int* __restrict__ seq_qlen, int C, int K) {
    const int s = blockIdx.x;
    const int qlen = seq_qlen[s], tok0 = seq_qstart[s];
    pdl_wait();
    pdl_trigger();
    float* kept = state + (size_t)seq_slot[s] * slot_stride + conv_offset;
    for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < C; c += gridDim.y * blockDim.x)
        for (int i = 0; i < K - 1; ++i) {            // ascending: what is read lies ahead
            const int rel = qlen - (K - 1) + i;
            kept[(size_t)i * C + c] = rel >= 0 ? to_float(proj[(size_t)(tok0 + rel) * ld + c])
                                               : kept[(size_t)(i + qlen) * C + c];
        }
}

// After the attention: every head's result (float32 [N, H dv]) turned back by its token's position
// (pairs (i, i + dv/2), angle -pos * fv[i]; fv null: as it is), times sigmoid(gate) where a gate
// (type T, row stride ld_gate; one number a feature, or one a head with gate_per_head) is given,
// rounded to the activation type.  One block a token.
template <typename T>
__global__ void attn_finish_kernel(const float* __restrict__ o, const int* __restrict__ positions,
                                   const float* __restrict__ fv, const T* __restrict__ gate,
                                   int ld_gate, T* __restrict__ out, int H, int dv,
                                   int gate_per_head) {
    const int n = blockIdx.x;
    const float fpos = (float)positions[n];
    const float* src = o + (size_t)n * H * dv;
    T* dst = out + (size_t)n * H * dv;
    const T* gt = gate ? gate + (size_t)n * ld_gate : nullptr;
    pdl_wait();
    pdl_trigger();
    if (fv != nullptr) {
        const int half = dv / 2, per = dv - half;
        for (int idx = threadIdx.x; idx < H * per; idx += blockDim.x) {
            const int h = idx / per, i = idx - h * per;
            const int a = h * dv + i, b = a + half;
            if (i < half) {
                float sn, cs, ra, rb;
                sincosf(fpos * fv[i], &sn, &cs);
                rope_rotate(src[a], src[b], cs, -sn, ra, rb);
                if (gt) {
                    ra *= 1.0f / (1.0f + expf(-to_float(gt[gate_per_head ? h : a])));
                    rb *= 1.0f / (1.0f + expf(-to_float(gt[gate_per_head ? h : b])));
                }
                dst[a] = from_float<T>(ra);
                dst[b] = from_float<T>(rb);
            } else {
                float x = src[b];
                if (gt) x *= 1.0f / (1.0f + expf(-to_float(gt[gate_per_head ? h : b])));
                dst[b] = from_float<T>(x);
            }
        }
    } else {
        for (int idx = threadIdx.x; idx < H * dv; idx += blockDim.x) {
            float x = src[idx];
            if (gt) x *= 1.0f / (1.0f + expf(-to_float(gt[gate_per_head ? idx / dv : idx])));
            dst[idx] = from_float<T>(x);
        }
    }
}

// The same in groups of four features (with `fv`: of four pairs, the angles formed once a token), for
// heads of whole groups at such addresses.  2,048 tokens, 16 heads of 128, turned: 10 us (14).
template <typename T>
__global__ void attn_finish_vec_kernel(const float* __restrict__ o, const int* __restrict__ positions,
                                       const float* __restrict__ fv, const T* __restrict__ gate,
                                       int ld_gate, T* __restrict__ out, int H, int dv,
                                       int gate_per_head) {
    __shared__ __align__(16) float tab[MAX_D];
    const int n = blockIdx.x, half = dv / 2;
    const float* src = o + (size_t)n * H * dv;
    T* dst = out + (size_t)n * H * dv;
    const T* gt = gate ? gate + (size_t)n * ld_gate : nullptr;
    if (fv != nullptr) angles(tab, fv, half, (float)positions[n]);
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    auto finish = [&](float4 v, int h, int at) {
        if (gt) {
            float4 g;
            if (gate_per_head) g.x = g.y = g.z = g.w = to_float(gt[h]);
            else g = load_four(gt + at);
            v.x *= 1.0f / (1.0f + expf(-g.x));
            v.y *= 1.0f / (1.0f + expf(-g.y));
            v.z *= 1.0f / (1.0f + expf(-g.z));
            v.w *= 1.0f / (1.0f + expf(-g.w));
        }
        store_four(dst + at, v);
    };
    if (fv == nullptr) {
        for (int i = threadIdx.x * 4; i < H * dv; i += blockDim.x * 4)
            finish(load_four(src + i), i / dv, i);
        return;
    }
    for (int idx = threadIdx.x; idx < H * half / 4; idx += blockDim.x) {
        const int h = idx / (half / 4), i = (idx - h * (half / 4)) * 4, at = h * dv + i;
        const float4 a = load_four(src + at), b = load_four(src + at + half);
        const float4 c = load_four(tab + i), s = load_four(tab + half + i);
        float4 x, y;
        rope_rotate(a.x, b.x, c.x, -s.x, x.x, y.x);
        rope_rotate(a.y, b.y, c.y, -s.y, x.y, y.y);
        rope_rotate(a.z, b.z, c.z, -s.z, x.z, y.z);
        rope_rotate(a.w, b.w, c.w, -s.w, x.w, y.w);
        finish(x, h, at);
        finish(y, h, at + half);
    }
}

template <typename T>
__global__ void __launch_bounds__(ROWS * 32)
attn_chunk_kernel(const T* __restrict__ q, int q_stride, void* __restrict__ out, int out_stride,
                  const T* __restrict__ k_pages, const T* __restrict__ v_pages,
                  const int* __restrict__ block_table, int table_stride, int num_pages,
                  const int* __restrict__ seq_slot, const int* __restrict__ seq_qstart,
                  const int* __restrict__ seq_qlen, const int* __restrict__ seq_pos0,
                  const WorkItem* __restrict__ items, const float* __restrict__ r1,
                  const float* __restrict__ r2, int heads, int kv_heads, int dk, int dv, int page,
                  float scale, Sight sight, int out_f32, int* __restrict__ status) {
    extern __shared__ float smem[];
    float* Ks = smem;                       // [TILE][dk + 1]; column dk: 0, or -inf without a page
    float* Vs = Ks + TILE * (dk + 1);       // [TILE][dv]
    float* Qs = Vs + TILE * dv;             // [ROWS][dk]

    const WorkItem it = items[blockIdx.x];
    if (it.kv_begin >= it.kv_end) {
        pdl_wait();
        return;
    }
    const int hk = blockIdx.y;
    const int g = heads / kv_heads;
    const int qlen = seq_qlen[it.seq], pos0 = seq_pos0[it.seq];
    const int slot = seq_slot[it.seq], tok0 = seq_qstart[it.seq];
    const int rows_total = qlen * g;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    const int r = it.row0 + warp;
    const bool active = r < rows_total;
    const int t = active ? r / g : 0;
    const int hq = hk * g + (active ? r % g : 0);
    const int pos = pos0 + t;
    const bool penalty = r1 != nullptr;
    const float pen1 = penalty ? r1[hq] : 0.0f, pen2 = penalty ? r2[hq] : 0.0f;

    pdl_wait();
    for (int i = lane; i < dk; i += 32)
        Qs[warp * dk + i] = active ? to_float(q[(size_t)(tok0 + t) * q_stride + hq * dk + i]) : 0.0f;

    // the tile's key range: from the chunk or window of its first token to its last token, and
    // the kept first keys
    const int last_row = min(it.row0 + ROWS, rows_total) - 1;
    const int max_pos = pos0 + last_row / g, min_pos = pos0 + it.row0 / g;
    const int k_hi = min(it.kv_end, max_pos + 1);
    const int k_lo_true = max(it.kv_begin, sight_lo(sight, min_pos));
    const int k_first = it.kv_begin > 0 ? 0 : sight_first(sight, k_lo_true);
    const TileWalk walk(k_lo_true, k_first, TILE);
    // this row's
    const int row_lo = max(it.kv_begin, sight_lo(sight, pos));
    const int row_first = it.kv_begin > 0 ? 0 : sight_first(sight, row_lo);
    const int row_hi = min(it.kv_end, pos + 1);

    float m = -INFINITY, l = 0.0f;
    float acc[MAX_D / 32];
#pragma unroll
    for (int i = 0; i < MAX_D / 32; ++i) acc[i] = 0.0f;

    for (int kt = walk.start; kt < k_hi; kt = walk.next(kt, TILE)) {
        __syncthreads();
        for (int j = warp; j < TILE; j += ROWS) {        // a warp a key: whole rows of the pages
            const int kpos = kt + j;
            bool held = true, inside = (kpos >= k_lo_true || kpos < k_first) && kpos < k_hi;
            size_t at = 0;
            if (inside) {
                const int page_id = block_table[(size_t)slot * table_stride + kpos / page];
                held = page_id >= 0 && page_id < num_pages;
                at = ((size_t)page_id * kv_heads + hk) * page + (size_t)(kpos % page);
            }
            const bool read = inside && held;
            for (int i = lane; i < dk; i += 32)
                Ks[j * (dk + 1) + i] = read ? to_float(k_pages[at * dk + i]) : 0.0f;
            for (int i = lane; i < dv; i += 32)
                Vs[j * dv + i] = read ? to_float(v_pages[at * sight.v_stride + i]) : 0.0f;
            if (lane == 0) {
                Ks[j * (dk + 1) + dk] = held ? 0.0f : -INFINITY;
                if (!held && status != nullptr) atomicExch(status, 2);
            }
        }
        __syncthreads();
        if (!active) continue;

        const int kpos = kt + lane;
        const float* kr = Ks + lane * (dk + 1);
        const bool valid = (kpos >= row_lo || kpos < row_first) && kpos < row_hi && kr[dk] == 0.0f;
        const float* qr = Qs + warp * dk;
        float s = 0.0f;
        for (int i = 0; i < dk; ++i) s = fmaf(qr[i], kr[i], s);
        s = valid ? sight_score(sight, s, scale, pen1, pen2, penalty, (float)(pos - kpos)) : -INFINITY;
        const float m_new = fmaxf(m, warp_max(s));
        if (m_new == -INFINITY) continue;
        const float p = valid ? expf(s - m_new) : 0.0f;
        const float corr = expf(m - m_new);
        l = l * corr + warp_sum(p);
#pragma unroll
        for (int i = 0; i < MAX_D / 32; ++i) acc[i] *= corr;
        for (int j = 0; j < TILE; ++j) {
            const float pj = __shfl_sync(0xffffffffu, p, j);
            if (pj == 0.0f) continue;
            const float* vr = Vs + j * dv;
#pragma unroll
            for (int i = 0; i < MAX_D / 32; ++i) {
                const int dd = lane + 32 * i;
                if (dd < dv) acc[i] = fmaf(pj, vr[dd], acc[i]);
            }
        }
        m = m_new;
    }
    pdl_trigger();
    if (!active) return;
    const float inv = sight_inverse(sight, hq, m, l);
    const size_t o = (size_t)(tok0 + t) * out_stride + hq * dv;
#pragma unroll
    for (int i = 0; i < MAX_D / 32; ++i) {
        const int dd = lane + 32 * i;
        if (dd < dv)
            store_out<T>(out, out_f32, o + dd,
                         acc[i] * inv * sight_gate<T>(sight, (size_t)(tok0 + t), hq, dv, dd));
    }
}


// ------------------------------------------------------------------------------------------
// The same attention for key and value rows that are whole 16-byte pieces (sizes that are a
// multiple of 8 in bfloat16, of 4 in float32): the next tile of keys and values is asked for in
// 16-byte loads into registers before the current one is worked on, a warp takes RW rows (it
// reads a key or a value from shared memory once for all of them), and shared memory is read as
// float4.  A row's sums are formed in the same order as in the kernel above whatever RW is.
// ------------------------------------------------------------------------------------------
template <typename T> struct Piece;                 // 16 bytes of T as floats
template <> struct Piece<float> {
    static constexpr int N = 4;
    static __device__ __forceinline__ void unpack(const uint4& u, float* f) {
        f[0] = __uint_as_float(u.x); f[1] = __uint_as_float(u.y);
        f[2] = __uint_as_float(u.z); f[3] = __uint_as_float(u.w);
    }
};
template <> struct Piece<__nv_bfloat16> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void unpack(const uint4& u, float* f) {
        const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            f[2 * i] = __uint_as_float(w[i] << 16);
            f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        }
    }
};

template <typename T, int RW, int NCH>
__global__ void __launch_bounds__(ROWS * 32, NCH <= 4 ? 2 : 1)
attn_chunk_vec_kernel(const T* __restrict__ q, int q_stride, void* __restrict__ out, int out_stride,
                      const T* __restrict__ k_pages, const T* __restrict__ v_pages,
                      const int* __restrict__ block_table, int table_stride, int num_pages,
                      const int* __restrict__ seq_slot, const int* __restrict__ seq_qstart,
                      const int* __restrict__ seq_qlen, const int* __restrict__ seq_pos0,
                      const WorkItem* __restrict__ items, const float* __restrict__ r1,
                      const float* __restrict__ r2, int heads, int kv_heads, int dk, int dv,
                      int page, float scale, Sight sight, int out_f32, int* __restrict__ status) {
    constexpr int PN = Piece<T>::N;
    extern __shared__ __align__(16) float smem[];
    const int ks = ((dk + 31) / 32) * 32 + 4;       // a key's stride: float4 reads without conflicts
    float* Ks = smem;                                // [TILE][ks]
    float* Vs = Ks + TILE * ks;                      // [TILE][dv]
    float* Qs = Vs + TILE * dv;                      // [ROWS * RW][dk]
    float* Held = Qs + ROWS * RW * dk;               // [TILE]: 0, or -inf for a key without a page

    const WorkItem it = items[blockIdx.x];
    if (it.kv_begin >= it.kv_end) {
        pdl_wait();
        return;
    }
    const int hk = blockIdx.y;
    const int g = heads / kv_heads;
    const int qlen = seq_qlen[it.seq], pos0 = seq_pos0[it.seq];
    const int slot = seq_slot[it.seq], tok0 = seq_qstart[it.seq];
    const int rows_total = qlen * g;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    bool active[RW];
    int tok[RW], hq[RW], pos[RW], row_lo[RW], row_hi[RW], row_first[RW];
    float pen1[RW], pen2[RW], m[RW], l[RW];
    bool any = false;
    const bool penalty = r1 != nullptr;
#pragma unroll
    for (int i = 0; i < RW; ++i) {
        const int r = it.row0 + warp * RW + i;
        active[i] = r < rows_total;
        any |= active[i];
        tok[i] = active[i] ? r / g : 0;
        hq[i] = hk * g + (active[i] ? r % g : 0);
        pos[i] = pos0 + tok[i];
        pen1[i] = penalty ? r1[hq[i]] : 0.0f;
        pen2[i] = penalty ? r2[hq[i]] : 0.0f;
        row_lo[i] = max(it.kv_begin, sight_lo(sight, pos[i]));
        row_first[i] = it.kv_begin > 0 ? 0 : sight_first(sight, row_lo[i]);
        row_hi[i] = min(it.kv_end, pos[i] + 1);
        m[i] = -INFINITY;
        l[i] = 0.0f;
    }
    const int last_row = min(it.row0 + ROWS * RW, rows_total) - 1;
    const int max_pos = pos0 + last_row / g, min_pos = pos0 + it.row0 / g;
    const int k_hi = min(it.kv_end, max_pos + 1);
    const int k_lo_true = max(it.kv_begin, sight_lo(sight, min_pos));
    const int k_first = it.kv_begin > 0 ? 0 : sight_first(sight, k_lo_true);
    const TileWalk walk(k_lo_true, k_first, TILE);

    const int ck = dk / PN, cv = dv / PN, per_key = ck + cv;
    uint4 pre[NCH];
    unsigned missing = 0;                            // bit c: piece c's key has no page

    pdl_wait();
    auto prefetch = [&](int kt) {
        missing = 0;
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
            const int e = threadIdx.x + c * (ROWS * 32);
            pre[c] = make_uint4(0u, 0u, 0u, 0u);
            if (e >= TILE * per_key) continue;
            const int j = e / per_key, w = e - j * per_key;
            const int kpos = kt + j;
            if ((kpos < k_lo_true && kpos >= k_first) || kpos >= k_hi) continue;
            const int page_id = block_table[(size_t)slot * table_stride + kpos / page];
            if (page_id < 0 || page_id >= num_pages) {
                missing |= 1u << c;
                continue;
            }
            const size_t at = ((size_t)page_id * kv_heads + hk) * page + (size_t)(kpos % page);
            const T* src = w < ck ? k_pages + at * dk + w * PN : v_pages + at * sight.v_stride + (w - ck) * PN;
            pre[c] = *reinterpret_cast<const uint4*>(src);
        }
    };
    prefetch(walk.start);
#pragma unroll
    for (int i = 0; i < RW; ++i)
        for (int d = lane; d < dk; d += 32)
            Qs[(warp * RW + i) * dk + d] =
                active[i] ? to_float(q[(size_t)(tok0 + tok[i]) * q_stride + hq[i] * dk + d]) : 0.0f;

    float acc[RW][MAX_D / 128][4];
#pragma unroll
    for (int i = 0; i < RW; ++i)
#pragma unroll
        for (int b = 0; b < MAX_D / 128; ++b)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][b][e] = 0.0f;

    for (int kt = walk.start; kt < k_hi; kt = walk.next(kt, TILE)) {
        __syncthreads();                             // the tile before this one has been used
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
            const int e = threadIdx.x + c * (ROWS * 32);
            if (e >= TILE * per_key) continue;
            const int j = e / per_key, w = e - j * per_key;
            float f[PN];
            Piece<T>::unpack(pre[c], f);
            float* dst = w < ck ? Ks + j * ks + w * PN : Vs + j * dv + (w - ck) * PN;
#pragma unroll
            for (int x = 0; x < PN; x += 4)
                *reinterpret_cast<float4*>(dst + x) = make_float4(f[x], f[x + 1], f[x + 2], f[x + 3]);
            if (w == 0) {
                const bool gone = (missing >> c) & 1u;
                Held[j] = gone ? -INFINITY : 0.0f;
                if (gone && status != nullptr) atomicExch(status, 2);
            }
        }
        __syncthreads();
        if (walk.next(kt, TILE) < k_hi) prefetch(walk.next(kt, TILE));   // in flight meanwhile
        if (!any) continue;

        const int kpos = kt + lane;
        const float4* kr = reinterpret_cast<const float4*>(Ks + lane * ks);
        float s[RW];
#pragma unroll
        for (int i = 0; i < RW; ++i) s[i] = 0.0f;
#pragma unroll 4
        for (int d = 0; d < dk / 4; ++d) {
            const float4 kk = kr[d];
#pragma unroll
            for (int i = 0; i < RW; ++i) {
                const float4 qq = reinterpret_cast<const float4*>(Qs + (warp * RW + i) * dk)[d];
                s[i] = fmaf(qq.x, kk.x, s[i]);
                s[i] = fmaf(qq.y, kk.y, s[i]);
                s[i] = fmaf(qq.z, kk.z, s[i]);
                s[i] = fmaf(qq.w, kk.w, s[i]);
            }
        }
        const bool held = Held[lane] == 0.0f;
        float p[RW];
        bool some = false;
#pragma unroll
        for (int i = 0; i < RW; ++i) {
            const bool valid = active[i] && (kpos >= row_lo[i] || kpos < row_first[i]) &&
                               kpos < row_hi[i] && held;
            const float sc = valid ? sight_score(sight, s[i], scale, pen1[i], pen2[i], penalty,
                                                 (float)(pos[i] - kpos))
                                   : -INFINITY;
            const float m_new = fmaxf(m[i], warp_max(sc));
            if (m_new == -INFINITY) {               // nothing of this tile is visible to the row
                p[i] = 0.0f;
                continue;
            }
            p[i] = valid ? expf(sc - m_new) : 0.0f;
            const float corr = expf(m[i] - m_new);
            l[i] = l[i] * corr + warp_sum(p[i]);
#pragma unroll
            for (int b = 0; b < MAX_D / 128; ++b)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[i][b][e] *= corr;
            m[i] = m_new;
            some = true;
        }
        if (!some) continue;
#pragma unroll 4
        for (int j = 0; j < TILE; ++j) {
            float pj[RW];
            bool zero = true;
#pragma unroll
            for (int i = 0; i < RW; ++i) {
                pj[i] = __shfl_sync(0xffffffffu, p[i], j);
                zero &= pj[i] == 0.0f;
            }
            if (zero) continue;                      // the same for the whole warp
#pragma unroll
            for (int b = 0; b < MAX_D / 128; ++b) {
                const int dd = 4 * lane + 128 * b;
                if (dd < dv) {
                    const float4 vv = *reinterpret_cast<const float4*>(Vs + j * dv + dd);
#pragma unroll
                    for (int i = 0; i < RW; ++i) {
                        if (pj[i] == 0.0f) continue;  // as the kernel above skips it
                        acc[i][b][0] = fmaf(pj[i], vv.x, acc[i][b][0]);
                        acc[i][b][1] = fmaf(pj[i], vv.y, acc[i][b][1]);
                        acc[i][b][2] = fmaf(pj[i], vv.z, acc[i][b][2]);
                        acc[i][b][3] = fmaf(pj[i], vv.w, acc[i][b][3]);
                    }
                }
            }
        }
    }
    pdl_trigger();
#pragma unroll
    for (int i = 0; i < RW; ++i) {
        if (!active[i]) continue;
        const float inv = sight_inverse(sight, hq[i], m[i], l[i]);
        const size_t o = (size_t)(tok0 + tok[i]) * out_stride + hq[i] * dv;
#pragma unroll
        for (int b = 0; b < MAX_D / 128; ++b) {
            const int dd = 4 * lane + 128 * b;
            if (dd < dv) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    store_out<T>(out, out_f32, o + dd + e,
                                 acc[i][b][e] * inv * sight_gate<T>(sight, (size_t)(tok0 + tok[i]),
                                                                    hq[i], dv, dd + e));
            }
        }
    }
}


// ------------------------------------------------------------------------------------------
// The same attention for long prompt portions, with the products tiled in registers: a block of
// four warps takes 64 rows, a warp 16 of them against the tile of 32 keys.  Lane (i, j) of a warp
// (i = lane / 8, j = lane % 8) holds rows i, i + 4, i + 8, i + 12 against keys j, j + 8, j + 16,
// j + 24: a step over four features is four 16-byte reads of q and four of k from shared memory
// for 64 multiply-adds (the kernel above: five reads for 16), and rows and keys that meet in one
// read lie 4 banks apart.  The weights go through shared memory once ([key][row], a warp's own
// 2 KB), and for the values lane (i, j) holds the same four rows against columns 4 j + 32 c.
// A row's score sums its features in ascending order, a row's sums over a tile's keys have an
// order of their own (fixed by the key's place in its tile), so a row's result does not depend on
// what shares its tile, its step or its batch.  Sizes as the kernel above.
// ------------------------------------------------------------------------------------------
constexpr int TROWS = 64;

template <typename T, int NC>
__global__ void __launch_bounds__(128, NC <= 4 ? 3 : 2)
attn_chunk_tiled_kernel(const T* __restrict__ q, int q_stride, void* __restrict__ out,
                        int out_stride, const T* __restrict__ k_pages,
                        const T* __restrict__ v_pages, const int* __restrict__ block_table,
                        int table_stride, int num_pages, const int* __restrict__ seq_slot,
                        const int* __restrict__ seq_qstart, const int* __restrict__ seq_qlen,
                        const int* __restrict__ seq_pos0, const WorkItem* __restrict__ items,
                        const float* __restrict__ r1, const float* __restrict__ r2, int heads,
                        int kv_heads, int dk, int dv, int page, float scale, Sight sight,
                        int out_f32, int* __restrict__ status) {
    constexpr int PN = Piece<T>::N;
    extern __shared__ __align__(16) float smem[];
    const int kst = dk + 4;                          // a key's and a query's stride
    float* Ks = smem;                                // [TILE][kst]
    float* Vs = Ks + TILE * kst;                     // [TILE][dv]
    float* Qs = Vs + TILE * dv;                      // [TROWS][kst]
    float* Ps = Qs + TROWS * kst;                    // [4 warps][TILE][16]
    float* Held = Ps + 4 * TILE * 16;                // [TILE]: 0, or -inf for a key without a page

    const WorkItem it = items[blockIdx.x];
    if (it.kv_begin >= it.kv_end) {
        pdl_wait();
        return;
    }
    const int hk = blockIdx.y;
    const int g = heads / kv_heads;
    const int qlen = seq_qlen[it.seq], pos0 = seq_pos0[it.seq];
    const int slot = seq_slot[it.seq], tok0 = seq_qstart[it.seq];
    const int rows_total = qlen * g;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int li = lane >> 3, lj = lane & 7;
    const bool penalty = r1 != nullptr;

    bool active[4];
    int tok[4], hq[4], pos[4], row_lo[4], row_hi[4], row_first[4];
    float pen1[4], pen2[4], m[4], l[4];
    bool mine = false;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int r = it.row0 + warp * 16 + li + 4 * e;
        active[e] = r < rows_total;
        mine |= active[e];
        tok[e] = active[e] ? r / g : 0;
        hq[e] = hk * g + (active[e] ? r % g : 0);
        pos[e] = pos0 + tok[e];
        pen1[e] = penalty ? r1[hq[e]] : 0.0f;
        pen2[e] = penalty ? r2[hq[e]] : 0.0f;
        row_lo[e] = max(it.kv_begin, sight_lo(sight, pos[e]));
        row_first[e] = it.kv_begin > 0 ? 0 : sight_first(sight, row_lo[e]);
        row_hi[e] = min(it.kv_end, pos[e] + 1);
        m[e] = -INFINITY;
        l[e] = 0.0f;
    }
    const bool any = __any_sync(0xffffffffu, mine);
    const int last_row = min(it.row0 + TROWS, rows_total) - 1;
    const int max_pos = pos0 + last_row / g, min_pos = pos0 + it.row0 / g;
    const int k_hi = min(it.kv_end, max_pos + 1);
    const int k_lo_true = max(it.kv_begin, sight_lo(sight, min_pos));
    const int k_first = it.kv_begin > 0 ? 0 : sight_first(sight, k_lo_true);
    const TileWalk walk(k_lo_true, k_first, TILE);
    const int ck = dk / PN, cv = dv / PN, per_key = ck + cv;

    pdl_wait();
    for (int idx = threadIdx.x; idx < TROWS * dk; idx += 128) {
        const int row = idx / dk, d = idx - row * dk;
        const int r = it.row0 + row;
        float x = 0.0f;
        if (r < rows_total)
            x = to_float(q[(size_t)(tok0 + r / g) * q_stride + (hk * g + r % g) * dk + d]);
        Qs[row * kst + d] = x;
    }

    float acc[4][NC][4];
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int x = 0; x < 4; ++x) acc[e][c][x] = 0.0f;

    float* Pw = Ps + warp * TILE * 16;
    for (int kt = walk.start; kt < k_hi; kt = walk.next(kt, TILE)) {
        __syncthreads();                             // the tile before this one has been used
        {
            // four threads a key: thread t takes the key's 16-byte pieces t % 4, t % 4 + 4, ...
            // (keys first, then values), so its key, its page and its row are found once a tile
            const int j = threadIdx.x >> 2, w0 = threadIdx.x & 3;
            const int kpos = kt + j;
            const bool inside = (kpos >= k_lo_true || kpos < k_first) && kpos < k_hi;
            bool gone = false;
            size_t at = 0;
            if (inside) {
                const int page_id = block_table[(size_t)slot * table_stride + kpos / page];
                gone = page_id < 0 || page_id >= num_pages;
                at = ((size_t)page_id * kv_heads + hk) * page + (size_t)(kpos % page);
            }
            const bool read = inside && !gone;
            const T* ksrc = k_pages + at * dk;
            const T* vsrc = v_pages + at * sight.v_stride;
            float* kdst = Ks + j * kst;
            float* vdst = Vs + j * dv;
            for (int w = w0; w < per_key; w += 16) {
                uint4 piece[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {        // four loads in flight a thread
                    const int ww = w + 4 * u;
                    piece[u] = make_uint4(0u, 0u, 0u, 0u);
                    if (read && ww < per_key)
                        piece[u] = *reinterpret_cast<const uint4*>(
                            ww < ck ? ksrc + ww * PN : vsrc + (ww - ck) * PN);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int ww = w + 4 * u;
                    if (ww >= per_key) continue;
                    float f[PN];
                    Piece<T>::unpack(piece[u], f);
                    float* dst = ww < ck ? kdst + ww * PN : vdst + (ww - ck) * PN;
#pragma unroll
                    for (int x = 0; x < PN; x += 4)
                        *reinterpret_cast<float4*>(dst + x) =
                            make_float4(f[x], f[x + 1], f[x + 2], f[x + 3]);
                }
            }
            if (w0 == 0) {
                Held[j] = gone ? -INFINITY : 0.0f;
                if (gone && status != nullptr) atomicExch(status, 2);
            }
        }
        __syncthreads();
        if (!any) continue;

        float s[4][4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int c = 0; c < 4; ++c) s[e][c] = 0.0f;
        const float* qb = Qs + (warp * 16 + li) * kst;
        const float* kb = Ks + lj * kst;
#pragma unroll 2
        for (int d = 0; d < dk; d += 4) {
            float4 qv[4], kv[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) qv[e] = *reinterpret_cast<const float4*>(qb + 4 * e * kst + d);
#pragma unroll
            for (int c = 0; c < 4; ++c) kv[c] = *reinterpret_cast<const float4*>(kb + 8 * c * kst + d);
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    s[e][c] = fmaf(qv[e].x, kv[c].x, s[e][c]);
                    s[e][c] = fmaf(qv[e].y, kv[c].y, s[e][c]);
                    s[e][c] = fmaf(qv[e].z, kv[c].z, s[e][c]);
                    s[e][c] = fmaf(qv[e].w, kv[c].w, s[e][c]);
                }
        }
        bool held[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) held[c] = Held[lj + 8 * c] == 0.0f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            float top = -INFINITY;
            bool valid[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int kpos = kt + lj + 8 * c;
                valid[c] = active[e] && (kpos >= row_lo[e] || kpos < row_first[e]) &&
                           kpos < row_hi[e] && held[c];
                s[e][c] = valid[c] ? sight_score(sight, s[e][c], scale, pen1[e], pen2[e], penalty,
                                                 (float)(pos[e] - kpos))
                                   : -INFINITY;
                top = fmaxf(top, s[e][c]);
            }
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 4));
            const float m_new = fmaxf(m[e], top);
            float sum = 0.0f, corr = 1.0f;
            if (m_new == -INFINITY) {                // nothing of this tile is visible to the row
#pragma unroll
                for (int c = 0; c < 4; ++c) s[e][c] = 0.0f;
            } else {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    s[e][c] = valid[c] ? expf(s[e][c] - m_new) : 0.0f;
                    sum += s[e][c];
                }
                corr = expf(m[e] - m_new);
                m[e] = m_new;
            }
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            sum += __shfl_xor_sync(0xffffffffu, sum, 4);
            l[e] = l[e] * corr + sum;
#pragma unroll
            for (int c = 0; c < NC; ++c)
#pragma unroll
                for (int x = 0; x < 4; ++x) acc[e][c][x] *= corr;
        }
        __syncwarp();                                // the weights of the tile before have been read
#pragma unroll
        for (int c = 0; c < 4; ++c)
            *reinterpret_cast<float4*>(Pw + (lj + 8 * c) * 16 + 4 * li) =
                make_float4(s[0][c], s[1][c], s[2][c], s[3][c]);
        __syncwarp();
        const float* vrow = Vs + 4 * lj;
        const float* prow = Pw + 4 * li;
#pragma unroll 4
        for (int key = 0; key < TILE; ++key, vrow += dv, prow += 16) {
            const float4 pv = *reinterpret_cast<const float4*>(prow);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                if (4 * lj + 32 * c < dv) {
                    const float4 vv = *reinterpret_cast<const float4*>(vrow + 32 * c);
                    acc[0][c][0] = fmaf(pv.x, vv.x, acc[0][c][0]); acc[0][c][1] = fmaf(pv.x, vv.y, acc[0][c][1]);
                    acc[0][c][2] = fmaf(pv.x, vv.z, acc[0][c][2]); acc[0][c][3] = fmaf(pv.x, vv.w, acc[0][c][3]);
                    acc[1][c][0] = fmaf(pv.y, vv.x, acc[1][c][0]); acc[1][c][1] = fmaf(pv.y, vv.y, acc[1][c][1]);
                    acc[1][c][2] = fmaf(pv.y, vv.z, acc[1][c][2]); acc[1][c][3] = fmaf(pv.y, vv.w, acc[1][c][3]);
                    acc[2][c][0] = fmaf(pv.z, vv.x, acc[2][c][0]); acc[2][c][1] = fmaf(pv.z, vv.y, acc[2][c][1]);
                    acc[2][c][2] = fmaf(pv.z, vv.z, acc[2][c][2]); acc[2][c][3] = fmaf(pv.z, vv.w, acc[2][c][3]);
                    acc[3][c][0] = fmaf(pv.w, vv.x, acc[3][c][0]); acc[3][c][1] = fmaf(pv.w, vv.y, acc[3][c][1]);
                    acc[3][c][2] = fmaf(pv.w, vv.z, acc[3][c][2]); acc[3][c][3] = fmaf(pv.w, vv.w, acc[3][c][3]);
                }
            }
        }
    }
    pdl_trigger();
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        if (!active[e]) continue;
        const float inv = sight_inverse(sight, hq[e], m[e], l[e]);
        const size_t o = (size_t)(tok0 + tok[e]) * out_stride + hq[e] * dv;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int col = 4 * lj + 32 * c;
            if (col < dv) {
#pragma unroll
                for (int x = 0; x < 4; ++x)
                    store_out<T>(out, out_f32, o + col + x,
                                 acc[e][c][x] * inv * sight_gate<T>(sight, (size_t)(tok0 + tok[e]),
                                                                    hq[e], dv, col + x));
            }
        }
    }
}


// ------------------------------------------------------------------------------------------
// The same attention on the tensor cores, for bfloat16 rows of D = 64 or 128 features (keys and
// values alike): mma.sync m16n8k16, a block of four warps takes 64 rows, a warp 16 of them against
// tiles of 32 keys that come through two stages of cp.async.  Nothing loses precision against the
// kernels above: the products of bfloat16 queries and keys are exact, and a softmax weight enters
// its product with the values as three bfloat16 terms whose sum is the float32 weight.  What the
// tensor cores add up is a tile's share only, the small terms first; the running sums of a row are
// float32 multiply-adds (acc <- acc * correction + tile's share).  Scores, cap, penalty, maximum and
// exponentials are those of the kernels above.  A row's tiles lie at
// absolute multiples of 32, so its result does not depend on what shares its block or its step (but
// on whether the step's tiles are of 32 or 64 rows).
// The kernel above runs the same work on the CUDA cores, where a prompt of 2,048 tokens of 16 heads
// of 128 on 4 kv heads takes 734 us with a window of 1,024 and a cap, 147 us here, 39 us of
// 512 tokens against 221 (its distance from 64 bits 2.5e-7 of the result against 4.7e-7); without
// window and cap 202 us against 1,141.  What bounds it: twelve warps an SM, each a chain of two
// products, a maximum and exponentials a tile; the tensor pipe is busy a third of the time.
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ void ldmatrix4(unsigned (&r)[4], const void* p) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void ldmatrix4_trans(unsigned (&r)[4], const void* p) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void mma16816(float (&c)[4], const unsigned (&a)[4], unsigned b0,
                                         unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ unsigned pack2(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const unsigned*>(&v);
}
// x and y as sums of three bfloat16 numbers each: all 24 bits of a float32 mantissa
__device__ __forceinline__ void split3(float x, float y, unsigned& a, unsigned& b, unsigned& c) {
    a = pack2(x, y);
    const float rx = x - __uint_as_float(a << 16), ry = y - __uint_as_float(a & 0xffff0000u);
    b = pack2(rx, ry);
    c = pack2(rx - __uint_as_float(b << 16), ry - __uint_as_float(b & 0xffff0000u));
}

constexpr int MKT = 32;           // keys of a tile

template <int D, int HALVES> constexpr size_t mma_smem() {
    return (size_t)4 * HALVES * MKT * (D + 8) * sizeof(__nv_bfloat16);
}

template <int D, int HALVES>
__global__ void __launch_bounds__(128, 3)
attn_chunk_mma_kernel(const __nv_bfloat16* __restrict__ q, int q_stride, void* __restrict__ out,
                      int out_stride, const __nv_bfloat16* __restrict__ k_pages,
                      const __nv_bfloat16* __restrict__ v_pages,
                      const int* __restrict__ block_table, int table_stride, int num_pages,
                      const int* __restrict__ seq_slot, const int* __restrict__ seq_qstart,
                      const int* __restrict__ seq_qlen, const int* __restrict__ seq_pos0,
                      const WorkItem* __restrict__ items, const float* __restrict__ r1,
                      const float* __restrict__ r2, int heads, int kv_heads, int page, float scale,
                      Sight sight, int out_f32, int parts, int* __restrict__ status) {
    using T = __nv_bfloat16;
    constexpr int LD = D + 8;                        // a row's stride: ldmatrix without conflicts
    constexpr int NT = MKT / 8, DT = D / 8, CH = D / 8;
    constexpr int TEAM = 128 / HALVES, WARPS = 4 / HALVES, MROWS = 16 * WARPS;
    extern __shared__ __align__(16) float smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int half = warp / WARPS, tid = threadIdx.x % TEAM;  // which tiles; thread of the half
    T* k_s = reinterpret_cast<T*>(smem) + half * 4 * MKT * LD;       // [2][MKT][LD]
    T* v_s = k_s + 2 * MKT * LD;                     // [2][MKT][LD]
    __shared__ int pages_all[HALVES][3][MKT];             // the pages of three tiles in a row
    __shared__ int gone_s;                           // a key inside the range had no page
    int (*pages_s)[MKT] = pages_all[half];
    auto half_sync = [&]() {
        asm volatile("bar.sync %0, %1;\n" ::"r"(1 + half), "n"(TEAM) : "memory");
    };

    WorkItem it = items[blockIdx.x / parts];         // (`parts` blocks share an item's rows)
    it.row0 += (int)(blockIdx.x % parts) * MROWS;
    if (it.kv_begin >= it.kv_end || it.row0 >= seq_qlen[it.seq] * (heads / kv_heads)) {
        pdl_wait();
        return;
    }
    const int hk = blockIdx.y;
    const int g = heads / kv_heads;
    const int qlen = seq_qlen[it.seq], pos0 = seq_pos0[it.seq];
    const int slot = seq_slot[it.seq], tok0 = seq_qstart[it.seq];
    const int rows_total = qlen * g;
    const int gid = lane >> 2, tig = lane & 3;
    const bool penalty = r1 != nullptr;

    // the rows of this thread: gid and gid + 8 of the warp's sixteen
    bool active[2];
    int tok[2], hq[2], pos[2], row_lo[2], row_hi[2], row_first[2];
    float pen1[2], pen2[2], m[2], l[2];
    int all_lo = 0, all_hi = 0x7fffffff;             // keys [all_lo, all_hi) are seen by every row
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int r = it.row0 + warp % WARPS * 16 + gid + 8 * e;
        active[e] = r < rows_total;
        tok[e] = active[e] ? r / g : 0;
        hq[e] = hk * g + (active[e] ? r % g : 0);
        pos[e] = pos0 + tok[e];
        pen1[e] = penalty ? r1[hq[e]] : 0.0f;
        pen2[e] = penalty ? r2[hq[e]] : 0.0f;
        row_lo[e] = max(it.kv_begin, sight_lo(sight, pos[e]));
        row_first[e] = it.kv_begin > 0 ? 0 : sight_first(sight, row_lo[e]);
        row_hi[e] = active[e] ? min(it.kv_end, pos[e] + 1) : 0;
        if (active[e]) {
            all_lo = max(all_lo, row_lo[e]);
            all_hi = min(all_hi, row_hi[e]);
        }
        m[e] = -INFINITY;
        l[e] = 0.0f;
    }
    const bool any = it.row0 + warp % WARPS * 16 < rows_total;
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
        all_lo = max(all_lo, __shfl_xor_sync(0xffffffffu, all_lo, o));
        all_hi = min(all_hi, __shfl_xor_sync(0xffffffffu, all_hi, o));
    }
    const int last_row = min(it.row0 + MROWS, rows_total) - 1;
    const int max_pos = pos0 + last_row / g, min_pos = pos0 + it.row0 / g;
    const int k_hi = min(it.kv_end, max_pos + 1);
    const int k_lo_true = max(it.kv_begin, sight_lo(sight, min_pos));
    const int k_first = it.kv_begin > 0 ? 0 : sight_first(sight, k_lo_true);
    const TileWalk walk(k_lo_true, k_first, MKT);
    // two halves: the first two warps take the tiles of even number, the others those of odd number
    // (by absolute place, so that a tile's half does not depend on what else the block holds)
    auto mine = [&](int kt) {
        while (HALVES == 2 && kt < k_hi && ((kt / MKT) & 1) != half) kt = walk.next(kt, MKT);
        return kt;
    };
    auto after = [&](int kt) { return mine(walk.next(kt, MKT)); };

    // the page of key kt + thread; -1 for keys that no row sees, -2 for a seen key without a page
    auto page_of = [&](int kt) {
        const int kpos = kt + tid;
        if (tid >= MKT || kt >= k_hi || (kpos < k_lo_true && kpos >= k_first) || kpos >= k_hi) return -1;
        const int id = block_table[(size_t)slot * table_stride + kpos / page];
        return id >= 0 && id < num_pages ? id : -2;
    };
    auto put_page = [&](int id, int which) {
        if (tid < MKT) pages_s[which][tid] = id;
        if (id == -2) {
            gone_s = 1;
            if (status != nullptr) atomicExch(status, 2);
        }
    };
    auto load_tile = [&](int kt, int which, int stage) {
        T* kd = k_s + stage * MKT * LD;
        T* vd = v_s + stage * MKT * LD;
#pragma unroll
        for (int i = 0; i < MKT * CH / TEAM; ++i) {
            const int c = tid + TEAM * i, j = c / CH, ch = c % CH;
            const int id = pages_s[which][j];
            const size_t at = id >= 0 ? ((size_t)id * kv_heads + hk) * page +
                                            (size_t)((kt + j) % page) : 0;
            const int bytes = id >= 0 ? 16 : 0;
            const unsigned ka = (unsigned)__cvta_generic_to_shared(kd + j * LD + ch * 8);
            const unsigned va = (unsigned)__cvta_generic_to_shared(vd + j * LD + ch * 8);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(ka),
                         "l"(k_pages + at * D + ch * 8), "r"(bytes) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(va),
                         "l"(v_pages + at * sight.v_stride + ch * 8), "r"(bytes) : "memory");
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };

    if (threadIdx.x == 0) gone_s = 0;
    const int start = mine(walk.start), second = after(start);
    const int page_a = page_of(start), page_b = page_of(second);
    __syncthreads();
    put_page(page_a, 0);
    put_page(page_b, 1);
    __syncthreads();
    pdl_wait();            // q, and the keys and values of this step's tokens, are just written
    load_tile(start, 0, 0);

    // q fragments straight from global memory (read once)
    unsigned qf[D / 16][4];
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const T* p = q + (size_t)(tok0 + tok[e]) * q_stride + hq[e] * D + kk * 16 + 2 * tig;
            qf[kk][e] = active[e] ? *reinterpret_cast<const unsigned*>(p) : 0u;
            qf[kk][e + 2] = active[e] ? *reinterpret_cast<const unsigned*>(p + 8) : 0u;
        }
    float acc[DT][4];
#pragma unroll
    for (int j = 0; j < DT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][e] = 0.0f;

    const int mat = lane >> 3, mr = lane & 7;
    const float inv_cap = sight.softcap > 0.0f ? 1.0f / sight.softcap : 0.0f;
    int stage = 0, which = 0;
    for (int kt = start; kt < k_hi; stage ^= 1) {
        const int next = after(kt), which_next = which == 2 ? 0 : which + 1;
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        half_sync();                 // this tile has landed, the one before it has been used
        int ahead = -1;
        if (next < k_hi) {
            load_tile(next, which_next, stage ^ 1);
            ahead = page_of(after(next));
        }
        if (any) {
            const T* kb = k_s + stage * MKT * LD;
            const T* vb = v_s + stage * MKT * LD;
            // q . k in two chains of half the features each, added in float32
            float s[NT][4];
#pragma unroll
            for (int j = 0; j < NT; j += 2) {
                float c[2][2][4];
#pragma unroll
                for (int i = 0; i < 16; ++i) c[i >> 3][(i >> 2) & 1][i & 3] = 0.0f;
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk) {
                    unsigned b[4];
                    ldmatrix4(b, kb + ((j + (mat >> 1)) * 8 + mr) * LD + kk * 16 + (mat & 1) * 8);
                    mma16816(c[kk & 1][0], qf[kk], b[0], b[1]);
                    mma16816(c[kk & 1][1], qf[kk], b[2], b[3]);
                }
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    s[j][x] = c[0][0][x] + c[1][0][x];
                    s[j + 1][x] = c[0][1][x] + c[1][1][x];
                }
            }
            const bool inside = kt >= all_lo && kt + MKT <= all_hi && gone_s == 0;
            // as sight_score: scale, penalty, cap
            if (!penalty) {
#pragma unroll
                for (int j = 0; j < NT; ++j)
#pragma unroll
                    for (int x = 0; x < 4; ++x) s[j][x] *= scale;
            } else {
#pragma unroll
                for (int j = 0; j < NT; ++j)
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        const int e = x >> 1;
                        const float dist = (float)(pos[e] - (kt + j * 8 + 2 * tig + (x & 1)));
                        s[j][x] *= scale;
                        s[j][x] -= sight.linear ? pen1[e] * dist : pen1[e] * log1pf(pen2[e] * dist);
                    }
            }
            if (sight.softcap > 0.0f) {
                float far = 0.0f;
#pragma unroll
                for (int j = 0; j < NT; ++j)
#pragma unroll
                    for (int x = 0; x < 4; ++x) far = fmaxf(far, fabsf(s[j][x]));
                if (__any_sync(0xffffffffu, far * inv_cap > TANH_NEAR)) {
#pragma unroll
                    for (int j = 0; j < NT; ++j)
#pragma unroll
                        for (int x = 0; x < 4; ++x)
                            s[j][x] = sight.softcap *
                                      (fabsf(s[j][x]) * inv_cap > TANH_NEAR
                                           ? tanhf(s[j][x] / sight.softcap)
                                           : tanh_near(s[j][x] * inv_cap));
                } else {
#pragma unroll
                    for (int j = 0; j < NT; ++j)
#pragma unroll
                        for (int x = 0; x < 4; ++x)
                            s[j][x] = sight.softcap * tanh_near(s[j][x] * inv_cap);
                }
            }
            if (!inside) {
#pragma unroll
                for (int j = 0; j < NT; ++j)
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        const int e = x >> 1, key = j * 8 + 2 * tig + (x & 1), kpos = kt + key;
                        const bool valid = (kpos >= row_lo[e] || kpos < row_first[e]) &&
                                           kpos < row_hi[e] && pages_s[which][key] >= 0;
                        if (!valid) s[j][x] = -INFINITY;
                    }
            }
            float corr[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float top = m[e];
#pragma unroll
                for (int j = 0; j < NT; ++j) top = fmaxf(top, fmaxf(s[j][2 * e], s[j][2 * e + 1]));
                top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
                top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
                // (a row that has seen nothing yet: every weight is exp(-inf) = 0)
                const float use = top == -INFINITY ? 0.0f : top;
                corr[e] = expf(m[e] - use);
                m[e] = top;
                float sum = 0.0f;
#pragma unroll
                for (int j = 0; j < NT; ++j)
#pragma unroll
                    for (int x = 2 * e; x < 2 * e + 2; ++x) {
                        s[j][x] = expf(s[j][x] - use);
                        sum += s[j][x];
                    }
                l[e] = l[e] * corr[e] + sum;
            }
            unsigned pw[3][MKT / 16][4];             // the weights' terms, largest first
#pragma unroll
            for (int ks = 0; ks < MKT / 16; ++ks)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float* p = &s[2 * ks + (i >> 1)][2 * (i & 1)];
                    split3(p[0], p[1], pw[0][ks][i], pw[1][ks][i], pw[2][ks][i]);
                }
#pragma unroll
            for (int jd = 0; jd < DT; jd += 2) {
                unsigned b[MKT / 16][4];
                float t0[4] = {0.0f, 0.0f, 0.0f, 0.0f}, t1[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                for (int ks = 0; ks < MKT / 16; ++ks)
                    ldmatrix4_trans(b[ks], vb + (ks * 16 + (mat & 1) * 8 + mr) * LD +
                                               (jd + (mat >> 1)) * 8);
#pragma unroll
                for (int term = 2; term >= 0; --term)
#pragma unroll
                    for (int ks = 0; ks < MKT / 16; ++ks) {
                        mma16816(t0, pw[term][ks], b[ks][0], b[ks][1]);
                        mma16816(t1, pw[term][ks], b[ks][2], b[ks][3]);
                    }
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    acc[jd][x] = fmaf(acc[jd][x], corr[x >> 1], t0[x]);
                    acc[jd + 1][x] = fmaf(acc[jd + 1][x], corr[x >> 1], t1[x]);
                }
            }
        }
        // (the pages of the tile before this one were last read before the barrier above)
        put_page(ahead, which == 0 ? 2 : which - 1);
        which = which_next;
        kt = next;
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    if (HALVES == 1) pdl_trigger();
    // the second half's sums join the first's
    float* joint = smem + tid;                       // [DT * 4 + 4][64]
    if (HALVES == 2) __syncthreads();
    if (half == 1) {
#pragma unroll
        for (int j = 0; j < DT; ++j)
#pragma unroll
            for (int x = 0; x < 4; ++x) joint[(4 * j + x) * 64] = acc[j][x];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            joint[(4 * DT + e) * 64] = m[e];
            joint[(4 * DT + 2 + e) * 64] = l[e];
        }
    }
    if (HALVES == 2) {
        __syncthreads();
        pdl_trigger();
        if (half == 1) return;
        float mine_f[2], other_f[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const float mo = joint[(4 * DT + e) * 64], top = fmaxf(m[e], mo);
            const float use = top == -INFINITY ? 0.0f : top;
            mine_f[e] = expf(m[e] - use);
            other_f[e] = expf(mo - use);
            l[e] = l[e] * mine_f[e] + joint[(4 * DT + 2 + e) * 64] * other_f[e];
            m[e] = top;
        }
#pragma unroll
        for (int j = 0; j < DT; ++j)
#pragma unroll
            for (int x = 0; x < 4; ++x)
                acc[j][x] = fmaf(acc[j][x], mine_f[x >> 1],
                                 joint[(4 * j + x) * 64] * other_f[x >> 1]);
    }
    const bool pairs = out_stride % 2 == 0 && (uintptr_t)out % (out_f32 ? 8 : 4) == 0;
    unsigned spoilt = 0;                             // rows that met an infinity or NaN
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        l[e] += __shfl_xor_sync(0xffffffffu, l[e], 1);
        l[e] += __shfl_xor_sync(0xffffffffu, l[e], 2);
        if (!active[e]) continue;
        const float inv = sight_inverse(sight, hq[e], m[e], l[e]);
        const size_t token = (size_t)(tok0 + tok[e]);
        const size_t o = token * out_stride + hq[e] * D;
        float zero = 0.0f;
#pragma unroll
        for (int j = 0; j < DT; ++j) {
            const int col = j * 8 + 2 * tig;
            const float a = acc[j][2 * e] * inv * sight_gate<T>(sight, token, hq[e], D, col);
            const float b = acc[j][2 * e + 1] * inv *
                            sight_gate<T>(sight, token, hq[e], D, col + 1);
            zero = fmaf(a, 0.0f, fmaf(b, 0.0f, zero));
            if (!pairs) {
                store_out<T>(out, out_f32, o + col, a);
                store_out<T>(out, out_f32, o + col + 1, b);
            } else if (out_f32) {
                store_pair((float*)out + o + col, a, b);
            } else {
                store_pair((T*)out + o + col, a, b);
            }
        }
        if (!(zero == 0.0f)) spoilt |= 1u << (gid + 8 * e);
    }
    spoilt = __reduce_or_sync(0xffffffffu, spoilt);
    if (spoilt == 0) return;
    __syncwarp();
    for (int row = 0; row < 16; ++row) {
        if (!((spoilt >> row) & 1u)) continue;
        const int r = it.row0 + warp % WARPS * 16 + row, t = r / g, h = hk * g + r % g;
        float mr, lr, res[D / 32];
        row_again<D>(q + (size_t)(tok0 + t) * q_stride + h * D, k_pages, v_pages,
                     block_table + (size_t)slot * table_stride, num_pages, hk, kv_heads, page,
                     pos0 + t, it.kv_begin, it.kv_end, scale, penalty ? r1[h] : 0.0f,
                     penalty ? r2[h] : 0.0f, penalty, sight, mr, lr, res);
        const float inv = sight_inverse(sight, h, mr, lr);
        const size_t o = (size_t)(tok0 + t) * out_stride + h * D;
#pragma unroll
        for (int i = 0; i < D / 32; ++i) {
            const int col = lane + 32 * i;
            store_out<T>(out, out_f32, o + col,
                         res[i] * inv * sight_gate<T>(sight, (size_t)(tok0 + t), h, D, col));
        }
    }
}

// ------------------------------------------------------------------------------------------
// Steps in which every sequence brings one token.  A block takes a sequence and a kv head; its
// eight warps share the key tiles of the token's chunk out among themselves (warp w takes tiles
// w, w + 8, ...) and each works alone: it asks for its tile's 32 key rows and 32 value rows at
// once (cp.async, 16 bytes a piece, into shared memory of its own), so a tile costs one trip to
// memory; then a lane takes its key's row, and the values come row by row as the weights are
// handed round.  All RW query heads of the group ride on every key read.  The
// warps' partial results (maximum, sum, weighted values) are merged in ascending order of the
// warps.  Sizes as the kernel above; RW >= heads / kv_heads.
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ void cp_async_16(void* dst, const void* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}

// What the kernel for single tokens does besides the attention when `on`: it turns its token's
// queries by position (in shared memory), turns and stores the token's key and value of its kv
// head in the pages before it reads them (write_kv; q's row is then [q (H dk) | k (G dk) |
// v (G dv) | ...]), and it finishes every head's result itself - turned back by position where fv
// is given, times sigmoid(gate) where a gate is given, rounded to T - as kv_write_rotated and
// attn_finish_kernel do around the other kernels, with the same arithmetic.
struct Fuse {
    int on;
    const float* fk;
    int rot;
    const float* fv;
    int write_kv;
    const void* gate;
    int ld_gate;
};

// The token's queries of `g` heads from h0 on into Qs [rw][dk] as float32 (zeros beyond them) and,
// with fuse.on, what Fuse says of queries, key and value.  Ends with a barrier of the block.
template <typename T>
__device__ __forceinline__ void decode_begin(
    float* Qs, int rw, int g, int h0, int hk, const T* __restrict__ q, int q_stride, int tok,
    int slot, int pos, T* k_pages, T* v_pages, const int* __restrict__ block_table,
    int table_stride, int num_pages, int heads, int kv_heads, int dk, int dv, int page,
    const Fuse& fuse, int* __restrict__ status) {
    for (int e = threadIdx.x; e < rw * dk; e += (int)blockDim.x) {
        const int i = e / dk, d = e - i * dk;
        Qs[e] = i < g ? to_float(q[(size_t)tok * q_stride + (h0 + i) * dk + d]) : 0.0f;
    }
    __syncthreads();
    if (fuse.on) {
        const float fpos = (float)pos;
        const int half = fuse.rot / 2;
        for (int e = threadIdx.x; e < g * half; e += (int)blockDim.x) {
            const int i = e / half, p = e - i * half;
            float sn, cs, ra, rb;
            sincosf(fpos * fuse.fk[p], &sn, &cs);
            rope_rotate(Qs[i * dk + p], Qs[i * dk + p + half], cs, sn, ra, rb);
            Qs[i * dk + p] = to_float(from_float<T>(ra));        // rounded as when q goes through memory
            Qs[i * dk + p + half] = to_float(from_float<T>(rb));
        }
        if (fuse.write_kv) {
            const int page_id = block_table[(size_t)slot * table_stride + pos / page];
            if (page_id < 0 || page_id >= num_pages) {           // never written outside the pool
                if (threadIdx.x == 0 && status != nullptr) atomicExch(status, 1);
            } else {
                const size_t at = ((size_t)page_id * kv_heads + hk) * page + (size_t)(pos % page);
                const T* ks = q + (size_t)tok * q_stride + heads * dk + hk * dk;
                const T* vs = q + (size_t)tok * q_stride + (heads + kv_heads) * dk + hk * dv;
                T* kd = k_pages + at * dk;
                T* vd = v_pages + at * dv;
                for (int i = threadIdx.x; i < dk - half; i += (int)blockDim.x) {
                    if (i < half) {
                        float sn, cs, ra, rb;
                        sincosf(fpos * fuse.fk[i], &sn, &cs);
                        rope_rotate(to_float(ks[i]), to_float(ks[i + half]), cs, sn, ra, rb);
                        kd[i] = from_float<T>(ra);
                        kd[i + half] = from_float<T>(rb);
                    } else {
                        kd[i + half] = ks[i + half];
                    }
                }
                if (fuse.fv != nullptr) {
                    const int vhalf = dv / 2;
                    for (int i = threadIdx.x; i < dv - vhalf; i += (int)blockDim.x) {
                        if (i < vhalf) {
                            float sn, cs, ra, rb;
                            sincosf(fpos * fuse.fv[i], &sn, &cs);
                            rope_rotate(to_float(vs[i]), to_float(vs[i + vhalf]), cs, sn, ra, rb);
                            vd[i] = from_float<T>(ra);
                            vd[i + vhalf] = from_float<T>(rb);
                        } else {
                            vd[i + vhalf] = vs[i + vhalf];
                        }
                    }
                } else {
                    for (int i = threadIdx.x; i < dv; i += (int)blockDim.x) vd[i] = vs[i];
                }
            }
        }
        __syncthreads();                             // the block reads what it has just stored
    }
}

// The warps' partial results (Pml [warps][rw][2] maximum and sum, Pacc [warps][rw][dv]) merged in
// ascending order of the warps, a warp a head, and finished.
template <typename T>
__device__ __forceinline__ void decode_finish(const float* Pml, float* Pacc, int rw, int warps,
                                              int g, int h0, int tok, int pos, void* out,
                                              int out_stride, int dv, const Sight& sight,
                                              int out_f32, const Fuse& fuse) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = warp; i < g; i += warps) {
        float top = -INFINITY;
        for (int w = 0; w < warps; ++w) top = fmaxf(top, Pml[(w * rw + i) * 2]);
        float sum = 0.0f, res[MAX_D / 32];
#pragma unroll
        for (int b = 0; b < MAX_D / 32; ++b) res[b] = 0.0f;
        for (int w = 0; w < warps; ++w) {
            const float mw = Pml[(w * rw + i) * 2];
            if (mw == -INFINITY) continue;
            const float f = expf(mw - top);
            sum = fmaf(Pml[(w * rw + i) * 2 + 1], f, sum);
#pragma unroll
            for (int b = 0; b < MAX_D / 32; ++b) {
                const int dd = lane + 32 * b;
                if (dd < dv) res[b] = fmaf(Pacc[(size_t)(w * rw + i) * dv + dd], f, res[b]);
            }
        }
        const float inv = sight_inverse(sight, h0 + i, top, sum);
        const size_t o = (size_t)tok * out_stride + (h0 + i) * dv;
        if (fuse.on) {
            // the head's result through shared memory (the place of the first warp's share of
            // this head, which only this warp reads), so that a lane finds its feature's pair
            float* fin = Pacc + (size_t)i * dv;
            __syncwarp();
#pragma unroll
            for (int b = 0; b < MAX_D / 32; ++b) {
                const int dd = lane + 32 * b;
                if (dd < dv) fin[dd] = res[b] * inv;
            }
            __syncwarp();
            const int vhalf = dv / 2;
            const T* gt = fuse.gate
                              ? (const T*)fuse.gate + (size_t)tok * fuse.ld_gate + (h0 + i) * dv
                              : nullptr;
#pragma unroll
            for (int b = 0; b < MAX_D / 32; ++b) {
                const int dd = lane + 32 * b;
                if (dd >= dv) continue;
                float x = fin[dd];
                if (fuse.fv != nullptr && dd < 2 * vhalf) {
                    const int p = dd < vhalf ? dd : dd - vhalf;
                    float sn, cs, ra, rb;
                    sincosf((float)pos * fuse.fv[p], &sn, &cs);
                    rope_rotate(fin[p], fin[p + vhalf], cs, -sn, ra, rb);
                    x = dd < vhalf ? ra : rb;
                }
                if (gt) x *= 1.0f / (1.0f + expf(-to_float(gt[dd])));
                ((T*)out)[o + dd] = from_float<T>(x);
            }
            continue;
        }
#pragma unroll
        for (int b = 0; b < MAX_D / 32; ++b) {
            const int dd = lane + 32 * b;
            if (dd < dv)
                store_out<T>(out, out_f32, o + dd,
                             res[b] * inv * sight_gate<T>(sight, (size_t)tok, h0 + i, dv, dd));
        }
    }
}

template <typename T, int RW>
__global__ void __launch_bounds__(ROWS * 32)
attn_chunk_decode_kernel(const T* __restrict__ q, int q_stride, void* __restrict__ out,
                         int out_stride, T* k_pages, T* v_pages,
                         const int* __restrict__ block_table,
                         int table_stride, int num_pages, const int* __restrict__ seq_slot,
                         const int* __restrict__ seq_qstart, const int* __restrict__ seq_pos0,
                         const float* __restrict__ r1, const float* __restrict__ r2, int heads,
                         int kv_heads, int dk, int dv, int page, float scale, Sight sight,
                         int out_f32, Fuse fuse, int* __restrict__ status) {
    constexpr int PN = Piece<T>::N;
    extern __shared__ __align__(16) float smem[];
    float* Qs = smem;                                // [RW][dk]
    float* Pml = Qs + RW * dk;                       // [ROWS warps][RW][2]
    float* Pacc = Pml + ROWS * RW * 2;               // [ROWS warps][RW][dv]
    // a warp's tile: key rows at a stride that keeps 16-byte reads of 8 lanes on different banks
    const int k_stride = ((dk * (int)sizeof(T) + 127) / 128) * 128 + 16;       // bytes
    // values that are the first dv features of the keys (one set of pages, rows of dk) are read
    // from the key tile
    const bool v_in_k = v_pages == k_pages && sight.v_stride == dk;
    const int tile_bytes = TILE * k_stride + (v_in_k ? 0 : TILE * dv * (int)sizeof(T));
    char* mine = reinterpret_cast<char*>(Pacc + ROWS * RW * dv) +
                 (size_t)(threadIdx.x >> 5) * tile_bytes;
    char* Kt = mine;
    const T* Vt = reinterpret_cast<const T*>(mine + TILE * k_stride);
    // a kv head with more than RW query heads is shared by several blocks, RW heads each
    const int parts = gridDim.y / kv_heads;
    const int seq = blockIdx.x, hk = blockIdx.y / parts;
    const int h0 = hk * (heads / kv_heads) + (blockIdx.y % parts) * RW;   // the block's first head
    const int g = min(RW, (hk + 1) * (heads / kv_heads) - h0);            // and how many it has
    const int pos = seq_pos0[seq], slot = seq_slot[seq], tok = seq_qstart[seq];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int lo = sight_lo(sight, pos), hi = pos + 1, first = sight_first(sight, lo);
    // the tiles: those of the kept first keys, then from the tile of `lo` on, dealt out in turn
    const TileWalk walk(lo, first, TILE);
    const int first_tiles = walk.jump_at > 0 ? walk.jump_at / TILE : 0;
    const int near0 = walk.jump_at > 0 ? walk.jump_to : walk.start;
    const int n_tiles = first_tiles + (hi - near0 + TILE - 1) / TILE;
    const bool penalty = r1 != nullptr;
    float pen1[RW], pen2[RW], m[RW], l[RW];
#pragma unroll
    for (int i = 0; i < RW; ++i) {
        const int hq = h0 + min(i, g - 1);
        pen1[i] = penalty ? r1[hq] : 0.0f;
        pen2[i] = penalty ? r2[hq] : 0.0f;
        m[i] = -INFINITY;
        l[i] = 0.0f;
    }
    pdl_wait();
    decode_begin<T>(Qs, RW, g, h0, hk, q, q_stride, tok, slot, pos, k_pages, v_pages, block_table,
                    table_stride, num_pages, heads, kv_heads, dk, dv, page, fuse, status);
    float acc[RW][MAX_D / 32];
#pragma unroll
    for (int i = 0; i < RW; ++i)
#pragma unroll
        for (int b = 0; b < MAX_D / 32; ++b) acc[i][b] = 0.0f;

    for (int ti = warp; ti < n_tiles; ti += ROWS) {
        const int kt = ti < first_tiles ? ti * TILE : near0 + (ti - first_tiles) * TILE;
        const int kpos = kt + lane;
        bool valid = (kpos >= lo || kpos < first) && kpos < hi;
        size_t row = 0;
        if (valid) {
            const int page_id = block_table[(size_t)slot * table_stride + kpos / page];
            if (page_id < 0 || page_id >= num_pages) {
                valid = false;
                if (status != nullptr) atomicExch(status, 2);
            } else {
                row = ((size_t)page_id * kv_heads + hk) * page + (size_t)(kpos % page);
            }
        }
        __syncwarp();                                // the tile before this one has been used
        {
            const int ck = dk / PN, cv = dv / PN;
            for (int e = lane; e < TILE * ck; e += 32) {
                const int j = e / ck, w = e - j * ck;
                const unsigned long long rj = __shfl_sync(0xffffffffu, (unsigned long long)row, j);
                const bool ok = __shfl_sync(0xffffffffu, (int)valid, j) != 0;
                if (ok) cp_async_16(Kt + j * k_stride + w * 16, k_pages + (size_t)rj * dk + w * PN);
            }
            for (int e = lane; e < (v_in_k ? 0 : TILE * cv); e += 32) {
                const int j = e / cv, w = e - j * cv;
                const unsigned long long rj = __shfl_sync(0xffffffffu, (unsigned long long)row, j);
                const bool ok = __shfl_sync(0xffffffffu, (int)valid, j) != 0;
                if (ok)
                    cp_async_16(mine + TILE * k_stride + ((size_t)j * dv + w * PN) * sizeof(T),
                                v_pages + (size_t)rj * sight.v_stride + w * PN);
            }
            asm volatile("cp.async.commit_group;\n" ::: "memory");
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            __syncwarp();
        }
        float s[RW];
#pragma unroll
        for (int i = 0; i < RW; ++i) s[i] = 0.0f;
        const uint4* kp = reinterpret_cast<const uint4*>(Kt + lane * k_stride);
#pragma unroll 4
        for (int piece = 0; piece < dk / PN; ++piece) {
            float f[PN];
            Piece<T>::unpack(valid ? kp[piece] : make_uint4(0u, 0u, 0u, 0u), f);
#pragma unroll
            for (int i = 0; i < RW; ++i) {
                const float4* q4 = reinterpret_cast<const float4*>(Qs + i * dk + piece * PN);
#pragma unroll
                for (int x = 0; x < PN / 4; ++x) {
                    const float4 qq = q4[x];
                    s[i] = fmaf(qq.x, f[4 * x + 0], s[i]);
                    s[i] = fmaf(qq.y, f[4 * x + 1], s[i]);
                    s[i] = fmaf(qq.z, f[4 * x + 2], s[i]);
                    s[i] = fmaf(qq.w, f[4 * x + 3], s[i]);
                }
            }
        }
        float p[RW];
        const float dist = (float)(pos - kpos);
#pragma unroll
        for (int i = 0; i < RW; ++i) {
            const float sc = valid ? sight_score(sight, s[i], scale, pen1[i], pen2[i], penalty, dist)
                                   : -INFINITY;
            const float m_new = fmaxf(m[i], warp_max(sc));
            if (m_new == -INFINITY) {
                p[i] = 0.0f;
                continue;
            }
            p[i] = valid ? expf(sc - m_new) : 0.0f;
            const float corr = expf(m[i] - m_new);
            l[i] = l[i] * corr + warp_sum(p[i]);
#pragma unroll
            for (int b = 0; b < MAX_D / 32; ++b) acc[i][b] *= corr;
            m[i] = m_new;
        }
#pragma unroll 4
        for (int j = 0; j < TILE; ++j) {
            float pj[RW];
            bool zero = true;
#pragma unroll
            for (int i = 0; i < RW; ++i) {
                pj[i] = __shfl_sync(0xffffffffu, p[i], j);
                zero &= pj[i] == 0.0f;
            }
            if (zero) continue;
            const T* vr = v_in_k ? reinterpret_cast<const T*>(Kt + j * k_stride) : Vt + (size_t)j * dv;
#pragma unroll
            for (int b = 0; b < MAX_D / 32; ++b) {
                const int dd = lane + 32 * b;
                if (dd < dv) {
                    const float vv = to_float(vr[dd]);
#pragma unroll
                    for (int i = 0; i < RW; ++i) acc[i][b] = fmaf(pj[i], vv, acc[i][b]);
                }
            }
        }
    }
    pdl_trigger();
#pragma unroll
    for (int i = 0; i < RW; ++i) {
        if (lane == 0) {
            Pml[(warp * RW + i) * 2] = m[i];
            Pml[(warp * RW + i) * 2 + 1] = l[i];
        }
#pragma unroll
        for (int b = 0; b < MAX_D / 32; ++b) {
            const int dd = lane + 32 * b;
            if (dd < dv) Pacc[(size_t)(warp * RW + i) * dv + dd] = acc[i][b];
        }
    }
    __syncthreads();
    decode_finish<T>(Pml, Pacc, RW, ROWS, g, h0, tok, pos, out, out_stride, dv, sight, out_f32, fuse);
}

// ------------------------------------------------------------------------------------------
// The same for bfloat16 rows of D = 64 or 128 features (keys and values alike), up to eight query
// heads a kv head, with both products on the tensor cores as attn_chunk_mma_kernel forms them (a
// block's heads are the first eight of a product's sixteen rows).  A warp's tiles are 16 keys and
// come through three stages of its own, so that two are on their way while one is worked on; a
// block of four warps leaves room for a second on its SM, eight warps serve steps of few sequences
// (four or eight partial results are merged: a row's bits depend on which, so on the step's size.  Four
// warps with two shares of the tiles each would give one order, and were slower: 64 sequences of 700
// keys of 64 features 15.8 -> 19.9 us, of one key on 16 kv heads 11.0 -> 14.7).
// Bound by memory and by the trips to it: 64 sequences of up to 700 keys (614 on average, 80 MB), 16
// heads on 4 kv heads of 128: 26 us, 3.0 TB/s (the kernel above, which asks for a tile, waits and works:
// 81).
// ------------------------------------------------------------------------------------------
constexpr int DKT = 16, DSTAGES = 3, DRW = 8;

template <int D, int WARPS> constexpr size_t decode_mma_smem() {
    return (size_t)(DRW * D + WARPS * DRW * 2) * sizeof(float) +
           (size_t)WARPS * DSTAGES * 2 * DKT * (D + 8) * sizeof(__nv_bfloat16);
}

template <int D, int WARPS>
__global__ void __launch_bounds__(WARPS * 32)
attn_chunk_decode_mma_kernel(const __nv_bfloat16* __restrict__ q, int q_stride,
                             void* __restrict__ out, int out_stride, __nv_bfloat16* k_pages,
                             __nv_bfloat16* v_pages, const int* __restrict__ block_table,
                             int table_stride, int num_pages, const int* __restrict__ seq_slot,
                             const int* __restrict__ seq_qstart, const int* __restrict__ seq_pos0,
                             const float* __restrict__ r1, const float* __restrict__ r2, int heads,
                             int kv_heads, int page, float scale, Sight sight, int out_f32,
                             Fuse fuse, int* __restrict__ status) {
    using T = __nv_bfloat16;
    constexpr int LD = D + 8, DT = D / 8, CH = D / 8;
    extern __shared__ __align__(16) float smem[];
    float* Qs = smem;                                // [DRW][D]
    float* Pml = Qs + DRW * D;                       // [WARPS][DRW][2]
    T* tiles = reinterpret_cast<T*>(Pml + WARPS * DRW * 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gid = lane >> 2, tig = lane & 3;
    T* mine = tiles + (size_t)warp * DSTAGES * 2 * DKT * LD;   // [stage][K, V][DKT][LD]
    const int seq = blockIdx.x, hk = blockIdx.y, g = heads / kv_heads, h0 = hk * g;
    const int pos = seq_pos0[seq], slot = seq_slot[seq], tok = seq_qstart[seq];
    const int lo = sight_lo(sight, pos), hi = pos + 1, first = sight_first(sight, lo);
    // the tiles: those of the kept first keys, then from the tile of `lo` on, dealt out in turn
    const TileWalk walk(lo, first, DKT);
    const int first_tiles = walk.jump_at > 0 ? walk.jump_at / DKT : 0;
    const int near0 = walk.jump_at > 0 ? walk.jump_to : walk.start;
    const int n_tiles = first_tiles + (hi - near0 + DKT - 1) / DKT;
    auto start_of = [&](int ti) {
        return ti < first_tiles ? ti * DKT : near0 + (ti - first_tiles) * DKT;
    };
    // lane j < 16 finds key j of a tile: its row in the pages, -1 for a key that is not seen
    auto row_of = [&](int ti) {
        long long row = -1;
        if (ti < n_tiles && lane < DKT) {
            const int kpos = start_of(ti) + lane;
            if ((kpos >= lo || kpos < first) && kpos < hi) {
                const int id = block_table[(size_t)slot * table_stride + kpos / page];
                if (id >= 0 && id < num_pages)
                    row = ((long long)id * kv_heads + hk) * page + kpos % page;
                else if (status != nullptr) atomicExch(status, 2);
            }
        }
        return row;
    };
    const bool penalty = r1 != nullptr;
    const int hq = h0 + min(gid, g - 1);
    const float pen1 = penalty ? r1[hq] : 0.0f, pen2 = penalty ? r2[hq] : 0.0f;
    long long next_row = row_of(warp);

    pdl_wait();
    decode_begin<T>(Qs, DRW, g, h0, hk, q, q_stride, tok, slot, pos, k_pages, v_pages, block_table,
                    table_stride, num_pages, heads, kv_heads, D, D, page, fuse, status);
    unsigned qf[D / 16][4];                          // (rounded already: what q went through)
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
        const float* p = Qs + gid * D + kk * 16 + 2 * tig;
        qf[kk][0] = pack2(p[0], p[1]);
        qf[kk][2] = pack2(p[8], p[9]);
        qf[kk][1] = qf[kk][3] = 0u;                  // rows 8 to 15
    }
    // which of a tile's keys are seen, of the tile worked on and the two behind it
    unsigned seen[DSTAGES];
    auto issue = [&](int ti, int stage) {
        T* kd = mine + (size_t)stage * 2 * DKT * LD;
        T* vd = kd + DKT * LD;
        const long long row = next_row;
        next_row = row_of(ti + WARPS);
#pragma unroll
        for (int i = 0; i < DKT * CH / 32; ++i) {
            const int c = lane + 32 * i, j = c / CH, ch = c % CH;
            const long long r = __shfl_sync(0xffffffffu, row, j);
            const size_t at = r >= 0 ? (size_t)r : 0;
            const int bytes = r >= 0 ? 16 : 0;
            const unsigned ka = (unsigned)__cvta_generic_to_shared(kd + j * LD + ch * 8);
            const unsigned va = (unsigned)__cvta_generic_to_shared(vd + j * LD + ch * 8);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(ka),
                         "l"(k_pages + at * D + ch * 8), "r"(bytes) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(va),
                         "l"(v_pages + at * sight.v_stride + ch * 8), "r"(bytes) : "memory");
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        return __ballot_sync(0xffffffffu, row >= 0);
    };
#pragma unroll
    for (int i = 0; i < DSTAGES - 1; ++i) seen[i] = issue(warp + i * WARPS, i);

    float m = -INFINITY, l = 0.0f, acc[DT][2];
#pragma unroll
    for (int j = 0; j < DT; ++j) acc[j][0] = acc[j][1] = 0.0f;
    const int mat = lane >> 3, mr = lane & 7;
    int stage = 0;
    for (int ti = warp; ti < n_tiles; ti += WARPS) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(DSTAGES - 2) : "memory");
        __syncwarp();                // this tile has landed, the one before it has been used
        const int free = stage == 0 ? DSTAGES - 1 : stage - 1;
        const unsigned mask = seen[0];
        seen[0] = seen[1];
        seen[1] = issue(ti + (DSTAGES - 1) * WARPS, free);
        const T* kb = mine + (size_t)stage * 2 * DKT * LD;
        const T* vb = kb + DKT * LD;
        stage = stage == DSTAGES - 1 ? 0 : stage + 1;
        float c[2][2][4];            // q . k in two chains of half the features each
#pragma unroll
        for (int i = 0; i < 16; ++i) c[i >> 3][(i >> 2) & 1][i & 3] = 0.0f;
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
            unsigned b[4];
            ldmatrix4(b, kb + ((mat >> 1) * 8 + mr) * LD + kk * 16 + (mat & 1) * 8);
            mma16816(c[kk & 1][0], qf[kk], b[0], b[1]);
            mma16816(c[kk & 1][1], qf[kk], b[2], b[3]);
        }
        const int kt = start_of(ti);
        float s[2][2];
        float top = m;
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const int key = 8 * j + 2 * tig + x;
                const float sc = sight_score(sight, c[0][j][x] + c[1][j][x], scale, pen1, pen2,
                                             penalty, (float)(pos - kt - key));
                s[j][x] = (mask >> key) & 1u ? sc : -INFINITY;
                top = fmaxf(top, s[j][x]);
            }
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
        const float use = top == -INFINITY ? 0.0f : top;
        const float corr = expf(m - use);
        m = top;
        float sum = 0.0f;
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                s[j][x] = expf(s[j][x] - use);
                sum += s[j][x];
            }
        l = l * corr + sum;
        unsigned pw[3][4];
#pragma unroll
        for (int j = 0; j < 2; ++j) split3(s[j][0], s[j][1], pw[0][2 * j], pw[1][2 * j], pw[2][2 * j]);
#pragma unroll
        for (int t = 0; t < 3; ++t) pw[t][1] = pw[t][3] = 0u;
#pragma unroll
        for (int jd = 0; jd < DT; jd += 2) {
            unsigned b[4];
            ldmatrix4_trans(b, vb + ((mat & 1) * 8 + mr) * LD + (jd + (mat >> 1)) * 8);
            float t0[4] = {0.0f, 0.0f, 0.0f, 0.0f}, t1[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int term = 2; term >= 0; --term) {
                mma16816(t0, pw[term], b[0], b[1]);
                mma16816(t1, pw[term], b[2], b[3]);
            }
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                acc[jd][x] = fmaf(acc[jd][x], corr, t0[x]);
                acc[jd + 1][x] = fmaf(acc[jd + 1][x], corr, t1[x]);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    pdl_trigger();
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    __syncthreads();                                 // the tiles' place now holds the partial results
    float* Pacc = reinterpret_cast<float*>(tiles);   // [WARPS][DRW][D]
    if (tig == 0) {
        Pml[(warp * DRW + gid) * 2] = m;
        Pml[(warp * DRW + gid) * 2 + 1] = l;
    }
    float zero = 0.0f;
#pragma unroll
    for (int j = 0; j < DT; ++j) {
        store_pair(Pacc + (size_t)(warp * DRW + gid) * D + j * 8 + 2 * tig, acc[j][0], acc[j][1]);
        zero = fmaf(acc[j][1], 0.0f, fmaf(acc[j][0], 0.0f, zero));
    }
    // heads that met an infinity or NaN: their result in the first warp's place
    if (__syncthreads_or(gid < g && !(zero == 0.0f))) {
        for (int i = warp; i < g; i += WARPS) {
            bool spoilt = false;
            for (int w = 0; w < WARPS; ++w)
                for (int c = lane; c < D; c += 32)
                    spoilt |= !(Pacc[(size_t)(w * DRW + i) * D + c] * 0.0f == 0.0f);
            if (!__any_sync(0xffffffffu, spoilt)) continue;
            float mr, lr, res[D / 32];
            row_again<D>(Qs + i * D, (const T*)k_pages, (const T*)v_pages,
                         block_table + (size_t)slot * table_stride, num_pages, hk, kv_heads, page,
                         pos, 0, hi, scale, penalty ? r1[h0 + i] : 0.0f,
                         penalty ? r2[h0 + i] : 0.0f, penalty, sight, mr, lr, res);
#pragma unroll
            for (int c = 0; c < D / 32; ++c) Pacc[(size_t)i * D + lane + 32 * c] = res[c];
            if (lane < WARPS) {
                Pml[(lane * DRW + i) * 2] = lane == 0 ? mr : -INFINITY;
                Pml[(lane * DRW + i) * 2 + 1] = lr;
            }
        }
        __syncthreads();
    }
    decode_finish<T>(Pml, Pacc, DRW, WARPS, g, h0, tok, pos, out, out_stride, D, sight, out_f32,
                     fuse);
}

}  // namespace

// rows of a tile: 8, or 32 when the step brings prompt portions (`wide`) and the sizes allow the
// kernel that gives a warp four rows
static bool vec_ok(int dtype, int dk, int dv) {
    const int pn = dtype == DE_BF16 ? 8 : 4;
    return dk % pn == 0 && dv % pn == 0 && dk <= MAX_DK && dv <= MAX_D;
}
// the kernel that gives a warp one or four rows holds a tile's 16-byte pieces in at most 16
// registers a thread
static bool vec_fits(int dtype, int dk, int dv) {
    const int pn = dtype == DE_BF16 ? 8 : 4;
    return vec_ok(dtype, dk, dv) && TILE * (dk / pn + dv / pn) <= 16 * ROWS * 32;
}
static size_t tiled_smem(int dk, int dv) {
    return (size_t)(TILE * (dk + 4) + TILE * dv + TROWS * (dk + 4) + 4 * TILE * 16 + TILE) *
           sizeof(float);
}
static int sm_count() {
    static int count = 0;
    if (count == 0) {
        int device = 0;
        if (cudaGetDevice(&device) != cudaSuccess ||
            cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
            count = 148;
    }
    return count;
}
// the tensor-core kernel's sizes: bfloat16, keys and values of 64 or of 128 features
static bool mma_ok(int dtype, int dk, int dv) {
    return dtype == DE_BF16 && dk == dv && (dk == 64 || dk == 128);
}
// `wide`: 0 for steps of single tokens, else the rows (tokens times query heads a kv head) of the
// step's longest portion (1: some portion): from 48 rows on 64 (the register-tiled kernel's,
// or the tensor-core kernel's first form), else 32; callers give a portion's rows only where tiles of
// 64 give every SM two blocks (tensor cores, 16 heads on 4 kv heads of 128: 1,024 tokens of 8 heads
// on 2, 128 blocks of 64 rows or 256 of 32, 100 against 79 us; 2,048 tokens of 16 heads, 512 or
// 1,024 blocks, 199 against 231).
DE_EXPORT int de_attn_chunk_rows(int dtype, int dk, int dv, int wide) {
    if (!(vec_ok(dtype, dk, dv) && wide)) return ROWS;
    if (mma_ok(dtype, dk, dv)) return wide >= 48 ? TROWS : TROWS / 2;
    if (wide >= 48 && tiled_smem(dk, dv) <= 200 * 1024) return TROWS;
    return vec_fits(dtype, dk, dv) ? ROWS * 4 : ROWS;
}

static size_t decode_smem(int dtype, int rw, int dk, int dv, int v_in_k) {
    const int size = dtype == DE_BF16 ? 2 : 4;
    const size_t tile = (size_t)TILE * (((dk * size + 127) / 128) * 128 + 16) +
                        (v_in_k ? 0 : (size_t)TILE * dv * size);
    return (size_t)(rw * dk + ROWS * rw * 2 + ROWS * rw * dv) * sizeof(float) + ROWS * tile;
}

// The query heads a block of the single-token kernel takes (0: the kernel does not take this
// shape).  Keys and values of their own: up to 8 query heads a kv head, all in one block, if the
// eight warps' tiles then fit an SM.  Values inside the keys (`v_in_k`): any number of heads;
// several blocks share a kv head, each with as many heads (up to 8) as fit.
static int decode_rows(int dtype, int heads, int kv_heads, int dk, int dv, int v_in_k) {
    if (!(vec_ok(dtype, dk, dv) && kv_heads > 0 && heads % kv_heads == 0)) return 0;
    const int g = heads / kv_heads;
    int rw = g <= 1 ? 1 : (g <= 2 ? 2 : (g <= 4 ? 4 : 8));
    if (!v_in_k) return g <= 8 && decode_smem(dtype, rw, dk, dv, 0) <= 200 * 1024 ? rw : 0;
    if (decode_smem(dtype, rw, dk, dv, v_in_k) <= 200 * 1024) return rw;
    while ((rw >>= 1) >= 1)
        if (decode_smem(dtype, rw, dk, dv, v_in_k) <= 216 * 1024) return rw;
    return 0;
}

// Whether steps of single tokens go to the kernel that takes a (sequence, kv head) a block, or a
// few blocks where a kv head has many query heads: rows of whole 16-byte pieces, and its eight
// tiles fit an SM.  v_in_k: the values are the first dv features of the keys.
DE_EXPORT int de_attn_chunk_decode_ok(int dtype, int heads, int kv_heads, int dk, int dv,
                                      int v_in_k) {
    return decode_rows(dtype, heads, kv_heads, dk, dv, v_in_k) > 0;
}

DE_EXPORT int de_attn_chunk_decode(int dtype, const void* q, int q_stride, void* out,
                                   int out_stride, void* k_pages, void* v_pages,
                                   const int* block_table, int table_stride, int num_pages,
                                   const int* seq_slot, const int* seq_qstart,
                                   const int* seq_pos0, int n_seqs, const float* r1,
                                   const float* r2, int heads, int kv_heads, int dk, int dv,
                                   int page, float scale, int chunk, int window, int keep_first,
                                   float softcap, int out_f32, int fused, const float* fk, int rot,
                                   const float* fv, int write_kv, const void* gate, int ld_gate,
                                   int v_stride, int linear, const float* sink,
                                   const void* out_gate, int ld_out_gate, int gate_per_head,
                                   float out_scale, int* status, void* stream) {
    if (n_seqs <= 0) return 0;
    // v_stride 0: values in rows of their own; else rows of v_pages are that many elements apart
    const int pn_v = dtype == DE_BF16 ? 8 : 4;
    if (v_stride != 0 && (v_stride < dv || v_stride % pn_v != 0 || fused)) return -2;
    const Sight sight = {chunk, window, keep_first, softcap, v_stride ? v_stride : dv, linear, sink,
                         out_gate, ld_out_gate, gate_per_head, out_scale};
    if (out_gate != nullptr && fused) return -2;     // a fused step has its own gate
    const Fuse fuse = {fused, fk, rot, fv, write_kv, gate, ld_gate};
    if (fused && (rot < 0 || rot % 2 || rot > dk || (fv != nullptr && dv % 2) || out_f32)) return -2;
    const int v_in_k = v_pages == k_pages && v_stride == dk;
    const int rw = decode_rows(dtype, heads, kv_heads, dk, dv, v_in_k);
    if (rw == 0 || (uintptr_t)k_pages % 16 != 0) return -2;
    cudaStream_t s = (cudaStream_t)stream;
    const int g = heads / kv_heads;
    const size_t smem = decode_smem(dtype, rw, dk, dv, v_in_k);
    if ((uintptr_t)v_pages % 16 != 0) return -2;
    if (g > rw && fused) return -2;         // a kv head's blocks would each store the token's key
    if (mma_ok(dtype, dk, dv) && g <= DRW && sight.v_stride % 8 == 0) {
        // four warps a block, two blocks an SM; eight where there is at most one block an SM (us with
        // four and eight, 700 keys, 4 kv heads of 128: 8 sequences 19.4 and 15.1, 37 sequences = 148
        // blocks 23.5 and 19.1, 48 sequences 25.8 and 31.6, 128 sequences 50 and 61)
        const bool few = (long long)n_seqs * kv_heads <= sm_count();
#define DECM(D, W)                                                                              \
    do {                                                                                        \
        auto kernel = attn_chunk_decode_mma_kernel<D, W>;                                       \
        const size_t bytes = decode_mma_smem<D, W>();                                           \
        const cudaError_t me = cudaFuncSetAttribute(                                            \
            kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);                   \
        if (me != cudaSuccess) return (int)me;                                                  \
        return de_launch(kernel, dim3(n_seqs, kv_heads), dim3(W * 32), bytes, s,                \
                         (const __nv_bfloat16*)q, q_stride, out, out_stride,                    \
                         (__nv_bfloat16*)k_pages, (__nv_bfloat16*)v_pages, block_table,         \
                         table_stride, num_pages, seq_slot, seq_qstart, seq_pos0, r1, r2,       \
                         heads, kv_heads, page, scale, sight, out_f32, fuse, status);           \
    } while (0)
        if (dk == 64) {
            if (few) DECM(64, 8);
            DECM(64, 4);
        }
        if (few) DECM(128, 8);
        DECM(128, 4);
#undef DECM
    }
    dim3 grid(n_seqs, kv_heads * ((g + rw - 1) / rw));
#define DEC(T, RW)                                                                              \
    do {                                                                                        \
        if (smem > 48 * 1024) {                                                                 \
            cudaError_t e = cudaFuncSetAttribute(attn_chunk_decode_kernel<T, RW>,               \
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize,   \
                                                 (int)smem);                                    \
            if (e != cudaSuccess) return (int)e;                                                \
        }                                                                                       \
        return de_launch(attn_chunk_decode_kernel<T, RW>, grid, dim3(ROWS * 32), smem, s,       \
                         (const T*)q, q_stride, out, out_stride, (T*)k_pages, (T*)v_pages,      \
                         block_table, table_stride, num_pages, seq_slot, seq_qstart, seq_pos0,  \
                         r1, r2, heads, kv_heads, dk, dv, page, scale, sight, out_f32, fuse,    \
                         status);                                                               \
    } while (0)
#define DEC_T(T)                                                                                \
    do {                                                                                        \
        if (rw == 1) DEC(T, 1);                                                                 \
        if (rw == 2) DEC(T, 2);                                                                 \
        if (rw == 4) DEC(T, 4);                                                                 \
        DEC(T, 8);                                                                              \
    } while (0)
    if (dtype == DE_BF16) DEC_T(__nv_bfloat16);
    DEC_T(float);
#undef DEC_T
#undef DEC
}

DE_EXPORT int de_kv_write_normed(int dtype, const void* proj, int ld, int k_col,
                                 const int* positions, const int* token_slot, int G, int dk,
                                 int dv, float eps, void* k_pages, void* v_pages,
                                 const int* block_table, int table_stride, int page, int num_pages,
                                 int n, int* status, void* stream) {
    if (n <= 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    const int threads = 64;
    if (dtype == DE_BF16)
        return de_launch(kv_write_normed_kernel<__nv_bfloat16>, dim3(n, G), dim3(threads), 0, s,
                         (const __nv_bfloat16*)proj, ld, k_col, positions, token_slot, G, dk, dv,
                         eps, (__nv_bfloat16*)k_pages, (__nv_bfloat16*)v_pages, block_table,
                         table_stride, page, num_pages, status);
    return de_launch(kv_write_normed_kernel<float>, dim3(n, G), dim3(threads), 0, s,
                     (const float*)proj, ld, k_col, positions, token_slot, G, dk, dv, eps,
                     (float*)k_pages, (float*)v_pages, block_table, table_stride, page, num_pages,
                     status);
}

DE_EXPORT int de_kv_write_rotated(int dtype, void* proj, int ld, const int* positions,
                                  const int* token_slot, const float* fk, int rot, const float* fv,
                                  int H, int G, int dk, int dv, void* k_pages, void* v_pages,
                                  const int* block_table, int table_stride, int page,
                                  int num_pages, int write_kv, int n, int* status, void* stream) {
    if (n <= 0) return 0;
    if (rot < 0 || rot % 2 || rot > dk || (fv != nullptr && dv % 2)) return -2;
    cudaStream_t s = (cudaStream_t)stream;
    const int work = (H + G) * dk + G * dv;
    const int threads = n >= 512 ? 128 : (work >= 2048 ? 512 : 256);
    // A group's features: eight of bfloat16 where everything is whole groups of them, else four.  As many
    // threads as groups, but at least four warps (8 + 2 heads of 64, 1,000 tokens 2.4 us; 3.1 by the two
    // that have groups, 2.55 by four in groups of four); in float32, while the tokens are one round of
    // six blocks of 256 an SM, more (12 + 2 heads of 64, 512 tokens 2.3 and 2.6, 999 tokens 3.5 and 3.1).
    auto groups = [&](int e, size_t bytes) {
        return rot % (2 * e) == 0 && (dk - rot) % e == 0 && dv % (fv != nullptr ? 2 * e : e) == 0 &&
               ld % e == 0 && dk <= MAX_D && dv <= MAX_D && (uintptr_t)proj % bytes == 0 &&
               (uintptr_t)k_pages % bytes == 0 && (uintptr_t)v_pages % bytes == 0;
    };
#define ROT(T, E)                                                                               \
    do {                                                                                        \
        const int items = (H + G) * ((dk - rot / 2) / E) + G * ((fv != nullptr ? dv / 2 : dv) / E); \
        const int fits = items >= 256 ? 256 : items <= 128 ? 128 : (items + 31) / 32 * 32;      \
        const int block = sizeof(T) == 4 && n <= 6 * sm_count() && work >= 1024 ? 256 : fits;   \
        return de_launch(kv_write_rotated_vec_kernel<T, E>, dim3(n), dim3(block), 0, s,         \
                         (T*)proj, ld, positions, token_slot, fk, rot, fv, H, G, dk, dv,        \
                         (T*)k_pages, (T*)v_pages, block_table, table_stride, page, num_pages,  \
                         write_kv, status);                                                     \
    } while (0)
    if (dtype == DE_BF16 && groups(8, 16)) ROT(__nv_bfloat16, 8);
    if (dtype == DE_BF16 && groups(4, 8)) ROT(__nv_bfloat16, 4);
    if (dtype != DE_BF16 && groups(4, 16)) ROT(float, 4);
#undef ROT
    if (dtype == DE_BF16)
        return de_launch(kv_write_rotated_kernel<__nv_bfloat16>, dim3(n), dim3(threads), 0, s,
                         (__nv_bfloat16*)proj, ld, positions, token_slot, fk, rot, fv, H, G, dk, dv,
                         (__nv_bfloat16*)k_pages, (__nv_bfloat16*)v_pages, block_table,
                         table_stride, page, num_pages, write_kv, status);
    return de_launch(kv_write_rotated_kernel<float>, dim3(n), dim3(threads), 0, s, (float*)proj, ld,
                     positions, token_slot, fk, rot, fv, H, G, dk, dv, (float*)k_pages,
                     (float*)v_pages, block_table, table_stride, page, num_pages, write_kv, status);
}

// Whether a step of n tokens goes in runs, where its sizes are whole groups: `heads` of q, k and v
// together.  Us, a token a block and in runs, a norm a head, what proj holds in the L2 as after its product:
// always from 128 tokens on for heads of 64 (48 heads, 650 tokens, 11.5 and 7.3), with taps (24 heads of
// 128, 128 tokens 6.2 and 4.9, 600 16.5 and 10.2) and in float32 (24 heads, 700 tokens 7.8 and 7.4).
// bfloat16 heads of 128 without taps: not while the runs' blocks leave SMs without one or hardly one each
// (20 heads, 128 tokens 3.2 and 4.0; 12 heads, 300 4.2 and 4.3, 400 5.0 and 4.4), nor where up to 24 heads'
// runs are two rounds of blocks, three an SM, and the tokens one, five an SM (20 heads, 592 tokens 6.4
// and 5.2, 600 6.5 and 7.2, 700 6.5 and 7.5, 750 9.1 and 7.7; with 48 heads 600 12.4 and 11.5).
static bool prepare_in_runs(int dtype, int n, int heads, int dk, bool taps, int sms) {
    if (n < 128) return false;
    if (dk == 64 || taps || dtype == DE_F32) return true;
    const int across = (heads + 7) / 8, blocks = (n + RUN - 1) / RUN * across;
    // (blocks of 512 threads, two an SM, for fewer than 512 tokens of 16 heads and more)
    if (n > (heads >= 16 && n < 512 ? 2 : 5) * sms) return true;
    return 4 * blocks >= 5 * sms && !(across <= 3 && blocks > 3 * sms);
}
DE_EXPORT int de_qkv_prepare_in_runs(int dtype, int n, int heads, int dk, int taps, int sms) {
    return prepare_in_runs(dtype, n, heads, dk, taps != 0, sms);
}

DE_EXPORT int de_qkv_prepare(int dtype, const void* proj, int ld, void* q_out,
                             const int* positions, const int* token_seq, const int* token_slot,
                             const int* seq_pos0, const float* bias, const float* taps, int by_tap, int K,
                             float* state, long long slot_stride, int conv_offset, int norm,
                             const float* q_weight, const float* k_weight, float eps,
                             const float* freq, int rot, float magnitude, int adjacent,
                             float temp_coef, int temp_every, int mix, const float* lambda,
                             float* v_first, int keep_here, int v_from_k, int H, int G, int dk,
                             int dv, void* k_pages, void* v_pages, const int* block_table,
                             int table_stride, int page, int num_pages, int n, int* status,
                             void* stream) {
    if (n <= 0) return 0;
    if (rot < 0 || rot % 2 || rot > dk || (rot > 0 && freq == nullptr) || norm < 0 || norm > 2 ||
        (norm == 2 && (q_weight == nullptr || k_weight == nullptr)) ||
        (q_weight == nullptr) != (k_weight == nullptr) || (v_from_k && dv != dk) || mix < 0 || mix > 2 ||
        (mix != 0 && v_first == nullptr) || (mix == 2 && lambda == nullptr) ||
        (taps != nullptr && (K < 1 || (K > 1 && state == nullptr))))
        return -2;
    if (by_tap && ((uintptr_t)taps % 16 || (uintptr_t)bias % 16)) return -2;
    const Prepare pp = {bias, taps, by_tap, K, state, slot_stride, conv_offset, norm, q_weight, k_weight,
                        eps, freq, rot, magnitude, adjacent, temp_coef, temp_every, mix, lambda,
                        v_first, keep_here, v_from_k};
    cudaStream_t s = (cudaStream_t)stream;
    const int C = (H + G) * dk + (v_from_k ? 0 : G * dv);
    const size_t four = dtype == DE_BF16 ? 8 : 16;   // bytes of a group of four
    if (dk == dv && (dk == 64 || dk == 128) && norm != 2 && mix == 0 && !keep_here &&
        (taps == nullptr || (K >= 2 && K <= 4)) && rot % (adjacent ? 4 : 8) == 0 && ld % 4 == 0 &&
        (uintptr_t)proj % four == 0 && (uintptr_t)q_out % four == 0 &&
        (uintptr_t)k_pages % four == 0 && (uintptr_t)v_pages % four == 0 &&
        prepare_in_runs(dtype, n, C / dk, dk, taps != nullptr, sm_count())) {
        const int heads = C / dk, per_block = dk == 64 ? 16 : 8;
        const dim3 grid((n + RUN - 1) / RUN, (heads + per_block - 1) / per_block);
#define PREP_RUNS(T, D, KK)                                                                     \
    return de_launch(qkv_prepare_runs_kernel<T, D, KK>, grid, dim3(256), 0, s, (const T*)proj,  \
                     ld, (T*)q_out, positions, token_seq, token_slot, seq_pos0, pp, H, G,       \
                     (T*)k_pages, (T*)v_pages, block_table, table_stride, page, num_pages, n,   \
                     status)
#define PREP_RUNS_K(T, D)                                                                       \
    do {                                                                                        \
        if (taps == nullptr) PREP_RUNS(T, D, 1);                                                \
        if (K == 2) PREP_RUNS(T, D, 2);                                                         \
        if (K == 3) PREP_RUNS(T, D, 3);                                                         \
        PREP_RUNS(T, D, 4);                                                                     \
    } while (0)
        if (dtype == DE_BF16) {
            if (dk == 64) PREP_RUNS_K(__nv_bfloat16, 64);
            PREP_RUNS_K(__nv_bfloat16, 128);
        }
        if (dk == 64) PREP_RUNS_K(float, 64);
        PREP_RUNS_K(float, 128);
#undef PREP_RUNS_K
#undef PREP_RUNS
    }
    const size_t smem = (size_t)(C + rot + H + G) * sizeof(float);
    if (smem > 200 * 1024) return -2;
    const int threads = C >= 2048 && n < 512 ? 512 : 256;
    const int pn = dtype == DE_BF16 ? 8 : 4;
    const bool vec = C % pn == 0 && ld % pn == 0 && (uintptr_t)proj % 16 == 0;
    const bool conv = taps != nullptr && K > 1;
#define PREP_C(T, V, CONV)                                                                      \
    do {                                                                                        \
        if (smem > 48 * 1024) {                                                                 \
            cudaError_t e = cudaFuncSetAttribute(qkv_prepare_kernel<T, V, CONV>,                \
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize,   \
                                                 (int)smem);                                    \
            if (e != cudaSuccess) return (int)e;                                                \
        }                                                                                       \
        return de_launch(qkv_prepare_kernel<T, V, CONV>, dim3(n), dim3(threads), smem, s,       \
                         (const T*)proj, ld, (T*)q_out, positions, token_seq, token_slot,       \
                         seq_pos0, pp, H, G, dk, dv, (T*)k_pages, (T*)v_pages, block_table,     \
                         table_stride, page, num_pages, status);                                \
    } while (0)
#define PREP(T, V)                                                                              \
    do {                                                                                        \
        if (conv) PREP_C(T, V, true);                                                           \
        PREP_C(T, V, false);                                                                    \
    } while (0)
    if (dtype == DE_BF16) {
        if (vec) PREP(__nv_bfloat16, true);
        PREP(__nv_bfloat16, false);
    }
    if (vec) PREP(float, true);
    PREP(float, false);
#undef PREP
#undef PREP_C
}

DE_EXPORT int de_conv_keep(int dtype, const void* proj, int ld, float* state, long long slot_stride,
                           int conv_offset, const int* seq_slot, const int* seq_qstart,
                           const int* seq_qlen, int n_seqs, int C, int K, void* stream) {
    if (n_seqs <= 0 || K <= 1) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    const dim3 grid(n_seqs, (C + 255) / 256);
    if (dtype == DE_BF16)
        return de_launch(conv_keep_kernel<__nv_bfloat16>, grid, dim3(256), 0, s,
                         (const __nv_bfloat16*)proj, ld, state, slot_stride, conv_offset, seq_slot,
                         seq_qstart, seq_qlen, C, K);
    return de_launch(conv_keep_kernel<float>, grid, dim3(256), 0, s, (const float*)proj,
                     ld, state, slot_stride, conv_offset, seq_slot, seq_qstart, seq_qlen, C, K);
}

DE_EXPORT int de_attn_finish(int dtype, const float* o, const int* positions, const float* fv,
                             const void* gate, int ld_gate, void* out, int n, int H, int dv,
                             int gate_per_head, void* stream) {
    if (n <= 0) return 0;
    if (fv != nullptr && dv % 2) return -2;
    cudaStream_t s = (cudaStream_t)stream;
    const int threads = n >= 512 ? 128 : (H * dv >= 2048 ? 512 : 256);
    const size_t four = dtype == DE_BF16 ? 8 : 16;   // bytes of a group of four
    // (rows of 640 and more: 16 heads of 40 and their turns 2.5 us by the general form, 1.9 so; of 4 heads
    // of 40 1.7 and 1.9, at 2,048 tokens 2.9 and 3.9: a block has more threads than groups)
    if (H * dv >= 640 && dv % (fv != nullptr ? 8 : 4) == 0 && dv <= MAX_D && (uintptr_t)o % 16 == 0 &&
        (uintptr_t)out % four == 0 &&
        (gate == nullptr || gate_per_head || (ld_gate % 4 == 0 && (uintptr_t)gate % four == 0))) {
#define FIN(T)                                                                                  \
    return de_launch(attn_finish_vec_kernel<T>, dim3(n), dim3(H * dv >= 1024 ? 256 : 128), 0, s, o, \
                     positions, fv, (const T*)gate, ld_gate, (T*)out, H, dv, gate_per_head)
        if (dtype == DE_BF16) FIN(__nv_bfloat16);
        FIN(float);
#undef FIN
    }
    if (dtype == DE_BF16)
        return de_launch(attn_finish_kernel<__nv_bfloat16>, dim3(n), dim3(threads), 0, s, o,
                         positions, fv, (const __nv_bfloat16*)gate, ld_gate, (__nv_bfloat16*)out, H,
                         dv, gate_per_head);
    return de_launch(attn_finish_kernel<float>, dim3(n), dim3(threads), 0, s, o, positions, fv,
                     (const float*)gate, ld_gate, (float*)out, H, dv, gate_per_head);
}

DE_EXPORT int de_attn_chunk(int dtype, const void* q, int q_stride, void* out, int out_stride,
                            const void* k_pages, const void* v_pages, const int* block_table,
                            int table_stride, int num_pages, const int* seq_slot,
                            const int* seq_qstart, const int* seq_qlen, const int* seq_pos0,
                            const int* items, int num_items, const float* r1, const float* r2,
                            int heads, int kv_heads, int dk, int dv, int page, float scale,
                            int chunk, int window, int keep_first, float softcap, int out_f32,
                            int tile_rows, int v_stride, int linear, const float* sink,
                            const void* out_gate, int ld_out_gate, int gate_per_head,
                            float out_scale, int* status, void* stream) {
    if (num_items <= 0) return 0;
    // v_stride 0: values in rows of their own; else rows of v_pages are that many elements apart
    if (v_stride != 0 && (v_stride < dv || (vec_ok(dtype, dk, dv) && v_stride % (dtype == DE_BF16 ? 8 : 4))))
        return -2;
    const Sight sight = {chunk, window, keep_first, softcap, v_stride ? v_stride : dv, linear, sink,
                         out_gate, ld_out_gate, gate_per_head, out_scale};
    if (dk <= 0 || dk > MAX_DK || dv <= 0 || dv > MAX_D || heads % kv_heads != 0) return -2;
    cudaStream_t s = (cudaStream_t)stream;
    if (tile_rows != ROWS && !((tile_rows == ROWS * 4 && vec_fits(dtype, dk, dv)) ||
                               (tile_rows == TROWS && vec_ok(dtype, dk, dv)) ||
                               (tile_rows == 2 * TROWS && mma_ok(dtype, dk, dv))))
        return -5;
    if ((tile_rows >= TROWS || tile_rows == TROWS / 2) && mma_ok(dtype, dk, dv) &&
        q_stride % 2 == 0 && (uintptr_t)q % 4 == 0 && (uintptr_t)k_pages % 16 == 0 &&
        (uintptr_t)v_pages % 16 == 0) {
        const int parts = tile_rows == 2 * TROWS ? 2 : 1;
        dim3 mgrid(num_items * parts, kv_heads);
#define MMA(D, HALVES)                                                                          \
    do {                                                                                        \
        auto kernel = attn_chunk_mma_kernel<D, HALVES>;                                         \
        const size_t bytes = mma_smem<D, HALVES>();                                             \
        const cudaError_t me = cudaFuncSetAttribute(                                            \
            kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);                   \
        if (me != cudaSuccess) return (int)me;                                                  \
        return de_launch(kernel, mgrid, dim3(128), bytes, s, (const __nv_bfloat16*)q, q_stride, \
                         out, out_stride, (const __nv_bfloat16*)k_pages,                        \
                         (const __nv_bfloat16*)v_pages, block_table, table_stride, num_pages,   \
                         seq_slot, seq_qstart, seq_qlen, seq_pos0, (const WorkItem*)items, r1,  \
                         r2, heads, kv_heads, page, scale, sight, out_f32, parts, status);      \
    } while (0)
        if (tile_rows >= TROWS) {
            if (dk == 64) MMA(64, 1);
            MMA(128, 1);
        }
        if (dk == 64) MMA(64, 2);
        MMA(128, 2);
#undef MMA
    }
    if (tile_rows == 2 * TROWS) return -5;
    if (tile_rows == TROWS) {
        if ((uintptr_t)k_pages % 16 != 0 || (uintptr_t)v_pages % 16 != 0) return -5;
        const size_t tsmem = tiled_smem(dk, dv);
        if (tsmem > 200 * 1024) return -5;
        const int nc = (dv + 31) / 32;
        dim3 tgrid(num_items, kv_heads);
#define TILED(T, NC)                                                                            \
    do {                                                                                        \
        if (tsmem > 48 * 1024) {                                                                \
            cudaError_t te = cudaFuncSetAttribute(attn_chunk_tiled_kernel<T, NC>,               \
                                                  cudaFuncAttributeMaxDynamicSharedMemorySize,  \
                                                  (int)tsmem);                                  \
            if (te != cudaSuccess) return (int)te;                                              \
        }                                                                                       \
        return de_launch(attn_chunk_tiled_kernel<T, NC>, tgrid, dim3(128), tsmem, s,            \
                         (const T*)q, q_stride, out, out_stride, (const T*)k_pages,             \
                         (const T*)v_pages, block_table, table_stride, num_pages, seq_slot,     \
                         seq_qstart, seq_qlen, seq_pos0, (const WorkItem*)items, r1, r2, heads, \
                         kv_heads, dk, dv, page, scale, sight, out_f32, status);                \
    } while (0)
#define TILED_N(T)                                                                              \
    do {                                                                                        \
        if (nc <= 1) TILED(T, 1);                                                               \
        if (nc <= 2) TILED(T, 2);                                                               \
        if (nc <= 4) TILED(T, 4);                                                               \
        TILED(T, 8);                                                                            \
    } while (0)
        if (dtype == DE_BF16) TILED_N(__nv_bfloat16);
        TILED_N(float);
#undef TILED_N
#undef TILED
    }
    if (vec_fits(dtype, dk, dv) && (uintptr_t)k_pages % 16 == 0 && (uintptr_t)v_pages % 16 == 0) {
        const int rw = tile_rows / ROWS;
        const int pn = dtype == DE_BF16 ? 8 : 4;
        const int pieces = TILE * (dk / pn + dv / pn);
        const int nch = (pieces + ROWS * 32 - 1) / (ROWS * 32);
        const size_t vsmem = (size_t)(TILE * (((dk + 31) / 32) * 32 + 4) + TILE * dv +
                                      ROWS * rw * dk + TILE) * sizeof(float);
        dim3 vgrid(num_items, kv_heads);
#define VEC(T, RW, NCH)                                                                         \
    do {                                                                                        \
        if (vsmem > 48 * 1024) {                                                                \
            cudaError_t ve = cudaFuncSetAttribute(attn_chunk_vec_kernel<T, RW, NCH>,            \
                                                  cudaFuncAttributeMaxDynamicSharedMemorySize,  \
                                                  (int)vsmem);                                  \
            if (ve != cudaSuccess) return (int)ve;                                              \
        }                                                                                       \
        return de_launch(attn_chunk_vec_kernel<T, RW, NCH>, vgrid, dim3(ROWS * 32), vsmem, s,   \
                         (const T*)q, q_stride, out, out_stride, (const T*)k_pages,             \
                         (const T*)v_pages, block_table, table_stride, num_pages, seq_slot,     \
                         seq_qstart, seq_qlen, seq_pos0, (const WorkItem*)items, r1, r2, heads, \
                         kv_heads, dk, dv, page, scale, sight, out_f32, status);                \
    } while (0)
#define VEC_N(T, RW)                                                                            \
    do {                                                                                        \
        if (nch <= 2) VEC(T, RW, 2);                                                            \
        if (nch <= 4) VEC(T, RW, 4);                                                            \
        if (nch <= 8) VEC(T, RW, 8);                                                            \
        VEC(T, RW, 16);                                                                         \
    } while (0)
        if (dtype == DE_BF16) {
            if (rw == 4) VEC_N(__nv_bfloat16, 4);
            VEC_N(__nv_bfloat16, 1);
        }
        if (rw == 4) VEC_N(float, 4);
        VEC_N(float, 1);
#undef VEC_N
#undef VEC
    }
    const size_t smem = (size_t)(TILE * (dk + 1) + TILE * dv + ROWS * dk) * sizeof(float);
    dim3 grid(num_items, kv_heads);
    cudaError_t e;
#define LAUNCH(T)                                                                               \
    do {                                                                                        \
        if (smem > 48 * 1024) {                                                                 \
            e = cudaFuncSetAttribute(attn_chunk_kernel<T>,                                      \
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);   \
            if (e != cudaSuccess) return (int)e;                                                \
        }                                                                                       \
        return de_launch(attn_chunk_kernel<T>, grid, dim3(ROWS * 32), smem, s, (const T*)q,     \
                         q_stride, out, out_stride, (const T*)k_pages, (const T*)v_pages,       \
                         block_table, table_stride, num_pages, seq_slot, seq_qstart, seq_qlen,  \
                         seq_pos0, (const WorkItem*)items, r1, r2, heads, kv_heads, dk, dv, page, \
                         scale, sight, out_f32, status);                                        \
    } while (0)
    if (dtype == DE_BF16) LAUNCH(__nv_bfloat16);
    LAUNCH(float);
#undef LAUNCH
}
