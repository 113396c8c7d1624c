// True 32-bit matrix product for the float32 path: out[n, m] = sum_k x[n, k] * w[m, k].
// IEEE float32 multiply-adds on the CUDA cores: no tensor cores, no TF32, no reduced-precision
// staging.  Every output element is formed in one way, whatever the number of rows and whichever of
// the kernels below runs, so a row's result does not depend on the batch it is in: k is cut into
// segments of 256, a segment's terms are one chain of fused multiply-adds in ascending order, and
// the segments' sums are added in ascending order.  (Segments let few rows spread over more warps,
// and a sum over k = 5,632 loses less than in one chain: 3.0e-7 of the result against 1.3e-6.)
//
// It stands where the reference calls F.linear in float32 with TF32 switched off
// (src/layers/linear.py:19-20, src/distengine/worker.py:427-428).

#include <atomic>

#include "common.cuh"

DE_DEFINE_PDL_SWITCH

namespace {

constexpr int SEG = 256;       // k of a segment

__device__ __forceinline__ void cp_async16_f32(void* smem, const void* gmem, bool pred) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    const int bytes = pred ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async4_f32(unsigned smem, const void* gmem, bool pred) {
    const int bytes = pred ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(smem), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// two IEEE multiply-adds in one instruction
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a,
                                     unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;\n" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long both(float a) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %1};\n" : "=l"(r) : "f"(a));
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

// ------------------------------------------------------------------------------------------
// Many rows: a block takes a tile of TILE rows of x by TILE rows of w; its GROUPS groups of threads
// form the whole tile each, over one segment of k in turn, a thread 8 x 8 outputs in two halves of
// four rows and columns.  A group brings steps of 16 k through two stages of its own of 4-byte
// cp.async that turn the operands ([k][row]), so that four neighbouring rows are one 16-byte read.
// The segments' sums are added to the block's sum in shared memory in ascending order: a group
// waits for the one whose segment comes before its own, adds, and goes on with its next segment.
// Bound by the multiply-add pipe and the reads of shared memory beside it.  Packed multiply-adds
// (fma.rn.f32x2) in a loop without loads run at 63 TFLOP/s on B200, single ones at 52; 1,000 rows
// against 11,264 x 2,048: 945 us = 48.8 TFLOP/s (tiles of 64 x 64 with 4 x 4 outputs a thread and
// single multiply-adds: 1,397 us; lanes that do not share reads: 1,115; steps of 8 k through four
// stages: 1,043).  Tiles of 64 with four groups: 1,037 us there, but 324 us at 300 rows against
// 382 (440 before) and 294 against 502 us (450) for 300 rows against 2,048 x 5,632.
// ------------------------------------------------------------------------------------------
constexpr int BK = 16, STAGES = 2;

template <int THREADS> __device__ __forceinline__ void group_sync(int g) {   // a group's threads
    asm volatile("bar.sync %0, %1;\n" ::"r"(1 + g), "n"(THREADS) : "memory");
}
// until the group before g has added; and: g may add now
template <int THREADS> __device__ __forceinline__ void link_wait(int g) {
    asm volatile("bar.sync %0, %1;\n" ::"r"(5 + g), "n"(2 * THREADS) : "memory");
}
template <int THREADS> __device__ __forceinline__ void link_pass(int g) {
    __threadfence_block();
    asm volatile("bar.arrive %0, %1;\n" ::"r"(5 + g), "n"(2 * THREADS) : "memory");
}

template <int TILE, int GROUPS>
struct Tiles {
    static constexpr int THREADS = TILE * TILE / 64;           // of a group
    static constexpr int LD = TILE + 4;                        // of a stage's rows of either operand
    static constexpr int STAGE = 2 * BK * LD;                  // floats
    static constexpr size_t SMEM = (size_t)(TILE * LD + GROUPS * STAGES * STAGE) * sizeof(float);
};

template <int TILE, int GROUPS>
__global__ void __launch_bounds__(Tiles<TILE, GROUPS>::THREADS * GROUPS,
                                  512 / (Tiles<TILE, GROUPS>::THREADS * GROUPS))
gemm_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ out,
                int n_rows, int m_cols, int k_dim, int ldx, int ldw, int ldo, int vec_out) {
    constexpr int THREADS = Tiles<TILE, GROUPS>::THREADS, LDT = Tiles<TILE, GROUPS>::LD;
    constexpr int STAGE = Tiles<TILE, GROUPS>::STAGE;
    constexpr int WN = TILE / 64;                  // warps of a group along the columns
    constexpr int RS = THREADS / 8, LOADS = TILE / RS;
    extern __shared__ __align__(16) float smem[];
    float* total = smem;                           // [TILE][LDT]
    const int tid = threadIdx.x % THREADS, group = threadIdx.x / THREADS;
    float* mine = smem + TILE * LDT + group * STAGES * STAGE;
    const int lane = tid & 31, warp = tid >> 5;
    const int row0 = blockIdx.y * TILE, col0 = blockIdx.x * TILE;
    // the thread's rows ty.., ty + 16.. and columns tx.., tx + 32..: lanes l and l ^ 1 read the same
    // rows, l and l ^ 2 the same columns, which is what lets a 16-byte read of a warp pass in two
    // wavefronts instead of four
    const int ty = warp / WN * 32 + (((lane >> 1) & 1) | ((lane >> 3) & 2)) * 4;
    const int tx = warp % WN * 64 + ((lane & 1) | ((lane >> 1) & 6)) * 4;
    // staging: thread t copies k = t % 8 of the rows t / 8, t / 8 + RS, ...
    const int l_k = tid & 7, l_row = tid >> 3;

    const int segments = (k_dim + SEG - 1) / SEG;
    // the next step of 16 k to bring, of this group's segments; past the last: zeros
    int n_k = group * SEG, n_slot = 0;
    const float* wp = w + (size_t)(col0 + l_row) * ldw + l_k;
    const float* xp = x + (size_t)(row0 + l_row) * ldx + l_k;
    const unsigned dst = (unsigned)__cvta_generic_to_shared(mine + l_k * LDT + l_row);
    const bool whole_w = col0 + TILE <= m_cols, whole_x = row0 + TILE <= n_rows;
    auto load = [&](const float* p, const float* base, int ld, int first, int limit, bool whole,
                    unsigned d) {
        if (whole && n_k + BK <= k_dim) {
#pragma unroll
            for (int i = 0; i < LOADS; ++i)
#pragma unroll
                for (int j = 0; j < BK; j += 8)
                    cp_async4_f32(d + 4 * (RS * i + j * LDT), p + (size_t)(RS * i) * ld + n_k + j,
                                  true);
        } else {
#pragma unroll
            for (int i = 0; i < LOADS; ++i)
#pragma unroll
                for (int j = 0; j < BK; j += 8) {
                    const bool ok = n_k + j + l_k < k_dim && first + RS * i < limit;
                    cp_async4_f32(d + 4 * (RS * i + j * LDT),
                                  ok ? p + (size_t)(RS * i) * ld + n_k + j : base, ok);
                }
        }
    };
    auto load_w = [&]() {
        load(wp, w, ldw, col0 + l_row, m_cols, whole_w, dst + 4 * (n_slot * STAGE + BK * LDT));
    };
    auto load_x = [&]() {
        load(xp, x, ldx, row0 + l_row, n_rows, whole_x, dst + 4 * (n_slot * STAGE));
    };
    auto advance = [&]() {
        n_slot = (n_slot + 1) % STAGES;
        n_k += BK;
        if (n_k % SEG == 0) n_k += (GROUPS - 1) * SEG;
    };

    pdl_wait();
#pragma unroll
    for (int t = 0; t < STAGES - 1; ++t) {
        load_w();
        load_x();
        advance();
        cp_async_commit();
    }

    int slot = 0;
    for (int seg = group; seg < segments; seg += GROUPS) {
        unsigned long long acc[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
        const int steps = min(SEG, k_dim - seg * SEG);
        for (int k0 = 0; k0 < steps; k0 += BK) {
            cp_async_wait<STAGES - 2>();
            group_sync<THREADS>(group);      // this step has landed; the stage refilled below is free
            load_w();
            load_x();
            advance();
            cp_async_commit();
            const float* ap = mine + slot * STAGE + ty;
            const float* bp = mine + slot * STAGE + BK * LDT + tx;
            slot = (slot + 1) % STAGES;
#pragma unroll
            for (int k = 0; k < BK; ++k) {
                const float4 a0 = *reinterpret_cast<const float4*>(ap + k * LDT);
                const float4 a1 = *reinterpret_cast<const float4*>(ap + k * LDT + 16);
                const float4 b0 = *reinterpret_cast<const float4*>(bp + k * LDT);
                const float4 b1 = *reinterpret_cast<const float4*>(bp + k * LDT + 32);
                const unsigned long long b[4] = {pair(b0.x, b0.y), pair(b0.z, b0.w),
                                                 pair(b1.x, b1.y), pair(b1.z, b1.w)};
                const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const unsigned long long aa = both(a[i]);
#pragma unroll
                    for (int j = 0; j < 4; ++j) fma2(acc[i][j], aa, b[j]);
                }
            }
        }
        // the block's sum takes the segments in ascending order; the last one writes the result
        if (seg > 0) link_wait<THREADS>(group);
        const bool last = seg == segments - 1;
        if (last) pdl_trigger();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = ty + (i & 3) + (i >> 2) * 16;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c = tx + 32 * h;
                float4 v;
                unpair(acc[i][2 * h], v.x, v.y);
                unpair(acc[i][2 * h + 1], v.z, v.w);
                float4* t = reinterpret_cast<float4*>(total + r * LDT + c);
                if (seg > 0) {
                    const float4 old = *t;
                    v.x += old.x; v.y += old.y; v.z += old.z; v.w += old.w;
                }
                if (!last) {
                    *t = v;
                    continue;
                }
                if (row0 + r >= n_rows) continue;
                float* o = out + (size_t)(row0 + r) * ldo + col0 + c;
                if (vec_out && col0 + c + 3 < m_cols) {
                    *reinterpret_cast<float4*>(o) = v;
                } else {
                    const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (col0 + c + q < m_cols) o[q] = e[q];
                }
            }
        }
        if (!last) link_pass<THREADS>((group + 1) % GROUPS);
    }
    cp_async_wait<0>();
}

// ------------------------------------------------------------------------------------------
// Few rows (decode steps): bound by streaming w.  A block takes COLS rows of w and up to T rows of
// x; its eight warps take one segment of k each (then the next eight), every warp alone: it brings
// steps of SM_K k through its own stages of 16-byte cp.async, and a lane forms two columns for its
// group's tokens, so that a read of shared memory serves several multiply-adds.  The segments'
// sums meet in shared memory and are added in ascending order.  Blocks walk the tiles of w with
// the grid's stride and the stages run on from one tile into the next.  Eight rows against
// 11,264 x 2,048: 25 us = 3.7 TB/s, against 2,048 x 5,632 15 us, against 32,000 x 2,048 54 us =
// 4.8 TB/s (one chain of k an output on 16 x 16 threads: 73, 45 and 196 us).  32 rows: 65, 38 and
// 154 us (140, 78 and 384), there the reads of shared memory are what it waits for.
// ------------------------------------------------------------------------------------------
constexpr int SM_WARPS = 8;

template <int T, int COLS, int SM_STAGES, int SM_K>
__global__ void __launch_bounds__(SM_WARPS * 32)
gemm_f32_small_kernel(const float* __restrict__ x, const float* __restrict__ w,
                      float* __restrict__ out, int n_rows, int m_cols, int k_dim, int ldx, int ldw,
                      int ldo, int col_tiles, int early) {
    constexpr int SM_LD = SM_K + 4;
    constexpr int PAIRS = COLS / 2;                          // lanes along the columns
    constexpr int TG = 32 / PAIRS;                           // groups of tokens
    constexpr int TL = T / TG;                               // tokens of a lane
    constexpr int OUTS = (T * COLS + SM_WARPS * 32 - 1) / (SM_WARPS * 32);   // a thread adds up
    constexpr int STAGE = (COLS + T) * SM_LD;                // floats
    extern __shared__ __align__(16) float smem[];
    float* part = smem;                                      // [2][WARPS][T][COLS]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float* mine = smem + 2 * SM_WARPS * T * COLS + warp * SM_STAGES * STAGE;
    // lanes l and l ^ 2 read the same columns, l and l ^ 1 the same tokens (see above)
    const int cp = PAIRS == 16 ? ((lane & 1) | ((lane >> 1) & 14))
                               : ((lane & 1) | ((lane >> 1) & 6));
    const int tg = PAIRS == 16 ? (lane >> 1) & 1 : (((lane >> 1) & 1) | ((lane >> 3) & 2));
    const int row0 = blockIdx.y * T;
    const int segments = (k_dim + SEG - 1) / SEG;
    const int rounds = (segments + SM_WARPS - 1) / SM_WARPS;
    constexpr int PER = SEG / SM_K;                          // stages of a segment
    const int my_tiles = (col_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;

    // the next stage to bring: a step of a segment (of this round), of a tile of w
    constexpr int PER_ROW = SM_K / 4, RS = 32 / PER_ROW;     // lanes a row, rows a copy
    const int l_row = lane / PER_ROW, l_k = (lane % PER_ROW) * 4;
    int n_step = 0, n_round = 0, n_tile = 0, n_slot = 0;
    auto stage_w = [&]() {
        const int gk = (n_round * SM_WARPS + warp) * SEG + n_step * SM_K + l_k;
        const int c0 = ((int)blockIdx.x + n_tile * (int)gridDim.x) * COLS + l_row;
        const bool in_k = n_tile < my_tiles && gk < k_dim;
        const float* p = w + (size_t)c0 * ldw + gk;
        float* d = mine + n_slot * STAGE + l_row * SM_LD + l_k;
#pragma unroll
        for (int i = 0; i < COLS; i += RS) {
            const bool ok = in_k && c0 + i < m_cols;
            cp_async16_f32(d + i * SM_LD, ok ? p + (size_t)i * ldw : w, ok);
        }
    };
    auto stage_x = [&]() {
        const int gk = (n_round * SM_WARPS + warp) * SEG + n_step * SM_K + l_k;
        const bool in_k = n_tile < my_tiles && gk < k_dim;
        const float* p = x + (size_t)(row0 + l_row) * ldx + gk;
        float* d = mine + n_slot * STAGE + (COLS + l_row) * SM_LD + l_k;
#pragma unroll
        for (int i = 0; i < T; i += RS) {
            const bool ok = in_k && row0 + i + l_row < n_rows;
            cp_async16_f32(d + i * SM_LD, ok ? p + (size_t)i * ldx : x, ok);
        }
    };
    auto advance = [&]() {
        n_slot = n_slot == SM_STAGES - 1 ? 0 : n_slot + 1;
        if (++n_step < PER) return;
        n_step = 0;
        if (++n_round < rounds) return;
        n_round = 0;
        ++n_tile;
    };
    auto first_w = [&]() {
#pragma unroll
        for (int t = 0; t < SM_STAGES - 1; ++t) {
            stage_w();
            advance();
        }
        n_step = n_round = n_tile = n_slot = 0;
    };
    if (early) first_w();
    pdl_wait();
    if (!early) first_w();
#pragma unroll
    for (int t = 0; t < SM_STAGES - 1; ++t) {
        stage_x();
        advance();
        cp_async_commit();
    }
    pdl_trigger();

    int slot = 0, flip = 0;
    for (int tile = 0; tile < my_tiles; ++tile) {
        float sum[OUTS];
#pragma unroll
        for (int o = 0; o < OUTS; ++o) sum[o] = 0.0f;
        for (int round = 0; round < rounds; ++round, flip ^= 1) {
            float acc[2][TL];
#pragma unroll
            for (int t = 0; t < TL; ++t) acc[0][t] = acc[1][t] = 0.0f;
            for (int step = 0; step < PER; ++step) {
                cp_async_wait<SM_STAGES - 2>();
                __syncwarp();                // every lane's copies have landed, the next stage is free
                stage_w();
                stage_x();
                advance();
                cp_async_commit();
                const float* wr = mine + slot * STAGE + cp * SM_LD;
                const float* xr = mine + slot * STAGE + (COLS + tg) * SM_LD;
                slot = slot == SM_STAGES - 1 ? 0 : slot + 1;
                if ((round * SM_WARPS + warp) * SEG + step * SM_K >= k_dim) continue;
#pragma unroll
                for (int k = 0; k < SM_K; k += 4) {
                    const float4 w0 = *reinterpret_cast<const float4*>(wr + k);
                    const float4 w1 = *reinterpret_cast<const float4*>(wr + PAIRS * SM_LD + k);
#pragma unroll
                    for (int t = 0; t < TL; ++t) {
                        const float4 a = *reinterpret_cast<const float4*>(xr + t * TG * SM_LD + k);
                        acc[0][t] = fmaf(a.x, w0.x, acc[0][t]);
                        acc[1][t] = fmaf(a.x, w1.x, acc[1][t]);
                        acc[0][t] = fmaf(a.y, w0.y, acc[0][t]);
                        acc[1][t] = fmaf(a.y, w1.y, acc[1][t]);
                        acc[0][t] = fmaf(a.z, w0.z, acc[0][t]);
                        acc[1][t] = fmaf(a.z, w1.z, acc[1][t]);
                        acc[0][t] = fmaf(a.w, w0.w, acc[0][t]);
                        acc[1][t] = fmaf(a.w, w1.w, acc[1][t]);
                    }
                }
            }
            // the round's segments in ascending order (the other half of `part` may still be read)
            float* p = part + flip * SM_WARPS * T * COLS;
            float* pw = p + warp * T * COLS + tg * COLS + cp;
#pragma unroll
            for (int t = 0; t < TL; ++t) {
                pw[t * TG * COLS] = acc[0][t];
                pw[t * TG * COLS + PAIRS] = acc[1][t];
            }
            __syncthreads();
            const int live = min(SM_WARPS, segments - round * SM_WARPS);
#pragma unroll
            for (int o = 0; o < OUTS; ++o) {
                const int idx = tid + o * SM_WARPS * 32;
                if (idx < T * COLS)
                    for (int g = 0; g < live; ++g) sum[o] += p[g * T * COLS + idx];
            }
        }
        const int c0 = ((int)blockIdx.x + tile * (int)gridDim.x) * COLS;
#pragma unroll
        for (int o = 0; o < OUTS; ++o) {
            const int idx = tid + o * SM_WARPS * 32;
            const int r = row0 + idx / COLS, c = c0 + idx % COLS;
            if (idx < T * COLS && r < n_rows && c < m_cols) out[(size_t)r * ldo + c] = sum[o];
        }
    }
    cp_async_wait<0>();
}

// ------------------------------------------------------------------------------------------
// Short sums (k of one or two segments), where the kernels above leave most of their warps without a
// segment: a thread forms its outputs over all of k, a segment at a time.  Bound by the trip to
// memory and, with many tiles, by the reads of shared memory (four and two multiply-adds a read).
// By tiles of 64 x 64: 4 x 4 outputs a thread on 16 x 16 threads, operands of any stride and address.
// 130 rows of 64 against 2,048 columns: 5.1 us (the few-row kernel 22).
// ------------------------------------------------------------------------------------------
constexpr int WT = 64, WK = 16;

template <bool VEC4>
__global__ void __launch_bounds__(256)
gemm_f32_wide_kernel(const float* __restrict__ x, const float* __restrict__ w,
                     float* __restrict__ out, int n_rows, int m_cols, int k_dim, int ldx, int ldw,
                     int ldo) {
    __shared__ float xs[WK][WT + 4];
    __shared__ float ws[WK][WT + 4];
    const int tid = threadIdx.x, ty = tid / 16, tx = tid % 16;
    const int row0 = blockIdx.y * WT, col0 = blockIdx.x * WT;
    const int l_row = tid / 4, l_k = (tid % 4) * 4;  // a thread stages 4 k of a row of each operand
    float acc[4][4], sum[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = sum[i][j] = 0.0f;

    pdl_wait();
    for (int k0 = 0; k0 < k_dim; k0 += WK) {
        float xv[4] = {0.f, 0.f, 0.f, 0.f}, wv[4] = {0.f, 0.f, 0.f, 0.f};
        const int gr = row0 + l_row, gc = col0 + l_row, gk = k0 + l_k;
        if (gr < n_rows) {
            const float* p = x + (size_t)gr * ldx + gk;
            if (VEC4 && gk + 3 < k_dim) {
                const float4 t = *reinterpret_cast<const float4*>(p);
                xv[0] = t.x; xv[1] = t.y; xv[2] = t.z; xv[3] = t.w;
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) if (gk + i < k_dim) xv[i] = p[i];
            }
        }
        if (gc < m_cols) {
            const float* p = w + (size_t)gc * ldw + gk;
            if (VEC4 && gk + 3 < k_dim) {
                const float4 t = *reinterpret_cast<const float4*>(p);
                wv[0] = t.x; wv[1] = t.y; wv[2] = t.z; wv[3] = t.w;
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) if (gk + i < k_dim) wv[i] = p[i];
            }
        }
        __syncthreads();                             // the step before this one has been used
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            xs[l_k + i][l_row] = xv[i];
            ws[l_k + i][l_row] = wv[i];
        }
        __syncthreads();
        if (k0 > 0 && k0 % SEG == 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    sum[i][j] += acc[i][j];
                    acc[i][j] = 0.0f;
                }
        }
#pragma unroll
        for (int k = 0; k < WK; ++k) {
            const float4 a = *reinterpret_cast<const float4*>(&xs[k][ty * 4]);
            const float4 b = *reinterpret_cast<const float4*>(&ws[k][tx * 4]);
            const float av[4] = {a.x, a.y, a.z, a.w};
            const float bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
    }
    pdl_trigger();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = row0 + ty * 4 + i;
        if (r >= n_rows) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int c = col0 + tx * 4 + j;
            if (c < m_cols) out[(size_t)r * ldo + c] = sum[i][j] + acc[i][j];
        }
    }
}

// By tiles of 16 x 16, an output a thread, k = 64 a stage of 16-byte cp.async, four stages.  24 rows of
// 64 against 2,048 columns: 3.0 us (the few-row kernel 5.7).
constexpr int NT = 16, NK = 64, NSTAGES = 4, NLD = NK + 4;

__global__ void __launch_bounds__(NT * NT)
gemm_f32_narrow_kernel(const float* __restrict__ x, const float* __restrict__ w,
                       float* __restrict__ out, int n_rows, int m_cols, int k_dim, int ldx,
                       int ldw, int ldo, int early) {
    extern __shared__ __align__(16) float smem[];
    float* xs = smem;                                // [STAGES][16][LD]
    float* ws = smem + NSTAGES * NT * NLD;
    const int tid = threadIdx.x, ty = tid / NT, tx = tid % NT;
    const int row0 = blockIdx.y * NT, col0 = blockIdx.x * NT;
    const int l_row = tid / 16, l_k = (tid % 16) * 4;
    const int steps = (k_dim + NK - 1) / NK;         // k_dim is a multiple of 4 here
    auto stage_w = [&](int step) {
        const int gk = step * NK + l_k, gc = col0 + l_row;
        const bool ok = step < steps && gc < m_cols && gk < k_dim;
        cp_async16_f32(ws + (step % NSTAGES * NT + l_row) * NLD + l_k,
                       ok ? w + (size_t)gc * ldw + gk : w, ok);
    };
    auto stage_x = [&](int step) {
        const int gk = step * NK + l_k, gr = row0 + l_row;
        const bool ok = step < steps && gr < n_rows && gk < k_dim;
        cp_async16_f32(xs + (step % NSTAGES * NT + l_row) * NLD + l_k,
                       ok ? x + (size_t)gr * ldx + gk : x, ok);
    };
    auto first_w = [&]() {
#pragma unroll
        for (int t = 0; t < NSTAGES - 1; ++t) stage_w(t);
    };
    if (early) first_w();
    pdl_wait();
    if (!early) first_w();
#pragma unroll
    for (int t = 0; t < NSTAGES - 1; ++t) {
        stage_x(t);
        cp_async_commit();
    }
    float acc = 0.0f, sum = 0.0f;
    for (int step = 0; step < steps; ++step) {
        cp_async_wait<NSTAGES - 2>();
        __syncthreads();                     // this step has landed; the stage refilled below is free
        stage_w(step + NSTAGES - 1);
        stage_x(step + NSTAGES - 1);
        cp_async_commit();
        if (step > 0 && step % (SEG / NK) == 0) {
            sum += acc;
            acc = 0.0f;
        }
        const float* xr = xs + (step % NSTAGES * NT + ty) * NLD;
        const float* wr = ws + (step % NSTAGES * NT + tx) * NLD;
#pragma unroll
        for (int k = 0; k < NK; k += 4) {
            const float4 a = *reinterpret_cast<const float4*>(xr + k);
            const float4 b = *reinterpret_cast<const float4*>(wr + k);
            acc = fmaf(a.x, b.x, acc);
            acc = fmaf(a.y, b.y, acc);
            acc = fmaf(a.z, b.z, acc);
            acc = fmaf(a.w, b.w, acc);
        }
    }
    cp_async_wait<0>();
    pdl_trigger();
    const int r = row0 + ty, c = col0 + tx;
    if (r < n_rows && c < m_cols) out[(size_t)r * ldo + c] = sum + acc;
}

int sm_count() {
    static int count = 0;
    if (count == 0) {
        int device = 0;
        if (cudaGetDevice(&device) != cudaSuccess ||
            cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
            count = 148;
    }
    return count;
}

// Lets a kernel's blocks have `smem` bytes of dynamic shared memory, once a device: `devices` (one a
// kernel) notes which.
template <typename F>
int allow_smem(F kernel, size_t smem, std::atomic<unsigned long long>& devices) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return (int)e;
    const unsigned long long bit = device < 64 ? 1ull << device : 0ull;
    if (devices.load() & bit) return 0;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    devices |= bit;
    return 0;
}

// Up to 32 rows (decode steps) the kernels ask for their first weights before the wait for the kernel
// before them, which must not have formed them; with more rows, they wait first.
int early_weights(int n_rows) { return n_rows <= 32; }

template <int TILE, int GROUPS>
int launch_tiles(const float* x, const float* w, float* out, int n_rows, int m_cols, int k_dim,
                 int ldx, int ldw, int ldo, cudaStream_t s) {
    using Shape = Tiles<TILE, GROUPS>;
    static std::atomic<unsigned long long> allowed{0};
    auto kernel = gemm_f32_kernel<TILE, GROUPS>;
    if (int e = allow_smem(kernel, Shape::SMEM, allowed)) return e;
    dim3 grid((m_cols + TILE - 1) / TILE, (n_rows + TILE - 1) / TILE);
    if (grid.y > 65535) return -3;
    const int vec_out = ldo % 4 == 0 && (uintptr_t)out % 16 == 0;
    return de_launch(kernel, grid, dim3(Shape::THREADS * GROUPS), Shape::SMEM, s, x, w, out, n_rows,
                     m_cols, k_dim, ldx, ldw, ldo, vec_out);
}

template <int T, int COLS, int SM_STAGES, int SM_K>
int launch_small(const float* x, const float* w, float* out, int n_rows, int m_cols, int k_dim,
                 int ldx, int ldw, int ldo, cudaStream_t s) {
    const size_t smem = ((size_t)2 * SM_WARPS * T * COLS +
                         (size_t)SM_WARPS * SM_STAGES * (COLS + T) * (SM_K + 4)) * sizeof(float);
    static std::atomic<unsigned long long> allowed{0};
    static std::atomic<int> blocks{0};               // of an SM
    auto kernel = gemm_f32_small_kernel<T, COLS, SM_STAGES, SM_K>;
    if (int e = allow_smem(kernel, smem, allowed)) return e;
    int per_sm = blocks.load();
    if (per_sm == 0) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, SM_WARPS * 32, smem) !=
                cudaSuccess || per_sm < 1) per_sm = 1;
        blocks = per_sm;
    }
    const int tiles = (m_cols + COLS - 1) / COLS, row_tiles = (n_rows + T - 1) / T;
    const int places = sm_count() * per_sm / row_tiles;
    dim3 grid(tiles < places ? tiles : (places < 1 ? 1 : places), row_tiles);
    return de_launch(kernel, grid, dim3(SM_WARPS * 32), smem, s, x, w, out, n_rows, m_cols, k_dim,
                     ldx, ldw, ldo, tiles, early_weights(n_rows));
}

int launch_wide(const float* x, const float* w, float* out, int n_rows, int m_cols, int k_dim,
                int ldx, int ldw, int ldo, bool vec, cudaStream_t s) {
    dim3 grid((m_cols + WT - 1) / WT, (n_rows + WT - 1) / WT);
    if (grid.y > 65535) return -3;
    return de_launch(vec ? gemm_f32_wide_kernel<true> : gemm_f32_wide_kernel<false>, grid, dim3(256),
                     0, s, x, w, out, n_rows, m_cols, k_dim, ldx, ldw, ldo);
}

int launch_narrow(const float* x, const float* w, float* out, int n_rows, int m_cols, int k_dim,
                  int ldx, int ldw, int ldo, cudaStream_t s) {
    static std::atomic<unsigned long long> allowed{0};
    const size_t smem = (size_t)NSTAGES * 2 * NT * NLD * sizeof(float);
    if (int e = allow_smem(gemm_f32_narrow_kernel, smem, allowed)) return e;
    dim3 grid((m_cols + NT - 1) / NT, (n_rows + NT - 1) / NT);
    if (grid.y > 65535) return -3;
    return de_launch(gemm_f32_narrow_kernel, grid, dim3(NT * NT), smem, s, x, w, out, n_rows, m_cols,
                     k_dim, ldx, ldw, ldo, early_weights(n_rows));
}

}  // namespace

DE_EXPORT int de_gemm_f32_small_rows() { return 32; }

namespace {
enum Form { NARROW, WIDE, FEW8, FEW16_WIDE, FEW16, FEW32_WIDE, FEW32, TILES64, TILES128 };

// `vec`: rows of whole 16-byte pieces at such addresses (NARROW and the FEW forms need them).
Form choose(int n_rows, int m_cols, int k_dim, bool vec) {
    auto tiles = [&](int rows, int cols) {
        return (long long)((n_rows + rows - 1) / rows) * ((m_cols + cols - 1) / cols);
    };
    const int sms = sm_count();
    // Short sums, few tiles: an output a thread (us at k = 64 / 256, against 2,048 columns: 1 row 2.1 /
    // 3.6, by FEW8 3.7 / 4.6; 24 rows 3.0 / 5.9, by FEW32 5.7 / 9.2; 64 rows 4.1 / 9.9, 9.8 / 16.8;
    // 130 rows, 1,152 tiles, go to WIDE, 5.1 / 14.7, by FEW32_WIDE 22 / 44.7).  From two segments on
    // FEW8 is faster for eight rows (k = 320: 4.5 and 4.8; 512: 6.1 and 4.7), and from three the others
    // (24 rows against 512 columns, k = 512: 5.5 and 9.0; 1,024: 9.3 and 6.4).  At k = 16 WIDE is as
    // fast from 128 tiles on and faster with many.
    if (vec && k_dim <= 512 && !(k_dim > 320 && n_rows <= 8) && tiles(16, 16) <= 704 &&
        (k_dim > 32 || tiles(16, 16) <= 128))
        return NARROW;
    // Short sums, more tiles: WIDE, or tiles of 128 with one of their two groups at work where these
    // are nearly whole rounds of one block an SM (us, 3.2 + 0.105 k a round; 2 + (8 + 0.058 a tile) k /
    // 256; measured at k = 64 / 256: 704 tiles of 64 14.9 / 50.0 and, two rounds, 19.0 / 57.7; 1,024
    // tiles 20.4 / 68.2 and, two rounds, 19.0 / 56.9).
    if (k_dim <= 320) {
        const float rounds = (float)((tiles(128, 128) + sms - 1) / sms);
        return rounds * (3.2f + 0.105f * k_dim) <
                       2.0f + (8.0f + 0.058f * tiles(64, 64)) * k_dim * (1.0f / 256)
                   ? TILES128 : WIDE;
    }
    // few rows, and somewhat more where tiles of 64 x 64 would leave a third of the SMs without one
    // (64 rows against 2,048 x 5,632: 74 against 152 us; 40 against 2,560 x 2,048: 40 against 61; 130
    // against 2,560 x 2,048, 120 tiles: 77 against 61; with k = 512 not: 24 rows against 11,264 45
    // against 34, 100 against 2,048 32 against 21).  (Zeros beyond k_dim add nothing to a chain, so
    // the kernels' results are the same bits.)
    if (vec && (n_rows <= (k_dim > 512 ? 32 : 16) ||
                (k_dim > 512 && n_rows <= 256 && tiles(64, 64) * 3 < 2LL * sms))) {
        // 32 columns a block where that still gives every SM two blocks' worth
        if (n_rows <= 8) return FEW8;
        if (n_rows <= 16) return tiles(16, 32) >= 2LL * sms ? FEW16_WIDE : FEW16;
        // (few columns: blocks of 16 rows are more blocks; 24 rows against 512 columns, k = 1,024: 6.4
        // against 10.0)
        if (tiles(16, 16) <= 128 && n_rows <= 64) return FEW16;
        return tiles(32, 32) >= 2LL * sms ? FEW32_WIDE : FEW32;
    }
    // tiles of 128: one block an SM; of 64: two, which take 0.54 of the time together.  The fewer
    // rounds of blocks decide.
    const long long wide = (tiles(128, 128) + sms - 1) / sms;
    const long long narrow = (tiles(64, 64) + 2 * sms - 1) / (2 * sms);
    return wide * 100 <= narrow * 54 ? TILES128 : TILES64;
}

int launch(Form form, const float* x, const float* w, float* out, int n_rows, int m_cols, int k_dim,
           int ldx, int ldw, int ldo, bool vec, cudaStream_t s) {
#define ARGS x, w, out, n_rows, m_cols, k_dim, ldx, ldw, ldo
    switch (form) {
        case NARROW: return launch_narrow(ARGS, s);
        case WIDE: return launch_wide(ARGS, vec, s);
        case FEW8: return launch_small<8, 16, 2, 64>(ARGS, s);
        case FEW16_WIDE: return launch_small<16, 32, 3, 32>(ARGS, s);
        case FEW16: return launch_small<16, 16, 4, 32>(ARGS, s);
        case FEW32_WIDE: return launch_small<32, 32, 2, 32>(ARGS, s);
        case FEW32: return launch_small<32, 16, 3, 32>(ARGS, s);
        case TILES64: return launch_tiles<64, 4>(ARGS, s);
        default: return launch_tiles<128, 2>(ARGS, s);
    }
#undef ARGS
}
}  // namespace

// Which kernel a product takes (a Form): operands of whole 16-byte pieces (`vec`) or not.
DE_EXPORT int de_gemm_f32_form(int n_rows, int m_cols, int k_dim, int vec) {
    return (int)choose(n_rows, m_cols, k_dim, vec != 0);
}

DE_EXPORT int de_gemm_f32(const float* x, const float* w, float* out, int n_rows, int m_cols,
                          int k_dim, int ldx, int ldw, int ldo, void* stream) {
    if (n_rows <= 0 || m_cols <= 0) return 0;
    if (k_dim <= 0) return -2;
    const bool vec4 = ldx % 4 == 0 && ldw % 4 == 0 && (uintptr_t)x % 16 == 0 &&
                      (uintptr_t)w % 16 == 0;
    return launch(choose(n_rows, m_cols, k_dim, vec4 && k_dim % 4 == 0), x, w, out, n_rows, m_cols,
                  k_dim, ldx, ldw, ldo, vec4, (cudaStream_t)stream);
}
