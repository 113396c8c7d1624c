// bfloat16 matrix product on the 5th-generation tensor cores: out[m, n] = sum_k x[m, k] * w[n, k],
// float32 accumulation in tensor memory, for prompt portions (many rows of x).
//
// A persistent kernel, one block per SM, each block walking over 128 x bn tiles of the output
// (bn a multiple of 32 up to 256, chosen by the host: the fewest rounds of tiles over the SMs, then
// the narrowest tile), with the roles split over warps:
//   * warp 0, one thread: moves 128 x 64 tiles of x and bn x 64 tiles of w into shared memory with
//     TMA (cp.async.bulk.tensor.2d, 128-byte swizzle, zero fill outside the matrices), 4 stages
//     deep, each stage guarded by a "full" mbarrier with a transaction count;
//   * warp 1, one thread: issues tcgen05.mma (kind::f16, M = 128, N = bn, K = 16; operands are
//     shared-memory descriptors), four per stage, hands the stage back with tcgen05.commit on its
//     "empty" mbarrier, and after a tile's last stage commits on the accumulator's "full" mbarrier;
//   * warps 2-5: the epilogue.  The accumulator is double-buffered in tensor memory (2 x 256
//     columns), so these warps read one tile with tcgen05.ld, convert, turn and store it while the
//     tensor core already works on the next.  The gated epilogue computes silu(gate) * up from the
//     two halves of the accumulator (src/layers/activation.py:6-9), so the activation costs no
//     pass over memory and the product's [gate | up] output is never written.
// Tiles are numbered with the rows of x fastest, so the blocks at work share a few tiles of w.
// No cluster launch; every block fetches its own tiles.
//
// Grouped form (routed experts): the rows of x are slots sorted by expert, 128 slots a tile of one
// expert (`tile_expert`, -1: a tile without an expert, which every role skips), w is the experts'
// matrices stacked ([experts * n_out, k]) and a tile takes its rows of w from its expert's part.
// `pair_of` tells which slots are taken (others are not stored) and, scattering, the output row of
// a slot.  An activation (by number, -1: none) is applied to the outputs, which are rounded to
// bfloat16 first as a product kernel followed by an activation kernel would.
//
// Every wait on an mbarrier is bounded: after SPIN_LIMIT polls a thread records status 3, stops
// waiting, and the block runs to its end (tensor memory is freed on every path); the host raises.
//
// Stands where the reference calls F.linear (src/layers/linear.py:19-20) on [1, T, H] inputs.

#include <cuda.h>

#include "common.cuh"
#include "tcgen05_common.cuh"
#include "tensor_maps.cuh"

DE_DEFINE_PDL_SWITCH

namespace {

constexpr int BM = 128;                // rows of x per tile = lanes of tensor memory
constexpr int BK = 64;                 // k per stage: 128 bytes of bfloat16 = one swizzle row
constexpr int THREADS = 192;           // producer warp, tensor-core warp, four epilogue warps
constexpr int A_BYTES = BM * BK * 2;   // 16 KB
constexpr int MAX_BN = 256;            // columns of an accumulator
constexpr int STAGES = 4;
constexpr int STAGE_BYTES = A_BYTES + MAX_BN * BK * 2;   // 48 KB: room for the widest tile of w
constexpr int SMEM_TILES = STAGES * STAGE_BYTES;

using namespace tc5;

// A warp's 32 rows of 32 columns on their way out: 16-byte pieces, their places within a row exchanged
// so that neither side meets a bank twice.
template <typename OutT> constexpr int OUT_PIECES = 32 * (int)sizeof(OutT) / 16;
template <typename OutT> constexpr int OUT_BYTES = 4 * 32 * 32 * (int)sizeof(OutT);     // four warps
template <typename OutT> __device__ __forceinline__ uint4* out_piece(uint4* stage, int row, int i) {
    constexpr int P = OUT_PIECES<OutT>;
    return stage + row * P + (i ^ ((P == 4 ? row >> 1 : row) & (P - 1)));
}

// Eight outputs of a row, of which `left` are the matrix's.
template <typename OutT>
__device__ __forceinline__ void store_eight(OutT* out, const float (&y)[8], int left, bool vec) {
    if (vec && left >= 8) {
        store8(out, y);
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (j < left) out[j] = from_float<OutT>(y[j]);
    }
}

// 32 outputs of every lane's row, columns c .. c + 31 of `out_tile` (of which `left` are the matrix's):
// by way of shared memory, so that lanes side by side write a row's bytes side by side (a lane a row
// writes 32 half sectors an instruction: what a round's last tiles, which nothing hides, waited for).
// 2,048 rows against 2,048 columns: float32 out with k = 128 6.1 us (8.5 so), bfloat16 out with k =
// 2,048 15.2 (15.6); 1,500 rows with k = 128 5.2 (6.9).
template <typename OutT>
__device__ __forceinline__ void store_columns(const float (&y)[32], OutT* out_tile, int ldo, int c,
                                              int left, bool vec, int dest, bool live, uint4* stage) {
    if (vec && c + 32 <= left) {
        constexpr int P = OUT_PIECES<OutT>, PER = 16 / (int)sizeof(OutT);
        const int lane = threadIdx.x & 31;
        const unsigned mask = __ballot_sync(0xffffffffu, live);
#pragma unroll
        for (int i = 0; i < P; ++i) {
            OutT four[PER];
#pragma unroll
            for (int j = 0; j < PER; ++j) four[j] = from_float<OutT>(y[i * PER + j]);
            *out_piece<OutT>(stage, lane, i) = *reinterpret_cast<const uint4*>(four);
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < P; ++i) {
            const int row = i * (32 / P) + lane / P;
            const int to = __shfl_sync(0xffffffffu, dest, row);
            if ((mask >> row) & 1)
                *reinterpret_cast<uint4*>(out_tile + (size_t)to * ldo + c + lane % P * PER) =
                    *out_piece<OutT>(stage, row, lane % P);
        }
        __syncwarp();
    } else if (live) {
        OutT* out_row = out_tile + (size_t)dest * ldo + c;
        for (int i = 0; i < 32; i += 8) {
            float eight[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) eight[j] = y[i + j];
            store_eight(out_row + i, eight, left - c - i, vec);
        }
    }
}

// silu(gate) * up; product outputs are rounded to bfloat16 before the activation, as a separate product
// and activation kernel would do
__device__ __forceinline__ float gated_output(unsigned gate, unsigned up) {
    const float g = __bfloat162float(__float2bfloat16_rn(__uint_as_float(gate)));
    const float u = __bfloat162float(__float2bfloat16_rn(__uint_as_float(up)));
    // fast division: a gate far below zero gives 0, the function's limit
    return __fdividef(g, 1.0f + __expf(-g)) * u;
}

// One tile's accumulator out of tensor memory: thread = row, which goes to row `dest`.  GATED: columns
// 0 .. bn/2-1 are gate outputs, bn/2 .. bn-1 the up outputs of the same features; bn/2 columns of
// silu(gate) * up go out.  `many` tiles a block: by way of shared memory; with few of them, whose last
// nothing hides, a gated tile's, half as many bytes, go out as they are formed, eight a lane at a time
// (2,048 rows against 2 x 1,024 with k = 256 9.8 us and 10.5, against 2 x 14,336 with k = 4,096, twelve
// tiles a block, 381 and 377).
template <bool GATED, typename OutT>
__device__ __forceinline__ void store_tile(unsigned lane_base, int bn, OutT* out_tile, int ldo, int dest,
                                           bool live, int cols_left, bool vec, uint4* stage, bool many,
                                           int act = -1) {
    const int cols = GATED ? bn / 2 : bn;
#pragma unroll 1
    for (int c = 0; c < cols; c += 32) {
        float y[32];
        if (GATED) {
            unsigned gate[32], up[32];
            tmem_load_32cols(lane_base + c, gate);
            tmem_load_32cols(lane_base + bn / 2 + c, up);
            tmem_wait_loads();
            if (!many) {
                if (live) {
                    OutT* out_row = out_tile + (size_t)dest * ldo + c;
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        float eight[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) eight[j] = gated_output(gate[i + j], up[i + j]);
                        store_eight(out_row + i, eight, cols_left - c - i, vec);
                    }
                }
                __syncwarp();
                continue;
            }
#pragma unroll
            for (int i = 0; i < 32; ++i) y[i] = gated_output(gate[i], up[i]);
        } else {
            unsigned v[32];
            tmem_load_32cols(lane_base + c, v);
            tmem_wait_loads();
#pragma unroll
            for (int i = 0; i < 32; ++i) y[i] = __uint_as_float(v[i]);
            if (act >= 0) {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    y[i] = de_activate(__bfloat162float(__float2bfloat16_rn(y[i])), act);
            }
        }
        store_columns<OutT>(y, out_tile, ldo, c, cols_left, vec, dest, live, stage);
    }
}

// map_w: the rows of w (GATED: the gate rows); map_up: the up rows (GATED only).
// GROUPED: see the head of this file; tile_expert [tiles_m], pair_of [m_rows], scatter: a slot's
// output row is its pair.
template <bool GATED, typename OutT, bool GROUPED = false>
__global__ void __launch_bounds__(THREADS, 1)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap map_x,
                    const __grid_constant__ CUtensorMap map_w,
                    const __grid_constant__ CUtensorMap map_up, OutT* __restrict__ out, int ldo,
                    int m_rows, int n_out, int k_dim, int bn, int tiles_m, int tiles_n,
                    int* status, const int* __restrict__ tile_expert,
                    const int* __restrict__ pair_of, int scatter, int act) {
    const int b_bytes = bn * BK * 2;
    const int out_cols = GATED ? bn / 2 : bn;             // output columns of a tile
    constexpr unsigned TMEM_COLS = 2 * MAX_BN;            // two accumulators
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // the tiles need 1024-byte alignment for the swizzle pattern
    unsigned char* tiles = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) unsigned long long full_bar[STAGES], empty_bar[STAGES];
    __shared__ __align__(8) unsigned long long acc_full[2], acc_empty[2];
    __shared__ unsigned tmem_base_slot;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k_steps = (k_dim + BK - 1) / BK;
    const int total = tiles_m * tiles_n;

    if (threadIdx.x == 0) {
#pragma unroll
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 4);                  // one arrival per epilogue warp
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) tmem_alloc(&tmem_base_slot, TMEM_COLS);
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const unsigned tmem_base = tmem_base_slot;

    bool ok = true;
    if (warp == 0) {
        // ---- producer: TMA loads, ahead of the tensor core by up to STAGES
        pdl_wait();                                        // x is the previous kernel's output
        if (lane == 0) {
            int it = 0;
            for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
                // grouped: the column tiles of a row tile run side by side (they share its rows, and the
                // row tiles of an expert, which follow one another, its weights)
                const int tile_m = GROUPED ? tile / tiles_n : tile % tiles_m;
                const int tile_n = GROUPED ? tile % tiles_n : tile / tiles_m;
                int w_row0 = tile_n * bn;
                if (GROUPED) {
                    const int e = tile_expert[tile_m];
                    if (e < 0) continue;
                    w_row0 += e * n_out;
                }
                for (int ks = 0; ks < k_steps; ++ks, ++it) {
                    const int s = it % STAGES;
                    if (it >= STAGES) ok = mbar_wait(&empty_bar[s], ((it / STAGES) - 1) & 1, status);
                    if (!ok) break;
                    unsigned char* a_tile = tiles + s * STAGE_BYTES;
                    unsigned char* b_tile = a_tile + A_BYTES;
                    mbar_expect_tx(&full_bar[s], A_BYTES + b_bytes);
                    tma_load_2d(a_tile, &map_x, &full_bar[s], ks * BK, tile_m * BM);
                    if (GATED) {
                        tma_load_2d(b_tile, &map_w, &full_bar[s], ks * BK, tile_n * (bn / 2));
                        tma_load_2d(b_tile + b_bytes / 2, &map_up, &full_bar[s], ks * BK,
                                    tile_n * (bn / 2));
                    } else {
                        tma_load_2d(b_tile, &map_w, &full_bar[s], ks * BK, w_row0);
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---- tensor core: four K = 16 steps per stage, accumulators in tensor memory
        if (GROUPED) pdl_wait();                           // tile_expert is a kernel's output
        if (lane == 0) {
            const unsigned idesc = instr_desc(BM, bn);
            int it = 0, local = -1;
            for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
                if (GROUPED && tile_expert[tile / tiles_n] < 0) continue;
                ++local;
                const int buf = local & 1;
                // the epilogue has read this accumulator's tile before last
                if (local >= 2) ok = mbar_wait(&acc_empty[buf], ((local >> 1) - 1) & 1, status);
                for (int ks = 0; ks < k_steps && ok; ++ks, ++it) {
                    const int s = it % STAGES;
                    ok = mbar_wait(&full_bar[s], (it / STAGES) & 1, status);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    const unsigned char* a_tile = tiles + s * STAGE_BYTES;
                    const unsigned long long a_desc = smem_desc(a_tile);
                    const unsigned long long b_desc = smem_desc(a_tile + A_BYTES);
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) {
                        // 16 elements of k are 32 bytes: the start addresses advance by 2
                        umma_bf16(tmem_base + buf * MAX_BN, a_desc + 2 * k, b_desc + 2 * k, idesc,
                                  ks > 0 || k > 0);
                    }
                    umma_commit(&empty_bar[s]);            // the stage is free when these are done
                }
                umma_commit(&acc_full[buf]);
            }
        }
    } else {
        // ---- epilogue: warp w reads the lanes 32 (w % 4) .. + 31 of the accumulator
        const int quarter = warp & 3;
        const bool vec = (ldo % 8 == 0) && ((reinterpret_cast<uintptr_t>(out) & 15) == 0);
        uint4* stage = reinterpret_cast<uint4*>(tiles + SMEM_TILES) + quarter * OUT_BYTES<OutT> / 64;
        int local = -1;
        if (GROUPED) pdl_wait();                           // tile_expert, pair_of: kernels' outputs
        for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
            const int tile_m = GROUPED ? tile / tiles_n : tile % tiles_m;
            const int tile_n = GROUPED ? tile % tiles_n : tile / tiles_m;
            if (GROUPED && tile_expert[tile_m] < 0) continue;
            ++local;
            const int buf = local & 1;
            ok = mbar_wait(&acc_full[buf], (local >> 1) & 1, status);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const int row = tile_m * BM + quarter * 32 + lane;
            const unsigned lane_base = tmem_base + buf * MAX_BN + ((unsigned)(quarter * 32) << 16);
            bool live = row < m_rows;
            int dest = row;
            if (GROUPED && live) {
                const int pair = pair_of[row];
                live = pair >= 0;
                if (scatter) dest = pair;
            }
            store_tile<GATED, OutT>(lane_base, bn, out + (size_t)tile_n * out_cols, ldo, dest, live,
                                    n_out - tile_n * out_cols, vec, stage,
                                    total > 3 * (int)gridDim.x, GROUPED ? act : -1);
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[buf]);
        }
    }
    __syncwarp();
    pdl_trigger();
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

// ---------------------------------------------------------------------------------- host side
// A [rows, k] bfloat16 matrix with row stride ld (elements), boxes of box_rows x 64.
int make_map(CUtensorMap* map, const void* base, int rows, int k, int ld, int box_rows) {
    return tensor_maps::get(map, base, rows, k, ld, box_rows, BK);
}

int sm_count() {
    static int count = 0;
    if (count == 0) {
        int device = 0;
        if (cudaGetDevice(&device) != cudaSuccess ||
            cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
            count <= 0)
            count = 148;
    }
    return count;
}

// The tile width: the candidate whose rounds of tiles over the SMs take least, a round of tiles bn wide
// taking about bn + `fixed` units.  Tiles narrower than 128 read too much of x and w per flop; they are
// candidates only when wider ones would leave SMs without a tile.
int best_width(int m_rows, int n_out, bool gated, int fixed) {
    const int tiles_m = (m_rows + BM - 1) / BM;
    const long sms = sm_count();
    auto tiles = [&](int bn) {
        const int cols = gated ? bn / 2 : bn;
        return (long)tiles_m * ((n_out + cols - 1) / cols);
    };
    int best = 0;
    long best_cost = 0;
    const bool small = tiles(128) < sms;
    const int step = gated ? 64 : 32;
    for (int bn = MAX_BN; bn >= (small ? step : 128); bn -= step) {
        const long cost = ((tiles(bn) + sms - 1) / sms) * (bn + fixed);
        if (best == 0 || cost < best_cost) {
            best = bn;
            best_cost = cost;
        }
    }
    return best;
}

// From k = 256 on a round hardly depends on the tiles' width: at k = 2,048 11.4 us for 128 columns, 12.2
// for 192, 13.4 for 256, at k = 4,096 23, 24.5 and 26.8, so the number of rounds decides and, among
// equals, the narrowest.  (By width + 16: 1,300 rows against 2 x 5,632 gated 79 us in seven rounds of
// 128, 53 in four of 256; 2,048 against 2 x 11,008 with k = 4,096 336 and 268; 1,024 against 2 x 5,632 64
// and 43.)  Of a smaller k a round is mostly its epilogue, at k = 64 1.45, 2.0 and 2.5 us, at k = 128 1.6, 2.0
// and 2.55: 1,300 rows against 12,288 in five rounds of 192 columns 11.8 and 12.3 us, in four of 256 12.4
// and 13.1 (with k = 256 14.2 and 14.1).
int choose_bn(int m_rows, int n_out, bool gated, int k_dim) {
    return best_width(m_rows, n_out, gated, k_dim < 256 ? 48 : 600);
}

template <bool GATED, typename OutT>
int launch(const void* x, int ldx, const void* w, int ldw, void* out, int ldo, int m_rows, int n_out,
           int k_dim, int* status, cudaStream_t s) {
    const int bn = choose_bn(m_rows, n_out, GATED, k_dim);
    CUtensorMap map_x, map_w, map_up;
    int code = make_map(&map_x, x, m_rows, k_dim, ldx, BM);
    if (code) return code;
    // gated: the gate rows and the up rows as matrices of their own, so that a tile at the edge
    // reads zeros and not the other's rows
    code = make_map(&map_w, w, n_out, k_dim, ldw, GATED ? bn / 2 : bn);
    if (code) return code;
    const void* up = GATED ? (const void*)((const __nv_bfloat16*)w + (size_t)n_out * ldw) : w;
    code = make_map(&map_up, up, n_out, k_dim, ldw, GATED ? bn / 2 : bn);
    if (code) return code;
    const size_t smem = (size_t)SMEM_TILES + OUT_BYTES<OutT> + 1024;
    auto kernel = gemm_tcgen05_kernel<GATED, OutT, false>;
    static bool sized = false;                 // per instantiation: the attribute is set once
    if (!sized) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (e != cudaSuccess) return (int)e;
        sized = true;
    }
    const int out_cols = GATED ? bn / 2 : bn;
    const int tiles_m = (m_rows + BM - 1) / BM, tiles_n = (n_out + out_cols - 1) / out_cols;
    const int total = tiles_m * tiles_n;
    const int grid = total < sm_count() ? total : sm_count();
    return de_launch(kernel, dim3(grid), dim3(THREADS), smem, s, map_x, map_w, map_up, (OutT*)out,
                     ldo, m_rows, n_out, k_dim, bn, tiles_m, tiles_n, status, (const int*)nullptr,
                     (const int*)nullptr, 0, -1);
}

}  // namespace

// How wide the tiles are for a product of these sizes.
DE_EXPORT int de_gemm_tcgen05_width(int m_rows, int n_out, int k_dim, int gated) {
    return choose_bn(m_rows, n_out, gated != 0, k_dim);
}
// How wide they would have to be if a tile took as long as its columns: the host decides with it whether
// a shape comes here.  By the width that the kernel takes, shapes would come that fill their rounds only
// so: 4,096 rows against 2,048 and 2,048 against 4,096, for which the library is the sooner one at every k
// (us, here and there, k = 128 7.9 and 6.7, 512 10.9 and 10.3, 2,048 26.5 and 24.8, 4,096 50.3 and 45.7).
DE_EXPORT int de_gemm_tcgen05_tile(int m_rows, int n_out, int gated) {
    return best_width(m_rows, n_out, gated != 0, 16);
}
DE_EXPORT int de_gemm_tcgen05_sms() { return sm_count(); }

// out_f32: float32 output (not with gated).  gated: w is [2 n_out, k] with the gate rows first; out
// is [m, n_out] = silu(x gate^T) * (x up^T).  x, w: bfloat16, rows contiguous, 16-byte aligned
// row starts.  `status` receives 3 if a wait inside the kernel ran out.
DE_EXPORT int de_gemm_tcgen05(const void* x, int ldx, const void* w, int ldw, void* out, int ldo,
                              int m_rows, int n_out, int k_dim, int out_f32, int gated, int* status,
                              void* stream) {
    if (m_rows <= 0 || n_out <= 0) return 0;
    if (k_dim <= 0 || k_dim % 8 != 0 || ldx % 8 != 0 || ldw % 8 != 0 || ((uintptr_t)x & 15) ||
        ((uintptr_t)w & 15))
        return -3;
    cudaStream_t s = (cudaStream_t)stream;
    if (gated) {
        if (out_f32) return -5;
        return launch<true, __nv_bfloat16>(x, ldx, w, ldw, out, ldo, m_rows, n_out, k_dim, status, s);
    }
    if (out_f32)
        return launch<false, float>(x, ldx, w, ldw, out, ldo, m_rows, n_out, k_dim, status, s);
    return launch<false, __nv_bfloat16>(x, ldx, w, ldw, out, ldo, m_rows, n_out, k_dim, status, s);
}

// The grouped product of the routed experts (see the head of this file): x [tiles * 128, k] rows
// of slots, w [experts * n_out, k] the experts' matrices stacked, tile_expert [tiles], pair_of
// [tiles * 128].  scatter = 0: out [tiles * 128, n_out] by slot; 1: out [pairs, n_out] by pair.
// act: an activation's number or -1.  bfloat16 in and out.
DE_EXPORT int de_gemm_tcgen05_grouped(const void* x, int ldx, const void* w, void* out, int ldo,
                                      const int* tile_expert, const int* pair_of, int tiles,
                                      int experts, int n_out, int k_dim, int scatter, int act,
                                      int* status, void* stream) {
    if (tiles <= 0 || n_out <= 0 || experts <= 0) return 0;
    if (k_dim <= 0 || k_dim % 8 != 0 || ldx % 8 != 0 || ((uintptr_t)x & 15) || ((uintptr_t)w & 15))
        return -3;
    const int m_rows = tiles * BM;
    // most reserved tiles may be without tokens: their rounds cost nothing, wider tiles would
    const int bn = best_width(m_rows, n_out, false, 16);
    CUtensorMap map_x, map_w;
    int code = make_map(&map_x, x, m_rows, k_dim, ldx, BM);
    if (code) return code;
    code = make_map(&map_w, w, experts * n_out, k_dim, k_dim, bn);
    if (code) return code;
    const size_t smem = (size_t)SMEM_TILES + OUT_BYTES<__nv_bfloat16> + 1024;
    auto kernel = gemm_tcgen05_kernel<false, __nv_bfloat16, true>;
    static bool sized = false;
    if (!sized) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (e != cudaSuccess) return (int)e;
        sized = true;
    }
    const int tiles_n = (n_out + bn - 1) / bn;
    const int total = tiles * tiles_n;
    const int grid = total < sm_count() ? total : sm_count();
    return de_launch(kernel, dim3(grid), dim3(THREADS), smem, (cudaStream_t)stream, map_x, map_w,
                     map_w, (__nv_bfloat16*)out, ldo, m_rows, n_out, k_dim, bn, tiles, tiles_n,
                     status, tile_expert, pair_of, scatter, act);
}
