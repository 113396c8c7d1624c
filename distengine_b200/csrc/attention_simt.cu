// Attention over the paged cache, float32 arithmetic on the CUDA cores, for float32 or bfloat16
// storage and any head size up to 256.  It serves the true 32-bit path and every head size that
// the tensor-core kernel does not take.  One kernel does prompt portions and decoded tokens: the
// host cuts the step into work items, each a tile of up to 8 query rows of one sequence and one
// kv head, with a range of keys.
//
// A row is (token, query head within the kv head's group); query head h reads kv head h / g
// (the reference expands k and v with repeat_interleave, src/layers/attention.py:35-36).
// score = (q . k) * scale, scale applied after the product (:38); a key is masked when its
// position is greater than the query's (:41-58) or, with a window, when it is `window` or more
// positions behind; softmax in float32 (:66-69) as a running maximum and sum over tiles of 32
// keys.  Keys come straight from the pages through the block table
// (position -> page, offset: src/distengine/paged_kv_cache.py:165-167); nothing is gathered or
// expanded in memory (the reference copies and expands, paged_kv_cache.py:197-214,318-321).
// A key inside a row's visible range whose page the block table does not hold is masked like a
// key outside the range (never scored as zeros) and recorded in the status word (code 2).
//
// Long key ranges of decoded tokens are cut into chunks that separate blocks work on; each writes
// an unnormalised partial result (accumulator, maximum, sum) into scratch memory, and
// `attn_combine` merges the chunks of a row in ascending order (in float32 steps of single tokens the
// block that finishes a row last does, after the rotation and the cache's write in the same kernel).

#include "common.cuh"

DE_DEFINE_PDL_SWITCH

namespace {

constexpr int ROWS = 8;        // query rows (warps) per block
constexpr int TILE = 32;       // keys per tile: one per lane
constexpr int MAX_D = 256;

struct WorkItem {              // 8 ints, built on the host
    int seq;                   // index into the step's sequence arrays
    int row0;                  // first row of the tile among the sequence's rows of this step
    int kv_begin, kv_end;      // key positions this item covers (before causal / window limits)
    int partial;               // slot in scratch, or -1: write the output directly
    int pad0, pad1, pad2;
};

struct CombineItem {           // 4 ints
    int seq, row0, first_partial, num_partials;
};

// A score as its row's maximum takes it: NaN as infinity, so that a tile of nothing but NaN is not one
// that the row does not see (fmaxf leaves NaN out), and the row's result is NaN in tiles of any height.
__device__ __forceinline__ float for_max(float s) { return s == s ? s : INFINITY; }

template <typename T>
__global__ void __launch_bounds__(ROWS * 32)
attn_simt_kernel(const T* __restrict__ q, int q_stride, T* __restrict__ out, int out_stride,
                 const T* __restrict__ k_pages, const T* __restrict__ v_pages,
                 const int* __restrict__ block_table, int table_stride, int num_pages,
                 const int* __restrict__ seq_slot, const int* __restrict__ seq_qstart,
                 const int* __restrict__ seq_qlen, const int* __restrict__ seq_pos0,
                 const WorkItem* __restrict__ items, float* __restrict__ partial_acc,
                 float* __restrict__ partial_ml, int partial_limit, int heads, int kv_heads, int d,
                 int page, float scale, int window, int* __restrict__ status) {
    extern __shared__ float smem[];
    float* Ks = smem;                       // [TILE][d + 1]; column d: 0, or -inf without a page
    float* Vs = Ks + TILE * (d + 1);        // [TILE][d]
    float* Qs = Vs + TILE * d;              // [ROWS][d]

    const WorkItem it = items[blockIdx.x];
    // (an item whose partial slot lies beyond the scratch it was given is skipped like padding)
    if (it.kv_begin >= it.kv_end || it.partial >= partial_limit) {
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

    pdl_wait();            // q, and the keys and values of this step's tokens, are just written
    for (int i = lane; i < d; i += 32)
        Qs[warp * d + i] = active ? to_float(q[(size_t)(tok0 + t) * q_stride + hq * d + i]) : 0.0f;

    // key range of the whole tile
    const int last_row = min(it.row0 + ROWS, rows_total) - 1;
    const int max_pos = pos0 + last_row / g, min_pos = pos0 + it.row0 / g;
    const int k_hi = min(it.kv_end, max_pos + 1);
    int k_lo_true = it.kv_begin;
    if (window > 0) k_lo_true = max(k_lo_true, min_pos - window + 1);
    const int k_lo = (k_lo_true / TILE) * TILE;       // tiles sit at absolute positions
    // key range of this warp's row
    int row_lo = it.kv_begin;
    if (window > 0) row_lo = max(row_lo, pos - window + 1);
    const int row_hi = min(it.kv_end, pos + 1);

    float m = -INFINITY, l = 0.0f;
    float acc[MAX_D / 32];
#pragma unroll
    for (int i = 0; i < MAX_D / 32; ++i) acc[i] = 0.0f;

    const size_t slab = (size_t)page * d;             // one (page, kv head)
    for (int kt = k_lo; kt < k_hi; kt += TILE) {
        __syncthreads();                              // the previous tile has been consumed
        for (int idx = threadIdx.x; idx < TILE * d; idx += ROWS * 32) {
            const int j = idx / d, dd = idx - j * d;
            const int kpos = kt + j;
            float kv = 0.0f, vv = 0.0f;
            bool held = true;
            if (kpos >= k_lo_true && kpos < k_hi) {
                const int page_id = block_table[(size_t)slot * table_stride + kpos / page];
                held = page_id >= 0 && page_id < num_pages;
                if (held) {
                    const size_t off =
                        ((size_t)page_id * kv_heads + hk) * slab + (size_t)(kpos % page) * d + dd;
                    kv = to_float(k_pages[off]);
                    vv = to_float(v_pages[off]);
                }
            }
            Ks[j * (d + 1) + dd] = kv;
            Vs[j * d + dd] = vv;
            if (dd == 0) {
                Ks[j * (d + 1) + d] = held ? 0.0f : -INFINITY;
                if (!held && status != nullptr) atomicExch(status, 2);
            }
        }
        __syncthreads();
        if (!active) continue;

        const int kpos = kt + lane;
        const float* kr = Ks + lane * (d + 1);
        const bool valid = kpos >= row_lo && kpos < row_hi && kr[d] == 0.0f;
        const float* qr = Qs + warp * d;
        float s = 0.0f;
        for (int dd = 0; dd < d; ++dd) s = fmaf(qr[dd], kr[dd], s);
        s = valid ? s * scale : -INFINITY;
        const float m_new = fmaxf(m, warp_max(for_max(s)));
        if (m_new == -INFINITY) continue;             // nothing of this tile is visible to the row
        const float p = valid ? expf(s - m_new) : 0.0f;
        const float corr = expf(m - m_new);           // 0 when m was -inf
        l = l * corr + warp_sum(p);
#pragma unroll
        for (int i = 0; i < MAX_D / 32; ++i) acc[i] *= corr;
        for (int j = 0; j < TILE; ++j) {
            const float pj = __shfl_sync(0xffffffffu, p, j);
            if (pj == 0.0f) continue;                 // uniform over the warp
            const float* vr = Vs + j * d;
#pragma unroll
            for (int i = 0; i < MAX_D / 32; ++i) {
                const int dd = lane + 32 * i;
                if (dd < d) acc[i] = fmaf(pj, vr[dd], acc[i]);
            }
        }
        m = m_new;
    }
    pdl_trigger();
    if (!active) return;

    if (it.partial < 0) {
        const float inv = l > 0.0f ? 1.0f / l : 0.0f;
        T* o = out + (size_t)(tok0 + t) * out_stride + hq * d;
#pragma unroll
        for (int i = 0; i < MAX_D / 32; ++i) {
            const int dd = lane + 32 * i;
            if (dd < d) o[dd] = from_float<T>(acc[i] * inv);
        }
    } else {
        const size_t idx = ((size_t)it.partial * kv_heads + hk) * ROWS + warp;
        float* pa = partial_acc + idx * d;
#pragma unroll
        for (int i = 0; i < MAX_D / 32; ++i) {
            const int dd = lane + 32 * i;
            if (dd < d) pa[dd] = acc[i];
        }
        if (lane == 0) {
            partial_ml[idx * 2] = m;
            partial_ml[idx * 2 + 1] = l;
        }
    }
}

// Row w of a tile: its partial results `first` .. `first + count - 1`, in ascending order, into o.  A warp.
template <typename T, int BLOCKS>                  // BLOCKS: of 32 features
__device__ __forceinline__ void merge_row(T* o, const float* partial_acc, const float* partial_ml,
                                          int first, int count, int kv_heads, int hk,
                                          int rows_per_tile, int w, int d) {
    const int lane = threadIdx.x & 31;
    float m = -INFINITY;
    for (int c = 0; c < count; ++c) {
        const size_t idx = ((size_t)(first + c) * kv_heads + hk) * rows_per_tile + w;
        m = fmaxf(m, __ldcg(partial_ml + idx * 2));
    }
    float l = 0.0f;
    float acc[BLOCKS];
#pragma unroll
    for (int i = 0; i < BLOCKS; ++i) acc[i] = 0.0f;
    // (everything is loaded without a branch on what was loaded before it)
#pragma unroll 4
    for (int c = 0; c < count; ++c) {
        const size_t idx = ((size_t)(first + c) * kv_heads + hk) * rows_per_tile + w;
        const float mc = __ldcg(partial_ml + idx * 2), lc = __ldcg(partial_ml + idx * 2 + 1);
        const bool any = mc != -INFINITY;         // else the chunk held no visible key
        const float f = any ? expf(mc - m) : 0.0f;
        if (any) l += lc * f;
        const float* pa = partial_acc + idx * d;
#pragma unroll
        for (int i = 0; i < BLOCKS; ++i) {
            const int dd = lane + 32 * i;
            const float v = dd < d ? __ldcg(pa + dd) : 0.0f;
            if (any) acc[i] = fmaf(v, f, acc[i]);
        }
    }
    const float inv = l > 0.0f ? 1.0f / l : 0.0f;
#pragma unroll
    for (int i = 0; i < BLOCKS; ++i) {
        const int dd = lane + 32 * i;
        if (dd < d) o[dd] = from_float<T>(acc[i] * inv);
    }
}

// The same attention for float32 pages whose rows are whole 16-byte pieces: tiles of keys and values
// come through three stages of 16-byte cp.async (eight threads a key, which look its page up once
// and a tile ahead), a warp takes RW rows and reads a key or a value from shared memory once for
// all of them.  A row's sums have the order of the kernel above - features ascending in a score,
// keys ascending in a weighted sum - so the two, and any RW, give the same bits.  Portions in tiles of
// 32 rows come here (RW 4), and tiles of 8 rows over few keys (RW 1, de_attn_simt_by_tiles).  The kernel
// above waits for one element's page and then its key at a time: a layer with a prompt of 400 tokens took
// 872 us by it, 325 by this one.
constexpr int STAGES = 3;

template <int RW, int VW, int NB>
__global__ void __launch_bounds__(ROWS * 32)
attn_simt_vec_kernel(const float* __restrict__ q, int q_stride, float* __restrict__ out,
                     int out_stride, const float* __restrict__ k_pages,
                     const float* __restrict__ v_pages, const int* __restrict__ block_table,
                     int table_stride, int num_pages, const int* __restrict__ seq_slot,
                     const int* __restrict__ seq_qstart, const int* __restrict__ seq_qlen,
                     const int* __restrict__ seq_pos0, const WorkItem* __restrict__ items,
                     float* __restrict__ partial_acc, float* __restrict__ partial_ml,
                     int partial_limit, int heads, int kv_heads, int d, int page, float scale,
                     int window, int aligned, int* __restrict__ status) {
    constexpr int TROWS = ROWS * RW;
    extern __shared__ __align__(16) float smem[];
    const int ks = d + 4;                             // a key's stride: 16-byte reads without conflicts
    const int stage_floats = TILE * (ks + d) + TILE;
    float* Qs = smem + STAGES * stage_floats;         // [TROWS][d]

    const WorkItem it = items[blockIdx.x];
    if (it.kv_begin >= it.kv_end || it.partial >= partial_limit) {
        pdl_wait();
        return;
    }
    const int hk = blockIdx.y;
    const int g = heads / kv_heads;
    const int qlen = seq_qlen[it.seq], pos0 = seq_pos0[it.seq];
    const int slot = seq_slot[it.seq], tok0 = seq_qstart[it.seq];
    const int rows_total = qlen * g;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    bool active[RW], any = false;
    int tok[RW], hq[RW], row_lo[RW], row_hi[RW];
#pragma unroll
    for (int i = 0; i < RW; ++i) {
        const int r = it.row0 + warp * RW + i;
        active[i] = r < rows_total;
        any |= active[i];
        tok[i] = active[i] ? r / g : 0;
        hq[i] = hk * g + (active[i] ? r % g : 0);
        const int pos = pos0 + tok[i];
        row_lo[i] = it.kv_begin;
        if (window > 0) row_lo[i] = max(row_lo[i], pos - window + 1);
        row_hi[i] = active[i] ? min(it.kv_end, pos + 1) : 0;
    }
    const int last_row = min(it.row0 + TROWS, rows_total) - 1;
    const int max_pos = pos0 + last_row / g, min_pos = pos0 + it.row0 / g;
    const int k_hi = min(it.kv_end, max_pos + 1);
    int k_lo_true = it.kv_begin;
    if (window > 0) k_lo_true = max(k_lo_true, min_pos - window + 1);
    const int k_lo = (k_lo_true / TILE) * TILE;       // tiles sit at absolute positions

    const int j = threadIdx.x >> 3, part = threadIdx.x & 7;    // this thread's key of a tile
    const int pieces = d >> 2;
    auto page_of = [&](int kt) {                      // of the key at kt + j; -2: outside the range
        const int kpos = kt + j;
        if (kpos < k_lo_true || kpos >= k_hi) return -2;
        return block_table[(size_t)slot * table_stride + kpos / page];
    };
    int next_page = page_of(k_lo);

    pdl_wait();            // q, and the keys and values of this step's tokens, are just written
    auto issue = [&](int kt, int stage) {
        float* kd = smem + stage * stage_floats + j * ks;
        float* vd = smem + stage * stage_floats + TILE * ks + j * d;
        const int page_id = next_page;
        next_page = page_of(kt + TILE);
        const bool read = page_id >= 0 && page_id < num_pages;
        const bool gone = page_id != -2 && !read;
        const size_t off = read ? (((size_t)page_id * kv_heads + hk) * page +
                                   (size_t)((kt + j) % page)) * d : 0;
        const int bytes = read ? 16 : 0;
        if (!aligned) {                               // pages that do not start at 16 bytes
            for (int c = part; c < d; c += 8) {
                kd[c] = read ? k_pages[off + c] : 0.0f;
                vd[c] = read ? v_pages[off + c] : 0.0f;
            }
        }
        for (int c = part; c < (aligned ? pieces : 0); c += 8) {
            const unsigned ka = (unsigned)__cvta_generic_to_shared(kd + 4 * c);
            const unsigned va = (unsigned)__cvta_generic_to_shared(vd + 4 * c);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(ka),
                         "l"(k_pages + off + 4 * c), "r"(bytes) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(va),
                         "l"(v_pages + off + 4 * c), "r"(bytes) : "memory");
        }
        if (part == 0) {
            smem[stage * stage_floats + TILE * (ks + d) + j] = gone ? -INFINITY : 0.0f;
            if (gone && status != nullptr) atomicExch(status, 2);
        }
    };
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (k_lo + s * TILE < k_hi) issue(k_lo + s * TILE, s);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
#pragma unroll
    for (int i = 0; i < RW; ++i)
        for (int dd = lane; dd < d; dd += 32)
            Qs[(warp * RW + i) * d + dd] =
                active[i] ? q[(size_t)(tok0 + tok[i]) * q_stride + hq[i] * d + dd] : 0.0f;

    float m[RW], l[RW], acc[RW][NB][VW];
#pragma unroll
    for (int i = 0; i < RW; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.0f;
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int e = 0; e < VW; ++e) acc[i][b][e] = 0.0f;
    }

    int stage = 0;
    for (int kt = k_lo; kt < k_hi; kt += TILE) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
        __syncthreads();                              // this tile has landed, the oldest is consumed
        const int free = stage == 0 ? STAGES - 1 : stage - 1;
        if (kt + (STAGES - 1) * TILE < k_hi) issue(kt + (STAGES - 1) * TILE, free);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        const float* Ks = smem + stage * stage_floats;
        const float* Vs = Ks + TILE * ks;
        stage = stage == STAGES - 1 ? 0 : stage + 1;
        if (!any) continue;

        const int kpos = kt + lane;
        const float4* kr = reinterpret_cast<const float4*>(Ks + lane * ks);
        float s[RW];
#pragma unroll
        for (int i = 0; i < RW; ++i) s[i] = 0.0f;
#pragma unroll 4
        for (int c = 0; c < pieces; ++c) {
            const float4 kk = kr[c];
#pragma unroll
            for (int i = 0; i < RW; ++i) {
                const float4 qq = reinterpret_cast<const float4*>(Qs + (warp * RW + i) * d)[c];
                s[i] = fmaf(qq.x, kk.x, s[i]);
                s[i] = fmaf(qq.y, kk.y, s[i]);
                s[i] = fmaf(qq.z, kk.z, s[i]);
                s[i] = fmaf(qq.w, kk.w, s[i]);
            }
        }
        const bool held = Vs[TILE * d + lane] == 0.0f;
        float p[RW];
        bool some = false;
#pragma unroll
        for (int i = 0; i < RW; ++i) {
            const bool valid = kpos >= row_lo[i] && kpos < row_hi[i] && held;
            const float sc = valid ? s[i] * scale : -INFINITY;
            const float m_new = fmaxf(m[i], warp_max(for_max(sc)));
            p[i] = 0.0f;
            if (m_new == -INFINITY) continue;         // nothing of this tile is visible to the row
            p[i] = valid ? expf(sc - m_new) : 0.0f;
            const float corr = expf(m[i] - m_new);    // 0 when m was -inf
            l[i] = l[i] * corr + warp_sum(p[i]);
#pragma unroll
            for (int b = 0; b < NB; ++b)
#pragma unroll
                for (int e = 0; e < VW; ++e) acc[i][b][e] *= corr;
            m[i] = m_new;
            some = true;
        }
        if (!some) continue;
#pragma unroll 4
        for (int key = 0; key < TILE; ++key) {
            float pj[RW];
            bool zero = true;
#pragma unroll
            for (int i = 0; i < RW; ++i) {
                pj[i] = __shfl_sync(0xffffffffu, p[i], key);
                zero &= pj[i] == 0.0f;
            }
            if (zero) continue;                       // uniform over the warp
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                const int dd = VW * lane + 32 * VW * b;
                if (dd >= d) continue;
                float v[VW];
                if (VW == 4) {
                    const float4 t = *reinterpret_cast<const float4*>(Vs + key * d + dd);
                    v[0] = t.x; v[1] = t.y; v[VW - 2] = t.z; v[VW - 1] = t.w;
                } else {
                    const float2 t = *reinterpret_cast<const float2*>(Vs + key * d + dd);
                    v[0] = t.x; v[1] = t.y;
                }
#pragma unroll
                for (int i = 0; i < RW; ++i) {
                    if (pj[i] == 0.0f) continue;
#pragma unroll
                    for (int e = 0; e < VW; ++e) acc[i][b][e] = fmaf(pj[i], v[e], acc[i][b][e]);
                }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    pdl_trigger();
#pragma unroll
    for (int i = 0; i < RW; ++i) {
        if (!active[i]) continue;
        float* o;
        float factor = 1.0f;
        if (it.partial < 0) {
            factor = l[i] > 0.0f ? 1.0f / l[i] : 0.0f;
            o = out + (size_t)(tok0 + tok[i]) * out_stride + hq[i] * d;
        } else {
            const size_t idx = ((size_t)it.partial * kv_heads + hk) * TROWS + warp * RW + i;
            o = partial_acc + idx * d;
            if (lane == 0) {
                partial_ml[idx * 2] = m[i];
                partial_ml[idx * 2 + 1] = l[i];
            }
        }
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int e = 0; e < VW; ++e) {
                const int dd = VW * lane + 32 * VW * b + e;
                if (dd < d) o[dd] = it.partial < 0 ? acc[i][b][e] * factor : acc[i][b][e];
            }
    }
}

// The same for tiles of 8 rows (decoded tokens, small portions), KEYS keys at a time, asked for at once,
// keys before values: a thread forms the scores of one key with RPT rows, a warp takes a row's maxima,
// weights and sums over the tiles of 32 keys, and then two rows' weighted sums over half of the
// features.  All sums in the order of the kernels above, so the same bits.
// Bound by the trips to memory that follow one another and by barriers.  A decode step of 8 sequences of
// 520 keys through 22 layers: 2,151 us with a warp a row through tiles of 32 keys, 2,000 so, 1,829 in one
// kernel with rotation, cache write and merge (`Fuse`; 16 us a layer instead of 28 for the three).
//
// With `fuse.on` (a step of single tokens, one tile of rows a sequence; an item's row0 and pad2 are then
// the token's position and its slot) a block also does what rope_kv_write and attn_combine do around it,
// in their arithmetic: it turns its queries, the block whose range ends with the token's own position
// turns that key and stores it and its value, and the block that finishes a tile last merges the
// tile's partial results.  No block waits for another.
// The code is kept small (a step streams all weights between two launches: instructions come from far)
// and so is the number of loads that wait for one another.
struct Fuse {
    int on;
    const float* inv_freq;     // or null: nothing is turned
    int rot, writes;           // writes 0: the cache is another run's
    int* counters;             // [sequences][kv heads], zero before and after
};

// `KEYS` rows of keys (`hide` given) or values of one kv head into `to`, eight threads a row; `skip`: a
// position that does not come from the pages.
template <int KEYS>
__device__ __noinline__ void copy_rows(const float* pages, float* to, int stride, float* hide,
                                       const int* table, int kt, int lo, int hi, int skip, int num_pages,
                                       int hk, int kv_heads, int page, int d, int aligned, int* status) {
    const int j0 = threadIdx.x >> 3, part = threadIdx.x & 7;
    int ids[KEYS / 32];
#pragma unroll
    for (int i = 0; i < KEYS / 32; ++i) {
        const int kpos = kt + j0 + 32 * i;
        ids[i] = kpos < lo || kpos >= hi ? -2 : table[kpos / page];      // -2: outside the range
    }
#pragma unroll
    for (int i = 0; i < KEYS / 32; ++i) {
        const int j = j0 + 32 * i;
        const bool read = ids[i] >= 0 && ids[i] < num_pages;
        const float* from = pages + (read ? (((size_t)ids[i] * kv_heads + hk) * page +
                                             (size_t)((kt + j) % page)) * d : 0);
        if (hide != nullptr && part == 0) {
            const bool gone = ids[i] != -2 && !read;
            hide[j] = gone ? -INFINITY : 0.0f;
            if (gone && status != nullptr) atomicExch(status, 2);
        }
        if (kt + j == skip && read) continue;
        if (aligned) {
            const unsigned at = (unsigned)__cvta_generic_to_shared(to + j * stride);
            for (int c = 4 * part; c < d; c += 32)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(at + 4 * c),
                             "l"(from + c), "r"(read ? 16 : 0) : "memory");
        } else {                                     // pages that do not start at 16 bytes
            for (int c = part; c < d; c += 8) to[j * stride + c] = read ? from[c] : 0.0f;
        }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}

template <int VW, int KEYS>
__global__ void __launch_bounds__(ROWS * 32, 3)
attn_simt_rows_kernel(const float* __restrict__ q, int q_stride, float* __restrict__ out,
                      int out_stride, const float* k_pages, const float* v_pages,
                      const int* __restrict__ block_table, int table_stride, int num_pages,
                      const int* __restrict__ seq_slot, const int* __restrict__ seq_qstart,
                      const int* __restrict__ seq_qlen, const int* __restrict__ seq_pos0,
                      const WorkItem* __restrict__ items, float* partial_acc, float* partial_ml,
                      int partial_limit, int heads, int kv_heads, int d, int page, float scale,
                      int window, int aligned, Fuse fuse, int* __restrict__ status) {
    constexpr int RPT = ROWS * KEYS / 256, NT = KEYS / TILE;   // rows of a thread's scores; tiles
    extern __shared__ __align__(16) float smem[];
    const int ks = d + 4;                            // a key's stride: 16-byte reads without conflicts
    float* Ks = smem;                                // [KEYS][ks]
    float* Vs = Ks + KEYS * ks;                      // [KEYS][d]
    float* Qs = Vs + KEYS * d;                       // [ROWS][d]
    float* Ps = Qs + ROWS * d;                       // [ROWS][KEYS]: scores, then weights
    float* hide = Ps + ROWS * KEYS;                  // [KEYS]: 0, or -inf without a page
    float* corr_s = hide + KEYS;                     // [ROWS][NT]
    float* l_s = corr_s + ROWS * NT;                 // [ROWS]
    float* turn_s = l_s + ROWS;                      // [d]: cosines, then sines (with fuse.on)

    const WorkItem it = items[blockIdx.x];
    if (it.kv_begin >= it.kv_end || it.partial >= partial_limit) {
        pdl_wait();
        return;
    }
    const int hk = blockIdx.y, g = heads / kv_heads;
    const int row0 = fuse.on ? 0 : it.row0, rows_total = fuse.on ? g : seq_qlen[it.seq] * g;
    const int pos0 = fuse.on ? it.row0 : seq_pos0[it.seq];
    const int slot = fuse.on ? it.pad2 : seq_slot[it.seq], tok0 = seq_qstart[it.seq];
    const int* table = block_table + (size_t)slot * table_stride;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int last_row = min(row0 + ROWS, rows_total) - 1;
    const int k_hi = min(it.kv_end, pos0 + last_row / g + 1);
    int k_lo_true = it.kv_begin;
    if (window > 0) k_lo_true = max(k_lo_true, pos0 + row0 / g - window + 1);
    const int k_lo = (k_lo_true / TILE) * TILE;      // tiles sit at absolute positions
    // the token's own key, if it is this block's to store; among the first keys it does not come from the
    // pages but from here, later ones are read back
    const int own = fuse.on && fuse.writes && pos0 >= k_lo_true && pos0 < k_hi ? pos0 : -1;
    const int skip = own < k_lo + KEYS ? own : -1;
    auto copy = [&](int kt, bool keys) {
        copy_rows<KEYS>(keys ? k_pages : v_pages, keys ? Ks : Vs, keys ? ks : d, keys ? hide : nullptr,
                        table, kt, k_lo_true, k_hi, skip, num_pages, hk, kv_heads, page, d, aligned,
                        status);
    };

    // Older keys, the only ones that a step's own cache holds here, are from kernels long before the last:
    // they are asked for before the wait.  Another run's cache got its newest key in this step, and
    // portions' keys were stored by the kernel before this one.
    const bool early = fuse.on && fuse.writes;
    if (!early) pdl_wait();
#pragma unroll 1
    for (int i = 0; i < 2; ++i) copy(k_lo, i == 0);
    const int half = fuse.on ? fuse.rot / 2 : 0;
    if ((int)threadIdx.x < half) {                   // (half <= MAX_D / 2)
        float sn = 0.0f, cs = 1.0f;
        if (fuse.inv_freq) sincosf((float)pos0 * fuse.inv_freq[threadIdx.x], &sn, &cs);
        turn_s[threadIdx.x] = cs;
        turn_s[half + threadIdx.x] = sn;
    }
    if (early) pdl_wait();
    if (fuse.on) __syncthreads();
    // queries, a warp a row; with fuse.on the warps go on with the token's own key and value
    const int qkv_rows = ROWS + (own >= 0 ? 2 : 0);
#pragma unroll 1
    for (int w = warp; w < qkv_rows; w += ROWS) {
        const int r = row0 + w;
        const bool active = w >= ROWS || r < rows_total;
        const int head = w == ROWS ? heads + hk : w > ROWS ? heads + kv_heads + hk : hk * g + r % g;
        const float* src = q + (size_t)(tok0 + (active && w < ROWS ? r / g : 0)) * q_stride +
                           (size_t)(active ? head : 0) * d;
        float *to = Qs + w * d, *to_page = nullptr;
        if (w >= ROWS) {
            // (its page is missing: the key is hidden, and the status says so)
            const int id = table[own / page];
            if (id < 0 || id >= num_pages) continue;
            const size_t at = (((size_t)id * kv_heads + hk) * page + (size_t)(own % page)) * d;
            to_page = const_cast<float*>(w == ROWS ? k_pages : v_pages) + at;
            to = skip < 0 ? nullptr : w == ROWS ? Ks + (own - k_lo) * ks : Vs + (own - k_lo) * d;
        }
        const int turned = w > ROWS ? 0 : half;      // pairs
#pragma unroll 1
        for (int i = lane; i < d - turned; i += 32) {
            const int c = i < turned ? i : i + turned;
            float a = active ? src[c] : 0.0f, b = 0.0f;
            if (i < turned) {
                b = active ? src[i + half] : 0.0f;
                rope_rotate(a, b, turn_s[i], turn_s[half + i], a, b);
                if (to != nullptr) to[i + half] = b;
            }
            if (to != nullptr) to[c] = a;
            if (to_page != nullptr) {
                to_page[c] = a;
                if (i < turned) to_page[i + half] = b;
            }
        }
    }
    // scores: key `key` with rows srow .. srow + RPT - 1
    const int key = threadIdx.x % KEYS, srow = threadIdx.x / KEYS * RPT;
    float m = -INFINITY, l = 0.0f;                   // of row `warp`
    // weighted sums: rows arow, arow + 1, features f .. f + VW - 1
    const int arow = 2 * (warp & 3), f = (warp >> 2) * 32 * VW + VW * lane;
    float acc[2][VW];
#pragma unroll
    for (int e = 0; e < VW; ++e) acc[0][e] = acc[1][e] = 0.0f;

#pragma unroll 1
    for (int kt = k_lo; kt < k_hi; kt += KEYS) {
        const bool more = kt + KEYS < k_hi;
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();                             // the keys have landed
        {
            const float4* kr = reinterpret_cast<const float4*>(Ks + key * ks);
            const float4* qr = reinterpret_cast<const float4*>(Qs + srow * d);
            float s[RPT];
#pragma unroll
            for (int i = 0; i < RPT; ++i) s[i] = 0.0f;
#pragma unroll 4
            for (int c = 0; c < d / 4; ++c) {
                const float4 kk = kr[c];
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    const float4 qq = qr[i * (d / 4) + c];
                    s[i] = fmaf(qq.x, kk.x, s[i]);
                    s[i] = fmaf(qq.y, kk.y, s[i]);
                    s[i] = fmaf(qq.z, kk.z, s[i]);
                    s[i] = fmaf(qq.w, kk.w, s[i]);
                }
            }
            const int kpos = kt + key;
            const bool held = hide[key] == 0.0f && kpos < it.kv_end;
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                const int r = row0 + srow + i, pos = pos0 + r / g;
                const bool valid = held && r < rows_total && kpos >= it.kv_begin && kpos <= pos &&
                                   (window <= 0 || kpos > pos - window);
                Ps[(srow + i) * KEYS + key] = valid ? s[i] * scale : -INFINITY;
            }
        }
        __syncthreads();                             // the scores are written, the keys have been used
        if (more) copy(kt + KEYS, true);
        else asm volatile("cp.async.commit_group;\n" ::: "memory");
        {
            float sc[NT], top[NT], corr[NT];
#pragma unroll
            for (int t = 0; t < NT; ++t) sc[t] = Ps[warp * KEYS + t * TILE + lane];
#pragma unroll
            for (int t = 0; t < NT; ++t) top[t] = warp_max(for_max(sc[t]));
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                const float m_new = fmaxf(m, top[t]);
                // (nothing of this tile is visible to the row, nor of those before: all weights are 0)
                const float use = m_new == -INFINITY ? 0.0f : m_new;
                corr[t] = m_new == -INFINITY ? 1.0f : expf(m - use);     // 0 when m was -inf
                sc[t] = sc[t] == -INFINITY ? 0.0f : expf(sc[t] - use);
                m = m_new;
            }
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                l = l * corr[t] + warp_sum(sc[t]);
                Ps[warp * KEYS + t * TILE + lane] = sc[t];
                if (lane == 0) corr_s[warp * NT + t] = corr[t];
            }
        }
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();                             // the weights are written, the values have landed
        if (f < d) {
#pragma unroll 1
            for (int k0 = 0; k0 < KEYS && kt + k0 < k_hi; k0 += 4) {
                if (k0 % TILE == 0) {
#pragma unroll
                    for (int i = 0; i < 2; ++i)
#pragma unroll
                        for (int e = 0; e < VW; ++e) acc[i][e] *= corr_s[(arow + i) * NT + k0 / TILE];
                }
                const float4 p0 = *reinterpret_cast<const float4*>(Ps + arow * KEYS + k0);
                const float4 p1 = *reinterpret_cast<const float4*>(Ps + (arow + 1) * KEYS + k0);
                const float p[2][4] = {{p0.x, p0.y, p0.z, p0.w}, {p1.x, p1.y, p1.z, p1.w}};
                float v[4][VW];
#pragma unroll
                for (int x = 0; x < 4; ++x)
#pragma unroll
                    for (int e = 0; e < VW; ++e) v[x][e] = Vs[(k0 + x) * d + f + e];
#pragma unroll
                for (int x = 0; x < 4; ++x)
#pragma unroll
                    for (int i = 0; i < 2; ++i)
#pragma unroll
                        for (int e = 0; e < VW; ++e) {
                            // (keys of weight 0 add nothing, whatever their values)
                            const float with = fmaf(p[i][x], v[x][e], acc[i][e]);
                            acc[i][e] = p[i][x] != 0.0f ? with : acc[i][e];
                        }
            }
        }
        __syncthreads();                             // the values have been used
        if (more) copy(kt + KEYS, false);
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    pdl_trigger();
    if (lane == 0) {
        l_s[warp] = l;
        if (it.partial >= 0 && row0 + warp < rows_total) {
            const size_t idx = ((size_t)it.partial * kv_heads + hk) * ROWS + warp;
            partial_ml[idx * 2] = m;
            partial_ml[idx * 2 + 1] = l;
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int r = row0 + arow + i;
        if (r >= rows_total || f >= d) continue;
        float factor = 1.0f;
        float* o = partial_acc + (((size_t)max(it.partial, 0) * kv_heads + hk) * ROWS + arow + i) * d + f;
        if (it.partial < 0) {
            factor = l_s[arow + i] > 0.0f ? 1.0f / l_s[arow + i] : 0.0f;
            o = out + (size_t)(tok0 + r / g) * out_stride + (hk * g + r % g) * d + f;
        }
#pragma unroll
        for (int e = 0; e < VW; ++e) o[e] = it.partial < 0 ? acc[i][e] * factor : acc[i][e];
    }
    if (!fuse.on || it.partial < 0) return;
    // the block that finishes the tile last merges its live partial results
    __shared__ int last_s;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        int* counter = fuse.counters + (size_t)it.seq * kv_heads + hk;
        last_s = atomicAdd(counter, 1) == it.pad1 - 1;
        if (last_s) *counter = 0;
    }
    __syncthreads();
    if (!last_s) return;
    __threadfence();
    if (warp < rows_total)
        merge_row<float, 2 * VW>(out + (size_t)tok0 * out_stride + (hk * g + warp) * d, partial_acc,
                                 partial_ml, it.pad0, it.pad1, kv_heads, hk, ROWS, warp, d);
}

// Merge the chunks of each row, in ascending order of the chunks.
template <typename T>
__global__ void __launch_bounds__(ROWS * 32)
attn_combine_kernel(T* __restrict__ out, int out_stride, const int* __restrict__ seq_qstart,
                    const int* __restrict__ seq_qlen, const CombineItem* __restrict__ items,
                    const float* __restrict__ partial_acc, const float* __restrict__ partial_ml,
                    int partial_limit, int heads, int kv_heads, int d, int rows_per_tile) {
    const CombineItem it = items[blockIdx.x];
    pdl_wait();
    pdl_trigger();
    if (it.num_partials <= 0) return;
    // slots beyond the scratch that was given: nothing is read, the rows are left as they are
    if (it.first_partial < 0 || it.first_partial > partial_limit - it.num_partials) return;
    const int hk = blockIdx.y;
    const int g = heads / kv_heads;
    const int rows_total = seq_qlen[it.seq] * g;
    // a warp a row, the rows of a tile over blockIdx.z
    for (int w = blockIdx.z * ROWS + (threadIdx.x >> 5); w < rows_per_tile; w += ROWS * gridDim.z) {
        const int r = it.row0 + w;
        if (r >= rows_total) continue;
        const int t = r / g, hq = hk * g + r % g;
        merge_row<T, MAX_D / 32>(out + (size_t)(seq_qstart[it.seq] + t) * out_stride + hq * d, partial_acc,
                     partial_ml, it.first_partial, it.num_partials, kv_heads, hk, rows_per_tile, w, d);
    }
}

}  // namespace

DE_EXPORT int de_attn_simt_rows_per_tile() { return ROWS; }

// shared memory of attn_simt_vec_kernel
static size_t vec_bytes(int d, int tile_rows) {
    return (size_t)(STAGES * (TILE * (2 * d + 4) + TILE) + tile_rows * d) * sizeof(float);
}
// Whether `blocks` of tiles of 8 float32 rows whose longest sees `keys` keys are sooner through tiles of 32
// keys (de_attn_simt with tile_rows -8) than a range at once, which costs a block some 1.5 us more before
// its first scores (us, 32 heads on 4 of 64: one portion of 10 tokens 5.4 and 6.9, four of 17 6.3 and 9.7, 10
// of 4 behind 1,000 58 and 46; 32 on 8 of 128, one of 10 5.9 and 6.7, one of 33 9.0 and 7.9) but then wins by
// a quarter to two fifths.  Up to one tile of keys unless that takes more rounds of blocks over the SMs,
// three of which an SM holds the other way; up to three tiles where it takes fewer (heads of 64: 480
// blocks of 43 keys 13.3 and 18.1).
DE_EXPORT int de_attn_simt_by_tiles(int d, int blocks, int keys) {
    if (d <= 0 || d > MAX_D || d % 4 != 0 || keys > 3 * TILE) return 0;
    int device = 0, sms = 148;
    if (cudaGetDevice(&device) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
        sms = 148;
    int places = (int)(227 * 1024 / (vec_bytes(d, ROWS) + 1024));
    places = places < 1 ? 1 : places > 8 ? 8 : places;       // (256 threads each)
    const int here = (blocks + places * sms - 1) / (places * sms);
    const int at_once = (blocks + 3 * sms - 1) / (3 * sms);
    return keys <= TILE ? here <= at_once : here < at_once;
}

static int launch_simt(int dtype, const void* q, int q_stride, void* out, int out_stride,
                       const void* k_pages, const void* v_pages, const int* block_table,
                       int table_stride, int num_pages, const int* seq_slot,
                       const int* seq_qstart, const int* seq_qlen, const int* seq_pos0,
                       const int* items, int num_items, float* partial_acc, float* partial_ml,
                       int partial_limit, int heads, int kv_heads, int d, int page, float scale,
                       int window, int* status, void* stream, int tile_rows = ROWS,
                       Fuse fuse = Fuse{0, nullptr, 0, 0, nullptr});
static int launch_combine(int dtype, void* out, int out_stride, const int* seq_qstart,
                          const int* seq_qlen, const int* items, int num_items,
                          const float* partial_acc, const float* partial_ml, int partial_limit,
                          int heads, int kv_heads, int d, int rows_per_tile, void* stream);

DE_EXPORT int de_attn_simt(int dtype, const void* q, int q_stride, void* out, int out_stride,
                           const void* k_pages, const void* v_pages, const int* block_table,
                           int table_stride, int num_pages, const int* seq_slot,
                           const int* seq_qstart, const int* seq_qlen, const int* seq_pos0,
                           const int* items, int num_items, float* partial_acc, float* partial_ml,
                           int heads, int kv_heads, int d, int page, float scale, int window,
                           int tile_rows, int* status, void* stream) {
    // (tile_rows -8: tiles of 8 rows, see de_attn_simt_by_tiles)
    return launch_simt(dtype, q, q_stride, out, out_stride, k_pages, v_pages, block_table,
                       table_stride, num_pages, seq_slot, seq_qstart, seq_qlen, seq_pos0, items,
                       num_items, partial_acc, partial_ml, 0x7fffffff, heads, kv_heads, d, page,
                       scale, window, status, stream, tile_rows);
}

// `partial_limit`: partial slots that the scratch holds (work items that name a slot beyond it are
// skipped); `status`: may be null.
static int launch_simt(int dtype, const void* q, int q_stride, void* out, int out_stride,
                       const void* k_pages, const void* v_pages, const int* block_table,
                       int table_stride, int num_pages, const int* seq_slot,
                       const int* seq_qstart, const int* seq_qlen, const int* seq_pos0,
                       const int* items, int num_items, float* partial_acc, float* partial_ml,
                       int partial_limit, int heads, int kv_heads, int d, int page, float scale,
                       int window, int* status, void* stream, int tile_rows, Fuse fuse) {
    if (num_items <= 0) return 0;
    if (d <= 0 || d > MAX_D || heads % kv_heads != 0) return -2;
    cudaStream_t s = (cudaStream_t)stream;
    const bool vec = dtype == DE_F32 && d % 4 == 0;
    const int aligned = (uintptr_t)k_pages % 16 == 0 && (uintptr_t)v_pages % 16 == 0;
    const bool by_tiles = tile_rows == -ROWS;        // tiles of 8 rows through the kernel for tiles of keys
    if (by_tiles) tile_rows = ROWS;
    if (by_tiles && (!vec || fuse.on)) return -5;
    if (tile_rows != ROWS && !(vec && tile_rows == 4 * ROWS)) return -5;
    if (vec) {
        const size_t bytes = vec_bytes(d, tile_rows);
#define LAUNCH_VEC(RW, VW, NB)                                                                  \
    do {                                                                                        \
        auto kernel = attn_simt_vec_kernel<RW, VW, NB>;                                         \
        if (bytes > 48 * 1024) {                                                                \
            const cudaError_t e = cudaFuncSetAttribute(                                         \
                kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);               \
            if (e != cudaSuccess) return (int)e;                                                \
        }                                                                                       \
        return de_launch(kernel, dim3(num_items, kv_heads), dim3(ROWS * 32), bytes, s,          \
                         (const float*)q, q_stride, (float*)out, out_stride,                    \
                         (const float*)k_pages, (const float*)v_pages, block_table,             \
                         table_stride, num_pages, seq_slot, seq_qstart, seq_qlen, seq_pos0,     \
                         (const WorkItem*)items, partial_acc, partial_ml, partial_limit, heads, \
                         kv_heads, d, page, scale, window, aligned, status);                    \
    } while (0)
        if (by_tiles) {
            if (d <= 64) LAUNCH_VEC(1, 2, 1);
            if (d <= 128) LAUNCH_VEC(1, 4, 1);
            LAUNCH_VEC(1, 4, 2);
        }
        if (tile_rows == ROWS) {
#define LAUNCH_ROWS(VW, KEYS)                                                                   \
    do {                                                                                        \
        auto kernel = attn_simt_rows_kernel<VW, KEYS>;                                          \
        const size_t need = (size_t)(KEYS * (2 * d + 4) + ROWS * d + ROWS * KEYS + KEYS +       \
                                     ROWS * (KEYS / TILE) + ROWS + d) * sizeof(float);          \
        if (need > 48 * 1024) {                                                                 \
            const cudaError_t e = cudaFuncSetAttribute(                                         \
                kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)need);                \
            if (e != cudaSuccess) return (int)e;                                                \
        }                                                                                       \
        return de_launch(kernel, dim3(num_items, kv_heads), dim3(ROWS * 32), need, s,           \
                         (const float*)q, q_stride, (float*)out, out_stride,                    \
                         (const float*)k_pages, (const float*)v_pages, block_table,             \
                         table_stride, num_pages, seq_slot, seq_qstart, seq_qlen, seq_pos0,     \
                         (const WorkItem*)items, partial_acc, partial_ml, partial_limit, heads, \
                         kv_heads, d, page, scale, window, aligned, fuse, status);              \
    } while (0)
            if (d <= 64) LAUNCH_ROWS(1, 128);
            if (d <= 128) LAUNCH_ROWS(2, 64);
            LAUNCH_ROWS(4, 32);
#undef LAUNCH_ROWS
        }
        if (d <= 64) LAUNCH_VEC(4, 2, 1);
        if (d <= 128) LAUNCH_VEC(4, 4, 1);
        LAUNCH_VEC(4, 4, 2);
#undef LAUNCH_VEC
    }
    const size_t smem = (size_t)(TILE * (d + 1) + TILE * d + ROWS * d) * sizeof(float);
    dim3 grid(num_items, kv_heads);
    cudaError_t e;
#define LAUNCH(T)                                                                               \
    do {                                                                                        \
        if (smem > 48 * 1024) {                                                                 \
            e = cudaFuncSetAttribute(attn_simt_kernel<T>,                                       \
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);   \
            if (e != cudaSuccess) return (int)e;                                                \
        }                                                                                       \
        return de_launch(attn_simt_kernel<T>, grid, dim3(ROWS * 32), smem, s, (const T*)q,      \
                         q_stride, (T*)out, out_stride, (const T*)k_pages, (const T*)v_pages,   \
                         block_table, table_stride, num_pages, seq_slot, seq_qstart, seq_qlen,  \
                         seq_pos0, (const WorkItem*)items, partial_acc, partial_ml,             \
                         partial_limit, heads, kv_heads, d, page, scale, window, status);       \
    } while (0)
    if (dtype == DE_BF16) LAUNCH(__nv_bfloat16);
    LAUNCH(float);
#undef LAUNCH
}

// A step of single tokens in float32 in one launch: qkv rows [q heads | k heads | v heads] as the product
// left them (`Fuse`); `items` as de_attn_simt takes them for tiles of 8 rows, up to 8 query heads a kv
// head; `counters`: int32 [tiles * kv_heads], zero before and after.
DE_EXPORT int de_attn_simt_decode(const void* qkv, int qkv_stride, void* out, int out_stride,
                                  void* k_pages, void* v_pages, const int* block_table,
                                  int table_stride, int num_pages, const int* seq_slot,
                                  const int* seq_qstart, const int* seq_qlen, const int* seq_pos0,
                                  const int* items, int num_items, float* partial_acc,
                                  float* partial_ml, int* counters, const float* inv_freq, int rot,
                                  int writes, int heads, int kv_heads, int d, int page, float scale,
                                  int window, int* status, void* stream) {
    if (d % 4 != 0 || kv_heads <= 0 || heads > ROWS * kv_heads || rot < 0 || rot % 2 || rot > d) return -2;
    return launch_simt(DE_F32, qkv, qkv_stride, out, out_stride, k_pages, v_pages, block_table,
                       table_stride, num_pages, seq_slot, seq_qstart, seq_qlen, seq_pos0, items,
                       num_items, partial_acc, partial_ml, 0x7fffffff, heads, kv_heads, d, page,
                       scale, window, status, stream, ROWS, Fuse{1, inv_freq, rot, writes, counters});
}

// `rows_per_tile`: rows of a tile in the partial layout (8 for the kernels above, 32 for the one of
// portions; the tensor-core kernel writes the same layout with its own tile height).
DE_EXPORT int de_attn_combine(int dtype, void* out, int out_stride, const int* seq_qstart,
                              const int* seq_qlen, const int* items, int num_items,
                              const float* partial_acc, const float* partial_ml, int heads,
                              int kv_heads, int d, int rows_per_tile, void* stream) {
    return launch_combine(dtype, out, out_stride, seq_qstart, seq_qlen, items, num_items,
                          partial_acc, partial_ml, 0x7fffffff, heads, kv_heads, d, rows_per_tile,
                          stream);
}

static int launch_combine(int dtype, void* out, int out_stride, const int* seq_qstart,
                          const int* seq_qlen, const int* items, int num_items,
                          const float* partial_acc, const float* partial_ml, int partial_limit,
                          int heads, int kv_heads, int d, int rows_per_tile, void* stream) {
    if (num_items <= 0) return 0;
    if (d <= 0 || d > MAX_D) return -2;
    cudaStream_t s = (cudaStream_t)stream;
    dim3 grid(num_items, kv_heads, (rows_per_tile + ROWS - 1) / ROWS);
    if (dtype == DE_BF16)
        return de_launch(attn_combine_kernel<__nv_bfloat16>, grid, dim3(ROWS * 32), 0, s,
                         (__nv_bfloat16*)out, out_stride, seq_qstart, seq_qlen,
                         (const CombineItem*)items, partial_acc, partial_ml, partial_limit, heads,
                         kv_heads, d, rows_per_tile);
    return de_launch(attn_combine_kernel<float>, grid, dim3(ROWS * 32), 0, s, (float*)out,
                     out_stride, seq_qstart, seq_qlen, (const CombineItem*)items, partial_acc,
                     partial_ml, partial_limit, heads, kv_heads, d, rows_per_tile);
}

// ------------------------------------------------------------------------------------------
// The variant that allocates nothing: see attention_static_scratch.h for who needs it and the
// rules.  The scratch for the partial results is this file-scope device array.  Its name is a
// device symbol: host code must not pass it to a kernel as if it were a pointer (on the host the
// name stands for a shadow object, not for device memory); the device address is looked up once
// per device with cudaGetSymbolAddress and that pointer is what the kernels get.
// ------------------------------------------------------------------------------------------
#include <cstdio>
#include <mutex>

#include "attention_static_scratch.h"

static __device__ __align__(256) float g_static_scratch[DE_ATTN_STATIC_SCRATCH_FLOATS];

namespace {
constexpr int MAX_DEVICES = 64;
float* g_scratch_address[MAX_DEVICES] = {};       // per device, filled at the first call there
std::mutex g_scratch_mutex;
thread_local char g_static_error[256] = "";

// The device address of the array on the current device; looked up at the first call on it.
int static_scratch_address(float** address) {
    int device = -1;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return (int)e;
    if (device < 0 || device >= MAX_DEVICES) return -11;
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (g_scratch_address[device] == nullptr) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_static_scratch);
        if (e != cudaSuccess) return (int)e;
        g_scratch_address[device] = static_cast<float*>(p);
    }
    *address = g_scratch_address[device];
    return 0;
}
}  // namespace

DE_EXPORT const char* de_attn_static_scratch_error(void) { return g_static_error; }

DE_EXPORT int de_attn_simt_static_scratch(
    int dtype, const void* q, int q_stride, void* out, int out_stride, const void* k_pages,
    const void* v_pages, const int* block_table, int table_stride, int num_pages,
    const int* seq_slot, const int* seq_qstart, const int* seq_qlen, const int* seq_pos0,
    const int* items, int num_items, const int* combine_items, int num_combine, int num_partials,
    int heads, int kv_heads, int head_dim, int page, float scale, int window, void* stream) {
    g_static_error[0] = '\0';
    if (num_items <= 0) return 0;
    if (head_dim <= 0 || head_dim > MAX_D || kv_heads <= 0 || heads % kv_heads != 0 ||
        num_partials < 0) {
        std::snprintf(g_static_error, sizeof(g_static_error),
                      "de_attn_simt_static_scratch: head_dim %d (1..%d), heads %d, kv_heads %d or "
                      "num_partials %d cannot be used", head_dim, MAX_D, heads, kv_heads,
                      num_partials);
        return -2;
    }
    const long long rows = (long long)num_partials * kv_heads * ROWS;
    const long long need = rows * (head_dim + 2);
    if (need > DE_ATTN_STATIC_SCRATCH_FLOATS) {
        std::snprintf(g_static_error, sizeof(g_static_error),
                      "de_attn_simt_static_scratch: %d partial results x %d kv heads x %d rows x "
                      "(head_dim %d + 2) = %lld floats, the built-in scratch array holds %d; use "
                      "de_attn_simt with scratch of your own, or fewer chunks",
                      num_partials, kv_heads, ROWS, head_dim, need, DE_ATTN_STATIC_SCRATCH_FLOATS);
        return DE_ATTN_STATIC_TOO_LARGE;
    }
    float* scratch = nullptr;
    const int status = static_scratch_address(&scratch);
    if (status != 0) {
        std::snprintf(g_static_error, sizeof(g_static_error),
                      "de_attn_simt_static_scratch: the scratch array's device address could not "
                      "be looked up (code %d)", status);
        return status;
    }
    float* partial_acc = scratch;                               // [rows][head_dim]
    float* partial_ml = scratch + rows * head_dim;              // [rows][2]
    // the kernels are told how many partial slots the array holds for this call: an item that
    // names a slot at or beyond num_partials writes and merges nothing
    int code = launch_simt(dtype, q, q_stride, out, out_stride, k_pages, v_pages, block_table,
                           table_stride, num_pages, seq_slot, seq_qstart, seq_qlen, seq_pos0,
                           items, num_items, partial_acc, partial_ml, num_partials, heads,
                           kv_heads, head_dim, page, scale, window, nullptr, stream);
    if (code != 0) return code;
    return launch_combine(dtype, out, out_stride, seq_qstart, seq_qlen, combine_items,
                          num_combine, partial_acc, partial_ml, num_partials, heads, kv_heads,
                          head_dim, ROWS, stream);
}
