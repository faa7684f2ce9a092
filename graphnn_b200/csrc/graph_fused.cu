// The structure2vec classifier of a batch of small and medium graphs in ONE kernel: input projection, all levels,
// pooling and (for small batches) the readout, with the node embeddings in shared memory from the first level to the
// pooled sum.
//
//     H0   = ReLU(X)                               X = W_in[tag] (one-hot tags) or a dense projection made beforehand
//     Hl+1 = ReLU((A * Hl) * W + X),  l = 0..L-1   Y[g] = sum (or mean) of HL over the nodes of graph g
//     logits = ReLU(Y * W1) * W2, softmax, argmax
//
// (examples/graph_classification/src/kernel_mean_field.cpp:31-47 of the reference.)  A batch of graphs is block
// diagonal, so a CTA that owns whole graphs never needs a row of another CTA: HBM sees the CSR, the tags and the
// results, and the neighbour sums read shared memory at 128 bytes per clock instead of L2.
//
// Bounded by the shared-memory reads of the gather (63 % of that pipe) and instruction issue (47 %); HBM and tensor pipe are
// idle most of the time.  Measured against one launch per level and the older kernel for d = 128: 64 small graphs, d = 64,
// 56 -> 16 us; 700 molecules, d = 128, 82 -> 44; 4,093 220 -> 142; 16,384 645 -> 437; 4,096 proteins, d = 64, 1856 -> 1345.
//
// Work split.  Every CTA owns a contiguous range of graphs that starts at an equal share of the nodes (found by a
// search in graph_ptr, no planning launch) and walks it in tiles of whole graphs of at most `cap` nodes.  A tile is up
// to cap/128 row blocks of 128 nodes.  Per level and row block:
//   gather  : d/4 lanes own one node row; they add the neighbour rows in CSR order (fp32), scale the sum by a power of
//             two taken from its own largest element, split it into an fp16 head and tail and store both as the
//             K-major MMA operand.  The scale is per row, so a graph's results do not depend on its neighbours in the tile.
//   product : one warp issues tcgen05.mma, A = the 128 rows, B = W^T (head and tail, scaled by its largest element):
//             tail*head, head*tail, head*head into one fp32 accumulator in tensor memory.  W and the sums are scaled by
//             powers of two (GfScales, and a scale per row of sums); fp16 head + tail then carry 22 bits of every element
//             within 2^-17 of its row's largest one and 2^-39 of that largest one below it: the TF32 head + tail pair
//             carries the same 22 bits, at twice the operand bytes and half the MMA rate.
//   drain   : once every row block of the level is multiplied (tensor memory holds the whole new H, so no second copy
//             in shared memory is needed): accumulator * 2^-k + X, ReLU, back into the H rows.
// d = 128 takes the product transposed, W^T (A operand, in tensor memory) times the row block's sums, in row blocks of 64: an
// accumulator lane is then a column, so H rows are read and written straight, and two CTAs share an SM.
// d <= 64: H rows are stored in 16-byte pieces XOR-swizzled by the row's low three bits: a row is read by its lanes, and
// written by lanes that own 32 different rows, without bank conflicts.
//
// Every wait is bounded and nobody leaves the sequence of barriers: after a time-out (recorded in the status word) the
// remaining waits return at once and the kernel runs to its end.
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "tcgen05.cuh"

namespace
{

struct GfParams {
    int64_t G;
    const int32_t* row_ptr;
    const int32_t* col_idx;
    const float* val;
    const int32_t* graph_ptr;
    const int32_t* tags;      // NULL: dense input, X rows at `x`
    const float* x;           // tags: W_in [num_tags x d]; dense: msg [N x d]
    int num_tags;
    const float* W;
    const void* w_image;      // W^T as scaled fp16 head / tail in the operand layout (gf_weight_image_kernel), or NULL
    const float* P;           // ReLU(W_in) * W, or NULL (the first level goes through the MMAs)
    int levels;               // MMA levels
    int pool_average;
    float* Y;                 // [G x d], or NULL when the readout runs here
    float* embed_out;
    const float* W1;          // readout in this kernel when logits != NULL
    const float* W2;
    int hidden, num_class;
    float* logits;
    float* probs;
    int32_t* pred;
    int cap, chunk_cap;
    uint32_t tm_cols;
    s2v_device_status* status;
    s2v_device_status* edge_status;   // where an edge that leaves its tile is reported
};

template <int D>
struct GfCfg {
    // d = 128: the product is taken transposed, (H_new)^T = W^T * S^T, with W^T as the A operand in tensor memory and row blocks
    // of 64: operand buffer and H rows of a 128-node tile then take 96 KB, and two CTAs fit an SM -- one gathers while the
    // other multiplies and drains.  (With W in shared memory, one tile per SM: 16 warps in lock step, 0.70 ms on 16,384 molecules.)
    static constexpr bool TR = D == 128;
    static constexpr int RB = TR ? 64 : 128;              // rows per row block
    static constexpr int MAXG = TR ? 56 : 64;             // graphs per tile
    static constexpr uint32_t CHUNK = TR ? 16 : 8;        // bytes of a chunk of four columns
    static constexpr int LPR = D / 4;                     // lanes (and 16-byte pieces) per row
    static constexpr uint32_t ROWB = D * 4;
    static constexpr uint32_t S_BYTES = RB * D * 4;       // fp16 head + tail of a row block
    static constexpr uint32_t W_BYTES = D * D * 4;
    static constexpr uint32_t OFF_S = 0, OFF_W = S_BYTES, OFF_H = S_BYTES + (TR ? 0u : W_BYTES);
    static constexpr uint32_t TM_WLO = 64, TM_ACC = 128;  // TR: tensor memory columns (W^T head at 0)
    static constexpr uint32_t PART_OFF = MAXG * ROWB < S_BYTES / 2 ? S_BYTES / 2 : MAXG * ROWB;   // pooling: partial sums behind the pooled rows
    // K chunks of 64 fp16 (one 128-byte swizzle row); d = 32 keeps head and tail side by side in one chunk
    static constexpr uint32_t S_LO = D == 32 ? 64 : S_BYTES / 2, W_LO = D == 32 ? 64 : W_BYTES / 2;
    static constexpr int SHIFT = D == 128 ? 5 : (D == 64 ? 4 : 3);
    static constexpr uint32_t IDESC = (1u << 4) | ((uint32_t)((TR ? RB : D) >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);   // f32 <- f16 x f16, M = 128, N = D (TR: RB)
};

__host__ __device__ constexpr uint32_t gf_up(uint32_t v, uint32_t a) { return (v + a - 1) / a * a; }

// Byte offsets behind the H rows (one row more than cap: a row of zeros, what an unused gather slot adds).
struct GfMap {
    uint32_t info, roww, tags, goff, rs, bar, ws, col, total;
};
template <int D>
__host__ __device__ inline GfMap gf_map(int cap, int chunk_cap, bool has_val)
{
    GfMap m;
    m.info = GfCfg<D>::OFF_H + (uint32_t)(cap + 1) * GfCfg<D>::ROWB;   // per row: first chunk of columns | entries << 16
    m.roww = m.info + 4u * (uint32_t)cap;                              // per row: its edge weight
    m.tags = m.roww + (has_val ? 4u * (uint32_t)cap : 0u);
    m.goff = m.tags + gf_up((GfCfg<D>::TR ? 4u : 2u) * (uint32_t)(cap + 1), 16);   // TR: byte offsets of the rows' X, else tags
    m.rs = m.goff + gf_up(4u * (GfCfg<D>::MAXG + 1), 16);              // per row: exponent of its operand scale (TR: what its products are multiplied by)
    m.bar = m.rs + (GfCfg<D>::TR ? 4u : 1u) * (uint32_t)cap;
    m.ws = m.bar + 160;                                                // what W was scaled by: GfScales
    m.col = m.ws + 8u * D + 16u;                                            // chunks of four local columns: 16-bit indices into H (TR: byte offsets)
    m.total = m.col + gf_up(GfCfg<D>::CHUNK * (uint32_t)chunk_cap, 16) + 1024;   // + slack to align the base to 1024 bytes
    return m;
}

// element (row n, k) of a K-major fp16 operand of `rows` rows: chunk k/64, 128-byte row, 16-byte pieces XOR-swizzled
__device__ __forceinline__ uint32_t gf_op_off(int n, int k, int rows)
{
    return (uint32_t)(k >> 6) * (uint32_t)(rows * 128) + (uint32_t)n * 128u + (uint32_t)((((k & 63) >> 3) ^ (n & 7)) * 16 + (k & 7) * 2);
}
// the tail of the same element: LO bytes behind, or (d = 32) in pieces 4..7 of the same 128-byte row
template <int D>
__device__ __forceinline__ uint32_t gf_op_off_lo(int n, int k, int rows, uint32_t lo)
{
    return D == 32 ? gf_op_off(n, k + 32, rows) : lo + gf_op_off(n, k, rows);
}

// 16-byte piece `piece` of row r of H: swizzled where a warp's lanes read or write the same piece of many rows (not at d = 128,
// where every access is a row's consecutive bytes)
template <int D>
__device__ __forceinline__ uint32_t gf_h(int r, int piece)
{
    return D == 128 ? (uint32_t)(r * 32 + piece) : (uint32_t)(((r << GfCfg<D>::SHIFT) + (r & 7)) ^ piece);
}
__device__ __forceinline__ ulonglong2 gf_lds(uint32_t addr)   // 16 bytes of shared memory
{
    ulonglong2 v;
    asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "r"(addr));
    return v;
}

// Power-of-two scale that brings a largest magnitude into [2^14, 2^15), from its exponent (clamped so that the scale and its
// inverse stay normal numbers), and the inverse.  _field: the exponent in its place in the bits.
__device__ __forceinline__ uint32_t gf_exponent_field(uint32_t max_bits) { return max(max_bits, 15u << 23) & 0x7f800000u; }
__device__ __forceinline__ float gf_scale_field(uint32_t e) { return __uint_as_float((268u << 23) - e); }
__device__ __forceinline__ float gf_unscale_field(uint32_t e) { return __uint_as_float(e - (14u << 23)); }
__device__ __forceinline__ float gf_unscale(uint32_t e) { return __uint_as_float((e - 14u) << 23); }

__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t pack2(float x, float y)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
// v < 0 ? 0 : v for values that are only added afterwards (NaN stays NaN; -0 becomes +0)
__device__ __forceinline__ float relu_max(float v)
{
    float r;
    asm("max.NaN.f32 %0, %1, 0f00000000;" : "=f"(r) : "f"(v));
    return r;
}
// two scaled values -> packed fp16 heads and tails (head rounded to nearest, tail = exact remainder rounded to nearest)
__device__ __forceinline__ void split_f16(uint64_t v, uint32_t& hi, uint32_t& lo)
{
    const float2 f = unpack2(v);
    const __half2 h = __floats2half2_rn(f.x, f.y);
    const float2 hf = __half22float2(h);
    const __half2 l = __floats2half2_rn(f.x - hf.x, f.y - hf.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}
__device__ __forceinline__ void mma_f16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        :
        : "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// A (two packed fp16 per column) in tensor memory
__device__ __forceinline__ void mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        :
        : "r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tc_ld_cols8(uint32_t addr, uint32_t* v)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(addr)
                 : "memory");
}

// first graph whose first node is at or behind `target` (graph_ptr ascending), found by one warp 32 probes at a time
__device__ __forceinline__ int64_t gf_lower_graph(const int32_t* graph_ptr, int64_t G, int64_t target)
{
    const int lane = threadIdx.x & 31;
    int64_t lo = 0, hi = G;   // answer in [lo, hi]
    while (hi > lo) {
        const int64_t step = (hi - lo + 31) / 32;
        const int64_t at = lo + step * lane;
        const bool below = at < hi && (int64_t)__ldg(graph_ptr + at) < target;
        const int n = __popc(__ballot_sync(0xffffffffu, below));
        if (n == 0) return lo;
        lo = lo + step * (n - 1) + 1;
        hi = lo + step - 1 < hi ? lo + step - 1 : hi;
    }
    return lo;
}

// Scales of W, powers of two.  Where all its rows and columns are of about one size, one for all of it, which the scale of a row of
// sums takes in.  Otherwise one on either side, W'[k][n] = W[k][n] / in[k] / out[n], so that the largest element of every column and
// (nearly) of every row of W' is 2^14 .. 2^15; the sums are then multiplied by in[k] before they are split and the products by out[n],
// and a result does not depend on the units its features are held in: with one scale, an output feature whose weights are 2^-24 of the
// largest has lost half of its 22 bits.  (A column below 2^-64 of its rows is not scaled up all the way.)  Of one size: no row or column
// (or the part of it that a warp or a thread holds) whose largest element is more than 2^EVEN below the largest of all; what is
// lost is then 2^-31 at most.  An infinite weight calls for two scales, to which infinities and NaN don't count.
// One scale without a look at the rows and columns: 335 us on 16,384 molecules (d = 128), 16.3 on 64 small graphs (d = 64); two always:
// 341 and 17.8; as it is: 338 and 16.8.
template <int D>
struct GfScales {
    float out[D];
    float in[D];
    float all;              // one scale: what the products are multiplied by (1 with scales on both sides)
    uint32_t uneven;        // scales on both sides
    uint32_t pad[2];
};
static_assert(sizeof(GfScales<64>) == 8 * 64 + 16, "its place in GfMap");
template <int D>
struct GfScaleWork {        // while W is converted (in the operand buffer's place)
    float down[D];          // 1 / in
    uint32_t row_max[D], col_max[D];
    uint32_t most, least;   // largest element; smallest of the rows' and columns' largest ones
    static constexpr uint32_t EVEN = 8;
    __device__ __forceinline__ void clear()
    {
        if (threadIdx.x < D) row_max[threadIdx.x] = col_max[threadIdx.x] = 0u;
        if (threadIdx.x == 0) { most = 0u; least = ~0u; }
    }
    // col: bits of the largest of the thread's elements, all of one column; row: the smallest of the rows' largest ones, as far as the warp sees them
    __device__ __forceinline__ void add(uint32_t col, uint32_t row)
    {
        const uint32_t w = __reduce_max_sync(0xffffffffu, col), l = min(row, __reduce_min_sync(0xffffffffu, col));
        if ((threadIdx.x & 31) == 0) {
            atomicMax(&most, w);
            atomicMin(&least, l);
        }
    }
    // behind a barrier: whether one scale will do (its exponent stays clear of the ends of the range)
    __device__ __forceinline__ bool even() const { return (least >> 23) + EVEN >= (most >> 23) && (most >> 23) >= 87u && (most >> 23) <= 167u; }
    __device__ __forceinline__ float all_up() const { return pow2(268u - (most >> 23)); }
    __device__ __forceinline__ float all_out() const { return pow2((most >> 23) - 14u); }
    __device__ __forceinline__ static uint32_t finite_bits(float v)
    {
        const uint32_t b = __float_as_uint(fabsf(v));
        return b < 0x7f800000u ? b : 0u;
    }
    __device__ __forceinline__ static float pow2(uint32_t biased) { return __uint_as_float(biased << 23); }
    // behind the rows' maxima, between two barriers (exponents that keep both scales normal numbers)
    __device__ __forceinline__ void finish_rows(GfScales<D>* s)
    {
        if (threadIdx.x >= D) return;
        const uint32_t e = min(max(row_max[threadIdx.x] >> 23, 15u), 253u);
        s->in[threadIdx.x] = pow2(e);
        down[threadIdx.x] = pow2(254u - e);
    }
    // behind a barrier after the columns' maxima: what brings a column's largest element to 2^14 .. 2^15
    __device__ __forceinline__ uint32_t col_exponent(int n) const { return max(col_max[n] >> 23, 63u); }
    __device__ __forceinline__ float col_up(int n) const { return pow2(268u - col_exponent(n)); }
    __device__ __forceinline__ void finish_cols(GfScales<D>* s) const
    {
        if (threadIdx.x < D) s->out[threadIdx.x] = pow2(col_exponent(threadIdx.x) - 14u);
    }
};

// W^T as the B operand: scaled fp16 head and tail.  Thread t converts pairs of consecutive k of one column n.
// `work` is cleared beforehand; contains barriers, so every thread of the CTA calls it.
template <int D, int THREADS>
__device__ __forceinline__ bool gf_convert_w(const float* __restrict__ W, unsigned char* dst, GfScales<D>* scales, GfScaleWork<D>* work, float& all)
{
    constexpr int PAIRS = D * D / 2, PER = (PAIRS + THREADS - 1) / THREADS;
    static_assert(THREADS % D == 0, "a thread stays in one column, a warp in one row");
    const int n = threadIdx.x % D;
    float a[PER][2];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int p = threadIdx.x + i * THREADS, k = p / D * 2;
        a[i][0] = p < PAIRS ? __ldg(W + k * D + n) : 0.f;
        a[i][1] = p < PAIRS ? __ldg(W + (k + 1) * D + n) : 0.f;
    }
    {
        float col = 0.f;
        uint32_t row = ~0u;
#pragma unroll
        for (int i = 0; i < PER; ++i) col = fmaxf(col, fmaxf(fabsf(a[i][0]), fabsf(a[i][1])));
        auto look = [&](auto first) {   // D / 32 warps hold a row; each looks at its share of the rows
#pragma unroll
            for (int i = decltype(first)::value; i < PER; i += D / 32)
#pragma unroll
                for (int h = 0; h < 2; ++h) row = min(row, __reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(a[i][h]))));
        };
        if (D == 32 || ((threadIdx.x >> 5) & 1) == 0) look(std::integral_constant<int, 0>{});
        else look(std::integral_constant<int, 1>{});
        if (threadIdx.x < PAIRS) work->add(__float_as_uint(col), row);   // (whole warps)
    }
    __syncthreads();
    float up = work->all_up();
    const bool even = work->even();
    all = even ? work->all_out() : 1.f;
    if (!even) {
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int p = threadIdx.x + i * THREADS, k = p / D * 2;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t w = __reduce_max_sync(0xffffffffu, work->finite_bits(a[i][h]));
                if (p < PAIRS && (threadIdx.x & 31) == 0) atomicMax(work->row_max + k + h, w);
            }
        }
        __syncthreads();
        work->finish_rows(scales);
        __syncthreads();
        uint32_t m = 0;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int p = threadIdx.x + i * THREADS, k = p / D * 2;
            if (p < PAIRS) {
                const float2 down = *reinterpret_cast<const float2*>(work->down + k);
                a[i][0] *= down.x;
                a[i][1] *= down.y;
                m = max(m, max(work->finite_bits(a[i][0]), work->finite_bits(a[i][1])));
            }
        }
        atomicMax(work->col_max + n, m);
        __syncthreads();
        work->finish_cols(scales);
        up = work->col_up(n);
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int p = threadIdx.x + i * THREADS, k = p / D * 2;
        if (p < PAIRS) {
            uint32_t hi, lo;
            split_f16(pack2(a[i][0] * up, a[i][1] * up), hi, lo);
            *reinterpret_cast<uint32_t*>(dst + gf_op_off(n, k, D)) = hi;
            *reinterpret_cast<uint32_t*>(dst + gf_op_off_lo<D>(n, k, D, GfCfg<D>::W_LO)) = lo;
        }
    }
    return !even;
}

// d = 128: W^T as the A operand in tensor memory: lane m = output feature, column c = the pair of input features 2c, 2c + 1.
// Each thread holds 64 input features of one output feature: warp w of eight has lanes 32 (w % 4) .. and the half w / 4.
__device__ __forceinline__ void gf_store_w_pairs(uint32_t tmem, const uint32_t (&hi)[32], const uint32_t (&lo)[32])
{
    const int warp = threadIdx.x >> 5;
    const uint32_t at = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(32 * (warp >> 2));
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        tc_st_cols8(at + 8 * h, hi + 8 * h);
        tc_st_cols8(at + GfCfg<128>::TM_WLO + 8 * h, lo + 8 * h);
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// image: word (c, m) at c * 128 + m, heads first, tails behind them
__device__ __forceinline__ void gf_load_w_t(const void* image, uint32_t tmem)
{
    const int warp = threadIdx.x >> 5, m = 32 * (warp & 3) + (threadIdx.x & 31);
    const uint32_t* w = static_cast<const uint32_t*>(image) + (32 * (warp >> 2)) * 128 + m;
    uint32_t hi[32], lo[32];
#pragma unroll
    for (int c = 0; c < 32; ++c) { hi[c] = __ldg(w + c * 128); lo[c] = __ldg(w + 64 * 128 + c * 128); }
    gf_store_w_pairs(tmem, hi, lo);
}
__device__ __forceinline__ bool gf_convert_w_t(const float* __restrict__ W, uint32_t tmem, GfScales<128>* scales, GfScaleWork<128>* work, float& all)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, m = 32 * (warp & 3) + lane, k0 = 64 * (warp >> 2);
    float a[64];
#pragma unroll
    for (int k = 0; k < 64; ++k) a[k] = __ldg(W + (k0 + k) * 128 + m);
    {
        float col = 0.f;
        uint32_t row = ~0u;
#pragma unroll
        for (int k = 0; k < 64; ++k) col = fmaxf(col, fabsf(a[k]));
        auto look = [&](auto first) {   // four warps hold a row; each looks at a quarter of the rows
#pragma unroll
            for (int k = decltype(first)::value; k < 64; k += 4) row = min(row, __reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(a[k]))));
        };
        switch (warp & 3) {
            case 0: look(std::integral_constant<int, 0>{}); break;
            case 1: look(std::integral_constant<int, 1>{}); break;
            case 2: look(std::integral_constant<int, 2>{}); break;
            default: look(std::integral_constant<int, 3>{});
        }
        work->add(__float_as_uint(col), row);
    }
    __syncthreads();
    float up = work->all_up();
    const bool even = work->even();
    all = even ? work->all_out() : 1.f;
    if (!even) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            uint32_t mine = 0;
#pragma unroll
            for (int k = 0; k < 32; ++k) {
                const uint32_t w = __reduce_max_sync(0xffffffffu, work->finite_bits(a[32 * h + k]));
                if (lane == k) mine = w;
            }
            atomicMax(work->row_max + k0 + 32 * h + lane, mine);
        }
        __syncthreads();
        work->finish_rows(scales);
        __syncthreads();
        uint32_t mx = 0;
#pragma unroll
        for (int k = 0; k < 64; k += 4) {
            const float4 down = *reinterpret_cast<const float4*>(work->down + k0 + k);
            a[k] *= down.x; a[k + 1] *= down.y; a[k + 2] *= down.z; a[k + 3] *= down.w;
#pragma unroll
            for (int u = 0; u < 4; ++u) mx = max(mx, work->finite_bits(a[k + u]));
        }
        atomicMax(work->col_max + m, mx);
        __syncthreads();
        work->finish_cols(scales);
        up = work->col_up(m);
    }
    uint32_t hi[32], lo[32];
#pragma unroll
    for (int c = 0; c < 32; ++c) split_f16(pack2(a[2 * c] * up, a[2 * c + 1] * up), hi[c], lo[c]);
    gf_store_w_pairs(tmem, hi, lo);
    return !even;
}

// The same into global memory, once per batch: [operand image | scales].
template <int D>
__global__ void __launch_bounds__(1024) gf_weight_image_kernel(const float* __restrict__ W, unsigned char* __restrict__ image)
{
    __shared__ __align__(16) GfScales<D> scales;
    __shared__ __align__(16) GfScaleWork<D> work;
    work.clear();
    __syncthreads();
    float all;
    bool uneven;
    if constexpr (D == 128) {
        uint32_t* const words = reinterpret_cast<uint32_t*>(image);
        const int m = threadIdx.x % 128;
        float a[8][2];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int c = threadIdx.x / 128 + 8 * i;
            a[i][0] = __ldg(W + (2 * c) * 128 + m);
            a[i][1] = __ldg(W + (2 * c + 1) * 128 + m);
        }
        float col = 0.f;
        uint32_t row = ~0u;
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                col = fmaxf(col, fabsf(a[i][h]));
                row = min(row, __reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(a[i][h]))));
            }
        work.add(__float_as_uint(col), row);
        __syncthreads();
        float up = work.all_up();
        const bool even = work.even();
        all = even ? work.all_out() : 1.f;
        uneven = !even;
        if (!even) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t w = __reduce_max_sync(0xffffffffu, work.finite_bits(a[i][h]));
                    if ((threadIdx.x & 31) == 0) atomicMax(work.row_max + 2 * (threadIdx.x / 128 + 8 * i) + h, w);
                }
            __syncthreads();
            work.finish_rows(&scales);
            __syncthreads();
            uint32_t mx = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float2 down = *reinterpret_cast<const float2*>(work.down + 2 * (threadIdx.x / 128 + 8 * i));
                a[i][0] *= down.x;
                a[i][1] *= down.y;
                mx = max(mx, max(work.finite_bits(a[i][0]), work.finite_bits(a[i][1])));
            }
            atomicMax(work.col_max + m, mx);
            __syncthreads();
            work.finish_cols(&scales);
            up = work.col_up(m);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int e = threadIdx.x + i * 1024;
            uint32_t hi, lo;
            split_f16(pack2(a[i][0] * up, a[i][1] * up), hi, lo);
            words[e] = hi;
            words[64 * 128 + e] = lo;
        }
    } else {
        uneven = gf_convert_w<D, 1024>(W, image, &scales, &work, all);
    }
    if (threadIdx.x == 0) {
        scales.all = all;
        scales.uneven = uneven ? 1u : 0u;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < (int)(sizeof(scales) / 4); e += 1024) reinterpret_cast<float*>(image + GfCfg<D>::W_BYTES)[e] = reinterpret_cast<const float*>(&scales)[e];
}

template <int WT>
__device__ __forceinline__ void gf_worker_sync()
{
    asm volatile("bar.sync 1, %0;" ::"n"(WT) : "memory");
}

// readout of NB graphs whose pooled rows lie in shared memory: layer 1 split over threads as (hidden unit, slice of k)
template <int D, int WT, int NB>
__device__ __forceinline__ void gf_readout(const GfParams& p, const float* y_s, float* scratch, int nb, int64_t g_first)
{
    const int tid = threadIdx.x, hidden = p.hidden, C = p.num_class;
    int slices = WT / hidden;
    slices = slices >= 8 ? 8 : (slices >= 4 ? 4 : (slices >= 2 ? 2 : 1));
    float* part = scratch;                                            // [slices][NB][hidden]
    float* hid = scratch + (slices > 1 ? slices * NB * hidden : 0);   // [NB][hidden]
    float* out_s = hid + NB * hidden;                                 // [NB][C]
    const int items = hidden * slices, kper = D / slices;
    for (int it = tid; it < items; it += WT) {
        const int h = it % hidden, sl = it / hidden;
        float acc[NB];
#pragma unroll
        for (int g = 0; g < NB; ++g) acc[g] = 0.f;
        const float* w = p.W1 + (int64_t)(sl * kper) * hidden + h;
        const float* y = y_s + sl * kper;
        constexpr int U = NB <= 4 ? 32 : 16;   // loads of W1 in flight
        for (int k = 0; k < kper; k += U) {
            float wv[U];
#pragma unroll
            for (int u = 0; u < U; ++u) wv[u] = k + u < kper ? __ldg(w + (int64_t)(k + u) * hidden) : 0.f;
#pragma unroll
            for (int u = 0; u < U; u += 4) {
                if (k + u >= kper) break;   // (kper is a multiple of four)
#pragma unroll
                for (int g = 0; g < NB; ++g) {
                    const float4 yv = *reinterpret_cast<const float4*>(y + g * D + k + u);
                    acc[g] = fmaf(yv.x, wv[u], acc[g]);
                    acc[g] = fmaf(yv.y, wv[u + 1], acc[g]);
                    acc[g] = fmaf(yv.z, wv[u + 2], acc[g]);
                    acc[g] = fmaf(yv.w, wv[u + 3], acc[g]);
                }
            }
        }
#pragma unroll
        for (int g = 0; g < NB; ++g) {
            if (slices > 1) part[(sl * NB + g) * hidden + h] = acc[g];
            else hid[g * hidden + h] = relu_ref(acc[g]);
        }
    }
    gf_worker_sync<WT>();
    if (slices > 1) {
        for (int e = tid; e < NB * hidden; e += WT) {
            float s = part[e];
            for (int sl = 1; sl < slices; ++sl) s += part[sl * NB * hidden + e];
            hid[e] = relu_ref(s);
        }
        gf_worker_sync<WT>();
    }
    const int warp = tid >> 5, lane = tid & 31;
    for (int gc = warp; gc < nb * C; gc += WT / 32) {   // one warp per (graph, class)
        const int g = gc / C, c = gc - g * C;
        float acc = 0.f;
        for (int h = lane; h < hidden; h += 32) acc = fmaf(hid[g * hidden + h], __ldg(p.W2 + (int64_t)h * C + c), acc);
#pragma unroll
        for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) out_s[gc] = acc;
    }
    gf_worker_sync<WT>();
    for (int g = tid; g < nb; g += WT) {
        const float* l = out_s + g * C;
        float mx = l[0];
        int best = 0;
        for (int c = 1; c < C; ++c)
            if (l[c] > mx) { mx = l[c]; best = c; }
        float s = 0.f;
        for (int c = 0; c < C; ++c) s += expf(l[c] - mx);
        for (int c = 0; c < C; ++c) {
            p.logits[(g_first + g) * C + c] = l[c];
            if (p.probs) p.probs[(g_first + g) * C + c] = expf(l[c] - mx) / s;
        }
        if (p.pred) p.pred[g_first + g] = best;
    }
}

// Neighbour sums with the columns (and weights) straight from global memory: tiles whose columns do not fit the chunk list, and tiles
// with a row whose edges carry different weights.  A row's lanes load its indices side by side, one each, the next ones on their way
// while these are summed, and hand them round by shuffles: five instructions per neighbour and lane where the list takes four.
// FIRST: sum of rows of P.  (Four broadcast loads, then four rows, one row at a time: 454 us instead of 270 on 1,000 graphs of 90 nodes
// with 50 neighbours each, 122 instead of 106 on 250 proteins with unequal weights; one launch per level 270 and 97; d = 64.)
struct GfFar {
    uint32_t rows, xo;         // shared memory: H, X offset (d = 128) or tag of each row
    const ulonglong2* P;
    int node0, nrows, cap;
    s2v_device_status* status;
};
// all lanes of a warp; col, val, n: the lane group's row (n = 0: none); c, w: its entry number sl, where it has one
template <int D, bool HAS_VAL, bool FIRST>
__device__ __noinline__ ulonglong2 gf_row_from_global(const GfFar f, const int32_t* col, const float* val, int n, int c, float w)
{
    using Cfg = GfCfg<D>;
    constexpr int LPR = Cfg::LPR;
    const int sl = threadIdx.x % LPR;
    const int most = __reduce_max_sync(0xffffffffu, n);
    ulonglong2 acc = make_ulonglong2(0ull, 0ull);
    for (int t = 0; t < most; t += LPR) {
        const int tn = t + LPR + sl;
        const int cn = tn < n ? __ldg(col + tn) : 0;
        const float wn = HAS_VAL && tn < n ? __ldg(val + tn) : 0.f;
        uint32_t e = (uint32_t)f.cap;   // past the end: the row of zeros
        if (t + sl < n) {
            e = (uint32_t)(c - f.node0);
            if (e >= (uint32_t)f.nrows) {
                f.status->code = S2V_ERR_BAD_CSR;
                f.status->where = 5;
                e = 0;
            }
        }
        if (FIRST) {
            if (Cfg::TR) {
                asm volatile("ld.shared.u32 %0, [%1];" : "=r"(e) : "r"(f.xo + 4 * e));
                e >>= 4;
            } else {
                uint16_t tag;
                asm volatile("ld.shared.u16 %0, [%1];" : "=h"(tag) : "r"(f.xo + 2 * e));
                e = (uint32_t)tag * LPR;
            }
        } else e = Cfg::TR ? e * LPR : (e << Cfg::SHIFT) + (e & 7u);
#pragma unroll
        for (int u0 = 0; u0 < LPR; u0 += 4) {
            if (t + u0 >= most) break;
            ulonglong2 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t eu = __shfl_sync(0xffffffffu, e, u0 + u, LPR);
                if (FIRST) v[u] = __ldg(f.P + eu + sl);
                else v[u] = gf_lds(f.rows + 16u * (Cfg::TR ? eu + sl : eu ^ (uint32_t)sl));
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (HAS_VAL) {
                    const float wu = __shfl_sync(0xffffffffu, w, u0 + u, LPR);
                    const uint64_t ww = pack2(wu, wu);
                    acc.x = fma2(ww, v[u].x, acc.x);
                    acc.y = fma2(ww, v[u].y, acc.y);
                } else {
                    acc.x = add2(acc.x, v[u].x);
                    acc.y = add2(acc.y, v[u].y);
                }
            }
        }
        c = cn;
        w = wn;
    }
    return acc;
}

// One row's sum with a weight per entry, columns and weights from the lists in shared memory (16,384 molecules with unequal weights:
// d = 128 577 us from global memory, 466 from the lists, 469 with one launch per level; d = 64 372, 324, 328).  chunk, weights: the row's first ones;
// most: chunks of the warp's longest row (a row with fewer, mine, adds nothing there).
template <int D, bool FIRST>
__device__ __noinline__ ulonglong2 gf_row_weighted(const GfFar f, uint32_t chunk, uint32_t weights, uint32_t mine, uint32_t most)
{
    using Cfg = GfCfg<D>;
    constexpr int LPR = Cfg::LPR;
    const uint32_t sl = threadIdx.x % LPR;
    ulonglong2 acc = make_ulonglong2(0ull, 0ull);
    for (uint32_t c = 0; c < most; ++c) {
        if (c >= mine) continue;
        uint32_t e[4];
        if (Cfg::TR) {
            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(e[0]), "=r"(e[1]), "=r"(e[2]), "=r"(e[3]) : "r"(chunk + 16 * c));
        } else {
            uint32_t lo, hi;
            asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(lo), "=r"(hi) : "r"(chunk + 8 * c));
            e[0] = lo & 0xffffu; e[1] = lo >> 16; e[2] = hi & 0xffffu; e[3] = hi >> 16;
        }
        const ulonglong2 w2 = gf_lds(weights + 16 * c);
        const float2 w01 = unpack2(w2.x), w23 = unpack2(w2.y);
        const float w[4] = {w01.x, w01.y, w23.x, w23.y};
        ulonglong2 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (FIRST) {
                uint32_t x;
                if (Cfg::TR) {
                    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(x) : "r"(f.xo + ((e[u] - Cfg::OFF_H) >> 7)));
                    x >>= 4;
                } else {
                    uint16_t tag;
                    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(tag) : "r"(f.xo + 2 * (e[u] >> Cfg::SHIFT)));
                    x = (uint32_t)tag * LPR;
                }
                v[u] = __ldg(f.P + x + sl);
            } else {
                v[u] = gf_lds(Cfg::TR ? f.rows - Cfg::OFF_H + e[u] + 16 * sl : f.rows + 16 * (e[u] ^ sl));
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint64_t ww = pack2(w[u], w[u]);
            acc.x = fma2(ww, v[u].x, acc.x);
            acc.y = fma2(ww, v[u].y, acc.y);
        }
    }
    return acc;
}

// READOUT: logits and predictions are made here, W converted and the first level multiplied (small batches).  Otherwise the pooled rows go
// out, and P and the image of W may have been made beforehand.  One kernel for both: 16,384 molecules 438 us and 700 of them 47 with eight loads
// of W1 at a time in the readout, 451 and 45.5 with sixteen (the registers of the main loops spill).
template <int D, int WARPS, bool HAS_VAL, bool READOUT>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 8 ? 2 : 1) s2v_graph_fused_kernel(const GfParams p)
{
    using Cfg = GfCfg<D>;
    constexpr int WT = WARPS * 32;
    constexpr int LPR = Cfg::LPR, GPW = 32 / LPR;   // lanes per row, row groups per warp
    constexpr int NG = WARPS * GPW;                 // row groups
    constexpr int RB = Cfg::RB, RPG = RB / NG;      // rows of a row block, per group
    constexpr int CW = D / (WARPS / 4);             // accumulator columns a warp drains (not TR)
    constexpr int LDC = CW >= 16 ? 16 : 8;          // columns per tcgen05.ld
    constexpr int ROUNDS = D == 128 || (D == 64 && WARPS == 8) ? 1 : (D == 32 && WARPS == 8 ? 3 : 2);   // rows per thread in the prologue

    extern __shared__ unsigned char gf_smem_raw[];
    unsigned char* smem = gf_smem_raw + ((1024u - (smem_u32(gf_smem_raw) & 1023u)) & 1023u);
    const GfMap map = gf_map<D>(p.cap, p.chunk_cap, HAS_VAL);
    uint32_t* const info_s = reinterpret_cast<uint32_t*>(smem + map.info);
    float* const roww = reinterpret_cast<float*>(smem + map.roww);
    uint16_t* const tag_s = reinterpret_cast<uint16_t*>(smem + map.tags);
    int* const goff = reinterpret_cast<int*>(smem + map.goff);
    uint8_t* const rs = smem + map.rs;
    float* const rsf = reinterpret_cast<float*>(smem + map.rs);
    uint32_t* const xo_s = reinterpret_cast<uint32_t*>(smem + map.tags);
    uint2* const chunks = reinterpret_cast<uint2*>(smem + map.col);
    uint4* const chunks_t = reinterpret_cast<uint4*>(smem + map.col);
    uint4* const p_chunks = reinterpret_cast<uint4*>(smem + Cfg::OFF_S);   // TR, first level: as long as `chunks_t`, which the launch keeps within S_BYTES
    float4* const H4 = reinterpret_cast<float4*>(smem + Cfg::OFF_H);
    const ulonglong2* const H2 = reinterpret_cast<const ulonglong2*>(smem + Cfg::OFF_H);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + map.bar);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + map.bar + 16);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + map.bar + 24);
    GfScales<D>* const scales = reinterpret_cast<GfScales<D>*>(smem + map.ws);
    GfScaleWork<D>* const scale_work = reinterpret_cast<GfScaleWork<D>*>(smem + Cfg::OFF_S);
    int* s_range = reinterpret_cast<int*>(smem + map.bar + 32);
    int* s_mixed = reinterpret_cast<int*>(smem + map.bar + 44);
    int* s_scan = reinterpret_cast<int*>(smem + map.bar + 64);   // WARPS totals
    const uint32_t bar_mma = smem_u32(bars), bar_full = bar_mma + 8;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nb_cta = gridDim.x;

    if (threadIdx.x == 0) {
        tc_mbar_init(bar_mma, 1);
        tc_mbar_init(bar_full, WARPS);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(p.tm_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // the CTA's graphs: one each when there are no more graphs than CTAs, else an equal share of the nodes
    if (warp == 1 || warp == 2) {
        int64_t g;
        const int64_t i = (int64_t)blockIdx.x + warp - 1;
        if (p.G <= nb_cta) g = i < p.G ? i : p.G;
        else g = i >= nb_cta ? p.G : (i == 0 ? 0 : gf_lower_graph(p.graph_ptr, p.G, (int64_t)__ldg(p.graph_ptr + p.G) * i / nb_cta));
        if (lane == 0) s_range[warp - 1] = (int)g;
    }
    if (threadIdx.x < LPR) H4[p.cap * LPR + threadIdx.x] = make_float4(0.f, 0.f, 0.f, 0.f);   // the row of zeros
    scale_work->clear();
    const uint32_t zero_entry = (uint32_t)p.cap << Cfg::SHIFT;
    if (threadIdx.x == 0) {
        // chunk 0: zero rows; P has a row of zeros behind the last tag
        if (Cfg::TR) {
            const uint32_t z = Cfg::OFF_H + (uint32_t)p.cap * Cfg::ROWB;
            chunks_t[0] = make_uint4(z, z, z, z);
            xo_s[p.cap] = (uint32_t)p.num_tags * Cfg::ROWB;
        } else {
            chunks[0] = make_uint2(zero_entry * 0x10001u, zero_entry * 0x10001u);
            tag_s[p.cap] = (uint16_t)p.num_tags;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    const int g_lo = s_range[0], g_hi = s_range[1];
    float inv_w;
    bool uneven;   // scales on both sides of W, in `scales`
    if (!READOUT && p.w_image) {
        const unsigned char* const image = static_cast<const unsigned char*>(p.w_image);
        if (Cfg::TR) gf_load_w_t(image, tmem_base);
        else
            for (int i = threadIdx.x; i < (int)(Cfg::W_BYTES / 16); i += WT)
                reinterpret_cast<uint4*>(smem + Cfg::OFF_W)[i] = __ldg(reinterpret_cast<const uint4*>(image) + i);
        if (threadIdx.x < sizeof(GfScales<D>) / 16)
            reinterpret_cast<float4*>(scales)[threadIdx.x] = __ldg(reinterpret_cast<const float4*>(image + Cfg::W_BYTES) + threadIdx.x);
        const GfScales<D>* const made = reinterpret_cast<const GfScales<D>*>(image + Cfg::W_BYTES);
        inv_w = __ldg(&made->all);
        uneven = __ldg(&made->uneven) != 0;
    } else {
        if constexpr (Cfg::TR) uneven = gf_convert_w_t(p.W, tmem_base, scales, scale_work, inv_w);
        else uneven = gf_convert_w<D, WT>(p.W, smem + Cfg::OFF_W, scales, scale_work, inv_w);
    }
    if (Cfg::TR) asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");

    uint32_t job = 0;      // row blocks multiplied so far (the same count in every warp)
    int bad_tag = 0;
    const int q = warp & 3, jc = warp >> 2;
    const int sub = lane / LPR, sl = lane % LPR;
    const int grp = warp * GPW + sub;
    const float4* __restrict__ X4 = reinterpret_cast<const float4*>(p.x);
    for (int g0 = g_lo; g0 < g_hi;) {
        // ---- the tile: whole graphs from g0 on, at most cap nodes and MAXG graphs (every warp works it out by itself)
        const int node0 = __ldg(p.graph_ptr + g0);
        int g1 = g0;
        while (g1 < g_hi && g1 - g0 < Cfg::MAXG) {
            const int gi = g1 + 1 + lane;
            const bool fits = gi <= g_hi && gi - g0 <= Cfg::MAXG && __ldg(p.graph_ptr + gi) - node0 <= p.cap;
            const unsigned bal = __ballot_sync(0xffffffffu, fits);
            const int n = bal == 0xffffffffu ? 32 : __ffs(~bal) - 1;
            g1 += n;
            if (n < 32) break;
        }
        if (g1 == g0) g1 = g0 + 1;
        int nrows = __ldg(p.graph_ptr + g1) - node0;
        if (nrows > p.cap) {   // a graph beyond the capacity: reported, truncated
            nrows = p.cap;
            p.status->code = S2V_ERR_UNSUPPORTED;
            p.status->where = 4;
        }
        if (nrows < 0) nrows = 0;
        const int ngr = g1 - g0;
        const int mt = (nrows + RB - 1) / RB;

        // ---- tile prologue: row structure, tags, graph offsets; then local columns in chunks of four, H0
        int rb[ROUNDS], rn[ROUNDS];
#pragma unroll
        for (int k = 0; k < ROUNDS; ++k) {
            const int r = k * WT + threadIdx.x;
            rb[k] = rn[k] = 0;
            if (r < nrows) {
                rb[k] = __ldg(p.row_ptr + node0 + r);
                rn[k] = __ldg(p.row_ptr + node0 + r + 1) - rb[k];
                if (rn[k] < 0) rn[k] = 0;
                if (p.tags) {
                    const int t = __ldg(p.tags + node0 + r);
                    bad_tag |= (unsigned)t >= (unsigned)p.num_tags ? 1 : 0;
                    const int ok = (unsigned)t >= (unsigned)p.num_tags ? 0 : t;
                    if (Cfg::TR) xo_s[r] = (uint32_t)ok * Cfg::ROWB;
                    else tag_s[r] = (uint16_t)ok;
                } else if (Cfg::TR) xo_s[r] = (uint32_t)r * Cfg::ROWB;
            }
        }
        if (Cfg::TR && threadIdx.x >= nrows && threadIdx.x < p.cap) xo_s[threadIdx.x] = 0;   // (looked up, never used)
        for (int k = threadIdx.x; k <= ngr; k += WT) {
            const int v = __ldg(p.graph_ptr + g0 + k) - node0;
            goff[k] = v < 0 ? 0 : (v > nrows ? nrows : v);
        }
        if (HAS_VAL && threadIdx.x == 0) *s_mixed = 0;
        if (!READOUT && Cfg::TR && p.P && threadIdx.x == 0) {
            const uint32_t z = (uint32_t)p.num_tags * Cfg::ROWB;
            p_chunks[0] = make_uint4(z, z, z, z);
        }
        int first[ROUNDS], carry = 1;   // chunk 0 is the chunk of zero rows
#pragma unroll
        for (int k = 0; k < ROUNDS; ++k) {
            const int c = (rn[k] + 3) >> 2;
            int incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            if (k > 0) gf_worker_sync<WT>();   // the totals of the previous round are read
            if (lane == 31) s_scan[warp] = incl;
            gf_worker_sync<WT>();
            int tot = lane < WARPS ? s_scan[lane] : 0;
            int before = lane < warp ? tot : 0;
            tot = __reduce_add_sync(0xffffffffu, tot);
            before = __reduce_add_sync(0xffffffffu, before);
            first[k] = carry + before + incl - c;
            carry += tot;
        }
        const bool cached = carry <= p.chunk_cap;   // uniform over the CTA
#pragma unroll
        for (int k = 0; k < ROUNDS; ++k) {
            const int r = k * WT + threadIdx.x;
            if (r < nrows) {
                const int c = (rn[k] + 3) >> 2;
                info_s[r] = c ? (uint32_t)first[k] | ((uint32_t)(rn[k] < 65535 ? rn[k] : 65535) << 16) : 0u;   // (a listed row is shorter)
                if (cached)
                    for (int t = 0; t < rn[k]; t += 4) {
                        uint32_t e[4], xe[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) e[u] = t + u < rn[k] ? (uint32_t)(__ldg(p.col_idx + rb[k] + t + u) - node0) : (uint32_t)p.cap;
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            if (e[u] >= (uint32_t)nrows && t + u < rn[k]) {   // an edge that leaves the tile
                                p.edge_status->code = S2V_ERR_BAD_CSR;
                                p.edge_status->where = 5;
                                e[u] = 0;
                            }
                            if (!READOUT && Cfg::TR) xe[u] = xo_s[e[u]];
                            e[u] = Cfg::TR ? Cfg::OFF_H + e[u] * Cfg::ROWB : (e[u] << Cfg::SHIFT) + (e[u] & 7u);
                        }
                        if (Cfg::TR) {
                            chunks_t[first[k] + (t >> 2)] = make_uint4(e[0], e[1], e[2], e[3]);
                            // the first level's list: offsets of the neighbours' table rows, in the operand buffer's place
                            if (!READOUT && p.P) p_chunks[first[k] + (t >> 2)] = make_uint4(xe[0], xe[1], xe[2], xe[3]);
                        }
                        else chunks[first[k] + (t >> 2)] = make_uint2(e[0] | (e[1] << 16), e[2] | (e[3] << 16));
                    }
                if (HAS_VAL) {
                    const float w0 = rn[k] > 0 ? __ldg(p.val + rb[k]) : 0.f;
                    bool mixed = false;
                    for (int t = 1; t < rn[k]; ++t) mixed |= __ldg(p.val + rb[k] + t) != w0;
                    roww[r] = w0;
                    if (mixed) *s_mixed = 1;
                }
            }
        }
        if (READOUT || !p.P) {
            for (int r = grp; r < nrows; r += NG) {
                int64_t xr = node0 + r;
                if (p.tags) {
                    const int t = __ldg(p.tags + xr);
                    xr = (unsigned)t >= (unsigned)p.num_tags ? 0 : t;
                }
                const float4 v = __ldg(X4 + xr * LPR + sl);
                H4[gf_h<D>(r, sl)] = make_float4(relu_ref(v.x), relu_ref(v.y), relu_ref(v.z), relu_ref(v.w));
            }
        }
        gf_worker_sync<WT>();
        // averaged messages give every edge of a row the same weight: the row is summed unweighted and scaled once
        const bool mixed = HAS_VAL && *s_mixed != 0;
        const bool listed = cached && !mixed;
        // different weights in a row: they are listed behind the columns, where there is room
        const uint32_t weights_at = smem_u32(smem + map.col) + gf_up(Cfg::CHUNK * (uint32_t)carry, 16);
        const bool weighted = mixed && cached && gf_up(Cfg::CHUNK * (uint32_t)carry, 16) + 16u * (uint32_t)carry <= Cfg::CHUNK * (uint32_t)p.chunk_cap;
        if (weighted) {
            float4* const wl = reinterpret_cast<float4*>(smem + map.col + gf_up(Cfg::CHUNK * (uint32_t)carry, 16));
            for (int r = threadIdx.x; r < nrows; r += WT) {
                const int b = __ldg(p.row_ptr + node0 + r), n = __ldg(p.row_ptr + node0 + r + 1) - b;
                float4* const to = wl + (info_s[r] & 0xffffu);
                for (int t = 0; t < n; t += 4) {
                    auto w = [&](int u) { return t + u < n ? __ldg(p.val + b + t + u) : 0.f; };
                    to[t >> 2] = make_float4(w(0), w(1), w(2), w(3));
                }
            }
            gf_worker_sync<WT>();
        }
        auto far_rows = [&]() {
            return GfFar{smem_u32(smem + Cfg::OFF_H), smem_u32(smem + map.tags), reinterpret_cast<const ulonglong2*>(p.P), node0, nrows, p.cap, p.edge_status};
        };
        auto weighted_row = [&](auto first, int r) {   // all lanes of a warp; r: the lane group's row, or beyond the last one
            const uint32_t inf = r < nrows ? info_s[r] : 0u, mine = ((inf >> 16) + 3) / 4;
            return gf_row_weighted<D, decltype(first)::value>(far_rows(), smem_u32(smem + map.col) + Cfg::CHUNK * (inf & 0xffffu), weights_at + 16u * (inf & 0xffffu),
                                                              mine, __reduce_max_sync(0xffffffffu, mine));
        };
        if (!READOUT && p.P) {   // first level: a sum of rows of P = ReLU(W_in) * W, no product
            const float4* __restrict__ P4 = reinterpret_cast<const float4*>(p.P);
            auto finish_first = [&](int r, ulonglong2 v) {
                if (r >= nrows) return;
                const float4 x = __ldg(X4 + (Cfg::TR ? (int64_t)(xo_s[r] / 16u) : (int64_t)tag_s[r] * LPR) + sl);
                const float2 f0 = unpack2(v.x), f1 = unpack2(v.y);
                H4[gf_h<D>(r, sl)] = make_float4(relu_max(f0.x + x.x), relu_max(f0.y + x.y), relu_max(f1.x + x.z), relu_max(f1.y + x.w));
            };
            if (Cfg::TR && listed) {
                // Two rows at a time, the third and fourth table row only where there is one.  The table rows' offsets are listed once per tile:
                // with a look-up of the tag per neighbour, and four rows read always, a batch of 4,093 molecules took 46.9 us for this level alone,
                // now 39.6.  (Four rows at a time: the registers spill, and what L1 the shared memory leaves goes to the spills: 178 us instead of 144.)
                const char* const Pl = reinterpret_cast<const char*>(p.P) + 16 * lane;
                const char* const Xl = reinterpret_cast<const char*>(p.x) + 16 * lane;
                auto table = [&](uint32_t off) { return __ldg(reinterpret_cast<const ulonglong2*>(Pl + off)); };
                constexpr int A = 2;
                for (int r = warp; r < nrows; r += A * WARPS) {
                    uint32_t inf[A];
                    uint4 c[A];
                    ulonglong2 v[A][2], t[A][2], x[A];
#pragma unroll
                    for (int a = 0; a < A; ++a) {
                        const int ra = r + a * WARPS;
                        inf[a] = ra < nrows ? info_s[ra] : 0u;
                        c[a] = p_chunks[inf[a] & 0xffffu];
                        x[a] = __ldg(reinterpret_cast<const ulonglong2*>(Xl + (ra < nrows ? xo_s[ra] : 0u)));
                    }
#pragma unroll
                    for (int a = 0; a < A; ++a) { v[a][0] = table(c[a].x); v[a][1] = table(c[a].y); }
#pragma unroll
                    for (int a = 0; a < A; ++a)
                        if (inf[a] >= 0x30000u) { t[a][0] = table(c[a].z); t[a][1] = table(c[a].w); }   // three neighbours or more
#pragma unroll
                    for (int a = 0; a < A; ++a) {
                        const int ra = r + a * WARPS;
                        if (ra >= nrows) break;
                        uint64_t s0 = add2(v[a][0].x, v[a][1].x), s1 = add2(v[a][0].y, v[a][1].y);
                        if (inf[a] >= 0x30000u) {
                            s0 = add2(add2(s0, t[a][0].x), t[a][1].x);
                            s1 = add2(add2(s1, t[a][0].y), t[a][1].y);
                            for (uint32_t k = 1; 4 * k < (inf[a] >> 16); ++k) {
                                const uint4 d = p_chunks[(inf[a] & 0xffffu) + k];
                                const ulonglong2 w0 = table(d.x), w1 = table(d.y), w2 = table(d.z), w3 = table(d.w);
                                s0 = add2(add2(add2(add2(s0, w0.x), w1.x), w2.x), w3.x);
                                s1 = add2(add2(add2(add2(s1, w0.y), w1.y), w2.y), w3.y);
                            }
                        }
                        if (HAS_VAL) {
                            const float w = roww[ra];
                            s0 = mul2(s0, pack2(w, w));
                            s1 = mul2(s1, pack2(w, w));
                        }
                        const float2 f0 = unpack2(add2(s0, x[a].x)), f1 = unpack2(add2(s1, x[a].y));
                        H4[ra * 32 + lane] = make_float4(relu_max(f0.x), relu_max(f0.y), relu_max(f1.x), relu_max(f1.y));
                    }
                }
            } else if (!Cfg::TR && listed) {
                for (int r = grp; r < nrows; r += NG) {
                    const float4 x = __ldg(X4 + (int64_t)tag_s[r] * LPR + sl);
                    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
                    const uint32_t inf = info_s[r];
                    for (uint32_t c = 0; c < ((inf >> 16) + 3) / 4; ++c) {
                        const uint2 e2 = chunks[(inf & 0xffffu) + c];
                        const uint32_t e[4] = {e2.x & 0xffffu, e2.x >> 16, e2.y & 0xffffu, e2.y >> 16};
                        float4 v[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) v[u] = __ldg(P4 + (int64_t)tag_s[e[u] >> Cfg::SHIFT] * LPR + sl);
#pragma unroll
                        for (int u = 0; u < 4; ++u) { acc.x += v[u].x; acc.y += v[u].y; acc.z += v[u].z; acc.w += v[u].w; }
                    }
                    if (HAS_VAL) { const float w = roww[r]; acc.x *= w; acc.y *= w; acc.z *= w; acc.w *= w; }
                    H4[gf_h<D>(r, sl)] =
                        make_float4(relu_max(acc.x + x.x), relu_max(acc.y + x.y), relu_max(acc.z + x.z), relu_max(acc.w + x.w));
                }
            } else if (HAS_VAL && weighted) {
                for (int rw = warp * GPW; rw < nrows; rw += NG) {   // warp-uniform
                    const int r = rw + sub;
                    const ulonglong2 v = weighted_row(std::true_type{}, r);
                    finish_first(r, v);
                }
            } else {
                const GfFar far = far_rows();
                auto span = [&](int r, int& b, int& n) {
                    b = n = 0;
                    if (r < nrows) { b = __ldg(p.row_ptr + node0 + r); n = __ldg(p.row_ptr + node0 + r + 1) - b; }
                };
                int b0, n0, b1, n1;   // this row's entries and the next one's
                span(grp, b0, n0);
                span(grp + NG, b1, n1);
                int c0 = sl < n0 ? __ldg(p.col_idx + b0 + sl) : 0;
                float w0 = HAS_VAL && sl < n0 ? __ldg(p.val + b0 + sl) : 0.f;
                for (int rw = warp * GPW; rw < nrows; rw += NG) {   // warp-uniform
                    const int r = rw + sub;
                    int b2, n2;
                    span(r + 2 * NG, b2, n2);
                    const int c1 = sl < n1 ? __ldg(p.col_idx + b1 + sl) : 0;
                    const float w1 = HAS_VAL && sl < n1 ? __ldg(p.val + b1 + sl) : 0.f;
                    const ulonglong2 v = gf_row_from_global<D, HAS_VAL, true>(far, p.col_idx + b0, p.val + b0, n0, c0, w0);
                    finish_first(r, v);
                    b0 = b1; n0 = n1; b1 = b2; n1 = n2; c0 = c1; w0 = w1;
                }
            }
            gf_worker_sync<WT>();
        }

        for (int lv = 0; lv < p.levels; ++lv) {
            // -------------------------------- gather, split, hand over --------------------------------
            for (int m = 0; m < mt; ++m) {
                const int rows_m = nrows - RB * m < RB ? nrows - RB * m : RB;
                uint64_t a0[RPG], a1[RPG];
                if (Cfg::TR && listed) {
                    // (the same, a warp per row and byte offsets in the list)
                    const uint32_t lane_addr = smem_u32(smem) + 16u * (uint32_t)lane;
                    uint32_t inf[RPG];
#pragma unroll
                    for (int i = 0; i < RPG; ++i) inf[i] = i * NG + warp < rows_m ? info_s[RB * m + i * NG + warp] : 0u;
#pragma unroll
                    for (int i = 0; i < RPG; ++i) {
                        a0[i] = a1[i] = 0ull;
                        if (i * NG + warp < rows_m) {
                            const uint4 c = chunks_t[inf[i] & 0xffffu];
                            const ulonglong2 v0 = gf_lds(lane_addr + c.x), v1 = gf_lds(lane_addr + c.y);
                            if (inf[i] < 0x30000u) {   // at most two neighbours: the row costs half the shared-memory reads
                                a0[i] = add2(v0.x, v1.x);
                                a1[i] = add2(v0.y, v1.y);
                            } else {
                                const ulonglong2 v2 = gf_lds(lane_addr + c.z), v3 = gf_lds(lane_addr + c.w);
                                a0[i] = add2(add2(add2(v0.x, v1.x), v2.x), v3.x);
                                a1[i] = add2(add2(add2(v0.y, v1.y), v2.y), v3.y);
                                for (uint32_t k = 1; 4 * k < (inf[i] >> 16); ++k) {
                                    const uint4 d = chunks_t[(inf[i] & 0xffffu) + k];
                                    const ulonglong2 w0 = gf_lds(lane_addr + d.x), w1 = gf_lds(lane_addr + d.y), w2 = gf_lds(lane_addr + d.z), w3 = gf_lds(lane_addr + d.w);
                                    a0[i] = add2(add2(add2(add2(a0[i], w0.x), w1.x), w2.x), w3.x);
                                    a1[i] = add2(add2(add2(add2(a1[i], w0.y), w1.y), w2.y), w3.y);
                                }
                            }
                            if (HAS_VAL) {
                                const float w = roww[RB * m + i * NG + warp];
                                a0[i] = mul2(a0[i], pack2(w, w));
                                a1[i] = mul2(a1[i], pack2(w, w));
                            }
                        }
                    }
                } else if (!Cfg::TR && listed) {
                    // every row's first chunk is fetched before the first row is summed; further chunks in a loop whose
                    // count is the warp's largest (a row without them reads the chunk of zero rows)
                    uint32_t inf[RPG];
                    uint2 ef[RPG];
                    const uint32_t slx = (uint32_t)sl * 0x10001u;
#pragma unroll
                    for (int i = 0; i < RPG; ++i) inf[i] = i * NG + grp < rows_m ? info_s[RB * m + i * NG + grp] : 0u;
#pragma unroll
                    for (int i = 0; i < RPG; ++i) ef[i] = chunks[inf[i] & 0xffffu];
#pragma unroll
                    for (int i = 0; i < RPG; ++i) {
                        a0[i] = a1[i] = 0ull;
                        if (i * NG + warp * GPW < rows_m) {   // warp-uniform
                            auto add_pair = [&](uint32_t e) {
                                e ^= slx;
                                const ulonglong2 v0 = H2[e & 0xffffu], v1 = H2[e >> 16];
                                a0[i] = add2(add2(a0[i], v0.x), v1.x);
                                a1[i] = add2(add2(a1[i], v0.y), v1.y);
                            };
                            auto add4 = [&](uint2 e2) {
                                e2.x ^= slx;
                                e2.y ^= slx;
                                const ulonglong2 v0 = H2[e2.x & 0xffffu], v1 = H2[e2.x >> 16], v2 = H2[e2.y & 0xffffu], v3 = H2[e2.y >> 16];
                                a0[i] = add2(add2(add2(add2(a0[i], v0.x), v1.x), v2.x), v3.x);
                                a1[i] = add2(add2(add2(add2(a1[i], v0.y), v1.y), v2.y), v3.y);
                            };
                            const uint32_t mine = inf[i] >> 16, most = __reduce_max_sync(0xffffffffu, mine);
                            if (most > 2) add4(ef[i]);
                            else add_pair(ef[i].x);
                            uint32_t c = 1;
                            auto next = [&]() { return chunks[4 * c < mine ? (inf[i] & 0xffffu) + c : 0u]; };
                            for (; 4 * c + 2 < most; ++c) add4(next());
                            if (4 * c < most) add_pair(next().x);   // one or two entries are left
                            if (HAS_VAL) {
                                const float w = i * NG + grp < rows_m ? roww[RB * m + i * NG + grp] : 0.f;
                                a0[i] = mul2(a0[i], pack2(w, w));
                                a1[i] = mul2(a1[i], pack2(w, w));
                            }
                        }
                    }
                }
                unsigned char* const s_hi = smem + Cfg::OFF_S + gf_op_off(grp, 4 * sl, RB);   // (row i*NG + grp: + i*NG*128, the same swizzle)
                unsigned char* const s_lo = smem + Cfg::OFF_S + gf_op_off_lo<D>(grp, 4 * sl, RB, Cfg::S_LO);
                auto largest = [](uint64_t v0, uint64_t v1) {
                    const float2 f0 = unpack2(v0), f1 = unpack2(v1);
                    return __float_as_uint(fmaxf(fmaxf(fabsf(f0.x), fabsf(f0.y)), fmaxf(fabsf(f1.x), fabsf(f1.y))));
                };
                // row i*NG + grp, mx: its largest element's bits (rows past the tile's last one are written too: finite, never read back)
                auto put_row = [&](int i, uint64_t v0, uint64_t v1, uint32_t mx) {
                    const uint32_t ex = gf_exponent_field(mx);
                    const float s = gf_scale_field(ex);
                    const uint64_t ss = pack2(s, s);
                    uint2 hi, lo;
                    split_f16(mul2(v0, ss), hi.x, lo.x);
                    split_f16(mul2(v1, ss), hi.y, lo.y);
                    *reinterpret_cast<uint2*>(s_hi + i * NG * 128) = hi;
                    *reinterpret_cast<uint2*>(s_lo + i * NG * 128) = lo;
                    if (sl == 0 && i * NG + grp < rows_m) {
                        if (Cfg::TR) rsf[RB * m + i * NG + grp] = gf_unscale_field(ex) * inv_w;
                        else rs[RB * m + i * NG + grp] = (uint8_t)(ex >> 23);
                    }
                };
                // the operand buffer is free once the previous row block of this level is multiplied
                auto wait_free = [&]() {
                    if (m > 0) tc_wait(bar_mma, (job - 1) & 1u, abort_flag, p.status, 40);
                };
                if (listed) {
                    wait_free();
                    if (uneven) {
                        const ulonglong2 in_scale = gf_lds(smem_u32(scales->in + 4 * sl));
#pragma unroll
                        for (int i = 0; i < RPG; ++i) {
                            a0[i] = mul2(a0[i], in_scale.x);
                            a1[i] = mul2(a1[i], in_scale.y);
                        }
                    }
                    // Rows whose maxima are taken side by side (a row past the end: zeros): shuffles are worth it (4,096 proteins 1402 -> 1320 us, together
                    // with the drain under the last product; one row at a time as everything else is now: 2,000 proteins, 16 warps, 703 us instead of 683; two rows at eight
                    // warps, 8,000 molecules at d = 64 192.4 -> 189.3, 16,000 at d = 32 183.8 -> 181.4), the one instruction of d = 128 is not (16,384 molecules 438 us,
                    // with two rows 447).
                    constexpr int SB = Cfg::TR ? 1 : (WARPS == 16 && RPG >= 4 ? 4 : 2);
                    static_assert(RPG % SB == 0, "whole batches");
#pragma unroll
                    for (int ib = 0; ib < RPG; ib += SB) {
                        if (ib * NG + warp * GPW >= rows_m) break;
                        uint32_t mx[SB];
#pragma unroll
                        for (int i = 0; i < SB; ++i) mx[i] = largest(a0[ib + i], a1[ib + i]);
                        if (LPR == 32) {
#pragma unroll
                            for (int i = 0; i < SB; ++i) mx[i] = __reduce_max_sync(0xffffffffu, mx[i]);
                        } else {
#pragma unroll
                            for (int o = LPR / 2; o; o >>= 1)
#pragma unroll
                                for (int i = 0; i < SB; ++i) mx[i] = max(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], o));
                        }
#pragma unroll
                        for (int i = 0; i < SB; ++i) put_row(ib + i, a0[ib + i], a1[ib + i], mx[i]);
                    }
                } else {
                    // one row after the other (nothing is held across the calls that sum them)
                    auto put_sum = [&](int i, ulonglong2 v) {
                        if (i == 0) wait_free();
                        if (uneven) {
                            const ulonglong2 in_scale = gf_lds(smem_u32(scales->in + 4 * sl));
                            v.x = mul2(v.x, in_scale.x);
                            v.y = mul2(v.y, in_scale.y);
                        }
                        uint32_t mx = largest(v.x, v.y);
#pragma unroll
                        for (int o = LPR / 2; o; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                        put_row(i, v.x, v.y, mx);
                    };
                    if (warp * GPW >= rows_m) wait_free();
                    else if (HAS_VAL && weighted) {
#pragma unroll 1
                        for (int i = 0; i * NG + warp * GPW < rows_m; ++i) put_sum(i, weighted_row(std::false_type{}, RB * m + i * NG + grp));
                    } else {
                        const GfFar far = far_rows();
                        auto span = [&](int i, int& b, int& n) {
                            b = n = 0;
                            if (i * NG + grp < rows_m) {
                                const int32_t* const rp = p.row_ptr + node0 + RB * m + i * NG + grp;
                                b = __ldg(rp);
                                n = __ldg(rp + 1) - b;
                            }
                        };
                        int b0, n0, b1, n1;   // this row's entries and the next one's
                        span(0, b0, n0);
                        span(1, b1, n1);
                        int c0 = sl < n0 ? __ldg(p.col_idx + b0 + sl) : 0;
                        float w0 = HAS_VAL && sl < n0 ? __ldg(p.val + b0 + sl) : 0.f;
#pragma unroll 1
                        for (int i = 0; i * NG + warp * GPW < rows_m; ++i) {   // warp-uniform
                            int b2, n2;
                            span(i + 2, b2, n2);
                            const int c1 = sl < n1 ? __ldg(p.col_idx + b1 + sl) : 0;
                            const float w1 = HAS_VAL && sl < n1 ? __ldg(p.val + b1 + sl) : 0.f;
                            put_sum(i, gf_row_from_global<D, HAS_VAL, false>(far, p.col_idx + b0, p.val + b0, n0, c0, w0));
                            b0 = b1; n0 = n1; b1 = b2; n1 = n2; c0 = c1; w0 = w1;
                        }
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // my stores -> visible to the tensor core
                __syncwarp();
                if (lane == 0) tc_mbar_arrive(bar_full);
                // one of the warps, another one for each row block, waits for all of them and issues the products
                if ((int)(job % WARPS) == warp) {
                    tc_wait(bar_full, job & 1u, abort_flag, p.status, 42);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (tc_elect()) {
                        const uint64_t s_desc = tc_b_desc(smem_u32(smem + Cfg::OFF_S)), w_desc = tc_b_desc(smem_u32(smem + Cfg::OFF_W));
                        const uint32_t acc = tmem_base + (Cfg::TR ? Cfg::TM_ACC + (uint32_t)(m * RB) : (uint32_t)(m * D));
#pragma unroll
                        for (int pass = 0; pass < 3; ++pass) {   // tail*head, head*tail, head*head: small terms first
                            const uint32_t s_off = pass == 0 ? Cfg::S_LO : 0u, w_off = pass == 1 ? Cfg::W_LO : 0u;
#pragma unroll
                            for (int ks = 0; ks < D / 16; ++ks) {
                                const uint32_t so = (uint32_t)(ks >> 2) * (uint32_t)(RB * 128) + (uint32_t)(ks & 3) * 32u;
                                const uint32_t wo = (uint32_t)(ks >> 2) * (uint32_t)(D * 128) + (uint32_t)(ks & 3) * 32u;
                                if (Cfg::TR) mma_f16_ts(acc, tmem_base + (pass == 1 ? Cfg::TM_WLO : 0u) + 8u * ks, s_desc + ((s_off + so) >> 4), Cfg::IDESC, (pass | ks) != 0);
                                else mma_f16_ss(acc, s_desc + ((s_off + so) >> 4), w_desc + ((w_off + wo) >> 4), Cfg::IDESC, (pass | ks) != 0);
                            }
                        }
                        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_mma) : "memory");
                    }
                    __syncwarp();
                }
                ++job;
            }
            // -------------------------------- drain: H = ReLU(acc * scale + X) --------------------------------
            // Units of LDC columns of 32 rows.  X of the next unit is on its way while one is worked on, the first unit's
            // during the wait.  H may be written once every warp has handed over its last row block (bar_full): the last product runs
            // under the drain of the row blocks before it, whose products every warp has seen complete.
            auto wait_last = [&]() {
                tc_wait(bar_mma, (job - 1) & 1u, abort_flag, p.status, 41);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            };
            auto wait_first = [&]() {
                if (mt > 1) {
                    tc_wait(bar_full, (job - 1) & 1u, abort_flag, p.status, 43);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                } else if (mt > 0) wait_last();
            };
            if constexpr (Cfg::TR) {
                // lane = output feature f, 16 nodes at a time (their scales and tags are broadcast reads); the rows of H are
                // written 128 bytes per instruction
                const int f = 32 * q + lane;
                const char* const Xf = reinterpret_cast<const char*>(p.x + f) + (p.tags ? 0 : (int64_t)node0 * Cfg::ROWB);
                float* const hcol = reinterpret_cast<float*>(smem + Cfg::OFF_H) + f;
                auto load_x = [&](int r0, float (&x)[16]) {
                    if (r0 >= nrows) return;
#pragma unroll
                    for (int i = 0; i < 16; i += 4) {
                        const uint4 o = *reinterpret_cast<const uint4*>(xo_s + r0 + i);
                        x[i] = __ldg(reinterpret_cast<const float*>(Xf + o.x));
                        x[i + 1] = __ldg(reinterpret_cast<const float*>(Xf + o.y));
                        x[i + 2] = __ldg(reinterpret_cast<const float*>(Xf + o.z));
                        x[i + 3] = __ldg(reinterpret_cast<const float*>(Xf + o.w));
                    }
                };
                float xa[16], xb[16];
                auto finish = [&](int r0, const float (&x)[16]) {
                    if (r0 >= nrows) return;   // warp-uniform
                    uint32_t v[16];
                    tc_ld_cols16(tmem_base + Cfg::TM_ACC + ((uint32_t)(32 * q) << 16) + (uint32_t)r0, v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (uneven) {
                        const float out_scale = scales->out[f];
#pragma unroll
                        for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * out_scale);
                    }
                    float* const h = hcol + r0 * 128;
#pragma unroll
                    for (int i = 0; i < 16; i += 4) {
                        const ulonglong2 c = *reinterpret_cast<const ulonglong2*>(rsf + r0 + i);
                        const float2 lo2 = unpack2(fma2(pack2(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), c.x, pack2(x[i], x[i + 1])));
                        const float2 hi2 = unpack2(fma2(pack2(__uint_as_float(v[i + 2]), __uint_as_float(v[i + 3])), c.y, pack2(x[i + 2], x[i + 3])));
                        h[i * 128] = relu_max(lo2.x);
                        h[(i + 1) * 128] = relu_max(lo2.y);
                        h[(i + 2) * 128] = relu_max(hi2.x);
                        h[(i + 3) * 128] = relu_max(hi2.y);
                    }
                };
                const int half = 32 * jc;   // my half of every row block: two groups of 16 nodes
                load_x(half, xa);
                wait_first();
                for (int m = 0; m < mt; ++m) {
                    if (m > 0 && m == mt - 1) wait_last();
                    load_x(64 * m + half + 16, xb);
                    finish(64 * m + half, xa);
                    if (m + 1 < mt) load_x(64 * (m + 1) + half, xa);
                    finish(64 * m + half + 16, xb);
                }
            } else {
                constexpr int UNITS = CW / LDC;
                float4 x[LDC / 4];
                auto x_row = [&](int m) -> const float4* {
                    const int r = 128 * m + 32 * q + lane;
                    const int64_t xr = r < nrows ? (p.tags ? (int64_t)tag_s[r] : (int64_t)node0 + r) : 0;
                    return X4 + xr * LPR + jc * (CW / 4);
                };
                const float4* xp = x_row(0);
#pragma unroll
                for (int c = 0; c < LDC / 4; ++c) x[c] = __ldg(xp + c);
                wait_first();
                for (int m = 0; m < mt; ++m) {
                    if (128 * m + 32 * q >= nrows) break;   // warp-uniform
                    if (m > 0 && m == mt - 1) wait_last();
                    const int r = 128 * m + 32 * q + lane;
                    const bool have = r < nrows;
                    const float c1 = have ? gf_unscale(rs[r]) * inv_w : 0.f;
                    const uint64_t cc = pack2(c1, c1);
                    const uint32_t acc_addr = tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)(m * D + jc * CW);
                    const uint32_t he = (uint32_t)((r << Cfg::SHIFT) + (r & 7));
                    const float4* xn = x_row(m + 1);
#pragma unroll
                    for (int h = 0; h < UNITS; ++h) {
                        uint32_t v[LDC];
                        if (LDC == 16) tc_ld_cols16(acc_addr + (uint32_t)(h * LDC), v);
                        else tc_ld_cols8(acc_addr + (uint32_t)(h * LDC), v);
                        float4 y[LDC / 4];
#pragma unroll
                        for (int c = 0; c < LDC / 4; ++c) y[c] = x[c];
                        const float4* nx = h + 1 < UNITS ? xp + (h + 1) * (LDC / 4) : xn;
#pragma unroll
                        for (int c = 0; c < LDC / 4; ++c) x[c] = __ldg(nx + c);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                        if (uneven) {
#pragma unroll
                            for (int c = 0; c < LDC; c += 4) {
                                const float4 o = *reinterpret_cast<const float4*>(scales->out + jc * CW + h * LDC + c);
                                v[c] = __float_as_uint(__uint_as_float(v[c]) * o.x);
                                v[c + 1] = __float_as_uint(__uint_as_float(v[c + 1]) * o.y);
                                v[c + 2] = __float_as_uint(__uint_as_float(v[c + 2]) * o.z);
                                v[c + 3] = __float_as_uint(__uint_as_float(v[c + 3]) * o.w);
                            }
                        }
                        if (have) {
#pragma unroll
                            for (int c = 0; c < LDC / 4; ++c) {
                                const float2 lo2 = unpack2(fma2(pack2(__uint_as_float(v[4 * c]), __uint_as_float(v[4 * c + 1])), cc, pack2(y[c].x, y[c].y)));
                                const float2 hi2 = unpack2(fma2(pack2(__uint_as_float(v[4 * c + 2]), __uint_as_float(v[4 * c + 3])), cc, pack2(y[c].z, y[c].w)));
                                H4[he ^ (uint32_t)(jc * (CW / 4) + h * (LDC / 4) + c)] = make_float4(relu_max(lo2.x), relu_max(lo2.y), relu_max(hi2.x), relu_max(hi2.y));
                            }
                        }
                    }
                    xp = xn;
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            gf_worker_sync<WT>();
        }
        // -------------------------------- node embeddings, pooling --------------------------------
        if (p.embed_out)
            for (int r = grp; r < nrows; r += NG)
                reinterpret_cast<float4*>(p.embed_out)[(int64_t)(node0 + r) * LPR + sl] = H4[gf_h<D>(r, sl)];
        // Graphs of up to 32 nodes are summed by one warp each; larger ones in pieces of 32 nodes (counted from the
        // graph's first node) by different warps, the partial sums added in order.
        float* const y_s = reinterpret_cast<float*>(smem + Cfg::OFF_S);                       // [Cfg::MAXG][D]
        float4* const part4 = reinterpret_cast<float4*>(smem + Cfg::OFF_S + Cfg::PART_OFF);   // pieces of graphs above 32 nodes
        int slot = 0;
        auto sum_rows = [&](int nb, int ne, float wgt) -> float4 {
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
            for (int n = nb + sub; n < ne; n += GPW) {
                const float4 v = H4[gf_h<D>(n, sl)];
                acc.x = fmaf(wgt, v.x, acc.x); acc.y = fmaf(wgt, v.y, acc.y);
                acc.z = fmaf(wgt, v.z, acc.z); acc.w = fmaf(wgt, v.w, acc.w);
            }
#pragma unroll
            for (int o = 16; o >= LPR; o >>= 1) {
                acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
                acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
                acc.z += __shfl_xor_sync(0xffffffffu, acc.z, o);
                acc.w += __shfl_xor_sync(0xffffffffu, acc.w, o);
            }
            return acc;
        };
        auto put_y = [&](int k, float4 acc) {
            if (sub != 0) return;
            if (READOUT) reinterpret_cast<float4*>(y_s)[k * LPR + sl] = acc;
            else reinterpret_cast<float4*>(p.Y)[(int64_t)(g0 + k) * LPR + sl] = acc;
        };
        for (int k = 0; k < ngr; ++k) {
            const int nb = goff[k], ne = goff[k + 1];
            const float wgt = p.pool_average ? (float)(1.0 / (double)(ne - nb)) : 1.0f;
            if (ne - nb <= 32) {
                if (k % WARPS == warp) put_y(k, sum_rows(nb, ne, wgt));
            } else {
                for (int c = 0; nb + 32 * c < ne; ++c, ++slot)
                    if ((k + c) % WARPS == warp) {
                        const float4 acc = sum_rows(nb + 32 * c, nb + 32 * c + 32 < ne ? nb + 32 * c + 32 : ne, wgt);
                        if (sub == 0) part4[slot * LPR + sl] = acc;
                    }
            }
        }
        gf_worker_sync<WT>();
        if (slot > 0) {
            slot = 0;
            for (int k = 0; k < ngr; ++k) {
                const int nb = goff[k], ne = goff[k + 1];
                if (ne - nb <= 32) continue;
                const int pieces = (ne - nb + 31) >> 5;
                if (k % WARPS == warp) {
                    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
                    for (int c = 0; c < pieces; ++c) {
                        const float4 v = part4[(slot + c) * LPR + sl];
                        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
                    }
                    put_y(k, acc);
                }
                slot += pieces;
            }
            gf_worker_sync<WT>();
        }
        if constexpr (READOUT) {
            float* scratch = reinterpret_cast<float*>(smem + Cfg::OFF_H);
            for (int gb = 0; gb < ngr; gb += 8) {
                const int nb = ngr - gb < 8 ? ngr - gb : 8;
                if (nb == 1) gf_readout<D, WT, 1>(p, y_s + gb * D, scratch, nb, (int64_t)g0 + gb);
                else if (nb <= 4) gf_readout<D, WT, 4>(p, y_s + gb * D, scratch, nb, (int64_t)g0 + gb);
                else gf_readout<D, WT, 8>(p, y_s + gb * D, scratch, nb, (int64_t)g0 + gb);
                gf_worker_sync<WT>();
            }
        }
        g0 = g1;
    }
    if (bad_tag) {
        p.status->code = S2V_ERR_INVALID_ARG;
        p.status->where = 3;
    }
    // ---- teardown: everyone is done with tensor memory before it is released
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(p.tm_cols) : "memory");
}

constexpr uint32_t gf_budget(int warps) { return (warps == 8 ? 113u : 227u) * 1024u; }   // shared memory of a CTA: two of eight warps share an SM

template <int D, int WARPS>
int gf_launch(s2v_ctx* ctx, cudaStream_t st, const GfParams& p, uint32_t smem, unsigned blocks)
{
    auto kern = p.logits ? (p.val ? s2v_graph_fused_kernel<D, WARPS, true, true> : s2v_graph_fused_kernel<D, WARPS, false, true>)
                         : (p.val ? s2v_graph_fused_kernel<D, WARPS, true, false> : s2v_graph_fused_kernel<D, WARPS, false, false>);
    S2V_CUDA_OK(ctx, s2v_allow_shared(kern, gf_budget(WARPS)));
    kern<<<blocks, WARPS * 32, smem, st>>>(p);
    S2V_CHECK_LAUNCH(ctx, "s2v_graph_fused_kernel");
    return S2V_OK;
}

}  // namespace

// Whether the kernel takes a batch whose largest graph has `max_nodes` nodes: its rows, the operand buffer and W have to
// fit the 227 KB a CTA may use (d = 128: 128 rows, d = 64: 640, d = 32: 1024), tags are kept in 16 bits.
bool s2v_graph_fused_supported(const s2v_ctx* ctx, int d, int max_nodes, int num_tags)
{
    const int most = d == 128 ? 128 : (d == 64 ? 640 : (d == 32 ? 1024 : 0));
    const int tags = d == 128 ? 1 << 23 : 1 << 16;   // held as 32-bit byte offsets of their W_in rows, or as 16-bit tags
    return max_nodes >= 1 && max_nodes <= most && num_tags < tags && ctx->smem_optin >= 227 * 1024;
}

size_t s2v_graph_fused_image_bytes(int d) { return sizeof(float) * ((size_t)d * (d + 2) + 4); }   // + GfScales

bool s2v_graph_fused_readout_ok(int d, int hidden, int num_class)
{
    // scratch of the readout (partial sums, hidden rows, logits of eight graphs) takes the H rows' place
    const int slices = hidden <= 64 ? 8 : (hidden <= 128 ? 4 : (hidden <= 256 ? 2 : 1));
    return sizeof(float) * 8 * ((size_t)hidden * (slices > 1 ? slices + 1 : 1) + num_class) <= (size_t)128 * 4 * d;
}

int s2v_launch_graph_fused(s2v_ctx* ctx, cudaStream_t st, const s2v_graph_fused_args& a)
{
    if (!s2v_graph_fused_supported(ctx, a.d, a.max_graph_nodes, a.num_tags)) return S2V_ERR_UNSUPPORTED;
    GfParams p{};
    p.G = a.G;
    p.row_ptr = a.row_ptr; p.col_idx = a.col_idx; p.val = a.val; p.graph_ptr = a.graph_ptr;
    p.tags = a.tags; p.x = a.x; p.num_tags = a.num_tags;
    p.W = a.W;
    p.levels = a.levels;
    p.pool_average = a.pool_average;
    p.Y = a.Y; p.embed_out = a.embed_out;
    p.W1 = a.W1; p.W2 = a.W2; p.hidden = a.hidden; p.num_class = a.num_class;
    p.logits = a.logits; p.probs = a.probs; p.pred = a.pred;
    p.status = ctx->dstatus_dev;
    p.edge_status = a.edge_status ? a.edge_status : ctx->dstatus_dev;
    if (a.P_scratch && a.levels >= 1 && !a.logits) {
        const int rc = s2v_launch_first_table_product(ctx, st, a.num_tags, a.d, a.x, a.W, a.P_scratch, true);
        if (rc != S2V_OK) return rc;
        p.P = a.P_scratch;
        p.levels = a.levels - 1;
    }
    if (a.image_scratch && !a.logits) {
        unsigned char* img = static_cast<unsigned char*>(a.image_scratch);
        if (a.d == 128) gf_weight_image_kernel<128><<<1, 1024, 0, st>>>(a.W, img);
        else if (a.d == 64) gf_weight_image_kernel<64><<<1, 1024, 0, st>>>(a.W, img);
        else gf_weight_image_kernel<32><<<1, 1024, 0, st>>>(a.W, img);
        S2V_CHECK_LAUNCH(ctx, "gf_weight_image_kernel");
        p.w_image = img;
    }
    // Rows per tile.  Small graphs: one row block per tile and (d <= 64) two 256-thread CTAs per SM, so that one CTA's
    // gather runs under the other's products and drains.  Larger graphs: as many rows as the batch gives each SM, up to
    // what fits, with 512 threads.
    const int need = (a.max_graph_nodes + 127) / 128 * 128;
    int warps = 16, per_sm = 1, cap = 128;
    if (a.d == 128) { warps = 8; per_sm = 2; }
    if (a.d == 64 && need == 128) { warps = 8; per_sm = 2; }
    if (a.d == 64 && need > 128) {
        const int64_t share = (a.N / ctx->sm_count + 127) / 128 * 128;
        cap = (int)(share < 640 ? share : 640);
        if (cap < need) cap = need;
    }
    if (a.d == 32) {
        if (need <= 640) {
            warps = 8; per_sm = 2;
            const int64_t share = (a.N / (2 * ctx->sm_count) + 127) / 128 * 128;
            cap = (int)(share < 640 ? share : 640);
            if (cap < need) cap = need;
        } else cap = 1024;
    }
    // What is left of the CTA's share of shared memory lists the columns (four to a chunk).  Six chunks per row, or what
    // the batch's mean asks for (1,000 graphs of 90 nodes, 30 neighbours each, d = 64: 199 us unlisted, 174).  Tiles get smaller as long as the list
    // would not hold a full one's (d = 32, averaged messages, 16,384 molecules: tiles of 640 rows take 179 us, of 512 152).
    const bool hv = a.val != nullptr;
    auto total = [&](int n) {
        return a.d == 128 ? gf_map<128>(cap, n, hv).total : (a.d == 64 ? gf_map<64>(cap, n, hv).total : gf_map<32>(cap, n, hv).total);
    };
    const uint32_t budget = gf_budget(warps);
    const uint32_t chunk = a.d == 128 ? GfCfg<128>::CHUNK : 8u;
    const double per_row = std::min(std::max(1.1, a.N > 0 ? 0.25 * (double)a.E / (double)a.N + 0.375 : 0.), 4096.);   // chunks: rows end inside one
    while (cap - 128 >= need && (budget - total(0)) / chunk < per_row * cap) cap -= 128;
    p.cap = cap;
    uint32_t cols = 32;
    while (cols < (uint32_t)(cap / 128 * a.d)) cols *= 2;
    p.tm_cols = a.d == 128 ? 256 : cols;   // d = 128: W^T and the accumulators of two row blocks
    const uint32_t left = (budget - total(0)) / 16 * 16, enough = (uint32_t)(cap * std::max(6.0, 1.25 * per_row)) / 2 * 2 * chunk;   // (more would take from the cache)
    p.chunk_cap = (int)((left < enough ? left : enough) / chunk);
    // the first level's list at d = 128 (p_chunks) has a chunk for each of these in the operand buffer, right in front of H
    static_assert((gf_budget(8) - GfCfg<128>::OFF_H - 128 * GfCfg<128>::ROWB) / GfCfg<128>::CHUNK <= GfCfg<128>::S_BYTES / GfCfg<128>::CHUNK, "cap = 128, two CTAs per SM");
    const uint32_t smem = total(p.chunk_cap);
    const int64_t most = (int64_t)ctx->sm_count * per_sm;
    const unsigned blocks = (unsigned)(a.G < most ? a.G : most);
    if (a.d == 128) return gf_launch<128, 8>(ctx, st, p, smem, blocks);
    if (a.d == 64) return warps == 8 ? gf_launch<64, 8>(ctx, st, p, smem, blocks) : gf_launch<64, 16>(ctx, st, p, smem, blocks);
    return warps == 8 ? gf_launch<32, 8>(ctx, st, p, smem, blocks) : gf_launch<32, 16>(ctx, st, p, smem, blocks);
}
