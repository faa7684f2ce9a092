// Long rows (hubs of a power-law graph) of the level kernels.  A level kernel gives a row to one warp, or part of one; a
// row of 10^4 or 10^5 entries keeps that warp -- and its CTA's pipeline behind it -- busy long after everyone else is done
// (R-MAT scale 20, d = 128: 11.3 ms, nearly all of it the longest rows).  So the rows above LONG_ROW entries are summed by whole
// CTAs ahead of the rest, together with the other rows of their groups of GROUP rows (what a warp of the main loop works on as one
// unit).  The sums go to the rows' places in `out`, which the level overwrites with the result afterwards, so no scratch memory is
// needed; the main loop reads such a group's sums from there instead of gathering.
//   * Up to LONG_BIG entries a warp sums a row, in slices of up to 64 columns with 4 KB of neighbour rows on their way; a longer
//     one, taken first, is streamed through a ring in shared memory by the whole CTA, where one warp would be bounded by latency.
//   * Entries are added one after the other in CSR order, as everywhere else in the level: a float sum of 10^5 entries
//     depends on its order in the fifth digit.
//   * In large levels (LongCfg::FRONT_ROWS) a kernel in front makes the sums, with the level kernel launched as its programmatic dependent: in level_tc.cu
//     for sparse matrices at d = 128, in level.cu where tcgen05 is switched off (level_stream.cu finishes such rows its own way).  The figures are of a time
//     when these two took every large level.  With the look and the sums inside, the registers of the main loop cost every level 1 - 5 %, also without a long row
//     (Erdos-Renyi, a million rows: d = 64 480 us inside, 474 in front, 473 without any of it; with edge weights 526, 473, 472;
//     d = 32 366, 351, 349; d = 128, half a million, 601, 584, 585; R-MAT 2^20, d = 128: 4.9 ms inside, 2.9 in front).  A second
//     launch costs up to 1 us: below, the level kernel does it for the rows it owns (30,000 rows, d = 64: 13.5 us, 14.1 in front).
#pragma once

#include "common.cuh"

namespace
{

constexpr int LONG_ROW = 256;      // below this a row is no longer than what the other warps of a tile work on
constexpr int LONG_BIG = 2048;      // above this a row is worth the whole CTA
constexpr int LONG_SCAN = 8;       // rows per thread and pass of the sums
enum { LONG_NONE, LONG_INSIDE, LONG_FRONT };   // where a level kernel's long rows are summed

template <int W> struct LongVec;
template <> struct LongVec<4> { using T = float4; };
template <> struct LongVec<2> { using T = float2; };
template <> struct LongVec<1> { using T = float; };
__device__ __forceinline__ void long_add(float4& a, float4 v) { a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w; }
__device__ __forceinline__ void long_fma(float4& a, float w, float4 v) { a.x = fmaf(w, v.x, a.x); a.y = fmaf(w, v.y, a.y); a.z = fmaf(w, v.z, a.z); a.w = fmaf(w, v.w, a.w); }
__device__ __forceinline__ void long_add(float2& a, float2 v) { a.x += v.x; a.y += v.y; }
__device__ __forceinline__ void long_add(float& a, float v) { a += v; }
__device__ __forceinline__ void long_fma(float2& a, float w, float2 v) { a.x = fmaf(w, v.x, a.x); a.y = fmaf(w, v.y, a.y); }
__device__ __forceinline__ void long_fma(float& a, float w, float v) { a = fmaf(w, v, a); }

// SL columns (H, out_row already point at the first of them) of one row by one warp; c: its first 32 indices, one per lane
template <int D, int SL, bool HAS_VAL>
__device__ __forceinline__ void long_row_by_warp(const float* __restrict__ H, const int32_t* __restrict__ col, const float* __restrict__ val, int n, int c,
                                                 float* out_row)
{
    using V = typename LongVec<SL / 32>::T;
    constexpr int U = 1024 / SL, STRIDE = D / (SL / 32);   // 4 KB in flight
    const int lane = threadIdx.x & 31;
    const V* __restrict__ Hv = reinterpret_cast<const V*>(H) + lane;
    V acc{};
    float w = HAS_VAL && lane < n ? __ldg(val + lane) : 0.f;
    for (int t = 0; t < n; t += 32) {
        const int cn = t + 32 + lane < n ? __ldg(col + t + 32 + lane) : 0;   // the next indices, on their way while these rows are summed
        const float wn = HAS_VAL && t + 32 + lane < n ? __ldg(val + t + 32 + lane) : 0.f;
#pragma unroll
        for (int u0 = 0; u0 < 32; u0 += U) {
            if (t + u0 >= n) break;
            V v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int cc = __shfl_sync(0xffffffffu, c, u0 + u);
                v[u] = V{};
                if (t + u0 + u < n) v[u] = __ldg(Hv + (int64_t)cc * STRIDE);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {   // (what lies past the end adds zeros)
                if (HAS_VAL) long_fma(acc, __shfl_sync(0xffffffffu, w, u0 + u), v[u]);
                else long_add(acc, v[u]);
            }
        }
        c = cn;
        w = wn;
    }
    reinterpret_cast<V*>(out_row)[lane] = acc;
}

// One row by the whole CTA: the threads copy the neighbour rows through a ring, TURN rows side by side, and the first D threads add one
// column each.  A stage costs about 300 cycles (wait, barrier, copies) and 6 to 10 per row, and a row of a large H takes 1.5 us to arrive: so
// stages of two turns where the ring has room for four of them (four, not three, where there is room for more), and up to eight stages.  (d = 128, ring of 80 KB, one row of 262,144 entries,
// us: stages of 16 rows 4,020, of 32 2,370; ring of 110 KB, stages of 48 rows 2,820, of 32 2,460; with four stages of 32 rows and each stage's indices loaded one stage ahead 5,900.)
template <int D, int THREADS, int BYTES, bool HAS_VAL>
__device__ __forceinline__ void long_row_by_cta(unsigned char* ring, const float* __restrict__ H, const int32_t* __restrict__ col,
                                                const float* __restrict__ val, int n, float* out_row)
{
    constexpr int PIECES = D / 4, TURN = THREADS / PIECES, FIT = BYTES / (TURN * 4 * D);
    constexpr int TURNS = FIT < 8 ? 1 : (FIT < 16 ? 2 : 4), STAGE = TURN * TURNS, NS = FIT / TURNS < 8 ? FIT / TURNS : 8;   // turns and rows per stage, stages
    static_assert(NS >= 3, "two stages on their way while one is added");
    const int piece = threadIdx.x % PIECES, row0 = threadIdx.x / PIECES;
    const int stages = (n + STAGE - 1) / STAGE;
    const uint32_t ring_addr = smem_u32(ring) + (uint32_t)(row0 * D + 4 * piece) * 4u;
    // a lane has its group's index of one turn of PIECES; those of the next PIECES turns are on their way
    auto indices = [&](int q0) {
        const uint32_t t = (uint32_t)((q0 + piece) * TURN + row0);
        return row0 < TURN && t < (uint32_t)n ? __ldg(col + t) : -1;
    };
    int c = indices(0), c_next = indices(PIECES), q = 0, slot = 0;
    auto issue = [&]() {
#pragma unroll
        for (int k = 0; k < TURNS; ++k, ++q) {
            if (q > 0 && q % PIECES == 0) {
                c = c_next;
                c_next = indices(q + PIECES);
            }
            const int cc = __shfl_sync(0xffffffffu, c, q % PIECES, PIECES);
            if (cc >= 0)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ring_addr + (uint32_t)((slot * TURNS + k) * TURN * D) * 4u), "l"(H + (int64_t)cc * D + 4 * piece)
                             : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        slot = slot + 1 < NS ? slot + 1 : 0;
    };
    for (int s = 0; s < NS - 1; ++s) issue();
    float acc = 0.f;
    int at = 0;
    for (int s = 0; s < stages; ++s) {
        asm volatile("cp.async.wait_group %0;" ::"n"(NS - 2) : "memory");
        __syncthreads();   // stage s has arrived, and everyone is done with the stage before it
        issue();
        if (threadIdx.x < D) {
            const float* p = reinterpret_cast<const float*>(ring) + at * STAGE * D + threadIdx.x;
            const int m = n - s * STAGE < STAGE ? n - s * STAGE : STAGE;
            constexpr int U = STAGE % 32 == 0 ? 32 : 16;
            int r = 0;
            for (; r + U <= m; r += U) {
                float v[U];
#pragma unroll
                for (int u = 0; u < U; ++u) v[u] = p[(r + u) * D];
#pragma unroll
                for (int u = 0; u < U; ++u) acc = HAS_VAL ? fmaf(__ldg(val + s * STAGE + r + u), v[u], acc) : acc + v[u];
            }
            for (; r < m; ++r) acc = HAS_VAL ? fmaf(__ldg(val + s * STAGE + r), p[r * D], acc) : acc + p[r * D];
        }
        at = at + 1 < NS ? at + 1 : 0;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (threadIdx.x < D) out_row[threadIdx.x] = acc;
    __syncthreads();
}

// The rows of a CTA that owns the row blocks blockIdx.x, blockIdx.x + gridDim.x, ... of RB rows each, by position.
template <int RB>
__device__ __forceinline__ int64_t long_row_of(int j) { return ((int64_t)blockIdx.x + (int64_t)(j / RB) * gridDim.x) * RB + j % RB; }
template <int RB>
__device__ __forceinline__ int long_rows_owned(int64_t n_rows)
{
    const int64_t blocks = (n_rows + RB - 1) / RB;
    return blocks > blockIdx.x ? (int)((blocks - 1 - blockIdx.x) / gridDim.x + 1) * RB : 0;
}

// Whether the CTA owns a long row.  A thread takes STEP consecutive rows at a time and looks at each of them only if they have more
// than LONG_ROW entries together.  load() issues the first loads; what they bring is looked at after the conversion of W.  The look is
// bounded by its own instructions, fetched and run once: with a load and a shuffle per row it took 2 us of every level.
template <int THREADS, int RB, typename RpT>
struct LongLook {
    static constexpr int STEP = 8, PER = RB / STEP, AHEAD = 2;
    static_assert(RB % STEP == 0 && THREADS % PER == 0, "whole groups, whole blocks");
    RpT a[AHEAD], z[AHEAD];
    static __device__ __forceinline__ int64_t row_of(int j) { return ((int64_t)(j / PER) * gridDim.x + blockIdx.x) * RB + j % PER * STEP; }
    __device__ __forceinline__ void load(int64_t n_rows, const RpT* __restrict__ row_ptr, int j0 = 0)
    {
#pragma unroll
        for (int k = 0; k < AHEAD; ++k) {
            const int64_t r = row_of(j0 + k * THREADS + (int)threadIdx.x);
            a[k] = z[k] = 0;
            if (r < n_rows) {
                a[k] = __ldg(row_ptr + r);
                z[k] = __ldg(row_ptr + (r + STEP < n_rows ? r + STEP : n_rows));
            }
        }
    }
    __device__ __forceinline__ bool any(int64_t n_rows, const RpT* __restrict__ row_ptr)
    {
        bool found = false;
        for (int j0 = 0;;) {
#pragma unroll
            for (int k = 0; k < AHEAD; ++k)
                if (z[k] - a[k] > LONG_ROW) {
                    const int64_t r0 = row_of(j0 + k * THREADS + (int)threadIdx.x), r1 = r0 + STEP < n_rows ? r0 + STEP : n_rows;
#pragma unroll 1
                    for (int64_t r = r0; r < r1; ++r) found |= __ldg(row_ptr + r + 1) - __ldg(row_ptr + r) > LONG_ROW;
                }
            j0 += THREADS * AHEAD;
            if (row_of(j0) >= n_rows) return found;
            load(n_rows, row_ptr, j0);
        }
    }
};

// Called by all THREADS threads of the CTA; BYTES of shared memory at `smem`.
template <int D, int THREADS, int RB, int GROUP, int BYTES, bool HAS_VAL, typename RpT>
__device__ __forceinline__ void sum_long_rows(unsigned char* smem, int64_t n_rows, const RpT* row_ptr, const int32_t* col_idx, const float* val,
                                           const float* H, float* out)
{
    constexpr int SL = D < 64 ? D : 64, SLICES = D / SL, LIST = 2 * ((THREADS * LONG_SCAN + GROUP - 1) / GROUP), RING = (16 + LIST + 127) / 128 * 128;
    static_assert(RB % GROUP == 0 && 32 % GROUP == 0 && THREADS % 32 == 0 && RING < BYTES, "whole groups per warp; the ring behind the list");
    int* const cnt = reinterpret_cast<int*>(smem);                  // groups listed, next slice to take
    uint16_t* const list = reinterpret_cast<uint16_t*>(smem + 16);
    const int lane = threadIdx.x & 31;
    const int owned = long_rows_owned<RB>(n_rows);
    for (int j0 = 0; j0 < owned; j0 += THREADS * LONG_SCAN) {
        __syncthreads();
        if (threadIdx.x == 0) cnt[0] = cnt[1] = 0;
        __syncthreads();
        for (int k = 0; k < LONG_SCAN; ++k) {
            const int j = k * THREADS + threadIdx.x;
            bool is_long = false;
            if (j0 + j < owned) {
                const int64_t r = long_row_of<RB>(j0 + j);
                is_long = r < n_rows && __ldg(row_ptr + r + 1) - __ldg(row_ptr + r) > LONG_ROW;
            }
            const unsigned marks = __ballot_sync(0xffffffffu, is_long) >> (lane / GROUP * GROUP);
            if (lane % GROUP == 0 && (marks & ((1u << GROUP) - 1u)) != 0) list[atomicAdd(cnt, 1)] = (uint16_t)(j / GROUP);
        }
        __syncthreads();
        const int n = cnt[0];
        // fewer groups than warps: the whole CTA on every long row, or most of its warps would look on
        const int big = n * SLICES < THREADS / 32 ? LONG_ROW : LONG_BIG;
        for (int i = 0; i < n; ++i) {   // the longest rows
            const int64_t r0 = long_row_of<RB>(j0 + list[i] * GROUP);
            for (int64_t r = r0; r < r0 + GROUP && r < n_rows; ++r) {
                const int64_t b = __ldg(row_ptr + r), len = __ldg(row_ptr + r + 1) - b;
                if (len > big)
                    long_row_by_cta<D, THREADS, BYTES - RING, HAS_VAL>(smem + RING, H, col_idx + b, HAS_VAL ? val + b : nullptr, (int)len, out + r * D);
            }
        }
        while (true) {   // the others: a warp for each slice of a group
            int i = 0;
            if (lane == 0) i = atomicAdd(cnt + 1, 1);
            i = __shfl_sync(0xffffffffu, i, 0);
            if (i >= n * SLICES) break;
            const int64_t r0 = long_row_of<RB>(j0 + list[i / SLICES] * GROUP);
            const int c0 = i % SLICES * SL;
            const int64_t ri = r0 + (lane <= GROUP ? lane : GROUP);
            const RpT rp = __ldg(row_ptr + (ri < n_rows ? ri : n_rows));
            int64_t b = __shfl_sync(0xffffffffu, rp, 0), e = __shfl_sync(0xffffffffu, rp, 1);
            int c = b + lane < e ? __ldg(col_idx + b + lane) : 0;
            for (int k = 0; k < GROUP; ++k) {
                const int64_t en = __shfl_sync(0xffffffffu, rp, k + 2 <= GROUP ? k + 2 : GROUP);
                const int cn = e + lane < en ? __ldg(col_idx + e + lane) : 0;   // the next row's first indices
                if (r0 + k < n_rows && e - b <= big)
                    long_row_by_warp<D, SL, HAS_VAL>(H + c0, col_idx + b, HAS_VAL ? val + b : nullptr, (int)(e - b), c, out + (r0 + k) * D + c0);
                b = e;
                e = en;
                c = cn;
            }
        }
    }
    __syncthreads();
}

// The same as a call, for the level kernels: their main loops keep their registers.
template <int D, int THREADS, int RB, int GROUP, int BYTES, bool HAS_VAL, typename RpT>
__device__ __noinline__ void sum_long_rows_call(unsigned char* smem, int64_t n_rows, const RpT* row_ptr, const int32_t* col_idx, const float* val,
                                                const float* H, float* out)
{
    sum_long_rows<D, THREADS, RB, GROUP, BYTES, HAS_VAL>(smem, n_rows, row_ptr, col_idx, val, H, out);
}

// Shared memory: with the CTAs of the level kernel beside it an SM keeps the split of its memory into cache and shared memory, so the
// kernel asks for no more per SM than the level kernel does (d = 64, 112 KB per CTA instead of 48: the level of a million rows 544 us
// instead of 474; d = 128, 48 KB instead of 112: R-MAT scale 20 4.76 ms instead of 2.91).
template <int D> struct LongCfg { static constexpr int THREADS = 512, CTAS = 2, BYTES = (D == 128 ? 112 : 48) << 10, FRONT_ROWS = 131072; };
// (d = 32 at 131,072 rows: R-MAT 137 us inside, 141 in front; Erdos-Renyi at 180,000: 43.2 and 41.7)
template <> struct LongCfg<32> { static constexpr int THREADS = 256, CTAS = 3, BYTES = 40 << 10, FRONT_ROWS = 160000; };
constexpr int LONG_RB = 128;
template <int D, int GROUP, bool HAS_VAL, typename RpT>
__global__ void __launch_bounds__(LongCfg<D>::THREADS, LongCfg<D>::CTAS)
long_rows_kernel(int64_t n_rows, const RpT* __restrict__ row_ptr, const int32_t* __restrict__ col_idx, const float* __restrict__ val,
                 const float* __restrict__ H, float* __restrict__ out)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    extern __shared__ __align__(128) unsigned char long_smem[];
    LongLook<LongCfg<D>::THREADS, LONG_RB, RpT> look;
    look.load(n_rows, row_ptr);
    if (__syncthreads_or(look.any(n_rows, row_ptr)))
        sum_long_rows<D, LongCfg<D>::THREADS, LONG_RB, GROUP, LongCfg<D>::BYTES, HAS_VAL>(long_smem, n_rows, row_ptr, col_idx, val, H, out);
}
template <int D, int GROUP, bool HAS_VAL, typename RpT>
int launch_long_rows(s2v_ctx* ctx, cudaStream_t st, int64_t n_rows, const RpT* row_ptr, const int32_t* col_idx, const float* val, const float* H, float* out)
{
    auto kern = long_rows_kernel<D, GROUP, HAS_VAL, RpT>;
    constexpr int BYTES = LongCfg<D>::BYTES;
    if (BYTES > (48 << 10)) S2V_CUDA_OK(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, BYTES));
    const int64_t blocks = (n_rows + LONG_RB - 1) / LONG_RB, most = (int64_t)LongCfg<D>::CTAS * ctx->sm_count;
    kern<<<(unsigned)(blocks < most ? blocks : most), LongCfg<D>::THREADS, BYTES, st>>>(n_rows, row_ptr, col_idx, val, H, out);
    S2V_CHECK_LAUNCH(ctx, "long_rows_kernel");
    return S2V_OK;
}
// The level kernel behind it may start while the sums are made.
template <typename... Params, typename... Args>
cudaError_t launch_behind_long_rows(void (*kern)(Params...), unsigned blocks, unsigned threads, size_t smem, cudaStream_t st, Args... args)
{
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = blocks;
    cfg.blockDim = threads;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<Params>(args)...);
}
__device__ __forceinline__ void long_rows_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// the sum that long_rows_kernel left in the row's place of `out`
__device__ __forceinline__ float4 long_row_sum(const float4* p)
{
    float4 v;
    asm volatile("ld.global.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    return v;
}

}  // namespace
