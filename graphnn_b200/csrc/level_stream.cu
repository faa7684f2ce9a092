// Fused structure2vec level for large matrices (d = 32, 64, 128):
//
//     out[i,:] = ReLU( (sum_{t in row i} val[t] * H[col_idx[t],:]) * W + X[i,:] )
//
// The sum is a gather of random rows of H, and what bounds it is how many bytes an SM keeps on their way: a kernel that only sums, with 2,048
// threads per SM, takes 333 us for a million rows with 8.4 million entries (d = 64, X read and out written), where level_tc.cu, whose warps
// gather, convert and store by turns, took 473.  So some warps do nothing but gather, and others take the sums through the tensor core and
// out.  Measured against the kernels it replaced from S2V_STREAM_ROWS rows on (us; other buffers each time and the L2 flushed; Erdos-Renyi, 8 entries a
// row, dense X): d = 32, a million rows, 361 -> 200; d = 64, a million, 483 -> 376; d = 128, half a million, 591 -> 416; R-MAT with 2^20 rows, d = 64,
// 1,830 -> 640, with 2^19, d = 128, 937 -> 580.  Rows of 2 entries: d = 64, a million, 216 -> 213 (of one 185 -> 207); d = 128: s2v_level_path.
//
// A tile is 16 units; a unit is what a warp sums at a time: a row for each group of d/4 lanes, two rows at d = 128.
//
//   gather warps  : take units one by one (a counter in shared memory).  Four 16-byte loads a lane go out together (d = 128: eight), and the
//                   next unit's indices and row offsets are on their way meanwhile.  Entries are added in CSR order.  A sum is split into a
//                   TF32 head and tail and stored as a row of the K-major B operand of its tile (four tiles in shared memory).  d = 32, 64:
//                   2 x 19 warps per SM at 40 registers (d = 64, a million rows, the same buffers each time: one CTA of 15 warps with eight
//                   loads each 404 us, this 367).  Instances with edge weights and those of d = 128 spill 4 to 16 bytes.
//                   d = 128: tensor memory holds W^T once, so one CTA per SM, 15 warps at 80 registers, with the unit
//                   behind the next one begun too.
//   MMA warp      : out^T = W^T * sum^T: W^T (A operand, head and tail; 128 / d copies below each other) stays in tensor memory, 3 * d/8
//                   tcgen05.mma of 128 x ROWS x 8 per tile (lo*hi, hi*lo, hi*hi) into one of several accumulators.  It also asks for the
//                   next tiles: the grid has a CTA per tile, and a running CTA takes over tiles whose CTAs have not started
//                   (clusterlaunchcontrol), so that an SM that starts late or has longer rows does fewer of them.
//   epilogue warps: an accumulator lane is an output column (the copies: of other rows), so X is read and out written 128 bytes per
//                   instruction, both past the L2's other contents, which is left to H (three levels in a row, where out is the next one's H:
//                   d = 64, 400,000 rows, 8 entries, 381 us, with ordinary stores 384; d = 32 206 and 209; d = 128 946 and 929; 131,072 and 200,000 rows
//                   0 to 1 % in its favour).
//
// Rows of more than LS_LONG entries would hold up their tile.  A kernel in front finishes them (sum, product, X, ReLU); this kernel, its
// programmatic dependent, does not wait for it before its own end and leaves those rows out.
//
// Every wait is bounded: on a time-out the kernel records S2V_ERR_DEVICE_TIMEOUT, raises a CTA-wide abort flag, waits (bounded again) for
// the tile requests that are on their way, frees its tensor memory and returns.
#include "common.cuh"
#include "long_rows.cuh"
#include "tcgen05.cuh"

namespace
{

constexpr int LS_RING = 16;                   // tiles that are known at a time
constexpr int LS_LONG = 128;                  // longer rows are left to the kernel in front
// ONE: one CTA per SM at every d, for grids that are to leave SMs free (CTAs go to every SM before one gets two).  24 gather warps with eight loads a lane at
// 64 registers, the most that AHEAD allows.  A million rows, 8 entries each, with one and with 20 SMs left, us: d = 64 404 and 443 (one CTA of the two 638 and 726,
// 16 warps 493 and 552; level_tc.cu 482 and 501), d = 32 218 and 242 (341 and 388); R-MAT 2^20, d = 64, 908 and 945 (963 and 1,097; 1,812 and 4,602).
// R-MAT 2^17 with one SM left loses (d = 64 137 -> 161): there is no room beside a CTA of the kernel in front.
template <int D, bool ONE = false>
struct LsCfg {
    static constexpr int SUB = 128 / D, LPR = D / 4;      // lane groups of a warp, lanes per group
    static constexpr int CTAS = D == 128 || ONE ? 1 : 2;  // per SM: tensor memory has 512 columns, W^T takes 2 d of them
    static constexpr int GW = D == 128 ? 15 : (ONE ? 24 : 19), EW = D == 128 ? 8 : 4, MW = GW + EW, THREADS = (MW + 1) * 32;   // gather and epilogue warps, number of the MMA warp
    static constexpr int R = D == 128 ? 2 : 1;            // rows per lane group and unit
    static constexpr int U = D == 128 || ONE ? 8 : 4;     // neighbours whose rows are on their way together
    static constexpr int HELD = D == 128 ? 3 : 2;         // units a gather warp has taken and not stored
    static constexpr int TN = 16, STAGES = 4, ROWS = TN * R * SUB, WROWS = TN * R;   // units per tile, tiles of operands, rows per tile and epilogue warp
    static constexpr int ACC = D == 32 ? 2 : 4;           // accumulators
    // While the MMA warp is at tile t, the tiles up to t - 2 are multiplied, at most STAGES tiles from t on are stored, and a gather warp holds
    // HELD units that are not; so no unit beyond tile t + AHEAD has been taken.  That far the tiles' numbers have to be known, or a warp
    // would wait for one with a unit of tile t in hand; and less than 2 * STAGES - 1 it has to be, or a warp would take the barrier of a stage
    // that is two phases behind for one that is ahead.
    static constexpr int AHEAD = 2 * STAGES - 2, ASKED = AHEAD + 2;   // tiles known, and asked for, ahead of the products
    static_assert((STAGES * TN + HELD * GW - 1) / TN <= AHEAD && ASKED <= 8 && AHEAD + ACC < LS_RING, "see above");
    static constexpr uint32_t HALF = TN * R * 512, STAGE_BYTES = 2 * HALF;       // operand head; the tail behind it
    static constexpr uint32_t TM_LO = D, TM_ACC = 2 * D, TM_COLS = 512 / CTAS;   // tensor memory: W^T head, tail, accumulators
    static_assert(TM_ACC + ACC * ROWS <= TM_COLS, "tensor memory");
    static constexpr uint32_t IDESC = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(ROWS >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);   // f32 <- tf32 x tf32, M = 128, N = ROWS
    static constexpr uint32_t OFF_FLAGS = STAGES * STAGE_BYTES;    // per tile and row: whether it is left out
    static constexpr uint32_t OFF_TILE = OFF_FLAGS + LS_RING * ROWS;
    static constexpr uint32_t OFF_RESP = OFF_TILE + 4 * LS_RING;   // answers to tile requests, 16 bytes each
    static constexpr uint32_t OFF_BAR = OFF_RESP + 16 * 8;
    enum { FULL = 0, EMPTY = FULL + STAGES, DONE = EMPTY + STAGES, READ = DONE + ACC, READY = READ + ACC, ANSWER = READY + LS_RING, BARS = ANSWER + 8 };
    static constexpr uint32_t OFF_MISC = OFF_BAR + 8 * BARS;
    static constexpr uint32_t SMEM = OFF_MISC + 32 + 1024;         // + slack to align the base to 1024 bytes
};

__device__ __forceinline__ uint64_t ls_add2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t ls_fma2(float w, uint64_t a, uint64_t c)
{
    uint64_t r, ww;
    asm("mov.b64 %0, {%1, %1};" : "=l"(ww) : "f"(w));
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(ww), "l"(a), "l"(c));
    return r;
}
__device__ __forceinline__ void ls_ld_cols8(uint32_t addr, uint32_t* v)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(addr)
                 : "memory");
}
// 16 bytes of a row.  (Volatile: the loads of a step stay together.  Under a condition, which the additions share, the compiler made one
// branch of both, and every load waited for the addition before it: d = 64, a million rows, 596 us instead of 404.  Lanes past the end of
// their row load its last entry again, or row 0; as one load for zeros, or at row 0 always, 378 and 382 us instead of 367, the same buffers each time.)
__device__ __forceinline__ ulonglong2 ls_row(const ulonglong2* p)
{
    ulonglong2 v;
    asm volatile("ld.global.nc.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p));
    return v;
}
// a request to take over a CTA that has not started; the answer arrives at `resp` on the barrier
__device__ __forceinline__ void ls_ask(uint32_t resp, uint32_t bar)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], 16;" ::"r"(bar) : "memory");
    asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(resp), "r"(bar) : "memory");
}
// the number of the CTA that was taken over, or -1
__device__ __forceinline__ int ls_answer(uint32_t resp)
{
    int x;
    asm volatile(
        "{\n\t.reg .b128 r;\n\t.reg .pred p;\n\t.reg .b32 a, b, c;\n\t"
        "ld.shared.b128 r, [%1];\n\t"
        "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n\t"
        "mov.b32 a, -1;\n\t"
        "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {a, b, c, _}, r;\n\t"
        "mov.b32 %0, a;\n\t}"
        : "=r"(x)
        : "r"(resp)
        : "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the slot is written again
    return x;
}

template <int D, bool HAS_VAL, int XMODE /*0 none, 1 dense, 2 table lookup*/, typename RpT, bool ONE>
__global__ void __launch_bounds__(LsCfg<D, ONE>::THREADS, LsCfg<D, ONE>::CTAS)
s2v_level_stream_kernel(int64_t n_rows, const RpT* __restrict__ row_ptr, const int32_t* __restrict__ col_idx, const float* __restrict__ val,
                        const float* __restrict__ H, const float* __restrict__ W, const float* X, const int32_t* __restrict__ x_index, int n_table,
                        float* out, int long_limit, int num_tiles, s2v_device_status* status)
{
    using Cfg = LsCfg<D, ONE>;
    constexpr int SUB = Cfg::SUB, LPR = Cfg::LPR, TN = Cfg::TN, ROWS = Cfg::ROWS, STAGES = Cfg::STAGES, ACC = Cfg::ACC, U = Cfg::U, WROWS = Cfg::WROWS;
    extern __shared__ unsigned char ls_smem_raw[];
    unsigned char* const smem = ls_smem_raw + ((1024u - (smem_u32(ls_smem_raw) & 1023u)) & 1023u);
    uint8_t* const flags = smem + Cfg::OFF_FLAGS;
    volatile int* const tiles = reinterpret_cast<volatile int*>(smem + Cfg::OFF_TILE);
    int* const next_unit = reinterpret_cast<int*>(smem + Cfg::OFF_MISC);
    volatile int* const abort_flag = reinterpret_cast<volatile int*>(smem + Cfg::OFF_MISC + 4);
    uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(smem + Cfg::OFF_MISC + 8);
    const uint32_t smem0 = smem_u32(smem);
    auto bar = [&](int i) { return smem0 + Cfg::OFF_BAR + 8u * (uint32_t)i; };
    const bool dealt = gridDim.x == (unsigned)num_tiles;   // tiles are taken over; else (SMs are left to others) every gridDim.x-th is this CTA's
    // the i-th request, i >= 1
    auto answer_at = [&](int i) { return smem0 + Cfg::OFF_RESP + 16u * (uint32_t)((i - 1) & 7); };
    auto answer_bar = [&](int i) { return bar(Cfg::ANSWER + ((i - 1) & 7)); };
    auto answer_phase = [&](int i) { return (uint32_t)((i - 1) >> 3) & 1u; };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) { tc_mbar_init(bar(Cfg::FULL + i), TN); tc_mbar_init(bar(Cfg::EMPTY + i), 1); }
        for (int i = 0; i < ACC; ++i) { tc_mbar_init(bar(Cfg::DONE + i), 1); tc_mbar_init(bar(Cfg::READ + i), 4); }
        for (int i = 0; i < LS_RING; ++i) tc_mbar_init(bar(Cfg::READY + i), 1);
        for (int i = 0; i < 8; ++i) tc_mbar_init(bar(Cfg::ANSWER + i), 1);
        *next_unit = Cfg::HELD == 3 ? 2 * Cfg::GW : 0;   // (d = 128: a warp's first two units go by its number)
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == Cfg::MW) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(Cfg::TM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp == Cfg::MW && lane == 0) {
        tiles[0] = (int)blockIdx.x;
        tc_mbar_arrive(bar(Cfg::READY));
        for (int i = 1; dealt && i <= Cfg::ASKED; ++i) ls_ask(answer_at(i), answer_bar(i));
    }
    if (warp >= Cfg::GW && warp < Cfg::MW) {
        // W^T: lane = output column (32 q + lane) % D, tensor memory column = input column
        constexpr int PART = D * 4 / Cfg::EW;
        const int q = warp & 3, part = (warp - Cfg::GW) >> 2;
        const float* const w = W + (32 * q + lane) % D;
        const uint32_t at = tmem + ((uint32_t)(32 * q) << 16);
#pragma unroll
        for (int c0 = 0; c0 < PART; c0 += 8) {
            const int c = PART * part + c0;
            uint32_t hi[8], lo[8];
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = __ldg(w + (int64_t)(c + u) * D);
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                hi[u] = tf32_rn(v[u]);
                lo[u] = tf32_rn(v[u] - __uint_as_float(hi[u]));
            }
            tc_st_cols8(at + c, hi);
            tc_st_cols8(at + Cfg::TM_LO + c, lo);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    auto tile_of = [&](int t, bool& ok) -> int {   // the CTA's t-th tile, -1: there is none
        ok = tc_wait(bar(Cfg::READY + (t & (LS_RING - 1))), (uint32_t)(t / LS_RING) & 1u, abort_flag, status, 60);
        return ok ? tiles[t & (LS_RING - 1)] : -1;
    };

    if (warp < Cfg::GW) {
        // =========================== gather ===========================
        const int sub = lane / LPR, sl = lane % LPR;
        const ulonglong2* __restrict__ H2 = reinterpret_cast<const ulonglong2*>(H) + sl;
        bool ok = true;
        // a unit's sums, row by row of the tile, as TF32 head and tail
        auto put = [&](int stage, int row, ulonglong2 a) {
            uint32_t hi[4], lo[4];
            tc_split(__uint_as_float((uint32_t)a.x), hi[0], lo[0]);
            tc_split(__uint_as_float((uint32_t)(a.x >> 32)), hi[1], lo[1]);
            tc_split(__uint_as_float((uint32_t)a.y), hi[2], lo[2]);
            tc_split(__uint_as_float((uint32_t)(a.y >> 32)), hi[3], lo[3]);
            unsigned char* const to = smem + (uint32_t)stage * Cfg::STAGE_BYTES + (uint32_t)(sl >> 3) * (ROWS * 128u) + (uint32_t)row * 128u +
                                      (uint32_t)(((sl & 7) ^ (row & 7)) * 16);
            *reinterpret_cast<uint4*>(to) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            *reinterpret_cast<uint4*>(to + Cfg::HALF) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        };
        // the operand is free once the tile STAGES before is multiplied
        auto wait_free = [&](int t) {
            if (ok && t >= STAGES) ok = tc_wait(bar(Cfg::EMPTY + t % STAGES), (uint32_t)(t / STAGES - 1) & 1u, abort_flag, status, 61);
            return ok;
        };
        auto stored = [&](int t) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) tc_mbar_arrive(bar(Cfg::FULL + t % STAGES));
        };
        if constexpr (Cfg::R == 1) {
            int unit, unit_x;   // the unit that is summed, the next one (below zero: there is none)
            RpT b = 0, e = 0;   // my row's entries: the next unit's from take() on
            int n = 0, c = 0;   // how many are summed here, one index per lane
            float w = 0.f;
            auto take = [&]() {   // the next unit, and its row offsets
                if (lane == 0) unit_x = atomicAdd(next_unit, 1);
                unit_x = __shfl_sync(0xffffffffu, unit_x, 0);
                const int tile = tile_of(unit_x / TN, ok);
                const int64_t row = (int64_t)tile * ROWS + unit_x % TN * SUB + sub;
                b = e = 0;
                if (tile < 0) unit_x = -1;
                else if (row < n_rows) {
                    b = __ldg(row_ptr + row);
                    e = __ldg(row_ptr + row + 1);
                }
            };
            auto window = [&](const int32_t* col, const float* vals) {   // a lane's index (and weight), where it has one
                if (HAS_VAL) w = sl < n ? __ldg(vals + sl) : 0.f;
                c = n > 0 ? __ldg(col + (sl < n ? sl : n - 1)) : 0;
            };
            auto start = [&]() {   // of the unit that has been taken: its first indices
                const bool left_out = e - b > (RpT)long_limit;
                if (sl == 0 && unit_x >= 0) flags[(unit_x / TN & (LS_RING - 1)) * ROWS + unit_x % TN * SUB + sub] = left_out ? 1 : 0;
                n = left_out ? 0 : (int)(e - b);
                window(col_idx + b, HAS_VAL ? val + b : nullptr);
            };
            take();
            start();
            while (unit_x >= 0) {
                unit = unit_x;
                const RpT at = b;
                int left = n;   // entries from the step on
                int most = SUB == 1 ? n : (int)__reduce_max_sync(0xffffffffu, (uint32_t)n);
                take();
                ulonglong2 acc = make_ulonglong2(0ull, 0ull);
                for (int t = 0; t < most; t += U, left -= U) {
                    if (t > 0 && t % LPR == 0) {
                        n = left;
                        window(col_idx + at + t, HAS_VAL ? val + at + t : nullptr);
                    }
                    ulonglong2 v[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) v[u] = ls_row(H2 + (int64_t)__shfl_sync(0xffffffffu, c, t % LPR + u, LPR) * LPR);
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const float wu = HAS_VAL ? __shfl_sync(0xffffffffu, w, t % LPR + u, LPR) : 0.f;
                        if (u < left) {
                            if (HAS_VAL) {
                                acc.x = ls_fma2(wu, v[u].x, acc.x);
                                acc.y = ls_fma2(wu, v[u].y, acc.y);
                            } else {
                                acc.x = ls_add2(acc.x, v[u].x);
                                acc.y = ls_add2(acc.y, v[u].y);
                            }
                        }
                    }
                }
                start();
                const int t = unit / TN;
                if (!wait_free(t)) break;
                put(t % STAGES, unit % TN * SUB + sub, acc);
                stored(t);
            }
        } else {
            // The unit that is summed, the next one (whose indices are on their way), the number of the one behind it (whose row offsets are);
            // below zero: the CTA has no such unit.  A lane group has two consecutive rows, whose entries are one range.
            int unit = -1, unit_x = -1, unit_r = warp;
            RpT b = 0, b_x = 0, rp_r;                             // first entry; row offset (one per lane)
            int m = 0, m_x = 0, n = 0, n_x = 0, c = 0, c_x = 0;   // entries of the first row, of both; index (one per lane)
            float w = 0.f, w_x = 0.f;
            auto offsets = [&]() {
                const int tile = tile_of(unit_r / TN, ok);
                int64_t row = (int64_t)tile * ROWS + (unit_r % TN * SUB + sub) * 2 + (sl < 2 ? sl : 2);
                if (tile < 0) { unit_r = -1; row = n_rows; }
                rp_r = __ldg(row_ptr + (row < n_rows ? row : n_rows));
            };
            auto prepare = [&](int then) {   // the unit behind becomes the next one; `then` (below zero: take one) the one behind
                unit_x = unit_r;
                b_x = __shfl_sync(0xffffffffu, rp_r, 0, LPR);
                const RpT mid = __shfl_sync(0xffffffffu, rp_r, 1, LPR), end = __shfl_sync(0xffffffffu, rp_r, 2, LPR);
                const bool long0 = mid - b_x > (RpT)long_limit, long1 = end - mid > (RpT)long_limit;
                m_x = long0 ? 0 : (int)(mid - b_x);
                n_x = m_x + (long1 ? 0 : (int)(end - mid));
                if (long0) b_x = mid;
                c_x = sl < n_x ? __ldg(col_idx + b_x + sl) : 0;
                if (HAS_VAL) w_x = sl < n_x ? __ldg(val + b_x + sl) : 0.f;
                if (unit_x < 0) return;
                if (sl < 2) flags[(unit_x / TN & (LS_RING - 1)) * ROWS + (unit_x % TN * SUB + sub) * 2 + sl] = (sl ? long1 : long0) ? 1 : 0;
                if (then < 0) {
                    if (lane == 0) then = atomicAdd(next_unit, 1);
                    then = __shfl_sync(0xffffffffu, then, 0);
                }
                unit_r = then;
                offsets();
            };
            offsets();
            prepare(Cfg::GW + warp);   // the first units by number
            while (unit_x >= 0) {
                unit = unit_x; b = b_x; m = m_x; n = n_x; c = c_x; w = w_x;
                const int most = SUB == 1 ? n : (int)__reduce_max_sync(0xffffffffu, (uint32_t)n);
                int cw = 0;   // the next window of indices
                float ww = 0.f;
                ulonglong2 first = make_ulonglong2(0ull, 0ull), acc = make_ulonglong2(0ull, 0ull);
                ulonglong2 v[U];
                auto fetch = [&](int t) {
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int cc = __shfl_sync(0xffffffffu, c, t % LPR + u, LPR);
                        v[u] = ls_row(H2 + (int64_t)cc * LPR);
                    }
                };
                auto add = [&](int t) {
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const float wu = HAS_VAL ? __shfl_sync(0xffffffffu, w, t % LPR + u, LPR) : 0.f;
                        if (t + u == m) { first = acc; acc = make_ulonglong2(0ull, 0ull); }
                        if (t + u < n) {
                            if (HAS_VAL) {
                                acc.x = ls_fma2(wu, v[u].x, acc.x);
                                acc.y = ls_fma2(wu, v[u].y, acc.y);
                            } else {
                                acc.x = ls_add2(acc.x, v[u].x);
                                acc.y = ls_add2(acc.y, v[u].y);
                            }
                        }
                    }
                };
                auto window = [&](int t) {   // indices t .. t + LPR - 1
                    cw = t + sl < n ? __ldg(col_idx + b + t + sl) : 0;
                    if (HAS_VAL) ww = t + sl < n ? __ldg(val + b + t + sl) : 0.f;
                };
                if (most > 0) fetch(0);   // (without an entry there may be no row 0, which lanes past their end read)
                if (most > LPR) window(LPR);
                prepare(-1);
                add(0);
                int t = U;
                for (; t < most; t += U) {
                    if (t % LPR == 0) {
                        c = cw;
                        w = ww;
                        if (t + LPR < most) window(t + LPR);
                    }
                    fetch(t);
                    add(t);
                }
                if (m >= t) { first = acc; acc = make_ulonglong2(0ull, 0ull); }   // (the second row's sum is empty and the first one's ended with the last step)
                const int tl = unit / TN, row = (unit % TN * SUB + sub) * 2;
                if (!wait_free(tl)) break;
                put(tl % STAGES, row, first);
                put(tl % STAGES, row + 1, acc);
                stored(tl);
            }
        }
    } else if (warp < Cfg::MW) {
        // =========================== epilogue ===========================
        const int q = warp & 3, f = (32 * q + lane) % D, r0 = 32 * q / D * WROWS;   // my column, the first of my WROWS rows of a tile
        const uint32_t acc_at = tmem + ((uint32_t)(32 * q) << 16) + Cfg::TM_ACC + (uint32_t)r0;
        for (int t = (warp - Cfg::GW) >> 2;; t += Cfg::EW / 4) {
            bool ok;
            const int tile = tile_of(t, ok);
            if (tile < 0) break;
            const int64_t row0 = (int64_t)tile * ROWS + r0;
            const int have = n_rows - row0 < WROWS ? (int)(n_rows - row0) : WROWS;   // (may be negative)
            float* const o = out + row0 * D + f;
            const float* const xp = X + (XMODE == 1 ? row0 * D : 0) + f;
            float x[WROWS];
#pragma unroll
            for (int i = 0; i < WROWS; ++i) {
                x[i] = 0.f;
                if (XMODE == 1 && i < have) x[i] = __ldcs(xp + D * i);
                if (XMODE == 2 && i < have) x[i] = __ldg(xp + (int64_t)tc_table_row(__ldg(x_index + row0 + i), n_table) * D);
            }
            if (!tc_wait(bar(Cfg::DONE + t % ACC), (uint32_t)(t / ACC) & 1u, abort_flag, status, 62)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            uint32_t leave = 0;   // bit i: my row i is left out
            {
                const uint32_t* const fl = reinterpret_cast<const uint32_t*>(flags + (t & (LS_RING - 1)) * ROWS + r0);
                uint32_t any = 0;
#pragma unroll
                for (int i = 0; i < WROWS / 4; ++i) any |= fl[i];
                if (any)
#pragma unroll
                    for (int i = 0; i < WROWS; ++i) leave |= (fl[i >> 2] >> (8 * (i & 3)) & 1u) << i;
            }
#pragma unroll
            for (int h = 0; h < WROWS; h += 8) {
                uint32_t v[8];
                ls_ld_cols8(acc_at + (uint32_t)(ROWS * (t % ACC) + h), v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (h + 8 == WROWS) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) tc_mbar_arrive(bar(Cfg::READ + t % ACC));
                }
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (h + i < have && !(leave >> (h + i) & 1u)) __stcs(o + D * (h + i), relu_ref(__uint_as_float(v[i]) + x[h + i]));
            }
        }
    } else {
        // =========================== products, tile requests ===========================
        int asked = dealt ? Cfg::ASKED : 0, answered = 0, known = 0;   // requests, answers, tiles that are published
        bool more = dealt, ok = true;                    // no request has been turned down yet
        for (int t = 0; ok; ++t) {
            while (ok && known < t + Cfg::AHEAD) {
                int tile = -1;
                while (ok && tile < 0 && answered < asked) {   // (after a refusal too: every tile that was handed over is this CTA's)
                    ++answered;
                    ok = tc_wait(answer_bar(answered), answer_phase(answered), abort_flag, status, 63);
                    if (ok) tile = ls_answer(answer_at(answered));
                    if (tile < 0) more = false;
                }
                if (!ok) break;
                ++known;
                if (!dealt && (int64_t)blockIdx.x + (int64_t)known * gridDim.x < num_tiles) tile = (int)(blockIdx.x + known * gridDim.x);
                if (lane == 0) {
                    tiles[known & (LS_RING - 1)] = tile;
                    tc_mbar_arrive(bar(Cfg::READY + (known & (LS_RING - 1))));
                }
                __syncwarp();
            }
            if (!ok || (t > 0 && tiles[t & (LS_RING - 1)] < 0)) break;
            for (; more && asked < t + Cfg::ASKED; ++asked)   // (the answer that lay in the slot has been read)
                if (lane == 0) ls_ask(answer_at(asked + 1), answer_bar(asked + 1));
            // (two tiles back: what Cfg::AHEAD counts on)
            if (t >= 2 && !(ok = tc_wait(bar(Cfg::EMPTY + (t - 2) % STAGES), (uint32_t)((t - 2) / STAGES) & 1u, abort_flag, status, 66))) break;
            const int stage = t % STAGES, a = t % ACC;
            ok = tc_wait(bar(Cfg::FULL + stage), (uint32_t)(t / STAGES) & 1u, abort_flag, status, 64);
            if (ok && t >= ACC) ok = tc_wait(bar(Cfg::READ + a), (uint32_t)(t / ACC - 1) & 1u, abort_flag, status, 65);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (tc_elect()) {
                const uint64_t desc = tc_b_desc(smem0 + (uint32_t)stage * Cfg::STAGE_BYTES);
                const uint32_t d_tmem = tmem + Cfg::TM_ACC + (uint32_t)(ROWS * a);
                uint32_t accumulate = 0;
#pragma unroll 1
                for (int pass = 0; pass < 3; ++pass) {   // tail*head, head*tail, head*head: small terms first
                    const uint32_t a_at = tmem + (pass == 1 ? Cfg::TM_LO : 0u), b_off = pass == 0 ? Cfg::HALF : 0u;
#pragma unroll
                    for (int ks = 0; ks < D / 8; ++ks) {
                        tc_mma(d_tmem, a_at + 8u * ks, desc + ((b_off + (uint32_t)(ks >> 2) * (ROWS * 128u) + (uint32_t)(ks & 3) * 32u) >> 4), Cfg::IDESC, accumulate);
                        accumulate = 1;
                    }
                }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar(Cfg::EMPTY + stage)) : "memory");
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar(Cfg::DONE + a)) : "memory");
            }
            __syncwarp();
        }
        // no answer may arrive once the CTA has gone (bounded like every wait, whatever the abort flag says)
        for (int i = answered + 1; i <= asked; ++i) {
            int spins = 0;
            while (!tc_mbar_try(answer_bar(i), answer_phase(i)))
                if (++spins > TC_WAIT_LIMIT) break;
        }
        __syncwarp();
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");   // what is launched behind this kernel counts on the long rows too
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == Cfg::MW) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Cfg::TM_COLS) : "memory");
}

// ---------------------------------------------------------------- rows of more than `long_limit` entries, finished
// A CTA looks through a block of rows.  Rows of more than LH_BIG entries come first, streamed through a ring in shared memory by the whole CTA,
// one after the other; then a warp sums a row at a time, rows of more than LH_MID entries before the others.  Where there are fewer of those
// than LH_FEW, the whole CTA takes the ones of more than LH_WARP entries too, or most of its warps would look on (half a million rows of one
// entry and 500 of 524, d = 128: 303 us without, 236 with).
constexpr int LH_THREADS = 512, LH_ROWS = 1024, LH_MID = 1024, LH_BIG = 2048, LH_WARP = 256, LH_FEW = 8;   // LH_ROWS: rows looked through by a CTA, at most
// What leaves the level kernel's CTAs room beside one or two of these.  (d = 128 with 108 KB: R-MAT 2^20 2,130 us instead of 1,600.)
template <int D> constexpr int LH_RING = (D == 128 ? 80 : 64) << 10;

// A row's sums (shared memory) times W, by a warp: D / 32 consecutive columns a lane
template <int D, int XMODE>
__device__ __forceinline__ void lh_finish(const float* sums, const float* __restrict__ W, const float* X, const int32_t* __restrict__ x_index, int n_table,
                                          float* out, int64_t r)
{
    constexpr int V = D / 32;
    const int at = (threadIdx.x & 31) * V;
    float acc[V];
#pragma unroll
    for (int i = 0; i < V; ++i) acc[i] = 0.f;
#pragma unroll 2
    for (int k = 0; k < D; k += 4) {
        const float4 s4 = *reinterpret_cast<const float4*>(sums + k);
        const float s[4] = {s4.x, s4.y, s4.z, s4.w};
        float w[4][V];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const float* const p = W + (k + u) * D + at;
            if constexpr (V == 4) *reinterpret_cast<float4*>(w[u]) = __ldg(reinterpret_cast<const float4*>(p));
            else if constexpr (V == 2) *reinterpret_cast<float2*>(w[u]) = __ldg(reinterpret_cast<const float2*>(p));
            else w[u][0] = __ldg(p);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int i = 0; i < V; ++i) acc[i] = fmaf(s[u], w[u][i], acc[i]);
    }
    const float* const x = XMODE == 0 ? nullptr : X + (XMODE == 1 ? r : (int64_t)tc_table_row(__ldg(x_index + r), n_table)) * D + at;
#pragma unroll
    for (int i = 0; i < V; ++i) out[r * D + at + i] = relu_ref(acc[i] + (XMODE == 0 ? 0.f : x[i]));
}

template <int D, bool HAS_VAL, int XMODE, typename RpT>
__global__ void __launch_bounds__(LH_THREADS, 2)
s2v_level_hub_kernel(int64_t n_rows, int rows_per_cta, const RpT* __restrict__ row_ptr, const int32_t* __restrict__ col_idx, const float* __restrict__ val,
                     const float* __restrict__ H, const float* __restrict__ W, const float* X, const int32_t* __restrict__ x_index, int n_table,
                     float* out, int long_limit)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    constexpr int WARPS = LH_THREADS / 32;
    extern __shared__ __align__(128) unsigned char lh_ring[];
    __shared__ uint16_t list[LH_ROWS + 1], big[LH_ROWS];   // longer rows from the front, shorter ones from the back
    __shared__ __align__(16) float sums[WARPS][D];
    __shared__ int cnt[4];                                 // longer, shorter, biggest rows; next one to take
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int64_t r0 = (int64_t)blockIdx.x * rows_per_cta; r0 < n_rows; r0 += (int64_t)gridDim.x * rows_per_cta) {
    __syncthreads();
    if (threadIdx.x < 4) cnt[threadIdx.x] = 0;
    __syncthreads();
    for (int j = threadIdx.x; j < rows_per_cta && r0 + j < n_rows; j += LH_THREADS) {
        const int64_t len = (int64_t)(__ldg(row_ptr + r0 + j + 1) - __ldg(row_ptr + r0 + j));
        if (len <= long_limit) continue;
        if (len > LH_BIG) big[atomicAdd(cnt + 2, 1)] = (uint16_t)j;
        else if (len > LH_MID) list[atomicAdd(cnt, 1)] = (uint16_t)j;
        else list[LH_ROWS - atomicAdd(cnt + 1, 1)] = (uint16_t)j;
    }
    __syncthreads();
    const int num_big = cnt[2], longer = cnt[0], total = longer + cnt[1];
    const int by_cta = num_big + (total < LH_FEW ? total : 0);
    auto row_of = [&](int i) { return r0 + list[i < longer ? i : LH_ROWS - (i - longer)]; };
    for (int i = 0; i < by_cta; ++i) {
        const int64_t r = i < num_big ? r0 + big[i] : row_of(i - num_big);
        const int64_t b = __ldg(row_ptr + r), len = __ldg(row_ptr + r + 1) - b;
        if (len <= LH_WARP) continue;
        long_row_by_cta<D, LH_THREADS, LH_RING<D>, HAS_VAL>(lh_ring, H, col_idx + b, HAS_VAL ? val + b : nullptr, (int)len, sums[0]);
        if (warp == WARPS - 1) lh_finish<D, XMODE>(sums[0], W, X, x_index, n_table, out, r);   // (done before this warp joins the next row)
    }
    __syncthreads();
    while (true) {
        int i = 0;
        if (lane == 0) i = atomicAdd(cnt + 3, 1);
        i = __shfl_sync(0xffffffffu, i, 0);
        if (i >= total) break;
        const int64_t r = row_of(i);
        const int64_t b = __ldg(row_ptr + r), len = __ldg(row_ptr + r + 1) - b;
        if (total < LH_FEW && len > LH_WARP) continue;
        const int c = lane < len ? __ldg(col_idx + b + lane) : 0;
        long_row_by_warp<D, D, HAS_VAL>(H, col_idx + b, HAS_VAL ? val + b : nullptr, (int)len, c, sums[warp]);
        __syncwarp();
        lh_finish<D, XMODE>(sums[warp], W, X, x_index, n_table, out, r);
        __syncwarp();
    }
    }
}

// ONE: some SMs are left to others (S2V_OPT_RESERVED_SMS); the kernel in front does not keep off them
template <int D, bool HAS_VAL, int XMODE, typename RpT, bool ONE>
int ls_launch_on(s2v_ctx* ctx, cudaStream_t st, bool long_rows, int64_t n_rows, const RpT* rp, const int32_t* ci, const float* val, const float* H,
                 const float* W, const float* X, const int32_t* x_index, int n_table, float* out)
{
    using Cfg = LsCfg<D, ONE && D != 128>;
    auto kern = s2v_level_stream_kernel<D, HAS_VAL, XMODE, RpT, ONE && D != 128>;
    S2V_CUDA_OK(ctx, s2v_allow_shared(kern, Cfg::SMEM));
    constexpr int64_t ROWS = Cfg::ROWS;
    const int64_t tiles = (n_rows + ROWS - 1) / ROWS;
    if (tiles >= (int64_t)INT32_MAX) return s2v_fail(ctx, S2V_ERR_UNSUPPORTED, "level: too many rows");
    const unsigned blocks = (unsigned)(!ONE || tiles < ctx->sm_count ? tiles : ctx->sm_count);
    const int limit = long_rows ? LS_LONG : 0x7fffffff;
    if (long_rows) {
        auto hubs = s2v_level_hub_kernel<D, HAS_VAL, XMODE, RpT>;
        S2V_CUDA_OK(ctx, s2v_allow_shared(hubs, LH_RING<D>));
        // about four CTAs per SM or more, so that they can be dealt out as they finish (eight: 2 us more for every level)
        const int64_t share = (n_rows / (4 * (int64_t)ctx->sm_count) + 63) / 64 * 64;
        const int per_cta = (int)(share < 64 ? 64 : (share > LH_ROWS ? LH_ROWS : share));
        const int64_t parts = (n_rows + per_cta - 1) / per_cta, resident = 2 * (int64_t)ctx->sm_count;
        hubs<<<(unsigned)(!ONE || parts < resident ? parts : resident), LH_THREADS, LH_RING<D>, st>>>(n_rows, per_cta, rp, ci, val, H, W, X, x_index, n_table,
                                                                                                    out, limit);
        S2V_CHECK_LAUNCH(ctx, "s2v_level_hub_kernel");
        S2V_CUDA_OK(ctx, launch_behind_long_rows(kern, blocks, Cfg::THREADS, Cfg::SMEM, st, n_rows, rp, ci, val, H, W, X, x_index, n_table, out, limit,
                                                 (int)tiles, ctx->dstatus_dev));
    } else
        kern<<<blocks, Cfg::THREADS, Cfg::SMEM, st>>>(n_rows, rp, ci, val, H, W, X, x_index, n_table, out, limit, (int)tiles, ctx->dstatus_dev);
    S2V_CHECK_LAUNCH(ctx, "s2v_level_stream_kernel");
    return S2V_OK;
}

template <int D, bool HAS_VAL, int XMODE, typename RpT>
int ls_launch(s2v_ctx* ctx, cudaStream_t st, bool long_rows, int64_t n_rows, const RpT* rp, const int32_t* ci, const float* val, const float* H,
              const float* W, const float* X, const int32_t* x_index, int n_table, float* out)
{
    return ctx->sm_count == ctx->sm_count_hw
               ? ls_launch_on<D, HAS_VAL, XMODE, RpT, false>(ctx, st, long_rows, n_rows, rp, ci, val, H, W, X, x_index, n_table, out)
               : ls_launch_on<D, HAS_VAL, XMODE, RpT, true>(ctx, st, long_rows, n_rows, rp, ci, val, H, W, X, x_index, n_table, out);
}

template <int D, typename RpT>
int ls_dispatch(s2v_ctx* ctx, cudaStream_t st, bool long_rows, int64_t n_rows, const RpT* rp, const int32_t* ci, const float* val, const float* H,
                const float* W, const float* X, const float* table, const int32_t* x_index, int n_table, float* out)
{
#define LS_GO(HV, XM) return ls_launch<D, HV, XM, RpT>(ctx, st, long_rows, n_rows, rp, ci, val, H, W, table ? table : X, x_index, n_table, out)
    if (val) {
        if (table) LS_GO(true, 2);
        if (X) LS_GO(true, 1);
        LS_GO(true, 0);
    }
    if (table) LS_GO(false, 2);
    if (X) LS_GO(false, 1);
    LS_GO(false, 0);
#undef LS_GO
}

}  // namespace

int s2v_launch_level_stream(s2v_ctx* ctx, cudaStream_t st, bool long_rows, int64_t n_rows, int d, const void* row_ptr, bool rp64, const int32_t* col_idx,
                            const float* val, const float* H, const float* W, const float* X, const float* table, const int32_t* x_index, int n_table,
                            float* out)
{
#define LS_D(DD)                                                                                                                                       \
    case DD:                                                                                                                                           \
        return rp64 ? ls_dispatch<DD>(ctx, st, long_rows, n_rows, (const int64_t*)row_ptr, col_idx, val, H, W, X, table, x_index, n_table, out)        \
                    : ls_dispatch<DD>(ctx, st, long_rows, n_rows, (const int32_t*)row_ptr, col_idx, val, H, W, X, table, x_index, n_table, out)
    switch (d) {
        LS_D(32);
        LS_D(64);
        LS_D(128);
        default: return S2V_ERR_UNSUPPORTED;
    }
#undef LS_D
}
