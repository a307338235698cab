// lstm_group_sm100.cu -- the recurrence of a factored-LSTM layer as many small thread-block
// clusters, each with a FEW chunk rows: the batch is spread over all clusters the device holds
// instead of being packed into 128-row tiles.
//
// A step is a chain of dependent stages, so its time is set by what each stage of one cluster has
// to move and compute for its own rows. With the rows as the M = 128 dimension of the
// contractions that amount does not shrink with the batch; here the operands are swapped. The
// WEIGHTS are the M dimension (128 hidden units per CTA, one accumulator block per gate) and the
// chunk rows are N = 16, 32 or 48 columns, and the recurrent half of the gate weights lives in
// TENSOR MEMORY as the A operand: an MMA then costs 12 to 20 cycles instead of the 40 that reading a
// 128-row A operand from shared memory takes whatever N is.
//
// A cluster has C = H / 128 CTAs (2 to 8). CTA j
//   * owns units 128 j .. 128 j + 127: their four gate weight blocks (hh half in tensor memory, x
//     half in shared memory) and, in registers, their cell state for the cluster's rows;
//   * projects: the CTAs form pairs (2p, 2p+1); pair p owns a contiguous part of the rows, CTA
//     2p + s computes projection columns 64 s .. 64 s + 63 of them (M = 64) from the complete
//     int8 rows. With an odd C the last CTA projects nothing.
// Per step two exchanges inside the cluster, both of 16-byte st.async stores (eight lanes write 128
// contiguous bytes) that complete on an mbarrier of the receiver: the int8 hidden slices go to the pair that
// owns the row, the f16 projections back to every CTA. The x half of the contraction runs meanwhile. With
// more than some thirty rows the cluster treats them as two groups, so that one is computed while the
// other travels.
//
//   warp 0       loader: resident weights, x_down rows of every step
//   warp 1       MMA issuer
//   warps 2-17   epilogues, four per tensor-memory lane quadrant: thread = hidden unit, a quarter
//                of the rows each (gates, cell update, int8 code); the same warps turn the
//                projection accumulators into f16 and send them
//
// A buffer is only overwritten after its reader has provably finished: a CTA sends h_t (of a group) after
// its gate contraction of step t, which needs hh_t from every pair, which a pair sends after its
// projection of h_{t-1} is complete; and the other way round for hh. Nobody leaves before the final
// cluster barrier. Clusters never wait for one another, so any number of them may run in waves.
//
// What bounds a step (B200, H = 768, cycles): with few rows (3 per cluster, 2790 cycles, 1.46 us)
// the chain: h exchange 600, projection 450 + read-back 250, hh exchange 500, contraction 500,
// cell update 430; with 47 (5500 cycles, 2.8 us for 1024 chunks; 0.2 more while the exchanges left in 16-byte
// pieces) the tensor pipe (x half 1450, projections 1400, hh half 1150), which waits for the second
// group's accumulators to be read and its hidden rows to arrive: the accumulators leave no tensor memory for a second set.
//
// Arithmetic and its order are those of the other single-launch forms (x_down half first, then the
// hh_down half in K steps of 16; int32 sums scaled by (1/127)*scale and rounded to f16): the bytes
// are the same.
#include <fluke/fluke.h>

#include "fluke_sm100.h"
#include "sm100_ptx.cuh"
#include "tma_host.cuh"

#include <cuda_fp16.h>

namespace fluke_sm100 {
namespace {

constexpr int kGThreads = 576;
constexpr int kGEpiWarps = 16;
constexpr int kGUnits = 128;       // hidden units per CTA = tensor-memory lanes
constexpr int kGRank = 128;        // factor rank the kernel is built for
constexpr int kGMaxCtas = 8;       // portable cluster size: H <= 1024
constexpr int kGTmemCols = 512;
constexpr int kGTmemW = 256;       // first column of the hh half of the gate weights: 4 gates x 64
constexpr int kGWxBytes = 4 * kGUnits * 256;  // x half of the gate weights in shared memory
constexpr int kGMaxSmem = 232448;

struct GroupDev {
    int T, B;
    int reverse;
    int rows;                  // chunk rows per cluster (the last one may have fewer)
    int n_own[2];              // rows of a group a pair projects
    const int8_t *dn;          // [R, H]
    const __half *w_up;        // [4H, 2R]
    const float *bias;         // [4H]
    const float *dn_scale;     // [R]
    float *c;                  // [B,H]
    int8_t *h_out;             // [T,B,H]
    int8_t *h_state;           // [B,H]: final hidden state
    long long *trace;          // trace builds only: [T][8] SM-clock stamps of CTA 0
};

// All of the following depends on the cluster size C = H / 128, which the kernel is compiled for: with
// operand addresses at fixed distances the issuer needs few instructions between MMAs (the 24 of a
// projection took 800 cycles to issue with C a variable).
// Rows of a group's hidden tile (and columns of its projection): what a pair projects of the group's n rows, as
// a multiple of 8.
__host__ __device__ constexpr int group_h_rows(int n, int C) { return ((n + C / 2 - 1) / (C / 2) + 7) / 8 * 8; }
// K blocks (128 hidden units, 32 columns) of the projection weights that fit in tensor memory beside
// the gate weights, the gate accumulators and the projections.
__host__ __device__ constexpr int group_dn_ts(int n0, int n1, int C) {
    const int fit = (kGTmemW - 4 * (n0 + n1) - group_h_rows(n0, C) - group_h_rows(n1, C)) / 32;
    return fit < C ? fit : C;
}
// Rows of a staging slot: a batch of four hidden rows, or the projected rows of a quarter of the warps.
__host__ __device__ constexpr int group_stage_rows(int n0, int n1, int C) {
    const int r = group_h_rows(n0 > n1 ? n0 : n1, C) / 4;
    return r > 4 ? r : 4;
}
struct GroupLayout {
    int x, hh, dn, h, stage, bars, misc, dynamic;
};
__host__ __device__ constexpr GroupLayout group_layout_slots(int n0, int n1, int C, int x_slots) {
    GroupLayout l = {};
    const int n = n0 + n1;
    l.x = kGWxBytes;                            // x_down rows: 2 K blocks [n x 128 B] per slot
    l.hh = l.x + x_slots * n * 256;             // hh_down rows, the same shape
    l.dn = l.hh + n * 256;                      // 64 projection rows: the K blocks not in tensor memory [64 x 128 B]
    l.h = l.dn + 8192 * (C - group_dn_ts(n0, n1, C));  // hidden rows of the pair, per group: C K blocks
    l.stage = l.h + (group_h_rows(n0, C) + group_h_rows(n1, C)) * C * kGUnits;  // 2 slots x 4 x [rows x 128 B]
    l.bars = l.stage + 8 * group_stage_rows(n0, n1, C) * 128;
    l.misc = l.bars + 15 * 8;
    l.dynamic = l.misc + 16 + 1024;             // slack for the manual 1024-byte alignment
    return l;
}
// x tiles of two steps where shared memory allows it, else of one.
__host__ __device__ constexpr int group_x_slots(int n0, int n1, int C) {
    return group_layout_slots(n0, n1, C, 2).dynamic <= kGMaxSmem ? 2 : 1;
}
__host__ __device__ constexpr GroupLayout group_layout(int n0, int n1, int C) {
    return group_layout_slots(n0, n1, C, group_x_slots(n0, n1, C));
}

// 16 bytes into a CTA of the cluster; completes 16 bytes of the transaction count of an mbarrier
// of the same CTA.
__device__ __forceinline__ void store_to_peer(uint32_t dst_cluster, uint4 v, uint32_t bar_cluster) {
    asm volatile(
        "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
        ::"r"(dst_cluster), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar_cluster)
        : "memory");
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void sts8(uint32_t addr, int v) {
    asm volatile("st.shared.u8 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void sts16(uint32_t addr, unsigned short v) {
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(addr), "h"(v) : "memory");
}

// Barrier of the four warps that share a staging slot.
__device__ __forceinline__ void quad_sync(int id) { asm volatile("barrier.cta.sync %0, 128;" ::"r"(id) : "memory"); }

template <int V>
struct Int { static constexpr int value = V; };  // a number that a lambda receives as a type

// N0 + N1: accumulator columns, i.e. chunk rows of a cluster at most. With N1 = 0 they are one group: the chain
// of a step is all there is to run. Otherwise the first N0 rows and the others are two groups that share the
// x part of the contraction (its MMAs read their A operand from shared memory, 40 cycles each whatever
// N is up to 64, so one for both) and go through the rest of the step one after the other: while
// one is exchanged, the other is projected or computed.
template <int N0, int N1, int C>
__global__ void __launch_bounds__(kGThreads, 1)
lstm_group_kernel(const __grid_constant__ CUtensorMap tm_w,    // w_up [4H, 2R] f16, boxes 128 x 64
                  const __grid_constant__ CUtensorMap tm_x,    // x_down [T, 2, B, 64] f16, boxes of NB rows
                  const __grid_constant__ CUtensorMap tm_dn,   // dn_hh [R, H] int8, boxes 64 x 128
                  const __grid_constant__ CUtensorMap tm_h0,   // h_0 [H/128, B, 128] int8, boxes of the first group's tile
                  const __grid_constant__ CUtensorMap tm_h1,   // and of the second's
                  const GroupDev p) {
    constexpr int G = N1 > 0 ? 2 : 1, NB = N0 + N1;
    constexpr int kXSlots = group_x_slots(N0, N1, C);
    constexpr int H = C * kGUnits;
    constexpr int kPad0 = group_h_rows(N0, C), kPad1 = group_h_rows(N1, C);
    constexpr int kDnTs = group_dn_ts(N0, N1, C);
    constexpr GroupLayout L = group_layout(N0, N1, C);
    constexpr int kCols = (N0 > N1 ? N0 : N1) / 4;   // rows of a group that an epilogue thread holds at most
    constexpr int kBatches = kCols / 4;              // it takes them four at a time
    constexpr int kSendP = kCols / 4;                // 16-byte stores per lane and step, projections
    constexpr int kStageRows = group_stage_rows(N0, N1, C);
    static_assert(N0 % 16 == 0 && N1 % 16 == 0 && 5 * NB <= kGTmemW, "accumulators beside the weights in tensor memory");
    extern __shared__ uint8_t smem_raw[];
    // every CTA of the cluster computes the same offset, so peers' buffers are at the same
    // shared-window offsets as this CTA's
    uint8_t *smem = reinterpret_cast<uint8_t *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L.bars);
    uint64_t *bar_once = &bars[0];       // resident weights loaded
    uint64_t *bar_x = &bars[1];          // [slots] x_down rows landed
    uint64_t *bar_x_free = &bars[3];     // [slots] x half of the contraction has read them
    uint64_t *bar_h = &bars[5];          // [G] complete hidden rows of the pair arrived
    uint64_t *bar_proj = &bars[7];       // [G] projection accumulator complete
    uint64_t *bar_hh = &bars[9];         // [G] hh_down rows arrived
    uint64_t *bar_acc = &bars[11];       // [G] gate accumulators complete
    uint64_t *bar_acc_free = &bars[13];  // [G] epilogue has read them
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + L.misc);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + L.misc + 4);

    const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x) >> 5, 0), lane = threadIdx.x & 31;
    const int rank = int(cluster_ctarank());
    const int pair = rank >> 1, half = rank & 1;
    const bool projects = rank < (C & ~1);
    const int m0 = (blockIdx.x / C) * p.rows;          // first chunk row of the cluster
    const int n_rows = min(p.rows, p.B - m0);          // and how many it has
    const int n0 = rank * kGUnits;
    // of group e: rows it has, rows of them this CTA projects
    auto rows_of = [&](int e) { return G == 1 ? n_rows : e == 0 ? min(n_rows, N0) : max(n_rows - N0, 0); };
    auto own_of = [&](int e) { return min(max(rows_of(e) - pair * p.n_own[e], 0), p.n_own[e]); };
    constexpr int h_group1 = kPad0 * H;                // byte offset of the second group's hidden rows
    auto time_of = [&](int i) { return p.reverse ? p.T - 1 - i : i; };
    if (threadIdx.x == 0) {
        for (int b = 0; b < 13; ++b) mbar_init(&bars[b], 1);
        for (int b = 13; b < 15; ++b) mbar_init(&bars[b], kGEpiWarps);
        *abort_flag = 0;
        fence_barrier_init();
        for (int e = 0; e < G; ++e) mbar_arrive_expect_tx(&bar_hh[e], uint32_t(rows_of(e)) * 256);
    }
    if (warp == 1) tmem_alloc(tmem_slot, kGTmemCols);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    if (warp >= 2) {
        // the hh half of the gate weights: warp = (lane quadrant, gate), thread = row of the block
        const int q = warp & 3, g = (warp - 2) >> 2;
        const uint4 *src = reinterpret_cast<const uint4 *>(
            p.w_up + (size_t(g) * H + n0 + q * 32 + lane) * (2 * kGRank));
        const uint32_t t_lane = tmem + (uint32_t(q * 32) << 16) + kGTmemW;
#pragma unroll 1
        for (int v = 0; v < 8; ++v) tmem_st_32x8(t_lane + g * 64 + v * 8, __ldg(src + 2 * v), __ldg(src + 2 * v + 1));
        if (projects) {
            // and K blocks g, g + 4, .. of the projection rows (M = 64: row 16 q + i in lane 32 q + i)
            const uint4 *dn = reinterpret_cast<const uint4 *>(p.dn + size_t(half * 64 + q * 16 + (lane & 15)) * H);
            for (int kb = g; kb < kDnTs; kb += 4)
#pragma unroll 1
                for (int v = 0; v < 4; ++v)
                    tmem_st_32x8(t_lane - 32 * (kb + 1) + v * 8, __ldg(dn + kb * 8 + 2 * v), __ldg(dn + kb * 8 + 2 * v + 1));
        }
        tmem_st_wait();
        tc_fence_before_sync();
    }
    __syncthreads();
    tc_fence_after_sync();
    // every barrier of the cluster is initialised before any CTA may store to a peer
    cluster_sync_all();

    if (warp == 0) {
        // ------------------------------ loader (one thread) -----------------------------
        if (elect_one()) {
            mbar_arrive_expect_tx(bar_once, kGWxBytes + (projects ? (C - kDnTs) * 8192 : 0));
            for (int g = 0; g < 4; ++g)
                for (int kb = 0; kb < 2; ++kb)
                    tma_load_2d(smem + (g * 2 + kb) * 16384, &tm_w, bar_once, kGRank + kb * 64, g * H + n0);
            if (projects) {
                for (int kb = kDnTs; kb < C; ++kb)
                    tma_load_2d(smem + L.dn + (kb - kDnTs) * 8192, &tm_dn, bar_once, kb * 128, half * 64);
                // step 0 projects the layer's initial hidden state
                for (int e = 0; e < G; ++e) {
                    mbar_arrive_expect_tx(&bar_h[e], uint32_t(e ? kPad1 : kPad0) * H);
                    tma_load_3d(smem + L.h + e * h_group1, e ? &tm_h1 : &tm_h0, &bar_h[e], 0, m0 + e * N0 + pair * p.n_own[e], 0);
                }
            }
            bool ok = true;
            for (int i = 0; i < p.T && ok; ++i) {
                const int s = i % kXSlots, u = i / kXSlots;
                if (u > 0) ok = mbar_wait(&bar_x_free[s], (u - 1) & 1, abort_flag, 96);
                if (!ok) break;
                mbar_arrive_expect_tx(&bar_x[s], NB * 256);
                tma_load_4d(smem + L.x + s * (NB * 256), &tm_x, &bar_x[s], 0, m0, 0, time_of(i));
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------ MMA issuer --------------------------------------
        // The whole warp walks the loop; one elected lane issues. Descriptors are uniform and the
        // K loops unrolled, so an MMA is issued every few cycles.
        constexpr uint32_t kIdescX = make_idesc<kKindF16>(128, NB);
        uint64_t d_wx = make_smem_desc_sw128(smem_u32(smem));
        uint64_t d_x0 = make_smem_desc_sw128(smem_u32(smem + L.x));
        uint64_t d_hh0 = make_smem_desc_sw128(smem_u32(smem + L.hh));
        uint64_t d_dn = make_smem_desc_sw128(smem_u32(smem + L.dn));
        uint64_t d_h0 = make_smem_desc_sw128(smem_u32(smem + L.h));
        bool ok = mbar_wait(bar_once, 0, abort_flag, 97);
        int i = 0;
        // The x half of gates [g0, g1). Its 32 MMAs read their A operand from shared memory (40 cycles
        // each, a third of a one-group step in all) and the tensor pipe works in order, so they are
        // issued in pieces for the times when it would wait.
        auto x_half = [&](auto from, auto to) {
            constexpr int g0 = decltype(from)::value, g1 = decltype(to)::value;
            const uint64_t d_x = d_x0 + uint64_t((i % kXSlots) * (NB * 16));
            if (elect_one()) {
#pragma unroll
                for (int g = g0; g < g1; ++g)
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        tc_mma<kKindF16>(tmem + g * NB, d_wx + uint64_t((g * 2 + (k >> 2)) * 1024 + 2 * (k & 3)),
                                         d_x + uint64_t((k >> 2) * (NB * 8) + 2 * (k & 3)), kIdescX, k != 0);
                if (g1 == 4) tc_commit(&bar_x_free[i % kXSlots]);
            }
            __syncwarp();
        };
        auto wait_x = [&]() {
            ok = ok && mbar_wait(&bar_x[i % kXSlots], (i / kXSlots) & 1, abort_flag, 99);
            if (i > 0) ok = ok && mbar_wait(bar_acc_free, (i - 1) & 1, abort_flag, 98);
            tc_fence_after_sync();
            return ok;
        };
        auto wait_h = [&](int e) {
            if (projects) ok = ok && mbar_wait<true>(&bar_h[e], i & 1, abort_flag, 100);
            return ok;
        };
        auto project = [&](auto group) {
            constexpr int e = decltype(group)::value;
            if (!projects) return true;
            fence_proxy_async_smem();   // the peers' stores are generic-proxy writes
            tc_fence_after_sync();
            FLUKE_STAMP(blockIdx.x == 0 && lane == 0, i * 8 + (e ? 2 : 3), clock64());
            if (elect_one()) {
                constexpr int kPad = e ? kPad1 : kPad0;
                constexpr uint32_t kIdesc = make_idesc<kKindI8>(64, kPad);
                const uint32_t t_proj = tmem + 4 * NB + (e ? kPad0 : 0);
                const uint64_t d_h = d_h0 + uint64_t(e * (h_group1 >> 4));
                // an MMA is 8 to 12 cycles with its weights in tensor memory, 27 from shared memory
#pragma unroll
                for (int kb = 0; kb < C; ++kb)
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint64_t rows = d_h + uint64_t(kb * kPad * 8 + 2 * k);
                        if (kb < kDnTs)
                            tc_mma_ts<kKindI8>(t_proj, tmem + kGTmemW - 32 * (kb + 1) + 8 * k, rows, kIdesc, (kb | k) != 0);
                        else
                            tc_mma<kKindI8>(t_proj, d_dn + uint64_t((kb - kDnTs) * 512 + 2 * k), rows, kIdesc, (kb | k) != 0);
                    }
                tc_commit(&bar_proj[e]);
                if (i + 1 < p.T) mbar_arrive_expect_tx(&bar_h[e], uint32_t(own_of(e)) * H);  // arm the next step
            }
            __syncwarp();
            return true;
        };
        auto hh_half = [&](auto group) {
            constexpr int e = decltype(group)::value;
            constexpr uint32_t kIdesc = make_idesc<kKindF16>(128, e ? N1 : N0);
            ok = ok && mbar_wait<true>(&bar_hh[e], i & 1, abort_flag, 101);
            if (!ok) return false;
            fence_proxy_async_smem();
            tc_fence_after_sync();
            FLUKE_STAMP(blockIdx.x == 0 && lane == 0, i * 8 + (e ? 7 : 6), clock64());
            if (elect_one()) {
                const uint64_t d_hh = d_hh0 + uint64_t(e * (N0 * 8));
#pragma unroll
                for (int g = 0; g < 4; ++g)
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        tc_mma_ts<kKindF16>(tmem + g * NB + e * N0, tmem + kGTmemW + g * 64 + k * 8,
                                            d_hh + uint64_t((k >> 2) * (NB * 8) + 2 * (k & 3)), kIdesc, 1u);
                tc_commit(&bar_acc[e]);
                if (i + 1 < p.T) mbar_arrive_expect_tx(&bar_hh[e], uint32_t(rows_of(e)) * 256);
            }
            __syncwarp();
            return true;
        };
        for (; i < p.T && ok; ++i) {
            // Fresh values in every step: hoisted out of the loop, the operands of its MMAs would fill
            // more registers than there are.
            asm volatile("" : "+l"(d_wx), "+l"(d_x0), "+l"(d_hh0), "+l"(d_dn), "+l"(d_h0));
            if constexpr (G == 1) {
                // half of the x part while the hidden state is computed and travels, half while the
                // projection is converted and travels
                if (!wait_x()) break;
                x_half(Int<0>{}, Int<2>{});
                if (!wait_h(0) || !project(Int<0>{})) break;
                x_half(Int<2>{}, Int<4>{});
                if (!hh_half(Int<0>{})) break;
            } else {
                // Pieces of the x part while the hidden rows of the groups travel, one gate while the second
                // projection is converted. 1024 chunks, gates in front of the first projection, between and
                // behind: 1-2-1 2.87 us per step, 1-1-2 3.02, 0-3-1 2.94, 1-3-0 3.02, 0-4-0 3.00.
                if (!wait_x()) break;
                x_half(Int<0>{}, Int<1>{});
                if (!wait_h(0)) break;
                project(Int<0>{});
                x_half(Int<1>{}, Int<3>{});
                if (!wait_h(1)) break;
                project(Int<1>{});
                x_half(Int<3>{}, Int<4>{});
                if (!hh_half(Int<0>{})) break;
                if (!hh_half(Int<1>{})) break;
            }
        }
    } else {
        // ------------------------------ epilogues ---------------------------------------
        const int q = warp & 3, ug = (warp - 2) >> 2;
        // gates: this warp's rows of a group (an even share, so that rows pair up)
        auto share_of = [&](int e) {
            const int most = G == 1 ? p.rows : e == 0 ? min(p.rows, N0) : p.rows - N0;
            return max((most + 3) / 4 + 1, 0) & ~1;
        };
        auto r0_of = [&](int e) { return e * N0 + ug * share_of(e); };   // in the cluster's rows
        auto my_rows_of = [&](int e) { return min(max(rows_of(e) - ug * share_of(e), 0), share_of(e)); };
        // projection: its columns (= rows) of the pair's accumulator
        auto pr0_of = [&](int e) { return ug * ((p.n_own[e] + 3) / 4); };
        auto my_pr_of = [&](int e) { return projects ? min(max(own_of(e) - pr0_of(e), 0), (p.n_own[e] + 3) / 4) : 0; };

        const int unit = n0 + q * 32 + lane;
        const float b_i = __ldg(p.bias + unit), b_f = __ldg(p.bias + H + unit);
        const float b_g = __ldg(p.bias + 2 * H + unit), b_o = __ldg(p.bias + 3 * H + unit);
        // one projection column per lane (16 lanes of a quadrant hold rows of an M = 64 accumulator)
        const int r_col = half * 64 + q * 16 + (lane & 15);
        const float sc = (1.0f / 127.0f) * __ldg(p.dn_scale + r_col);  // operand order of the dequant GEMM: sa * sb
        float2 c2[G][kCols / 2];
#pragma unroll
        for (int e = 0; e < G; ++e)
#pragma unroll
            for (int j = 0; j < kCols / 2; ++j) {
                const float *cp = p.c + int64_t(m0 + r0_of(e) + 2 * j) * H + unit;
                const int n = my_rows_of(e);
                c2[e][j] = make_float2(2 * j < n ? cp[0] : 0.f, 2 * j + 1 < n ? cp[H] : 0.f);
            }

        // What a CTA sends leaves in rows of 128 bytes, eight lanes each: the network between the SMs moves 64
        // contiguous bytes to one CTA in the time of 16 (20.7 against 9.5 B per cycle and SM, measured with
        // six CTAs sending to each other). A warp holds 32 bytes of a row, so the four warps of a quarter stage
        // together, in two slots in turn: the barrier after one batch is staged also says that the slot of
        // the batch before has been read.
        const uint32_t stage = smem_u32(smem + L.stage) + ug * (kStageRows * 128);
        uint32_t slot = 0;
        auto next_slot = [&]() { slot ^= 4 * kStageRows * 128; };
        // The stores of every step go to the same places: addresses are worked out once. A destination is
        // 16-byte aligned; its low bits hold the peer's rank (the peer's mbarrier address follows from
        // it), 8 marks one that exists. Lane 8 j + c stores piece c of the swizzled row.
        uint32_t hs_dst[G][kBatches];   // lanes 0-15: row q of a batch of four, to both CTAs of the pair
#pragma unroll
        for (int e = 0; e < G; ++e)
#pragma unroll
            for (int b = 0; b < (e ? N1 : N0) / 16; ++b) {
                const int row = 4 * b + q, at = ug * share_of(e) + row;
                const int pr = at / p.n_own[e], lr = at - pr * p.n_own[e];
                const uint32_t to = uint32_t(2 * pr + (lane >> 3));
                hs_dst[e][b] = lane < 16 && row < my_rows_of(e)
                    ? map_to_rank(smem_u32(smem + L.h + e * h_group1 + rank * ((e ? kPad1 : kPad0) * 128)) + lr * 128 + (lane & 7) * 16, to) | 8u | to
                    : 0u;
            }
        // ceil(ceil(N / pairs) / 4) rows to C CTAs each: at most 12 (row, CTA) per 16 rows (C = 3), 16 per store
        uint32_t ps_src[kSendP], ps_dst[G][kSendP];
#pragma unroll
        for (int s = 0; s < kSendP; ++s) {
            const int id = 16 * s + 4 * q + (lane >> 3), row = id / C;
            int to = id - row * C + rank;   // start with a different peer in every CTA
            if (to >= C) to -= C;
            ps_src[s] = row * 128;
#pragma unroll
            for (int e = 0; e < G; ++e)
                ps_dst[e][s] = row < my_pr_of(e)
                    ? map_to_rank(smem_u32(smem + L.hh + half * (NB * 128)) +
                                      (e * N0 + pair * p.n_own[e] + pr0_of(e) + row) * 128 + (lane & 7) * 16, uint32_t(to)) | 8u | uint32_t(to)
                    : 0u;
        }
        // the piece of a staged row that belongs at a destination of the 128-byte swizzle
        auto piece = [&](uint32_t dst) { return (uint32_t(lane) ^ (dst >> 7)) & 7u; };
        auto send = [&](uint32_t dst, uint4 v, uint64_t *bar) {
            store_to_peer(dst & ~15u, v, map_to_rank(smem_u32(bar), dst & 7u));
        };
        const uint32_t t_lane = tmem + (uint32_t(q * 32) << 16);
        int i = 0;
        // A warp whose wait ran out walks the remaining steps without waiting, sending or storing: the
        // three it shares a slot with meet it at every barrier until their own waits give up.
        bool ok = true;
        const int64_t plane = int64_t(p.reverse ? -p.B : p.B) * H;
        int8_t *h_out = p.h_out + int64_t(time_of(0)) * p.B * H;

        // ---- projection of group e's h_{i-1}: int32 -> f16, to every CTA of the cluster ----
        auto project_epilogue = [&](auto group) {
            constexpr int e = decltype(group)::value;
            const int my_pr = my_pr_of(e);
            if (my_pr > 0) {
                ok = ok && mbar_wait(&bar_proj[e], i & 1, abort_flag, 102);
                next_slot();
                FLUKE_STAMP(blockIdx.x == 0 && threadIdx.x == 64 && e == 0, i * 8 + 4, clock64());
                tc_fence_after_sync();
                const uint32_t t_proj = t_lane + 4 * NB + (e ? kPad0 : 0) + pr0_of(e);
                for (int c = 0; c < my_pr; c += 4) {
                    uint32_t a[4];
                    tmem_ld_32x4(t_proj + c, a);
                    tmem_ld_wait();
                    if (lane < 16) {
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            if (c + j < my_pr)
                                sts16(stage + slot + (c + j) * 128 + q * 32 + lane * 2, __half_as_ushort(__float2half_rn(float(int(a[j])) * sc)));
                    }
                }
                tc_fence_before_sync();
                quad_sync(1 + ug);
#pragma unroll
                for (int s = 0; s < (e ? N1 : N0) / 16; ++s)
                    if (const uint32_t dst = ok ? ps_dst[e][s] : 0u) send(dst, lds128(stage + slot + ps_src[s] + piece(dst) * 16), &bar_hh[e]);
                FLUKE_STAMP(blockIdx.x == 0 && threadIdx.x == 64 && e == 0, i * 8 + 5, clock64());
            }
        };

        // ---- gates, cell update, hidden code of group e ----
        auto gate_epilogue = [&](auto group) {
            constexpr int e = decltype(group)::value;
            constexpr int kB = (e ? N1 : N0) / 16;
            const int my_rows = my_rows_of(e), r0 = r0_of(e);
            ok = ok && mbar_wait(&bar_acc[e], i & 1, abort_flag, 103);
            FLUKE_STAMP(blockIdx.x == 0 && threadIdx.x == 64 && e == 0, i * 8 + 0, clock64());
            tc_fence_after_sync();
            // Four rows at a time, and each batch is sent as soon as it is staged (and stored, 128 bytes of a
            // row by eight lanes), so that the exchange runs beside the arithmetic. Two batches are read at the
            // start, which hands the accumulators back before the arithmetic.
            static_assert(kB <= 2, "two batches are in registers");
            uint32_t a[2][4][4];
            auto load4 = [&](int b) {
#pragma unroll
                for (int g = 0; g < 4; ++g) tmem_ld_32x4(t_lane + g * NB + r0 + 4 * b, a[b & 1][g]);
            };
            load4(0);
            if (kB > 1) load4(1);
            tmem_ld_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (e == G - 1 && lane == 0) mbar_arrive(bar_acc_free);
#pragma unroll
            for (int b = 0; b < kB; ++b) {
                const auto &v = a[b & 1];
                if (b > 0 && 4 * b >= my_rows) break;
                next_slot();
                if (4 * b < my_rows) {
                    auto codes = [&](int j) {
                        return lstm_cell_codes(v[0][2 * j], v[0][2 * j + 1], v[1][2 * j], v[1][2 * j + 1], v[2][2 * j], v[2][2 * j + 1],
                                               v[3][2 * j], v[3][2 * j + 1], make_float2(b_i, b_i), make_float2(b_f, b_f),
                                               make_float2(b_g, b_g), make_float2(b_o, b_o), c2[e][2 * b + j]);
                    };
                    auto stage_codes = [&](int j, int2 h) {
                        sts8(stage + slot + 2 * j * 128 + q * 32 + lane, h.x);
                        sts8(stage + slot + (2 * j + 1) * 128 + q * 32 + lane, h.y);
                    };
                    // Both pairs side by side: two chains. The second is left out where its rows do not exist.
                    // With the branch against without, us per step, x_down included: C = 6 7 rows per cluster 1.53 :
                    // 1.62, 14 rows 1.67 : 1.70, 20 rows 2.25 : 2.37; C = 7 and 8 alike (7 rows 1.57 : 1.67, 1.63 :
                    // 1.70), 10 rows 1 % slower. Two groups, 47 rows: 3.02 : 2.98, so not there. C = 2 and 3 go without:
                    // between -5 % (7 rows 1.47 : 1.55) and +1 % (10 and 16 rows).
                    if (G > 1 || C < 4 || 4 * b + 2 < my_rows) {
                        const int2 h0 = codes(0), h1 = codes(1);
                        stage_codes(0, h0);
                        stage_codes(1, h1);
                    } else {
                        stage_codes(0, codes(0));
                    }
                }
                quad_sync(1 + ug);
                if (const uint32_t dst = ok ? hs_dst[e][b] : 0u) {
                    const uint4 v = lds128(stage + slot + q * 128 + piece(dst) * 16);
                    if (i + 1 < p.T) send(dst, v, &bar_h[e]);
                    if (lane < 8) {
                        const size_t off = size_t(m0 + r0 + 4 * b + q) * H + n0 + piece(dst) * 16;
                        *reinterpret_cast<uint4 *>(h_out + off) = v;
                        if (i + 1 == p.T) *reinterpret_cast<uint4 *>(p.h_state + off) = v;
                    }
                }
            }
            FLUKE_STAMP(blockIdx.x == 0 && threadIdx.x == 64 && e == 0, i * 8 + 1, clock64());
        };

        for (; i < p.T; ++i, h_out += plane) {
            project_epilogue(Int<0>{});
            if constexpr (G > 1) project_epilogue(Int<1>{});
            gate_epilogue(Int<0>{});
            if constexpr (G > 1) gate_epilogue(Int<1>{});
        }
#pragma unroll
        for (int e = 0; e < G; ++e)
#pragma unroll
            for (int j = 0; j < kCols / 2; ++j) {
                float *cp = p.c + int64_t(m0 + r0_of(e) + 2 * j) * H + unit;
                const int n = my_rows_of(e);
                if (2 * j < n) cp[0] = c2[e][j].x;
                if (2 * j + 1 < n) cp[H] = c2[e][j].y;
            }
    }

    // Nobody leaves (and frees shared memory that a peer's store may still target) before every
    // CTA of the cluster is done.
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after_sync();
        tmem_dealloc(tmem, kGTmemCols);
    }
}

// ---- host side ---------------------------------------------------------------------------------

constexpr int kGMinRows = 2;  // fewer rows than this per cluster do not make a step shorter

struct GroupPlan {
    int kernel;       // index in kGroupKernels
    int rows;         // rows per cluster
    int tiles;        // clusters
};

using group_kernel_fn = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, GroupDev);
struct GroupKernel { int n0, n1; group_kernel_fn fn[kGMaxCtas + 1]; };
// Rows per cluster from which two groups are the faster: see group_kernel_for.
constexpr int group_two_from(int C) { return C == 3 ? 17 : 18 + 2 * C; }
template <int N0, int N1, int C>
constexpr group_kernel_fn group_kernel_fits() {
    constexpr bool kUsed = N1 == 0 || N0 + N1 > 32 || group_two_from(C) <= N0 + N1;
    if constexpr (kUsed && group_layout(N0, N1, C).dynamic <= kGMaxSmem) return lstm_group_kernel<N0, N1, C>;
    else return nullptr;
}
template <int N0, int N1>
constexpr GroupKernel group_kernels() {
    return {N0, N1, {nullptr, nullptr, group_kernel_fits<N0, N1, 2>(), group_kernel_fits<N0, N1, 3>(), group_kernel_fits<N0, N1, 4>(),
                     group_kernel_fits<N0, N1, 5>(), group_kernel_fits<N0, N1, 6>(), group_kernel_fits<N0, N1, 7>(),
                     group_kernel_fits<N0, N1, 8>()}};
}
const GroupKernel kGroupKernels[] = {group_kernels<16, 0>(), group_kernels<32, 0>(), group_kernels<16, 16>(), group_kernels<16, 32>()};

// The kernel for `rows` rows per cluster of hidden size H, or -1. One group has the shorter chain, two hide
// half of it: the longer the exchanges (more CTAs), the more rows it takes for two to be the faster. Step of one
// group against two, in us: H = 256, 20 rows 2.09 : 2.16, 28 rows 2.30 : 2.22; H = 384 (one pair of CTAs
// projects all rows), 17 rows 2.19 : 2.19, 20 rows 2.40 : 2.21; H = 512, 26 rows 2.36 : 2.35, 32 rows 2.52 : 2.36;
// H = 768, 28 rows 2.52 : 2.56, 32 rows 2.65 : 2.56; H = 1024, 32 rows 2.75 : 2.80.
inline int group_kernel_for(int rows, int H) {
    const int C = H / kGUnits;
    const int k = rows <= 16 ? 0 : rows <= 32 ? (rows < group_two_from(C) ? 1 : 2) : 3;
    return rows <= 48 && kGroupKernels[k].fn[C] ? k : -1;
}

// Clusters of C CTAs of kernel k that the device runs at once with the largest shared memory a CTA can
// have (0: the form is not available).
int group_capacity(int k, int C) {
    static int known[64][sizeof(kGroupKernels) / sizeof(kGroupKernels[0])][kGMaxCtas + 1];  // n + 1, or -1
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return 0;
    int &slot = known[dev][k][C];
    if (slot == 0) {
        int n = 0;
        const void *fn = reinterpret_cast<const void *>(kGroupKernels[k].fn[C]);
        bool ok = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kGMaxSmem) == cudaSuccess;
        if (ok) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(C);
            cfg.blockDim = dim3(kGThreads);
            cfg.dynamicSmemBytes = kGMaxSmem;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = C;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            ok = cudaOccupancyMaxActiveClusters(&n, fn, &cfg) == cudaSuccess && n > 0;
        }
        cudaGetLastError();  // a refused attribute must not linger as the thread's last error
        slot = ok ? n + 1 : -1;
    }
    return slot > 0 ? slot - 1 : 0;
}

// How B rows of hidden size H are spread: as few waves of clusters as the largest row count that
// fits shared memory allows, then evenly over all clusters of those waves.
bool group_plan(int B, int H, GroupPlan *g) {
    if (H % kGUnits) return false;
    const int C = H / kGUnits;
    if (C < 2 || C > kGMaxCtas) return false;
    int max_rows = 48;
    while (max_rows > 0 && (g->kernel = group_kernel_for(max_rows, H)) < 0) max_rows -= 16;
    if (max_rows < 16) return false;
    const int cap = group_capacity(g->kernel, C);
    if (cap < 1) return false;
    const int waves = (B + cap * max_rows - 1) / (cap * max_rows);
    int tiles = cap * waves;
    if (tiles > (B + kGMinRows - 1) / kGMinRows) tiles = (B + kGMinRows - 1) / kGMinRows;
    g->rows = (B + tiles - 1) / tiles;
    g->tiles = (B + g->rows - 1) / g->rows;
    g->kernel = group_kernel_for(g->rows, H);
    return g->kernel >= 0 && group_capacity(g->kernel, C) > 0;
}

}  // namespace
}  // namespace fluke_sm100

// Runs the recurrence of one layer (x_down already computed) with the batch spread over small
// clusters, and writes the final hidden state. Returns -2 when the shape or the device is not covered.
extern "C" int fluke_sm100_lstm_layer_group(const void *layer, const void *x_down, void *stream) {
    using namespace fluke_sm100;
    const fluke_flstm_layer_t *l = static_cast<const fluke_flstm_layer_t *>(layer);
    const int T = l->T, B = l->B, H = l->H, R = l->R;
    GroupPlan g;
    if (R != kGRank || !group_plan(B, H, &g)) return -2;
    const GroupKernel &kn = kGroupKernels[g.kernel];
    const int C = H / kGUnits;

    GroupDev p;
    p.T = T; p.B = B; p.reverse = l->reverse;
    p.rows = g.rows;
    const int in_group[2] = {kn.n1 ? min(g.rows, kn.n0) : g.rows, kn.n1 ? max(g.rows - kn.n0, 0) : 0};
    for (int e = 0; e < 2; ++e) p.n_own[e] = max((in_group[e] + C / 2 - 1) / (C / 2), 1);
    p.dn = static_cast<const int8_t *>(l->dn_hh_i8);
    p.w_up = static_cast<const __half *>(l->w_up_f16);
    p.bias = static_cast<const float *>(l->bias_f32);
    p.dn_scale = static_cast<const float *>(l->dn_hh_scale);
    p.c = static_cast<float *>(l->c_f32);
    p.h_out = static_cast<int8_t *>(l->h_out_i8);
    p.h_state = static_cast<int8_t *>(l->h_i8);
    p.trace = trace_buffer();

    CUtensorMap tm_w, tm_x, tm_dn, tm_h[2];
    int rc = make_tmap_2d(&tm_w, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, l->w_up_f16, 4 * uint64_t(H), 2 * R, uint64_t(2 * R) * 2,
                          kGUnits, 64, true);
    if (rc) return rc;
    {
        // both K blocks of a row range in one box: the 128-byte blocks of a row are a dimension
        const uint64_t dims[4] = {64, uint64_t(B), 2, uint64_t(T)};
        const uint64_t strides[3] = {uint64_t(R) * 2, 128, uint64_t(B) * R * 2};
        const uint32_t box[4] = {64, uint32_t(kn.n0 + kn.n1), 2, 1};
        rc = make_tmap_nd(&tm_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, x_down, 4, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
        if (rc) return rc;
    }
    rc = make_tmap_2d(&tm_dn, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, l->dn_hh_i8, R, H, H, 64, 128, true);
    if (rc) return rc;
    for (int e = 0; e < 2; ++e) {
        const uint64_t dims[3] = {128, uint64_t(B), uint64_t(C)};
        const uint64_t strides[2] = {uint64_t(H), 128};
        const uint32_t box[3] = {128, uint32_t(group_h_rows(e && kn.n1 ? kn.n1 : kn.n0, C)), uint32_t(C)};
        rc = make_tmap_nd(&tm_h[e], CU_TENSOR_MAP_DATA_TYPE_UINT8, l->h_i8, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
        if (rc) return rc;
    }

    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(g.tiles * C);
    cfg.blockDim = dim3(kGThreads);
    cfg.dynamicSmemBytes = group_layout(kn.n0, kn.n1, C).dynamic;
    cfg.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, kn.fn[C], tm_w, tm_x, tm_dn, tm_h[0], tm_h[1], p);
}
