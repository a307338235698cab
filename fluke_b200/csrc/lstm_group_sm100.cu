// lstm_group_sm100.cu -- the recurrence of a factored-LSTM layer as many small thread-block
// clusters, each with a FEW chunk rows: the batch is spread over all clusters the device holds
// instead of being packed into 128-row tiles.
//
// A step is a chain of dependent stages, so its time is set by what each stage of one cluster has
// to move and compute for its own rows. With the rows as the M = 128 dimension of the
// contractions that amount does not shrink with the batch; here the operands are swapped. The
// WEIGHTS are the M dimension (128 hidden units per CTA, one accumulator block per gate) and the
// chunk rows are N = 16, 32 or 48 columns, and the recurrent half of the gate weights lives in
// TENSOR MEMORY as the A operand: an MMA then costs N/2 cycles (8 for N = 16) instead of the 33 that
// reading a 128-row A operand from shared memory takes whatever N is.
//
// A cluster has C = H / 128 CTAs (2 to 8). CTA j
//   * owns units 128 j .. 128 j + 127: their four gate weight blocks (hh half in tensor memory, x
//     half in shared memory) and, in registers, their cell state for the cluster's rows;
//   * projects: the CTAs form pairs (2p, 2p+1); pair p owns a contiguous part of the rows, CTA
//     2p + s computes projection columns 64 s .. 64 s + 63 of them (M = 64) from the complete
//     int8 rows. With an odd C the last CTA projects nothing.
// Per step two exchanges inside the cluster, both of 16-byte st.async stores that complete on an
// mbarrier of the receiver: the int8 hidden slices go to the pair that owns the row, the
// f16 projections back to every CTA. The x half of the next step's contraction runs meanwhile.
//
//   warp 0       loader: resident weights, x_down rows of every step
//   warp 1       MMA issuer
//   warps 2-17   epilogues, four per tensor-memory lane quadrant: thread = hidden unit, a quarter
//                of the rows each (gates, cell update, int8 code); the same warps turn the
//                projection accumulators into f16 and send them
//
// A buffer is only overwritten after its reader has provably finished: a CTA sends h_t after its
// gate contraction of step t, which needs hh_t from every pair, which a pair sends after its
// projection of h_{t-1} is complete; and the other way round for hh. Nobody leaves before the final
// cluster barrier. Clusters never wait for one another, so any number of them may run in waves.
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

struct GroupDev {
    int T, B, H;
    int reverse;
    int rows;                  // chunk rows per cluster (the last cluster may have fewer)
    int n_own, n_pad;          // rows a pair projects; the same rounded up to a multiple of 8
    int dn_ts;                 // K blocks of the projection weights kept in tensor memory
    const int8_t *dn;          // [R, H]
    const __half *w_up;        // [4H, 2R]
    const float *bias;         // [4H]
    const float *dn_scale;     // [R]
    float *c;                  // [B,H]
    int8_t *h_out;             // [T,B,H]
    int8_t *h_state;           // [B,H]: final hidden state
    long long *trace;          // trace builds only: [T][8] SM-clock stamps of CTA 0
};

// Shared-memory layout; the row-dependent parts are sized at launch.
struct GroupLayout {
    int x, hh, dn, h, stage, bars, misc, dynamic;
};
// K blocks (128 hidden units, 32 columns) of the projection weights that fit in tensor memory beside
// the gate weights and the accumulators.
__host__ __device__ constexpr int group_dn_ts(int nb, int H, int n_pad) {
    const int fit = (kGTmemW - 4 * nb - n_pad) / 32;
    return fit < H / kGUnits ? fit : H / kGUnits;
}
__host__ __device__ constexpr GroupLayout group_layout(int nb, int H, int n_pad) {
    GroupLayout l = {};
    l.x = kGWxBytes;                  // x_down rows of two steps: 2 K blocks [nb x 128 B] each
    l.hh = l.x + 2 * nb * 256;        // hh_down rows, the same shape
    l.dn = l.hh + nb * 256;           // 64 projection rows: the other K blocks [64 x 128 B]
    l.h = l.dn + 64 * (H - 128 * group_dn_ts(nb, H, n_pad));              // hidden rows of the pair: H/128 K blocks [n_pad x 128 B]
    l.stage = l.h + n_pad * H;        // 16 warps x (nb/4 rows x 32 B)
    l.bars = l.stage + nb * 128;
    l.misc = l.bars + 10 * 8;
    l.dynamic = l.misc + 16 + 1024;   // slack for the manual 1024-byte alignment
    return l;
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

template <int NB>
__global__ void __launch_bounds__(kGThreads, 1)
lstm_group_kernel(const __grid_constant__ CUtensorMap tm_w,    // w_up [4H, 2R] f16, boxes 128 x 64
                  const __grid_constant__ CUtensorMap tm_x,    // x_down [T, 2, B, 64] f16, boxes of NB rows
                  const __grid_constant__ CUtensorMap tm_dn,   // dn_hh [R, H] int8, boxes 64 x 128
                  const __grid_constant__ CUtensorMap tm_h0,   // h_0 [H/128, B, 128] int8, boxes of n_pad rows
                  const GroupDev p) {
    constexpr int kCols = NB / 4;                    // rows an epilogue thread holds at most
    constexpr int kBatches = kCols / 4;              // it takes them four at a time
    constexpr int kSendP = NB / 16;                  // 16-byte stores per lane and step, projections
    static_assert(NB % 16 == 0 && 4 * NB + NB <= kGTmemW, "accumulators beside the weights in tensor memory");
    extern __shared__ uint8_t smem_raw[];
    // every CTA of the cluster computes the same offset, so peers' buffers are at the same
    // shared-window offsets as this CTA's
    uint8_t *smem = reinterpret_cast<uint8_t *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const GroupLayout L = group_layout(NB, p.H, p.n_pad);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L.bars);
    uint64_t *bar_once = &bars[0];       // resident weights loaded
    uint64_t *bar_x = &bars[1];          // [2] x_down rows landed
    uint64_t *bar_x_free = &bars[3];     // [2] x half of the contraction has read them
    uint64_t *bar_h = &bars[5];          // complete hidden rows of the pair arrived
    uint64_t *bar_proj = &bars[6];       // projection accumulator complete
    uint64_t *bar_hh = &bars[7];         // hh_down rows arrived
    uint64_t *bar_acc = &bars[8];        // gate accumulators complete
    uint64_t *bar_acc_free = &bars[9];   // epilogue has read them
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + L.misc);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + L.misc + 4);

    const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x) >> 5, 0), lane = threadIdx.x & 31;
    const int C = p.H / kGUnits;
    const int rank = int(cluster_ctarank());
    const int pair = rank >> 1, half = rank & 1;
    const bool projects = rank < (C & ~1);
    const int m0 = (blockIdx.x / C) * p.rows;          // first chunk row of the cluster
    const int n_rows = min(p.rows, p.B - m0);          // and how many it has
    const int n_own = min(max(n_rows - pair * p.n_own, 0), p.n_own);  // rows this CTA projects
    const int n0 = rank * kGUnits;
    auto time_of = [&](int i) { return p.reverse ? p.T - 1 - i : i; };

    if (threadIdx.x == 0) {
        for (int b = 0; b < 9; ++b) mbar_init(&bars[b], 1);
        mbar_init(bar_acc_free, kGEpiWarps);
        *abort_flag = 0;
        fence_barrier_init();
        mbar_arrive_expect_tx(bar_hh, uint32_t(n_rows) * 256);
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
            p.w_up + (size_t(g) * p.H + n0 + q * 32 + lane) * (2 * kGRank));
        const uint32_t t_lane = tmem + (uint32_t(q * 32) << 16) + kGTmemW;
#pragma unroll 1
        for (int v = 0; v < 8; ++v) tmem_st_32x8(t_lane + g * 64 + v * 8, __ldg(src + 2 * v), __ldg(src + 2 * v + 1));
        if (projects) {
            // and K blocks g, g + 4, .. of the projection rows (M = 64: row 16 q + i in lane 32 q + i)
            const uint4 *dn = reinterpret_cast<const uint4 *>(p.dn + size_t(half * 64 + q * 16 + (lane & 15)) * p.H);
            for (int kb = g; kb < p.dn_ts; kb += 4)
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
            mbar_arrive_expect_tx(bar_once, kGWxBytes + (projects ? (C - p.dn_ts) * 8192 : 0));
            for (int g = 0; g < 4; ++g)
                for (int kb = 0; kb < 2; ++kb)
                    tma_load_2d(smem + (g * 2 + kb) * 16384, &tm_w, bar_once, kGRank + kb * 64, g * p.H + n0);
            if (projects) {
                for (int kb = p.dn_ts; kb < C; ++kb)
                    tma_load_2d(smem + L.dn + (kb - p.dn_ts) * 8192, &tm_dn, bar_once, kb * 128, half * 64);
                // step 0 projects the layer's initial hidden state
                mbar_arrive_expect_tx(bar_h, uint32_t(p.n_pad) * p.H);
                tma_load_3d(smem + L.h, &tm_h0, bar_h, 0, m0 + pair * p.n_own, 0);
            }
            bool ok = true;
            for (int i = 0; i < p.T && ok; ++i) {
                if (i > 1) ok = mbar_wait(&bar_x_free[i & 1], ((i >> 1) - 1) & 1, abort_flag, 96);
                if (!ok) break;
                mbar_arrive_expect_tx(&bar_x[i & 1], NB * 256);
                tma_load_4d(smem + L.x + (i & 1) * (NB * 256), &tm_x, &bar_x[i & 1], 0, m0, 0, time_of(i));
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------ MMA issuer --------------------------------------
        // The whole warp walks the loop; one elected lane issues. Descriptors are uniform and the
        // K loops unrolled, so an MMA is issued every few cycles.
        constexpr uint32_t kIdescGate = make_idesc<kKindF16>(128, NB);
        const uint32_t idesc_proj = make_idesc<kKindI8>(64, 0) | (uint32_t(p.n_pad >> 3) << 17);
        uint64_t d_wx = make_smem_desc_sw128(smem_u32(smem));
        uint64_t d_hh = make_smem_desc_sw128(smem_u32(smem + L.hh));
        uint64_t d_dn = make_smem_desc_sw128(smem_u32(smem + L.dn));
        uint64_t d_h = make_smem_desc_sw128(smem_u32(smem + L.h));
        uint64_t d_x = 0;
        const uint32_t t_proj = tmem + 4 * NB;
        // The x half of gates [g0, g1). Its 32 MMAs read their A operand from shared memory (33
        // cycles each, a third of a step in all) and the tensor pipe works in order: half of them go in front
        // of the projection, while the hidden state is computed and travels, half behind it, while
        // the projection is converted and travels.
        auto x_half = [&](int g0, int g1) {
#pragma unroll
            for (int g = g0; g < g1; ++g)
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    tc_mma<kKindF16>(tmem + g * NB, d_wx + uint64_t((g * 2 + (k >> 2)) * 1024 + 2 * (k & 3)),
                                     d_x + uint64_t((k >> 2) * (NB * 8) + 2 * (k & 3)), kIdescGate, k != 0);
        };
        bool ok = mbar_wait(bar_once, 0, abort_flag, 97);
        for (int i = 0; i < p.T && ok; ++i) {
            if (i > 0) ok = mbar_wait(bar_acc_free, (i - 1) & 1, abort_flag, 98);
            if (!ok) break;
            ok = mbar_wait(&bar_x[i & 1], (i >> 1) & 1, abort_flag, 99);
            if (!ok) break;
            tc_fence_after_sync();
            // Fresh values in every step: hoisted out of the loop, the operands of its MMAs would fill
            // more registers than there are.
            d_x = make_smem_desc_sw128(smem_u32(smem + L.x)) + uint64_t((i & 1) * (NB * 16));
            asm volatile("" : "+l"(d_wx), "+l"(d_x), "+l"(d_hh), "+l"(d_dn), "+l"(d_h));
            if (elect_one()) x_half(0, 2);
            __syncwarp();
            if (projects) {
                ok = mbar_wait<true>(bar_h, i & 1, abort_flag, 100);
                if (!ok) break;
                fence_proxy_async_smem();   // the peers' stores are generic-proxy writes
                tc_fence_after_sync();
                FLUKE_STAMP(blockIdx.x == 0 && lane == 0, i * 8 + 3, clock64());
                if (elect_one()) {
                    // an MMA is 8 to 12 cycles with its weights in tensor memory, 24 from shared memory
                    for (int kb = 0; kb < p.dn_ts; ++kb)
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            tc_mma_ts<kKindI8>(t_proj, tmem + kGTmemW - 32 * (kb + 1) + 8 * k,
                                               d_h + uint64_t(kb * p.n_pad * 8 + 2 * k), idesc_proj, (kb | k) != 0);
                    for (int kb = p.dn_ts; kb < C; ++kb)
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            tc_mma<kKindI8>(t_proj, d_dn + uint64_t((kb - p.dn_ts) * 512 + 2 * k),
                                            d_h + uint64_t(kb * p.n_pad * 8 + 2 * k), idesc_proj, (kb | k) != 0);
                    tc_commit(bar_proj);
                    if (i + 1 < p.T) mbar_arrive_expect_tx(bar_h, uint32_t(n_own) * p.H);  // arm the next step
                }
                __syncwarp();
            }
            if (elect_one()) {
                x_half(2, 4);
                tc_commit(&bar_x_free[i & 1]);
            }
            __syncwarp();
            ok = mbar_wait<true>(bar_hh, i & 1, abort_flag, 101);
            if (!ok) break;
            fence_proxy_async_smem();
            tc_fence_after_sync();
            FLUKE_STAMP(blockIdx.x == 0 && lane == 0, i * 8 + 6, clock64());
            if (elect_one()) {
#pragma unroll
                for (int g = 0; g < 4; ++g)
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        tc_mma_ts<kKindF16>(tmem + g * NB, tmem + kGTmemW + g * 64 + k * 8,
                                            d_hh + uint64_t((k >> 2) * (NB * 8) + 2 * (k & 3)), kIdescGate, 1u);
                tc_commit(bar_acc);
                if (i + 1 < p.T) mbar_arrive_expect_tx(bar_hh, uint32_t(n_rows) * 256);
            }
            __syncwarp();
        }
    } else {
        // ------------------------------ epilogues ---------------------------------------
        const int q = warp & 3, ug = (warp - 2) >> 2;
        // gates: this warp's rows of the cluster (an even share, so that rows pair up)
        const int share = ((p.rows + 3) / 4 + 1) & ~1;
        const int r0 = ug * share;
        const int my_rows = min(max(n_rows - r0, 0), share);
        // projection: its columns (= rows) of the pair's accumulator
        const int p_share = (p.n_own + 3) / 4;
        const int pr0 = ug * p_share;
        const int my_pr = projects ? min(max(n_own - pr0, 0), p_share) : 0;

        const int unit = n0 + q * 32 + lane;
        const float b_i = __ldg(p.bias + unit), b_f = __ldg(p.bias + p.H + unit);
        const float b_g = __ldg(p.bias + 2 * p.H + unit), b_o = __ldg(p.bias + 3 * p.H + unit);
        // one projection column per lane (16 lanes of a quadrant hold rows of an M = 64 accumulator)
        const int r_col = half * 64 + q * 16 + (lane & 15);
        const float sc = (1.0f / 127.0f) * __ldg(p.dn_scale + r_col);  // operand order of the dequant GEMM: sa * sb
        float2 c2[kCols / 2];
#pragma unroll
        for (int j = 0; j < kCols / 2; ++j) {
            const float *cp = p.c + int64_t(m0 + r0 + 2 * j) * p.H + unit;
            c2[j] = make_float2(2 * j < my_rows ? cp[0] : 0.f, 2 * j + 1 < my_rows ? cp[p.H] : 0.f);
        }

        // The stores of every step go to the same places: addresses are worked out once. An item of
        // the hidden slice is (row, 16 units, projection half); of the projection (row, 8 columns, CTA).
        const uint32_t stage = smem_u32(smem + L.stage) + (warp - 2) * (kCols * 32);
        // A destination is 16-byte aligned; its low bits hold the peer's rank (the peer's mbarrier
        // address follows from it), 8 marks an item that exists.
        uint32_t hs_dst[kBatches];   // lanes 0-15, one store per batch of four rows
#pragma unroll
        for (int b = 0; b < kBatches; ++b) {
            const int row = 4 * b + (lane >> 2), ch = (lane >> 1) & 1;
            const int pr = (r0 + row) / p.n_own, lr = (r0 + row) - pr * p.n_own;
            const uint32_t to = uint32_t(2 * pr + (lane & 1));
            hs_dst[b] = lane < 16 && row < my_rows
                ? map_to_rank(smem_u32(smem + L.h + rank * (p.n_pad * 128)) + sw128_offset(lr, 2 * q + ch), to) | 8u | to
                : 0u;
        }
        // ceil(ceil(NB / pairs) / 4) rows of 2 C items each: at most 24 items per 16 rows (C = 3)
        uint32_t ps_src[kSendP], ps_dst[kSendP];
#pragma unroll
        for (int s = 0; s < kSendP; ++s) {
            const int id = lane + 32 * s, row = id / (2 * C), rest = id - row * 2 * C, ch = rest >= C ? 1 : 0;
            int to = rest - ch * C + rank;   // start with a different peer in every CTA
            if (to >= C) to -= C;
            ps_src[s] = stage + row * 32 + ch * 16;
            ps_dst[s] = row < my_pr
                ? map_to_rank(smem_u32(smem + L.hh + half * (NB * 128)) + sw128_offset(pair * p.n_own + pr0 + row, 2 * q + ch),
                              uint32_t(to)) | 8u | uint32_t(to)
                : 0u;
        }
        auto send = [&](uint32_t dst, uint32_t src, uint64_t *bar) {
            if (dst) store_to_peer(dst & ~15u, lds128(src), map_to_rank(smem_u32(bar), dst & 7u));
        };
        // the hidden slice's 16-byte pieces in global memory: lane = (row, 16 units)
        const bool g_ok = (lane >> 1) < my_rows;
        const uint32_t g_src = stage + lane * 16;
        const int64_t g_off = int64_t(m0 + r0 + (lane >> 1)) * p.H + n0 + q * 32 + (lane & 1) * 16;

        const uint32_t t_lane = tmem + (uint32_t(q * 32) << 16);
        bool ok = true;
        for (int i = 0; i < p.T && ok; ++i) {
            if (my_pr > 0) {
                // ---- projection of h_{i-1}: int32 -> f16, to every CTA of the cluster ----
                ok = mbar_wait(bar_proj, i & 1, abort_flag, 102);
                if (!ok) break;
                FLUKE_STAMP(blockIdx.x == 0 && threadIdx.x == 64, i * 8 + 4, clock64());
                tc_fence_after_sync();
                for (int c = 0; c < my_pr; c += 4) {
                    uint32_t a[4];
                    tmem_ld_32x4(t_lane + 4 * NB + pr0 + c, a);
                    tmem_ld_wait();
                    if (lane < 16) {
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            if (c + j < my_pr)
                                sts16(stage + (c + j) * 32 + lane * 2, __half_as_ushort(__float2half_rn(float(int(a[j])) * sc)));
                    }
                }
                tc_fence_before_sync();
                __syncwarp();
#pragma unroll
                for (int s = 0; s < kSendP; ++s)
                    send(ps_dst[s], ps_src[s], bar_hh);
                FLUKE_STAMP(blockIdx.x == 0 && threadIdx.x == 64, i * 8 + 5, clock64());
                __syncwarp();
            }
            // ---- gates, cell update, hidden code ----
            ok = mbar_wait(bar_acc, i & 1, abort_flag, 103);
            if (!ok) break;
            FLUKE_STAMP(blockIdx.x == 0 && threadIdx.x == 64, i * 8 + 0, clock64());
            tc_fence_after_sync();
            // Four rows at a time: the next four leave tensor memory while these are computed, and
            // each batch is sent as soon as it is staged, so the exchange runs beside the arithmetic.
            uint32_t a[2][4][4];
            auto load4 = [&](int b) {
#pragma unroll
                for (int g = 0; g < 4; ++g) tmem_ld_32x4(t_lane + g * NB + r0 + 4 * b, a[b & 1][g]);
            };
            load4(0);
#pragma unroll
            for (int b = 0; b < kBatches; ++b) {
                tmem_ld_wait();
                if (b + 1 < kBatches) {
                    load4(b + 1);
                } else {
                    // all reads of the step are done: the x half of the next one may overwrite
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_acc_free);
                }
                const auto &v = a[b & 1];
                if (4 * b < my_rows) {
                    int2 h[2];
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        h[j] = lstm_cell_codes(v[0][2 * j], v[0][2 * j + 1], v[1][2 * j], v[1][2 * j + 1], v[2][2 * j], v[2][2 * j + 1],
                                               v[3][2 * j], v[3][2 * j + 1], make_float2(b_i, b_i), make_float2(b_f, b_f),
                                               make_float2(b_g, b_g), make_float2(b_o, b_o), c2[2 * b + j]);
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        sts8(stage + (4 * b + 2 * j) * 32 + lane, h[j].x);
                        sts8(stage + (4 * b + 2 * j + 1) * 32 + lane, h[j].y);
                    }
                    __syncwarp();
                    if (i + 1 < p.T) send(hs_dst[b], stage + b * 128 + (lane >> 1) * 16, bar_h);
                }
            }
            FLUKE_STAMP(blockIdx.x == 0 && threadIdx.x == 64, i * 8 + 1, clock64());
            FLUKE_STAMP(blockIdx.x == 0 && threadIdx.x == 64, i * 8 + 2, clock64());
            if (g_ok) {
                const uint4 v = lds128(g_src);
                *reinterpret_cast<uint4 *>(p.h_out + int64_t(time_of(i)) * p.B * p.H + g_off) = v;
                if (i + 1 == p.T) *reinterpret_cast<uint4 *>(p.h_state + g_off) = v;
            }
            __syncwarp();
        }
#pragma unroll
        for (int j = 0; j < kCols / 2; ++j) {
            float *cp = p.c + int64_t(m0 + r0 + 2 * j) * p.H + unit;
            if (2 * j < my_rows) cp[0] = c2[j].x;
            if (2 * j + 1 < my_rows) cp[p.H] = c2[j].y;
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
    int nb;       // row columns of the kernel (16, 32 or 48)
    int rows;     // rows per cluster
    int tiles;    // clusters
    int n_own, n_pad;
};

constexpr int group_pad8(int v) { return (v + 7) / 8 * 8; }

inline int group_smem(int nb, int rows, int H) {
    const int n_pairs = H / kGUnits / 2;
    return group_layout(nb, H, group_pad8((rows + n_pairs - 1) / n_pairs)).dynamic;
}

using group_kernel_fn = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, GroupDev);
inline group_kernel_fn group_kernel(int nb) {
    return nb == 16 ? lstm_group_kernel<16> : nb == 32 ? lstm_group_kernel<32> : lstm_group_kernel<48>;
}

// Clusters of C CTAs of the NB-row kernel that the device runs at once with the largest shared
// memory a CTA can have (0: the form is not available).
int group_capacity(int nb, int C) {
    static int known[64][3][kGMaxCtas + 1];  // n + 1, or -1
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return 0;
    int &slot = known[dev][nb / 16 - 1][C];
    if (slot == 0) {
        int n = 0;
        const void *fn = reinterpret_cast<const void *>(group_kernel(nb));
        bool ok = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448) == cudaSuccess;
        if (ok) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(C);
            cfg.blockDim = dim3(kGThreads);
            cfg.dynamicSmemBytes = 232448;
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
    int max_nb = 48;
    while (max_nb >= 16 && group_smem(max_nb, max_nb, H) > 232448) max_nb -= 16;
    if (max_nb < 16) return false;
    const int cap = group_capacity(max_nb, C);
    if (cap < 1) return false;
    const int waves = (B + cap * max_nb - 1) / (cap * max_nb);
    int tiles = cap * waves;
    if (tiles > (B + kGMinRows - 1) / kGMinRows) tiles = (B + kGMinRows - 1) / kGMinRows;
    g->rows = (B + tiles - 1) / tiles;
    g->tiles = (B + g->rows - 1) / g->rows;
    g->nb = (g->rows + 15) / 16 * 16;
    if (group_capacity(g->nb, C) < 1) return false;
    g->n_own = (g->rows + C / 2 - 1) / (C / 2);
    g->n_pad = group_pad8(g->n_own);
    return true;
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
    const int C = H / kGUnits;

    GroupDev p;
    p.T = T; p.B = B; p.H = H; p.reverse = l->reverse;
    p.rows = g.rows; p.n_own = g.n_own; p.n_pad = g.n_pad; p.dn_ts = group_dn_ts(g.nb, H, g.n_pad);
    p.dn = static_cast<const int8_t *>(l->dn_hh_i8);
    p.w_up = static_cast<const __half *>(l->w_up_f16);
    p.bias = static_cast<const float *>(l->bias_f32);
    p.dn_scale = static_cast<const float *>(l->dn_hh_scale);
    p.c = static_cast<float *>(l->c_f32);
    p.h_out = static_cast<int8_t *>(l->h_out_i8);
    p.h_state = static_cast<int8_t *>(l->h_i8);
    p.trace = trace_buffer();

    CUtensorMap tm_w, tm_x, tm_dn, tm_h0;
    int rc = make_tmap_2d(&tm_w, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, l->w_up_f16, 4 * uint64_t(H), 2 * R, uint64_t(2 * R) * 2,
                          kGUnits, 64, true);
    if (rc) return rc;
    {
        // both K blocks of a row range in one box: the 128-byte blocks of a row are a dimension
        const uint64_t dims[4] = {64, uint64_t(B), 2, uint64_t(T)};
        const uint64_t strides[3] = {uint64_t(R) * 2, 128, uint64_t(B) * R * 2};
        const uint32_t box[4] = {64, uint32_t(g.nb), 2, 1};
        rc = make_tmap_nd(&tm_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, x_down, 4, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
        if (rc) return rc;
    }
    rc = make_tmap_2d(&tm_dn, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, l->dn_hh_i8, R, H, H, 64, 128, true);
    if (rc) return rc;
    {
        const uint64_t dims[3] = {128, uint64_t(B), uint64_t(C)};
        const uint64_t strides[2] = {uint64_t(H), 128};
        const uint32_t box[3] = {128, uint32_t(g.n_pad), uint32_t(C)};
        rc = make_tmap_nd(&tm_h0, CU_TENSOR_MAP_DATA_TYPE_UINT8, l->h_i8, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
        if (rc) return rc;
    }

    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(g.tiles * C);
    cfg.blockDim = dim3(kGThreads);
    cfg.dynamicSmemBytes = group_layout(g.nb, H, g.n_pad).dynamic;
    cfg.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, group_kernel(g.nb), tm_w, tm_x, tm_dn, tm_h0, p);
}
