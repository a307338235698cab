// lstm_group_sm100.cu -- the recurrence of a factored-LSTM layer as many small thread-block
// clusters, each with a FEW chunk rows: the batch is spread over all clusters the device holds
// instead of being packed into 128-row tiles.
//
// A step is a chain of dependent stages, so its time is set by what each stage of one cluster has
// to move and compute for its own rows. With the rows as the M = 128 dimension of the
// contractions that amount does not shrink with the batch; here the operands are swapped. The
// WEIGHTS are the M dimension (128 hidden units per CTA, one accumulator block per gate) and the
// chunk rows the columns, and the recurrent half of the gate weights lives in
// TENSOR MEMORY as the A operand: an MMA of 16 columns then costs 12 cycles instead of the 42 that reading a
// 128-row A operand from shared memory takes (32 columns 18 against 44, 48 columns 24 against 48).
//
// A cluster has C = H / 128 CTAs (2 to 8). CTA j owns units 128 j .. 128 j + 127: their four gate weight
// blocks (hh half in tensor memory, x half in shared memory) and, in registers, their cell state for the
// cluster's rows. What is exchanged for the projection of the hidden rows depends on how many rows there are:
//
//   GATHER, up to 16 rows: every CTA sends the int8 codes of its units to all CTAs and projects the complete
//   rows itself (M = 128 projection columns, K = H). One exchange per step. (Clusters of eight, from 9 rows on: see group_by_pair.)
//
//   SPLIT, two groups of up to 16 or 24 rows: a CTA projects only its own units (K = 128), so hidden codes do not
//   leave it. Its int32 partial sums go, four rows at a time, to the CTA that adds up those rows (integer sums,
//   exact in any order), which sends the f16 result to all. Projecting complete rows takes 24 MMAs per group
//   at H = 768 and 96 KB of weights, this 4 and 16 KB; what one group waits for is the other's time.
//
// All exchanges between CTAs are 16-byte st.async stores that complete on an mbarrier of the receiver; SPLIT: what stays in the CTA
// is stored there and announced by an arrival per warp.
//
//   warp 0       loader: resident weights, x_down rows of every step; SPLIT: also the TMA stores of h_out
//   warp 1       MMA issuer
//   warps 2-17   four per tensor-memory lane quadrant: thread = hidden unit and projection column. GATHER: each has a quarter
//                of the rows; SPLIT: eight warps per group, each half of its rows. They turn the projections into f16 (SPLIT:
//                send, add up, send) and compute gates, cell update and int8 codes
//
// A buffer is only overwritten after its reader has provably finished. SPLIT: a CTA sends partial sums of step t + 1
// after its gate contraction of step t, for which every owner of rows has read its partial sums of step t; an owner
// sends hh_{t+1} after every CTA's projection of h_t, i.e. after every CTA's contraction of step t. GATHER: a
// CTA sends h_t after it has received h_{t-1} of every CTA, which each sent after its projection of h_{t-2}: two
// slots of hidden rows. By pair: a CTA sends h_t after its contraction of step t, which needs hh_t of every pair, sent after its
// projection of h_{t-1}; and hh the other way round. The final hidden state goes where the initial one was read: of a CTA's
// own units only (SPLIT), or after every CTA's initial rows have landed (GATHER, before the first cluster barrier).
// Nobody leaves before the final cluster barrier. Clusters never wait for one another, so any number of them may run in waves.
//
// What bounds a step (B200, H = 768; cycles of one CTA by clock stamps, which add up to its period and lengthen it by 2 to 4 %). 2 rows
// per cluster, 2160 (1820 at H = 384): the chain of projection 500, its conversion 140, 110 until the issuer sees it, hh half 470, cell update and staging
// 490, exchange 430 (200 at H = 384). 14 rows, 2850: 500, 270, 130, 450, 1040 (the cell updates) and 440. 47 rows, 4500: first group's projection 460, its partial
// sums sent 310, on the way 480 to 800, read and added up 300, converted and sent 300 to 430, on the way 490, contraction 720, cell updates 950 (24 rows, eight
// warps), 230 until the issuer has seen the last warp's codes; the second group's chain runs beside it, and the tensor pipe works 3370 of them (x part 1540,
// hh half 1460, projections 370). The layer ends with the slowest cluster: 1024 chunks 2.66 us per step, x_down included, in layers of 400 steps (2.86 at commit
// f537a30, before own shares stayed out of the network), at the 1.83 GHz that the nanosecond timer gives inside the kernel (the driver reports 1965 MHz
// meanwhile). That is below the power limit: in a loop of seconds the gain is 5 % instead of 7 (five layers of 1000 steps 15.15 -> 14.37 ms).
// The cell updates live on few instructions: when places in the swizzle were worked out per row instead of by one exclusive or, 1024 chunks took 0.14 us
// more, 700 0.09.
//
// The operand rows that are zero (see group_form) add zero times a weight to another group's or step's accumulators: with
// finite weights nothing. A CTA whose recurrent gate weights are not all finite (0 x inf is NaN) issues other MMAs, see
// issue_exact: an infinite weight reaches the rows of its unit through their own factors only.
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

constexpr int kGUnits = 128;       // hidden units per CTA = tensor-memory lanes
constexpr int kGRank = 128;        // factor rank the kernel is built for
constexpr int kGMaxCtas = 8;       // portable cluster size: H <= 1024
constexpr int kGEpiWarps = 16;
constexpr int kGThreads = 32 * (2 + kGEpiWarps);
constexpr int kGTmemCols = 512;
constexpr int kGTmemW = 256;       // first column of the hh half of the gate weights: 4 gates x 64
constexpr int kGWxBytes = 4 * kGUnits * 256;  // x half of the gate weights in shared memory
constexpr int kGMaxSmem = 232448;

struct GroupDev {
    int T, B;
    int reverse;
    int rows;                  // chunk rows per cluster (the last one may have fewer)
    const int8_t *dn;          // [R, H]
    const float *bias;         // [4H]
    const float *dn_scale;     // [R]
    float *c;                  // [B,H]
    int8_t *h_out;             // [T,B,H]
    int8_t *h_state;           // [B,H]: final hidden state
    long long *trace;          // trace builds only: [T][16] SM-clock stamps of CTA 0
};

// The forms of the kernel: chunk rows per cluster up to 8, 16, 32 and 48. GATHER is one group of rows, SPLIT two. Step of the kernel of commit 31278fa, of one and
// two groups, which exchanged hidden rows between pairs of CTAs and projected them there, against these as they are now, us, x_down included, layers of 400 steps:
// H = 768 32 chunks (2 rows per cluster) 1.45 : 1.23, 170 (8) 1.56 : 1.44, 300 (14) 1.66 : 1.72, 500 (23) 2.40 : 1.96, 700 (32) 2.62 : 2.02, 1024 (47) 2.97 : 2.66; H = 384 32
// (2) 1.37 : 1.04, 387 (9) 1.55 : 1.39, 731 (17) 2.29 : 1.90; H = 256 594 (9) 1.48 : 1.37, 1122 (17) 1.73 : 1.54, 2376 (36) 2.69 : 2.64; H = 512 288 (9) 1.52 : 1.46, 544 (17) 2.09 : 1.79,
// 1472 (46) 2.91 : 2.72; H = 640 234 1.57 : 1.53, 442 2.18 : 1.83, 858 2.87 : 2.58; H = 896 153 1.72 : 1.68, 289 2.38 : 1.99, 561 3.06 : 2.55; H = 1024 700 (47), where it took two waves from
// 577 chunks on, 4.85 : 2.70. The left figures are of its own day, those in front of the first semicolon of longer layers, whose set-up is less per step (300 chunks of 777
// steps take 1.68 now). The limits are the same for every cluster size.
// Everything below depends on the form V, the cluster size C = H / 128 and the steps per x MMA, which the kernel is compiled
// for: with operand addresses at fixed distances the issuer needs few instructions between MMAs.
constexpr int kGForms = 4;
struct GroupForm {
    int most;           // rows per cluster
    bool gather;
    int groups, rows;   // groups, and chunk rows of each at most
    int n;              // columns of the MMAs of one group: M = 128 takes multiples of 16
    int acc;            // accumulator columns of a gate in a step
    int proj;           // columns of projection accumulators
};
// 8 rows: the columns of an x MMA are two or four steps' rows, see x_half. Two groups of 24 rows: an MMA of
// the first group also covers the first columns of the second, with operand rows that are zero, before that
// group's own MMAs; the second group's covers unused columns. They take turns with one projection accumulator.
__host__ __device__ constexpr GroupForm group_form(int V) {
    return V == 0   ? GroupForm{8, true, 1, 8, 16, 8, 16}
           : V == 1 ? GroupForm{16, true, 1, 16, 16, 16, 16}
           : V == 2 ? GroupForm{32, false, 2, 16, 16, 32, 32}
                    : GroupForm{48, false, 2, 24, 32, 56, 32};
}
// Steps whose x part one MMA covers: for each form and cluster size a kernel of the fewest and, where it pays, one of more. Up to 8 rows: MMAs of an
// A operand in shared memory take as long for 32 columns (44 cycles) as for the sixteen that there are at least (42), and what is issued of them before
// the hidden codes arrive holds the issuer up: with 16 such MMAs per step it saw codes that had travelled for 200 cycles after 430. Four steps per MMA are 8 per step, and twice the accumulators, which clusters of
// two and three have the tensor memory for beside all projection weights. Two steps against four, us per step, x_down included: H = 384 32 chunks 1.156 :
// 1.044, 120 1.186 : 1.078, 172 1.188 : 1.088, 250 1.200 : 1.160, 344 1.235 : 1.238; H = 256 32 1.137 : 1.027, 300 1.182 : 1.109, 528 1.222 : 1.202. With
// more CTAs some projection weights have to give way: H = 512 32 chunks 1.166 : 1.125, but 200 1.269 : 1.339; H = 640 200 1.366 : 1.467.
// 17 to 32 rows: an MMA of 64 columns takes 48 cycles, one of 32 takes 44, and while they run little else gets at the shared memory (a step without any x part takes
// 10 % less at H = 768, 15 % at H = 512). One step against two: H = 768 360 chunks 2.031 : 1.941, 500 2.063 : 1.989, 700 2.103 : 2.037; H = 384 900 2.062 : 1.934; H =
// 256 1200 2.045 : 1.827; H = 512 700 2.047 : 1.835; H = 640 600 2.063 : 1.885; H = 896 400 2.060 : 2.050; clusters of eight 300 2.089 : 2.138.
// 9 to 16 rows, where the larger accumulators leave tensor memory for all projection weights: H = 256 600 chunks 1.455 : 1.369, 1000 1.545 : 1.507; H = 384 400
// 1.485 : 1.395, 600 1.569 : 1.547, 680 1.589 : 1.593; H = 512 300 1.494 : 1.462, 500 1.657 : 1.654. Without: H = 640 230 1.547 : 1.546, 260 1.555 : 1.569, 300 1.569 : 1.621, 400
// 1.685 : 1.772; H = 768 200 1.606 : 1.667, 300 1.758 : 1.842; clusters of seven lack the shared memory for the weights that would go there. (All pairs in layers of
// 400 steps, each as it was measured when it was chosen.)
constexpr int group_x_steps(int V, int C, bool most) {
    if (V == 0) return most && C <= 3 ? 4 : 2;
    return most && ((V == 1 && C <= 4) || (V == 2 && C <= 7)) ? 2 : 1;
}
// Which of the two. Windows of several steps begin before the first one or end behind the last, so a layer of few steps pays for more than its
// own; and with many rows in its form the wider accumulators cost more than they save. Fewest : most, us of a layer, x_down included.
// Up to 8 rows, H = 384 86 chunks (2 rows) 1 step 12.4 : 12.7, H = 256 132 8 steps 19.6 : 19.2; H = 384 301 chunks (7 rows) 100 steps 127.2 : 127.3, 344 (8) 400 steps 485 : 492.
// 9 to 16 rows, H = 512 448 chunks (14) 1 step 13.2 : 13.7; H = 384 602 (14) 10 steps 26.1 : 26.5, 24 steps 46.3 : 46.5 and in long layers 0.7 % less; H = 256 924 (14) 16 steps
// 34.3 : 34.1; H = 512 384 (12) 48 steps 80.4 : 80.1, 448 (14) 400 steps 627 : 634; H = 384 688 (16) 400 steps 612 : 619. 17 to 32 rows, H = 256 2112 chunks 1 step 12.5 : 13.0, 1848 8
// steps 27.0 : 26.4; H = 640 700 8 steps 26.7 : 26.4; H = 768 704 1 step 12.7 : 13.3, 8 steps 26.7 : 27.0, 20 steps 50.6 : 50.4; H = 896 448 20 steps 49.0 : 50.1, 100 to 400 steps
// within 1 % of each other.
bool group_most_x_steps(int T, int rows, int V, int C) {
    if (V == 1) return T >= 16 && rows <= (C == 2 ? 16 : C == 3 ? 14 : 12);
    if (V == 2) return T >= (C <= 5 ? 8 : 16);
    return T >= 8 && rows <= (C == 2 ? 8 : 6);
}
// The x_down rows of a cluster in shared memory. A tile is the rows of one step in one of the two K blocks of 64. Up to 8 rows: per K block a ring of
// tiles, of which the first steps - 1 are repeated behind it, so that the rows of a window of steps are contiguous wherever it begins. More rows, two
// steps: two windows of two tiles per K block. Else: two steps.
struct GroupX {
    int steps;          // that an x MMA covers
    int slots;          // windows (with one step: steps) that are loaded ahead, a power of two
    int tile;           // bytes
    int slot;           // from a slot to the next
    int kb;             // from the first K block to the second
    int bytes;          // all of it
};
__host__ __device__ constexpr GroupX group_x(int V, int steps) {
    const int tile = group_form(V).groups * group_form(V).rows * 128;
    if (V == 0) {
        const int slots = 2 * steps, ring = slots + steps - 1;
        return GroupX{steps, slots, tile, tile, ring * tile, 2 * ring * tile};
    }
    return GroupX{steps, 2, tile, 2 * steps * tile, steps * tile, 2 * 2 * steps * tile};
}
// Accumulator columns from gate to gate.
__host__ __device__ constexpr int group_stride(int V, int X) { return group_form(V).acc * (V == 0 ? X : 1); }
// Columns of all gate accumulators. Two steps of more than 8 rows: six places of a gate's columns hold the four gates of a step and two of the next.
__host__ __device__ constexpr int group_acc_cols(int V, int X) { return (V > 0 && X == 2 ? 6 : 4) * group_stride(V, X); }
// K steps (32 units, 8 columns) of the projection weights that fit in tensor memory beside the gate weights, the gate
// accumulators and the projections.
__host__ __device__ constexpr int group_dn_ts(int V, int C, int X) {
    const GroupForm f = group_form(V);
    const int fit = (kGTmemW - group_acc_cols(V, X) - f.proj) / 8, all = f.gather ? 4 * C : 4;
    return fit < all ? fit : all;
}
// Four rows of a group are projected as one piece (16 bytes per projection column). The pieces of all groups are dealt to
// the C CTAs in turn; the owner adds up what the C CTAs have of it.
__host__ __device__ constexpr int group_own_pieces(int V, int C) {
    return (group_form(V).groups * group_form(V).rows / 4 + C - 1) / C;
}
// GATHER with clusters of eight and 9 to 16 rows: rows are projected BY PAIR. Pair (2p, 2p + 1) of CTAs receives the codes of a
// quarter of the rows, projects 64 columns per CTA (M = 64) and sends the f16 result to all: two exchanges, but half of the
// bytes. Two such clusters share the network between the SMs of a GPC; all to all, the last code is 840 cycles old when
// the slowest arrives, 535 where a cluster is alone in its GPC. Us per step, x_down included, all to all against by pair: 9 rows 1.89 : 1.66,
// 12 rows 1.98 : 1.71, 14 rows 2.13 : 1.79, 16 rows 2.19 : 1.87 (the kernel of 31278fa, by pair as well: 1.76, 1.88, 1.95, 2.04).
// Smaller clusters stay with all to all: an odd number of CTAs has no pairs, a pair of fewer than eight would own more than one
// row per quarter of its gate warps, and there all to all was the faster against that kernel (H = 768, 14 rows 1.61 : 1.66).
// Up to 8 rows two steps per x MMA make up for it (H = 1024, 8 rows 1.69 : 1.73 against that kernel).
__host__ __device__ constexpr bool group_by_pair(int V, int C) { return V == 1 && C == 8; }
// mbarriers of a CTA, as indices
enum : int {
    kBarOnce = 0,      // x half of the gate weights loaded
    kBarX = 1,         // [slots] x_down rows landed
    kBarXFree = 5,     // [slots] the x part of the contraction has read them
    kBarAccFree = 9,   // the gate warps have read all accumulators
    kBarProj = 10,     // [G] projection accumulator complete
    kBarAcc = 12,      // [G] gate accumulators complete
    kBarHh = 14,       // [G] hh_down rows in place
    kBarCode = 16,     // SPLIT [G]: hidden codes of this CTA's units in place
    kBarSum = 18,      // SPLIT [G]: partial sums of the CTA's own pieces arrived
    kBarSent = 20,     // SPLIT: the projection accumulator has been read
    kBarStored = 21,   // SPLIT: the TMA stores have read the hidden codes
    kBarStart = 22,    // resident projection weights and the initial hidden rows loaded
    kBarH = 16,        // GATHER [2], by pair [1]: hidden rows of all CTAs arrived
    kBarW = 24,        // set-up [4]: recurrent weights of a gate landed in shared memory
    kBarWRead = 28,    // set-up [4]: and have been read from there
    kBarX4 = 32,       // up to 8 rows, four steps per x MMA [8]: in place of kBarX
    kBarX4Free = 40,   // and of kBarXFree
    kGBars = 48
};

struct GroupLayout {
    int x, hh, dn, h, recv, stage, bars, misc, dynamic;
};
__host__ __device__ constexpr GroupLayout group_layout(int V, int C, int X) {
    const GroupForm f = group_form(V);
    GroupLayout l = {};
    l.x = kGWxBytes;                              // x_down rows, see x_half
    l.hh = l.x + group_x(V, X).bytes;
    // hh_down rows: per group 2 K blocks [n x 128 B]; 8 rows: [24 x 128 B], the rows in front and behind are zero
    l.dn = l.hh + (f.rows == 8 ? 24 : f.groups * f.n) * 256;
    // projection weights [128 x 128 B] (by pair [64 x 128 B]) of the K blocks that are not all in tensor memory
    l.h = l.dn + (group_by_pair(V, C) ? 8192 : 16384) * ((f.gather ? C : 1) - group_dn_ts(V, C, X) / 4);
    // int8 hidden rows. GATHER: two slots of C K blocks [rows x 128 B], by pair one of [8 x 128 B]; else this CTA's units, per
    // group [rows x 128 B]. An MMA of more columns reads on behind them
    l.recv = l.h + (group_by_pair(V, C) ? C * 1024 : (f.gather ? 2 * C : f.groups) * f.rows * 128);
    // partial sums of the CTA's own pieces: per piece and source CTA [128 columns][4 rows] int32
    l.stage = l.recv + (f.gather ? 0 : group_own_pieces(V, C) * C * 2048);
    // GATHER: two slots x four quarters x [2 rows x 128 B], by pair [4 rows x 128 B]; else per warp [2 rows x 64 B]
    l.bars = l.stage + (group_by_pair(V, C) ? 4096 : 2048);
    l.misc = l.bars + kGBars * 8;
    l.dynamic = l.misc + 16 + 1024;               // slack for the manual 1024-byte alignment
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
__device__ __forceinline__ int2 lds64(uint32_t addr) {
    int2 v;
    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
    return v;
}
// n arrivals at once
__device__ __forceinline__ void mbar_arrive_n(uint64_t *bar, int n) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(n) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t addr, uint4 v) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ int lds8(uint32_t addr) {
    int v;
    asm volatile("ld.shared.s8 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void sts8(uint32_t addr, int v) {
    asm volatile("st.shared.u8 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void sts16(uint32_t addr, unsigned short v) {
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(addr), "h"(v) : "memory");
}

// Adds zero times the halves of w to sum: NaN from the first that is infinite or NaN on, else zero.
__device__ __forceinline__ void add_zero_times(__half2 &sum, uint4 w) {
    const __half2 zero = __half2half2(__ushort_as_half(0));
    const uint32_t words[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) sum = __hfma2(*reinterpret_cast<const __half2 *>(&words[j]), zero, sum);
}

// Barrier of the four warps that share a staging slot.
__device__ __forceinline__ void quad_sync(int id) { asm volatile("barrier.cta.sync %0, 128;" ::"r"(id) : "memory"); }

template <int V>
struct Int { static constexpr int value = V; };  // a number that a lambda receives as a type

// What the kernel and its MMA issuer know at compile time.
template <int V, int C, int STEPS>
struct GroupConst {
    static constexpr GroupForm F = group_form(V);
    static constexpr GroupLayout L = group_layout(V, C, STEPS);
    static constexpr bool kGather = F.gather;
    static constexpr int G = F.groups, NB = G * F.rows, S = group_stride(V, STEPS), H = C * kGUnits;
    static constexpr bool kTwoSteps = V == 0 && STEPS == 2;    // an x MMA covers two steps
    static constexpr bool kFourSteps = STEPS == 4;   // or four
    static constexpr bool kTwoStepsWide = V > 0 && STEPS == 2;   // two steps of more than 8 rows, see x_half
    static constexpr int kAcc = group_acc_cols(V, STEPS);         // columns of the gate accumulators; the projections' follow
    static constexpr GroupX X = group_x(V, STEPS);
    static constexpr int kXSlots = X.slots;
    static constexpr int kBarXAt = kFourSteps ? kBarX4 : kBarX, kBarXFreeAt = kFourSteps ? kBarX4Free : kBarXFree;
    static constexpr bool kByPair = group_by_pair(V, C);
    static constexpr bool kPeerHh = !kGather || kByPair;      // hh_down rows come from peers
    static constexpr int kTile = (kByPair ? 8 : F.rows) * 128;     // bytes of a group's hidden rows in one K block
    static constexpr int kHhTile = (F.rows == 8 ? 24 : F.n) * 128;   // and of its hh_down rows
    static constexpr bool kZeroRows = kHhTile > F.rows * 128; // some of which are zero
    static constexpr int kDnRows = kByPair ? 64 : kGRank;     // projection columns of a CTA
    static constexpr int kPieces = F.rows / 4;                // pieces of a group
    static constexpr int kPairs = kGather ? F.rows / 8 : F.rows / 4;   // pairs of rows of a gate thread
    static constexpr int kDnTs = group_dn_ts(V, C, STEPS);
    static constexpr int kDnCol = kGTmemW - 8 * kDnTs;        // first column of the projection weights in tensor memory
    static constexpr bool kOneProj = F.proj < G * F.n;        // the groups share the projection accumulator
    static_assert(kAcc + F.proj + 8 * kDnTs <= kGTmemW, "accumulators beside the weights in tensor memory");
    static_assert(L.dynamic <= kGMaxSmem, "shared memory of a CTA");
    static_assert((kXSlots & (kXSlots - 1)) == 0 && X.tile == NB * 128, "slots by masks, tiles as the tensor map loads them");
    static_assert(V != 0 || X.kb == (kXSlots + X.steps - 1) * X.slot, "a window of the ring ends in front of the other K block");
    static_assert(V == 0 || (X.kb == X.steps * X.tile && X.slot == 2 * X.kb), "a window's K blocks in front of the next window");
    static_assert(L.hh - L.x == (V == 0 ? 2 * X.kb : kXSlots * X.slot), "x_down rows end where the hh_down rows begin");
    static_assert(kXSlots <= kBarXFreeAt - kBarXAt && kXSlots <= (kFourSteps ? kGBars : kBarAccFree) - kBarXFreeAt, "a barrier per slot");
    static_assert(kBarX4 >= kBarWRead + 4 && L.misc - L.bars == kGBars * 8, "barriers one after the other");
    static_assert(!kByPair || (C % 2 == 0 && F.rows <= 2 * C), "a pair's rows are one per quarter of the gate warps");
};
// The MMA issuer, warp 1. The whole warp walks the loop; one elected lane issues. Descriptors are uniform and the
// K loops unrolled, so an MMA is issued every few cycles. kExact: for weights that are not finite.
template <int V, int C, int STEPS, bool kExact>
__device__ __forceinline__ void issue(uint8_t *smem, uint32_t tmem, const GroupDev &p, int n_rows, int own_rows, uint32_t hh_bytes0, uint32_t hh_bytes1) {
    using K = GroupConst<V, C, STEPS>;
    constexpr GroupForm F = K::F;
    constexpr GroupLayout L = K::L;
    constexpr bool kGather = K::kGather, kByPair = K::kByPair, kTwoSteps = K::kTwoSteps, kFourSteps = K::kFourSteps, kOneProj = K::kOneProj;
    constexpr int G = K::G, NB = K::NB, S = K::S, H = K::H, kXSlots = K::kXSlots, kTile = K::kTile, kHhTile = K::kHhTile;
    constexpr int kDnTs = K::kDnTs, kDnCol = K::kDnCol;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L.bars);
    uint64_t *bar_once = bars + kBarOnce, *bar_x = bars + K::kBarXAt, *bar_x_free = bars + K::kBarXFreeAt, *bar_acc_free = bars + kBarAccFree;
    uint64_t *bar_proj = bars + kBarProj, *bar_acc = bars + kBarAcc, *bar_hh = bars + kBarHh, *bar_code = bars + kBarCode;
    uint64_t *bar_sent = bars + kBarSent, *bar_stored = bars + kBarStored, *bar_h = bars + kBarH;
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + L.misc + 4);
    [[maybe_unused]] const int lane = threadIdx.x & 31;
    auto rows_of = [&](int e) { return min(max(n_rows - F.rows * e, 0), F.rows); };
    const bool both = G > 1 && n_rows > F.rows;        // the last cluster may have nothing in its second group
    constexpr uint32_t kIdescX = make_idesc<kKindF16>(128, K::X.steps * NB);
    constexpr uint32_t kIdescHh = make_idesc<kKindF16>(128, F.n);
    constexpr uint32_t kIdescP = make_idesc<kKindI8>(128, F.n);
    uint64_t d_wx = make_smem_desc_sw128(smem_u32(smem));
    uint64_t d_x0 = make_smem_desc_sw128(smem_u32(smem + L.x));
    uint64_t d_hh = make_smem_desc_sw128(smem_u32(smem + L.hh));
    uint64_t d_dn = make_smem_desc_sw128(smem_u32(smem + L.dn));
    uint64_t d_h0 = make_smem_desc_sw128(smem_u32(smem + L.h));
    bool ok = mbar_wait(bars + kBarStart, 0, abort_flag, 97) && mbar_wait(bar_once, 0, abort_flag, 97);
    int i = 0;
    // MMAs [from, to) of the x part of a step. They read their A operand from shared memory (42 cycles
    // each, 48 with 48 columns) and the tensor pipe works in order, so they are issued in pieces for the times when it
    // would wait. With up to 8 rows, where the 32 MMAs of a step would take longer than all of its waits, an MMA covers
    // the rows of two or four steps. Two: even steps compute gates 0 and 1 of themselves and the next, odd ones gates 2 and
    // 3. Slot s of five holds step s mod 4, so that a step's rows and the next one's are sixteen contiguous ones. Four: step i computes gate
    // i mod 4 of itself and the next three, whose rows are contiguous in a ring of eight slots of which the first three are repeated behind it.
    // More than 8 rows, two steps: step i computes gates 0 and 1 (i even) or 2 and 3 of itself and the next, side by side. What has been read makes room for them
    // if even steps lie behind the odd ones of their window: gates 0 and 1 in places 0, 1 and 3, 4 of the six, 2 and 3 in 1, 2 and 4, 5, so that gate g of step i
    // is at place 3 (g mod 2) + g / 2 + (1 if i is even). A window is loaded as one tile of both steps' rows per K block, each step twice.
    constexpr int kX = kFourSteps ? 8 : kTwoSteps || K::kTwoStepsWide ? 16 : 32;
    auto x_half = [&](auto from, auto to, int i, bool release = true, int gate = 0) {
        constexpr int first = decltype(from)::value, end = decltype(to)::value;
        const int slot = (K::kTwoStepsWide ? i + 1 : i) & (kXSlots - 1);
        const uint64_t d_x = d_x0 + uint64_t(slot * (K::X.slot >> 4));
        const int g0 = kFourSteps ? (kExact ? gate : i & 3) : kTwoSteps || K::kTwoStepsWide ? 2 * (i & 1) : 0;
        if (elect_one()) {
#pragma unroll
            for (int m = first; m < end; ++m) {
                const int g = m >> 3, k = m & 7;
                tc_mma<kKindF16>(tmem + (K::kTwoStepsWide ? 3 * g + (i & 1) : g0 + g) * S, d_wx + uint64_t(((g0 + g) * 2 + (k >> 2)) * 1024 + 2 * (k & 3)),
                                 d_x + uint64_t((k >> 2) * (K::X.kb >> 4) + 2 * (k & 3)), kIdescX, k != 0);
            }
            if (end == kX && release) tc_commit(&bar_x_free[slot]);
        }
        __syncwarp();
    };
    auto wait_x = [&](int step) {
        const int n = K::kTwoStepsWide ? step + 1 : step;
        if (step < p.T) ok = ok && mbar_wait(&bar_x[n & (kXSlots - 1)], (n / kXSlots) & 1, abort_flag, 99);
        return ok;
    };
    auto wait_acc = [&]() {
        if (i > 0) ok = ok && mbar_wait(bar_acc_free, (i - 1) & 1, abort_flag, 98);
        tc_fence_after_sync();
        return ok;
    };
    // projection u overwrites what projection u - 1 left
    auto wait_sent = [&](int u) {
        if (kOneProj && u > 0) ok = ok && mbar_wait(bar_sent, (u - 1) & 1, abort_flag, 106);
        return ok;
    };
    // projection of h_{i-1}. SPLIT: this CTA's K block for the rows of a group
    auto project = [&](auto group, int i) {
        constexpr int e = decltype(group)::value;
        if (e > 0 && !both) return true;
        if (i > 0) ok = ok && mbar_wait(&bar_code[e], (i - 1) & 1, abort_flag, 100);
        if (!ok) return false;
        tc_fence_after_sync();
        FLUKE_STAMP(blockIdx.x == 0 && lane == 0, i * 16 + e, clock64());
        if (elect_one()) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint64_t rows = d_h0 + uint64_t(e * (kTile >> 4) + 2 * k);
                constexpr int kTo = K::kAcc + (kOneProj ? 0 : e * F.n);
                if (k < kDnTs) tc_mma_ts<kKindI8>(tmem + kTo, tmem + kDnCol + 8 * k, rows, kIdescP, k != 0);
                else tc_mma<kKindI8>(tmem + kTo, d_dn + uint64_t(2 * k), rows, kIdescP, k != 0);
            }
            tc_commit(&bar_proj[e]);
        }
        __syncwarp();
        return true;
    };
    // GATHER: all K blocks. Hidden rows of step u are in slot u mod 2, by pair in the only one
    auto project_all = [&]() {
        if (i > 0) ok = ok && mbar_wait<true>(&bar_h[kByPair ? 0 : (i + 1) & 1], (kByPair ? i - 1 : (i - 1) >> 1) & 1, abort_flag, 100);
        if (!ok) return false;
        FLUKE_STAMP(blockIdx.x == 0 && lane == 0, i * 16 + 11, clock64());
        fence_proxy_async_smem();   // the peers' stores are generic-proxy writes
        tc_fence_after_sync();
        FLUKE_STAMP(blockIdx.x == 0 && lane == 0, i * 16 + 0, clock64());
        if (elect_one()) {
            const uint64_t d_h = d_h0 + uint64_t((kByPair ? 0 : (i + 1) & 1) * (C * kTile >> 4));
            constexpr uint32_t kIdesc = make_idesc<kKindI8>(K::kDnRows, kByPair ? 8 : F.n);
#pragma unroll
            for (int kb = 0; kb < C; ++kb)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint64_t rows = d_h + uint64_t(kb * (kTile >> 4) + 2 * k);
                    if (4 * kb + k < kDnTs) tc_mma_ts<kKindI8>(tmem + K::kAcc, tmem + kDnCol + 8 * (4 * kb + k), rows, kIdesc, (kb | k) != 0);
                    else tc_mma<kKindI8>(tmem + K::kAcc, d_dn + uint64_t((kb - kDnTs / 4) * (K::kDnRows * 8) + 2 * k), rows, kIdesc, (kb | k) != 0);
                }
            tc_commit(&bar_proj[0]);
            if (kByPair && i > 0 && i + 1 < p.T) mbar_arrive_expect_tx(&bar_h[0], uint32_t(own_rows) * H);  // for h_i
            if (!kByPair && i > 0 && i + 2 < p.T) mbar_arrive_expect_tx(&bar_h[(i + 1) & 1], uint32_t(n_rows) * H);  // for h_{i+1}
        }
        __syncwarp();
        FLUKE_STAMP(blockIdx.x == 0 && lane == 0, i * 16 + 1, clock64());
        return true;
    };
    auto hh_half = [&](auto group) {
        constexpr int e = decltype(group)::value;
        if (e > 0 && !both) return true;
        // Several steps per x MMA: neighbouring steps' columns get rows that are zero. All of it is worked out in front of the wait.
        uint64_t rows[4];
        uint32_t cols[4];
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            rows[g] = d_hh;
            cols[g] = tmem + (K::kTwoStepsWide ? 3 * (g & 1) + (g >> 1) + 1 - (i & 1) : g) * S + F.rows * e;
            if (kTwoSteps) rows[g] += (i ^ (g >> 1)) & 1 ? 0 : 64;
            if (kFourSteps) {
                const int at = kExact ? 0 : (i - g) & 3;
                rows[g] += at < 3 ? 64 : 0;
                cols[g] += at < 3 ? 8 * at : 16;
                asm volatile("" : "+l"(rows[g]), "+r"(cols[g]));
            }
        }
        ok = ok && mbar_wait<true>(&bar_hh[e], i & 1, abort_flag, 101);
        if (!ok) return false;
        if (K::kPeerHh) fence_proxy_async_smem();
        tc_fence_after_sync();
        FLUKE_STAMP(blockIdx.x == 0 && lane == 0, i * 16 + 3 + e, clock64());
        if (elect_one()) {
#pragma unroll
            for (int g = 0; g < 4; ++g)
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    tc_mma_ts<kKindF16>(cols[g], tmem + kGTmemW + g * 64 + k * 8,
                                        rows[g] + uint64_t((2 * e + (k >> 2)) * (kHhTile >> 4) + 2 * (k & 3)), kIdescHh, 1u);
            tc_commit(&bar_acc[e]);
            if (K::kPeerHh && i + 1 < p.T) mbar_arrive_expect_tx(&bar_hh[e], kGather ? uint32_t(n_rows) * 256 : e == 0 ? hh_bytes0 : hh_bytes1);
        }
        __syncwarp();
        return true;
    };
    // Two groups of 24 rows, kExact: 48 rows in three MMAs of sixteen, the middle one of the first group's last eight and the second's
    // first eight (the distance of eight rows from the next is the descriptor's), when both groups are there.
    auto hh_both = [&]() {
        for (int e = 0; e < 2; ++e) ok = ok && mbar_wait<true>(&bar_hh[e], i & 1, abort_flag, 101);
        if (!ok) return false;
        fence_proxy_async_smem();
        tc_fence_after_sync();
        if (elect_one()) {
            constexpr uint32_t kIdesc = make_idesc<kKindF16>(128, 16);
            constexpr uint64_t kGroup = 2 * kHhTile >> 4;   // from a group's rows to the other's
            const uint64_t rows[3] = {d_hh, d_hh + 128 + ((kGroup - 128 - 64) << 32), d_hh + kGroup + 64};
#pragma unroll 1
            for (int g = 0; g < 4; ++g)
#pragma unroll
                for (int b = 0; b < 3; ++b)
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        tc_mma_ts<kKindF16>(tmem + g * S + 16 * b, tmem + kGTmemW + g * 64 + k * 8,
                                            rows[b] + uint64_t((k >> 2) * (kHhTile >> 4) + 2 * (k & 3)), kIdesc, 1u);
            for (int e = 0; e < 2; ++e) {
                tc_commit(&bar_acc[e]);
                if (i + 1 < p.T) mbar_arrive_expect_tx(&bar_hh[e], e == 0 ? hh_bytes0 : hh_bytes1);
            }
        }
        __syncwarp();
        return true;
    };
    if constexpr (kTwoSteps) {
        // gates 2 and 3 of step 0: as the second step of the one before it
        if (ok) ok = mbar_wait(&bar_x[0], 0, abort_flag, 99);
        if (ok) x_half(Int<0>{}, Int<16>{}, -1, false);
    }
    if constexpr (K::kTwoStepsWide) {
        // gates 2 and 3 of step 0: as the second step of a window that begins before it
        if (wait_x(-1)) x_half(Int<0>{}, Int<kX>{}, -1);
    }
    if constexpr (kFourSteps) {
        // gates 1, 2 and 3 of the first steps, as of steps before them: whatever is in the slots enters columns that nothing reads
        for (int w = -3; w < 0 && wait_x(w + 3); ++w) x_half(Int<0>{}, Int<kX>{}, w, false, w & 3);
    }
    for (; i < p.T && ok; ++i) {
        // Fresh values in every step: hoisted out of the loop, the operands of its MMAs would fill
        // more registers than there are.
        asm volatile("" : "+l"(d_wx), "+l"(d_x0), "+l"(d_hh), "+l"(d_dn), "+l"(d_h0));
        constexpr int kFirstX = kFourSteps ? 4 : kTwoSteps ? 10 : kByPair ? 16 : kGather ? (K::kTwoStepsWide ? 12 : 24) : 2;
        if constexpr (kGather) {
            // Most of the x part while the hidden state is computed and travels, the rest while the projection is converted. Us per step (x_down
            // included). One step per MMA, 20 / 24 / 28 of 32 in front: H = 768 200 chunks 1.62 / 1.57 / 1.64, 300 1.74 / 1.70 / 1.73; H = 896 180 1.71 / 1.70 / 1.74. Two
            // steps, up to 8 rows, 8 / 10 / 12 of 16: H = 768 32 chunks 1.19 / 1.19 / 1.23, 100 1.29 / 1.27 / 1.30; H = 1024 60 1.42 / 1.40 / 1.44; more rows, 10 / 12 / 14
            // of 16: H = 384 600 1.533 / 1.529 / 1.525; H = 256 600 1.363 / 1.361 / 1.354, 1000 1.486 / 1.494 / 1.474; H = 512 300 1.480 / 1.479 / 1.482, 500 1.645 / 1.642 / 1.639. Four
            // steps, 3 / 4 / 5 of 8 within 1 % of each other. By pair 12 / 16 / 20 of 32: 135 chunks 1.68 / 1.66 / 1.73, 240 1.86 / 1.87 / 1.88.
            if (!wait_x(kFourSteps ? i + 3 : kTwoSteps ? i + 1 : i) || !wait_acc()) break;
            FLUKE_STAMP(blockIdx.x == 0 && lane == 0, i * 16 + 15, clock64());
            // Two steps per MMA: the zero rows of the step before have spoilt the accumulators of this step's gates that its x MMAs
            // computed. Once more from the same slots; the step before may be gone from its, it enters columns that have been read.
            if (kExact && kTwoSteps && i > 0) x_half(Int<0>{}, Int<kX>{}, i - 1, false);
            if constexpr (kExact && kFourSteps) {
                // all gates of this step from this step's window: what the zero rows spoil is never used. The last gate behind the projection: in front of it
                // as well, H = 384 32 chunks 1.491 -> 1.629 us per step, H = 256 528 1.529 -> 1.694 (two steps per MMA 1.544 and 1.606).
                for (int g = 0; g < 3; ++g) x_half(Int<0>{}, Int<kX>{}, i, false, g);
                if (!project_all()) break;
                x_half(Int<0>{}, Int<kX>{}, i, true, 3);
            } else {
                x_half(Int<0>{}, Int<kFirstX>{}, i);
                FLUKE_STAMP(blockIdx.x == 0 && lane == 0, i * 16 + 10, clock64());
                if (!project_all()) break;
                x_half(Int<kFirstX>{}, Int<kX>{}, i);
            }
            if (!hh_half(Int<0>{})) break;
        } else {
            // A group's projection as soon as its codes are there, pieces of the x part in between. A wait for
            // what has long been there takes 100 cycles and more while the gate warps keep the units of the SM busy that
            // serve both, so such waits stand where the issuer has time (1024 chunks 3.07 -> 2.89 us per step when it was done).
            // MMAs in front of the second projection, us per step (x_down included). One step per MMA, 0 / 2 / 4 / 8, before own shares stayed in the CTA: H = 768 900
            // chunks 2.76 / 2.76 / 2.77 / 2.83, 1024 2.93 / 2.93 / 2.96 / 2.94; H = 384 1500 2.71 / 2.71 / 2.71 / 2.71; H = 1024 300 2.17 / 2.16 / 2.16 / 2.18, 700 2.90 / 2.91 / 2.92 /
            // 2.98. Four in front of the first as well took 0.3 us more. Two steps per MMA, 0 / 1 / 2 / 4 of 16: H = 768 500 1.958 / 1.960 / 1.964 / 1.966, 700 2.022 / 2.023 / 2.017 /
            // 2.037; H = 384 900 1.912 / 1.908 / 1.923 / 1.918; H = 512 700 1.850 / 1.857 / 1.841 / 1.843; H = 640 600 1.888 / 1.878 / 1.883 / 1.902; H = 256 1200 1.824 / 1.833 / 1.816 / 1.829. The
            // last quarter behind the wait for the stores, of 16 from 8 / 12 / 14 on: H = 768 700 2.032 / 2.017 / 2.033; H = 256 1200 1.836 / 1.816 / 1.818; others within 0.8 %.
            if (!wait_x(i) || !wait_sent(both ? 2 * i : i)) break;
            if (!project(Int<0>{}, i)) break;
            if (!wait_acc()) break;
            x_half(Int<0>{}, Int<kFirstX>{}, i);
            if (both && !wait_sent(2 * i + 1)) break;
            if (!project(Int<1>{}, i)) break;
            constexpr int kLastX = kX - kX / 4;
            x_half(Int<kFirstX>{}, Int<kLastX>{}, i);
            // the gate warps overwrite the hidden codes once the hh half is complete
            if (i > 0) ok = ok && mbar_wait(bar_stored, (i - 1) & 1, abort_flag, 104);
            x_half(Int<kLastX>{}, Int<kX>{}, i);
            if (kExact && both) {
                if (!hh_both()) break;
                continue;
            }
            if (!hh_half(Int<0>{})) break;
            if (!hh_half(Int<1>{})) break;
        }
    }
}
// Out of line: as a branch or a second loop in the kernel it cost the other weights 1 to 3 % of a step.
template <int V, int C, int STEPS>
__device__ __noinline__ void issue_exact(uint8_t *smem, uint32_t tmem, GroupDev p, int n_rows, uint32_t hh_bytes0, uint32_t hh_bytes1) {
    issue<V, C, STEPS, GroupConst<V, C, STEPS>::kZeroRows>(smem, tmem, p, n_rows, 0, hh_bytes0, hh_bytes1);
}

// A row of the recurrent weights of a gate from its place in shared memory (two K blocks of 64 in the 128-byte swizzle) to its lane of tensor
// memory; returns whether one of them is not finite, where that matters. All eight loads go ahead of the stores: unrolled once the set-up of a layer
// with few rows takes 0.5 us more. Out of line because it runs once: in the kernel either form of the loop moved the code of the steps, and each made another form
// of them 0.6 to 1.6 % slower (us per step, unrolled 8 : 1 : this; H = 384 32 chunks 1.163 : 1.179 : 1.155, H = 768 300 1.757 : 1.743 : 1.738, H = 1024 240
// 1.892 : 1.863 : 1.861; the largest losses of this one 256 64 1.126 : 1.146 : 1.143, 768 170 1.441 : 1.440 : 1.455).
template <int V, int C, int STEPS>
__device__ __noinline__ bool recurrent_weights(uint32_t row, uint32_t t_w, int lane) {
    using K = GroupConst<V, C, STEPS>;
    __half2 zeros[2] = {__half2half2(__ushort_as_half(0)), __half2half2(__ushort_as_half(0))};
#pragma unroll
    for (int v = 0; v < 8; ++v) {
        const uint32_t at = row + (v >> 2) * 16384;
        const uint4 lo = lds128(at + (((2 * (v & 3)) ^ (lane & 7)) << 4)), hi = lds128(at + (((2 * (v & 3) + 1) ^ (lane & 7)) << 4));
        tmem_st_32x8(t_w + v * 8, lo, hi);
        if (K::kZeroRows) {
            add_zero_times(zeros[0], lo);
            add_zero_times(zeros[1], hi);
        }
    }
    const __half2 sum = __hadd2(zeros[0], zeros[1]);
    return K::kZeroRows && (__hisnan(__low2half(sum)) || __hisnan(__high2half(sum)));
}

// The groups of chunk rows share the x part of the contraction (its MMAs read their A operand from shared memory, so
// one for both) and go through the rest of the step one after the other: while one is exchanged, the other
// is projected or computed.
template <int V, int C, int STEPS>
__global__ void __launch_bounds__(kGThreads, 1)
lstm_group_kernel(const __grid_constant__ CUtensorMap tm_w,    // w_up [4H, 2R] f16, boxes 128 x 64
                  const __grid_constant__ CUtensorMap tm_x,    // x_down [T, 2, B, 64] f16, boxes of all rows
                  const __grid_constant__ CUtensorMap tm_dn,   // dn_hh [R, H] int8, boxes 128 x 128
                  const __grid_constant__ CUtensorMap tm_h0,   // h_0 [H/128, B, 128] int8, boxes of a group's rows; GATHER: of all K blocks
                  const __grid_constant__ CUtensorMap tm_o,    // SPLIT: h_out [T, B, H], boxes of the first group's rows x 128
                  const __grid_constant__ CUtensorMap tm_ol,   // and of the second's
                  const GroupDev p) {
    using K = GroupConst<V, C, STEPS>;
    constexpr GroupForm F = K::F;
    constexpr GroupLayout L = K::L;
    constexpr bool kGather = K::kGather, kByPair = K::kByPair, kTwoSteps = K::kTwoSteps, kFourSteps = K::kFourSteps, kOneProj = K::kOneProj;
    constexpr int G = K::G, S = K::S, H = K::H, kXSlots = K::kXSlots, kTile = K::kTile, kHhTile = K::kHhTile;
    constexpr int kPieces = K::kPieces, kPairs = K::kPairs, kDnTs = K::kDnTs, kDnCol = K::kDnCol;
    extern __shared__ uint8_t smem_raw[];
    // every CTA of the cluster computes the same offset, so peers' buffers are at the same
    // shared-window offsets as this CTA's
    uint8_t *smem = reinterpret_cast<uint8_t *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L.bars);
    uint64_t *bar_once = bars + kBarOnce, *bar_x = bars + K::kBarXAt, *bar_x_free = bars + K::kBarXFreeAt, *bar_acc_free = bars + kBarAccFree;
    uint64_t *bar_proj = bars + kBarProj, *bar_acc = bars + kBarAcc, *bar_hh = bars + kBarHh, *bar_code = bars + kBarCode;
    uint64_t *bar_sum = bars + kBarSum, *bar_sent = bars + kBarSent, *bar_stored = bars + kBarStored, *bar_h = bars + kBarH;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + L.misc);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + L.misc + 4);

    const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x) >> 5, 0), lane = threadIdx.x & 31;
    const int rank = int(cluster_ctarank());
    const int m0 = (blockIdx.x / C) * p.rows;          // first chunk row of the cluster
    const int n_rows = min(p.rows, p.B - m0);          // and how many it has
    const int n0 = rank * kGUnits;
    auto rows_of = [&](int e) { return min(max(n_rows - F.rows * e, 0), F.rows); };
    // by pair: rows per pair, and those of this one
    const int pair = rank >> 1, half = rank & 1;
    const int per_pair = kByPair ? (p.rows + C / 2 - 1) / (C / 2) : 0;
    const int own_rows = kByPair ? min(max(n_rows - pair * per_pair, 0), per_pair) : 0;
    // pieces of a group that this CTA adds up, and bytes of hh_down rows that the group receives from peers
    auto pieces_below = [&](unsigned n) { return (n + unsigned(C - 1 - rank)) / C; };   // own ones among the first n of all groups
    auto pieces_of = [&](int e) { return (unsigned(rows_of(e)) + 3) / 4; };
    auto own_pieces = [&](int e) { return int(pieces_below(kPieces * e + pieces_of(e)) - pieces_below(kPieces * e)); };
    auto hh_bytes = [&](int e) {
        const unsigned rows = rows_of(e), pieces = pieces_of(e);
        const bool owns_last = pieces > 0 && (kPieces * e + pieces - 1) % C == unsigned(rank);   // which may have fewer than four rows
        return (rows - 4 * own_pieces(e) + (owns_last ? 4 * pieces - rows : 0)) * 256;
    };
    const bool both = G > 1 && n_rows > F.rows;        // the last cluster may have nothing in its second group
    auto time_of = [&](int i) { return p.reverse ? p.T - 1 - i : i; };
    if (threadIdx.x == 0) {
        auto arrivals = [&](int b) {   // warps that arrive, or one arrival with the expected bytes
            if (b == kBarAccFree) return kGather || both ? kGEpiWarps : kGEpiWarps / 2;
            if (b >= kBarWRead && b < kBarWRead + 4) return 4;
            if (b >= kBarWRead) return 1;
            if (kGather) return !kByPair && b == kBarHh ? kGEpiWarps : 1;
            return b == kBarCode || b == kBarCode + 1 || b == kBarSent ? kGEpiWarps / 2 : 1;
        };
#pragma unroll
        for (int b = 0; b < (kFourSteps ? kGBars : kBarX4); ++b)
            if (kGather || (b / 2 != kBarSum / 2 && b / 2 != kBarHh / 2)) mbar_init(&bars[b], arrivals(b));
        *abort_flag = 0;
        fence_barrier_init();
        if constexpr (kByPair) {
            mbar_arrive_expect_tx(&bar_hh[0], uint32_t(n_rows) * 256);
            if (p.T > 1) mbar_arrive_expect_tx(&bar_h[0], uint32_t(own_rows) * H);
        } else if constexpr (kGather) {
            for (int s = 0; s < 2; ++s)
                if (s + 1 < p.T) mbar_arrive_expect_tx(&bar_h[s], uint32_t(n_rows) * H);
        }
    }
    // SPLIT: the barriers whose counts are those of the CTA's own pieces, by a second thread. Code that runs once costs its instruction fetches, and all
    // that the first thread does stands in front of the loads of the weights (pieces counted one by one by that thread: 330 cycles later).
    if (!kGather && threadIdx.x == 64) {
        for (int e = 0; e < 2; ++e) {
            const int n = own_pieces(e);
            mbar_init(&bar_hh[e], 1 + (kGEpiWarps / 2) * n);
            mbar_init(&bar_sum[e], 1 + 4 * n);
            fence_barrier_init();
            if (e > 0 && !both) break;
            mbar_arrive_expect_tx(&bar_hh[e], hh_bytes(e));
            if (n > 0) mbar_arrive_expect_tx(&bar_sum[e], uint32_t(n) * (C - 1) * 2048);
        }
    }
    if (K::kZeroRows) {
        for (int o = threadIdx.x * 16; o < L.dn - L.hh; o += kGThreads * 16)
            *reinterpret_cast<uint4 *>(smem + L.hh + o) = make_uint4(0, 0, 0, 0);
        fence_proxy_async_smem();
    }
    if (warp == 1) tmem_alloc(tmem_slot, kGTmemCols);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    uint64_t *bar_w = bars + kBarW, *bar_w_read = bars + kBarWRead, *bar_start = bars + kBarStart;
    if (warp == 0 && elect_one()) {
        // The recurrent half of the gate weights comes by way of the places of the x half: read by the threads from global memory,
        // one row per lane, every load touched 32 lines. Layer of one step, us, x_down included, that against this: H = 384 32 chunks 16.7 : 14.6,
        // H = 768 300 20.7 : 17.1, 500 18.7 : 15.1, 1024 19.5 : 16.6, H = 1024 200 20.6 : 16.6.
        for (int g = 0; g < 4; ++g) {
            mbar_arrive_expect_tx(&bar_w[g], 32768);
            for (int kb = 0; kb < 2; ++kb) tma_load_2d(smem + (g * 2 + kb) * 16384, &tm_w, &bar_w[g], kb * 64, g * H + n0);
        }
        // what stays, and the initial hidden rows
        constexpr int kDnTile = K::kDnRows * 128, kDnTiles = (L.h - L.dn) / kDnTile;   // the last K blocks
        mbar_arrive_expect_tx(bar_once, kGWxBytes);
        mbar_arrive_expect_tx(bar_start, kDnTiles * kDnTile + (kGather ? C : G) * kTile);
        for (int b = 0; b < kDnTiles; ++b)
            tma_load_2d(smem + L.dn + b * kDnTile, &tm_dn, bar_start, kGather ? (kDnTs / 4 + b) * kGUnits : n0, kByPair ? half * 64 : 0);
        // step 0 projects the layer's initial hidden state
        for (int e = 0; e < G; ++e)
            tma_load_3d(smem + L.h + (kByPair ? 0 : kGather ? C : e) * kTile, &tm_h0, bar_start, 0,
                        kByPair ? m0 + pair * per_pair : m0 + F.rows * e, kGather ? 0 : rank);
        for (int g = 0; g < 4; ++g) {
            if (!mbar_wait(&bar_w_read[g], 0, abort_flag, 108)) break;
            for (int kb = 0; kb < 2; ++kb)
                tma_load_2d(smem + (g * 2 + kb) * 16384, &tm_w, bar_once, kGRank + kb * 64, g * H + n0);
        }
    }
    bool non_finite = false;   // one of the recurrent gate weights
    if (warp >= 2) {
        // warp = (lane quadrant, gate), thread = row of the block: first projection weights, then the hh half of the gate weights
        const int q = warp & 3, g = (warp - 2) >> 2;
        const uint32_t t_lane = tmem + (uint32_t(q * 32) << 16);
        // K steps g, g + 4, .. of the projection rows, of all units or this CTA's
        // (M = 64: row 16 q + i in lane 32 q + i)
        const int dn_row = kByPair ? half * 64 + q * 16 + (lane & 15) : q * 32 + lane;
        const uint4 *dn = reinterpret_cast<const uint4 *>(p.dn + size_t(dn_row) * H + (kGather ? 0 : n0));
#pragma unroll 1
        for (int s = g; s < kDnTs; s += 4) tmem_st_32x8(t_lane + kDnCol + s * 8, __ldg(dn + 2 * s), __ldg(dn + 2 * s + 1));
        if (__all_sync(0xffffffffu, mbar_wait(&bar_w[g], 0, abort_flag, 109)))
            non_finite = recurrent_weights<V, C, STEPS>(smem_u32(smem) + g * 32768 + (q * 32 + lane) * 128, t_lane + kGTmemW + g * 64, lane);
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_w_read[g]);
        tmem_st_wait();
        tc_fence_before_sync();
    }
    bool finite = true;
    if constexpr (K::kZeroRows) finite = !__syncthreads_or(non_finite);
    else __syncthreads();
    tc_fence_after_sync();
    // GATHER: a CTA loads the initial hidden rows of its peers' units too, and a layer of one step stores the final ones, of its
    // own units and to the same place, without having heard from them: no CTA passes the barrier before they have landed.
    if (kGather && warp < 2) mbar_wait(bar_start, 0, abort_flag, 97);
    // Every barrier of the cluster is initialised before any CTA may store to a peer: each warp passes this once. SPLIT: what a role prepares without
    // its peers stands in front of it, where there is time: behind it the set-up of sixteen warps held the issuer up for 900 cycles. (GATHER, which has
    // less of it: no gain, and steps up to 1 % slower from where the code then lies.)
    auto peers_ready = [&]() { cluster_sync_all(); };
    if (kGather) peers_ready();

    if (warp == 0) {
        // ------------------------------ loader (one thread) -----------------------------
        bool ok = true;
        auto load_x = [&](int i) {
            const int s = (K::kTwoStepsWide ? i + 1 : i) & (kXSlots - 1), u = (K::kTwoStepsWide ? i + 1 : i) / kXSlots;
            if (u > 0) ok = ok && mbar_wait(&bar_x_free[s], (u - 1) & 1, abort_flag, 96);
            if (!ok) return;
            if constexpr (kTwoSteps || kFourSteps) {
                const bool twice = s < K::X.steps - 1;   // the last slots repeat the first
                mbar_arrive_expect_tx(&bar_x[s], 2 * K::X.tile * (twice ? 2 : 1));
                for (int kb = 0; kb < 2; ++kb)
                    for (int n = 0; n < (twice ? 2 : 1); ++n)
                        tma_load_4d(smem + L.x + kb * K::X.kb + (s + kXSlots * n) * K::X.slot, &tm_x, &bar_x[s], 0, m0, kb, time_of(i));
            } else if constexpr (K::kTwoStepsWide) {
                // steps i and i + 1, the odd one in front
                const int from = max(i, 0), to = min(i + 2, p.T);
                mbar_arrive_expect_tx(&bar_x[s], 2 * K::X.tile * (to - from));
                for (int t = from; t < to; ++t)
                    for (int kb = 0; kb < 2; ++kb)
                        tma_load_4d(smem + L.x + s * K::X.slot + kb * K::X.kb + (1 - (t & 1)) * K::X.tile, &tm_x, &bar_x[s], 0, m0, kb, time_of(t));
            } else {
                mbar_arrive_expect_tx(&bar_x[s], 2 * K::X.tile);
                tma_load_4d(smem + L.x + s * K::X.slot, &tm_x, &bar_x[s], 0, m0, 0, time_of(i));
            }
        };
        constexpr int kEarly = K::kTwoStepsWide ? 1 : 0;   // windows that begin before step 0
        if constexpr (!kGather) {
            if (elect_one())
                for (int i = -kEarly; i < min(p.T, kXSlots - kEarly); ++i) load_x(i);
            __syncwarp();
            peers_ready();
        }
        if (elect_one()) {
            if constexpr (kGather) {
                for (int i = -kEarly; i < p.T && ok; ++i) load_x(i);
            } else {
                // between the loads the stores of the hidden rows
                for (int i = 0; i < p.T && ok; ++i) {
                    if (K::kTwoStepsWide && i + 1 < p.T) load_x(i + 1);   // of two tiles, the other one is in use
                    for (int e = 0; e < (both ? 2 : 1) && ok; ++e) {
                        ok = mbar_wait(&bar_code[e], i & 1, abort_flag, 107);
                        if (ok) tma_store_3d(e > 0 ? &tm_ol : &tm_o, smem + L.h + e * kTile, n0, m0 + F.rows * e, time_of(i));
                    }
                    tma_store_commit();
                    if (!K::kTwoStepsWide && i + kXSlots < p.T) load_x(i + kXSlots);
                    tma_store_wait_read<0>();
                    mbar_arrive(bar_stored);
                }
                tma_store_wait_all<0>();
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (!kGather) peers_ready();
        if (!K::kZeroRows || finite) issue<V, C, STEPS, false>(smem, tmem, p, n_rows, own_rows, hh_bytes(0), hh_bytes(1));
        else issue_exact<V, C, STEPS>(smem, tmem, p, n_rows, hh_bytes(0), hh_bytes(1));
    } else {
        // ------------------------------ gates -------------------------------------------
        // thread = hidden unit. GATHER: a quarter of the rows; SPLIT: half of the rows of one group, eight warps each, so
        // that one group's waits are the other's time
        const int q = warp & 3;
        const int e = kGather ? 0 : (warp - 2) >> 3, part = ((warp - 2) >> 2) & (kGather ? 3 : 1);
        constexpr int kParts = kGather ? 4 : 2;
        constexpr int kShare = F.rows / kParts;
        const int r0 = part * kShare, my_rows = min(max(rows_of(e) - r0, 0), kShare);
        const int unit = n0 + q * 32 + lane;
        const float b_i = __ldg(p.bias + unit), b_f = __ldg(p.bias + H + unit);
        const float b_g = __ldg(p.bias + 2 * H + unit), b_o = __ldg(p.bias + 3 * H + unit);
        float *c_at = p.c + int64_t(m0 + F.rows * e + r0) * H + unit;
        float2 c2[kPairs];
#pragma unroll
        for (int j = 0; j < kPairs; ++j)
            c2[j] = make_float2(2 * j < my_rows ? c_at[int64_t(2 * j) * H] : 0.f, 2 * j + 1 < my_rows ? c_at[int64_t(2 * j + 1) * H] : 0.f);
        const uint32_t t_lane = tmem + (uint32_t(q * 32) << 16);
        bool ok = true;
        using Acc = uint32_t[4][4];   // [gate][row] of two pairs
        auto codes = [&](const Acc &a, int k, float2 &c) {
            return lstm_cell_codes(a[0][2 * k], a[0][2 * k + 1], a[1][2 * k], a[1][2 * k + 1], a[2][2 * k], a[2][2 * k + 1],
                                   a[3][2 * k], a[3][2 * k + 1], make_float2(b_i, b_i), make_float2(b_f, b_f),
                                   make_float2(b_g, b_g), make_float2(b_o, b_o), c);
        };

        if constexpr (kByPair) {
            // What a CTA sends leaves in rows of 128 bytes, eight lanes each (see below). The four warps of a quarter stage together, one
            // projected row or four rows of codes, in two slots in turn: the barrier after one batch is staged also
            // says that the slot of the batch before has been read.
            const uint32_t stage = smem_u32(smem + L.stage) + part * 512;
            uint32_t slot = 0;
            // the pair's row `part` of this CTA's columns: lanes 8 j .. 8 j + 7 of warps 0 and 1 send it to the CTA 4 q + j behind this one
            const bool projects = part < own_rows;
            const int p_row = pair * per_pair + part;
            const uint32_t p_to = uint32_t((4 * q + (lane >> 3) + rank) % C);
            const uint32_t p_dst = map_to_rank(smem_u32(smem + L.hh + half * kHhTile) + p_row * 128 + (lane & 7) * 16, p_to);
            const uint32_t p_bar = map_to_rank(smem_u32(bar_hh), p_to);
            // codes: row q of the quarter, lanes 0-7 to the first CTA of the pair that owns it, 8-15 to the second
            const int h_row = r0 + q, h_pair = h_row / per_pair, h_own = h_row - h_pair * per_pair;
            const bool sends = lane < 16 && q < my_rows;
            const uint32_t h_to = sends ? uint32_t(2 * h_pair + (lane >> 3)) : uint32_t(rank);
            const uint32_t h_dst = map_to_rank(smem_u32(smem + L.h) + rank * kTile + h_own * 128 + (lane & 7) * 16, h_to);
            const uint32_t h_bar = map_to_rank(smem_u32(bar_h), h_to);
            // the piece of a staged row that belongs at a place of the 128-byte swizzle
            const uint32_t p_src = stage + ((lane ^ p_row) & 7) * 16, h_src = stage + q * 128 + ((lane ^ h_own) & 7) * 16;
            const int64_t at = int64_t(m0 + h_row) * H + n0 + ((lane ^ h_own) & 7) * 16;
            const float sc = (1.0f / 127.0f) * __ldg(p.dn_scale + half * 64 + q * 16 + (lane & 15));  // operand order of the dequant GEMM: sa * sb
            int8_t *h_out = p.h_out + int64_t(time_of(0)) * p.B * H + at;
            const int64_t plane = int64_t(p.reverse ? -p.B : p.B) * H;
            // A warp whose wait ran out goes on without waiting, sending or storing, as below.
            for (int i = 0; i < p.T; ++i, h_out += plane) {
                // ---- projection of the pair's h_{i-1}: int32 -> f16, to every CTA ----
                if (projects) {
                    ok = ok && mbar_wait(&bar_proj[0], i & 1, abort_flag, 102);
                    slot ^= 2048;
                    tc_fence_after_sync();
                    uint32_t v, next;
                    tmem_ld_32x2(t_lane + K::kAcc + part, v, next);
                    tmem_ld_wait();
                    if (lane < 16) sts16(stage + slot + q * 32 + lane * 2, __half_as_ushort(__float2half_rn(float(int(v)) * sc)));
                    tc_fence_before_sync();
                    quad_sync(1 + part);
                    if (ok && q < 2) store_to_peer(p_dst, lds128(p_src + slot), p_bar);
                }
                // ---- gates, cell update, hidden codes: all four rows, sent as soon as they are staged ----
                ok = ok && mbar_wait(&bar_acc[0], i & 1, abort_flag, 103);
                Acc a;
                if (my_rows > 0) {
                    tc_fence_after_sync();
#pragma unroll
                    for (int g = 0; g < 4; ++g) tmem_ld_32x4(t_lane + g * S + r0, a[g]);
                    tmem_ld_wait();
                    tc_fence_before_sync();
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_acc_free);
                if (my_rows == 0) continue;
                slot ^= 2048;
                auto stage_pair = [&](int j) {
                    const int2 h = codes(a, j, c2[j]);
                    sts8(stage + slot + 2 * j * 128 + q * 32 + lane, h.x);
                    sts8(stage + slot + (2 * j + 1) * 128 + q * 32 + lane, h.y);
                };
                stage_pair(0);
                if (my_rows > 2) stage_pair(kPairs - 1);
                quad_sync(1 + part);
                if (ok && sends) {
                    const uint4 v = lds128(h_src + slot);
                    if (i + 1 < p.T) store_to_peer(h_dst, v, h_bar);
                    if (lane < 8) {
                        *reinterpret_cast<uint4 *>(h_out) = v;
                        if (i + 1 == p.T) *reinterpret_cast<uint4 *>(p.h_state + at) = v;
                    }
                }
            }
        } else if constexpr (kGather) {
            // Two rows at a time leave as rows of 128 bytes, eight lanes each: the network between the SMs moves 64
            // contiguous bytes to one CTA in the time of 16 (20.7 against 9.5 B per cycle and SM, measured with
            // six CTAs sending to each other). A warp holds 32 bytes of a row, so the four warps of a quarter stage
            // together, in two slots in turn: the barrier after one batch is staged also says that the slot of
            // the batch before has been read.
            const uint32_t stage = smem_u32(smem + L.stage) + part * 256;
            uint32_t slot = 0;
            // lanes 0-15 send to the CTA q behind this one, 16-31 to that q + 4 behind; the last sixteen of the four warps store
            const int s_row = (lane >> 3) & 1, s_to = q + 4 * (lane >> 4), s_piece = (lane ^ (r0 + s_row)) & 7;
            const uint32_t to = uint32_t((s_to + rank) % C);
            // Piece c of row r lies at place c ^ (r & 7) of the 128-byte swizzle. A share starts at a multiple of its size, a power of
            // two, so the row j rows on has its place at exclusive or j.
            const uint32_t dst = map_to_rank(smem_u32(smem + L.h) + rank * kTile + (r0 + s_row) * 128 + (lane & 7) * 16, to);
            const uint32_t src = stage + s_row * 128 + s_piece * 16;
            const uint32_t dst_bar = map_to_rank(smem_u32(bar_h), to);
            const float sc = (1.0f / 127.0f) * __ldg(p.dn_scale + q * 32 + lane);   // operand order of the dequant GEMM: sa * sb
            const uint32_t hh = smem_u32(smem + L.hh) + (q >> 1) * kHhTile + (F.rows == 8 ? 1024 : 0) + r0 * 128 +
                                (((q & 1) * 4 + (lane >> 3)) ^ (r0 & 7)) * 16 + (lane & 7) * 2;
            const int64_t at = int64_t(m0 + r0 + s_row) * H + n0;   // plus the piece
            int8_t *h_out = p.h_out + int64_t(time_of(0)) * p.B * H + at;
            const int64_t plane = int64_t(p.reverse ? -p.B : p.B) * H;
            // A warp whose wait ran out walks the remaining steps without waiting, sending or storing: the
            // three it shares a slot with meet it at every barrier until their own waits give up.
            for (int i = 0; i < p.T; ++i, h_out += plane) {
                // ---- projection of h_{i-1}: int32 -> f16, into the operand of the hh half ----
                ok = ok && mbar_wait(&bar_proj[0], i & 1, abort_flag, 102);
                FLUKE_STAMP(blockIdx.x == 0 && warp == 2 && lane == 0, i * 16 + 6, clock64());
                if (my_rows > 0) {
                    tc_fence_after_sync();
                    uint32_t v[4];
                    tmem_ld_32x4(t_lane + K::kAcc + r0, v);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 2 * kPairs; ++j)
                        if (j < my_rows)
                            sts16((hh ^ (j << 4)) + j * 128, __half_as_ushort(__float2half_rn(float(int(v[j])) * sc)));
                    tc_fence_before_sync();
                    fence_proxy_async_smem();
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_hh);
                FLUKE_STAMP(blockIdx.x == 0 && warp == 2 && lane == 0, i * 16 + 7, clock64());
                // ---- gates, cell update, hidden codes ----
                uint32_t cols[4];
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    cols[g] = t_lane + (K::kTwoStepsWide ? 3 * (g & 1) + (g >> 1) + 1 - (i & 1) : g) * S + r0 + (kTwoSteps ? ((i ^ (g >> 1)) & 1) * 8 : 0);
                    if (kFourSteps) {
                        cols[g] += 8 * (finite ? (i - g) & 3 : 0);
                        asm volatile("" : "+r"(cols[g]));   // worked out in front of the wait
                    }
                }
                ok = ok && mbar_wait(&bar_acc[0], i & 1, abort_flag, 103);
                FLUKE_STAMP(blockIdx.x == 0 && warp == 2 && lane == 0, i * 16 + 12, clock64());
                Acc a;
                if (my_rows > 0) {
                    tc_fence_after_sync();
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        if (kPairs > 1) tmem_ld_32x4(cols[g], a[g]);
                        else tmem_ld_32x2(cols[g], a[g][0], a[g][1]);
                    }
                    tmem_ld_wait();
                    tc_fence_before_sync();
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_acc_free);
#pragma unroll
                for (int j = 0; j < kPairs; ++j) {
                    if (2 * j >= my_rows) break;
                    slot ^= 1024;
                    const int2 h = codes(a, j, c2[j]);
                    sts8(stage + slot + q * 32 + lane, h.x);
                    sts8(stage + slot + 128 + q * 32 + lane, h.y);
                    quad_sync(1 + part);
                    if (ok && 2 * j + s_row < my_rows) {
                        const uint4 v = lds128((src ^ (j << 5)) + slot);
                        if (s_to < C && i + 1 < p.T) store_to_peer(dst + (i & 1) * (C * kTile) + j * 256, v, dst_bar + (i & 1) * 8);
                        if (s_to == 7) {
                            const int off = 2 * j * H + ((s_piece ^ (2 * j)) << 4);
                            *reinterpret_cast<uint4 *>(h_out + off) = v;
                            if (i + 1 == p.T) *reinterpret_cast<uint4 *>(p.h_state + at + off) = v;
                        }
                    }
                }
                FLUKE_STAMP(blockIdx.x == 0 && warp == 2 && lane == 0, i * 16 + 8, clock64());
            }
        } else if (e == 0 || both) {
            // The codes go straight into the operand of the projection (128-byte swizzle), from where the issuer also stores them.
            // Twelve rows on is four on in the swizzle: exclusive or 4, and exclusive or j mod 8 for the rows behind.
            const uint32_t code = smem_u32(smem + L.h) + e * kTile + r0 * 128 + (((q * 2 + (lane >> 4)) ^ (r0 & 7)) << 4) + (lane & 15);
            auto code_at = [&](int j) { return (code ^ ((j & 7) << 4)) + j * 128; };
            const uint32_t t_acc = t_lane + F.rows * e + r0;
            const uint32_t t_proj = t_lane + K::kAcc + (kOneProj ? 0 : e * F.n) + part * 4;
            const float sc = (1.0f / 127.0f) * __ldg(p.dn_scale + q * 32 + lane);   // operand order of the dequant GEMM: sa * sb
            const uint32_t recv = smem_u32(smem + L.recv) + uint32_t(q * 32 + lane) * 16;
            const uint32_t bar_sum_e = smem_u32(&bar_sum[e]), bar_hh_e = smem_u32(&bar_hh[e]);
            const uint32_t stage = smem_u32(smem + L.stage) + (warp - 2) * 128;
            const uint32_t hh = smem_u32(smem + L.hh) + (2 * e + (q >> 1)) * kHhTile;
            const int s_row = 2 * part + ((lane >> 2) & 1), s_piece = (q & 1) * 4 + (lane & 3);
            const int own = own_pieces(e);
            // Where the projected pieces and the rows of hh_down go. What stays in the CTA is stored there by itself: st.async takes it through the
            // network like the rest, whose bytes bound the step where several clusters share a GPC (clusters of 1024 chunks had periods of 4520 to 5080
            // cycles). Us per step of short runs, below the power limit, in the network : kept out, H = 768 700 chunks 2.138 : 2.114, 900 2.801 : 2.673, 1024 2.942 : 2.716; H = 1024 500 2.776 : 2.657, 700 2.911 :
            // 2.823; H = 384 900 2.041 : 2.074, 1500 2.685 : 2.615; H = 512 1400 2.863 : 2.728. Up to 16 rows (GATHER) it costs 2 to 8 %: 300 chunks 1.730 : 1.814.
            uint32_t p_to[kPieces / 2], p_bar[kPieces / 2];
            int p_own = 0;   // one bit per piece that the CTA adds up itself
#pragma unroll
            for (int k = 0; k < kPieces / 2; ++k) {
                const uint32_t n = uint32_t(kPieces * e + 2 * k + part), to = n % C;
                p_to[k] = map_to_rank(recv + ((n / C) * C + rank) * 2048, to);
                if (to == rank) p_own |= 1 << k, p_to[k] = recv + ((n / C) * C + rank) * 2048;
                p_bar[k] = map_to_rank(bar_sum_e, to);
            }
            int p_arrivals = 0;   // of those that there are
#pragma unroll
            for (int k = 0; k < kPieces / 2; ++k) p_arrivals += (p_own >> k & 1) && 4 * (2 * k + part) < rows_of(e);
            if (p_arrivals == 0) p_own = 0;
            // Every other eight columns' pieces have rows 2 and 3 in front: what a warp reads of them, two rows of 32 columns, then lies in all banks instead
            // of half of them. The sums stood 440 to 600 cycles behind their arrival, now 380 (us per step: H = 768 400 chunks 2.076 -> 2.052, 900 2.827 ->
            // 2.793; H = 384 1500 2.738 -> 2.689; H = 512 1400 2.960 -> 2.813; H = 768 1024 2.954 -> 2.959).
            const bool swap = lane & 8;
            // the first of the group's pieces that this CTA adds up
            const int k_first = (rank + C * ((kPieces * e + C - 1 - rank) / C)) - kPieces * e, rows_e = rows_of(e);
            const uint32_t mine_first = recv + ((part ^ (swap ? 1 : 0)) * 8) + ((kPieces * e + k_first) / C) * C * 2048;
            uint32_t hh_to[(C + 3) / 4], bar_to[(C + 3) / 4];
#pragma unroll
            for (int d = 0; d < C; d += 4) {
                int to = d + (lane >> 3) + rank;            // start with a different peer in every CTA
                if (to >= C) to -= C;
                if (to >= C) to = 0;
                hh_to[d / 4] = map_to_rank(hh, to);
                bar_to[d / 4] = map_to_rank(bar_hh_e, to);
            }
            peers_ready();
            for (int i = 0; i < p.T && ok; ++i) {
                // ---- projection of this CTA's h_{i-1}: every other piece to its owner ----
                ok = mbar_wait(&bar_proj[e], i & 1, abort_flag, 102);
                if (!ok) break;
                tc_fence_after_sync();
                uint32_t v[kPieces / 2][4];
#pragma unroll
                for (int k = 0; k < kPieces / 2; ++k) tmem_ld_32x4(t_proj + 8 * k, v[k]);
                tmem_ld_wait();
                tc_fence_before_sync();
                if (kOneProj) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_sent);
                }
                FLUKE_STAMP(blockIdx.x == 0 && (warp == 2 || warp == 10) && lane == 0, i * 16 + 6 + e, clock64());
#pragma unroll
                for (int k = 0; k < kPieces / 2; ++k) {
                    if (4 * (2 * k + part) >= rows_of(e)) continue;
                    const uint4 w = make_uint4(swap ? v[k][2] : v[k][0], swap ? v[k][3] : v[k][1], swap ? v[k][0] : v[k][2], swap ? v[k][1] : v[k][3]);
                    if (p_own >> k & 1) sts128(p_to[k], w);
                    else store_to_peer(p_to[k], w, p_bar[k]);
                }
                // announced behind the last of the pieces: in between it held the others up (H = 768 900 chunks 2.659 -> 2.621, 1024 2.706 -> 2.682; H = 384
                // 1500 2.600 -> 2.633, others the same)
                if (p_own) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive_n(&bar_sum[e], p_arrivals);
                }
                // ---- the CTA's own pieces: summed, converted, to every CTA (two of the four rows) ----
                if (own > 0) {
                    ok = mbar_wait<true>(&bar_sum[e], i & 1, abort_flag, 105);
                    if (!ok) break;
                    if (q == 0 && part == 0 && lane == 0 && i + 1 < p.T)   // for the next step
                        mbar_arrive_expect_tx(&bar_sum[e], uint32_t(own) * (C - 1) * 2048);
                    FLUKE_STAMP(blockIdx.x == 0 && (warp == 2 || warp == 10) && lane == 0, i * 16 + 9 + e, clock64());
                    uint32_t at_mine = mine_first;
#pragma unroll 1
                    for (int k = k_first; 4 * k < rows_e; k += C, at_mine += C * 2048) {
                        int s0 = 0, s1 = 0;
#pragma unroll
                        for (int j = 0; j < C; ++j) {
                            const int2 w = lds64(at_mine + j * 2048);
                            s0 += w.x;
                            s1 += w.y;
                        }
                        __syncwarp();   // the piece before has left the staging rows
                        sts16(stage + lane * 2, __half_as_ushort(__float2half_rn(float(s0) * sc)));
                        sts16(stage + 64 + lane * 2, __half_as_ushort(__float2half_rn(float(s1) * sc)));
                        __syncwarp();
                        const uint4 w = lds128(stage + (lane & 7) * 16);
                        const int row = 4 * k + s_row;
                        const uint32_t at = row * 128 + ((s_piece ^ (row & 7)) << 4);
#pragma unroll
                        for (int d = 0; d < C; d += 4)
                            if (d + (lane >> 3) < C && row < rows_e) {
                                if (d == 0 && lane < 8) sts128(hh + at, w);
                                else store_to_peer(hh_to[d / 4] + at, w, bar_to[d / 4]);
                            }
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&bar_hh[e]);
                    }
                }
                // ---- gates, cell update, hidden codes ----
                ok = mbar_wait(&bar_acc[e], i & 1, abort_flag, 103);
                FLUKE_STAMP(blockIdx.x == 0 && (warp == 2 || warp == 10) && lane == 0, i * 16 + 12 + e, clock64());
                if (!ok) break;
                tc_fence_after_sync();
                Acc a[kPairs / 2];
#pragma unroll
                for (int b = 0; b < kPairs / 2; ++b)
#pragma unroll
                    for (int g = 0; g < 4; ++g)
                        tmem_ld_32x4(t_acc + (K::kTwoStepsWide ? 3 * (g & 1) + (g >> 1) + 1 - (i & 1) : g) * S + 4 * b, a[b][g]);
                tmem_ld_wait();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_acc_free);
#pragma unroll
                for (int j = 0; j < kPairs; ++j) {
                    const int2 h = codes(a[j / 2], j & 1, c2[j]);   // of rows that the group does not have as well: nothing reads them
                    sts8(code_at(2 * j), h.x);
                    sts8(code_at(2 * j + 1), h.y);
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar_code[e]);
                FLUKE_STAMP(blockIdx.x == 0 && (warp == 2 || warp == 10) && lane == 0, i * 16 + (e == 0 ? 15 : 11), clock64());
            }
            // the last codes are the final hidden state
            if (ok)
                for (int j = 0; j < my_rows; ++j) p.h_state[int64_t(m0 + F.rows * e + r0 + j) * H + unit] = int8_t(lds8(code_at(j)));
        } else {
            peers_ready();
        }
#pragma unroll
        for (int j = 0; j < kPairs; ++j) {
            if (2 * j < my_rows) c_at[int64_t(2 * j) * H] = c2[j].x;
            if (2 * j + 1 < my_rows) c_at[int64_t(2 * j + 1) * H] = c2[j].y;
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
    int form;         // see group_form
    int rows;         // rows per cluster
    int tiles;        // clusters
    bool most;        // the kernel of most steps per x MMA
};

using group_kernel_fn = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, GroupDev);
struct GroupKernel { group_kernel_fn fn; int smem; };
template <int V, int C, bool MOST>
constexpr GroupKernel group_kernel() {
    constexpr int steps = group_x_steps(V, C, MOST);
    return {lstm_group_kernel<V, C, steps>, group_layout(V, C, steps).dynamic};
}
#define FLUKE_GROUP_KERNELS(V, MOST) \
    {{}, {}, group_kernel<V, 2, MOST>(), group_kernel<V, 3, MOST>(), group_kernel<V, 4, MOST>(), group_kernel<V, 5, MOST>(), group_kernel<V, 6, MOST>(), \
     group_kernel<V, 7, MOST>(), group_kernel<V, 8, MOST>()}
#define FLUKE_GROUP_FORMS(MOST) \
    {FLUKE_GROUP_KERNELS(0, MOST), FLUKE_GROUP_KERNELS(1, MOST), FLUKE_GROUP_KERNELS(2, MOST), FLUKE_GROUP_KERNELS(3, MOST)}
const GroupKernel kGroupKernels[2][kGForms][kGMaxCtas + 1] = {FLUKE_GROUP_FORMS(false), FLUKE_GROUP_FORMS(true)};
#undef FLUKE_GROUP_FORMS
#undef FLUKE_GROUP_KERNELS

// Clusters of C CTAs of form V that the device runs at once with the largest shared memory a CTA can
// have (0: the form is not available).
int group_capacity(int V, int C) {
    static int known[64][kGForms][kGMaxCtas + 1];  // n + 1, or -1
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return 0;
    int &slot = known[dev][V][C];
    if (slot == 0) {
        int n = 0;
        // both kernels of the form at once: a caller that has run a long layer may capture a short one
        const void *fn = nullptr;
        bool ok = true;
        for (int most = 0; most < 2 && ok; ++most) {
            fn = reinterpret_cast<const void *>(kGroupKernels[most][V][C].fn);
            ok = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kGMaxSmem) == cudaSuccess;
        }
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

// How B rows of hidden size H are spread over clusters for T steps: as few waves of clusters as the largest row count allows, then
// evenly over all clusters of those waves.
bool group_plan(int T, int B, int H, GroupPlan *g) {
    if (H % kGUnits) return false;
    const int C = H / kGUnits;
    if (C < 2 || C > kGMaxCtas) return false;
    const int cap = group_capacity(kGForms - 1, C);
    if (cap < 1) return false;
    const int per_wave = cap * group_form(kGForms - 1).most;
    const int waves = (B + per_wave - 1) / per_wave;
    int tiles = cap * waves;
    if (tiles > (B + kGMinRows - 1) / kGMinRows) tiles = (B + kGMinRows - 1) / kGMinRows;
    g->rows = (B + tiles - 1) / tiles;
    g->tiles = (B + g->rows - 1) / g->rows;
    g->form = 0;
    while (g->rows > group_form(g->form).most) ++g->form;
    g->most = group_most_x_steps(T, g->rows, g->form, C);
    return group_capacity(g->form, C) > 0;
}

}  // namespace
}  // namespace fluke_sm100

extern "C" int fluke_sm100_lstm_small_clusters(int T, int B, int H, int *x_steps) {
    using namespace fluke_sm100;
    GroupPlan g;
    if (T < 1 || B < 1 || H < 1 || !group_plan(T, B, H, &g)) return 0;
    if (x_steps) *x_steps = group_x_steps(g.form, H / kGUnits, g.most);
    return g.rows;
}

// Runs the recurrence of one layer (x_down already computed) with the batch spread over small
// clusters, and writes the final hidden state. Returns -2 when the shape or the device is not covered.
extern "C" int fluke_sm100_lstm_layer_group(const void *layer, const void *x_down, void *stream) {
    using namespace fluke_sm100;
    const fluke_flstm_layer_t *l = static_cast<const fluke_flstm_layer_t *>(layer);
    const int T = l->T, B = l->B, H = l->H, R = l->R;
    GroupPlan g;
    if (R != kGRank || !group_plan(T, B, H, &g)) return -2;
    const int C = H / kGUnits;
    const GroupForm f = group_form(g.form);
    const GroupKernel &kn = kGroupKernels[g.most][g.form][C];

    GroupDev p;
    p.T = T; p.B = B; p.reverse = l->reverse;
    p.rows = g.rows;
    p.dn = static_cast<const int8_t *>(l->dn_hh_i8);
    p.bias = static_cast<const float *>(l->bias_f32);
    p.dn_scale = static_cast<const float *>(l->dn_hh_scale);
    p.c = static_cast<float *>(l->c_f32);
    p.h_out = static_cast<int8_t *>(l->h_out_i8);
    p.h_state = static_cast<int8_t *>(l->h_i8);
    p.trace = trace_buffer();

    CUtensorMap tm_w, tm_x, tm_dn, tm_h0, tm_o[2] = {};
    int rc = make_tmap_2d(&tm_w, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, l->w_up_f16, 4 * uint64_t(H), 2 * R, uint64_t(2 * R) * 2,
                          kGUnits, 64, true);
    if (rc) return rc;
    {
        // both K blocks of a row range in one box: the 128-byte blocks of a row are a dimension
        const uint64_t dims[4] = {64, uint64_t(B), 2, uint64_t(T)};
        const uint64_t strides[3] = {uint64_t(R) * 2, 128, uint64_t(B) * R * 2};
        const uint32_t box[4] = {64, uint32_t(f.groups * f.rows), group_x_steps(g.form, C, g.most) > 1 ? 1u : 2u, 1};
        rc = make_tmap_nd(&tm_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, x_down, 4, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
        if (rc) return rc;
    }
    const bool by_pair = group_by_pair(g.form, C);
    rc = make_tmap_2d(&tm_dn, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, l->dn_hh_i8, R, H, H, by_pair ? 64 : kGRank, 128, true);
    if (rc) return rc;
    {
        const uint64_t dims[3] = {128, uint64_t(B), uint64_t(C)};
        const uint64_t strides[2] = {uint64_t(H), 128};
        const uint32_t box[3] = {128, by_pair ? 8u : uint32_t(f.rows), uint32_t(f.gather ? C : 1)};
        rc = make_tmap_nd(&tm_h0, CU_TENSOR_MAP_DATA_TYPE_UINT8, l->h_i8, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
        if (rc) return rc;
    }
    // boxes of exactly the rows a group has: the rows behind them are another cluster's
    for (int e = 0; e < 2 && !f.gather; ++e) {
        const int box_rows = e == 0 ? min(g.rows, f.rows) : max(g.rows - f.rows, 1);
        rc = make_tmap_3d(&tm_o[e], CU_TENSOR_MAP_DATA_TYPE_UINT8, l->h_out_i8, T, B, H, H, uint64_t(B) * H, box_rows, 128, true);
        if (rc) return rc;
    }

    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(g.tiles * C);
    cfg.blockDim = dim3(kGThreads);
    cfg.dynamicSmemBytes = kn.smem;
    cfg.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&cfg, kn.fn, tm_w, tm_x, tm_dn, tm_h0, tm_o[0], tm_o[1], p);
}
