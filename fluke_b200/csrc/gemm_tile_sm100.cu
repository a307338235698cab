// gemm_tile_sm100.cu -- the GEMM family of gemm_sm100.cu for problems with few output tiles: one
// CTA per 128 x BN tile, everything of the tile in flight at once.
//
// The persistent kernel gives a CTA a whole 128 KB weight tile and 256 accumulator columns per
// step. With a few hundred rows that leaves most SMs idle and makes the busy ones run a long chain: a
// 128 KB load, 16 MMAs of 128 cycles, an epilogue over 128 columns per warp. Here a tile is 32 or 64
// output columns wide (64 = one head for the rotary form; gate and up rows stacked for the
// gated form): the load is 96 KB in two pieces, an MMA takes 33 to 45 cycles, eight epilogue warps
// hold 16 or 32 columns each and store them straight from registers. Two CTAs fit an SM. What is left
// of the time is latency (launch, first TMA load, MMA chain, stores).
//
// Row-major K-major operands as in gemm_sm100.cu; K a multiple of 128 bytes (the tensor maps walk the
// 128-byte K blocks of a row as a dimension of their own). Arithmetic per element is that of the
// persistent kernel's epilogues, in the same order: the bits are the same.

namespace fluke_sm100 {
namespace {

constexpr int kTileThreads = 320;  // warp 0 loader, warp 1 MMA issuer, warps 2-9 epilogue

struct GemmTileDev {
    int M, N, ld_out;
    int nkb, half_kb;        // K blocks of 128 bytes; blocks per load
    __half *out;
    const float *scale_a;
    float const_scale_a;
    const float *scale_b, *scale_b2;
    const float *sin_tab, *cos_tab;
    int seqlen, qk_cols;
};

// 16 accumulator rows x BN columns in the 16-lane x 256-bit shape: r[4 j + 2 k], r[4 j + 2 k + 1] are
// columns 8 j + 2 t, + 1 of row g + 8 k (g = lane / 4, t = lane % 4).
template <int BN>
__device__ __forceinline__ void tmem_ld_16rows(uint32_t taddr, uint32_t (&r)[BN / 2]) {
    static_assert(BN == 32 || BN == 64, "tile widths");
    if constexpr (BN == 32) tmem_ld_16x256_x4(taddr, r);
    else tmem_ld_16x256_x8(taddr, r);
}

// Byte offset of 16-byte piece c of row r in a staging tile of 2 BN bytes per row, swizzled so that
// both the fragment stores and the row reads are free of bank conflicts.
template <int BN>
__device__ __forceinline__ uint32_t tile_offset(uint32_t r, uint32_t c) {
    if constexpr (BN == 64) return sw128_offset(r, c);
    else return r * 64u + ((c ^ ((r >> 1) & 3u)) << 4);
}

// BN: output columns per CTA (32 or 64; 64 for the rotary form).
template <int KIND, int EPI, int BN>
__global__ void __launch_bounds__(kTileThreads, 2)
gemm_tile_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
                 const __grid_constant__ CUtensorMap tm_b2, const GemmTileDev p) {
    constexpr bool kDual = EPI == FLUKE_SM100_EPI_SILU;
    constexpr int N_MMA = kDual ? 2 * BN : BN;
    constexpr uint32_t kIdesc = make_idesc<KIND>(128, N_MMA);
    constexpr uint32_t kTmemCols = N_MMA <= 32 ? 32 : N_MMA <= 64 ? 64 : 128;
    constexpr int kABytes = 128 * 128, kBBytes = N_MMA * 128;  // one K block
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ uint64_t full_bar[2], done_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_word;
    volatile int *abort_flag = &abort_word;

    const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x) >> 5, 0), lane = threadIdx.x & 31;
    const int m0 = blockIdx.y * 128, n0 = blockIdx.x * BN;
    const int pieces = p.nkb > p.half_kb ? 2 : 1;
    uint8_t *sa = smem, *sb = smem + 2 * p.half_kb * kABytes;

    if (threadIdx.x == 0) {
        mbar_init(&full_bar[0], 1);
        mbar_init(&full_bar[1], 1);
        mbar_init(&done_bar, 1);
        abort_word = 0;
        fence_barrier_init();
        tma_prefetch_desc(&tm_a);
        tma_prefetch_desc(&tm_b);
        if (kDual) tma_prefetch_desc(&tm_b2);
    }
    if (warp == 1) {
        tmem_alloc(&tmem_slot, kTmemCols);
        dependency_trigger();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = tmem_slot;
    dependency_wait();

    if (warp == 0) {
        if (elect_one()) {
            for (int h = 0; h < pieces; ++h) {
                // blocks past the end of K read as zeros and are not multiplied
                mbar_arrive_expect_tx(&full_bar[h], p.half_kb * (kABytes + kBBytes));
                const int kb0 = h * p.half_kb;
                tma_load_3d(sa + kb0 * kABytes, &tm_a, &full_bar[h], 0, m0, kb0);
                if constexpr (kDual) {
                    // [gate rows of all blocks of the piece | up rows of all blocks of the piece]
                    tma_load_3d(sb + kb0 * kBBytes, &tm_b, &full_bar[h], 0, n0, kb0);
                    tma_load_3d(sb + kb0 * kBBytes + p.half_kb * (kBBytes / 2), &tm_b2, &full_bar[h], 0, n0, kb0);
                } else {
                    tma_load_3d(sb + kb0 * kBBytes, &tm_b, &full_bar[h], 0, n0, kb0);
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        bool ok = true;
        for (int h = 0; h < pieces && ok; ++h) {
            ok = mbar_wait(&full_bar[h], 0, abort_flag, 112);
            if (!ok) break;
            tc_fence_after_sync();
            if (elect_one()) {
                const int kb0 = h * p.half_kb, n = min(p.half_kb, p.nkb - kb0);
                const uint64_t ad = make_smem_desc_sw128(smem_u32(sa + kb0 * kABytes));
                const uint64_t bd = make_smem_desc_sw128(smem_u32(sb + kb0 * kBBytes));
                for (int kb = 0; kb < n; ++kb)
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint64_t a = ad + uint64_t(kb * (kABytes >> 4) + 2 * k);
                        if constexpr (kDual) {
                            const uint64_t g = bd + uint64_t(kb * (kBBytes >> 5) + 2 * k);
                            constexpr uint32_t kIdescHalf = make_idesc<KIND>(128, BN);
                            tc_mma<KIND>(tmem, a, g, kIdescHalf, (h | kb | k) != 0);
                            tc_mma<KIND>(tmem + BN, a, g + uint64_t(p.half_kb * (kBBytes >> 5)), kIdescHalf, (h | kb | k) != 0);
                        } else {
                            tc_mma<KIND>(tmem, a, bd + uint64_t(kb * (kBBytes >> 4) + 2 * k), kIdesc, (h | kb | k) != 0);
                        }
                    }
                if (h == pieces - 1) tc_commit(&done_bar);
            }
            __syncwarp();
        }
    } else {
        // Warp = 16 rows x all columns, in the 16-lane x 256-bit shape (as in the persistent kernel):
        // column factors and rotary tables are read in whole 32-byte sectors, the results go through
        // shared memory (the A tile's, which the MMAs have finished with) as 8 x 8 fragments and
        // leave in whole rows.
        const int q = warp & 3, hr = (warp - 2) >> 2;
        const int g8 = lane >> 2, t4 = lane & 3;
        const int r0 = q * 32 + hr * 16;   // first of the warp's rows in the tile
        const uint32_t t_base = tmem + (uint32_t(r0) << 16);
        float2 sa2[2];
        int rows[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            rows[k] = m0 + r0 + g8 + 8 * k;
            const float v = p.scale_a ? (rows[k] < p.M ? p.scale_a[rows[k]] : 0.f) : p.const_scale_a;
            sa2[k] = make_float2(v, v);
        }
        float2 sc[BN / 8], x2[kDual ? BN / 8 : 1];
#pragma unroll
        for (int j = 0; j < BN / 8; ++j) {
            sc[j] = *reinterpret_cast<const float2 *>(p.scale_b + n0 + 8 * j + 2 * t4);
            if constexpr (kDual) {
                sc[j] = make_float2(0.5f * sc[j].x, 0.5f * sc[j].y);  // the gated form works on gate / 2
                x2[j] = *reinterpret_cast<const float2 *>(p.scale_b2 + n0 + 8 * j + 2 * t4);
            }
        }
        constexpr bool kRot = EPI == FLUKE_SM100_EPI_ROTARY;
        static_assert(!kRot || BN == 64, "a rotary tile is one head");
        const bool rotate = kRot && n0 < p.qk_cols;
        float2 sn[2][kRot ? 4 : 1], cs[2][kRot ? 4 : 1];
        if constexpr (kRot) {
            if (rotate) {
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const int pos = rows[k] < p.M ? rows[k] % p.seqlen : 0;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        sn[k][j] = *reinterpret_cast<const float2 *>(p.sin_tab + pos * 32 + 8 * j + 2 * t4);
                        cs[k][j] = *reinterpret_cast<const float2 *>(p.cos_tab + pos * 32 + 8 * j + 2 * t4);
                    }
                }
            }
        }
        if (mbar_wait(&done_bar, 0, abort_flag, 113)) {
            tc_fence_after_sync();
            uint8_t *staging = sa + (warp - 2) * (16 * BN * 2);
            uint32_t a[BN / 2], u[kDual ? BN / 2 : 1];
            tmem_ld_16rows<BN>(t_base, a);
            if constexpr (kDual) tmem_ld_16rows<BN>(t_base + BN, u);
            tmem_ld_wait();
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                uint32_t w[BN / 8];
                auto acc = [&](int j) { return acc_to_float2<KIND>(a[4 * j + 2 * k], a[4 * j + 2 * k + 1]); };
                if constexpr (kRot) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float2 x0 = mul2(mul2(acc(j), sa2[k]), sc[j]);
                        const float2 x1 = mul2(mul2(acc(j + 4), sa2[k]), sc[j + 4]);
                        float2 lo = x0, hi = x1;
                        if (rotate) {
                            const float2 m = mul2(x1, sn[k][j]);
                            lo = fma2(x0, cs[k][j], make_float2(-m.x, -m.y));
                            hi = fma2(x0, sn[k][j], mul2(x1, cs[k][j]));
                        }
                        w[j] = pack_half2(lo.x, lo.y);
                        w[j + 4] = pack_half2(hi.x, hi.y);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < BN / 8; ++j) {
                        float2 o;
                        if constexpr (kDual) {
                            const float2 h = mul2(mul2(acc(j), sa2[k]), sc[j]);
                            const float2 up = mul2(mul2(acc_to_float2<KIND>(u[4 * j + 2 * k], u[4 * j + 2 * k + 1]), sa2[k]), x2[j]);
                            o = mul2(fma2(h, make_float2(tanh_approx(h.x), tanh_approx(h.y)), h), up);
                        } else if constexpr (EPI == FLUKE_SM100_EPI_DEQUANT) {
                            o = mul2(acc(j), mul2(sa2[k], sc[j]));
                        } else {
                            o = mul2(mul2(acc(j), sa2[k]), sc[j]);
                        }
                        w[j] = pack_half2(o.x, o.y);
                    }
                }
#pragma unroll
                for (int c = 0; c < BN / 32; ++c) {
                    const uint32_t f[4] = {w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]};
                    stmatrix_x4(staging + tile_offset<BN>(8 * k + (lane & 7), 4 * c + (lane >> 3)), f);
                }
            }
            __syncwarp();
            constexpr int kLanes = BN / 8;   // 16-byte pieces of a row
#pragma unroll
            for (int i = 0; i < 16 * kLanes / 32; ++i) {
                const int r = i * (32 / kLanes) + lane / kLanes, c = lane % kLanes, row = m0 + r0 + r;
                const uint4 v = *reinterpret_cast<const uint4 *>(staging + tile_offset<BN>(r, c));
                if (row < p.M) *reinterpret_cast<uint4 *>(p.out + int64_t(row) * p.ld_out + n0 + 8 * c) = v;
            }
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, kTmemCols);
    }
}

// Shared memory of a CTA with `rows_b` weight rows: both operands' K blocks, rounded up to two equal
// loads, and the slack for the manual 1024-byte alignment.
inline int tile_smem(int K, int rows_b) { return (K / 128 + 1) / 2 * 2 * (128 + rows_b) * 128 + 1024; }

template <int KIND, int EPI, int BN>
int tile_launch(const fluke_sm100_gemm_t *g, cudaStream_t stream) {
    constexpr bool kDual = EPI == FLUKE_SM100_EPI_SILU;
    constexpr int kMaxK = EPI == FLUKE_SM100_EPI_SILU || EPI == FLUKE_SM100_EPI_ROTARY ? 512 : 1024;   // as the persistent kernel
    if (g->K > kMaxK) return (int)cudaErrorInvalidValue;
    GemmTileDev p;
    p.M = g->M; p.N = g->N; p.ld_out = g->ld_out;
    p.nkb = g->K / 128; p.half_kb = (p.nkb + 1) / 2;
    p.out = static_cast<__half *>(g->out);
    p.scale_a = g->scale_a; p.const_scale_a = g->const_scale_a;
    p.scale_b = g->scale_b; p.scale_b2 = g->scale_b2;
    p.sin_tab = g->sin_tab; p.cos_tab = g->cos_tab;
    p.seqlen = g->seqlen > 0 ? g->seqlen : 1;
    p.qk_cols = g->qk_cols;
    const uint64_t da[3] = {128, uint64_t(g->M), uint64_t(p.nkb)}, db[3] = {128, uint64_t(g->N), uint64_t(p.nkb)};
    const uint64_t strides[2] = {uint64_t(g->K), 128};
    const uint32_t box_a[3] = {128, 128, uint32_t(p.half_kb)}, box_b[3] = {128, BN, uint32_t(p.half_kb)};
    CUtensorMap tm_a, tm_b, tm_b2;
    int rc = make_tmap_nd(&tm_a, CU_TENSOR_MAP_DATA_TYPE_UINT8, g->a, 3, da, strides, box_a, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    rc = make_tmap_nd(&tm_b, CU_TENSOR_MAP_DATA_TYPE_UINT8, g->b, 3, db, strides, box_b, CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    tm_b2 = tm_b;
    if (kDual) {
        rc = make_tmap_nd(&tm_b2, CU_TENSOR_MAP_DATA_TYPE_UINT8, g->b2, 3, db, strides, box_b, CU_TENSOR_MAP_SWIZZLE_128B);
        if (rc) return rc;
    }
    constexpr int kRowsB = kDual ? 2 * BN : BN;
    rc = configure_smem<gemm_tile_kernel<KIND, EPI, BN>>(tile_smem(kMaxK, kRowsB));
    if (rc) return rc;
    return launch_dependent(gemm_tile_kernel<KIND, EPI, BN>, dim3(g->N / BN, (g->M + 127) / 128), kTileThreads, tile_smem(g->K, kRowsB), stream,
                            tm_a, tm_b, tm_b2, p);
}

}  // namespace
}  // namespace fluke_sm100
