// Projection / FFN GEMM with fused epilogue for sm_100a:  y = epilogue(x . w^T + bias (+ residual)).
//
// Persistent, warp-specialised CTA (one per SM):
//   warp 0      : TMA producer   — x tile [TM x 64] and w tile [BN x 64] of KSUB k-blocks into one stage of a STAGES-deep
//                                   ring of 128-byte-swizzled shared memory; completion on the stage's `full` mbarrier.
//   warp 1      : UMMA issuer    — owns the TMEM allocation (2 accumulators of BN fp32 columns); one elected lane
//                                   issues 4 x tcgen05.mma (TM x BN x 16) per k-block, commits the stage's `empty`
//                                   barrier, and commits `acc_full` after the last k-block of a tile.
//   warps 2..   : epilogue       — tcgen05.ld of the accumulator (a thread owns one row: lane = row), bias / GELU /
//                                   residual in registers, TMA store.  Four warps (BN = 32), or eight, of which two share
//                                   a quarter of the rows and split the columns.  While they drain accumulator b, the
//                                   issuer fills b^1.
// Used where a launch has few tiles; what bounds it there is one tile's serial chain of stages.  The hand-shake of a stage
// (wait, fence, UMMAs, commit) takes ~270 clocks whatever it holds, measured with the loads left out and a single UMMA per
// k-block (5.1 of the 7 us that 36 more k-blocks take on a 128 x 64 tile).  Hence several k-blocks per stage, each operand
// fetched by one 3-D TMA box: 3072 -> 768 at 41 rows on 64 x 32 tiles 10.2 us with one k-block per stage, 7.5 / 6.7 / 6.3 with
// two / three / four.  A k-block then takes 155-165 clocks of 1965 MHz (slope from 3072 to 6144 deep), of which its loads alone,
// with the UMMAs left out, would take 101-121 (24 and 144 CTAs): it is still the chain that binds, not the way from L2.
// Algorithmic work per launch: 2*M*N*K flop; HBM traffic at least (M*K + N*K + M*N (+ M*N residual)) elements.
#include "linear_common.cuh"

namespace b200 {
namespace lin {

// TM = rows of a tile (128, or 64), BN = its columns, KSUB = 64-deep k-blocks per pipeline stage.
template <int TM, int BN, int KSUB, int STAGES, bool FOLD>
struct Cfg {
    static constexpr int EPI_WARPS = BN >= 64 ? 8 : 4;          // every epilogue warp drains at least 32 columns
    static constexpr int THREADS = 64 + 32 * EPI_WARPS;
    static constexpr int COLS = BN / (EPI_WARPS / 4);           // accumulator columns drained by one epilogue warp
    static constexpr int RPW = TM / 4;                          // rows of the tile in a warp's TMEM lanes
    static constexpr int A_BLOCK = TM * BK * 2;                 // one k-block of the tile's rows of x
    static constexpr int B_BLOCK = BN * BK * 2;
    static constexpr int A_BYTES = KSUB * A_BLOCK;
    static constexpr int B_BYTES = KSUB * B_BLOCK;
    static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr int OUT_OFFSET = STAGES * STAGE_BYTES;               // output staging strips (TMA store)
    static constexpr int BAR_OFFSET = OUT_OFFSET + EPI_WARPS * kStageBytesPerWarp;
    static constexpr int BIAS_OFFSET = BAR_OFFSET + 512;         // per-epilogue-warp bias slice: COLS floats
    static constexpr int SMEM_BYTES = BIAS_OFFSET + EPI_WARPS * vec_strips<FOLD>() * COLS * 4 + 1024;  // + slack for 1024-byte alignment
    static constexpr int TMEM_COLS = 2 * BN;                    // 64, 128, 256 or 512: powers of two
    static_assert((2 * STAGES + 4) * 8 + 8 <= 512, "barriers");
};

// FEW: the whole launch has fewer rows than TM (p.x_rows of them in a load box).
template <int TM, int BN, int KSUB, int STAGES, bool FOLD, bool FEW>
__global__ void __launch_bounds__(Cfg<TM, BN, KSUB, STAGES, FOLD>::THREADS, 1)
linear_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w,
              const __grid_constant__ CUtensorMap tm_y, const LinearParams p) {
    using C = Cfg<TM, BN, KSUB, STAGES, FOLD>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::BAR_OFFSET);
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;
    uint64_t* acc_empty = acc_full + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], C::EPI_WARPS);
        }
        *abort_flag = 0;
        mbar_fence_init();
        prefetch_tmap(&tm_x);
        prefetch_tmap(&tm_w);
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, C::TMEM_COLS);
        tmem_relinquish();
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        // The weights on their way from HBM into L2 while the previous kernel of the stream drains, as in the pair kernel:
        // a prefetch reads nothing into this kernel, so it needs no order against an earlier kernel that writes them.
        const int k_boxes = (p.num_k_blocks + KSUB - 1) / KSUB;
        for (int b = blockIdx.x; b < k_boxes * p.num_n_tiles; b += gridDim.x) {
            if (KSUB == 1) tma_prefetch_l2_2d(&tm_w, (b % k_boxes) * BK, (b / k_boxes) * BN);
            else tma_prefetch_l2_3d(&tm_w, 0, (b / k_boxes) * BN, (b % k_boxes) * KSUB);
        }
    }
    pdl_wait();   // inputs come from earlier kernels; the output may still be read by one

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        if (elect_one()) {
            uint32_t st = 0, ph = 0;
            bool ok = true;
            const uint32_t stage_tx = FEW ? static_cast<uint32_t>(KSUB * p.x_rows * BK * 2 + C::B_BYTES) : C::STAGE_BYTES;
            for (int tile = blockIdx.x; ok && tile < p.num_tiles; tile += gridDim.x) {
                const int m_blk = tile / p.num_n_tiles;
                const int n_blk = tile % p.num_n_tiles;
                for (int kb = 0; kb < p.num_k_blocks; kb += KSUB) {
                    if (!mbar_wait(&empty[st], ph ^ 1u, abort_flag)) { ok = false; break; }
                    uint8_t* a = smem + st * C::STAGE_BYTES;
                    uint8_t* b = a + C::A_BYTES;
                    mbar_expect_tx(&full[st], stage_tx);
                    if (KSUB == 1) {
                        tma_load_2d(a, &tm_x, &full[st], kb * BK, m_blk * TM);
                        tma_load_2d(b, &tm_w, &full[st], kb * BK, n_blk * BN);
                    } else {   // maps with K split into blocks of 64: (inside the block, row, block)
                        tma_load_3d(a, &tm_x, &full[st], 0, m_blk * TM, kb);
                        tma_load_3d(b, &tm_w, &full[st], 0, n_blk * BN, kb);
                    }
                    if (++st == STAGES) { st = 0; ph ^= 1u; }
                }
            }
            if (!ok) {
                // Give copies already in flight time to land before the CTA's shared memory is released.
                for (int i = 0; i < 64; ++i) nanosleep(10000);
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------ UMMA issuer
        if (elect_one()) {
            uint32_t st = 0, ph = 0, tcount = 0;
            bool ok = true;
            // (with fewer rows than TM the UMMA reads on into whatever follows a k-block in the stage: rows that are not stored)
            const uint64_t a_step = static_cast<uint64_t>(FEW ? p.x_rows * BK * 2 : C::A_BLOCK) >> 4;
            const uint64_t a_desc0 = make_smem_desc_sw128(smem_u32(smem));
            const uint64_t b_desc0 = make_smem_desc_sw128(smem_u32(smem + C::A_BYTES));
            for (int tile = blockIdx.x; ok && tile < p.num_tiles; tile += gridDim.x, ++tcount) {
                const uint32_t buf = tcount & 1u;
                const uint32_t aph = (tcount >> 1) & 1u;
                if (!mbar_wait(&acc_empty[buf], aph ^ 1u, abort_flag)) { ok = false; break; }
                tcgen05_fence_after();
                const uint32_t d_tmem = tmem_base + buf * BN;
                for (int kb = 0; kb < p.num_k_blocks; kb += KSUB) {
                    if (!mbar_wait(&full[st], ph, abort_flag)) { ok = false; break; }
                    tcgen05_fence_after();
                    const uint64_t a_desc = a_desc0 + static_cast<uint64_t>(st * (C::STAGE_BYTES >> 4));
                    const uint64_t b_desc = b_desc0 + static_cast<uint64_t>(st * (C::STAGE_BYTES >> 4));
#pragma unroll
                    for (int sub = 0; sub < KSUB; ++sub) {
#pragma unroll
                        for (int k = 0; k < BK / 16; ++k) {
                            // 16 elements along K = 32 bytes inside the 128-byte swizzled row: +2 in (address >> 4) units
                            umma_f16_ss(d_tmem, a_desc + static_cast<uint64_t>(sub) * a_step + static_cast<uint64_t>(2 * k),
                                        b_desc + static_cast<uint64_t>(sub * (C::B_BLOCK >> 4) + 2 * k), p.idesc,
                                        (kb | sub | k) != 0 ? 1u : 0u);
                        }
                    }
                    umma_commit(&empty[st]);
                    if (++st == STAGES) { st = 0; ph ^= 1u; }
                }
                if (ok) umma_commit(&acc_full[buf]);
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------ epilogue
        const int ew = warp - 2;
        const int quarter = warp & 3;  // TMEM lanes 32*quarter .. 32*quarter+31 are the ones this warp may read
        const int half = ew >> 2;      // which COLS-wide part of the BN columns
        constexpr int COLS = C::COLS;
        constexpr int CHUNKS = COLS / 32;
        float* vec_w = reinterpret_cast<float*>(smem + C::BIAS_OFFSET) + ew * vec_strips<FOLD>() * COLS;  // private to this warp
        WarpEpilogue<CHUNKS, false, FOLD, C::RPW> epi{p, &tm_y, nullptr, smem + C::OUT_OFFSET + ew * kStageBytesPerWarp, nullptr,
                                        abort_flag, lane, 0u};
        uint32_t tcount = 0;
        bool ok = true;
        for (int tile = blockIdx.x; ok && tile < p.num_tiles; tile += gridDim.x, ++tcount) {
            const int m_blk = tile / p.num_n_tiles;
            const int n_blk = tile % p.num_n_tiles;
            const uint32_t buf = tcount & 1u;
            const uint32_t aph = (tcount >> 1) & 1u;
            // Stage this tile's bias slice while the accumulator is still being produced.
            const long long row = static_cast<long long>(m_blk) * TM + quarter * C::RPW + lane;
            epi.begin_tile(n_blk * BN + half * COLS, static_cast<int>(row) - lane);
            stage_vectors<FOLD>(p, vec_w, n_blk * BN + half * COLS, COLS, lane);
            if (!mbar_wait(&acc_full[buf], aph, abort_flag)) { ok = false; break; }
            __syncwarp();  // tcgen05.ld is warp-collective
            tcgen05_fence_after();
            const uint32_t tacc = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + buf * BN;
            epi.template run<COLS>(vec_w, tacc, row, n_blk * BN, half * COLS);
            // This warp has read everything it needs from accumulator `buf`.
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[buf]);
        }
        // this warp's tile stores have read their strips; the writes themselves are complete when the grid is
        if (lane == 0) tma_store_wait_read<0>();
        __syncwarp();
    }

    // ---------------------------------------------------------------- teardown (also the exit of an aborted CTA)
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 1) {
        tcgen05_fence_after();
        tmem_dealloc(tmem_base, C::TMEM_COLS);
    }
    if (threadIdx.x == 0 && *abort_flag != 0 && p.status != nullptr) atomicOr(p.status, 1u);
}

int device_sm_count() {
    static std::atomic<int> sms[kMaxDevices];   // 0 = not looked up yet; every thread would store the same value
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= kMaxDevices) return 148;
    int v = sms[dev].load(std::memory_order_relaxed);
    if (v == 0) {
        int n = 0, major = 0;
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
        v = (major == 10) ? n : -1;
        sms[dev].store(v, std::memory_order_relaxed);
    }
    return v;
}

template <int TM, int BN, int KSUB, int STAGES, bool FOLD, bool FEW = false>
int launch_linear_t(const B200LinearDesc& d, cudaStream_t stream, int sm_count) {
    using C = Cfg<TM, BN, KSUB, STAGES, FOLD>;
    const int x_rows = FEW ? static_cast<int>((d.M + 7) / 8 * 8) : TM;
    if (x_rows > TM || (FEW && KSUB == 1)) return B200_ERR_PARAM;
    CUtensorMap tx, tw, ty;
    if (KSUB == 1) {
        const uint64_t xd[2] = {static_cast<uint64_t>(d.K), static_cast<uint64_t>(d.M)};
        const uint64_t xs[1] = {static_cast<uint64_t>(d.ldx) * 2};
        const uint32_t xb[2] = {BK, TM};
        const uint64_t wd[2] = {static_cast<uint64_t>(d.K), static_cast<uint64_t>(d.N)};
        const uint64_t ws[1] = {static_cast<uint64_t>(d.ldw) * 2};
        const uint32_t wb[2] = {BK, BN};
        if (!get_tensor_map(&tx, d.x, 2, xd, xs, xb) || !get_tensor_map(&tw, d.w_nk, 2, wd, ws, wb)) return B200_ERR_DRIVER;
    } else {
        // K as (K / 64) blocks of 64 (the caller has checked that K is a multiple of 64): a box covers KSUB k-blocks, which
        // land one behind the other, each in the layout the UMMA descriptors expect.  Blocks beyond K read as zeros.
        const uint64_t xd[3] = {BK, static_cast<uint64_t>(d.M), static_cast<uint64_t>(d.K / BK)};
        const uint64_t xs[2] = {static_cast<uint64_t>(d.ldx) * 2, BK * 2};
        const uint32_t xb[3] = {BK, static_cast<uint32_t>(x_rows), KSUB};
        const uint64_t wd[3] = {BK, static_cast<uint64_t>(d.N), static_cast<uint64_t>(d.K / BK)};
        const uint64_t ws[2] = {static_cast<uint64_t>(d.ldw) * 2, BK * 2};
        const uint32_t wb[3] = {BK, BN, KSUB};
        if (!get_tensor_map(&tx, d.x, 3, xd, xs, xb) || !get_tensor_map(&tw, d.w_nk, 3, wd, ws, wb)) return B200_ERR_DRIVER;
    }
    ty = tx;   // placeholder when the output is fp32 (stored directly, map unused)
    if (d.out_dtype != B200_F32) {
        const uint64_t yd[2] = {static_cast<uint64_t>(d.N), static_cast<uint64_t>(d.M)};
        const uint64_t ys[1] = {static_cast<uint64_t>(d.ldy) * 2};
        const uint32_t yb[2] = {32, C::RPW};
        if (!get_tensor_map(&ty, d.y, 2, yd, ys, yb, 64)) return B200_ERR_DRIVER;
    }

    LinearParams p;
    p.bias = d.bias;
    p.residual = d.residual;
    p.y = d.y;
    p.M = static_cast<int>(d.M);
    p.N = static_cast<int>(d.N);
    p.K = static_cast<int>(d.K);
    p.ldr = d.ldr;
    p.ldy = d.ldy;
    p.dtype = d.dtype;
    p.out_dtype = d.out_dtype;
    p.epilogue = d.epilogue;
    p.num_n_tiles = (p.N + BN - 1) / BN;
    p.num_tiles = ((p.M + TM - 1) / TM) * p.num_n_tiles;
    p.num_k_blocks = (p.K + BK - 1) / BK;
    p.idesc = make_idesc_f16(TM, BN, d.dtype == B200_BF16 ? 1 : 0, 0, 0);
    p.status = device_status_ptr();
    p.out_stats = d.out_stats;
    p.ln_in_stats = d.ln_in_stats;
    p.ln_c1 = d.ln_c1;
    p.ln_c2 = d.ln_c2;
    p.res_ln_stats = d.res_ln_stats;
    p.res_ln_gamma = d.res_ln_gamma;
    p.res_ln_beta = d.res_ln_beta;
    p.ln_eps = d.ln_eps;
    p.k_slots = (p.K + 31) / 32;
    p.n_slots = (p.N + 31) / 32;
    p.x_rows = x_rows;

    static PerDeviceOnce attr_once;
    int dev = 0;
    cudaGetDevice(&dev);
    if (!attr_once.ensure(dev, []() {
            return cudaFuncSetAttribute(linear_kernel<TM, BN, KSUB, STAGES, FOLD, FEW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        C::SMEM_BYTES) == cudaSuccess;
        }))
        return B200_ERR_LAUNCH;
    const int grid = p.num_tiles < sm_count ? p.num_tiles : sm_count;
    launch_kernel(linear_kernel<TM, BN, KSUB, STAGES, FOLD, FEW>, dim3(grid), dim3(C::THREADS), C::SMEM_BYTES, stream, tx, tw, ty, p);
    count_launch();
    return check_launch();
}

// KSUB / KSTAGES: the multi-block pipeline, for a K of whole 64-deep blocks (its maps split K into such blocks).
template <int BN, int STAGES, int KSUB, int KSTAGES>
int launch_linear(const B200LinearDesc& d, cudaStream_t stream, int sm_count, bool multi_block) {
    if (wants_fold(d)) return launch_linear_t<128, BN, 1, STAGES - 1, true>(d, stream, sm_count);
    if (KSUB > 1 && multi_block) return launch_linear_t<128, BN, KSUB, KSTAGES, false>(d, stream, sm_count);
    return launch_linear_t<128, BN, 1, STAGES, false>(d, stream, sm_count);
}

// Tile choice.  With few tiles a launch is one tile's serial chain (one-wave rules below); beyond, estimated time ~ waves *
// (columns per tile * cost per column + fixed per-tile cost) + tail, in units of accumulator columns per SM.
struct TileChoice {
    bool pair;
    int bn;
    int tm = 128;               // rows of a single-CTA tile
    bool multi_block = false;   // several k-blocks per pipeline stage where the tile has such a form (K of whole blocks)
};
TileChoice choose_tile(const B200LinearDesc& d, int sm_count) {
    const int64_t M = d.M, N = d.N;
    const int64_t k_blocks = (d.K + BK - 1) / BK;
    const bool whole = !wants_fold(d) && d.K % BK == 0;
    // Stages of several k-blocks pay from about eight blocks on (us per launch at 512, 320, 128 deep, one block -> several:
    // 128 x 64 tiles, 768 columns + residual, 512 rows 4.43 -> 4.32 at 512, 3.38 -> 3.41 at 128; 2304 columns, 256 rows 3.63 ->
    // 3.66 at 320; 128 x 128, 2304 columns, 1024 rows 4.22 -> 4.57 at 320): a shorter chain is over before the ring is full.
    const bool deep = whole && k_blocks >= 8;
    auto tiles = [&](int64_t tm, int64_t tn) { return ((M + tm - 1) / tm) * ((N + tn - 1) / tn); };
    // Few rows: a launch is bound by its latencies (hand-over, first loads, the serial chain of k-blocks of one tile, drain),
    // so the smallest tile that still fits one wave is the fastest: the more SMs fetch operands at once, the shorter each
    // one's chain.  12 launches in turn on weights of their own, us per launch, 128 x 64 tiles with one k-block per
    // stage -> the tile below:  M = 41: 768 -> 768 5.4 -> 3.5, 768 -> 2304 4.7 -> 3.4, 768 -> 3072 5.1 -> 3.8,
    // 3072 -> 768 13.3 -> 7.7;  M = 256: 5.9 -> 3.7, 5.0 -> 4.2, 5.5 -> 5.1, 12.5 -> 7.1;  M = 1024: 768 -> 768 5.9 -> 5.1,
    // 3072 -> 768 13.1 -> 10.7 (128 x 64).  One tile more than SMs and the next wider one is ahead: 768 -> 3072 at 128 rows
    // 4.9 on 192 tiles of 64 x 32, 4.5 on 96 of 64 x 64.  All tiles add a row's products up in the same order, so the choice
    // changes no bit of the result.
    if (whole && k_blocks >= 2 && tiles(64, 32) <= sm_count) return {false, 32, 64};   // (64 deep: 2.6 us on 128 x 64, 3.2 on these)
    if (deep && tiles(64, 64) <= sm_count) return {false, 64, 64};
    if (whole && tiles(128, 64) <= sm_count) return {false, 64, 128, deep};
    // 128 x 128 drains two chunks per warp, and a residual of the second is not fetched ahead: 768 -> 2304 at 1024 rows
    // 5.8 against 6.5 us on pair tiles, 768 -> 768 with a residual at 2048 rows 7.8 against 6.7.  A k-block takes it longer
    // than a pair tile: 1024 deep still ahead (768 rows, 3072 columns: 6.7 against 7.2), 3072 deep behind (6144 rows, 256
    // columns: 13.5 against 12.8).
    if (whole && k_blocks <= 16 && d.epilogue != B200_EPI_BIAS_RESIDUAL && tiles(128, 128) <= sm_count)
        return {false, 128, 128, deep};

    // More than one wave.  Costs per column relative to 256-wide pair tiles, for pair tiles 256, 192, 128, 64 and single-CTA
    // tiles 256, 128, 64 wide; the narrower ones fetch more rows of x per flop and hand more stages over.  For a deep K they
    // are fitted to the measured choice between tiles at 129 .. 65536 rows, 768- and 1024-wide models; GELU hides better
    // behind 192-wide tiles' twelve epilogue warps.  The tail is the last tile's epilogue, which nothing hides: 128 columns per
    // warp on 256-wide tiles, 64 on 192- and 128-wide ones; it weighs less the longer the mainloop.  us per launch, 256 wide ->
    // chosen: 768 -> 3072 + GELU at 4096 rows 18.6 -> 17.7, 5120 23.6 -> 20.9, 8192 32.9 -> 30.5, 16384 63.4 -> 61.4;  768 -> 2304
    // at 2048 rows 8.9 -> 8.5 (128 wide);  768 -> 768 + residual at 16384 rows 21.4 -> 19.4, 32768 39.9 -> 38.5;  1024 -> 3072 at
    // 5120 rows 25.7 -> 24.3.  Where the 256-wide tile stays ahead, 192 wide: 1024 -> 3072 at 16384 rows 74.7 | 76.5, at 10240
    // 46.5 | 48.0;  768 -> 768 + residual at 65536 rows 75.6 | 76.4.
    // Otherwise (a short K, a K that is not in whole blocks, LayerNorm folding: one k-block per stage) narrow tiles cost more and
    // a tail says nothing: 776 -> 3072 + GELU at 4096 rows 24.2 us on 256-, 25.7 on 192-wide tiles, 776 -> 768 + residual
    // at 5120 rows 13.2 | 14.8 on 128-wide ones.
    const double pair_cost[2][4] = {{1.0, 1.17, 1.50, 2.50}, {1.0, d.epilogue == B200_EPI_BIAS_GELU ? 1.05 : 1.10, 1.28, 2.10}};
    const double single_cost[3] = {1.35, 1.50, 1.90};
    auto tail = [&](int bn) {
        if (!deep || M <= 128) return 0.0;   // (up to 128 rows only single-CTA tiles compete, and the weights' bytes decide)
        return (bn == 256 ? 200.0 : (bn == 64 ? 50.0 : 100.0)) * 12.0 / static_cast<double>(k_blocks);
    };
    TileChoice best = {false, 128, 128, deep};
    double best_t = 1e300;
    auto consider = [&](bool pair, int bn, int64_t n_tiles, int64_t slots, double cost) {
        const double t = static_cast<double>((n_tiles + slots - 1) / slots) * (bn * cost + 16.0) + tail(bn);
        if (t < best_t) {
            best_t = t;
            best = {pair, bn, 128, deep};
        }
    };
    const int pair_bn[4] = {256, 192, 128, 64}, single_bn[3] = {256, 128, 64};
    for (int i = 0; i < 4 && M > 128; ++i) {
        const int pairs = max_active_pairs(pair_bn[i]);
        if (pairs > 0) consider(true, pair_bn[i], tiles(256, pair_bn[i]), pairs, pair_cost[deep ? 1 : 0][i]);
    }
    for (int i = 0; i < 3; ++i) consider(false, single_bn[i], tiles(128, single_bn[i]), sm_count, single_cost[i]);
    return best;
}

int validate_linear_desc(const B200LinearDesc* d) {
    if (!d || !d->x || !d->w_nk || !d->y) return B200_ERR_PARAM;
    if (d->M <= 0 || d->N <= 0 || d->K <= 0) return B200_ERR_PARAM;
    if (d->M > (1ll << 30) || d->N > (1ll << 30) || d->K > (1ll << 30)) return B200_ERR_UNSUPPORTED;
    if (!is_half_dtype(d->dtype)) return B200_ERR_PARAM;
    if (d->out_dtype != B200_F16 && d->out_dtype != B200_BF16 && d->out_dtype != B200_F32) return B200_ERR_PARAM;
    if (d->epilogue < B200_EPI_BIAS || d->epilogue > B200_EPI_BIAS_TANH) return B200_ERR_PARAM;
    if (d->epilogue == B200_EPI_BIAS_RESIDUAL && !d->residual) return B200_ERR_PARAM;
    if ((d->K % 8) || (d->N % 8) || (d->ldx % 8) || (d->ldw % 8) || (d->ldy % 8)) return B200_ERR_PARAM;
    if (d->ldx < d->K || d->ldw < d->K || d->ldy < d->N) return B200_ERR_PARAM;
    if (!aligned16(d->x) || !aligned16(d->w_nk) || !aligned16(d->y)) return B200_ERR_PARAM;
    if (d->bias && !aligned16(d->bias)) return B200_ERR_PARAM;
    if (d->epilogue == B200_EPI_BIAS_RESIDUAL && ((d->ldr % 8) || d->ldr < d->N || !aligned16(d->residual)))
        return B200_ERR_PARAM;
    if (d->ln_in_stats && (!d->ln_c1 || !d->ln_c2)) return B200_ERR_PARAM;
    if (d->res_ln_stats && (!d->res_ln_gamma || !d->res_ln_beta || d->epilogue != B200_EPI_BIAS_RESIDUAL))
        return B200_ERR_PARAM;
    return B200_OK;
}

}  // namespace lin
}  // namespace b200

extern "C" int b200_linear_fwd(const B200LinearDesc* d, b200_stream_t stream_) {
    using namespace b200;
    using namespace b200::lin;
    const int valid = validate_linear_desc(d);
    if (valid != B200_OK) return valid;
    const int sms = device_sm_count();
    if (sms <= 0) return B200_ERR_NOT_SM100;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    const bool whole = d->K % BK == 0;
    TileChoice tc;
    if (d->block_n == 0) {
        tc = choose_tile(*d, sms);
    } else if (d->block_n > 0) {
        tc = {d->M > 128, d->block_n, 128, whole};
    } else {
        tc = {false, -d->block_n, 128, whole};
    }
    if (tc.pair) {
        switch (tc.bn) {
            case 256: return launch_linear_pair<256>(*d, stream, sms, tc.multi_block);
            case 192: return launch_linear_pair<192>(*d, stream, sms, tc.multi_block);
            case 128: return launch_linear_pair<128>(*d, stream, sms, tc.multi_block);
            case 64: return launch_linear_pair<64>(*d, stream, sms, tc.multi_block);
            default: return B200_ERR_PARAM;
        }
    }
    if (tc.tm == 64) {
        if (tc.bn == 64) return launch_linear_t<64, 64, 4, 3, false>(*d, stream, sms);
        // Up to 48 rows fetch only the rows that exist, rounded up to the swizzle's eight: rows beyond M are written to shared
        // memory as zeros at the cost of loaded ones.  us per launch at 16 rows: 768 -> 2304 3.8 -> 3.2, 768 -> 3072 4.6 -> 3.5;
        // at 41 rows 768 -> 3072 3.95 -> 3.75; at 56 rows and more there is nothing left to gain.
        return d->M <= 48 ? launch_linear_t<64, 32, 4, 4, false, true>(*d, stream, sms)
                          : launch_linear_t<64, 32, 4, 4, false>(*d, stream, sms);
    }
    switch (tc.bn) {
        case 256: return launch_linear<256, 4, 1, 4>(*d, stream, sms, tc.multi_block);
        case 128: return launch_linear<128, 6, 2, 3>(*d, stream, sms, tc.multi_block);
        case 64: return launch_linear<64, 8, 2, 4>(*d, stream, sms, tc.multi_block);
        default: return B200_ERR_PARAM;
    }
}
