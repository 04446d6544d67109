// float32 GEMM on the tensor cores: out[M,N] = act(X[M,K] . W[N,K]^T + bias) (+ residual), float32 operands and result.
//
// A float32 number is the sum of three bfloat16 numbers (rounded to nearest one after the other: 3 x 8 significant
// bits and their signs hold all 24), and a product of two of them is nine products of bfloat16 numbers. The six that
// are not below 2^-24 of the product go to tcgen05.mma; the three left out are below half a unit in the last place
// of the float32 product, with either sign. The tensor core adds into a float32 accumulator, but cuts off instead of
// rounding, so an accumulator may take few additions: every k block of 32 has an accumulator of its own, into which
// the small products go first (while it is small, so is what is cut off) and the two steps of leading products last;
// the sums of the k blocks are then added in float32 registers, rounded to nearest. Measured against 64-bit results
// with normal operands, the error is 0.1 (K = 6,400) to 0.6 (K = 36) of that of one chain of float32 fused
// multiply-adds per output (gemm_simt.cu).
//
// TMA brings float32 tiles of 128 features x 32 k (128-byte swizzle) into a staging ring; four warps (or eight, taking
// turns) split them, a thread a feature, and put the three planes into tensor memory, where tcgen05.mma takes its first
// operand from: shared memory, whose bandwidth bounds these MMAs, then serves only the tokens' planes. Up to 32 tokens
// those are split in the kernel as well (64-byte rows, 64-byte swizzle); above, a kernel before this one writes them once
// for all tiles (split_rows_kernel) and TMA brings them. The features are the 128 lanes of the accumulator and the tokens
// its columns, so a decode step of a few tokens wastes no tensor-core rows and the stores of a warp are 128 consecutive
// bytes of a row. The epilogue warps take every k block's accumulator out of TMEM while the next ones are at work. A
// cluster of blocks may share a tile's K; the partial tiles are then added over distributed shared memory in rank order.
//
// A sum that is not finite is computed again, product by product, with float32 fused multiply-adds: an infinity has
// no three parts (and neither has a number that rounds to infinity in bfloat16), so such sums come out as NaN here.
#include "common.cuh"
#include "tcgen05.cuh"

namespace {

constexpr int BM = 128;          // output features per tile (accumulator lanes)
constexpr int BK = 32;           // k elements per stage: one 128-byte swizzle row of float32, a 64-byte row of bfloat16
constexpr int PLANE_ROW = BK * 2;                       // bytes of a row of an operand plane
constexpr int W_COLS = 3 * BK / 2;                      // TMEM columns of a feature tile's three planes

template <int BN> struct SplitConfig {
    static constexpr bool X_SPLIT = BN >= 64;                            // the tokens' planes come from global memory
    static constexpr int EPI_WARPS = BN >= 128 ? 8 : 4;                  // two per lane quarter for the widest tile
    static constexpr int EPI_COLS = BN * 4 / EPI_WARPS;                  // columns an epilogue thread owns
    static constexpr int CONV_GROUPS = 2;                                // of four warps, k blocks taken in turn
    static constexpr int X_WARPS = X_SPLIT ? 1 : 4;                      // one thread that fetches planes, or warps that split, k blocks taken in turn
    // The widest tile has five whole warpgroups (the fetching warps and one that idles, two of epilogue, two that split), which
    // share the registers by their needs: 128 x 40 + 256 x 144 + 256 x 72 of the launch's 640 x 96. With 128 for everybody and
    // the sums live through the other warps' code, the epilogue's loads went one by one: with a residual 1,000 rows of 1,280 x
    // 5,120 took 127 us, now 107, and 5,120 x 1,280 142, now 107; plain products 103 / 101 and 92 / 93. What bounds those is what an
    // SM fetches, 40 KB a k block of 0.79 us (51 KB/us, 7.5 TB/s in all): half the MMAs take 2 % off.
    static constexpr bool GROUPED = BN >= 128;
    static constexpr int FIRST_EPI = GROUPED ? 4 : 2, FIRST_CONV = FIRST_EPI + EPI_WARPS, LAST_CONV = FIRST_CONV + 4 * CONV_GROUPS;
    static constexpr int FIRST_X = GROUPED ? 2 : LAST_CONV;
    static constexpr int THREADS = 32 * (GROUPED ? LAST_CONV : FIRST_X + X_WARPS);        // 18 warps: 96 registers a thread
    static constexpr int STAGING_BYTES = (BM + (X_SPLIT ? 0 : BN)) * BK * 4;
    static constexpr int OPERAND_BYTES = BN * PLANE_ROW * 3;
    static constexpr int STAGINGS = BN >= 64 ? 6 : 8;
    static constexpr int OPERANDS = 4;
    static constexpr int ACCS = BN >= 128 ? 2 : 4;
    static constexpr int TMEM_COLS = ACCS * BN + OPERANDS * W_COLS <= 256 ? 256 : 512;
    static constexpr int RING_BYTES = STAGINGS * STAGING_BYTES + OPERANDS * OPERAND_BYTES;
    static constexpr int SMEM_BYTES = RING_BYTES + 1024 /*alignment slack*/ + 256 /*barriers*/;
    // a slot of a ring always falls to the same warp, which therefore never waits for a phase but the slot's next one
    static_assert(OPERANDS % CONV_GROUPS == 0 && STAGINGS % CONV_GROUPS == 0 && (X_SPLIT || (OPERANDS % X_WARPS == 0 && STAGINGS % X_WARPS == 0)), "turns");
    static_assert(OPERANDS % ACCS == 0, "an accumulator's number follows from its operands' slot");
    static_assert(ACCS * BN + OPERANDS * W_COLS <= 512, "tensor memory");
    static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");
    // the partial tiles of a cluster lie over the rings, which nobody uses any more by then
    static_assert((BM + 8) * BN * 4 <= RING_BYTES, "the reduce buffer fits");
};

struct SplitParams {
    const float* X;
    const float* W;
    const uint8_t* planes;       // tiles of 64 and 128 tokens: their bfloat16 planes (split_rows_kernel)
    const float* bias;           // [N] or null
    const float* residual;       // [M, ldr] or null; may be out itself
    float* out;                  // [M, ldo]
    int* error_flag;
    int M, N, K, ldx, ldw, ldr, ldo, act, kblocks_per_split;
};

// K-major operand whose rows are 32 bfloat16 (64 bytes) under the 64-byte swizzle: 8-row groups 512 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_sw64(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(512 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;
    return d;
}

// Two neighbouring values to two bfloat16 in one register (the first in the lower half), and what is left of them.
__device__ __forceinline__ uint32_t take_bf16x2(float& a, float& b) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    a -= __uint_as_float(r << 16);
    b -= __uint_as_float(r & 0xffff0000u);
    return r;
}

__device__ __forceinline__ void bulk_load(void* smem_dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(tc::smem_u32(smem_dst)), "l"(src), "r"(bytes), "r"(tc::smem_u32(bar)) : "memory");
}

// A warp's wait: every lane asks (one asking for all and telling them measured 10 to 20 % slower), one decision.
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, volatile int* abort) {
    return __all_sync(0xffffffffu, tc::mbar_wait(bar, parity, abort));
}

// Which 16-byte piece of its row (of BN floats) feature lf's piece c lies at in the reduce buffer: c ^ this.
template <int BN> __device__ __forceinline__ int split_swizzle(int lf) { return BN >= 32 ? (lf & 7) : ((lf >> 1) & 3); }

__device__ __noinline__ float plain_dot(const float* x, const float* w, int K) {
    float s = 0.f;
    for (int k = 0; k < K; ++k) s = fmaf(x[k], w[k], s);
    return s;
}

// The result of COUNT tokens m0.. of feature n (inside the matrix) from their sums v. A function that is called, not
// copied into every place, and with one loop an activation: 64 copies of every activation behind one another ran from
// instruction memory at 16 us a tile (K = 64: 21.6 us for 64 rows, against 5.6 for one).
template <int COUNT>
__device__ __noinline__ void finish(const SplitParams& p, int m0, int n, const float* v, float bias) {
    float u[COUNT], res[COUNT];                           // the residual is read before anything is written: it may be out itself
#pragma unroll
    for (int j = 0; j < COUNT; ++j) {
        u[j] = v[j];
        res[j] = (p.residual && m0 + j < p.M) ? p.residual[(size_t)(m0 + j) * p.ldr + n] : 0.f;
    }
    bool fine = true;
#pragma unroll
    for (int j = 0; j < COUNT; ++j) fine &= isfinite(u[j]);
    if (!fine)
#pragma unroll
        for (int j = 0; j < COUNT; ++j)
            if (!isfinite(u[j]) && m0 + j < p.M) u[j] = plain_dot(p.X + (size_t)(m0 + j) * p.ldx, p.W + (size_t)n * p.ldw, p.K);
    if (p.act == DD_ACT_NONE) {
#pragma unroll
        for (int j = 0; j < COUNT; ++j) u[j] = u[j] + bias;
    } else if (p.act == DD_ACT_GELU_NEW) {
#pragma unroll
        for (int j = 0; j < COUNT; ++j) u[j] = dd_activation(u[j] + bias, DD_ACT_GELU_NEW);
    } else {
#pragma unroll
        for (int j = 0; j < COUNT; ++j) u[j] = dd_activation(u[j] + bias, p.act);
    }
#pragma unroll
    for (int j = 0; j < COUNT; ++j)
        if (m0 + j < p.M) p.out[(size_t)(m0 + j) * p.ldo + n] = u[j] + res[j];
}

template <int BN>
__global__ void __launch_bounds__(SplitConfig<BN>::THREADS, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                  const __grid_constant__ SplitParams p) {
    using C = SplitConfig<BN>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* staging = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* operands = staging + C::STAGINGS * C::STAGING_BYTES;
    uint64_t* staged = reinterpret_cast<uint64_t*>(staging + C::RING_BYTES);     // float32 tiles have landed
    uint64_t* staging_free = staged + C::STAGINGS;
    // The MMA thread's path (waits, issues, commits) is serial, and with a few tokens it is what bounds a k block: it waits
    // for one barrier for both operands, and one commit says that the operands are free and the accumulator is full.
    uint64_t* split_done = staging_free + C::STAGINGS;                           // features' planes in TMEM, tokens' in shared memory
    uint64_t* mma_done = split_done + C::OPERANDS;
    uint64_t* acc_free = mma_done + C::OPERANDS;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_free + C::ACCS);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    dd_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = (int)tc::cluster_size(), rank = (int)tc::cluster_rank();
    const int tiles_n = (p.N + BM - 1) / BM;
    const int n_tiles = tiles_n * ((p.M + BN - 1) / BN);
    const int total_kblocks = (p.K + BK - 1) / BK;
    const int kb_begin = rank * p.kblocks_per_split;
    const int n_kblocks = max(0, min(total_kblocks, kb_begin + p.kblocks_per_split) - kb_begin);
    // a cluster works on one tile; without clusters a block walks over tiles and its rings run on across them
    const int first_tile = blockIdx.x / S, tile_step = gridDim.x / S;
    const int n_its = (first_tile < n_tiles ? (n_tiles - 1 - first_tile) / tile_step + 1 : 0) * n_kblocks;      // k blocks this block takes

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::STAGINGS; ++s) {
            tc::mbar_init(&staged[s], 1);
            tc::mbar_init(&staging_free[s], C::X_SPLIT ? 4 : 5);
        }
        for (int s = 0; s < C::OPERANDS; ++s) {
            tc::mbar_init(&split_done[s], 5);             // four warps of features and one of tokens (or its fetching thread)
            tc::mbar_init(&mma_done[s], 1);
        }
        for (int a = 0; a < C::ACCS; ++a) tc::mbar_init(&acc_free[a], C::EPI_WARPS);
        *abort_flag = 0;
        tc::fence_barrier_init();
        tc::fence_proxy_async();
    }
    if (warp == 1) {
        tc::tmem_alloc(tmem_slot, C::TMEM_COLS);
        tc::tmem_relinquish();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_w = tmem_base + C::ACCS * BN;     // the features' planes, behind the accumulators

    // the two barriers at which the blocks of a cluster exchange their sums, for the warps that have none
    auto stand_by = [&] {
        if (S == 1) return;
        __syncwarp();
        tc::fence_before_sync();
        tc::cluster_arrive();
        tc::cluster_wait();
        tc::cluster_arrive();
        tc::cluster_wait();
    };
    // one thread: the tokens' planes that a kernel before this one wrote (X_SPLIT). A k block's three planes of BN tokens lie in
    // memory as they lie in shared memory, one piece
    auto fetch_planes = [&] {
        dd_grid_wait();
        int it = 0;
        bool ok = true;
        for (int tile = first_tile; tile < n_tiles && ok; tile += tile_step) {
            const uint8_t* from = p.planes + ((size_t)(tile / tiles_n) * total_kblocks + kb_begin) * C::OPERAND_BYTES;
            for (int i = 0; i < n_kblocks; ++i, ++it, from += C::OPERAND_BYTES) {
                const int s = it % C::OPERANDS;
                if (!tc::mbar_wait(&mma_done[s], ((it / C::OPERANDS) & 1) ^ 1, abort_flag)) { ok = false; break; }
                tc::mbar_expect_tx(&split_done[s], C::OPERAND_BYTES);
                bulk_load(operands + s * C::OPERAND_BYTES, from, C::OPERAND_BYTES, &split_done[s]);
            }
        }
    };
    if (warp < C::FIRST_EPI) {
        if constexpr (C::GROUPED) asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (warp == 0) {
            if (tc::elect_one()) {
                tc::prefetch_tensormap(&map_w);
                if (!C::X_SPLIT) tc::prefetch_tensormap(&map_x);
                // weights do not depend on the kernel before this one
                const int ahead = first_tile < n_tiles ? min(n_kblocks, C::STAGINGS) : 0;
                for (int i = 0; i < ahead; ++i) {
                    tc::mbar_expect_tx(&staged[i], C::STAGING_BYTES);
                    tc::tma_load_2d(staging + i * C::STAGING_BYTES, &map_w, (kb_begin + i) * BK, (first_tile % tiles_n) * BM, &staged[i]);
                }
                if (!C::X_SPLIT) dd_grid_wait();
                int it = 0;
                bool ok = true;
                for (int tile = first_tile; tile < n_tiles && ok; tile += tile_step) {
                    const int n0 = (tile % tiles_n) * BM, m0 = (tile / tiles_n) * BN;
                    for (int i = 0; i < n_kblocks; ++i, ++it) {
                        const int s = it % C::STAGINGS;
                        uint8_t* to = staging + s * C::STAGING_BYTES;
                        if (it >= ahead) {
                            if (!tc::mbar_wait(&staging_free[s], ((it / C::STAGINGS) & 1) ^ 1, abort_flag)) { ok = false; break; }
                            tc::mbar_expect_tx(&staged[s], C::STAGING_BYTES);
                            tc::tma_load_2d(to, &map_w, (kb_begin + i) * BK, n0, &staged[s]);
                        }
                        if (!C::X_SPLIT) tc::tma_load_2d(to + BM * BK * 4, &map_x, (kb_begin + i) * BK, m0, &staged[s]);
                    }
                }
            }
        } else if (warp == 1) {
            if (tc::elect_one()) {
                constexpr uint32_t idesc = tc::idesc_bf16_f32(BM, BN);
                // plane of W, plane of X: the products in ascending order of size
                constexpr int pw[6] = {2, 0, 1, 1, 0, 0}, px[6] = {0, 2, 1, 0, 1, 0};
                for (int it = 0; it < n_its; ++it) {
                    const int acc = it % C::ACCS, s = it % C::OPERANDS;
                    if (!tc::mbar_wait(&acc_free[acc], ((it / C::ACCS) & 1) ^ 1, abort_flag) ||
                        !tc::mbar_wait(&split_done[s], (it / C::OPERANDS) & 1, abort_flag)) break;
                    tc::fence_after_sync();
                    const uint32_t w_cols = tmem_w + s * W_COLS;
                    const uint32_t x_addr = tc::smem_u32(operands + s * C::OPERAND_BYTES);
#pragma unroll
                    for (int j = 0; j < 6; ++j)
#pragma unroll
                        for (int k = 0; k < BK / 16; ++k)
                            tc::mma_bf16_a_tmem(tmem_base + acc * BN, w_cols + pw[j] * (BK / 2) + k * 8,
                                                smem_desc_sw64(x_addr + px[j] * BN * PLANE_ROW + k * 32), idesc, (j > 0 || k > 0) ? 1u : 0u);
                    tc::mma_commit(&mma_done[s]);
                }
            }
        } else if (C::GROUPED && warp == C::FIRST_X) {
            if (tc::elect_one()) fetch_planes();
        }
        stand_by();
    } else if (warp < C::FIRST_CONV) {
        if constexpr (C::GROUPED) asm volatile("setmaxnreg.inc.sync.aligned.u32 144;");
        float sum[C::EPI_COLS];                           // this feature's sums
        dd_grid_wait();                                   // the residual is an earlier kernel's data
        const int quarter = warp & 3;
        const int c_begin = warp >= C::FIRST_EPI + 4 ? C::EPI_COLS : 0;
        const uint32_t lane_addr = tmem_base + c_begin + ((uint32_t)(quarter * 32) << 16);
        int it = 0;
        bool ok = true;
        for (int tile = first_tile; tile < n_tiles; tile += tile_step) {
#pragma unroll
            for (int j = 0; j < C::EPI_COLS; ++j) sum[j] = 0.f;
            for (int i = 0; i < n_kblocks; ++i, ++it) {
                const int acc = it % C::ACCS;
                ok = warp_wait(&mma_done[it % C::OPERANDS], (it / C::OPERANDS) & 1, abort_flag);
                if (!ok) break;
                tc::fence_after_sync();
                constexpr int CHUNK = C::EPI_COLS >= 32 ? 32 : 16;
#pragma unroll
                for (int c0 = 0; c0 < C::EPI_COLS; c0 += CHUNK) {
                    uint32_t r[CHUNK];
                    if (CHUNK == 32) tc::tmem_ld_x32(lane_addr + acc * BN + c0, r);
                    else tc::tmem_ld_x16(lane_addr + acc * BN + c0, r);
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < CHUNK; ++j) sum[c0 + j] += __uint_as_float(r[j]);
                }
                tc::fence_before_sync();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&acc_free[acc]);
            }
            if (!ok || S > 1) break;
            const int n = (tile % tiles_n) * BM + quarter * 32 + lane, m0 = (tile / tiles_n) * BN + c_begin;
            const float bias = (p.bias && n < p.N) ? __ldg(p.bias + n) : 0.f;
#pragma unroll
            for (int c0 = 0; c0 < C::EPI_COLS; c0 += 16) {
                if (n >= p.N || m0 + c0 >= p.M) break;
                float v[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = sum[c0 + j];
                finish<16>(p, m0 + c0, n, v, bias);
            }
            __syncwarp();
        }
        if (S > 1) {
            // The blocks of the cluster add their partial tiles: block r owns every S-th slice of the 128 features and gets
            // the others' rows of BN tokens into its shared memory. The rings are free once every block is through its k blocks.
            const int slice = (BM + S - 1) / S;
            float* reduce_buf = reinterpret_cast<float*>(staging);
            __syncwarp();
            tc::fence_before_sync();
            tc::cluster_arrive();
            tc::cluster_wait();
            const int tile = first_tile, n0 = (tile % tiles_n) * BM, m0 = (tile / tiles_n) * BN;
            const int epi = (int)threadIdx.x - 32 * C::FIRST_EPI;                // 0 .. 32 * EPI_WARPS - 1
            {
                const int f = quarter * 32 + lane;
                const int owner = f / slice, lf = f - owner * slice;
                const uint32_t remote = tc::map_to_rank(reduce_buf + ((size_t)rank * slice + lf) * BN, (uint32_t)owner);
                const int sw = split_swizzle<BN>(lf);
#pragma unroll
                for (int q = 0; q < C::EPI_COLS / 4; ++q)
                    if (m0 + c_begin + 4 * q < p.M)
                        tc::st_cluster_f32x4(remote + (uint32_t)(((c_begin / 4 + q) ^ sw) * 16), __float_as_uint(sum[4 * q]),
                                             __float_as_uint(sum[4 * q + 1]), __float_as_uint(sum[4 * q + 2]), __float_as_uint(sum[4 * q + 3]));
            }
            tc::cluster_arrive();
            tc::cluster_wait();
            {
                const int first_feature = rank * slice;
                const int my_features = max(0, min(slice, BM - first_feature));
                const int items = my_features * min(BN / 4, (p.M - m0 + 3) / 4);
                for (int item = epi; item < items; item += 32 * C::EPI_WARPS) {
                    const int lf = item % my_features, c = item / my_features;
                    const int n = n0 + first_feature + lf, m = m0 + 4 * c;
                    const float bias = (p.bias && n < p.N) ? __ldg(p.bias + n) : 0.f;
                    const float* mine = reduce_buf + (size_t)lf * BN + 4 * (c ^ split_swizzle<BN>(lf));
                    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                    for (int r = 0; r < S; ++r) {
                        const float4 a = *reinterpret_cast<const float4*>(mine + (size_t)r * slice * BN);
                        v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
                    }
                    if (n >= p.N) continue;
                    const float u[4] = {v.x, v.y, v.z, v.w};
                    finish<4>(p, m, n, u, bias);
                }
            }
        }
    } else if (warp < C::LAST_CONV) {
        if constexpr (C::GROUPED) asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
        // A thread splits the 32 k of one feature; the swizzle puts the pieces that neighbouring lanes read side by side
        // into different banks.
        const int quarter = warp & 3, row = quarter * 32 + lane, group = (warp - C::FIRST_CONV) >> 2;
        for (int it = group; it < n_its; it += C::CONV_GROUPS) {
            const int ss = it % C::STAGINGS, os = it % C::OPERANDS;
            if (!warp_wait(&staged[ss], (it / C::STAGINGS) & 1, abort_flag)) break;
            const uint8_t* from = staging + ss * C::STAGING_BYTES + row * (BK * 4);
            float x[BK];
#pragma unroll
            for (int g = 0; g < BK / 4; ++g) {
                const float4 u = *reinterpret_cast<const float4*>(from + ((g ^ (row & 7)) << 4));
                x[4 * g] = u.x; x[4 * g + 1] = u.y; x[4 * g + 2] = u.z; x[4 * g + 3] = u.w;
            }
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&staging_free[ss]);
            if (!warp_wait(&mma_done[os], ((it / C::OPERANDS) & 1) ^ 1, abort_flag)) break;
            tc::fence_after_sync();
            const uint32_t to = tmem_w + os * W_COLS + ((uint32_t)(quarter * 32) << 16);
#pragma unroll
            for (int plane = 0; plane < 3; ++plane) {
                uint32_t w[BK / 2];
#pragma unroll
                for (int j = 0; j < BK / 2; ++j) w[j] = take_bf16x2(x[2 * j], x[2 * j + 1]);
                tc::tmem_st_x16(to + plane * (BK / 2), w);
            }
            tc::tmem_st_wait();
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&split_done[os]);
        }
        stand_by();
    } else if (C::X_SPLIT) {
        if (tc::elect_one()) fetch_planes();
        stand_by();
    } else {
        // Eight values of a token's row at a time: 32 bytes of staging, 16 bytes of each plane.
        for (int it = warp - C::FIRST_X; it < n_its; it += C::X_WARPS) {
            const int ss = it % C::STAGINGS, os = it % C::OPERANDS;
            if (!warp_wait(&staged[ss], (it / C::STAGINGS) & 1, abort_flag) ||
                !warp_wait(&mma_done[os], ((it / C::OPERANDS) & 1) ^ 1, abort_flag)) break;
#pragma unroll
            for (int item = lane; item < BN * (BK / 8); item += 32) {
                const int row = item % BN, g = item / BN;
                const uint8_t* from = staging + ss * C::STAGING_BYTES + (BM + row) * (BK * 4);
                const float4 u = *reinterpret_cast<const float4*>(from + (((2 * g) ^ (row & 7)) << 4));
                const float4 v = *reinterpret_cast<const float4*>(from + (((2 * g + 1) ^ (row & 7)) << 4));
                float x[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
                uint8_t* to = operands + os * C::OPERAND_BYTES + row * PLANE_ROW + ((g ^ ((row >> 1) & 3)) << 4);
#pragma unroll
                for (int plane = 0; plane < 3; ++plane) {
                    uint4 w;
                    w.x = take_bf16x2(x[0], x[1]);
                    w.y = take_bf16x2(x[2], x[3]);
                    w.z = take_bf16x2(x[4], x[5]);
                    w.w = take_bf16x2(x[6], x[7]);
                    *reinterpret_cast<uint4*>(to + plane * BN * PLANE_ROW) = w;
                }
            }
            tc::fence_proxy_async();                      // what was written is read by the tensor core
            __syncwarp();
            if (lane == 0) {
                tc::mbar_arrive(&split_done[os]);
                tc::mbar_arrive(&staging_free[ss]);
            }
        }
        stand_by();
    }
    __syncwarp();
    tc::fence_before_sync();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag) atomicOr(p.error_flag, 8);
    if (warp == 1) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem_base, C::TMEM_COLS);
    }
}

// The three bfloat16 planes of X [M,K] in tiles of ROWS tokens x 32 k, each as it lies in shared memory: three planes of
// ROWS rows of 64 bytes under the 64-byte swizzle; [token tiles][k blocks] of them, zeros behind K, rows past the last
// token left as they are (nobody reads their columns of the product).
template <int ROWS>
__global__ void __launch_bounds__(256) split_rows_kernel(const float* X, int ldx, uint8_t* planes, int M, int K, int kblocks) {
    dd_launch_dependents();
    dd_grid_wait();
    // neighbouring threads: the four pieces of eight k of a row's k block, then the next rows
    const int t = blockIdx.x * 256 + threadIdx.x, g = t & 3, m = t >> 2, kb = blockIdx.y, k = kb * BK + 8 * g;
    if (m >= M) return;
    const float* from = X + (size_t)m * ldx + k;          // K and ldx are multiples of 4
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 u = k < K ? *reinterpret_cast<const float4*>(from) : zero;
    const float4 v = k + 4 < K ? *reinterpret_cast<const float4*>(from + 4) : zero;
    float x[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
    const int row = m % ROWS;
    uint8_t* to = planes + ((size_t)(m / ROWS) * kblocks + kb) * (3 * ROWS * PLANE_ROW) + row * PLANE_ROW + ((g ^ ((row >> 1) & 3)) << 4);
#pragma unroll
    for (int plane = 0; plane < 3; ++plane) {
        uint4 w;
        w.x = take_bf16x2(x[0], x[1]);
        w.y = take_bf16x2(x[2], x[3]);
        w.z = take_bf16x2(x[4], x[5]);
        w.w = take_bf16x2(x[6], x[7]);
        *reinterpret_cast<uint4*>(to + plane * ROWS * PLANE_ROW) = w;
    }
}

typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_fn() {
    static const EncodeTiled fn = [] {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
            sym = nullptr;
        return reinterpret_cast<EncodeTiled>(sym);
    }();
    return fn;
}

// rows x K float32 matrix with row stride ld elements; boxes of box_rows x 32, 128-byte swizzle
int make_map(CUtensorMap* map, const void* base, int rows, int K, int ld, int box_rows, const char* what) {
    EncodeTiled enc = encode_fn();
    if (!enc) return dd_fail("dd_gemm_split: cuTensorMapEncodeTiled is not available from this driver");
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
    cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
    cuuint32_t elem[2] = {1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, elem,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return dd_fail("dd_gemm_split: cannot describe %s to TMA (driver error %d)", what, (int)r);
    return 0;
}

template <int BN>
int launch(const SplitParams& p, int splits, int sm_count, cudaStream_t s) {
    using C = SplitConfig<BN>;
    static const cudaError_t configured =
        cudaFuncSetAttribute(gemm_split_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
    if (configured != cudaSuccess)
        return dd_fail("dd_gemm_split: shared memory of %d bytes refused: %s", C::SMEM_BYTES, cudaGetErrorString(configured));
    CUtensorMap mw, mx;
    if (int e = make_map(&mw, p.W, p.N, p.K, p.ldw, BM, "the weight matrix")) return e;
    if (C::X_SPLIT) {
        const int kblocks = dd_ceil_div(p.K, BK);
        if (!p.planes || ((uintptr_t)p.planes & 127)) return dd_fail("dd_gemm_split: tiles of %d tokens need aligned scratch for the tokens' planes", BN);
        if (kblocks > 65535) return dd_fail("dd_gemm_split: K=%d is too long", p.K);
        dd_launch(split_rows_kernel<BN>, dim3(dd_ceil_div((long long)p.M * 4, 256), kblocks), dim3(256), 0, s, p.X, p.ldx, const_cast<uint8_t*>(p.planes),
                  p.M, p.K, kblocks);
        if (int e = dd_check_launch("dd_gemm_split (planes)")) return e;
        mx = mw;                                          // not used
    } else if (int e = make_map(&mx, p.X, p.M, p.K, p.ldx, BN, "the activations")) return e;
    const int tiles = dd_ceil_div(p.N, BM) * dd_ceil_div(p.M, BN);
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(splits > 1 ? tiles * splits : (tiles < sm_count ? tiles : sm_count));
    config.blockDim = dim3(C::THREADS);
    config.dynamicSmemBytes = C::SMEM_BYTES;
    config.stream = s;
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeClusterDimension;
    attrs[0].val.clusterDim.x = splits;
    attrs[0].val.clusterDim.y = 1;
    attrs[0].val.clusterDim.z = 1;
    attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[1].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attrs;
    config.numAttrs = dd_pdl_enabled ? 2 : 1;
    cudaError_t e = cudaLaunchKernelEx(&config, gemm_split_kernel<BN>, mw, mx, p);
    if (e != cudaSuccess) return dd_fail("dd_gemm_split (cluster of %d): %s", splits, cudaGetErrorString(e));
    return dd_check_launch("dd_gemm_split");
}

}  // namespace

// The token tile (16, 32, 64 or 128) and how many blocks of a cluster share a tile's K (at most 8).
DD_API int dd_gemm_split_plan(int M, int N, int K, int sm_count, int* token_tile) {
    const int bn = M <= 16 ? 16 : (M <= 32 ? 32 : (M <= 64 ? 64 : 128));
    const int tiles = dd_ceil_div(N, BM) * dd_ceil_div(M, bn), kblocks = dd_ceil_div(K, BK);
    int splits = tiles > 0 ? sm_count / tiles : 1;
    if (splits > 8) splits = 8;
    if (splits > kblocks / 4) splits = kblocks / 4;
    if (splits < 1) splits = 1;
    if (token_tile) *token_tile = bn;
    return splits;
}

// X [M,K] and W [N,K] float32, 16-byte aligned, row strides and K multiples of 4; bias [N] or null; residual [M,N] (row
// stride ldr, may be out itself) or null; out [M,N] float32. token_tile and splits: see dd_gemm_split_plan. planes: scratch
// for tiles of 64 and 128 tokens, 192 bytes for each token (rounded up to whole tiles) and 32 k, 128-byte aligned.
DD_API int dd_gemm_split(const float* X, int ldx, const float* W, int ldw, const float* bias, const float* residual, int ldr,
                         float* out, int ldo, int M, int N, int K, int act, int token_tile, int splits, int sm_count,
                         void* planes, int* error_flag, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (M == 1) ldx = K;                                         // (the stride of a single row may be anything)
    if (N == 1) ldw = K;
    if (ldx < K || ldw < K) return dd_fail("dd_gemm_split: rows of %d elements lie over one another (strides %d, %d)", K, ldx, ldw);
    if (K <= 0 || K % 4 || ldx % 4 || ldw % 4 || (((uintptr_t)X | (uintptr_t)W) & 15))
        return dd_fail("dd_gemm_split: K=%d and the row strides (%d, %d) must be multiples of 4 and the operands 16-byte aligned", K, ldx, ldw);
    const int kblocks = dd_ceil_div(K, BK);
    if (splits < 1 || splits > 8 || splits > kblocks) return dd_fail("dd_gemm_split: bad split count %d for %d k blocks", splits, kblocks);
    if (sm_count < 1) return dd_fail("dd_gemm_split: bad SM count %d", sm_count);
    SplitParams p = {X, W, (const uint8_t*)planes, bias, residual, out, error_flag, M, N, K, ldx, ldw, ldr, ldo, act, dd_ceil_div(kblocks, splits)};
    splits = dd_ceil_div(kblocks, p.kblocks_per_split);          // no empty split
    cudaStream_t s = (cudaStream_t)stream;
    switch (token_tile) {
        case 16: return launch<16>(p, splits, sm_count, s);
        case 32: return launch<32>(p, splits, sm_count, s);
        case 64: return launch<64>(p, splits, sm_count, s);
        case 128: return launch<128>(p, splits, sm_count, s);
    }
    return dd_fail("dd_gemm_split: token tile %d is not one of 16, 32, 64, 128", token_tile);
}
