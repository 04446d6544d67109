// float32 GEMM for a step of up to 8 rows and a large matrix: out[M,N] = act(X[M,K] . W[N,K]^T + bias) (+ residual), float32
// multiply-adds on the CUDA cores.
//
// What bounds it: 4 us of start, first bytes and last sums for any size, then the stream of the weights (4 bytes for 8
// multiply-adds: at 6 TB/s a third of what the CUDA cores do) and the reads of X from shared memory, which hold large matrices
// to 4.7 TB/s. Nobody has anything to wait for but its own weights. A warp owns R rows of W (and their results) at a time; a lane owns every
// 32nd group of four k of them, copies those 16 bytes a row itself through a ring (cp.async, the first stages before the
// kernel before this one is done) and multiplies R x 4 weights with 8 x 4 values of X from shared memory, so a value that is
// read serves R rows. It keeps R x 8 sums (pairs: fma.rn.f32x2); the lanes' sums are added in float64 and rounded once. With
// chains of K / 64 multiply-adds the error against 64 bits is 0.95e-7 for K = 1,600 and 6,400, where the split product on the
// tensor cores (gemm_split_tcgen05.cu), which serves more rows, has 1.04e-7 and 1.24e-7. Where X does not fit beside the rings
// (8 x 1,792 values) the blocks of a cluster share K and send their sums, as float64 too, to the block that finishes them: two
// barriers of the cluster a round, and where a matrix takes several rounds the split product is ahead (4,096 x 4,096 at 8 rows
// 18.4 us, here 27.6). Registers of 512 threads: 112 and 122 for R = 2 and 3, all 128 and 24 bytes of spills for R = 4.
//
// 8 rows, split product / this one, us: 4,800 x 1,600 11.9 / 9.3, 6,400 x 1,600 14.2 / 11.0, 3,072 x 1,024 13.7 / 5.8 (parts/linear.py
// says which products come here). With the weights in TMA boxes of R rows x 256 k a warp 10.1, 11.8, 6.2; 8 warps of 3 to 6 rows
// each 9.5, 11.2, 6.1 (50,257 x 1,600: 75.7 us, now 68.3); two blocks of 8 warps an SM 10.5, 11.0, 5.7.
#include "common.cuh"
#include "tcgen05.cuh"
#include <atomic>

namespace {

constexpr int MR = 8, WARPS = 16, THREADS = WARPS * 32, BOX_K = 256, SUB_K = 128, MAX_BOXES = 7, MAX_SPLITS = 8;
constexpr int X_BYTES = MAX_BOXES * MR * BOX_K * 4;
constexpr int STREAM_BYTES = 9 * 1024;                       // of a warp's ring, at most
template <int R> struct StreamConfig {
    static constexpr int STAGE_BYTES = R * BOX_K * 4;
    static constexpr int STAGES = STREAM_BYTES / STAGE_BYTES;
    static constexpr int OUTS = R * MR;
    static constexpr int SMEM_BYTES = X_BYTES + WARPS * STAGES * STAGE_BYTES;
    static constexpr int MOST_BYTES = SMEM_BYTES + MAX_SPLITS * WARPS * OUTS * 8;         // with the sums of a cluster's blocks
    static_assert(MOST_BYTES <= 226 * 1024 && STAGES >= 2, "shared memory");
};

struct StreamParams {
    const float* W;
    const float* bias;           // [N] or null
    const float* residual;       // [M, ldr] or null; may be out itself
    float* out;                  // [M, ldo]
    int* error_flag;
    int M, N, K, ldw, ldr, ldo, act, slice;     // slice: the k of a block of the cluster, a multiple of SUB_K
};

__device__ __forceinline__ void fma_pair(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool live) {
    const int bytes = live ? 16 : 0;                       // zeros beyond the matrix
    asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void st_cluster_f64(uint32_t addr, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}

// A lane's sums of one row for 8 tokens -> the whole sum of token lane >> 2, in all four lanes of that token.
__device__ __forceinline__ double token_sum(const unsigned long long* acc, int lane) {
    double v[MR];
#pragma unroll
    for (int m = 0; m < MR; ++m) {
        float lo, hi;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(acc[m]));
        v[m] = (double)lo + (double)hi;
    }
#pragma unroll
    for (int n = MR / 2, o = 16; n > 0; n >>= 1, o >>= 1) {
        const bool upper = lane & o;
#pragma unroll
        for (int j = 0; j < n; ++j) {
            const double give = upper ? v[j] : v[j + n], keep = upper ? v[j + n] : v[j];
            v[j] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
    return v[0];
}

__device__ __forceinline__ void finish(const StreamParams& p, int m, int n, double sum) {
    if (m >= p.M || n >= p.N) return;
    const float res = p.residual ? p.residual[(size_t)m * p.ldr + n] : 0.f;
    p.out[(size_t)m * p.ldo + n] = dd_activation((float)sum + (p.bias ? p.bias[n] : 0.f), p.act) + res;
}

template <int R>
__global__ void __launch_bounds__(THREADS, 1)
gemm_stream_kernel(const __grid_constant__ CUtensorMap map_x, const StreamParams p) {
    using C = StreamConfig<R>;
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t x_full[MAX_BOXES];
    __shared__ int abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = (int)tc::cluster_size(), rank = (int)tc::cluster_rank();
    const int cluster = blockIdx.x / S, clusters = gridDim.x / S;
    const int groups = (p.N + R - 1) / R;
    const int k0 = rank * p.slice, subs = (min(p.slice, p.K - k0) + SUB_K - 1) / SUB_K, boxes = (subs + 1) / 2;
    // the groups of R rows are dealt out over the clusters first, then over the warps
    const int first = cluster + clusters * warp, step = clusters * WARPS;
    const int mine = first < groups ? (groups - 1 - first) / step + 1 : 0, rounds = (groups - 1 - cluster) / step + 1;
    uint8_t* ring = smem + X_BYTES + warp * C::STAGES * C::STAGE_BYTES;

    dd_launch_dependents();
    if (threadIdx.x == 0) {
        for (int i = 0; i < MAX_BOXES; ++i) tc::mbar_init(&x_full[i], 1);
        abort_flag = 0;
        tc::fence_barrier_init();
        tc::fence_proxy_async();
    }
    __syncthreads();
    const int total = mine * boxes;
    // the next box of this warp, in the order in which it is used; a lane copies what it will read itself, so that nobody but
    // the lane waits for it
    int fetched = 0, fetch_stage = 0, fetch_box = 0, fetch_n = first * R;
    auto fetch = [&] {
        if (fetched < total) {
            const int k = k0 + fetch_box * BOX_K + lane * 4;
            const float* from = p.W + (size_t)fetch_n * p.ldw + k;
            const uint32_t to = tc::smem_u32(ring) + fetch_stage * C::STAGE_BYTES + lane * 16;
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const bool live = fetch_n + r < p.N && k + h * SUB_K < p.K;
                    cp_async16(to + (r * BOX_K + h * SUB_K) * 4, live ? from + (size_t)r * p.ldw + h * SUB_K : p.W, live);
                }
            ++fetched;
            if (++fetch_stage == C::STAGES) fetch_stage = 0;
            if (++fetch_box == boxes) { fetch_box = 0; fetch_n += step * R; }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int i = 0; i < C::STAGES - 1; ++i) fetch();
    dd_grid_wait();              // X and the residual are earlier kernels' results
    if (threadIdx.x == 0)
        for (int i = 0; i < boxes; ++i) {
            tc::mbar_expect_tx(&x_full[i], MR * BOX_K * 4);
            tc::tma_load_2d(smem + i * MR * BOX_K * 4, &map_x, k0 + i * BOX_K, 0, &x_full[i]);       // rows past the last token read as zeros
        }

    bool ok = true;
    int stage = 0;
    for (int round = 0; round < rounds; ++round) {
        const bool work = round < mine;
        const int n0 = (first + round * step) * R;
        unsigned long long acc[R][MR];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int m = 0; m < MR; ++m) acc[r][m] = 0ull;
        if (work) {
#pragma unroll 1
            for (int b = 0; b < boxes; ++b) {
                if (round == 0) ok = ok && __all_sync(0xffffffffu, tc::mbar_wait(&x_full[b], 0, &abort_flag));
                if (!ok) break;
                fetch();                                     // into the stage that the box before has left
                asm volatile("cp.async.wait_group %0;" ::"n"(C::STAGES - 1) : "memory");
                const ulonglong2* w = reinterpret_cast<const ulonglong2*>(ring + stage * C::STAGE_BYTES) + lane;
                const ulonglong2* x = reinterpret_cast<const ulonglong2*>(smem + b * MR * BOX_K * 4) + lane;
                const int here = min(2, subs - 2 * b);
#pragma unroll 1
                for (int h = 0; h < here; ++h, w += 32, x += 32) {
                    ulonglong2 xv[MR];
#pragma unroll
                    for (int m = 0; m < MR; ++m) xv[m] = x[m * (BOX_K / 4)];
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const ulonglong2 wv = w[r * (BOX_K / 4)];
#pragma unroll
                        for (int m = 0; m < MR; ++m) fma_pair(acc[r][m], xv[m].x, wv.x);
#pragma unroll
                        for (int m = 0; m < MR; ++m) fma_pair(acc[r][m], xv[m].y, wv.y);
                    }
                }
                if (++stage == C::STAGES) stage = 0;
            }
        }
        if (S == 1) {
            if (work) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const double sum = token_sum(acc[r], lane);
                    if ((lane & 3) == (r & 3)) finish(p, lane >> 2, n0 + r, sum);
                }
            }
            continue;
        }
        // The cluster's sums of this round's groups: those of warp w are finished by block w % S, which adds them in rank order.
        double* sums = reinterpret_cast<double*>(smem + C::SMEM_BYTES);
        __syncwarp();
        tc::cluster_arrive();
        tc::cluster_wait();                                  // every block is there, and through with the round before
        if (work) {
            const uint32_t to = tc::map_to_rank(sums + ((size_t)rank * WARPS + warp) * C::OUTS, (uint32_t)(warp % S));
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const double sum = token_sum(acc[r], lane);
                if ((lane & 3) == (r & 3)) st_cluster_f64(to + (r * MR + (lane >> 2)) * 8, sum);
            }
        }
        __syncwarp();
        tc::cluster_arrive();
        tc::cluster_wait();
        if (work && warp % S == rank) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if ((lane & 3) != (r & 3)) continue;
                double sum = 0.0;
                for (int s = 0; s < S; ++s) sum += sums[((size_t)s * WARPS + warp) * C::OUTS + r * MR + (lane >> 2)];
                finish(p, lane >> 2, n0 + r, sum);
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (!ok && lane == 0) atomicOr(p.error_flag, 8);
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

// rows x K float32 matrix with row stride ld elements; boxes of box_rows x BOX_K as they lie
int make_map(CUtensorMap* map, const void* base, int rows, int K, int ld, int box_rows, const char* what) {
    EncodeTiled enc = encode_fn();
    if (!enc) return dd_fail("dd_gemm_stream: cuTensorMapEncodeTiled is not available from this driver");
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
    cuuint32_t box[2] = {(cuuint32_t)BOX_K, (cuuint32_t)box_rows};
    cuuint32_t elem[2] = {1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return dd_fail("dd_gemm_stream: cannot describe %s to TMA (driver error %d)", what, (int)r);
    return 0;
}

cudaLaunchConfig_t launch_config(int smem, int splits, cudaStream_t s, cudaLaunchAttribute* attrs) {
    cudaLaunchConfig_t config = {};
    config.blockDim = dim3(THREADS);
    config.dynamicSmemBytes = smem;
    config.stream = s;
    attrs[0].id = cudaLaunchAttributeClusterDimension;
    attrs[0].val.clusterDim.x = splits;
    attrs[0].val.clusterDim.y = 1;
    attrs[0].val.clusterDim.z = 1;
    attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[1].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attrs;
    config.numAttrs = dd_pdl_enabled ? 2 : 1;
    return config;
}

template <int R> int smem_bytes(int splits) {
    return StreamConfig<R>::SMEM_BYTES + (splits > 1 ? splits * WARPS * StreamConfig<R>::OUTS * 8 : 0);
}

constexpr int MAX_DEVICES = 16;             // whose answers are kept; of others they are asked for anew

int device() {
    int d = -1;
    return cudaGetDevice(&d) == cudaSuccess ? d : -1;
}

// The kernel's shared memory, once a device (two threads that both ask set the same).
template <int R> cudaError_t configure() {
    static std::atomic<bool> configured[MAX_DEVICES];
    const int d = device();
    const bool kept = d >= 0 && d < MAX_DEVICES;
    if (kept && configured[d].load(std::memory_order_acquire)) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(gemm_stream_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, StreamConfig<R>::MOST_BYTES);
    if (kept && e == cudaSuccess) configured[d].store(true, std::memory_order_release);
    return e;
}

// Clusters that are resident at once: of four blocks fewer than a quarter of the SMs' number, and a second wave of them
// doubles the time. Of every R the same: each takes more than half of an SM's shared memory, so one block fits.
int resident_clusters(int splits, int sm_count) {
    static std::atomic<int> resident[MAX_DEVICES][MAX_SPLITS + 1];
    static_assert(StreamConfig<2>::SMEM_BYTES > 114 * 1024 && StreamConfig<3>::SMEM_BYTES > 114 * 1024 && StreamConfig<4>::SMEM_BYTES > 114 * 1024, "one block an SM");
    const int d = device();
    const bool kept = d >= 0 && d < MAX_DEVICES;
    int n = kept ? resident[d][splits].load(std::memory_order_relaxed) : 0;
    if (!n) {
        cudaLaunchAttribute attrs[2];
        cudaLaunchConfig_t config = launch_config(smem_bytes<4>(splits), splits, nullptr, attrs);
        config.gridDim = dim3(splits);
        config.numAttrs = 1;
        if (configure<4>() != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, gemm_stream_kernel<4>, &config) != cudaSuccess || n < 1) {
            cudaGetLastError();
            n = sm_count / splits;
        } else if (kept) resident[d][splits].store(n, std::memory_order_relaxed);
    }
    return n < sm_count / splits ? n : sm_count / splits;
}

template <int R>
int launch(const CUtensorMap& map_x, const StreamParams& p, int splits, int clusters, cudaStream_t s) {
    if (cudaError_t e = configure<R>()) return dd_fail("dd_gemm_stream: shared memory refused: %s", cudaGetErrorString(e));
    cudaLaunchAttribute attrs[2];
    cudaLaunchConfig_t config = launch_config(smem_bytes<R>(splits), splits, s, attrs);
    const int groups = dd_ceil_div(p.N, R);
    config.gridDim = dim3((groups < clusters ? groups : clusters) * splits);
    cudaError_t e = cudaLaunchKernelEx(&config, gemm_stream_kernel<R>, map_x, p);
    if (e != cudaSuccess) return dd_fail("dd_gemm_stream (cluster of %d): %s", splits, cudaGetErrorString(e));
    return dd_check_launch("dd_gemm_stream");
}

}  // namespace

// How many clusters of so many blocks dd_gemm_stream takes to be resident at once on the current device's first sm_count SMs.
DD_API int dd_gemm_stream_clusters(int splits, int sm_count) {
    return splits < 1 || splits > MAX_SPLITS || sm_count < splits ? 0 : resident_clusters(splits, sm_count);
}

// X [M,K] (M up to 8) and W [N,K] float32, 16-byte aligned, row strides and K multiples of 4, rows that do not lie over one
// another; bias [N] or null; residual [M,N] (row stride ldr, may be out itself) or null; out [M,N] float32.
DD_API int dd_gemm_stream(const float* X, int ldx, const float* W, int ldw, const float* bias, const float* residual, int ldr,
                          float* out, int ldo, int M, int N, int K, int act, int sm_count, int* error_flag, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (M > MR) return dd_fail("dd_gemm_stream: takes up to %d rows (got %d)", MR, M);
    if (M == 1) ldx = K;                                         // (the stride of a single row may be anything)
    if (N == 1) ldw = K;
    if (ldx < K || ldw < K) return dd_fail("dd_gemm_stream: rows of %d elements lie over one another (strides %d, %d)", K, ldx, ldw);
    if (K <= 0 || K % 4 || ldx % 4 || ldw % 4 || (((uintptr_t)X | (uintptr_t)W) & 15))
        return dd_fail("dd_gemm_stream: K=%d and the row strides (%d, %d) must be multiples of 4 and the operands 16-byte aligned", K, ldx, ldw);
    // the blocks of a cluster that share K, and how much of it each takes (no empty slice)
    int splits = dd_ceil_div(K, MAX_BOXES * BOX_K);
    if (splits > MAX_SPLITS || splits > sm_count) return dd_fail("dd_gemm_stream: K=%d is too long", K);
    const int slice = dd_ceil_div(dd_ceil_div(K, splits), SUB_K) * SUB_K;
    splits = dd_ceil_div(K, slice);
    // How many rows of W a warp takes at a time: the fewest rows one after the other when the groups are dealt out over all
    // warps that are resident, and the widest group for that (6,400 x 1,600: 3, in one round; 50,257 x 1,600: 2, in eleven).
    const int clusters = resident_clusters(splits, sm_count);
    int rows = 0, best = 0;
    for (int r = 4; r >= 2; --r) {
        const int cost = dd_ceil_div(dd_ceil_div(N, r), clusters * WARPS) * r;
        if (!rows || cost < best) { rows = r; best = cost; }
    }
    CUtensorMap mx;
    if (int e = make_map(&mx, X, M, K, ldx, MR, "the activations")) return e;
    const StreamParams p = {W, bias, residual, out, error_flag, M, N, K, ldw, ldr, ldo, act, slice};
    cudaStream_t s = (cudaStream_t)stream;
    if (rows == 2) return launch<2>(mx, p, splits, clusters, s);
    if (rows == 3) return launch<3>(mx, p, splits, clusters, s);
    return launch<4>(mx, p, splits, clusters, s);
}
