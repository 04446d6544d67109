// Paged causal attention for float32 caches: a kernel for prompt portions and one for single tokens. Both take head
// sizes that are multiples of 4 up to 128, any key/value groups, a window, a chunked mask and a gate per head, with the
// meaning that attention_rows.cu gives them (that kernel serves all other sizes and options and is the reference of
// these two). Everything is float32 multiply-add on the CUDA cores: scores, softmax (expf) and the weighted value sum.
//
// The general kernel spends a warp on one query of one head and reads every key and value row again for each of them:
// 1,100 us for 1,000 tokens x 20 heads of 64, where the multiply-adds alone need 38. Here a block of a prompt owns 64
// queries of a head and reads each block of 64 keys once for all of them into shared memory (cp.async, the next block's
// keys under this block's softmax and values, its values under the next scores); a thread holds 4 x 8 scores and 4
// queries' pieces of the output in registers: 106 us. What bounds it now are the reads of shared memory (12 of 16 bytes
// for 128 multiply-adds a thread, 56 us) and the few warps that hide them (registers: three blocks an SM). A single
// token's block reads whole rows by groups of lanes, eight key and eight value rows of a group in flight at once, every
// group with a running maximum and sum of its own; a token's keys may be cut over the blocks of a cluster, whose results
// meet in the shared memory of the first (no scratch, no second launch), and the step's own key and value are taken from
// the projection and written to the cache here: 8 requests x 25 heads, 70 keys, in a graph 5.7 us against 34 for the
// general kernel, its merge and the cache write; at 1,000 keys 31 us (3.3 TB/s).
#include "common.cuh"
#include <math_constants.h>

namespace {

struct Pages {
    const int* block_table;      // [entries, max_blocks]
    int max_blocks, page_size, n_pages, kv_heads, d;
    int page_shift;              // log2 of the page size where that is a power of two, else -1
    // element offset of a key's row in the cache (its head kh), -1 without a page; the value row lies value_plane() further on
    __device__ __forceinline__ long long key_row(int entry, int key, int kh) const {
        const int blk = page_shift >= 0 ? key >> page_shift : key / page_size;
        const int page = blk < max_blocks ? block_table[(size_t)entry * max_blocks + blk] : -1;
        if (page < 0 || page >= n_pages) return -1;
        return ((long long)page * 2 * kv_heads + kh) * page_size * d + (long long)(key - blk * page_size) * d;
    }
    __device__ __forceinline__ long long value_plane() const { return (long long)kv_heads * page_size * d; }
};

struct Mask {
    int window, chunk;
    // the first key that a query at pos sees
    __device__ __forceinline__ int first_seen(int pos) const {
        int lo = window > 0 ? max(0, pos - window + 1) : 0;
        if (chunk > 0) lo = max(lo, pos - pos % chunk);
        return lo;
    }
};

__device__ __forceinline__ float logistic(float v) { return 1.0f / (1.0f + expf(-v)); }

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool live) {
    const int bytes = live ? 16 : 0;                       // zeros where there is nothing to copy
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t cluster_size() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// Four values to the same place in the shared memory of the cluster's first block.
__device__ __forceinline__ void send4(const float* where, float4 v) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(remote) : "r"((unsigned)__cvta_generic_to_shared(where)));
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(remote), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

// ---- prompt portions ----
// Two float32 multiply-adds with one instruction (registers in pairs): the multiply-add rate stays, the issue slots that
// the loads and the softmax need are freed.
typedef unsigned long long pair_t;
__device__ __forceinline__ pair_t pair_of(float lo, float hi) {
    pair_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpair(pair_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ void fma2(pair_t& acc, pair_t a, pair_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b)); }
__device__ __forceinline__ void mul2(pair_t& v, pair_t f) { asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(f)); }
struct Quad { pair_t lo, hi; };
__device__ __forceinline__ Quad load_quad(const float* p) {
    Quad r;
    asm("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(r.lo), "=l"(r.hi) : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
    return r;
}

constexpr int BQ = 64, BKV = 64, THREADS = 128;
template <int D> struct PromptSmem { static constexpr int BYTES = (3 * BQ * (D + 4) + BQ * (BKV + 4)) * 4 + 2 * BKV * 8; };
constexpr int PROMPT_SPLITS = 4;                            // blocks that may share a tile's keys

// D: columns of the tiles (a head has d <= D elements, the rest is zero). Threads: 16 rows of 8; a thread's queries are
// ty + 16 i and its keys tx + 8 j, so that the 16-byte reads of a warp (rows padded by 16 bytes) meet no bank twice.
// The blocks of a cluster take a tile's key blocks in turn; what they found meets in the first one's shared memory. (One
// block a tile left 1.6 of three possible blocks on an SM for 1,000 tokens x 20 heads and the SMs with the last tiles busy
// twice as long as the others: 148 us.)
template <int D>
__global__ void __launch_bounds__(THREADS, D <= 64 ? 3 : 1)
attention_f32_prompt_kernel(const float* __restrict__ q, int q_stride, const float* __restrict__ cache, const int* __restrict__ entry_start,
                            const int* __restrict__ entry_pos0, int n_entries, float* __restrict__ out, int out_stride, int H, Pages pages,
                            Mask mask, float scale, const float* __restrict__ gate, int gate_stride, int* __restrict__ error_flag) {
    constexpr int LD = D + 4, LP = BKV + 4, NC = D / 4, OJ = D / 32;
    extern __shared__ __align__(16) float smem[];
    float* sQ = smem;
    float* sK = sQ + BQ * LD;
    float* sV = sK + BKV * LD;
    float* sP = sV + BKV * LD;
    long long* rows_of = reinterpret_cast<long long*>(sP + BQ * LP);       // [2][BKV] key rows' offsets, blocks alternating
    dd_launch_dependents();
    dd_grid_wait();
    // which tile of which entry; a long prompt's last tiles, which see the most keys, come first, all heads' side by side
    const int S = (int)cluster_size(), rank = (int)cluster_rank();
    int e = 0, tile = blockIdx.x / S / H, len = 0;
    for (; e < n_entries; ++e) {
        len = entry_start[e + 1] - entry_start[e];
        const int n = (len + BQ - 1) / BQ;
        if (tile < n) { tile = n - 1 - tile; break; }
        tile -= n;
    }
    if (e == n_entries) return;
    const int h = blockIdx.x / S % H, kh = h / (H / pages.kv_heads), d = pages.d;
    const int q0 = tile * BQ, rows = min(BQ, len - q0), row0 = entry_start[e] + q0;
    const int pos_first = entry_pos0[e] + q0, pos_last = pos_first + rows - 1;
    const int kv_lo = mask.first_seen(pos_first);
    const int n_blocks = (pos_last - kv_lo) / BKV + 1;
    const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
    const long long value_plane = pages.value_plane();

    auto look_up = [&](int b, int turn) {                   // the key rows of block b
        if (b < n_blocks && tid < BKV) {
            const int key = kv_lo + b * BKV + tid;
            long long at = -1;
            if (key <= pos_last) {
                at = pages.key_row(e, key, kh);
                if (at < 0) atomicOr(error_flag, 4);
            }
            rows_of[(turn & 1) * BKV + tid] = at;
        }
    };
    auto load = [&](int b, int turn, float* dst, long long plane) {
        if (b < n_blocks)
            for (int i = tid; i < BKV * NC; i += THREADS) {
                const int r = i / NC, c = i % NC * 4;
                const long long at = rows_of[(turn & 1) * BKV + r];
                const bool live = at >= 0 && c < d;
                cp_async16(dst + r * LD + c, cache + (live ? at + plane + c : 0), live);
            }
        cp_commit();
    };
    for (int i = tid; i < BQ * NC; i += THREADS) {
        const int r = i / NC, c = i % NC * 4;
        const bool live = r < rows && c < d;
        cp_async16(sQ + r * LD + c, q + (live ? (size_t)(row0 + r) * q_stride + (size_t)h * d + c : 0), live);
    }
    look_up(rank, 0);
    __syncthreads();
    load(rank, 0, sK, 0);                                   // (group: queries and the first keys)
    load(rank, 0, sV, value_plane);

    pair_t o[4][2 * OJ];
    float m[4], l[4];
    int lo[4], hi[4];                                       // the keys a query sees
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int pos = pos_first + ty + 16 * i;
        lo[i] = mask.first_seen(pos);
        hi[i] = pos;
        m[i] = -CUDART_INF_F;
        l[i] = 0.f;
#pragma unroll
        for (int j = 0; j < 2 * OJ; ++j) o[i][j] = 0;
    }
    int turn = 0;
    for (int b = rank; b < n_blocks; b += S, ++turn) {
        look_up(b + S, turn + 1);
        cp_wait<1>();
        __syncthreads();                                    // this block's keys are there, the next one's rows looked up
        // A score is the sum of pieces of 16 elements, each from its even and its odd ones: shorter chains of additions
        // are less far from the exact sum (and from the sums that the single-token kernel makes in other orders).
        float s[4][8];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) s[i][j] = 0.f;
#pragma unroll 1
        for (int c0 = 0; c0 < D; c0 += 16) {
            pair_t part[4][8];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) part[i][j] = 0;
#pragma unroll
            for (int c = c0; c < c0 + 16; c += 4) {
                Quad a[4], k[8];
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] = load_quad(sQ + (ty + 16 * i) * LD + c);
#pragma unroll
                for (int j = 0; j < 8; ++j) k[j] = load_quad(sK + (tx + 8 * j) * LD + c);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        fma2(part[i][j], a[i].lo, k[j].lo);
                        fma2(part[i][j], a[i].hi, k[j].hi);
                    }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    float even, odd;
                    unpair(part[i][j], even, odd);
                    s[i][j] += even + odd;
                }
        }
        __syncthreads();                                    // everybody is through with the keys
        load(b + S, turn + 1, sK, 0);
        bool live[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) live[j] = rows_of[(turn & 1) * BKV + tx + 8 * j] >= 0;
        const int key0 = kv_lo + b * BKV + tx;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float top = -CUDART_INF_F;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int key = key0 + 8 * j;
                s[i][j] = live[j] && key >= lo[i] && key <= hi[i] ? s[i][j] * scale : -CUDART_INF_F;
                top = fmaxf(top, s[i][j]);
            }
#pragma unroll
            for (int x = 1; x < 8; x <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, x));
            const float m_new = fmaxf(m[i], top);
            const bool none = m_new == -CUDART_INF_F;       // no key seen yet
            const float corr = none ? 1.f : expf(m[i] - m_new);
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float p = none ? 0.f : expf(s[i][j] - m_new);
                sum += p;
                sP[(ty + 16 * i) * LP + tx + 8 * j] = p;
            }
#pragma unroll
            for (int x = 1; x < 8; x <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
            l[i] = l[i] * corr + sum;
            m[i] = m_new;
#pragma unroll
            for (int j = 0; j < 2 * OJ; ++j) mul2(o[i][j], pair_of(corr, corr));
        }
        cp_wait<1>();
        __syncthreads();                                    // this block's values and weights are there
#pragma unroll 2
        for (int k = 0; k < BKV; k += 4) {
            float4 p[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) p[i] = *reinterpret_cast<const float4*>(sP + (ty + 16 * i) * LP + k);
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int j = 0; j < OJ; ++j) {
                    const Quad v = load_quad(sV + (k + u) * LD + 4 * tx + 32 * j);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float w = u == 0 ? p[i].x : u == 1 ? p[i].y : u == 2 ? p[i].z : p[i].w;
                        fma2(o[i][2 * j], pair_of(w, w), v.lo);
                        fma2(o[i][2 * j + 1], pair_of(w, w), v.hi);
                    }
                }
        }
        __syncthreads();                                    // everybody is through with the values and the weights
        load(b + S, turn + 1, sV, value_plane);
    }
    float acc[4][4 * OJ];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2 * OJ; ++j) unpair(o[i][j], acc[i][2 * j], acc[i][2 * j + 1]);
    if (S > 1) {
        // the blocks have the same threads at the same places of the tile: a thread's values go to its like in the first block
        constexpr int PIECES = 4 * OJ + 2;                  // of four values: outputs, maxima, sums
        static_assert((PROMPT_SPLITS - 1) * PIECES * THREADS * 16 <= PromptSmem<D>::BYTES, "the others' results fit");
        float4* met = reinterpret_cast<float4*>(smem);
        cp_wait<0>();
        __syncwarp();
        cluster_arrive();
        cluster_wait();                                     // every block is through with its tiles
        if (rank) {
            float4* to = met + (size_t)(rank - 1) * PIECES * THREADS + tid;
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < OJ; ++j)
                    send4(reinterpret_cast<float*>(to + (i * OJ + j) * THREADS), make_float4(acc[i][4 * j], acc[i][4 * j + 1], acc[i][4 * j + 2], acc[i][4 * j + 3]));
            send4(reinterpret_cast<float*>(to + 4 * OJ * THREADS), make_float4(m[0], m[1], m[2], m[3]));
            send4(reinterpret_cast<float*>(to + (4 * OJ + 1) * THREADS), make_float4(l[0], l[1], l[2], l[3]));
        }
        __syncwarp();
        cluster_arrive();
        cluster_wait();
        if (rank) return;
        for (int r = 0; r < S - 1; ++r) {
            const float4* from = met + (size_t)r * PIECES * THREADS + tid;
            const float4 m4 = from[4 * OJ * THREADS], l4 = from[(4 * OJ + 1) * THREADS];
            const float ms[4] = {m4.x, m4.y, m4.z, m4.w}, ls[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (ms[i] == -CUDART_INF_F) continue;
                const float top = fmaxf(m[i], ms[i]);
                const float mine = expf(m[i] - top), theirs = expf(ms[i] - top);
                m[i] = top;
                l[i] = l[i] * mine + ls[i] * theirs;
#pragma unroll
                for (int j = 0; j < OJ; ++j) {
                    const float4 v = from[(i * OJ + j) * THREADS];
                    acc[i][4 * j] = acc[i][4 * j] * mine + v.x * theirs;
                    acc[i][4 * j + 1] = acc[i][4 * j + 1] * mine + v.y * theirs;
                    acc[i][4 * j + 2] = acc[i][4 * j + 2] * mine + v.z * theirs;
                    acc[i][4 * j + 3] = acc[i][4 * j + 3] * mine + v.w * theirs;
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = ty + 16 * i;
        if (r >= rows) continue;
        float inv = l[i] > 0.f ? 1.0f / l[i] : (l[i] == 0.f ? 0.f : l[i]);
        if (gate) inv *= logistic(gate[(size_t)(row0 + r) * gate_stride + h]);
        float* to = out + (size_t)(row0 + r) * out_stride + (size_t)h * d;
#pragma unroll
        for (int j = 0; j < OJ; ++j) {
            const int c = 4 * tx + 32 * j;
            if (c < d) *reinterpret_cast<float4*>(to + c) = make_float4(acc[i][4 * j] * inv, acc[i][4 * j + 1] * inv, acc[i][4 * j + 2] * inv, acc[i][4 * j + 3] * inv);
        }
    }
}

// ---- single tokens ----
constexpr int DECODE_WARPS = 8, BATCH = 8;

// D: 16, 32, 64 or 128; LANES lanes hold a row of D elements, 4 each. Blocks: tokens, their heads, the pieces of the keys.
template <int D>
__global__ void __launch_bounds__(32 * DECODE_WARPS)
attention_f32_decode_kernel(const float* __restrict__ q, const float* __restrict__ k_new, const float* __restrict__ v_new, int q_stride,
                            float* __restrict__ cache, const int* __restrict__ positions, float* __restrict__ out, int out_stride, int H,
                            Pages pages, Mask mask, float scale, const float* __restrict__ gate, int gate_stride, int* __restrict__ error_flag) {
    constexpr int LANES = D / 4, GROUPS = 32 / LANES;      // keys a warp reads at once
    constexpr int MOST = 8;                                 // blocks of a cluster
    __shared__ __align__(16) float part_o[DECODE_WARPS * GROUPS][D];
    __shared__ float part_m[DECODE_WARPS * GROUPS], part_l[DECODE_WARPS * GROUPS];
    __shared__ __align__(16) float all_o[MOST][D];
    __shared__ float all_m[MOST], all_l[MOST];
    dd_launch_dependents();
    dd_grid_wait();
    const int S = (int)cluster_size(), rank = (int)cluster_rank();
    const int row = blockIdx.x / S, t = row / H, h = row % H;
    if (S > 1) cluster_arrive();                            // "my shared memory exists"
    const int ratio = H / pages.kv_heads, kh = h / ratio, d = pages.d;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, group = lane / LANES, c = lane % LANES * 4;
    const bool mine = c < d;                                // this lane's four elements are inside the head
    const int pos = positions[t];
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const long long value_plane = pages.value_plane();
    const float* own_k = k_new ? k_new + (size_t)t * q_stride + (size_t)kh * d : nullptr;
    const float* own_v = v_new ? v_new + (size_t)t * q_stride + (size_t)kh * d : nullptr;
    if (own_k && rank == S - 1 && h == kh * ratio && warp == DECODE_WARPS - 1 && lane < LANES && mine) {
        const long long at = pos >= 0 ? pages.key_row(t, pos, kh) : -1;
        if (at < 0) {
            if (c == 0) atomicOr(error_flag, 2);
        } else {
            *reinterpret_cast<float4*>(cache + at + c) = *reinterpret_cast<const float4*>(own_k + c);
            *reinterpret_cast<float4*>(cache + at + value_plane + c) = *reinterpret_cast<const float4*>(own_v + c);
        }
    }
    const float4 qv = mine ? *reinterpret_cast<const float4*>(q + (size_t)t * q_stride + (size_t)h * d + c) : zero;

    const int lo = mask.first_seen(pos);
    // whole rounds of a warp's keys for every warp of every block: a piece starts on a multiple of a round
    constexpr int ROUND = DECODE_WARPS * GROUPS * BATCH;
    const int span = pos + 1 - lo;
    int per = (span + S - 1) / S;
    per = (per + GROUPS * BATCH - 1) / (GROUPS * BATCH) * (GROUPS * BATCH);
    const int k_end = min(pos + 1, lo + (rank + 1) * per);
    float m = -CUDART_INF_F, l = 0.f;
    float4 o = zero;
    for (int base = lo + rank * per + warp * GROUPS * BATCH + group; base - group < k_end; base += ROUND) {
        float4 kv[BATCH], vv[BATCH];
        bool live[BATCH];
        const float* kp[BATCH];
        const float* vp[BATCH];
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            const int key = base + u * GROUPS;
            live[u] = key < k_end;
            kp[u] = vp[u] = nullptr;
            if (live[u]) {
                if (own_k && key == pos) {
                    kp[u] = own_k;
                    vp[u] = own_v;
                } else {
                    const long long at = pages.key_row(t, key, kh);
                    if (at < 0) {
                        atomicOr(error_flag, 4);
                        live[u] = false;
                    } else {
                        kp[u] = cache + at;
                        vp[u] = cache + at + value_plane;
                    }
                }
            }
        }
#pragma unroll
        for (int u = 0; u < BATCH; ++u) kv[u] = live[u] && mine ? *reinterpret_cast<const float4*>(kp[u] + c) : zero;
#pragma unroll
        for (int u = 0; u < BATCH; ++u) vv[u] = live[u] && mine ? *reinterpret_cast<const float4*>(vp[u] + c) : zero;
        float s[BATCH], top = m;
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            s[u] = fmaf(qv.w, kv[u].w, fmaf(qv.z, kv[u].z, fmaf(qv.y, kv[u].y, qv.x * kv[u].x)));
#pragma unroll
            for (int x = 1; x < LANES; x <<= 1) s[u] += __shfl_xor_sync(0xffffffffu, s[u], x);
            s[u] = live[u] ? s[u] * scale : -CUDART_INF_F;
            top = fmaxf(top, s[u]);
        }
        if (top == -CUDART_INF_F) continue;                 // (no shuffles below: groups may part here until the next round)
        const float corr = expf(m - top);
        l *= corr;
        o.x *= corr; o.y *= corr; o.z *= corr; o.w *= corr;
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            const float p = live[u] ? expf(s[u] - top) : 0.f;
            l += p;
            o.x = fmaf(p, vv[u].x, o.x);
            o.y = fmaf(p, vv[u].y, o.y);
            o.z = fmaf(p, vv[u].z, o.z);
            o.w = fmaf(p, vv[u].w, o.w);
        }
        m = top;
    }
    __syncwarp();
    const int slot = warp * GROUPS + group;
    *reinterpret_cast<float4*>(&part_o[slot][c]) = o;
    if (c == 0) {
        part_m[slot] = m;
        part_l[slot] = l;
    }
    __syncthreads();
    // the block's result, then the cluster's: an element a thread
    const int i = threadIdx.x;
    float top = -CUDART_INF_F, sum = 0.f, acc = 0.f;
    if (i < D) {
#pragma unroll
        for (int x = 0; x < DECODE_WARPS * GROUPS; ++x) top = fmaxf(top, part_m[x]);
        for (int x = 0; x < DECODE_WARPS * GROUPS; ++x) {
            if (part_m[x] == -CUDART_INF_F) continue;
            const float w = expf(part_m[x] - top);
            sum = fmaf(part_l[x], w, sum);
            acc = fmaf(part_o[x][i], w, acc);
        }
    }
    if (S > 1) {
        __syncwarp();
        cluster_wait();
        if (i < D) {
            auto send = [&](const float* where, float v) {
                uint32_t remote;
                asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(remote) : "r"((unsigned)__cvta_generic_to_shared(where)));
                asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(v) : "memory");
            };
            send(&all_o[rank][i], acc);
            if (i == 0) {
                send(&all_m[rank], top);
                send(&all_l[rank], sum);
            }
        }
        __syncwarp();
        cluster_arrive();
        cluster_wait();
        if (rank != 0) return;
        if (i < D) {
            top = -CUDART_INF_F;
            for (int r = 0; r < S; ++r) top = fmaxf(top, all_m[r]);
            sum = acc = 0.f;
            for (int r = 0; r < S; ++r) {
                if (all_m[r] == -CUDART_INF_F) continue;
                const float w = expf(all_m[r] - top);
                sum = fmaf(all_l[r], w, sum);
                acc = fmaf(all_o[r][i], w, acc);
            }
        }
    }
    if (i < d) {
        float inv = sum == 0.f ? 0.f : 1.0f / sum;
        if (gate) inv *= logistic(gate[(size_t)t * gate_stride + h]);
        out[(size_t)t * out_stride + (size_t)h * d + i] = acc * inv;
    }
}

int shift_of(int page_size) { return page_size > 0 && !(page_size & (page_size - 1)) ? __builtin_ctz(page_size) : -1; }

int check_sizes(const char* what, int n_heads, int kv_heads, int d, int page_size, const void* q, int q_stride, const void* cache, int window, int chunk) {
    if (d <= 0 || d % 4 || d > 128) return dd_fail("%s: head size %d is not a multiple of 4 up to 128", what, d);
    if (n_heads <= 0 || kv_heads <= 0 || n_heads % kv_heads || page_size <= 0)
        return dd_fail("%s: %d heads, %d key/value heads, pages of %d tokens", what, n_heads, kv_heads, page_size);
    if (q_stride % 4 || (((uintptr_t)q | (uintptr_t)cache) & 15)) return dd_fail("%s: rows must be 16-byte aligned", what);
    if (window < 0 || chunk < 0) return dd_fail("%s: window %d and chunk %d must not be negative", what, window, chunk);
    return 0;
}

template <typename... KArgs, typename... Args>
int launch_clusters(const char* what, void (*kernel)(KArgs...), long long blocks, int splits, int threads, int smem, cudaStream_t s, Args... args) {
    if (blocks * splits > 0x7fffffffLL) return dd_fail("%s: %lld x %d blocks are more than one launch takes", what, blocks, splits);
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3((unsigned)(blocks * splits));
    config.blockDim = dim3(threads);
    config.dynamicSmemBytes = smem;
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
    const cudaError_t e = cudaLaunchKernelEx(&config, kernel, static_cast<KArgs>(args)...);
    if (e != cudaSuccess) return dd_fail("%s (clusters of %d): %s", what, splits, cudaGetErrorString(e));
    return dd_check_launch(what);
}

template <int D>
int launch_prompt(const float* q, int q_stride, const float* cache, const int* entry_start, const int* entry_pos0, int n_entries, int n_tokens,
                  float* out, int out_stride, int H, int splits, const Pages& pages, const Mask& mask, float scale, const float* gate,
                  int gate_stride, int* error_flag, cudaStream_t s) {
    static const cudaError_t configured =
        cudaFuncSetAttribute(attention_f32_prompt_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, PromptSmem<D>::BYTES);
    if (configured != cudaSuccess) return dd_fail("dd_attention_f32_prompt: shared memory refused: %s", cudaGetErrorString(configured));
    return launch_clusters("dd_attention_f32_prompt", attention_f32_prompt_kernel<D>, ((long long)dd_ceil_div(n_tokens, BQ) + n_entries) * H, splits,
                           THREADS, PromptSmem<D>::BYTES, s, q, q_stride, cache, entry_start, entry_pos0, n_entries, out, out_stride, H, pages, mask,
                           scale, gate, gate_stride, error_flag);
}

template <int D>
int launch_decode(const float* q, const float* k_new, const float* v_new, int q_stride, float* cache, const int* positions, float* out,
                  int out_stride, int n_tokens, int H, int splits, const Pages& pages, const Mask& mask, float scale, const float* gate,
                  int gate_stride, int* error_flag, cudaStream_t s) {
    return launch_clusters("dd_attention_f32_decode", attention_f32_decode_kernel<D>, (long long)n_tokens * H, splits, 32 * DECODE_WARPS, 0, s, q,
                           k_new, v_new, q_stride, cache, positions, out, out_stride, H, pages, mask, scale, gate, gate_stride, error_flag);
}
}  // namespace

// Runs of consecutive tokens: entry e's are rows entry_start[e] .. entry_start[e + 1] - 1 of q, at positions
// entry_pos0[e] on, against the pages of row e of block_table, which hold this step's keys and values already. q and gate
// as in dd_attention_rows. n_tokens: rows of q (at least those of the entries). splits: blocks (at most 4) that share a
// tile's keys.
DD_API int dd_attention_f32_prompt(const float* q, int q_stride, const float* cache, const int* entry_start, const int* entry_pos0, int n_entries,
                                   int n_tokens, const int* block_table, int max_blocks, float* out, int out_stride, int n_heads, int kv_heads,
                                   int head_dim, int page_size, int n_pages, int window, int chunk, float scale, int splits, const float* gate,
                                   int gate_stride, int* error_flag, void* stream) {
    if (n_tokens <= 0 || n_entries <= 0) return 0;
    if (int e = check_sizes("dd_attention_f32_prompt", n_heads, kv_heads, head_dim, page_size, q, q_stride, cache, window, chunk)) return e;
    if (splits < 1 || splits > PROMPT_SPLITS) return dd_fail("dd_attention_f32_prompt: %d splits", splits);
    if (out_stride % 4 || ((uintptr_t)out & 15)) return dd_fail("dd_attention_f32_prompt: rows of the result must be 16-byte aligned");
    const Pages pages = {block_table, max_blocks, page_size, n_pages, kv_heads, head_dim, shift_of(page_size)};
    const Mask mask = {window, chunk};
    cudaStream_t s = (cudaStream_t)stream;
    if (head_dim <= 32) return launch_prompt<32>(q, q_stride, cache, entry_start, entry_pos0, n_entries, n_tokens, out, out_stride, n_heads, splits, pages, mask, scale, gate, gate_stride, error_flag, s);
    if (head_dim <= 64) return launch_prompt<64>(q, q_stride, cache, entry_start, entry_pos0, n_entries, n_tokens, out, out_stride, n_heads, splits, pages, mask, scale, gate, gate_stride, error_flag, s);
    return launch_prompt<128>(q, q_stride, cache, entry_start, entry_pos0, n_entries, n_tokens, out, out_stride, n_heads, splits, pages, mask, scale, gate, gate_stride, error_flag, s);
}

// One query a token; token t is at positions[t] and belongs to row t of block_table. k_new, v_new: null (its key and value
// are in the cache), or row views of q's stride with them, which are then written to the cache. splits: blocks (at most 8)
// that share a token's keys.
DD_API int dd_attention_f32_decode(const float* q, const float* k_new, const float* v_new, int q_stride, float* cache, const int* positions,
                                   int n_tokens, const int* block_table, int max_blocks, float* out, int out_stride, int n_heads, int kv_heads,
                                   int head_dim, int page_size, int n_pages, int window, int chunk, float scale, int splits, const float* gate,
                                   int gate_stride, int* error_flag, void* stream) {
    if (n_tokens <= 0) return 0;
    if (int e = check_sizes("dd_attention_f32_decode", n_heads, kv_heads, head_dim, page_size, q, q_stride, cache, window, chunk)) return e;
    if ((!k_new) != (!v_new) || (((uintptr_t)k_new | (uintptr_t)v_new) & 15)) return dd_fail("dd_attention_f32_decode: keys and values come together, 16-byte aligned");
    if (splits < 1 || splits > 8) return dd_fail("dd_attention_f32_decode: %d splits", splits);
    const Pages pages = {block_table, max_blocks, page_size, n_pages, kv_heads, head_dim, shift_of(page_size)};
    const Mask mask = {window, chunk};
    cudaStream_t s = (cudaStream_t)stream;
    if (head_dim <= 16) return launch_decode<16>(q, k_new, v_new, q_stride, cache, positions, out, out_stride, n_tokens, n_heads, splits, pages, mask, scale, gate, gate_stride, error_flag, s);
    if (head_dim <= 32) return launch_decode<32>(q, k_new, v_new, q_stride, cache, positions, out, out_stride, n_tokens, n_heads, splits, pages, mask, scale, gate, gate_stride, error_flag, s);
    if (head_dim <= 64) return launch_decode<64>(q, k_new, v_new, q_stride, cache, positions, out, out_stride, n_tokens, n_heads, splits, pages, mask, scale, gate, gate_stride, error_flag, s);
    return launch_decode<128>(q, k_new, v_new, q_stride, cache, positions, out, out_stride, n_tokens, n_heads, splits, pages, mask, scale, gate, gate_stride, error_flag, s);
}
