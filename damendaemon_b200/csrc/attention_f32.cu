// Paged causal attention of prompt portions over float32 caches: head sizes that are multiples of 4 up to 128, any
// key/value groups, a window, a chunked mask and a gate per head, with the meaning that attention_rows.cu gives them (that
// kernel serves all other sizes and options and is the reference; single tokens go to attention_tokens.cu). Everything is
// float32 multiply-add on the CUDA cores: scores, softmax (expf) and the weighted value sum.
//
// The general kernel spends a warp on one query of one head and reads every key and value row again for each of them:
// 1,100 us for 1,000 tokens x 20 heads of 64, where the multiply-adds alone need 38. Here a block owns 64 queries of a head
// and reads each block of 64 keys once for all of them into shared memory (cp.async, the next block's keys under this
// block's softmax and values, its values under the next scores); a thread holds 4 x 8 scores and 4 queries' pieces of the
// output in registers: 106 us. What bounds it now are the reads of shared memory (12 of 16 bytes for 128 multiply-adds a
// thread, 56 us) and the few warps that hide them (registers: three blocks an SM).
#include "attention_cores.cuh"

namespace {

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool live) {
    const int bytes = live ? 16 : 0;                       // zeros where there is nothing to copy
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

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
// A key that a query does not see is not part of its sum, whatever its row holds: a weight of zero would make NaN of an
// infinite value. Blocks of keys that some query of the tile does not see are looked through for such values (each thread
// its own copies, the answer rides on the barrier that is there anyway) and then added pair by pair.
template <int D>
__global__ void __launch_bounds__(THREADS, D <= 64 ? 3 : 1)
attention_f32_prompt_kernel(const float* q, int q_stride, const float* cache, const int* entry_start, const int* entry_pos0, int n_entries,
                            float* out, int out_stride, int H, Pages pages, Mask mask, float scale, const float* gate, int gate_stride,
                            int* error_flag) {
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
    const int kv_lo = mask.first_seen(pos_first), lo_last = mask.first_seen(pos_last);
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
                const float p = s[i][j] == -CUDART_INF_F ? 0.f : expf(s[i][j] - m_new);     // (a NaN stays one, also where it is alone)
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
        const int first = kv_lo + b * BKV, last = min(first + BKV - 1, pos_last);
        bool odd = false;
        if (last > pos_first || first < lo_last) {          // a mask's border runs through the block
            float test = 0.f;
            for (int i = tid; i < BKV * NC; i += THREADS) {
                const float4 v = *reinterpret_cast<const float4*>(sV + i / NC * LD + i % NC * 4);
                test = fmaf(v.x, 0.f, fmaf(v.y, 0.f, fmaf(v.z, 0.f, fmaf(v.w, 0.f, test))));
            }
            odd = test != 0.f;                              // 0, or NaN if some value is not finite
        }
        if (__syncthreads_or(odd)) {                        // this block's values and weights are there
#pragma unroll 1
            for (int k = 0; k < BKV; ++k)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (first + k < lo[i] || first + k > hi[i]) continue;
                    const float w = sP[(ty + 16 * i) * LP + k];
#pragma unroll
                    for (int j = 0; j < OJ; ++j) {
                        const Quad v = load_quad(sV + k * LD + 4 * tx + 32 * j);
                        fma2(o[i][2 * j], pair_of(w, w), v.lo);
                        fma2(o[i][2 * j + 1], pair_of(w, w), v.hi);
                    }
                }
        } else
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
                if (ls[i] == 0.f) continue;                // no key seen there (a sum of NaN counts)
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
    if (int e = check_sizes("dd_attention_f32_prompt", n_heads, kv_heads, head_dim, page_size, q, q_stride, 4, cache, window, chunk)) return e;
    if (splits < 1 || splits > PROMPT_SPLITS) return dd_fail("dd_attention_f32_prompt: %d splits", splits);
    if (out_stride % 4 || ((uintptr_t)out & 15)) return dd_fail("dd_attention_f32_prompt: rows of the result must be 16-byte aligned");
    const Pages pages = {block_table, max_blocks, page_size, n_pages, kv_heads, head_dim, shift_of(page_size)};
    const Mask mask = {window, chunk};
    cudaStream_t s = (cudaStream_t)stream;
    if (head_dim <= 32) return launch_prompt<32>(q, q_stride, cache, entry_start, entry_pos0, n_entries, n_tokens, out, out_stride, n_heads, splits, pages, mask, scale, gate, gate_stride, error_flag, s);
    if (head_dim <= 64) return launch_prompt<64>(q, q_stride, cache, entry_start, entry_pos0, n_entries, n_tokens, out, out_stride, n_heads, splits, pages, mask, scale, gate, gate_stride, error_flag, s);
    return launch_prompt<128>(q, q_stride, cache, entry_start, entry_pos0, n_entries, n_tokens, out, out_stride, n_heads, splits, pages, mask, scale, gate, gate_stride, error_flag, s);
}
