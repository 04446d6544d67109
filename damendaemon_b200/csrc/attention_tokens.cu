// Paged causal attention of single tokens (a decode step), for float32 and bfloat16 caches on the CUDA cores: rows of a
// head of up to 128 elements that are whole 16-byte pieces, any key/value groups, a window, a chunked mask and a gate per
// head, with the meaning that attention_rows.cu gives them (that kernel is the reference). Scores, softmax and the
// weighted sum are float32 whatever the storage type.
//
// A block owns a token's head and reads its keys with whole rows by groups of lanes, eight key and eight value rows of a
// group in flight at once; every group keeps a running maximum and sum of its own, and the groups meet at the end (in the
// warp by shuffles, in the block through shared memory). A token's keys may be cut over the blocks of a cluster, whose
// results meet in the shared memory of the first: no scratch, no second launch. The step's own key and value are taken
// from the projection and written to the cache here, and all other keys are earlier steps': the first eight rows of every
// group (of heads of 64: 128 keys of a block in float32, 256 in bfloat16) are requested before the kernel waits for the
// projection. Beside that projection, us: float32, 8 requests x 25 heads at 70 keys 34 -> 6 (the general kernel, its merge
// and the cache write before); bfloat16, 8 requests x 25 heads on 5 at 400 keys 32 -> 6.4. What bounds it is the chain
// position -> page -> rows -> merge with few tokens; with long contexts a batch's instructions and the wait for its rows,
// which two blocks an SM do not hide: bfloat16, 8 requests x 32 heads of 128 on 8, 4,000 and 16,000 keys 99 and 374 (general
// kernel 175 and 618), float32 180 and 709 (797 for the longer); 8 x 25 heads of 64 in float32, 4,000 keys 106 (222). The
// figures of the rule for the pieces are beside it (parts/paged_attention.py).
#include "attention_cores.cuh"

namespace {
constexpr int WARPS = 8, BATCH = 8;
constexpr int MOST = 8;                                     // blocks of a cluster

template <typename T> struct Piece;                          // 16 bytes of a row
template <> struct Piece<float> {
    static constexpr int N = 4;
    __device__ static void unpack(const uint4& w, float* x) {
        x[0] = __uint_as_float(w.x); x[1] = __uint_as_float(w.y); x[2] = __uint_as_float(w.z); x[3] = __uint_as_float(w.w);
    }
    __device__ static float exp(float x) { return expf(x); }
};
template <> struct Piece<__nv_bfloat16> {
    static constexpr int N = 8;
    __device__ static void unpack(const uint4& w, float* x) {
        const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            x[2 * i] = __uint_as_float(u[i] << 16);
            x[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
        }
    }
    __device__ static float exp(float x) { return __expf(x); }
};

// D: 16, 32, 64 or 128, the elements that LANES lanes hold of a row (a head has d <= D). Blocks: tokens, their heads, the
// pieces of the keys.
template <typename T, int D>
__global__ void __launch_bounds__(32 * WARPS, 2)
attention_tokens_kernel(const T* q, const T* k_new, const T* v_new, int q_stride, T* cache, const int* positions, T* out, int out_stride, int H,
                        Pages pages, Mask mask, float scale, const T* gate, int gate_stride, int* error_flag) {
    constexpr int E = Piece<T>::N, LANES = D / E, GROUPS = 32 / LANES;      // GROUPS keys a warp reads at once
    constexpr int KEYS = GROUPS * BATCH;                    // keys of a warp's batch
    __shared__ __align__(16) float part_o[WARPS][D];
    __shared__ float part_m[WARPS], part_l[WARPS];
    __shared__ __align__(16) float all_o[MOST][D];
    __shared__ float all_m[MOST], all_l[MOST];
    dd_launch_dependents();
    const int S = (int)cluster_size(), rank = (int)cluster_rank();
    const int row = blockIdx.x / S, t = row / H, h = row % H;
    if (S > 1) cluster_arrive();                            // "my shared memory exists"
    const int ratio = H / pages.kv_heads, kh = h / ratio, d = pages.d;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, group = lane / LANES, c = lane % LANES * E;
    const bool mine = c < d;                                // this lane's elements are inside the head
    const long long value_plane = pages.value_plane();
    const T* own_k = k_new ? k_new + (size_t)t * q_stride + (size_t)kh * d : nullptr;
    const T* own_v = v_new ? v_new + (size_t)t * q_stride + (size_t)kh * d : nullptr;
    const uint4 nothing = make_uint4(0, 0, 0, 0);
    // positions and the block table are the step's inputs, and with the step's own key at hand the cache is read at earlier
    // steps' keys only: all that is known before the projection is done
    if (!own_k) dd_grid_wait();
    const int pos = positions[t];
    const int lo = mask.first_seen(pos);
    int per = (pos + 1 - lo + S - 1) / S;
    per = (per + KEYS - 1) / KEYS * KEYS;                   // a piece of the keys is whole batches
    const int k_end = min(pos + 1, lo + (rank + 1) * per);
    uint4 kv[BATCH], vv[BATCH];
    uint32_t live = 0;                                      // bit u: key u of the batch exists
    auto fetch = [&](int base) {                            // a batch's rows, but for the step's own key's
        // all pages are asked for before the first of them is looked at (with a look between, the answers come one after the
        // other), and a key's place in its page is worked out once: a batch of 128 keys of 128 elements takes 2.6 us, 5.7 before
        Pages::Place place[BATCH];
#pragma unroll
        for (int u = 0; u < BATCH; ++u) place[u] = pages.place(t, min(base + u * GROUPS, k_end - 1));
        live = 0;
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            const int key = base + u * GROUPS;
            kv[u] = vv[u] = nothing;
            if (key >= k_end) continue;
            if (own_k && key == pos) {
                live |= 1u << u;
                continue;
            }
            const long long at = pages.row_at(place[u], kh);
            if (at < 0) {
                atomicOr(error_flag, 4);
                continue;
            }
            live |= 1u << u;
            if (mine) {
                kv[u] = *reinterpret_cast<const uint4*>(cache + at + c);
                vv[u] = *reinterpret_cast<const uint4*>(cache + at + value_plane + c);
            }
        }
    };
    int base = lo + rank * per + warp * KEYS + group;
    if (base - group < k_end) fetch(base);
    if (own_k) dd_grid_wait();

    float qv[E];
    Piece<T>::unpack(mine ? *reinterpret_cast<const uint4*>(q + (size_t)t * q_stride + (size_t)h * d + c) : nothing, qv);
    if (own_k && rank == S - 1 && h == kh * ratio && warp == WARPS - 1 && lane < LANES && mine) {
        const long long at = pos >= 0 ? pages.key_row(t, pos, kh) : -1;
        if (at < 0) {
            if (c == 0) atomicOr(error_flag, 2);
        } else {
            *reinterpret_cast<uint4*>(cache + at + c) = *reinterpret_cast<const uint4*>(own_k + c);
            *reinterpret_cast<uint4*>(cache + at + value_plane + c) = *reinterpret_cast<const uint4*>(own_v + c);
        }
    }
    float m = -CUDART_INF_F, l = 0.f, o[E];
#pragma unroll
    for (int i = 0; i < E; ++i) o[i] = 0.f;
    while (base - group < k_end) {                          // the same count for a warp's lanes
        float s[BATCH], top = m;
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            if (own_k && base + u * GROUPS == pos && mine) {
                kv[u] = *reinterpret_cast<const uint4*>(own_k + c);
                vv[u] = *reinterpret_cast<const uint4*>(own_v + c);
            }
            float k[E];
            Piece<T>::unpack(kv[u], k);
            s[u] = qv[0] * k[0];
#pragma unroll
            for (int i = 1; i < E; ++i) s[u] = fmaf(qv[i], k[i], s[u]);
        }
#pragma unroll
        for (int x = 1; x < LANES; x <<= 1)
#pragma unroll
            for (int u = 0; u < BATCH; ++u) s[u] += __shfl_xor_sync(0xffffffffu, s[u], x);
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            s[u] = live >> u & 1 ? s[u] * scale : -CUDART_INF_F;
            top = fmaxf(top, s[u]);
        }
        if (top != -CUDART_INF_F) {
            const float corr = Piece<T>::exp(m - top);
            l *= corr;
#pragma unroll
            for (int i = 0; i < E; ++i) o[i] *= corr;
#pragma unroll
            for (int u = 0; u < BATCH; ++u) {
                const float p = live >> u & 1 ? Piece<T>::exp(s[u] - top) : 0.f;
                float v[E];
                Piece<T>::unpack(vv[u], v);
                l += p;
#pragma unroll
                for (int i = 0; i < E; ++i) o[i] = fmaf(p, v[i], o[i]);
            }
            m = top;
        } else {                                            // no score above -infinity: none at all, or NaN, which must not get lost
#pragma unroll
            for (int u = 0; u < BATCH; ++u)
                if (isnan(s[u])) l = s[u];
        }
        __syncwarp();
        base += WARPS * KEYS;
        if (base - group < k_end) fetch(base);
    }
    // the warp's groups, then the block's warps, then the cluster's blocks
    float top = m;
#pragma unroll
    for (int x = LANES; x < 32; x <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, x));
    const float mine_in_warp = m == -CUDART_INF_F ? 0.f : Piece<T>::exp(m - top);
    l *= mine_in_warp;
#pragma unroll
    for (int i = 0; i < E; ++i) o[i] *= mine_in_warp;
#pragma unroll
    for (int x = LANES; x < 32; x <<= 1) {
        l += __shfl_xor_sync(0xffffffffu, l, x);
#pragma unroll
        for (int i = 0; i < E; ++i) o[i] += __shfl_xor_sync(0xffffffffu, o[i], x);
    }
    if (group == 0) {
#pragma unroll
        for (int i = 0; i < E; ++i) part_o[warp][c + i] = o[i];
        if (c == 0) {
            part_m[warp] = top;
            part_l[warp] = l;
        }
    }
    __syncthreads();
    const int i = threadIdx.x;
    float sum = 0.f, acc = 0.f;
    if (i < D) {
        top = -CUDART_INF_F;
#pragma unroll
        for (int x = 0; x < WARPS; ++x) top = fmaxf(top, part_m[x]);
#pragma unroll
        for (int x = 0; x < WARPS; ++x) {
            const float w = part_m[x] == -CUDART_INF_F ? 0.f : Piece<T>::exp(part_m[x] - top);
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
                const float w = all_m[r] == -CUDART_INF_F ? 0.f : Piece<T>::exp(all_m[r] - top);
                sum = fmaf(all_l[r], w, sum);
                acc = fmaf(all_o[r][i], w, acc);
            }
        }
    }
    if (i < d) {
        float inv = sum == 0.f ? 0.f : 1.0f / sum;
        if (gate) inv *= logistic(dd_to_f32(gate[(size_t)t * gate_stride + h]));
        out[(size_t)t * out_stride + (size_t)h * d + i] = dd_from_f32<T>(acc * inv);
    }
}

template <typename T>
int launch(const void* q, const void* k_new, const void* v_new, int q_stride, void* cache, const int* positions, void* out, int out_stride,
           int n_tokens, int H, int splits, const Pages& pages, const Mask& mask, float scale, const void* gate, int gate_stride,
           int* error_flag, cudaStream_t s) {
#define DD_TOKENS(D)                                                                                                                       \
    return launch_clusters("dd_attention_tokens", attention_tokens_kernel<T, D>, (long long)n_tokens * H, splits, 32 * WARPS, 0, s, (const T*)q, \
                           (const T*)k_new, (const T*)v_new, q_stride, (T*)cache, positions, (T*)out, out_stride, H, pages, mask, scale,   \
                           (const T*)gate, gate_stride, error_flag)
    if (pages.d <= 16) DD_TOKENS(16);
    if (pages.d <= 32) DD_TOKENS(32);
    if (pages.d <= 64) DD_TOKENS(64);
    DD_TOKENS(128);
#undef DD_TOKENS
}
}  // namespace

// One query a token; token t is at positions[t] and belongs to row t of block_table. k_new, v_new: null (its key and value
// are in the cache), or row views of q's stride with them, which are then written to the cache. splits: blocks (at most 8)
// that share a token's keys.
DD_API int dd_attention_tokens(const void* q, const void* k_new, const void* v_new, int q_stride, void* cache, const int* positions,
                               int n_tokens, const int* block_table, int max_blocks, void* out, int out_stride, int n_heads, int kv_heads,
                               int head_dim, int page_size, int n_pages, int window, int chunk, float scale, int splits, const void* gate,
                               int gate_stride, int dtype, int* error_flag, void* stream) {
    if (n_tokens <= 0) return 0;
    if (dtype != DD_F32 && dtype != DD_BF16) return dd_fail("dd_attention_tokens: unknown dtype %d", dtype);
    if (int e = check_sizes("dd_attention_tokens", n_heads, kv_heads, head_dim, page_size, q, q_stride, dtype == DD_F32 ? 4 : 2, cache, window, chunk)) return e;
    if ((!k_new) != (!v_new) || (((uintptr_t)k_new | (uintptr_t)v_new) & 15)) return dd_fail("dd_attention_tokens: keys and values come together, 16-byte aligned");
    if (splits < 1 || splits > MOST) return dd_fail("dd_attention_tokens: %d splits", splits);
    const Pages pages = {block_table, max_blocks, page_size, n_pages, kv_heads, head_dim, shift_of(page_size)};
    const Mask mask = {window, chunk};
    if (dtype == DD_F32)
        return launch<float>(q, k_new, v_new, q_stride, cache, positions, out, out_stride, n_tokens, n_heads, splits, pages, mask, scale, gate,
                             gate_stride, error_flag, (cudaStream_t)stream);
    return launch<__nv_bfloat16>(q, k_new, v_new, q_stride, cache, positions, out, out_stride, n_tokens, n_heads, splits, pages, mask, scale, gate,
                                 gate_stride, error_flag, (cudaStream_t)stream);
}
