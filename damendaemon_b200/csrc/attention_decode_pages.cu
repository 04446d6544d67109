// Decode attention that streams whole cache pages with TMA, for bfloat16 caches with head size 64, as many
// key/value heads as heads, and pages of 16, 32, 64 or 128 tokens.
//
// In the cache a page holds the keys of all heads side by side and then the values ([page][K|V][head][slot][64]):
// the keys of G neighbouring heads are one run of G x page_size rows of 128 bytes. A block owns (token, group of
// G <= 8 heads, split of the token's pages); one warp asks TMA for one box of G x page_size rows of keys and one
// of values per page, as many pages ahead as the ring holds, so a block moves its bytes in pieces of tens of KB with two instructions
// each (copying the same bytes 16 at a time, one key row per 8 lanes, the memory system delivered 4.5 TB/s;
// in boxes of this size it delivers 5.4). The 128-byte swizzle of the tensor map is the layout ldmatrix wants.
// Each of the other warps owns one head of the group for all pages, so nothing is merged inside the block:
// scores and P.V on mma.sync m16n8k16 with the keys (and then the dimensions of the values) as its 16 rows and the single
// query (the weights) in every column, running maximum and sum in float32, base 2 (damendaemon/kernels.py:147-178; split
// merge by log-sum-exp kernels.py:190-210).
//
// With k_new/v_new the step's own key and value replace the cache row of the token's position in shared memory
// and are written to the cache by the warp that owns the head. Rows of the last page beyond the position are
// zeroed in shared memory (values) or masked by index (scores), so stale cache contents never reach the result.
// A token whose position is negative sees no key and gets zeros; one beyond the block table sees the keys that have
// pages, and the missing ones are reported (error bits 2 and 4) as a missing page is.
// n_splits is the most splits a token's pages may be cut into (the grid's third dimension); when the grid then holds
// more blocks than can be resident at once, the kernel gives each token its share of them, by its number of pages
// among all tokens' pages (see the kernel), and the blocks beyond a token's count leave at once.
// Every wait on a barrier is bounded (error bit 8).
#include "common.cuh"
#include "tcgen05.cuh"
#include <math_constants.h>

namespace {
constexpr int D = 64, TILE = 16, MAX_GROUP = 8;      // heads of a block: a warp each, and one that requests pages
constexpr int MAX_STAGES = 3;                 // deeper rings are no faster and leave fewer blocks an SM (see the kernel)

struct Params {
    const __nv_bfloat16* q;
    const __nv_bfloat16* k_new;
    const __nv_bfloat16* v_new;
    __nv_bfloat16* cache;
    const int* tok_entry;
    const int* tok_pos;
    const int* block_table;
    __nv_bfloat16* out;
    float* part_o;
    float* part_ml;
    int* counters;
    int* error_flag;
    int q_stride, out_stride, max_blocks, H, G, P, n_pages, window, stages;
    int chunk;                   // > 0: a query sees only the keys of its own chunk of this many positions
    const __nv_bfloat16* gate;   // null, or rows of gate_stride elements, one per head: sigmoid(gate) multiplies the head's output
    int gate_stride;
    int n_tokens, log2_P;
    int deal;                    // 1: more blocks in the grid than can be resident, so the splits are dealt out (see the kernel)
    float inv_block_budget;      // 1 / blocks that can be resident at once: the key splits are dealt out against them
    float scale_log2e;
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
// 16 rows of A times one column of B, which every column of B repeats (a lane's fragment does not depend on its column):
// every column of the result is the same, so one of a row's two accumulators in a lane is kept (row quad in c0, row
// quad + 8 in c1) and the other is fed with zeros and dropped.
__device__ __forceinline__ void mma_bf16_column(float& c0, float& c1, const uint32_t* a, uint32_t b0, uint32_t b1) {
    float d1, d3;
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%2,%1,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%10,%1,%10};"
                 : "+f"(c0), "+f"(c1), "=f"(d1), "=f"(d3)
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
    asm volatile("" ::"f"(d1), "f"(d3));      // the two dead accumulators count as used
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
// byte offset of 16-byte chunk c of key row r in a tile of 128-byte rows under the 128-byte swizzle
__device__ __forceinline__ uint32_t tile_off(int r, int c) { return (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4)); }

// What bounds it: a step of a few tokens is a chain of latencies, not a stream (8 tokens x 25 heads x 540 keys are 28 MB, 4.4 us of
// the memory's rate, and the kernel took 11.6 us of a layer). So nothing but data makes anybody wait: a warp of its own
// looks the pages up (the first 64 entries of the table are read beside the position, not after it) and requests them,
// the head warps follow it through full and empty barriers of the ring without a barrier of the block, keys and value
// dimensions are the 16 rows of mma.sync (8 of them a tile of 16 keys, not 16), and a head's splits are merged by
// the warp that finishes last, through a counter per head: before, the blocks' barriers, fences and the last block's
// walk over all its heads were 4.4 us behind the last key. Whole passes, before and now: 8 requests from 512 keys on
// (xl, 64 steps) 129.7 / 117.8 ms, 64 from 256 keys on 204.1 / 195.8, 32 of 16 to 800 keys (medium) 48.9 / 44.4.
// With pages of 16 tokens, three stages of groups of up to six heads (75 KB) and 80 registers leave three blocks an SM; groups of
// seven and eight (87 and 99 KB) leave two. Measured with 16 heads in groups of six (medium) and 25 in groups of seven (xl):
// 104 registers and two blocks 45.9 ms (118.0), two stages 44.5 (122.3), four 46.2; a spilled register costs more than any.
// Groups of eight (288 threads) take two blocks' registers, 96 a thread.
template <int MOST>
__global__ void __launch_bounds__((MOST + 1) * 32, MOST < 8 ? 3 : 2)
attention_decode_pages_kernel(const __grid_constant__ CUtensorMap map_kv, const __grid_constant__ CUtensorMap map_last, const Params p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int box_bytes = p.G * p.P * 128;                 // keys (or values) of the group's heads in one page
    uint64_t* full = reinterpret_cast<uint64_t*>(tiles + (size_t)p.stages * 2 * box_bytes);
    uint64_t* empty = full + MAX_STAGES;
    volatile int* stage_page = reinterpret_cast<volatile int*>(empty + MAX_STAGES);     // the page a stage holds, -1: none
    __shared__ int abort_flag;
    dd_launch_dependents();

    // Positions, entries and the block table are this step's inputs, not an earlier kernel's results: they are read
    // while the kernel before this one is still running.
    // The grid holds the most splits a token may need (gridDim.z, the slowest index, so that the splits every token
    // has are launched first); how many a token gets is decided here, from all tokens' positions, so that blocks do
    // about equal work whatever the contexts are: the step's pages x head groups are dealt out over the blocks that
    // can be resident at once, a token takes its share rounded to the nearest count, and the blocks beyond it leave.
    // (One split per token with contexts spread over 1..1000 made the kernel as long as its longest token: 61 us for
    // 64 tokens x 20 heads against 44 us with the long ones cut in three; with equal contexts nothing changes.)
    const int split = blockIdx.z, g = blockIdx.y, t = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int quad = lane >> 2, t4 = lane & 3;
    const int head0 = g * p.G;                              // first head of the group
    const int group_heads = min(p.G, p.H - head0);
    const CUtensorMap* map = group_heads == p.G ? &map_kv : &map_last;      // boxes of the last group's few heads
    const int pos = p.tok_pos[t];
    // without tok_entry token t is entry t (a step of single tokens in entry order): one trip to L2 less before the pages
    const int* bt = p.block_table + (size_t)(p.tok_entry ? p.tok_entry[t] : t) * p.max_blocks;
    int held[2] = {-1, -1};                                 // the page warp: entries lane and 32 + lane of a short table
    const bool short_table = p.max_blocks <= 64;
    if (warp == p.G) {
        if (short_table) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
                if (i * 32 + lane < p.max_blocks) held[i] = bt[i * 32 + lane];
        }
        if (lane == 0) {
            for (int s = 0; s < p.stages; ++s) {
                tc::mbar_init(&full[s], 1);
                tc::mbar_init(&empty[s], group_heads);
            }
            abort_flag = 0;
            tc::fence_barrier_init();
            tc::fence_proxy_async();
            tc::prefetch_tensormap(map);
        }
    }
    __syncthreads();                                        // the only one: from here every warp goes at its own pace

    // (page sizes are powers of two, and the block budget's reciprocal comes from the host: a chain of integer
    // divisions here, a hundred cycles each, stood between the positions and the first page request)
    const int span = p.max_blocks << p.log2_P;              // positions the block table can describe
    auto pages_of = [&](int position, int* first) {
        if (position < 0) {                                 // no key is visible from before the first one
            if (first) *first = 0;
            return 0;
        }
        position = min(position, span - 1);
        int from = p.window > 0 ? max(0, position - p.window + 1) : 0;
        if (p.chunk > 0) from = max(from, position - position % p.chunk);
        if (first) *first = from >> p.log2_P;
        return (position >> p.log2_P) - (from >> p.log2_P) + 1;
    };
    // every warp adds up the pages of all tokens for itself (a load per lane and five shuffles for up to 32 tokens):
    // no barrier and no shared memory stand between the positions and the first page request
    int total_pages = 0;
    if (p.deal) {
        for (int i = lane; i < p.n_tokens; i += 32) total_pages += pages_of(p.tok_pos[i], nullptr);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) total_pages += __shfl_xor_sync(0xffffffffu, total_pages, o);
    }
    int lo = p.window > 0 ? max(0, pos - p.window + 1) : 0;
    if (p.chunk > 0) lo = max(lo, pos - pos % p.chunk);
    int first_page = 0;
    const int my_pages = pages_of(pos, &first_page);
    const int last_page = first_page + my_pages - 1;
    // A position beyond the table: its own key has no page (to be written to, where it comes with the step), nor have the
    // other visible keys from the table's end on. The keys that have pages are attended to.
    if (warp == p.G && split == 0 && lane == 0 && pos >= span)
        atomicOr(p.error_flag, (p.k_new != nullptr ? 2 : 4) | (pos > max(lo, span) ? 4 : 0));
    // pages a block should take: all pages x groups over the blocks that can be resident (every block of a token does
    // the same arithmetic on the same numbers, so they agree whatever the rounding)
    int n_splits = gridDim.z;               // few tokens: every token may have all the splits, the blocks fit anyway
    if (p.deal) {
        const float share = fmaxf(1.f, ceilf((float)total_pages * (float)gridDim.y * p.inv_block_budget));
        n_splits = max(1, (int)(((float)my_pages + 0.5f * share) / share));
        n_splits = min(n_splits, (int)gridDim.z);
        if (split >= n_splits) return;
    }
    const int per = (my_pages + n_splits - 1) / n_splits;                // pages per split, rounded up
    const int page0 = first_page + split * per;
    const int n_mine = max(0, min(last_page + 1, page0 + per) - page0);

    if (warp == p.G) {
        // ---- the page warp: looks up and requests ----
        // With k_new/v_new given the pages hold earlier steps' keys and values only (this step's own row is patched in
        // below), so they are requested while the projection that produces the queries is still running.
        // Without them the step's row is in the cache already, written by some kernel of this step: then the wait comes first.
        if (p.k_new == nullptr) dd_grid_wait();
        bool ok = true;
        int s = 0, phase = 1;                               // the first round of the ring finds its stages free
#pragma unroll 1
        for (int i0 = 0; i0 < n_mine && ok; i0 += 32) {
            const int blk = page0 + i0 + lane;
            int page = -1;
            if (short_table) {
                const int low = __shfl_sync(0xffffffffu, held[0], blk & 31), high = __shfl_sync(0xffffffffu, held[1], blk & 31);
                page = blk < 32 ? low : (blk < p.max_blocks ? high : -1);
            } else if (i0 + lane < n_mine && blk < p.max_blocks) page = bt[blk];
            if (i0 + lane < n_mine && (page < 0 || page >= p.n_pages)) {
                // (the step's own key finds no place to be written to, and the page's other keys cannot be read)
                const bool own = p.k_new != nullptr && blk == pos >> p.log2_P;
                atomicOr(p.error_flag, own ? 2 | (pos > max(lo, blk << p.log2_P) ? 4 : 0) : 4);
                page = -1;
            }
#pragma unroll 1
            for (int i = i0; i < min(n_mine, i0 + 32) && ok; ++i) {
                const int id = __shfl_sync(0xffffffffu, page, i - i0);
                if (lane == 0) {
                    ok = tc::mbar_wait(&empty[s], phase, &abort_flag);
                    if (ok) {
                        stage_page[s] = id;
                        if (id < 0) tc::mbar_arrive(&full[s]);                  // a missing page (error bit set): nothing to wait for
                        else {
                            uint8_t* dst = tiles + (size_t)s * 2 * box_bytes;
                            tc::mbar_expect_tx(&full[s], 2 * group_heads * p.P * 128);
                            tc::tma_load_2d(dst, map, 0, ((id * 2 + 0) * p.H + head0) * p.P, &full[s]);
                            tc::tma_load_2d(dst + box_bytes, map, 0, ((id * 2 + 1) * p.H + head0) * p.P, &full[s]);
                        }
                    }
                }
                ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
                if (++s == p.stages) { s = 0; phase ^= 1; }
            }
        }
        if (!ok && lane == 0) atomicOr(p.error_flag, 8);
        return;
    }
    if (warp >= group_heads) return;

    // ---- a warp owns a head of the group ----
    dd_grid_wait();              // the queries and this step's keys and values are the kernel before this one's work
    const int h = head0 + warp;
    // the query as the B operand, the same in every column
    uint32_t qf[D / 16][2];
    float m = -CUDART_INF_F, l = 0.f, o[D / 16][2];         // o: dimensions 16 j + quad and 16 j + 8 + quad, in every lane of the quad
    {
        const __nv_bfloat16* qp = p.q + (size_t)t * p.q_stride + (size_t)h * D;
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
            qf[ks][0] = *reinterpret_cast<const uint32_t*>(qp + ks * 16 + 2 * t4);
            qf[ks][1] = *reinterpret_cast<const uint32_t*>(qp + ks * 16 + 8 + 2 * t4);
            o[ks][0] = o[ks][1] = 0.f;
        }
    }

    const size_t head_plane = (size_t)p.P * D, page_stride = 2 * (size_t)p.H * head_plane;
    bool ok = true;
    int s = 0, phase = 0;
#pragma unroll 1
    for (int i = 0; i < n_mine; ++i) {
        ok = __all_sync(0xffffffffu, tc::mbar_wait(&full[s], phase, &abort_flag));
        if (!ok) break;
        const int page = stage_page[s];
        const int key0 = (page0 + i) * p.P;                 // first key of the page
        uint8_t* kh = tiles + (size_t)s * 2 * box_bytes + (size_t)warp * p.P * 128;
        uint8_t* vh = kh + box_bytes;
        if (page >= 0) {
            if (key0 + p.P > pos) {
                // the page of the token's own position: its new key and value, and zeros for the unwritten slots
                const int slot = pos - key0;
                if (p.k_new != nullptr && lane < 16) {
                    const int c = lane & 7;
                    const __nv_bfloat16* src = (lane < 8 ? p.k_new : p.v_new) + (size_t)t * p.q_stride + (size_t)h * D + c * 8;
                    const uint4 v = *reinterpret_cast<const uint4*>(src);
                    *reinterpret_cast<uint4*>((lane < 8 ? kh : vh) + tile_off(slot, c)) = v;
                    __nv_bfloat16* dst = p.cache + (size_t)page * page_stride + (size_t)h * head_plane + (size_t)slot * D + c * 8;
                    *reinterpret_cast<uint4*>(lane < 8 ? dst : dst + (size_t)p.H * head_plane) = v;
                }
                for (int r = slot + 1 + (lane >> 3); r < p.P; r += 4)
                    *reinterpret_cast<uint4*>(vh + tile_off(r, lane & 7)) = make_uint4(0, 0, 0, 0);
                tc::fence_proxy_async();                    // (the token's last page: no later request writes over it, as it stands)
                __syncwarp();
            }
#pragma unroll 1
            for (int tt = 0; tt < p.P / TILE; ++tt) {
                const int base = key0 + tt * TILE;
                if (base > pos || base + TILE <= lo) continue;          // no live key in this tile
                const uint8_t* kt = kh + tt * TILE * 128;
                const uint8_t* vt = vh + tt * TILE * 128;
                // scores of 16 keys (the rows of A), in two independent parts: keys quad and quad + 8 in each lane of the quad
                float part[2][2];
                const int mi = lane >> 3;
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks) {
                    uint32_t a[4];
                    ldmatrix_x4(smem_addr(kt + tile_off((mi & 1) * 8 + (lane & 7), 2 * ks + (mi >> 1))), a);
                    float* c = part[ks & 1];
                    if (ks < 2) c[0] = c[1] = 0.f;
                    mma_bf16_column(c[0], c[1], a, qf[ks][0], qf[ks][1]);
                }
                const int key = base + quad;
                const float s0 = key <= pos && key >= lo ? (part[0][0] + part[1][0]) * p.scale_log2e : -CUDART_INF_F;
                const float s1 = key + 8 <= pos && key + 8 >= lo ? (part[0][1] + part[1][1]) * p.scale_log2e : -CUDART_INF_F;
                float mx = fmaxf(s0, s1);
#pragma unroll
                for (int x = 4; x < 32; x <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
                const float m_new = fmaxf(m, mx);               // the tile holds at least one live key
                const float corr = exp2f(m - m_new);
                m = m_new;
                const float p0 = exp2f(s0 - m_new), p1 = exp2f(s1 - m_new);
                l = l * corr + (p0 + p1);
                // the weights as the B operand: a lane gets keys 2 t4, 2 t4 + 1 and the same + 8 from the quads that hold them
                const uint32_t mine = pack_bf16(p0, p1);
                const uint32_t even = __shfl_sync(0xffffffffu, mine, 8 * t4), odd = __shfl_sync(0xffffffffu, mine, 8 * t4 + 4);
                const uint32_t w0 = __byte_perm(even, odd, 0x5410), w1 = __byte_perm(even, odd, 0x7632);
#pragma unroll
                for (int j = 0; j < D / 16; ++j) {
                    uint32_t a[4];
                    ldmatrix_x4_trans(smem_addr(vt + tile_off((mi >> 1) * 8 + (lane & 7), 2 * j + (mi & 1))), a);
                    o[j][0] *= corr;
                    o[j][1] *= corr;
                    mma_bf16_column(o[j][0], o[j][1], a, w0, w1);
                }
            }
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&empty[s]);          // this warp is done with the stage
        if (++s == p.stages) { s = 0; phase ^= 1; }
    }
    if (!ok && lane == 0) atomicOr(p.error_flag, 8);

    // every lane of a quad holds the same: lane t4 stores dimensions 16 t4 + quad and 16 t4 + 8 + quad
#pragma unroll
    for (int x = 4; x < 32; x <<= 1) l += __shfl_xor_sync(0xffffffffu, l, x);
    const int d = 16 * t4 + quad;
    const float o0 = t4 == 0 ? o[0][0] : (t4 == 1 ? o[1][0] : (t4 == 2 ? o[2][0] : o[3][0]));
    const float o1 = t4 == 0 ? o[0][1] : (t4 == 1 ? o[1][1] : (t4 == 2 ? o[2][1] : o[3][1]));
    if (n_splits == 1) {
        float inv = l != 0.f ? 1.f / l : 0.f;
        if (p.gate) inv *= 1.0f / (1.0f + __expf(-__bfloat162float(p.gate[(size_t)t * p.gate_stride + h])));
        __nv_bfloat16* dst = p.out + (size_t)t * p.out_stride + (size_t)h * D + d;
        dst[0] = __float2bfloat16_rn(o0 * inv);
        dst[8] = __float2bfloat16_rn(o1 * inv);
        return;
    }
    const size_t first = ((size_t)t * p.H + h) * gridDim.z;     // the scratch is laid out for the most splits
    {
        float* dst = p.part_o + (first + split) * D + d;
        dst[0] = o0;
        dst[8] = o1;
        if (lane == 0) *reinterpret_cast<float2*>(p.part_ml + 2 * (first + split)) = make_float2(m, l);
        __threadfence();
    }
    __syncwarp();
    int last = 0;
    if (lane == 0) last = atomicAdd(&p.counters[t * p.H + h], 1) == n_splits - 1;
    if (!__shfl_sync(0xffffffffu, last, 0)) return;
    __threadfence();
    // The warp that finished last merges the head: a lane per two output dimensions, the partial maxima and sums of eight
    // splits in eight lanes, everything of eight splits requested together and merged with a running maximum.
    float Mx = -CUDART_INF_F, Lx = 0.f, a0 = 0.f, a1 = 0.f;
    for (int sp0 = 0; sp0 < n_splits; sp0 += 8) {
        const int mine = sp0 + (lane & 7);
        float2 ml = make_float2(-CUDART_INF_F, 0.f), oo[8];
        if (mine < n_splits) ml = __ldcg(reinterpret_cast<const float2*>(p.part_ml + 2 * (first + mine)));
#pragma unroll
        for (int u = 0; u < 8; ++u)
            oo[u] = sp0 + u < n_splits ? __ldcg(reinterpret_cast<const float2*>(p.part_o + (first + sp0 + u) * D) + lane) : make_float2(0.f, 0.f);
        // a split without a live key has the sum 0 and adds nothing, whatever its scratch holds; a NaN sum goes on to the result
        const bool live = ml.y != 0.f;
        float cm = live ? ml.x : -CUDART_INF_F;
#pragma unroll
        for (int x = 4; x > 0; x >>= 1) cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, x));
        cm = fmaxf(cm, Mx);
        if (!__any_sync(0xffffffffu, live)) continue;
        const float keep = Mx == -CUDART_INF_F ? 0.f : exp2f(Mx - cm);
        Mx = cm;
        const float w = live ? exp2f(ml.x - Mx) : 0.f;
        float sum = live ? ml.y * w : 0.f;
#pragma unroll
        for (int x = 4; x > 0; x >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
        Lx = Lx * keep + sum;
        a0 *= keep;
        a1 *= keep;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const float wu = __shfl_sync(0xffffffffu, w, u);
            if (wu != 0.f) {
                a0 += oo[u].x * wu;
                a1 += oo[u].y * wu;
            }
        }
    }
    const float gated = p.gate ? 1.0f / (1.0f + __expf(-__bfloat162float(p.gate[(size_t)t * p.gate_stride + h]))) : 1.0f;
    const float inv = Lx != 0.f ? gated / Lx : 0.f;
    *reinterpret_cast<uint32_t*>(p.out + (size_t)t * p.out_stride + (size_t)h * D + 2 * lane) = pack_bf16(a0 * inv, a1 * inv);
    if (lane == 0) p.counters[t * p.H + h] = 0;
}

typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_fn() {
    static EncodeTiled fn = nullptr;
    if (!fn) {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiled>(sym);
    }
    return fn;
}

// Heads per block, spread evenly over the groups: up to seven (a warp each, 256 box rows at most), since the fewer and
// larger the boxes the better they stream (64 tokens x 25 heads: a step of 195 ms in groups of 7, 214 in groups of 5); up to
// eight for 31 and 32 heads, four groups of them instead of five full ones of seven (us a layer of a whole step, seven / eight:
// 32 tokens at 540 keys 82.4 / 74.8, 64 at 900 146.6 / 129.5, 64 at 16 to 768 keys 94.4 / 96.0). Where groups of seven leave
// places free, they stay: three groups of six and not two of eight for 16 heads, since three smaller blocks share an SM (64
// at 16 to 768 keys 54.6 / 58.4, at 900 73.6 / 72.1; 24 heads 67.9 / 71.3, at 900 92.9 / 100.9); and one of six or more groups
// saved brings nothing (40 heads, 32 tokens at 900 keys 131.0 / 134.4);
// up to four while a step has so few tokens that its blocks, in eight splits, stay below 1.35 an SM: then it is the
// chain of a block's pages that counts (1 token x 16 heads: 0.5 to 2 % of a whole step, 5 tokens 2 %).
void grouping(int n_tokens, int n_heads, int page_size, int sm_count, int* group, int* n_groups) {
    int most = MAX_GROUP < 256 / page_size ? MAX_GROUP : 256 / page_size;
    const int sevens = dd_ceil_div(n_heads, 7);
    if (most > 7 && (sevens > 5 || dd_ceil_div(n_heads, sevens) < 7)) most = 7;
    if (most > 4 && (long long)n_tokens * dd_ceil_div(n_heads, 4) * 8 * 20 <= 27ll * sm_count) most = 4;
    *n_groups = dd_ceil_div(n_heads, most);
    *group = dd_ceil_div(n_heads, *n_groups);
}
}  // namespace

// 1 if dd_attention_decode_pages takes the problem.
DD_API int dd_attention_decode_pages_supported(int n_heads, int n_kv_heads, int head_dim, int page_size, int dtype) {
    return dtype == DD_BF16 && n_heads == n_kv_heads && n_heads > 0 && head_dim == D &&
           (page_size == 16 || page_size == 32 || page_size == 64 || page_size == 128);
}

// The most key splits a token of dd_attention_decode_pages may need when the longest context is `context` keys (the
// kernel's n_splits argument: the grid is laid out for it; how many splits each token really gets the kernel decides
// from all tokens' positions). At most eight, which merge in one trip to L2 (measured at 8 tokens x 25 heads x 768
// keys: 8 splits, all blocks resident, 13 us; a second wave of blocks 18 us).
DD_API int dd_attention_decode_pages_splits(int n_tokens, int n_heads, int page_size, int context, int sm_count) {
    int group = 0, n_groups = 0;
    grouping(n_tokens < 1 ? 1 : n_tokens, n_heads, page_size, sm_count, &group, &n_groups);
    const int pages = dd_ceil_div(context < 1 ? 1 : context, page_size);
    // A token gets pages / (all pages x groups / resident blocks) splits: with equal contexts that is resident blocks
    // / (tokens x groups); a token 2.5 times as long as the average gets 2.5 times as many, and the grid allows for
    // that much. More would only add blocks that leave at once, and while those wait for a place the next kernel
    // cannot start its prologue (64 tokens, 8 splits allowed, 1 taken: 58 us against 56).
    int splits = dd_ceil_div(5ll * 2 * sm_count, 2ll * (n_tokens < 1 ? 1 : n_tokens) * n_groups);
    // at most eight, which merge in one trip to L2, unless the context is so long that more splits still leave a block 16
    // pages (one token of 16,384 keys x 25 heads: 118 us in 8 splits, 32 blocks in all)
    const int most = pages / 16 > 8 ? pages / 16 : 8;
    if (splits > most) splits = most;
    if (splits > pages) splits = pages;
    return splits < 1 ? 1 : splits;
}

// The arguments of dd_attention_decode (attention_decode.cu).
DD_API int dd_attention_decode_pages(const void* q, int q_stride, const void* k_new, const void* v_new, void* cache,
                                     const int* tok_entry, const int* tok_pos, const int* block_table, int max_blocks,
                                     void* out, int out_stride, float* part_o, float* part_ml, int* counters, int n_tokens,
                                     int n_heads, int n_kv_heads, int head_dim, int page_size, int n_pages, int window,
                                     float scale, int n_splits, int* error_flag, void* stream, int chunk, const void* gate,
                                     int gate_stride) {
    if (n_tokens <= 0) return 0;
    if (!dd_attention_decode_pages_supported(n_heads, n_kv_heads, head_dim, page_size, DD_BF16))
        return dd_fail("dd_attention_decode_pages: needs heads == key/value heads, head size 64 and pages of 16, 32, 64 or 128 "
                       "tokens (got %d, %d, %d, %d)", n_heads, n_kv_heads, head_dim, page_size);
    if (n_splits < 1 || n_splits > 65535 || (n_splits > 1 && (!part_o || !part_ml || !counters)))
        return dd_fail("dd_attention_decode_pages: n_splits=%d needs scratch and counters", n_splits);
    if (q_stride % 8 || out_stride % 8 || ((uintptr_t)q & 15) || ((uintptr_t)cache & 15) || ((uintptr_t)out & 3))
        return dd_fail("dd_attention_decode_pages: rows must be 16-byte aligned");
    if (n_tokens > 65535) return dd_fail("dd_attention_decode_pages: too many tokens");
    if ((k_new == nullptr) != (v_new == nullptr) || ((uintptr_t)k_new & 15) || ((uintptr_t)v_new & 15))
        return dd_fail("dd_attention_decode_pages: k_new and v_new come together, 16-byte aligned");
    EncodeTiled enc = encode_fn();
    if (!enc) return dd_fail("dd_attention_decode_pages: cuTensorMapEncodeTiled is not available from this driver");
    Params p;
    static int sm_count = 0;
    if (!sm_count) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev);
        if (sm_count <= 0) sm_count = 148;
    }
    int n_groups = 0;
    grouping(n_tokens, n_heads, page_size, sm_count, &p.G, &n_groups);
    const int box_bytes = p.G * page_size * 128;
    // Stages for two blocks an SM, and the splits are dealt out for two, also where the groups are so small that three of
    // MAX_STAGES fit (up to six heads of 16 tokens): a budget of three has not been measured.
    p.stages = (106 * 1024) / (2 * box_bytes);
    int blocks_per_sm = 2;
    if (p.stages < 2) {                                               // large pages: one block per SM
        p.stages = (210 * 1024) / (2 * box_bytes);
        blocks_per_sm = 1;
    }
    p.inv_block_budget = 1.0f / (float)(blocks_per_sm * sm_count);
    p.deal = (long long)n_tokens * n_groups * n_splits > (long long)blocks_per_sm * sm_count;
    p.log2_P = page_size == 16 ? 4 : (page_size == 32 ? 5 : (page_size == 64 ? 6 : 7));
    if (p.stages > MAX_STAGES) p.stages = MAX_STAGES;
    if (p.stages < 2) return dd_fail("dd_attention_decode_pages: a page of %d heads x %d tokens does not fit twice into shared memory", p.G, page_size);
    const int smem = p.stages * 2 * box_bytes + 1024 + MAX_STAGES * (2 * 8 + 4);
    static int configured = 0;
    if (configured < smem) {
        cudaError_t e = cudaFuncSetAttribute(attention_decode_pages_kernel<7>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(attention_decode_pages_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return dd_fail("dd_attention_decode_pages: shared memory of %d bytes refused: %s", smem, cudaGetErrorString(e));
        configured = smem;
    }
    CUtensorMap maps[2];
    cuuint64_t dims[2] = {(cuuint64_t)D, (cuuint64_t)n_pages * 2 * n_heads * page_size};
    cuuint64_t strides[1] = {(cuuint64_t)D * 2};
    cuuint32_t elem[2] = {1, 1};
    for (int i = 0; i < 2; ++i) {
        // the last group may hold fewer heads: a box of its own reads no neighbour's rows (25 heads in groups of 7: 28 were read)
        cuuint32_t box[2] = {(cuuint32_t)D, (cuuint32_t)((i ? n_heads - (n_groups - 1) * p.G : p.G) * page_size)};
        CUresult r = enc(&maps[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, cache, dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return dd_fail("dd_attention_decode_pages: cannot describe the cache to TMA (driver error %d)", (int)r);
    }
    p.q = (const __nv_bfloat16*)q; p.k_new = (const __nv_bfloat16*)k_new; p.v_new = (const __nv_bfloat16*)v_new;
    p.cache = (__nv_bfloat16*)cache; p.tok_entry = tok_entry; p.tok_pos = tok_pos; p.block_table = block_table;
    p.out = (__nv_bfloat16*)out; p.part_o = part_o; p.part_ml = part_ml; p.counters = counters; p.error_flag = error_flag;
    p.q_stride = q_stride; p.out_stride = out_stride; p.max_blocks = max_blocks; p.H = n_heads; p.P = page_size;
    p.n_pages = n_pages; p.window = window; p.chunk = chunk; p.gate = (const __nv_bfloat16*)gate; p.gate_stride = gate_stride;
    p.scale_log2e = scale * 1.4426950408889634f;
    p.n_tokens = n_tokens;
    const dim3 grid(n_tokens, n_groups, n_splits), block((p.G + 1) * 32);
    cudaStream_t s = (cudaStream_t)stream;
    if (p.G < 8) dd_launch(attention_decode_pages_kernel<7>, dim3(grid), dim3(block), (size_t)smem, s, maps[0], maps[1], p);
    else dd_launch(attention_decode_pages_kernel<8>, dim3(grid), dim3(block), (size_t)smem, s, maps[0], maps[1], p);
    return dd_check_launch("dd_attention_decode_pages");
}
