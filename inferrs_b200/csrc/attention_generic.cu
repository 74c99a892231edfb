// Grouped-query attention over the paged cache, for any head size: 32-bit arithmetic
// throughout.  Two kernels: one warp per (token, query head) for everything, and for
// 32-bit activations whose heads hold a multiple of four numbers, 128 at most, one
// CTA per tile of tokens and key/value head (below).
//
// A token at position `pos` of its request sees the keys lo..pos of that request,
// lo = 0, pos - window + 1, or (window < 0) the first position of pos's chunk of -window positions.  Values may
// have another size than keys.  This step's keys are already in the cache when the
// kernel runs, so a prompt portion and a decoded token are the same case.  Keys are
// taken 32 at a time in ascending order from a multiple of 32, with an online
// softmax; the order of every sum depends only on (pos, window), never on what else
// is in the batch or on which pages hold the keys.
//
// This is the kernel of the true 32-bit path and the fallback of the bfloat16 path
// for head sizes that its tensor-core kernels do not take.
//
// Two options serve attention whose heads' scores are mixed before the softmax and penalised by distance.
// JOINT: a query head holds one vector per key/value head, side by side (n_kv_heads * head_dim numbers), and its
// score against a token is the sum of its products with all of the token's key heads; values are still those
// of the head's own group.  dist_bias [n_heads, bias_len]: dist_bias[h, pos - j] is taken off head h's score
// against key j (a distance beyond the table reads its last entry).
//
// Three more options, each a number per head (absent: not applied).  head_scale[h] multiplies head h's scaled score
// (a learned temperature).  slopes[h] * (pos - j) is taken off the score (a bias that grows linearly with the
// distance).  sinks[h]: every row's softmax gets one more term, exp(sinks[h]), in its denominator only; no key or
// value belongs to it, and neither the scale nor the factor nor the slope touches it.  The other options (a cap on the
// scores, a sequence's first keys beside the window, a gate per head) are those of IbScoreOptions.
#include "common.cuh"

#define ATT_WARPS 4

template <int DPL, bool JOINT>  // DPL value elements per lane: v_dim <= 32 * DPL
__global__ void paged_attention_generic_kernel(
    const act_t* __restrict__ q, const act_t* __restrict__ k_pages, const act_t* __restrict__ v_pages,
    const int* __restrict__ block_table, int max_pages, int page_size, int n_pages,
    const int* __restrict__ row_request, const int* __restrict__ positions, int n_heads, int n_kv_heads,
    int head_dim, int v_dim, float scale, int window, act_t* __restrict__ out,
    const float* __restrict__ dist_bias, int bias_len, const IbScoreOptions opt) {
    extern __shared__ float smem[];
    ib_grid_dependency_sync();
    const int row = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int head = blockIdx.y * ATT_WARPS + warp;
    if (head >= n_heads) return;  // whole warps leave; only warp-level syncs follow
    const int d = head_dim;
    const int dq = JOINT ? n_kv_heads * d : d;      // numbers of a query head
    float* qs = smem + warp * dq;
    const int pos = positions[row];
    const int req = row_request[row];
    const int lo = ib_first_visible(pos, window);
    const int kvh = head / (n_heads / n_kv_heads);
    const int* bt = block_table + (long)req * max_pages;

    const act_t* qr = q + ((long)row * n_heads + head) * dq;
    for (int e = lane; e < dq; e += 32) qs[e] = ib_to_float(qr[e]);
    const float* bias_h = dist_bias ? dist_bias + (long)head * bias_len : nullptr;
    const float scale_h = opt.head_scale ? scale * opt.head_scale[head] : scale;
    const float slope_h = opt.slopes ? opt.slopes[head] : 0.0f;
    __syncwarp();

    float acc[DPL];
#pragma unroll
    for (int k = 0; k < DPL; ++k) acc[k] = 0.0f;
    float m = -INFINITY, l = 0.0f;

    const int n_kept = ib_kept_tiles(opt.keep_first, lo / 32, 32);
    for (int i = 0; ; ++i) {
        const int j0 = ib_nth_tile(i, n_kept, lo / 32) * 32;
        if (j0 > pos) break;
        const int j = j0 + lane;
        const bool valid = ib_visible(j, lo, pos, opt.keep_first);
        float s = -INFINITY;
        long off = 0;      // the key's place counted in heads' rows; times d its key, times v_dim its value
        if (valid) {
            const int page = bt[j / page_size];
            if (page >= 0 && page < n_pages) {
                off = ((long)page * n_kv_heads + kvh) * page_size + (j % page_size);
                float dot = 0.0f;
                if (JOINT) {
                    for (int c = 0; c < n_kv_heads; ++c) {
                        const act_t* kr = k_pages + (((long)page * n_kv_heads + c) * page_size + (j % page_size)) * d;
                        const float* qc = qs + c * d;
                        for (int e = 0; e < d; ++e) dot = fmaf(qc[e], ib_to_float(kr[e]), dot);
                    }
                } else {
                    const act_t* kr = k_pages + off * d;
                    for (int e = 0; e < d; ++e) dot = fmaf(qs[e], ib_to_float(kr[e]), dot);
                }
                s = dot * scale_h - slope_h * (float)(pos - j);
                if (bias_h) s -= bias_h[pos - j < bias_len ? pos - j : bias_len - 1];
                if (opt.cap > 0.0f) s = opt.cap * tanhf(s / opt.cap);
            }
        }
        const float m_new = fmaxf(m, ib_warp_max(s));
        const float p = (s == -INFINITY) ? 0.0f : expf(s - m_new);
        const float corr = (m == -INFINITY) ? 0.0f : expf(m - m_new);
        l = l * corr + ib_warp_sum(p);
#pragma unroll
        for (int k = 0; k < DPL; ++k) acc[k] *= corr;
        const int n_in_chunk = (pos - j0 + 1 < 32) ? pos - j0 + 1 : 32;
        for (int jj = 0; jj < n_in_chunk; ++jj) {
            const float pj = __shfl_sync(0xffffffffu, p, jj);
            const long voff = __shfl_sync(0xffffffffu, off, jj);
            if (pj == 0.0f) continue;  // masked key (uniform over the warp)
            const act_t* vr = v_pages + voff * v_dim;
#pragma unroll
            for (int k = 0; k < DPL; ++k) {
                const int e = lane + 32 * k;
                if (e < v_dim) acc[k] = fmaf(pj, ib_to_float(vr[e]), acc[k]);
            }
        }
        m = m_new;
    }
    if (opt.sinks) {        // the place without a key: it adds to the denominator and to nothing else
        const float sink = opt.sinks[head];
        const float m_new = fmaxf(m, sink);
        const float corr = (m == -INFINITY) ? 0.0f : expf(m - m_new);
        l = l * corr + expf(sink - m_new);
#pragma unroll
        for (int k = 0; k < DPL; ++k) acc[k] *= corr;
    }
    const float inv = (l > 0.0f ? 1.0f / l : 0.0f) * ib_head_gate(opt, row, head);
    act_t* dst = out + row * opt.out_ld + (long)head * v_dim;
#pragma unroll
    for (int k = 0; k < DPL; ++k) {
        const int e = lane + 32 * k;
        if (e < v_dim) dst[e] = ib_from_float<act_t>(acc[k] * inv);
    }
}

// ---- tiles of tokens against tiles of keys, 32-bit activations -----------------------------------------------------
// A CTA takes the query heads of one key/value head for a few tokens that follow one another in the step; 32 keys and
// values at a time come into shared memory by cp.async, the next ones while these are worked on, and serve all of the
// CTA's queries.  (One warp per token and head read every key once per query head, each lane a key of its own, 4 bytes at
// a time: 32 sectors a load.)  A warp owns QPW queries from the scores to the output: a lane has one key for the scores
// and the softmax, four value numbers for the output, so nothing is exchanged between warps.
// Tokens of several requests may meet in a tile: each run of one request's tokens is walked by itself.
// A row's sums: four partial sums per score (numbers 0, 4, 8, ... of the head, 1, 5, 9, ... and so on), keys in ascending
// tiles of 32 from a multiple of 32; a tile of which a row sees nothing leaves its sums as they are.  They depend on
// the row's position and options only, as above.
#if !IB_ACT_BF16
namespace gat {

constexpr int KEYS = 32, PLD = KEYS + 4, MAX_DIM = 128;

__device__ __forceinline__ void copy16(float* dst, const float* src, bool there) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(there ? 16 : 0) : "memory");
}

static size_t smem_bytes(int warps, int qpw, int d, int dv) {
    return sizeof(float) * (2 * KEYS * (d + 4 + dv) + warps * qpw * (d + PLD));
}

template <int WARPS, int QPW>
__global__ void __launch_bounds__(32 * WARPS, 1) tile_kernel(
    const float* __restrict__ q, const float* __restrict__ k_pages, const float* __restrict__ v_pages,
    const int* __restrict__ block_table, int max_pages, int page_size, int n_pages, const int* __restrict__ row_request,
    const int* __restrict__ positions, int n_rows, int tokens, int n_heads, int n_kv_heads, int d, int dv, float scale,
    int window, float* __restrict__ out, const IbScoreOptions opt) {
    extern __shared__ __align__(16) float smem[];
    __shared__ int s_req[WARPS * QPW], s_pos[WARPS * QPW], q_pos[WARPS * QPW], q_lo[WARPS * QPW];
    __shared__ float q_scale[WARPS * QPW], q_slope[WARPS * QPW], q_m[WARPS * QPW], q_l[WARPS * QPW], q_corr[WARPS * QPW];
    const int group = n_heads / n_kv_heads, kvh = blockIdx.y;
    const int kld = d + 4, row0 = blockIdx.x * tokens;
    const int rows = n_rows - row0 < tokens ? n_rows - row0 : tokens;
    float* ks = smem;                                   // [2][KEYS][d + 4]
    float* vs = ks + 2 * KEYS * kld;                    // [2][KEYS][dv]
    float* qs = vs + 2 * KEYS * dv;                     // [queries][d]
    float* ps = qs + WARPS * QPW * d;                   // [queries][PLD]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
    ib_grid_dependency_sync();
    if (tid < rows) {
        s_req[tid] = row_request[row0 + tid];
        s_pos[tid] = positions[row0 + tid];
    }
    for (int m = warp; m < rows * group; m += WARPS) {
        const float* src = q + ((long)(row0 + m / group) * n_heads + kvh * group + m % group) * d;
        for (int e = lane; e < d; e += 32) qs[m * d + e] = src[e];
    }
    __syncthreads();

    for (int a = 0, b; a < rows; a = b) {               // tokens a .. b - 1 of the tile: one request's
        const int req = s_req[a];
        int lo_min = ib_first_visible(s_pos[a], window), pos_max = s_pos[a];
        for (b = a + 1; b < rows && s_req[b] == req; ++b) {
            const int lo = ib_first_visible(s_pos[b], window);
            lo_min = lo < lo_min ? lo : lo_min;
            pos_max = s_pos[b] > pos_max ? s_pos[b] : pos_max;
        }
        const int* bt = block_table + (long)req * max_pages;
        const int t_first = lo_min / KEYS, n_kept = ib_kept_tiles(opt.keep_first, t_first, KEYS);
        const int n_tiles = n_kept + (pos_max >= 0 ? pos_max / KEYS : -1) + 1 - t_first;
        auto place = [&](int j) -> long {               // of key j of this request, counted in heads' rows; -1: nowhere
            if (j > pos_max) return -1;
            const int page = bt[j / page_size];
            return page >= 0 && page < n_pages ? ((long)page * n_kv_heads + kvh) * page_size + j % page_size : -1;
        };
        auto fetch = [&](int i) {
            float* kd = ks + (i & 1) * KEYS * kld;
            float* vd = vs + (i & 1) * KEYS * dv;
            const int j0 = ib_nth_tile(i, n_kept, t_first) * KEYS;
            const long mine = place(j0 + lane);
#pragma unroll 1
            for (int j = warp; j < KEYS; j += WARPS) {
                const long at = __shfl_sync(0xffffffffu, mine, j);
                if (lane * 4 < d) copy16(kd + j * kld + lane * 4, at >= 0 ? k_pages + at * d + lane * 4 : k_pages, at >= 0);
                if (lane * 4 < dv) copy16(vd + j * dv + lane * 4, at >= 0 ? v_pages + at * dv + lane * 4 : v_pages, at >= 0);
            }
        };
        if (lane < QPW) {                               // the warp's own queries (a warp that has none of them: none)
            const int m = warp * QPW + lane, r = m / group, head = kvh * group + m % group;
            const bool mine = r >= a && r < b;
            q_pos[m] = mine ? s_pos[r] : -1;
            q_lo[m] = mine ? ib_first_visible(s_pos[r], window) : 0;
            q_scale[m] = mine && opt.head_scale ? scale * opt.head_scale[head] : scale;
            q_slope[m] = mine && opt.slopes ? opt.slopes[head] : 0.0f;
            q_m[m] = -INFINITY;
            q_l[m] = 0.0f;
        }
        __syncwarp();
        float acc[QPW][4];
        int last = -1;                                  // the furthest key that a query of this warp sees
#pragma unroll
        for (int c = 0; c < QPW; ++c) {
            acc[c][0] = acc[c][1] = acc[c][2] = acc[c][3] = 0.0f;
            last = q_pos[warp * QPW + c] > last ? q_pos[warp * QPW + c] : last;
        }
        if (n_tiles > 0) fetch(0);
        asm volatile("cp.async.commit_group;" ::: "memory");
        for (int i = 0; i < n_tiles; ++i) {
            if (i + 1 < n_tiles) fetch(i + 1);
            asm volatile("cp.async.commit_group;" ::: "memory");
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();
            const int j0 = ib_nth_tile(i, n_kept, t_first) * KEYS, j = j0 + lane;
            if (j0 <= last) {
                const float* kr = ks + ((i & 1) * KEYS + lane) * kld;
                const float* qr = qs + warp * QPW * d;
                float4 dot[QPW];
#pragma unroll
                for (int c = 0; c < QPW; ++c) dot[c] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
                for (int e = 0; e < d; e += 4) {
                    const float4 kv = *reinterpret_cast<const float4*>(kr + e);
#pragma unroll
                    for (int c = 0; c < QPW; ++c) {
                        const float4 qv = *reinterpret_cast<const float4*>(qr + c * d + e);
                        dot[c].x = fmaf(qv.x, kv.x, dot[c].x);
                        dot[c].y = fmaf(qv.y, kv.y, dot[c].y);
                        dot[c].z = fmaf(qv.z, kv.z, dot[c].z);
                        dot[c].w = fmaf(qv.w, kv.w, dot[c].w);
                    }
                }
                float* own = ps + warp * QPW * PLD + lane;
#pragma unroll
                for (int c = 0; c < QPW; ++c) own[c * PLD] = (dot[c].x + dot[c].y) + (dot[c].z + dot[c].w);
                const bool there = place(j) >= 0;
#pragma unroll 1
                for (int c = 0; c < QPW; ++c) {         // (a loop: unrolled four times it is more code than it saves)
                    const int m = warp * QPW + c, pos = q_pos[m];
                    float s = -INFINITY;
                    if (there && ib_visible(j, q_lo[m], pos, opt.keep_first)) {
                        s = own[c * PLD] * q_scale[m] - q_slope[m] * (float)(pos - j);
                        if (opt.cap > 0.0f) s = opt.cap * tanhf(s / opt.cap);
                    }
                    const float m_run = q_m[m], m_new = fmaxf(m_run, ib_warp_max(s));
                    const float p = (s == -INFINITY) ? 0.0f : expf(s - m_new);
                    const float corr = (m_run == -INFINITY) ? 0.0f : expf(m_run - m_new);
                    const float l = q_l[m] * corr + ib_warp_sum(p);
                    __syncwarp();
                    own[c * PLD] = p;
                    if (lane == 0) {
                        q_m[m] = m_new;
                        q_l[m] = l;
                        q_corr[m] = corr;
                    }
                }
                __syncwarp();
#pragma unroll
                for (int c = 0; c < QPW; ++c) {
                    const float corr = q_corr[warp * QPW + c];
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[c][e] *= corr;
                }
                if (lane * 4 < dv) {
                    const float* vr = vs + (i & 1) * KEYS * dv + lane * 4;
                    const float* pr = ps + warp * QPW * PLD;
#pragma unroll 1
                    for (int jj = 0; jj < KEYS; jj += 4) {
                        float4 vv[4];
#pragma unroll
                        for (int g = 0; g < 4; ++g) vv[g] = *reinterpret_cast<const float4*>(vr + (jj + g) * dv);
#pragma unroll
                        for (int c = 0; c < QPW; ++c) {
                            const float4 p4 = *reinterpret_cast<const float4*>(pr + c * PLD + jj);
                            const float p[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
                            for (int g = 0; g < 4; ++g) {
                                if (p[g] != 0.0f) {     // a masked key's value is not looked at
                                    acc[c][0] = fmaf(p[g], vv[g].x, acc[c][0]);
                                    acc[c][1] = fmaf(p[g], vv[g].y, acc[c][1]);
                                    acc[c][2] = fmaf(p[g], vv[g].z, acc[c][2]);
                                    acc[c][3] = fmaf(p[g], vv[g].w, acc[c][3]);
                                }
                            }
                        }
                    }
                }
            }
            __syncthreads();                            // this tile's buffer may be filled again
        }
        __syncwarp();
        float* own = ps + warp * QPW * PLD;             // 1 / denominator and the last correction, a lane per query
        if (lane < QPW) {
            const int m = warp * QPW + lane, r = m / group, head = kvh * group + m % group;
            float l = q_l[m], corr = 1.0f;
            if (r >= a && r < b) {
                if (opt.sinks) {                        // adds to the denominator and to nothing else
                    const float sink = opt.sinks[head], m_new = fmaxf(q_m[m], sink);
                    corr = (q_m[m] == -INFINITY) ? 0.0f : expf(q_m[m] - m_new);
                    l = l * corr + expf(sink - m_new);
                }
                own[lane] = (l > 0.0f ? 1.0f / l : 0.0f) * ib_head_gate(opt, row0 + r, head);
            }
            own[QPW + lane] = corr;
        }
        __syncwarp();
#pragma unroll
        for (int c = 0; c < QPW; ++c) {
            const int m = warp * QPW + c, r = m / group, head = kvh * group + m % group;
            if (r < a || r >= b || lane * 4 >= dv) continue;
            float* dst = out + (row0 + r) * opt.out_ld + (long)head * dv + lane * 4;
#pragma unroll
            for (int e = 0; e < 4; ++e) dst[e] = acc[c][e] * own[QPW + c] * own[c];
        }
        __syncwarp();
    }
}

// One token and key/value head per CTA, up to G query heads: the same sums as above in the same order, laid out for a
// single token, whose chain of tiles is all there is to wait for.  Four tiles at a time and four warps per query head
// (four heads side by side at most, PER of them after one another): each warp takes the scores of one tile of 32 keys, the
// running maximum goes over the tiles in order, and a thread owns one value number of a head.  The next keys are on
// their way while values are summed, the next values during the scores.  Bound by the instructions of that chain.
template <int G>
__global__ void __launch_bounds__(128 * (G < 4 ? G : 4), 1) token_kernel(
    const float* __restrict__ q, const float* __restrict__ k_pages, const float* __restrict__ v_pages,
    const int* __restrict__ block_table, int max_pages, int page_size, int n_pages, const int* __restrict__ row_request,
    const int* __restrict__ positions, int n_heads, int n_kv_heads, int d, int dv, float scale, int window,
    float* __restrict__ out, const IbScoreOptions opt) {
    constexpr int SIDE = G < 4 ? G : 4, PER = G / SIDE, THREADS = 128 * SIDE;
    extern __shared__ __align__(16) float smem[];
    __shared__ float s_max[G][4], s_sum[G][4], s_corr[G][4], s_m[G], s_l[G];
    __shared__ __align__(16) float ps[G][4 * KEYS];
    const int group = n_heads / n_kv_heads, kvh = blockIdx.y, row = blockIdx.x;
    const int kld = d + 4, tid = threadIdx.x, lane = tid & 31, tile = (tid >> 5) & 3, c0 = (tid >> 7) * PER;
    float* ks = smem;                                   // [4 * KEYS][d + 4]
    float* vs = ks + 4 * KEYS * kld;                    // [4 * KEYS][dv]
    float* qs = vs + 4 * KEYS * dv;                     // [G][d]
    ib_grid_dependency_sync();
    const int pos = positions[row], req = row_request[row];
    const int* bt = block_table + (long)req * max_pages;
    const int lo = ib_first_visible(pos, window), t_first = lo / KEYS;
    const int n_kept = ib_kept_tiles(opt.keep_first, t_first, KEYS);
    const int n_tiles = n_kept + (pos >= 0 ? pos / KEYS : -1) + 1 - t_first;
    // the place of this lane's key in tile i, counted in heads' rows; -1: nowhere
    auto place = [&](int i) -> long {
        const int j = i < n_tiles ? ib_nth_tile(i, n_kept, t_first) * KEYS + lane : pos + 1;
        if (j > pos) return -1;
        const int page = bt[j / page_size];
        return page >= 0 && page < n_pages ? ((long)page * n_kv_heads + kvh) * page_size + j % page_size : -1;
    };
    auto fetch = [&](float* dst, int ld, const float* pages, int n, long at) {
        const float* mine = at >= 0 ? pages + at * n : nullptr;
        dst += tile * KEYS * ld + lane * 4;
#pragma unroll 2
        for (int j = tid >> 7; j < KEYS; j += SIDE) {   // the warps of a tile share its rows
            const float* src = reinterpret_cast<const float*>(__shfl_sync(0xffffffffu, (unsigned long long)mine, j));
            if (lane * 4 < n) copy16(dst + j * ld, src ? src + lane * 4 : pages, src != nullptr);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    long at = place(tile);
    fetch(ks, kld, k_pages, d, at);
    fetch(vs, dv, v_pages, dv, at);
    for (int e = tid; e < group * d; e += THREADS) qs[e] = q[((long)row * n_heads + kvh * group) * d + e];
    if (tid < G) {
        s_m[tid] = -INFINITY;
        s_l[tid] = 0.0f;
    }
    float acc[PER];
#pragma unroll
    for (int c = 0; c < PER; ++c) acc[c] = 0.0f;
    for (int i0 = 0; i0 < n_tiles; i0 += 4) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");            // the keys
        __syncthreads();
        const int j = ib_nth_tile(i0 + tile, n_kept, t_first) * KEYS + lane;
        const bool seen = at >= 0 && ib_visible(j, lo, pos, opt.keep_first);
        const float* kr = ks + (tile * KEYS + lane) * kld;
#pragma unroll 1
        for (int c = c0; c < c0 + PER && c < group; ++c) {
            const float* qr = qs + c * d;
            float4 dot = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
            for (int e = 0; e < d; e += 4) {
                const float4 kv = *reinterpret_cast<const float4*>(kr + e), qv = *reinterpret_cast<const float4*>(qr + e);
                dot.x = fmaf(qv.x, kv.x, dot.x);
                dot.y = fmaf(qv.y, kv.y, dot.y);
                dot.z = fmaf(qv.z, kv.z, dot.z);
                dot.w = fmaf(qv.w, kv.w, dot.w);
            }
            float s = -INFINITY;
            if (seen) {
                const int head = kvh * group + c;
                s = ((dot.x + dot.y) + (dot.z + dot.w)) * (opt.head_scale ? scale * opt.head_scale[head] : scale) -
                    (opt.slopes ? opt.slopes[head] : 0.0f) * (float)(pos - j);
                if (opt.cap > 0.0f) s = opt.cap * tanhf(s / opt.cap);
            }
            ps[c][tile * KEYS + lane] = s;
            const float top = ib_warp_max(s);
            if (lane == 0) s_max[c][tile] = top;
        }
        __syncthreads();                                                // everyone has left the keys
        at = place(i0 + 4 + tile);
        fetch(ks, kld, k_pages, d, at);
#pragma unroll 1
        for (int c = c0; c < c0 + PER && c < group; ++c) {
            float before = s_m[c];                                      // the maximum over the tiles before this one
            for (int t = 0; t < tile; ++t) before = fmaxf(before, s_max[c][t]);
            const float mine = fmaxf(before, s_max[c][tile]), s = ps[c][tile * KEYS + lane];
            if (lane == 0) s_corr[c][tile] = (before == -INFINITY) ? 0.0f : expf(before - mine);
            const float p = (s == -INFINITY) ? 0.0f : expf(s - mine), sum = ib_warp_sum(p);
            ps[c][tile * KEYS + lane] = p;
            if (lane == 0) s_sum[c][tile] = sum;
        }
        asm volatile("cp.async.wait_group 1;" ::: "memory");            // the values
        __syncthreads();                                                // ... and the probabilities
        if (tid < group) {                                              // (read again after the next round's barriers)
            float l = s_l[tid], m = s_m[tid];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                l = l * s_corr[tid][t] + s_sum[tid][t];
                m = fmaxf(m, s_max[tid][t]);
            }
            s_l[tid] = l;
            s_m[tid] = m;
        }
        const int e = tid & 127;
        if (e < dv) {
#pragma unroll 1
            for (int t = 0; t < 4; ++t) {
#pragma unroll
                for (int c = 0; c < PER; ++c) {
                    if (c0 + c >= group) continue;
                    acc[c] *= s_corr[c0 + c][t];
#pragma unroll 4
                    for (int jj = 0; jj < KEYS; jj += 4) {
                        const float4 p = *reinterpret_cast<const float4*>(&ps[c0 + c][t * KEYS + jj]);
                        const float* vr = vs + (t * KEYS + jj) * dv + e;
                        if (p.x != 0.0f) acc[c] = fmaf(p.x, vr[0], acc[c]);      // a masked key's value is not looked at
                        if (p.y != 0.0f) acc[c] = fmaf(p.y, vr[dv], acc[c]);
                        if (p.z != 0.0f) acc[c] = fmaf(p.z, vr[2 * dv], acc[c]);
                        if (p.w != 0.0f) acc[c] = fmaf(p.w, vr[3 * dv], acc[c]);
                    }
                }
            }
        }
        __syncthreads();                                                // everyone has left the values
        fetch(vs, dv, v_pages, dv, at);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int c = 0; c < PER; ++c) {
        if (c0 + c >= group) continue;
        const int head = kvh * group + c0 + c, e = tid & 127;
        float l = s_l[c0 + c], co = 1.0f;
        if (opt.sinks) {
            const float m = s_m[c0 + c], m_new = fmaxf(m, opt.sinks[head]);
            co = (m == -INFINITY) ? 0.0f : expf(m - m_new);
            l = l * co + expf(opt.sinks[head] - m_new);
        }
        const float inv = (l > 0.0f ? 1.0f / l : 0.0f) * ib_head_gate(opt, row, head);
        if (e < dv) out[row * opt.out_ld + (long)head * dv + e] = acc[c] * co * inv;
    }
}

static size_t token_smem_bytes(int g, int d, int dv) {
    return sizeof(float) * (4 * KEYS * (d + 4 + dv) + g * d);
}

}  // namespace gat
#endif

IB_EXPORT int ib_paged_attention_generic(const void* q, const void* k_pages, const void* v_pages,
                                         const int* block_table, int max_pages, int page_size, int n_pages,
                                         const int* row_request, const int* positions, int n_rows,
                                         int n_requests, int n_heads, int n_kv_heads, int head_dim, int v_dim, float scale, int window, void* out,
                                         int joint, const float* dist_bias, int bias_len, const float* head_scale,
                                         const float* slopes, const float* sinks, float cap, int keep_first,
                                         const void* gate, long gate_ld, long out_ld, cudaStream_t stream) {
    if (n_rows <= 0) return IB_OK;
    if (n_heads <= 0 || n_kv_heads <= 0 || n_heads % n_kv_heads || head_dim <= 0 || page_size <= 0 || max_pages <= 0)
        return IB_ERR_ARGUMENT;
    if (v_dim <= 0) return IB_ERR_ARGUMENT;
    if (dist_bias != nullptr && bias_len <= 0) return IB_ERR_ARGUMENT;
    if (keep_first < 0 || out_ld < (long)n_heads * v_dim || (gate != nullptr && gate_ld < n_heads)) return IB_ERR_ARGUMENT;
    const IbScoreOptions opt = {head_scale, slopes, sinks, cap, keep_first, (const act_t*)gate, gate_ld, out_ld};
    const int dq = joint ? n_kv_heads * head_dim : head_dim;
    if (head_dim > 512 || v_dim > 512 || dq > 2048) return IB_ERR_UNSUPPORTED;
#if !IB_ACT_BF16
    // Tiles of 32 queries where the step brings more than two tokens a request on average, else a token a CTA (a tile's
    // requests are walked one after another).  Measured on a B200, 16 query heads of 128 on 8, launch included: four tokens
    // behind 41 to 208 keys 19 us (a warp per token and head: 60 us), behind 2,048 keys 92 us; prompts of 33 to 200
    // tokens 62 us (a warp per token and head: 195 us).
    const int group = n_heads / n_kv_heads;
    if (!joint && dist_bias == nullptr && group <= 32 && head_dim % 4 == 0 && v_dim % 4 == 0 && head_dim <= gat::MAX_DIM &&
        v_dim <= gat::MAX_DIM && n_kv_heads <= 65535 && (uintptr_t)k_pages % 16 == 0 && (uintptr_t)v_pages % 16 == 0) {
        const bool many = n_rows > 2 * n_requests;
        const int tokens = many ? 32 / group : 1;
        const dim3 tiles((n_rows + tokens - 1) / tokens, n_kv_heads);
#define IB_LAUNCH_TILES(WARPS, QPW)                                                                                       \
    do {                                                                                                                  \
        static IbDeviceSet allowed;                                                                                       \
        const int e = ib_allow_dynamic_smem(allowed, gat::tile_kernel<WARPS, QPW>,                                        \
                                            gat::smem_bytes(WARPS, QPW, gat::MAX_DIM, gat::MAX_DIM));                     \
        if (e) return e;                                                                                                  \
        ib_launch(gat::tile_kernel<WARPS, QPW>, tiles, 32 * WARPS, gat::smem_bytes(WARPS, QPW, head_dim, v_dim), stream,  \
                  (const float*)q, (const float*)k_pages, (const float*)v_pages, block_table, max_pages, page_size,       \
                  n_pages, row_request, positions, n_rows, tokens, n_heads, n_kv_heads, head_dim, v_dim, scale, window,   \
                  (float*)out, opt);                                                                                      \
        return ib_launch_status();                                                                                        \
    } while (0)
        if (many || group > 8) IB_LAUNCH_TILES(8, 4);
#undef IB_LAUNCH_TILES
#define IB_LAUNCH_TOKENS(G)                                                                                               \
    do {                                                                                                                  \
        static IbDeviceSet allowed;                                                                                       \
        const int e = ib_allow_dynamic_smem(allowed, gat::token_kernel<G>,                                                \
                                            gat::token_smem_bytes(G, gat::MAX_DIM, gat::MAX_DIM));                        \
        if (e) return e;                                                                                                  \
        ib_launch(gat::token_kernel<G>, tiles, 128 * (G < 4 ? G : 4), gat::token_smem_bytes(G, head_dim, v_dim), stream, (const float*)q,   \
                  (const float*)k_pages, (const float*)v_pages, block_table, max_pages, page_size, n_pages, row_request,  \
                  positions, n_heads, n_kv_heads, head_dim, v_dim, scale, window, (float*)out, opt);                      \
        return ib_launch_status();                                                                                        \
    } while (0)
        if (group > 4) IB_LAUNCH_TOKENS(8);
        if (group > 2) IB_LAUNCH_TOKENS(4);
        if (group > 1) IB_LAUNCH_TOKENS(2);
        IB_LAUNCH_TOKENS(1);
#undef IB_LAUNCH_TOKENS
    }
#endif
    const dim3 grid(n_rows, (n_heads + ATT_WARPS - 1) / ATT_WARPS);
    const size_t smem = (size_t)ATT_WARPS * dq * sizeof(float);
#define IB_LAUNCH_ATT_J(DPL, JOINT)                                                                             \
    ib_launch(paged_attention_generic_kernel<DPL, JOINT>, grid, 32 * ATT_WARPS, smem, stream,                   \
        (const act_t*)q, (const act_t*)k_pages, (const act_t*)v_pages, block_table, max_pages, page_size,       \
        n_pages, row_request, positions, n_heads, n_kv_heads, head_dim, v_dim, scale, window, (act_t*)out,      \
        dist_bias, bias_len, opt)
#define IB_LAUNCH_ATT(DPL) do { if (joint) IB_LAUNCH_ATT_J(DPL, true); else IB_LAUNCH_ATT_J(DPL, false); } while (0)
    if (v_dim <= 32) IB_LAUNCH_ATT(1);
    else if (v_dim <= 64) IB_LAUNCH_ATT(2);
    else if (v_dim <= 128) IB_LAUNCH_ATT(4);
    else if (v_dim <= 256) IB_LAUNCH_ATT(8);
    else IB_LAUNCH_ATT(16);
#undef IB_LAUNCH_ATT
#undef IB_LAUNCH_ATT_J
    return ib_launch_status();
}
