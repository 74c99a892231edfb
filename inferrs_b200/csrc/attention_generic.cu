// Grouped-query attention over the paged cache, for any head size: 32-bit arithmetic
// throughout.  One warp per (token, query head) for everything, and for 32-bit
// activations whose heads hold a multiple of four numbers, 128 at most, one CTA per
// tile of tokens, or per token, and key/value head (below).
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
// 32 keys and values at a time come into shared memory by cp.async, the next ones while these are worked on, and serve all
// of the CTA's queries.  (One warp per token and head read every key once per query head, each lane a key of its own, 4
// bytes at a time: 32 sectors a load.)  Two forms: tile_kernel takes the query heads of one key/value head for several
// tokens that follow one another in a request, token_kernel for one token.
// A row's sums are the same in both: four partial sums per score (numbers 0, 4, 8, ... of the head, 1, 5, 9, ... and so
// on), the score's slope, factor and cap by score() below, keys in ascending tiles of 32 from a multiple of 32; a tile of
// which a row sees nothing leaves its sums as they are.  They depend on the row's position and options only, as above.
#if !IB_ACT_BF16
namespace gat {

constexpr int KEYS = 32, PLD = KEYS + 4, MAX_DIM = 128;
constexpr int WARPS = 8, QPW = 4, QUERIES = WARPS * QPW;   // of tile_kernel: warps, queries of a warp
constexpr int SHORT_RUN = 2;                               // rows of a request that go to token_kernel in a step of both
constexpr int SMS = 148;
constexpr size_t SM_BYTES = 228 * 1024;

// 16 bytes, or zeros where there are none
__device__ __forceinline__ void copy16(float* dst, const float* src, bool there) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(there ? 16 : 0) : "memory");
}

// A product's score.  Written so that the compiler has no choice of what to contract: both forms must round alike.
__device__ __forceinline__ float score(float dot, float scale, float slope, int distance, float cap) {
    const float s = fmaf(-slope, (float)distance, __fmul_rn(dot, scale));
    return cap > 0.0f ? cap * tanhf(s / cap) : s;
}

static size_t tile_smem_bytes(int d, int dv) { return sizeof(float) * (2 * KEYS * (d + 4 + dv) + QUERIES * (d + PLD)); }
static size_t token_smem_bytes(int g, int t, int d, int dv) { return sizeof(float) * (t * KEYS * (d + 4 + dv) + g * d); }

// Up to `tokens` rows of one request and one key/value head at a time.  A warp owns QPW queries from the scores to the
// output: a lane has one key for the scores and the softmax, four value numbers for the output, so nothing is exchanged
// between warps; bound by its instructions.  The step's rows are cut into windows of `tokens` (blockIdx.x), and of the runs of
// one request's rows in its window a CTA takes every gridDim.z-th: a CTA for all of them walks one request after the
// other while most of its warps have no query (four prompts of 33 to 200 tokens, 16 heads on 16: 60 us, now 51).  shared:
// runs of up to SHORT_RUN rows, counted beyond the window's edges, are token_kernel's.
// FEWEST: CTAs per SM.  Two pay where there are as many (a prompt of 2,048 tokens: 1,485 us with one, 1,145 with two), one has
// the registers to be faster by itself.
template <int FEWEST>
__global__ void __launch_bounds__(32 * WARPS, FEWEST) tile_kernel(
    const float* __restrict__ q, const float* __restrict__ k_pages, const float* __restrict__ v_pages,
    const int* __restrict__ block_table, int max_pages, int page_size, int n_pages, const int* __restrict__ row_request,
    const int* __restrict__ positions, int n_rows, int tokens, int shared, int n_heads, int n_kv_heads, int d, int dv,
    float scale, int window, float* __restrict__ out, const IbScoreOptions opt) {
    extern __shared__ __align__(16) float smem[];
    __shared__ int s_run[QUERIES + 1], s_req[QUERIES], s_pos[QUERIES], q_pos[QUERIES], q_lo[QUERIES];
    __shared__ float q_scale[QUERIES], q_slope[QUERIES], q_m[QUERIES], q_l[QUERIES], q_corr[QUERIES];
    const int group = n_heads / n_kv_heads, kvh = blockIdx.y, kld = d + 4;
    float* ks = smem;                                   // [2][KEYS][d + 4]
    float* vs = ks + 2 * KEYS * kld;                    // [2][KEYS][dv]
    float* qs = vs + 2 * KEYS * dv;                     // [queries][d]
    float* ps = qs + QUERIES * d;                       // [queries][PLD]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
    const int window0 = blockIdx.x * tokens, in_window = min(tokens, n_rows - window0);
    ib_grid_dependency_sync();
    if (tid >= 32 && tid - 32 < in_window) s_pos[tid - 32] = positions[window0 + tid - 32];
    if (warp == 0) {
        // the window's rows, a lane each, and the two before and behind it: this CTA's runs as first row * 64 + rows
        const int mine = row_request[window0 + min(lane, in_window - 1)];
        const int beside = lane < SHORT_RUN ? window0 - 1 - lane : window0 + in_window + lane - SHORT_RUN;
        const bool known = shared && lane < 2 * SHORT_RUN && beside >= 0 && beside < n_rows;
        const int other = known ? row_request[beside] : -1;
        const int edge = __shfl_sync(0xffffffffu, mine, lane < SHORT_RUN ? 0 : in_window - 1);
        const unsigned joins = __ballot_sync(0xffffffffu, known && other == edge);
        const int left = __ffs(~(joins & ((1u << SHORT_RUN) - 1))) - 1, right = __ffs(~(joins >> SHORT_RUN)) - 1;
        const int ahead = __shfl_up_sync(0xffffffffu, mine, 1);
        const bool starts = lane < in_window && (lane == 0 || mine != ahead);
        const unsigned all = __ballot_sync(0xffffffffu, starts), behind = lane < 31 ? all >> (lane + 1) : 0u;
        const int end = behind ? lane + __ffs(behind) : in_window;
        const int len = end - lane + (lane == 0 ? left : 0) + (end == in_window ? right : 0);
        const unsigned taken = __ballot_sync(0xffffffffu, starts && !(shared && len <= SHORT_RUN));
        const int nth = __popc(taken & ((1u << lane) - 1)), slots = gridDim.z;
        if ((taken >> lane & 1) && nth % slots == blockIdx.z) {
            s_run[nth / slots] = lane * 64 + end - lane;
            s_req[nth / slots] = mine;
        }
        if (lane == 0) s_run[QUERIES] = (__popc(taken) + slots - 1 - (int)blockIdx.z) / slots;
    }
    __syncthreads();
    for (int run = 0; run < s_run[QUERIES]; ++run) {
        const int in0 = s_run[run] / 64, row0 = window0 + in0, rows = s_run[run] % 64, req = s_req[run];
        const int* pos_of = s_pos + in0;
        if (run > 0) __syncthreads();                   // everyone has left the run before
        for (int m = warp; m < rows * group; m += WARPS) {
            const float* src = q + ((long)(row0 + m / group) * n_heads + kvh * group + m % group) * d;
            for (int e = lane; e < d; e += 32) qs[m * d + e] = src[e];
        }
        __syncthreads();
        int lo_min = ib_first_visible(pos_of[0], window), pos_max = pos_of[0];
        for (int r = 1; r < rows; ++r) {
            const int lo = ib_first_visible(pos_of[r], window);
            lo_min = lo < lo_min ? lo : lo_min;
            pos_max = pos_of[r] > pos_max ? pos_of[r] : pos_max;
        }
        const int* bt = block_table + (long)req * max_pages;
        const int t_first = lo_min / KEYS, n_kept = ib_kept_tiles(opt.keep_first, t_first, KEYS);
        const int n_tiles = n_kept + (pos_max >= 0 ? pos_max / KEYS : -1) + 1 - t_first;
        auto place = [&](int j) -> long {                   // of key j of this request, counted in heads' rows; -1: nowhere
            if (j > pos_max) return -1;
            const int page = bt[j / page_size];
            return page >= 0 && page < n_pages ? ((long)page * n_kv_heads + kvh) * page_size + j % page_size : -1;
        };
        auto fetch = [&](int i) {
            float* kd = ks + (i & 1) * KEYS * kld;
            float* vd = vs + (i & 1) * KEYS * dv;
            const long mine = place(ib_nth_tile(i, n_kept, t_first) * KEYS + lane);
#pragma unroll 1
            for (int j = warp; j < KEYS; j += WARPS) {
                const long at = __shfl_sync(0xffffffffu, mine, j);
                if (lane * 4 < d) copy16(kd + j * kld + lane * 4, at >= 0 ? k_pages + at * d + lane * 4 : k_pages, at >= 0);
                if (lane * 4 < dv) copy16(vd + j * dv + lane * 4, at >= 0 ? v_pages + at * dv + lane * 4 : v_pages, at >= 0);
            }
        };
        if (lane < QPW) {                                   // the warp's own queries (position -1: none)
            const int m = warp * QPW + lane, r = m / group, head = kvh * group + m % group;
            const bool there = r < rows;
            q_pos[m] = there ? pos_of[r] : -1;
            q_lo[m] = there ? ib_first_visible(pos_of[r], window) : 0;
            q_scale[m] = there && opt.head_scale ? scale * opt.head_scale[head] : scale;
            q_slope[m] = there && opt.slopes ? opt.slopes[head] : 0.0f;
            q_m[m] = -INFINITY;
            q_l[m] = 0.0f;
            q_corr[m] = 1.0f;
        }
        __syncwarp();
        float acc[QPW][4];
        int last = -1;                                      // the furthest key that a query of this warp sees
#pragma unroll
        for (int c = 0; c < QPW; ++c) {
            acc[c][0] = acc[c][1] = acc[c][2] = acc[c][3] = 0.0f;
            last = max(last, q_pos[warp * QPW + c]);
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
                for (int c = 0; c < QPW; ++c) {             // (a loop: unrolled four times it is more code than it saves)
                    const int m = warp * QPW + c, pos = q_pos[m];
                    float s = -INFINITY;
                    if (there && ib_visible(j, q_lo[m], pos, opt.keep_first))
                        s = score(own[c * PLD], q_scale[m], q_slope[m], pos - j, opt.cap);
                    const float m_run = q_m[m], m_new = fmaxf(m_run, ib_warp_max(s));
                    const float p = (s == -INFINITY) ? 0.0f : expf(s - m_new);
                    const float corr = (m_run == -INFINITY) ? 0.0f : expf(m_run - m_new);
                    const float l = fmaf(q_l[m], corr, ib_warp_sum(p));
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
                    const int keys = last + 1 - j0 < KEYS ? last + 1 - j0 : KEYS;
#pragma unroll 1
                    for (int jj = 0; jj < keys; jj += 4) {
                        float4 vv[4];
#pragma unroll
                        for (int g = 0; g < 4; ++g) vv[g] = *reinterpret_cast<const float4*>(vr + (jj + g) * dv);
#pragma unroll
                        for (int c = 0; c < QPW; ++c) {
                            const float4 p4 = *reinterpret_cast<const float4*>(pr + c * PLD + jj);
                            const float p[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
                            for (int g = 0; g < 4; ++g) {
                                if (p[g] != 0.0f) {         // a masked key's value is not looked at
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
            __syncthreads();                                // this tile's buffer may be filled again
        }
        __syncwarp();
        float* own = ps + warp * QPW * PLD;                 // 1 / denominator and the last correction, a lane per query
        if (lane < QPW) {
            const int m = warp * QPW + lane, r = m / group, head = kvh * group + m % group;
            float l = q_l[m], corr = 1.0f;
            if (r < rows) {
                if (opt.sinks) {                            // adds to the denominator and to nothing else
                    const float sink = opt.sinks[head], m_new = fmaxf(q_m[m], sink);
                    corr = (q_m[m] == -INFINITY) ? 0.0f : expf(q_m[m] - m_new);
                    l = fmaf(l, corr, expf(sink - m_new));
                }
                own[lane] = (l > 0.0f ? 1.0f / l : 0.0f) * ib_head_gate(opt, row0 + r, head);
            }
            own[QPW + lane] = corr;
        }
        __syncwarp();
#pragma unroll
        for (int c = 0; c < QPW; ++c) {
            const int m = warp * QPW + c, r = m / group, head = kvh * group + m % group;
            if (r >= rows || lane * 4 >= dv) continue;
            float* dst = out + (row0 + r) * opt.out_ld + (long)head * dv + lane * 4;
#pragma unroll
            for (int e = 0; e < 4; ++e) dst[e] = acc[c][e] * own[QPW + c] * own[c];
        }
    }
}

// One token and key/value head per CTA, up to G query heads: T tiles at a time and T warps per query head (four heads side by
// side at most, PER of them after one another): each warp takes the scores of one tile of 32 keys, the running maximum
// goes over the tiles in order, and a thread owns 4 / T value numbers of each of its heads.  The next keys are on their way
// while values are summed, the next values during the scores.  Bound by the instructions of that chain: few rows want T = 4,
// many T = 1, with which six CTAs of heads of 128 share an SM instead of one (16 heads on 16 behind 1,000 keys, T = 4 / 1: one
// row 51 / 146 us, 256 rows 1,191 / 706; 256 rows behind 8 keys 263 with T = 4 and all of its tiles, 33 with T = 1).
// shared: only the rows of runs of up to SHORT_RUN rows of one request.
template <int G, int T>
__global__ void __launch_bounds__(32 * T * (G < 4 ? G : 4), 1024 / (32 * T * (G < 4 ? G : 4))) token_kernel(
    const float* __restrict__ q, const float* __restrict__ k_pages, const float* __restrict__ v_pages,
    const int* __restrict__ block_table, int max_pages, int page_size, int n_pages, const int* __restrict__ row_request,
    const int* __restrict__ positions, int n_rows, int shared, int n_heads, int n_kv_heads, int d, int dv, float scale,
    int window, float* __restrict__ out, const IbScoreOptions opt) {
    constexpr int SIDE = G < 4 ? G : 4, PER = G / SIDE, LINE = 32 * T, THREADS = LINE * SIDE, NV = 4 / T;
    extern __shared__ __align__(16) float smem[];
    __shared__ float s_max[G][T], s_sum[G][T], s_corr[G][T], s_m[G], s_l[G];
    __shared__ __align__(16) float ps[G][T * KEYS];
    const int group = n_heads / n_kv_heads, kvh = blockIdx.y, row = blockIdx.x;
    const int kld = d + 4, tid = threadIdx.x, lane = tid & 31, tile = (tid >> 5) % T, side = tid / LINE, c0 = side * PER;
    float* ks = smem;                                   // [T * KEYS][d + 4]
    float* vs = ks + T * KEYS * kld;                    // [T * KEYS][dv]
    float* qs = vs + T * KEYS * dv;                     // [G][d]
    // a row's place and the keys and values of earlier steps are fetched while the kernel ahead still runs
    ib_grid_dependency_launch();
    const int req = row_request[row], pos = positions[row];
    if (shared) {
        const int beside = row - SHORT_RUN + lane;
        const bool known = lane <= 2 * SHORT_RUN && beside >= 0 && beside < n_rows;
        const unsigned same = __ballot_sync(0xffffffffu, (known ? row_request[beside] : -1) == req && known);
        if (__clz(~(same << (32 - SHORT_RUN))) + __ffs(~(same >> SHORT_RUN)) - 1 > SHORT_RUN) {
            ib_grid_dependency_wait();
            return;
        }
    }
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
    // own: the row's own key, the last of the last tile
    auto fetch = [&](float* dst, int ld, const float* pages, int n, int i, long at, bool own, bool others) {
        const float* mine = at >= 0 ? pages + at * n : nullptr;
        dst += tile * KEYS * ld + lane * 4;
        auto copy = [&](int j) {                        // the warps of a tile share its rows
            const float* src = reinterpret_cast<const float*>(__shfl_sync(0xffffffffu, (unsigned long long)mine, j));
            if (lane * 4 < n) copy16(dst + j * ld, src ? src + lane * 4 : pages, src != nullptr);
        };
        if (i < n_tiles - 1) {
            if (others) {
#pragma unroll 2
                for (int j = side; j < KEYS; j += SIDE) copy(j);
            }
        } else if (i == n_tiles - 1) {                  // the last tile ends with the row's own key
            const int last = pos % KEYS;
            if (others) {
#pragma unroll 1
                for (int j = side; j < last; j += SIDE) copy(j);
            }
            if (own && last % SIDE == side) copy(last);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    long at = place(tile);
    const bool early = row == 0 || row_request[row - 1] != req;         // no key but its own is this step's
    if (early) {
        fetch(ks, kld, k_pages, d, tile, at, false, true);
        fetch(vs, dv, v_pages, dv, tile, at, false, true);
    }
    ib_grid_dependency_wait();
    q = ib_after_wait(q);
    fetch(ks, kld, k_pages, d, tile, at, true, !early);
    fetch(vs, dv, v_pages, dv, tile, at, true, !early);
    for (int e = tid; e < group * d; e += THREADS) qs[e] = q[((long)row * n_heads + kvh * group) * d + e];
    for (int c = tid; c < G; c += THREADS) {
        s_m[c] = -INFINITY;
        s_l[c] = 0.0f;
    }
    const int e0 = (tid % LINE) * NV;                   // this thread's value numbers
    float acc[PER][NV];
#pragma unroll
    for (int c = 0; c < PER; ++c)
#pragma unroll
        for (int k = 0; k < NV; ++k) acc[c][k] = 0.0f;
    for (int i0 = 0; i0 < n_tiles; i0 += T) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");            // the keys
        __syncthreads();
        const bool live = i0 + tile < n_tiles;                          // (the warp has a tile in this round)
        if (live) {
            const int j = ib_nth_tile(i0 + tile, n_kept, t_first) * KEYS + lane;
            const bool seen = at >= 0 && ib_visible(j, lo, pos, opt.keep_first);
            const float* kr = ks + (tile * KEYS + lane) * kld;
            float4 dot[PER];
#pragma unroll
            for (int c = 0; c < PER; ++c) dot[c] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
            for (int e = 0; e < d; e += 4) {
                const float4 kv = *reinterpret_cast<const float4*>(kr + e);
#pragma unroll
                for (int c = 0; c < PER; ++c) {
                    const float4 qv = *reinterpret_cast<const float4*>(qs + (c0 + c) * d + e);
                    dot[c].x = fmaf(qv.x, kv.x, dot[c].x);
                    dot[c].y = fmaf(qv.y, kv.y, dot[c].y);
                    dot[c].z = fmaf(qv.z, kv.z, dot[c].z);
                    dot[c].w = fmaf(qv.w, kv.w, dot[c].w);
                }
            }
#pragma unroll
            for (int c = 0; c < PER; ++c) {
                if (c0 + c >= group) continue;
                const int head = kvh * group + c0 + c;
                float s = -INFINITY;
                if (seen)
                    s = score((dot[c].x + dot[c].y) + (dot[c].z + dot[c].w),
                              opt.head_scale ? scale * opt.head_scale[head] : scale, opt.slopes ? opt.slopes[head] : 0.0f,
                              pos - j, opt.cap);
                ps[c0 + c][tile * KEYS + lane] = s;
                const float top = ib_warp_max(s);
                if (lane == 0) s_max[c0 + c][tile] = top;
            }
        }
        __syncthreads();                                                // everyone has left the keys
        at = place(i0 + T + tile);
        fetch(ks, kld, k_pages, d, i0 + T + tile, at, true, true);
        if (live) {
#pragma unroll
            for (int c_ = 0; c_ < PER; ++c_) {
                const int c = c0 + c_;
                if (c >= group) continue;
                float before = s_m[c];                                  // the maximum over the tiles before this one
                for (int t = 0; t < tile; ++t) before = fmaxf(before, s_max[c][t]);
                const float mine = fmaxf(before, s_max[c][tile]), s = ps[c][tile * KEYS + lane];
                if (lane == 0) s_corr[c][tile] = (before == -INFINITY) ? 0.0f : expf(before - mine);
                const float p = (s == -INFINITY) ? 0.0f : expf(s - mine), sum = ib_warp_sum(p);
                ps[c][tile * KEYS + lane] = p;
                if (lane == 0) s_sum[c][tile] = sum;
            }
        }
        asm volatile("cp.async.wait_group 1;" ::: "memory");            // the values
        __syncthreads();                                                // ... and the probabilities
        const int n_live = min(T, n_tiles - i0);
        if (tid < group) {                                              // (read again after the next round's barriers)
            float l = s_l[tid], m = s_m[tid];
#pragma unroll
            for (int t = 0; t < T; ++t)
                if (t < n_live) {
                    l = fmaf(l, s_corr[tid][t], s_sum[tid][t]);
                    m = fmaxf(m, s_max[tid][t]);
                }
            s_l[tid] = l;
            s_m[tid] = m;
        }
        if (e0 < dv) {
#pragma unroll 1
            for (int t = 0; t < n_live; ++t) {
#pragma unroll
                for (int c = 0; c < PER; ++c)
                    if (c0 + c < group)
#pragma unroll
                        for (int k = 0; k < NV; ++k) acc[c][k] *= s_corr[c0 + c][t];
                const float* vr = vs + t * KEYS * dv + e0;
                auto four = [&](int jj) {
                    float v[4][NV];
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        if constexpr (NV == 4) {
                            const float4 x = *reinterpret_cast<const float4*>(vr + g * dv);
                            v[g][0] = x.x; v[g][1] = x.y; v[g][2] = x.z; v[g][3] = x.w;
                        } else if constexpr (NV == 2) {
                            const float2 x = *reinterpret_cast<const float2*>(vr + g * dv);
                            v[g][0] = x.x; v[g][1] = x.y;
                        } else {
                            v[g][0] = vr[g * dv];
                        }
                    }
                    vr += 4 * dv;
#pragma unroll
                    for (int c = 0; c < PER; ++c) {
                        if (c0 + c >= group) continue;
                        const float4 p4 = *reinterpret_cast<const float4*>(&ps[c0 + c][t * KEYS + jj]);
                        const float p[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
                        for (int g = 0; g < 4; ++g)
                            if (p[g] != 0.0f)                           // a masked key's value is not looked at
#pragma unroll
                                for (int k = 0; k < NV; ++k) acc[c][k] = fmaf(p[g], v[g][k], acc[c][k]);
                    }
                };
                if (i0 + t < n_tiles - 1) {
                    constexpr int AT_ONCE = NV == 4 ? 4 : 8;
#pragma unroll AT_ONCE
                    for (int jj = 0; jj < KEYS; jj += 4) four(jj);
                } else {
#pragma unroll 1
                    for (int jj = 0; jj <= pos % KEYS; jj += 4) four(jj);
                }
            }
        }
        __syncthreads();                                                // everyone has left the values
        fetch(vs, dv, v_pages, dv, i0 + T + tile, at, true, true);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int c = 0; c < PER; ++c) {
        if (c0 + c >= group) continue;
        const int head = kvh * group + c0 + c;
        float l = s_l[c0 + c], co = 1.0f;
        if (opt.sinks) {
            const float m = s_m[c0 + c], m_new = fmaxf(m, opt.sinks[head]);
            co = (m == -INFINITY) ? 0.0f : expf(m - m_new);
            l = fmaf(l, co, expf(opt.sinks[head] - m_new));
        }
        const float inv = (l > 0.0f ? 1.0f / l : 0.0f) * ib_head_gate(opt, row, head);
        if (e0 < dv)
#pragma unroll
            for (int k = 0; k < NV; ++k) out[row * opt.out_ld + (long)head * dv + e0 + k] = acc[c][k] * co * inv;
    }
}

struct Step {
    const float* q;
    const float* k_pages;
    const float* v_pages;
    const int* block_table;
    int max_pages, page_size, n_pages;
    const int* row_request;
    const int* positions;
    int n_rows, n_requests, n_heads, n_kv_heads, d, dv;
    float scale;
    int window;
    float* out;
    IbScoreOptions opt;
    cudaStream_t stream;
};

// Shared memory that a CTA asks for: no SM is to take more CTAs than the fullest one has to, since those that come before the
// kernel ahead has left its SMs would crowd on the free ones otherwise.
static size_t spread(size_t smem, long ctas) {
    const size_t share = SM_BYTES / ((ctas + SMS - 1) / SMS + 1);
    return smem > share ? smem : share;
}

template <int FEWEST>
static int launch_tiles(const Step& s, int tokens, int slots, bool shared) {
    static IbDeviceSet allowed;
    if (const int e = ib_allow_dynamic_smem(allowed, tile_kernel<FEWEST>, SM_BYTES / 2)) return e;
    const int windows = (s.n_rows + tokens - 1) / tokens;
    ib_launch(tile_kernel<FEWEST>, dim3(windows, s.n_kv_heads, slots), 32 * WARPS,
              spread(tile_smem_bytes(s.d, s.dv), (long)windows * s.n_kv_heads), s.stream, s.q, s.k_pages, s.v_pages, s.block_table,
              s.max_pages, s.page_size, s.n_pages, s.row_request, s.positions, s.n_rows, tokens, (int)shared, s.n_heads, s.n_kv_heads,
              s.d, s.dv, s.scale, s.window, s.out, s.opt);
    return ib_launch_status();
}

template <int G, int T>
static int launch_tokens(const Step& s, bool shared) {
    static IbDeviceSet allowed;
    constexpr size_t half = SM_BYTES / 2;
    const size_t most = token_smem_bytes(G, T, MAX_DIM, MAX_DIM);
    if (const int e = ib_allow_dynamic_smem(allowed, token_kernel<G, T>, most > half ? most : half)) return e;
    const size_t smem = token_smem_bytes(G, T, s.d, s.dv);
    ib_launch(token_kernel<G, T>, dim3(s.n_rows, s.n_kv_heads), 32 * T * (G < 4 ? G : 4),
              shared ? smem : spread(smem, (long)s.n_rows * s.n_kv_heads), s.stream, s.q, s.k_pages, s.v_pages, s.block_table,
              s.max_pages, s.page_size, s.n_pages, s.row_request, s.positions, s.n_rows, (int)shared, s.n_heads, s.n_kv_heads, s.d, s.dv,
              s.scale, s.window, s.out, s.opt);
    return ib_launch_status();
}

// CTAs of token_kernel<G, T> that an SM holds, by shared memory and by 64 registers a thread
static long resident(int g, int t, int d, int dv) {
    const long by_memory = 227 * 1024 / ((long)token_smem_bytes(g, t, d, dv) + 4 * g * KEYS * t + 1280);
    const long by_threads = 1024 / (32 * t * (g < 4 ? g : 4));
    return by_memory < by_threads ? by_memory : by_threads;
}

// As many tiles at a time as leave all CTAs room at once; one beside tile_kernel, where most CTAs leave at once.
template <int G>
static int launch_tokens(const Step& s, bool shared) {
    const long per_sm = ((long)s.n_kv_heads * s.n_rows + SMS - 1) / SMS;
    if (!shared && per_sm <= resident(G, 4, s.d, s.dv)) return launch_tokens<G, 4>(s, shared);
    if (!shared && per_sm <= resident(G, 2, s.d, s.dv)) return launch_tokens<G, 2>(s, shared);
    return launch_tokens<G, 1>(s, shared);
}

static int launch_tokens(const Step& s, bool shared) {
    const int group = s.n_heads / s.n_kv_heads;
    return group > 4   ? launch_tokens<8>(s, shared)
           : group > 2 ? launch_tokens<4>(s, shared)
           : group > 1 ? launch_tokens<2>(s, shared)
                       : launch_tokens<1>(s, shared);
}

// Which form takes the step; the bits are the same.  us on a B200, launches included; in brackets a warp per token and head.
//   * More than eight query heads a key/value head: tiles, of a single token in steps of them (16 heads on 1, 64 tokens
//     behind 1,000 keys 140 (835); behind 8 keys 8 (10)).  Runs of a window side by side while they are short, when a CTA's
//     start is what they wait for (32 heads on 2, 128 requests of 1 to 8 tokens 25, one after the other 38 (18)).
//   * Few rows a request: tokens.  16 heads on 8: one token behind 1,000 keys 45 (485), 64 tokens 145 (1,004), 64 behind
//     2,048 keys beside a prompt of 200 351 (3,238; tiles alone 1,059).  "Few" is up to eight on average, two for a request by
//     itself; while no row sees more than 128 keys, up to 8 + 4 a head of the group: 32 prompts of 10 tokens 14 (32; tiles 17), 16
//     of 20 tokens 15 (56; tiles 14), of 32 heads on 4 16 (76; tiles 22).
//   * Else tiles: a prompt of 512 tokens 126 (1,388; tokens 215), a token behind 900 keys and a prompt of 400 141 (1,042;
//     tokens 184).
//   * Where single tokens alone would be more CTAs than two per SM, both: runs of one or two rows as tokens, the others as
//     tiles.
static int launch(const Step& s) {
    const int group = s.n_heads / s.n_kv_heads;
    const bool singles = s.n_rows <= 2 * s.n_requests;
    const int tokens = group > 8 && singles ? 1 : QUERIES / group;
    const long tiles = (long)((s.n_rows + tokens - 1) / tokens) * s.n_kv_heads;
    const bool few_keys = (long)s.max_pages * s.page_size <= 128;
    if (group > 8) {
        if (!few_keys || singles || s.n_requests < 2) return launch_tiles<1>(s, tokens, 1, false);
        return launch_tiles<2>(s, tokens, tokens, false);
    }
    const long few_rows = (few_keys ? 8 + 4 * group : s.n_requests > 1 ? 8 : 2) * (long)s.n_requests;
    if (s.n_rows <= few_rows) return launch_tokens(s, false);
    const int slots = s.n_requests < 1 ? 1 : s.n_requests < 4 ? s.n_requests : 4;
    const bool both = (long)s.n_requests * s.n_kv_heads > 2 * SMS;
    if (both)
        if (const int e = launch_tokens(s, true)) return e;
    return tiles <= SMS ? launch_tiles<1>(s, tokens, slots, both) : launch_tiles<2>(s, tokens, slots, both);
}

}  // namespace gat
#endif

IB_EXPORT int ib_paged_attention_generic(const void* q, const void* k_pages, const void* v_pages,
                                         const int* block_table, int max_pages, int page_size, int n_pages,
                                         const int* row_request, const int* positions, int n_rows,
                                         int n_requests, int n_heads, int n_kv_heads, int head_dim, int v_dim, float scale,
                                         int window, void* out,
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
    const int group = n_heads / n_kv_heads;
    if (!joint && dist_bias == nullptr && group <= gat::QUERIES && head_dim % 4 == 0 && v_dim % 4 == 0 && head_dim <= gat::MAX_DIM &&
        v_dim <= gat::MAX_DIM && n_kv_heads <= 65535 && (uintptr_t)k_pages % 16 == 0 && (uintptr_t)v_pages % 16 == 0) {
        const gat::Step step = {(const float*)q, (const float*)k_pages, (const float*)v_pages, block_table, max_pages, page_size,
                                n_pages, row_request, positions, n_rows, n_requests, n_heads, n_kv_heads, head_dim, v_dim, scale,
                                window, (float*)out, opt, stream};
        return gat::launch(step);
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
