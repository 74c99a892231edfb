// y[t, f] = sum_k x[t, k] * w[f, k]  for 32-bit x, w and y on the fifth-generation tensor cores, without giving up
// any of the 32 bits.
//
// A float32 number has 24 significant bits and bfloat16 has 8, with the same range of exponents: every finite number is exactly
// the sum of three bfloat16 numbers (the number rounded to eight bits, what is left rounded again, and the rest: at most 2^-8
// and 2^-17 of it, of either sign).  A product of two numbers is then nine products of their pieces, each exact in
// float32.  Eight are taken; the ninth is below 2^-34 of the product.  The tensor cores' float32 accumulators round towards
// zero, so the one of the largest product is not kept longer than 64 of k: then its value is added to a float32 sum in
// registers, which rounds to nearest.  The seven others have accumulators of their own (two: by size) for a segment of K,
// which are added to each other before they join that sum.
//
// Error against 64 bits, of the result's norm, six products of cut pieces / these / a chain of fused multiply-adds: normal x
// and w, K 512 1.2e-7 / 8.3e-8 / 4.1e-7, K 4,096 1.4e-7 / 1.0e-7 / 1.2e-6; positive ones, K 4,096 1.2e-7 / 7.9e-8 / 8.4e-7; all
// numbers 1 + 2^-7 - 2^-23, K 512 4.7e-7 / 1.8e-9 / 1.2e-7; sums of a single product 6e-8 / 2.5e-8 / 2.5e-8 (rounded once).  Cutting
// and leaving out the products of the second and third pieces loses up to 2^-21 of a product, always on one side.  What
// these cost beside the six: 0 to 1 % up to 64 rows, 2 to 4 % beyond (512 rows, 4,096 features over 1,024: 42.6 -> 43.9 us;
// 2,048 rows 155 -> 164).
//
// The order of the sums depends on K alone, so a row's bits do not depend on how many rows the batch has, where the row
// stands in it or how the work is cut: the ceil(K / 64) blocks fall into eight segments of equal length (the last may
// be short or empty), a segment's blocks are added in ascending order, and the eight segments pair by pair, the pairs
// pair by pair, and so on.  A cluster of 2, 4 or 8 CTAs can therefore share a tile's K: each adds up a branch
// of that tree, and the branches meet through distributed shared memory.
//
// Roles in a CTA (tile_rows <= 128 rows of W as the M of the products, BN tokens as their N):
//   warp 0      TMA producer: 32 of k of W and x, as float32, per stage of the ring
//   warp 1      issuer of the products, owner of the tensor-memory allocation
//   warps 2-3   x's pieces, to three swizzled tiles in shared memory (the products' B operand); beyond 16 tokens two more
//               warps at the end, on the SM's other schedulers
//   warps 4-7   W's pieces: a thread reads its row from the stage and writes the three pieces to tensor memory (the
//               products' A operand, so that W's pieces never pass through shared memory again)
//   warps 8-    the sums: four warps, or beyond 16 tokens eight with half of the tokens each
//
// What bounds it (512 rows, 4,096 features over 1,024): 44 us = 98 TFLOP/s, where a chain of multiply-adds took 110 to 160 us
// (36 TFLOP/s); 2,048 rows 105.  The tensor pipe is busy 40 % of the time, the issue slots 53, memory hands over 0.4 TB/s: the
// warps that make the pieces and add up are what a block of 64 of k waits for.  With two warps for x's pieces instead of
// four 45.8 us, with four summing warps instead of eight 63.5.  Up to 16 rows: a row 7 to 10 us, the way of x
// and the cluster's exchange; memory takes 1.3 to 4 of them.
//
// Infinities and NaN: the pieces of an infinity are no numbers, so a result that is not finite is computed again as
// one chain of fused multiply-adds, by the thread that would store it.  Numbers below 2^-110 have pieces that bfloat16 holds only
// partly, an absolute error of 2^-134 times the other factor: a result below 2^-90, which may be made of such numbers,
// is computed again too (but for zeros: rows of zeros are common, and only numbers below 2^-133 vanish).
//
// Every wait on an mbarrier is bounded (about two seconds); a wait that runs out records a code in the library's error
// word, the CTA lets outstanding copies land, frees its tensor memory and returns.
#include <cuda.h>

#include "common.cuh"
#include "sm100.cuh"

namespace split3 {

using namespace sm100;

constexpr int BM = 128;                 // rows of W per tile at most (the products' M)
constexpr int KS = 32;                  // k per stage of the ring: 32 floats = one 128-byte swizzle row
constexpr int BK = 64;                  // k per block: two stages, one round of products
constexpr int SEGMENTS = 8;
constexpr int SUM_WARP0 = 8;           // the first of the warps that add up
constexpr int W_STAGE = BM * KS * 4;

__device__ int g_error = 0;             // 0 ok; else (role code) of the first wait that ran out
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, int code) {
    return mbar_wait_bounded(bar, parity, &g_error, code);
}

struct Params {
    const float* x;
    const float* w;
    float* y;
    long ldx, ldw, ldy;
    int n_tok, n_out, k, tile_rows;
    int blocks, blocks_per_segment;     // of BK: in K, in a segment
};

__device__ __forceinline__ void cluster_arrive() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// one lane of a warp that is here as a whole; the compiler knows that it is one, and keeps what it computes for the
// tensor cores' descriptors out of the lanes' own registers
__device__ __forceinline__ bool elect_one() {
    unsigned ok;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok));
    return ok != 0;
}
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void st_cluster(unsigned local_addr, unsigned rank, float v) {
    unsigned remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local_addr), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(v) : "memory");
}

// Two neighbouring numbers of K as three pairs of bfloat16, the first in the low half.  Every piece is what is left, rounded
// to nearest; the differences are exact.  (Beyond 3.39e38 the first piece is an infinity: see `finished`.)
__device__ __forceinline__ unsigned pack_pair(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const unsigned*>(&v);
}
__device__ __forceinline__ void split_pair(float a, float b, unsigned& p0, unsigned& p1, unsigned& p2) {
    p0 = pack_pair(a, b);
    const float a1 = a - __uint_as_float(p0 << 16), b1 = b - __uint_as_float(p0 & 0xffff0000u);
    p1 = pack_pair(a1, b1);
    p2 = pack_pair(a1 - __uint_as_float(p1 << 16), b1 - __uint_as_float(p1 & 0xffff0000u));
}

// The result of one row and feature as one chain of fused multiply-adds: what infinities and NaN make of it, and numbers
// whose pieces are too small for bfloat16.
__device__ __noinline__ float chain(const float* x, const float* w, int k) {
    float s = 0.0f;
    for (int i = 0; i < k; ++i) s = fmaf(x[i], w[i], s);
    return s;
}
__device__ __forceinline__ float finished(const Params& p, float v, int tok, int feature) {
    const float a = fabsf(v);
    return a <= 3.402823466e38f && (a >= 8.077935669e-28f || a == 0.0f) ? v : chain(p.x + (long)tok * p.ldx, p.w + (long)feature * p.ldw, p.k);
}

// A segment's sum joins those before it: like the carry of a binary counter, so that equal powers of two of segments
// are added to each other.  A thread has C numbers: 16, all waiting sums in registers; or 32, single segments in tensor memory, pairs
// in shared memory (where the cluster's parts come later) and fours in registers.
template <int C> struct Waiting {
    float v[C <= 16 ? 3 : 1][C];
    unsigned tmem;                      // of this warp's lanes
    float* pairs;                       // of this thread: C numbers BM apart

    template <int L> __device__ __forceinline__ void add(float (&s)[C]) {
        if constexpr (C > 16 && L == 0) {
            unsigned t[32];
            tmem_ld32_issue(tmem, t);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < C; ++j) s[j] = __uint_as_float(t[j]) + s[j];
        } else if constexpr (C > 16 && L == 1) {
#pragma unroll
            for (int j = 0; j < C; ++j) s[j] = pairs[j * BM] + s[j];
        } else {
#pragma unroll
            for (int j = 0; j < C; ++j) s[j] = v[C <= 16 ? L : 0][j] + s[j];
        }
    }
    template <int L> __device__ __forceinline__ void put(const float (&s)[C]) {
        if constexpr (C > 16 && L == 0) {
            unsigned t[32];
#pragma unroll
            for (int j = 0; j < C; ++j) t[j] = __float_as_uint(s[j]);
            tmem_st32(tmem, t);
            tmem_st_wait();
        } else if constexpr (C > 16 && L == 1) {
#pragma unroll
            for (int j = 0; j < C; ++j) pairs[j * BM] = s[j];
        } else {
#pragma unroll
            for (int j = 0; j < C; ++j) v[C <= 16 ? L : 0][j] = s[j];
        }
    }
    // `n`: segments that this CTA has summed before; `last`: s is complete once everything that waits has joined
    __device__ __forceinline__ void join(float (&s)[C], int n, bool last) {
        if (!(n & 1)) { if (!last) put<0>(s); return; }
        add<0>(s);
        if (!(n & 2)) { if (!last) put<1>(s); return; }
        add<1>(s);
        if (!(n & 4)) { if (!last) put<2>(s); return; }
        add<2>(s);
    }
};

template <int BN, int STAGES>
constexpr size_t smem_bytes() {
    return 1024 + (size_t)STAGES * (W_STAGE + BN * KS * 4) + 2 * 3 * BN * BK * 2 + (size_t)BN * BM * 4 + 256;
}

constexpr int sum_warps(int bn) { return bn <= 16 ? 4 : 8; }
constexpr int x_warps(int bn) { return bn <= 16 ? 2 : 4; }
constexpr int threads_of(int bn) { return 32 * (SUM_WARP0 + sum_warps(bn) + x_warps(bn) - 2); }

template <int BN, int STAGES>
__global__ void __launch_bounds__(threads_of(BN), (BN <= 16 ? 2 : 1)) split_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                           const __grid_constant__ CUtensorMap map_x,
                                                                           const Params p) {
    constexpr int X_STAGE = BN * KS * 4, PIECE = BN * BK * 2;
    constexpr int A_COLS = 3 * BK / 2;                       // one block of W's pieces in tensor memory
    // accumulators: of the largest product per block parity, and of the others (two sizes side by side)
    constexpr int TMEM_ACC = 2 * A_COLS, TMEM_SMALL = TMEM_ACC + 2 * BN, TMEM_WAITING = TMEM_SMALL + 2 * BN;
    constexpr int TMEM_COLS = BN <= 16 ? 256 : 512;
    constexpr int X_WARPS = x_warps(BN), SUM_WARPS = sum_warps(BN), C = BN * 4 / SUM_WARPS;         // C: tokens of a thread that adds up
    static_assert(TMEM_WAITING + (C > 16 ? BN : 0) <= TMEM_COLS && (C == 16 || C == 32), "");
    static_assert((2 * STAGES + 7) * 8 + 8 <= 256, "");
    extern __shared__ unsigned char raw_smem[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(raw_smem) + 1023) & ~(uintptr_t)1023);
    unsigned char* w_ring = smem;
    unsigned char* x_ring = w_ring + STAGES * W_STAGE;
    unsigned char* pieces = x_ring + STAGES * X_STAGE;       // x's: [block parity][piece][BN][64], swizzled
    float* recv = reinterpret_cast<float*>(pieces + 2 * 3 * PIECE);   // [rank of the sender][BN][rows owned]
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(recv + BN * BM);
    const unsigned full0 = smem_u32(bars), empty0 = smem_u32(bars + STAGES);
    const unsigned ready0 = smem_u32(bars + 2 * STAGES);     // per block parity: both operands' pieces are there
    const unsigned done0 = smem_u32(bars + 2 * STAGES + 2);  // ... the products of a block are done
    const unsigned taken0 = smem_u32(bars + 2 * STAGES + 4); // ... the accumulator has been read
    const unsigned small0 = smem_u32(bars + 2 * STAGES + 6); // a segment's small products have been read
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(bars + 2 * STAGES + 7);

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int splits = gridDim.z;
    const int tok0 = blockIdx.y * BN, feat0 = blockIdx.x * p.tile_rows;
    const int my_segments = SEGMENTS / splits;
    const int first = (int)blockIdx.z * my_segments * p.blocks_per_segment;
    int n_blocks = my_segments * p.blocks_per_segment;
    if (n_blocks > p.blocks - first) n_blocks = p.blocks - first;
    if (n_blocks < 0) n_blocks = 0;

    ib_grid_dependency_launch();
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 4 + X_WARPS); }
        for (int s = 0; s < 2; ++s) { mbar_init(ready0 + 8 * s, 4 + X_WARPS); mbar_init(done0 + 8 * s, 1); mbar_init(taken0 + 8 * s, SUM_WARPS); }
        mbar_init(small0, SUM_WARPS);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const unsigned tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    bool ok = true;
    // A CTA's shared memory may be written by its cluster only once the CTA runs and, beyond 32 tokens, keeps nothing there
    // any more: every CTA says so and looks at the others' word just before its first store to them.
    if (splits > 1 && BN <= 32) cluster_arrive();

    const int q = warp & 3;                                  // the quarter of the 128 lanes that this warp may touch
    const int row = q * 32 + lane;

    if (warp == 0) {
        if (lane == 0) {
            // weights that no other CTA reads again leave the L2 cache first
            const unsigned long long pol = policy_evict_first();
            const unsigned stage_bytes = (unsigned)(p.tile_rows * KS * 4 + X_STAGE);
            auto load_w = [&](int t, int s) {
                const unsigned dst = smem_u32(w_ring + s * W_STAGE);
                const int k0 = first * BK + t * KS;          // beyond K: zeros
                if (gridDim.y == 1) tma_load_2d_hint(dst, &map_w, k0, feat0, full0 + 8 * s, pol);
                else tma_load_2d(dst, &map_w, k0, feat0, full0 + 8 * s);
            };
            auto load_x = [&](int t, int s) {
                tma_load_2d(smem_u32(x_ring + s * X_STAGE), &map_x, first * BK + t * KS, tok0, full0 + 8 * s);
            };
            const int n = 2 * n_blocks, head = n < STAGES ? n : STAGES;
            for (int t = 0; t < head; ++t) {                 // weights: no kernel writes them
                mbar_expect_tx(full0 + 8 * t, stage_bytes);
                load_w(t, t);
            }
            ib_grid_dependency_wait();
            for (int t = 0; t < head; ++t) load_x(t, t);
            for (int t = head; t < n; ++t) {
                const int s = t % STAGES;
                if (!mbar_wait(empty0 + 8 * s, ((t / STAGES) - 1) & 1, 1)) { ok = false; break; }
                mbar_expect_tx(full0 + 8 * s, stage_bytes);
                load_w(t, s);
                load_x(t, s);
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            const unsigned idesc1 = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(BN >> 3) << 17) | ((unsigned)(BM >> 4) << 24);
            const unsigned idesc2 = idesc1 + ((unsigned)(BN >> 3) << 17);        // two pieces of x side by side
            int m = 0, segment = 0;
            for (int i = 0; i < n_blocks; ++i) {
                const int s = i & 1;
                if (!mbar_wait(ready0 + 8 * s, (i >> 1) & 1, 2)) { ok = false; break; }
                if (i >= 2 && !mbar_wait(taken0 + 8 * s, ((i >> 1) - 1) & 1, 3)) { ok = false; break; }
                if (m == 0 && segment > 0 && !mbar_wait(small0, (segment - 1) & 1, 9)) { ok = false; break; }
                fence_after();
                const unsigned a = tmem + s * A_COLS, d = tmem + TMEM_ACC + s * BN, small = tmem + TMEM_SMALL;
                const unsigned long long b = desc_k_major(smem_u32(pieces + s * 3 * PIECE));
                // (a product waits for the one before it that adds to the same accumulator, for about 90 cycles whatever its
                // width: few wide ones, and the largest product's between the small ones')
#pragma unroll
                for (int k = 0; k < BK / 16; ++k) {
                    const unsigned a0 = a + k * 8, a1 = a0 + BK / 2, a2 = a1 + BK / 2;
                    const unsigned long long b0 = b + (unsigned long long)((k * 32) >> 4), b1 = b0 + (unsigned long long)(PIECE >> 4),
                                             b2 = b1 + (unsigned long long)(PIECE >> 4);
                    umma_ts(small, a0, b1, idesc2, (m | k) != 0);
                    umma_ts(d, a0, b0, idesc1, k != 0);
                    umma_ts(small, a1, b0, idesc2, 1);
                    umma_ts(small + BN, a2, b0, idesc1, 1);
                    umma_ts(small + BN, a1, b2, idesc1, 1);
                    umma_ts(small, a2, b1, idesc1, 1);
                }
                umma_commit(done0 + 8 * s);
                if (++m == p.blocks_per_segment) { m = 0; ++segment; }
            }
        }
    } else if (warp < 4 || warp >= SUM_WARP0 + SUM_WARPS) {
        const int part = warp < 4 ? warp - 2 : warp - (SUM_WARP0 + SUM_WARPS) + 2;
        const int r0 = ((lane >> 3) & 1) + ((lane >> 4) & 1) * 4 + (part & 1) * 2 + (part >> 1) * 8;
        for (int i = 0; i < n_blocks && ok; ++i) {
            const int b = i & 1;
            if (i >= 2 && !mbar_wait(done0 + 8 * b, ((i >> 1) - 1) & 1, 6)) ok = false;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int t = 2 * i + h, s = t % STAGES;
                if (ok && !mbar_wait(full0 + 8 * s, (t / STAGES) & 1, 7)) ok = false;
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                float4 v[BN / (4 * X_WARPS)];                // four numbers of a row at a time, all asked for together
                const int c = lane & 7;                      // (a warp's rows differ in bit 2: its stores meet all banks)
#pragma unroll
                for (int j = 0; j < BN / (4 * X_WARPS); ++j) {
                    const int r = r0 + j * 4 * X_WARPS;
                    v[j] = *reinterpret_cast<const float4*>(x_ring + s * X_STAGE + r * 128 + ((c ^ (r & 7)) << 4));
                }
#pragma unroll
                for (int j = 0; j < BN / (4 * X_WARPS); ++j) {
                    const int r = r0 + j * 4 * X_WARPS;
                    uint2 w0, w1, w2;
                    split_pair(v[j].x, v[j].y, w0.x, w1.x, w2.x);
                    split_pair(v[j].z, v[j].w, w0.y, w1.y, w2.y);
                    unsigned char* dst = pieces + b * 3 * PIECE + r * 128 + (((h * 4 + (c >> 1)) ^ (r & 7)) << 4) + (c & 1) * 8;
                    *reinterpret_cast<uint2*>(dst) = w0;
                    *reinterpret_cast<uint2*>(dst + PIECE) = w1;
                    *reinterpret_cast<uint2*>(dst + 2 * PIECE) = w2;
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(empty0 + 8 * s);
            }
            if (!ok) break;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the products read what was just written
            __syncwarp();
            if (lane == 0) mbar_arrive(ready0 + 8 * b);
        }
    } else if (warp < 8) {
        const bool busy = q * 32 < p.tile_rows;              // whole warps
        for (int i = 0; i < n_blocks && ok; ++i) {
            const int b = i & 1;
            if (i >= 2 && !mbar_wait(done0 + 8 * b, ((i >> 1) - 1) & 1, 4)) ok = false;   // the pieces are free again
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int t = 2 * i + h, s = t % STAGES;
                if (ok && !mbar_wait(full0 + 8 * s, (t / STAGES) & 1, 5)) ok = false;
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                if (busy) {
                    const unsigned char* src = w_ring + s * W_STAGE + row * 128;
                    unsigned p0[16], p1[16], p2[16];
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const float4 v = *reinterpret_cast<const float4*>(src + ((c ^ (row & 7)) << 4));
                        split_pair(v.x, v.y, p0[2 * c], p1[2 * c], p2[2 * c]);
                        split_pair(v.z, v.w, p0[2 * c + 1], p1[2 * c + 1], p2[2 * c + 1]);
                    }
                    if (h == 0) fence_after();
                    const unsigned dst = tmem + ((unsigned)(q * 32) << 16) + b * A_COLS + h * 16;
                    tmem_st16(dst, p0);
                    tmem_st16(dst + BK / 2, p1);
                    tmem_st16(dst + BK, p2);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(empty0 + 8 * s);
            }
            if (!ok) break;
            tmem_st_wait();
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(ready0 + 8 * b);
        }
    } else {
        ib_grid_dependency_wait();                           // y may still be read by the kernel before; x, if read again
        const int col0 = ((warp - SUM_WARP0) >> 2) * C;      // this warp's tokens
        const unsigned lanes = tmem + ((unsigned)(q * 32) << 16) + col0;
        const int feature = feat0 + row;
        Waiting<C> waiting;
        waiting.tmem = lanes + TMEM_WAITING;
        waiting.pairs = recv + col0 * BM + row;
        float sum[C];
        auto add = [&](unsigned at) {
            if constexpr (C == 16) {
                float v[16];
                tmem_ld16(at, v);
#pragma unroll
                for (int j = 0; j < 16; ++j) sum[j] += v[j];
            } else {
                unsigned v[32];
                tmem_ld32_issue(at, v);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 32; ++j) sum[j] += __uint_as_float(v[j]);
            }
        };
        int i = 0;
        for (int g = 0; g < my_segments && ok; ++g) {
#pragma unroll
            for (int j = 0; j < C; ++j) sum[j] = 0.0f;
            for (int m = 0; m < p.blocks_per_segment && i < n_blocks; ++m, ++i) {
                const int b = i & 1;
                ok = mbar_wait(done0 + 8 * b, (i >> 1) & 1, 8);
                ok = __all_sync(0xffffffffu, ok);            // one answer per warp: the loads below are warp-wide
                if (!ok) break;
                fence_after();
                if (m == p.blocks_per_segment - 1 || i == n_blocks - 1) {   // the segment's last: its small products join once
#pragma unroll
                    for (int h = 0; h < C; h += 16) {
                        float v[16], u[16];
                        tmem_ld16(lanes + TMEM_SMALL + BN + h, v);
                        tmem_ld16(lanes + TMEM_SMALL + h, u);
#pragma unroll
                        for (int j = 0; j < 16; ++j) sum[h + j] += v[j] + u[j];
                    }
                    fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(small0);
                }
                add(lanes + TMEM_ACC + b * BN);
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(taken0 + 8 * b);
            }
            if (ok) waiting.join(sum, g, g == my_segments - 1);
        }
        if (splits == 1) {
            if (ok && row < p.tile_rows && feature < p.n_out) {
                float* y = p.y + (long)(tok0 + col0) * p.ldy + feature;
#pragma unroll
                for (int j = 0; j < C; ++j, y += p.ldy)
                    if (tok0 + col0 + j < p.n_tok) *y = finished(p, sum[j], tok0 + col0 + j, feature);
            }
        } else {
            // every CTA of the cluster owns an equal share of the tile's rows: its neighbours' branches of the sums come
            // straight into its shared memory, one cluster barrier follows, and it adds them up and stores
            const int owned = p.tile_rows / splits;
            const unsigned my_rank = cluster_rank();
            if (BN > 32) cluster_arrive();
            cluster_wait();
            if (ok && row < p.tile_rows) {
                const unsigned owner = (unsigned)(row / owned);
                float* slot = recv + ((size_t)my_rank * BN + col0) * owned + (row - (int)owner * owned);
#pragma unroll
                for (int j = 0; j < C; ++j)
                    if (tok0 + col0 + j < p.n_tok) st_cluster(smem_u32(slot + j * owned), owner, sum[j]);
            }
            cluster_arrive();
            cluster_wait();
            if (ok && g_error == 0) {
                const int per = BN * owned;
                for (int idx = (int)threadIdx.x - 32 * SUM_WARP0; idx < per; idx += 32 * SUM_WARPS) {
                    const int tok = tok0 + idx / owned, f = feat0 + (int)my_rank * owned + idx % owned;
                    if (tok >= p.n_tok || f >= p.n_out) continue;
                    const float* part = recv + idx;
                    float v;
                    if (splits == 2) v = part[0] + part[per];
                    else if (splits == 4) v = (part[0] + part[per]) + (part[2 * per] + part[3 * per]);
                    else v = ((part[0] + part[per]) + (part[2 * per] + part[3 * per])) +
                             ((part[4 * per] + part[5 * per]) + (part[6 * per] + part[7 * per]));
                    p.y[(long)tok * p.ldy + f] = finished(p, v, tok, f);
                }
            }
        }
    }
    if (splits > 1 && (warp < SUM_WARP0 || warp >= SUM_WARP0 + SUM_WARPS)) {      // the other warps' part in the cluster's two barriers
        if (BN > 32) cluster_arrive();
        cluster_wait();
        cluster_arrive();
        cluster_wait();
    }

    if (!ok) {   // a wait of this CTA ran out: copies still in flight get time to land before it leaves
        const unsigned long long t0 = global_ns();
        while (global_ns() - t0 < 2000000ull) __nanosleep(1000);
    }
    fence_before();
    __syncthreads();
    if (warp == 1) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

// a row-major float32 matrix [rows, k] with row stride ld (numbers), boxes of [box_rows, 32]
static bool make_map(CUtensorMap* map, const void* base, long rows, long k, long ld, int box_rows) {
    EncodeTiled enc = encode_fn();
    if (enc == nullptr) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
    const cuuint32_t box[2] = {(cuuint32_t)KS, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, elem,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN, int STAGES>
static int launch(const CUtensorMap& mw, const CUtensorMap& mx, const Params& p, int splits, cudaStream_t stream) {
    static IbDeviceSet allowed;
    constexpr size_t smem = smem_bytes<BN, STAGES>();
    static_assert(smem <= (BN <= 16 ? 113 : 227) * 1024, "");
    if (const int e = ib_allow_dynamic_smem(allowed, split_kernel<BN, STAGES>, smem)) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((p.n_out + p.tile_rows - 1) / p.tile_rows, (p.n_tok + BN - 1) / BN, splits);
    cfg.blockDim = dim3(threads_of(BN));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = splits;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ib_pdl_enabled ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, split_kernel<BN, STAGES>, mw, mx, p);
    return e == cudaSuccess ? ib_launch_status() : (int)e;
}

// How a product is cut: CTAs per tile and rows of W per tile.
struct Cut { int splits, tile_rows; };

static Cut choose_cut(int n_tok, int n_out, int blocks, int bn) {
    const long tiles = (long)((n_out + BM - 1) / BM) * ((n_tok + bn - 1) / bn);
    // CTAs that run at a time, per CTA of an SM (clusters want their SMs in one part of the chip: fewer with larger ones)
    const int resident[4] = {148, 148, 136, 120};            // splits 1, 2, 4, 8
    if (bn <= 16) {
        // as many parts as the GPU holds at once, two CTAs an SM (1 to 16 tokens, us: 1,024 features over 2,048 eight 8.0, four
        // 10.1; over 3,072 9.9; 6,144 over 1,024 four 10.9, eight 14.2; lower tiles, so that more SMs have one, lose: 1,024
        // over 3,072 in 128 / 96 / 32 rows 9.9 / 10.3 / 11.7)
        for (int l = 3; l > 0; --l)
            if (tiles << l <= 2 * (resident[l] + 12)) return {1 << l, BM};
        return {1, BM};
    }
    // else the time of the fullest SM, us: its blocks, and what a wave of CTAs pays at its ends (least where the segments are
    // shared by eight: none is added to another by the CTA itself).  Fitted to 32 to 2,048 rows of 4,096 and 6,144
    // features over 1,024, of 1,024 over 2,048 and 3,072 in 1 / 2 / 4 / 8 parts: 64 tiles over 1,024 21.7 / 18.2 / 23.0 /
    // 40.4, over 3,072 52.7 / 33.1 / 38.1 / 59.9; 192 tiles over 1,024 44.6 / 53.6 / 68.0 / 106.8; 8 tiles over 2,048 36.4 / 24.3 /
    // 14.2 / 10.0
    const float ends[4] = {6.5f, 9.8f, 7.5f, 5.0f};
    Cut best = {1, BM};
    float least = 0.0f;
    for (int l = 0; l < 4; ++l) {
        const long waves = ((tiles << l) + resident[l] - 1) / resident[l];
        const float t = waves * ((float)((blocks + (1 << l) - 1) >> l) * 0.93f + ends[l]);
        if (l == 0 || t < least) { least = t; best.splits = 1 << l; }
    }
    return best;
}

}  // namespace split3

int ib_pdl_enabled = 0;
IB_EXPORT void ib_gemm_split_set_pdl(int on) { ib_pdl_enabled = on; }

// x [n_tok, k] (row stride ldx), w [n_out, k] (row stride ldw), y [n_tok, n_out] (row stride ldy), all float32.
// IB_ERR_UNSUPPORTED: rows that do not start on 16 bytes.  splits and tile_rows: 0 lets the function choose.
IB_EXPORT int ib_gemm_tn_split(const float* x, long ldx, const float* w, long ldw, float* y, long ldy, int n_tok, int n_out,
                               int k, int splits, int tile_rows, cudaStream_t stream) {
    if (n_tok <= 0 || n_out <= 0) return IB_OK;
    if (k <= 0) return IB_ERR_ARGUMENT;
    if ((ldx % 4) || (ldw % 4) || ((uintptr_t)x % 16) || ((uintptr_t)w % 16)) return IB_ERR_UNSUPPORTED;
    split3::Params p;
    p.x = x; p.w = w; p.y = y; p.ldx = ldx; p.ldw = ldw; p.ldy = ldy;
    p.n_tok = n_tok; p.n_out = n_out; p.k = k;
    p.blocks = (k + split3::BK - 1) / split3::BK;
    p.blocks_per_segment = (p.blocks + split3::SEGMENTS - 1) / split3::SEGMENTS;
    const int bn = n_tok <= 16 ? 16 : n_tok <= 32 ? 32 : 64;
    if ((n_tok + bn - 1) / bn > 65535) return IB_ERR_UNSUPPORTED;
    const split3::Cut cut = split3::choose_cut(n_tok, n_out, p.blocks, bn);
    if (splits == 0) { splits = cut.splits; if (tile_rows == 0) tile_rows = cut.tile_rows; }
    if (tile_rows == 0) tile_rows = split3::BM;
    if ((splits != 1 && splits != 2 && splits != 4 && splits != 8) || tile_rows < 8 || tile_rows > split3::BM || tile_rows % 8)
        return IB_ERR_ARGUMENT;
    p.tile_rows = tile_rows;
    CUtensorMap mw, mx;
    if (!split3::make_map(&mw, w, n_out, k, ldw, tile_rows) || !split3::make_map(&mx, x, n_tok, k, ldx, bn)) return IB_ERR_UNSUPPORTED;
    switch (bn) {
        case 16: return split3::launch<16, 5>(mw, mx, p, splits, stream);
        case 32: return split3::launch<32, 8>(mw, mx, p, splits, stream);
        default: return split3::launch<64, 6>(mw, mx, p, splits, stream);
    }
}

// The error word of the kernels above: 0, or the code of the first wait that ran out.  Reading it synchronises with the
// device; `reset` clears it.
IB_EXPORT int ib_gemm_split_error(int reset) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, split3::g_error, sizeof(int)) != cudaSuccess) return -1;
    if (reset && v != 0) {
        const int zero = 0;
        cudaMemcpyToSymbol(split3::g_error, &zero, sizeof(int));
    }
    return v;
}
IB_EXPORT int ib_gemm_split_error_async(int* out, cudaStream_t stream) {
    return (int)cudaMemcpyFromSymbolAsync(out, split3::g_error, sizeof(int), 0, cudaMemcpyDeviceToHost, stream);
}
