// y[n, m] = sum_k x[n, k] * w[m, k]   (weights stored [out, in], no bias)
//
// Plain fused multiply-adds: no tensor cores, no reduced-precision mode.  Every output element is one chain of fused
// multiply-adds over k in ascending order, in every kernel below, so its value does not depend on how many rows the
// batch has, where the row stands in it or which kernel took it.  This is the matrix product of the true 32-bit path;
// with other element types it also serves 32-bit weights met by bfloat16 activations.
//
// Two kernels:
//   * tiles: BM x BN outputs per CTA, TM x TN per thread, k in blocks of 16 through two shared buffers stored
//     transposed, so that a thread's operands of one k are 16-byte reads.  Bound by the multiply-adds; two rows'
//     chains go through one packed instruction (fma.rn.f32x2), which rounds each half as fmaf does.
//   * rows: up to 32 rows.  Bound by streaming w (and, for few outputs, by the chain itself: four cycles per k).  A ring
//     of cp.async stages keeps w's bytes in flight, the first of them asked for before the kernel before this one
//     has ended; a thread owns one output feature and up to eight rows.
#include "common.cuh"

namespace simt {

template <typename T> __device__ __forceinline__ void load4(const T* p, float* v);
template <> __device__ __forceinline__ void load4<float>(const float* p, float* v) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
template <> __device__ __forceinline__ void load4<__nv_bfloat16>(const __nv_bfloat16* p, float* v) {
    const uint2 t = *reinterpret_cast<const uint2*>(p);
    v[0] = __uint_as_float(t.x << 16); v[1] = __uint_as_float(t.x & 0xffff0000u);
    v[2] = __uint_as_float(t.y << 16); v[3] = __uint_as_float(t.y & 0xffff0000u);
}

__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ void fma2(unsigned long long& c, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}

constexpr int BK = 16, DEPTH = 2;

// Four k of ROWS rows from row0 on, this thread's share: registers, zeros beyond the matrix.
template <typename T, int ROWS, int NT, bool VEC>
__device__ __forceinline__ void fetch(const T* __restrict__ src, long ld, int row0, int n, int k0, int k_dim,
                                      float (*v)[4]) {
#pragma unroll
    for (int i = 0; i < ROWS * 4 / NT; ++i) {
        const int idx = threadIdx.x + i * NT, r = row0 + (idx >> 2), k = k0 + (idx & 3) * 4;
        const T* p = src + (long)r * ld + k;
        if (VEC) {                                      // k_dim is a multiple of 4
            v[i][0] = v[i][1] = v[i][2] = v[i][3] = 0.0f;
            if (r < n && k < k_dim) load4<T>(p, v[i]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) v[i][j] = (r < n && k + j < k_dim) ? ib_to_float(p[j]) : 0.0f;
        }
    }
}

// ... to shared memory as [k][row]; the row's place is turned by eight per group of four k, so that the 32 lanes of a
// store (eight rows, four groups) meet 32 banks.
template <int ROWS, int NT>
__device__ __forceinline__ void stash(float* dst, const float (*v)[4]) {
#pragma unroll
    for (int i = 0; i < ROWS * 4 / NT; ++i) {
        const int idx = threadIdx.x + i * NT, r = idx >> 2, g = idx & 3;
#pragma unroll
        for (int j = 0; j < 4; ++j) dst[(g * 4 + j) * ROWS + (r ^ (g * 8))] = v[i][j];
    }
}

template <typename XT, typename WT, typename OT, int BM, int BN, int TM, int TN, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN)) tiles_kernel(
    const XT* __restrict__ x, const WT* __restrict__ w, OT* __restrict__ y, int n_rows, int n_out, int k_dim, long ldx,
    long ldw, long ldy, long bx, long bw, long by, int vec_y) {
    constexpr int NX = BN / TN, NT = (BM / TM) * NX;    // threads along the outputs, threads
    static_assert(TM % 4 == 0 && TN % 4 == 0 && BM * 4 % NT == 0 && BN * 4 % NT == 0 && BM % 32 == 0 && BN % 32 == 0, "");
    __shared__ __align__(16) float xs[2][BK * BM];
    __shared__ __align__(16) float ws[2][BK * BN];
    // blockIdx.z numbers the products of a batch: operand b starts bx, bw, by elements after operand b - 1
    x += (long)blockIdx.z * bx;
    w += (long)blockIdx.z * bw;
    y += (long)blockIdx.z * by;
    const int tx = threadIdx.x % NX, ty = threadIdx.x / NX;
    const int row0 = blockIdx.y * BM, col0 = blockIdx.x * BN;
    unsigned long long acc[TM / 2][TN];
#pragma unroll
    for (int i = 0; i < TM / 2; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;

    // blocks 1 .. DEPTH of k on their way in registers while block 0 is worked on
    float xv[DEPTH][BM * 4 / NT][4], wv[DEPTH][BN * 4 / NT][4];
    fetch<XT, BM, NT, VEC>(x, ldx, row0, n_rows, 0, k_dim, xv[0]);
    fetch<WT, BN, NT, VEC>(w, ldw, col0, n_out, 0, k_dim, wv[0]);
    stash<BM, NT>(xs[0], xv[0]);
    stash<BN, NT>(ws[0], wv[0]);
#pragma unroll
    for (int d = 0; d < DEPTH; ++d) {
        fetch<XT, BM, NT, VEC>(x, ldx, row0, n_rows, (d + 1) * BK, k_dim, xv[d]);
        fetch<WT, BN, NT, VEC>(w, ldw, col0, n_out, (d + 1) * BK, k_dim, wv[d]);
    }
    __syncthreads();
    for (int base = 0; base < k_dim; base += DEPTH * BK) {
#pragma unroll
        for (int d = 0; d < DEPTH; ++d) {           // DEPTH is even: buffer and registers are known per d
            const int k0 = base + d * BK;
            if (k0 >= k_dim) break;
            if (k0 + BK < k_dim) {                  // into the buffer that every thread left before the last barrier
                stash<BM, NT>(xs[(d & 1) ^ 1], xv[d]);
                stash<BN, NT>(ws[(d & 1) ^ 1], wv[d]);
                fetch<XT, BM, NT, VEC>(x, ldx, row0, n_rows, k0 + (DEPTH + 1) * BK, k_dim, xv[d]);
                fetch<WT, BN, NT, VEC>(w, ldw, col0, n_out, k0 + (DEPTH + 1) * BK, k_dim, wv[d]);
            }
#pragma unroll
            for (int kk = 0; kk < BK; ++kk) {
                const float* xr = xs[d & 1] + kk * BM;
                const float* wr = ws[d & 1] + kk * BN;
                unsigned long long a[TM / 2], b[TN];
#pragma unroll
                for (int i = 0; i < TM / 4; ++i) {
                    const ulonglong2 t =
                        *reinterpret_cast<const ulonglong2*>(xr + ((i * (BM / (TM / 4)) + ty * 4) ^ ((kk >> 2) * 8)));
                    a[2 * i] = t.x; a[2 * i + 1] = t.y;
                }
#pragma unroll
                for (int j = 0; j < TN / 4; ++j) {
                    const float4 t =
                        *reinterpret_cast<const float4*>(wr + ((j * (BN / (TN / 4)) + tx * 4) ^ ((kk >> 2) * 8)));
                    b[4 * j] = pack2(t.x, t.x); b[4 * j + 1] = pack2(t.y, t.y);
                    b[4 * j + 2] = pack2(t.z, t.z); b[4 * j + 3] = pack2(t.w, t.w);
                }
#pragma unroll
                for (int i = 0; i < TM / 2; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) fma2(acc[i][j], a[i], b[j]);
            }
            __syncthreads();
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gr = row0 + (i / 4) * (BM / (TM / 4)) + ty * 4 + (i & 3);
        if (gr >= n_rows) continue;
#pragma unroll
        for (int j = 0; j < TN / 4; ++j) {
            const int gc = col0 + j * (BN / (TN / 4)) + tx * 4;
            float v[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                float lo, hi;
                unpack2(acc[i / 2][4 * j + c], lo, hi);
                v[c] = (i & 1) ? hi : lo;
            }
            OT* dst = y + (long)gr * ldy + gc;
            if (sizeof(OT) == 4 && vec_y && gc + 3 < n_out) {
                *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (gc + c < n_out) dst[c] = ib_from_float<OT>(v[c]);
            }
        }
    }
}

__device__ __forceinline__ void copy16(float* dst, const float* src, bool there) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(there ? 16 : 0) : "memory");
}

// RT rows (n_rows of them real) times FT features per CTA, RPT rows and one feature per thread, a ring of STAGES with
// KT k each.  Rows of a stage lie KT + 4 floats apart: eight lanes that read 16 bytes of eight features meet 32 banks.
// A thread's chain takes four cycles per k, so its operands are read from shared memory AHEAD groups of four k early.
constexpr int ROWS_THREADS = 128, AHEAD = 4;

template <int RT, int FT, int RPT, int KT, int STAGES>
__global__ void __launch_bounds__(ROWS_THREADS) rows_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                            float* __restrict__ y, int n_rows, int n_out, int k_dim,
                                                            long ldx, long ldw, long ldy, long bx, long bw, long by) {
    constexpr int LD = KT + 4, NG = KT / (4 * AHEAD);
    static_assert(FT * RT / RPT <= ROWS_THREADS && KT % (4 * AHEAD) == 0, "");
    extern __shared__ __align__(16) float ring[];       // STAGES of (FT features, then RT rows)
    x += (long)blockIdx.z * bx;
    w += (long)blockIdx.z * bw;
    y += (long)blockIdx.z * by;
    const int f0 = blockIdx.x * FT, tid = threadIdx.x;
    const int n_stages = (k_dim + KT - 1) / KT;
    auto fetch_w = [&](int s) {
        float* dst = ring + (s % STAGES) * (FT + RT) * LD;
#pragma unroll 4
        for (int i = tid; i < FT * (KT / 4); i += ROWS_THREADS) {
            const int r = i / (KT / 4), k = s * KT + (i % (KT / 4)) * 4;
            const bool there = f0 + r < n_out && k < k_dim;
            copy16(dst + r * LD + (i % (KT / 4)) * 4, there ? w + (long)(f0 + r) * ldw + k : w, there);
        }
    };
    auto fetch_x = [&](int s) {
        float* dst = ring + ((s % STAGES) * (FT + RT) + FT) * LD;
#pragma unroll 4
        for (int i = tid; i < RT * (KT / 4); i += ROWS_THREADS) {
            const int r = i / (KT / 4), k = s * KT + (i % (KT / 4)) * 4;
            const bool there = r < n_rows && k < k_dim;
            copy16(dst + r * LD + (i % (KT / 4)) * 4, there ? x + (long)r * ldx + k : x, there);
        }
    };
    ib_grid_dependency_launch();
    for (int s = 0; s < STAGES - 1 && s < n_stages; ++s) fetch_w(s);        // weights: no kernel writes them
    ib_grid_dependency_wait();
    for (int s = 0; s < STAGES - 1 && s < n_stages; ++s) fetch_x(s);
    asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
    for (int s = 1; s < STAGES - 1; ++s) asm volatile("cp.async.commit_group;" ::: "memory");

    const int f = tid % FT, g = tid / FT;
    const bool busy = g * RPT < RT;
    float acc[RPT];
#pragma unroll
    for (int r = 0; r < RPT; ++r) acc[r] = 0.0f;
    for (int s = 0; s < n_stages; ++s) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();                                // stage s is there, and everyone has left stage s - 1
        if (s + STAGES - 1 < n_stages) { fetch_w(s + STAGES - 1); fetch_x(s + STAGES - 1); }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (!busy) continue;
        const float* wr = ring + ((s % STAGES) * (FT + RT) + f) * LD;
        const float* xr = ring + ((s % STAGES) * (FT + RT) + FT + g * RPT) * LD;
        float4 b[2][AHEAD], a[2][RPT][AHEAD];
        auto read = [&](int n, int buf) {
#pragma unroll
            for (int q = 0; q < AHEAD; ++q) {
                b[buf][q] = *reinterpret_cast<const float4*>(wr + (n * AHEAD + q) * 4);
#pragma unroll
                for (int r = 0; r < RPT; ++r)
                    a[buf][r][q] = *reinterpret_cast<const float4*>(xr + r * LD + (n * AHEAD + q) * 4);
            }
        };
        read(0, 0);
#pragma unroll
        for (int n = 0; n < NG; ++n) {                  // beyond k_dim: zeros
            if (n + 1 < NG) read(n + 1, (n + 1) & 1);
#pragma unroll
            for (int q = 0; q < AHEAD; ++q) {
                const float4 v = b[n & 1][q];
#pragma unroll
                for (int r = 0; r < RPT; ++r) acc[r] = fmaf(a[n & 1][r][q].x, v.x, acc[r]);
#pragma unroll
                for (int r = 0; r < RPT; ++r) acc[r] = fmaf(a[n & 1][r][q].y, v.y, acc[r]);
#pragma unroll
                for (int r = 0; r < RPT; ++r) acc[r] = fmaf(a[n & 1][r][q].z, v.z, acc[r]);
#pragma unroll
                for (int r = 0; r < RPT; ++r) acc[r] = fmaf(a[n & 1][r][q].w, v.w, acc[r]);
            }
        }
    }
    if (!busy || f0 + f >= n_out) return;
#pragma unroll
    for (int r = 0; r < RPT; ++r)
        if (g * RPT + r < n_rows) y[(long)(g * RPT + r) * ldy + f0 + f] = acc[r];
}

struct Product {
    const void* x;
    const void* w;
    void* y;
    int n_rows, n_out, k_dim;
    long ldx, ldw, ldy;
    int batch;
    long bx, bw, by;
    cudaStream_t stream;
};

template <typename XT, typename WT, typename OT, int BM, int BN, int TM, int TN, bool VEC>
static int launch_tiles(const Product& p) {
    const dim3 grid((p.n_out + BN - 1) / BN, (p.n_rows + BM - 1) / BM, p.batch);
    const int vec_y = sizeof(OT) == 4 && p.ldy % 4 == 0 && p.by % 4 == 0 && (uintptr_t)p.y % 16 == 0;
    // Launched the plain way: CTAs that come while the kernel before them still holds SMs would crowd on the others (403
    // rows: 325 us for a product that takes 140 on a free machine).
    tiles_kernel<XT, WT, OT, BM, BN, TM, TN, VEC><<<grid, (BM / TM) * (BN / TN), 0, p.stream>>>(
        (const XT*)p.x, (const WT*)p.w, (OT*)p.y, p.n_rows, p.n_out, p.k_dim, p.ldx, p.ldw, p.ldy, p.bx, p.bw, p.by, vec_y);
    return ib_launch_status();
}

template <int RT, int FT, int RPT, int KT, int STAGES>
static int launch_rows(const Product& p) {
    static IbDeviceSet allowed;
    constexpr size_t SM_BYTES = 228 * 1024, most = SM_BYTES / 2;
    static_assert(STAGES * (FT + RT) * (KT + 4) * sizeof(float) <= most, "");
    if (const int e = ib_allow_dynamic_smem(allowed, rows_kernel<RT, FT, RPT, KT, STAGES>, most)) return e;
    const dim3 grid((p.n_out + FT - 1) / FT, 1, p.batch);
    // A CTA asks for so much shared memory that no SM takes more CTAs than the fullest one has to: those that come before
    // the kernel ahead has left its SMs would crowd on the free ones otherwise.
    const size_t share = SM_BYTES / ((size_t)((grid.x * (long)grid.z + 147) / 148) + 1);
    size_t smem = (size_t)STAGES * (FT + RT) * (KT + 4) * sizeof(float);
    if (smem < share) smem = share;
    ib_launch(rows_kernel<RT, FT, RPT, KT, STAGES>, grid, ROWS_THREADS, smem, p.stream, (const float*)p.x, (const float*)p.w,
              (float*)p.y, p.n_rows, p.n_out, p.k_dim, p.ldx, p.ldw, p.ldy, p.bx, p.bw, p.by);
    return ib_launch_status();
}

// How the work is cut.  Times on a B200 with cold weights, launch included (a launch of next to nothing: 6 us).
//   * Up to 32 rows of float32 whose rows start on 16 bytes: rows_kernel.  Few features per CTA where the product has
//     few, so that every SM streams; more where it has many, so that x is fetched less often and a thread takes
//     several rows per read of w (4 rows, K 1,024: 1,024 features 8 a CTA; 4,096: 14 us with 16, 18 with 32 and four rows a
//     thread; 151,936: 127 us with 32 and two rows a thread, 177 with 8: 4.9 TB/s; tiles 41 and 301 us).  At 32 rows and
//     many features the tiles are ahead (315 against 397 us).
//   * Else tiles of 64 x 64 (8 x 4 a thread), or of 32 x 64 (4 x 4) where those leave SMs idle.  CTAs on the fullest SM and
//     the measured time of 1,024 k: 64 x 64 about 15 + 25 a CTA, 32 x 64 about 8 + 19 a CTA and not below 35.  403 rows:
//     4,096 x 1,024 113 us, 6,144 x 1,024 140 us (36 TFLOP/s), 1,024 x 3,072 121 us; before, with one 64 x 64 kernel of
//     4 x 4 a thread and nothing in flight, 242, 283 and 511 us.  2,048 rows: 48 TFLOP/s.
static int launch_f32(const Product& p) {
    const bool vec = p.k_dim % 4 == 0 && p.ldx % 4 == 0 && p.ldw % 4 == 0 && p.bx % 4 == 0 && p.bw % 4 == 0 &&
                     (uintptr_t)p.x % 16 == 0 && (uintptr_t)p.w % 16 == 0;
    if (!vec) return launch_tiles<float, float, float, 64, 64, 8, 4, false>(p);
    const long features = (long)p.n_out * p.batch;
    const int size = features < 2048 ? 0 : features < 32768 ? 1 : 2;
    if (p.n_rows <= 4 && size == 1) return launch_rows<4, 16, 1, 128, 4>(p);
    if (p.n_rows <= 4 && size == 2) return launch_rows<4, 32, 2, 128, 3>(p);
    if (p.n_rows <= 8 && size == 0) return launch_rows<8, 8, 1, 256, 3>(p);
    if (p.n_rows <= 8 && size == 1) return launch_rows<8, 16, 2, 128, 4>(p);
    if (p.n_rows <= 8) return launch_rows<8, 32, 4, 64, 4>(p);
    if (p.n_rows <= 16 && size == 0) return launch_rows<16, 8, 1, 128, 4>(p);
    if (p.n_rows <= 16 && size == 1) return launch_rows<16, 16, 2, 128, 4>(p);
    if (p.n_rows <= 16) return launch_rows<16, 64, 8, 64, 3>(p);
    if (p.n_rows <= 32 && size == 0) return launch_rows<32, 8, 2, 128, 4>(p);
    if (p.n_rows <= 32 && size == 1) return launch_rows<32, 16, 4, 128, 3>(p);
    constexpr long SMS = 148;
    const long across = (p.n_out + 63) / 64 * (long)p.batch;
    const long per64 = (across * ((p.n_rows + 63) / 64) + SMS - 1) / SMS;
    const long per32 = (across * ((p.n_rows + 31) / 32) + SMS - 1) / SMS;
    const long t32 = 8 + 19 * per32;
    return (t32 > 35 ? t32 : 35) < 15 + 25 * per64 ? launch_tiles<float, float, float, 32, 64, 4, 4, true>(p)
                                                   : launch_tiles<float, float, float, 64, 64, 8, 4, true>(p);
}

template <typename XT, typename WT, typename OT>
static int launch_mixed(const Product& p) {
    const bool vec = p.k_dim % 4 == 0 && p.ldx % 4 == 0 && p.ldw % 4 == 0 && p.bx % 4 == 0 && p.bw % 4 == 0 &&
                     (uintptr_t)p.x % (4 * sizeof(XT)) == 0 && (uintptr_t)p.w % (4 * sizeof(WT)) == 0;
    // Rows that do not start on whole loads come number by number: threads are what such a product lacks, so its tiles are low
    // (bfloat16, 1,001 features over 1,023, 64 rows: 64 x 64 98 us, 32 x 64 46).
    return vec ? launch_tiles<XT, WT, OT, 64, 64, 8, 4, true>(p) : launch_tiles<XT, WT, OT, 32, 64, 4, 4, false>(p);
}

static int launch(const Product& p, int x_is_f32, int w_is_f32, int y_is_f32) {
    if (x_is_f32 && w_is_f32 && y_is_f32) return launch_f32(p);
#if IB_ACT_BF16
    if (!x_is_f32 && !w_is_f32 && !y_is_f32) return launch_mixed<act_t, __nv_bfloat16, act_t>(p);
    if (!x_is_f32 && !w_is_f32 && y_is_f32) return launch_mixed<act_t, __nv_bfloat16, float>(p);
    if (!x_is_f32 && w_is_f32 && !y_is_f32) return launch_mixed<act_t, float, act_t>(p);
    if (!x_is_f32 && w_is_f32 && y_is_f32) return launch_mixed<act_t, float, float>(p);
    if (x_is_f32 && w_is_f32 && !y_is_f32) return launch_mixed<float, float, act_t>(p);
#endif
    return IB_ERR_UNSUPPORTED;
}

}  // namespace simt

// x is act_t or float (x_is_f32), w is bfloat16 or float (w_is_f32), y is act_t or float (y_is_f32).
IB_EXPORT int ib_gemm_tn_simt(const void* x, int x_is_f32, const void* w, int w_is_f32, void* y, int y_is_f32,
                              int n_rows, int n_out, int k_dim, long ldx, long ldw, long ldy, cudaStream_t stream) {
    if (n_rows <= 0 || n_out <= 0) return IB_OK;
    if (k_dim <= 0) return IB_ERR_ARGUMENT;
    const simt::Product p = {x, w, y, n_rows, n_out, k_dim, ldx, ldw, ldy, 1, 0, 0, 0, stream};
    return simt::launch(p, x_is_f32, w_is_f32, y_is_f32);
}

// A batch of such products, y_b = x_b w_b^T for b < batch: operand b starts bx, bw, by elements after operand b - 1
// (so the heads of one activation tensor, or of one weight tensor, are multiplied in place).
IB_EXPORT int ib_gemm_tn_simt_batched(const void* x, int x_is_f32, const void* w, int w_is_f32, void* y, int y_is_f32,
                                      int n_rows, int n_out, int k_dim, long ldx, long ldw, long ldy, int batch, long bx,
                                      long bw, long by, cudaStream_t stream) {
    if (n_rows <= 0 || n_out <= 0 || batch <= 0) return IB_OK;
    if (k_dim <= 0 || batch > 65535) return IB_ERR_ARGUMENT;
    const simt::Product p = {x, w, y, n_rows, n_out, k_dim, ldx, ldw, ldy, batch, bx, bw, by, stream};
    return simt::launch(p, x_is_f32, w_is_f32, y_is_f32);
}
