// exp(M) phi of every walker by the dynamicOrder Taylor series
// (LogHop2isSD2isOperation::applyToRight, logHop2isSD2isOperation.cpp:38-45,
// 159-195), FP64, one kernel for the whole series and, where asked, the
// one-body product that follows it.
//
// A CTA holds 16 columns (24 where that is all the walker has) of one walker
// and all n rows: the current term in
// shared memory (the right operand of the next order), the running sum in
// the registers that also define the accumulator layout (a warp owns 16 rows
// and all columns).  M is streamed through three or four cp.async stages of 8
// columns, once per order; the walkers in flight (148 SMs times n^2 16 bytes per
// walker, 39 MB at n = 128) stay in L2, so memory sees M once.  The CTAs of one
// walker form a cluster: the stopping test is the walker's largest term, so
// each order from `checkFrom` on ends with one exchange of maxima over
// distributed shared memory.
//
// Bound: the FP64 matrix rate.  Per order 8 n^2 N flops per walker against
// n^2 16 bytes of M from L2 (16 bytes per cycle and SM at n = 256, 8 at 128) and
// 32 bytes per cycle and SM of fragment loads, both far below their limits.
// Phase times, series and one-body product, one GEMM and one accumulation launch per
// order up to the cap against this: n = 128, N = 32, 2048 walkers 7.44 and 2.49 ms
// (23.6 TFLOP/s at a mean order of 6.35, the matrix pipe busy 66 % of the time);
// n = 64, N = 16, 512 walkers 0.761 and 0.109; n = 90, N = 21, 300 walkers 1.17 and
// 0.269; n = 256, N = 64, 512 walkers 7.37 and 5.83.  These read the panels of a
// symmetric M: the mirrored rows cost loads here (n = 256 with a full M 5.59 against
// 6.01 then), and the M-build that writes the panels has half the products (2.87 ->
// 1.40, 0.117 -> 0.058, 0.123 -> 0.075, 5.68 -> 2.64 ms).
#include <cooperative_groups.h>
#include <math_constants.h>

#include <algorithm>
#include <atomic>

#include "dmma.cuh"
#include "once.cuh"
#include "taylor_f64.cuh"

namespace cg = cooperative_groups;

extern std::atomic<long long> g_launch_count;

namespace {

constexpr int TF_COLS = 16;      // columns of phi per CTA (8 NJ, NJ = 2; 24 for a walker of 17..24)
constexpr int TF_BK = 8;         // columns of M per stage
constexpr int TF_MAXN = 256;     // 16 rows per warp, 16 warps
constexpr int TF_MAXCL = 8;      // CTAs per walker (portable cluster size)

__host__ __device__ constexpr int tf_rows(int n) { return (n + 15) / 16 * 16; }
// leading dimensions (elements) that keep fragment loads conflict-free: rows
// contiguous 2 mod 8 (complex) or 4 mod 16 (real); contraction contiguous 4 mod 8
__host__ __device__ constexpr int tf_lda(int n) { return tf_rows(n) + 2; }
__host__ __device__ constexpr int tf_ldt(int n) { return tf_rows(n) + 4; }
__host__ __device__ constexpr size_t tf_stage(int n) { return (size_t)TF_BK * tf_lda(n) * sizeof(zd); }
__host__ __device__ constexpr size_t tf_smem(int n, int stages, int cols)
{
    return stages * tf_stage(n) + (size_t)cols * tf_ldt(n) * sizeof(zd);
}

template <int NJ>
struct TfAcc {
    double r[2][NJ][2], i[2][NJ][2];   // 8-row block, 8-column block, column parity
};

// One n x n matrix times the term in shared memory, accumulated into c.  The
// stream of M stages is cyclic: stage `it` of the stream is tile it % KT, so
// that the next order's first tiles are already on their way at an order's
// end.  REAL: the matrix is real (its tile is 8-byte elements, leading
// dimension rows + 4).  PACKED: the matrix is complex symmetric, its lower
// triangle packed by columns; a tile's rows above the diagonal block come from
// the mirrored entries, 8 neighbouring threads taking one row's 8 columns (128
// contiguous bytes).
template <bool REAL, bool PACKED, int STAGES, int NJ>
struct TfStream {
    const void *base;
    int n, npad, KT, it;
    unsigned st0;
    size_t stage;
    int r, k0;                 // this thread's row and first column of a tile

    __device__ __forceinline__ void start(const void *m, int n_, unsigned st0_, size_t stage_)
    {
        base = m; n = n_; npad = tf_rows(n_); KT = (n_ + TF_BK - 1) / TF_BK; it = 0; st0 = st0_; stage = stage_;
        r = threadIdx.x % npad;
        k0 = threadIdx.x / npad;   // 0 or 1: the CTA has 2 npad threads
#pragma unroll
        for (int s = 0; s < STAGES - 1; ++s) fill(s);
    }
    __device__ __forceinline__ void fill(int at)
    {
        constexpr int E = REAL ? 8 : 16;
        const int kt = at % KT, slot = at % STAGES;
        const int ld = REAL ? npad + 4 : npad + 2;
        const unsigned dst = st0 + (unsigned)(slot * stage);
        const int c0 = kt * TF_BK;
        if (!PACKED) {
#pragma unroll
            for (int t = 0; t < TF_BK / 2; ++t) {
                const int kk = k0 + 2 * t, k = c0 + kk;
                const bool ok = r < n && k < n;
                cp_async_elem<E>(dst + (unsigned)((kk * ld + r) * E), (const char *)base + (ok ? (k * n + r) * E : 0), ok);
            }
        } else {
            const int n8 = (n + 7) / 8 * 8;
            if (r >= c0) {
                const int e0 = c0 * n8 - c0 * (c0 - 8) / 2 + (r - c0), len = n8 - c0;
                const bool ok = r < n8;
#pragma unroll
                for (int t = 0; t < TF_BK / 2; ++t) {
                    const int kk = k0 + 2 * t;
                    cp_async_elem<E>(dst + (unsigned)((kk * ld + r) * E),
                                     (const char *)base + (ok ? (e0 + kk * len) * E : 0), ok);
                }
            }
            const int kk = threadIdx.x % TF_BK, dr = npad / 4;   // 2 npad / TF_BK rows a pass
            int rr = threadIdx.x / TF_BK;
#pragma unroll
            for (int t = 0; t < 4; ++t, rr += dr)
                if (rr < c0) {
                    const int j0 = rr & ~7;
                    const int e = j0 * n8 - j0 * (j0 - 8) / 2 + (rr - j0) * (n8 - j0) + (c0 - j0) + kk;
                    cp_async_elem<E>(dst + (unsigned)((kk * ld + rr) * E), (const char *)base + e * E, true);
                }
        }
        cp_async_commit();
    }
    __device__ __forceinline__ void product(const unsigned char *smem, const zd *T, int ldt, int wr, int fr, int fk,
                                            int nb, TfAcc<NJ> &c)
    {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < NJ; ++j) c.r[i][j][0] = c.r[i][j][1] = c.i[i][j][0] = c.i[i][j][1] = 0.0;
        // all 8-column blocks (no branch between the products), or the first ones
        if (nb == NJ) stages<true>(smem, T, ldt, wr, fr, fk, nb, c);
        else stages<false>(smem, T, ldt, wr, fr, fk, nb, c);
    }
    template <bool FULL>
    __device__ __forceinline__ void stages(const unsigned char *smem, const zd *T, int ldt, int wr, int fr, int fk,
                                           int nb, TfAcc<NJ> &c)
    {
        for (int kt = 0; kt < KT; ++kt, ++it) {
            cp_async_wait<STAGES - 2>();
            __syncthreads();
            fill(it + STAGES - 1);
            const unsigned char *sp = smem + (it % STAGES) * stage;
#pragma unroll
            for (int k4 = 0; k4 < TF_BK; k4 += 4) {
                double ar[2], ai[2], an[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    if constexpr (REAL) {
                        ar[i] = ((const double *)sp)[(k4 + fk) * (npad + 4) + wr + 8 * i + fr];
                    } else {
                        const zd v = ((const zd *)sp)[(k4 + fk) * (npad + 2) + wr + 8 * i + fr];
                        ar[i] = v.x; ai[i] = v.y; an[i] = -v.y;
                    }
                }
#pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    if (!FULL && j >= nb) continue;
                    const zd b = T[(size_t)(8 * j + fr) * ldt + kt * TF_BK + k4 + fk];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        dmma(c.r[i][j][0], c.r[i][j][1], ar[i], b.x);
                        dmma(c.i[i][j][0], c.i[i][j][1], ar[i], b.y);
                        if constexpr (!REAL) {
                            dmma(c.r[i][j][0], c.r[i][j][1], an[i], b.y);
                            dmma(c.i[i][j][0], c.i[i][j][1], ai[i], b.x);
                        }
                    }
                }
            }
        }
    }
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;\n" ::: "memory"); }

template <bool PACKED, int MAXT, int MINB, int STAGES, int NJ>
__global__ void __launch_bounds__(MAXT, MINB)
taylor_f64_kernel(TaylorF64 a)
{
    constexpr int COLS = 8 * NJ;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ double wmax[16], cmax[2][TF_MAXCL];
    const int n = a.n, N = a.N;
    const int cs = (N + COLS - 1) / COLS, w = blockIdx.x / cs, rank = blockIdx.x % cs;
    if (a.mask && !a.mask[w]) return;   // the whole cluster
    // the peers' shared memory may be written to once all of them have started:
    // said here, waited for before the first store, which is orders away
    if (cs > 1) cluster_arrive();
    const int kFirst = max(1, a.checkFrom);
    const int col0 = rank * COLS, ncols = min(COLS, N - col0), nb = (ncols + 7) / 8;
    const int ldt = tf_ldt(n);
    const size_t stage = tf_stage(n);
    zd *T = (zd *)(smem + STAGES * stage);
    const unsigned st0 = (unsigned)__cvta_generic_to_shared(smem);
    const int tid = threadIdx.x, NT = blockDim.x, lane = tid & 31, warp = tid >> 5;
    const int wr = warp * 16, fr = lane >> 2, fk = lane & 3;

    TfStream<false, PACKED, STAGES, NJ> ms;
    ms.start(a.M + (size_t)w * a.Mstride, n, st0, stage);
    const zd *src = a.src + ((size_t)w * N + col0) * n;
    for (int e = tid; e < COLS * tf_rows(n); e += NT) {
        const int r = e % tf_rows(n), c = e / tf_rows(n);
        T[(size_t)c * ldt + r] = (r < n && c < ncols) ? src[(size_t)c * n + r] : make_double2(0.0, 0.0);
    }
    __syncthreads();
    TfAcc<NJ> sum, c;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const zd v = T[(size_t)(8 * j + 2 * fk + h) * ldt + wr + 8 * i + fr];
                sum.r[i][j][h] = v.x;
                sum.i[i][j][h] = v.y;
            }

    int k = 1;
    for (;; ++k) {
        ms.product(smem, T, ldt, wr, fr, fk, nb, c);
        const double inv = 1.0 / k;
        double mx = 0.0;   // largest |term|^2
        __syncthreads();   // every warp is done with the previous term
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < NJ; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const double x = c.r[i][j][h] * inv, y = c.i[i][j][h] * inv;
                    sum.r[i][j][h] += x;
                    sum.i[i][j][h] += y;
                    T[(size_t)(8 * j + 2 * fk + h) * ldt + wr + 8 * i + fr] = make_double2(x, y);
                    double s = fma(x, x, y * y);
                    // |z| of an infinity with a NaN is infinite
                    if (!(s <= 1e300) && (isinf(x) || isinf(y))) s = CUDART_INF;
                    mx = fmax(mx, s);
                }
        if (k < a.checkFrom) continue;
        mx = warp_max(mx);
        if (lane == 0) wmax[warp] = mx;
        __syncthreads();
        double all = 0.0;
        for (int q = 0; q < NT / 32; ++q) all = fmax(all, wmax[q]);
        if (cs > 1) {
            cg::cluster_group cl = cg::this_cluster();
            if (k == kFirst) cluster_wait();
            if (tid < cs) cl.map_shared_rank(&cmax[k & 1][0], tid)[rank] = all;
            cl.sync();
            for (int q = 0; q < cs; ++q) all = fmax(all, cmax[k & 1][q]);
        }
        const bool done = all <= a.acc * a.acc;
        if (!done && k < a.kmax) continue;
        if (rank == 0 && tid == 0) {
            if (a.order) a.order[w] = k;
            if (!done) atomicOr(a.status + w, (int)ST_TAYLOR_CAP);
        }
        break;
    }

    if (a.postZ || a.postR) {
        cp_async_wait<0>();
        __syncthreads();   // the series' stages and the last term are free
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < NJ; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    T[(size_t)(8 * j + 2 * fk + h) * ldt + wr + 8 * i + fr] =
                        make_double2(sum.r[i][j][h], sum.i[i][j][h]);
        if (a.postR) {
            TfStream<true, false, STAGES, NJ> ps;
            ps.start(a.postR, n, st0, stage);
            ps.product(smem, T, ldt, wr, fr, fk, nb, sum);
        } else {
            TfStream<false, false, STAGES, NJ> ps;
            ps.start(a.postZ, n, st0, stage);
            ps.product(smem, T, ldt, wr, fr, fk, nb, sum);
        }
    }
    zd *dst = a.dst + ((size_t)w * N + col0) * n;
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int cc = 8 * j + 2 * fk + h;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int r = wr + 8 * i + fr;
                if (cc < ncols && r < n) dst[(size_t)cc * n + r] = make_double2(sum.r[i][j][h], sum.i[i][j][h]);
            }
        }
    cp_async_wait<0>();
}

}  // namespace

bool taylor_f64_supported(int n, int N) { return n <= TF_MAXN && N <= TF_COLS * TF_MAXCL; }

template <bool PACKED, int MAXT, int MINB, int STAGES, int NJ = 2>
static cudaError_t launch(const TaylorF64 &a, cudaStream_t s)
{
    const auto kernel = taylor_f64_kernel<PACKED, MAXT, MINB, STAGES, NJ>;
    static std::atomic<unsigned long long> attr{0};
    cudaError_t r = each_device_once(attr, [] {
        return cudaFuncSetAttribute(taylor_f64_kernel<PACKED, MAXT, MINB, STAGES, NJ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)tf_smem(MAXT / 2, STAGES, 8 * NJ));
    });
    if (r != cudaSuccess) return r;
    const int cs = (a.N + 8 * NJ - 1) / (8 * NJ);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)cs * (unsigned)a.W);
    cfg.blockDim = dim3((unsigned)(2 * tf_rows(a.n)));
    cfg.dynamicSmemBytes = tf_smem(a.n, STAGES, 8 * NJ);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)cs;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    r = cudaLaunchKernelEx(&cfg, kernel, a);
    return r != cudaSuccess ? r : cudaGetLastError();
}

// A walker of 17 to 24 columns, n <= 96: one CTA of 24 columns (168 registers)
// instead of a cluster of 16 and 8, which streams M twice and meets at each order
// (n, N, walkers: 96, 20, 2048 1297 -> 963 us; 64, 24, 2048 579 -> 420; 90, 21, 300
// 277 -> 253; 32, 20, 1000 117 -> 102; 48, 24, 100 57 -> 51).  Small matrices of
// no more walkers than SMs stay on two SMs each (40, 18, 64: 40 us against 45; 32, 20,
// 148: 38 and 40), and wider walkers on 16 columns a CTA: 24 gain where waves are
// full (96, 48, 1000 1036 -> 978) and lose where they are not (90, 45, 300 355 -> 368).
//
// Otherwise 128 registers a thread, four stages.  192 threads (n = 81..96) take 96
// registers so that three CTAs are resident instead of two, 288 (n = 129..144) two
// instead of one: n = 90, N = 21, 300 walkers 303 -> 277 us; n = 64 and 128, whose
// number of CTAs stays the same, 98 us either way and 2.47 against 2.49 ms.  Above
// that one CTA per SM has three stages: n = 256 6.00 -> 5.81 ms (n = 64 and 128 with
// three: 98 us and 2.51 ms).
cudaError_t taylor_f64(const TaylorF64 &a, cudaStream_t s)
{
    g_launch_count++;
    const int nt = 2 * tf_rows(a.n);
    if (nt <= 192 && a.N > 16 && a.N <= 24 && (a.n > 40 || a.W > 148))
        return a.packed ? launch<true, 192, 2, 4, 3>(a, s) : launch<false, 192, 2, 4, 3>(a, s);
    if (nt == 192 || nt == 288) return a.packed ? launch<true, 288, 2, 4>(a, s) : launch<false, 288, 2, 4>(a, s);
    if (nt <= 256) return a.packed ? launch<true, 256, 2, 4>(a, s) : launch<false, 256, 2, 4>(a, s);
    return a.packed ? launch<true, 512, 1, 3>(a, s) : launch<false, 512, 1, 3>(a, s);
}
