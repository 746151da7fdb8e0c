// Batched complex FP64 GEMM (plain form) on the FP64 matrix instruction
// (mma.sync.m8n8k4.f64).  tcgen05 has no FP64 kind; the warp-level FP64
// product runs at the rate of the FP64 pipe (37.0 TFLOP/s measured, against
// 33.9 for a bare chain of DFMAs), and its fragments take each operand value
// from shared memory once per warp: a 32 x 16 complex warp tile reads 3 KB
// per 512 matrix-pipe cycles, where the register-tiled DFMA form before it was
// bound by its fragment loads.  One B200, scalar tiles and the first form of
// these: M-build (16384 x 2048 x 640, real A) 4.14 and 2.83 ms, one-body product of
// 1024 128 x 56 walkers 0.465 and 0.27 ms.  Without a branch between the products
// of a warp whose tile lies inside C, 10 % more.  Now 8704 x 2048 x 640, real A, takes
// 1.43 ms (31.9 TFLOP/s, the matrix pipe busy 90 % of the time) and the force 640 x
// 2048 x 4096 0.71 ms (30.2, 89 %); what is left is barriers and the copies' address
// arithmetic.  Small outputs are bound by their operands too: 32 x 32 x 128, real A,
// 2048 walkers 0.047 ms (22.8 TFLOP/s, pipe 74 %, 3.1 TB/s).
#include "zgemm.cuh"

#include <algorithm>
#include <atomic>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>

#include "dmma.cuh"
#include "once.cuh"

extern std::atomic<long long> g_launch_count;

namespace {

template <bool REAL> struct Elem { typedef zd T; };
template <> struct Elem<true> { typedef double T; };

// One operand's tile: R rows (its m or n extent) by BK of the contraction.
// KC: the contraction index is the contiguous one in memory.  The shared
// layout keeps memory's order, so that neighbouring threads copy neighbouring
// elements, and its leading dimension makes a fragment load (8 rows x 4 k)
// touch every bank once: 4 mod 8 (complex) or 4 / 12 mod 16 (real) elements
// with k contiguous, 2 mod 8 or 4 mod 16 with the rows contiguous.
template <int R, int BK, bool KC, bool REAL>
struct TileLayout {
    typedef typename Elem<REAL>::T T;
    static constexpr int LD = KC ? BK + 4 : R + (REAL ? 4 : 2);
    static constexpr int COUNT = KC ? R * LD : BK * LD;
    static constexpr size_t BYTES = (COUNT * sizeof(T) + 15) / 16 * 16;
    static __device__ __forceinline__ int at(int r, int k) { return KC ? r * LD + k : k * LD + r; }
};

// REAL: 0 both operands complex, 1 A real, 2 B real, 3 both real; a real
// operand takes two real products per complex one in place of four.
template <int BM_, int BN_, int WM_, int WN_, int BK_, int STAGES_, int MINB_>
struct Tile {
    static constexpr int BM = BM_, BN = BN_, WM = WM_, WN = WN_, BK = BK_, STAGES = STAGES_, MINB = MINB_;
    static constexpr int NT = 32 * (BM / WM) * (BN / WN);
};

template <class TL, int OPA, int OPB, int REAL>
struct GemmShape {
    typedef TileLayout<TL::BM, TL::BK, OPA != OP_N, (REAL & 1) != 0> LA;
    typedef TileLayout<TL::BN, TL::BK, OPB == OP_N, (REAL & 2) != 0> LB;
    static constexpr size_t STAGE = LA::BYTES + LB::BYTES;
    static constexpr size_t SMEM = STAGE * TL::STAGES;
};

template <int R, int BK, int NT, bool KC, bool REAL>
struct Loader {
    typedef TileLayout<R, BK, KC, REAL> L;
    typedef typename L::T T;
    static constexpr int N = R * BK / NT;   // elements per thread
    static_assert(R * BK % NT == 0 && (KC ? NT % BK == 0 : (NT % R == 0 || R % NT == 0)), "tile split");
    const T *base;
    const T *safe;
    long long ld;
    int r0, k0, rows, K;

    __device__ __forceinline__ Loader(const void *P, long long ld_, int tile, int ext, int K_)
    {
        const int t = threadIdx.x;
        // thread t's first element; the t-th of its N is rstep / kstep further
        k0 = KC ? t % BK : t / R;
        r0 = KC ? t / BK : t % R;
        ld = ld_;
        rows = ext - tile;
        K = K_;
        safe = (const T *)P;
        base = (const T *)P + (KC ? (long long)(tile + r0) * ld + k0 : (long long)k0 * ld + tile + r0);
    }
    // tile number kt of the contraction into the stage at `dst`
    __device__ __forceinline__ void load(unsigned dst, int kt) const
    {
        const T *p = base + (KC ? (long long)kt * BK : (long long)kt * BK * ld);
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int dr = KC ? i * (NT / BK) : (R > NT ? (i % (R / NT)) * NT : 0);
            const int dk = KC ? 0 : (R > NT ? i / (R / NT) : i * (NT / R));
            const bool ok = r0 + dr < rows && kt * BK + k0 + dk < K;
            const T *q = p + (KC ? (long long)dr * ld : (long long)dk * ld + dr);
            cp_async_elem<(int)sizeof(T)>(dst + (unsigned)(L::at(r0 + dr, k0 + dk) * sizeof(T)), ok ? q : safe, ok);
        }
    }
};

// C_b = alpha op(A_b) op(B_b) + beta C_b, one BM x BN tile per CTA, BK columns
// of the contraction per stage, STAGES cp.async stages in flight.  Each warp
// owns a WM x WN block as 8 x 8 accumulator fragments; a fragment row or
// column that lies outside C takes no products, so a ragged edge costs its
// 8-row granule only.
template <class TL, int OPA, int OPB, int REAL, bool SCALE>
__global__ void __launch_bounds__(TL::NT, TL::MINB)
zgemm_kernel(ZGemmArgs a)
{
    constexpr int BM = TL::BM, BN = TL::BN, WM = TL::WM, WN = TL::WN, BK = TL::BK, ST = TL::STAGES, NT = TL::NT;
    constexpr int MI = WM / 8, NI = WN / 8;
    constexpr bool RA = (REAL & 1) != 0, RB = (REAL & 2) != 0;
    typedef GemmShape<TL, OPA, OPB, REAL> SH;
    typedef typename SH::LA LA;
    typedef typename SH::LB LB;
    // the second part's tiles follow the first one's in x: z, the batch, is limited
    // to 65535
    const int b = blockIdx.z, tilesM = a.parts > 1 ? gridDim.x >> 1 : gridDim.x;
    const bool second = blockIdx.x >= tilesM;
    const int bx = second ? blockIdx.x - tilesM : blockIdx.x;
    if (a.mask && a.mask[b] == 0) return;
    if (a.skip && a.skip[b] != 0) return;
    const int m = second ? a.m1 : a.m, n = second ? a.n1 : a.n;
    // a quadratic form's rows get longer downwards: the longest start first
    const int tileM = (a.quad ? tilesM - 1 - bx : bx) * BM, tileN = blockIdx.y * BN;
    if (tileM >= m || tileN >= n) return;
    if (a.lower && tileM + BM <= tileN) return;
    int k = second ? a.k1 : a.k;
    const int kBegin = a.ksum ? b * a.k : 0;   // this piece's place in the contraction
    if (a.quad || a.ksum) {
        const int kAll = a.ksum ? a.ksum : a.k;
        k = max(0, min(a.k, (a.quad ? min(kAll, tileM + BM) : kAll) - kBegin));
    }

    extern __shared__ __align__(16) unsigned char smem[];
    const unsigned smem0 = (unsigned)__cvta_generic_to_shared(smem);
    const char *Ab = (const char *)a.A + ((size_t)b * a.strideA + (second ? a.offA1 : 0)) * sizeof(typename LA::T);
    const char *Bb = (const char *)a.B + ((size_t)b * a.strideB + (second ? a.offB1 : 0)) * sizeof(typename LB::T);
    const Loader<BM, BK, NT, OPA != OP_N, RA> la(Ab, a.lda, tileM, m, k);
    const Loader<BN, BK, NT, OPB == OP_N, RB> lb(Bb, a.ldb, tileN, n, k);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wm = (warp % (BM / WM)) * WM, wn = (warp / (BM / WM)) * WN;
    const int fr = lane >> 2, fk = lane & 3;
    // fragments of this warp that meet C
    const int mb = (m - tileM - wm + 7) / 8, nb = (n - tileN - wn + 7) / 8;

    double cr[MI][NI][2], ci[MI][NI][2];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NI; ++j) cr[i][j][0] = cr[i][j][1] = ci[i][j][0] = ci[i][j][1] = 0.0;

    const int KT = (k + BK - 1) / BK;
    // first stage of the diagonal block (KT: it lies in a later piece)
    const int left = a.quad ? tileM - kBegin : 0;
    const int ktDiag = left <= 0 ? -1 : left >= k ? KT : left / BK;
    static_assert(BM % BK == 0, "a diagonal block starts a stage");
#pragma unroll
    for (int s = 0; s < ST - 1; ++s) {
        if (s < KT) {
            la.load(smem0 + s * (unsigned)SH::STAGE, s);
            lb.load(smem0 + s * (unsigned)SH::STAGE + (unsigned)LA::BYTES, s);
        }
        cp_async_commit();
    }
    // FULL: every fragment of the warp meets C, so that no branch stands
    // between the products
    const zd *scale = SCALE ? a.scaleB + (size_t)b * a.strideScale + (second ? a.offScale1 : 0) : nullptr;
    zd scl[BK / 4];   // this lane's factors of a stage, fetched while the stage arrives
    auto products = [&](auto full, const typename LA::T *As, const typename LB::T *Bs) {
        constexpr bool FULL = decltype(full)::value;
#pragma unroll
        for (int k4 = 0; k4 < BK; k4 += 4) {
            double ar[MI], ai[MI], an[MI];
            const zd sc = SCALE ? scl[k4 / 4] : make_double2(0.0, 0.0);
#pragma unroll
            for (int i = 0; i < MI; ++i) {
                if constexpr (RA) {
                    ar[i] = As[LA::at(wm + 8 * i + fr, k4 + fk)];
                } else {
                    const zd v = As[LA::at(wm + 8 * i + fr, k4 + fk)];
                    ar[i] = v.x;
                    ai[i] = OPA == OP_C ? -v.y : v.y;
                    an[i] = OPA == OP_C ? v.y : -v.y;
                }
            }
#pragma unroll
            for (int j = 0; j < NI; ++j) {
                if (!FULL && j >= nb) continue;
                double br, bi = 0.0;
                if constexpr (RB) {
                    br = Bs[LB::at(wn + 8 * j + fr, k4 + fk)];
                } else {
                    const zd v = Bs[LB::at(wn + 8 * j + fr, k4 + fk)];
                    br = v.x;
                    bi = OPB == OP_C ? -v.y : v.y;
                    if constexpr (SCALE) {
                        br = v.x * sc.x - v.y * sc.y;
                        bi = v.x * sc.y + v.y * sc.x;
                    }
                }
#pragma unroll
                for (int i = 0; i < MI; ++i) {
                    if (!FULL && i >= mb) continue;
                    dmma(cr[i][j][0], cr[i][j][1], ar[i], br);
                    if constexpr (!RB) dmma(ci[i][j][0], ci[i][j][1], ar[i], bi);
                    if constexpr (!RA && !RB) dmma(cr[i][j][0], cr[i][j][1], an[i], bi);
                    if constexpr (!RA) dmma(ci[i][j][0], ci[i][j][1], ai[i], br);
                }
            }
        }
    };
    auto twice = [&] {
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
            for (int j = 0; j < NI; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) { cr[i][j][h] *= 2.0; ci[i][j][h] *= 2.0; }
    };
    const bool full = mb >= MI && nb >= NI;
    int slot = 0, fill = ST - 1;
    for (int kt = 0; kt < KT; ++kt) {
        if constexpr (SCALE) {
#pragma unroll
            for (int q = 0; q < BK / 4; ++q) {
                const int kk = kt * BK + 4 * q + fk;
                scl[q] = kk < k ? __ldg(scale + kk) : make_double2(0.0, 0.0);
            }
        }
        cp_async_wait<ST - 2>();
        __syncthreads();
        if (kt + ST - 1 < KT) {
            la.load(smem0 + fill * (unsigned)SH::STAGE, kt + ST - 1);
            lb.load(smem0 + fill * (unsigned)SH::STAGE + (unsigned)LA::BYTES, kt + ST - 1);
        }
        cp_async_commit();
        if (kt == ktDiag) twice();
        const typename LA::T *As = (const typename LA::T *)(smem + slot * SH::STAGE);
        const typename LB::T *Bs = (const typename LB::T *)(smem + slot * SH::STAGE + LA::BYTES);
        if (full) products(std::true_type{}, As, Bs);
        else products(std::false_type{}, As, Bs);
        slot = slot + 1 == ST ? 0 : slot + 1;
        fill = fill + 1 == ST ? 0 : fill + 1;
    }
    if (ktDiag == KT) twice();

    zd *Cb = a.C + (size_t)b * a.strideC + (second ? a.offC1 : 0);
    const bool beta0 = (a.beta.x == 0.0 && a.beta.y == 0.0);
#pragma unroll
    for (int j = 0; j < NI; ++j) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int gj = tileN + wn + 8 * j + 2 * fk + h;
            if (gj >= n) continue;
#pragma unroll
            for (int i = 0; i < MI; ++i) {
                const int gi = tileM + wm + 8 * i + fr;
                if (gi >= m) continue;
                zd v = zmul(a.alpha, make_double2(cr[i][j][h], ci[i][j][h]));
                zd *c = Cb + gi + (size_t)gj * a.ldc;
                if (!beta0) zfma(v, a.beta, *c);
                *c = v;
            }
        }
    }
}

template <class TL, int OPA, int OPB, int REAL = 0, bool SCALE = false>
cudaError_t launch3(const ZGemmArgs &a, cudaStream_t s)
{
    typedef GemmShape<TL, OPA, OPB, REAL> SH;
    const int m = a.parts > 1 ? std::max(a.m, a.m1) : a.m, n = a.parts > 1 ? std::max(a.n, a.n1) : a.n;
    dim3 grid((m + TL::BM - 1) / TL::BM * a.parts, (n + TL::BN - 1) / TL::BN, a.batch);
    static std::atomic<unsigned long long> attr{0};
    const cudaError_t r = each_device_once(attr, [] {
        return cudaFuncSetAttribute(zgemm_kernel<TL, OPA, OPB, REAL, SCALE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)SH::SMEM);
    });
    if (r != cudaSuccess) return r;
    zgemm_kernel<TL, OPA, OPB, REAL, SCALE><<<grid, TL::NT, SH::SMEM, s>>>(a);
    return cudaGetLastError();
}

// The operator pairs and real operands that the engine's products have.
template <class TL, bool ONE_REAL = false>
cudaError_t launch2(const ZGemmArgs &a, cudaStream_t s)
{
    const int real = (a.a_real ? 1 : 0) | (a.b_real ? 2 : 0);
#define ZG_CASE(OA, OB, R) \
    if (a.opA == OA && a.opB == OB && real == R) return launch3<TL, OA, OB, R>(a, s);
    ZG_CASE(OP_N, OP_N, 1) ZG_CASE(OP_N, OP_N, 2) ZG_CASE(OP_N, OP_T, 1) ZG_CASE(OP_C, OP_N, 2) ZG_CASE(OP_T, OP_N, 1)
    if constexpr (!ONE_REAL) {
        ZG_CASE(OP_N, OP_N, 0) ZG_CASE(OP_N, OP_T, 0) ZG_CASE(OP_N, OP_T, 3) ZG_CASE(OP_C, OP_N, 0)
        ZG_CASE(OP_T, OP_N, 0) ZG_CASE(OP_T, OP_T, 0) ZG_CASE(OP_T, OP_C, 0)
    }
#undef ZG_CASE
    return cudaErrorInvalidValue;
}

}  // namespace

// ----------------------------------------------------------- autotuner
// Candidate tile shapes; the default rule picks one by size, the autotuner
// (when enabled) times every candidate once per problem shape and keeps the
// fastest.  Timing runs are synchronous, so shapes are tuned on first use
// outside stream capture; captured launches reuse the cached choice.
namespace {

// Measured on one B200, TFLOP/s of the three tiles (32 x 32 | 64 x 32 | 64 x 64):
// M-build 16384 x 2048 x 640, real A: - | - | 30.4; 128 x 32 x 128 x 2048
// walkers: 30.3 | 30.6 | 26.9; 56 x 56 x 128 x 1024: 23.8 | 23.4 | 20.8;
// 32 x 32 x 128 x 2048: 28.2 | 15.4 | 9.3; 14 x 14 x 32 x 100: 6.5 us each.
constexpr int NCAND = 3;
typedef Tile<32, 32, 16, 16, 8, 4, 4> TileS;
typedef Tile<64, 32, 32, 16, 8, 4, 3> TileM;
typedef Tile<64, 64, 32, 16, 16, 3, 2> TileL;
// The largest for one real operand and a long contraction: half the products per
// stage leave room for 32 columns of it in two stages, half the barriers (TileL
// and this, in one run: 4096 x 2048 x 4096, real A, 4.24 and 4.09 ms; 4096 x 640 x 4096,
// real B, 1.54 and 1.48; the complex form loses, 4.21 and 4.56).
typedef Tile<64, 64, 32, 16, 32, 2, 2> TileLR;

cudaError_t launch_cand(int c, const ZGemmArgs &a, cudaStream_t s)
{
    switch (c) {
    case 0: return launch2<TileS>(a, s);
    case 1: return launch2<TileM>(a, s);
    default:
        if ((a.a_real != 0) != (a.b_real != 0) && a.k >= 256) return launch2<TileLR, true>(a, s);
        return launch2<TileL>(a, s);
    }
}

// Time of the last-finishing SM in products: waves of CTAs (148 SMs,
// MINB CTAs each) times the whole tile, over the tile's measured rate on
// shapes that fill it (the smaller tiles pay more fragment loads and barriers
// per product; half of the largest one's warps lose their branch-free loop where
// the rows end inside it: 56 x 128 x 56, 1024 walkers, 144 us against 137).  A tile counts in full where C covers part of it: the warps
// outside C leave their SM quadrant's matrix pipe idle (32 x 32 outputs: 0.076
// ms in 32 x 32 tiles, 0.140 in 64 x 32, 0.232 in 64 x 64).
template <class TL>
double tile_cost(const ZGemmArgs &a, double rate)
{
    // a quadratic form's pieces end where the row block ends: their total length
    // over the slots, and half the longest for the last ones to finish
    if (a.quad) {
        const double t = (double)((a.m + TL::BM - 1) / TL::BM) * ((a.n + TL::BN - 1) / TL::BN) / (148.0 * TL::MINB);
        const double all = a.ksum ? a.ksum : a.k, piece = a.k;
        return std::max(piece, 0.5 * t * all + 0.5 * piece) * TL::MINB * TL::BM * TL::BN / rate;
    }
    double tiles = (double)((a.m + TL::BM - 1) / TL::BM) * ((a.n + TL::BN - 1) / TL::BN);
    if (a.parts > 1) tiles += (double)((a.m1 + TL::BM - 1) / TL::BM) * ((a.n1 + TL::BN - 1) / TL::BN);
    tiles *= a.batch * (a.lower ? 0.5 : 1.0);
    double waves = tiles / (148.0 * TL::MINB);
    // beyond a few waves the ragged last one overlaps the stragglers
    waves = waves < 4.0 ? (double)(long long)(waves + 0.999999) : waves + 0.5;
    return waves * a.k * TL::MINB * TL::BM * TL::BN / rate;
}

// C = A diag(scale) B in one tile per column block, so that C may be B: 32 x 32 up
// to 32 rows, 64 x 64 up to 64, 128 x 32 above.  The factors meet B's fragments in
// registers: 95 us for 1024 64 x 56 pairs of spins against 80 without them, and
// against 41 for a pass of its own over the walkers.
typedef Tile<128, 32, 32, 16, 8, 4, 2> TileTall;
template <int REAL>
cudaError_t launch_scaled(const ZGemmArgs &a, cudaStream_t s)
{
    const int m = a.parts > 1 ? std::max(a.m, a.m1) : a.m;
    if (m <= 32) return launch3<TileS, OP_N, OP_N, REAL, true>(a, s);
    if (m <= 64) return launch3<TileL, OP_N, OP_N, REAL, true>(a, s);
    if (m <= 128) return launch3<TileTall, OP_N, OP_N, REAL, true>(a, s);
    return cudaErrorInvalidValue;
}

double cand_cost(const ZGemmArgs &a, int *cand)
{
    const bool ragged = a.m < 256 && a.m % 64 != 0;
    const double c[NCAND] = {tile_cost<TileS>(a, 0.93), tile_cost<TileM>(a, 0.95),
                             tile_cost<TileL>(a, ragged ? 0.9 : 1.0)};
    int best = 0;
    for (int i = 1; i < NCAND; ++i)
        if (c[i] < c[best]) best = i;
    if (cand) *cand = best;
    return c[best];
}

std::mutex g_tune_mu;
typedef std::tuple<int, int, int, int, int, int, int, int, int, int> TuneKey;
TuneKey tune_key(const ZGemmArgs &a)
{
    return TuneKey(a.m, a.n, a.k, a.opA, a.opB, a.a_real, a.b_real, a.batch, a.lower + 2 * a.quad + 4 * a.parts, a.ksum);
}
std::map<TuneKey, int> g_tuned;
std::atomic<int> g_autotune{0};

}  // namespace

// A piece more costs its output written and read once more (as much as 40 elements of
// the contraction) and the stages in flight at its start (32); the sum is a
// launch.  The pieces take at most 256 MB.  In one piece and in those chosen: force
// 277 x 300 x 1890 72 us (two equal pieces) and 42 (six; the best of a sweep over
// pieces and tiles is 37); forms 1890 x 300 164 and 113 (five; 109), 1024 x 512 74
// and 58 (four; 55), 4096 x 640 911 and 748 (four; 725), 16384 x 512 9.69 ms and
// 8.54 (two; 8.43), 16384 x 1280 20.6 ms in one, within 0.3% of the best.
int zgemm_pieces(const ZGemmArgs &a)
{
    int best = 1;
    double bestCost = 0.0;
    for (int p = 1; p <= 8 && (p == 1 || (double)a.m * a.n * p <= (1 << 24)); ++p) {
        ZGemmArgs s = a;
        if (zgemm_split(s, p, 0) != p) continue;
        double cost = cand_cost(s, nullptr) * (s.k + 32.0) / s.k;
        if (p > 1) cost += (double)a.m * a.n / 148.0 * 40.0 * p + (a.quad ? 0.0 : 2e5);
        if (p == 1 || cost < bestCost) { best = p; bestCost = cost; }
    }
    return best;
}

int zgemm_split(ZGemmArgs &a, int pieces, long long strideC)
{
    if (pieces <= 1) return 1;
    const int all = a.k;
    a.k = (all + pieces - 1) / pieces;
    if (a.quad) a.k = (a.k + 63) / 64 * 64;
    a.ksum = all;
    a.batch = (all + a.k - 1) / a.k;
    a.strideA = a.opA == OP_N ? a.lda * a.k : a.k;
    a.strideB = a.opB == OP_N ? a.k : a.ldb * a.k;
    a.strideC = strideC;
    return a.batch;
}

void zgemm_set_autotune(int on) { g_autotune = on; }

int zgemm_tuned_choice(const ZGemmArgs &a)
{
    const TuneKey key = tune_key(a);
    std::lock_guard<std::mutex> lock(g_tune_mu);
    auto it = g_tuned.find(key);
    return it == g_tuned.end() ? -1 : it->second;
}

cudaError_t zgemm_batched(const ZGemmArgs &a, cudaStream_t stream)
{
    g_launch_count++;
    if (a.m <= 0 || a.n <= 0 || a.batch <= 0) return cudaSuccess;
    if (a.k <= 0) return cudaErrorInvalidValue;
    if (a.scaleB) {
        if (a.opA != OP_N || a.opB != OP_N || a.b_real || a.lower || a.quad) return cudaErrorInvalidValue;
        return a.a_real ? launch_scaled<1>(a, stream) : launch_scaled<0>(a, stream);
    }
    const TuneKey key = tune_key(a);
    int choice = -1;
    {
        std::lock_guard<std::mutex> lock(g_tune_mu);
        auto it = g_tuned.find(key);
        if (it != g_tuned.end()) choice = it->second;
    }
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(stream, &cs);
    if (choice < 0 && g_autotune && cs == cudaStreamCaptureStatusNone && a.beta.x == 0.0 &&
        a.beta.y == 0.0) {
        // time every candidate (the output is simply rewritten each time)
        cudaEvent_t e0, e1;
        cudaEventCreate(&e0);
        cudaEventCreate(&e1);
        float best = 1e30f;
        for (int c = 0; c < NCAND; ++c) {
            if (launch_cand(c, a, stream) != cudaSuccess) { cudaGetLastError(); continue; }
            cudaEventRecord(e0, stream);
            for (int r = 0; r < 3; ++r) launch_cand(c, a, stream);
            cudaEventRecord(e1, stream);
            cudaEventSynchronize(e1);
            float ms = 0.f;
            cudaEventElapsedTime(&ms, e0, e1);
            if (ms < best) { best = ms; choice = c; }
        }
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        std::lock_guard<std::mutex> lock(g_tune_mu);
        g_tuned[key] = choice;
    }
    if (choice < 0) cand_cost(a, &choice);
    return launch_cand(choice, a, stream);
}
