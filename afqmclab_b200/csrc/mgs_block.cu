// Gram-Schmidt stabilisation of a walker (SD::stabilize / SD2is::stabilize,
// SD.cpp:42-56, SD2is.cpp:48-76) in panels of eight columns, FP64 arithmetic.
//
// One CTA per walker, 32 rows per warp, one row per lane.  Panel p first loses
// its components along every finished panel Q_j in turn, as the modified
// Gram-Schmidt does column by column: W = Q_j^H P (each warp its rows' share, the
// shares added in shared memory) and P -= Q_j W, both on the FP64 matrix
// instruction.  Its own columns then follow one another: one reduction gives a
// column's norm and its products with the panel's later columns.  The
// finished panels come back from memory (L2) one ahead of their use, or stay
// in shared memory up to 40 KB (QS; always for the mixed form, whose columns
// are rounded to fp32 only on the way out).
//
// Bound: instruction issue and latency of the columns' reductions (35 % of the
// issue slots and 33 % of the matrix pipe busy at 128 x 56) over the walkers that
// share an SM, three at n = 128.  Against one column at a time over
// all later ones (us per launch, one B200): 128 x 56, 1024 walkers 568 -> 341; 200 x
// 80, 1024: 3670 -> 1295; 288 x 120, 1024: 12600 -> 3300; 128 x 32, 2048: 349 -> 252 (fp32
// walkers 348 -> 306); 256 x 64, 512: 1227 -> 557; 32 x 14, 100: 20 -> 16.
#include <atomic>

#include "dmma.cuh"
#include "once.cuh"
#include "walker_kernels.cuh"

extern std::atomic<long long> g_launch_count;

namespace {

constexpr int MB_LDW = 9;           // leading dimension of a share of W
constexpr int MB_LDT = 10;          // of T_j
constexpr int MB_MAXN = 512;        // 16 warps
constexpr size_t MB_QS_BYTES = 40 * 1024;   // finished panels kept in shared memory up to this size

__host__ __device__ constexpr int mb_ld(int nw) { return 32 * nw + 1; }

struct MbLayout {
    int nw, ld;
    size_t q, wpart, t, dpart, r, bytes;
};
__host__ __device__ inline MbLayout mb_layout(int n, int ncol, bool qs)
{
    MbLayout L;
    L.nw = (n + 31) / 32;
    L.ld = mb_ld(L.nw);
    size_t at = (size_t)8 * L.ld * sizeof(zd);                                   // the panel
    L.q = at;
    at += (size_t)(qs ? (ncol + 7) / 8 * 8 : 16) * L.ld * sizeof(zd);           // all finished panels, or two stages
    L.wpart = at;
    at += (size_t)2 * L.nw * 8 * MB_LDW * sizeof(zd);                           // [parity][warp]: shares of W
    L.t = at;
    at += (size_t)((ncol + 7) / 8) * 8 * MB_LDT * sizeof(zd);                   // [panel][k][row]: T_j
    L.dpart = at;
    at += (size_t)2 * L.nw * 16 * sizeof(double);                               // [parity][warp]: shares of a column's products
    L.r = at;
    at += (size_t)ncol * sizeof(double);
    L.bytes = at;
    return L;
}

// The sums over the warp of 16 values per lane: lane t receives value
// mb_value(t) (lanes 2 i and 2 i + 1 the same one).
__device__ __forceinline__ int mb_value(int lane) { return lane >> 1; }
__device__ __forceinline__ double mb_reduce16(double (&x)[16], int lane)
{
#pragma unroll
    for (int h = 8; h >= 1; h >>= 1) {
        const bool up = lane & (2 * h);
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (i < h) {
                const double give = up ? x[i] : x[i + h], keep = up ? x[i + h] : x[i];
                x[i] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * h);
            }
    }
    return x[0] + __shfl_xor_sync(0xffffffffu, x[0], 1);
}

// F32: the walkers are the mixed form's fp32 planes [re n x ncol | im n x ncol].
template <bool F32, bool QS>
__global__ void __launch_bounds__(MB_MAXN, 1)
mgs_block_kernel(int n, int ncol, int nup, int ndn, int isSD2is, void *wfv, zd *logw, const int *alive, int *status)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int w = blockIdx.x;
    if (alive && !alive[w]) return;
    const MbLayout L = mb_layout(n, ncol, QS);
    const int nw = L.nw, ld = L.ld;
    zd *P = (zd *)smem, *Q = (zd *)(smem + L.q), *wpart = (zd *)(smem + L.wpart);
    zd *Tm = (zd *)(smem + L.t);
    double *dpart = (double *)(smem + L.dpart), *rS = (double *)(smem + L.r);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, fr = lane >> 2, fk = lane & 3;
    const int row = 32 * warp + lane, r0 = 32 * warp;
    const bool mine = row < n;
    const size_t ws = (size_t)n * ncol;
    zd *g = F32 ? nullptr : (zd *)wfv + (size_t)w * ws;
    float *g32 = F32 ? (float *)wfv + (size_t)w * 2 * ws : nullptr;
    const int np = (ncol + 7) / 8;
    int turn = 0;   // parity of the shared reduction buffers

    zd nx[8];   // the next panel's row
    auto fetch = [&](int p) {
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int col = 8 * p + c;
            const size_t e = row + (size_t)n * col;
            if (!(mine && col < ncol)) nx[c] = make_double2(0.0, 0.0);
            else if (F32) nx[c] = make_double2(g32[e], g32[ws + e]);
            else nx[c] = g[e];
        }
    };
    // this warp's rows of finished panel j into stage j & 1
    auto stage = [&](int j) {
        const unsigned q0 = (unsigned)__cvta_generic_to_shared(Q + (size_t)(j & 1) * 8 * ld + row);
#pragma unroll
        for (int c = 0; c < 8; ++c)
            cp_async_elem<16>(q0 + (unsigned)(c * ld * sizeof(zd)), mine ? g + row + (size_t)n * (8 * j + c) : g, mine);
        cp_async_commit();
    };

    // Q^H P over the CTA's rows in the right operand's layout: wb[q] is entry
    // (4 q + fk, fr)
    auto product = [&](const zd *Qj, zd (&wb)[2]) {
        double x[2][4][2];   // [even / odd rows][Re Re, Im Im, Re Im, Im Re]
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int t = 0; t < 4; ++t) x[q][t][0] = x[q][t][1] = 0.0;
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int rr = r0 + 8 * b + 4 * q + fk;
                const zd a = Qj[fr * ld + rr], v = P[fr * ld + rr];
                dmma(x[q][0][0], x[q][0][1], a.x, v.x);
                dmma(x[q][1][0], x[q][1][1], a.y, v.y);
                dmma(x[q][2][0], x[q][2][1], a.x, v.y);
                dmma(x[q][3][0], x[q][3][1], a.y, v.x);
            }
        zd *mineW = wpart + (size_t)(turn * nw + warp) * 8 * MB_LDW;
#pragma unroll
        for (int h = 0; h < 2; ++h)
            mineW[(2 * fk + h) * MB_LDW + fr] =
                make_double2((x[0][0][h] + x[1][0][h]) + (x[0][1][h] + x[1][1][h]),
                             (x[0][2][h] + x[1][2][h]) - (x[0][3][h] + x[1][3][h]));
        if (nw > 1) __syncthreads(); else __syncwarp();
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const zd *s = wpart + (size_t)turn * nw * 8 * MB_LDW + fr * MB_LDW + 4 * q + fk;
            zd v = s[0];
            for (int t = 1; t < nw; ++t) v = zadd(v, s[(size_t)t * 8 * MB_LDW]);
            wb[q] = v;
        }
        turn ^= 1;
    };

    fetch(0);
    for (int p = 0; p < np; ++p) {
        if (!QS && p > 0) stage(0);
#pragma unroll
        for (int c = 0; c < 8; ++c) P[c * ld + row] = nx[c];
        if (p + 1 < np) fetch(p + 1);
        __syncwarp();
        double pr[4][2], pi[4][2];   // the panel's rows as accumulators: 8-row block, column 2 fk + h
        if (p > 0) {
#pragma unroll
            for (int b = 0; b < 4; ++b)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const zd v = P[(2 * fk + h) * ld + r0 + 8 * b + fr];
                    pr[b][h] = v.x;
                    pi[b][h] = v.y;
                }
        }
        for (int j = 0; j < p; ++j) {
            const zd *Qj = Q + (size_t)(QS ? j : (j & 1)) * 8 * ld;
            if (!QS) {
                if (j + 1 < p) {
                    stage(j + 1);
                    cp_async_wait<1>();
                } else {
                    cp_async_wait<0>();
                }
                __syncwarp();
            }
            zd wb[2];
            product(Qj, wb);
            // T_j W, back through shared memory into the right operand's layout (the
            // buffer of this warp's next share, which nobody else reads yet)
            zd *own = wpart + (size_t)(turn * nw + warp) * 8 * MB_LDW;
            double t0[2] = {0.0, 0.0}, t1[2] = {0.0, 0.0}, t2[2] = {0.0, 0.0}, t3[2] = {0.0, 0.0};
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const zd a = Tm[((size_t)8 * j + 4 * q + fk) * MB_LDT + fr];
                dmma(t0[0], t0[1], a.x, wb[q].x);
                dmma(t1[0], t1[1], a.y, wb[q].y);
                dmma(t2[0], t2[1], a.x, wb[q].y);
                dmma(t3[0], t3[1], a.y, wb[q].x);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) own[(2 * fk + h) * MB_LDW + fr] = make_double2(t1[h] - t0[h], -(t2[h] + t3[h]));
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 2; ++q) wb[q] = own[fr * MB_LDW + 4 * q + fk];   // -T_j W
#pragma unroll
            for (int b = 0; b < 4; ++b)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const zd a = Qj[(4 * q + fk) * ld + r0 + 8 * b + fr];
                    dmma(pr[b][0], pr[b][1], a.x, wb[q].x);
                    dmma(pi[b][0], pi[b][1], a.x, wb[q].y);
                    dmma(pr[b][0], pr[b][1], -a.y, wb[q].y);
                    dmma(pi[b][0], pi[b][1], a.y, wb[q].x);
                }
#pragma unroll
            for (int b = 0; b < 4; ++b)
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    P[(2 * fk + h) * ld + r0 + 8 * b + fr] = make_double2(pr[b][h], pi[b][h]);
            __syncwarp();
        }
        // the panel's own columns, a row per lane
        zd v[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) v[c] = P[c * ld + row];
        const int cols = min(8, ncol - 8 * p);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            if (c >= cols) continue;
            double x[16];
            x[0] = fma(v[c].x, v[c].x, v[c].y * v[c].y);
            x[15] = 0.0;
#pragma unroll
            for (int j = 1; j < 8; ++j) {
                // conj(v_c) v_(c + j) at 2 j - 1, 2 j
                if (c + j < 8) {
                    x[2 * j - 1] = fma(v[c].x, v[c + j].x, v[c].y * v[c + j].y);
                    x[2 * j] = fma(v[c].x, v[c + j].y, -v[c].y * v[c + j].x);
                } else {
                    x[2 * j - 1] = x[2 * j] = 0.0;
                }
            }
            double s = mb_reduce16(x, lane);
            if (nw > 1) {
                double *mineD = dpart + (size_t)(turn * nw + warp) * 16;
                if (!(lane & 1)) mineD[mb_value(lane)] = s;
                __syncthreads();
                const double *d = dpart + (size_t)turn * nw * 16 + mb_value(lane);
                s = d[0];
                for (int t = 1; t < nw; ++t) s += d[16 * t];
                turn ^= 1;
            }
            const double r2 = __shfl_sync(0xffffffffu, s, 0), r = sqrt(r2);
            const double inv = r > 0.0 ? 1.0 / r : 0.0;
            if (tid == 0) rS[8 * p + c] = r;
            v[c] = zscale(v[c], inv);
#pragma unroll
            for (int j = 1; j < 8; ++j)
                if (c + j < 8) {
                    const double dx = __shfl_sync(0xffffffffu, s, 2 * (2 * j - 1)) * inv;
                    const double dy = __shfl_sync(0xffffffffu, s, 2 * (2 * j)) * inv;
                    v[c + j].x -= dx * v[c].x - dy * v[c].y;
                    v[c + j].y -= dx * v[c].y + dy * v[c].x;
                }
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const size_t e = row + (size_t)n * (8 * p + c);
            if (QS) Q[(size_t)(8 * p + c) * ld + row] = v[c];
            if (mine && c < cols) {
                if (F32) {
                    g32[e] = (float)v[c].x;
                    g32[ws + e] = (float)v[c].y;
                } else {
                    g[e] = v[c];
                }
            }
        }
        if (p + 1 < np) {
            // T of this panel: its Gram matrix G from the copy in P, then
            // (1 + L) T = 1 by rows, a column per lane (the same in every warp)
#pragma unroll
            for (int c = 0; c < 8; ++c) P[c * ld + row] = v[c];
            __syncwarp();
            zd wb[2];
            product(P, wb);
            zd *own = wpart + (size_t)(turn * nw + warp) * 8 * MB_LDW;   // G(k, col) at col * MB_LDW + k
#pragma unroll
            for (int q = 0; q < 2; ++q) own[fr * MB_LDW + 4 * q + fk] = wb[q];
            __syncwarp();
            if (warp == 0 && lane < 8) {
                zd t[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    zd x = make_double2(i == lane ? 1.0 : 0.0, 0.0);
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        if (k < i) {
                            const zd l = own[k * MB_LDW + i];
                            zfma(x, zneg(l), t[k]);
                        }
                    t[i] = x;
                    Tm[((size_t)8 * p + lane) * MB_LDT + i] = x;   // T(i, lane)
                }
            }
            // read first after the next panel's first barrier (or by this warp)
            __syncwarp();
        }
        __syncwarp();   // the warp's other lanes read these rows from here on
    }
    if (warp == 0) {
        __syncwarp();
        const int nmin = nup < ndn ? nup : ndn;
        double logR = 0.0, logRmin = 0.0;
        bool bad = false;
        for (int c = lane; c < ncol; c += 32) {
            const double r = rS[c], lr = log(r);
            bad = bad || r == 0.0;
            logR += lr;
            if (c < nmin) logRmin += lr;
        }
        logR = warp_sum(logR);
        logRmin = warp_sum(logRmin);
        bad = __any_sync(0xffffffffu, bad);
        if (lane == 0) {
            zd lw = logw[w];
            if (!isSD2is) lw.x += logR;
            else if (nup == ndn) lw.x += 2.0 * logR;
            else lw.x += logR + logRmin;
            logw[w] = lw;
            if (bad && status) atomicOr(status + w, (int)ST_ZERO_NORM);
        }
    }
}

template <bool F32, bool QS>
cudaError_t launch(int W, int n, int ncol, int nup, int ndn, int isSD2is, void *wf, zd *logw, const int *alive,
                   int *status, cudaStream_t s)
{
    static std::atomic<unsigned long long> attr{0};
    const cudaError_t r = each_device_once(attr, [] {
        return cudaFuncSetAttribute(mgs_block_kernel<F32, QS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    });
    if (r != cudaSuccess) return r;
    const MbLayout L = mb_layout(n, ncol, QS);
    mgs_block_kernel<F32, QS><<<W, 32 * L.nw, L.bytes, s>>>(n, ncol, nup, ndn, isSD2is, wf, logw, alive, status);
    return cudaPeekAtLastError();
}

}  // namespace

bool launch_mgs_block(int W, int n, int ncol, int nup, int ndn, int isSD2is, void *wf, bool f32, zd *logw,
                      const int *alive, int *status, cudaStream_t s)
{
    const size_t limit = 227 * 1024;
    if (n > MB_MAXN) return false;
    const bool fits = mb_layout(n, ncol, true).bytes <= limit;
    const bool qs = f32 || (fits && (size_t)n * ncol * sizeof(zd) <= MB_QS_BYTES);
    if (!(qs ? fits : mb_layout(n, ncol, false).bytes <= limit)) return false;
    g_launch_count++;
    if (f32) launch<true, true>(W, n, ncol, nup, ndn, isSD2is, wf, logw, alive, status, s);
    else if (qs) launch<false, true>(W, n, ncol, nup, ndn, isSD2is, wf, logw, alive, status, s);
    else launch<false, false>(W, n, ncol, nup, ndn, isSD2is, wf, logw, alive, status, s);
    return true;
}
