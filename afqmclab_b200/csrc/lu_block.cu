// Log-determinant and inverse of the overlap blocks by a blocked in-place
// Gauss-Jordan elimination on the FP64 matrix instruction (same contract as
// launch_lu_logdet_inverse; logDeterminant, tensor_2d_common_fun.cpp:75-105).
//
// The matrix stays in registers as 8 x 8 accumulator blocks: warp i owns block
// row i, a CTA up to 8 block columns (64 columns; blocks of 65 to 128 columns
// are split over a cluster of two CTAs).  Panel p is block column p.  Its
// eight elimination steps run on the panel alone, one row per lane, with
// zgetf2's pivot rule (first position of the largest |re| + |im|; rows stay
// where they are and carry their position in the interchanged matrix).  The
// panel's own in-place result G then updates every other block column at once:
// with B the eight pivot rows before the update,
//     A <- A with the pivot rows zeroed + G B        (rank 8, matrix products)
// and the panel's columns become G.  After the last panel the matrix is the
// inverse up to the interchanges.
//
// The next panel's column block is updated first, and panel warps of their own
// factor it while the others finish this update.  The step of the panel is a
// chain of about 25 dependent operations (a pivot search, a reciprocal, one
// exchange through shared memory), which bounds the kernel: for 1024 matrices of 56
// columns the warps spend half their time at the barriers behind it, the matrix
// pipe is busy 22 % and the issue slots 28 % of the time.  Hence one warp reduction
// per search (lb_rank) and the hardware's reciprocal start (lb_rcp); with the
// compute warps as panel warps the registers spilled.  Rows that tie in the rank
// are told apart by all 64 bits: at once where one warp holds the rows, else by
// one more pass over the panel (lb_again); the test costs nothing up to 64 columns
// and 3 to 4 % on 80 and 120.
//
// Against the element-wise kernels it replaces (us per launch, one B200): 14
// columns, 100 matrices 35 -> 17; 16 columns, 512 matrices 31 -> 17; 56, 1024: 203
// -> 183; 64, 512: 131 -> 109; 80, 1024: 1459 -> 822; 120, 1024: 2867 -> 1464.
// Error against extended precision over random matrices of 4 to 120 columns, the
// element-wise kernels' as 1 (geometric mean, 120 to 900 matrices a size): inverse
// 1.03 to 1.2, log-determinant 0.7 to 1.1; both are some N eps.
#include <cooperative_groups.h>

#include <atomic>

#include "dmma.cuh"
#include "lu_block.cuh"
#include "lu_common.cuh"
#include "once.cuh"

namespace cg = cooperative_groups;

extern std::atomic<long long> g_launch_count;

namespace {

// C: CTAs per block; NCB: block columns per CTA (8, or 4 for up to 32 columns, whose
// fewer registers let six CTAs share an SM).
template <int C, int NCB>
struct LbShared {
    static constexpr int ROWS = 8 * NCB * C, LDG = ROWS + 2;   // 2 mod 8: conflict-free fragment loads
    static constexpr int LB_LDB = 8 * NCB + 2;
    zd G[2][8][LDG];        // [panel parity][column][row]
    zd B[8][LB_LDB];        // the pivot rows
    zd crow[2][2 * C][9];   // [step parity][warp]: the candidate's reciprocal, the rest of its panel row, its value
    int4 rank[2];           // [step parity]: each panel warp's best rank
    zd piv[ROWS];           // the pivots, by step
    int slot[2][ROWS];      // [panel parity][row]: the panel step that the row was pivot of, or -1
    int pv[ROWS], rowOf[ROWS], pos[ROWS];   // by step: pivot position before its interchange, pivot row; by row: final position
    int sing;
    double ln;   // of the pivots recorded here: sum of log |pivot|, product of the phases
    zd ph;
};

__device__ __forceinline__ void bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// Whether any of the barrier's threads votes for it.
__device__ __forceinline__ bool bar_any(int id, int threads, bool vote)
{
    int r;
    asm volatile("{\n.reg .pred p, q;\nsetp.ne.s32 p, %3, 0;\nbar.red.or.pred q, %1, %2, p;\nselp.s32 %0, 1, 0, q;\n}\n"
                 : "=r"(r)
                 : "r"(id), "r"(threads), "r"((int)vote)
                 : "memory");
    return r != 0;
}

// The steps of panel p on the panel warps' rows a (row prow at position pos; the
// step that takes it as pivot in myslot).  The row rotates by one register per
// step, so that the current column is always a[0] and the step is one loop body
// with static register indices.  One warp (NCB = 4) chooses by rank and by all bits in the same
// step.  Several choose by rank; tied: a row ties with a chosen one, and the
// panel has to be done again by all bits (EXACT).
template <bool EXACT, int C, int NCB>
__device__ __forceinline__ void lb_steps(LbShared<C, NCB> &sh, LbShared<C, NCB> *peer, int p, int Ns, int pw, int prow,
                                         zd (&a)[8], int &pos, int &myslot, bool &tied)
{
    const int pwarp = prow >> 5, lane = prow & 31, steps = min(8, Ns - 8 * p);
#pragma unroll 1
    for (int c = 0; c < steps; ++c) {
        const int k = 8 * p + c;
        const unsigned u = lb_rank(a[0], pos, prow < Ns && pos >= k);
        unsigned best = __reduce_max_sync(0xffffffffu, u);
        if constexpr (EXACT) {
            best = lb_exact(a[0], u, best);
        } else if constexpr (NCB == 4) {
            if (__any_sync(0xffffffffu, lb_rival(u, best))) best = lb_exact(a[0], u, best);
        }
        double d;
        const zd qr = lb_rcp(a[0], d);
        zd *cw = sh.crow[c & 1][pwarp];
        if (u == best && u != 0) {
            cw[0] = (d > 1e-280 && d < 1e280) ? qr : lb_rcp_any(a[0]);
#pragma unroll
            for (int j = 1; j < 8; ++j) cw[j] = a[j];
            cw[8] = a[0];
        }
        const zd *pr = sh.crow[c & 1][0];
        if (pw > 1) {
            if (lane == 0) ((unsigned *)&sh.rank[c & 1])[pwarp] = best;
            bar_sync(1, 32 * pw);
            const int4 v = sh.rank[c & 1];
            const unsigned t[4] = {(unsigned)v.x, (unsigned)v.y, pw > 2 ? (unsigned)v.z : 0u,
                                   pw > 3 ? (unsigned)v.w : 0u};
            int bw = 0;
            best = t[0];
#pragma unroll
            for (int q = 1; q < 2 * C; ++q)
                if (t[q] > best) { best = t[q]; bw = q; }
            if constexpr (EXACT) {   // the warps' candidates by all bits, then the lower position
                const unsigned top = best;
                unsigned long long v = lb_bits(sh.crow[c & 1][bw][8]);
#pragma unroll
                for (int q = 0; q < 2 * C; ++q) {
                    if (!lb_tied(t[q], top)) continue;
                    const unsigned long long vq = lb_bits(sh.crow[c & 1][q][8]);
                    if (vq > v || (vq == v && t[q] > best)) { v = vq; best = t[q]; bw = q; }
                }
            }
            pr = sh.crow[c & 1][bw];
        } else {
            __syncwarp();
        }
        if constexpr (!EXACT && NCB == 8) tied = tied || lb_rival(u, best);
        const int key = 127 - (int)(best & 127u);   // the pivot's position
        const zd q = pr[0];
        if (pwarp == 0 && lane == 0) {
            const zd a0 = pr[8];
            sh.piv[k] = a0;
            sh.pv[k] = key;
        }
        const bool isP = pos == key;
        if (pos == k) pos = key;
        if (isP) {
            pos = k;
            myslot = c;
            sh.rowOf[k] = prow;
            if constexpr (C > 1) peer->rowOf[k] = prow;
        }
        // the pivot row becomes q times itself, the others lose f times it
        const zd f = isP ? zneg(q) : zmul(a[0], q);
#pragma unroll
        for (int j = 1; j < 8; ++j) {
            const zd pj = pr[j];
            const zd base = isP ? make_double2(0.0, 0.0) : a[j];
            a[j - 1].x = fma(-f.x, pj.x, fma(f.y, pj.y, base.x));
            a[j - 1].y = fma(-f.x, pj.y, fma(-f.y, pj.x, base.y));
        }
        a[7] = zneg(f);
    }
}

struct LbRow {
    zd a[8];
    int pos, slot;
};

// Panel p once more from its columns, the pivots chosen by all bits: about one
// panel in 700 of random 56 x 56 matrices, and matrices with equal entries.  Out
// of line: inside the loop above it cost 8 % without ever running.
template <int C, int NCB>
__device__ __noinline__ LbRow lb_again(LbShared<C, NCB> &sh, LbShared<C, NCB> *peer, int p, int Ns, int pw, int prow, int pos)
{
    LbRow row;
    row.pos = pos;
    row.slot = -1;
    bool tied;
    zd a[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) a[c] = prow < Ns ? sh.G[p & 1][c][prow] : make_double2(0.0, 0.0);
    lb_steps<true>(sh, peer, p, Ns, pw, prow, a, row.pos, row.slot, tied);
#pragma unroll
    for (int c = 0; c < 8; ++c) row.a[c] = a[c];
    return row;
}

// NBK: spin blocks per walker.
template <int NBK, int C, int LB_NCB>
__global__ void __launch_bounds__(LB_NCB == 4 ? 160 : 320 * C, LB_NCB == 4 ? 6 : C == 1 ? 2 : 1)
lu_block_kernel(int nbw, Blocks bl, const zd *S, zd *Sinv, float *Sinv32, long long s32, const int *active, const zd *logw,
                zd logwAdd, zd logwT, zd *logov, int *alive, int *surv, zd *logwOut, double *weight, int *status,
                int mode, int wantInverse)
{
    static_assert(NBK == 1 || C == 1, "two spin blocks are not split");
    typedef LbShared<C, LB_NCB> SH;
    constexpr int LDG = SH::LDG, LB_LDB = SH::LB_LDB;
    extern __shared__ __align__(16) unsigned char smem[];
    SH &sh = *(SH *)smem;
    cg::cluster_group cl = cg::this_cluster();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, fr = lane >> 2, fk = lane & 3;
    const int w = blockIdx.x / (NBK * C), rank = blockIdx.x % (NBK * C);
    const int b = rank / C, half = rank % C;
    const bool act = (active == nullptr) || active[w] != 0;
    const int Ns = b == 0 ? bl.Ns[0] : bl.Ns[1];
    const long long sOff = b == 0 ? bl.sOff[0] : bl.sOff[1];
    const bool inv = wantInverse && (Sinv || Sinv32);
    if (tid == 0) { sh.sing = 0; sh.ln = 0.0; sh.ph = make_double2(1.0, 0.0); }
    if constexpr (C > 1) cl.sync();   // the peer runs and has cleared its flag before it is written to

    auto sync_all = [&]() {
        if constexpr (C > 1) cl.sync(); else __syncthreads();
    };

    if (act && Ns > 0) {   // uniform over a block's CTAs
        const int nb = (Ns + 7) / 8, cb = (nb + C - 1) / C, jb0 = half * cb, ncb = min(cb, nb - jb0);
        const int pw = (Ns + 31) / 32;          // panel warps
        const int r = 8 * warp + fr;            // accumulator row
        const int pwarp = warp - nbw;           // panel warp, from 0; negative in the others
        const int prow = 32 * pwarp + lane;     // panel row
        SH *peer = &sh;
        if constexpr (C > 1) peer = cl.map_shared_rank(&sh, rank ^ 1);

        int pos = prow;                          // position of this lane's panel row

        // the steps of panel p on the columns in G[p & 1], in place
        auto factor = [&](int p) {
            zd (*G)[LDG] = sh.G[p & 1];
            zd a[8];
            if (C > 1 && p > 0 && prow < Ns) pos = sh.pos[prow];   // the other CTA may have had the last panel
#pragma unroll
            for (int c = 0; c < 8; ++c) a[c] = prow < Ns ? G[c][prow] : make_double2(0.0, 0.0);
            int myslot = -1;
            const int steps = min(8, Ns - 8 * p), pos0 = pos;
            bool tied = false;
            lb_steps<false>(sh, peer, p, Ns, pw, prow, a, pos, myslot, tied);
            if (LB_NCB == 8 && bar_any(1, 32 * pw, tied)) {
                LbRow row = lb_again(sh, peer, p, Ns, pw, prow, pos0);
#pragma unroll
                for (int c = 0; c < 8; ++c) a[c] = row.a[c];
                pos = row.pos;
                myslot = row.slot;
            }
            if (prow < Ns) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int c = (j + steps) & 7;   // register j holds panel column c
                    G[c][prow] = a[j];
                    if constexpr (C > 1) peer->G[p & 1][c][prow] = a[j];
                }
                sh.slot[p & 1][prow] = myslot;
                sh.pos[prow] = pos;
                if constexpr (C > 1) {
                    peer->slot[p & 1][prow] = myslot;
                    peer->pos[prow] = pos;
                }
            }
        };
        // eight finished columns (register block j) from a panel buffer to memory
        auto copy_out = [&](int j) {
            zd (*G)[LDG] = sh.G[j & 1];
            for (int c = warp; c < 8; c += blockDim.x >> 5) {
                const int k = 8 * (jb0 + j) + c;
                if (k >= Ns) continue;
                const size_t col = (size_t)Ns * sh.rowOf[k];
                if (Sinv32) {
                    float *Xr = Sinv32 + (size_t)w * s32 + 2 * sOff + col, *Xi = Xr + (size_t)Ns * Ns;
                    for (int i = lane; i < Ns; i += 32) {
                        const zd v = G[c][i];
                        Xr[i] = (float)v.x;
                        Xi[i] = (float)v.y;
                    }
                } else {
                    zd *X = Sinv + (size_t)w * bl.sStride + sOff + col;
                    for (int i = lane; i < Ns; i += 32) X[i] = G[c][i];
                }
            }
        };
        if (warp >= nbw) {
            // the panel warps; iteration -1 factors panel 0
#pragma unroll 1
            for (int p = -1; p < nb; ++p) {
                if (p >= 0) sync_all();
                const int jn = p + 1 < nb ? p + 1 - jb0 : -1;
                if (jn >= 0 && jn < ncb) {
                    bar_sync(2, blockDim.x);   // the panel's columns are stored
                    if (pwarp < pw) factor(p + 1);
                }
            }
            if (pwarp == 0) {
                // log-determinant of the pivots recorded here, while the last
                // update runs
                double ln = 0.0;
                zd ph = make_double2(1.0, 0.0);
                bool zero = false;
                const int k1 = min(Ns, 8 * (jb0 + ncb));
                for (int k = 8 * jb0 + lane; k < k1; k += 32) {
                    const zd d = sh.piv[k];
                    zero = zero || zeq0(d);
                    const double ad = zabs(d);
                    ln += log(ad);
                    zd t = make_double2(d.x / ad, d.y / ad);
                    if (sh.pv[k] != k) t = zneg(t);
                    ph = zmul(ph, t);
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    ln += __shfl_xor_sync(0xffffffffu, ln, o);
                    zd t;
                    t.x = __shfl_xor_sync(0xffffffffu, ph.x, o);
                    t.y = __shfl_xor_sync(0xffffffffu, ph.y, o);
                    ph = zmul(ph, t);
                }
                if (lane == 0) { sh.ln = ln; sh.ph = ph; }
                if (zero) {
                    sh.sing = 1;
                    if constexpr (C > 1) peer->sing = 1;
                }
            }
            sync_all();
            if (inv)
                for (int j = 0; j < ncb; ++j) {
                    __syncthreads();
                    copy_out(j);
                }
        } else {
            double cr[LB_NCB][2], ci[LB_NCB][2];
            const zd *Sg = S + (size_t)w * bl.sStride + sOff;
#pragma unroll
            for (int j = 0; j < LB_NCB; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int c = 8 * (jb0 + j) + 2 * fk + h;
                    const zd v = (j < ncb && r < Ns && c < Ns) ? Sg[r + (size_t)Ns * c] : make_double2(0.0, 0.0);
                    cr[j][h] = v.x;
                    ci[j][h] = v.y;
                }
#pragma unroll 1
            for (int p = -1; p < nb; ++p) {
                const int jp = p - jb0;   // the panel's own block here, if in [0, ncb)
                double ar[2], ai[2], an[2];
                if (p >= 0) {
                    sync_all();   // panel p's result everywhere; the last update is done
                    zd (*G)[LDG] = sh.G[p & 1];
                    const int s = r < Ns ? sh.slot[p & 1][r] : -1;
                    if (s >= 0) {
#pragma unroll
                        for (int j = 0; j < LB_NCB; ++j)
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                sh.B[s][8 * j + 2 * fk + h] = make_double2(cr[j][h], ci[j][h]);
                                cr[j][h] = ci[j][h] = 0.0;
                            }
                    }
#pragma unroll
                    for (int j = 0; j < LB_NCB; ++j)
                        if (j == jp) {
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                const zd v = r < Ns ? G[2 * fk + h][r] : make_double2(0.0, 0.0);
                                cr[j][h] = v.x;
                                ci[j][h] = v.y;
                            }
                        }
                    const int steps = min(8, Ns - 8 * p);
                    for (int e = tid; e < (8 - steps) * LB_LDB; e += 32 * nbw)
                        sh.B[steps + e / LB_LDB][e % LB_LDB] = make_double2(0.0, 0.0);
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const zd v = r < Ns ? G[4 * q + fk][r] : make_double2(0.0, 0.0);
                        ar[q] = v.x; ai[q] = v.y; an[q] = -v.y;
                    }
                    bar_sync(3, 32 * nbw);   // B complete
                }
                auto update = [&](int j) {   // j: unrolled index
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const zd v = sh.B[4 * q + fk][8 * j + fr];
                        dmma(cr[j][0], cr[j][1], ar[q], v.x);
                        dmma(ci[j][0], ci[j][1], ar[q], v.y);
                        dmma(cr[j][0], cr[j][1], an[q], v.y);
                        dmma(ci[j][0], ci[j][1], ai[q], v.x);
                    }
                };
                const int jn = p + 1 < nb ? p + 1 - jb0 : -1;   // the next panel's block here
                const bool next = jn >= 0 && jn < ncb;
                if (next) {
#pragma unroll
                    for (int j = 0; j < LB_NCB; ++j)
                        if (j == jn) {
                            if (p >= 0) update(j);
#pragma unroll
                            for (int h = 0; h < 2; ++h)
                                sh.G[(p + 1) & 1][2 * fk + h][r] = make_double2(cr[j][h], ci[j][h]);
                        }
                    bar_arrive(2, blockDim.x);
                }
                if (p >= 0) {
#pragma unroll
                    for (int j = 0; j < LB_NCB; ++j)
                        if (j < ncb && j != jp && !(next && j == jn) && (inv || j > jp)) update(j);
                }
            }
            sync_all();
            if (inv) {
                // entry (row, column k) of the registers is entry (pos[row], rowOf[k])
                // of the inverse: eight columns at a time through a panel buffer,
                // so that the stores run along a column
                const int pr = r < Ns ? sh.pos[r] : 0;
                const bool sing = sh.sing != 0;
#pragma unroll
                for (int j = 0; j < LB_NCB; ++j) {
                    if (j >= ncb) continue;
                    if (r < Ns) {
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            sh.G[j & 1][2 * fk + h][pr] = sing ? make_double2(0.0, 0.0) : make_double2(cr[j][h], ci[j][h]);
                    }
                    __syncthreads();
                    copy_out(j);
                }
            }
        }
    }
    if constexpr (NBK == 2 || C == 2) cl.sync(); else __syncthreads();
    if (rank == 0 && tid == 0) {
        // the blocks' CTAs hold the parts; without an active walker they are zero
        zd ldB[NBK];
        int sgB[NBK];
        double ln = sh.ln;
        zd ph = sh.ph;
        if constexpr (C == 2) {
            const SH *o = cl.map_shared_rank(&sh, 1);
            ln += o->ln;
            ph = zmul(ph, o->ph);
        }
        ldB[0] = zadd(make_double2(ln, 0.0), zlog(ph));
        sgB[0] = sh.sing;
        if constexpr (NBK == 2) {
            const SH *o = cl.map_shared_rank(&sh, 1);
            ldB[1] = zadd(make_double2(o->ln, 0.0), zlog(o->ph));
            sgB[1] = o->sing;
        }
        lu_walker_finish(w, act, NBK, bl.mult, ldB, sgB, logw, logwAdd, logwT, logov, alive, surv, logwOut, weight,
                         status, mode);
    }
    if constexpr (NBK * C > 1) cl.sync();   // rank 1's shared memory stays until rank 0 has read it
}

template <int NBK, int C, int NCB>
cudaError_t launch(int W, int maxNs, const Blocks &bl, const zd *S, zd *Sinv, float *Sinv32, long long s32,
                   const int *active, const zd *logw, zd logwAdd, zd logwT, zd *logov, int *alive, int *surv,
                   zd *logwOut, double *weight, int *status, int mode, int inv, cudaStream_t s)
{
    static std::atomic<unsigned long long> attr{0};
    cudaError_t r = each_device_once(attr, [] {
        return cudaFuncSetAttribute(lu_block_kernel<NBK, C, NCB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)sizeof(LbShared<C, NCB>));
    });
    if (r != cudaSuccess) return r;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(NBK * C) * (unsigned)W);
    const int nbw = (maxNs + 7) / 8;   // one warp per block row, then the panel warps
    cfg.blockDim = dim3(32u * (unsigned)(nbw + (maxNs + 31) / 32));
    cfg.dynamicSmemBytes = sizeof(LbShared<C, NCB>);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = NBK * C;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = NBK * C > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, lu_block_kernel<NBK, C, NCB>, nbw, bl, S, Sinv, Sinv32, s32, active, logw, logwAdd,
                              logwT, logov, alive, surv, logwOut, weight, status, mode, inv);
}

}  // namespace

bool lu_block_supported(const Blocks &bl)
{
    if (bl.nblk == 1) return bl.Ns[0] <= 128;
    return bl.nblk == 2 && bl.Ns[0] <= 64 && bl.Ns[1] <= 64;
}

cudaError_t lu_block(int W, const Blocks &bl, const zd *S, zd *Sinv, float *Sinv32, const int *active, const zd *logw,
                     zd logwAdd, zd logwT, zd *logov, int *alive, int *surv, zd *logwOut, double *weight, int *status,
                     int mode, bool wantInverse, cudaStream_t s)
{
    g_launch_count++;
    const int maxNs = bl.nblk == 2 && bl.Ns[1] > bl.Ns[0] ? bl.Ns[1] : bl.Ns[0], inv = wantInverse ? 1 : 0;
    const long long s32 = sinv32_stride(bl);
#define LB_ARGS W, maxNs, bl, S, Sinv, Sinv32, s32, active, logw, logwAdd, logwT, logov, alive, surv, logwOut, weight, status, mode, inv, s
    if (maxNs <= 32) return bl.nblk == 2 ? launch<2, 1, 4>(LB_ARGS) : launch<1, 1, 4>(LB_ARGS);
    if (bl.nblk == 2) return launch<2, 1, 8>(LB_ARGS);
    return maxNs <= 64 ? launch<1, 1, 8>(LB_ARGS) : launch<1, 2, 8>(LB_ARGS);
#undef LB_ARGS
}
