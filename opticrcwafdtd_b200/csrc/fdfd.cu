// fdfd.cu -- orf_fdfd2d_*: the 2D TE frequency-domain solver with its adjoint
// (toolbox/+orf/fdfd2D.m:1-19) on the device.
//
//   (1/s_x) d/dx((1/s_x) dE/dx) + (1/s_z) d/dz((1/s_z) dE/dz) + k0^2 eps E = -J
//
// on the FDTD's E_y points, E = 0 outside the grid, stretched-coordinate PML
// s = 1 + i a (depth / L)^3 (e^{-i w t}), discretised with the 5-point
// stencil.  Ordered line by line along the longer axis, the matrix A is block
// tridiagonal: blocks of m = min(nx, nz) unknowns (one line across the
// shorter axis), tridiagonal diagonal blocks, diagonal couplings to the
// neighbouring lines.  M = diag(s_x s_z) A is complex symmetric, and M is what
// is factored: A E = -J is M E = -s J, and the adjoint A.' lam = g is
// M u = g, lam = s u, so one set of factors and one kind of sweep serve both.
//
// Factorisation.  The lines are cut into S segments, with one separator line
// between neighbours.  Each segment is eliminated line by line,
//   D_0 = M_00,  D_b = M_bb - E_b D_{b-1}^{-1} E_b   (E_b: the line couplings),
// by its own thread-block cluster, every D_b inverted and kept; the last
// segment runs from its far end.  The separators' Schur complement is block
// tridiagonal, with dense blocks made of the corner blocks of the segments'
// inverses; those of the segments with two separators come from
//   L_b = -D_b^{-1} E_b L_{b-1} ([last, first]),  F_b = F_{b-1} - L_b.' E_b L_{b-1}
// ([first, first]) by matrix products over all segments at once.  The
// separators are then eliminated from both ends towards the middle one.
// A chain of nb inversions becomes one of about nb / S + S / 2: with one
// segment (a cluster of 16 CTAs on 16 of the 148 SMs) the 501 x 221 guide took
// 400 ms, with 15 segments of 8 CTAs 25.
// A segment between two separators is a closed cavity and can be nearly
// singular where the whole operator is not.  So a factorisation with several
// segments is tried on one right-hand side: if the residual is not that of a
// stable solve, the operator is factored again as one segment.  Each solve of an
// operator in several segments checks its residual too, is refined while that
// is above rounding and falls, and has the operator factored again as one
// segment where it does not come down.
//
// A solve is a forward and a backward sweep of every segment (for the
// separators' right-hand side), the separators' two sweeps, and a second pair
// of segment sweeps with the separators' values known.
#include <cooperative_groups.h>

#include <math_constants.h>

#include <complex>
#include <limits>

#include "runtime.cuh"

namespace cg = cooperative_groups;

namespace orf {
namespace {

constexpr int kFdMaxM = 384;      // largest block (the shorter grid axis)
constexpr unsigned kFull = 0xffffffffu;

struct FdfdDev {
    int m, nb;                 // block size, number of lines
    const double2* diag;       // [nb][m]
    const double2* wc;         // [nb][m]: coupling of p - 1 and p inside the line (entry 0 unused)
    const double2* eb;         // [nb][m]: coupling of line b - 1 and b at p (line 0 unused)
    double2* inv;              // [nb][m][m]: D_b^{-1}, row-major
    int* fault;                // a zero or NaN pivot (singular block, permittivity that is not a number)
    double2* xrow;             // [clusters][kPanel][m]: pivot rows of a panel
};

// Lines a .. a+n-1, eliminated upwards (dir 1) or downwards (dir -1); dense:
// one line whose block is given as a matrix.
struct FdSeg {
    int a, n, dir, pad;
    const double2* dense;
};

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double cabs2(double2 a) { return a.x * a.x + a.y * a.y; }
// c + a b and c - a b
__device__ __forceinline__ double2 cfma(double2 a, double2 b, double2 c) {
    return make_double2(fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y)));
}
__device__ __forceinline__ double2 cfms(double2 a, double2 b, double2 c) {
    return make_double2(fma(-a.x, b.x, fma(a.y, b.y, c.x)), fma(-a.x, b.y, fma(-a.y, b.x, c.y)));
}

// Block inversions by Gauss-Jordan elimination with partial pivoting, blocked:
// pivots are chosen and applied kPanel columns at a time.  CTA c of a cluster
// holds rows [c R, c R + R) of the block in registers (thread (j, h) holds
// column j of the rows of group h).  Per panel:
//   - every CTA pushes its rows' entries of the panel columns into the shared
//     memory of every CTA of the cluster (cluster barrier);
//   - every CTA runs the panel's pivot steps on that copy (thread r holds row
//     r; the pivot is the row of largest magnitude not yet used, compared on
//     the leading 32 bits of |.|^2, the lowest row on a tie: every CTA decides
//     the same).  A step is one barrier of the warps that hold rows: each warp
//     publishes its candidate row, every warp picks the best of them;
//   - the owners write the panel's pivot rows (old values, every column) to a
//     global scratch and, after a second cluster barrier, every CTA reads them
//     (from L2: the fan-out of up to eight whole rows would go through one
//     SM's port);
//   - the rank-kPanel update of the own rows, whose coefficients are what the
//     pivot steps left in the copy's rows.
// Rows are never exchanged: the inverse is the result with its rows in pivot
// order and its columns in the inverse order, written row by row in its true
// place and read back for the next line's Schur complement.
// A panel of a 221-point block takes 12.7 us: the pivot steps 5.1 (0.64 each: the
// reduction, a barrier, and the FP64 latency of a reciprocal and two products
// in a row), the update 3.9 (FP64 units, a third of their rate), the two
// exchanges 3.6.
constexpr int kPanel = 8;

inline size_t fd_factor_smem(int m, int R) {   // s_recv[2][m][W + 1], s_ex[4][m], s_own[R][W + 1], s_pn[R][W + 1]
    return ((size_t)2 * (m + R) * (kPanel + 1) + (size_t)m * 4) * sizeof(double2);
}

template <int RS, int TPC, int NT>
__global__ void __launch_bounds__(NT, 1) k_fdfd_factor(FdfdDev P, const FdSeg* __restrict__ segs) {
    cg::cluster_group cl = cg::this_cluster();
    const int C = (int)cl.num_blocks();
    const int c = (int)cl.block_rank();
    const int cid = (int)(blockIdx.x / C);
    const FdSeg seg = segs[cid];
    const int m = P.m;
    const int mp = (m + 31) / 32 * 32;
    const int R = (m + C - 1) / C;
    const int r0 = c * R;
    const int nr = max(0, min(m, r0 + R) - r0);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int nt = (int)blockDim.x;                     // TPC x mp threads (at most NT)
    const int nrw = mp / 32;                            // warps that hold rows of the panel copy
    const int j = t % mp, h = t / mp;
    const int q0 = h * RS;
    const int r1 = r0 + q0;
    const int nq = max(0, min(RS, nr - q0));
    const bool col = j < m;
    constexpr int W = kPanel, MW = kFdMaxM / 32, WP = W + 1;   // (rows of the copy padded: no bank conflicts)
    double2* xrow = P.xrow + (size_t)cid * W * m;
    // the push: thread t takes entries pq, pq + NPQ, .. for CTAs pc, pc + NPC, ..
    constexpr int NPC = 2;
    const int NPQ = nt / NPC, pq = t % NPQ, pc = t / NPQ;

    extern __shared__ double2 s_dyn[];
    double2* s_recv = s_dyn;                         // [2][m][WP]: the panel columns, every row (old values)
    double2* s_ex = s_recv + (size_t)2 * m * WP;     // [TPC][m]: exchange of a finished block's columns
    double2* s_own = s_ex + (size_t)4 * m;            // [R][WP]: the own rows' panel entries, before the push
    double2* s_pn = s_own + (size_t)R * WP;           // [R][WP]: the own rows' panel entries after the pivot steps
    __shared__ double2 s_cand[2][MW][W];             // a warp's candidate row, by step parity
    __shared__ int2 s_ckey[2][MW];                   // its key and row, 1 / |candidate|^2
    __shared__ double s_cinv[2][MW];
    __shared__ signed char s_kown[32];               // index among the panel's pivots of an own row, or -1
    __shared__ int s_piv[kFdMaxM], s_ipiv[kFdMaxM];

    double2 a[RS];
#pragma unroll
    for (int u = 0; u < RS; ++u) a[u] = make_double2(0.0, 0.0);
    int par = 0;

    cl.sync();   // every CTA of the cluster runs: its shared memory may be written
    for (int it = 0; it < seg.n; ++it) {
        const int b = seg.dir > 0 ? seg.a + it : seg.a + seg.n - 1 - it;
        if (col) {
            const double2* e = P.eb + (size_t)(seg.dir > 0 ? b : b + 1) * m;   // to the line before (it > 0)
            const double2 ej = it > 0 ? e[j] : make_double2(0.0, 0.0);
#pragma unroll
            for (int u = 0; u < RS; ++u) {
                if (u >= nq) break;
                const int p = r1 + u;
                if (seg.dense) {
                    a[u] = seg.dense[(size_t)p * m + j];
                    continue;
                }
                const size_t o = (size_t)b * m + p;
                double2 v = make_double2(0.0, 0.0);
                if (it > 0) {
                    const double2 s = cmul(cmul(e[p], a[u]), ej);
                    v = make_double2(-s.x, -s.y);
                }
                if (j == p) v = cadd(v, P.diag[o]);
                else if (j == p - 1) v = cadd(v, P.wc[o]);
                else if (j == p + 1) v = cadd(v, P.wc[o + 1]);
                a[u] = v;
            }
        }
        bool myused = false;   // row t (thread t < m) is the pivot row of an earlier column
        for (int k0 = 0; k0 < m; k0 += W, par ^= 1) {
            const int we = min(W, m - k0);
            double2* pan = s_recv + (size_t)par * m * WP;
            // ---- the panel entries of the own rows into every CTA of the
            // cluster.  (Buffer par was last read in the update two panels ago;
            // every CTA has since passed a cluster barrier of the panel before.)
            // (columns past the last one are zero)
            if (j >= k0 && j < k0 + W) {
#pragma unroll
                for (int u = 0; u < RS; ++u)
                    if (u < nq) s_own[(q0 + u) * WP + (j - k0)] = col ? a[u] : make_double2(0.0, 0.0);
            }
            __syncthreads();
            for (int q = pq; q < nr * WP; q += NPQ)
                for (int c2 = pc; c2 < C; c2 += NPC) cl.map_shared_rank(pan, c2)[r0 * WP + q] = s_own[q];
            cl.sync();   // the whole panel is here
            // ---- the panel's pivot steps on the copy: thread r holds row r
            if (warp < nrw) {
                double2 pr[W];
                int myk = -1;
#pragma unroll
                for (int l = 0; l < W; ++l) pr[l] = t < m ? pan[t * WP + l] : make_double2(0.0, 0.0);
#pragma unroll
                for (int aa = 0; aa < W; ++aa) {
                    if (aa >= we) break;
                    const int sp = aa & 1;
                    // (the sign bit cleared: a NaN has a key too, and every row is
                    // used once; every row forms its reciprocal while the warps agree)
                    const double dd = cabs2(pr[aa]);
                    const int key = t < m && !myused ? __double2hiint(dd) & 0x7fffffff : -1;
                    const int wkey = __reduce_max_sync(kFull, key);
                    const double inv_dd = dd == 0.0 ? 0.0 : 1.0 / dd;
                    const int wl = __ffs(__ballot_sync(kFull, key == wkey)) - 1;
                    if (lane == wl) {
                        s_ckey[sp][warp] = make_int2(wkey, t);
                        s_cinv[sp][warp] = inv_dd;
#pragma unroll
                        for (int l = 0; l < W; ++l) s_cand[sp][warp][l] = pr[l];
                    }
                    asm volatile("bar.sync 1, %0;" ::"r"(32 * nrw) : "memory");   // the row warps
                    const int2 ck = lane < nrw ? s_ckey[sp][lane] : make_int2(-2, 0);
                    const int bk = __reduce_max_sync(kFull, ck.x);
                    const int bw = __ffs(__ballot_sync(kFull, ck.x == bk)) - 1;
                    const int p = __shfl_sync(kFull, ck.y, bw);
                    const double2* prw = s_cand[sp][bw];
                    const double pinv = s_cinv[sp][bw];
                    const double2 ip = make_double2(prw[aa].x * pinv, -prw[aa].y * pinv);   // 1 / pivot
                    if (t == 0) s_piv[k0 + aa] = p;
                    // others: row -= (f / pivot) pivot row; the pivot row: divided by the pivot
                    const bool me = t == p;
                    double2 g = cmul(pr[aa], ip);
                    g = me ? ip : make_double2(-g.x, -g.y);
                    myused = myused || me;
                    myk = me ? aa : myk;
#pragma unroll
                    for (int l0 = 1; l0 < W; ++l0) {   // the next step's column first
                        const int l = (aa + l0) % W;
                        const double2 base = me ? make_double2(0.0, 0.0) : pr[l];
                        pr[l] = cfma(g, prw[l], base);
                    }
                    pr[aa] = g;
                    // a zero or NaN pivot (as bits: a quiet NaN's key, no further FP64 comparison)
                    if (me && (dd == 0.0 || bk >= 0x7ff80000)) atomicExch(P.fault, 1);
                }
                if (t >= r0 && t < r0 + nr) {
                    s_kown[t - r0] = (signed char)myk;
#pragma unroll
                    for (int l = 0; l < W; ++l) s_pn[(t - r0) * WP + l] = pr[l];
                }
            }
            __syncthreads();
            // ---- the panel's pivot rows (old values, every column) through the
            // scratch rows.  (They were last read before this panel's first
            // cluster barrier.)
            if (col) {
#pragma unroll
                for (int u = 0; u < RS; ++u) {
                    if (u >= nq) break;
                    const int ki = s_kown[q0 + u];
                    if (ki >= 0) __stcg(xrow + (size_t)ki * m + j, a[u]);
                }
            }
            __threadfence();
            cl.sync();   // the pivot rows are in memory
            // ---- the rank-kPanel update of the own rows, four at a time: after
            // the pivot steps the copy's entries of a row are the coefficients
            // of the pivot rows in its update, P^-1 for a pivot row (whose old
            // values count for nothing more) and -A[r, K0] P^-1 for the others
            if (col) {
                double2 rk[W];
#pragma unroll
                for (int l = 0; l < W; ++l) rk[l] = l < we ? __ldcg(xrow + l * m + j) : make_double2(0.0, 0.0);
                const bool inpan = j >= k0 && j < k0 + we;
#pragma unroll
                for (int u0 = 0; u0 < RS; u0 += 4) {
                    if (u0 >= nq) break;
#pragma unroll
                    for (int u = u0; u < u0 + 4; ++u)
                        if (s_kown[min(q0 + u, R - 1)] >= 0) a[u] = make_double2(0.0, 0.0);
#pragma unroll
                    for (int l = 0; l < W; ++l)
#pragma unroll
                        for (int u = u0; u < u0 + 4; ++u)   // (rows past nq: values never used)
                            a[u] = cfma(s_pn[min(q0 + u, R - 1) * WP + l], rk[l], a[u]);
                    if (inpan) {
#pragma unroll
                        for (int u = u0; u < u0 + 4; ++u) a[u] = s_pn[min(q0 + u, R - 1) * WP + (j - k0)];
                    }
                }
            }
        }
        // ---- the inverse: row ipiv[r] is row r of what the threads hold,
        // with column j taken from column ipiv[j]
        __syncthreads();
        if (t < m) s_ipiv[s_piv[t]] = t;
        __syncthreads();
        static_assert(TPC <= 4, "s_ex");
        const int src = col ? s_ipiv[j] : 0;
#pragma unroll
        for (int u = 0; u < RS; ++u) {
            if (col) s_ex[(size_t)h * m + j] = a[u];
            __syncthreads();
            if (col) a[u] = s_ex[(size_t)h * m + src];
            __syncthreads();
        }
        double2* out = P.inv + (size_t)b * m * m;
        if (col) {
#pragma unroll
            for (int u = 0; u < RS; ++u)
                if (u < nq) __stcg(out + (size_t)s_ipiv[r1 + u] * m + j, a[u]);
        }
        if (it + 1 < seg.n) {
            __threadfence();
            cl.sync();   // every CTA's rows of the inverse are in memory
            if (col) {
#pragma unroll
                for (int u = 0; u < RS; ++u)
                    if (u < nq) a[u] = __ldcg(out + (size_t)(r1 + u) * m + j);
            }
        }
    }
    cl.sync();   // no CTA leaves while another may still write its shared memory
}

// C = C0 + sign op(A) diag(e) op(B) of m x m complex matrices, a batch of
// problems per launch (blockIdx.z): 32 x 32 tiles by 128 threads, 2 x 4 results
// a thread, the next 8 columns of op(A) and rows of op(B) loaded into registers
// while the current ones (two shared buffers, one barrier a round) are
// multiplied.  Bound by the FP64 units and, for one or two problems, by a
// tile's own chain of rounds: 28 problems of 221^2 in 0.15 ms (16 TFLOP/s), one in 38 us.
struct FdGemm {
    const double2 *A, *B, *C0, *e;   // C0 null: zero; e null: ones
    double2* C;
    int ta, tb;                      // op is the transpose
    double sign;
};
constexpr int kGT = 32, kGK = 8, kGN = 128;
__global__ void __launch_bounds__(kGN) k_fd_gemm(const FdGemm* __restrict__ probs, int m) {
    const FdGemm g = probs[blockIdx.z];
    __shared__ double2 As[2][kGK][kGT + 1], Bs[2][kGK][kGT + 1];
    constexpr int NL = kGT * kGK / kGN;   // loads of each operand per thread and round
    const int t = threadIdx.x, tx = t & 7, ty = t >> 3;
    const int i0 = blockIdx.y * kGT, j0 = blockIdx.x * kGT;
    const double2 zero = make_double2(0.0, 0.0);
    // element (k, i) of op(A) and (k, j) of op(B), the fast index along memory
    int ka[NL], ia[NL], kb[NL], jb[NL];
#pragma unroll
    for (int s = 0; s < NL; ++s) {
        const int e = t + kGN * s;
        ka[s] = g.ta ? e / kGT : e % kGK;
        ia[s] = g.ta ? e % kGT : e / kGK;
        kb[s] = g.tb ? e % kGK : e / kGT;
        jb[s] = g.tb ? e / kGK : e % kGT;
    }
    double2 ra[NL], rb[NL];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int s = 0; s < NL; ++s) {
            const int k = k0 + ka[s], i = i0 + ia[s];
            ra[s] = i < m && k < m ? __ldg(g.ta ? g.A + (size_t)k * m + i : g.A + (size_t)i * m + k) : zero;
        }
#pragma unroll
        for (int s = 0; s < NL; ++s) {
            const int k = k0 + kb[s], j = j0 + jb[s];
            const bool v = j < m && k < m;
            rb[s] = v ? __ldg(g.tb ? g.B + (size_t)j * m + k : g.B + (size_t)k * m + j) : zero;
            if (g.e && v) rb[s] = cmul(rb[s], __ldg(g.e + k));
        }
    };
    double2 acc[2][4];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[r][q] = zero;
    fetch(0);
    int buf = 0;
    for (int k0 = 0; k0 < m; k0 += kGK, buf ^= 1) {
#pragma unroll
        for (int s = 0; s < NL; ++s) {
            As[buf][ka[s]][ia[s]] = ra[s];
            Bs[buf][kb[s]][jb[s]] = rb[s];
        }
        __syncthreads();   // (the other buffer was read in the round before last's compute, a barrier ago)
        if (k0 + kGK < m) fetch(k0 + kGK);
#pragma unroll
        for (int k = 0; k < kGK; ++k) {
            double2 av[2], bv[4];
#pragma unroll
            for (int r = 0; r < 2; ++r) av[r] = As[buf][k][ty + 16 * r];
#pragma unroll
            for (int q = 0; q < 4; ++q) bv[q] = Bs[buf][k][tx + 8 * q];
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[r][q] = cfma(av[r], bv[q], acc[r][q]);
        }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int i = i0 + ty + 16 * r, j = j0 + tx + 8 * q;
            if (i >= m || j >= m) continue;
            const size_t o = (size_t)i * m + j;
            const double2 v = make_double2(g.sign * acc[r][q].x, g.sign * acc[r][q].y);
            g.C[o] = g.C0 ? cadd(g.C0[o], v) : v;
        }
}

// The separators' system: Kd[j] = M_jj - E [last, last] E - E [first, first] E
// and T[j] = -E L E (the block of separators j and j-1), one row per block.
struct FdSepIn {
    int line;                        // the separator's line
    int hasT;
    const double2 *last, *first;     // corner blocks of the segments before and after
    const double2* L;                // [last, first] of the segment before (hasT)
};
__global__ void k_fd_assemble(FdfdDev P, const FdSepIn* __restrict__ sep, double2* Kd, double2* T) {
    const int m = P.m, q = blockIdx.y, p = blockIdx.x;
    const FdSepIn s = sep[q];
    const double2 *e0 = P.eb + (size_t)s.line * m, *e1 = e0 + m;   // couplings to the line before and after
    const double2* ea = s.hasT ? P.eb + (size_t)(sep[q - 1].line + 1) * m : nullptr;
    for (int j = threadIdx.x; j < m; j += blockDim.x) {
        const size_t o = (size_t)p * m + j;
        double2 v = make_double2(0.0, 0.0);
        if (j == p) v = P.diag[(size_t)s.line * m + p];
        else if (j == p - 1) v = P.wc[(size_t)s.line * m + p];
        else if (j == p + 1) v = P.wc[(size_t)s.line * m + p + 1];
        v = csub(v, cmul(cmul(e0[p], s.last[o]), e0[j]));
        v = csub(v, cmul(cmul(e1[p], s.first[o]), e1[j]));
        Kd[(size_t)q * m * m + o] = v;
        if (s.hasT) {
            const double2 w = cmul(cmul(e0[p], s.L[o]), ea[j]);
            T[(size_t)q * m * m + o] = make_double2(-w.x, -w.y);
        }
    }
}
__global__ void k_fd_transpose(const double2* __restrict__ a, double2* __restrict__ b, int m) {
    __shared__ double2 s[16][17];
    const size_t o = (size_t)blockIdx.z * m * m;
    int i = blockIdx.y * 16 + threadIdx.y, j = blockIdx.x * 16 + threadIdx.x;
    if (i < m && j < m) s[threadIdx.y][threadIdx.x] = a[o + (size_t)i * m + j];
    __syncthreads();
    i = blockIdx.x * 16 + threadIdx.y;
    j = blockIdx.y * 16 + threadIdx.x;
    if (i < m && j < m) b[o + (size_t)i * m + j] = s[threadIdx.x][threadIdx.y];
}

// Products of m x m matrices with vectors by a cluster: CTA c owns the rows
// (and the vector entries) [c R, c R + R), warp w of it the rows w, w + NT/32,
// .., a lane NQ columns of each.  A matrix's rows wait in registers, loaded
// before the vector is known; the vector's entries are pushed into the shared
// memory of every CTA (one cluster barrier per product).
template <int NQ, int RW, int NT>
struct FdMv {
    static constexpr int NW = NT / 32;
    int m, R, r0, nr, lane, warp;
    double2 M[RW][NQ];
    __device__ void load(const double2* __restrict__ A) {   // A: [m][m]
#pragma unroll
        for (int r = 0; r < RW; ++r) {
            const int row = warp + r * NW;
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const int cc = lane + 32 * q;
                M[r][q] = row < nr && cc < m ? __ldcg(A + (size_t)(r0 + row) * m + cc) : make_double2(0.0, 0.0);
            }
        }
    }
    __device__ void dot(const double2* v, double2 (&acc)[RW]) const {   // per lane
#pragma unroll
        for (int r = 0; r < RW; ++r) acc[r] = make_double2(0.0, 0.0);
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const int cc = lane + 32 * q;
            const double2 x = cc < m ? v[cc] : make_double2(0.0, 0.0);
#pragma unroll
            for (int r = 0; r < RW; ++r) acc[r] = cfma(M[r][q], x, acc[r]);
        }
    }
    // Sums over the warp.  Halves of the warp take one row each (RW 2), then
    // half of those the real and half the imaginary part, so a value is
    // exchanged once per level: lane returns the sum of part() of row().
    __device__ int row() const { return warp + (RW == 2 ? (lane >> 4) * NW : 0); }
    __device__ int part() const { return (RW == 2 ? lane >> 3 : lane >> 4) & 1; }
    __device__ bool writes() const { return (lane & (RW == 2 ? 7 : 15)) == 0 && row() < nr; }
    __device__ double reduce(const double2 (&acc)[RW]) const {
        static_assert(RW <= 2, "two rows at most");
        double2 v = acc[0];
        int o = 16;
        if constexpr (RW == 2) {
            const bool up = (lane & 16) != 0;
            const double2 keep = up ? acc[1] : acc[0], give = up ? acc[0] : acc[1];
            v.x = keep.x + __shfl_xor_sync(kFull, give.x, 16);
            v.y = keep.y + __shfl_xor_sync(kFull, give.y, 16);
            o = 8;
        }
        const bool im = (lane & o) != 0;
        double u = (im ? v.y : v.x) + __shfl_xor_sync(kFull, im ? v.x : v.y, o);
#pragma unroll
        for (int q = 8; q > 0; q >>= 1)
            if (q < o) u += __shfl_xor_sync(kFull, u, q);
        return u;
    }
};
// entry p of a vector, as its two parts
__device__ __forceinline__ double* part_of(double2* v, size_t p, int part) { return reinterpret_cast<double*>(v + p) + part; }

// Forward and backward sweep of every segment (a cluster each): X of the
// segment's lines for right-hand side f, with E = 0 on the separators
// (seps 0) or with their values in X (seps 1).
//   w_b = f_b - E_b y_{b-1},  y_b = D_b^{-1} w_b,  x_b = y_b - D_b^{-1} E_{b+1} x_{b+1}
// A product takes 3 us on the 501 x 221 guide (the 15 clusters read the
// inverses at 3.8 TB/s); a second matrix on its way through shared memory
// made it 3.5.
template <int NQ, int RW, int NT>
__global__ void __launch_bounds__(NT, 1) k_fdfd_sweep(FdfdDev P, const FdSeg* __restrict__ segs,
                                                      const double2* __restrict__ f, double2* X, int seps) {
    cg::cluster_group cl = cg::this_cluster();
    const int C = (int)cl.num_blocks(), c = (int)cl.block_rank();
    const FdSeg seg = segs[blockIdx.x / C];
    const int m = P.m, t = threadIdx.x;
    FdMv<NQ, RW, NT> mv;
    mv.m = m;
    mv.R = (m + C - 1) / C;
    mv.r0 = c * mv.R;
    mv.nr = max(0, min(m, mv.r0 + mv.R) - mv.r0);
    mv.lane = t & 31;
    mv.warp = t >> 5;
    __shared__ double2 s_full[2][kFdMaxM];   // the vector multiplied, by step parity
    __shared__ double2 s_y[32];              // the own entries of the last product
    cl.sync();   // every CTA of the cluster runs: its shared memory may be written
    const int d = seg.dir, first = d > 0 ? seg.a : seg.a + seg.n - 1;
    // couplings of line b to the one before (prev) and after it, in the order of elimination
    auto e_prev = [&](int b) { return P.eb + (size_t)(d > 0 ? b : b + 1) * m; };
    auto e_next = [&](int b) { return P.eb + (size_t)(d > 0 ? b + 1 : b) * m; };
    // thread t pushes entry t % nr of the vector to CTA t / nr
    const int npush = mv.nr * C;
    int par = 0;
    const double2 zero = make_double2(0.0, 0.0);
    constexpr int NPU = ((NQ > 8 ? 24 * 16 : 32 * 8) + NT - 1) / NT;   // pushes per thread at most
    // separators next to the segment (seps)
    const bool sp0 = seps && seg.a > 0, sp1 = seps && seg.a + seg.n < P.nb;

    // the entry this thread pushes, and what forms it: f and the coupling are
    // loaded a step ahead
    static_assert(NPU == 1, "one entry per thread");
    const bool pushes = t < npush;
    const int c2 = pushes ? t / mv.nr : 0, prow = pushes ? t - c2 * mv.nr : 0, pp = mv.r0 + prow;
    double2* const dst[2] = {cl.map_shared_rank(&s_full[0][0], c2) + pp, cl.map_shared_rank(&s_full[1][0], c2) + pp};
    double2 fv = zero, ev = zero;
    auto ahead_fwd = [&](int i) {   // step i of the forward sweep
        if (!pushes || i >= seg.n) return;
        const int b = first + d * i;
        fv = __ldg(f + (size_t)b * m + pp);
        if (i > 0) ev = __ldg(e_prev(b) + pp);
        if (sp0 && b == seg.a) fv = cfms(P.eb[(size_t)b * m + pp], X[(size_t)(b - 1) * m + pp], fv);
        if (sp1 && b == seg.a + seg.n - 1) fv = cfms(P.eb[(size_t)(b + 1) * m + pp], X[(size_t)(b + 1) * m + pp], fv);
    };
    auto ahead_back = [&](int i) {
        if (pushes && i >= 0) ev = __ldg(e_next(first + d * i) + pp);
    };
    mv.load(P.inv + (size_t)first * m * m);
    ahead_fwd(0);
    // ---- forward
    for (int i = 0; i < seg.n; ++i) {
        const int b = first + d * i;
        if (pushes) *dst[par] = i > 0 ? cfms(ev, s_y[prow], fv) : fv;
        if (i + 1 < seg.n) ahead_fwd(i + 1);
        else ahead_back(seg.n - 2);
        cl.sync();
        double2 acc[RW];
        mv.dot(s_full[par], acc);
        // the next matrix: the next line's, or (backward) the last line but one's
        if (i + 1 < seg.n) mv.load(P.inv + (size_t)(b + d) * m * m);
        else if (seg.n > 1) mv.load(P.inv + (size_t)(b - d) * m * m);
        const double y = mv.reduce(acc);
        if (mv.writes()) {
            *part_of(s_y, mv.row(), mv.part()) = y;
            *part_of(X, (size_t)b * m + mv.r0 + mv.row(), mv.part()) = y;
        }
        __syncthreads();
        par ^= 1;
    }
    // ---- backward (s_y: x of the last line)
    for (int i = seg.n - 2; i >= 0; --i) {
        const int b = first + d * i;
        if (pushes) *dst[par] = cmul(ev, s_y[prow]);
        ahead_back(i - 1);
        const double y = mv.writes() ? *part_of(X, (size_t)b * m + mv.r0 + mv.row(), mv.part()) : 0.0;
        cl.sync();
        double2 acc[RW];
        mv.dot(s_full[par], acc);
        if (i > 0) mv.load(P.inv + (size_t)(b - d) * m * m);
        const double x = y - mv.reduce(acc);
        if (mv.writes()) {
            *part_of(s_y, mv.row(), mv.part()) = x;
            *part_of(X, (size_t)b * m + mv.r0 + mv.row(), mv.part()) = x;
        }
        __syncthreads();
        par ^= 1;
    }
    cl.sync();   // no CTA leaves while another may still write its shared memory
}

// The separators' sweeps, cluster 0 from the first one and cluster 1 from the
// last one to the middle: phase 0 forward,
//   z_j = r_j - Y z of the one before,  V_j = Inv_j z_j,
// phase 1 the middle one (both clusters) and back, x_j = V_j - Y_j.' x_next.
// r_j = f_j - E x of the lines beside it (the segments' first sweeps).
struct FdRed {
    int J, mid;
    const int* line;                 // [J]
    const double2 *Y, *YT;           // [J][m][m]: z of the next separator towards mid -= Y_j z_j
    double2 *V, *Z;                  // [J][m], [2][m]: what reaches the middle one from each side
};
template <int NQ, int RW, int NT>
__global__ void __launch_bounds__(NT, 1) k_fdfd_red(FdfdDev P, FdRed D, const double2* __restrict__ f, double2* X,
                                                    int phase) {
    cg::cluster_group cl = cg::this_cluster();
    const int C = (int)cl.num_blocks(), c = (int)cl.block_rank(), side = (int)(blockIdx.x / C);
    const int m = P.m, t = threadIdx.x;
    FdMv<NQ, RW, NT> mv;
    mv.m = m;
    mv.R = (m + C - 1) / C;
    mv.r0 = c * mv.R;
    mv.nr = max(0, min(m, mv.r0 + mv.R) - mv.r0);
    mv.lane = t & 31;
    mv.warp = t >> 5;
    __shared__ double2 s_full[2][kFdMaxM];
    __shared__ double2 s_y[32];
    cl.sync();   // every CTA of the cluster runs: its shared memory may be written
    const int npush = mv.nr * C;
    int par = 0;
    constexpr int NPU = ((NQ > 8 ? 24 * 16 : 32 * 8) + NT - 1) / NT;
    const int d = side == 0 ? 1 : -1, j0 = side == 0 ? 0 : D.J - 1;
    const int n = side == 0 ? D.mid : D.J - 1 - D.mid;   // separators before the middle one
    auto rhs = [&](int j, int p) {
        const int b = D.line[j];
        double2 r = f[(size_t)b * m + p];
        r = cfms(P.eb[(size_t)b * m + p], X[(size_t)(b - 1) * m + p], r);
        return cfms(P.eb[(size_t)(b + 1) * m + p], X[(size_t)(b + 1) * m + p], r);
    };
    // the vector of a product, entry by entry
    auto push = [&](auto&& value) {
#pragma unroll
        for (int u = 0; u < NPU; ++u) {
            const int q = t + u * NT;
            if (q >= npush) break;
            const int c2 = q / mv.nr, row = q - c2 * mv.nr;
            cl.map_shared_rank(&s_full[par][0], c2)[mv.r0 + row] = value(row, mv.r0 + row);
        }
        cl.sync();
    };
    double2 acc[RW];
    if (phase == 0) {
        if (n > 0) mv.load(D.Y + (size_t)j0 * m * m);
        for (int i = 0; i < n; ++i) {
            const int j = j0 + d * i;
            push([&](int row, int p) {
                const double2 r = rhs(j, p);
                return i > 0 ? csub(r, s_y[row]) : r;
            });
            mv.dot(s_full[par], acc);
            mv.load(P.inv + (size_t)D.line[j] * m * m);
            const double y = mv.reduce(acc);   // (s_y was read before the push's cluster barrier)
            if (mv.writes()) {
                *part_of(s_y, mv.row(), mv.part()) = y;
                if (i + 1 == n) *part_of(D.Z, (size_t)side * m + mv.r0 + mv.row(), mv.part()) = y;
            }
            mv.dot(s_full[par], acc);
            if (i + 1 < n) mv.load(D.Y + (size_t)(j + d) * m * m);
            const double v = mv.reduce(acc);
            if (mv.writes()) *part_of(D.V, (size_t)j * m + mv.r0 + mv.row(), mv.part()) = v;
            __syncthreads();
            par ^= 1;
        }
    } else {
        mv.load(P.inv + (size_t)D.line[D.mid] * m * m);
        push([&](int row, int p) {
            (void)row;
            double2 r = rhs(D.mid, p);
            if (D.mid > 0) r = csub(r, D.Z[p]);
            if (D.mid < D.J - 1) r = csub(r, D.Z[m + p]);
            return r;
        });
        mv.dot(s_full[par], acc);
        if (n > 0) mv.load(D.YT + (size_t)(D.mid - d) * m * m);
        const double xm = mv.reduce(acc);
        if (mv.writes()) {
            *part_of(s_y, mv.row(), mv.part()) = xm;
            if (side == 0) *part_of(X, (size_t)D.line[D.mid] * m + mv.r0 + mv.row(), mv.part()) = xm;
        }
        __syncthreads();
        par ^= 1;
        for (int i = n - 1; i >= 0; --i) {
            const int j = j0 + d * i;
            push([&](int row, int) { return s_y[row]; });
            mv.dot(s_full[par], acc);
            if (i > 0) mv.load(D.YT + (size_t)(j - d) * m * m);
            const double v = mv.writes() ? *part_of(D.V, (size_t)j * m + mv.r0 + mv.row(), mv.part()) : 0.0;
            const double x = v - mv.reduce(acc);
            if (mv.writes()) {
                *part_of(s_y, mv.row(), mv.part()) = x;
                *part_of(X, (size_t)D.line[j] * m + mv.r0 + mv.row(), mv.part()) = x;
            }
            __syncthreads();
            par ^= 1;
        }
    }
    cl.sync();   // no CTA leaves while another may still write its shared memory
}

__device__ __forceinline__ double2 fd_scaled(double2 a, int e) {
    return e == 0 ? a : make_double2(scalbn(a.x, e), scalbn(a.y, e));
}
// bits of the largest |re| or |im| (infinity's where an entry is not finite)
__global__ void k_fd_biggest(const double2* __restrict__ v, size_t n, unsigned long long* big) {
    double a = 0.0;
    bool nan = false;
    for (size_t o = blockIdx.x * (size_t)blockDim.x + threadIdx.x; o < n; o += (size_t)gridDim.x * blockDim.x) {
        const double2 x = v[o];
        nan = nan || x.x != x.x || x.y != x.y;
        a = fmax(a, fmax(fabs(x.x), fabs(x.y)));
    }
    if (nan) a = CUDART_INF;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a = fmax(a, __shfl_xor_sync(kFull, a, o));
    if ((threadIdx.x & 31) == 0) atomicMax(big, (unsigned long long)__double_as_longlong(a));
}

// The caller's vector (i + nx k) and the block layout (b m + p), with the
// scaling by s = s_x(i) s_z(k): f = -s J (mode 0) or g (mode 1); E = x or s x.
// f is taken by 2^-ex and the result by 2^ex.  k_fd_in clears mx for the residual
// that follows.
struct FdMap {
    int nx, nz, along_x;
    const double2 *sx, *sz;
    __device__ size_t at(int i, int k) const { return along_x ? (size_t)i * nz + k : (size_t)k * nx + i; }
};
__global__ void k_fd_in(FdMap mp, const double2* __restrict__ v, double2* __restrict__ f, int mode,
                        int ex, unsigned long long* mx) {
    if (blockIdx.x == 0 && threadIdx.x < 3) mx[threadIdx.x] = 0;
    for (size_t g = blockIdx.x * (size_t)blockDim.x + threadIdx.x; g < (size_t)mp.nx * mp.nz;
         g += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(g % mp.nx), k = (int)(g / mp.nx);
        double2 x = fd_scaled(v[g], -ex);
        if (mode == 0) {
            x = cmul(cmul(mp.sx[i], mp.sz[k]), x);
            x = make_double2(-x.x, -x.y);
        }
        f[mp.at(i, k)] = x;
    }
}
__global__ void k_fd_out(FdMap mp, const double2* __restrict__ x, double2* __restrict__ v, int mode,
                         int ex) {
    for (size_t g = blockIdx.x * (size_t)blockDim.x + threadIdx.x; g < (size_t)mp.nx * mp.nz;
         g += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(g % mp.nx), k = (int)(g / mp.nx);
        const double2 y = x[mp.at(i, k)];
        v[g] = fd_scaled(mode == 0 ? y : cmul(cmul(mp.sx[i], mp.sz[k]), y), ex);
    }
}
// r = f - M x and the largest |r|^2, |x|^2 and |f|^2 (bits of non-negative
// doubles order as integers)
__global__ void k_fd_residual(FdfdDev P, const double2* __restrict__ f, const double2* __restrict__ x,
                              double2* __restrict__ r, unsigned long long* mx) {
    const size_t N = (size_t)P.nb * P.m;
    double v[3] = {0.0, 0.0, 0.0};
    bool nan = false;
    for (size_t o = blockIdx.x * (size_t)blockDim.x + threadIdx.x; o < N; o += (size_t)gridDim.x * blockDim.x) {
        const int b = (int)(o / P.m), p = (int)(o - (size_t)b * P.m);
        const double2 xo = x[o], fo = f[o];
        double2 s = cfms(P.diag[o], xo, fo);
        if (p > 0) s = cfms(P.wc[o], x[o - 1], s);
        if (p + 1 < P.m) s = cfms(P.wc[o + 1], x[o + 1], s);
        if (b > 0) s = cfms(P.eb[o], x[o - P.m], s);
        if (b + 1 < P.nb) s = cfms(P.eb[o + P.m], x[o + P.m], s);
        r[o] = s;
        const double a[3] = {cabs2(s), cabs2(xo), cabs2(fo)};
        for (int q = 0; q < 3; ++q) {
            nan = nan || !(a[q] >= 0.0);
            v[q] = fmax(v[q], a[q]);
        }
    }
    if (nan) v[0] = CUDART_INF;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[q] = fmax(v[q], __shfl_xor_sync(kFull, v[q], o));
        if ((threadIdx.x & 31) == 0) atomicMax(mx + q, (unsigned long long)__double_as_longlong(v[q]));
    }
}
// x += dx; clears mx for the residual that follows
__global__ void k_fd_add(double2* __restrict__ x, const double2* __restrict__ dx, size_t n, unsigned long long* mx) {
    if (blockIdx.x == 0 && threadIdx.x < 3) mx[threadIdx.x] = 0;
    for (size_t o = blockIdx.x * (size_t)blockDim.x + threadIdx.x; o < n; o += (size_t)gridDim.x * blockDim.x)
        x[o] = cadd(x[o], dx[o]);
}
// the right-hand side a factorisation is tried on: of magnitude one everywhere, no pattern
// (the index hashed with the multipliers and shifts of the xxHash32 finaliser)
__global__ void k_fd_probe(double2* f, size_t n, unsigned long long* mx) {
    if (blockIdx.x == 0 && threadIdx.x < 3) mx[threadIdx.x] = 0;
    for (size_t o = blockIdx.x * (size_t)blockDim.x + threadIdx.x; o < n; o += (size_t)gridDim.x * blockDim.x) {
        unsigned h = (unsigned)o * 2654435761u;
        h ^= h >> 15;
        h *= 2246822519u;
        h ^= h >> 13;
        f[o] = make_double2((double)(h & 0xffffu) / 32768.0 - 1.0, (double)(h >> 16) / 32768.0 - 1.0);
    }
}

// Shape for block size m: CTAs of a cluster (rows per CTA: at most 32, 24 for
// the 16 of a non-portable cluster).
int fd_shape(int m, int* C) {
    static const int kC[4] = {2, 4, 8, 16}, kM[4] = {64, 128, 256, kFdMaxM};
    for (int q = 0; q < 4; ++q)
        if (m <= kM[q]) {
            *C = kC[q];
            return ORF_OK;
        }
    set_error("fdfd2D: the shorter grid axis has %d points, above the %d this solver takes", m, kFdMaxM);
    return ORF_ETOOLARGE;
}

// limit: the most dynamic shared memory any launch of this kernel asks for (0:
// none).  The attribute belongs to the kernel, not to a launch, so every launch
// sets the same value: one that followed the block size would lower what
// another host thread is about to launch with.
template <class K, class... Args>
cudaError_t launch_cluster(K kern, int clusters, int C, int threads, size_t smem, size_t limit, cudaStream_t s,
                           int* most, Args... args) {
    if (C > 8) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return e;
    }
    if (limit > 0) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit);
        if (e != cudaSuccess) return e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(C * clusters), 1, 1);
    cfg.blockDim = dim3((unsigned)threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)C;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (most) return cudaOccupancyMaxActiveClusters(most, kern, &cfg);   // resident at once; no launch
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

// the factor kernel of block size m (most: only ask how many clusters fit)
cudaError_t launch_factor(const FdfdDev& P, int C, const FdSeg* segs, int n, cudaStream_t s, int* most) {
    const int mp = (P.m + 31) / 32 * 32, R = (P.m + C - 1) / C;
    const size_t smem = fd_factor_smem(P.m, R);
    // (the largest block of each kernel: fd_shape)
    if (C <= 4) return launch_cluster(k_fdfd_factor<8, 4, 512>, n, C, 4 * mp, smem, fd_factor_smem(128, 32), s, most, P, segs);
    if (C == 8) return launch_cluster(k_fdfd_factor<16, 2, 512>, n, C, 2 * mp, smem, fd_factor_smem(256, 32), s, most, P, segs);
    return launch_cluster(k_fdfd_factor<24, 1, 384>, n, C, mp, smem, fd_factor_smem(kFdMaxM, 24), s, most, P, segs);
}
cudaError_t launch_sweep(const FdfdDev& P, int C, const FdSeg* segs, int n, const double2* f, double2* X, int seps,
                         cudaStream_t s) {
    if (C == 2) return launch_cluster(k_fdfd_sweep<2, 2, 512>, n, C, 512, 0, 0, s, nullptr, P, segs, f, X, seps);
    if (C == 4) return launch_cluster(k_fdfd_sweep<4, 2, 512>, n, C, 512, 0, 0, s, nullptr, P, segs, f, X, seps);
    if (C == 8) return launch_cluster(k_fdfd_sweep<8, 2, 512>, n, C, 512, 0, 0, s, nullptr, P, segs, f, X, seps);
    return launch_cluster(k_fdfd_sweep<12, 2, 384>, n, C, 384, 0, 0, s, nullptr, P, segs, f, X, seps);
}
cudaError_t launch_red(const FdfdDev& P, int C, const FdRed& D, const double2* f, double2* X, int phase,
                       cudaStream_t s) {
    if (C == 2) return launch_cluster(k_fdfd_red<2, 2, 512>, 2, C, 512, 0, 0, s, nullptr, P, D, f, X, phase);
    if (C == 4) return launch_cluster(k_fdfd_red<4, 2, 512>, 2, C, 512, 0, 0, s, nullptr, P, D, f, X, phase);
    if (C == 8) return launch_cluster(k_fdfd_red<8, 2, 512>, 2, C, 512, 0, 0, s, nullptr, P, D, f, X, phase);
    return launch_cluster(k_fdfd_red<12, 2, 384>, 2, C, 384, 0, 0, s, nullptr, P, D, f, X, phase);
}

// Segments for nb lines when `most` clusters run at once: the chain is
// nb / S inversions in the segments and S / 2 at the separators (each with two
// matrix products behind it), so as many as fit, up to about sqrt(2 nb).
int fd_segments(int nb, int most) {
    int best = 1;
    double best_t = nb;
    for (int S = 2; S <= most && nb - (S - 1) >= 4 * S; ++S) {
        const double t = std::ceil((double)(nb - (S - 1)) / S) * (S > 2 ? 1.15 : 1.0) + 1.2 * (S / 2);
        if (t < best_t) {
            best_t = t;
            best = S;
        }
    }
    return best;
}

using cplx = std::complex<double>;

// s at the integer points (half = false) or at the half points u = -1/2 ..
// n-1/2 (half = true) of one axis: s = 1 + i a (depth / L)^3 inside the
// npml-cell layers, depth = npml - u below the low edge, u - (n-1-npml)
// above the high edge (the FDTD's CPML convention), a = 2 ln(1/R) / (k0 L)
std::vector<cplx> fd_stretch(int n, int npml, double d, double k0, double R, bool half) {
    const int npts = half ? n + 1 : n;
    std::vector<cplx> s(npts, cplx(1.0, 0.0));
    if (npml <= 0) return s;
    const double L = npml * d;
    const double a = 2.0 * std::log(1.0 / R) / (k0 * L);
    const double lo = npml, hi = (n - 1) - npml;
    for (int q = 0; q < npts; ++q) {
        const double u = half ? q - 0.5 : (double)q;
        double depth = 0.0;
        if (u < lo) depth = lo - u;
        else if (u > hi) depth = u - hi;
        const double r = depth * d / L;
        s[q] = cplx(1.0, a * r * r * r);
    }
    return s;
}

}  // namespace
}  // namespace orf

using namespace orf;

struct orf_fdfd {
    orf_ctx* ctx = nullptr;
    int nx = 0, nz = 0, m = 0, nb = 0, C = 8;
    bool along_x = true;   // blocks are lines of constant x (m = nz)
    int S = 1, planned = 1;   // segments of the factors, and as chosen for the grid
    double mnorm = 0.0;    // scale of |M|: its largest row sum, the two couplings along an axis taken together
    Arena ar;
    double2 *diag = nullptr, *wc = nullptr, *eb = nullptr, *sx = nullptr, *sz = nullptr;
    double2 *inv = nullptr, *vin = nullptr, *vout = nullptr, *xrow = nullptr;
    double2 *f = nullptr, *x = nullptr, *r = nullptr, *dx = nullptr, *Y = nullptr, *YT = nullptr, *V = nullptr,
            *Z = nullptr;
    unsigned long long* mx = nullptr;   // largest |r|^2, |x|^2, |f|^2; the caller's largest entry (k_fd_biggest)
    double* h_mx = nullptr;             // the same on the host (pinned)
    int scale = 0;                      // of f
    double eta = -1.0;                  // residual of the last solve (-1: none taken)
    bool singular = false;              // a zero or NaN pivot in the last factorisation
    FdSeg* segs = nullptr;
    int *line = nullptr, *fault = nullptr;
    cudaEvent_t copied = nullptr;       // the result has reached the staging buffer
    ~orf_fdfd() {
        if (ar.base) {
            cudaStreamSynchronize(ctx->stream);
            ar.release();
        }
        if (copied) cudaEventDestroy(copied);
        host_mapped_free(h_mx);
        if (ctx) ctx_release(ctx);
    }
    FdfdDev dev() const { return FdfdDev{m, nb, diag, wc, eb, inv, fault, xrow}; }
    FdMap map() const { return FdMap{nx, nz, along_x ? 1 : 0, sx, sz}; }
    size_t N() const { return (size_t)nx * nz; }
    // (i, k) of the grid <-> entry b * m + p of the block layout
    size_t at(int i, int k) const { return along_x ? (size_t)i * m + k : (size_t)k * m + i; }
    // x of M x = f for the right-hand side in `rhs`, into `out`
    int solve(const double2* rhs, double2* out) {
        cudaStream_t st = ctx->stream;
        const FdfdDev P = dev();
        ORF_CUDA(launch_sweep(P, C, segs, S, rhs, out, 0, st));
        if (S > 1) {
            const FdRed D{S - 1, (S - 1) / 2, line, Y, YT, V, Z};
            ORF_CUDA(launch_red(P, C, D, rhs, out, 0, st));
            ORF_CUDA(launch_red(P, C, D, rhs, out, 1, st));
            ORF_CUDA(launch_sweep(P, C, segs, S, rhs, out, 1, st));
        }
        return ORF_OK;
    }
    // f of the caller's right-hand side (in vin), taken by 2^-scale
    int rhs(int mode) {
        k_fd_in<<<296, 256, 0, ctx->stream>>>(map(), vin, f, mode, scale, mx);
        ORF_CUDA(cudaGetLastError());
        return ORF_OK;
    }
    // r = f - M x on the stream; its size reaches the host with it (mx cleared by
    // the kernel that formed f or x)
    int residual() {
        cudaStream_t st = ctx->stream;
        k_fd_residual<<<296, 256, 0, st>>>(dev(), f, x, r, mx);
        ORF_CUDA(cudaGetLastError());
        ORF_CUDA(cudaMemcpyAsync(h_mx, mx, 3 * sizeof *mx, cudaMemcpyDeviceToHost, st));
        return ORF_OK;
    }
    // its size against rounding, |r| / (|M| |x| + |f|) with the largest entries,
    // once the stream has reached it
    double eta_now() const {
        const double den = mnorm * std::sqrt(h_mx[1]) + std::sqrt(h_mx[2]);
        return h_mx[0] == 0.0 ? 0.0 : std::sqrt(h_mx[0]) / den;
    }
    int refine() {
        ORF_TRY(solve(r, dx));
        k_fd_add<<<296, 256, 0, ctx->stream>>>(x, dx, N(), mx);
        ORF_CUDA(cudaGetLastError());
        return ORF_OK;
    }
    template <class Out>
    int settle(int mode, Out&& out);
    int scaled(int mode, bool* finite);
    int factor(int nseg);
    int refuse_singular() const {
        if (!singular) return ORF_OK;
        set_error("fdfd2D: the operator is singular (a zero or NaN pivot in the block elimination)");
        return ORF_EINVAL;
    }
};

namespace {
// A solve with a residual above kEtaRefine takes a step of refinement: as one
// segment the residuals are 6e-17 .. 6e-16 (error against an exact solve 2e-14
// .. 1.4e-13 on grids of 150 x 92 .. 600 x 250), as 15 segments 1e-16 .. 5e-15
// (up to 3e-12), and 1e-17 .. 2e-16 (2e-14 .. 9e-14) after the step.  Above
// kEtaAccept it takes up to kRefineSteps in all while the residual falls; if it
// still ends above, the operator is factored again as one segment (whose solves
// are refined above kEtaAccept only).  So is a factorisation whose trial solve
// has a residual above kEtaTrial.
constexpr double kEtaRefine = 1e-16, kEtaAccept = 1e-15, kEtaTrial = 1e-11;
constexpr int kRefineSteps = 3;
}  // namespace

// The residual's squares vanish or overflow, or it is not a number: the right-hand
// side brought to [1, 2) by a power of two, and solved again.  The result is the same to the bit as at an
// ordinary magnitude.  finite: false where an entry is not, or all are zero (there
// is nothing to refine).
int orf_fdfd::scaled(int mode, bool* finite) {
    cudaStream_t st = ctx->stream;
    ORF_CUDA(cudaMemsetAsync(mx + 3, 0, sizeof *mx, st));
    k_fd_biggest<<<296, 256, 0, st>>>(vin, N(), mx + 3);
    ORF_CUDA(cudaGetLastError());
    ORF_CUDA(cudaMemcpyAsync(h_mx + 3, mx + 3, sizeof *mx, cudaMemcpyDeviceToHost, st));
    ORF_CUDA(cudaStreamSynchronize(st));
    *finite = std::isfinite(h_mx[3]) && h_mx[3] > 0.0;
    if (!*finite) return ORF_OK;
    scale = std::ilogb(h_mx[3]);
    ORF_TRY(rhs(mode));
    ORF_TRY(solve(f, x));
    ORF_TRY(residual());
    ORF_CUDA(cudaStreamSynchronize(st));
    return ORF_OK;
}

// From the first x of M x = f to the one handed over by out(beside), which enqueues
// the copy, then beside, and waits for the copy: refined as above, the residual of
// the refined x taken while the host moves the result (out runs again in the rare
// case that more is to do).
template <class Out>
int orf_fdfd::settle(int mode, Out&& out) {
    ORF_TRY(residual());
    ORF_CUDA(cudaStreamSynchronize(ctx->stream));
    if (!(h_mx[2] > 1e-200 && h_mx[2] < 1e200) || !std::isfinite(eta_now())) {
        bool finite = false;
        ORF_TRY(scaled(mode, &finite));
        if (!finite) {
            eta = h_mx[3] == 0.0 ? 0.0 : std::numeric_limits<double>::quiet_NaN();
            return out([]() -> int { return ORF_OK; });
        }
    }
    eta = eta_now();
    if (eta <= (S > 1 ? kEtaRefine : kEtaAccept)) return out([]() -> int { return ORF_OK; });
    for (int k = 0; k < kRefineSteps; ++k) {
        const double before = eta;
        ORF_TRY(refine());
        ORF_TRY(out([this] { return residual(); }));
        ORF_CUDA(cudaStreamSynchronize(ctx->stream));
        eta = eta_now();
        if (eta <= kEtaAccept) return ORF_OK;
        if (!(eta < before)) break;   // it falls no more (or is not a number)
    }
    if (S == 1) return ORF_OK;
    ORF_TRY(factor(1));
    ORF_TRY(refuse_singular());
    ORF_TRY(rhs(mode));
    ORF_TRY(solve(f, x));
    return settle(mode, out);
}

// Factor the operator as nseg segments.
int orf_fdfd::factor(int nseg) {
    cudaStream_t st = ctx->stream;
    const FdfdDev P = dev();
    const size_t mm = (size_t)m * m;
    S = nseg;
    const int J = S - 1;
    // the segments' lines: equal shares of the lines that are not separators
    std::vector<FdSeg> hs(S);
    std::vector<int> sep(J);
    {
        int a = 0;
        for (int s = 0; s < S; ++s) {
            const int n = (int)((int64_t)(nb - J) * (s + 1) / S - (int64_t)(nb - J) * s / S);
            hs[s] = FdSeg{a, n, s > 0 && s == S - 1 ? -1 : 1, 0, nullptr};
            a += n;
            if (s < J) sep[s] = a++;
        }
    }
    ORF_CUDA(cudaMemsetAsync(fault, 0, sizeof(int), st));
    ORF_CUDA(cudaMemcpyAsync(segs, hs.data(), S * sizeof(FdSeg), cudaMemcpyHostToDevice, st));
    ORF_CUDA(launch_factor(P, C, segs, S, st, nullptr));
    Arena tmp;   // the separators' blocks and the corner blocks of the segments' inverses
    struct Release {
        Arena& a;
        cudaStream_t s;
        ~Release() {
            if (a.base) {
                cudaStreamSynchronize(s);
                a.release();
            }
        }
    } rel{tmp, st};
    if (J > 0) {
        ORF_CUDA(cudaMemcpyAsync(line, sep.data(), J * sizeof(int), cudaMemcpyHostToDevice, st));
        const int nin = std::max(0, S - 2);   // segments with two separators: 1 .. S-2
        double2 *Kd, *T, *L, *F;
        FdGemm* d_g;
        FdSepIn* d_sep;
        FdSeg* d_dense;
        int tmax = 0;
        for (int s = 1; s <= nin; ++s) tmax = std::max(tmax, hs[s].n);
        const int mid = J / 2;
        // ---- the batches of matrix products, in order: the corner blocks
        // (step t: L_t of every segment, F of step t - 1), then the separators'
        tmp.add(&Kd, J * mm);
        tmp.add(&T, J * mm);
        tmp.add(&L, (size_t)std::max(1, 3 * nin) * mm);
        tmp.add(&F, (size_t)std::max(1, nin) * mm);
        tmp.add(&d_g, (size_t)2 * nin * (tmax + 1) + 2 * J + 1);
        tmp.add(&d_sep, J);
        tmp.add(&d_dense, J);
        ORF_TRY(tmp.alloc());
        std::vector<FdGemm> g;
        std::vector<std::pair<int, int>> batch;   // [first, end) in g
        auto Lp = [&](int s, int t) -> double2* {   // L_t of segment s
            return t == 0 ? inv + (size_t)hs[s].a * mm : L + ((size_t)3 * (s - 1) + t % 3) * mm;
        };
        for (int t = 1; t <= tmax; ++t) {
            const int g0 = (int)g.size();
            for (int s = 1; s <= nin; ++s) {
                const int n = hs[s].n;
                const double2* e = eb + (size_t)(hs[s].a + t) * m;
                if (t < n) g.push_back(FdGemm{inv + (size_t)(hs[s].a + t) * mm, Lp(s, t - 1), nullptr, e, Lp(s, t), 0, 0, -1.0});
                if (t >= 2 && t - 1 < n) {
                    double2* Fs = F + (size_t)(s - 1) * mm;
                    g.push_back(FdGemm{Lp(s, t - 1), Lp(s, t - 2), t == 2 ? Lp(s, 0) : Fs, e - m, Fs, 1, 0, -1.0});
                }
            }
            batch.push_back({g0, (int)g.size()});
        }
        const size_t nspike = batch.size();
        // ---- elimination of the separators: the blocks of each step
        std::vector<FdSepIn> si(J);
        std::vector<FdSeg> dense;
        std::vector<int> dense_n;
        for (int q = 0; q < J; ++q) {
            // segment q before the separator (its last line eliminated last),
            // segment q + 1 after it (the last segment runs downwards)
            // (a segment has four lines at least: F of every one with two separators)
            const double2* first = q + 1 == S - 1 ? inv + (size_t)hs[S - 1].a * mm : F + (size_t)q * mm;
            si[q] = FdSepIn{sep[q], q > 0 ? 1 : 0, inv + (size_t)(sep[q] - 1) * mm, first,
                            q > 0 ? Lp(q, hs[q].n - 1) : nullptr};
        }
        for (int i = 0; i <= std::max(mid, J - 1 - mid); ++i) {
            const int lo = i, hi = J - 1 - i;
            const bool l = lo < mid, h = hi > mid;
            int n = 0;
            if (l) dense.push_back(FdSeg{sep[lo], 1, 1, 0, Kd + (size_t)lo * mm}), ++n;
            if (h) dense.push_back(FdSeg{sep[hi], 1, 1, 0, Kd + (size_t)hi * mm}), ++n;
            if (!l && !h) {
                dense.push_back(FdSeg{sep[mid], 1, 1, 0, Kd + (size_t)mid * mm});
                dense_n.push_back(1);
                break;
            }
            dense_n.push_back(n);
            const int g0 = (int)g.size();
            if (l) g.push_back(FdGemm{T + (size_t)(lo + 1) * mm, inv + (size_t)sep[lo] * mm, nullptr, nullptr, Y + (size_t)lo * mm, 0, 0, 1.0});
            if (h) g.push_back(FdGemm{T + (size_t)hi * mm, inv + (size_t)sep[hi] * mm, nullptr, nullptr, Y + (size_t)hi * mm, 1, 0, 1.0});
            batch.push_back({g0, (int)g.size()});
            // (the two updates may meet in the middle block: one launch each)
            if (l) {
                double2* K = Kd + (size_t)(lo + 1) * mm;
                g.push_back(FdGemm{Y + (size_t)lo * mm, T + (size_t)(lo + 1) * mm, K, nullptr, K, 0, 1, -1.0});
                batch.push_back({(int)g.size() - 1, (int)g.size()});
            }
            if (h) {
                double2* K = Kd + (size_t)(hi - 1) * mm;
                g.push_back(FdGemm{Y + (size_t)hi * mm, T + (size_t)hi * mm, K, nullptr, K, 0, 0, -1.0});
                batch.push_back({(int)g.size() - 1, (int)g.size()});
            }
        }
        ORF_CUDA(cudaMemcpyAsync(d_g, g.data(), g.size() * sizeof(FdGemm), cudaMemcpyHostToDevice, st));
        ORF_CUDA(cudaMemcpyAsync(d_sep, si.data(), J * sizeof(FdSepIn), cudaMemcpyHostToDevice, st));
        ORF_CUDA(cudaMemcpyAsync(d_dense, dense.data(), dense.size() * sizeof(FdSeg), cudaMemcpyHostToDevice, st));
        const unsigned nt = (unsigned)((m + kGT - 1) / kGT);
        size_t bq = 0;
        auto products = [&]() -> cudaError_t {
            const auto [a, b] = batch[bq++];
            if (b > a) k_fd_gemm<<<dim3(nt, nt, (unsigned)(b - a)), kGN, 0, st>>>(d_g + a, m);
            return cudaGetLastError();
        };
        while (bq < nspike) ORF_CUDA(products());
        k_fd_assemble<<<dim3((unsigned)m, (unsigned)J), 128, 0, st>>>(P, d_sep, Kd, T);
        ORF_CUDA(cudaGetLastError());
        int dq = 0;
        for (size_t i = 0; i < dense_n.size(); ++i) {
            ORF_CUDA(launch_factor(P, C, d_dense + dq, dense_n[i], st, nullptr));
            dq += dense_n[i];
            if (i + 1 < dense_n.size())
                for (int q = 0; q < 1 + dense_n[i]; ++q) ORF_CUDA(products());
        }
        const unsigned tt = (unsigned)((m + 15) / 16);
        k_fd_transpose<<<dim3(tt, tt, (unsigned)J), dim3(16, 16), 0, st>>>(Y, YT, m);
        ORF_CUDA(cudaGetLastError());
    }
    int flt = 0;
    ORF_CUDA(cudaMemcpyAsync(&flt, fault, sizeof(int), cudaMemcpyDeviceToHost, st));
    ORF_CUDA(cudaStreamSynchronize(st));
    singular = flt != 0;
    return ORF_OK;
}

extern "C" int32_t orf_fdfd2d_factor(orf_ctx* ctx, const orf_fdfd2d* pr, orf_fdfd** out) {
    if (!out) {
        set_error("out is null");
        return ORF_EINVAL;
    }
    *out = nullptr;
    if (!ctx || !pr || !pr->eps) {
        set_error("ctx, problem and eps are required");
        return ORF_EINVAL;
    }
    const int nx = pr->nx, nz = pr->nz;
    if (nx < 3 || nz < 3 || !(pr->dx > 0) || !(pr->lambda0 > 0)) {
        set_error("fdfd2D: needs at least 3 x 3 points, dx > 0 and lambda0 > 0");
        return ORF_EINVAL;
    }
    if (pr->npml_x < 0 || pr->npml_z < 0 || 2 * pr->npml_x >= nx || 2 * pr->npml_z >= nz) {
        set_error("fdfd2D: Npml must leave interior points on both axes");
        return ORF_EINVAL;
    }
    if (!(pr->pml_reflection > 0 && pr->pml_reflection < 1)) {
        set_error("fdfd2D: PmlReflection must lie in (0, 1)");
        return ORF_EINVAL;
    }
    ORF_ON_DEVICE(ctx->device);
    auto F = std::make_unique<orf_fdfd>();
    F->nx = nx;
    F->nz = nz;
    F->along_x = nz <= nx;
    F->m = F->along_x ? nz : nx;
    F->nb = F->along_x ? nx : nz;
    ORF_TRY(fd_shape(F->m, &F->C));
    const int m = F->m, nb = F->nb;
    const size_t N = F->N();

    // ---- M = diag(s_x s_z) A, symmetric
    const double d = pr->dx, k0 = 2.0 * kPi / pr->lambda0, R = pr->pml_reflection;
    const auto sxi = fd_stretch(nx, pr->npml_x, d, k0, R, false), sxh = fd_stretch(nx, pr->npml_x, d, k0, R, true);
    const auto szi = fd_stretch(nz, pr->npml_z, d, k0, R, false), szh = fd_stretch(nz, pr->npml_z, d, k0, R, true);
    std::vector<double2> hd(N), hw(N), he(N);
    const double h2 = 1.0 / (d * d);
    auto d2 = [](cplx v) { return make_double2(v.real(), v.imag()); };
    std::vector<cplx> rxh(nx + 1), rzh(nz + 1);
    for (int i = 0; i <= nx; ++i) rxh[i] = h2 / sxh[i];
    for (int k = 0; k <= nz; ++k) rzh[k] = h2 / szh[k];
    for (int k = 0; k < nz; ++k)
        for (int i = 0; i < nx; ++i) {
            const cplx cx = szi[k] * rxh[i], cz = sxi[i] * rzh[k];   // to (i-1, k), to (i, k-1)
            const size_t g = (size_t)i + (size_t)nx * k;
            const cplx eps(pr->eps[2 * g], pr->eps[2 * g + 1]);
            const cplx ax = szi[k] * (rxh[i] + rxh[i + 1]), az = sxi[i] * (rzh[k] + rzh[k + 1]);
            const cplx dg = -(ax + az) + k0 * k0 * eps * sxi[i] * szi[k];
            const size_t o = F->at(i, k);
            hd[o] = d2(dg);
            hw[o] = d2(F->along_x ? cz : cx);
            he[o] = d2(F->along_x ? cx : cz);
            F->mnorm = std::max(F->mnorm, std::abs(dg) + std::abs(ax) + std::abs(az));
        }

    F->ctx = ctx;
    ctx_retain(ctx);
    cudaStream_t st = ctx->stream;
    int most = 1;
    {
        FdfdDev P{};
        P.m = m;
        P.nb = nb;
        ORF_CUDA(launch_factor(P, F->C, nullptr, 1, st, &most));
    }
    int S = fd_segments(nb, most);
    F->planned = S;
    Arena& ar = F->ar;
    auto carve = [&]() {
        const int J = S - 1;
        ar = Arena{};
        ar.add(&F->diag, N);
        ar.add(&F->wc, N + 1);
        ar.add(&F->eb, N + m);   // (read one line past the last, unused)
        ar.add(&F->sx, nx);
        ar.add(&F->sz, nz);
        ar.add(&F->inv, (size_t)nb * m * m);
        ar.add(&F->vin, N);
        ar.add(&F->vout, N);
        ar.add(&F->f, N);
        ar.add(&F->x, N);
        ar.add(&F->r, N);
        ar.add(&F->dx, N);
        ar.add(&F->Y, (size_t)J * m * m);
        ar.add(&F->YT, (size_t)J * m * m);
        ar.add(&F->V, (size_t)J * m);
        ar.add(&F->Z, (size_t)2 * m);
        ar.add(&F->mx, 4);
        ar.add(&F->segs, S);
        ar.add(&F->line, J);
        ar.add(&F->fault, 1);
        ar.add(&F->xrow, (size_t)S * kPanel * m);
        return ar.alloc();
    };
    {
        void *h = nullptr, *d = nullptr;
        ORF_TRY(host_mapped_alloc(4 * sizeof(double), &h, &d));
        F->h_mx = static_cast<double*>(h);
        ORF_CUDA(cudaEventCreateWithFlags(&F->copied, cudaEventDisableTiming));
    }
    int rc = carve();
    if (rc == ORF_ENOMEM_DEVICE && S > 1) {   // one segment needs no memory for separators
        S = 1;
        rc = carve();
    }
    ORF_TRY(rc);
    ORF_CUDA(cudaMemcpyAsync(F->diag, hd.data(), N * sizeof(double2), cudaMemcpyHostToDevice, st));
    ORF_CUDA(cudaMemcpyAsync(F->wc, hw.data(), N * sizeof(double2), cudaMemcpyHostToDevice, st));
    ORF_CUDA(cudaMemcpyAsync(F->eb, he.data(), N * sizeof(double2), cudaMemcpyHostToDevice, st));
    std::vector<double2> hx(nx), hz(nz);
    for (int i = 0; i < nx; ++i) hx[i] = d2(sxi[i]);
    for (int k = 0; k < nz; ++k) hz[k] = d2(szi[k]);
    ORF_CUDA(cudaMemcpyAsync(F->sx, hx.data(), nx * sizeof(double2), cudaMemcpyHostToDevice, st));
    ORF_CUDA(cudaMemcpyAsync(F->sz, hz.data(), nz * sizeof(double2), cudaMemcpyHostToDevice, st));
    add_h2d(ctx, (int64_t)((3 * N + nx + nz) * sizeof(double2)));
    rc = F->factor(S);
    if (rc == ORF_ENOMEM_DEVICE && S > 1) {   // (the separators' blocks; every other error is the caller's to see)
        S = 1;
        rc = F->factor(S);
    }
    ORF_TRY(rc);
    if (S > 1) {
        // a segment that is nearly singular by itself shows in a trial solve
        double trial = 0.0;
        if (!F->singular) {
            k_fd_probe<<<296, 256, 0, st>>>(F->f, N, F->mx);
            ORF_CUDA(cudaGetLastError());
            ORF_TRY(F->solve(F->f, F->x));
            ORF_TRY(F->residual());
            ORF_CUDA(cudaStreamSynchronize(st));
            trial = F->eta_now();
        }
        if (F->singular || !(trial <= kEtaTrial)) ORF_TRY(F->factor(1));
    }
    ORF_TRY(F->refuse_singular());
    *out = F.release();
    return ORF_OK;
}

extern "C" int32_t orf_fdfd2d_solve(orf_fdfd* F, const double* rhs, double* x, int32_t transpose) {
    if (!F || !rhs || !x) {
        set_error("fdfd handle, rhs and x are required");
        return ORF_EINVAL;
    }
    ORF_TRY(F->refuse_singular());   // (found by an earlier solve)
    ORF_ON_DEVICE(F->ctx->device);
    const size_t bytes = F->N() * sizeof(double2);
    const int mode = transpose ? 1 : 0;
    cudaStream_t st = F->ctx->stream;
    void* stage = nullptr;
    ORF_TRY(pinned_stage_acquire(&stage));
    struct Release {
        void* s;
        cudaStream_t st;
        ~Release() {
            cudaStreamSynchronize(st);   // (after an error a copy may still be on its way)
            pinned_stage_release(s);
        }
    } rel{stage, st};
    ORF_TRY(copy_h2d_staged(F->vin, rhs, bytes, stage, st));
    add_h2d(F->ctx, (int64_t)bytes);
    F->scale = 0;
    ORF_TRY(F->rhs(mode));
    auto result = [&](auto&& beside) -> int {   // of the solve so far, into the caller's array
        k_fd_out<<<296, 256, 0, st>>>(F->map(), F->x, F->vout, mode, F->scale);
        ORF_CUDA(cudaGetLastError());
        const char* src = reinterpret_cast<const char*>(F->vout);
        for (size_t off = 0; off < bytes; off += kStageBytes) {
            const size_t n = std::min(kStageBytes, bytes - off);
            ORF_CUDA(cudaMemcpyAsync(stage, src + off, n, cudaMemcpyDeviceToHost, st));
            ORF_CUDA(cudaEventRecord(F->copied, st));
            if (off + n == bytes) ORF_TRY(beside());
            ORF_CUDA(cudaEventSynchronize(F->copied));
            std::memcpy(reinterpret_cast<char*>(x) + off, stage, n);
        }
        return ORF_OK;
    };
    ORF_TRY(F->solve(F->f, F->x));
    // (planned as one segment: no residual is taken)
    ORF_TRY(F->planned > 1 ? F->settle(mode, result) : result([]() -> int { return ORF_OK; }));
    add_d2h(F->ctx, (int64_t)bytes);
    return ORF_OK;
}

extern "C" void orf_fdfd2d_release(orf_fdfd* F) {
    if (!F) return;
    DeviceScope ds(F->ctx->device);
    delete F;
}

extern "C" int32_t orf_fdfd2d_info(const orf_fdfd* F, int32_t* block, int32_t* nblocks, int32_t* cluster) {
    if (!F) {
        set_error("fdfd handle is null");
        return ORF_EINVAL;
    }
    if (block) *block = F->m;
    if (nblocks) *nblocks = F->nb;
    if (cluster) *cluster = F->C;
    return ORF_OK;
}

extern "C" int32_t orf_fdfd2d_segments(const orf_fdfd* F, int32_t* planned, int32_t* segments) {
    if (!F) {
        set_error("fdfd handle is null");
        return ORF_EINVAL;
    }
    if (planned) *planned = F->planned;
    if (segments) *segments = F->S;
    return ORF_OK;
}

extern "C" int32_t orf_fdfd2d_residual(const orf_fdfd* F, double* residual) {
    if (!F || !residual) {
        set_error("fdfd handle and residual are required");
        return ORF_EINVAL;
    }
    *residual = F->eta;
    return ORF_OK;
}
