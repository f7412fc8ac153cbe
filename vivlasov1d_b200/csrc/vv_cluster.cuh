// The implicit time step (and the GMRES solve alone) of one instance by one
// thread-block cluster, in one launch.
//
// The multi-kernel step is bound by latency on small and medium grids: a
// GMRES iteration there is seven or eight dependent launches inside a
// conditional graph loop, 50-60 us whatever the grid's size, while the data
// of an iteration (the vector, its half spectrum, a few basis vectors) is a
// few hundred KB.  Here a cluster of C CTAs owns the instance for the whole
// step: CTA r keeps v rows [r rows, (r + 1) rows) of the vector in work in
// shared memory, in place through every stage (stencil output -> row FFTs ->
// v solves -> inverse row FFTs -> Gram-Schmidt), and the CTAs meet at
// hardware cluster barriers: two in a preconditioner application, one per
// reduction.  The basis stays in global memory (L2).  Every CTA runs the
// scalar work of GMRES and of the Picard loop (Givens rotations, convergence
// tests, the Poisson solve) redundantly from the same reduced values, so all
// decisions are uniform without a broadcast.
//
// The v solve of mode k.  The LU sweeps are linear recurrences
//   y_j = b_j - l_j y_{j-1},   x_j = d_j y_j - m_j x_{j+1},
// l_j = lambda alpha_j d_{j-1}, m_j = lambda gamma_j d_j, d the LU reciprocals.
// A thread owns a chunk of rows of a mode, sweeps it with a zero carry, and
// the chunks are joined through (a, b): out = b + a in, a = prod(-l).  The
// diagonal of A_k is four times its off-diagonals plus 1/ht, so |l| is at
// most about 2 - sqrt(3) and a decays below the rounding of the sum within
// a few tens of rows: a chunk takes its carry from the `klev` chunks before
// it (the host finds, from the actual multipliers, the number of rows
// over which every product falls below 1e-18, 1e-10 in FP32), read from the
// neighbouring CTAs' shared memory, instead of a scan over the whole line.
//
// Algorithm and arithmetic are those of the multi-kernel path (vv_bracket.cuh,
// vv_pcj.cuh, vv_vec.cuh): factored stencils, FP64 residual, moments, Poisson
// and reductions, the basis unnormalised with 1/||V_q|| applied where it is
// read; the sums run in another order.
#pragma once
#include <cooperative_groups.h>
#include "vv_bracket.cuh"
#include "vv_pc.cuh"
#include "vv_pcj.cuh"
#include "vv_vec.cuh"

namespace vv {

constexpr int CL_THREADS = 512;
constexpr int CL_WARPS = CL_THREADS / 32;
constexpr int CL_MAXC = 16;        // CTAs of a cluster
constexpr int CL_RESTART = 32;     // longest GMRES cycle (the back substitution runs on one warp)
constexpr int CL_CHUNK = 16;       // most rows of a tridiagonal chunk (a thread's registers)
constexpr int CL_NXMAX = 512;      // longest x row (the DFT's outputs per lane, the column strips)

enum ClMode { CL_STEP = 0, CL_GMRES = 1 };

// one instance (device-resident table)
struct ClInst {
    DevState* ds;
    int nx, nv, fam;               // fam: M = nx/2 for the FFT rows, 0 for the direct DFT
    int rows, nch, klev;           // v rows per CTA, row chunks per mode and CTA, carry levels
    int kv, dsm;                   // basis vectors kept in shared memory; 1: the LU reciprocals too
    size_t ncell;
    double ht_inv, fscale, hv;     // fscale: f1 (J1, J4) or f2 (J2)
    double cA1, cA2;               // scheme constants (Coef<SCHEME>)
    int scheme;
    const double *h0, *v;
    double* hxp;
    const void *tw;                // W^k = exp(-2 pi i k / nx), k < nx
    const void *dinv, *lam;        // slot-ordered LU reciprocals [nv][slots] and eigenvalues [slots]
    const void *alpha, *gamma;
    const double* green;           // circulant inverse of the Laplacian on mean-free profiles: phi = green * b
    PoissonParams po;
    double *f, *fh, *phi, *phih, *h1c, *h1h, *h2c, *h2h, *n, *u, *e, *a;
    double *Fh, *fl;
    void *V, *bT, *xT;
};

// rows of M complex numbers = P1 x P2, padded so that the column reads of
// both FFT passes fall on distinct banks: sample n at slot n + n / P2
template <int M> struct ClFft;
template <> struct ClFft<32> { static constexpr int P1 = 8, P2 = 4, RS = 44; };
template <> struct ClFft<64> { static constexpr int P1 = 8, P2 = 8, RS = 72; };
template <> struct ClFft<128> { static constexpr int P1 = 16, P2 = 8, RS = 152; };
template <> struct ClFft<256> { static constexpr int P1 = 16, P2 = 16, RS = 272; };

// mode of slot s: the FFT leaves Z_{k1 + P1 k2} at k1 (P2 + 1) + k2, slot
// s = k1 P2 + k2 (slot 0 holds the real pair X_0, X_M); DFT rows: s itself
template <int M> __host__ __device__ inline int cl_mode(int s) {
    if constexpr (M == 0) return s;
    else return s / ClFft<M>::P2 + ClFft<M>::P1 * (s % ClFft<M>::P2);
}
__host__ __device__ inline int cl_mode_of(int M, int s) {
    switch (M) {
        case 32: return cl_mode<32>(s);
        case 64: return cl_mode<64>(s);
        case 128: return cl_mode<128>(s);
        case 256: return cl_mode<256>(s);
        default: return s;
    }
}
__host__ __device__ inline int cl_row_slots(int fam, int nx) {
    switch (fam) {
        case 32: return ClFft<32>::RS;
        case 64: return ClFft<64>::RS;
        case 128: return ClFft<128>::RS;
        case 256: return ClFft<256>::RS;
        default: return (nx / 2 + 1) | 1;
    }
}
__host__ __device__ inline int cl_slots(int fam, int nx) { return fam ? fam : nx / 2 + 1; }

// scalar state of the solve, one copy per CTA
struct ClState {
    double rtol, atol, dtol, haptol, rnorm0, ttol, res;
    double snes_atol, pred, prev, scal[2], tt;
    int it, its, reason, active, restart, max_it, npad, breakdown;
    int pic_i, pic_stop, pic_revert, pic_rule, pic_max, ksp_failures, gmres_total, ncycles;
    double grs[CL_RESTART + 2], cc[CL_RESTART + 2], ss[CL_RESTART + 2], vsc[CL_RESTART + 2];
    double hcol[CL_RESTART + 2], cf[CL_RESTART + 2], nrs[CL_RESTART + 2];
    alignas(16) double dot[(CL_RESTART + 2) * CL_WARPS];   // this CTA's partial multi-dots (read by the cluster)
    double nrm[CL_WARPS];                      // ... partial norms
    double red[CL_WARPS];
    double hh[(CL_RESTART + 2) * (CL_RESTART + 1)];
    int gmres_its[MAX_PICARD_DEV], ksp_reason[MAX_PICARD_DEV];
    double residual[MAX_PICARD_DEV + 1];
};

// byte offsets of the dynamic shared memory (the same in every CTA): first the
// arrays whose sizes follow from nx alone
struct ClLay {
    int st, tw, lam, col, mp, h1, h1h, gr, row, lu, tri, W, U, d, v;
    int band;       // rows of FP64 the band buffer U holds (the residual's blocks)
    size_t bytes;
};
__host__ __device__ constexpr int cl_al(int b) { return (b + 15) & ~15; }
// kv, dsm: as in ClInst
__host__ __device__ inline ClLay cl_layout(int fam, int nx, int rows, int nch, int tsz, int kv, int dsm) {
    ClLay L;
    const int sl = cl_slots(fam, nx);
    L.st = 0;
    L.tw = cl_al((int)sizeof(ClState));
    L.lam = L.tw + cl_al((fam ? fam : nx) * 2 * tsz);
    L.col = L.lam + cl_al(sl * 2 * tsz);
    L.mp = L.col + cl_al(3 * nx * 8);
    L.h1 = L.mp + cl_al(3 * nx * 8);
    L.h1h = L.h1 + cl_al(nx * 8);
    L.gr = L.h1h + cl_al(nx * 8);
    L.row = L.gr + cl_al(2 * nx * 8);
    L.lu = L.row + cl_al(3 * rows * 8);
    L.tri = L.lu + cl_al(2 * rows * tsz);
    L.W = L.tri + 4 * nch * sl * 2 * tsz;
    int w = rows * cl_row_slots(fam, nx) * 2 * tsz;
    const int s1 = 5 * cl_al(nx * 8) + cl_al(CL_THREADS * 8);    // Poisson scratch
    const int s2 = CL_WARPS * 32 * 3 * 8;                         // moment partials
    if (w < s1) w = s1;
    if (w < s2) w = s2;
    L.U = L.W + cl_al(w);
    // the band of the stencils: rows + 4 of the GMRES precision, in FP64 at least
    // min(rows, 16) + 4
    const int fr = (rows < 16 ? rows : 16) + 4;
    int u = cl_al((rows + 4) * nx * tsz);
    if (u < fr * nx * 8) u = cl_al(fr * nx * 8);
    L.band = u / (nx * 8);
    L.d = L.U + u;
    L.v = L.d + (dsm ? cl_al((rows + 1) * sl * 2 * tsz) : 0);
    L.bytes = (size_t)L.v + (size_t)kv * cl_al(rows * nx * tsz);
    return L;
}

namespace cg = cooperative_groups;

// arrive (release) + wait (acquire) of the cluster's hardware barrier: the
// CTAs' shared and global writes before it are visible after it.  Not the
// .aligned form: the lanes of a warp may come from loops of different lengths.
VV_DEV void cl_sync() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;\n" ::: "memory");
}
// ... ordering the shared memory alone.  The full release waits until the
// warp's global stores are done (2400 cycles after a basis vector was stored,
// 500 without stores; this one 140-250): most barriers of an iteration pass
// only shared memory to the neighbours.
VV_DEV void cl_sync_shared() {
    __syncwarp();
    asm volatile(
        "fence.release.sync_restrict::shared::cta.cluster;\n\t"
        "barrier.cluster.arrive.relaxed;\n\t"
        "barrier.cluster.wait.acquire;\n\t"
        "fence.acquire.sync_restrict::shared::cluster.cluster;\n" ::: "memory");
}

extern __shared__ __align__(16) unsigned char cl_smem[];

template <typename T, int M> struct ClRun {
    using C = typename Cplx<T>::type;
    static constexpr int VN = M ? 16 / (int)sizeof(T) : 1;   // reals of a Gram-Schmidt item
    const ClInst& I;
    const int C_, rank, nv, r0, nr;
    int nxr;                       // nx where it is not 2 M
    int oRow, oLu, oTri, oW, oU, oD, oV, band;
    bool tri_ready;

    VV_DEV ClRun(const ClInst& inst, int csize, int crank)
        : I(inst), C_(csize), rank(crank), nv(inst.nv), r0(min(crank * inst.rows, inst.nv)),
          nr(max(0, min(inst.rows, inst.nv - crank * inst.rows))), nxr(inst.nx), tri_ready(false) {
        const ClLay L = cl_layout(M, NX(), I.rows, I.nch, (int)sizeof(T), I.kv, I.dsm);
        oRow = L.row; oLu = L.lu; oTri = L.tri; oW = L.W; oU = L.U; oD = L.d; oV = L.v;
        band = L.band;
    }
    // nx, modes per row and slots per row: constants of the FFT rows
    VV_DEV int NX() const {
        if constexpr (M != 0) return 2 * M;
        else return nxr;
    }
    VV_DEV int SL() const { return cl_slots(M, NX()); }
    VV_DEV int RS() const { return cl_row_slots(M, NX()); }
    // the arrays of the shared memory (shared-space addresses: 32-bit)
    template <typename P> VV_DEV static P* at(int o) { return reinterpret_cast<P*>(cl_smem + o); }
    VV_DEV static ClState* st() { return at<ClState>(0); }
    VV_DEV int oTw() const { return cl_al((int)sizeof(ClState)); }
    VV_DEV int oLam() const { return oTw() + cl_al((M ? M : NX()) * 2 * (int)sizeof(T)); }
    VV_DEV int oCol() const { return oLam() + cl_al(SL() * 2 * (int)sizeof(T)); }
    VV_DEV int oMp() const { return oCol() + cl_al(3 * NX() * 8); }
    VV_DEV int oH1() const { return oMp() + cl_al(3 * NX() * 8); }
    VV_DEV int oH1h() const { return oH1() + cl_al(NX() * 8); }
    VV_DEV int oGr() const { return oH1h() + cl_al(NX() * 8); }
    VV_DEV C* W() const { return at<C>(oW); }
    VV_DEV T* U() const { return at<T>(oU); }
    VV_DEV C* stw() const { return at<C>(oTw()); }
    VV_DEV C* lams() const { return at<C>(oLam()); }
    VV_DEV double* colc() const { return at<double>(oCol()); }   // stencil coefficients (FP64: the residual reads them too)
    VV_DEV double* rowc() const { return at<double>(oRow); }
    VV_DEV T* lurow() const { return at<T>(oLu); }               // alpha and gamma of the LU sweeps
    VV_DEV C* tri() const { return at<C>(oTri); }
    VV_DEV double* mp() const { return at<double>(oMp()); }
    VV_DEV double* h1s() const { return at<double>(oH1()); }
    VV_DEV double* h1hs() const { return at<double>(oH1h()); }
    VV_DEV double* gr() const { return at<double>(oGr()); }
    // LU reciprocals of this CTA's rows (shared memory or global); the row
    // before is readable if r0 > 0
    VV_DEV const C* dtab() const {
        return I.dsm ? at<const C>(oD) + SL() : reinterpret_cast<const C*>(I.dinv) + (ptrdiff_t)r0 * SL();
    }

    template <typename P> VV_DEV P* peer(P* p, int r) const {
        return cg::this_cluster().map_shared_rank(p, r);
    }
    VV_DEV int tid() const { return threadIdx.x; }
    VV_DEV int warp() const { return threadIdx.x >> 5; }
    VV_DEV int lane() const { return threadIdx.x & 31; }

    // address (in T) of real sample i of row r
    VV_DEV int wreal(int r, int i) const {
        if constexpr (M != 0) {
            const int n = i >> 1;
            return 2 * (r * RS() + n + n / ClFft<M>::P2) + (i & 1);
        } else {
            return 2 * r * RS() + i;
        }
    }

    // ---- set-up --------------------------------------------------------------
    VV_DEV void stage() {
        const int nx = NX(), sl = SL(), rows = I.rows;
        const C* tw = reinterpret_cast<const C*>(I.tw);
        for (int k = tid(); k < (M ? M : nx); k += CL_THREADS) stw()[k] = tw[k];
        for (int i = tid(); i < nx; i += CL_THREADS) gr()[i] = gr()[nx + i] = I.green[i];   // twice: no wrap in the convolution
        for (int k = tid(); k < sl; k += CL_THREADS) lams()[k] = reinterpret_cast<const C*>(I.lam)[k];
        if (I.dsm) {
            const C* src = reinterpret_cast<const C*>(I.dinv) + (ptrdiff_t)r0 * sl;
            C* dst = at<C>(oD) + sl;
            for (int k = tid() - (r0 > 0 ? sl : 0); k < nr * sl; k += CL_THREADS) dst[k] = src[k];
        }
        // row coefficients A1, alpha-, alpha+ of the stencil; alpha and gamma of the LU sweeps
        for (int r = tid(); r < nr; r += CL_THREADS) {
            const int j = r0 + r;
            double a[5];
#pragma unroll
            for (int d = 0; d < 5; ++d) {
                const int jj = j - 2 + d;
                a[d] = (jj >= 0 && jj < nv) ? I.h0[jj] : 0.0;
            }
            double am, aq;
            const double Dam = a[2] - a[1], Dap = a[3] - a[2], A1 = a[3] - a[1], Cm = a[2] - a[0], Cp = a[4] - a[2];
            if (I.scheme == 1) Coef<1>::row(Dam, Dap, A1, Cm, Cp, am, aq);
            else if (I.scheme == 2) Coef<2>::row(Dam, Dap, A1, Cm, Cp, am, aq);
            else Coef<4>::row(Dam, Dap, A1, Cm, Cp, am, aq);
            rowc()[r] = A1;
            rowc()[rows + r] = am;
            rowc()[2 * rows + r] = aq;
            lurow()[r] = reinterpret_cast<const T*>(I.alpha)[j];
            lurow()[rows + r] = reinterpret_cast<const T*>(I.gamma)[j];
        }
        if (tid() == 0) {
            const DevState* s = I.ds;
            ClState* S = st();
            S->its = 0;
            S->reason = R_ITERATING;
            S->rtol = s->rtol; S->atol = s->atol; S->dtol = s->dtol; S->haptol = s->haptol;
            S->restart = s->restart; S->max_it = s->max_it;
            S->snes_atol = s->snes_atol; S->pic_max = s->pic_max_iter;
            S->rnorm0 = 0.0; S->ttol = 0.0; S->res = 0.0;
            S->ncycles = 0; S->gmres_total = 0; S->ksp_failures = 0;
            S->pic_i = 0; S->pic_stop = 0; S->pic_revert = 0; S->pic_rule = 0;
        }
        __syncthreads();
    }

    VV_DEV int left(int i) const { return i == 0 ? NX() - 1 : i - 1; }
    VV_DEV int right(int i) const { return i + 1 == NX() ? 0 : i + 1; }
    // column coefficients B1, beta-, beta+ from the profile sb (nx doubles)
    VV_DEV void columns(const double* sb) {
        const int nx = NX();
        for (int i = tid(); i < nx; i += CL_THREADS) {
            const int m1 = left(i), p1 = right(i);
            const double b = sb[i], bl = sb[m1], br = sb[p1];
            const double Dbm = b - bl, Dbp = br - b, B1 = br - bl, Bm = b - sb[left(m1)], Bp = sb[right(p1)] - b;
            double bm, bq;
            if (I.scheme == 1) Coef<1>::col(Dbm, Dbp, B1, Bm, Bp, bm, bq);
            else if (I.scheme == 2) Coef<2>::col(Dbm, Dbp, B1, Bm, Bp, bm, bq);
            else Coef<4>::col(Dbm, Dbp, B1, Bm, Bp, bm, bq);
            colc()[i] = B1;
            colc()[nx + i] = bm;
            colc()[2 * nx + i] = bq;
        }
        __syncthreads();
    }

    // ---- stencil ---------------------------------------------------------------
    // W = hti d + tsc [x, h] on the local rows [rb, rb + n): x from a band in
    // shared memory (band row k holds local row rb + k - 2), a thread one column
    // down a run of rows through a register window (6 shared loads per output).
    // d: the time derivative's operand, x itself or (Pre) ctr(r, col) at local row r;
    // returns the thread's sum of squares then.
    template <typename R, bool Pre, typename Ctr>
    VV_DEV double stencil(const R* bnd, int rb, int n, R hti, R tsc, Ctr ctr) {
        const int nx = NX(), rows = I.rows;
        const int nxp = (nx + 31) & ~31, nseg = CL_THREADS / nxp;
        const int sg = tid() / nxp, c = tid() - sg * nxp;
        const int seg = (n + nseg - 1) / nseg;
        const R cA1 = R(I.cA1), cA2 = R(I.cA2);
        T* Wt = reinterpret_cast<T*>(W());
        double acc = 0.0;
        const int k0 = sg * seg, k1 = min(n, k0 + seg);
        if (sg < nseg && c < nx && k0 < k1) {
            const int m1 = left(c), m2 = left(m1), p1 = right(c), p2 = right(p1);
            const R B1 = R(colc()[c]), bm = R(colc()[nx + c]), bq = R(colc()[2 * nx + c]);
            const R* b = bnd + k0 * nx;
            R w0 = b[c], w1 = b[nx + c], w2 = b[2 * nx + c], w3 = b[3 * nx + c];
            R l0 = b[nx + m1], l1 = b[2 * nx + m1], q0 = b[nx + p1], q1 = b[2 * nx + p1];
            constexpr int PF = Pre ? 4 : 1;   // rows whose operand is loaded ahead (global memory)
            R d[PF];
#pragma unroll 1
            for (int kb = k0; kb < k1; kb += PF) {
                if constexpr (Pre) {
#pragma unroll
                    for (int u = 0; u < PF; ++u) d[u] = kb + u < k1 ? ctr(rb + kb + u, c) : R(0);
                }
#pragma unroll
                for (int u = 0; u < PF; ++u) {
                    if (kb + u >= k1) break;
                    const R w4 = b[4 * nx + c], l2 = b[3 * nx + m1], q2 = b[3 * nx + p1];
                    const int r = rb + kb + u, j = r0 + r;
                    const R xl = b[2 * nx + m2], xr = b[2 * nx + p2];
                    const R A1 = R(rowc()[r]), am = R(rowc()[rows + r]), ap = R(rowc()[2 * rows + r]);
                    R y = hti * (Pre ? d[u] : w2);
                    const R ax = cA1 * (q1 - l1) + cA2 * (xr - xl);
                    const R bx = cA1 * (w3 - w1) + cA2 * (w4 - w0);
                    R s = A1 * ax - B1 * bx;
                    s += am * (l0 - q0);
                    s += ap * (l2 - q2);
                    s += bm * (l0 - l2);
                    s += bq * (q0 - q2);
                    if (j >= 2 && j < nv - 2) y += tsc * s;
                    Wt[wreal(r, c)] = T(y);
                    if constexpr (Pre) acc += (double)y * (double)y;
                    w0 = w1; w1 = w2; w2 = w3; w3 = w4;
                    l0 = l1; l1 = l2; q0 = q1; q1 = q2;
                    b += nx;
                }
            }
        }
        __syncthreads();
        return acc;
    }
    // W = sc J x for the field x in U (its halo rows from the neighbours' U)
    VV_DEV void jvp(double sc) {
        const int nx = NX(), rows = I.rows;
        // a quarter of the threads a halo row
        const int h = tid() / (CL_THREADS / 4), r = h < 2 ? h - 2 : nr + h - 2, j = r0 + r;
        if (nr > 0 && j >= 0 && j < nv) {
            const int o = h < 2 ? (rows > 1 || h == 1 ? rank - 1 : rank - 2) : j / rows;
            const int own = h < 2 && rows == 1 ? 0 : j - o * rows;
            const T* src = peer(U(), o) + (own + 2) * nx;
            T* dst = U() + (r + 2) * nx;
            for (int i = tid() % (CL_THREADS / 4); i < nx; i += CL_THREADS / 4) dst[i] = src[i];
        }
        __syncthreads();
        stencil<T, false>(U(), 0, nr, T(I.ht_inv * sc), T(I.fscale * (0.5 * sc)), 0);
    }

    // ---- row transforms (in place) ------------------------------------------------
    // FFT rows: a warp transforms rw rows, 32 / P2 at most, fewer when that
    // spreads them over all warps.  Pass 1: lane = (row, m2), the P1-point DFTs and
    // twiddles; pass 2: lane = (row, k1), the P2-point DFTs and the real split, the
    // partner mode M - k = (P1 - k1) + P1 (P2 - 1 - k2) from lane P1 - k1.
    VV_DEV static C c_make2(T x, T y) { C r; r.x = x; r.y = y; return r; }
    VV_DEV static C shfl_c(C v, int src) {
        return c_make2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
    }
    VV_DEV int rows_per_warp() const {
        constexpr int P2 = M ? ClFft<M ? M : 32>::P2 : 1;
        return min(32 / P2, (nr + CL_WARPS - 1) / CL_WARPS);
    }
    VV_DEV void rfft() {
        if constexpr (M != 0) {
            constexpr int P1 = ClFft<M>::P1, P2 = ClFft<M>::P2, RS = ClFft<M>::RS;
            const int ln = lane(), rw = rows_per_warp();
#pragma unroll 1
            for (int g = warp() * rw; g < nr; g += CL_WARPS * rw) {
                const int ge = min(nr, g + rw);
                {
                    const int r = g + ln / P2, m2 = ln % P2;
                    C a[P1];
                    C* row = W() + r * RS + m2;
                    if (r < ge) {
#pragma unroll
                        for (int m1 = 0; m1 < P1; ++m1) a[m1] = row[m1 * (P2 + 1)];
                        reg_dft<P1, -1>(a);
                        row[0] = a[0];
#pragma unroll
                        for (int k1 = 1; k1 < P1; ++k1)
                            row[k1 * (P2 + 1)] = c_mul(a[k1], tw_half<M, -1>(stw(), m2 * k1));
                    }
                }
                __syncwarp();
                const int k1 = ln % P1, pl = (ln & ~(P1 - 1)) | ((P1 - k1) & (P1 - 1));
#pragma unroll 1
                for (int rr = g; rr < ge; rr += 32 / P1) {
                    const int r = rr + ln / P1;
                    const bool on = r < ge;
                    C* row = W() + r * RS + k1 * (P2 + 1);
                    C b[P2];
#pragma unroll
                    for (int m2 = 0; m2 < P2; ++m2) b[m2] = on ? row[m2] : c_make2(0, 0);
                    reg_dft<P2, -1>(b);
#pragma unroll
                    for (int k2 = 0; k2 < P2; ++k2) {
                        C z = shfl_c(b[P2 - 1 - k2], pl);
                        if (k1 == 0) z = b[(P2 - k2) % P2];
                        // X_k = E + w O of Z_k and Z_{M-k}; slot 0: X_0 and X_M
                        const C zk = b[k2], zc = c_conj(z);
                        const C E = c_scale(c_add(zk, zc), (T)0.5), D = c_sub(zk, zc);
                        C x = c_add(E, c_mul(stw()[k1 + P1 * k2], c_make2((T)0.5 * D.y, (T)-0.5 * D.x)));
                        if (k2 == 0 && k1 == 0) x = c_make2(zk.x + zk.y, zk.x - zk.y);
                        if (on) row[k2] = x;
                    }
                }
                __syncwarp();
            }
        } else {
            dft_rows();
        }
        __syncthreads();
    }
    VV_DEV void irfft() {
        if constexpr (M != 0) {
            constexpr int P1 = ClFft<M>::P1, P2 = ClFft<M>::P2, RS = ClFft<M>::RS;
            const int ln = lane(), rw = rows_per_warp();
            const T s = (T)(1.0 / (double)M);
#pragma unroll 1
            for (int g = warp() * rw; g < nr; g += CL_WARPS * rw) {
                const int ge = min(nr, g + rw);
                const int k1 = ln % P1, pl = (ln & ~(P1 - 1)) | ((P1 - k1) & (P1 - 1));
#pragma unroll 1
                for (int rr = g; rr < ge; rr += 32 / P1) {
                    const int r = rr + ln / P1;
                    const bool on = r < ge;
                    C* row = W() + r * RS + k1 * (P2 + 1);
                    C x[P2], b[P2];
#pragma unroll
                    for (int k2 = 0; k2 < P2; ++k2) x[k2] = on ? row[k2] : c_make2(0, 0);
#pragma unroll
                    for (int k2 = 0; k2 < P2; ++k2) {
                        C y = shfl_c(x[P2 - 1 - k2], pl);
                        if (k1 == 0) y = x[(P2 - k2) % P2];
                        // Z_k = E + i O of X_k and X_{M-k}
                        const C xk = x[k2], xc = c_conj(y);
                        const C E = c_scale(c_add(xk, xc), (T)0.5);
                        const C O = c_mul(c_conj(stw()[k1 + P1 * k2]), c_scale(c_sub(xk, xc), (T)0.5));
                        b[k2] = c_make2(E.x - O.y, E.y + O.x);
                        if (k2 == 0 && k1 == 0) b[0] = c_make2((T)0.5 * (xk.x + xk.y), (T)0.5 * (xk.x - xk.y));
                    }
                    reg_dft<P2, +1>(b);
                    if (on) {
                        row[0] = b[0];
#pragma unroll
                        for (int m2 = 1; m2 < P2; ++m2) row[m2] = c_mul(b[m2], tw_half<M, +1>(stw(), m2 * k1));
                    }
                }
                __syncwarp();
                {
                    const int r = g + ln / P2, m2 = ln % P2;
                    C a[P1];
                    C* row = W() + r * RS + m2;
                    if (r < ge) {
#pragma unroll
                        for (int q = 0; q < P1; ++q) a[q] = row[q * (P2 + 1)];
                        reg_dft<P1, +1>(a);
#pragma unroll
                        for (int m1 = 0; m1 < P1; ++m1) row[m1 * (P2 + 1)] = c_scale(a[m1], s);
                    }
                }
                __syncwarp();
            }
        } else {
            idft_rows();
        }
        __syncthreads();
    }
    // any nx: the direct DFT (x_n and x_{nx-n} share a twiddle).  A warp takes 32
    // modes of four rows, so that a gathered twiddle serves four products (the
    // gathers from shared memory bound it); the outputs stay in registers until
    // the block has read its rows.
    static constexpr int DR = 4;
    VV_DEV void dft_rows() {
        const int nx = NX(), rs = RS(), nm = SL(), nT = (nm + 31) >> 5, half = (nx - 1) >> 1;
        const int RB = DR * (CL_WARPS / nT);   // rows per round
        const int t = warp() % nT, k = lane() + 32 * t, kk = k < nm ? k : 0;
#pragma unroll 1
        for (int rb = 0; rb < nr; rb += RB) {
            const int r = rb + DR * (warp() / nT), re = min(nr, rb + RB);
            const bool on = warp() / nT < CL_WARPS / nT && r < re;
            T re_[DR], im[DR];
            if (on) {
                const T* row[DR];
#pragma unroll
                for (int d = 0; d < DR; ++d) {
                    row[d] = reinterpret_cast<const T*>(W() + min(r + d, re - 1) * rs);
                    const T xh = (nx & 1) ? T(0) : row[d][nx >> 1];
                    re_[d] = row[d][0] + ((kk & 1) ? -xh : xh);
                    im[d] = T(0);
                }
                int i = 0;
#pragma unroll 2
                for (int n = 1; n <= half; ++n) {
                    i += kk;
                    if (i >= nx) i -= nx;
                    const C w = stw()[i];
#pragma unroll
                    for (int d = 0; d < DR; ++d) {
                        const T a = row[d][n], b = row[d][nx - n];
                        re_[d] += (a + b) * w.x;
                        im[d] += (a - b) * w.y;
                    }
                }
            }
            __syncthreads();
            if (on && k < nm) {
#pragma unroll
                for (int d = 0; d < DR; ++d)
                    if (r + d < re) W()[(r + d) * rs + k] = c_make2(re_[d], im[d]);
            }
        }
    }
    // lane's samples n and nx - n
    VV_DEV void idft_rows() {
        const int nx = NX(), rs = RS(), nm = SL(), nT = (nm + 31) >> 5, K = (nx - 1) >> 1;
        const int RB = DR * (CL_WARPS / nT);
        const int t = warp() % nT, n = lane() + 32 * t, nn = n < nm ? n : 0;
        const T s = (T)(1.0 / (double)nx);
#pragma unroll 1
        for (int rb = 0; rb < nr; rb += RB) {
            const int r = rb + DR * (warp() / nT), re = min(nr, rb + RB);
            const bool on = warp() / nT < CL_WARPS / nT && r < re;
            T A[DR], B[DR], e[DR];
            if (on) {
                const C* X[DR];
#pragma unroll
                for (int d = 0; d < DR; ++d) {
                    X[d] = W() + min(r + d, re - 1) * rs;
                    const T XN = (nx & 1) ? T(0) : X[d][nx >> 1].x;
                    e[d] = X[d][0].x + ((nn & 1) ? -XN : XN);
                    A[d] = B[d] = T(0);
                }
                int i = 0;
#pragma unroll 2
                for (int k = 1; k <= K; ++k) {
                    i += nn;
                    if (i >= nx) i -= nx;
                    const C w = stw()[i];
#pragma unroll
                    for (int d = 0; d < DR; ++d) {
                        const C x = X[d][k];
                        A[d] += x.x * w.x;
                        B[d] += x.y * w.y;
                    }
                }
            }
            __syncthreads();
            if (on && n < nm) {
#pragma unroll
                for (int d = 0; d < DR; ++d)
                    if (r + d < re) {
                        T* row = reinterpret_cast<T*>(W() + (r + d) * rs);
                        row[n] = (e[d] + T(2) * (A[d] + B[d])) * s;
                        if (n > 0 && 2 * n != nx) row[nx - n] = (e[d] + T(2) * (A[d] - B[d])) * s;
                    }
            }
        }
    }

    // ---- v solves ------------------------------------------------------------------
    VV_DEV static C lmul(C lam, T al, C d) { return c_mul(c_rmul(lam, al), d); }
    // the carry into a chunk from `levels` chunks before it (fwd) or after it,
    // the farthest first: (rr, cc) its CTA and chunk
    VV_DEV C carry(const C* a, const C* b, int rr, int cc, int dir, int levels, int s) const {
        const int G = I.nch, sl = SL();
        C v = c_make2(0, 0);
        const C *pa = peer(a, rr), *pb = peer(b, rr);
#pragma unroll 2
        for (int t = 0; t < levels; ++t) {
            const int o = cc * sl + s;
            v = c_add(pb[o], c_mul(pa[o], v));
            cc += dir;
            if (cc == G || cc < 0) {
                cc = dir > 0 ? 0 : G - 1;
                rr += dir;
                if (t + 1 < levels) {
                    pa = peer(a, rr);
                    pb = peer(b, rr);
                }
            }
        }
        return v;
    }
    VV_DEV void solve_v() {
        const int G = I.nch, sl = SL(), rs = RS();
        const int c = tid() / sl, s = tid() - c * sl;
        const bool on = c < G;
        const int ra = on ? c * nr / G : 0, len = on ? (c + 1) * nr / G - ra : 0;
        const C* dv = dtab() + ra * sl + s;
        const T* al = lurow() + ra;
        const T* ga = al + I.rows;
        C* col = W() + ra * rs + s;
        if constexpr (M != 0) col += s / ClFft<M>::P2;
        C* const af = tri();
        C* const bf = af + G * sl;
        C* const ab = bf + G * sl;
        C* const bb = ab + G * sl;
        const int me = c * sl + s;
        const C lam = on ? lams()[s] : c_make2(0, 0);
        const C zero = c_make2(0, 0);
        const C dm = len > 0 && r0 + ra > 0 ? dv[-sl] : zero;   // the row before the chunk
        if (!tri_ready && on) {   // the carries' multipliers, the same at every application
            C a = c_make2(1, 0), e = a, d = dm;
#pragma unroll 1
            for (int u = 0; u < len; ++u) {
                a = c_sub(zero, c_mul(lmul(lam, al[u], d), a));
                d = dv[u * sl];
                e = c_sub(zero, c_mul(lmul(lam, ga[u], d), e));
            }
            af[me] = a;
            ab[me] = e;
        }
        tri_ready = true;
        {   // forward with a zero carry
            C y = zero, d = dm;
            C* w = col;
            const C* dp = dv;
#pragma unroll 2
            for (int u = 0; u < len; ++u, w += rs, dp += sl) {
                y = c_sub(*w, c_mul(lmul(lam, al[u], d), y));
                d = *dp;
                *w = y;
            }
            if (on) bf[me] = y;
        }
        cl_sync_shared();
        {   // the carry, then y and the backward sweep with a zero carry
            C p = zero, d = dm;
            if (len > 0) {
                const int g = rank * G + c, lv = min(I.klev, g), q = g - lv, rr = q / G;
                p = carry(af, bf, rr, q - rr * G, 1, lv, s);
            }
            C* w = col;
            const C* dp = dv;
#pragma unroll 2
            for (int u = 0; u < len; ++u, w += rs, dp += sl) {
                p = c_sub(zero, c_mul(lmul(lam, al[u], d), p));
                d = *dp;
                *w = c_add(*w, p);
            }
            C x = zero;
#pragma unroll 2
            for (int u = len - 1; u >= 0; --u) {
                w -= rs;
                dp -= sl;
                d = *dp;
                x = c_sub(c_mul(d, *w), c_mul(lmul(lam, ga[u], d), x));
                *w = x;
            }
            if (on) bb[me] = x;
        }
        cl_sync_shared();
        if (len > 0) {
            const int g = rank * G + c, lv = min(I.klev, C_ * G - 1 - g), q = g + lv, rr = q / G;
            C p = carry(ab, bb, rr, q - rr * G, -1, lv, s);
            C* w = col + len * rs;
            const C* dp = dv + len * sl;
#pragma unroll 2
            for (int u = len - 1; u >= 0; --u) {
                w -= rs;
                dp -= sl;
                p = c_sub(zero, c_mul(lmul(lam, ga[u], *dp), p));
                *w = c_add(*w, p);
            }
        }
        __syncthreads();
    }
    // W = P^-1 W
    VV_DEV void precondition() {
        rfft();
        solve_v();
        irfft();
    }

    // ---- reductions ----------------------------------------------------------------
    // sum over the cluster of every thread's v, in warp 0 (the same bits in
    // every CTA).  Shared memory written before the call is visible after it;
    // global memory too with `global` (its barrier waits for the stores)
    VV_DEV double cluster_sum(double v, bool global) {
        v = warp_sum(v);
        if (lane() == 0) st()->nrm[warp()] = v;
        if (global) cl_sync();
        else cl_sync_shared();
        double t = 0.0;
        if (warp() == 0) {
            for (int k = lane(); k < C_ * CL_WARPS; k += 32) t += peer(st()->nrm, k / CL_WARPS)[k % CL_WARPS];
            t = warp_sum(t);
        }
        return t;
    }

    // Gram-Schmidt items: VN consecutive reals of this CTA's rows
    VV_DEV int items() const { return nr * NX() / VN; }
    VV_DEV int waddr(int e) const {
        if constexpr (M != 0) {
            constexpr int GX = 2 * M / VN;
            return wreal(e / GX, (e % GX) * VN);
        } else {
            const int r = e / NX();
            return wreal(r, e - r * NX());
        }
    }
    struct Vec { T v[VN]; };
    VV_DEV Vec ldw(int e) const {
        Vec o;
        const T* p = reinterpret_cast<const T*>(W()) + waddr(e);
        if constexpr (M != 0) {
#pragma unroll
            for (int k = 0; k < VN / 2; ++k) {
                const C c = *reinterpret_cast<const C*>(p + 2 * k);
                o.v[2 * k] = c.x;
                o.v[2 * k + 1] = c.y;
            }
        } else {
            o.v[0] = *p;
        }
        return o;
    }
    VV_DEV static Vec ldg(const T* p) {
        Vec o;
        if constexpr (VN == 1) {
            o.v[0] = *p;
        } else if constexpr (VN == 2) {
            const double2 q = *reinterpret_cast<const double2*>(p);
            o.v[0] = q.x;
            o.v[1] = q.y;
        } else {
            const float4 q = *reinterpret_cast<const float4*>(p);
            o.v[0] = q.x;
            o.v[1] = q.y;
            o.v[2] = q.z;
            o.v[3] = q.w;
        }
        return o;
    }
    VV_DEV static void stg(T* p, const Vec& o) {
        if constexpr (VN == 1) *p = o.v[0];
        else if constexpr (VN == 2) *reinterpret_cast<double2*>(p) = make_double2(o.v[0], o.v[1]);
        else *reinterpret_cast<float4*>(p) = make_float4(o.v[0], o.v[1], o.v[2], o.v[3]);
    }

    // this CTA's rows of V_q: in shared memory for q < kv, else in global memory
    VV_DEV T* vec(int q) const {
        return q < I.kv ? at<T>(oV + q * cl_al(I.rows * NX() * (int)sizeof(T)))
                        : reinterpret_cast<T*>(I.V) + (size_t)q * I.ncell + (size_t)r0 * NX();
    }
    // partial dots <w, V_q>, q < m, of this CTA's items, per warp: a thread holds
    // its w (converted once: the FP32 basis is converted to FP64 for every
    // product, at 16 a cycle per SM the bound of this pass) and runs down the
    // basis, QU vectors' loads in flight
    template <int NI, int QU> VV_DEV void dots(int m) {
        ClState* S = st();
        const int E = items(), last = E - 1;
        if (E == 0) {   // a CTA past the last row: nothing of its W or V was ever written
            for (int q = lane(); q < m; q += 32) S->dot[q * CL_WARPS + warp()] = 0.0;
            return;
        }
#pragma unroll 1
        for (int b = 0; b < E; b += NI * CL_THREADS) {
            double w[NI][VN];
            int o[NI];
#pragma unroll
            for (int k = 0; k < NI; ++k) {
                const int e = b + tid() + k * CL_THREADS;
                o[k] = min(e, last) * VN;
                const Vec v = ldw(min(e, last));
#pragma unroll
                for (int i = 0; i < VN; ++i) w[k][i] = e < E ? (double)v.v[i] : 0.0;
            }
#pragma unroll 1
            for (int q0 = 0; q0 < m; q0 += QU) {
                Vec x[QU][NI];
#pragma unroll
                for (int u = 0; u < QU; ++u) {
                    const T* v = vec(min(q0 + u, m - 1));
#pragma unroll
                    for (int k = 0; k < NI; ++k) x[u][k] = ldg(v + o[k]);
                }
                double t[QU];
#pragma unroll
                for (int u = 0; u < QU; ++u) {
                    t[u] = 0.0;
                    if (q0 + u < m) {
#pragma unroll
                        for (int k = 0; k < NI; ++k)
#pragma unroll
                            for (int i = 0; i < VN; ++i) t[u] += w[k][i] * (double)x[u][k].v[i];
                    }
                }
#pragma unroll
                for (int s = 16; s > 0; s >>= 1)
#pragma unroll
                    for (int u = 0; u < QU; ++u) t[u] += __shfl_xor_sync(0xffffffffu, t[u], s);
                if (lane() == 0) {
#pragma unroll
                    for (int u = 0; u < QU; ++u)
                        if (q0 + u < m) {
                            double* d = S->dot + (q0 + u) * CL_WARPS + warp();
                            *d = b ? *d + t[u] : t[u];
                        }
                }
            }
        }
    }
    // hcol_q = vsc_q <w, V_q>, q < m, w in W, in every CTA
    VV_DEV void multidot(int m) {
        ClState* S = st();
        if (I.rows * NX() <= CL_THREADS * VN) dots<1, 4>(m);
        else dots<4, 2>(m);
        cl_sync_shared();
        // 16 threads per dot, one per CTA
        const int q = tid() / CL_MAXC, r = tid() % CL_MAXC;
        double t = 0.0;
        if (q < m && r < C_) {
            const double2* d = reinterpret_cast<const double2*>(peer(S->dot, r) + q * CL_WARPS);
            double2 v[CL_WARPS / 2];
#pragma unroll
            for (int p = 0; p < CL_WARPS / 2; ++p) v[p] = d[p];
#pragma unroll
            for (int p = 0; p < CL_WARPS / 2; ++p) t += v[p].x + v[p].y;
        }
#pragma unroll
        for (int o = CL_MAXC / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (q < m && r == 0) {
            const double h = t * S->vsc[q];
            S->hcol[q] = h;
            S->cf[q] = -h * S->vsc[q];
        }
        __syncthreads();
    }

    // Gram-Schmidt update and solution update (one body, its instructions are
    // fetched by both): two items of a thread at a time, four vectors' loads in
    // flight.
    //   ORTH   V_m = w + sum_q cf_q V_q, w in W; kept in U too (the next
    //          operand); returns the sum of its squares
    //   SOLN   x (+)= sum_q nrs_q V_q at the end of a cycle that goes on, kept
    //          in U too (the restart's operand)
    //   INTOF  ... of the step's last cycle: fl <- f, f -= x unless the solve failed
    enum { ORTH, SOLN, INTOF };
    VV_DEV double combine(int mode, int m, bool first) {
        ClState* S = st();
        const int E = items();
        const double* cf = mode == ORTH ? S->cf : S->nrs;
        T* out = mode == ORTH ? vec(m) : reinterpret_cast<T*>(I.xT) + (size_t)r0 * NX();
        T* u = U() + 2 * NX();
        double* f = I.f + (size_t)r0 * NX();
        double* fl = I.fl + (size_t)r0 * NX();
        const bool ok = S->reason >= 0;
        double acc = 0.0;
#pragma unroll 1
        for (int e0 = tid(); e0 < E; e0 += 2 * CL_THREADS) {
            const int e1 = e0 + CL_THREADS < E ? e0 + CL_THREADS : e0;
            double w[2][VN];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                Vec v;
#pragma unroll
                for (int i = 0; i < VN; ++i) v.v[i] = T(0);
                if (mode == ORTH) v = ldw(k ? e1 : e0);
                else if (!first) v = ldg(out + (k ? e1 : e0) * VN);
#pragma unroll
                for (int i = 0; i < VN; ++i) w[k][i] = (double)v.v[i];
            }
#pragma unroll 1
            for (int q0 = 0; q0 < m; q0 += 4) {
                Vec v[4][2];
                double cq[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int q = min(q0 + c, m - 1);
                    const T* p = vec(q);
                    cq[c] = q0 + c < m ? cf[q] : 0.0;
                    v[c][0] = ldg(p + e0 * VN);
                    v[c][1] = ldg(p + e1 * VN);
                }
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (q0 + c < m) {
#pragma unroll
                        for (int k = 0; k < 2; ++k)
#pragma unroll
                            for (int i = 0; i < VN; ++i) w[k][i] += cq[c] * (double)v[c][k].v[i];
                    }
            }
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                if (k && e1 == e0) break;
                const int e = k ? e1 : e0;
                Vec o;
#pragma unroll
                for (int i = 0; i < VN; ++i) {
                    o.v[i] = (T)w[k][i];
                    acc += w[k][i] * w[k][i];
                }
                if (mode == INTOF) {
#pragma unroll
                    for (int i = 0; i < VN; ++i) {
                        const double fv = f[e * VN + i];
                        fl[e * VN + i] = fv;
                        if (ok) f[e * VN + i] = fv - (double)o.v[i];
                    }
                } else {
                    stg(out + e * VN, o);
                    stg(u + e * VN, o);
                }
            }
        }
        return acc;
    }

    // ---- GMRES (KSPGMRES's control flow) -------------------------------------------
    VV_DEV static int converged(int n, double rnorm) {
        ClState* S = st();
        if (n == 0) {
            S->rnorm0 = rnorm;
            S->ttol = fmax(S->rtol * rnorm, S->atol);
        }
        if (isnan(rnorm) || isinf(rnorm)) return R_NANORINF;
        if (rnorm <= S->ttol) return rnorm < S->atol ? R_ATOL : R_RTOL;
        if (rnorm >= S->dtol * S->rnorm0) return R_DTOL;
        return R_ITERATING;
    }
    // the previous rotations applied to the new column (one thread)
    VV_DEV void rotate() {
        ClState* S = st();
        const int it = S->it;
        double* hc = S->hh + it * (CL_RESTART + 2);
        double hj = S->hcol[0];
#pragma unroll 1
        for (int j = 1; j <= it; ++j) {
            const double hn = S->hcol[j], c = S->cc[j - 1], sn = S->ss[j - 1];
            hc[j - 1] = c * hj + sn * hn;
            hj = c * hn - sn * hj;
        }
        hc[it] = hj;
    }
    // the step's rotation and the convergence test from ||w||^2 (one thread)
    VV_DEV void arnoldi(double s2) {
        ClState* S = st();
        const int it = S->it;
        double* hc = S->hh + it * (CL_RESTART + 2);
        const double tt = sqrt(s2), hj = hc[it], g = S->grs[it], t2 = hj * hj + s2;
        const double ri = rsqrt(t2), c = hj * ri, sn = tt * ri;
        S->vsc[it + 1] = (tt != 0.0) ? rsqrt(s2) : 1.0;
        hc[it + 1] = tt;
        // KSPGMRES's happy breakdown: tt < min(haptol, |tt / grs|)
        const bool hapend = tt < S->haptol && tt < fabs(tt / g);
        bool null = false;
        double res = 0.0;
        if (!hapend) {
            if (t2 == 0.0) {
                S->reason = R_NULL;
                null = true;
                res = S->res;
            } else {
                S->cc[it] = c;
                S->ss[it] = sn;
                S->grs[it + 1] = -(sn * g);
                S->grs[it] = c * g;
                hc[it] = c * hj + sn * tt;
                res = fabs(sn * g);
            }
        }
        S->res = res;
        S->it = it + 1;
        const int its = S->its + 1;
        S->its = its;
        int reason = R_NULL;
        if (!null) {
            reason = converged(its, res);
            if (hapend && reason == R_ITERATING) reason = R_BREAKDOWN;
            S->reason = reason;
        }
        S->active = (reason == R_ITERATING && it + 1 < S->restart && its < S->max_it) ? 1 : 0;
    }
    // KSPGMRESBuildSoln's triangular solve, by columns on one warp (the
    // diagonal's reciprocals by one division across the lanes)
    VV_DEV void backsolve() {
        if (warp() != 0) return;
        ClState* S = st();
        const int last = S->it - 1, ld = CL_RESTART + 2, l = lane();
        int npad = 0, breakdown = 0;
        if (last >= 0) {
            const double dg = l <= last ? S->hh[l * ld + l] : 1.0;
            breakdown = __any_sync(0xffffffffu, dg == 0.0) ? 1 : 0;
            if (!breakdown) {
                const double inv = 1.0 / dg;
                double t = l <= last ? S->grs[l] : 0.0;
#pragma unroll 1
                for (int k = last; k >= 0; --k) {
                    const double h = l < k ? S->hh[k * ld + l] : 0.0;
                    t -= h * __shfl_sync(0xffffffffu, t * inv, k);
                }
                npad = last + 1;
                if (l <= last) S->nrs[l] = t * inv * S->vsc[l];
            }
        }
        if (l == 0) {
            S->npad = npad;
            if (breakdown) S->reason = R_BREAKDOWN;
            if (S->its >= S->max_it && S->reason == R_ITERATING) S->reason = R_ITS;
        }
    }
    // start of a cycle from the residual in W (keep_b: the right-hand side,
    // kept in bT for the restarts of a step's solve): V_0, its norm
    VV_DEV void cycle_head(bool keep_b) {
        ClState* S = st();
        T* V0 = vec(0);
        T* bT = reinterpret_cast<T*>(I.bT) + (size_t)r0 * NX();
        T* u = U() + 2 * NX();
        const int E = items();
        double acc = 0.0;
#pragma unroll 1
        for (int e = tid(); e < E; e += CL_THREADS) {
            const Vec w = ldw(e);
            stg(V0 + e * VN, w);
            stg(u + e * VN, w);
            if (keep_b) stg(bT + e * VN, w);
#pragma unroll
            for (int k = 0; k < VN; ++k) acc += (double)w.v[k] * (double)w.v[k];
        }
        const double ss2 = cluster_sum(acc, false);
        if (tid() == 0) {
            const double res = sqrt(ss2);
            S->ncycles += 1;
            S->it = 0;
            S->grs[0] = res;
            S->res = res;
            S->vsc[0] = (res != 0.0) ? 1.0 / res : 1.0;
            if (res == 0.0) {
                S->reason = R_ATOL;
                S->active = 0;
            } else {
                S->reason = converged(S->its, res);
                S->active = (S->reason == R_ITERATING && S->its < S->max_it) ? 1 : 0;
            }
        }
        __syncthreads();
    }

    // ---- the rest of a Picard pass ------------------------------------------------
    // scratch of the x profiles (in W, free between the solves)
    VV_DEV double* scr(int k) const { return at<double>(oW + k * cl_al(NX() * 8)); }

    // (A phi)_i of the Laplacian, phi in scr(0)
    VV_DEV double laplace(const double* sp, int i) const {
        const int m1 = left(i), p1 = right(i);
        return (I.po.la2 * (sp[left(m1)] + sp[right(p1)]) + I.po.la1 * (sp[m1] + sp[p1]) + I.po.la0 * sp[i]) *
               (I.po.hx2_inv / I.po.lden);
    }
    // scr(2) = the right-hand side b = -(n~ - mean n) charge of the density in scr(1)
    VV_DEV void poisson_rhs() {
        const int nx = NX();
        const double* sn = scr(1);
        double t = 0.0;
        for (int i = lane(); i < nx; i += 32) t += sn[i];
        const double nmean = warp_sum(t) * I.po.inv_nx;   // the same in every warp
        for (int i = tid(); i < nx; i += CL_THREADS) {
            double d = sn[i];
            if (I.po.ravg) {
                const int m1 = left(i), p1 = right(i);
                d = ((((I.po.ra2 * sn[left(m1)] + I.po.ra1 * sn[m1]) + I.po.ra0 * d) + I.po.ra1 * sn[p1]) +
                     I.po.ra2 * sn[right(p1)]) / I.po.rden;
            }
            scr(2)[i] = -(d - nmean) * I.po.charge;
        }
        __syncthreads();
    }
    // from phi in scr(0) and b in scr(2): the norm of the Poisson residual
    // (scal[0]); phi - mean phi in scr(3)
    VV_DEV void poisson_tail() {
        const int nx = NX();
        const double* sp = scr(0);
        double a = 0.0;
        for (int i = lane(); i < nx; i += 32) a += sp[i];
        const double pmean = warp_sum(a) * I.po.inv_nx;
        double r2 = 0.0;
        for (int i = tid(); i < nx; i += CL_THREADS) {
            const double r = laplace(sp, i) - scr(2)[i];
            r2 += r * r;
            scr(3)[i] = sp[i] - pmean;
        }
        r2 = block_sum(r2, st()->red);
        if (tid() == 0) st()->scal[0] = sqrt(r2);
        __syncthreads();
    }
    // scr(0) (+)= green * src, CL_THREADS / nx threads per point
    VV_DEV void convolve(const double* src, bool add) {
        const int nx = NX(), P = CL_THREADS / nx, part = tid() / nx, i = tid() - part * nx;
        double* sc = scr(5);
        if (part < P) {
            const int ma = part * nx / P, mb = (part + 1) * nx / P;
            const double* g = gr() + nx + i;   // green at i - m
            double a0 = 0.0, a1 = 0.0;
            int m = ma;
#pragma unroll 2
            for (; m + 1 < mb; m += 2) {
                a0 += g[-m] * src[m];
                a1 += g[-m - 1] * src[m + 1];
            }
            if (m < mb) a0 += g[-m] * src[m];
            sc[tid()] = a0 + a1;
        }
        __syncthreads();
        if (tid() < nx) {
            double p = add ? scr(0)[tid()] : 0.0;
            for (int k = 0; k < P; ++k) p += sc[k * nx + tid()];
            scr(0)[tid()] = p;
        }
        __syncthreads();
    }

    // moments of f, Poisson, h1 (h1s) and the Poisson residual's norm (scal[0])
    // in every CTA; rank 0 writes the state's profiles
    VV_DEV void moments() {
        const int nx = NX();
        double* tmp = at<double>(oW);   // [seg][3][nx]
        const int ns = (nx + 31) >> 5, nseg = max(1, CL_WARPS / ns);
        {
            const int sg = warp() / ns, c = (warp() - sg * ns) * 32 + lane();
            if (sg < nseg && c < nx) {
                double a0 = 0.0, a1 = 0.0, a2 = 0.0;
                const double* f = I.f + (size_t)r0 * nx + c;
#pragma unroll 4
                for (int r = sg; r < nr; r += nseg) {
                    const double fv = f[r * nx], vj = I.v[r0 + r];
                    a0 += fv;
                    a1 += vj * fv;
                    a2 += (vj * vj) * fv;
                }
                tmp[sg * 3 * nx + c] = a0;
                tmp[(sg * 3 + 1) * nx + c] = a1;
                tmp[(sg * 3 + 2) * nx + c] = a2;
            }
        }
        __syncthreads();
        for (int i = tid(); i < 3 * nx; i += CL_THREADS) {
            double t = 0.0;
            for (int s = 0; s < nseg; ++s) t += tmp[s * 3 * nx + i];
            mp()[i] = t;
        }
        cl_sync();   // f of the neighbours' rows too (the residual's halo)
        // the sums over the CTAs (velocity and energy density: rank 0 only), then
        // the Poisson equation in every CTA: phi = green * b by direct convolution
        // (nx^2 products over the block: fewer cycles than the FFT pair's chain of
        // stages), refined once: the convolution's rounding is white in x and the
        // Laplacian of it, without the second pass, is the floor of the residual
        double *sp = scr(0), *sn = scr(1);
        for (int i = tid(); i < (rank == 0 ? 3 * nx : nx); i += CL_THREADS) {
            double t = 0.0;
#pragma unroll 4
            for (int r = 0; r < C_; ++r) t += peer(mp(), r)[i];
            (i < nx ? sn : i < 2 * nx ? scr(3) - nx : scr(4) - 2 * nx)[i] = t * I.hv;
        }
        __syncthreads();
        if (rank == 0)
            for (int i = tid(); i < nx; i += CL_THREADS) {
                const double s0 = sn[i], s1 = scr(3)[i], s2 = scr(4)[i];
                if (I.n) I.n[i] = s0;
                if (I.u) I.u[i] = s1;
                if (I.e) I.e[i] = s2;
                if (I.a) I.a[i] = s0 * s0 / (s0 * s2 - s1 * s1);   // Toolbox.pyx:164-165
            }
        poisson_rhs();
#pragma unroll 1
        for (int k = 0; k < 2; ++k) {
            convolve(k ? scr(3) : scr(2), k != 0);
            if (k) break;
            for (int i = tid(); i < nx; i += CL_THREADS) scr(3)[i] = scr(2)[i] - laplace(sp, i);
            __syncthreads();
        }
        poisson_tail();
        for (int i = tid(); i < nx; i += CL_THREADS) {
            const double h = scr(3)[i];
            h1s()[i] = h;
            if (rank == 0) {
                I.phi[i] = sp[i];
                I.h1c[i] = h;
            }
        }
        __syncthreads();
    }
    // h's x profile from h1s and the history profiles, its column coefficients
    VV_DEV void profile() {
        double* sb = scr(0);
        for (int i = tid(); i < NX(); i += CL_THREADS) {
            double b = 0.5 * h1s()[i] + 0.5 * h1hs()[i];
            b += 0.5 * (I.h2c ? I.h2c[i] : 0.0);
            b += 0.5 * (I.h2h ? (I.h2c ? I.h2c[i] : I.h2h[i]) : 0.0);   // make_history: h2h <- h2c
            sb[i] = b;
        }
        __syncthreads();
        columns(sb);
    }
    // W = R(f) (rounded to T); ||R||^2 in warp 0.  Fave = (Fh + F)/2 staged in
    // FP64 by blocks of the rows the band buffer holds
    VV_DEV double residual() {
        const int nx = NX();
        const double* F = I.f;
        const double* Fh = I.Fh;
        double* bnd = at<double>(oU);
        const int RB = band - 4;
        double acc = 0.0;
#pragma unroll 1
        for (int rb = 0; rb < nr; rb += RB) {
            const int n = min(RB, nr - rb), cnt = (n + 4) * nx;
            // rows rb - 2 .. rb + n + 1 of the grid are consecutive in memory
            const ptrdiff_t o0 = (ptrdiff_t)(r0 + rb - 2) * nx, total = (ptrdiff_t)I.ncell;
#pragma unroll 4
            for (int e = tid(); e < cnt; e += CL_THREADS) {
                const ptrdiff_t o = o0 + e;
                const bool in = o >= 0 && o < total;
                const double a = in ? Fh[o] : 0.0, b = in ? F[o] : 0.0;
                bnd[e] = 0.5 * a + 0.5 * b;
            }
            __syncthreads();
            const double *Fb = F + (size_t)r0 * nx, *Hb = Fh + (size_t)r0 * nx;
            acc += stencil<double, true>(bnd, rb, n, I.ht_inv, I.fscale,
                                         [&](int r, int c) { return Fb[r * nx + c] - Hb[r * nx + c]; });
        }
        return cluster_sum(acc, false);
    }

    // make_history and update_previous (run_base.py:749-763); the Poisson
    // residual of the state's phi and n (scal[0])
    VV_DEV void prologue() {
        const int nx = NX();
        const size_t base = (size_t)r0 * nx;
        const int cnt = nr * nx;
#pragma unroll 4
        for (int i = tid(); i < cnt; i += CL_THREADS) {
            const double fv = I.f[base + i];
            I.fh[base + i] = fv;
            I.Fh[base + i] = fv;
        }
        for (int i = tid(); i < nx; i += CL_THREADS) {
            const double h1 = I.h1c[i], phi = I.phi[i];
            h1s()[i] = h1;
            h1hs()[i] = h1;
            scr(0)[i] = phi;
            scr(1)[i] = I.n[i];
            if (rank == 0) {
                I.h1h[i] = h1;
                const double h2 = I.h2c ? I.h2c[i] : 0.0;
                if (I.h2c && I.h2h) I.h2h[i] = h2;
                if (I.phih) I.phih[i] = phi;
                I.hxp[nx + i] = h1;
                I.hxp[2 * nx + i] = h2;
                I.hxp[3 * nx + i] = I.h2h ? (I.h2c ? h2 : I.h2h[i]) : 0.0;
            }
        }
        __syncthreads();
        poisson_rhs();
        poisson_tail();
        cl_sync();   // Fh of the neighbours' rows
    }
    // the operator's h and the right-hand side of a solve alone
    VV_DEV void load_rhs() {
        const int nx = NX();
        for (int i = tid(); i < nx; i += CL_THREADS) {
            double b = 0.5 * I.hxp[i] + 0.5 * I.hxp[nx + i];
            b += 0.5 * I.hxp[2 * nx + i];
            b += 0.5 * I.hxp[3 * nx + i];
            mp()[i] = b;
        }
        __syncthreads();
        columns(mp());
        load_b(false);
    }
    // W = b, or b - W
    VV_DEV void load_b(bool minus) {
        const T* bT = reinterpret_cast<const T*>(I.bT) + (size_t)r0 * NX();
        const int E = items();
#pragma unroll 1
        for (int e = tid(); e < E; e += CL_THREADS) {
            const Vec b = ldg(bT + e * VN);
            T* p = reinterpret_cast<T*>(W()) + waddr(e);
#pragma unroll
            for (int k = 0; k < VN; ++k) p[k] = minus ? (T)((double)b.v[k] - (double)p[k]) : b.v[k];
        }
        __syncthreads();
    }

    // The step (or the solve) as one loop around the preconditioner, so that
    // every stage is compiled once (the instructions of an iteration have to
    // stay in the instruction cache):
    //   PASS     end of a Picard pass (or its start, the prologue): moments,
    //            profile, residual, the stop rules -> right-hand side
    //   RHS      W = P^-1 R -> first cycle
    //   ARNOLDI  W = P^-1 J v_it -> Gram-Schmidt
    //   RESTART  W = P^-1 J x -> b - W -> next cycle
    VV_DEV void run(int mode) {
        enum { PASS, RHS, ARNOLDI, RESTART, HEAD };
        ClState* S = st();
        const bool step = mode == CL_STEP;
        int phase = step ? PASS : HEAD;
        bool first_pass = true, reverting = false, first_cycle = true;
        if (step) prologue();
        else load_rhs();
#pragma unroll 1
        for (;;) {
            if (phase == PASS) {
                if (!first_pass) {
                    moments();
                    if (reverting) break;
                }
                if (rank == 0)
                    for (int i = tid(); i < NX(); i += CL_THREADS) I.hxp[i] = h1s()[i];
                profile();
                // the cluster barrier of moments() (or the prologue) ordered the neighbours' f before this
                const double f2 = residual();
                if (tid() == 0) {
                    const double pred = sqrt(f2) + S->scal[0];
                    if (first_pass) S->residual[0] = S->pred = pred;
                    else picard(pred);
                    if (!S->pic_stop) {
                        S->its = 0;
                        S->reason = R_ITERATING;
                    }
                }
                __syncthreads();
                if (S->pic_stop) {
                    if (!S->pic_revert) break;
                    const size_t base = (size_t)r0 * NX();
                    for (int i = tid(); i < nr * NX(); i += CL_THREADS) I.f[base + i] = I.fl[base + i];
                    __syncthreads();
                    reverting = true;
                    continue;
                }
                first_pass = false;
                first_cycle = true;
                phase = RHS;
            }
            if (phase == ARNOLDI || phase == RESTART) jvp(phase == ARNOLDI ? S->vsc[S->it] : 1.0);
            if (phase != HEAD) precondition();
            int comb = ORTH, m = 0;
            if (phase == ARNOLDI) {
                m = S->it + 1;
                multidot(m);
                // one warp's first lane runs the rotations while the others start the update
                if (tid() == CL_THREADS - 32) rotate();
            } else {
                if (phase == RESTART) load_b(true);
                cycle_head(phase == RHS);
                comb = SOLN;
            }
            bool done = false;
#pragma unroll 1
            for (;;) {
                if (comb != ORTH) {   // no further iteration in this cycle
                    if (S->active) break;
                    backsolve();
                    __syncthreads();
                    m = S->npad;
                    done = S->reason != R_ITERATING;
                    if (done && step) comb = INTOF;
                }
                const double acc = combine(comb, m, first_cycle);
                if (comb != ORTH) break;
                const double s2 = cluster_sum(acc, false);
                if (tid() == 0) arnoldi(s2);
                __syncthreads();
                comb = SOLN;
            }
            if (S->active) {
                phase = ARNOLDI;
                continue;
            }
            first_cycle = false;
            if (done) {
                if (!step) break;
                __syncthreads();
                phase = PASS;
            } else {
                cl_sync_shared();   // x of the neighbours' rows (U)
                phase = RESTART;
            }
        }
    }
    // the stop rules of run_nonlinear_matrixfree_split_mp.py:158-163 (thread 0)
    VV_DEV static void picard(double pred) {
        ClState* S = st();
        const int k = S->pic_i;
        if (k < MAX_PICARD_DEV) {
            S->gmres_its[k] = S->its;
            S->ksp_reason[k] = S->reason;
        }
        S->gmres_total += S->its;
        if (S->reason < 0) S->ksp_failures += 1;
        const int i = k + 1;
        S->pic_i = i;
        S->prev = S->pred;
        S->pred = pred;
        if (i <= MAX_PICARD_DEV) S->residual[i] = pred;
        const bool rose = pred > S->prev && i > 1;
        const bool small = pred < S->snes_atol;
        const bool maxed = i >= S->pic_max || i >= MAX_PICARD_DEV;
        if (rose || small || maxed) {
            S->pic_rule = rose ? 1 : (small ? 2 : 3);
            S->pic_revert = pred > S->prev ? 1 : 0;
            S->pic_stop = 1;
        }
    }

    VV_DEV void report(int mode) {
        if (rank != 0) return;
        __syncthreads();
        DevState* s = I.ds;
        const ClState* S = st();
        if (mode == CL_STEP) {
            const int np = min(S->pic_i, MAX_PICARD_DEV);
            for (int k = tid(); k <= np; k += CL_THREADS) {
                s->residual[k] = S->residual[k];
                if (k < np) {
                    s->gmres_its[k] = S->gmres_its[k];
                    s->ksp_reason[k] = S->ksp_reason[k];
                }
            }
        }
        if (tid() != 0) return;
        s->it = S->it;
        s->its = S->its;
        s->reason = S->reason;
        s->active = 0;
        s->res = S->res;
        s->ncycles = S->ncycles;
        if (mode == CL_STEP) {
            s->pic_i = S->pic_i;
            s->pic_stop = S->pic_stop;
            s->pic_revert = S->pic_revert;
            s->pic_stop_rule = S->pic_rule;
            s->ksp_failures = S->ksp_failures;
            s->gmres_total = S->gmres_total;
            s->pic_active = 0;
            s->pred = S->pred;
            s->prev = S->prev;
            s->have_set = 1;
        }
    }
};

// one cluster per instance of rows of kind M; order: the instances in the
// order in which the clusters are placed (the longest first)
template <typename T, int M>
__global__ void __launch_bounds__(CL_THREADS, 1) k_cl_run(const ClInst* __restrict__ tab, const int* __restrict__ order,
                                                          int mode) {
    const int csize = (int)cg::this_cluster().num_blocks(), crank = (int)cg::this_cluster().block_rank();
    const int cid = blockIdx.x / csize;
    // the description in shared memory: its fields are read again after every barrier
    __shared__ ClInst I;
    static_assert(sizeof(ClInst) % 4 == 0, "copied by words");
    const unsigned* src = reinterpret_cast<const unsigned*>(tab + (order ? order[cid] : cid));
    for (int k = threadIdx.x; k < (int)(sizeof(ClInst) / 4); k += CL_THREADS)
        reinterpret_cast<unsigned*>(&I)[k] = src[k];
    __syncthreads();
    ClRun<T, M> r(I, csize, crank);
    r.stage();
    r.run(mode);
    r.report(mode);
    cl_sync();   // no CTA leaves while a neighbour may read its shared memory
}

}  // namespace vv
