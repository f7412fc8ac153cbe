// Tensor-product kinetic preconditioner of one grid in the v-major layout,
// spec[j * (M + 1) + k] (row j, mode k = 0..M, M = nx/2 a power of two): rows are
// read and written whole by every stage, no transposes.
//
//   x transforms  rows of M = P1 P2 P3 complex samples in place in shared memory:
//                 three passes of register DFTs (two up to M = 256, vv_pcj.cuh)
//                 and the real split.
//   v solves      a block takes 32 modes x TL_WARPS chunks of 8 or 16 rows; a thread
//                 sweeps one chunk of one mode with its rows in registers, and a
//                 chunk takes its carry from the `lev` chunks before it, as in
//                 vv_cluster.cuh: |l| <= 2 - sqrt(3) but for the 1/ht term, so the
//                 products of the LU multipliers over lev chunks are below 1e-18
//                 (1e-9 in FP32; the host finds lev from the multipliers).  The
//                 block's first and last lev chunks only provide carries and are
//                 recomputed by the neighbours: nothing waits on another block,
//                 at 1 + 2 lev / (TL_WARPS - 2 lev) times the reads.
//
// Bytes: 48 B/cell in FP64 over the three stages (the solves read their overlap
// and the LU reciprocals on top: 1.33 x 32 + 16 B per complex unknown).  No stage
// is at HBM yet: by these bytes 87, 136 and 94 us at 2048 x 8192 are 47, 55 and
// 44% of the measured 6.54 TB/s.  Few warps are in flight (23-33% of the SM's:
// shared memory and registers) and they wait for loads (long scoreboard), in the
// solves because a block loads everything, then sweeps, then stores.
#pragma once
#include "vv_common.cuh"
#include "vv_pc.cuh"
#include "vv_pcj.cuh"

namespace vv {

// ---- rows of 512..2048 complex samples ---------------------------------------------
template <int M> struct FftL;
template <> struct FftL<512> { static constexpr int P1 = 8, P2 = 8, P3 = 8; };
template <> struct FftL<1024> { static constexpr int P1 = 16, P2 = 8, P3 = 8; };
template <> struct FftL<2048> { static constexpr int P1 = 16, P2 = 16, P3 = 8; };
constexpr int FL_THREADS = 128;

// Z_{k1 + P1 k2 + P1 P2 k3} (and sample (m1 P2 + m2) P3 + m3) at
// k1 S1 + k2 (P3 + 1) + k3, S1 = P2 (P3 + 1) + 1: every pass and the split read
// distinct banks
template <int M> struct RowL {
    static constexpr int P1 = FftL<M>::P1, P2 = FftL<M>::P2, P3 = FftL<M>::P3;
    static constexpr int S2 = P3 + 1, S1 = P2 * S2 + 1, RS = P1 * S1;
    // rows per block: about the number that gives every thread one P1-point DFT
    static constexpr int RB = (FL_THREADS * P1 / M) > 0 ? FL_THREADS * P1 / M : 1;
    VV_DEV static int slot(int k) { return (k % P1) * S1 + (k / P1 % P2) * S2 + k / (P1 * P2); }
};
inline size_t fl_smem(int M, size_t csz) {
    switch (M) {
        case 512: return (size_t)RowL<512>::RB * RowL<512>::RS * csz;
        case 1024: return (size_t)RowL<1024>::RB * RowL<1024>::RS * csz;
        case 2048: return (size_t)RowL<2048>::RB * RowL<2048>::RS * csz;
        default: return 0;
    }
}
inline int fl_rows(int M) {
    switch (M) {
        case 512: return RowL<512>::RB;
        case 1024: return RowL<1024>::RB;
        case 2048: return RowL<2048>::RB;
        default: return 0;
    }
}

// W_M^(q) from the table tw[k] = exp(-2 pi i k / nx), nx = 2 M
template <int SIGN, typename C> VV_DEV C tw_row(const C* __restrict__ tw, int q) {
    C w = __ldg(tw + 2 * q);
    if (SIGN > 0) w.y = -w.y;
    return w;
}

template <typename TI, typename R, int M>
__global__ void __launch_bounds__(FL_THREADS) k_rfftl(const TI* __restrict__ X, typename Cplx<R>::type* __restrict__ spec,
                                                      PcParams p) {
    using C = typename Cplx<R>::type;
    using L = RowL<M>;
    constexpr int P1 = L::P1, P2 = L::P2, P3 = L::P3, RB = L::RB;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* buf = reinterpret_cast<C*>(smem_raw);
    const C* tw = reinterpret_cast<const C*>(p.tw);
    const int j0 = blockIdx.x * RB, nr = min(RB, p.nv - j0);
    for (int u = threadIdx.x; u < nr * (P2 * P3); u += FL_THREADS) {
        const int r = u / (P2 * P3), m = u % (P2 * P3);   // m = P3 m2 + m3
        const auto* row = reinterpret_cast<const typename Pair<TI>::type*>(X + (size_t)(j0 + r) * p.nx) + m;
        C a[P1];
#pragma unroll
        for (int m1 = 0; m1 < P1; ++m1) {
            const auto v = row[m1 * (P2 * P3)];
            a[m1] = c_make<C>((double)v.x, (double)v.y);
        }
        reg_dft<P1, -1>(a);
        C* b = buf + r * L::RS + (m / P3) * L::S2 + m % P3;
        b[0] = a[0];
#pragma unroll
        for (int k1 = 1; k1 < P1; ++k1) b[k1 * L::S1] = c_mul(a[k1], tw_row<-1>(tw, m * k1));
    }
    __syncthreads();
    for (int u = threadIdx.x; u < nr * (P1 * P3); u += FL_THREADS) {
        const int r = u / (P1 * P3), k1 = u / P3 % P1, m3 = u % P3;
        C* b = buf + r * L::RS + k1 * L::S1 + m3;
        C a[P2];
#pragma unroll
        for (int m2 = 0; m2 < P2; ++m2) a[m2] = b[m2 * L::S2];
        reg_dft<P2, -1>(a);
        b[0] = a[0];
#pragma unroll
        for (int k2 = 1; k2 < P2; ++k2) b[k2 * L::S2] = c_mul(a[k2], tw_row<-1>(tw, P1 * m3 * k2));
    }
    __syncthreads();
    for (int u = threadIdx.x; u < nr * (P1 * P2); u += FL_THREADS) {
        const int r = u / (P1 * P2), k1 = u / P2 % P1, k2 = u % P2;
        C* b = buf + r * L::RS + k1 * L::S1 + k2 * L::S2;
        C a[P3];
#pragma unroll
        for (int m3 = 0; m3 < P3; ++m3) a[m3] = b[m3];
        reg_dft<P3, -1>(a);
#pragma unroll
        for (int k3 = 0; k3 < P3; ++k3) b[k3] = a[k3];
    }
    __syncthreads();
    for (int u = threadIdx.x; u < nr * (M / 2 + 1); u += FL_THREADS) {
        const int r = u / (M / 2 + 1), k = u % (M / 2 + 1), kc = M - k;
        const C* b = buf + r * L::RS;
        const C zk = b[L::slot(k)], zc = b[L::slot(k == 0 ? 0 : kc)];
        C* out = spec + (size_t)(j0 + r) * (M + 1);
        auto split = [&](C a, C c, C w) {
            const C cc = c_conj(c);
            const C E = c_scale(c_add(a, cc), (R)0.5), D = c_sub(a, cc);
            C t;
            t.x = (R)0.5 * D.y;
            t.y = (R)-0.5 * D.x;
            return c_add(E, c_mul(w, t));
        };
        out[k] = split(zk, zc, __ldg(tw + k));
        if (kc != k) out[kc] = split(zc, zk, k == 0 ? c_make<C>(-1.0, 0.0) : __ldg(tw + kc));
    }
}

// normalised inverse (the imaginary parts of X_0 and X_M are ignored)
template <typename R, typename TO, int M>
__global__ void __launch_bounds__(FL_THREADS) k_irfftl(const typename Cplx<R>::type* __restrict__ spec, TO* __restrict__ Y,
                                                       PcParams p) {
    using C = typename Cplx<R>::type;
    using L = RowL<M>;
    constexpr int P1 = L::P1, P2 = L::P2, P3 = L::P3, RB = L::RB;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* buf = reinterpret_cast<C*>(smem_raw);
    const C* tw = reinterpret_cast<const C*>(p.tw);
    const int j0 = blockIdx.x * RB, nr = min(RB, p.nv - j0);
    if (p.yidx) Y += (size_t)(*p.yidx + p.yoff) * p.ystride;
    for (int u = threadIdx.x; u < nr * (M / 2 + 1); u += FL_THREADS) {
        const int r = u / (M / 2 + 1), k = u % (M / 2 + 1), kc = M - k;
        const C* in = spec + (size_t)(j0 + r) * (M + 1);
        C xk = in[k], xc = in[kc];
        if (k == 0) {
            xk.y = 0;
            xc.y = 0;
        }
        C* b = buf + r * L::RS;
        auto unsplit = [&](C a, C c, C w) {
            const C cc = c_conj(c);
            const C E = c_scale(c_add(a, cc), (R)0.5);
            const C O = c_mul(c_conj(w), c_scale(c_sub(a, cc), (R)0.5));
            C z;
            z.x = E.x - O.y;
            z.y = E.y + O.x;
            return z;
        };
        b[L::slot(k)] = unsplit(xk, xc, __ldg(tw + k));
        if (k != 0 && kc != k) b[L::slot(kc)] = unsplit(xc, xk, __ldg(tw + kc));
    }
    __syncthreads();
    for (int u = threadIdx.x; u < nr * (P1 * P2); u += FL_THREADS) {
        const int r = u / (P1 * P2), k1 = u / P2 % P1, k2 = u % P2;
        C* b = buf + r * L::RS + k1 * L::S1 + k2 * L::S2;
        C a[P3];
#pragma unroll
        for (int k3 = 0; k3 < P3; ++k3) a[k3] = b[k3];
        reg_dft<P3, +1>(a);
        b[0] = a[0];
#pragma unroll
        for (int m3 = 1; m3 < P3; ++m3) b[m3] = c_mul(a[m3], tw_row<+1>(tw, P1 * m3 * k2));
    }
    __syncthreads();
    for (int u = threadIdx.x; u < nr * (P1 * P3); u += FL_THREADS) {
        const int r = u / (P1 * P3), k1 = u / P3 % P1, m3 = u % P3;
        C* b = buf + r * L::RS + k1 * L::S1 + m3;
        C a[P2];
#pragma unroll
        for (int k2 = 0; k2 < P2; ++k2) a[k2] = b[k2 * L::S2];
        reg_dft<P2, +1>(a);
#pragma unroll
        for (int m2 = 0; m2 < P2; ++m2) b[m2 * L::S2] = c_mul(a[m2], tw_row<+1>(tw, (P3 * m2 + m3) * k1));
    }
    __syncthreads();
    const R s = (R)(1.0 / (double)M);
    for (int u = threadIdx.x; u < nr * (P2 * P3); u += FL_THREADS) {
        const int r = u / (P2 * P3), m = u % (P2 * P3);
        const C* b = buf + r * L::RS + (m / P3) * L::S2 + m % P3;
        C a[P1];
#pragma unroll
        for (int k1 = 0; k1 < P1; ++k1) a[k1] = b[k1 * L::S1];
        reg_dft<P1, +1>(a);
        auto* row = reinterpret_cast<typename Pair<TO>::type*>(Y + (size_t)(j0 + r) * p.nx) + m;
#pragma unroll
        for (int m1 = 0; m1 < P1; ++m1) {
            typename Pair<TO>::type o;
            o.x = (TO)(a[m1].x * s);
            o.y = (TO)(a[m1].y * s);
            row[m1 * (P2 * P3)] = o;
        }
    }
}

// rows of 32..256 complex samples: the batch's row transforms, one item per block
template <typename TI, typename R, int M>
__global__ void __launch_bounds__(FJ_THREADS) k_rfftj1(const TI* __restrict__ X, typename Cplx<R>::type* __restrict__ spec,
                                                       PcParams p) {
    rfftj_block<TI, R, M>(X, spec, p, blockIdx.x);
}
template <typename R, typename TO, int M>
__global__ void __launch_bounds__(FJ_THREADS) k_irfftj1(const typename Cplx<R>::type* __restrict__ spec,
                                                        TO* __restrict__ Y, PcParams p) {
    if (p.yidx) Y += (size_t)(*p.yidx + p.yoff) * p.ystride;
    irfftj_block<R, TO, M>(spec, Y, p, blockIdx.x);
}

// ---- v solves ------------------------------------------------------------------------
constexpr int TL_WARPS = 16;
template <typename R> constexpr size_t tl_smem(int ch) { return (size_t)TL_WARPS * ch * 32 * 2 * sizeof(R); }

// x = A_k^-1 b (ADJ: A_k^-H b) for 32 modes and a run of rows, out of place.
//   A:   y_j = b_j - l_j y_{j-1}, l_j = lambda alpha_j d_{j-1};  x_j = d_j y_j - m_j x_{j+1}, m_j = lambda gamma_j d_j
//   A^H: w_j = conj(d_j) (b_j - conj(lambda gamma_{j-1}) w_{j-1});  z_j = w_j - conj(l_{j+1}) z_{j+1}
// lev: chunks a carry reaches over; dinv v-major, staged by cp.async (the four
// sweeps read it again).  Rows outside the line are zero, and so are the
// multipliers across its ends.
template <typename R, bool ADJ, int TL_CH>
__global__ void __launch_bounds__(32 * TL_WARPS, sizeof(R) == 4 || TL_CH == 8 ? 2 : 1)
k_tridiagl(const typename Cplx<R>::type* __restrict__ in, typename Cplx<R>::type* __restrict__ out,
           const typename Cplx<R>::type* __restrict__ dinvJ, TriParams p, int lev) {
    using C = typename Cplx<R>::type;
    __shared__ C sa[TL_WARPS][32], sb[TL_WARPS][32];
    __shared__ R sal[TL_WARPS * TL_CH + 1], sga[TL_WARPS * TL_CH + 1];   // alpha, gamma of the block's rows (from one before)
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* sd = reinterpret_cast<C*>(smem_raw);
    const int lane = threadIdx.x & 31, c = threadIdx.x >> 5;
    const int nm = p.nmodes, nv = p.nv, k = blockIdx.x * 32 + lane, kk = min(k, nm - 1);
    const int useful = TL_WARPS - 2 * lev;                       // chunks this block stores
    const int jb = ((int)blockIdx.y * useful - lev) * TL_CH;     // the block's first row (may lie outside the line)
    const int q0 = c * TL_CH, j0 = jb + q0;                      // this chunk's, in the block and in the line
    const C lam = reinterpret_cast<const C*>(p.lambda)[kk];
    const C zero = c_make<C>(0.0, 0.0);
    C y[TL_CH];
#pragma unroll
    for (int u = 0; u < TL_CH; ++u) {
        const int j = j0 + u;
        const bool on = j >= 0 && j < nv;
        const size_t o = (size_t)(on ? j : 0) * nm + kk;
        if (on) cp_async_elem(&sd[(q0 + u) * 32 + lane], &dinvJ[o]);
        else sd[(q0 + u) * 32 + lane] = zero;
        y[u] = on ? in[o] : zero;
    }
    cp_async_commit();
    for (int t = threadIdx.x; t <= TL_WARPS * TL_CH; t += 32 * TL_WARPS) {
        const int j = jb - 1 + t;
        // alpha_j couples rows j-1, j; gamma_j rows j, j+1: zero across the ends
        sal[t] = j >= 1 && j < nv ? reinterpret_cast<const R*>(p.alpha)[j] : R(0);
        sga[t] = j >= 0 && j + 1 < nv ? reinterpret_cast<const R*>(p.gamma)[j] : R(0);
    }
    cp_async_wait0();
    __syncthreads();
    auto d = [&](int u) -> C { return sd[(q0 + u) * 32 + lane]; };   // u = -1: the chunk before (none before the block's first)
    auto fwd = [&](int u) -> C {   // multiplier of y_{j-1}
        if (!ADJ) return q0 + u > 0 ? c_mul(c_rmul(lam, sal[q0 + u + 1]), d(u - 1)) : zero;
        return c_mul(c_conj(d(u)), c_conj(c_rmul(lam, sga[q0 + u])));
    };
    auto bwd = [&](int u) -> C {   // multiplier of x_{j+1}
        if (!ADJ) return c_mul(c_rmul(lam, sga[q0 + u + 1]), d(u));
        return q0 + u + 2 <= TL_WARPS * TL_CH ? c_conj(c_mul(c_rmul(lam, sal[q0 + u + 2]), d(u))) : zero;
    };
    C a = c_make<C>(1.0, 0.0), t = zero;
#pragma unroll
    for (int u = 0; u < TL_CH; ++u) {
        const C l = fwd(u);
        const C b = ADJ ? c_mul(c_conj(d(u)), y[u]) : y[u];
        t = c_sub(b, c_mul(l, t));
        y[u] = t;
        a = c_sub(zero, c_mul(l, a));
    }
    sa[c][lane] = a;
    sb[c][lane] = t;
    __syncthreads();
    C v = zero;
    for (int q = max(0, c - lev); q < c; ++q) v = c_add(sb[q][lane], c_mul(sa[q][lane], v));
    __syncthreads();
    // the carry, then the backward sweep from the chunk's end
#pragma unroll
    for (int u = 0; u < TL_CH; ++u) {
        v = c_sub(zero, c_mul(fwd(u), v));
        y[u] = c_add(y[u], v);
    }
    a = c_make<C>(1.0, 0.0);
    t = zero;
#pragma unroll
    for (int u = TL_CH - 1; u >= 0; --u) {
        const C m = bwd(u);
        const C b = ADJ ? y[u] : c_mul(d(u), y[u]);
        t = c_sub(b, c_mul(m, t));
        y[u] = t;
        a = c_sub(zero, c_mul(m, a));
    }
    sa[c][lane] = a;
    sb[c][lane] = t;
    __syncthreads();
    if (c < lev || c >= lev + useful || k >= nm) return;
    v = zero;
    for (int q = min(TL_WARPS - 1, c + lev); q > c; --q) v = c_add(sb[q][lane], c_mul(sa[q][lane], v));
#pragma unroll
    for (int u = TL_CH - 1; u >= 0; --u) {
        const int j = j0 + u;
        v = c_sub(zero, c_mul(bwd(u), v));
        if (j >= 0 && j < nv) out[(size_t)j * nm + k] = c_add(y[u], v);
    }
}

}  // namespace vv
