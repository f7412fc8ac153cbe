// Tensor-product potential preconditioner (`tensor_potential`):
// TensorProductPotential.pyx:157-183 (the FFT - solve - iFFT sequence),
// TensorProductPotentialFast.pyx:43-266 (FFT along v, banded matrices from
// phi, zgbtrf/zgbtrs with KL = KU = 1), eigenvalues TensorProduct.pyx:109-116
// for n = nv.
//
//   P^-1 X = irFFT_v [ A_k^-1 (rFFT_v X)_k ],  k = 0..nv/2,
//
// A_k (nx x nx, tridiagonal, no periodic corner entries):
//   A[i][i-1] = lambda_k (phi_i - phi_{i-1}) a,
//   A[i][i]   = lambda_k 2 (phi_{i+1} - phi_{i-1}) a + 1/ht,
//   A[i][i+1] = lambda_k (phi_{i+1} - phi_i) a,     a = hx^-1 hv^-1 / 24,
// with periodic differences of phi, built from the phi of make_history.
//
// The v transforms run as the x-row kernels on the transposed field (rows of
// length nv); A_k is solved by Gaussian elimination with partial pivoting
// (the pivot rule of LAPACK's band LU: swap when |sub|_1 > |diag|_1), one
// thread per mode; the factors are made once per phi.
#pragma once
#include "vv_common.cuh"

namespace vv {

// dst[c*rows + r] = src[r*cols + c] (rows x cols -> cols x rows), 32 x 32
// tiles through shared memory, block (32, 8); dst may be a GMRES basis base
// pointer: dst += (*yidx + yoff) * ystride
template <typename TI, typename TO>
__global__ void k_transpose(const TI* __restrict__ src, TO* __restrict__ dst, int rows, int cols,
                            const int* __restrict__ yidx, int yoff, size_t ystride) {
    __shared__ TO t[32][33];
    if (yidx) dst += (size_t)(*yidx + yoff) * ystride;
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {
        const int r = r0 + k, c = c0 + threadIdx.x;
        if (r < rows && c < cols) t[k][threadIdx.x] = (TO)src[(size_t)r * cols + c];
    }
    __syncthreads();
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {
        const int c = c0 + k, r = r0 + threadIdx.x;
        if (c < cols && r < rows) dst[(size_t)c * rows + r] = t[threadIdx.x][k];
    }
}

struct PotParams {
    int nx, nmv;           // x points, v modes (nv/2 + 1)
    double arak, ht_inv;   // hx^-1 hv^-1 / 24, 1/ht
    const double* phi;     // nx: the potential of make_history
    const double2* lam;    // nmv: shifted eigenvalues for n = nv
};

template <typename C>
VV_DEV double c_abs1(C a) { return fabs((double)a.x) + fabs((double)a.y); }
template <typename C>
VV_DEV C c_div(C a, C b) {
    using R = decltype(a.x);
    const R den = b.x * b.x + b.y * b.y;
    C r;
    r.x = (a.x * b.x + a.y * b.y) / den;
    r.y = (a.y * b.x - a.x * b.y) / den;
    return r;
}

// Factors of every mode's A_k, kept until phi changes (update_matrices): the
// elimination with partial pivoting of a tridiagonal solver with row
// interchanges (the fill-in of an interchange is the second super-diagonal),
// tables [row][mode].  Its divisions (540 cycles each) stay out of the
// applications.
template <typename C> struct PotLu {
    C *fact, *dinv, *du, *dl;      // multiplier, 1/U_ii, U_{i,i+1}, U_{i,i+2}
    unsigned char* swap;           // rows i and i+1 interchanged
};

// one thread per mode, in FP64; lu32 (optional): rounded copies
static __global__ void k_pcv_factor(PotLu<double2> lu, PotLu<float2> lu32, PotParams p) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= p.nmv) return;
    const int n = p.nx, m = p.nmv;
    const double2 lam = p.lam[k], zero = make_double2(0.0, 0.0);
    // bands (TensorProductPotentialFast.pyx:228-260): A[i][i], A[i][i+1] and A[i+1][i] (equal)
    auto diag = [&](int i) {
        const int im = i == 0 ? n - 1 : i - 1, ip = i + 1 == n ? 0 : i + 1;
        const double2 dg = c_rmul(c_rmul(c_rmul(lam, 2.0), p.phi[ip] - p.phi[im]), p.arak);
        return make_double2(dg.x + p.ht_inv, dg.y);
    };
    auto off = [&](int i) {
        return i + 1 < n ? c_rmul(c_rmul(c_rmul(lam, 1.0), p.phi[i + 1] - p.phi[i]), p.arak) : zero;
    };
    double2 d = diag(0), u = off(0);   // row i as the elimination left it
    for (int i = 0; i < n; ++i) {
        double2 f = zero, di = d, dui = u, dli = zero;
        unsigned char sw = 0;
        if (i + 1 < n) {
            const double2 l = off(i), dn = diag(i + 1), un = off(i + 1);
            if (c_abs1(d) >= c_abs1(l)) {
                f = c_div(l, d);
                d = c_sub(dn, c_mul(f, u));
                u = un;
            } else {
                sw = 1;
                f = c_div(d, l);
                di = l;
                dui = dn;
                dli = un;
                d = c_sub(u, c_mul(f, dn));
                const double2 t = c_mul(f, un);
                u = make_double2(-t.x, -t.y);
            }
        }
        const double2 inv = c_div(make_double2(1.0, 0.0), di);
        const size_t q = (size_t)i * m + k;
        lu.fact[q] = f;
        lu.dinv[q] = inv;
        lu.du[q] = dui;
        lu.dl[q] = dli;
        lu.swap[q] = sw;
        if (lu32.fact) {
            lu32.fact[q] = make_float2((float)f.x, (float)f.y);
            lu32.dinv[q] = make_float2((float)inv.x, (float)inv.y);
            lu32.du[q] = make_float2((float)dui.x, (float)dui.y);
            lu32.dl[q] = make_float2((float)dli.x, (float)dli.y);
        }
    }
}

// One mode's elimination and back substitution, row i of b at b + i bs, of the
// factors at i m.  A chain of two complex multiply-adds per row; the next rows'
// operands are loaded while it runs (PV_CH rows ahead).
constexpr int PV_CH = 4;
template <typename C>
VV_DEV void pcv_chain(C* b, int bs, const C* fact, const C* dinv, const C* du, const C* dl, const unsigned char* swap,
                      int n, int m) {
    const C zero = c_make<C>(0.0, 0.0);
    {   // forward: b <- L^-1 P b
        C f[2][PV_CH], r[2][PV_CH];
        unsigned char w[2][PV_CH];
        auto load = [&](int s, int i0) {
#pragma unroll
            for (int u = 0; u < PV_CH; ++u) {
                const int i = min(i0 + u, n - 1);
                f[s][u] = fact[(size_t)i * m];
                w[s][u] = swap[(size_t)i * m];
                r[s][u] = b[(size_t)min(i + 1, n - 1) * bs];
            }
        };
        C cur = b[0];
        load(0, 0);
        int i0 = 0;
        auto run = [&](int s) {
            load(s ^ 1, i0 + PV_CH);
#pragma unroll
            for (int u = 0; u < PV_CH; ++u) {
                const int i = i0 + u;
                if (i + 1 < n) {
                    const C nx = r[s][u];
                    const bool sw = w[s][u] != 0;
                    b[(size_t)i * bs] = sw ? nx : cur;
                    cur = sw ? c_sub(cur, c_mul(f[s][u], nx)) : c_sub(nx, c_mul(f[s][u], cur));
                }
            }
            i0 += PV_CH;
        };
        while (i0 < n - 1) {
            run(0);
            if (i0 < n - 1) run(1);
        }
        b[(size_t)(n - 1) * bs] = cur;
    }
    {   // back substitution
        C d[2][PV_CH], u1[2][PV_CH], u2[2][PV_CH], r[2][PV_CH];
        auto load = [&](int s, int i0) {
#pragma unroll
            for (int u = 0; u < PV_CH; ++u) {
                const int i = max(i0 - u, 0);
                const size_t q = (size_t)i * m;
                d[s][u] = dinv[q];
                u1[s][u] = du[q];
                u2[s][u] = dl[q];
                r[s][u] = b[(size_t)i * bs];
            }
        };
        C x1 = zero, x2 = zero;   // x_{i+1}, x_{i+2}
        int i0 = n - 1;
        load(0, i0);
        auto run = [&](int s) {
            load(s ^ 1, i0 - PV_CH);
#pragma unroll
            for (int u = 0; u < PV_CH; ++u) {
                const int i = i0 - u;
                if (i >= 0) {
                    const C x = c_mul(d[s][u], c_sub(c_sub(r[s][u], c_mul(u2[s][u], x2)), c_mul(u1[s][u], x1)));
                    b[(size_t)i * bs] = x;
                    x2 = x1;
                    x1 = x;
                }
            }
            i0 -= PV_CH;
        };
        while (i0 >= 0) {
            run(0);
            if (i0 >= 0) run(1);
        }
    }
}

// A_k c = b in place on spec[k*nx ..], one thread per mode (a warp 32 of them),
// for systems too long for shared memory
template <typename R>
__global__ void __launch_bounds__(32) k_pcv_solve(typename Cplx<R>::type* __restrict__ spec,
                                                  PotLu<typename Cplx<R>::type> lu, int n, int m) {
    const int k = blockIdx.x * 32 + threadIdx.x;
    if (k >= m) return;
    pcv_chain(spec + (size_t)k * n, 1, lu.fact + k, lu.dinv + k, lu.du + k, lu.dl + k, lu.swap + k, n, m);
}

// The same with a block's `mb` modes whole in shared memory: there are only
// nv/2 + 1 chains, so a chain that waits for L2 every PV_CH rows leaves the chip
// idle; here all operands are in flight at once and the chain reads shared memory
// (50 x 101 in FP64: 17.4 -> 11.8 us; staging tiles of 8 rows ahead of the chain,
// a barrier per tile, took 36).
constexpr int PV_THREADS = 128;
constexpr size_t PV_SMEM = 48 * 1024;
inline size_t pcv_smem(size_t csz, int n, int mb) { return (size_t)n * mb * (5 * csz + 1); }
template <typename R>
__global__ void __launch_bounds__(PV_THREADS) k_pcv_solve_sm(typename Cplx<R>::type* __restrict__ spec,
                                                             PotLu<typename Cplx<R>::type> lu, int n, int m, int mb) {
    using C = typename Cplx<R>::type;
    extern __shared__ __align__(16) unsigned char pv_raw[];
    const int e1 = n * mb, k0 = blockIdx.x * mb, on = min(mb, m - k0);
    C* b = reinterpret_cast<C*>(pv_raw);
    C *f = b + e1, *d = f + e1, *u1 = d + e1, *u2 = u1 + e1;
    unsigned char* w = reinterpret_cast<unsigned char*>(u2 + e1);
    for (int e = threadIdx.x; e < n * on; e += PV_THREADS) {
        const int i = e / on, l = e - i * on, t = i * mb + l;
        const size_t q = (size_t)i * m + k0 + l;
        f[t] = lu.fact[q];
        d[t] = lu.dinv[q];
        u1[t] = lu.du[q];
        u2[t] = lu.dl[q];
        w[t] = lu.swap[q];
        const int lb = e / n, ib = e - lb * n;   // a mode's rows are contiguous
        b[ib * mb + lb] = spec[(size_t)k0 * n + e];
    }
    __syncthreads();
    const int l = threadIdx.x;
    if (l < on) pcv_chain(b + l, mb, f + l, d + l, u1 + l, u2 + l, w + l, n, mb);
    __syncthreads();
    for (int e = threadIdx.x; e < n * on; e += PV_THREADS) {
        const int lb = e / n, ib = e - lb * n;
        spec[(size_t)k0 * n + e] = b[ib * mb + lb];
    }
}

}  // namespace vv
