// Cluster-resident step: launch, shapes and tables (vv_cluster.h).
#include "vv_cluster.h"
#include "vv_cluster.cuh"

#include <algorithm>
#include <mutex>
#include <vector>

namespace vv {

namespace {

template <typename T> const void* kernel_t(int fam) {
    switch (fam) {
        case 32: return (const void*)k_cl_run<T, 32>;
        case 64: return (const void*)k_cl_run<T, 64>;
        case 128: return (const void*)k_cl_run<T, 128>;
        case 256: return (const void*)k_cl_run<T, 256>;
        default: return (const void*)k_cl_run<T, 0>;
    }
}
const void* kernel_of(bool fp32, int fam) { return fp32 ? kernel_t<float>(fam) : kernel_t<double>(fam); }

// slot s of row j: mode cl_mode_of(fam, s); slot 0 of an FFT row holds the
// real pair (X_0, X_M), whose matrices are 1/ht I (their eigenvalues vanish)
template <typename C>
__global__ void k_cl_table(const C* __restrict__ dinv, const C* __restrict__ lambda, C* __restrict__ dinv_s,
                           C* __restrict__ lam_s, int fam, int slots, int nv, double ht) {
    const size_t n = (size_t)nv * slots;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
        const int j = (int)(t / slots), s = (int)(t - (size_t)j * slots);
        const int k = cl_mode_of(fam, s);
        dinv_s[t] = fam && s == 0 ? c_make<C>(ht, 0.0) : dinv[(size_t)k * nv + j];
        if (j == 0) lam_s[s] = fam && s == 0 ? c_make<C>(0.0, 0.0) : lambda[k];
    }
}

}  // namespace

int cl_family(int nx, bool pow2) {
    const int M = nx / 2;
    return pow2 && M >= 32 && M <= 256 ? M : 0;
}

// set up for the kernels that are asked for: the attributes load a kernel, which
// costs milliseconds
size_t cl_smem_limit(bool fp32, int fam) {
    static std::mutex mu;
    static size_t limit[64][2][5] = {};
    int dev = 0, q = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    for (int m = 32; m <= fam; m *= 2) ++q;
    std::lock_guard<std::mutex> lock(mu);
    size_t& l = limit[dev][fp32 ? 1 : 0][q];
    if (l == 0) {
        int optin = 0;
        cudaFuncAttributes fa;
        const void* k = kernel_of(fp32, fam);
        if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
            cudaFuncGetAttributes(&fa, k) != cudaSuccess)
            return cudaGetLastError(), 0;
        const int dyn = optin - (int)fa.sharedSizeBytes;
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) != cudaSuccess ||
            cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
            return cudaGetLastError(), 0;
        l = (size_t)dyn;
    }
    return l;
}

ClShape cl_shape(int nx, int nv, bool pow2, int ctas, int tsz, size_t smem_limit) {
    ClShape s{};
    if (nx > CL_NXMAX || ctas < 1 || ctas > CL_MAXC) return s;
    s.fam = cl_family(nx, pow2);
    s.slots = cl_slots(s.fam, nx);
    s.rows = (nv + ctas - 1) / ctas;
    // chunks of about eight rows, of at most CL_CHUNK, one thread per (chunk, slot)
    const int most = CL_THREADS / s.slots;
    if (most < 1) return ClShape{};
    s.nch = std::max(1, std::min(most, (s.rows + 7) / 8));
    if ((s.rows + s.nch - 1) / s.nch > CL_CHUNK) return ClShape{};
    auto bytes = [&]() { return cl_layout(s.fam, nx, s.rows, s.nch, tsz, s.kv, s.dsm).bytes; };
    if (bytes() > smem_limit) return ClShape{};
    // what is left of the shared memory: the LU reciprocals, then basis vectors
    s.dsm = 1;
    if (bytes() > smem_limit) s.dsm = 0;
    while (s.kv < CL_RESTART + 1 && (++s.kv, bytes() <= smem_limit)) {}
    while (s.kv > 0 && bytes() > smem_limit) --s.kv;
    s.smem = bytes();
    s.ctas = ctas;
    return s;
}

int cl_resident(bool fp32, int fam, int ctas) {
    const size_t smem = cl_smem_limit(fp32, fam);
    if (smem == 0) return 0;
    // the answer of each kind is kept: the query costs about a millisecond
    struct Key {
        int dev, fp32, fam, ctas, n;
    };
    static std::mutex mu;
    static std::vector<Key> seen;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    std::lock_guard<std::mutex> lock(mu);
    for (const Key& k : seen)
        if (k.dev == dev && k.fp32 == (int)fp32 && k.fam == fam && k.ctas == ctas) return k.n;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(CL_THREADS);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)ctas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel_of(fp32, fam), &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    seen.push_back({dev, (int)fp32, fam, ctas, n});
    return n;
}

int cl_levels(const ClShape& s, int nv, const double* lf, const double* lb, double tol) {
    const int total = s.ctas * s.nch;
    std::vector<double> pf(total), pb(total);
    for (int g = 0; g < total; ++g) {
        const int r0 = g / s.nch * s.rows, c = g % s.nch;
        const int nr = std::max(0, std::min(s.rows, nv - r0));
        double a = 1.0, b = 1.0;
        for (int j = r0 + c * nr / s.nch; j < r0 + (c + 1) * nr / s.nch; ++j) {
            a *= lf[j];
            b *= lb[j];
        }
        pf[g] = a;
        pb[g] = b;
    }
    // a carry from lev chunks leaves out what their product scales
    int lev = 1;
    for (; lev < total; ++lev) {
        bool fits = true;
        for (int g = 0; g + lev <= total && fits; ++g) {
            double a = 1.0, b = 1.0;
            for (int q = 0; q < lev; ++q) {
                a *= pf[g + q];
                b *= pb[g + q];
            }
            fits = a <= tol * tol && b <= tol * tol;
        }
        if (fits) break;
    }
    return lev;
}

cudaError_t cl_tables(bool fp32, const ClShape& s, int nv, const void* dinv, const void* lambda, void* dinv_s,
                      void* lam_s, double ht, cudaStream_t st) {
    const unsigned g = (unsigned)std::min<size_t>(1024, ((size_t)nv * s.slots + 255) / 256);
    if (fp32)
        k_cl_table<float2><<<g, 256, 0, st>>>((const float2*)dinv, (const float2*)lambda, (float2*)dinv_s,
                                              (float2*)lam_s, s.fam, s.slots, nv, ht);
    else
        k_cl_table<double2><<<g, 256, 0, st>>>((const double2*)dinv, (const double2*)lambda, (double2*)dinv_s,
                                               (double2*)lam_s, s.fam, s.slots, nv, ht);
    return cudaGetLastError();
}

cudaError_t cl_launch(bool fp32, int fam, const ClInst* tab, const int* order, int n, int ctas, size_t smem, int mode,
                      cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(n * ctas));
    cfg.blockDim = dim3(CL_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)ctas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    void* args[] = {(void*)&tab, (void*)&order, (void*)&mode};
    return cudaLaunchKernelExC(&cfg, kernel_of(fp32, fam), args);
}

}  // namespace vv
