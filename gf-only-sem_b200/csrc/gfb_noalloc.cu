// gfb_noalloc.cu -- element internal force for callers that cannot allocate
// device memory.
//
// gfb_element_residual (gfb_solver.cu) allocates device buffers for every
// call: the inputs and output, the cell geometry in the time loop's layout,
// the node table and the GLL derivative table.  Some callers cannot do that:
// code that embeds the kernel in a time loop whose device memory is owned by a
// caching pool (allocating behind the pool's back fragments it and can fail
// under memory pressure), code that must not trigger the implicit device
// synchronisation of cudaMalloc/cudaFree inside a latency-critical loop, and
// code running where the allocator is intercepted or forbidden.  Those callers
// already hold device buffers for their inputs and output, in the reference's
// layout; the kernel here reads and writes exactly those.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <vector>

#include "../../include/gfb.h"
#include "gfb_internal.h"

namespace {

struct GllTables {
    double w[6];
    double D[36];
    bool ok;
};

GllTables make_tables(int ngll) {
    GllTables t{};
    std::vector<double> w, D;
    t.ok = gfb::gll_tables_for(ngll, w, D);
    if (t.ok) {
        std::copy(w.begin(), w.end(), t.w);
        std::copy(D.begin(), D.end(), t.D);
    }
    return t;
}

// The tables of each ngll, computed once.
const GllTables& tables(int ngll) {
    static const GllTables t[4] = {make_tables(3), make_tables(4), make_tables(5), make_tables(6)};
    return t[ngll - 3];
}

template <int NG>
struct DirectShape {
    static constexpr int NN = NG * NG * NG;
    static constexpr int NNP = (NN + 31) / 32 * 32;
    static constexpr int CELLS = NNP <= 32 ? 4 : (NNP <= 64 ? 2 : 1);
    static constexpr int THREADS = NNP * CELLS;
};

// K_e u of independent cells straight from the caller's arrays (element_cpu.cpp:
// 19-162), one thread per GLL point, a cell (several below ngll 5) per block.
// A call is a few hundred cells, so it is bound by latency: one launch, every
// input fetched once by coalesced loads that are all in flight together, the
// fluxes in the shared memory the geometry came in.  600 cells at ngll 5 take
// 8.0 us per call in a stream of calls, 14.3 when a first kernel repacked the
// inputs into a scratch array.
template <int NG>
__global__ void __launch_bounds__(DirectShape<NG>::THREADS)
    elem_direct_kernel(int n_elem, const double* dxi_dx, const double* jacobian, const double* lambda_, const double* mu_,
                       const double* u, double* r, const __grid_constant__ GllTables t) {
    using S = DirectShape<NG>;
    constexpr int NN = S::NN, CELLS = S::CELLS, THREADS = S::THREADS;
    __shared__ double s_geo[CELLS * NN * 9];  // dxi_dx [cell][p][9], then fluxes [cell][axis][component][p]
    __shared__ double s_u[CELLS * NN * 3];
    __shared__ double sD[NG * NG];
    const int tid = threadIdx.x, el = tid / S::NNP, p = tid - el * S::NNP;
    const int e0 = blockIdx.x * CELLS, nc = min(CELLS, n_elem - e0);
    const bool active = p < NN && el < nc;
    const size_t q0 = (size_t)e0 * NN, q = q0 + (size_t)el * NN + p;
#pragma unroll
    for (int x = 0; x < (CELLS * NN * 9 + THREADS - 1) / THREADS; ++x) {
        const int at = x * THREADS + tid;
        if (at < nc * NN * 9) s_geo[at] = dxi_dx[q0 * 9 + at];
    }
#pragma unroll
    for (int x = 0; x < (CELLS * NN * 3 + THREADS - 1) / THREADS; ++x) {
        const int at = x * THREADS + tid;
        if (at < nc * NN * 3) s_u[at] = u[q0 * 3 + at];
    }
    if (tid < NG * NG) sD[tid] = t.D[tid];
    double jac = 0.0, lam = 0.0, mu = 0.0;
    if (active) {
        jac = jacobian[q];
        lam = lambda_[q];
        mu = mu_[q];
    }
    __syncthreads();
    const int i = p / (NG * NG), j = (p / NG) % NG, k = p % NG;
    double dd[9];
    double* fl = s_geo + el * NN * 9;
    if (active) {
#pragma unroll
        for (int x = 0; x < 9; ++x) dd[x] = fl[p * 9 + x];
    }
    __syncthreads();  // the geometry is in registers
    if (active) {
        const double* ue = s_u + el * NN * 3;
        double gx[3] = {0, 0, 0}, gy[3] = {0, 0, 0}, gz[3] = {0, 0, 0};
#pragma unroll
        for (int s = 0; s < NG; ++s) {
            const double a = sD[i * NG + s], b = sD[j * NG + s], c = sD[k * NG + s];
            const double* ua = ue + 3 * ((s * NG + j) * NG + k);
            const double* ub = ue + 3 * ((i * NG + s) * NG + k);
            const double* uc = ue + 3 * ((i * NG + j) * NG + s);
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                gx[x] += a * ua[x];
                gy[x] += b * ub[x];
                gz[x] += c * uc[x];
            }
        }
        // physical gradient with the reference's reading of dxi_dx
        double gr[3][3];
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            gr[x][0] = gx[x] * dd[0] + gy[x] * dd[1] + gz[x] * dd[2];
            gr[x][1] = gx[x] * dd[3] + gy[x] * dd[4] + gz[x] * dd[5];
            gr[x][2] = gx[x] * dd[6] + gy[x] * dd[7] + gz[x] * dd[8];
        }
        // weight detJ w_i w_j w_k (element_cpu.cpp:108); mu <= 0: the point
        // adds nothing (element_cpu.cpp:42-43)
        const bool on = mu > 0.0;
        const double jw = jac * t.w[i] * t.w[j] * t.w[k];
        const double tr = lam * (gr[0][0] + gr[1][1] + gr[2][2]), m2 = 2.0 * mu;
        double sg[3][3];
        sg[0][0] = m2 * gr[0][0] + tr;
        sg[1][1] = m2 * gr[1][1] + tr;
        sg[2][2] = m2 * gr[2][2] + tr;
        sg[0][1] = sg[1][0] = mu * (gr[0][1] + gr[1][0]);
        sg[0][2] = sg[2][0] = mu * (gr[0][2] + gr[2][0]);
        sg[1][2] = sg[2][1] = mu * (gr[1][2] + gr[2][1]);
        // flux along reference axis a: jw * sigma . (dd[a], dd[3+a], dd[6+a])
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int x = 0; x < 3; ++x)
                fl[(a * 3 + x) * NN + p] =
                    on ? jw * (sg[x][0] * dd[a] + sg[x][1] * dd[3 + a] + sg[x][2] * dd[6 + a]) : 0.0;
    }
    __syncthreads();
    if (!active) return;
    double acc[3] = {0, 0, 0};
#pragma unroll
    for (int s = 0; s < NG; ++s) {
        const double a = sD[s * NG + i], b = sD[s * NG + j], c = sD[s * NG + k];
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            acc[x] += a * fl[x * NN + (s * NG + j) * NG + k];
            acc[x] += b * fl[(3 + x) * NN + (i * NG + s) * NG + k];
            acc[x] += c * fl[(6 + x) * NN + (i * NG + j) * NG + s];
        }
    }
#pragma unroll
    for (int x = 0; x < 3; ++x) r[q * 3 + x] = -acc[x];
}

template <int NG>
gfb_status run(int n_elem, const double* dxi_dx, const double* jacobian, const double* lambda_, const double* mu,
               const double* u, double* r, const GllTables& t, cudaStream_t stream) {
    using S = DirectShape<NG>;
    elem_direct_kernel<NG><<<(n_elem + S::CELLS - 1) / S::CELLS, S::THREADS, 0, stream>>>(n_elem, dxi_dx, jacobian,
                                                                                         lambda_, mu, u, r, t);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        char msg[256];
        snprintf(msg, sizeof(msg), "element residual (no-alloc): element kernel launch failed: %s",
                 cudaGetErrorString(e));
        return gfb::set_error(GFB_ERR_CUDA, msg);
    }
    return GFB_OK;
}

// Largest call per ngll, part of the interface (include/gfb.h).
int max_cells_for(int ngll) {
    constexpr int kMax[4] = {3106, 1310, 671, 388};
    return kMax[ngll - 3];
}

}  // namespace

extern "C" {

gfb_status gfb_element_residual_noalloc(int32_t n_elem, const double* dxi_dx, const double* jacobian,
                                        const double* lambda_, const double* mu, int32_t ngll, const double* u,
                                        double* r, void* stream) {
    if (!dxi_dx || !jacobian || !lambda_ || !mu || !u || !r)
        return gfb::set_error(GFB_ERR_INVALID, "element residual (no-alloc): missing device pointer");
    if (ngll < 3 || ngll > 6)
        return gfb::set_error(GFB_ERR_UNSUPPORTED, "element residual (no-alloc): ngll must be 3..6");
    if (n_elem <= 0) return gfb::set_error(GFB_ERR_INVALID, "element residual (no-alloc): n_elem must be > 0");
    if (n_elem > max_cells_for(ngll)) {
        char msg[256];
        snprintf(msg, sizeof(msg),
                 "element residual (no-alloc): %d cells exceed the maximum of %d cells at ngll=%d; split the call",
                 n_elem, max_cells_for(ngll), ngll);
        return gfb::set_error(GFB_ERR_INVALID, msg);
    }
    // an error left by an earlier, unrelated call would otherwise be read
    // back after this call's launch and reported as its own: clear it (a
    // sticky error of a broken context comes back at the launch anyway)
    (void)cudaGetLastError();
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return gfb::set_error(GFB_ERR_NO_DEVICE, "no current CUDA device");
    const GllTables& t = tables(ngll);
    if (!t.ok) return gfb::set_error(GFB_ERR_INVALID, "GLL tables failed");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    switch (ngll) {
        case 3: return run<3>(n_elem, dxi_dx, jacobian, lambda_, mu, u, r, t, s);
        case 4: return run<4>(n_elem, dxi_dx, jacobian, lambda_, mu, u, r, t, s);
        case 5: return run<5>(n_elem, dxi_dx, jacobian, lambda_, mu, u, r, t, s);
        default: return run<6>(n_elem, dxi_dx, jacobian, lambda_, mu, u, r, t, s);
    }
}

}  // extern "C"
