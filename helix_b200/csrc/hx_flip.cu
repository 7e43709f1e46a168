// Stage kernels for coupling operators with transverse (spin-flip) parts and
// for any Hilbert dimension up to 4096.
//
// Coupling operators V_j = diag(v_j) + sum_i w_ji sigma_x(i) (the reference's
// compiled model has one collective V = Dlong sum s_z + Dtrans sum_i sigma_x(i),
// src/initialize.cu:95-147).  Commutators then mix elements within a slab:
//
//   [V,X]_rc = (v_r - v_c) X_rc + sum_i w_i (X_{r^2^i,c} - X_{r,c^2^i})
//   {V,X}_rc = (v_r + v_c) X_rc + sum_i w_i (X_{r^2^i,c} + X_{r,c^2^i})
//
// so, as in the reference (getdRhoSparse, src/liouville.cu:778-860), each
// stage runs in two passes:
//   comm_kernel:     B_{j,n} = [V_j, u_n] and A_{j,n} = {V_j, u_n} for every
//                    bath j and ADO n (both from the same flip loads)
//   combine_kernel:  out_n = base_n + alpha * ( -i[H,u_n] - g_n u_n
//                      - i sum_{m up} B_{j(m), n+e_m}
//                      - i sum_{m down} a_{n,m} B_{j(m), n-e_m}
//                      - sum_j b_{n,j} A_{j, n-e_j0}
//                      - sum_j (Xi_j [V_j, B_{j,n}] + i kappa_j {V_j, B_{j,n}}) )
// The buffer holds B for all (j, n), then A for all (j, n).
// A thread owns E rows of one column, so log2 E row flips are in its registers
// and every other flip asks for E partners at once (L1/L2: a slab of d = 1024
// is 16 MB).  Bound by the 20 reads of 16 bytes per element and pass; with one
// element per thread and one flip after the other they waited on each other.
// Per step at d = 1024, 10 ADOs: 2.99 ms with one element per thread, 2.03 with
// four rows (two rows 3.2, eight rows 2.99: fewer warps hide the latency).

#include <cuda_runtime.h>

#include <cstdint>

#include "hx_internal.h"

namespace hx {

namespace {

// Element, row and column of a thread: E consecutive rows of one column.
struct FlipAt {
    long long n;  // ADO
    int r, c;     // first row, column
    int e;        // first element in the slab; + d per row
};

template <int LOGE>
__device__ __forceinline__ FlipAt flip_at(long long q, int logd)
{
    FlipAt t;
    t.n = q >> (2 * logd - LOGE);
    const int in = static_cast<int>(q - (t.n << (2 * logd - LOGE)));
    t.c = in & ((1 << logd) - 1);
    t.r = (in >> logd) << LOGE;
    t.e = (t.r << logd) + t.c;
    return t;
}

// rowp[k], colp[k]: the partners of the thread's rows under a flip of bit b.
template <int LOGE>
__device__ __forceinline__ void flip_partners(const double2* __restrict__ X, const double2* x, int e, int b, int logd,
                                              double2* rowp, double2* colp)
{
    constexpr int E = 1 << LOGE;
    const int D = 1 << logd;
    if (b >= LOGE) {
        const double2* p = X + (e ^ (1 << (b + logd)));
#pragma unroll
        for (int k = 0; k < E; ++k) rowp[k] = __ldg(p + k * D);
    } else {
#pragma unroll
        for (int k = 0; k < E; ++k) {
            // a register of the thread: k ^ 2^b, by selects (b is not a constant)
            rowp[k] = x[k ^ 1];
            if (LOGE > 1 && b == 1) rowp[k] = x[k ^ (LOGE > 1 ? 2 : 0)];
            if (LOGE > 2 && b == 2) rowp[k] = x[k ^ (LOGE > 2 ? 4 : 0)];
        }
    }
    const double2* p = X + (e ^ (1 << b));
#pragma unroll
    for (int k = 0; k < E; ++k) colp[k] = __ldg(p + k * D);
}

template <int LOGE>
__global__ void __launch_bounds__(256, LOGE ? 3 : 4)
    comm_kernel(FlipArgs a, const double2* __restrict__ u, double2* __restrict__ B)
{
    constexpr int E = 1 << LOGE;
    const int D = 1 << a.logd;
    const long long D2 = static_cast<long long>(D) * D;
    const long long HD2 = a.H * D2;
    const long long total = static_cast<long long>(a.J) * HD2;
    const long long q = blockIdx.x * 256ll + threadIdx.x;
    if (q >= (HD2 >> LOGE)) return;
    const FlipAt t = flip_at<LOGE>(q, a.logd);
    const double2* un = u + t.n * D2;
    double2 x[E];
#pragma unroll
    for (int k = 0; k < E; ++k) x[k] = __ldg(un + t.e + k * D);
    for (int j = 0; j < a.J; ++j) {
        // P = V u, Q = u V
        double2 P[E], Q[E];
        const double vc = __ldg(a.vdiag + j * D + t.c);
#pragma unroll
        for (int k = 0; k < E; ++k) {
            const double vr = __ldg(a.vdiag + j * D + t.r + k);
            P[k] = make_double2(vr * x[k].x, vr * x[k].y);
            Q[k] = make_double2(vc * x[k].x, vc * x[k].y);
        }
#pragma unroll 1
        for (int b = 0; b < a.logd; ++b) {
            const double w = __ldg(a.vflip + j * a.logd + b);
            if (w == 0.0) continue;
            double2 pr[E], pc[E];
            flip_partners<LOGE>(un, x, t.e, b, a.logd, pr, pc);
#pragma unroll
            for (int k = 0; k < E; ++k) {
                P[k].x = fma(w, pr[k].x, P[k].x);
                P[k].y = fma(w, pr[k].y, P[k].y);
                Q[k].x = fma(w, pc[k].x, Q[k].x);
                Q[k].y = fma(w, pc[k].y, Q[k].y);
            }
        }
        const long long idx = static_cast<long long>(j) * HD2 + t.n * D2 + t.e;
#pragma unroll
        for (int k = 0; k < E; ++k) {
            B[idx + k * D] = make_double2(P[k].x - Q[k].x, P[k].y - Q[k].y);
            B[total + idx + k * D] = make_double2(P[k].x + Q[k].x, P[k].y + Q[k].y);
        }
    }
}

template <int LOGE>
__global__ void __launch_bounds__(256, LOGE ? 3 : 4)
    combine_kernel(FlipArgs a, const double2* __restrict__ u, const double2* __restrict__ B, const double2* rho,
                   double2* out, double alpha, int base_kind)
{
    constexpr int E = 1 << LOGE;
    const int D = 1 << a.logd;
    const long long D2 = static_cast<long long>(D) * D;
    const long long HD2 = a.H * D2;
    const long long q = blockIdx.x * 256ll + threadIdx.x;
    if (q >= (HD2 >> LOGE)) return;
    const FlipAt t = flip_at<LOGE>(q, a.logd);
    const double2* un = u + t.n * D2;
    double2 acc[E];
    // -g u - i (E_r - E_c) u - i sum_i h_i (u_{r^i,c} - u_{r,c^i})
    {
        double2 x[E];
#pragma unroll
        for (int k = 0; k < E; ++k) x[k] = __ldg(un + t.e + k * D);
        const double g = __ldg(a.gsum + t.n), ec = __ldg(a.hdiag + t.c);
#pragma unroll
        for (int k = 0; k < E; ++k) {
            const double dE = __ldg(a.hdiag + t.r + k) - ec;
            acc[k].x = fma(dE, x[k].y, -g * x[k].x);
            acc[k].y = fma(-dE, x[k].x, -g * x[k].y);
        }
        for (int b = 0; b < a.logd; ++b) {
            const double h = __ldg(a.hflip + b);
            if (h == 0.0) continue;
            double2 pr[E], pc[E];
            flip_partners<LOGE>(un, x, t.e, b, a.logd, pr, pc);
#pragma unroll
            for (int k = 0; k < E; ++k) {
                acc[k].x = fma(h, pr[k].y - pc[k].y, acc[k].x);
                acc[k].y = fma(-h, pr[k].x - pc[k].x, acc[k].y);
            }
        }
    }
    const int32_t* edges = a.edges + t.n * 2 * a.M;
    for (int j = 0; j < a.J; ++j) {
        const double2* Bj = B + static_cast<long long>(j) * HD2;
        const int m0 = __ldg(a.bath_off + j), m1 = __ldg(a.bath_off + j + 1);
        // up and down neighbours: -i B_up, -i a B_down
#pragma unroll 2
        for (int m = m0; m < m1; ++m) {
            const int up = __ldg(edges + m), dn = __ldg(edges + a.M + m);
            const double w = dn < a.H ? __ldg(a.acoef + t.n * a.M + m) : 0.0;
            double2 yu[E], yd[E];
#pragma unroll
            for (int k = 0; k < E; ++k) {
                yu[k] = up < a.H ? __ldg(Bj + up * D2 + t.e + k * D) : make_double2(0.0, 0.0);
                yd[k] = dn < a.H ? __ldg(Bj + dn * D2 + t.e + k * D) : make_double2(0.0, 0.0);
            }
#pragma unroll
            for (int k = 0; k < E; ++k) {
                acc[k].x += fma(w, yd[k].y, yu[k].y);
                acc[k].y -= fma(w, yd[k].x, yu[k].x);
            }
        }
        // theta2: -b {V_j, u_{n-e_j0}} = -b A_{j, n-e_j0}
        const int dn0 = __ldg(edges + a.M + m0);
        if (dn0 < a.H) {
            const double bw = __ldg(a.bcoef + t.n * a.J + j);
            const double2* An = Bj + static_cast<long long>(a.J) * HD2 + dn0 * D2 + t.e;
#pragma unroll
            for (int k = 0; k < E; ++k) {
                const double2 y = __ldg(An + k * D);
                acc[k].x = fma(-bw, y.x, acc[k].x);
                acc[k].y = fma(-bw, y.y, acc[k].y);
            }
        }
        // Xi and counter: -Xi [V, B_n] - i kappa {V, B_n} = (-Xi - i kappa) V B_n + (Xi - i kappa) B_n V
        const double2* Bn = Bj + t.n * D2;
        const double xi = __ldg(a.xi + j), ka = __ldg(a.counter + j);
        double2 y[E];
        const double vc = __ldg(a.vdiag + j * D + t.c);
#pragma unroll
        for (int k = 0; k < E; ++k) y[k] = __ldg(Bn + t.e + k * D);
#pragma unroll
        for (int k = 0; k < E; ++k) {
            const double vr = __ldg(a.vdiag + j * D + t.r + k);
            const double cr = -xi * (vr - vc), ci = -ka * (vr + vc);
            acc[k].x = fma(cr, y[k].x, fma(-ci, y[k].y, acc[k].x));
            acc[k].y = fma(cr, y[k].y, fma(ci, y[k].x, acc[k].y));
        }
#pragma unroll 1
        for (int b = 0; b < a.logd; ++b) {
            const double w = __ldg(a.vflip + j * a.logd + b);
            if (w == 0.0) continue;
            double2 pr[E], pc[E];
            flip_partners<LOGE>(Bn, y, t.e, b, a.logd, pr, pc);
            const double wx = w * xi, wk = w * ka;
#pragma unroll
            for (int k = 0; k < E; ++k) {
                acc[k].x = fma(-wx, pr[k].x - pc[k].x, fma(wk, pr[k].y + pc[k].y, acc[k].x));
                acc[k].y = fma(-wx, pr[k].y - pc[k].y, fma(-wk, pr[k].x + pc[k].x, acc[k].y));
            }
        }
    }
#pragma unroll
    for (int k = 0; k < E; ++k) {
        const long long idx = t.n * D2 + t.e + k * D;
        double2 base = make_double2(0.0, 0.0);
        if (base_kind == kBaseSelf) base = __ldg(un + t.e + k * D);
        else if (base_kind == kBaseRho) base = rho[idx];
        out[idx] = make_double2(fma(alpha, acc[k].x, base.x), fma(alpha, acc[k].y, base.y));
    }
}

template <int LOGE>
void launch_flip_t(const FlipArgs& a, const double2* u, double2* B, const double2* rho, double2* out, double alpha,
                   int base_kind, cudaStream_t s)
{
    const long long threads = (a.H << (2 * a.logd)) >> LOGE;
    const unsigned grid = static_cast<unsigned>((threads + 255) / 256);
    comm_kernel<LOGE><<<grid, 256, 0, s>>>(a, u, B);
    combine_kernel<LOGE><<<grid, 256, 0, s>>>(a, u, B, rho, out, alpha, base_kind);
}

}  // namespace

void launch_flip_stage(const FlipArgs& a, const double2* u, double2* B, const double2* rho, double2* out,
                       double alpha, int base_kind, cudaStream_t s)
{
    // four rows per thread once that still fills the GPU
    if (a.logd >= 2 && (a.H << (2 * a.logd)) >= 4 * 148 * 512) launch_flip_t<2>(a, u, B, rho, out, alpha, base_kind, s);
    else launch_flip_t<0>(a, u, B, rho, out, alpha, base_kind, s);
}

}  // namespace hx
