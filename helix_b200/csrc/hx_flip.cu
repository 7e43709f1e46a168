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
// Every commutator and anti-commutator is summed from the differences and sums
// of its terms, and every group of terms by itself: V u and u V apart lose the
// digits that a common part of V's diagonal takes, and one running sum is
// rounded at its full size by every flip (twice the error of a right-hand side).
// A thread owns E rows of one column, so log2 E row flips are in its registers
// and every other flip asks for E partners at once (L1/L2: a slab of d = 1024
// is 16 MB).  Bound by the 20 reads of 16 bytes per element and pass; with one
// element per thread and one flip after the other they waited on each other.
// Per step at d = 1024, 10 ADOs: 2.99 ms with one element per thread, 2.03 with
// four rows (two rows 3.2, eight rows 2.99: fewer warps hide the latency); 1.91
// as it is now, 2.31 with flips in H too.  Couplings with flips at d <= 32 run
// whole steps in one launch (flip_run_kernel).

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "hx_internal.h"
#include "hx_run.cuh"

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

// f(k, w, row partner, column partner) for the thread's rows and every flip of weight w != 0.  Row partners of the
// low log2 E bits are the thread's own rows (in x), which are not needed afterwards.
template <int LOGE, typename F>
__device__ __forceinline__ void for_flips(const double2* __restrict__ X, const double2* x, int e,
                                          const double* __restrict__ weight, int logd, F f)
{
    constexpr int E = 1 << LOGE;
    const int D = 1 << logd;
#pragma unroll
    for (int b = 0; b < LOGE; ++b) {
        const double w = __ldg(weight + b);
        if (w == 0.0) continue;
        const double2* p = X + (e ^ (1 << b));
        double2 colp[E];
#pragma unroll
        for (int k = 0; k < E; ++k) colp[k] = __ldg(p + k * D);
#pragma unroll
        for (int k = 0; k < E; ++k) f(k, w, x[k ^ (1 << b)], colp[k]);
    }
#pragma unroll 1
    for (int b = LOGE; b < logd; ++b) {
        const double w = __ldg(weight + b);
        if (w == 0.0) continue;
        const double2 *p = X + (e ^ (1 << (b + logd))), *q = X + (e ^ (1 << b));
        double2 rowp[E], colp[E];
#pragma unroll
        for (int k = 0; k < E; ++k) rowp[k] = __ldg(p + k * D);
#pragma unroll
        for (int k = 0; k < E; ++k) colp[k] = __ldg(q + k * D);
#pragma unroll
        for (int k = 0; k < E; ++k) f(k, w, rowp[k], colp[k]);
    }
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
    for (int j = 0; j < a.J; ++j) {
        double2 x[E];
#pragma unroll
        for (int k = 0; k < E; ++k) x[k] = __ldg(un + t.e + k * D);
        // C = [V, u] and A = {V, u}, each from the differences and sums of its terms: V u and u V apart lose the
        // digits that a common part of V's diagonal takes
        double2 C[E], A[E];
        const double vc = __ldg(a.vdiag + j * D + t.c);
#pragma unroll
        for (int k = 0; k < E; ++k) {
            const double vr = __ldg(a.vdiag + j * D + t.r + k);
            C[k] = make_double2((vr - vc) * x[k].x, (vr - vc) * x[k].y);
            A[k] = make_double2((vr + vc) * x[k].x, (vr + vc) * x[k].y);
        }
        for_flips<LOGE>(un, x, t.e, a.vflip + j * a.logd, a.logd, [&](int k, double w, double2 pr, double2 pc) {
            C[k].x = fma(w, pr.x - pc.x, C[k].x);
            C[k].y = fma(w, pr.y - pc.y, C[k].y);
            A[k].x = fma(w, pr.x + pc.x, A[k].x);
            A[k].y = fma(w, pr.y + pc.y, A[k].y);
        });
        const long long idx = static_cast<long long>(j) * HD2 + t.n * D2 + t.e;
#pragma unroll
        for (int k = 0; k < E; ++k) {
            B[idx + k * D] = C[k];
            B[total + idx + k * D] = A[k];
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
    // every group of terms is summed by itself and then added: the sum so far is rounded once per group
    double2 acc[E];
    // - i sum_i h_i (u_{r^i,c} - u_{r,c^i}) - i (E_r - E_c) u - g u
    {
        double2 x[E];
#pragma unroll
        for (int k = 0; k < E; ++k) {
            x[k] = __ldg(un + t.e + k * D);
            acc[k] = make_double2(0.0, 0.0);
        }
        for_flips<LOGE>(un, x, t.e, a.hflip, a.logd, [&](int k, double h, double2 pr, double2 pc) {
            acc[k].x = fma(h, pr.y - pc.y, acc[k].x);
            acc[k].y = fma(-h, pr.x - pc.x, acc[k].y);
        });
        const double g = __ldg(a.gsum + t.n), ec = __ldg(a.hdiag + t.c);
#pragma unroll
        for (int k = 0; k < E; ++k) {
            const double2 y = __ldg(un + t.e + k * D);
            const double dE = __ldg(a.hdiag + t.r + k) - ec;
            acc[k].x += fma(dE, y.y, -g * y.x);
            acc[k].y += fma(-dE, y.x, -g * y.y);
        }
    }
    const int32_t* edges = a.edges + t.n * 2 * a.M;
    for (int j = 0; j < a.J; ++j) {
        const double2* Bj = B + static_cast<long long>(j) * HD2;
        const int m0 = __ldg(a.bath_off + j), m1 = __ldg(a.bath_off + j + 1);
        // up and down neighbours: -i B_up, -i a B_down
        double2 s[E];
#pragma unroll
        for (int k = 0; k < E; ++k) s[k] = make_double2(0.0, 0.0);
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
                s[k].x += fma(w, yd[k].x, yu[k].x);
                s[k].y += fma(w, yd[k].y, yu[k].y);
            }
        }
#pragma unroll
        for (int k = 0; k < E; ++k) {
            acc[k].x += s[k].y;
            acc[k].y -= s[k].x;
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
        for (int k = 0; k < E; ++k) {
            y[k] = __ldg(Bn + t.e + k * D);
            const double vr = __ldg(a.vdiag + j * D + t.r + k);
            const double cr = -xi * (vr - vc), ci = -ka * (vr + vc);
            s[k].x = fma(cr, y[k].x, -ci * y[k].y);
            s[k].y = fma(cr, y[k].y, ci * y[k].x);
        }
        for_flips<LOGE>(Bn, y, t.e, a.vflip + j * a.logd, a.logd, [&](int k, double w, double2 pr, double2 pc) {
            s[k].x = fma(w, fma(-xi, pr.x - pc.x, ka * (pr.y + pc.y)), s[k].x);
            s[k].y = fma(w, fma(-xi, pr.y - pc.y, -ka * (pr.x + pc.x)), s[k].y);
        });
#pragma unroll
        for (int k = 0; k < E; ++k) {
            acc[k].x += s[k].x;
            acc[k].y += s[k].y;
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

// Whole integrator steps in one cooperative launch (d <= 32), a CTA per ADO:
// grid barriers between the stages, the last CTA records rho_0 and the
// observables.  With C_j = [V_j, u_n], S_j the sum of the up neighbours and of
// the down neighbours times a, and u_d the Drude mode's down neighbour, a bath
// contributes
//   [V_j, T_j] + {V_j, A_j},   T_j = -i S_j - xi_j C_j,  A_j = -b_j u_d - i kappa_j C_j,
// and S_j, u_d are sums of neighbours of u, not of their commutators: the
// slab, T_j and A_j in shared memory, two block barriers per bath, and no
// commutator leaves the CTA.  Commutators and anti-commutators are formed from
// the differences and sums of their terms, as in the two passes above.  A
// thread keeps its elements of the slab and of the Horner base in registers.
template <int LOGD> struct FlipRunShape {
    static constexpr int D = 1 << LOGD, D2 = D * D;
    static constexpr int T = D2 > 512 ? 512 : (D2 < 32 ? 32 : D2);
    static constexpr int E = D2 > T ? D2 / T : 1;  // elements of a thread, T / D rows apart
};

// y += sum_b w_b (X_{r^b,c} -+ X_{r,c^b}) at element e of a slab: the flips of a commutator, or of an
// anti-commutator (PLUS).
template <int LOGD, bool PLUS>
__device__ __forceinline__ void slab_flips(const double2* X, int e, const double* w, double2& y)
{
#pragma unroll
    for (int b = 0; b < LOGD; ++b) {
        const double h = w[b];
        if (h == 0.0) continue;
        const double2 p = X[e ^ (1 << (LOGD + b))], q = X[e ^ (1 << b)];
        y.x = fma(h, PLUS ? p.x + q.x : p.x - q.x, y.x);
        y.y = fma(h, PLUS ? p.y + q.y : p.y - q.y, y.y);
    }
}

template <int LOGD>
__global__ void __launch_bounds__(FlipRunShape<LOGD>::T)
    flip_run_kernel(FlipArgs a, double2* rho, double2* ua, double2* ub, double dt, int order, int nsteps,
                    unsigned* gcount, int* error_flag, StepWait w, double2* trace, double* obs)
{
    using S = FlipRunShape<LOGD>;
    constexpr int D = S::D, D2 = S::D2, T = S::T, E = S::E;
    extern __shared__ __align__(16) unsigned char smem[];
    double2* X = reinterpret_cast<double2*>(smem);     // [D2] the slab
    double2* sT = X + D2;                              // [D2]
    double2* sA = sT + D2;                             // [D2]
    double* sE = reinterpret_cast<double*>(sA + D2);   // [D] diagonal of H
    double* sH = sE + D;                               // [LOGD] its flips
    double* sV = sH + LOGD;                            // [J][D]
    double* sW = sV + a.J * D;                         // [J][LOGD]
    const int tid = threadIdx.x;
    const bool watch = trace != nullptr || obs != nullptr;
    const bool watcher = watch && blockIdx.x == gridDim.x - 1;
    const bool on = tid < D2 && !watcher;
    const long long n = blockIdx.x;
    for (int i = tid; i < D; i += T) sE[i] = a.hdiag[i];
    for (int i = tid; i < a.J * D; i += T) sV[i] = a.vdiag[i];
    if (tid < LOGD) sH[tid] = a.hflip[tid];
    for (int i = tid; i < a.J * LOGD; i += T) sW[i] = a.vflip[i];
    const double g = watcher ? 0.0 : a.gsum[n];
    const int32_t* edges = a.edges + (watcher ? 0 : n) * 2 * a.M;
    const int c = tid & (D - 1);
    double2 x[E], base[E];
#pragma unroll
    for (int k = 0; k < E; ++k) x[k] = base[k] = on ? __ldcg(rho + n * D2 + tid + T * k) : make_double2(0.0, 0.0);
    __syncthreads();
    unsigned passed = 0;
    double2* bufs[2] = {ua, ub};
    const double2* in = rho;
    for (int step = 0; step < nsteps; ++step) {
        for (int st = 1; st <= order; ++st) {
            const double alpha = dt / static_cast<double>(order - st + 1);
            double2* out = (st == order) ? rho : bufs[(st - 1) & 1];
            if (!watcher) {
                double2 acc[E];
                if (on)
#pragma unroll
                    for (int k = 0; k < E; ++k) X[tid + T * k] = x[k];
                __syncthreads();
                if (on)
#pragma unroll
                    for (int k = 0; k < E; ++k) {
                        // -g X - i [H, X]
                        const int e = tid + T * k;
                        const double dE = sE[e >> LOGD] - sE[c];
                        double2 h = make_double2(dE * x[k].x, dE * x[k].y);
                        slab_flips<LOGD, false>(X, e, sH, h);
                        acc[k] = make_double2(fma(-g, x[k].x, h.y), fma(-g, x[k].y, -h.x));
                    }
                for (int j = 0; j < a.J; ++j) {
                    const double* V = sV + j * D;
                    const double* W = sW + j * LOGD;
                    const double xi = __ldg(a.xi + j), ka = __ldg(a.counter + j);
                    const int m0 = __ldg(a.bath_off + j), m1 = __ldg(a.bath_off + j + 1);
                    double2 t[E], s[E], d[E], sum[E];
                    if (on) {
#pragma unroll
                        for (int k = 0; k < E; ++k) s[k] = d[k] = make_double2(0.0, 0.0);
#pragma unroll 2
                        for (int m = m0; m < m1; ++m) {
                            const int up = __ldg(edges + m), dn = __ldg(edges + a.M + m);
                            if (up < a.H)
#pragma unroll
                                for (int k = 0; k < E; ++k) {
                                    const double2 v = __ldcg(in + static_cast<long long>(up) * D2 + tid + T * k);
                                    s[k].x += v.x;
                                    s[k].y += v.y;
                                }
                            if (dn < a.H) {
                                const double wd = __ldg(a.acoef + n * a.M + m);
#pragma unroll
                                for (int k = 0; k < E; ++k) {
                                    const double2 v = __ldcg(in + static_cast<long long>(dn) * D2 + tid + T * k);
                                    s[k].x = fma(wd, v.x, s[k].x);
                                    s[k].y = fma(wd, v.y, s[k].y);
                                    if (m == m0) {
                                        const double b = __ldg(a.bcoef + n * a.J + j);
                                        d[k] = make_double2(b * v.x, b * v.y);
                                    }
                                }
                            }
                        }
#pragma unroll
                        for (int k = 0; k < E; ++k) {
                            const int e = tid + T * k;
                            const double dv = V[e >> LOGD] - V[c], sv = V[e >> LOGD] + V[c];
                            double2 comm = make_double2(dv * x[k].x, dv * x[k].y);
                            slab_flips<LOGD, false>(X, e, W, comm);
                            t[k] = make_double2(fma(-xi, comm.x, s[k].y), fma(-xi, comm.y, -s[k].x));
                            d[k] = make_double2(fma(ka, comm.y, -d[k].x), fma(-ka, comm.x, -d[k].y));
                            sum[k] = make_double2(fma(dv, t[k].x, sv * d[k].x), fma(dv, t[k].y, sv * d[k].y));
                        }
                    }
                    if (j > 0) __syncthreads();  // the flips of the bath before are done
                    if (on)
#pragma unroll
                        for (int k = 0; k < E; ++k) {
                            sT[tid + T * k] = t[k];
                            sA[tid + T * k] = d[k];
                        }
                    __syncthreads();
                    if (on)
#pragma unroll
                        for (int k = 0; k < E; ++k) {
                            slab_flips<LOGD, false>(sT, tid + T * k, W, sum[k]);
                            slab_flips<LOGD, true>(sA, tid + T * k, W, sum[k]);
                            acc[k].x += sum[k].x;
                            acc[k].y += sum[k].y;
                        }
                }
                if (on)
#pragma unroll
                    for (int k = 0; k < E; ++k) {
                        x[k] = make_double2(fma(alpha, acc[k].x, base[k].x), fma(alpha, acc[k].y, base[k].y));
                        __stcg(out + n * D2 + tid + T * k, x[k]);
                        if (st == order) base[k] = x[k];
                    }
            }
            in = out;
            const bool last = step + 1 == nsteps && st == order;
            if (last && !watcher) {
                if (watch) grid_arrive(gcount);  // the watcher waits for the last state; nobody else does
                break;
            }
            ++passed;
            if (!grid_barrier(gcount, passed, w)) {
                run_gave_up(error_flag, w, nsteps, step, st == order);
                return;
            }
            if (watcher && st == order) {
                if (trace)
                    for (int i = tid; i < D2; i += T) trace[static_cast<long long>(step) * D2 + i] = __ldcg(rho + i);
                if (obs && tid < 32)
                    warp_observables<LOGD>(
                        a.hdiag, a.hflip, [&](int r0, int c0) { return __ldcg(rho + (r0 << LOGD) + c0); }, obs + 3 * step);
            }
        }
    }
    grid_reset(gcount, watch, watcher, static_cast<unsigned>(nsteps * order));
}

template <int LOGD>
size_t flip_run_smem(int J)
{
    constexpr size_t D = FlipRunShape<LOGD>::D;
    return 3 * D * D * sizeof(double2) + sizeof(double) * (D + LOGD + J * (D + LOGD));
}

constexpr size_t kFlipRunSmem = 227 * 1024;
constexpr long long kFlipRunMost = 3000;  // ADOs

template <int LOGD>
bool prepare_flip_run_t(const FlipArgs& a, int sms)
{
    const size_t smem = flip_run_smem<LOGD>(a.J);
    if (smem > kFlipRunSmem) return false;
    static std::atomic<bool> raised[64];
    int dev = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    if (!raised[dev].load()) {
        if (cudaFuncSetAttribute(flip_run_kernel<LOGD>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(kFlipRunSmem)) != cudaSuccess)
            return false;
        raised[dev].store(true);
    }
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, flip_run_kernel<LOGD>, FlipRunShape<LOGD>::T, smem) !=
        cudaSuccess)
        return false;
    return a.H <= static_cast<long long>(per_sm) * sms - 1;  // and the watcher
}

template <int LOGD>
int launch_flip_run_t(const FlipArgs& a, double2* rho, double2* ua, double2* ub, double dt, int order, int nsteps,
                      unsigned* gcount, int* error_flag, StepWait w, double2* trace, double* obs, cudaStream_t s)
{
    FlipArgs args = a;
    void* params[] = {&args, &rho, &ua, &ub, &dt, &order, &nsteps, &gcount, &error_flag, &w, &trace, &obs};
    return cudaLaunchCooperativeKernel(reinterpret_cast<void*>(flip_run_kernel<LOGD>),
                                       dim3(static_cast<unsigned>(a.H + (trace || obs ? 1 : 0))),
                                       dim3(FlipRunShape<LOGD>::T), params, flip_run_smem<LOGD>(a.J), s) == cudaSuccess
               ? 1
               : -1;
}

}  // namespace

#define HX_FLIP_SWITCH(CALL, NONE) \
    switch (a.logd) {              \
    case 1: return CALL(1);        \
    case 2: return CALL(2);        \
    case 3: return CALL(3);        \
    case 4: return CALL(4);        \
    case 5: return CALL(5);        \
    default: return NONE;          \
    }

// Whole steps while every ADO has a CTA of its own (at d = 32 an SM of its own).  us per step, two passes against a
// run, one bath: d = 4, 20 ADOs 38 and 14; d = 16, 120 ADOs 42 and 17, 560 50 and 26; d = 32, 35 ADOs 50 and 27, 120
// 55 and 27; five baths, d = 32, 66 ADOs 95 and 70.  Thousands of arrivals at every barrier take longer than the two
// launches: d = 4, 1771 ADOs 42 and 26, 3654 42 and 47, so the line lies at 3000 (d <= 4 alone has room for more).
// At d = 64 the two passes with four rows per thread were ahead
// of a CTA per ADO at any count (per four steps 275 and 517 at 20 ADOs, 502 and 626 at 126).
bool prepare_flip_run(const FlipArgs& a, int sms)
{
    if (a.H > kFlipRunMost) return false;
#define HX_CALL(L) prepare_flip_run_t<L>(a, sms)
    HX_FLIP_SWITCH(HX_CALL, false)
#undef HX_CALL
}

int launch_flip_run(const FlipArgs& a, double2* rho, double2* ua, double2* ub, double dt, int order, int nsteps,
                    unsigned* gcount, int* error_flag, StepWait w, double2* trace, double* obs, cudaStream_t s)
{
#define HX_CALL(L) launch_flip_run_t<L>(a, rho, ua, ub, dt, order, nsteps, gcount, error_flag, w, trace, obs, s)
    HX_FLIP_SWITCH(HX_CALL, -1)
#undef HX_CALL
}

void launch_flip_stage(const FlipArgs& a, const double2* u, double2* B, const double2* rho, double2* out,
                       double alpha, int base_kind, cudaStream_t s)
{
    // four rows per thread once that still fills the GPU
    if (a.logd >= 2 && (a.H << (2 * a.logd)) >= 4 * 148 * 512) launch_flip_t<2>(a, u, B, rho, out, alpha, base_kind, s);
    else launch_flip_t<0>(a, u, B, rho, out, alpha, base_kind, s);
}

}  // namespace hx
