// Stage kernels for general sparse Hermitian operators (H and every V_j in
// compressed rows), any Hilbert dimension up to 4096, double precision.
//
// The reference validates System::from_sparse but executes only its compiled
// model (src/helix.cpp:166-258,335-347); its right-hand side
// (getdRhoSparse, src/liouville.cu:778-860) applies V through SpMM and
// transposes.  Here the operator products are gathers along CSR rows: for a
// Hermitian operator A,
//   (A X)_rc = sum_{p in row r} A_p X_{col p, c}
//   (X A)_rc = sum_k X_rk A_kc = sum_{p in row c} X_{r, col p} conj(A_p)
// so both sides of a commutator use the rows of A.  As in the flip path
// (hx_flip.cu) each stage runs in two passes:
//   csr_comm_kernel:    B_{j,n} = [V_j, u_n] and A_{j,n} = {V_j, u_n} for
//                       every bath j and ADO n (B for all (j, n), then A)
//   csr_combine_kernel: out_n = base_n + alpha * ( -i[H,u_n] - g_n u_n
//                         - i sum_{m up} B_{j(m), n+e_m}
//                         - i sum_{m down} a_{n,m} B_{j(m), n-e_m}
//                         - sum_j b_{n,j} A_{j, n-e_j0}
//                         + sum_j ((-Xi_j - i kappa_j) V_j B_{j,n} + (Xi_j - i kappa_j) B_{j,n} V_j) )
// the last line being -Xi [V, B] - i kappa {V, B}.  One thread per element;
// the gathered rows and columns of a slab are read through L1/L2.
// Bound by the latency of index, value and gather one after the other, so two
// entries are asked for at once, in the registers that leave six CTAs per SM
// (first pass) and five (second).  us per step, one entry at a time and five
// CTAs, two entries and four, and now: d = 128, three baths, 13 ADOs 263, 303 and
// 252, 28 ADOs 477, 472 and 425; d = 256, 3 ADOs 205, 224 and 194, 10 ADOs 652, 673
// and 586; d = 512, 10 ADOs 2536, 2492 and 2300.  Six CTAs for both spill (d = 128, 6
// ADOs 84 -> 93).  Four entries, or four rows of a column per thread, take the
// registers of the warps that hide the latency.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "hx_internal.h"

namespace hx {

namespace {

__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// a * conj(b)
__device__ __forceinline__ double2 cmulc(double2 a, double2 b)
{
    return make_double2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}

// (A X)_rc and (X A)_rc of operator k for slab X (row-major, d = 2^logd), U entries at a time.
struct Sides {
    double2 left, right;
};

template <int U>
__device__ __forceinline__ Sides sides(const CsrArgs& a, int k, const double2* __restrict__ X, int r, int c)
{
    const int D = 1 << a.logd;
    const int32_t* ptr = a.ptr + static_cast<long long>(k) * (D + 1);
    double2 L = make_double2(0.0, 0.0), R = make_double2(0.0, 0.0);
    const int r1 = __ldg(ptr + r + 1), c1 = __ldg(ptr + c + 1);
#pragma unroll U
    for (int p = __ldg(ptr + r); p < r1; ++p) {
        const double2 v = __ldg(a.val + p);
        const double2 x = __ldg(X + (static_cast<long long>(__ldg(a.col + p)) << a.logd) + c);
        const double2 t = cmul(v, x);
        L.x += t.x;
        L.y += t.y;
    }
#pragma unroll U
    for (int p = __ldg(ptr + c); p < c1; ++p) {
        const double2 v = __ldg(a.val + p);
        const double2 x = __ldg(X + (static_cast<long long>(r) << a.logd) + __ldg(a.col + p));
        const double2 t = cmulc(x, v);
        R.x += t.x;
        R.y += t.y;
    }
    return Sides{L, R};
}

template <int U>
__global__ void __launch_bounds__(256, 6) csr_comm_kernel(CsrArgs a, const double2* __restrict__ u, double2* __restrict__ B)
{
    const int D = 1 << a.logd;
    const long long D2 = static_cast<long long>(D) * D;
    const long long HD2 = a.H * D2;
    const long long total = static_cast<long long>(a.J) * HD2;
    for (long long ne = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; ne < HD2;
         ne += static_cast<long long>(gridDim.x) * blockDim.x) {
        const long long n = ne >> (2 * a.logd);
        const long long e = ne & (D2 - 1);
        const int r = static_cast<int>(e >> a.logd), c = static_cast<int>(e & (D - 1));
        for (int j = 0; j < a.J; ++j) {
            const Sides s = sides<U>(a, 1 + j, u + n * D2, r, c);
            const long long idx = static_cast<long long>(j) * HD2 + ne;
            B[idx] = make_double2(s.left.x - s.right.x, s.left.y - s.right.y);
            B[total + idx] = make_double2(s.left.x + s.right.x, s.left.y + s.right.y);
        }
    }
}

template <int U>
__global__ void __launch_bounds__(256, U == 1 ? 4 : 5)
    csr_combine_kernel(CsrArgs a, const double2* __restrict__ u, const double2* __restrict__ B, const double2* rho,
                       double2* out, double alpha, int base_kind)
{
    const int D = 1 << a.logd;
    const long long D2 = static_cast<long long>(D) * D;
    const long long total = a.H * D2;
    const long long HD2 = a.H * D2;
    for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
         idx += static_cast<long long>(gridDim.x) * blockDim.x) {
        const long long n = idx >> (2 * a.logd);
        const long long e = idx & (D2 - 1);
        const int r = static_cast<int>(e >> a.logd), c = static_cast<int>(e & (D - 1));
        const double2* un = u + n * D2;
        const double2 x = un[e];
        // -g u - i [H, u]
        const double g = a.gsum[n];
        const Sides h = sides<U>(a, 0, un, r, c);
        const double cr = h.left.x - h.right.x, ci = h.left.y - h.right.y;
        double re = -g * x.x + ci;
        double im = -g * x.y - cr;
        const int32_t* edges = a.edges + n * 2 * a.M;
        for (int j = 0; j < a.J; ++j) {
            const double2* Bj = B + static_cast<long long>(j) * HD2;
            // up and down neighbours: -i B_up, -i a B_down
            double sr = 0.0, si = 0.0;
            for (int m = a.bath_off[j]; m < a.bath_off[j + 1]; ++m) {
                const int up = edges[m];
                if (up < a.H) {
                    const double2 y = __ldg(Bj + static_cast<long long>(up) * D2 + e);
                    sr += y.x;
                    si += y.y;
                }
                const int dn = edges[a.M + m];
                if (dn < a.H) {
                    const double w = a.acoef[n * a.M + m];
                    const double2 y = __ldg(Bj + static_cast<long long>(dn) * D2 + e);
                    sr += w * y.x;
                    si += w * y.y;
                }
            }
            re += si;
            im -= sr;
            // theta2: -b {V_j, u_{n-e_j0}} = -b A_{j, n-e_j0}
            const int dn0 = edges[a.M + a.bath_off[j]];
            if (dn0 < a.H) {
                const double b = a.bcoef[n * a.J + j];
                const double2 y = __ldg(Bj + static_cast<long long>(a.J) * HD2 + static_cast<long long>(dn0) * D2 + e);
                re -= b * y.x;
                im -= b * y.y;
            }
            // -Xi [V, B_n] - i kappa {V, B_n} = (-Xi - i kappa) V B + (Xi - i kappa) B V
            const double xi = a.xi[j], ka = a.counter[j];
            const Sides s = sides<U>(a, 1 + j, Bj + n * D2, r, c);
            re += -xi * s.left.x + ka * s.left.y + xi * s.right.x + ka * s.right.y;
            im += -xi * s.left.y - ka * s.left.x + xi * s.right.y - ka * s.right.x;
        }
        double2 base;
        if (base_kind == kBaseSelf) base = x;
        else if (base_kind == kBaseRho) base = rho[idx];
        else base = make_double2(0.0, 0.0);
        out[idx] = make_double2(base.x + alpha * re, base.y + alpha * im);
    }
}

// out[0] = Re Tr(H rho_0) = Re sum_r sum_{p in row r} conj(H_p) rho0_{r, col p} (H is Hermitian), so the
// reads run along rows of rho_0; out[1..2] = Tr rho_0.  A warp per row, the blocks' sums in scratch[3 b ..],
// added pairwise in a fixed order by the block that finishes last (*ticket counts them and goes back to zero; one
// after the other they are rounded at the size of the total all the way): one block over columns of rho_0 took 55 us
// for a dense H of d = 256, this takes 10.
constexpr int kObsBlocks = 64;

__global__ void __launch_bounds__(256)
    csr_observables_kernel(const double2* __restrict__ rho0, int logd, const int32_t* __restrict__ ptr,
                           const int32_t* __restrict__ col, const double2* __restrict__ val, double* scratch,
                           unsigned* ticket, double* out)
{
    const int D = 1 << logd, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double s[3] = {0.0, 0.0, 0.0};  // per lane: energy; lane 0: trace
    for (int r = blockIdx.x * 8 + warp; r < D; r += gridDim.x * 8) {
        const double2* row = rho0 + (static_cast<long long>(r) << logd);
        const int p1 = __ldg(ptr + r + 1);
#pragma unroll 4
        for (int p = __ldg(ptr + r) + lane; p < p1; p += 32) {
            const double2 y = row[__ldg(col + p)], v = __ldg(val + p);
            s[0] += v.x * y.x + v.y * y.y;
        }
        if (lane == 0) {
            s[1] += row[r].x;
            s[2] += row[r].y;
        }
    }
    __shared__ double red[8][3];
    for (int off = 16; off > 0; off >>= 1) s[0] += __shfl_down_sync(0xffffffffu, s[0], off);
    if (lane == 0)
        for (int q = 0; q < 3; ++q) red[warp][q] = s[q];
    __syncthreads();
    __shared__ bool last;
    if (threadIdx.x == 0) {
        for (int q = 0; q < 3; ++q) {
            scratch[3 * blockIdx.x + q] = ((red[0][q] + red[1][q]) + (red[2][q] + red[3][q])) +
                                          ((red[4][q] + red[5][q]) + (red[6][q] + red[7][q]));
        }
        __threadfence();
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last || warp >= 3) return;
    __threadfence();
    double t = 0.0;
#pragma unroll
    for (int b = lane; b < kObsBlocks; b += 32)
        if (b < static_cast<int>(gridDim.x)) t += __ldcg(scratch + 3 * b + warp);
    for (int off = 16; off > 0; off >>= 1) t += __shfl_down_sync(0xffffffffu, t, off);
    if (lane == 0) out[warp] = t;
    if (threadIdx.x == 0) *ticket = 0u;
}

unsigned grid_for(long long n)
{
    const long long g = (n + 255) / 256;
    return static_cast<unsigned>(g < 148ll * 64 ? g : 148ll * 64);
}

}  // namespace

void launch_csr_stage(const CsrArgs& a, const double2* u, double2* B, const double2* rho, double2* out, double alpha,
                      int base_kind, cudaStream_t s)
{
    // the rows of small matrices are too short for two entries side by side (d = 4, two baths, 4845 ADOs 83 us a step
    // with two, 67 with one)
    const unsigned grid = grid_for(a.H << (2 * a.logd));
    if (a.logd >= 6) {
        csr_comm_kernel<2><<<grid, 256, 0, s>>>(a, u, B);
        csr_combine_kernel<2><<<grid, 256, 0, s>>>(a, u, B, rho, out, alpha, base_kind);
    } else {
        csr_comm_kernel<1><<<grid, 256, 0, s>>>(a, u, B);
        csr_combine_kernel<1><<<grid, 256, 0, s>>>(a, u, B, rho, out, alpha, base_kind);
    }
}

void launch_observables_csr(const double2* rho0, int logd, const int32_t* ptr, const int32_t* col,
                            const double2* val, double* scratch, double* out, cudaStream_t s)
{
    const int blocks = std::min(kObsBlocks, std::max(1, (1 << logd) / 8));
    csr_observables_kernel<<<blocks, 256, 0, s>>>(rho0, logd, ptr, col, val, scratch,
                                                  reinterpret_cast<unsigned*>(scratch + 3 * kObsBlocks), out);
}

size_t observables_csr_scratch() { return 3 * kObsBlocks + 1; }

}  // namespace hx
