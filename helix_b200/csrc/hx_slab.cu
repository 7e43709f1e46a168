// Stage kernels for sparse Hermitian operators (compressed rows) at d <= 64,
// where a slab fits in shared memory.
//
// Same mathematics as the two-pass path (hx_csr.cu; reference
// getdRhoSparse, src/liouville.cu:778-860), arranged so that no commutator of
// an ADO leaves its CTA.  With C_j = [V_j, u_n], S_j the sum of the up
// neighbours and of the down neighbours times a, and u_d the Drude mode's down
// neighbour, everything a bath contributes is
//   V_j P_j + Q_j V_j,   P_j = -i S_j - b_j u_d - (xi_j + i kappa_j) C_j,
//                        Q_j = +i S_j - b_j u_d + (xi_j - i kappa_j) C_j,
// and S_j, u_d are sums of neighbours of u, not of their commutators: 2 (J + 1)
// + 2 J sparse products per ADO inside one CTA instead of [V_j, u_n] and
// {V_j, u_n} of every bath and ADO through memory and back.
//
//  * left products (A X)_rc run with the columns over the lanes, right
//    products (X A)_rc = sum_p X_{r, col p} conj(A_p) with the rows over the
//    lanes: the operator's entries are the same for a whole warp in both, and
//    the slab (element (r, c) at r d + (c ^ (r & 7))) is read free of bank
//    conflicts along rows and along columns;
//  * the two kinds of accumulators meet once per ADO, through shared memory;
//  * the operators' entries stay in shared memory.
//
// slab_kernel runs one stage per launch, after a gather pass
// (slab_gather_kernel) has summed the neighbours.
//
// Bound by shared memory (16 bytes per element and entry) and, for few ADOs,
// by one CTA's time per ADO.  us per step, two passes against this: d = 64, six
// baths, 91 ADOs 660 and 450; d = 32, four baths, 165 ADOs 285 and 183.

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>

#include "hx_internal.h"

namespace hx {

namespace {

template <int LOGD> struct SlabShape {
    static constexpr int D = 1 << LOGD;
    static constexpr int T = LOGD >= 5 ? 512 : (D * D < 32 ? 32 : D * D);  // threads
    static constexpr int NC = D >= 64 ? D / 32 : 1;                         // elements of a thread along the lanes
    static constexpr int LANES = D >= 32 ? 32 : D;
    static constexpr int GROUPS = T >= D * D ? D : T / LANES;               // lines of the matrix side by side
    static constexpr int NR = D / GROUPS;                                   // lines per thread
    static constexpr int E = NR * NC;
};

template <int LOGD>
__device__ __forceinline__ int slab_at(int r, int c)
{
    return (r << LOGD) + (c ^ (r & (LOGD >= 3 ? 7 : 0)));
}

// Shared-memory view of the operators: 0 = H, 1 + j = V_j.
struct SlabOps {
    const double2* val;
    const int* col;
    const int* ptr;  // [(J + 1)(D + 1)]
};

// y[k] += f sum_p A_p X[col p][c0 + 32 k] over row r (left product), or
// y[k] += f sum_p X[r0 + 32 k][col p] conj(A_p) over row c (right product).
template <int LOGD, bool RIGHT>
__device__ __forceinline__ void slab_product(const SlabOps& o, int op, const double2* X, int line, int at, double2* y)
{
    constexpr int D = 1 << LOGD, NC = SlabShape<LOGD>::NC;
    const int p1 = o.ptr[op * (D + 1) + line + 1];
#pragma unroll 4
    for (int p = o.ptr[op * (D + 1) + line]; p < p1; ++p) {
        const double2 a = o.val[p];
        const int q = o.col[p];
#pragma unroll
        for (int k = 0; k < NC; ++k) {
            const double2 x = X[RIGHT ? slab_at<LOGD>(at + 32 * k, q) : slab_at<LOGD>(q, at + 32 * k)];
            const double im = RIGHT ? -a.y : a.y;
            y[k].x = fma(a.x, x.x, fma(-im, x.y, y[k].x));
            y[k].y = fma(a.x, x.y, fma(im, x.x, y[k].y));
        }
    }
}

// z[k] += the product, summed by itself first: the sum over the baths is rounded once per bath, not per entry.
// Error of a right-hand side (relative, random states): d = 32, five baths 3.2e-16 entry by entry, 1.4e-16 so (the
// two passes 1.5e-16); d = 64, two baths 2.1e-16 and 1.0e-16.  It costs 5% of a step with six baths (430 us, 451).
template <int LOGD, bool RIGHT>
__device__ __forceinline__ void slab_add(const SlabOps& o, int op, const double2* X, int line, int at, double2* z)
{
    constexpr int NC = SlabShape<LOGD>::NC;
    double2 y[NC];
#pragma unroll
    for (int k = 0; k < NC; ++k) y[k] = make_double2(0.0, 0.0);
    slab_product<LOGD, RIGHT>(o, op, X, line, at, y);
#pragma unroll
    for (int k = 0; k < NC; ++k) {
        z[k].x += y[k].x;
        z[k].y += y[k].y;
    }
}

// One ADO: out_n = base_n + alpha L(u)_n, S_j and b_j u_d from the gather buffer.
template <int LOGD>
__device__ __forceinline__ void slab_ado(const CsrArgs& a, const SlabOps& o, double2* X, double2* W, long long n,
                                         const double2* u, const double2* gather, const double2* base, double2* out,
                                         double alpha, int base_kind)
{
    using S = SlabShape<LOGD>;
    constexpr int D = S::D, NC = S::NC, NR = S::NR, E = S::E;
    constexpr long long D2 = static_cast<long long>(D) * D;
    const int tid = threadIdx.x;
    const bool on = tid < D * D;
    const int lane = tid & (S::LANES - 1), line = tid / S::LANES;  // element (line + GROUPS i, lane + 32 k)
    double2 L[E], R[E], y[E];
    if (on)
#pragma unroll
        for (int i = 0; i < NR; ++i)
#pragma unroll
            for (int k = 0; k < NC; ++k)
                X[slab_at<LOGD>(line + S::GROUPS * i, lane + 32 * k)] =
                    __ldcg(u + n * D2 + ((line + S::GROUPS * i) << LOGD) + lane + 32 * k);
    __syncthreads();
    const double g = a.gsum[n];
    if (on)
#pragma unroll
        for (int i = 0; i < NR; ++i) {
            const int r = line + S::GROUPS * i;
            double2 l[NC], q[NC];
#pragma unroll
            for (int k = 0; k < NC; ++k) l[k] = q[k] = make_double2(0.0, 0.0);
            slab_product<LOGD, false>(o, 0, X, r, lane, l);
            slab_product<LOGD, true>(o, 0, X, r, lane, q);
#pragma unroll
            for (int k = 0; k < NC; ++k) {
                // -i H X - g X, + i X H
                const double2 x = X[slab_at<LOGD>(r, lane + 32 * k)];
                L[i * NC + k] = make_double2(fma(-g, x.x, l[k].y), fma(-g, x.y, -l[k].x));
                R[i * NC + k] = make_double2(-q[k].y, q[k].x);
            }
        }
    const long long HD2 = a.H * D2;
    for (int j = 0; j < a.J; ++j) {
        // C_j: left part in registers, right part through W
        if (on)
#pragma unroll
            for (int i = 0; i < NR; ++i) {
                const int r = line + S::GROUPS * i;
                double2 l[NC], q[NC];
#pragma unroll
                for (int k = 0; k < NC; ++k) l[k] = q[k] = make_double2(0.0, 0.0);
                slab_product<LOGD, false>(o, 1 + j, X, r, lane, l);
                slab_product<LOGD, true>(o, 1 + j, X, r, lane, q);
#pragma unroll
                for (int k = 0; k < NC; ++k) {
                    y[i * NC + k] = l[k];
                    W[slab_at<LOGD>(lane + 32 * k, r)] = q[k];
                }
            }
        __syncthreads();
        // P_j into W, Q_j kept
        const double xi = a.xi[j], ka = a.counter[j];
        if (on)
#pragma unroll
            for (int i = 0; i < NR; ++i)
#pragma unroll
                for (int k = 0; k < NC; ++k) {
                    const int r = line + S::GROUPS * i, c = lane + 32 * k, e = (r << LOGD) + c;
                    const double2 s = __ldcg(gather + j * HD2 + n * D2 + e), d = __ldcg(gather + (a.J + j) * HD2 + n * D2 + e);
                    const double2 q = W[slab_at<LOGD>(r, c)], l = y[i * NC + k];
                    const double cx = l.x - q.x, cy = l.y - q.y;
                    // P = -i S - b u_d - (xi + i kappa) C, Q = i S - b u_d + (xi - i kappa) C
                    W[slab_at<LOGD>(r, c)] = make_double2(s.y - d.x - xi * cx + ka * cy, -s.x - d.y - xi * cy - ka * cx);
                    y[i * NC + k] = make_double2(-s.y - d.x + xi * cx + ka * cy, s.x - d.y + xi * cy - ka * cx);
                }
        __syncthreads();
        if (on)
#pragma unroll
            for (int i = 0; i < NR; ++i) slab_add<LOGD, false>(o, 1 + j, W, line + S::GROUPS * i, lane, L + i * NC);
        __syncthreads();
        if (on)
#pragma unroll
            for (int i = 0; i < NR; ++i)
#pragma unroll
                for (int k = 0; k < NC; ++k) W[slab_at<LOGD>(line + S::GROUPS * i, lane + 32 * k)] = y[i * NC + k];
        __syncthreads();
        if (on)
#pragma unroll
            for (int i = 0; i < NR; ++i) slab_add<LOGD, true>(o, 1 + j, W, line + S::GROUPS * i, lane, R + i * NC);
        __syncthreads();
    }
    // right products meet the left ones
    if (on)
#pragma unroll
        for (int i = 0; i < NR; ++i)
#pragma unroll
            for (int k = 0; k < NC; ++k) W[slab_at<LOGD>(lane + 32 * k, line + S::GROUPS * i)] = R[i * NC + k];
    __syncthreads();
    if (on)
#pragma unroll
        for (int i = 0; i < NR; ++i)
#pragma unroll
            for (int k = 0; k < NC; ++k) {
                const int r = line + S::GROUPS * i, c = lane + 32 * k;
                const long long e = n * D2 + (r << LOGD) + c;
                const double2 q = W[slab_at<LOGD>(r, c)], l = L[i * NC + k];
                double2 v = make_double2(0.0, 0.0);
                if (base_kind == kBaseSelf) v = X[slab_at<LOGD>(r, c)];
                else if (base_kind == kBaseRho) v = __ldcg(base + e);
                __stcg(out + e, make_double2(fma(alpha, l.x + q.x, v.x), fma(alpha, l.y + q.y, v.y)));
            }
}

// The operators into shared memory; returns what follows them.
template <int LOGD>
__device__ __forceinline__ SlabOps slab_ops(const CsrArgs& a, int nnz, unsigned char* smem)
{
    constexpr int D = 1 << LOGD;
    double2* val = reinterpret_cast<double2*>(smem);
    int* col = reinterpret_cast<int*>(val + nnz);
    int* ptr = col + nnz;
    for (int i = threadIdx.x; i < nnz; i += blockDim.x) {
        val[i] = a.val[i];
        col[i] = a.col[i];
    }
    for (int i = threadIdx.x; i < (a.J + 1) * (D + 1); i += blockDim.x) ptr[i] = a.ptr[i];
    return SlabOps{val, col, ptr};
}

template <int LOGD>
__global__ void __launch_bounds__(SlabShape<LOGD>::T)
    slab_kernel(CsrArgs a, int nnz, const double2* u, const double2* gather, const double2* rho, double2* out,
                double alpha, int base_kind)
{
    constexpr int D2 = 1 << (2 * LOGD);
    extern __shared__ __align__(16) unsigned char smem[];
    double2* X = reinterpret_cast<double2*>(smem);
    const SlabOps o = slab_ops<LOGD>(a, nnz, smem + 2 * D2 * sizeof(double2));
    slab_ado<LOGD>(a, o, X, X + D2, blockIdx.x, u, gather, rho, out, alpha, base_kind);
}

// S_j of every ADO and bath into G[j][n], b_j u_d into G[J + j][n].
__global__ void __launch_bounds__(256) slab_gather_kernel(CsrArgs a, const double2* __restrict__ u, double2* __restrict__ G)
{
    const long long D2 = 1ll << (2 * a.logd), HD2 = a.H * D2;
    const long long q = blockIdx.x * 256ll + threadIdx.x;
    if (q >= HD2) return;
    const long long n = q >> (2 * a.logd), e = q & (D2 - 1);
    const int j = blockIdx.y;
    const int32_t* edges = a.edges + n * 2 * a.M;
    const int m0 = __ldg(a.bath_off + j), m1 = __ldg(a.bath_off + j + 1);
    double2 s = make_double2(0.0, 0.0), d = s;
#pragma unroll 4
    for (int m = m0; m < m1; ++m) {
        const int up = __ldg(edges + m), dn = __ldg(edges + a.M + m);
        if (up < a.H) {
            const double2 v = __ldg(u + up * D2 + e);
            s.x += v.x;
            s.y += v.y;
        }
        if (dn < a.H) {
            const double2 v = __ldg(u + dn * D2 + e);
            const double w = __ldg(a.acoef + n * a.M + m);
            s.x = fma(w, v.x, s.x);
            s.y = fma(w, v.y, s.y);
            if (m == m0) {
                const double b = __ldg(a.bcoef + n * a.J + j);
                d = make_double2(b * v.x, b * v.y);
            }
        }
    }
    G[j * HD2 + q] = s;
    G[(a.J + j) * HD2 + q] = d;
}

template <int LOGD>
size_t slab_smem(int J, int nnz)
{
    constexpr size_t D = size_t(1) << LOGD;
    return 2 * D * D * sizeof(double2) + static_cast<size_t>(nnz) * (sizeof(double2) + sizeof(int)) +
           sizeof(int) * (J + 1) * (D + 1);
}

constexpr size_t kSlabSmem = 227 * 1024;

template <int LOGD>
bool prepare_slab_t(int J, int nnz)
{
    if (slab_smem<LOGD>(J, nnz) > kSlabSmem) return false;
    static std::atomic<bool> raised[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    if (raised[dev].load()) return true;
    if (cudaFuncSetAttribute(slab_kernel<LOGD>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(kSlabSmem)) != cudaSuccess)
        return false;
    raised[dev].store(true);
    return true;
}

}  // namespace

#define HX_SLAB_SWITCH(CALL) \
    switch (a.logd) {        \
    case 1: return CALL(1);  \
    case 2: return CALL(2);  \
    case 3: return CALL(3);  \
    case 4: return CALL(4);  \
    case 5: return CALL(5);  \
    case 6: return CALL(6);  \
    default: return 0;       \
    }

// At d = 64 the two-pass kernels, which spread every ADO over the GPU, stay ahead while most SMs would have no
// slab, whatever the number of baths: us per step, two passes against a slab per CTA, 35 ADOs of one bath 91 and 123, of
// four 189 and 271; 45 ADOs of one 124 and 122, of four 280 and 275; 55 of one 148 and 130, of three 287 and 229; 91 of
// six 629 and 453; at d = 32 a slab per CTA is ahead from 2 ADOs (per four steps 299 and 297) on, 20 ADOs 531 and 436.
// At d = 2 and 4 a CTA per slab of 4 or 16 elements leaves most of its threads idle, and with thousands of them the
// two passes are ahead: d = 2, 1330 ADOs 42 and 42, 3654 42 and 48, 52360 72 and 173; d = 4, 1330 50 and 46, 2300 50
// and 54, 10660 82 and 107, two baths 1820 66 and 60, 3003 67 and 73.  At d = 8 the slabs stay ahead (10660 199 and
// 164).
int prepare_slab(const CsrArgs& a, int nnz)
{
    if (a.logd == 6 && a.H < 45) return 0;
    if (a.logd <= 2 && a.H > (a.logd == 1 ? 1024 : 2000)) return 0;
#define HX_CALL(L) (prepare_slab_t<L>(a.J, nnz) ? 1 : 0)
    HX_SLAB_SWITCH(HX_CALL)
#undef HX_CALL
}

int launch_slab_stage(const CsrArgs& a, int nnz, const double2* u, double2* G, const double2* rho, double2* out,
                      double alpha, int base_kind, cudaStream_t s)
{
    const long long HD2 = a.H << (2 * a.logd);
    slab_gather_kernel<<<dim3(static_cast<unsigned>((HD2 + 255) / 256), static_cast<unsigned>(a.J)), 256, 0, s>>>(a, u, G);
#define HX_CALL(L)                                                                                                     \
    (slab_kernel<L><<<static_cast<unsigned>(a.H), SlabShape<L>::T, slab_smem<L>(a.J, nnz), s>>>(a, nnz, u, G, rho, out, \
                                                                                                alpha, base_kind),     \
     2)
    HX_SLAB_SWITCH(HX_CALL)
#undef HX_CALL
}

}  // namespace hx
