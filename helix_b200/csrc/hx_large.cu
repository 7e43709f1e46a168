// Stage kernels for Hilbert dimension 128 <= d <= 1024 with diagonal couplings,
// in double precision (the plain propagator) or in single precision with
// complex64 storage (the mixed-precision propagator, whose tier-0 ADO runs in
// double precision in ado0_kernel).
//
// Mathematics as in fused_kernel (hx_fused.cu): out_n = base_n + alpha L(u)_n
// with L the reference right-hand side (getdRhoSparse, src/liouville.cu:749-869)
// for diagonal couplings V_j and H = diag(E) + sum_i h_i sigma_x(i).  A slab of
// d = 256 is 1 MB in double precision, too large for shared memory, so:
//
//  * one CTA computes one 64 x 64 tile of one ADO, held in shared memory
//    (tile_kernel; with packed slabs the tiles on and above the diagonal);
//    consecutive CTAs take the tiles of one ADO, so the rest of its slab is in
//    L2 while they run;
//  * flips of the six low bits of row and column read shared memory or
//    registers, flips of the higher bits another tile through L2;
//  * neighbour terms are elementwise (diagonal V) and read through L2; the up
//    term of tier L-1 (neighbours in the top tier) comes from
//    large_upterm_kernel, which walks the top tier tile by tile.
//
// With a dense H (HX_FLAG_DENSE_H, complex64 path) the diagonal table keeps
// the real diagonal of H and the commutator with the rest of H (no flip
// terms) comes from the product Y_n = X_n H_off of every ADO, computed before
// the stage by the tensor-core GEMM (hx_tcgemm.cu) as one [H d x 2d] x
// [2d x 2d] real product in 3-term TF32 split form.  Every ADO is Hermitian,
// so H_off X_n = Y_n^dagger and -i[H_off, X_n]_rc = -i(conj(Y_cr) - Y_rc): one
// product per ADO, not two (dense_tile_kernel).
//
// The reference has no precision other than the compiled one
// (src/legacy_compile_options.h:6); the complex64 path is the
// mixed-precision extension of this propagator.

#include <cuda_runtime.h>

#include <cstdint>

#include "hx_internal.h"

namespace hx {

namespace {

__device__ __forceinline__ uint32_t l_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

template <typename R>
__device__ __forceinline__ C2<R> mk(R x, R y)
{
    C2<R> v;
    v.x = x;
    v.y = y;
    return v;
}

// ---------------------------------------------------------------------------
// Stage of a dense H on full slabs (complex64): no flips, the commutator with
// H_off comes from Y_n = X_n H_off.  The term at (r, c) needs Y_rc and Y_cr,
// and the result is Hermitian, so a CTA takes a pair of 64 x 64 tiles (I, J)
// and (J, I), I <= J: it reads both tiles of Y, but the slab, the neighbours,
// the up terms and the base of the upper tile only, and writes the result and
// its conjugate transpose.  The transposed tiles pass through shared memory
// (element (r, c) at r 65 + c), so every access to memory is a run of columns.
// Bound by HBM: 12 of the 16 slabs' bytes of the element by element form.
// d = 256, 969 ADOs: 384 us a stage, where bands that computed both triangles
// took 635.
template <int LOGD, bool PAULI>
__global__ void __launch_bounds__(512, 2)
    dense_tile_kernel(LargeArgs<float> a, const float2* __restrict__ u, const float2* rho, float2* out, double alpha_d,
                      int base_kind)
{
    constexpr int D = 1 << LOGD, NBK = D / 64, NT = NBK * (NBK + 1) / 2, E = 4;
    constexpr long long D2 = static_cast<long long>(D) * D;
    extern __shared__ __align__(128) unsigned char smem[];
    float2* sT = reinterpret_cast<float2*>(smem);                            // [64][65] Y of tile (J, I), then the result
    double* sE = reinterpret_cast<double*>(smem + 64 * 65 * sizeof(float2));  // [D] (PAULI)
    float* sX = reinterpret_cast<float*>(sE + (PAULI ? D : 0));              // [D] (PAULI)
    float* sV = sX + (PAULI ? D : 0);                                        // [J][D] (general couplings)
    float* sWc = sV + (PAULI ? 0 : a.J * D);                                 // [2M] (twice the weights with PAULI)
    float* sWa = sWc + 2 * a.M;                                              // [2M]
    int* sSlab = reinterpret_cast<int*>(sWa + 2 * a.M);                      // [2M]
    int* sBit = sSlab + 2 * a.M;                                             // [2M] spin (PAULI) or bath

    const int tid = threadIdx.x;
    const long long n = a.first_ado + static_cast<long long>(blockIdx.x) / NT;
    int J = 0, I = static_cast<int>(blockIdx.x % NT);
    while (I > J) I -= ++J;
    const int c = tid & 63, r0 = tid >> 6;  // rows r0 + 8 k of the tile
    const int gc = J * 64 + c, gr0 = I * 64 + r0;
    const long long own = n * D2 + (static_cast<long long>(gr0) << LOGD) + gc;   // + 8 D k
    const long long mir = n * D2 + (static_cast<long long>(J * 64 + r0) << LOGD) + I * 64 + c;  // the transposed tile
#pragma unroll
    for (int k = 0; k < 8; ++k) sT[(r0 + 8 * k) * 65 + c] = __ldcs(a.dense_y + mir + 8ll * D * k);
    const int Q = a.ent_count[n];
    for (int q = tid; q < Q; q += 512) {
        const long long e = n * 2 * a.M + q;
        const int j = a.ent_bath[e] & 0xffff;
        sSlab[q] = a.ent_slab[e];
        sBit[q] = PAULI ? a.vbit[j] : j;
        sWc[q] = static_cast<float>(PAULI ? 2.0 * a.ent_wc[e] : a.ent_wc[e]);
        sWa[q] = static_cast<float>(PAULI ? 2.0 * a.ent_wa[e] : a.ent_wa[e]);
    }
    if (PAULI) {
        for (int i = tid; i < D; i += 512) {
            sE[i] = a.hdiag[i];
            sX[i] = static_cast<float>(a.xsum[i]);
        }
    } else {
        for (int i = tid; i < a.J * D; i += 512) sV[i] = a.vdiag[i];
    }
    const float g = static_cast<float>(a.gsum[n]);
    const int slot = a.slot ? a.slot[n] : -1;
    const float alpha = static_cast<float>(alpha_d);
    __syncthreads();
    float2 o[8];
#pragma unroll
    for (int k0 = 0; k0 < 8; k0 += E) {
        float2 x[E], acc[E];
#pragma unroll
        for (int k = 0; k < E; ++k) {
            x[k] = __ldg(u + own + 8ll * D * (k0 + k));
            acc[k] = __ldcs(a.dense_y + own + 8ll * D * (k0 + k));
        }
#pragma unroll
        for (int k = 0; k < E; ++k) {
            const int r = gr0 + 8 * (k0 + k);
            float tr, ti;
            if (PAULI) {
                tr = sX[r ^ gc];
                ti = static_cast<float>(sE[gc] - sE[r]);
            } else {
                const float2 t = __ldg(a.diag + (static_cast<long long>(r) << LOGD) + gc);
                tr = t.x;
                ti = t.y;
            }
            tr -= g;
            // -i [H_off, X] = -i (conj(Y_cr) - Y_rc)
            const float2 yrc = acc[k], ycr = sT[c * 65 + r0 + 8 * (k0 + k)];
            acc[k].x = tr * x[k].x - ti * x[k].y - (yrc.y + ycr.y);
            acc[k].y = tr * x[k].y + ti * x[k].x + (yrc.x - ycr.x);
        }
        const float2* ub = u + own - n * D2 + 8ll * D * k0;
#pragma unroll 1
        for (int q = 0; q < Q; ++q) {
            const float2* src = ub + sSlab[q] * D2;
            const float wc = sWc[q], wa = sWa[q];
            const int bit = sBit[q];
            float2 y[E];
            float wr[E], wi[E];
#pragma unroll
            for (int k = 0; k < E; ++k) {
                const int r = gr0 + 8 * (k0 + k);
                if (PAULI) {
                    // equal bits: only -{V, y} wa; different bits: only -i [V, y] wc
                    const int br = (r >> bit) & 1;
                    const bool same = br == ((gc >> bit) & 1);
                    wr[k] = same ? (br ? -wa : wa) : 0.f;
                    wi[k] = same ? 0.f : (br ? -wc : wc);
                } else {
                    const float vr = sV[bit * D + r], vc = sV[bit * D + gc];
                    wr[k] = -(vr + vc) * wa;
                    wi[k] = -(vr - vc) * wc;
                }
                y[k] = mk<float>(0.f, 0.f);
                if (wr[k] != 0.f || wi[k] != 0.f) y[k] = __ldg(src + 8ll * D * k);
            }
#pragma unroll
            for (int k = 0; k < E; ++k) {
                acc[k].x += wr[k] * y[k].x - wi[k] * y[k].y;
                acc[k].y += wr[k] * y[k].y + wi[k] * y[k].x;
            }
        }
        if (slot >= 0) {
#pragma unroll
            for (int k = 0; k < E; ++k) {
                const float2 w = __ldcs(a.U + slot * D2 + own - n * D2 + 8ll * D * (k0 + k));
                acc[k].x += w.x;
                acc[k].y += w.y;
            }
        }
#pragma unroll
        for (int k = 0; k < E; ++k) {
            float2 b = mk<float>(0.f, 0.f);
            if (base_kind == kBaseSelf) b = x[k];
            else if (base_kind == kBaseRho) b = __ldcs(rho + own + 8ll * D * (k0 + k));
            o[k0 + k] = mk<float>(b.x + alpha * acc[k].x, b.y + alpha * acc[k].y);
        }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) __stcs(out + own + 8ll * D * k, o[k]);
    if (I == J) return;
    __syncthreads();  // every Y of the tile is read
#pragma unroll
    for (int k = 0; k < 8; ++k) sT[(r0 + 8 * k) * 65 + c] = mk<float>(o[k].x, -o[k].y);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 8; ++k) __stcs(out + mir + 8ll * D * k, sT[c * 65 + r0 + 8 * k]);
}

// Element (r, c) of a Hermitian-packed slab, any r, c (one load, no branch
// around it, so several lookups can be in flight at once).
template <typename C>
__device__ __forceinline__ C packed_at(const C* __restrict__ slab, int r, int c, int logd)
{
    const bool lower = r > c;
    const C v = __ldg(slab + herm_index(lower ? c : r, lower ? r : c, logd));
    C w;
    w.x = v.x;
    w.y = lower ? -v.y : v.y;
    return w;
}

// ---------------------------------------------------------------------------
// Tile kernel, on full slabs (FULL) or Hermitian-packed ones (layout in
// hx_internal.h).  A CTA computes one 64 x 64 tile (I, J), packed I <= J, of one ADO.  What bounds a stage
// is the traffic between L2 and the SMs (64 bytes a cycle each): per element
// its own value, the flip partners outside the tile, the neighbours, the base
// and the result.  A square tile keeps the six low bits of row and column
// inside, so 2 (log2 d - 6) partners come through L2 where bands of whole rows
// needed log2 d - log2(2048 / d) and the scattered lower halves of the rows:
//
//  * double: the lanes of a warp are 4 rows x 8 columns, so a partner tile is
//    read in pieces of 128 bytes directly and of 64 bytes where it lies below
//    the diagonal (conjugates of the transposed tile): no load is scattered;
//  * complex64: the lanes are one row of 32 columns, and the partner tiles on
//    and below the diagonal come through shared memory, two asked for at the
//    start and used after everything else (64 x 65 buffers, so the transposed
//    read is free of bank conflicts).  Read directly they were 33 of the 46
//    wavefronts of global loads per 32 elements.  Not staged where the tables
//    leave no room for the buffers at two CTAs per SM;
//  * the sum is kept times i: then a flip and a commutator entry are one
//    packed multiply-add in complex64, and an entry whose weight is zero on
//    all of a warp's rows is left out (the kernel issues 61% of the time);
//  * a thread owns 8 elements of one column, 8 rows apart, in NP passes: the
//    flips of the rows of a pass are in registers, the other flips inside the
//    tile in shared memory (element (r, c) at r 64 + (c ^ (r & 7)): free of
//    bank conflicts for the mirrored writes of a diagonal tile too);
//  * with sigma_z couplings the weights come from index bits and the diagonal
//    term from two d-entry tables instead of a third slab-sized stream;
//  * the diagonal term comes last: started with it, the sum was rounded at its
//    size by every flip and neighbour (error of a right-hand side at d = 128
//    1.57e-16 against 1.07e-16, of a complex64 step 2.4e-7 against 1.7e-7; d =
//    256 in double 4% faster so, in complex64 1% slower);
//  * diagonal tiles compute their upper triangle only.
//
// d = 256, 969 ADOs: 0.68 ms a stage in double, 0.44 in complex64 (bands of
// rows: 0.94 and 0.56; complex64 without staged tiles and packed arithmetic
// 0.48).  Double is at 77% of the load-store unit's wavefronts and 8.8 TB/s
// between L2 and the SMs.  Full slabs, us per step, bands of 4096 / d rows
// against tiles: d = 256, 165 ADOs 1260 and 855 in double, 614 and 475 in
// complex64; d = 128, 680 ADOs 1226 and 814; 604 and 465.  The 64 registers of two CTAs per SM are the limit: one
// pass of 8 rows in double spills or leaves one CTA (0.85 ms).
template <typename R, int LOGD> struct TileShape;
template <int LOGD> struct TileShape<double, LOGD> { static constexpr int NP = 2, MINB = 2, LR = LOGD == 7 ? 1 : 4; };
template <int LOGD> struct TileShape<float, LOGD> { static constexpr int NP = 1, MINB = 2, LR = 1; };
constexpr int kTileT = 512;

// Element (r, c), r <= c, of a packed slab is at packed_row(r) + c.
template <int LOGD>
__device__ __forceinline__ int packed_row(int r)
{
    constexpr int D = 1 << LOGD;
    return r < D / 2 ? r * D : (D - 1 - r) * (D + 1) + 1;
}

template <int LOGD, bool FULL>
__device__ __forceinline__ int row_at(int r)
{
    return FULL ? r << LOGD : packed_row<LOGD>(r);
}

// z += w y and x - y, elementwise: one packed instruction each in complex64 (the same roundings).
__device__ __forceinline__ void add_scaled(double2& z, double w, const double2& y)
{
    z.x += w * y.x;
    z.y += w * y.y;
}
__device__ __forceinline__ double2 minus(const double2& x, const double2& y) { return make_double2(x.x - y.x, x.y - y.y); }
__device__ __forceinline__ uint64_t bits2(const float2& v)
{
    uint64_t b;
    asm("mov.b64 %0, {%1, %2};" : "=l"(b) : "f"(v.x), "f"(v.y));
    return b;
}
__device__ __forceinline__ float2 fma2(const float2& a, const float2& b, const float2& c)
{
    uint64_t d;
    float2 v;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(bits2(a)), "l"(bits2(b)), "l"(bits2(c)));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(d));
    return v;
}
__device__ __forceinline__ void add_scaled(float2& z, float w, const float2& y) { z = fma2(make_float2(w, w), y, z); }
// z += (wx y.x, wy y.y)
__device__ __forceinline__ void add_scaled2(float2& z, float wx, float wy, const float2& y)
{
    z = fma2(make_float2(wx, wy), y, z);
}
__device__ __forceinline__ void add_scaled2(double2& z, double wx, double wy, const double2& y)
{
    z.x += wx * y.x;
    z.y += wy * y.y;
}
__device__ __forceinline__ float2 minus(const float2& x, const float2& y) { return fma2(y, make_float2(-1.f, -1.f), x); }

// z += i (weight at the k-th row) y for one neighbour entry with a sigma_z
// coupling.  Where the spin's bits of row and column agree only -{V, y} wa
// counts, else only -i [V, y] wc (twice the weights are given).  T: the bit of
// k that the spin's row bit is, or -1 when all the rows of the pass share it.
template <typename R, int E, int T>
__device__ __forceinline__ void tile_entry(C2<R>* z, const C2<R>* src, int step, const bool* on, int k0, int br0,
                                           int bc, R wc, R wa)
{
    C2<R> y[E];
    const bool same0 = br0 == bc;  // at rows whose bit is br0
    const R wr0 = same0 ? (br0 ? -wa : wa) : R(0), wi0 = same0 ? R(0) : (br0 ? -wc : wc);
    const R wr1 = same0 ? R(0) : (br0 ? wa : -wa), wi1 = same0 ? (br0 ? wc : -wc) : R(0);  // at the others
    const bool need0 = wr0 != R(0) || wi0 != R(0), need1 = wr1 != R(0) || wi1 != R(0);
    // 3% of a complex64 step; in double, where issue slots are not short, the branch costs 1.5%
    if (sizeof(R) == sizeof(float) && !need0 && (T < 0 || !need1)) return;
#pragma unroll
    for (int k = 0; k < E; ++k) {
        const bool other = T >= 0 && ((k >> (T < 0 ? 0 : T)) & 1);
        y[k] = mk<R>(0, 0);
        if (on[k] && (other ? need1 : need0)) y[k] = __ldg(src + k * step);
    }
    if (same0) {
#pragma unroll
        for (int k = 0; k < E; ++k) {
            if (T >= 0 && ((k >> (T < 0 ? 0 : T)) & 1)) {
                add_scaled(z[k], -wi1, y[k]);
            } else {
                z[k].x -= wr0 * y[k].y;
                z[k].y += wr0 * y[k].x;
            }
        }
    } else {
#pragma unroll
        for (int k = 0; k < E; ++k) {
            if (T >= 0 && ((k >> (T < 0 ? 0 : T)) & 1)) {
                z[k].x -= wr1 * y[k].y;
                z[k].y += wr1 * y[k].x;
            } else {
                add_scaled(z[k], -wi0, y[k]);
            }
        }
    }
}

// Flip f of tile (I, J), f = 2 i for bit 6 + i of the row and 2 i + 1 of the column: the partner's tile
// (A, B), true when it is not stored as such (on or below the diagonal).
__device__ __forceinline__ bool flip_tile(int f, int I, int J, int& A, int& B)
{
    const int m = 1 << (f >> 1);
    A = f & 1 ? I : I ^ m;
    B = f & 1 ? J ^ m : J;
    return A >= B;
}

// Ask for the stored tile (B, A), B <= A, of a packed slab into the 64 x 65 buffer dst (the upper triangle
// only when A == B).
template <typename R, int LOGD>
__device__ __forceinline__ void stage_tile(const C2<R>* __restrict__ un, int A, int B, C2<R>* dst)
{
    constexpr int D = 1 << LOGD;
    const int j = threadIdx.x & 63, i0 = threadIdx.x >> 6;  // rows i0 + 8 k
    const C2<R>* src = un + packed_row<LOGD>(B * 64 + i0) + A * 64 + j;
    const int step = B * 64 < D / 2 ? 8 * D : -8 * (D + 1);
    const uint32_t at = l_addr(dst + i0 * 65 + j);
#pragma unroll
    for (int k = 0; k < 8; ++k)
        if (A != B || i0 + 8 * k <= j)
            asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(
                             at + k * 8 * 65 * static_cast<uint32_t>(sizeof(C2<R>))),
                         "l"(src + k * step), "n"(sizeof(C2<R>))
                         : "memory");
}

template <typename R, int LOGD, bool PAULI, bool STAGED, bool FULL>
__global__ void __launch_bounds__(kTileT, TileShape<R, LOGD>::MINB)
    tile_kernel(LargeArgs<R> a, const C2<R>* __restrict__ u, const C2<R>* rho, C2<R>* out, double alpha_d,
                     int base_kind)
{
    using C = C2<R>;
    constexpr int D = 1 << LOGD, NP = TileShape<R, LOGD>::NP, E = 8 / NP, NBK = D / 64,
                  NT = FULL ? NBK * NBK : NBK * (NBK + 1) / 2;
    constexpr int LR = FULL ? 1 : TileShape<R, LOGD>::LR, LC = 32 / LR;  // rows and columns of a warp's lanes
    constexpr long long P = FULL ? static_cast<long long>(D) * D : static_cast<long long>(D / 2) * (D + 1);
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr int F = 2 * (LOGD - 6);
    C* sx = reinterpret_cast<C*>(smem);                                // [64][64] the tile
    C* sT = sx + 4096;                                                 // [2][64][65] partner tiles, when staged
    double* sE = reinterpret_cast<double*>(sT + (STAGED ? 2 * 64 * 65 : 0));  // [D] E_r (PAULI)
    R* sX = reinterpret_cast<R*>(sE + (PAULI ? D : 0));                // [D] -4 sum of xi over differing bits (PAULI)
    R* sV = sX + (PAULI ? D : 0);                                      // [J][D] (general couplings)
    R* sH = sV + (PAULI ? 0 : a.J * D);                                // [LOGD]
    R* sWc = sH + LOGD;                                                // [2M] (twice the weights with PAULI)
    R* sWa = sWc + 2 * a.M;                                            // [2M]
    int* sSlab = reinterpret_cast<int*>(sWa + 2 * a.M);                // [2M]
    int* sBit = sSlab + 2 * a.M;                                       // [2M] spin (PAULI) or bath

    const int tid = threadIdx.x;
    const bool halves = NP == 2 && a.halves;
    const unsigned blk = halves ? blockIdx.x >> 1 : blockIdx.x;
    const long long n = a.first_ado + static_cast<long long>(blk) / NT;
    int J = 0, I = static_cast<int>(blk % NT);
    if constexpr (FULL) {
        J = I % NBK;
        I /= NBK;
    } else {
        while (I > J) I -= ++J;  // tile (I, J) of the upper triangle, column by column
    }
    const C* un = u + n * P;
    const int warp = tid >> 5, lane = tid & 31;
    const int r0 = lane / LC + LR * (warp / (2 * LR));  // rows r0 + 8 k of the tile
    // the second half of the rows is stored shifted by -r mod 8 elements: shifting the columns of a thread
    // the other way keeps eight lanes on one 128-byte line
    const int c = (lane % LC + LC * (warp % (2 * LR)) + (FULL || I * 64 < D / 2 ? 0 : r0)) & 63;
    const bool diag = !FULL && I == J;
    const int gc = J * 64 + c, gr0 = I * 64 + r0;
    const int own = row_at<LOGD, FULL>(gr0) + gc;     // packed position of element k: own + k * step
    const int step = FULL || I * 64 < D / 2 ? 8 * D : -8 * (D + 1);

    // ---- the tile (both triangles of a diagonal one)
    [[maybe_unused]] int fl = 0;  // the next flip to stage, or past the last one
    {
        C x[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (!diag || r0 + 8 * k <= c) x[k] = __ldg(un + own + k * step);
        if constexpr (STAGED) {
#pragma unroll 1
            for (int b = 0; b < 2; ++b) {
                int A, B;
                while (fl < F && !flip_tile(fl, I, J, A, B)) ++fl;
                if (fl < F) stage_tile<R, LOGD>(un, A, B, sT + b * 64 * 65);
                asm volatile("cp.async.commit_group;" ::: "memory");
                ++fl;
            }
        }
        const int Q = a.ent_count[n];
        for (int q = tid; q < Q; q += kTileT) {
            const long long src = n * 2 * a.M + q;
            const int j = a.ent_bath[src] & 0xffff;
            sSlab[q] = a.ent_slab[src];
            sBit[q] = PAULI ? a.vbit[j] : j;
            sWc[q] = static_cast<R>(PAULI ? 2.0 * a.ent_wc[src] : a.ent_wc[src]);
            sWa[q] = static_cast<R>(PAULI ? 2.0 * a.ent_wa[src] : a.ent_wa[src]);
        }
        if (PAULI) {
            for (int i = tid; i < D; i += kTileT) {
                sE[i] = a.hdiag[i];
                sX[i] = static_cast<R>(a.xsum[i]);
            }
        } else {
            for (int i = tid; i < a.J * D; i += kTileT) sV[i] = a.vdiag[i];
        }
        if (tid < LOGD) sH[tid] = a.hflip[tid];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int r = r0 + 8 * k;
            if (diag && r > c) continue;
            sx[r * 64 + (c ^ (r & 7))] = x[k];
            if (diag && r < c) sx[c * 64 + (r ^ (c & 7))] = mk<R>(x[k].x, -x[k].y);
        }
    }
    const int Q = a.ent_count[n];
    const R g = static_cast<R>(a.gsum[n]);
    const int slot = a.slot ? a.slot[n] : -1;
    const R alpha = static_cast<R>(alpha_d);
    __syncthreads();

#pragma unroll 1
    for (int k0 = halves ? static_cast<int>(blockIdx.x & 1) * E : 0, k1 = halves ? k0 + E : 8; k0 < k1; k0 += E) {
        if (NP > 1 && diag && !__any_sync(0xffffffffu, r0 + 8 * k0 <= c)) break;  // the warp's rows are below its columns
        C z[E];  // i times the sum
        bool on[E];
        const C* sp = sx + (r0 + 8 * k0) * 64;  // the pass's first row; + 512 per k
        const int cs = c ^ (r0 & 7);
#pragma unroll
        for (int k = 0; k < E; ++k) {
            on[k] = !diag || r0 + 8 * (k0 + k) <= c;
            z[k] = mk<R>(0, 0);
        }
        {
            C x[E];
#pragma unroll
            for (int k = 0; k < E; ++k) x[k] = sp[cs + 512 * k];
            // ---- flips inside the tile: z += h (row partner - column partner)
#pragma unroll
            for (int b = 0; b < 6; ++b) {
                const R h = sH[b];
                const C* rp = sx + (((r0 + 8 * k0) ^ (1 << b)) * 64);  // row partners not in registers (no bit of k)
                const int rs = cs ^ (b < 3 ? (1 << b) : 0);
#pragma unroll
                for (int k = 0; k < E; ++k) {
                    C rowp;
                    if (b >= 3 && (1 << (b - 3)) < E) rowp = x[k ^ (1 << (b - 3))];
                    else rowp = rp[rs + 512 * k];
                    const C colp = sp[(cs ^ (1 << b)) + 512 * k];
                    add_scaled(z[k], h, minus(rowp, colp));
                }
            }
        }
        // ---- flips of the higher bits: the same place in another tile, through L2
#pragma unroll 1
        for (int f = 0; f < F; ++f) {
            int A, B;  // the partner's tile
            if (flip_tile(f, I, J, A, B) && STAGED) continue;
            const R h = sH[6 + (f >> 1)];
            const R w = f & 1 ? -h : h;
            C y[E];
            if (!FULL && A == B) {
                const int rb = A * 64 + r0 + 8 * k0, cb = B * 64 + c;
#pragma unroll
                for (int k = 0; k < E; ++k) y[k] = on[k] ? packed_at(un, rb + 8 * k, cb, LOGD) : mk<R>(0, 0);
            } else {
                // above the diagonal directly, below it the transposed place
                const bool up = FULL || A < B;
                const int at = up ? row_at<LOGD, FULL>(A * 64 + r0) + B * 64 + c : packed_row<LOGD>(B * 64 + c) + A * 64 + r0;
                const int st = up ? (FULL || A * 64 < D / 2 ? 8 * D : -8 * (D + 1)) : 8;
                const C* src = un + at + k0 * st;
#pragma unroll
                for (int k = 0; k < E; ++k) y[k] = on[k] ? __ldg(src + k * st) : mk<R>(0, 0);
            }
            const R wy = !FULL && A > B ? -w : w;
#pragma unroll
            for (int k = 0; k < E; ++k) {
                z[k].x += w * y[k].x;
                z[k].y += wy * y[k].y;
            }
        }
        // ---- neighbour entries, E loads in flight
        const C* ub = u + own + k0 * step;
#pragma unroll 1
        for (int q = 0; q < Q; ++q) {
            const C* src = ub + static_cast<long long>(sSlab[q]) * P;
            const R wc = sWc[q], wa = sWa[q];
            const int bit = sBit[q];
            if (PAULI) {
                const int br0 = ((gr0 + 8 * k0) >> bit) & 1, bc = (gc >> bit) & 1;
                if (bit == 3 && E > 1) tile_entry<R, E, 0>(z, src, step, on, k0, br0, bc, wc, wa);
                else if (bit == 4 && E > 2) tile_entry<R, E, 1>(z, src, step, on, k0, br0, bc, wc, wa);
                else if (bit == 5 && E > 4) tile_entry<R, E, 2>(z, src, step, on, k0, br0, bc, wc, wa);
                else tile_entry<R, E, -1>(z, src, step, on, k0, br0, bc, wc, wa);
            } else {
                const R* vj = sV + bit * D;
                const R vc = vj[gc];
                C y[E];
#pragma unroll
                for (int k = 0; k < E; ++k) {
                    const R vr = vj[gr0 + 8 * (k0 + k)];
                    y[k] = mk<R>(0, 0);
                    if (on[k] && ((vr + vc) * wa != R(0) || (vr - vc) * wc != R(0))) y[k] = __ldg(src + k * step);
                }
#pragma unroll
                for (int k = 0; k < E; ++k) {
                    const R vr = vj[gr0 + 8 * (k0 + k)];
                    const R ar = -(vr + vc) * wa, ai = -(vr - vc) * wc;
                    z[k].x -= ar * y[k].y + ai * y[k].x;
                    z[k].y += ar * y[k].x - ai * y[k].y;
                }
            }
        }
        // ---- the flips from staged tiles: conjugates of the transposed place
        if constexpr (STAGED) {
            int buf = 0;
#pragma unroll 1
            for (int f = 0; f < F; ++f) {
                int A, B;
                if (!flip_tile(f, I, J, A, B)) continue;
                asm volatile("cp.async.wait_group 1;" ::: "memory");
                __syncthreads();
                const C* t = sT + buf * 64 * 65;
                const R h = sH[6 + (f >> 1)];
                const R w = f & 1 ? -h : h;
                if (A != B) {
#pragma unroll
                    for (int k = 0; k < E; ++k) {
                        const C y = t[c * 65 + r0 + 8 * k];
                        add_scaled2(z[k], w, -w, y);
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < E; ++k) {
                        const int r = r0 + 8 * k;
                        const C y = t[r <= c ? r * 65 + c : c * 65 + r];
                        z[k].x += w * y.x;
                        z[k].y += r <= c ? w * y.y : -w * y.y;
                    }
                }
                int A2, B2;
                while (fl < F && !flip_tile(fl, I, J, A2, B2)) ++fl;
                if (fl < F) {
                    __syncthreads();  // every warp has read the buffer
                    stage_tile<R, LOGD>(un, A2, B2, sT + buf * 64 * 65);
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
                ++fl;
                buf ^= 1;
            }
        }
        // ---- up term of tier L-1, summed by large_upterm_kernel
        C y[E];
        if (slot >= 0) {
            const C* Un = a.U + static_cast<long long>(slot) * P + own + k0 * step;
#pragma unroll
            for (int k = 0; k < E; ++k) y[k] = on[k] ? __ldcs(Un + k * step) : mk<R>(0, 0);
#pragma unroll
            for (int k = 0; k < E; ++k) {
                z[k].x -= y[k].y;
                z[k].y += y[k].x;
            }
        }
        // ---- diagonal term, last: everything before is rounded at its own, smaller size
#pragma unroll
        for (int k = 0; k < E; ++k) {
            const int r = gr0 + 8 * (k0 + k);
            const C x = sp[cs + 512 * k];
            R tr, ti;
            if (PAULI) {
                tr = sX[r ^ gc];
                ti = static_cast<R>(sE[gc] - sE[r]);
            } else {
                const C t = on[k] ? __ldg(a.diag + own + (k0 + k) * step) : mk<R>(0, 0);
                tr = t.x;
                ti = t.y;
            }
            tr -= g;
            z[k].x -= tr * x.y + ti * x.x;
            z[k].y += tr * x.x - ti * x.y;
        }
        // ---- Horner epilogue
        C* on_ = out + n * P + own + k0 * step;
        const C* rn = rho + n * P + own + k0 * step;
#pragma unroll
        for (int k = 0; k < E; ++k) {
            y[k] = mk<R>(0, 0);
            if (base_kind == kBaseSelf) y[k] = sp[cs + 512 * k];
            else if (base_kind == kBaseRho && on[k]) y[k] = __ldcs(rn + k * step);
        }
#pragma unroll
        for (int k = 0; k < E; ++k)
            if (on[k]) __stcs(on_ + k * step, mk<R>(y[k].x + alpha * z[k].y, y[k].y - alpha * z[k].x));
    }
}

// Up term of tier L-1 in the working precision, tile-major so the top-tier
// data of the resident tiles stays in L2 (as upterm_kernel, hx_upterm.cu).
constexpr int kUpWarps = 8, kUpTile = 32;

// A warp takes SLOTS slots side by side and asks for MODES neighbours of each at a time.
template <typename R, int SLOTS, int MODES>
__global__ void __launch_bounds__(kUpWarps * 32)
    large_upterm_kernel(LargeUpArgs<R> a, const C2<R>* __restrict__ u, C2<R>* __restrict__ U)
{
    using C = C2<R>;
    const int D = 1 << a.logd;
    // elements per stored slab: d^2, or the packed upper triangle
    const long long D2 = a.herm ? herm_elems(a.logd) : static_cast<long long>(D) * D;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long e = static_cast<long long>(blockIdx.y) * kUpTile + lane;
    if (e >= D2) return;
    int r, c;
    if (a.herm) {
        herm_coords(static_cast<int>(e), a.logd, r, c);
    } else {
        r = static_cast<int>(e >> a.logd);
        c = static_cast<int>(e & (D - 1));
        if (a.upper && (c >> 6) < (r >> 6)) return;  // a tile that nobody reads
    }
    const C* ue = u + e;
    const int s0 = (blockIdx.x * kUpWarps + warp) * SLOTS;
    const int ns = min(a.S - s0, SLOTS);
    if (ns <= 0) return;
    const int32_t* slab[SLOTS];
    R re[SLOTS], im[SLOTS];
#pragma unroll
    for (int t = 0; t < SLOTS; ++t) {
        slab[t] = a.slab + static_cast<long long>(s0 + min(t, ns - 1)) * a.M;
        re[t] = im[t] = 0;
    }
    for (int j = 0; j < a.J; ++j) {
        const R del = __ldg(a.vdiag + j * D + r) - __ldg(a.vdiag + j * D + c);
        if (del == R(0)) continue;
        const int m1 = __ldg(a.bath_off + j + 1);
        R sr[SLOTS], si[SLOTS];
#pragma unroll
        for (int t = 0; t < SLOTS; ++t) sr[t] = si[t] = 0;
        for (int m = __ldg(a.bath_off + j); m < m1; m += MODES) {
            C y[MODES][SLOTS];
#pragma unroll
            for (int i = 0; i < MODES; ++i)
#pragma unroll
                for (int t = 0; t < SLOTS; ++t)
                    if (m + i < m1) y[i][t] = __ldg(ue + static_cast<long long>(__ldg(slab[t] + m + i)) * D2);
#pragma unroll
            for (int i = 0; i < MODES; ++i)
#pragma unroll
                for (int t = 0; t < SLOTS; ++t)
                    if (m + i < m1) {
                        sr[t] += y[i][t].x;
                        si[t] += y[i][t].y;
                    }
        }
#pragma unroll
        for (int t = 0; t < SLOTS; ++t) {
            re[t] += del * si[t];  // -i del S
            im[t] -= del * sr[t];
        }
    }
#pragma unroll
    for (int t = 0; t < SLOTS; ++t)
        if (t < ns) U[static_cast<long long>(s0 + t) * D2 + e] = mk<R>(re[t], im[t]);
}

template <typename R, int SLOTS, int MODES>
void launch_upterm_t(const LargeUpArgs<R>& a, const C2<R>* u, C2<R>* U, cudaStream_t s)
{
    const long long D2 = a.herm ? herm_elems(a.logd) : 1ll << (2 * a.logd);
    constexpr int per = kUpWarps * SLOTS;
    const dim3 grid((a.S + per - 1) / per, static_cast<unsigned>((D2 + kUpTile - 1) / kUpTile));
    large_upterm_kernel<R, SLOTS, MODES><<<grid, kUpWarps * 32, 0, s>>>(a, u, U);
}

// Tier-0 ADO of the mixed-precision propagator in double precision: its own
// slab u0, H and diagonal terms in FP64; its (up) neighbours come from the
// complex64 hierarchy and are accumulated in FP64.  Writes the FP64 result
// and its complex64 copy (slot 0 of the complex64 output).
__global__ void __launch_bounds__(256)
    ado0_kernel(Ado0Args a, const double2* __restrict__ u0, const float2* __restrict__ u, const double2* rho0,
                double2* out0, float2* out32, double alpha, int base_kind)
{
    const int D = 1 << a.logd;
    const long long D2 = a.herm ? herm_elems(a.logd) : static_cast<long long>(D) * D;
    const long long ge = blockIdx.x * 256ll + threadIdx.x;
    if (ge >= D2) return;
    int r, c;
    if (a.herm) {
        herm_coords(static_cast<int>(ge), a.logd, r, c);
    } else {
        r = static_cast<int>(ge >> a.logd);
        c = static_cast<int>(ge & (D - 1));
    }
    const double2 x = u0[ge];
    const double2 t = a.diag[ge];
    double hr = 0.0, hi = 0.0;
    for (int i = 0; i < a.logd; ++i) {
        double2 p, q;
        if (a.herm) {
            p = packed_at(u0, r ^ (1 << i), c, a.logd);
            q = packed_at(u0, r, c ^ (1 << i), a.logd);
        } else {
            p = u0[ge ^ (static_cast<long long>(D) << i)];
            q = u0[ge ^ (1ll << i)];
        }
        hr += a.hflip[i] * (p.x - q.x);
        hi += a.hflip[i] * (p.y - q.y);
    }
    double ax = t.x * x.x - t.y * x.y + hi;
    double ay = t.x * x.y + t.y * x.x - hr;
    if (a.dense_z) {
        // -i [H_off, X] = -i (conj(Z_cr) - Z_rc) of ADO 0 from its FP64 product Z = X H_off (X, H Hermitian);
        // the diagonal terms -2 Im Z_rr sum to -2 Im Tr(X H_off) = 0, so the commutator stays traceless
        const double2 zrc = a.dense_z[ge], zcr = a.dense_z[(static_cast<long long>(c) << a.logd) + r];
        ax -= zrc.y + zcr.y;
        ay += zrc.x - zcr.x;
    }
    const int Q = a.ent_count[0];
    for (int q = 0; q < Q; ++q) {
        const int j = a.ent_bath[q] & 0xffff;
        const double vr = a.vdiag[j * D + r], vc = a.vdiag[j * D + c];
        const double ar = -(vr + vc) * a.ent_wa[q], ai = -(vr - vc) * a.ent_wc[q];
        if (ar == 0.0 && ai == 0.0) continue;
        const float2 yf = u[static_cast<long long>(a.ent_slab[q]) * D2 + ge];
        const double yx = yf.x, yy = yf.y;
        ax += ar * yx - ai * yy;
        ay += ar * yy + ai * yx;
    }
    double2 b;
    if (base_kind == kBaseSelf) b = x;
    else if (base_kind == kBaseRho) b = rho0[ge];
    else b = make_double2(0.0, 0.0);
    const double2 o = make_double2(b.x + alpha * ax, b.y + alpha * ay);
    out0[ge] = o;
    out32[ge] = make_float2(static_cast<float>(o.x), static_cast<float>(o.y));
}

// Z = X H, d x d complex FP64 (ADO 0 of a dense-H stage): 32 x 16 output
// tiles, two outputs of one row per thread, K staged through shared memory 32
// at a time with the next block's loads under way.  d^3 complex multiply-adds
// in d^2 / 512 CTAs (d = 256: 48 us with 64 CTAs of 16 x 4 outputs a warp,
// 18 so).
__global__ void __launch_bounds__(256) zgemm_kernel(const double2* __restrict__ x, const double2* __restrict__ h,
                                                    double2* __restrict__ z, int logd)
{
    constexpr int TM = 32, TN = 16, TK = 32;
    __shared__ double2 sa[TM][TK + 1];
    __shared__ double2 sb[TK][TN];
    const int D = 1 << logd;
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
    const int tid = threadIdx.x, col = tid & 7, row = tid >> 3;  // outputs (row, col) and (row, col + 8)
    double2 ra[4], rb[2];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int e = tid + 256 * i;
            ra[i] = __ldg(x + (static_cast<long long>(m0 + (e >> 5)) << logd) + k0 + (e & 31));
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int e = tid + 256 * i;
            rb[i] = __ldg(h + (static_cast<long long>(k0 + (e >> 4)) << logd) + n0 + (e & 15));
        }
    };
    double2 acc[2] = {make_double2(0.0, 0.0), make_double2(0.0, 0.0)};
    fetch(0);
    for (int k0 = 0; k0 < D; k0 += TK) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i) sa[(tid + 256 * i) >> 5][(tid + 256 * i) & 31] = ra[i];
#pragma unroll
        for (int i = 0; i < 2; ++i) sb[(tid + 256 * i) >> 4][(tid + 256 * i) & 15] = rb[i];
        __syncthreads();
        if (k0 + TK < D) fetch(k0 + TK);
#pragma unroll 8
        for (int kk = 0; kk < TK; ++kk) {
            const double2 av = sa[row][kk];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const double2 b = sb[kk][col + 8 * j];
                acc[j].x = fma(av.x, b.x, fma(-av.y, b.y, acc[j].x));
                acc[j].y = fma(av.x, b.y, fma(av.y, b.x, acc[j].y));
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) z[(static_cast<long long>(m0 + row) << logd) + n0 + col + 8 * j] = acc[j];
}

__global__ void d2f_kernel(const double2* __restrict__ in, float2* __restrict__ out, long long n)
{
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x)
        out[i] = make_float2(static_cast<float>(in[i].x), static_cast<float>(in[i].y));
}

__global__ void vec_d2f_kernel(const double* __restrict__ in, float* __restrict__ out, long long n)
{
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x)
        out[i] = static_cast<float>(in[i]);
}

template <typename R, int LOGD>
size_t tile_smem(int M, int J, bool pauli, bool staged)
{
    const size_t D = size_t(1) << LOGD;
    return (4096 + (staged ? 2 * 64 * 65 : 0)) * sizeof(C2<R>) + (pauli ? D * (sizeof(double) + sizeof(R)) : J * D * sizeof(R)) +
           sizeof(R) * (LOGD + 4 * M) + sizeof(int) * 4 * M;
}

// Stage of a dense H; launch = false: raise the shared-memory limit only.
template <int LOGD>
bool launch_dense(const LargeArgs<float>& a, const float2* u, const float2* rho, float2* out, double alpha, int base,
                  cudaStream_t s, bool launch)
{
    const size_t D = size_t(1) << LOGD;
    const size_t smem = 64 * 65 * sizeof(float2) + (a.pauli ? D * (sizeof(double) + sizeof(float)) : a.J * D * sizeof(float)) +
                        sizeof(float) * 4 * a.M + sizeof(int) * 4 * a.M;
    if (smem > 227 * 1024) return false;
    auto* kernel = a.pauli ? dense_tile_kernel<LOGD, true> : dense_tile_kernel<LOGD, false>;
    if (!launch)
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) == cudaSuccess;
    constexpr long long kBlocks = (1 << LOGD) / 64;
    const long long nb = (a.H - a.first_ado) * (kBlocks * (kBlocks + 1) / 2);
    if (nb > 0) kernel<<<static_cast<unsigned>(nb), 512, smem, s>>>(a, u, rho, out, alpha, base);
    return true;
}

// A CTA per half of a tile's rows (double): always while the tiles do not fill the SMs, then while the SM with the most
// halves has less to do than the one with the most tiles, as long as there are few rounds.  us a step, tiles and halves:
// d = 128, 28 ADOs (84 tiles) 111 and 96, 66 (198) 148 and 132, but 120 (360) 179 and 185; d = 256, 15 ADOs (150) 155 and
// 141, 29 (290: two tiles or four halves on an SM) 188 and 198, 45 (450) 232 and 222, 165 (1650) 627 and 663; d = 512, 5
// ADOs (180) 196 and 174, 9 (324) 239 and 230, 13 (468) 308 and 297.
inline bool half_tiles(long long tiles, int logd)
{
    constexpr long long kSms = 148;
    if (tiles <= kSms) return true;
    if (tiles > (logd == 7 ? 3 * kSms / 2 : 13 * kSms / 4)) return false;
    return (2 * tiles + kSms - 1) / kSms < 2 * ((tiles + kSms - 1) / kSms);
}

template <typename R, int LOGD>
bool launch_t(const LargeArgs<R>& a, const C2<R>* u, const C2<R>* rho, C2<R>* out, double alpha, int base,
              cudaStream_t s, bool launch)
{
    using Kernel = void (*)(LargeArgs<R>, const C2<R>*, const C2<R>*, C2<R>*, double, int);
    // complex64: partner tiles are staged where two CTAs per SM still find room for the buffers
    constexpr bool kStage = sizeof(R) == sizeof(float);
    // one coupling: the two tables of the sigma_z form are longer than the operator's, which may be what fits
    const bool pauli = a.pauli && tile_smem<R, LOGD>(a.M, a.J, true, false) <= 227 * 1024;
    const bool staged = kStage && a.herm && tile_smem<R, LOGD>(a.M, a.J, pauli, true) <= 113 * 1024;
    const size_t smem = tile_smem<R, LOGD>(a.M, a.J, pauli, staged);
    Kernel kernel;
    if (!a.herm) kernel = pauli ? tile_kernel<R, LOGD, true, false, true> : tile_kernel<R, LOGD, false, false, true>;
    else if (staged) kernel = pauli ? tile_kernel<R, LOGD, true, kStage, false> : tile_kernel<R, LOGD, false, kStage, false>;
    else kernel = pauli ? tile_kernel<R, LOGD, true, false, false> : tile_kernel<R, LOGD, false, false, false>;
    if (smem > 227 * 1024) return false;
    // the limit is raised when a context is made, outside any capture
    if (!launch)
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) == cudaSuccess;
    // packed slabs: the tiles of the upper triangle
    constexpr long long kBlocks = (1 << LOGD) / 64;
    const long long nb = (a.H - a.first_ado) * (a.herm ? kBlocks * (kBlocks + 1) / 2 : kBlocks * kBlocks);
    if (nb <= 0) return true;
    LargeArgs<R> t = a;
    t.halves = sizeof(R) == sizeof(double) && half_tiles(nb, LOGD) ? 1 : 0;
    kernel<<<static_cast<unsigned>(t.halves ? 2 * nb : nb), kTileT, smem, s>>>(t, u, rho, out, alpha, base);
    return true;
}

template <typename R>
bool dispatch(const LargeArgs<R>& a, const C2<R>* u, const C2<R>* rho, C2<R>* out, double alpha, int base,
              cudaStream_t s, bool launch)
{
    if constexpr (sizeof(R) == sizeof(float))
        if (a.dense) {
            switch (a.logd) {
            case 7: return launch_dense<7>(a, u, rho, out, alpha, base, s, launch);
            case 8: return launch_dense<8>(a, u, rho, out, alpha, base, s, launch);
            case 9: return launch_dense<9>(a, u, rho, out, alpha, base, s, launch);
            case 10: return launch_dense<10>(a, u, rho, out, alpha, base, s, launch);
            default: return false;
            }
        }
    switch (a.logd) {
    case 7: return launch_t<R, 7>(a, u, rho, out, alpha, base, s, launch);
    case 8: return launch_t<R, 8>(a, u, rho, out, alpha, base, s, launch);
    case 9: return launch_t<R, 9>(a, u, rho, out, alpha, base, s, launch);
    case 10: return launch_t<R, 10>(a, u, rho, out, alpha, base, s, launch);
    default: return false;
    }
}

}  // namespace

bool large_supported(int logd, int M, int J)
{
    if (logd < 7 || logd > 10) return false;
    const size_t need = 4096 * sizeof(double2) + 16 + sizeof(double) * 4 * M + sizeof(double) * (J * (1 << logd) + logd + 1) +
                        sizeof(int) * 4 * M + 16;
    return need <= 227 * 1024;
}

template <typename R>
bool prepare_large(const LargeArgs<R>& a)
{
    return dispatch<R>(a, nullptr, nullptr, nullptr, 0.0, 0, nullptr, false);
}

template <typename R>
bool launch_large(const LargeArgs<R>& a, const C2<R>* u, const C2<R>* rho, C2<R>* out, double alpha, int base_kind,
                  cudaStream_t s)
{
    return dispatch<R>(a, u, rho, out, alpha, base_kind, s, true);
}

template <typename R>
void launch_large_upterm(const LargeUpArgs<R>& a, const C2<R>* u, C2<R>* U, cudaStream_t s)
{
    if (a.S <= 0) return;
    // few slots: four modes of one slot at a time, else the warps wait on one neighbour after the other.  us a step in
    // double, four slots side by side and this: d = 128, 28 modes 1 slot 112 and 92, 12 modes 12 slots 162 and 140, 14
    // modes 14 slots 179 and 171, but 8 modes 36 slots 214 and 219; d = 256, 8 modes 8 slots 224 and 206, 36 slots 626
    // and 644; eight modes at a time 116, 152, 179, 241, 220 and 726.
    if (a.S <= 16) launch_upterm_t<R, 1, 4>(a, u, U, s);
    else launch_upterm_t<R, 4, 1>(a, u, U, s);
}

template bool prepare_large<double>(const LargeArgs<double>&);
template bool prepare_large<float>(const LargeArgs<float>&);
template bool launch_large<double>(const LargeArgs<double>&, const double2*, const double2*, double2*, double, int,
                                   cudaStream_t);
template bool launch_large<float>(const LargeArgs<float>&, const float2*, const float2*, float2*, double, int,
                                  cudaStream_t);
template void launch_large_upterm<double>(const LargeUpArgs<double>&, const double2*, double2*, cudaStream_t);
template void launch_large_upterm<float>(const LargeUpArgs<float>&, const float2*, float2*, cudaStream_t);

void launch_zgemm(const double2* x, const double2* h, double2* z, int logd, cudaStream_t s)
{
    zgemm_kernel<<<dim3(1u << (logd - 4), 1u << (logd - 5)), 256, 0, s>>>(x, h, z, logd);
}

void launch_ado0(const Ado0Args& a, const double2* u0, const float2* u, const double2* rho0, double2* out0,
                 float2* out32, double alpha, int base_kind, cudaStream_t s)
{
    const long long D2 = a.herm ? herm_elems(a.logd) : 1ll << (2 * a.logd);
    ado0_kernel<<<static_cast<unsigned>((D2 + 255) / 256), 256, 0, s>>>(a, u0, u, rho0, out0, out32, alpha, base_kind);
}

void launch_d2f(const double2* in, float2* out, long long n, cudaStream_t s)
{
    d2f_kernel<<<148 * 8, 256, 0, s>>>(in, out, n);
}

void launch_vec_d2f(const double* in, float* out, long long n, cudaStream_t s)
{
    vec_d2f_kernel<<<static_cast<unsigned>(n < 148 * 256 ? (n + 255) / 256 : 148), 256, 0, s>>>(in, out, n);
}

}  // namespace hx
