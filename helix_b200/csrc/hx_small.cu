// Kernels for small slabs (d <= 16): small_step_kernel, whole integrator steps
// in one launch, and small_kernel, one stage per launch with sigma_z couplings
// (single right-hand sides, and hierarchies too large for the resident CTAs).
//
// Same mathematics as stage_kernel (hx_stage.cu): small_kernel evaluates
// out_n = base_n + alpha L(u)_n for every ADO n, L being the reference
// right-hand side (getdRhoSparse, src/liouville.cu:749-869).  At d = 16 a
// slab is 256 elements (4 KB), so a stage is bound by the latency of its
// gathers, not by bandwidth.  The generic kernel walks baths and modes and
// waits on each neighbour read in turn; here every ADO carries the compacted
// neighbour entry list of the fused kernels (slab, spin bit, commutator and
// anti-commutator weight; up neighbours of every tier included), and each
// thread issues the reads of kBatch entries before it consumes any, so a
// stage costs a few L2 round trips instead of one per entry.
//
//  * one CTA per ADO, one thread per element (d^2 threads, at least a warp);
//  * the slab goes to shared memory once for the transverse-field flips;
//  * diagonal term from two d-entry tables: Re T = -4 sum_j xi_j
//    [bit_j(r) != bit_j(c)] (over r ^ c) and Im T = -(E_r - E_c);
//  * sigma_z weights from the index bits, as in the fused kernels.

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>

#include "hx_internal.h"
#include "hx_run.cuh"

namespace hx {

namespace {

constexpr int kBatch = 8;  // neighbour reads in flight per thread

// Sum over the spins of h_b (X_{r^b, c} - X_{r, c^b}) at element e of the slab xs.
template <int LOGD>
__device__ __forceinline__ double2 flip_sum(const double2* xs, int e, const double* h)
{
    double hr = 0.0, hi = 0.0;
#pragma unroll
    for (int b = 0; b < LOGD; ++b) {
        const double2 rp = xs[e ^ (1 << (LOGD + b))];
        const double2 cp = xs[e ^ (1 << b)];
        hr = fma(h[b], rp.x - cp.x, hr);
        hi = fma(h[b], rp.y - cp.y, hi);
    }
    return make_double2(hr, hi);
}

// (tr + i ti) x - i f
__device__ __forceinline__ double2 diag_term(double tr, double ti, double2 x, double2 f)
{
    return make_double2(fma(tr, x.x, fma(-ti, x.y, f.y)), fma(tr, x.y, fma(ti, x.x, -f.x)));
}

// One neighbour entry with a sigma_z coupling on spin `bit`: -{V, y} wa where
// the bits of r and c agree, -i [V, y] wc where they differ (wc2, wa2: twice
// the weights).
__device__ __forceinline__ void add_entry(double2& acc, int r, int c, int bit, double wc2, double wa2, double2 y)
{
    const int br = (r >> bit) & 1;
    const bool same = br == ((c >> bit) & 1);
    const double w2 = same ? wa2 : wc2;
    const double w = br ? -w2 : w2;
    acc.x = fma(w, same ? y.x : -y.y, acc.x);
    acc.y = fma(w, same ? y.y : y.x, acc.y);
}

template <int LOGD>
__global__ void __launch_bounds__((1 << (2 * LOGD)) < 32 ? 32 : (1 << (2 * LOGD)))
    small_kernel(FusedArgs a, const double2* __restrict__ u, const double2* rho, double2* out, double alpha,
                 int base_kind)
{
    constexpr int D = 1 << LOGD, D2 = D * D;
    extern __shared__ __align__(16) unsigned char smem[];
    double2* sx = reinterpret_cast<double2*>(smem);  // [D2]
    double* sE = reinterpret_cast<double*>(sx + D2);  // [D]
    double* sX = sE + D;                              // [D]
    double* sH = sX + D;                              // [LOGD]
    double* sWc = sH + LOGD;                          // [2M]
    double* sWa = sWc + 2 * a.M;                      // [2M]
    int* sSlab = reinterpret_cast<int*>(sWa + 2 * a.M);
    int* sBit = sSlab + 2 * a.M;

    const int tid = threadIdx.x;
    const long long n = static_cast<long long>(blockIdx.x);
    const bool active = tid < D2;
    const int e = active ? tid : 0;
    const int r = e >> LOGD, c = e & (D - 1);
    const double2 x = active ? __ldg(u + n * D2 + e) : make_double2(0.0, 0.0);
    if (active) sx[e] = x;
    const int Q = a.ent_count[n];
    for (int q = tid; q < Q; q += blockDim.x) {
        const long long src = n * 2 * a.M + q;
        sSlab[q] = a.ent_slab[src];
        sBit[q] = a.vbit[a.ent_bath[src] & 0xffff];
        sWc[q] = a.ent_wc[src];
        sWa[q] = a.ent_wa[src];
    }
    if (tid < D) {
        sE[tid] = a.hdiag[tid];
        double s = 0.0;
        for (int j = 0; j < a.J; ++j)
            if ((tid >> a.vbit[j]) & 1) s += a.xi[j];
        sX[tid] = 4.0 * s;
    }
    if (tid < LOGD) sH[tid] = a.hflip[tid];
    const double g = a.gsum[n];
    __syncthreads();
    if (!active) return;

    // diagonal and transverse field
    double2 acc = diag_term(-sX[r ^ c] - g, sE[c] - sE[r], x, flip_sum<LOGD>(sx, e, sH));

    // neighbour entries, kBatch reads in flight
    const double2* ue = u + e;
    for (int q0 = 0; q0 < Q; q0 += kBatch) {
        double2 y[kBatch];
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
            const int q = q0 + i;
            y[i] = make_double2(0.0, 0.0);
            if (q < Q) {
                const int bit = sBit[q];
                const bool same = ((r >> bit) & 1) == ((c >> bit) & 1);
                if (same ? sWa[q] != 0.0 : sWc[q] != 0.0) y[i] = __ldg(ue + static_cast<long long>(sSlab[q]) * D2);
            }
        }
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
            const int q = q0 + i;
            if (q < Q) add_entry(acc, r, c, sBit[q], 2.0 * sWc[q], 2.0 * sWa[q], y[i]);
        }
    }

    double2 base = make_double2(0.0, 0.0);
    if (base_kind == kBaseSelf) base = x;
    else if (base_kind == kBaseRho) base = __ldcs(rho + n * D2 + e);
    __stcs(out + n * D2 + e, make_double2(fma(alpha, acc.x, base.x), fma(alpha, acc.y, base.y)));
}

template <int LOGD>
void launch_small_t(const FusedArgs& a, const double2* u, const double2* rho, double2* out, double alpha, int base,
                    cudaStream_t s)
{
    constexpr int D = 1 << LOGD, D2 = D * D;
    const int threads = D2 < 32 ? 32 : D2;
    const size_t smem = small_smem(LOGD, a.M);
    small_kernel<LOGD><<<static_cast<unsigned>(a.H), threads, smem, s>>>(a, u, rho, out, alpha, base);
}

// Elements of a slab that one thread of small_step_kernel owns, and threads per slab.
template <int LOGD> struct RunShape {
    static constexpr int E = LOGD == 4 ? 2 : 1;
    static constexpr int TA = (1 << (2 * LOGD)) / E;
};
constexpr int kRunThreads = 512;
constexpr int kRunBatch = 4;  // staged entries read back side by side

// A run of whole integrator steps (all m Horner stages of each) for small
// slabs in one launch, with the observables and the rho_0 trace of every step.
// A stage of these hierarchies is a few microseconds of dependent latency
// (neighbour reads through L2, one exchange of the slab in shared memory, one
// barrier over the grid), so what pays is to do nothing else between stages:
//
//  * one CTA per SM holds apc slabs at a time, per times; the stage input, the
//    stage output and the Horner base of its own slabs stay in shared memory
//    for the whole run, its tables too.  114 arrivals at a barrier instead of
//    455 (d = 16, 455 ADOs) and no launch between steps;
//  * a read of a slab that another SM has just written takes about 1,500
//    cycles, so a thread asks for every neighbour element it will need at
//    once (cp.async into its own places of a staging area, no registers held,
//    no barrier to read them back) and works out the transverse field of its
//    own slab meanwhile.  Four entries at a time in registers cost 7,300
//    cycles for the 14 entries of a tier L-1 ADO;
//  * ADOs are dealt to the CTAs by their number of entries (a.order, most
//    first): a CTA that drew several of tier L-1 made the others wait;
//  * the last CTA only watches: after the barrier that ends a step it copies
//    rho_0 and reduces the observables while the others are in the next step,
//    so a recorded step costs what an unrecorded one does.  It arrives at
//    every barrier, so rho is not rewritten under it;
//  * SOLO: a hierarchy of at most kSoloElems elements stays in one CTA, its
//    neighbour reads go to shared memory and the barriers are block barriers
//    (an extra warp does the watching).
//
// Per step at d = 16, 455 ADOs with every step recorded: 37.2 us with a launch
// per step and a pass for the observables, 20.5 us here (of a stage's 9,300
// cycles the grid barrier takes 2,600, the slowest CTA's entries 4,900); one
// recorded step of 15 ADOs at d = 4, call to result: 54 -> 32 us.
// Per ADO the arithmetic is small_kernel's, in the same order (PAULI), so the
// two give the same bits.  Without PAULI the couplings are general diagonals
// and the diagonal term comes from the table a.diag.
template <int LOGD, bool PAULI, bool SOLO>
__global__ void __launch_bounds__(kRunThreads, 1)
    small_step_kernel(FusedArgs a, RunClosure cl, double2* rho, double2* ua, double2* ub, double dt, int order, int nsteps,
                     int apc, int per, int cap, unsigned* gcount, StepWait w, double2* trace, double* obs)
{
    constexpr int D = 1 << LOGD, D2 = D * D, E = RunShape<LOGD>::E, TA = RunShape<LOGD>::TA;
    extern __shared__ __align__(16) unsigned char smem[];
    const int NL = per * apc, TP = NL * D2, M2 = 2 * a.M;
    double2* sx = reinterpret_cast<double2*>(smem);      // [2][TP] stage input, stage output
    double2* sb = sx + 2 * TP;                           // [TP] Horner base
    double2* sS = sb + TP;                               // [cap][D2] staged neighbour slabs
    double2* sW = sS + (SOLO ? 0 : cap * D2);                             // [NL][2M] commutator, anti-commutator weight
    double* sG = reinterpret_cast<double*>(sW + NL * M2);  // [NL]
    double* sH = sG + NL;                                // [LOGD]
    double* sV = sH + LOGD;                              // PAULI: E[D], X[D]; else [J][D]
    int2* sN = reinterpret_cast<int2*>(sV + (PAULI ? 2 * D : a.J * D));  // [NL][2M] neighbour's first element, spin or bath
    int* sQ = reinterpret_cast<int*>(sN + NL * M2);      // [NL]
    int* sA = sQ + NL;                                   // [NL] the ADO of each local slab, or -1
    int* sK = sA + NL;                                   // [NL] its slab of closure coefficients, or -1
    int* sO = sK + NL;                                   // [apc] first staging place of each group of TA threads
    int* sC = sO + apc;                                  // [apc] entries it stages at a time

    const int tid = threadIdx.x;
    const bool watch = trace != nullptr || obs != nullptr;
    const int G = static_cast<int>(gridDim.x);           // arrivals per barrier
    const int GC = SOLO ? 1 : G - (watch ? 1 : 0);       // computing CTAs
    const bool watcher = watch && (SOLO ? tid >= static_cast<int>(blockDim.x) - 32
                                        : static_cast<int>(blockIdx.x) == GC);
    const bool active = tid < apc * TA && !watcher;
    const int la = tid / TA, lg = tid & (TA - 1);
    const int c = lg & (D - 1);
    int m[E], rr[E];  // of element lg + TA k: row ^ column, row
#pragma unroll
    for (int k = 0; k < E; ++k) {
        rr[k] = (lg + TA * k) >> LOGD;
        m[k] = rr[k] ^ c;
    }

    if (SOLO || !watcher) {
        for (int l = tid; l < NL; l += blockDim.x) {
            const int at = l * GC + static_cast<int>(blockIdx.x);
            const int n = at < a.H ? (SOLO ? at : a.order[at]) : -1;
            sA[l] = n;
            sQ[l] = n >= 0 ? a.ent_count[n] : 0;
            sG[l] = n >= 0 ? a.gsum[n] : 0.0;
            sK[l] = n >= 0 && cl.slot ? cl.slot[n] : -1;
        }
        if (PAULI) {
            if (tid < D) {
                sV[tid] = a.hdiag[tid];
                double s = 0.0;
                for (int j = 0; j < a.J; ++j)
                    if ((tid >> a.vbit[j]) & 1) s += a.xi[j];
                sV[D + tid] = 4.0 * s;
            }
        } else {
            for (int i = tid; i < a.J * D; i += blockDim.x) sV[i] = a.vdiag[i];
        }
        if (tid < LOGD) sH[tid] = a.hflip[tid];
        __syncthreads();
        for (int i = tid; i < NL * M2; i += blockDim.x) {
            const int l = i / M2, q = i - l * M2;
            if (q < sQ[l]) {
                const long long src = static_cast<long long>(sA[l]) * M2 + q;
                const int j = a.ent_bath[src] & 0xffff;
                const double wc = a.ent_wc[src], wa = a.ent_wa[src];
                // spin (or bath), and whether the commutator and the anti-commutator weight are nonzero
                sN[i] = make_int2(a.ent_slab[src] * D2,
                                  (PAULI ? a.vbit[j] : j) | (wc != 0.0 ? 1 << 8 : 0) | (wa != 0.0 ? 1 << 9 : 0));
                sW[i] = PAULI ? make_double2(2.0 * wc, 2.0 * wa) : make_double2(wc, wa);
            }
        }
        if (!SOLO && tid == 0) {
            // a thread group keeps its places for all its slabs (they are its own threads' only); every
            // entry of the largest of them when that fits for all groups together, else equal shares
            int sum = 0;
            for (int k = 0; k < apc; ++k) {
                int most = 1;
                for (int j = 0; j < per; ++j) most = max(most, sQ[j * apc + k]);
                sO[k] = sum;
                sC[k] = most;
                sum += most;
            }
            for (int k = 0; sum > cap && k < apc; ++k) {
                sC[k] = cap / apc;
                sO[k] = k * sC[k];
            }
        }
        for (int i = tid; i < TP; i += blockDim.x) {
            const int n = sA[i / D2];
            if (n >= 0) sx[i] = sb[i] = __ldcg(rho + n * D2 + (i & (D2 - 1)));
        }
        __syncthreads();
    }
    double tr0[E], ti[E];
#pragma unroll
    for (int k = 0; k < E; ++k) {
        tr0[k] = ti[k] = 0.0;
        if (active) {
            if (PAULI) {
                tr0[k] = -sV[D + m[k]];
                ti[k] = sV[c] - sV[rr[k]];
            } else {
                const double2 t = __ldg(a.diag + lg + TA * k);
                tr0[k] = t.x;
                ti[k] = t.y;
            }
        }
    }

    int cur = 0;
    unsigned passed = 0;  // barriers
    double2* bufs[2] = {ua, ub};
    const double2* in = rho;
    for (int step = 0; step < nsteps; ++step) {
        for (int st = 1; st <= order; ++st) {
            const double alpha = dt / static_cast<double>(order - st + 1);
            double2* out = (st == order) ? rho : bufs[(st - 1) & 1];
            const double2* xin = sx + cur * TP;
            double2* xout = sx + (cur ^ 1) * TP;
            if (SOLO && watcher && st == 1 && step > 0) {
                // xin of this stage is the state after the step before
                if (trace)
                    for (int i = tid & 31; i < D2; i += 32) trace[static_cast<long long>(step - 1) * D2 + i] = xin[i];
                if (obs) warp_observables<LOGD>(a.hdiag, a.hflip, [&](int r0, int c0) { return xin[(r0 << LOGD) + c0]; }, obs + 3 * (step - 1));
            }
            for (int j = 0; active && j < per; ++j) {
                const int l = j * apc + la;
                const int n = sA[l];
                if (n < 0) break;
                const double2* xs = xin + l * D2;
                const double g = sG[l];
                const int Q = sQ[l];
                const int2* nb = sN + l * M2;
                const double2* wt = sW + l * M2;
                const double2* ue = (SOLO ? xin : in) + lg;
                double2* mine = SOLO ? nullptr : sS + sO[la] * D2 + lg;
                const uint32_t mine32 = SOLO ? 0u : static_cast<uint32_t>(__cvta_generic_to_shared(mine));
                const int C = SOLO ? Q : sC[la];
                // whether entry p has a nonzero weight at this thread's element k
                auto need = [&](int2 p, int k) -> bool {
                    if (PAULI) return (p.y >> (((m[k] >> (p.y & 31)) & 1) ? 8 : 9)) & 1;
                    const int v = (p.y & 255) * D;
                    const double vr = sV[v + rr[k]], vc = sV[v + c];
                    return (vr != vc && (p.y & (1 << 8))) || (vr + vc != 0.0 && (p.y & (1 << 9)));
                };
                auto ask = [&](int q0) {
                    const int q1 = min(Q, q0 + C);
#pragma unroll 4
                    for (int q = q0; q < q1; ++q) {
                        const int2 p = nb[q];
#pragma unroll
                        for (int k = 0; k < E; ++k)
                            if (need(p, k))
                                cp_async16(mine32 + static_cast<uint32_t>((q - q0) * D2 + TA * k) * 16u, ue + p.x + TA * k);
                    }
                };
                if (!SOLO) ask(0);
                double2 x[E], acc[E], kc[E];
                const int ks = sK[l];
#pragma unroll
                for (int k = 0; k < E; ++k) {
                    x[k] = xs[lg + TA * k];
                    kc[k] = ks >= 0 ? __ldg(cl.coef + ks * D2 + lg + TA * k) : make_double2(0.0, 0.0);
                }
#pragma unroll
                for (int k = 0; k < E; ++k) {
                    // flips of the rows that this thread owns too are in registers
                    double hr = 0.0, hi = 0.0;
#pragma unroll
                    for (int b = 0; b < LOGD; ++b) {
                        const int step_b = 1 << (LOGD + b);  // element distance of the row flip
                        const double2 rp = step_b >= TA ? x[(k ^ (step_b / TA)) & (E - 1)] : xs[(lg + TA * k) ^ step_b];
                        const double2 cp = xs[(lg + TA * k) ^ (1 << b)];
                        hr = fma(sH[b], rp.x - cp.x, hr);
                        hi = fma(sH[b], rp.y - cp.y, hi);
                    }
                    acc[k] = diag_term(tr0[k] - g + kc[k].x, ti[k] + kc[k].y, x[k], make_double2(hr, hi));
                }
                for (int q0 = 0; q0 < Q; q0 += C) {
                    if (!SOLO) {
                        if (q0 > 0) ask(q0);
                        cp_async_wait();
                    }
                    const int q1 = min(Q, q0 + C);
                    for (int qb = q0; qb < q1; qb += kRunBatch) {
                        double2 y[kRunBatch][E], ww[kRunBatch];
                        int2 p[kRunBatch];
#pragma unroll
                        for (int i = 0; i < kRunBatch; ++i) {
                            const int q = min(qb + i, q1 - 1);
                            p[i] = nb[q];
                            ww[i] = wt[q];
#pragma unroll
                            for (int k = 0; k < E; ++k) {
                                y[i][k] = make_double2(0.0, 0.0);
                                if (qb + i < q1 && need(p[i], k))
                                    y[i][k] = SOLO ? ue[p[i].x + TA * k] : mine[(q - q0) * D2 + TA * k];
                            }
                        }
#pragma unroll
                        for (int i = 0; i < kRunBatch; ++i)
#pragma unroll
                            for (int k = 0; k < E; ++k) {
                                if (PAULI) {
                                    add_entry(acc[k], rr[k], c, p[i].y & 31, ww[i].x, ww[i].y, y[i][k]);
                                } else {
                                    const int v = (p[i].y & 255) * D;
                                    const double vr = sV[v + rr[k]], vc = sV[v + c];
                                    const double ar = -(vr + vc) * ww[i].y, ai = -(vr - vc) * ww[i].x;
                                    acc[k].x = fma(ar, y[i][k].x, fma(-ai, y[i][k].y, acc[k].x));
                                    acc[k].y = fma(ar, y[i][k].y, fma(ai, y[i][k].x, acc[k].y));
                                }
                            }
                    }
                }
#pragma unroll
                for (int k = 0; k < E; ++k) {
                    const int i = l * D2 + lg + TA * k;
                    const double2 b = sb[i];
                    const double2 o = make_double2(fma(alpha, acc[k].x, b.x), fma(alpha, acc[k].y, b.y));
                    if (!SOLO) __stcg(out + n * D2 + lg + TA * k, o);
                    xout[i] = o;
                    if (st == order) sb[i] = o;
                }
            }
            cur ^= 1;
            in = out;
            if (SOLO) {
                __syncthreads();
                continue;
            }
            const bool last = step + 1 == nsteps && st == order;
            if (last && !watcher) {
                if (watch) grid_arrive(gcount);  // the watcher waits for the last state; nobody else does
                break;
            }
            ++passed;
            if (!grid_barrier(gcount, passed, w)) {
                run_gave_up(a.error_flag, w, nsteps, step, st == order);
                return;
            }
            if (watcher && st == order) {
                if (trace)
                    for (int i = tid; i < D2; i += blockDim.x) trace[static_cast<long long>(step) * D2 + i] = __ldcg(rho + i);
                if (obs && tid < 32)
                    warp_observables<LOGD>(a.hdiag, a.hflip, [&](int r0, int c0) { return __ldcg(rho + (r0 << LOGD) + c0); }, obs + 3 * step);
            }
        }
    }
    if (SOLO) {
        const double2* xs = sx + cur * TP;
        for (int i = tid; i < a.H * D2; i += blockDim.x) rho[i] = xs[i];
        if (watcher) {
            if (trace)
                for (int i = tid & 31; i < D2; i += 32) trace[static_cast<long long>(nsteps - 1) * D2 + i] = xs[i];
            if (obs) warp_observables<LOGD>(a.hdiag, a.hflip, [&](int r0, int c0) { return xs[(r0 << LOGD) + c0]; }, obs + 3 * (nsteps - 1));
        }
        return;
    }
    grid_reset(gcount, watch, watcher, static_cast<unsigned>(nsteps * order));
}

// order[k] = the ADO with the k-th most entries (ties by index): ranks by
// counting, one thread per ADO, once per context.  A hundred thousand ADOs at most fit a run (d = 2).
__global__ void run_order_kernel(const int* __restrict__ count, int H, int32_t* order)
{
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= H) return;
    const int q = count[n];
    int rank = 0;
    for (int i = 0; i < H; ++i) {
        const int qi = __ldg(count + i);
        rank += (qi > q || (qi == q && i < n)) ? 1 : 0;
    }
    order[rank] = n;
}

// Shape of a run: one CTA while a stage in it costs less than a barrier over
// the grid (us per step, one CTA against the grid: 4.8 and 9.7 at 280
// elements, 8.9 and 10.1 at 960, 12.2 and 11.2 at 1344, 13.6 and 10.8 at
// 1792, so the line lies near 1000), else one CTA per SM, at least 256 elements in each (fewer arrivals), and as few
// slabs one after the other as kRunThreads allow.
struct RunPlan {
    int apc = 0, per = 0, cap = 0, grid = 0, threads = 0;
    bool solo = false;
    size_t smem = 0;
};

constexpr int kSoloElems = 1024;
constexpr size_t kRunSmem = 227 * 1024;

size_t run_smem(int logd, int M, int J, bool pauli, int apc, int per)
{
    const size_t D = size_t(1) << logd, NL = static_cast<size_t>(apc) * per;
    return 3 * NL * D * D * sizeof(double2) + NL * 2 * M * (sizeof(double2) + sizeof(int2)) +
           sizeof(double) * (NL + logd + (pauli ? 2 * D : J * D)) + sizeof(int) * (3 * NL + 2 * apc);
}

bool plan_run(int logd, int M, int J, bool pauli, long long H, int sms, bool solo, RunPlan& p)
{
    const int d2 = 1 << (2 * logd);
    const int ta = logd == 4 ? RunShape<4>::TA : d2;  // threads per slab
    if (solo && H * d2 <= kSoloElems) {
        p.apc = static_cast<int>(std::min<long long>(H, (kRunThreads - 32) / ta));
        p.per = static_cast<int>((H + p.apc - 1) / p.apc);
        p.solo = true;
        p.grid = 1;
        p.threads = ((p.apc * ta + 31) & ~31) + 32;
        p.smem = run_smem(logd, M, J, pauli, p.apc, p.per);
        if (p.smem <= kRunSmem) return true;
    }
    const int ctas = sms - 1;  // and the watcher
    if (ctas < 1) return false;
    const int most = kRunThreads / ta;
    const long long each = std::max<long long>((H + ctas - 1) / ctas, std::max(1, 256 / d2));
    if (each > 64ll * most) return false;
    p.per = static_cast<int>((each + most - 1) / most);
    // general couplings read their weights per element and entry, and one round of slabs is what a run gains on
    // them: us a step, run against a launch per stage, d = 16, one bath, 495 ADOs 29 and 37, 715 (two rounds) 42
    // and 37, 1716 71 and 59; d = 8 924 22 and 34, 3003 (three rounds) 45 and 42
    if (!pauli && p.per > 1) return false;
    p.apc = static_cast<int>((each + p.per - 1) / p.per);
    p.solo = false;
    p.grid = static_cast<int>((H + static_cast<long long>(p.apc) * p.per - 1) / (static_cast<long long>(p.apc) * p.per));
    p.threads = (p.apc * ta + 31) & ~31;
    p.smem = run_smem(logd, M, J, pauli, p.apc, p.per);
    if (p.smem > kRunSmem) return false;
    // staging: every entry that the slabs in hand can have, or what is left of the shared memory
    const size_t slab = static_cast<size_t>(d2) * sizeof(double2);
    p.cap = static_cast<int>(std::min<size_t>(static_cast<size_t>(p.apc) * 2 * M, (kRunSmem - p.smem) / slab));
    p.smem += p.cap * slab;
    // with less room than three entries per slab in hand the run waits on every entry by itself: d = 16, 12 modes,
    // 1820 ADOs 120 us a step, 68 with a launch per stage; 1716 ADOs, where 18 entries fit, 47 and 67
    return p.cap >= std::min(3, 2 * M) * p.apc;  // (one mode has two entries at most)
}

template <int LOGD, bool PAULI, bool SOLO>
int launch_run_t(const RunPlan& p, const FusedArgs& a, const RunClosure& cl, double2* rho, double2* ua, double2* ub, double dt, int order,
                 int nsteps, unsigned* gcount, StepWait w, double2* trace, double* obs, cudaStream_t s)
{
    auto* kernel = small_step_kernel<LOGD, PAULI, SOLO>;
    FusedArgs args = a;
    RunClosure clo = cl;
    int apc = p.apc, per = p.per, cap = p.cap;
    void* params[] = {&args, &clo, &rho, &ua, &ub, &dt, &order, &nsteps, &apc, &per, &cap, &gcount, &w, &trace, &obs};
    const dim3 grid(static_cast<unsigned>(p.grid + (!SOLO && (trace || obs) ? 1 : 0))), block(static_cast<unsigned>(p.threads));
    const cudaError_t e = SOLO ? cudaLaunchKernel(reinterpret_cast<void*>(kernel), grid, block, params, p.smem, s)
                               : cudaLaunchCooperativeKernel(reinterpret_cast<void*>(kernel), grid, block, params, p.smem, s);
    return e == cudaSuccess ? 1 : -1;
}

template <int LOGD>
int launch_run_d(const RunPlan& p, const FusedArgs& a, const RunClosure& cl, double2* rho, double2* ua, double2* ub, double dt, int order,
                 int nsteps, unsigned* gcount, StepWait w, double2* trace, double* obs, cudaStream_t s, bool dry)
{
    if (dry) {  // creation: raise the shared-memory limits (function attributes, not to be set in a capture)
        static std::atomic<bool> raised[2][64];  // by couplings, device
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
        if (raised[a.pauli ? 1 : 0][dev].load()) return 1;
        auto raise = [](const void* f) {
            return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kRunSmem)) ==
                   cudaSuccess;
        };
        const bool ok = a.pauli ? raise(reinterpret_cast<const void*>(small_step_kernel<LOGD, true, true>)) &&
                                      raise(reinterpret_cast<const void*>(small_step_kernel<LOGD, true, false>))
                                : raise(reinterpret_cast<const void*>(small_step_kernel<LOGD, false, true>)) &&
                                      raise(reinterpret_cast<const void*>(small_step_kernel<LOGD, false, false>));
        if (ok) raised[a.pauli ? 1 : 0][dev].store(true);
        return ok ? 1 : -1;
    }
    if (a.pauli)
        return p.solo ? launch_run_t<LOGD, true, true>(p, a, cl, rho, ua, ub, dt, order, nsteps, gcount, w, trace, obs, s)
                      : launch_run_t<LOGD, true, false>(p, a, cl, rho, ua, ub, dt, order, nsteps, gcount, w, trace, obs, s);
    return p.solo ? launch_run_t<LOGD, false, true>(p, a, cl, rho, ua, ub, dt, order, nsteps, gcount, w, trace, obs, s)
                  : launch_run_t<LOGD, false, false>(p, a, cl, rho, ua, ub, dt, order, nsteps, gcount, w, trace, obs, s);
}

}  // namespace

size_t small_smem(int logd, int M)
{
    const size_t D = size_t(1) << logd;
    return D * D * sizeof(double2) + sizeof(double) * (2 * D + logd + 4 * M) + sizeof(int) * 4 * M;
}

bool small_supported(int logd, int M, int pauli) { return pauli && logd >= 1 && logd <= 4 && small_smem(logd, M) <= 48 * 1024; }

int launch_small_run(const FusedArgs& a, const RunClosure& cl, double2* rho, double2* ua, double2* ub, double dt, int order, int nsteps,
                     unsigned* gcount, int sms, cudaStream_t s, bool dry, double2* trace, double* obs, StepWait w)
{
    RunPlan p;
    if (order < 2) return 0;  // order 1 writes rho while neighbours read it
    // a wait that is to run out needs the grid barriers
    if (!plan_run(a.logd, a.M, a.J, a.pauli != 0, a.H, sms, w.skew == 0, p)) return 0;
    switch (a.logd) {
    case 1: return launch_run_d<1>(p, a, cl, rho, ua, ub, dt, order, nsteps, gcount, w, trace, obs, s, dry);
    case 2: return launch_run_d<2>(p, a, cl, rho, ua, ub, dt, order, nsteps, gcount, w, trace, obs, s, dry);
    case 3: return launch_run_d<3>(p, a, cl, rho, ua, ub, dt, order, nsteps, gcount, w, trace, obs, s, dry);
    case 4: return launch_run_d<4>(p, a, cl, rho, ua, ub, dt, order, nsteps, gcount, w, trace, obs, s, dry);
    default: return 0;
    }
}

void launch_run_order(const int* ent_count, long long H, int32_t* order, cudaStream_t s)
{
    run_order_kernel<<<static_cast<unsigned>((H + 127) / 128), 128, 0, s>>>(ent_count, static_cast<int>(H), order);
}

bool launch_small(const FusedArgs& a, const double2* u, const double2* rho, double2* out, double alpha, int base_kind,
                  cudaStream_t s)
{
    switch (a.logd) {
    case 1: launch_small_t<1>(a, u, rho, out, alpha, base_kind, s); return true;
    case 2: launch_small_t<2>(a, u, rho, out, alpha, base_kind, s); return true;
    case 3: launch_small_t<3>(a, u, rho, out, alpha, base_kind, s); return true;
    case 4: launch_small_t<4>(a, u, rho, out, alpha, base_kind, s); return true;
    default: return false;
    }
}

}  // namespace hx
