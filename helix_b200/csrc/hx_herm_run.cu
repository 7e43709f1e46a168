// Whole integrator steps in one launch for d = 32 and 64 on Hermitian-packed
// slabs, while the three state buffers stay in L2.
//
// Same mathematics as herm_kernel (hx_fused.cu): out_n = base_n + alpha L(u)_n
// for every ADO n, L being the reference right-hand side (getdRhoSparse,
// src/liouville.cu:749-869) for diagonal couplings.  With a launch for the up
// terms and one for the stage, a small hierarchy spends its time on the
// latency of dependent reads: 19 + 16 us a stage at d = 32, 816 ADOs, where the
// data would pass in 3.  Here the CTAs stay resident over all stages of a run:
//
//  * a CTA takes one ADO at a time, E packed elements per thread; ADOs are
//    dealt to the CTAs by their number of entries (a.order, most first, every
//    other round backwards), and MINB CTAs share an SM so that one reads
//    while the other computes;
//  * a thread asks for its elements of KB neighbour entries, of the slab and
//    of the Horner base at once, so one read latency covers them all; the
//    transverse field is worked out from the unpacked swizzled slab
//    (herm_kernel's layout) while they are under way.  Up neighbours are
//    entries like the others (they hit L2), so there is no up-term pass;
//  * a barrier over the grid separates the stages, and the last CTA only
//    watches (records rho_0 and the observables), as in small_step_kernel;
//  * a closure's term is a second diagonal coefficient of the top-tier ADOs.
//
// us per step, a launch per pass against a run: 92 and 25 at d = 32, 136 ADOs
// (a stage's 12,000 cycles: grid barrier 2,600, the slowest CTA's entries and
// flips the rest), 111 and 61 at 816 ADOs (bound by the 128 bytes a cycle of
// shared memory: 13 reads of 16 bytes per element for the flips), 168 and 115
// at d = 64, 325 ADOs.

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>

#include "hx_internal.h"
#include "hx_run.cuh"

namespace hx {

namespace {

template <int LOGD, int TS, int E, int KB, int MINB, bool PAULI>
__global__ void __launch_bounds__(TS, MINB)
    herm_run_kernel(FusedArgs a, RunClosure cl, double2* rho, double2* ua, double2* ub, double dt, int order,
                    int nsteps, int per, unsigned* gcount, StepWait w, double2* trace, double* obs)
{
    constexpr int D = 1 << LOGD, D2 = D * D, P = (D / 2) * (D + 1);
    constexpr bool kExact = P % TS == 0;
    extern __shared__ __align__(16) unsigned char smem[];
    const int M2 = 2 * a.M;
    double2* full = reinterpret_cast<double2*>(smem);     // [D2] unpacked slab
    double2* sW = full + D2;                              // [per][2M] commutator, anti-commutator weight
    double* sG = reinterpret_cast<double*>(sW + per * M2);  // [per]
    double* sH = sG + per;                                // [LOGD]
    double* sV = sH + LOGD;                               // [J][D] (general couplings)
    int2* sN = reinterpret_cast<int2*>(sV + (PAULI ? 0 : a.J * D));  // [per][2M] neighbour slab, spin or bath | flags
    int* sQ = reinterpret_cast<int*>(sN + per * M2);      // [per]
    int* sA = sQ + per;                                   // [per] the ADO, or -1
    int* sK = sA + per;                                   // [per] its slab of closure coefficients, or -1

    const int tid = threadIdx.x;
    const bool watch = trace != nullptr || obs != nullptr;
    const int G = static_cast<int>(gridDim.x);            // arrivals per barrier
    const int GC = G - (watch ? 1 : 0);                   // computing CTAs
    const bool watcher = watch && static_cast<int>(blockIdx.x) == GC;
    if (!watcher) {
        for (int j = tid; j < per; j += TS) {
            const int at = j * GC + ((j & 1) ? GC - 1 - static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x));
            const int n = at < a.H ? a.order[at] : -1;
            sA[j] = n;
            sQ[j] = n >= 0 ? a.ent_count[n] : 0;
            sG[j] = n >= 0 ? a.gsum[n] : 0.0;
            sK[j] = n >= 0 && cl.slot ? cl.slot[n] : -1;
        }
        if (!PAULI)
            for (int i = tid; i < a.J * D; i += TS) sV[i] = a.vdiag[i];
        if (tid < LOGD) sH[tid] = a.hflip[tid];
        __syncthreads();
        for (int i = tid; i < per * M2; i += TS) {
            const int j = i / M2, q = i - j * M2;
            if (q < sQ[j]) {
                const long long src = static_cast<long long>(sA[j]) * M2 + q;
                const int b = a.ent_bath[src] & 0xffff;
                const double wc = a.ent_wc[src], wa = a.ent_wa[src];
                sN[i] = make_int2(a.ent_slab[src] * P,
                                  (PAULI ? a.vbit[b] : b) | (wc != 0.0 ? 1 << 8 : 0) | (wa != 0.0 ? 1 << 9 : 0));
                sW[i] = PAULI ? make_double2(2.0 * wc, 2.0 * wa) : make_double2(wc, wa);
            }
        }
        __syncthreads();
    }

    // this thread's packed elements: row and column
    int rc[E];
#pragma unroll
    for (int k = 0; k < E; ++k) {
        int r = 0, c = 0;
        if (kExact || tid + TS * k < P) herm_coords(tid + TS * k, LOGD, r, c);
        rc[k] = (r << 8) | c;
    }

    double2 x[E], b[E];   // stage input, Horner base
    unsigned passed = 0;  // barriers
    double2* bufs[2] = {ua, ub};
    const double2* in = rho;
    for (int step = 0; step < nsteps; ++step) {
        for (int st = 1; st <= order; ++st) {
            const double alpha = dt / static_cast<double>(order - st + 1);
            double2* out = (st == order) ? rho : bufs[(st - 1) & 1];
            for (int j = 0; !watcher && j < per; ++j) {
                const int n = sA[j];
                if (n < 0) break;  // uniform
                const int o0 = n * P + tid;
                const int Q = sQ[j];
                const int2* nb = sN + j * M2;
                const double2* wt = sW + j * M2;
                const double2* ue = in + tid;
                double2 acc[E], y[KB][E];
                // a CTA's only ADO stays in its registers from stage to stage
                if (per > 1 || (step == 0 && st == 1)) {
#pragma unroll
                    for (int k = 0; k < E; ++k) {
                        x[k] = make_double2(0.0, 0.0);
                        if (kExact || tid + TS * k < P) x[k] = __ldcg(in + o0 + TS * k);
                    }
                }
                // whether entry p has a nonzero weight at this thread's element k
                auto need = [&](int2 p, int k) -> bool {
                    if (!kExact && tid + TS * k >= P) return false;
                    const int r = rc[k] >> 8, c = rc[k] & 255;
                    if (PAULI) return (p.y >> (9 - (((r ^ c) >> (p.y & 31)) & 1))) & 1;
                    const int v = (p.y & 255) * D;
                    const double vr = sV[v + r], vc = sV[v + c];
                    return (vr != vc && (p.y & (1 << 8))) || (vr + vc != 0.0 && (p.y & (1 << 9)));
                };
                auto ask = [&](int q0) {
#pragma unroll
                    for (int i = 0; i < KB; ++i) {
                        if (q0 + i >= Q) break;
                        const int2 p = nb[q0 + i];
#pragma unroll
                        for (int k = 0; k < E; ++k) {
                            y[i][k] = make_double2(0.0, 0.0);
                            if (need(p, k)) y[i][k] = __ldcg(ue + p.x + TS * k);
                        }
                    }
                };
                ask(0);
#pragma unroll
                for (int k = 0; k < E; ++k) {
                    if (st == 1) b[k] = x[k];
                    else if (per > 1 && (kExact || tid + TS * k < P)) b[k] = __ldcg(rho + o0 + TS * k);
                }
                const int ks = sK[j];
                const double g = sG[j];
                // ---- unpack the slab: (r, c) and its mirror (c, r) = conj
                if (j > 0) __syncthreads();  // the flips of the ADO before are done
#pragma unroll
                for (int k = 0; k < E; ++k)
                    if (kExact || tid + TS * k < P) {
                        const int r = rc[k] >> 8, c = rc[k] & 255;
                        full[(r << LOGD) | (c ^ (r & 7))] = x[k];
                        if (r != c) full[(c << LOGD) | (r ^ (c & 7))] = make_double2(x[k].x, -x[k].y);
                    }
                __syncthreads();
                // ---- diagonal and transverse field
#pragma unroll
                for (int k = 0; k < E; ++k) {
                    const int r = rc[k] >> 8, c = rc[k] & 255;
                    const int sl = (r << LOGD) | (c ^ (r & 7));
                    double hr = 0.0, hi = 0.0;
#pragma unroll
                    for (int f = 0; f < LOGD; ++f) {
                        const double h = sH[f];
                        const double2 rowp = full[sl ^ (1 << (LOGD + f)) ^ (f < 3 ? (1 << f) : 0)];
                        const double2 colp = full[sl ^ (1 << f)];
                        hr = fma(h, rowp.x - colp.x, hr);
                        hi = fma(h, rowp.y - colp.y, hi);
                    }
                    double2 T = make_double2(0.0, 0.0);
                    if (kExact || tid + TS * k < P) T = __ldg(a.diag + tid + TS * k);
                    T.x -= g;
                    if (ks >= 0 && (kExact || tid + TS * k < P)) {
                        const double2 kc = __ldg(cl.coef + static_cast<long long>(ks) * P + tid + TS * k);
                        T.x += kc.x;
                        T.y += kc.y;
                    }
                    acc[k].x = fma(T.x, x[k].x, fma(-T.y, x[k].y, hi));
                    acc[k].y = fma(T.x, x[k].y, fma(T.y, x[k].x, -hr));
                }
                // ---- neighbour entries
                for (int q0 = 0; q0 < Q; q0 += KB) {
                    if (q0 > 0) ask(q0);
#pragma unroll
                    for (int i = 0; i < KB; ++i) {
                        if (q0 + i >= Q) break;
                        const int2 p = nb[q0 + i];
                        const double2 ww = wt[q0 + i];
#pragma unroll
                        for (int k = 0; k < E; ++k) {
                            const int r = rc[k] >> 8, c = rc[k] & 255;
                            if (PAULI) {
                                // equal bits: -{V, y} wa; different bits: -i [V, y] wc (2 wc, 2 wa in ww)
                                const int bit = p.y & 31, br = (r >> bit) & 1;
                                if (!(p.y & (1 << 9))) {  // commutator only: y is zero where the bits agree
                                    const double wk = br ? -ww.x : ww.x;
                                    acc[k].x = fma(-wk, y[i][k].y, acc[k].x);
                                    acc[k].y = fma(wk, y[i][k].x, acc[k].y);
                                } else {
                                    const bool same = br == ((c >> bit) & 1);
                                    const double w2 = same ? ww.y : ww.x;
                                    const double wk = br ? -w2 : w2;
                                    acc[k].x = fma(wk, same ? y[i][k].x : -y[i][k].y, acc[k].x);
                                    acc[k].y = fma(wk, same ? y[i][k].y : y[i][k].x, acc[k].y);
                                }
                            } else {
                                const int v = (p.y & 255) * D;
                                const double vr = sV[v + r], vc = sV[v + c];
                                const double ar = -(vr + vc) * ww.y, ai = -(vr - vc) * ww.x;
                                acc[k].x = fma(ar, y[i][k].x, fma(-ai, y[i][k].y, acc[k].x));
                                acc[k].y = fma(ar, y[i][k].y, fma(ai, y[i][k].x, acc[k].y));
                            }
                        }
                    }
                }
                // ---- Horner epilogue
#pragma unroll
                for (int k = 0; k < E; ++k) {
                    x[k] = make_double2(fma(alpha, acc[k].x, b[k].x), fma(alpha, acc[k].y, b[k].y));
                    if (kExact || tid + TS * k < P) __stcg(out + o0 + TS * k, x[k]);
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
                run_gave_up(a.error_flag, w, nsteps, step, st == order);
                return;
            }
            if (watcher && st == order) {
                if (trace)
                    for (int i = tid; i < P; i += TS) trace[static_cast<long long>(step) * P + i] = __ldcg(rho + i);
                if (obs && tid < 32)
                    warp_observables<LOGD>(
                        a.hdiag, a.hflip, [&](int r, int c) { return __ldcg(rho + (r <= c ? herm_index(r, c, LOGD) : herm_index(c, r, LOGD))); },
                        obs + 3 * step);
            }
        }
    }
    grid_reset(gcount, watch, watcher, static_cast<unsigned>(nsteps * order));
}

// Shape of a run.
struct HermRunPlan {
    bool wide = false;  // d = 32: one CTA per SM holds every ADO, with more neighbour reads in flight
    int per = 0, grid = 0;
    size_t smem = 0;
};

constexpr size_t kHermRunSmem = 227 * 1024;

bool plan_herm_run(int logd, int M, int J, bool pauli, long long H, int sms, HermRunPlan& p)
{
    if ((logd != 5 && logd != 6) || sms < 2 || H < 1 || H * herm_elems(logd) > INT32_MAX) return false;
    p.wide = logd == 5 && H <= sms - 1;
    const int share = logd == 5 && !p.wide ? 2 : 1;  // CTAs per SM
    const long long ctas = static_cast<long long>(share) * sms - 1;  // and the watcher
    p.grid = static_cast<int>(std::min(H, ctas));
    p.per = static_cast<int>((H + p.grid - 1) / p.grid);
    const size_t D = size_t(1) << logd, per = static_cast<size_t>(p.per);
    p.smem = D * D * sizeof(double2) + per * 2 * M * (sizeof(double2) + sizeof(int2)) +
             sizeof(double) * (per + logd + (pauli ? 0 : J * D)) + sizeof(int) * 3 * per;
    return p.smem <= kHermRunSmem / share - 1024 * (share - 1);
}

template <int LOGD, int TS, int E, int KB, int MINB, bool PAULI>
int launch_herm_run_t(const HermRunPlan& p, const FusedArgs& a, const RunClosure& cl, double2* rho, double2* ua,
                      double2* ub, double dt, int order, int nsteps, unsigned* gcount, StepWait w, double2* trace,
                      double* obs, cudaStream_t s, bool dry)
{
    auto* kernel = herm_run_kernel<LOGD, TS, E, KB, MINB, PAULI>;
    if (dry) {  // creation: raise the shared-memory limit (a function attribute, not to be set in a capture)
        static std::atomic<bool> raised[64];
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
        if (raised[dev].load()) return 1;
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(kHermRunSmem / MINB)) != cudaSuccess)
            return -1;
        raised[dev].store(true);
        return 1;
    }
    FusedArgs args = a;
    RunClosure clo = cl;
    int per = p.per;
    void* params[] = {&args, &clo, &rho, &ua, &ub, &dt, &order, &nsteps, &per, &gcount, &w, &trace, &obs};
    const dim3 grid(static_cast<unsigned>(p.grid + (trace || obs ? 1 : 0)));
    return cudaLaunchCooperativeKernel(reinterpret_cast<void*>(kernel), grid, dim3(TS), params, p.smem, s) == cudaSuccess
               ? 1
               : -1;
}

}  // namespace

int launch_herm_run(const FusedArgs& a, const RunClosure& cl, double2* rho, double2* ua, double2* ub, double dt,
                    int order, int nsteps, unsigned* gcount, int sms, cudaStream_t s, bool dry, double2* trace,
                    double* obs, StepWait w)
{
    HermRunPlan p;
    if (order < 2) return 0;  // order 1 writes rho while neighbours read it
    if (!plan_herm_run(a.logd, a.M, a.J, a.pauli != 0, a.H, sms, p)) return 0;
#define HX_RUN(L, TS, E, KB, MINB)                                                                                    \
    (a.pauli ? launch_herm_run_t<L, TS, E, KB, MINB, true>(p, a, cl, rho, ua, ub, dt, order, nsteps, gcount, w,       \
                                                           trace, obs, s, dry)                                       \
             : launch_herm_run_t<L, TS, E, KB, MINB, false>(p, a, cl, rho, ua, ub, dt, order, nsteps, gcount, w,      \
                                                            trace, obs, s, dry))
    if (a.logd == 6) return HX_RUN(6, 704, 3, 2, 1);
    return p.wide ? HX_RUN(5, 544, 1, 16, 1) : HX_RUN(5, 544, 1, 4, 2);
#undef HX_RUN
}

// The line between a run and a launch per pass: a run saves the launches and
// the up-term pass, but its CTAs hide less latency than herm_kernel's.  us per
// step, launches against run: d = 32, 1.1 MiB of state 91 and 23, 6.6 MiB 106
// and 61, 13.8 MiB 120 and 105, 24 MiB 171 and 192, 31 MiB 226 and 235; d = 64,
// 6 MiB 134 and 60, 14.4 MiB 142 and 107, 23 MiB 160 and 169, so the line lies
// at 18 MiB for both.  (Runs of several contexts on several streams wait for
// one another, their launches overlap: 24 contexts of 816 ADOs at d = 32 take
// 59 us a step and context in runs and 37 without, of 136 ADOs 23 and 24;
// HX_SMALL_STEP=0 leaves the runs out, and a batch never uses them.)
bool herm_run_fits(int logd, int M, int J, int pauli, long long H, int sms)
{
    HermRunPlan p;
    const long long state = H * herm_elems(logd) * static_cast<long long>(sizeof(double2));
    return plan_herm_run(logd, M, J, pauli != 0, H, sms, p) && state <= 18ll << 20;
}

}  // namespace hx
