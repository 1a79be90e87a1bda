// One Arnoldi step's classical Gram-Schmidt in a single cooperative kernel
// (pamp.h:317-345 without re-orthogonalisation; BLASIntegrationFunctor block
// InnerProduct + zgemv + norm, functors.h:182-241):
//     h = V_{0..J}^H w,   w <- w - V h,   beta = ||w||,   Hessenberg column J, breakdown test.
// The grid has up to one CTA per SM (co-resident by the cooperative launch).  CTA b owns the
// element chunk [b*C, (b+1)*C) of every basis vector: it reads its chunk of V once into
// shared memory (when it fits), forms its partial inner products, and after a grid
// barrier every CTA sums all CTAs' partials (as integers: the same h everywhere), updates its chunk of w from the cached V and writes its share of
// ||w||^2; CTA 0 writes the Hessenberg column and the counters.  beta = ||w|| is formed from
// those shares by the next solve, the first kernel that needs it (see launch_solve_inv).
// Versus separate dot / update / finalize kernels this reads V once instead of twice and
// removes two launches and two last-block reductions per Arnoldi step.
#include "gbprop_internal.h"
#include "gbprop_device.cuh"

#include <algorithm>
#include <cfloat>

namespace gbprop {

constexpr int kFuseThreads = 512;
constexpr int kCgsMaxGrid = 256;               // partial sums per value (see to_fixed)
constexpr long kBarrierSpinLimit = 1L << 24;   // polls (each an L2 round trip) before a barrier gives up

// Grid barrier for a co-resident grid on a counter that only grows within an Arnoldi step
// (zeroed before the step's first launch): barrier number t of the step completes when the
// counter reaches (t + 1) * nblocks.  One acquire-release atomic per CTA and acquire polls
// (1.2 us per barrier over 152 CTAs, against 2.3 us with full fences around a volatile
// sense flag).  Bounded: after kBarrierSpinLimit polls (or the handle's Ctrl::wait_limit, see
// wait_budget) it records ctrl->wait_timeout and returns false.
__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ bool grid_barrier(unsigned* bar, unsigned nblocks, unsigned t, Ctrl* ctrl) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        unsigned old;
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(bar) : "memory");
        const unsigned target = (t + 1) * nblocks;
        const long lim = wait_budget(ctrl, kBarrierSpinLimit);
        long it = 0;
        while ((int)(ld_acquire_gpu(bar) - target) < 0) {
            if (++it > lim) {
                ctrl->wait_timeout = 1;
                ok = 0;
                break;
            }
        }
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// complex conj(v) * x accumulated in FP64
__device__ __forceinline__ void acc_dot64(double& ar, double& ai, double vr, double vi, double xr, double xi) {
    ar = fma(vr, xr, ar);
    ar = fma(vi, xi, ar);
    ai = fma(vr, xi, ai);
    ai = fma(-vi, xr, ai);
}

// Phase C (CTA 0): the Hessenberg column J and the counters (pamp.h:305-345).  beta of the next
// vector, its breakdown test and 1/beta are formed from the ||w||^2 partials by the next solve
// (the first kernel that needs them), which saves a grid barrier here; H(J, J-1) = beta_J,
// recorded by the solve of this Arnoldi step, is written now.
__device__ __forceinline__ void cgs_finish(Ctrl* ctrl, double* H, const double* hs, int m, int J, int b) {
    if (b != 0) return;
    const int nv = J + 1;
    for (int k = threadIdx.x; k < nv; k += blockDim.x) {
        H[2 * ((size_t)k * m + J)] = hs[2 * k];
        H[2 * ((size_t)k * m + J) + 1] = hs[2 * k + 1];
        ctrl->h[2 * k] = hs[2 * k];
        ctrl->h[2 * k + 1] = hs[2 * k + 1];
    }
    if (threadIdx.x == 0) {
        ctrl->nbasis = nv;
        ctrl->operator_count++;
        if (J == 0) ctrl->inner_product_count++;
        if (J > 0) {
            H[2 * ((size_t)J * m + J - 1)] = ctrl->beta;
            H[2 * ((size_t)J * m + J - 1) + 1] = 0.0;
        }
    }
}

// The end of a step with re-orthogonalisation (CTA 0; its warp 0 holds the norms): the column, the
// counters, the next beta and its breakdown test, as launch_arnoldi_finalize leaves them.
__device__ __forceinline__ void cgs_finish_dorth(Ctrl* ctrl, double* H, const double* ht, unsigned* bar, unsigned tb,
                                                 int m, int J, int b, int passes, int again, double pre2, double orig2,
                                                 double resid2, double brk_tol) {
    const int nv = J + 1;
    if (b != 0) return;
    for (int k = threadIdx.x; k < nv; k += kFuseThreads) {
        H[2 * ((size_t)k * m + J)] = ht[2 * k];
        H[2 * ((size_t)k * m + J) + 1] = ht[2 * k + 1];
        ctrl->h[2 * k] = ht[2 * k];
        ctrl->h[2 * k + 1] = ht[2 * k + 1];
    }
    if (threadIdx.x != 0) return;
    const double resid = sqrt(resid2);
    bar[1] = tb;
    ctrl->nbasis = nv;
    ctrl->operator_count++;
    if (J == 0) ctrl->inner_product_count++;
    // after the third pass the reference counts once more and stops (pamp.h:372-381)
    ctrl->orthogonalization_count += passes + (again && passes == 3 ? 1 : 0);
    ctrl->ro_count = passes;
    ctrl->ro_go = again;
    ctrl->pre_norm = sqrt(pre2);
    ctrl->orig_norm = sqrt(orig2);
    ctrl->resid_norm = resid;
    if (!isfinite(resid)) ctrl->nonfinite = 1;
    if (J + 1 >= m) return;
    if (fabs(resid) < brk_tol) {
        ctrl->broken = 1;
        ctrl->breakdown_count++;
    } else {
        H[2 * ((size_t)(J + 1) * m + J)] = resid;
        H[2 * ((size_t)(J + 1) * m + J) + 1] = 0.0;
        ctrl->beta = resid;
        set_inv_beta(ctrl, resid);
    }
}

// h[0..nvals) = sums over the CTAs' partials (two components per vector and CTA), every CTA the
// same values: tpv threads per value, a power of two <= 32, so that a value's threads are
// consecutive lanes of one warp; up to kRound partials per lane and round in fixed point.
__device__ __forceinline__ void cgs_sum_partials(const double* part, int G, int nvals, double* h) {
    constexpr int kRound = 10;
    const int tid = threadIdx.x;
    int tpv = 32;
    while (tpv > 1 && tpv * nvals > kFuseThreads) tpv >>= 1;
    const int v = tid / tpv, q = tid % tpv;
    const double* p = part + (size_t)(v >> 1) * G * 2 + (v & 1);       // value v: component v & 1 of vector v >> 1
    double total = 0.0;
    for (int g0 = 0; g0 < G; g0 += kRound * tpv) {
        double t[kRound];
        int e = 0;
#pragma unroll
        for (int u = 0; u < kRound; ++u) {
            const int g = g0 + q + u * tpv;
            t[u] = v < nvals && g < G ? __ldcg(p + (size_t)g * 2) : 0.0;
            e = max(e, exp_field(t[u]));
        }
        for (int o = 1; o < tpv; o <<= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
        long long f = 0;
#pragma unroll
        for (int u = 0; u < kRound; ++u) f += to_fixed<2>(t[u], e);
        for (int o = 1; o < tpv; o <<= 1) f += shfl_xor_ll(f, o);
        total = g0 ? total + from_fixed<2>(f, e) : from_fixed<2>(f, e);
    }
    if (v < nvals && q == 0) h[v] = total;
}

// DORTH: re-orthogonalisation inside the kernel (pamp.h:353-400): a pass is dot, barrier, update,
// barrier, and every CTA takes the same decision from the same sums.  The column, the counters and the
// next beta are then complete here (brk_tol: the happy-breakdown threshold), so the next solve
// reads ctrl->inv_beta.  bar[1] holds the step's barriers used so far.  Against nine launches per Arnoldi step
// (dot, update, three conditional passes of both, finalize), most of which find nothing to do:
// a 16 x 300 step of m = 20 took 57 us of Gram-Schmidt per vector with those.
template <bool CACHE, bool DORTH>
__global__ void __launch_bounds__(kFuseThreads) k_arnoldi_cgs(const double2* __restrict__ V, long n, int J, int m,
                                                              double2* __restrict__ w, double* __restrict__ part,
                                                              unsigned* bar, Ctrl* ctrl, double* H, int update,
                                                              int chunk, double brk_tol) {
    using C = double2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double hs[2 * (kMaxBasis + 1)];
    __shared__ double ht[DORTH ? 2 * kMaxBasis : 1];   // the column, summed over the passes
    __shared__ double red[kFuseThreads / 32];
    __shared__ int s_again;
    __shared__ __align__(8) unsigned long long s_bar;
    const int nv = J + 1, G = gridDim.x, b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long i0 = (long)b * chunk;
    const int cl = (int)max(0L, min((long)chunk, n - i0));
    // shared memory: w chunk | cached rows of V
    C* ws = reinterpret_cast<C*>(smem_raw);
    C* cache = reinterpret_cast<C*>(smem_raw + (((size_t)chunk * sizeof(C) + 15) & ~(size_t)15));
    // With the cache, the CTA's basis rows (written by kernels before the predecessor) are
    // copied in by bulk asynchronous copies issued before the dependency wait; w, the
    // predecessor's output, follows it and carries the barrier's one arrival (rows start on
    // 16-byte boundaries: 16-byte elements)
    const bool tma = CACHE && cl > 0;
    const unsigned row = (unsigned)cl * 16;
    if (tma) {
        if (tid == 0) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&s_bar)) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncthreads();
        if (tid == 0) {
            asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;"
                         :: "r"(smem_u32(&s_bar)), "r"(row * (unsigned)nv) : "memory");
            for (int k = 0; k < nv; ++k) bulk_g2s(cache + (size_t)k * chunk, V + (size_t)k * n + i0, row, &s_bar);
        }
    }
    pdl_wait();
    if (ctrl->broken) {                              // uniform: written only between launches
        if (tma) {
            if (tid == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(smem_u32(&s_bar)) : "memory");
            mbar_wait0(&s_bar);                      // copies in flight land before exit
        }
        return;
    }
    const bool rnd = ctrl->round_matvec & 2;        // precision probe (FP64 handles)
    unsigned tb = DORTH ? *(volatile const unsigned*)(bar + 1) : (unsigned)J;   // the step's next barrier
    if (tma) {
        if (tid == 0) {
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                         :: "r"(smem_u32(&s_bar)), "r"(row) : "memory");
            bulk_g2s(ws, w + i0, row, &s_bar);
        }
        if (!__syncthreads_and(mbar_wait0(&s_bar, wait_budget(ctrl, kInvWaitLimit)))) {
            if (tid == 0) ctrl->wait_timeout = 1;
            mbar_wait0(&s_bar);                      // copies in flight land before exit
            return;
        }
    } else {
        for (int i = tid; i < cl; i += kFuseThreads) ws[i] = w[i0 + i];
        __syncthreads();
    }
    double orig2 = 0.0, resid2 = 0.0;                  // warp 0: squared norms before and after a pass
    double pre2 = 0.0;                                 // before the first
    int passes = 0, again = 0;
    for (;;) {
        // ---- phase A: partial inner products, one warp per basis vector.  The FP64 pipe retires
        // one warp instruction per 16 SM cycles and its dependent latency is about as long, so two
        // accumulator pairs per warp keep it busy; the lanes' sums are added in fixed point. --------
        for (int k = warp; k < nv; k += kFuseThreads / 32) {
            double ar = 0.0, ai = 0.0, br = 0.0, bi = 0.0;
            const C* vk = V + (size_t)k * n + i0;
            int i = lane;
            const C* ck = cache + (size_t)k * chunk;     // (staged rows when CACHE)
            for (; i + 96 < cl; i += 128) {
                C v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = CACHE ? ck[i + 32 * u] : vk[i + 32 * u];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const C x = ws[i + 32 * u];
                    if (u & 1) acc_dot64(br, bi, v[u].x, v[u].y, x.x, x.y);
                    else acc_dot64(ar, ai, v[u].x, v[u].y, x.x, x.y);
                }
            }
            for (; i + 32 < cl; i += 64) {
                const C v = CACHE ? ck[i] : vk[i], u = CACHE ? ck[i + 32] : vk[i + 32];
                const C x = ws[i], y = ws[i + 32];
                acc_dot64(ar, ai, v.x, v.y, x.x, x.y);
                acc_dot64(br, bi, u.x, u.y, y.x, y.y);
            }
            if (i < cl) {
                const C v = CACHE ? ck[i] : vk[i];
                const C x = ws[i];
                acc_dot64(ar, ai, v.x, v.y, x.x, x.y);
            }
            if (cl > 32) {
                ar += br;
                ai += bi;
            }
            ar = warp_fixed_sum(ar);
            ai = warp_fixed_sum(ai);
            if (lane == 0) {
                part[((size_t)k * G + b) * 2] = ar;
                part[((size_t)k * G + b) * 2 + 1] = ai;
            }
        }
        if (DORTH && passes == 0) {
            // ||w||^2 before the first pass, as one more vector's partial
            double t = 0.0;
            for (int i = tid; i < cl; i += kFuseThreads) {
                const C x = ws[i];
                t = fma(x.x, x.x, t);
                t = fma(x.y, x.y, t);
            }
            t = warp_fixed_sum(t);
            if (lane == 0) red[warp] = t;
            __syncthreads();
            if (warp == 0) {
                t = warp_fixed_sum(lane < kFuseThreads / 32 ? red[lane] : 0.0);
                if (lane == 0) {
                    part[((size_t)nv * G + b) * 2] = t;
                    part[((size_t)nv * G + b) * 2 + 1] = 0.0;
                }
            }
        }
        if (!grid_barrier(bar, G, tb++, ctrl)) return;

        // ---- phase B: h = sum of the partials -----------------------------------------------
        cgs_sum_partials(part, G, 2 * nv + (DORTH && passes == 0 ? 1 : 0), hs);
        __syncthreads();
        if (DORTH) {
            if (passes == 0) pre2 = orig2 = hs[2 * nv];
            for (int k = tid; k < 2 * nv; k += kFuseThreads) ht[k] = passes ? ht[k] + hs[k] : hs[k];
        }

        double nrm = 0.0;
        if (update) {
            // w -= V h on this chunk; ||w||^2 partial
            for (int i = tid; i < cl; i += kFuseThreads) {
                C r = ws[i];
                double sr0 = 0.0, si0 = 0.0, sr1 = 0.0, si1 = 0.0;
                int k = 0;
                for (; k + 1 < nv; k += 2) {
                    const C a = CACHE ? cache[(size_t)k * chunk + i] : V[(size_t)k * n + i0 + i];
                    const C c = CACHE ? cache[(size_t)(k + 1) * chunk + i] : V[(size_t)(k + 1) * n + i0 + i];
                    sr0 = fma(a.x, hs[2 * k], sr0);
                    sr0 = fma(-a.y, hs[2 * k + 1], sr0);
                    si0 = fma(a.x, hs[2 * k + 1], si0);
                    si0 = fma(a.y, hs[2 * k], si0);
                    sr1 = fma(c.x, hs[2 * k + 2], sr1);
                    sr1 = fma(-c.y, hs[2 * k + 3], sr1);
                    si1 = fma(c.x, hs[2 * k + 3], si1);
                    si1 = fma(c.y, hs[2 * k + 2], si1);
                }
                if (k < nv) {
                    const C a = CACHE ? cache[(size_t)k * chunk + i] : V[(size_t)k * n + i0 + i];
                    sr0 = fma(a.x, hs[2 * k], sr0);
                    sr0 = fma(-a.y, hs[2 * k + 1], sr0);
                    si0 = fma(a.x, hs[2 * k + 1], si0);
                    si0 = fma(a.y, hs[2 * k], si0);
                }
                r.x -= (sr0 + sr1);
                r.y -= (si0 + si1);
                if (rnd) r = make_double2(f2d_fast(d2f_fast(r.x)), f2d_fast(d2f_fast(r.y)));
                if (DORTH) ws[i] = r;
                else w[i0 + i] = r;
                nrm = fma(r.x, r.x, nrm);
                nrm = fma(r.y, r.y, nrm);
            }
            nrm = warp_fixed_sum(nrm);
            if (lane == 0) red[warp] = nrm;
            __syncthreads();
            if (warp == 0) {
                const double t = warp_fixed_sum(lane < kFuseThreads / 32 ? red[lane] : 0.0);
                // (without DORTH: for the next solve's beta)
                if (lane == 0) part[(size_t)(DORTH ? nv + 1 : nv) * G * 2 + b] = t;
            }
        }
        if (!DORTH) break;
        if (!grid_barrier(bar, G, tb++, ctrl)) return;
        if (warp == 0) {
            const double t = warp_fixed_sum_of(part + (size_t)(nv + 1) * G * 2, G, 1);
            if (passes > 0) orig2 = resid2;
            resid2 = t;
            if (lane == 0) s_again = t < 0.717 * 0.717 * orig2;      // pamp.h:369
        }
        __syncthreads();
        again = s_again;
        // the reference loop runs at most MaxOrthogonalizationCount = 3 passes (pamp.h:75,375)
        if (!again || passes == 3) break;
        ++passes;
    }
    if constexpr (!DORTH) {
        cgs_finish(ctrl, H, hs, m, J, b);
    } else {
        for (int i = tid; i < cl; i += kFuseThreads) w[i0 + i] = ws[i];
        cgs_finish_dorth(ctrl, H, ht, bar, tb, m, J, b, passes, again, pre2, orig2, resid2, brk_tol);
    }
}

// The same step with the inner products in 56-bit fixed point, for chunks of up to kFixedChunk elements whose
// basis rows are in shared memory.  A complex product is four FP64 instructions of 64 cycles of a
// sub-partition, or 12 integer multiply-adds of about 5: every row of V and w is split into two signed
// 29-bit digits at the largest exponent of the CTA's chunk, and
//     a x = a1 x1 2^58 + (a1 x0 + a0 x1) 2^29 + a0 x0
// summed without its last part.  An entry is rounded to 2^-57 of its chunk's largest and a product's
// dropped part is below 2^-56 of the two chunks' largest, both of either sign: h errs by that of ||v|| ||w||, where
// FP64 rounds every partial sum to 2^-53 (measured at 64 x 1000 and 23 x 437: 2^-54 to 2^-56 of ||w||, FP64
// 2^-53 to 2^-54).  A conversion costs what the products of a pair do, so a row is converted once, by the launch that
// meets it first, and its digits are kept for the step's later ones (Vd, ev: the step's launches share their
// chunks).
// w - V h keeps every element's own digits, however small it is beside the others of its chunk: a row whose h_k is
// within 2^-kSmallRow of the scale of w (the largest h, or ||w|| where it is known) is subtracted in FP64, its real and
// imaginary part each -- the real parts of the last two or three for a Hermitian operator, whose other h_k are
// rounding noise -- and the others in FP32, from rows converted with the digits (Vf): 2^-24 of |V_ki h_k| each,
// together below 2^-53 max|h| |V_ki|, what the h themselves leave open.  (With digits here too half of the elements of a
// 64 x 1000 step, emulated, err by 2^39 times what FP64 leaves them; so they by 2, and where w is tens of
// orders below its largest by up to 2^11, from the h_k of rows that hardly overlap with w.)
// Measured, a launch with its timing events, mean over the 30 vectors of 64 x 1000: FP64 products 27.1 us,
// digits formed by every launch 22.0, kept 18.0 (w - V h in digits too, without the small elements' own), this 18.2.
// At vector 15 the inner products take 6k cycles, arriving rows 3k, the barrier 2.5k and the sums over CTAs 3.3k.
constexpr int kSmallRow = 36;
constexpr int kRowBias = 120;                          // Vf holds V 2^120, |V| <= 1: entries down to 2^-246
constexpr int kFixedOwn = 2;
constexpr int kFixedChunk = kFixedOwn * kFuseThreads;
constexpr int kGsBias = 2 * (1075 + 3) - 29;           // exponent of a product of two digits pairs' sums

template <bool DORTH, int PER_SM>
__global__ void __launch_bounds__(kFuseThreads, PER_SM) k_arnoldi_cgs_fixed(const double2* __restrict__ V, long n, int J, int m,
                                                                    double2* __restrict__ w, double* __restrict__ part,
                                                                    int4* __restrict__ Vd, float2* __restrict__ Vf,
                                                                    int* __restrict__ ev_rows,
                                                                    unsigned* bar, Ctrl* ctrl, double* H, int update,
                                                                    int chunk, double brk_tol) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double hs[2 * (kMaxBasis + 1)];
    __shared__ double ht[DORTH ? 2 * kMaxBasis : 1];   // the column, summed over the passes
    __shared__ double red[kFuseThreads / 32];
    __shared__ int2 s_e[kFuseThreads / 32];
    __shared__ int s_ev[kMaxBasis];                    // the rows' exponents
    __shared__ float2 s_hf[64];                        // the column's small entries 2^(1023 - s_hx), zero for the others
    __shared__ unsigned s_big[2][2];                   // rows whose real, imaginary parts are the others
    __shared__ int s_hx, s_again;
    __shared__ __align__(8) unsigned long long s_bar;
    const int nv = J + 1, G = gridDim.x, b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long i0 = (long)b * chunk;
    const int cl = (int)max(0L, min((long)chunk, n - i0));
    // shared memory: w chunk | rows of V as digits; w and the newest row as they came and then as digits
    double2* ws = reinterpret_cast<double2*>(smem_raw);
    double2* cache = reinterpret_cast<double2*>(smem_raw + (size_t)chunk * sizeof(double2));
    int4* wd = reinterpret_cast<int4*>(ws);
    int4* cd = reinterpret_cast<int4*>(cache);
    // rows of V before the dependency wait, w after it (see k_arnoldi_cgs)
    const bool tma = cl > 0;
    const unsigned row = (unsigned)cl * 16;
    if (tma) {
        if (tid == 0) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&s_bar)) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncthreads();
        if (tid == 0) {
            asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;"
                         :: "r"(smem_u32(&s_bar)), "r"(row * (unsigned)nv) : "memory");
            for (int k = 0; k < J; ++k) bulk_g2s(cd + (size_t)k * chunk, Vd + (size_t)k * n + i0, row, &s_bar);
            bulk_g2s(cache + (size_t)J * chunk, V + (size_t)J * n + i0, row, &s_bar);
        }
    }
    pdl_wait();
    if (ctrl->broken) {                              // uniform: written only between launches
        if (tma) {
            if (tid == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(smem_u32(&s_bar)) : "memory");
            mbar_wait0(&s_bar);                      // copies in flight land before exit
        }
        return;
    }
    const bool rnd = ctrl->round_matvec & 2;        // precision probe (FP64 handles)
    if (tid < J) s_ev[tid] = ev_rows[tid * G + b];
    unsigned tb = DORTH ? *(volatile const unsigned*)(bar + 1) : (unsigned)J;   // the step's next barrier
    if (tma) {
        if (tid == 0) {
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                         :: "r"(smem_u32(&s_bar)), "r"(row) : "memory");
            bulk_g2s(ws, w + i0, row, &s_bar);
        }
        if (!__syncthreads_and(mbar_wait0(&s_bar, wait_budget(ctrl, kInvWaitLimit)))) {
            if (tid == 0) ctrl->wait_timeout = 1;
            mbar_wait0(&s_bar);                      // copies in flight land before exit
            return;
        }
    }
    double2 r[kFixedOwn];                              // this thread's elements of w
    double2 v0[kFixedOwn], v1[kFixedOwn];              // and of the two newest rows
#pragma unroll
    for (int u = 0; u < kFixedOwn; ++u) {
        const int i = tid + u * kFuseThreads;
        r[u] = i < cl ? ws[i] : make_double2(0.0, 0.0);
        v0[u] = i < cl ? cache[(size_t)J * chunk + i] : make_double2(0.0, 0.0);
        v1[u] = i < cl && J > 0 ? V[(size_t)(J - 1) * n + i0 + i] : make_double2(0.0, 0.0);
    }
    double orig2 = 0.0, resid2 = 0.0;                  // warp 0: squared norms before and after a pass
    double pre2 = 0.0;                                 // before the first
    int passes = 0, again = 0;
    for (;;) {
        // ---- digits of w and, in the first pass, of the newest row -----------------------------
        const bool first = passes == 0;
        int ew = 0, ev = 0;
#pragma unroll
        for (int u = 0; u < kFixedOwn; ++u) {
            ew = max(ew, max(exp_field(r[u].x), exp_field(r[u].y)));
            ev = max(ev, max(exp_field(v0[u].x), exp_field(v0[u].y)));
        }
        ew = (int)__reduce_max_sync(0xffffffffu, (unsigned)ew);
        ev = (int)__reduce_max_sync(0xffffffffu, (unsigned)ev);
        if (lane == 0) s_e[warp] = make_int2(ew, ev);
        __syncthreads();
        const int2 em = lane < kFuseThreads / 32 ? s_e[lane] : make_int2(0, 0);
        ew = (int)__reduce_max_sync(0xffffffffu, (unsigned)em.x);
        ev = (int)__reduce_max_sync(0xffffffffu, (unsigned)em.y);
#pragma unroll
        for (int u = 0; u < kFixedOwn; ++u) {
            const int i = tid + u * kFuseThreads;
            if (i >= cl) break;
            const int2 x = split29(to_fixed<3>(r[u].x, ew)), y = split29(to_fixed<3>(r[u].y, ew));
            wd[i] = make_int4(x.x, x.y, y.x, y.y);
            if (!first) continue;
            const int2 p = split29(to_fixed<3>(v0[u].x, ev)), q = split29(to_fixed<3>(v0[u].y, ev));
            const int4 v = make_int4(p.x, p.y, q.x, q.y);
            cd[(size_t)J * chunk + i] = v;
            Vd[(size_t)J * n + i0 + i] = v;
            Vf[(size_t)J * n + i0 + i] = make_float2(d2f_fast<kRowBias>(v0[u].x), d2f_fast<kRowBias>(v0[u].y));
        }
        if (first && tid == 0) s_ev[J] = ev_rows[J * G + b] = ev;
        __syncthreads();
        // ---- phase A: partial inner products, one warp per basis vector --------------------------
        for (int k = warp; k < nv; k += kFuseThreads / 32) {
            const int4* dk = cd + (size_t)k * chunk;
            const int ek = s_ev[k];
            // (at most 2 kFixedChunk / 32 products of 2^54, twice as many of 2^55)
            long long r1 = 0, r0 = 0, i1 = 0, i0s = 0;
            auto add = [&](const int4 v, const int4 x) {
                mad_wide(r1, v.x, x.x);
                mad_wide(r0, v.x, x.y);
                mad_wide(r0, v.y, x.x);
                mad_wide(r1, v.z, x.z);
                mad_wide(r0, v.z, x.w);
                mad_wide(r0, v.w, x.z);
                const int a = -v.z, c = -v.w;
                mad_wide(i1, v.x, x.z);
                mad_wide(i0s, v.x, x.w);
                mad_wide(i0s, v.y, x.z);
                mad_wide(i1, a, x.x);
                mad_wide(i0s, a, x.y);
                mad_wide(i0s, c, x.x);
            };
#pragma unroll 4
            for (int i = lane; i < cl; i += 32) add(dk[i], wd[i]);
            const bool bad = ek == 2047 || ew == 2047;
            const double nan = __hiloint2double(0x7ff80000, 0);
            const double ar = warp_fixed_sum(bad ? nan : from_digits(r1, r0, ek + ew - kGsBias));
            const double ai = warp_fixed_sum(bad ? nan : from_digits(i1, i0s, ek + ew - kGsBias));
            if (lane == 0) {
                part[((size_t)k * G + b) * 2] = ar;
                part[((size_t)k * G + b) * 2 + 1] = ai;
            }
        }
        if (DORTH && passes == 0) {
            // ||w||^2 before the first pass, as one more vector's partial
            double t = 0.0;
#pragma unroll
            for (int u = 0; u < kFixedOwn; ++u) t = fma(r[u].y, r[u].y, fma(r[u].x, r[u].x, t));
            t = warp_fixed_sum(t);
            if (lane == 0) red[warp] = t;
            __syncthreads();
            if (warp == 0) {
                t = warp_fixed_sum(lane < kFuseThreads / 32 ? red[lane] : 0.0);
                if (lane == 0) {
                    part[((size_t)nv * G + b) * 2] = t;
                    part[((size_t)nv * G + b) * 2 + 1] = 0.0;
                }
            }
        }
        if (!grid_barrier(bar, G, tb++, ctrl)) return;

        // ---- phase B: h = sum of the partials -----------------------------------------------
        cgs_sum_partials(part, G, 2 * nv + (DORTH && passes == 0 ? 1 : 0), hs);
        __syncthreads();
        if (DORTH) {
            if (passes == 0) pre2 = orig2 = hs[2 * nv];
            for (int k = tid; k < 2 * nv; k += kFuseThreads) ht[k] = passes ? ht[k] + hs[k] : hs[k];
        }
        if (update) {
            // which rows are subtracted in FP64, and the others' entries in FP32
            if (warp == 0) {
                int e[2][2], hx = 0;
#pragma unroll
                for (int u = 0; u < 2; ++u)
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const int k = lane + 32 * u;
                        e[u][c] = k < nv ? exp_field(hs[2 * k + c]) : 0;
                        hx = max(hx, e[u][c]);
                    }
                hx = (int)__reduce_max_sync(0xffffffffu, (unsigned)hx);
                if (DORTH) hx = max(hx, (exp_field(passes ? resid2 : pre2) + 1023) / 2);
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int k = lane + 32 * u;
                    float g[2] = {0.f, 0.f};
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const bool big = e[u][c] != 0 && e[u][c] >= hx - kSmallRow;
                        const unsigned mask = __ballot_sync(0xffffffffu, big);
                        if (lane == 0) s_big[c][u] = mask;
                        if (k < nv && !big) g[c] = d2f_fast(scale_pow2(hs[2 * k + c], 1023 - hx));
                    }
                    s_hf[k] = make_float2(g[0], g[1]);
                }
                if (lane == 0) s_hx = hx;
            }
            __syncthreads();
            const int hx = s_hx;
            const unsigned long long big[2] = {s_big[0][0] | (unsigned long long)s_big[0][1] << 32,
                                               s_big[1][0] | (unsigned long long)s_big[1][1] << 32};
            double nrm = 0.0;
#pragma unroll
            for (int u = 0; u < kFixedOwn; ++u) {
                const int i = tid + u * kFuseThreads;
                if (i >= cl) break;
                float sr = 0.f, si = 0.f;
                const float2* vf = Vf + i0 + i;
                for (int k0 = 0; k0 < nv; k0 += 8) {          // eight loads in flight, also in the last round
                    float2 v[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) v[q] = k0 + q < nv ? vf[(size_t)(k0 + q) * n] : make_float2(0.f, 0.f);
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const float2 g = s_hf[k0 + q];
                        sr = fmaf(v[q].x, g.x, sr);
                        sr = fmaf(-v[q].y, g.y, sr);
                        si = fmaf(v[q].x, g.y, si);
                        si = fmaf(v[q].y, g.x, si);
                    }
                }
                double dr = scale_pow2(f2d_fast<kRowBias>(sr), hx - 1023), di = scale_pow2(f2d_fast<kRowBias>(si), hx - 1023);
                auto sub = [&](int k, double2 v) {
                    if (big[0] >> k & 1) {
                        dr = fma(v.x, hs[2 * k], dr);
                        di = fma(v.y, hs[2 * k], di);
                    }
                    if (big[1] >> k & 1) {
                        dr = fma(-v.y, hs[2 * k + 1], dr);
                        di = fma(v.x, hs[2 * k + 1], di);
                    }
                };
                sub(J, v0[u]);
                if (J > 0) sub(J - 1, v1[u]);
                // (an operator that is not Hermitian has more of them: four loads in flight)
                for (unsigned long long rows = (big[0] | big[1]) & ((1ull << max(J - 1, 0)) - 1); rows != 0;) {
                    int k[4];
                    double2 v[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        k[q] = __ffsll((long long)rows) - 1;      // -1: none left
                        rows &= rows - 1;
                        v[q] = k[q] >= 0 ? V[(size_t)k[q] * n + i0 + i] : make_double2(0.0, 0.0);
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (k[q] >= 0) sub(k[q], v[q]);
                }
                if (hx == 2047) dr = di = __hiloint2double(0x7ff80000, 0);
                r[u].x -= dr;
                r[u].y -= di;
                if (rnd) r[u] = make_double2(f2d_fast(d2f_fast(r[u].x)), f2d_fast(d2f_fast(r[u].y)));
                if (!DORTH) w[i0 + i] = r[u];
                nrm = fma(r[u].x, r[u].x, nrm);
                nrm = fma(r[u].y, r[u].y, nrm);
            }
            nrm = warp_fixed_sum(nrm);
            if (lane == 0) red[warp] = nrm;
            __syncthreads();
            if (warp == 0) {
                const double t = warp_fixed_sum(lane < kFuseThreads / 32 ? red[lane] : 0.0);
                // (without DORTH: for the next solve's beta)
                if (lane == 0) part[(size_t)(DORTH ? nv + 1 : nv) * G * 2 + b] = t;
            }
        }
        if (!DORTH) break;
        if (!grid_barrier(bar, G, tb++, ctrl)) return;
        if (warp == 0) {
            const double t = warp_fixed_sum_of(part + (size_t)(nv + 1) * G * 2, G, 1);
            if (passes > 0) orig2 = resid2;
            resid2 = t;
            if (lane == 0) s_again = t < 0.717 * 0.717 * orig2;      // pamp.h:369
        }
        __syncthreads();
        again = s_again;
        // the reference loop runs at most MaxOrthogonalizationCount = 3 passes (pamp.h:75,375)
        if (!again || passes == 3) break;
        ++passes;
    }
    if constexpr (!DORTH) {
        cgs_finish(ctrl, H, hs, m, J, b);
    } else {
#pragma unroll
        for (int u = 0; u < kFixedOwn; ++u) {
            const int i = tid + u * kFuseThreads;
            if (i < cl) w[i0 + i] = r[u];
        }
        cgs_finish_dorth(ctrl, H, ht, bar, tb, m, J, b, passes, again, pre2, orig2, resid2, brk_tol);
    }
}

// ---------------------------------------------------------------------------
// Complex64 basis (FP32-mixed path).  The same phases, with every inner product, partial
// sum and norm share formed by error-free FP32 transformations (hi + lo pairs): on this
// GPU the FP64 pipe retires two thread operations per clock per SM, so FP64 adds in
// reductions (every lane of every warp) cost as much as the products themselves.  The
// first vector comes split into FP32 pairs (v0s, float4 re_hi, im_hi, re_lo, im_lo);
// partials are float4 (re_hi, re_lo, im_hi, im_lo) per (vector, CTA).  Only single
// threads touch FP64 (the Hessenberg entries).
constexpr int kCgsWarps = kFuseThreads / 32;
constexpr int kCgsItems = 64;

template <bool CACHE>
__global__ void __launch_bounds__(kFuseThreads) k_arnoldi_cgs32(const float2* __restrict__ V,
                                                                const float4* __restrict__ v0s, long n, int J,
                                                                int m, float2* __restrict__ w,
                                                                float4* __restrict__ part, unsigned* bar,
                                                                Ctrl* ctrl, double* H, int update, int chunk) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ float4 psum[kCgsItems];
    __shared__ float2 hf[kMaxBasis + 1], hl[kMaxBasis + 1];
    __shared__ double hs[2 * (kMaxBasis + 1)];
    __shared__ float2 red[kCgsWarps];
    __shared__ __align__(8) unsigned long long s_bar;
    const int nv = J + 1, G = gridDim.x, b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long i0 = (long)b * chunk;
    const int cl = (int)max(0L, min((long)chunk, n - i0));
    float2* ws = reinterpret_cast<float2*>(smem_raw);
    float4* c0 = reinterpret_cast<float4*>(smem_raw + (((size_t)chunk * sizeof(float2) + 15) & ~(size_t)15));
    float2* cache = reinterpret_cast<float2*>(reinterpret_cast<unsigned char*>(c0) + (v0s ? (size_t)chunk * 16 : 0));
    // With the cache, the CTA's whole share (w, the first vector, every basis row) arrives by
    // bulk asynchronous copies issued at once, so phase A waits one memory latency instead
    // of one per unrolled load round.  Row starts are 16-byte aligned when n is even (chunk
    // is a multiple of 8).
    const bool tma = CACHE && (n & 1) == 0 && cl > 0;
    const int k_first = v0s ? 1 : 0;                 // rows of V read (row 0 replaced by v0s)
    // The basis rows and the split first vector were written by kernels before the
    // predecessor, so their copies are issued before the dependency wait (overlapping the
    // predecessor's tail); w, the predecessor's output, and the control block after it.  The
    // barrier's single arrival comes with w's bytes, so the phase cannot complete early.
    const unsigned row = (unsigned)cl * 8;
    if (tma) {
        if (tid == 0) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&s_bar)) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncthreads();
        if (tid == 0) {
            const unsigned bytes = row * (unsigned)((v0s ? 2 : 0) + (nv - k_first));
            if (bytes)
                asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;"
                             :: "r"(smem_u32(&s_bar)), "r"(bytes) : "memory");
            if (v0s) bulk_g2s(c0, v0s + i0, 2 * row, &s_bar);
            for (int k = k_first; k < nv; ++k) bulk_g2s(cache + (size_t)k * chunk, V + (size_t)k * n + i0, row, &s_bar);
        }
    }
    pdl_wait();
    if (ctrl->broken) {                              // uniform: written only between launches
        if (tma) {
            if (tid == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(smem_u32(&s_bar)) : "memory");
            mbar_wait0(&s_bar);                      // copies in flight land before exit
        }
        return;
    }
    if (tma) {
        if (tid == 0) {
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                         :: "r"(smem_u32(&s_bar)), "r"(row) : "memory");
            bulk_g2s(ws, w + i0, row, &s_bar);
        }
        if (!__syncthreads_and(mbar_wait0(&s_bar, wait_budget(ctrl, kInvWaitLimit)))) {
            if (tid == 0) ctrl->wait_timeout = 1;
            mbar_wait0(&s_bar);                      // copies in flight land before exit
            return;
        }
    } else {
        for (int i = tid; i < cl; i += kFuseThreads) ws[i] = w[i0 + i];
        __syncthreads();
    }

    // ---- phase A: partials of conj(v_k) . w; with fewer vectors than warps each vector's
    // chunk is cut into S slices (one warp each), summed in slice order afterwards
    const int S = nv >= kCgsWarps ? 1 : max(1, min(kCgsWarps / nv, cl / 32));
    const int sl = ((cl + S - 1) / S + 31) & ~31;
    for (int it = warp; it < nv * S; it += kCgsWarps) {
        const int k = it / S;
        const int e0 = min(cl, (it % S) * sl), e1 = min(cl, e0 + sl);
        float rh = 0.f, rl = 0.f, ih = 0.f, il = 0.f, sh = 0.f, sl2 = 0.f, th = 0.f, tl = 0.f;
        if (v0s && k == 0) {
            for (int i = e0 + lane; i < e1; i += 32) {
                const float4 a = tma ? c0[i] : v0s[i0 + i];
                if (CACHE && !tma) c0[i] = a;
                const float2 x = ws[i];
                // conj(a) x with a = hi + lo: re = ar xr + ai xi, im = ar xi - ai xr
                acc_prod(rh, rl, a.x, a.z, x.x);
                acc_prod(sh, sl2, a.y, a.w, x.y);
                acc_prod(ih, il, a.x, a.z, x.y);
                acc_prod(th, tl, -a.y, -a.w, x.x);
            }
        } else {
            const float2* vk = tma ? cache + (size_t)k * chunk : V + (size_t)k * n + i0;
            const bool fill = CACHE && !tma;
            int i = e0 + lane;
            for (; i + 96 < e1; i += 128) {
                float2 v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = vk[i + 32 * u];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (fill) cache[(size_t)k * chunk + i + 32 * u] = v[u];
                    const float2 x = ws[i + 32 * u];
                    if (u & 1) {
                        acc_prod(sh, sl2, v[u].x, 0.f, x.x);
                        acc_prod(sh, sl2, v[u].y, 0.f, x.y);
                        acc_prod(th, tl, v[u].x, 0.f, x.y);
                        acc_prod(th, tl, -v[u].y, 0.f, x.x);
                    } else {
                        acc_prod(rh, rl, v[u].x, 0.f, x.x);
                        acc_prod(rh, rl, v[u].y, 0.f, x.y);
                        acc_prod(ih, il, v[u].x, 0.f, x.y);
                        acc_prod(ih, il, -v[u].y, 0.f, x.x);
                    }
                }
            }
            for (; i < e1; i += 32) {
                const float2 v = vk[i];
                if (fill) cache[(size_t)k * chunk + i] = v;
                const float2 x = ws[i];
                acc_prod(rh, rl, v.x, 0.f, x.x);
                acc_prod(rh, rl, v.y, 0.f, x.y);
                acc_prod(ih, il, v.x, 0.f, x.y);
                acc_prod(ih, il, -v.y, 0.f, x.x);
            }
        }
        acc_pair(rh, rl, sh, sl2);
        acc_pair(ih, il, th, tl);
        warp_pair_sum(rh, rl);
        warp_pair_sum(ih, il);
        if (lane == 0) {
            const float4 r = make_float4(rh, rl, ih, il);
            if (S == 1) part[(size_t)k * G + b] = r;
            else psum[it] = r;
        }
    }
    if (S > 1) {
        __syncthreads();
        if (tid < nv) {
            float4 a = psum[tid * S];
            for (int q = 1; q < S; ++q) {
                const float4 c = psum[tid * S + q];
                acc_pair(a.x, a.y, c.x, c.y);
                acc_pair(a.z, a.w, c.z, c.w);
            }
            part[(size_t)tid * G + b] = a;
        }
    }
    if (!grid_barrier(bar, G, J, ctrl)) return;   // the launch's only barrier: number J of the step

    // ---- phase B: h_k = sum over the CTAs' partials, every CTA in the same fixed order:
    // tpv consecutive lanes per vector, lane q taking partials q, q + tpv, ... (four loads in
    // flight), then a compensated shuffle tree inside the group
    {
        int tpv = 32;
        while (tpv > 1 && tpv * nv > kFuseThreads) tpv >>= 1;
        const int k = tid / tpv, q = tid % tpv;
        float rh = 0.f, rl = 0.f, ih = 0.f, il = 0.f;
        if (k < nv) {
            // all of a lane's partials in flight at once (12 per round covers G <= 12 tpv);
            // zero padding leaves a compensated sum unchanged
            constexpr int kRound = 12;
            const float4* p = part + (size_t)k * G;
            for (int g0 = q; g0 < G; g0 += kRound * tpv) {
                float4 c[kRound];
#pragma unroll
                for (int u = 0; u < kRound; ++u) {
                    const int g = g0 + u * tpv;
                    c[u] = g < G ? __ldcg(p + g) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
                for (int u = 0; u < kRound; ++u) {
                    acc_pair(rh, rl, c[u].x, c[u].y);
                    acc_pair(ih, il, c[u].z, c[u].w);
                }
            }
        }
        for (int o = 1; o < tpv; o <<= 1) {
            const float a = __shfl_xor_sync(0xffffffffu, rh, o), c = __shfl_xor_sync(0xffffffffu, rl, o);
            const float d = __shfl_xor_sync(0xffffffffu, ih, o), e = __shfl_xor_sync(0xffffffffu, il, o);
            acc_pair(rh, rl, a, c);
            acc_pair(ih, il, d, e);
        }
        if (k < nv && q == 0) {
            float h1, l1, h2, l2;
            two_sum(rh, rl, h1, l1);                 // normalised pairs
            two_sum(ih, il, h2, l2);
            hf[k] = make_float2(h1, h2);
            hl[k] = make_float2(l1, l2);
            hs[2 * k] = (double)h1 + (double)l1;
            hs[2 * k + 1] = (double)h2 + (double)l2;
        }
    }
    __syncthreads();

    if (update) {
        // w -= V h on this chunk (the first vector's product to first order in the low
        // parts); ||w||^2 partial as an exact-square compensated sum
        float nh = 0.f, nl = 0.f;
        for (int i = tid; i < cl; i += kFuseThreads) {
            float2 r = ws[i];
            float sr = 0.f, si = 0.f, cr = 0.f, ci = 0.f;
            int k = 0;
            if (v0s) {
                const float4 a = CACHE ? c0[i] : v0s[i0 + i];
                const float2 H0 = hf[0], L0 = hl[0];
                acc_prod(sr, cr, H0.x, L0.x, a.x);
                acc_prod(sr, cr, -H0.y, -L0.y, a.y);
                acc_prod(si, ci, H0.y, L0.y, a.x);
                acc_prod(si, ci, H0.x, L0.x, a.y);
                cr = __fmaf_rn(a.z, H0.x, __fmaf_rn(-a.w, H0.y, cr));
                ci = __fmaf_rn(a.z, H0.y, __fmaf_rn(a.w, H0.x, ci));
                k = 1;
            }
            for (; k < nv; ++k) {
                const float2 vk = CACHE ? cache[(size_t)k * chunk + i] : V[(size_t)k * n + i0 + i];
                const float2 Hk = hf[k], Lk = hl[k];
                sr = fmaf(vk.x, Hk.x, sr);
                sr = fmaf(-vk.y, Hk.y, sr);
                si = fmaf(vk.x, Hk.y, si);
                si = fmaf(vk.y, Hk.x, si);
                cr = fmaf(vk.x, Lk.x, cr);
                cr = fmaf(-vk.y, Lk.y, cr);
                ci = fmaf(vk.x, Lk.y, ci);
                ci = fmaf(vk.y, Lk.x, ci);
            }
            r.x = r.x - (sr + cr);
            r.y = r.y - (si + ci);
            w[i0 + i] = r;
            acc_prod(nh, nl, r.x, 0.f, r.x);
            acc_prod(nh, nl, r.y, 0.f, r.y);
        }
        warp_pair_sum(nh, nl);
        if (lane == 0) red[warp] = make_float2(nh, nl);
        __syncthreads();
        if (tid == 0) {
            float a = 0.f, c = 0.f;
            for (int q = 0; q < kCgsWarps; ++q) acc_pair(a, c, red[q].x, red[q].y);
            part[(size_t)nv * G + b] = make_float4(a, c, 0.f, 0.f);   // for the next solve's beta
        }
    }
    cgs_finish(ctrl, H, hs, m, J, b);
}

size_t arnoldi_cgs_smem(int prec, long n, int nv, int grid, int with_v0, int cache) {
    const size_t es = prec == 0 ? sizeof(double2) : sizeof(float2);
    const long chunk = ((n + grid - 1) / grid + 7) / 8 * 8;
    size_t b = (((size_t)chunk * es + 15) & ~(size_t)15);
    if (with_v0) b += (size_t)chunk * 16;
    if (cache) b += (size_t)nv * chunk * es;
    return b;
}

static int cgs_chunk(long n, int grid) { return (int)(((n + grid - 1) / grid + 7) / 8 * 8); }

// Fixed point wherever the rows are in shared memory and a thread holds its elements of w (up to 1024 a CTA: all
// but long vectors of small bases).
static bool cgs_fixed(int cache, int chunk) { return cache && chunk <= kFixedChunk; }

// Alone a CTA has its SM to itself and takes 108 registers, 120 with re-orthogonalisation; a batch's members share SMs
// with each other's CTAs and solves, so theirs stays within 64 (8 words spilled): alone 64 x 1000 18.7 us a vector with
// the first and 19.5 with the second, 12 uneven problems 7.65 and 7.54 ms.
static decltype(&k_arnoldi_cgs_fixed<false, 1>) cgs_kernel_fixed(int dorth, int batch) {
    return dorth ? k_arnoldi_cgs_fixed<true, 1> : batch ? k_arnoldi_cgs_fixed<false, 2> : k_arnoldi_cgs_fixed<false, 1>;
}

static decltype(&k_arnoldi_cgs<true, false>) cgs_kernel64(int cache, int dorth) {
    return dorth ? (cache ? k_arnoldi_cgs<true, true> : k_arnoldi_cgs<false, true>)
                 : (cache ? k_arnoldi_cgs<true, false> : k_arnoldi_cgs<false, false>);
}

template <typename Kern, typename... Args>
static cudaError_t cgs_coop_launch(Kern kern, int grid, size_t smem, cudaStream_t s, Args... args) {
    cudaError_t e = allow_max_smem(kern);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kFuseThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // the kernels call pdl_wait
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

cudaError_t launch_arnoldi_cgs(int prec, const void* V, const void* v0, long n, int J, int m, void* w,
                               double* part, unsigned* bar, Ctrl* ctrl, double* H, int update, int grid, int cache,
                               int dorth, double brk_tol, void* Vd, int* ev_rows, int batch, cudaStream_t s) {
    count_launch();
    const int chunk = cgs_chunk(n, grid);
    const size_t smem = arnoldi_cgs_smem(prec, n, J + 1, grid, v0 != nullptr, cache);
    if (prec == 0) {
        if (Vd && cgs_fixed(cache, chunk))
            return cgs_coop_launch(cgs_kernel_fixed(dorth, batch), grid, smem, s, (const double2*)V, n, J, m, (double2*)w, part, (int4*)Vd,
                                   (float2*)((int4*)Vd + (size_t)m * n), ev_rows, bar, ctrl, H, update, chunk, brk_tol);
        auto kern = cgs_kernel64(cache, dorth);
        return cgs_coop_launch(kern, grid, smem, s, (const double2*)V, n, J, m, (double2*)w, part, bar, ctrl, H, update,
                               chunk, brk_tol);
    }
    if (dorth) return cudaErrorInvalidValue;
    auto kern = cache ? k_arnoldi_cgs32<true> : k_arnoldi_cgs32<false>;
    return cgs_coop_launch(kern, grid, smem, s, (const float2*)V, (const float4*)v0, n, J, m, (float2*)w,
                           (float4*)part, bar, ctrl, H, update, chunk);
}

size_t arnoldi_cgs_digits_bytes(int prec, long n, int m, int grid, int cache) {
    return prec == 0 && cgs_fixed(cache, cgs_chunk(n, grid)) ? (size_t)m * n * (sizeof(int4) + sizeof(float2)) : 0;
}

// resident CTAs per SM of the FP64 form (of both where it may be the fixed-point one)
static cudaError_t cgs_occupancy64(long n, int grid, int cache, int dorth, int batch, size_t smem, int* per_sm) {
    auto kern = cgs_kernel64(cache, dorth);
    allow_max_smem(kern);
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, kern, kFuseThreads, smem);
    if (e == cudaSuccess && cgs_fixed(cache, cgs_chunk(n, grid))) {
        int fixed = 0;
        auto fk = cgs_kernel_fixed(dorth, batch);
        allow_max_smem(fk);
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fixed, fk, kFuseThreads, smem);
        *per_sm = std::min(*per_sm, fixed);
    }
    return e;
}

// Grid of co-resident CTAs for this configuration: one CTA per SM, or one per 32 elements where
// those are fewer -- a warp of a smaller chunk takes as long, and every CTA sums all CTAs' partials
// (0 when the cooperative form cannot run: no cooperative launch support or shared memory too large).
int arnoldi_cgs_grid(int prec, long n, int m, int with_v0, int cache, int dorth) {
    int dev = 0, sms = 0, coop = 0, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (!coop || sms <= 0 || (dorth && prec != 0)) return 0;
    const int grid = (int)std::min<long>(std::min(sms, kCgsMaxGrid), std::max<long>(1, (n + 31) / 32));
    const size_t smem = arnoldi_cgs_smem(prec, n, m, grid, with_v0, cache);
    if (smem + 8192 > (size_t)optin) return 0;
    int per_sm = 0;
    cudaError_t e;
    if (prec == 0) {
        e = cgs_occupancy64(n, grid, cache, dorth, 0, smem, &per_sm);
    } else {
        auto kern = cache ? k_arnoldi_cgs32<true> : k_arnoldi_cgs32<false>;
        allow_max_smem(kern);
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kFuseThreads, smem);
    }
    cudaGetLastError();
    if (e != cudaSuccess || per_sm < 1) return 0;
    return grid;
}

// Grid of the cooperative form for a problem inside a batch, where other problems fill the
// GPU: the fewest CTAs whose chunk of V fits in shared memory (V read once per Arnoldi step),
// else one CTA per ~2048 elements without the cache; 0 when neither is co-resident.
int arnoldi_cgs_grid_batch(int prec, long n, int m, int with_v0, int* cache) {
    int dev = 0, sms = 0, coop = 0, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (!coop || sms <= 0) return 0;
    sms = std::min(sms, kCgsMaxGrid);
    for (int c = 1; c >= 0; --c) {
        int grid = c ? 1 : (int)std::min<long>(sms, std::max<long>(1, (n + 2047) / 2048));
        if (c)
            while (grid <= sms && arnoldi_cgs_smem(prec, n, m, grid, with_v0, 1) + 4096 > (size_t)optin) ++grid;
        if (grid > sms) continue;
        const size_t smem = arnoldi_cgs_smem(prec, n, m, grid, with_v0, c);
        if (smem + 4096 > (size_t)optin) continue;
        int per_sm = 0;
        cudaError_t e;
        if (prec == 0) {
            e = cgs_occupancy64(n, grid, c, 0, 1, smem, &per_sm);
        } else {
            auto kern = c ? k_arnoldi_cgs32<true> : k_arnoldi_cgs32<false>;
            allow_max_smem(kern);
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kFuseThreads, smem);
        }
        cudaGetLastError();
        if (e != cudaSuccess || per_sm < 1 || grid > per_sm * sms) continue;
        *cache = c;
        return grid;
    }
    return 0;
}

}  // namespace gbprop
