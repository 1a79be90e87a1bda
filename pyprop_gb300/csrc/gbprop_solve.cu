// Banded triangular solves along r (ztbsv 'U','N' / 'U','C' in the reference,
// piram/piram/blitzblas.h:454-487, called from overlapmatrix.cpp:137-229):
//   * k_solve_rows  -- banded approximate inverse of the overlap factor applied in FP32
//                      with refinement from FP32-pair and FP64 residuals (the runtime's default);
//   * k_solve_ir    -- FP32 block back-substitution + FP64 refinement (fallback for
//                      factors whose inverse decays too slowly);
//   * k_solve       -- the block back-substitution in one precision.
#include "gbprop_internal.h"
#include "gbprop_device.cuh"

#include <cfloat>
#include <cmath>

namespace gbprop {

// ---------------------------------------------------------------------------
// parallel banded triangular solve (ztbsv 'U','N' / 'U','C' along r)
// ---------------------------------------------------------------------------
constexpr int kPitch = 33;   // smem pitch of the block-interleaved row buffer

// One warp solves U~ x = b for one row held in smem in block-interleaved e order
// (element e = B*L + i at buf[i*kPitch + B]); lane B owns block B.
//   1) local back-substitution of the block with rows pre-scaled by 1/U(e,e);
//   2) warp-shuffle suffix scan of the kd-vector recurrence t_B = y_B[0:kd] - F_B t_{B+1};
//   3) correction x_B -= G_B t_{B+1}.
template <typename T, int KD>
__device__ __forceinline__ void warp_block_solve(const SolveTab<T>& tab, cx<T>* buf, int lane) {
    using C = cx<T>;
    const int n = tab.n, L = tab.L, P = tab.P;
    const int B = lane;
    C win[KD];
#pragma unroll
    for (int d = 0; d < KD; ++d) win[d] = mk<T>(0, 0);
    for (int i = L - 1; i >= 0; --i) {
        const int e = B * L + i;
        const int idx = i * kPitch + B;
        const T inv = tab.invd[i * 32 + B];
        C x = mk<T>(0, 0);
        if (e < n) {
            const C b = buf[idx];
            T sr = b.x * inv, si = b.y * inv;
#pragma unroll
            for (int d = KD; d >= 1; --d) {
                const T u = tab.ud[((d - 1) * L + i) * 32 + B];
                sr = fma(-u, win[d - 1].x, sr);
                si = fma(-u, win[d - 1].y, si);
            }
            x = mk<T>(sr, si);
            buf[idx] = x;
        }
#pragma unroll
        for (int d = KD - 1; d >= 1; --d) win[d] = win[d - 1];
        win[0] = x;
    }
    C a[KD];
#pragma unroll
    for (int c = 0; c < KD; ++c) a[c] = (B * L + c < n && B < P) ? buf[c * kPitch + B] : mk<T>(0, 0);
    for (int lev = 0; lev < tab.levels; ++lev) {
        const int s = 1 << lev;
        C nb[KD];
#pragma unroll
        for (int c = 0; c < KD; ++c) {
            nb[c].x = __shfl_down_sync(0xffffffffu, a[c].x, s);
            nb[c].y = __shfl_down_sync(0xffffffffu, a[c].y, s);
        }
        if (B + s < P) {
            const T* M = tab.mlev + ((size_t)(lev * 32 + B) * KD) * KD;
#pragma unroll
            for (int r = 0; r < KD; ++r) {
                T ar = a[r].x, ai = a[r].y;
#pragma unroll
                for (int c = 0; c < KD; ++c) {
                    const T mv = M[r * KD + c];
                    ar = fma(mv, nb[c].x, ar);
                    ai = fma(mv, nb[c].y, ai);
                }
                a[r] = mk<T>(ar, ai);
            }
        }
    }
    C t[KD];
#pragma unroll
    for (int c = 0; c < KD; ++c) {
        t[c].x = __shfl_down_sync(0xffffffffu, a[c].x, 1);
        t[c].y = __shfl_down_sync(0xffffffffu, a[c].y, 1);
    }
    if (B + 1 < P) {
        for (int i = 0; i < L; ++i) {
            const int e = B * L + i;
            if (e >= n) break;
            const int idx = i * kPitch + B;
            C x = buf[idx];
#pragma unroll
            for (int c = 0; c < KD; ++c) {
                const T gv = tab.g[(c * L + i) * 32 + B];
                x.x = fma(-gv, t[c].x, x.x);
                x.y = fma(-gv, t[c].y, x.y);
            }
            buf[idx] = x;
        }
    }
    __syncwarp();
}

// Working-precision solve (the complex64 Krylov basis of the mixed path), one warp per row.
template <typename T, int KD, typename TI, typename TO, typename TV>
__global__ void __launch_bounds__(32) k_solve(SolveTab<T> tab, const TI* in, TO* out,
                                              TV* __restrict__ vstore, const Ctrl* __restrict__ ctrl,
                                              int scale_mode, int check_broken) {
    using C = cx<T>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* buf = reinterpret_cast<C*>(smem_raw);
    if (check_broken && ctrl->broken) return;
    const int l = blockIdx.x, lane = threadIdx.x;
    const int n = tab.n, L = tab.L;
    const double sc = scale_mode ? ctrl->inv_beta : 1.0;
    const size_t base = (size_t)l * n;
    for (int p = lane; p < n; p += 32) {
        TI v = in[base + p];
        double re = (double)v.x, im = (double)v.y;
        if (scale_mode) { re *= sc; im *= sc; }
        C c = mk<T>((T)re, (T)im);
        if (vstore) vstore[base + p] = conv<TV>(c);
        const int e = tab.dir ? (n - 1 - p) : p;
        const int B = e / L, i = e - B * L;
        buf[i * kPitch + B] = c;
    }
    __syncwarp();
    warp_block_solve<T, KD>(tab, buf, lane);
    for (int p = lane; p < n; p += 32) {
        const int e = tab.dir ? (n - 1 - p) : p;
        const int Bq = e / L, i = e - Bq * L;
        out[base + p] = conv<TO>(buf[i * kPitch + Bq]);
    }
}

// FP64-accurate solve for the FP64 path: FP32 block solve of the (power-of-two
// scaled) residual, refined three times with FP64 residuals r = b - U~ x
// (mixed-precision iterative refinement: each pass multiplies the error by the
// FP32 solve's relative accuracy, c*eps32*cond(U) ~ 1e-5 for the B-spline overlap
// factors, so three passes reach the FP64 level).  One CTA per row; the FP64 work
// is the residual band products (2*(kd+1) FMA per element per pass).
constexpr int kIrThreads = 256;
constexpr int kIrRefinements = 3;

template <int KD, typename TI, typename TO, typename TV>
__global__ void __launch_bounds__(kIrThreads) k_solve_ir(SolveTab<float> tab, const double* __restrict__ udp,
                                                         const TI* in, TO* out, TV* __restrict__ vstore,
                                                         const Ctrl* __restrict__ ctrl, int scale_mode,
                                                         int check_broken, int stage_tables, int stage_udp) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n = tab.n, L = tab.L, dir = tab.dir;
    double2* bd = reinterpret_cast<double2*>(smem_raw);
    double2* xd = bd + n;
    double2* rd = xd + n;
    float2* rf = reinterpret_cast<float2*>(rd + n);
    float* tsm = reinterpret_cast<float*>(rf + (size_t)L * kPitch);  // FP32 solve tables (when staged)
    const int nud = KD * L * 32, ninv = L * 32, ng = KD * L * 32, nm = max(tab.levels, 1) * 32 * KD * KD;
    double* ud_smem = reinterpret_cast<double*>(tsm + (stage_tables ? nud + ninv + ng + nm : 0));
    const double* ud_s = stage_udp ? ud_smem : udp;                    // (KD+1) x n FP64 diagonals
    __shared__ float s_red[kIrThreads / 32];
    if (check_broken && ctrl->broken) return;
    const int l = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // stage the solve tables (shared by every row; L2-resident) in shared memory
    SolveTab<float> st = tab;
    if (stage_tables) {
        float* p_ud = tsm;
        float* p_inv = p_ud + nud;
        float* p_g = p_inv + ninv;
        float* p_m = p_g + ng;
        for (int k = tid; k < nud; k += kIrThreads) p_ud[k] = tab.ud[k];
        for (int k = tid; k < ninv; k += kIrThreads) p_inv[k] = tab.invd[k];
        for (int k = tid; k < ng; k += kIrThreads) p_g[k] = tab.g[k];
        for (int k = tid; k < nm; k += kIrThreads) p_m[k] = tab.mlev[k];
        st.ud = p_ud;
        st.invd = p_inv;
        st.g = p_g;
        st.mlev = p_m;
    }
    if (stage_udp)
        for (int k = tid; k < (KD + 1) * n; k += kIrThreads) ud_smem[k] = udp[k];
    const double sc = scale_mode ? ctrl->inv_beta : 1.0;
    const size_t base = (size_t)l * n;
    for (int p = tid; p < n; p += kIrThreads) {
        const TI v = in[base + p];
        double2 b = make_double2((double)v.x, (double)v.y);
        if (scale_mode) { b.x *= sc; b.y *= sc; }
        if (vstore) vstore[base + p] = conv<TV>(b);
        bd[p] = b;
        rd[p] = b;
        xd[p] = make_double2(0.0, 0.0);
    }
    __syncthreads();
    for (int it = 0; it <= kIrRefinements; ++it) {
        if (it > 0) {
            // r = b - U~ x in FP64 (physical coordinates)
            for (int p = tid; p < n; p += kIrThreads) {
                double rr = bd[p].x, ri = bd[p].y;
                if (dir == 0) {
#pragma unroll
                    for (int d = 0; d <= KD; ++d) {
                        if (p + d < n) {
                            const double u = ud_s[(size_t)d * n + p];
                            rr = fma(-u, xd[p + d].x, rr);
                            ri = fma(-u, xd[p + d].y, ri);
                        }
                    }
                } else {
#pragma unroll
                    for (int d = 0; d <= KD; ++d) {
                        if (p - d >= 0) {
                            const double u = ud_s[(size_t)d * n + p - d];
                            rr = fma(-u, xd[p - d].x, rr);
                            ri = fma(-u, xd[p - d].y, ri);
                        }
                    }
                }
                rd[p] = make_double2(rr, ri);
            }
            __syncthreads();
        }
        // power-of-two scale so that the FP32 right-hand side is O(1)
        float mx = 0.f;
        for (int p = tid; p < n; p += kIrThreads) mx = fmaxf(mx, fmaxf(fabsf((float)rd[p].x), fabsf((float)rd[p].y)));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (lane == 0) s_red[warp] = mx;
        __syncthreads();
        mx = 0.f;
#pragma unroll
        for (int w = 0; w < kIrThreads / 32; ++w) mx = fmaxf(mx, s_red[w]);
        if (mx == 0.f) break;                       // exact solution reached (or zero rhs)
        int ex;
        frexpf(mx, &ex);
        const double scale = ldexp(1.0, -ex), unscale = ldexp(1.0, ex);
        for (int p = tid; p < n; p += kIrThreads) {
            const int e = dir ? (n - 1 - p) : p;
            const int B = e / L, i = e - B * L;
            rf[i * kPitch + B] = make_float2((float)(rd[p].x * scale), (float)(rd[p].y * scale));
        }
        __syncthreads();
        if (warp == 0) warp_block_solve<float, KD>(st, rf, lane);
        __syncthreads();
        for (int p = tid; p < n; p += kIrThreads) {
            const int e = dir ? (n - 1 - p) : p;
            const int B = e / L, i = e - B * L;
            const float2 dlt = rf[i * kPitch + B];
            xd[p].x += (double)dlt.x * unscale;
            xd[p].y += (double)dlt.y * unscale;
        }
        __syncthreads();
    }
    for (int p = tid; p < n; p += kIrThreads) out[base + p] = conv<TO>(xd[p]);
}

template <typename T, int KD>
static cudaError_t solve_kd(const SolveTab<T>& tab, int nrows, const void* in, int in_prec, void* out, int out_prec,
                            void* vstore, int v_prec, const Ctrl* ctrl, int scale_mode, int check_broken,
                            cudaStream_t s) {
    const size_t smem = (size_t)tab.L * kPitch * sizeof(cx<T>);
    dim3 grid(nrows), block(32);
    // in/out/vstore precision combinations used by the runtime
#define GB_SOLVE_CASE(TI_, TO_, TV_)                                                                             \
    {                                                                                                            \
        auto kern = k_solve<T, KD, TI_, TO_, TV_>;                                                               \
        if (smem > 48 * 1024) {                                                                                  \
            cudaError_t ea = allow_max_smem(kern);                                                               \
            if (ea != cudaSuccess) return ea;                                                                    \
        }                                                                                                        \
        kern<<<grid, block, smem, s>>>(tab, (const TI_*)in, (TO_*)out, (TV_*)vstore, ctrl, scale_mode,           \
                                       check_broken);                                                            \
        return cudaGetLastError();                                                                               \
    }
    // combinations the runtime uses (the complex64 Krylov basis of the mixed path)
    const int key = in_prec * 4 + out_prec * 2 + v_prec;
    switch (key) {
        case 3: GB_SOLVE_CASE(double2, float2, float2)
        case 7: GB_SOLVE_CASE(float2, float2, float2)
        default: return cudaErrorInvalidValue;
    }
#undef GB_SOLVE_CASE
}

template <typename T>
static cudaError_t solve_dispatch(const SolveTab<T>& tab, int nrows, const void* in, int in_prec, void* out,
                                  int out_prec, void* vstore, int v_prec, const Ctrl* ctrl, int scale_mode,
                                  int check_broken, cudaStream_t s) {
    switch (tab.kd) {
#define GB_KD(K) \
    case K: return solve_kd<T, K>(tab, nrows, in, in_prec, out, out_prec, vstore, v_prec, ctrl, scale_mode, check_broken, s);
        GB_KD(1) GB_KD(2) GB_KD(3) GB_KD(4) GB_KD(5) GB_KD(6) GB_KD(7) GB_KD(8)
#undef GB_KD
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_solve(int arith, const void* tab, int nrows, const void* in, int in_prec, void* out, int out_prec,
                         void* vstore, int v_prec, const Ctrl* ctrl, int scale_mode, int check_broken,
                         cudaStream_t s) {
    count_launch();
    if (arith == 0) return cudaErrorInvalidValue;     // FP64 solves go through the refined kernels
    return solve_dispatch(*(const SolveTab<float>*)tab, nrows, in, in_prec, out, out_prec, vstore, v_prec, ctrl,
                          scale_mode, check_broken, s);
}

template <int KD>
static cudaError_t solve_ir_kd(const SolveTab<float>& tab, const double* udp, int nrows, const void* in, int in_prec,
                               void* out, int out_prec, void* vstore, int v_prec, const Ctrl* ctrl, int scale_mode,
                               int check_broken, cudaStream_t s) {
    // shared memory: b, x, r rows + FP32 work row are required; the solve tables and the FP64
    // diagonals are staged only while they fit (otherwise read through L1/L2)
    const size_t limit = 220 * 1024;
    const size_t base = (size_t)3 * tab.n * sizeof(double2) + (size_t)tab.L * kPitch * sizeof(float2);
    const size_t tabb = ((size_t)KD * tab.L * 32 * 2 + (size_t)tab.L * 32 +
                         (size_t)(tab.levels > 0 ? tab.levels : 1) * 32 * KD * KD) * sizeof(float);
    const size_t udb = (size_t)(KD + 1) * tab.n * sizeof(double);
    const int stage_tables = base + tabb <= limit;
    const int stage_udp = base + (stage_tables ? tabb : 0) + udb <= limit;
    const size_t smem = base + (stage_tables ? tabb : 0) + (stage_udp ? udb : 0);
    if (smem > limit) return cudaErrorInvalidValue;
    dim3 grid(nrows), block(kIrThreads);
#define GB_IR_CASE(TI_, TO_, TV_)                                                                                \
    {                                                                                                            \
        auto kern = k_solve_ir<KD, TI_, TO_, TV_>;                                                               \
        if (smem > 48 * 1024) {                                                                                  \
            cudaError_t ea = allow_max_smem(kern);                                                               \
            if (ea != cudaSuccess) return ea;                                                                    \
        }                                                                                                        \
        kern<<<grid, block, smem, s>>>(tab, udp, (const TI_*)in, (TO_*)out, (TV_*)vstore, ctrl, scale_mode,      \
                                       check_broken, stage_tables, stage_udp);                                   \
        return cudaGetLastError();                                                                               \
    }
    // combinations the runtime uses: refined solves store double2 (or nothing)
    const int key = in_prec * 4 + out_prec * 2 + v_prec;
    switch (key) {
        case 0: GB_IR_CASE(double2, double2, double2)
        case 2: GB_IR_CASE(double2, float2, double2)
        case 4: GB_IR_CASE(float2, double2, double2)
        case 6: GB_IR_CASE(float2, float2, double2)
        default: return cudaErrorInvalidValue;
    }
#undef GB_IR_CASE
}

cudaError_t launch_solve_ir(const void* tabf, const double* udp, int nrows, const void* in, int in_prec, void* out,
                            int out_prec, void* vstore, int v_prec, const Ctrl* ctrl, int scale_mode, int check_broken,
                            cudaStream_t s) {
    count_launch();
    const SolveTab<float>& tab = *(const SolveTab<float>*)tabf;
    switch (tab.kd) {
#define GB_KD(K) \
    case K: return solve_ir_kd<K>(tab, udp, nrows, in, in_prec, out, out_prec, vstore, v_prec, ctrl, scale_mode, check_broken, s);
        GB_KD(1) GB_KD(2) GB_KD(3) GB_KD(4) GB_KD(5) GB_KD(6) GB_KD(7) GB_KD(8)
#undef GB_KD
        default: return cudaErrorInvalidValue;
    }
}

// ---------------------------------------------------------------------------
// solve through the banded approximate inverse (all threads busy, no recursion)
// ---------------------------------------------------------------------------
// CTA (chunk c, row group g) produces x on q in [q0, q0 + cl), q0 = c * chunk, for up to `rg`
// angular rows.  With P refinement passes, pass k (0..P) forms M r on [q0, q0 + R_k),
// R_k = cl + (P-k)(w+kd), and adds it to x:
//     r = b                 (pass 0, FP32)
//     r = b - U~ x          (later passes)
// x on R_k needs r on R_k + w, which needs the previous x on R_k + w + kd = R_{k-1}, so the
// chunk's halo is recomputed instead of exchanged.
//   * FP64-accurate solve (R64): x0 is exact in FP32, so the first residual is formed from FP32
//     pairs (U~ = uh + ul, b = bh + bl; error-free products and sums); the last ones are in FP64.
//   * complex64 solve of the mixed path's basis: P = 1 with the FP32-pair residual.  The
//     refinement makes the operator seen by the basis U^-1 to ~1e-13 (the FP32 band of M alone
//     perturbs it by ~1e-7, which shifts high eigenvalues systematically).  A double2 operand (the
//     FP64 first vector) is used as hi + lo, a complex64 operand as stored, so the solve acts on
//     exactly the vector kept in the basis.
//
// U is real and the same for every row, so the rows' real and imaginary parts are columns of one
// right-hand side and the band product of a CTA is a banded matrix times a (radial) x (2 rows)
// matrix: it runs on the tensor cores (mma.sync m16n8k16, bfloat16 operands, FP32 accumulation), M
// and r each split exactly into three bfloat16 parts, six products (the other three are below FP32's
// resolution).  A warp owns sixteen outputs of eight columns; M comes in fragment order (InvTab), one
// 16-byte load per lane, part and k step, through L1 and L2: a CTA uses an entry once per pass.  A
// lane's accumulators are one row's real and imaginary part of two outputs.  (Two TF32 parts, three
// products, take as many instructions with the splitting of M and leave 2^-22 instead of 2^-24 of the
// product: states that fall off towards the origin by tens of orders keep the error of that as noise
// in the operator's stiff modes, 50 times more in a step of the 64 x 1000 hydrogen operator.)
// What bounds it: the FP64 residual, 2 (kd+1) FP64 warp instructions per 32 complex elements at 16 SM
// cycles each, on the chunk and w halo elements; then the latency of the barrier-separated phases.
// The form before this one gave a thread two complex outputs of one row and fed FP32 FMAs from shared
// memory at 8 bytes per FMA per lane, which bound it.  (Sharing an M entry among the lanes of all rows
// instead does not help FMAs: a broadcast costs the register-side bandwidth of the loads all the same.)
// Measured, FP64, a launch with its timing events: 64 x 1000 27.6 us before, 18.5 now; no pipe above 21%
// busy, DRAM 1.7 MB a launch.  Balanced matvec of that size (two solves and the band) 65 -> 45.5 us.
//
// beta of an Arnoldi vector (the norm partials of the previous Gram-Schmidt launch) is formed by a
// warp of its own.  The FP64-accurate solve runs on the unscaled vector meanwhile and multiplies v
// and x by 1/beta when it stores them; the complex64 solve needs v rounded first and waits for an
// FP32-pair reciprocal square root.
//
// Worker warps: 16 for a problem alone (one CTA per SM; its phases are latency-bound), 8 inside a
// batch, where two or three CTAs of different problems share an SM (InvTab::warps).
constexpr int kRowWarps = 16;                        // most worker warps
constexpr int kRowBlock = 32 * kRowWarps + 32;       // + the warp that forms 1/beta
// The FP64 solve's FP32 and bfloat16 numbers stand for 2^-kBias of themselves (free in the integer conversions): a
// row of up to 2^50 leaves FP32 room for U^-1 above, one of 2^-100 for its residuals and their parts below
constexpr int kBias = 40;

__device__ __forceinline__ void worker_sync(int nw) { asm volatile("bar.sync 1, %0;" :: "r"(32 * nw) : "memory"); }

template <bool SMEM, typename T> __device__ __forceinline__ T row_ld(const T* p) { return SMEM ? *p : __ldg(p); }

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint4& a, unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}

// M fragments of one block, this lane's: the leading and middle parts of the first kSolveFrags k steps
__device__ __forceinline__ void load_frags(uint4 (&a)[2 * kSolveFrags], const uint4* frag) {
#pragma unroll
    for (int i = 0; i < kSolveFrags; ++i) {
        a[2 * i] = __ldg(frag + i * 96);
        a[2 * i + 1] = __ldg(frag + i * 96 + 32);
    }
}

// Sixteen outputs of eight planes: o[0], o[1] = planes 2j, 2j+1 (j = lane % 4) of output lane / 4,
// o[2], o[3] of output lane / 4 + 8.  frag: the block's M fragments (this lane's), a: what load_frags
// took of them; r: this lane's plane (lane / 4) of the leading parts, as pairs of entries, from the
// block's first output on + lane % 4; the middle and last parts `part` words further each.
__device__ __forceinline__ void band_tile(float (&o)[4], const uint4* frag, uint4 (&a)[2 * kSolveFrags], int ks,
                                          const unsigned* r, int part) {
    float c1[4] = {0.f, 0.f, 0.f, 0.f}, c2[4] = {0.f, 0.f, 0.f, 0.f}, c3[4] = {0.f, 0.f, 0.f, 0.f};
    float c4[4] = {0.f, 0.f, 0.f, 0.f}, c5[4] = {0.f, 0.f, 0.f, 0.f}, c6[4] = {0.f, 0.f, 0.f, 0.f};
    for (int k0 = 0;;) {
        uint4 al[kSolveFrags];
#pragma unroll
        for (int i = 0; i < kSolveFrags; ++i) al[i] = __ldg(frag + i * 96 + 64);
#pragma unroll
        for (int i = 0; i < kSolveFrags; ++i) {
            const unsigned h0 = r[8 * i], h1 = r[8 * i + 4], m0 = r[8 * i + part], m1 = r[8 * i + 4 + part];
            const unsigned l0 = r[8 * i + 2 * part], l1 = r[8 * i + 4 + 2 * part];
            mma_bf16(c1, a[2 * i], h0, h1);
            mma_bf16(c2, a[2 * i], m0, m1);
            mma_bf16(c3, a[2 * i + 1], h0, h1);
            mma_bf16(c4, a[2 * i + 1], m0, m1);
            mma_bf16(c5, a[2 * i], l0, l1);
            mma_bf16(c6, al[i], h0, h1);
        }
        k0 += kSolveFrags;
        if (k0 >= ks) break;
        r += 8 * kSolveFrags;
        frag += 96 * kSolveFrags;
        load_frags(a, frag);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) o[j] = c1[j] + ((c2[j] + c3[j]) + (c4[j] + (c5[j] + c6[j])));
}

// a plane's entry as its three bfloat16 parts (v = h + m + l exactly), `part` halves apart
__device__ __forceinline__ void put_split(unsigned short* r, int part, float v) {
    const unsigned h = __float_as_uint(v) & 0xffff0000u;
    const float v1 = __fsub_rn(v, __uint_as_float(h));
    const unsigned m = __float_as_uint(v1) & 0xffff0000u;
    const float v2 = __fsub_rn(v1, __uint_as_float(m));
    r[0] = (unsigned short)(h >> 16);
    r[part] = (unsigned short)(m >> 16);
    r[2 * part] = (unsigned short)(__float_as_uint(v2) >> 16);
}

template <int KD, bool R64, bool STAGE>
__global__ void __launch_bounds__(kRowBlock) k_solve_rows(InvTab tab, int nl, const void* in, int in_prec, void* out,
                                                          int out_prec, void* vstore, float4* v0s, Ctrl* ctrl, int dir,
                                                          int scale_mode, int check_broken, const void* bpart, int bG) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned s_red[kRowWarps];
    __shared__ int s_e[kRowWarps];                     // powers of two of scaled rows (FP64 solve)
    __shared__ double s_ib;                            // 1/beta (FP64 solve)
    __shared__ float2 s_ibf;                           // 1/beta as an FP32 pair (complex64 solve)
    __shared__ int s_brk, s_skip;
    constexpr int UP = inv_upitch(KD);                 // entries of a row of U~'s tables
    const int n = tab.n, w = tab.w, P = R64 ? tab.refine : 1, ks = tab.ks;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = (int)(blockDim.x >> 5) - 1;
    const int q0 = blockIdx.x * tab.chunk, left = n - q0;
    const int lg = tab.lg, rmask = (1 << lg) - 1, l0 = blockIdx.y << lg;
    const int rows = min(1 << lg, nl - l0);
    const int lnt = max(lg - 2, 0);                    // log2 of the plane groups of a tile column
    int cl, R0, RB;
    inv_region(n, q0, tab.chunk, P, w, KD, &cl, &R0, &RB);
    const int PL = tab.pl;                             // from a plane's leading part to its next
    const int PQ = tab.pq, PX = tab.px, PD = tab.pd, PB = tab.pb;
    const InvLayout& ly = tab.ly;
    const double* const Us = reinterpret_cast<const double*>(smem_raw + ly.u);
    const float2* const Ufs = reinterpret_cast<const float2*>(smem_raw + ly.uf);
    double2* const bq = reinterpret_cast<double2*>(smem_raw + ly.b);      // R64: right-hand side [row][q]
    float4* const bf = reinterpret_cast<float4*>(smem_raw + ly.b);        // complex64: FP32 pairs [row][q]
    double2* const xd = reinterpret_cast<double2*>(smem_raw + ly.x);      // R64: iterate [row][q]
    unsigned short* const r16 = reinterpret_cast<unsigned short*>(smem_raw + ly.r16);   // residual planes
    float2* const x0f = reinterpret_cast<float2*>(smem_raw + ly.x0);      // first iterate [row][q]
    const uint4* const Mg = reinterpret_cast<const uint4*>(tab.mf) + (size_t)(q0 >> 4) * ks * 96 + lane;
    const bool late = scale_mode && bpart;             // beta comes from norm partials

    if (warp == nw) {
        // this warp forms 1/beta
        pdl_wait();
        const bool writer = blockIdx.x == 0 && blockIdx.y == 0 && !(check_broken == 1 && ctrl->broken);
        if constexpr (R64) {
            if (late) {
                const double beta = gs_beta(bpart, bG);
                if (lane == 0) {
                    s_brk = gs_record_beta(ctrl, beta, writer);
                    s_ib = 1.0 / beta;
                }
            }
            __syncthreads();
        } else if (late) {
            const float2 t = gs_norm2_pair(reinterpret_cast<const float4*>(bpart), bG);
            if (lane == 0) {
                s_brk = t.x < (float)DBL_EPSILON || (t.x == (float)DBL_EPSILON && t.y < 0.f);
                s_ibf = inv_sqrt_pair(t.x, t.y);
            }
            __syncthreads();
            if (lane == 0 && writer) gs_record_beta(ctrl, sqrt((double)t.x + (double)t.y), true);
        }
        return;
    }
    // ---- workers.  The first tile's M fragments are on their way before the wait; everything
    // below reads what earlier kernels wrote.
    uint4 fr[2 * kSolveFrags];
    const int ft = warp >> lnt;                        // the warp's first block of outputs
    if (16 * ft < R0) {
        load_frags(fr, Mg + ft * ks * 96);
#pragma unroll
        for (int i = 0; i < kSolveFrags; ++i) prefetch_l1(Mg + ft * ks * 96 + i * 96 + 64);
    }
    if (STAGE) {
        // U~'s slices: contiguous rows of R0p entries (sizes and addresses multiples of 16 bytes)
        const int nc = ((R0 + 3) & ~3) * UP / 2;
        const double2* gf = reinterpret_cast<const double2*>(tab.uf + (size_t)q0 * UP);
        const double2* gu = reinterpret_cast<const double2*>(tab.u + (size_t)q0 * UP);
        for (int i = tid; i < nc; i += (32 * nw)) {
            cp_async16(smem_raw + ly.uf + 16 * i, gf + i);
            if (R64) cp_async16(smem_raw + ly.u + 16 * i, gu + i);
        }
    }
    pdl_wait();
    const int gdir = dir ? -1 : 1;
    const size_t gbase = (size_t)l0 * n + (dir ? n - 1 - q0 : q0);
    auto gidx = [&](int row, int q) { return gbase + (long)(row * n + gdir * q); };
    // 1: after a happy breakdown, 2: a step of this call gave up on a wait -- nothing is written.  One
    // read for the CTA: this launch's first CTA may set ctrl->broken while others start
    int skip = 0;
    if (tid == 0)
        skip = check_broken == 1   ? *(volatile const int*)&ctrl->broken
               : check_broken == 2 ? *(volatile const int*)&ctrl->wait_timeout
                                   : 0;
    // zeros past the chunk's data: the residual past the right-hand side (a tile reads 16 ks entries
    // from its first output on; planes without a row are zero), the iterates past the last element
    auto zero_tails = [&]() {
        if (tid == 0) s_skip = skip;
        for (int g = warp; g < max(2 << lg, 8); g += nw) {
            const int t0 = g < 2 * rows ? RB : 0;
            unsigned short* rr = r16 + g * PQ;
            if ((t0 & 1) && lane < 3) rr[lane * PL + t0] = 0;
            for (int i = ((t0 + 1) >> 1) + lane; i < (PQ >> 1); i += 32) {
                reinterpret_cast<unsigned*>(rr)[i] = 0;
                reinterpret_cast<unsigned*>(rr + PL)[i] = 0;
                reinterpret_cast<unsigned*>(rr + 2 * PL)[i] = 0;
            }
        }
        if (warp >= nw / 2) {
            const int xde = (min(left, cl + (P >= 2 ? P - 1 : 1) * (w + KD)) + 15) & ~15;
            for (int row = warp - nw / 2; row < rows; row += nw / 2) {
                for (int q = ((R0 + 15) & ~15) + lane; q < PX; q += 32) x0f[row * PX + q] = make_float2(0.f, 0.f);
                if (R64)
                    for (int q = xde + lane; q < PD; q += 32) xd[row * PD + q] = make_double2(0.0, 0.0);
            }
        }
    };
    const int probe = R64 && check_broken == 1 ? ctrl->round_matvec : 0;

    // right-hand side: a warp takes 32-element segments of the rows, kPre of them loaded at once
    constexpr int kPre = 3;
    const int nbs = ((RB + 31) >> 5) << lg;
    double fin = 1.0;                                  // R64: factor of x and v at the end, if scale_mode
    bool rescaled = false;                             // R64: rows of b are scaled, row r by 2^-s_e[r]
    if constexpr (R64) {
        if (scale_mode && !late) fin = ctrl->inv_beta;
        auto keep = [&](int it, double2 b) {
            const int row = it & rmask, q = (it >> lg) * 32 + lane;
            if (row < rows && q < RB) {
                bq[row * PB + q] = b;
                unsigned short* rr = r16 + 2 * row * PQ + q;
                put_split(rr, PL, d2f_fast<kBias>(b.x));
                put_split(rr + PQ, PL, d2f_fast<kBias>(b.y));
            }
        };
        unsigned hmax = 0;                             // (a warp's items are of one row: 2^lg <= nw)
        for (int i0 = warp;;) {
            double2 pre[kPre];
#pragma unroll
            for (int u = 0; u < kPre; ++u) {
                const int it = i0 + u * nw, row = it & rmask, q = (it >> lg) * 32 + lane;
                pre[u] = make_double2(0.0, 0.0);
                if (row < rows && q < RB) {
                    if (in_prec == 0) pre[u] = reinterpret_cast<const double2*>(in)[gidx(row, q)];
                    else {
                        const float2 t = reinterpret_cast<const float2*>(in)[gidx(row, q)];
                        pre[u] = make_double2(f2d_fast(t.x), f2d_fast(t.y));
                    }
                }
            }
            if (i0 == warp) zero_tails();              // while the first loads are in flight
#pragma unroll
            for (int u = 0; u < kPre; ++u) {
                keep(i0 + u * nw, pre[u]);
                hmax = max(hmax, max((unsigned)__double2hiint(pre[u].x) & 0x7fffffffu,
                                     (unsigned)__double2hiint(pre[u].y) & 0x7fffffffu));
            }
            i0 += kPre * nw;
            if (i0 >= nbs) break;
        }
        hmax = __reduce_max_sync(0xffffffffu, hmax);
        if (lane == 0) s_red[warp] = hmax;
        if (STAGE) cp_async_wait_all();
        worker_sync(nw);
        // a row whose largest exponent leaves the range where the FP32 residuals (down to 2^-50 of it) and their
        // bfloat16 parts stay normal is scaled by a power of two, and its x back at the end.  Every row by its own:
        // beside a row of magnitude 1 one of 1e-39 would lose everything to FP32's exponent range, and wave functions'
        // tails are such rows.  s_red[v] is of row v & rmask
        const unsigned hv = s_red[lane & (nw - 1)];
        if (__any_sync(0xffffffffu, hv != 0 && hv - ((1022u - 100u) << 20) >= (151u << 20))) {     // outside -100 .. 50
            unsigned hr = hv;
            for (int o = 1 << lg; o < nw; o <<= 1) hr = max(hr, __shfl_xor_sync(0xffffffffu, hr, o));
            const int e = (int)(hr >> 20) - 1022;
            const int er = hr != 0 && hr < 0x7ff00000u && (e < -100 || e > 50) ? e : 0;      // of row lane & rmask
            rescaled = __any_sync(0xffffffffu, er != 0);                                    // (the same in every warp)
            if (rescaled) {
                if (warp == 0 && lane <= rmask) s_e[lane] = er;
                const int row = warp & rmask, ew = -__shfl_sync(0xffffffffu, er, row);
#pragma unroll 1
                for (int it = warp; it < nbs && ew != 0 && row < rows; it += nw) {
                    const int q = (it >> lg) * 32 + lane;
                    if (q >= RB) break;
                    const double2 b = bq[row * PB + q];
                    keep(it, make_double2(scale_pow2(b.x, ew), scale_pow2(b.y, ew)));
                }
                worker_sync(nw);
            }
        }
    } else {
        if (in_prec == 0) {
            // the FP64 first vector (once per step): scaled in FP64, kept as hi + lo
            zero_tails();
            const double sc = scale_mode ? ctrl->inv_beta : 1.0;
            for (int it = warp; it < nbs; it += nw) {
                const int row = it & rmask, q = (it >> lg) * 32 + lane;
                if (row >= rows || q >= RB) continue;
                const size_t gi = gidx(row, q);
                double2 b = reinterpret_cast<const double2*>(in)[gi];
                if (scale_mode) { b.x *= sc; b.y *= sc; }
                const float2 hi = make_float2(d2f_fast(b.x), d2f_fast(b.y));
                const float2 lo = make_float2(d2f_fast(b.x - f2d_fast(hi.x)), d2f_fast(b.y - f2d_fast(hi.y)));
                if (q < cl) {
                    if (vstore) reinterpret_cast<double2*>(vstore)[gi] = b;
                    if (v0s) v0s[gi] = make_float4(hi.x, hi.y, lo.x, lo.y);
                }
                unsigned short* rr = r16 + 2 * row * PQ + q;
                put_split(rr, PL, hi.x);
                put_split(rr + PQ, PL, hi.y);
                bf[row * PB + q] = make_float4(hi.x, hi.y, lo.x, lo.y);
            }
        } else {
            // a complex64 vector: scaled by 1/beta as an FP32 pair, rounded once
            const float2* src = reinterpret_cast<const float2*>(in);
            float sh = 1.f, sl = 0.f;
            int brk = 0;
            for (int i0 = warp;;) {
                float2 pre[kPre];
#pragma unroll
                for (int u = 0; u < kPre; ++u) {
                    const int it = i0 + u * nw, row = it & rmask, q = (it >> lg) * 32 + lane;
                    pre[u] = row < rows && q < RB ? src[gidx(row, q)] : make_float2(0.f, 0.f);
                }
                if (i0 == warp) {
                    zero_tails();                      // while the first loads are in flight
                    if (late) {
                        __syncthreads();               // with the warp that forms 1/beta
                        sh = s_ibf.x;
                        sl = s_ibf.y;
                        brk = s_brk;
                    } else if (scale_mode) {
                        sh = ctrl->inv_beta_f[0];
                        sl = ctrl->inv_beta_f[1];
                    }
                }
#pragma unroll
                for (int u = 0; u < kPre; ++u) {
                    const int it = i0 + u * nw, row = it & rmask, q = (it >> lg) * 32 + lane;
                    if (row >= rows || q >= RB) continue;
                    float2 v = pre[u];
                    if (scale_mode) v = make_float2(mul_pair(v.x, sh, sl), mul_pair(v.y, sh, sl));
                    if (vstore && q < cl && !brk) reinterpret_cast<float2*>(vstore)[gidx(row, q)] = v;
                    unsigned short* rr = r16 + 2 * row * PQ + q;
                    put_split(rr, PL, v.x);
                    put_split(rr + PQ, PL, v.y);
                    bf[row * PB + q] = make_float4(v.x, v.y, 0.f, 0.f);
                }
                i0 += kPre * nw;
                if (i0 >= nbs) break;
            }
        }
        if (STAGE) cp_async_wait_all();
        worker_sync(nw);
        if (late && s_brk) return;                     // uniform: the same beta in every CTA
    }
    if (s_skip) {
        if (R64) __syncthreads();
        return;
    }

    const bool pair = !R64 || P >= 2;                  // the first residual comes from FP32 pairs
    const double* const ub = STAGE ? Us : tab.u + (size_t)q0 * UP;
    const float2* const ufb = STAGE ? Ufs : tab.uf + (size_t)q0 * UP;
    for (int k = 0; k <= P; ++k) {
        const int Rk = min(left, cl + (P - k) * (w + KD));
        if (k > 0) {
            if (16 * ft < Rk) load_frags(fr, Mg + ft * ks * 96);
            const int Rr = min(left, Rk + w), nrs = ((Rr + 31) >> 5) << lg;
            for (int it = warp; it < nrs; it += nw) {
                const int row = it & rmask, q = (it >> lg) * 32 + lane;
                if (row >= rows || q >= Rr) continue;
                unsigned short* rr = r16 + 2 * row * PQ + q;
                if (k == 1 && pair) {
                    // r = b - U~ x0, x0 exact in FP32, from FP32 pairs: relative error ~2^-48 |b| / |r|,
                    // far below what a pass needs whose result is refined again or rounded to FP32
                    const float2* xp = x0f + row * PX + q;
                    const float2* up = ufb + q * UP;
                    float4 b;                          // b's FP32 pairs
                    if constexpr (R64) {
                        const double2 v = bq[row * PB + q];
                        b = make_float4(d2f_fast<kBias>(v.x), d2f_fast<kBias>(v.y), d2f_low<kBias>(v.x), d2f_low<kBias>(v.y));
                    } else {
                        b = bf[row * PB + q];
                    }
                    float hr = 0.f, lr = 0.f, hi = 0.f, li = 0.f;
#pragma unroll
                    for (int d = 0; d <= KD; ++d) {
                        const float2 u = row_ld<STAGE>(up + d);
                        const float2 xv = xp[d];
                        acc_prod(hr, lr, u.x, u.y, xv.x);
                        acc_prod(hi, li, u.x, u.y, xv.y);
                    }
                    float s, e;
                    two_sum(b.x, -hr, s, e);
                    put_split(rr, PL, __fadd_rn(s, __fadd_rn(e, __fsub_rn(b.z, lr))));
                    two_sum(b.y, -hi, s, e);
                    put_split(rr + PQ, PL, __fadd_rn(s, __fadd_rn(e, __fsub_rn(b.w, li))));
                } else if constexpr (R64) {
                    const double2* xp = xd + row * PD + q;
                    const double* up = ub + q * UP;
                    double2 r = bq[row * PB + q];
#pragma unroll
                    for (int d = 0; d <= KD; ++d) {
                        const double u = row_ld<STAGE>(up + d);
                        const double2 xv = xp[d];
                        r.x = fma(-u, xv.x, r.x);
                        r.y = fma(-u, xv.y, r.y);
                    }
                    put_split(rr, PL, d2f_fast<kBias>(r.x));
                    put_split(rr + PQ, PL, d2f_fast<kBias>(r.y));
                }
            }
            if (R64 && k == P) __syncthreads();        // with the warp that forms 1/beta
            else worker_sync(nw);
        }
        const bool last = k == P;
        if (R64 && last && late) {
            if (s_brk) return;                         // uniform: the same beta in every CTA
            fin *= s_ib;
        }
        const bool rnd = R64 && (probe & 2);           // precision probe
        const int nt = (warp & ((1 << lnt) - 1)), row = 4 * nt + (lane & 3);
        const unsigned* rt = reinterpret_cast<const unsigned*>(r16) + (8 * nt + (lane >> 2)) * (PQ >> 1) + (lane & 3);
        for (int bk = ft; 16 * bk < Rk; bk += nw >> lnt) {
            const uint4* frag = Mg + bk * ks * 96;
            if (bk != ft) load_frags(fr, frag);
            float d[4];
            band_tile(d, frag, fr, ks, rt + 8 * bk, PL >> 1);
            if (row >= rows) continue;
            const int q = 16 * bk + (lane >> 2);
            if (k == 0 && pair) {
                float2* xp = x0f + row * PX + q;
                xp[0] = make_float2(d[0], d[1]);
                xp[8] = make_float2(d[2], d[3]);
            } else if constexpr (R64) {
                double2 x[2];
#pragma unroll
                for (int j = 0; j < 2; ++j) x[j] = make_double2(f2d_fast<kBias>(d[2 * j]), f2d_fast<kBias>(d[2 * j + 1]));
                double2* xp = xd + row * PD + q;
                if (k == 1 && pair) {
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const float2 x0 = x0f[row * PX + q + 8 * j];
                        x[j].x += f2d_fast<kBias>(x0.x);
                        x[j].y += f2d_fast<kBias>(x0.y);
                    }
                } else if (k > 0) {
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const double2 xo = xp[8 * j];
                        x[j].x += xo.x;
                        x[j].y += xo.y;
                    }
                }
                if (!last) {
                    xp[0] = x[0];
                    xp[8] = x[1];
                    continue;
                }
                if (scale_mode) {
#pragma unroll
                    for (int j = 0; j < 2; ++j) x[j] = make_double2(x[j].x * fin, x[j].y * fin);
                }
                if (rescaled) {
                    const int e = s_e[row];
#pragma unroll
                    for (int j = 0; j < 2; ++j) x[j] = make_double2(scale_pow2(x[j].x, e), scale_pow2(x[j].y, e));
                }
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    if (q + 8 * j >= cl) break;
                    const size_t gi = gidx(row, q + 8 * j);
                    // (the integer conversions: an FP64 conversion instruction costs what an FMA does)
                    const float2 f = make_float2(d2f_fast(x[j].x), d2f_fast(x[j].y));
                    if (out_prec) reinterpret_cast<float2*>(out)[gi] = f;
                    else reinterpret_cast<double2*>(out)[gi] = rnd ? make_double2(f2d_fast(f.x), f2d_fast(f.y)) : x[j];
                }
            } else {
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    if (q + 8 * j >= cl) break;
                    const float2 x0 = x0f[row * PX + q + 8 * j];
                    reinterpret_cast<float2*>(out)[gidx(row, q + 8 * j)] =
                        make_float2(__fadd_rn(x0.x, d[2 * j]), __fadd_rn(x0.y, d[2 * j + 1]));
                }
            }
        }
        if (R64 && last && vstore) {
            // the basis vector v = in / beta
            const int e = rescaled ? s_e[warp & rmask] : 0;
            const int nvs = ((cl + 31) >> 5) << lg;
            for (int it = warp; it < nvs; it += nw) {
                const int row = it & rmask, q = (it >> lg) * 32 + lane;
                if (row >= rows || q >= cl) continue;
                const double2 b = bq[row * PB + q];
                double2 v = make_double2(b.x * fin, b.y * fin);
                if (e) v = make_double2(scale_pow2(v.x, e), scale_pow2(v.y, e));
                reinterpret_cast<double2*>(vstore)[gidx(row, q)] = v;
            }
        }
        if (!last) worker_sync(nw);
    }
}

template <int KD, bool R64, bool STAGE>
static cudaError_t solve_rows_launch(const InvTab& tab, int nl, const void* in, int in_prec, void* out, int out_prec,
                                     void* vstore, Ctrl* ctrl, int dir, int scale_mode, int check_broken,
                                     cudaStream_t s, float4* v0s, const void* bpart, int bG) {
    const size_t smem = tab.ly.bytes;
    auto kern = k_solve_rows<KD, R64, STAGE>;
    if (smem > 48 * 1024) {
        cudaError_t ea = allow_max_smem(kern);
        if (ea != cudaSuccess) return ea;
    }
    dim3 grid(tab.nchunks, (nl + (1 << tab.lg) - 1) >> tab.lg), block(32 * tab.warps + 32);
    cudaError_t el = launch_pdl(kern, grid, block, smem, s, tab, nl, in, in_prec, out, out_prec, vstore, v0s, ctrl,
                                dir, scale_mode, check_broken, bpart, bG);
    return el != cudaSuccess ? el : cudaGetLastError();
}

template <int KD>
static cudaError_t solve_rows_kd(const InvTab& tab, int nl, int refine64, const void* in, int in_prec, void* out,
                                 int out_prec, void* vstore, Ctrl* ctrl, int dir, int scale_mode, int check_broken,
                                 cudaStream_t s, float4* v0s, const void* bpart, int bG) {
#define GB_ROWS(R64_, STAGE_)                                                                                       \
    return solve_rows_launch<KD, R64_, STAGE_>(tab, nl, in, in_prec, out, out_prec, vstore, ctrl, dir, scale_mode, \
                                               check_broken, s, v0s, bpart, bG)
    if (refine64) {
        if (tab.stage) GB_ROWS(true, true);
        GB_ROWS(true, false);
    }
    if (tab.stage) GB_ROWS(false, true);
    GB_ROWS(false, false);
#undef GB_ROWS
}

cudaError_t launch_solve_inv(const InvTab& tab, int nrows, int refine64, const void* in, int in_prec, void* out,
                             int out_prec, void* vstore, int v_prec, Ctrl* ctrl, int dir, int scale_mode,
                             int check_broken, cudaStream_t s, float4* v0s, const void* bpart, int bG) {
    count_launch();
    // the combinations the runtime uses: FP64-accurate solves store v in FP64 (or not at all), the
    // complex64 solve gives complex64 and stores v as it came (the split only of an FP64 vector)
    if (refine64 ? (vstore && v_prec != 0) || v0s : out_prec != 1 || (vstore && v_prec != in_prec) || (v0s && in_prec) || (bpart && !in_prec))
        return cudaErrorInvalidValue;
    switch (tab.kd) {
#define GB_KD(K)                                                                                                 \
    case K:                                                                                                      \
        return solve_rows_kd<K>(tab, nrows, refine64, in, in_prec, out, out_prec, vstore, ctrl, dir, scale_mode, \
                                check_broken, s, v0s, bpart, bG);
        GB_KD(1) GB_KD(2) GB_KD(3) GB_KD(4) GB_KD(5) GB_KD(6) GB_KD(7) GB_KD(8)
#undef GB_KD
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace gbprop
