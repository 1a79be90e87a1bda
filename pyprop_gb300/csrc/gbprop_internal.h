// Internal declarations shared by the host runtime (gbprop_api.cpp) and the
// CUDA kernels (gbprop_kernels.cu).  Not part of the C ABI.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace gbprop {

constexpr int kMaxBasis = 45;       // largest krylov_basis_size a handle accepts (7 m*m complex in smem)
constexpr int kWarp = 32;
constexpr int kSolveLanes = 32;     // radial blocks per l-row in the parallel solve
constexpr int kMaxKd = 8;           // largest band half-width of the overlap factor (order 9)

template <typename T> struct cx_of;
template <> struct cx_of<double> { using type = double2; };
template <> struct cx_of<float> { using type = float2; };
template <typename T> using cx = typename cx_of<T>::type;

// Tables of the parallel upper-band triangular solve U x = b in "e" coordinates
// (e = p for U^-1, e = n-1-p for U^-T), block-interleaved so that lane B of a
// warp reads entry (.., i, B) coalesced.  Built on the host in FP64.
//   n       radial length,  kd  superdiagonals,  L  block length,  P  blocks (<= 32)
//   ud      ((d-1)*L + i)*32 + B : U(e, e+d) / U(e, e), d = 1..kd, zero outside the block
//   invd    i*32 + B             : 1 / U(e, e), zero for e >= n
//   g       (c*L + i)*32 + B     : coupling of x_e to x_{(B+1)L + c} (within-block solve of
//                                  the block's upper-right corner), zero for the last block
//   mlev    ((lev*32 + B)*kd + r)*kd + c : suffix-scan operators of the kd-vector recurrence
//                                  t_B = y_B[0:kd] - F_B t_{B+1}, lev = 0..levels-1
template <typename T> struct SolveTab {
    int n, kd, L, P, levels, dir;
    const T* ud;
    const T* invd;
    const T* g;
    const T* mlev;
};

// Banded approximate inverse of one direction of the overlap-factor solve, in solve
// coordinates q (q = p for U x = b, q = n-1-p for U^T x = b), where both directions
// are upper triangular:  U~(q, q+d), d = 0..kd  and  M(q, q+j) ~ U~^-1(q, q+j), j = 0..w.
// U^-1 of a B-spline overlap factor decays geometrically away from the diagonal, so
// w is chosen (on the host) where the dropped part is below 2^-26 of the kept one.
//   mf  bfloat16, blocks of sixteen outputs, ks steps of sixteen columns (16 ks >= w + 16, a multiple
//       of kSolveFrags steps, which the kernel loads at once) and three parts whose sum is the FP32
//       M(r, c), in the fragment order of mma.m16n8k16: entry (((B*ks + s)*3 + part)*32 + lane)*8 + e with
//       r = 16B + lane/4 + 8 (e/2 % 2), c = 16B + 16s + 2 (lane%4) + e%2 + 8 (e/4); zero outside the band
//       and the matrix
//   u   q*inv_upitch(kd) + d  FP64 (an odd row length: a warp's rows lie in different banks), zero
//       where q + d >= n; npad rows, npad = n rounded up to 4
//   uf  the same entries split into FP32 pairs u = uf.x + uf.y, for the error-free residuals
// Each CTA owns `chunk` radial elements (a multiple of 16) of `rg` rows and recomputes the halo its
// refinement passes need; stage = 1 copies the chunk's slices of U~ into shared memory (16-byte
// asynchronous copies: q0 and npad are multiples of 4).
// (five k steps are the inverse bands of orders 7 and 8, 52 to 63 columns, in one round of loads; orders 4 to 6, which
// have three or four, multiply one or two blocks of zeros, order 9 with six a second round of five)
constexpr int kSolveFrags = 5;
__host__ __device__ constexpr int inv_upitch(int kd) { return (kd + 1) | 1; }

// Byte offsets of a solve CTA's shared memory: U~ slices (staged) | right-hand side (FP64 complex, or
// complex FP32 pairs) | FP64 iterate | residual in bfloat16 parts | FP32 first iterate.
struct InvLayout {
    int u, uf, b, x, r16, x0, bytes;
};

struct InvTab {
    int n, kd, w, npad;
    int ks;                 // k steps of a block
    int lg;                 // log2 of the rows per CTA
    int warps;              // worker warps per CTA (8 or 16), at least as many as rows
    int chunk, nchunks;
    int refine;             // refinement passes of the FP64-accurate solve
    int stage;
    int pq, px, pd, pb, pl; // shared-memory pitches (inv_shape)
    InvLayout ly;
    const unsigned short* mf;
    const double* u;
    const float2* uf;
};

// Region of the CTA whose chunk starts at q0, for P refinement passes: cl elements written,
// x kept on [q0, q0 + R0), right-hand side read on [q0, q0 + RB).
__host__ __device__ inline void inv_region(int n, int q0, int chunk, int P, int w, int kd, int* cl, int* R0, int* RB) {
    const int left = n - q0;
    *cl = chunk < left ? chunk : left;
    const int r0 = *cl + P * (w + kd);
    *R0 = r0 < left ? r0 : left;
    const int rb = *R0 + w;
    *RB = rb < left ? rb : left;
}

// Shared-memory pitches and offsets of a solve CTA (the same for every chunk, sized by the first):
// residual entries per plane (8 mod 64: the eight planes and four pairs of columns of a B fragment lie
// in 32 banks), x0 complex64 per row (4 mod 16) and x complex128 per row (2 mod 8), whose four rows by
// four or two columns an accumulator fragment stores together, b complex per row.
inline void inv_shape(InvTab& t, int r64) {
    int cl, R0, RB;
    const int P = r64 ? t.refine : 1;
    inv_region(t.n, 0, t.chunk, P, t.w, t.kd, &cl, &R0, &RB);
    const int r0 = (R0 + 15) & ~15;
    const int d = P >= 2 ? cl + (P - 1) * (t.w + t.kd) : R0;      // the FP64 iterate starts after an FP32-pair pass
    const int rd = ((d < R0 ? d : R0) + 15) & ~15;
    const int vq = r0 + 16 * t.ks > RB ? r0 + 16 * t.ks : RB;
    t.pq = ((vq - 8 + 63) & ~63) + 8;
    t.px = ((r0 + t.kd - 4 + 15) & ~15) + 4;
    t.pd = ((rd + t.kd - 2 + 7) & ~7) + 2;
    t.pb = RB;
    const int rows = 1 << t.lg, ub = ((R0 + 3) & ~3) * inv_upitch(t.kd) * 8;
    int o = 0;
    t.ly.u = o;
    if (t.stage && r64) o += ub;
    t.ly.uf = o;
    if (t.stage) o += ub;
    t.ly.b = o;
    o += rows * t.pb * 16;
    t.ly.x = o;
    if (r64) o += rows * t.pd * 16;
    t.ly.r16 = o;
    t.pl = 2 * (rows < 4 ? 4 : rows) * t.pq;         // whole groups of eight planes
    o += 3 * t.pl * 2;                               // (a multiple of 16 bytes: 8 planes, pq a multiple of 8)
    t.ly.x0 = o;
    o += rows * t.px * 8;
    t.ly.bytes = o;
}

// Term list of the tensor-potential matvec, grouped by destination row l:
//   y[l][i] += coef_t * s_t * sum_d slot[t][d][i] * x[src_t][i + d - kb]
// slots are real bands stored diagonal-major: (slot*(2kb+1) + d)*nr + i = A(i, i+d-kb).
template <typename T> struct BandOp {
    int nl, nr, kb, nterms;
    int variant;             // tile shape of the band kernel (chosen by the autotuner)
    const int* row_ptr;      // nl + 1
    const int* t_src;        // nterms
    const int* t_slot;       // nterms
    const int* t_timedep;    // nterms: 0 static, k >= 1 scaled by time function k
    const double* t_coef;    // 2 * nterms (re, im)
    const T* slots;
    const T* slots_lo;       // FP32 only: slot - (float)slot, the coefficients' rounding remainder
    // the same terms as nl x maxt descriptors: source row (-1: none), slot, time function (0: static), 1
    // where the factor is i instead of 1
    int maxt;
    const int4* desc;
    // FP64, variants 11 and 12 only (else null): the slots as 58-bit fixed-point numbers (see split29) at each
    // row's largest exponent
    int nslots;
    const int2* fslots;
    const int* fexp;         // nslots x nr
};

// Device control block of one handle.  Every field is written by kernels only, except
// inject_lu, wait_limit and round_matvec (set by the host through gbprop_debug_set).
struct Ctrl {
    int step;               // index of the current entry of the schedule array
    int broken;             // happy breakdown seen in the current step
    int nbasis;             // Krylov vectors built in the current step
    int scaling_order;      // s of the last scaling-and-squaring
    // error flags (sticky until the host reports them; kept adjacent: copied and cleared as one)
    int lu_info;            // last non-zero LU info of the Pade solve
    int nonfinite;          // a NaN/Inf norm was seen
    int wait_timeout;       // a bounded device-side wait (bulk-copy staging, grid barrier) gave up
    int inject_lu;          // test hook: the next exponentials report a zero pivot (host-set)
    long long wait_limit;   // polls of a launch's first bounded wait: 0 = default, < 0 = give up at once
    int round_matvec;       // precision probe (host-set): bit 0 band outputs, bit 1 solve and
                            // Gram-Schmidt outputs of FP64 handles rounded to complex64
    int ro_go;              // re-orthogonalisation requested for the current vector
    int ro_count;           // re-orthogonalisation passes done for the current vector
    long long operator_count;
    long long inner_product_count;
    long long orthogonalization_count;
    long long breakdown_count;
    long long step_count;
    double beta0;           // ||U psi|| at the start of the step
    double beta;            // current residual norm
    double inv_beta;        // 1 / beta (the reference scales by the reciprocal)
    float inv_beta_f[2];    // inv_beta as an FP32 pair (hi, lo) for the complex64 solve
    double orig_norm;       // ||w|| before Gram-Schmidt (re-orthogonalisation rule; updated per pass)
    double pre_norm;        // ||w|| of the operator output, before any Gram-Schmidt pass
    double resid_norm;      // ||w|| after Gram-Schmidt
    double err_est;         // |y[m-1]|^2
    double h[2 * kMaxBasis];
    double h3[2 * kMaxBasis];
    double y[2 * kMaxBasis];
};

// Up to this many distinct time functions per handle (the consolidated TensorPotentials of
// one problem, each scaled by its own f(t), TensorPotential.py:98-100).
constexpr int kMaxTimeFuncs = 4;

// Values of the time functions at one instant: s[k] scales the terms of time function k + 1.
struct Scalings {
    double s[kMaxTimeFuncs];
};

// Schedule entry per step: the time functions at the step start and the complex time step.
struct SchedEntry {
    Scalings scaling;
    double dt_re;
    double dt_im;
};

// Message returned by gbprop_last_error() on the calling thread.
void set_last_error(const char* msg);

// Launch counter shared by all launchers (process-wide).
void count_launch(int n = 1);
long long launch_count();

// ---- launchers (gbprop_kernels.cu) -------------------------------------------
// All return the cudaGetLastError() of their launch.
// Parallel banded triangular solve, one warp per l-row.
//   in_prec/out_prec/v_prec: 0 = complex128, 1 = complex64;  arith: 0 = double, 1 = float
//   scale_mode 1 multiplies the input by ctrl->inv_beta; vstore (if not null) receives the
//   scaled input; check_broken skips the launch body after a happy breakdown.
cudaError_t launch_solve(int arith, const void* tab, int nrows, const void* in, int in_prec,
                         void* out, int out_prec, void* vstore, int v_prec, const Ctrl* ctrl,
                         int scale_mode, int check_broken, cudaStream_t s);
// FP64-accurate solve: FP32 block solve + FP64 iterative refinement, one CTA per row.
// tabf: SolveTab<float> of the direction; udp: (kd+1) x nr diagonals U(i, i+d) in FP64.
cudaError_t launch_solve_ir(const void* tabf, const double* udp, int nrows, const void* in, int in_prec, void* out,
                            int out_prec, void* vstore, int v_prec, const Ctrl* ctrl, int scale_mode, int check_broken,
                            cudaStream_t s);
// Solve through the banded approximate inverse of the overlap factor (see InvTab):
// x = M b in FP32, then `refine` passes x += M (b - U~ x), the last with FP64 residuals when
// refine64 is set (FP64-accurate result).  refine64 = 0 is the complex64 solve of the mixed
// path's Krylov basis: one refinement whose residual is formed with error-free FP32 products
// and sums, complex64 output.  in and out must not overlap (a chunk's halo is read by its
// neighbour).  check_broken 2: nothing is written once ctrl->wait_timeout is set.  Grid: (tab.nchunks, row groups); arguments as launch_solve.
// v0s (complex64 solve of the FP64 first vector only, may be null) receives the scaled input
// split into FP32 pairs, float4 (re_hi, im_hi, re_lo, im_lo) per element.  bpart (scale_mode
// 1, may be null): the cooperative Gram-Schmidt kernel's bG per-CTA ||w||^2 partials (double,
// or float4 FP32 pairs for refine64 = 0); the solve forms beta from them, records it in ctrl
// (breakdown test, 1/beta) and scales by 1/beta, instead of reading ctrl->inv_beta.
cudaError_t launch_solve_inv(const InvTab& tab, int nrows, int refine64, const void* in, int in_prec, void* out,
                             int out_prec, void* vstore, int v_prec, Ctrl* ctrl, int dir, int scale_mode,
                             int check_broken, cudaStream_t s, float4* v0s = nullptr, const void* bpart = nullptr,
                             int bG = 0);
// sched (device, may be null): the time functions come from sched[ctrl->step]; else `scaling`.
cudaError_t launch_band_apply(int arith, const void* op, const void* x, void* y, const SchedEntry* sched,
                              const Ctrl* ctrl, const Scalings& scaling, int check_broken, cudaStream_t s);
cudaError_t launch_tbmv(int arith, int kd, const void* ud_phys, int nl, int nr, const void* in, int in_prec,
                        void* out, int out_prec, cudaStream_t s);
cudaError_t launch_norm(int prec, const void* x, long n, double* partials, unsigned* counter, Ctrl* ctrl,
                        cudaStream_t s);
// x <- x / ||x|| (FP64 state): a k_norm launch and a scaling launch.
cudaError_t launch_renormalize(double2* x, long n, double* partials, unsigned* counter, Ctrl* ctrl,
                               cudaStream_t s);
// v0 (complex64 basis only, may be null): FP64 copy of the first basis vector, used in
// place of V row 0 by the dot, the update and the combination.
// v0: the FP64 first vector of a complex64 basis; v0s: its FP32-pair split (hi, lo), read
// instead when given (written by the inverse-band solve of that vector)
cudaError_t launch_cgs_dot(int prec, const void* V, const double2* v0, const float4* v0s, long n, int nv,
                           const void* w, double* partials, unsigned* counter, Ctrl* ctrl, int mode, int want_norm,
                           cudaStream_t s);
// Stateless block inner product into a caller buffer (out: 2nv doubles, + ||w||^2 when want_norm).
size_t block_inner_scratch_doubles(long n, int nvals);
cudaError_t launch_block_inner(int prec, const void* V, long n, int nv, const void* w, int want_norm, double* out,
                               double* partials, unsigned* counter, cudaStream_t s);
// mode: bit 0 re-orthogonalisation pass, bit 1 double orthogonalisation requested, bit 2 the
// last block also finalizes Arnoldi step nv - 1 (H column, beta, breakdown; H, m, brk_tol as
// launch_arnoldi_finalize)
cudaError_t launch_cgs_update(int prec, const void* V, const double2* v0, const float4* v0s, long n, int nv, void* w,
                              double* partials, unsigned* counter, Ctrl* ctrl, int mode, cudaStream_t s,
                              double* H = nullptr, int m = 0, double brk_tol = 0.0);
// brk_tol: happy-breakdown threshold on the new basis norm (pAMP: sqrt(eps), pamp.h:79;
// Expokit: 1e-7).
cudaError_t launch_arnoldi_finalize(Ctrl* ctrl, double* H, int m, int J, int double_orth, double brk_tol,
                                    cudaStream_t s);
// One Arnoldi step's Gram-Schmidt (dot, update, norm, Hessenberg column, breakdown) as a
// single cooperative kernel of `grid` co-resident CTAs (gbprop_cgs.cu).  part: at least
// arnoldi_cgs_part_doubles(grid) doubles; bar: two words, zero before the first launch.
// update = 0 forms only the Hessenberg column (last vector).  cache: keep V's chunk in
// shared memory between the two passes.
// dorth (FP64): re-orthogonalisation passes inside, and the column, the next beta and the breakdown
// test (brk_tol) complete on return, as launch_arnoldi_finalize leaves them.
// The complex64 form takes the first vector as FP32 pairs (v0s, see launch_solve_inv) and
// forms every sum with error-free FP32 transformations.  batch: the grid is arnoldi_cgs_grid_batch's.
cudaError_t launch_arnoldi_cgs(int prec, const void* V, const void* v0, long n, int J, int m, void* w,
                               double* part, unsigned* bar, Ctrl* ctrl, double* H, int update, int grid, int cache,
                               int dorth, double brk_tol, void* Vd, int* ev_rows, int batch, cudaStream_t s);
// FP64, rows cached: the fixed-point form's digits and FP32 values of the step's basis vectors,
// arnoldi_cgs_digits_bytes bytes at Vd (0: it does not apply), and their chunks' exponents, kMaxBasis * grid at
// ev_rows.  Null: the FP64 form.
size_t arnoldi_cgs_digits_bytes(int prec, long n, int m, int grid, int cache);
// Grid size for the cooperative Gram-Schmidt (0 if it cannot run co-resident).
int arnoldi_cgs_grid(int prec, long n, int m, int with_v0, int cache, int dorth);
int arnoldi_cgs_grid_batch(int prec, long n, int m, int with_v0, int* cache);
inline size_t arnoldi_cgs_part_doubles(int grid) { return (size_t)(2 * (kMaxBasis + 1) + 1) * grid; }
cudaError_t launch_step_begin(Ctrl* ctrl, double* H, int m, cudaStream_t s);
// max_cluster: 16 lets one problem's exponential spread over a thread-block cluster; 1 keeps it on
// one CTA (batches, where other problems fill the GPU).
// df32 = 1 (FP32-mixed handles): the cluster form in double-float arithmetic (gbprop_expm.cu).
cudaError_t launch_expm(Ctrl* ctrl, double* H, int m, const SchedEntry* sched, int max_cluster, cudaStream_t s,
                        int df32 = 0);
// krylov_exponentiation_method = 1 (pamp.h:567-607): y from the eigen-decomposition, one CTA.
cudaError_t launch_expm_eig(Ctrl* ctrl, double* H, int m, const SchedEntry* sched, cudaStream_t s);
// cluster: 16 or 8 CTAs, or 1 (one CTA, for batches; when expm_df_single_fits(m))
cudaError_t launch_expm_df(Ctrl* ctrl, double* H, int m, const SchedEntry* sched, int cluster, cudaStream_t s);
bool expm_df_single_fits(int m);
cudaError_t launch_combine(int prec, const void* V, const double2* v0, long n, const Ctrl* ctrl, void* out,
                           cudaStream_t s);
cudaError_t launch_step_end(Ctrl* ctrl, cudaStream_t s);
// out[0..2] = max of the members' (lu_info, nonfinite, wait_timeout); out[3] = 1 + the first
// member with any of them set (0 if none).  One CTA.
cudaError_t launch_gather_flags(Ctrl* const* ctrls, int count, int* out, cudaStream_t s);
cudaError_t launch_tensor_multiply_ref(int storage, const double2* V, int npairs, const int* pairs, int kb,
                                       double scaling, const double2* src, double2* dst, int nl, int nr,
                                       cudaStream_t s);
cudaError_t launch_zero(void* p, size_t bytes, cudaStream_t s);

int grid_reduce_blocks();
int band_variant_count();
constexpr int kBandFixed = 11;               // the first of the fixed-point forms
// fixed-point form of FP64 slots (nslots x (2 kb + 1) x nr) and the row exponents (nslots x nr)
cudaError_t launch_band_fixed_slots(const double* slots, int nslots, int nr, int width, int2* digits, int* exps,
                                    cudaStream_t s);
bool band_variant_vec_ok(int v, int nr);    // the variant's radial-size condition (even nr for 6, 7, 8)
// Bound states of banded generalized symmetric problems (gbprop_bound.cu; see gbprop_bound_states)
cudaError_t launch_bound_states(const double* Hb, const double* Sb, int n, int kd, int nrows, double emax,
                                int max_states, int* counts, double* energies, double* vectors, cudaStream_t s,
                                int* ntasks);
size_t partials_capacity();

}  // namespace gbprop
