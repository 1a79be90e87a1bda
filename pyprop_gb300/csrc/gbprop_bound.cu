// Field-free bound states on the GPU: the eigenpairs with E < emax of the generalized
// symmetric banded problems H_l c = E S c, one per angular row l (the static, angular-diagonal
// TensorPotentials in the B-spline overlap metric).  The reference's hydrogen analysis solves
// them with a dense generalized eigensolver per l
// (examples/tensor/helium_stabilization_sae/analysis.py:92-160); here the band structure is
// used directly:
//   * inertia: the number of eigenvalues below sigma is the number of negative pivots of the
//     banded LDL^T factorisation of H - sigma S (Sylvester's law of inertia, S positive
//     definite), O(n kd^2) per count with a sliding window of the last kd rows of L in
//     registers;
//   * bisection on that count for every wanted eigenvalue, one CTA per (row, index): a round
//     evaluates all midpoints that the next 5 to 7 bisections can meet, a thread each.  A count is a
//     serial chain of n rows (an FP64 instruction occupies its SM sub-partition for 64 cycles whether
//     one lane or all are active), so shifts are free up to the warps that fill the GPU: about 9 rounds
//     with 127 shifts where one after the other are 60 counts;
//   * inverse iteration at the converged eigenvalue (three banded LDL^T solves, the factor kept
//     in a global scratch array), normalised in the S metric: one warp per state, the rows after a
//     solved one updated by the lanes that own them.
// Measured (33 rows x 800 B-splines): 128 ms with one thread per state, 22 ms now; bound by the chain of
// n rows of dependent FP64 instructions a count, about 11 counts in sequence.
// Bands are diagonal-major: A[d * n + i] = A(i, i + d - kd), d = 0..2kd (symmetric; only the
// lower half and the diagonal are read).
#include "gbprop_internal.h"
#include "../../include/gbprop.h"

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <string>
#include <vector>

namespace gbprop {

namespace {

constexpr int kBoundThreads = 128;

// Banded LDL^T of A = H - sigma S, row by row: li[m] = L(i, i-KD+m), d_i the pivot.
// Returns the number of negative pivots; with Lout != null the factor rows are stored by the threads
// with `store`
// (Lout[i * (KD+1) + m] = L(i, i-KD+m), Lout[i * (KD+1) + KD] = 1 / d_i).
template <int KD>
__device__ int band_ldlt(const double* __restrict__ Hb, const double* __restrict__ Sb, int n, double sigma,
                         double* __restrict__ Lout, bool store) {
    double W[KD][KD];           // L rows of the previous KD rows (row r: W[r][m] = L(i-KD+r, i-2KD+r+m))
    double dp[KD], ip[KD];      // their pivots and inverse pivots
#pragma unroll
    for (int r = 0; r < KD; ++r) {
        dp[r] = 1.0;
        ip[r] = 0.0;            // rows before the start: no contribution
#pragma unroll
        for (int m = 0; m < KD; ++m) W[r][m] = 0.0;
    }
    int neg = 0;
    const double tiny = 1e-280;
    for (int i = 0; i < n; ++i) {
        double li[KD];
#pragma unroll
        for (int m = 0; m < KD; ++m) {
            const int j = i - KD + m;
            double a = 0.0;
            if (j >= 0) a = __ldg(Hb + (size_t)m * n + i) - sigma * __ldg(Sb + (size_t)m * n + i);
#pragma unroll
            for (int p = 0; p < m; ++p) a = fma(-li[p] * dp[p], W[m][p + KD - m], a);
            li[m] = a * ip[m];
        }
        double d = __ldg(Hb + (size_t)KD * n + i) - sigma * __ldg(Sb + (size_t)KD * n + i);
#pragma unroll
        for (int m = 0; m < KD; ++m) d = fma(-li[m] * li[m], dp[m], d);
        if (!(fabs(d) >= tiny)) d = (d < 0.0) ? -tiny : tiny;   // exact zero (or NaN): a tiny pivot
        neg += d < 0.0;
        const double id = 1.0 / d;
        if (Lout && store) {
#pragma unroll
            for (int m = 0; m < KD; ++m) Lout[(size_t)i * (KD + 1) + m] = li[m];
            Lout[(size_t)i * (KD + 1) + KD] = id;
        }
#pragma unroll
        for (int r = 0; r + 1 < KD; ++r) {
            dp[r] = dp[r + 1];
            ip[r] = ip[r + 1];
#pragma unroll
            for (int m = 0; m < KD; ++m) W[r][m] = W[r + 1][m];
        }
        dp[KD - 1] = d;
        ip[KD - 1] = id;
#pragma unroll
        for (int m = 0; m < KD; ++m) W[KD - 1][m] = li[m];
    }
    return neg;
}

template <int KD>
__global__ void __launch_bounds__(32) k_bound_count(const double* __restrict__ Hb, const double* __restrict__ Sb,
                                                    int n, int nrows, double emax, int* __restrict__ counts) {
    const int l = blockIdx.x;
    const int c = band_ldlt<KD>(Hb + (size_t)l * (2 * KD + 1) * n, Sb, n, emax, nullptr, false);
    if (threadIdx.x == 0) counts[l] = c;
}

// One CTA of 2^levels threads per (row, index k): the k-th smallest eigenvalue below emax by
// bisection on the inertia.  First the threads look for a lower end among the doublings of
// min(-1, emax - |emax| - 1); then a round evaluates the 2^levels - 1 midpoints that the next
// `levels` bisections can meet, thread j the node j of that tree, and walks down it.  The midpoints and
// with them the eigenvalue are those of plain bisection, bit for bit.
template <int KD>
__global__ void __launch_bounds__(kBoundThreads) k_bound_bisect(const double* __restrict__ Hb,
                                                                const double* __restrict__ Sb, int n,
                                                                const int2* __restrict__ tasks, double emax,
                                                                int levels, double* __restrict__ energy) {
    __shared__ int s_first;
    __shared__ unsigned char s_above[kBoundThreads];   // node j: more than k eigenvalues below its midpoint
    const int t = blockIdx.x, tid = threadIdx.x, nt = blockDim.x;
    const int l = tasks[t].x, k = tasks[t].y;
    const double* H = Hb + (size_t)l * (2 * KD + 1) * n;
    const double start = fmin(-1.0, emax - fabs(emax) - 1.0);
    double lo = start;
    // the first doubling with no eigenvalue below it (at most 64 of them)
    if (tid == 0) s_first = 64;
    __syncthreads();
    for (int i0 = 0; i0 < 64; i0 += nt) {
        const int i = i0 + tid;
        if (i < 64 && !(band_ldlt<KD>(H, Sb, n, ldexp(start, i), nullptr, false) > 0)) atomicMin(&s_first, i);
        __syncthreads();
        const int f = s_first;
        __syncthreads();
        lo = ldexp(start, f);
        if (f < 64) break;
    }
    double hi = emax;
    for (int it = 0; it < 200; it += levels) {
        // thread j >= 1: node j, its path from the root the bits of j below the leading one
        double a = lo, b = hi, mid = 0.5 * (a + b);
        for (int q = 30 - __clz(max(tid, 1)); q >= 0; --q) {
            if ((tid >> q) & 1) b = mid;
            else a = mid;
            mid = 0.5 * (a + b);
        }
        if (tid > 0) s_above[tid] = band_ldlt<KD>(H, Sb, n, mid, nullptr, false) > k;
        __syncthreads();
        bool done = false;
        int node = 1;
        for (int q = 0; q < levels && it + q < 200; ++q) {
            mid = 0.5 * (lo + hi);
            if (!(mid > lo && mid < hi)) {             // adjacent doubles: converged
                done = true;
                break;
            }
            const bool above = s_above[node];
            if (above) hi = mid;
            else lo = mid;
            node = 2 * node + (above ? 1 : 0);
        }
        __syncthreads();
        if (done) break;
    }
    if (tid == 0) energy[t] = 0.5 * (lo + hi);
}

// Inverse iteration at the converged eigenvalue: x <- (H - E S)^-1 S x three times from a fixed
// pseudo-random start, then x / sqrt(x^T S x).  One warp per state; scratch: (KD+1) n doubles for
// the factor and n for S x, per task.  The sweeps go 32 rows at a time, a lane per row: once a row is
// solved its value is broadcast and the lanes of the KD rows that follow subtract their share.
template <int KD>
__global__ void __launch_bounds__(32) k_bound_vector(const double* __restrict__ Hb, const double* __restrict__ Sb,
                                                     int n, const int2* __restrict__ tasks, int max_states,
                                                     const double* __restrict__ energy, double* __restrict__ scratch,
                                                     double* __restrict__ vectors) {
    constexpr unsigned kAll = 0xffffffffu;
    const int t = blockIdx.x, lane = threadIdx.x;
    const int l = tasks[t].x;
    const double* H = Hb + (size_t)l * (2 * KD + 1) * n;
    double* L = scratch + (size_t)t * (KD + 2) * n;
    double* sx = L + (size_t)(KD + 1) * n;
    double* x = vectors + ((size_t)l * max_states + tasks[t].y) * n;
    band_ldlt<KD>(H, Sb, n, energy[t], L, lane == 0);
    for (int i = lane; i < n; i += 32) {             // start: hashed values in [0.5, 1.5)
        unsigned h = (unsigned)i * 2654435761u + 0x9e3779b9u * (unsigned)(t + 1);
        h ^= h >> 15;
        h *= 0x2c1b3c6du;
        h ^= h >> 12;
        x[i] = 0.5 + (double)(h >> 8) * (1.0 / 16777216.0);
    }
    __threadfence_block();
    __syncwarp();
    auto sym_mul = [&](double* y) {                   // y = S x (symmetric band)
        for (int i = lane; i < n; i += 32) {
            double v = 0.0;
#pragma unroll
            for (int d = 0; d <= 2 * KD; ++d) {
                const int j = i + d - KD;
                if (j >= 0 && j < n) {
                    // S(i, j) from the lower half and the diagonal: S(i, j) = S(j, i) for j > i
                    const double s = d <= KD ? __ldg(Sb + (size_t)d * n + i) : __ldg(Sb + (size_t)(2 * KD - d) * n + j);
                    v = fma(s, x[j], v);
                }
            }
            y[i] = v;
        }
        __threadfence_block();
        __syncwarp();
    };
    const int nb = (n + 31) / 32;
    for (int pass = 0; pass < 3; ++pass) {
        sym_mul(sx);
        // forward: z_i = b_i - sum_m L(i, i-KD+m) z_{i-KD+m}, x_i = z_i / d_i
        double z = 0.0;                                // the lane's solved row of the previous block
        for (int b = 0; b < nb; ++b) {
            const int i = 32 * b + lane;
            double c[KD];                              // c[e-1] = L(i, i-e)
#pragma unroll
            for (int e = 1; e <= KD; ++e) c[e - 1] = i < n ? L[(size_t)i * (KD + 1) + KD - e] : 0.0;
            const double id = i < n ? L[(size_t)i * (KD + 1) + KD] : 0.0;
            double v = i < n ? sx[i] : 0.0;
#pragma unroll 2
            for (int s = -KD; s < 32; ++s) {
                const double zs = __shfl_sync(kAll, s < 0 ? z : v, s < 0 ? s + 32 : s);
                const int e = lane - s;
                double ce = 0.0;
#pragma unroll
                for (int u = 1; u <= KD; ++u) ce = e == u ? c[u - 1] : ce;
                if (e >= 1 && e <= KD) v = fma(-ce, zs, v);
            }
            z = v;
            if (i < n) x[i] = v * id;
        }
        __threadfence_block();
        __syncwarp();
        // backward: x_i = y_i - sum_{j=i+1}^{i+KD} L(j, i) x_j
        z = 0.0;
        double mx = 0.0;
        for (int b = nb - 1; b >= 0; --b) {
            const int i = 32 * b + lane;
            double c[KD];                              // c[e-1] = L(i+e, i)
#pragma unroll
            for (int e = 1; e <= KD; ++e) c[e - 1] = i + e < n ? L[(size_t)(i + e) * (KD + 1) + KD - e] : 0.0;
            double v = i < n ? x[i] : 0.0;
#pragma unroll 2
            for (int s = 31 + KD; s >= 0; --s) {
                const double zs = __shfl_sync(kAll, s > 31 ? z : v, s > 31 ? s - 32 : s);
                const int e = s - lane;
                double ce = 0.0;
#pragma unroll
                for (int u = 1; u <= KD; ++u) ce = e == u ? c[u - 1] : ce;
                if (e >= 1 && e <= KD) v = fma(-ce, zs, v);
            }
            z = v;
            if (i < n) {
                x[i] = v;
                mx = fmax(mx, fabs(v));
            }
        }
        // rescale (the solve amplifies by 1/|E - E_k|)
        for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(kAll, mx, o));
        const double s = mx > 0.0 ? 1.0 / mx : 0.0;
        for (int i = lane; i < n; i += 32) x[i] *= s;
        __threadfence_block();
        __syncwarp();
    }
    sym_mul(sx);
    double nrm = 0.0;
    for (int i = lane; i < n; i += 32) nrm = fma(x[i], sx[i], nrm);
    for (int o = 16; o > 0; o >>= 1) nrm += __shfl_xor_sync(kAll, nrm, o);
    const double s = nrm > 0.0 ? 1.0 / sqrt(nrm) : 0.0;
    for (int i = lane; i < n; i += 32) x[i] *= s;
}

template <int KD>
cudaError_t bound_kd(const double* Hb, const double* Sb, int n, int nrows, double emax, int max_states,
                     int* counts_host, double* energies_host, double* vectors, cudaStream_t s, int* ntasks_out) {
    int* d_counts = nullptr;
    cudaError_t e = cudaMallocAsync((void**)&d_counts, sizeof(int) * nrows, s);
    if (e != cudaSuccess) return e;
    count_launch();
    k_bound_count<KD><<<nrows, 32, 0, s>>>(Hb, Sb, n, nrows, emax, d_counts);
    if ((e = cudaGetLastError()) == cudaSuccess)
        e = cudaMemcpyAsync(counts_host, d_counts, sizeof(int) * nrows, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaFreeAsync(d_counts, s);
    if (e != cudaSuccess) return e;
    std::vector<int2> tasks;
    for (int l = 0; l < nrows; ++l) {
        const int c = counts_host[l] < max_states ? counts_host[l] : max_states;
        for (int k = 0; k < c; ++k) tasks.push_back(make_int2(l, k));
    }
    const int nt = (int)tasks.size();
    *ntasks_out = nt;
    for (int i = 0; i < nrows * max_states; ++i) energies_host[i] = 0.0;
    if (nt == 0) return cudaSuccess;
    int2* d_tasks = nullptr;
    double *d_energy = nullptr, *d_scratch = nullptr;
    e = cudaMallocAsync((void**)&d_tasks, sizeof(int2) * nt, s);
    if (e == cudaSuccess) e = cudaMallocAsync((void**)&d_energy, sizeof(double) * nt, s);
    if (e == cudaSuccess) e = cudaMallocAsync((void**)&d_scratch, sizeof(double) * (size_t)nt * (KD + 2) * n, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_tasks, tasks.data(), sizeof(int2) * nt, cudaMemcpyHostToDevice, s);
    // threads per state: as many warps as give every SM sub-partition one, 32 to kBoundThreads
    int levels = 7;
    while (levels > 5 && (long)nt << (levels - 5) > 4 * grid_reduce_blocks()) --levels;
    if (e == cudaSuccess) {
        count_launch();
        k_bound_bisect<KD><<<nt, 1 << levels, 0, s>>>(Hb, Sb, n, d_tasks, emax, levels, d_energy);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
        count_launch();
        k_bound_vector<KD><<<nt, 32, 0, s>>>(Hb, Sb, n, d_tasks, max_states, d_energy, d_scratch, vectors);
        e = cudaGetLastError();
    }
    std::vector<double> en(nt);
    if (e == cudaSuccess) e = cudaMemcpyAsync(en.data(), d_energy, sizeof(double) * nt, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    for (int t = 0; t < nt && e == cudaSuccess; ++t) energies_host[tasks[t].x * max_states + tasks[t].y] = en[t];
    cudaFreeAsync(d_tasks, s);
    cudaFreeAsync(d_energy, s);
    cudaFreeAsync(d_scratch, s);
    return e;
}

}  // namespace

cudaError_t launch_bound_states(const double* Hb, const double* Sb, int n, int kd, int nrows, double emax,
                                int max_states, int* counts, double* energies, double* vectors, cudaStream_t s,
                                int* ntasks) {
    switch (kd) {
        case 1: return bound_kd<1>(Hb, Sb, n, nrows, emax, max_states, counts, energies, vectors, s, ntasks);
        case 2: return bound_kd<2>(Hb, Sb, n, nrows, emax, max_states, counts, energies, vectors, s, ntasks);
        case 3: return bound_kd<3>(Hb, Sb, n, nrows, emax, max_states, counts, energies, vectors, s, ntasks);
        case 4: return bound_kd<4>(Hb, Sb, n, nrows, emax, max_states, counts, energies, vectors, s, ntasks);
        case 5: return bound_kd<5>(Hb, Sb, n, nrows, emax, max_states, counts, energies, vectors, s, ntasks);
        case 6: return bound_kd<6>(Hb, Sb, n, nrows, emax, max_states, counts, energies, vectors, s, ntasks);
        case 7: return bound_kd<7>(Hb, Sb, n, nrows, emax, max_states, counts, energies, vectors, s, ntasks);
        case 8: return bound_kd<8>(Hb, Sb, n, nrows, emax, max_states, counts, energies, vectors, s, ntasks);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace gbprop
