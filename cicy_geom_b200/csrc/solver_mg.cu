// Chain-aggregation multigrid (CAMG) preconditioned conjugate gradient for the
// DEA systems (device).
//
// Why: in a CNT resistor network the element resistors along one CNT conduct
// 1e4-1e9 times better than the tunnelling junctions between CNTs, so after the
// chain block-Jacobi has equilibrated every CNT the remaining error is "one
// potential per CNT", a graph Laplacian over CNTs with junction conductances
// spanning five orders of magnitude.  One-level preconditioners take thousands
// of iterations on it; a coarse space with one unknown per chain block removes
// it.  The hierarchy:
//
//   level 0   the free-node system; smoother: the chain blocks (explicit
//             tridiagonal inverses in the cluster kernels, LDL^T factors in the
//             grid kernel), damped by kOmega0 so 2 M^-1 - A stays
//             positive definite on floating islands (bipartite trees of CNTs
//             that no prescribed node reaches, where the undamped block smoother
//             would make the V-cycle singular)
//   level 1   one unknown per chain block (aggregate = block)
//   level l+1 pairwise aggregates of level l: three rounds of handshake
//             matching on the strongest coupling |a_ij| (ties: smaller j), then
//             every unmatched row joins the pair of its strongest neighbour
//   coarsest  dense inverse (Gauss-Jordan, 1e-8 diagonal regularisation,
//             variables with a vanishing pivot dropped) of up to kMgDenseMax rows,
//             by one CTA in shared memory, for the grid kernel of up to
//             kMgDenseGridMax, by the grid; otherwise an l1-Jacobi step
//
// Coarse operators are Galerkin products P^T A P with piecewise-constant P (the
// grid kernel's first one smoothed, see coarsen_smoothed): a warp or a CTA per
// aggregate gathers its members' cross-aggregate couplings, sorts them by coarse
// column and gather position and sums each column's run in that order
// (deterministic).  The host reads each level's size and entries, and the size of
// each product of the smoothed level.  Their diagonals come from summed row
// sums, diag_J = sum_{I in J} rowsum_I - sum_{J' != J} A_JJ', so the large
// intra-aggregate conductances never cancel in floating point and an aggregate
// with no outside coupling gets an exact zero row.  Levels >= 1 are smoothed by
// l1-Jacobi (1 / (|d| + sum |a|)), which makes the symmetric V(1,1)-cycle an SPD
// preconditioner.
//
// The solve is one persistent launch: a 16-CTA cluster (k_mg_pcg<true>) up to
// kMgClusterMaxRows rows, a cooperative grid with the operators in shared memory
// (k_mg_pcg_sm) above, clusters of 16, 8 or 4 CTAs in a batch (k_mg_batch).
// Level-0 rows are split over CTAs at block boundaries (the block smoother only
// reads rows of its own CTA); coarse levels are spread over all threads or dealt by
// entries.  Per CG iteration the barriers
// are: 1 after the pre-smoother and r.r, one per restriction, one after the
// coarse solve, one per prolongation above level 1, one after the post-smoother
// and r.z, one after p.q.  The stopping rule, FP64 true-residual replacement and
// the first-iteration behaviour are those of the one-level kernel (solver.cu).
#include <algorithm>
#include <cmath>
#include <vector>

#include "batch_shape.h"
#include "solver.cuh"
#include "trace.cuh"

namespace cicy {

namespace {

constexpr int kMgThreads = 256;
constexpr int kMgClusterThreads = 1024;
constexpr int kMgClusterCtas = 16;            // non-portable cluster size
// Largest system for the one-cluster kernel.  The shared-memory-resident grid kernel, with its fused
// rows, smoothed prolongator and larger dense coarsest, is faster as soon as the cluster's hierarchy
// has a third level: solve in ms, cluster / grid, 333 rows 0.33 / 0.35, 409 0.29 / 0.29, 448 0.34 / 0.36,
// 488 0.49 / 0.33, 1,552 0.90 / 0.40, 3,992 1.05 / 0.54, 10.2k 1.47 / 0.72, 18.5k 2.44 / 1.03; whole calls
// of 1,600 - 6,400 CNTs 3.7 - 7.3 against 2.7 - 4.9.  Several contexts at once gain too, although seven
// clusters fit at once and the grid takes up to every SM: eight threads with a context each make 491 calls/s
// with clusters up to 20,000 rows and 790 so on 1,000 CNTs, 240 and 318 on 6,400.
constexpr int kMgClusterMaxRows = 450;
constexpr int kMgMaxRestarts = 24;
constexpr double kOmega0 = 0.95;

int grid_for(long long n, int threads = 256) {
    long long b = (n + threads - 1) / threads;
    if (b < 1) b = 1;
    if (b > 148LL * 32) b = 148LL * 32;
    return (int)b;
}

// ---------------------------------------------------------------------------
// Setup kernels

__global__ void k_block_of_row(int n, const int32_t* __restrict__ is_start, const int32_t* __restrict__ start_scan,
                               int32_t* __restrict__ agg) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        agg[i] = start_scan[i] + is_start[i] - 1;
}

// Row sums of the level-0 matrix (diagonal included); a row sum at rounding level
// of its diagonal is an unconnected (floating) row: exactly 0.
__global__ void k_rowsum0(int n, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci, const double* __restrict__ v,
                          double* __restrict__ rs) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double s = 0, d = 0;
        for (int k = rp[i]; k < rp[i + 1]; k++) {
            s += v[k];
            if (ci[k] == i) d = v[k];
        }
        rs[i] = (fabs(s) <= 1e-13 * fabs(d)) ? 0.0 : s;
    }
}

// The setup's row kernels take `lanes` (a power of two up to 32) threads per row: rows have 2-5
// couplings on the chain level and hundreds on the lower levels of dense networks, where one
// thread per row read them one uncoalesced entry after another (47.7k-CNT / 5 um realisation:
// k_strongest 8.6 ms and k_rr_fill 9.7 ms in all, now 0.78 and 0.66 ms).
struct RowLanes {
    int first, step, lane;  // first row and row stride of the group, lane within it
};
__device__ __forceinline__ RowLanes row_lanes(int lanes) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    return RowLanes{t / lanes, (int)(gridDim.x * blockDim.x) / lanes, t % lanes};
}
int lanes_of(long long entries, int rows) {  // about two entries per thread
    int l = 1;
    while (l < 32 && 2LL * l * rows < entries) l <<= 1;
    return l;
}

// Strongest neighbour of each row (|a_ij| largest, ties: smaller j); with
// free_only, among unmatched rows and only for unmatched rows.
__global__ void k_strongest(int n, int lanes, int free_only, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                            const double* __restrict__ v, const int32_t* __restrict__ mate, int32_t* __restrict__ best) {
    const RowLanes g = row_lanes(lanes);
    const unsigned mask = lanes >= 32 ? 0xffffffffu : (((1u << lanes) - 1) << ((threadIdx.x & 31) & ~(lanes - 1)));
    for (int i = g.first; i < n; i += g.step) {
        int bj = -1;
        double bs = -1.0;
        if (!(free_only && mate[i] >= 0)) {
            for (int k = rp[i] + g.lane; k < rp[i + 1]; k += lanes) {
                const int j = ci[k];
                if (free_only && mate[j] >= 0) continue;
                const double s = fabs(v[k]);
                if (s > bs || (s == bs && j < bj)) {
                    bs = s;
                    bj = j;
                }
            }
        }
        for (int o = lanes / 2; o > 0; o >>= 1) {
            const double s = __shfl_xor_sync(mask, bs, o, lanes);
            const int j = __shfl_xor_sync(mask, bj, o, lanes);
            if (s > bs || (s == bs && j < bj)) {
                bs = s;
                bj = j;
            }
        }
        if (g.lane == 0) best[i] = bj;
    }
}

__global__ void k_handshake(int n, const int32_t* __restrict__ best, int32_t* __restrict__ mate) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int j = best[i];
        if (mate[i] < 0 && j >= 0 && best[j] == i) mate[i] = j;
    }
}

__global__ void k_pair_rep(int n, const int32_t* __restrict__ mate, int32_t* __restrict__ rep) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        rep[i] = mate[i] >= 0 ? min(i, mate[i]) : i;
}

// Unmatched rows join the pair of their strongest neighbour (pairs' representatives
// are never rewritten here, so reading rep[j] is race-free).
__global__ void k_join(int n, const int32_t* __restrict__ mate, const int32_t* __restrict__ best, int32_t* __restrict__ rep) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int j = best[i];
        if (mate[i] < 0 && j >= 0 && mate[j] >= 0) rep[i] = rep[j];
    }
}

__global__ void k_is_rep(int n, const int32_t* __restrict__ rep, int32_t* __restrict__ flag) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) flag[i] = rep[i] == i ? 1 : 0;
}

__global__ void k_agg_ids(int n, const int32_t* __restrict__ rep, const int32_t* __restrict__ id, int32_t* __restrict__ agg) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) agg[i] = id[rep[i]];
}

__global__ void k_fill_neg(int n, int32_t* __restrict__ a) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) a[i] = -1;
}

// Dense coarsest matrix (M zeroed before), then its inverse in place by Gauss-Jordan
// without pivoting (SPD up to floating islands).
__global__ void k_dense_coarse(int nc, int lanes, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci, const double* __restrict__ v,
                               const double* __restrict__ diag, double* __restrict__ M) {
    const RowLanes g = row_lanes(lanes);
    for (int i = g.first; i < nc; i += g.step) {
        for (int k = rp[i] + g.lane; k < rp[i + 1]; k += lanes) M[(size_t)i * nc + ci[k]] = v[k];
        if (g.lane == 0) M[(size_t)i * nc + i] = diag[i];
    }
}

// Blocked in-place Gauss-Jordan (32 pivots per block).  For pivot block b with the others o:
// four warps invert the Schur-complemented diagonal block D = S_bb two pivots at a time (dropping a
// variable whose pivot vanishes: its row and column of D^-1 are zero), then the CTA applies the
// block step S_bo <- D^-1 S_bo, S_ob <- -S_ob D^-1, S_oo <- S_oo - S_ob D^-1 S_bo, S_bb <- D^-1:
// the unblocked elimination's result with 4 barriers per block instead of 2 per pivot.
constexpr int kGjBlock = 32;
constexpr int kGjDS = kGjBlock + 1;  // row stride of a diagonal block in shared memory

constexpr int kGjThreads = 512;

// A 32 x 32 block inverted in place by the CTA's first four warps (kGjInvert threads): thread t holds
// column t % 32 of rows 8 (t / 32) .. + 7 in a; a smaller block is padded with the identity, which
// stays decoupled; a variable whose pivot is not above thr is dropped (its row and column of the
// inverse are zero).  The chain of pivots bounds it, so two are taken at a time: the warp that holds
// both rows inverts their 2 x 2 block (one division) and publishes the new rows, every thread in the
// two columns its old entries (two banks in turn: one barrier a pair), and all update.  A block of
// the grid Gauss-Jordan took 9.3 us with single pivots and 512 threads, 11 with one warp and shuffles.
constexpr int kGjInvert = 128;
struct GjBank {
    double row[2][kGjBlock];   // new pivot rows
    double2 col[kGjBlock];     // old pivot columns
};
__device__ __forceinline__ void gj_invert(double (&a)[8], GjBank (&bank)[2], double thr) {
    const int w = threadIdx.x >> 5, j = threadIdx.x & 31;
#pragma unroll 1
    for (int q = 0; q < 4; q++) {  // the warp that holds the pivots
#pragma unroll
        for (int h = 0; h < 4; h++) {
            const int k = 8 * q + 2 * h;
            GjBank& B = bank[h & 1];
            if (j == k)
#pragma unroll
                for (int e = 0; e < 8; e++) B.col[8 * w + e].x = a[e];
            if (j == k + 1)
#pragma unroll
                for (int e = 0; e < 8; e++) B.col[8 * w + e].y = a[e];
            if (w == q) {
                const double u = a[2 * h], v = a[2 * h + 1];
                const double p11 = __shfl_sync(0xffffffffu, u, k), p12 = __shfl_sync(0xffffffffu, u, k + 1);
                const double p21 = __shfl_sync(0xffffffffu, v, k), p22 = __shfl_sync(0xffffffffu, v, k + 1);
                const double det = p11 * p22 - p12 * p21;
                double i11 = 0, i12 = 0, i21 = 0, i22 = 0;
                if (p11 > thr && det > thr * p11) {  // det / p11: the second pivot after the first
                    const double inv = 1.0 / det;
                    i11 = p22 * inv;
                    i12 = -p12 * inv;
                    i21 = -p21 * inv;
                    i22 = p11 * inv;
                } else if (p11 > thr) {
                    i11 = 1.0 / p11;
                } else if (p22 > thr) {
                    i22 = 1.0 / p22;
                }
                B.row[0][j] = j == k ? i11 : j == k + 1 ? i12 : i11 * u + i12 * v;
                B.row[1][j] = j == k ? i21 : j == k + 1 ? i22 : i21 * u + i22 * v;
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");
            const double r0 = B.row[0][j], r1 = B.row[1][j];
            const bool own = j == k || j == k + 1;
#pragma unroll
            for (int e = 0; e < 8; e++) {
                const double2 c = B.col[8 * w + e];
                a[e] = (own ? 0.0 : a[e]) - c.x * r0 - c.y * r1;
            }
            if (w == q) {
                a[2 * h] = r0;
                a[2 * h + 1] = r1;
            }
        }
    }
}
static_assert(kGjInvert == 128 && kGjBlock == 32, "gj_invert: four warps of eight rows");

__global__ void __launch_bounds__(kGjThreads) k_gauss_jordan(int n, double* __restrict__ M) {
    extern __shared__ double S[];  // n * n, then Cb (n x 32), Rb (32 x n), D (32 x 33), f (32)
    __shared__ GjBank gj_bank[2];
    double* Cb = S + (size_t)n * n;
    double* Rb = Cb + (size_t)n * kGjBlock;
    double* D = Rb + (size_t)kGjBlock * n;
    __shared__ double dmax_s;
    const int t = threadIdx.x;
    for (int e = t; e < n * n; e += kGjThreads) S[e] = M[e];
    __syncthreads();
    if (t == 0) {
        double m = 0;
        for (int i = 0; i < n; i++) m = fmax(m, fabs(S[i * n + i]));
        dmax_s = m;
    }
    __syncthreads();
    const double thr = 1e-12 * dmax_s;
    for (int i = t; i < n; i += kGjThreads) S[i * n + i] *= (1.0 + 1e-8);
    __syncthreads();
    constexpr int DS = kGjDS;
    for (int b0 = 0; b0 < n; b0 += kGjBlock) {
        const int m = min(kGjBlock, n - b0);
        for (int e = t; e < kGjBlock * kGjBlock; e += kGjThreads) {
            const int r = e / kGjBlock, c = e % kGjBlock;
            D[r * DS + c] = (r < m && c < m) ? S[(b0 + r) * n + b0 + c] : (r == c ? 1.0 : 0.0);
        }
        for (int e = t; e < n * m; e += kGjThreads) Cb[(e / m) * kGjBlock + e % m] = S[(e / m) * n + b0 + e % m];
        __syncthreads();
        if (t < kGjInvert) {
            double a[8];
#pragma unroll
            for (int e = 0; e < 8; e++) a[e] = D[(8 * (t >> 5) + e) * kGjDS + (t & 31)];
            gj_invert(a, gj_bank, thr);
#pragma unroll
            for (int e = 0; e < 8; e++) D[(8 * (t >> 5) + e) * kGjDS + (t & 31)] = a[e];
        }
        __syncthreads();
        // Rb = D^-1 S_bo (columns outside the block)
        for (int e = t; e < m * n; e += kGjThreads) {
            const int ii = e / n, jc = e % n;
            if (jc >= b0 && jc < b0 + m) continue;
            double acc = 0;
            for (int kk = 0; kk < m; kk++) acc += D[ii * DS + kk] * S[(b0 + kk) * n + jc];
            Rb[ii * n + jc] = acc;
        }
        __syncthreads();
        for (int e = t; e < n * n; e += kGjThreads) {
            const int i = e / n, jc = e % n;
            const bool ib = i >= b0 && i < b0 + m, jb = jc >= b0 && jc < b0 + m;
            double v;
            if (ib) {
                v = jb ? D[(i - b0) * DS + (jc - b0)] : Rb[(i - b0) * n + jc];
            } else if (jb) {
                double acc = 0;
                for (int kk = 0; kk < m; kk++) acc += Cb[i * kGjBlock + kk] * D[kk * DS + (jc - b0)];
                v = -acc;
            } else {
                double acc = 0;
                for (int kk = 0; kk < m; kk++) acc += Cb[i * kGjBlock + kk] * Rb[kk * n + jc];
                v = S[e] - acc;
            }
            S[e] = v;
        }
        __syncthreads();
    }
    for (int e = t; e < n * n; e += kGjThreads) M[e] = S[e];
}

__global__ void k_ra_fill(int nc, int lanes, const int32_t* __restrict__ mptr, const int32_t* __restrict__ midx, const int32_t* __restrict__ rp,
                          const int32_t* __restrict__ ci, const double* __restrict__ v, const double* __restrict__ diag,
                          const int32_t* __restrict__ ra_ptr, int32_t* __restrict__ ra_col, double* __restrict__ ra_val) {
    const RowLanes g = row_lanes(lanes);
    for (int J = g.first; J < nc; J += g.step) {
        int e = ra_ptr[J];
        for (int m = mptr[J]; m < mptr[J + 1]; m++) {
            const int I = midx[m], b = rp[I], len = rp[I + 1] - b;
            if (g.lane == 0) {
                ra_col[e] = I;
                ra_val[e] = diag[I];
            }
            e++;
            for (int k = g.lane; k < len; k += lanes) {
                ra_col[e + k] = ci[b + k];
                ra_val[e + k] = v[b + k];
            }
            e += len;
        }
    }
}

// Fused restriction rows of level l >= 1 into level l + 1 (grid kernel): row J holds
// the members of aggregate J (column m < n: r_l[m], weight 1), then for each member I its
// diagonal and couplings (column n + c: z_l[c], weight -a), the rows of P^T A_l, so
// r_{l+1} = P^T (r_l - A_l z_l) is one gathered dot product.  rr_ptr = mptr + ra_ptr, both
// prefix sums (ra_ptr: the P^T A_l row lengths).
__global__ void k_rr_fill(int nc, int n, int lanes, const int32_t* __restrict__ mptr, const int32_t* __restrict__ midx,
                          const int32_t* __restrict__ rp, const int32_t* __restrict__ ci, const double* __restrict__ v,
                          const double* __restrict__ diag, const int32_t* __restrict__ ra_ptr, int32_t* __restrict__ rr_ptr,
                          int32_t* __restrict__ rr_col, double* __restrict__ rr_val) {
    const RowLanes g = row_lanes(lanes);
    for (int J = g.first; J < nc; J += g.step) {
        const int m0 = mptr[J], m1 = mptr[J + 1];
        int e = m0 + ra_ptr[J];
        if (g.lane == 0) {
            rr_ptr[J] = e;
            if (J == nc - 1) rr_ptr[nc] = mptr[nc] + ra_ptr[nc];
        }
        for (int m = g.lane; m < m1 - m0; m += lanes) {
            rr_col[e + m] = midx[m0 + m];
            rr_val[e + m] = 1.0;
        }
        e += m1 - m0;
        for (int m = m0; m < m1; m++) {
            const int I = midx[m], b = rp[I], len = rp[I + 1] - b;
            if (g.lane == 0) {
                rr_col[e] = n + I;
                rr_val[e] = -diag[I];
            }
            e++;
            for (int k = g.lane; k < len; k += lanes) {
                rr_col[e + k] = n + ci[b + k];
                rr_val[e + k] = -v[b + k];
            }
            e += len;
        }
    }
}

// Fused prolongation-smoother rows of level l (1 <= l < coarsest): row I holds its diagonal
// and off-diagonal couplings twice, on z_l (column c < n) and on the coarse correction
// (column n + aggregate of c), so w = r_l - A_l (z_l + P zc) is one gathered dot product.
__global__ void k_pq_fill(int n, int lanes, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci, const double* __restrict__ v,
                          const double* __restrict__ diag, const int32_t* __restrict__ agg, int32_t* __restrict__ pq_ptr,
                          int32_t* __restrict__ pq_col, double* __restrict__ pq_val) {
    const RowLanes g = row_lanes(lanes);
    for (int I = g.first; I < n; I += g.step) {
        const int b = rp[I], len = rp[I + 1] - b;
        int e = 2 * (b + I);
        if (g.lane == 0) {
            pq_ptr[I] = e;
            if (I == n - 1) pq_ptr[n] = 2 * (rp[n] + n);
            pq_col[e] = I;
            pq_val[e] = diag[I];
            pq_col[e + 1] = n + agg[I];
            pq_val[e + 1] = diag[I];
        }
        e += 2;
        for (int k = g.lane; k < len; k += lanes) {
            const int c = ci[b + k];
            pq_col[e + 2 * k] = c;
            pq_val[e + 2 * k] = v[b + k];
            pq_col[e + 2 * k + 1] = n + agg[c];
            pq_val[e + 2 * k + 1] = v[b + k];
        }
    }
}

// ---------------------------------------------------------------------------
// Solve kernel

constexpr int kGroup = 8;  // lanes cooperating on one coarse row

struct MgArgs {
    int n;
    const int32_t* rp;
    const int32_t* ci;
    const double* val;
    const double* b;
    double* x;
    const double* x0;  // when set, the solve starts from x0 (batched solves); else r = b - A x is given
    double *r, *z0, *z, *w, *p, *q;
    const double* tinv;
    const int32_t *row_off, *row_base, *row_m;
    const int32_t* cta_row;
    int levels;            // number of levels including level 0
    const MgLevel* lv;     // device descriptors
    const double* cinv;    // dense inverse of the coarsest level, or nullptr
    double omega0;
    double* partA;  // 4 x CTAs: r.r, p.q, then partB (r.z), r.r's second bank
    double* partB;
    double* stats;
    unsigned long long* bar;  // monotonic arrival counter (zeroed before the launch)
    long long spin_limit;     // polls of a barrier wait before it gives up
    int* err;
    double tol;
    long long max_iter;
    int max_restarts;
    int cap_b;  // stop at |r| <= tol min(|r0|, |b|) (batched solves); else |r| <= tol |r0| (Direct_Electrifying.cpp:1571, 1619)
};

// Grid barrier on a monotonic counter: one release-reduction per CTA (no return
// value to wait for; the release orders the CTA's writes, which __syncthreads
// gathered under thread 0, before the arrival), then an acquire spin until all
// CTAs of this round arrived.  Bounded: after `limit` polls the CTA records
// DEV_TIMEOUT and returns false.
__device__ __forceinline__ bool mg_sync(unsigned long long* bar, unsigned long long& target, int* err, int* s_ok, long long limit) {
    __syncthreads();
    if (threadIdx.x == 0) {
        target += gridDim.x;
        asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(bar) : "memory");
        long long spins = 0;
        int ok = 1;
        while (true) {
            unsigned long long v;
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(bar) : "memory");
            if (v >= target) break;
            if (++spins > limit || ((spins & 1023) == 0 && *((volatile int*)err) != 0)) {
                atomicCAS(err, 0, (int)DEV_TIMEOUT);
                ok = 0;
                break;
            }
        }
        *s_ok = ok;
    }
    __syncthreads();
    return *s_ok != 0;
}

// Dense inverse of a coarsest level too large for one CTA: blocked Gauss-Jordan (32 pivots
// per block, the drop rule and regularisation of k_gauss_jordan) over the whole grid, one
// cooperative launch with one grid barrier per block.  CTA (pr, pc) of a P x P grid keeps the tile
// [r0, r1) x [c0, c1) of the matrix in registers.  Block step b: every CTA reads the diagonal block
// D = S_bb, its rows' part of the column panel S[:, b] and its columns' part of the row panel
// S[b, :] (global, double-buffered; the tiles that hold the panels wrote them at the end of step
// b - 1), inverts D, forms X = D^-1 S_bj (columns of the block: D^-1) and updates its tile:
// S_ij = (j in the block ? 0 : S_ij) - S_ib X_bj outside the block's rows, X in them.
//
// A block step is bound by the pivot chain, its panel reads and the barrier.  Column strips, one
// per CTA, had every CTA read the whole column panel: 41 MB of L2 reads a block at 1,088 rows
// against 7 MB so: with the pivots two at a time (gj_invert) 883 -> 611 us in all, 753 rows 510 -> 327.
constexpr int kGjgThreads = 512;
constexpr int kMgDenseGridMax = 1280;  // largest dense coarsest
constexpr int kGjgTile = 112;          // largest tile edge: the CTA grid has at least n / 112 rows

// RT, CT: tile rows / 32 and columns / 16 (thread t holds rows t / 16 + 32 a, columns t % 16 + 16 b).
template <int RT, int CT>
__global__ void __launch_bounds__(kGjgThreads) k_gauss_jordan_grid(int n, int P, double* __restrict__ M, double* __restrict__ panel,
                                                                   unsigned long long* bar, unsigned long long* dmax_bits, int* err,
                                                                   long long limit) {
    constexpr int TR = 32 * RT, TC = 16 * CT;
    extern __shared__ double gsm[];  // column panel part (32 x TR), row panel part (32 x TC), X (32 x TC)
    double* const PI = gsm;
    double* const RB = PI + kGjBlock * TR;
    double* const X = RB + kGjBlock * TC;
    __shared__ double Dm[kGjBlock * kGjDS];
    __shared__ GjBank gj_bank[2];
    __shared__ int s_ok;
    const int t = threadIdx.x, ty = t >> 4, tx = t & 15;
    const int pr = blockIdx.x / P, pc = blockIdx.x % P;
    const int r0 = n * pr / P, nr = n * (pr + 1) / P - r0, c0 = n * pc / P, nc = n * (pc + 1) / P - c0;
    const size_t half = (size_t)n * kGjBlock;  // panel: column panels 0, 1 (kk * n + i), row panels 0, 1 (kk * n + j)
    double S[RT][CT];
    double dm = 0;
#pragma unroll
    for (int a = 0; a < RT; a++)
#pragma unroll
        for (int b = 0; b < CT; b++) {
            const int i = r0 + ty + 32 * a, j = c0 + tx + 16 * b;
            const bool in = ty + 32 * a < nr && tx + 16 * b < nc;
            double v = in ? M[(size_t)i * n + j] : 0.0;
            if (in && i == j) {
                dm = fmax(dm, fabs(v));
                v *= (1.0 + 1e-8);
            }
            S[a][b] = v;
        }
    if (dm > 0) atomicMax(dmax_bits, (unsigned long long)__double_as_longlong(dm));  // non-negative: the bits order as the values
    // the panels of block b0 from the tiles that hold them
    auto publish = [&](int b0, int bank) {
        const int m = min(kGjBlock, n - b0);
#pragma unroll
        for (int a = 0; a < RT; a++)
#pragma unroll
            for (int b = 0; b < CT; b++) {
                if (ty + 32 * a >= nr || tx + 16 * b >= nc) continue;
                const int i = r0 + ty + 32 * a, j = c0 + tx + 16 * b;
                if (j >= b0 && j < b0 + m) panel[bank * half + (size_t)(j - b0) * n + i] = S[a][b];
                if (i >= b0 && i < b0 + m) panel[(2 + bank) * half + (size_t)(i - b0) * n + j] = S[a][b];
            }
    };
    publish(0, 0);
    unsigned long long target = 0;
    if (!mg_sync(bar, target, err, &s_ok, limit)) return;
    const double thr = 1e-12 * __longlong_as_double((long long)__ldcg(dmax_bits));
    const int nblk = (n + kGjBlock - 1) / kGjBlock;
    for (int bk = 0; bk < nblk; bk++) {
        const int b0 = bk * kGjBlock, m = min(kGjBlock, n - b0);
        const double* cp = panel + (bk & 1) * half;
        const double* rp = panel + (2 + (bk & 1)) * half;
        // four warps invert the diagonal block while the others fetch the panels
        if (t < kGjInvert) {
            double a[8];
            const int w8 = 8 * (t >> 5), j = t & 31;
#pragma unroll
            for (int e = 0; e < 8; e++) a[e] = (w8 + e < m && j < m) ? __ldcg(&rp[(size_t)(w8 + e) * n + b0 + j]) : (w8 + e == j ? 1.0 : 0.0);
            gj_invert(a, gj_bank, thr);
#pragma unroll
            for (int e = 0; e < 8; e++) Dm[(w8 + e) * kGjDS + j] = a[e];
        } else {
            constexpr int T = kGjgThreads - kGjInvert;
            for (int e0 = t - kGjInvert; e0 < kGjBlock * (TR + TC); e0 += 4 * T) {
                double v[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int e = e0 + u * T, f = e - kGjBlock * TR;
                    v[u] = 0;
                    if (f < 0) {
                        if (e / TR < m && e % TR < nr) v[u] = __ldcg(&cp[(size_t)(e / TR) * n + r0 + e % TR]);
                    } else if (f < kGjBlock * TC) {
                        if (f / TC < m && f % TC < nc) v[u] = __ldcg(&rp[(size_t)(f / TC) * n + c0 + f % TC]);
                    }
                }
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (e0 + u * T < kGjBlock * (TR + TC)) PI[e0 + u * T] = v[u];  // (the row panel's part follows the column panel's)
            }
        }
        __syncthreads();
        {  // X: rows ty of the block (0 past it)
            double x[CT] = {};
#pragma unroll 8
            for (int kk = 0; kk < kGjBlock; kk++) {
                const double d = Dm[ty * kGjDS + kk];
#pragma unroll
                for (int b = 0; b < CT; b++) x[b] += d * RB[kk * TC + tx + 16 * b];
            }
#pragma unroll
            for (int b = 0; b < CT; b++) {
                const int jb = c0 + tx + 16 * b - b0;
                X[ty * TC + tx + 16 * b] = ty >= m ? 0.0 : jb >= 0 && jb < m ? Dm[ty * kGjDS + jb] : x[b];
            }
        }
#pragma unroll
        for (int b = 0; b < CT; b++) {
            const int jb = c0 + tx + 16 * b - b0;
            if (jb >= 0 && jb < m)
#pragma unroll
                for (int a = 0; a < RT; a++) S[a][b] = 0.0;
        }
        __syncthreads();
#pragma unroll 4
        for (int kk = 0; kk < kGjBlock; kk++) {
            double pv[RT], xv[CT];
#pragma unroll
            for (int a = 0; a < RT; a++) pv[a] = PI[kk * TR + ty + 32 * a];
#pragma unroll
            for (int b = 0; b < CT; b++) xv[b] = X[kk * TC + tx + 16 * b];
#pragma unroll
            for (int a = 0; a < RT; a++)
#pragma unroll
                for (int b = 0; b < CT; b++) S[a][b] -= pv[a] * xv[b];
        }
#pragma unroll
        for (int a = 0; a < RT; a++) {  // the block's own rows take X
            const int ib = r0 + ty + 32 * a - b0;
            if (ty + 32 * a < nr && ib >= 0 && ib < m)
#pragma unroll
                for (int b = 0; b < CT; b++) S[a][b] = X[ib * TC + tx + 16 * b];
        }
        if (bk + 1 < nblk) {
            publish(b0 + kGjBlock, (bk + 1) & 1);
            if (!mg_sync(bar, target, err, &s_ok, limit)) return;
        }
    }
#pragma unroll
    for (int a = 0; a < RT; a++)
#pragma unroll
        for (int b = 0; b < CT; b++)
            if (ty + 32 * a < nr && tx + 16 * b < nc) M[(size_t)(r0 + ty + 32 * a) * n + c0 + tx + 16 * b] = S[a][b];
}

// Cluster variant: the hardware cluster barrier (release/acquire at cluster
// scope orders the global-memory writes of all CTAs of the cluster).
template <bool CL>
__device__ __forceinline__ bool sync_all(unsigned long long* bar, unsigned long long& target, int* err, int* s_ok, long long limit) {
    if constexpr (CL) {
        asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
        return true;
    } else {
        return mg_sync(bar, target, err, s_ok, limit);
    }
}

__device__ __forceinline__ void mg_reduce1(double a, double* sm, double& ra) {
    a = warp_sum(a);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) sm[w] = a;
    __syncthreads();
    if (w == 0) {
        const int nw = blockDim.x >> 5;
        double x = lane < nw ? sm[lane] : 0.0;
        x = warp_sum(x);
        if (lane == 0) sm[64] = x;
    }
    __syncthreads();
    ra = sm[64];
    __syncthreads();
}

__device__ __forceinline__ double mg_sum_partials(const double* part, int nb, double* sm) {
    if (threadIdx.x < 32) {
        double a = 0;
        for (int i = threadIdx.x; i < nb; i += 32) a += __ldcg(&part[i]);
        a = warp_sum(a);
        if (threadIdx.x == 0) sm[66] = a;
    }
    __syncthreads();
    const double s = sm[66];
    __syncthreads();
    return s;
}

__device__ __forceinline__ double group_sum(double v, unsigned mask) {
    for (int o = kGroup / 2; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o, kGroup);
    return v;
}

// Gathered dot products of the solve phases.  The entries of a chunk (U per
// thread) have their column indices and values loaded first and their vector
// entries second, so a chunk costs two dependent L2 round trips instead of two
// per entry; the sum still runs in entry order.  Vectors other CTAs write are
// read with __ldcg (L2).
template <int U>
__device__ __forceinline__ double gather_dot(const int32_t* __restrict__ ci, const double* __restrict__ v, const double* x, int b, int e,
                                             int first = 0, int step = 1) {
    double s = 0;
    for (int k0 = b + first; k0 < e; k0 += U * step) {
        int c[U];
        double w[U], xv[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int k = k0 + u * step;
            c[u] = k < e ? ci[k] : 0;
            w[u] = k < e ? v[k] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; u++) xv[u] = (k0 + u * step < e) ? __ldcg(&x[c[u]]) : 0.0;
#pragma unroll
        for (int u = 0; u < U; u++) s += w[u] * xv[u];
    }
    return s;
}

// sum_k v[k] (x[ci[k]] + y[cg[k]])
template <int U>
__device__ __forceinline__ double gather_dot2(const int32_t* __restrict__ ci, const int32_t* __restrict__ cg, const double* __restrict__ v,
                                              const double* x, const double* y, int b, int e, int first = 0, int step = 1) {
    double s = 0;
    for (int k0 = b + first; k0 < e; k0 += U * step) {
        int c[U], g[U];
        double w[U], xv[U], yv[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int k = k0 + u * step;
            c[u] = k < e ? ci[k] : 0;
            g[u] = k < e ? cg[k] : 0;
            w[u] = k < e ? v[k] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const bool ok = k0 + u * step < e;
            xv[u] = ok ? __ldcg(&x[c[u]]) : 0.0;
            yv[u] = ok ? __ldcg(&y[g[u]]) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; u++) s += w[u] * (xv[u] + yv[u]);
    }
    return s;
}

// sum_m x[idx[m]]
template <int U>
__device__ __forceinline__ double gather_sum(const int32_t* __restrict__ idx, const double* x, int b, int e, int first, int step) {
    double s = 0;
    for (int k0 = b + first; k0 < e; k0 += U * step) {
        int c[U];
        double xv[U];
#pragma unroll
        for (int u = 0; u < U; u++) c[u] = (k0 + u * step < e) ? idx[k0 + u * step] : 0;
#pragma unroll
        for (int u = 0; u < U; u++) xv[u] = (k0 + u * step < e) ? __ldcg(&x[c[u]]) : 0.0;
#pragma unroll
        for (int u = 0; u < U; u++) s += xv[u];
    }
    return s;
}

__device__ __forceinline__ double block_apply(const MgArgs& a, const double* __restrict__ v, int i) {
    const int off = a.row_off[i], base = a.row_base[i], m = a.row_m[i];
    double s = 0;
    for (int j = 0; j < m; j++) s += a.tinv[off + j] * v[base + j];
    return s;
}

// Partials of r.r.  A residual replacement sums r.r twice with no barrier between the reads of the
// first sum's partials and the writes of the second's, so the two take different banks; a bank is
// written again only after the barriers of an iteration.
__device__ __forceinline__ double* residual_bank(const MgArgs& a, int restarts, int nctas) {
    return a.partA + (restarts & 1 ? 3 * nctas : 0);
}

// One MG-PCG solve by `nctas` CTAs (this is CTA `cta` of them).
template <bool CL>
__device__ void mg_pcg_body(const MgArgs& a, int cta, int nctas) {
    __shared__ double sm[72];
    __shared__ MgLevel lv[kMgMaxLevels];
    __shared__ double rc[kMgDenseMax];
    __shared__ int s_ok;
    if (threadIdx.x < a.levels) lv[threadIdx.x] = a.lv[threadIdx.x];
    __syncthreads();
    const int C = a.levels - 1;
    const int nb = nctas;
    const int gt = cta * blockDim.x + threadIdx.x, gs = nctas * blockDim.x;
    const int grp = gt / kGroup, glane = gt % kGroup, ngrp = gs / kGroup;
    const unsigned gmask = ((1u << kGroup) - 1) << ((threadIdx.x & 31) & ~(kGroup - 1));
    const int r_lo = a.cta_row[cta], r_hi = a.cta_row[cta + 1];
    if (a.x0) {  // start from x0: x = x0, r = b - A x0 (own rows; x0 is read-only, no barrier needed)
        for (int i = r_lo + threadIdx.x; i < r_hi; i += blockDim.x) {
            double s = 0;
            for (int kk = a.rp[i]; kk < a.rp[i + 1]; kk++) s += a.val[kk] * a.x0[a.ci[kk]];
            a.x[i] = a.x0[i];
            a.r[i] = a.b[i] - s;
        }
    }
    unsigned long long target = 0;
    double R0 = 0, rr = 0, rz = 0, beta = 0, bnorm = 0;
    if (a.cap_b) {  // |b| (partB is next written after the first barrier of the loop)
        double bb_l = 0;
        for (int i = r_lo + threadIdx.x; i < r_hi; i += blockDim.x) bb_l += a.b[i] * a.b[i];
        double s0;
        mg_reduce1(bb_l, sm, s0);
        if (threadIdx.x == 0) a.partB[cta] = s0;
        if (!sync_all<CL>(a.bar, target, a.err, &s_ok, a.spin_limit)) return;
        bnorm = sqrt(mg_sum_partials(a.partB, nb, sm));
    }
    long long k = 0;
    int restarts = 0;
    bool fresh = true;      // p = z, q = A z on the next direction update
    bool recursive = false; // r is the recursively updated residual (not b - A x)
    while (true) {
        // ---- pre-smoother z0 = w M0^-1 r on own rows; r.r ----
        __syncthreads();
        double rr_l = 0;
        for (int i = r_lo + threadIdx.x; i < r_hi; i += blockDim.x) {
            a.z0[i] = a.omega0 * block_apply(a, a.r, i);
            const double ri = a.r[i];
            rr_l += ri * ri;
        }
        double s0;
        mg_reduce1(rr_l, sm, s0);
        double* const part = residual_bank(a, restarts, nb);
        if (threadIdx.x == 0) part[cta] = s0;
        if (!sync_all<CL>(a.bar, target, a.err, &s_ok, a.spin_limit)) return;
        rr = mg_sum_partials(part, nb, sm);
        if (k == 0 && !recursive && restarts == 0) R0 = a.tol * (a.cap_b ? fmin(sqrt(rr), bnorm) : sqrt(rr));
        if (k > 0 && sqrt(rr) <= R0) {
            if (!recursive || restarts >= a.max_restarts) break;
            // the recursive residual met the test: replace it by the FP64 true residual
            for (int i = r_lo + threadIdx.x; i < r_hi; i += blockDim.x) {
                a.r[i] = a.b[i] - gather_dot<4>(a.ci, a.val, a.x, a.rp[i], a.rp[i + 1]);
            }
            restarts++;
            recursive = false;
            fresh = true;
            continue;
        }
        if (k >= a.max_iter) break;
        // ---- restriction 0 -> 1 inside the CTA (its blocks are its own rows) ----
        {
            const MgLevel& F = lv[0];
            const MgLevel& G = lv[1];
            for (int i = r_lo + threadIdx.x; i < r_hi; i += blockDim.x) {
                a.w[i] = a.r[i] - gather_dot<4>(a.ci, a.val, a.z0, a.rp[i], a.rp[i + 1]);
            }
            __syncthreads();
            const bool smooth = (C > 1) || a.cinv == nullptr;
            if (r_hi > r_lo) {
                const int b0 = F.agg[r_lo], b1 = F.agg[r_hi - 1];
                for (int J = b0 + threadIdx.x; J <= b1; J += blockDim.x) {
                    double s = 0;
                    for (int m = F.mptr[J]; m < F.mptr[J + 1]; m++) s += a.w[F.midx[m]];
                    G.r[J] = s;
                    if (smooth) G.z[J] = G.l1inv[J] * s;
                }
            }
            if (!sync_all<CL>(a.bar, target, a.err, &s_ok, a.spin_limit)) return;
        }
        // ---- restrictions l -> l+1 (l >= 1): r_{l+1} = P^T r_l - (P^T A_l) z_l ----
        for (int l = 1; l < C; l++) {
            const MgLevel& F = lv[l];
            const MgLevel& G = lv[l + 1];
            const bool smooth = (l + 1 < C) || a.cinv == nullptr;
            for (int J = grp; J < G.n; J += ngrp) {
                double s = gather_sum<2>(F.midx, F.r, F.mptr[J], F.mptr[J + 1], glane, kGroup) -
                           gather_dot<4>(F.ra_col, F.ra_val, F.z, F.ra_ptr[J], F.ra_ptr[J + 1], glane, kGroup);
                s = group_sum(s, gmask);
                if (glane == 0) {
                    G.r[J] = s;
                    if (smooth) G.z[J] = G.l1inv[J] * s;
                }
            }
            if (!sync_all<CL>(a.bar, target, a.err, &s_ok, a.spin_limit)) return;
        }
        // ---- coarsest: dense inverse, one warp per row ----
        if (a.cinv) {
            const MgLevel& Cl = lv[C];
            const int nC = Cl.n;
            const int wpb = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
            if (cta * wpb < nC) {
                for (int j = threadIdx.x; j < nC; j += blockDim.x) rc[j] = __ldcg(&Cl.r[j]);
                __syncthreads();
                for (int i = cta * wpb + warp; i < nC; i += nctas * wpb) {
                    const double* row = a.cinv + (size_t)i * nC;
                    double s = 0;
                    for (int j = lane; j < nC; j += 32) s += row[j] * rc[j];
                    s = warp_sum(s);
                    if (lane == 0) Cl.zf[i] = s;
                }
            }
            if (!sync_all<CL>(a.bar, target, a.err, &s_ok, a.spin_limit)) return;
        }
        // ---- prolongation + l1-Jacobi post-smoother, levels C-1 .. 1 ----
        for (int l = C - 1; l >= 1; l--) {
            const MgLevel& F = lv[l];
            const double* zc = lv[l + 1].zf;
            for (int I = grp; I < F.n; I += ngrp) {
                double w = -gather_dot2<4>(F.ci, F.cagg, F.val, F.z, zc, F.rp[I], F.rp[I + 1], glane, kGroup);
                w = group_sum(w, gmask);
                if (glane == 0) {
                    const double zp = __ldcg(&F.z[I]) + __ldcg(&zc[F.agg[I]]);
                    w += __ldcg(&F.r[I]) - F.diag[I] * zp;
                    F.zf[I] = zp + F.l1inv[I] * w;
                }
            }
            if (!sync_all<CL>(a.bar, target, a.err, &s_ok, a.spin_limit)) return;
        }
        // ---- level-0 post-smoother: z = z0 + P z1, z += w M0^-1 (r - A z); r.z ----
        {
            const double* zc = lv[1].zf;
            const int32_t* agg = lv[0].agg;
            const int32_t* cagg = lv[0].cagg;
            for (int i = r_lo + threadIdx.x; i < r_hi; i += blockDim.x) {
                a.w[i] = a.r[i] - gather_dot2<4>(a.ci, cagg, a.val, a.z0, zc, a.rp[i], a.rp[i + 1]);
                a.z[i] = a.z0[i] + __ldcg(&zc[agg[i]]);
            }
            __syncthreads();
            double rz_l = 0;
            for (int i = r_lo + threadIdx.x; i < r_hi; i += blockDim.x) {
                const double zi = a.z[i] + a.omega0 * block_apply(a, a.w, i);
                a.z[i] = zi;
                rz_l += a.r[i] * zi;
            }
            mg_reduce1(rz_l, sm, s0);
            if (threadIdx.x == 0) a.partB[cta] = s0;
            if (!sync_all<CL>(a.bar, target, a.err, &s_ok, a.spin_limit)) return;
            const double rz_new = mg_sum_partials(a.partB, nb, sm);
            beta = fresh ? 0.0 : rz_new / rz;
            rz = rz_new;
        }
        // ---- q = A z + beta q, p = z + beta p; p.q ----
        double pq_l = 0;
        for (int i = r_lo + threadIdx.x; i < r_hi; i += blockDim.x) {
            const double w = gather_dot<4>(a.ci, a.val, a.z, a.rp[i], a.rp[i + 1]);
            const double zi = a.z[i];
            const double qi = fresh ? w : w + beta * a.q[i];
            const double pi = fresh ? zi : zi + beta * a.p[i];
            a.q[i] = qi;
            a.p[i] = pi;
            pq_l += pi * qi;
        }
        mg_reduce1(pq_l, sm, s0);
        if (threadIdx.x == 0) a.partA[nb + cta] = s0;
        if (!sync_all<CL>(a.bar, target, a.err, &s_ok, a.spin_limit)) return;
        const double pq = mg_sum_partials(a.partA + nb, nb, sm);
        fresh = false;
        k++;
        // ---- x += alpha p, r -= alpha q ----
        const double alpha = rz / pq;
        for (int i = r_lo + threadIdx.x; i < r_hi; i += blockDim.x) {
            a.x[i] += alpha * a.p[i];
            a.r[i] -= alpha * a.q[i];
        }
        recursive = true;
    }
    if (cta == 0 && threadIdx.x == 0) {
        a.stats[0] = (double)k;
        a.stats[1] = rr;
        a.stats[2] = R0;
        a.stats[3] = (double)restarts;
    }
}

template <bool CL>
__global__ void __launch_bounds__(CL ? kMgClusterThreads : kMgThreads) k_mg_pcg(MgArgs a) {
    mg_pcg_body<CL>(a, blockIdx.x, gridDim.x);
}

// Batched solves: every cluster (of `ctas` CTAs) takes the next system of the queue and
// runs the MG-PCG on it; `slots` passes the index from cluster rank 0 to the others.
__global__ void __launch_bounds__(kMgClusterThreads) k_mg_batch(const MgArgs* __restrict__ all, int count, int ctas, int* queue, int* slots) {
    const int cl = blockIdx.x / ctas, rank = blockIdx.x % ctas;
    while (true) {
        if (rank == 0 && threadIdx.x == 0) slots[cl] = atomicAdd(queue, 1);
        asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
        const int s = __ldcg(&slots[cl]);
        asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
        if (s >= count) return;
        const MgArgs a = all[s];
        mg_pcg_body<true>(a, rank, ctas);
    }
}

// ---------------------------------------------------------------------------
// Shared-memory-resident grid kernel for systems above one cluster's size: one CTA per SM
// (cooperative launch).
//
// An iteration is a dozen phases between grid barriers, each a gathered sparse product of a few
// thousand entries a CTA, so it is bound by the latency of its dependent loads and barriers.  Every
// operator of the V-cycle is static during the solve: each CTA copies once, at launch, the rows it
// owns into shared memory (a set that does not fit the budget is read from global memory), and a
// phase costs one round trip for the vector entries other CTAs wrote, plus its barrier.
//
// Rows of the coarse levels are dealt by their entries, not their number, and a CTA spreads the
// entries over all its threads: products first, into shared memory, then the rows' sums.  With rows
// dealt by number and two to 32 lanes a row the CTA holding a level's longest rows kept the others
// waiting 2-10 us a phase.  The chain blocks are applied by their LDL^T factors, one thread a chain:
// two values a row instead of the chain's length (which large systems read from L2), and no inverses
// to set up (0.1-0.4 ms a network).
//
// An iteration of the 25k-CNT network's passes (64.7k, 28.4k rows) takes 44 and 40 us (57 and 47
// with rows dealt by number and dense blocks), of a 47.7k-CNT / 5 um realisation (313k, 246k rows)
// 86 and 90 us (160 and 123).  Measured and left: 1,024 threads (47, 43, 85, 88 us); one flag word a
// CTA polled by a thread each instead of the counter (90 us); values stored with their iteration's
// number and polled, without barriers (46, 41, 107, 98 us).
constexpr int kSmThreads = 512;
constexpr int kSmBytes = 200 * 1024;
constexpr int kSmProd = 4096;  // products of a phase held at once
constexpr int kSmAux = kSmThreads;  // rows of a phase held at once

struct MgSmLevel {
    int n;
    const int32_t* rr_ptr;  // fused restriction rows into level l + 1 (1 <= l < coarsest)
    const int32_t* rr_col;
    const double* rr_val;
    const int32_t* pq_ptr;  // fused prolongation-smoother rows of level l (1 <= l < coarsest)
    const int32_t* pq_col;
    const double* pq_val;
    const int32_t* agg;
    const double* l1inv;
    double* r;
    double* z;
    double* zf;
};

struct MgSmArgs {
    const MgSmLevel* lv;   // levels 0 .. coarsest
    const int32_t* mptr0;  // level-0 aggregates (the chain blocks): first row of each, then n
    const double* lfac;    // LDL^T factors of the chain blocks (0 at a block's first row, and one 0 past the last row)
    const double* ipiv;
    int smem_bytes;        // dynamic shared memory of the launch
};

// Rows [lo, hi) of one fused operator.  ptr[i - lo] - sub and ptr[i - lo + 1] - sub bound the
// entries of row i in col / val; agg and l1inv are indexed by i - lo.  lanes: threads per row sum.
struct SmRows {
    int lo, hi, sub, lanes;
    const int32_t* ptr;
    const int32_t* col;
    const double* val;
    const int32_t* agg;
    const double* l1inv;
};

// The CTA's level-0 rows [lo, hi): CSR (entries rp_sub-based), column aggregates, chain factors,
// aggregates alo .. ahi with their row ranges (mptr_sub-based), and the CG vectors of its rows.
struct SmL0 {
    int lo, hi, alo, ahi;
    int rp_sub, mptr_sub;
    const int32_t *rp, *ci, *cagg, *agg, *mptr;
    const double *val, *lf, *ip, *b, *l1;
    double *r, *x, *p, *q, *z, *z0, *w;
};

struct SmPlan {
    SmL0 l0;
    SmRows R[kMgMaxLevels];  // restriction rows into level l + 1 (index l)
    SmRows Q[kMgMaxLevels];  // prolongation rows of level l
    int clo, chi;            // coarsest rows of this CTA (dense inverse rows)
    const double* cinv;      // its rows, (i - clo) * nC based
    double *prod, *aux;
};

struct SmStage {  // one copy from global into shared memory
    void* dst;
    const void* src;
    int count, elem, rebase;  // elem 4: int32 (minus rebase), 8: double
};

// Sum of v over all threads of the grid, between grid barriers (mg_sync): every CTA publishes its
// partial before the barrier and adds up all of them, in the same order, after it.
__device__ __forceinline__ bool sm_sum(const MgArgs& a, double* part, unsigned long long& target, double v, double* sm, int* s_ok, double& total) {
    const int nb = gridDim.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = warp_sum(v);
    if (lane == 0) sm[warp] = v;
    __syncthreads();
    if (warp == 0) {
        v = warp_sum(lane < kSmThreads / 32 ? sm[lane] : 0.0);
        if (lane == 0) part[blockIdx.x] = v;
    }
    if (!mg_sync(a.bar, target, a.err, s_ok, a.spin_limit)) return false;
    v = warp_sum((int)threadIdx.x < nb ? __ldcg(&part[threadIdx.x]) : 0.0);
    if (lane == 0) sm[32 + warp] = v;
    __syncthreads();
    total = 0;
    for (int w = 0; w < (nb + 31) / 32; w++) total += sm[32 + w];
    return true;
}

// The CTA's part of one fused operator: out(row, sum, aux) for each of its rows, where sum is
// sum_k val[k] v(col[k]) with v(c) = v0[c] for c < n, else v1[c - n], and aux the row's two values
// of pre(row) (loaded with the entries).
template <bool kAux, class Pre, class Out>
__device__ __forceinline__ void sm_rows(const SmRows& R, double* prod, double* aux, int n, const double* v0, const double* v1, double* sm, Pre pre,
                                        Out out) {
    const int tid = threadIdx.x, nr = R.hi - R.lo;
    for (int i0 = 0; i0 < nr;) {
        const int e0 = R.ptr[i0] - R.sub;
        int i1 = min(nr, i0 + kSmAux);
        if (R.ptr[i1] - R.sub - e0 > kSmProd) {  // as many rows as fit, at least one
            int lo = i0 + 1, hi = i1;
            while (hi - lo > 1) {
                const int m = (lo + hi) >> 1;
                if (R.ptr[m] - R.sub - e0 <= kSmProd) lo = m; else hi = m;
            }
            i1 = lo;
        }
        const int E = R.ptr[i1] - R.sub - e0;
        double2 t = make_double2(0, 0);
        if (kAux && i0 + tid < i1) t = pre(i0 + tid);
        double long_sum = 0;  // a row of more than kSmProd entries: one thread's share of it
        for (int k0 = tid; k0 < E; k0 += 4 * kSmThreads) {
            int c[4];
            double w[4], x[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int k = k0 + u * kSmThreads;
                c[u] = k < E ? R.col[e0 + k] : 0;
                w[u] = k < E ? R.val[e0 + k] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < 4; u++) x[u] = k0 + u * kSmThreads < E ? (c[u] < n ? __ldcg(&v0[c[u]]) : __ldcg(&v1[c[u] - n])) : 0.0;
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int k = k0 + u * kSmThreads;
                if (E > kSmProd) long_sum += w[u] * x[u];
                else if (k < E) prod[k] = w[u] * x[u];
            }
        }
        if (kAux && i0 + tid < i1) {
            aux[2 * tid] = t.x;
            aux[2 * tid + 1] = t.y;
        }
        if (E > kSmProd) {
            long_sum = warp_sum(long_sum);
            if ((tid & 31) == 0) sm[tid >> 5] = long_sum;
        }
        __syncthreads();
        if (E > kSmProd) {
            if (tid == 0) {
                double s = 0;
                for (int w = 0; w < kSmThreads / 32; w++) s += sm[w];
                out(i0, s, kAux ? aux[0] : 0.0, kAux ? aux[1] : 0.0);
            }
        } else {
            const int lanes = R.lanes, gl = tid % lanes;
            for (int i = i0 + tid / lanes; i < i1; i += kSmThreads / lanes) {
                const int e = R.ptr[i + 1] - R.sub - e0;
                double s = 0;
                for (int k = R.ptr[i] - R.sub - e0 + gl; k < e; k += lanes) s += prod[k];
                const unsigned mask = lanes >= 32 ? 0xffffffffu : (((1u << lanes) - 1) << ((tid & 31) & ~(lanes - 1)));
                for (int o = lanes / 2; o > 0; o >>= 1) s += __shfl_xor_sync(mask, s, o, lanes);
                if (gl == 0) out(i, s, kAux ? aux[2 * (i - i0)] : 0.0, kAux ? aux[2 * (i - i0) + 1] : 0.0);
            }
        }
        i0 = i1;
        if (i0 < nr) __syncthreads();
    }
}

// One chain: w = (L D L^T)^-1 r over its rows [m0, m1) (r may be w).  lf is 0 at a chain's first
// row, and lf[m1] (the next chain's first row) is readable.
template <class Out>
__device__ __forceinline__ void chain_solve(const double* r, const double* lf, const double* ip, double* w, int m0, int m1, Out out) {
    double y = 0;
    for (int k0 = m0; k0 < m1; k0 += 4) {
        double rv[4], lv[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int k = min(k0 + u, m1 - 1);
            rv[u] = r[k];
            lv[u] = lf[k];
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (k0 + u < m1) {
                y = rv[u] - lv[u] * y;
                w[k0 + u] = y;
            }
    }
    y = 0;
    for (int k0 = m1 - 1; k0 >= m0; k0 -= 4) {
        double yv[4], lv[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int k = max(k0 - u, m0);
            yv[u] = w[k] * ip[k];
            lv[u] = lf[k + 1];
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (k0 - u >= m0) {
                y = yv[u] - lv[u] * y;
                out(k0 - u, y);
            }
    }
}

// Copies of one CTA: seven of level 0's rows, nine of each level between it and the coarsest (four of
// its restriction rows, five of its prolongation rows), five of level 0's matrix, x and the dense inverse.
constexpr int kSmMaxStages = 7 + 9 * (kMgMaxLevels - 2) + 5;

__global__ void __launch_bounds__(kSmThreads, 1) k_mg_pcg_sm(MgArgs a, MgSmArgs sa) {
    extern __shared__ __align__(16) unsigned char sm_dyn[];
    __shared__ double sm[64];
    __shared__ MgSmLevel lv[kMgMaxLevels];
    __shared__ SmPlan P;
    __shared__ SmStage st[kSmMaxStages];
    __shared__ int n_st, s_ok;
    __shared__ int cut[kMgMaxLevels][4];
    __shared__ double rc[kMgDenseGridMax];
    const int cta = blockIdx.x, nb = gridDim.x, tid = threadIdx.x;
    const int C = a.levels - 1;
    if (tid < a.levels) lv[tid] = sa.lv[tid];
    __syncthreads();
    // ---- this CTA's rows of every level: an equal share of entries + 4 rows ----
    if (tid < 4 * C && tid >= 4) {
        const int l = tid >> 2, n = (tid & 2) ? lv[l].n : lv[l + 1].n, c = cta + (tid & 1);
        const int32_t* ptr = (tid & 2) ? lv[l].pq_ptr : lv[l].rr_ptr;
        const long long want = (ptr[n] + 4LL * n) * c / nb;
        int lo = 0, hi = n;  // first row whose share starts at or after `want`
        while (lo < hi) {
            const int m = (lo + hi) >> 1;
            if (ptr[m] + 4LL * m < want) lo = m + 1; else hi = m;
        }
        cut[l][tid & 3] = c == nb ? n : lo;
    }
    __syncthreads();
    // ---- placement (thread 0), then the copies (all threads) ----
    if (tid == 0) {
        const unsigned int cap = (unsigned int)sa.smem_bytes;
        unsigned int used = 0;
        int ns = 0;
        auto take = [&](size_t bytes) -> unsigned char* {
            const unsigned int u = (used + 15u) & ~15u;
            if (u + bytes > cap) return nullptr;
            used = u + (unsigned int)bytes;
            return sm_dyn + u;
        };
        // room for a copy of `count` entries of `elem` bytes and its record, or null
        auto copy = [&](const void* src, int count, int elem, int rebase) -> unsigned char* {
            unsigned char* m = count > 0 && ns < kSmMaxStages ? take((size_t)elem * count) : nullptr;
            if (m) st[ns++] = SmStage{m, src, count, elem, rebase};
            return m;
        };
        // dst: the staged copy, or `src` itself when it does not fit
        auto stage_i = [&](const int32_t*& dst, const int32_t* src, int count, int rebase) {
            unsigned char* m = copy(src, count, 4, rebase);
            dst = m ? reinterpret_cast<const int32_t*>(m) : src;
            return m != nullptr;
        };
        auto stage_d = [&](const double*& dst, const double* src, int count) {
            unsigned char* m = copy(src, count, 8, 0);
            dst = m ? reinterpret_cast<const double*>(m) : src;
        };
        auto stage_v = [&](double* src, int count) {
            unsigned char* m = copy(src, count, 8, 0);
            return m ? reinterpret_cast<double*>(m) : src;
        };
        auto vec = [&](double* src, int count) {
            unsigned char* m = count > 0 ? take(8 * (size_t)count) : nullptr;
            return m ? reinterpret_cast<double*>(m) : src;
        };
        SmL0& L = P.l0;
        const MgLevel& G0 = a.lv[0];
        L.lo = a.cta_row[cta];
        L.hi = a.cta_row[cta + 1];
        const int nr = L.hi - L.lo;
        P.prod = reinterpret_cast<double*>(take(8 * kSmProd));
        P.aux = reinterpret_cast<double*>(take(16 * kSmAux));
        // what every phase of level 0 reads: residual, smoothed vectors, chain factors and ranges
        L.r = stage_v(a.r + L.lo, nr);
        L.z0 = vec(a.z0 + L.lo, nr);
        L.w = vec(a.w + L.lo, nr);
        L.z = vec(a.z + L.lo, nr);
        stage_d(L.lf, sa.lfac + L.lo, nr > 0 ? nr + 1 : 0);
        stage_d(L.ip, sa.ipiv + L.lo, nr);
        L.alo = nr > 0 ? G0.agg[L.lo] : 0;
        L.ahi = nr > 0 ? G0.agg[L.hi - 1] + 1 : 0;
        stage_i(L.agg, G0.agg + L.lo, nr, 0);
        L.mptr_sub = stage_i(L.mptr, sa.mptr0 + L.alo, nr > 0 ? L.ahi - L.alo + 1 : 0, L.lo) ? 0 : L.lo;
        stage_d(L.l1, lv[1].l1inv + L.alo, L.ahi - L.alo);
        const int ent0 = nr > 0 ? a.rp[L.lo] : 0, ent = nr > 0 ? a.rp[L.hi] - ent0 : 0;
        L.rp_sub = stage_i(L.rp, a.rp + L.lo, nr > 0 ? nr + 1 : 0, ent0) ? 0 : ent0;
        // coarse operators, the coarsest (most often waited for) first: row data, then entries
        for (int l = C - 1; l >= 1; l--) {
            for (int q = 0; q < 2; q++) {
                SmRows& R = q ? P.Q[l] : P.R[l];
                const MgSmLevel& F = lv[l];
                const int32_t* ptr = q ? F.pq_ptr : F.rr_ptr;
                R.lo = cut[l][2 * q];
                R.hi = cut[l][2 * q + 1];
                const int rows = R.hi - R.lo, e0 = ptr[R.lo], E = ptr[R.hi] - e0;
                R.sub = stage_i(R.ptr, ptr + R.lo, rows > 0 ? rows + 1 : 0, e0) ? 0 : e0;
                stage_d(R.l1inv, (q ? F.l1inv : lv[l + 1].l1inv) + R.lo, rows);
                if (q) stage_i(R.agg, F.agg + R.lo, rows, 0);
                stage_i(R.col, (q ? F.pq_col : F.rr_col) + e0, E, 0);
                stage_d(R.val, (q ? F.pq_val : F.rr_val) + e0, E);
                R.lanes = 32;
                while (R.lanes > 2 && (R.lanes * rows > kSmThreads || R.lanes * rows > E)) R.lanes >>= 1;
            }
        }
        // level-0 matrix, the vectors only their own rows use, dense inverse rows
        stage_i(L.ci, a.ci + ent0, ent, 0);
        stage_d(L.val, a.val + ent0, ent);
        stage_i(L.cagg, G0.cagg + ent0, ent, 0);
        L.q = vec(a.q + L.lo, nr);
        L.p = vec(a.p + L.lo, nr);
        L.x = stage_v(a.x + L.lo, nr);
        L.b = a.b + L.lo;
        const int nC = lv[C].n;
        P.clo = (int)((long long)nC * cta / nb);
        P.chi = (int)((long long)nC * (cta + 1) / nb);
        P.cinv = nullptr;
        if (a.cinv) stage_d(P.cinv, a.cinv + (size_t)P.clo * nC, (P.chi - P.clo) * nC);
        n_st = ns;
    }
    __syncthreads();
    for (int q = 0; q < n_st; q++) {
        const SmStage S = st[q];
        if (S.elem == 8) {
            double* d = static_cast<double*>(S.dst);
            const double* g = static_cast<const double*>(S.src);
            for (int i = tid; i < S.count; i += kSmThreads) d[i] = g[i];
        } else {
            int32_t* d = static_cast<int32_t*>(S.dst);
            const int32_t* g = static_cast<const int32_t*>(S.src);
            for (int i = tid; i < S.count; i += kSmThreads) d[i] = g[i] - S.rebase;
        }
    }
    __syncthreads();
    const SmL0& L = P.l0;
    const int lo = L.lo, hi = L.hi, nr = hi - lo;
    // out(row, sum) of own rows: sum_q val[q] v(ci[q]), v(c) = vs[c - lo] for the CTA's own rows (shared
    // memory), else the global vector vg; with zc, each entry also adds zc[cagg[q]].  Four entries at
    // a time: indices and weights first, vector entries second.
    auto own_rows = [&](const double* vs, const double* vg, const double* zc, auto out) {
        for (int li = tid; li < nr; li += kSmThreads) {
            const int e = L.rp[li + 1] - L.rp_sub;
            double s = 0;
            for (int q0 = L.rp[li] - L.rp_sub; q0 < e; q0 += 4) {
                int c[4], g[4];
                double w[4], x[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int q = q0 + u;
                    c[u] = q < e ? L.ci[q] : lo;
                    w[u] = q < e ? L.val[q] : 0.0;
                    g[u] = zc && q < e ? L.cagg[q] : -1;
                }
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    x[u] = (c[u] >= lo && c[u] < hi) ? vs[c[u] - lo] : __ldcg(&vg[c[u]]);
                    if (g[u] >= 0) x[u] += __ldcg(&zc[g[u]]);
                }
#pragma unroll
                for (int u = 0; u < 4; u++) s += w[u] * x[u];
            }
            out(li, s);
        }
    };
    auto chains = [&](const double* r, double* w, auto out) {  // one thread a chain
        for (int j = tid; j < L.ahi - L.alo; j += kSmThreads)
            chain_solve(r, L.lf, L.ip, w, L.mptr[j] - L.mptr_sub, L.mptr[j + 1] - L.mptr_sub, out);
    };
    unsigned long long target = 0;
    double R0 = 0, rr = 0, rz = 0, beta = 0;
    long long k = 0;
    int restarts = 0;
    bool fresh = true;
    bool recursive = false;
    while (true) {
        // ---- pre-smoother z0 = w M0^-1 r on own rows; r.r ----
        __syncthreads();
        chains(L.r, L.w, [&](int li, double z) { L.z0[li] = a.omega0 * z; });
        __syncthreads();
        double rr_l = 0;
        for (int li = tid; li < nr; li += kSmThreads) {
            a.z0[lo + li] = L.z0[li];
            const double ri = L.r[li];
            rr_l += ri * ri;
        }
        if (!sm_sum(a, residual_bank(a, restarts, nb), target, rr_l, sm, &s_ok, rr)) return;
        if (k == 0 && !recursive && restarts == 0) R0 = a.tol * sqrt(rr);
        if (k > 0 && sqrt(rr) <= R0) {
            if (!recursive || restarts >= a.max_restarts) break;
            // the recursive residual met the test: replace it by the FP64 true residual
            own_rows(L.x, a.x, nullptr, [&](int li, double s) { L.r[li] = L.b[li] - s; });
            restarts++;
            recursive = false;
            fresh = true;
            continue;
        }
        if (k >= a.max_iter) break;
        // ---- w = r - A z0; level 0 -> 1 over the own aggregates (the chain blocks) ----
        own_rows(L.z0, a.z0, nullptr, [&](int li, double s) { L.w[li] = L.r[li] - s; });
        __syncthreads();
        {
            const MgSmLevel& G = lv[1];
            const bool smooth = (C > 1) || a.cinv == nullptr;
            for (int j = tid; j < L.ahi - L.alo; j += kSmThreads) {
                const int m1 = L.mptr[j + 1] - L.mptr_sub;
                double v = 0;
                for (int m = L.mptr[j] - L.mptr_sub; m < m1; m++) v += L.w[m];
                G.r[L.alo + j] = v;
                if (smooth) G.z[L.alo + j] = L.l1[j] * v;
            }
        }
        if (!mg_sync(a.bar, target, a.err, &s_ok, a.spin_limit)) return;
        // ---- r_{l+1} = P^T (r_l - A_l z_l) and its l1-Jacobi smoothing ----
        for (int l = 1; l < C; l++) {
            const SmRows& R = P.R[l];
            const MgSmLevel& G = lv[l + 1];
            const bool smooth = (l + 1 < C) || a.cinv == nullptr;
            sm_rows<false>(R, P.prod, P.aux, lv[l].n, lv[l].r, lv[l].z, sm, [](int) { return make_double2(0, 0); },
                    [&](int j, double v, double, double) {
                        G.r[R.lo + j] = v;
                        if (smooth) G.z[R.lo + j] = R.l1inv[j] * v;
                    });
            if (!mg_sync(a.bar, target, a.err, &s_ok, a.spin_limit)) return;
        }
        // ---- dense inverse of the coarsest level (r_C staged once), one warp per row; without one its correction is z ----
        if (a.cinv) {
            const MgSmLevel& Cl = lv[C];
            const int nC = Cl.n, warp = tid >> 5, lane = tid & 31;
            for (int j = tid; j < nC; j += kSmThreads) rc[j] = __ldcg(&Cl.r[j]);
            __syncthreads();
            for (int i = P.clo + warp; i < P.chi; i += kSmThreads / 32) {
                const double* row = P.cinv + (size_t)(i - P.clo) * nC;
                double v = 0;
                for (int j = lane; j < nC; j += 32) v += row[j] * rc[j];
                v = warp_sum(v);
                if (lane == 0) Cl.zf[i] = v;
            }
            if (!mg_sync(a.bar, target, a.err, &s_ok, a.spin_limit)) return;
        }
        // ---- zp = z_l + P zc, zf_l = zp + D^-1 (r_l - A_l zp) ----
        for (int l = C - 1; l >= 1; l--) {
            const SmRows& Q = P.Q[l];
            const MgSmLevel& F = lv[l];
            const double* zc = lv[l + 1].zf;
            sm_rows<true>(Q, P.prod, P.aux, F.n, F.z, zc, sm,
                    [&](int i) { return make_double2(__ldcg(&F.z[Q.lo + i]) + __ldcg(&zc[Q.agg[i]]), __ldcg(&F.r[Q.lo + i])); },
                    [&](int i, double v, double zp, double r) { F.zf[Q.lo + i] = zp + Q.l1inv[i] * (r - v); });
            if (!mg_sync(a.bar, target, a.err, &s_ok, a.spin_limit)) return;
        }
        // ---- level-0 post-smoother: z = z0 + P z1, z += w M0^-1 (r - A z); r.z ----
        {
            const double* zc = lv[1].zf;
            for (int li = tid; li < nr; li += kSmThreads) L.z[li] = L.z0[li] + __ldcg(&zc[L.agg[li]]);
            own_rows(L.z0, a.z0, zc, [&](int li, double s) { L.w[li] = L.r[li] - s; });
            __syncthreads();
            chains(L.w, L.w, [&](int li, double z) { L.z[li] += a.omega0 * z; });
            __syncthreads();
            double rz_l = 0, rz_new;
            for (int li = tid; li < nr; li += kSmThreads) {
                const double zi = L.z[li];
                a.z[lo + li] = zi;
                rz_l += L.r[li] * zi;
            }
            if (!sm_sum(a, a.partB, target, rz_l, sm, &s_ok, rz_new)) return;
            beta = fresh ? 0.0 : rz_new / rz;
            rz = rz_new;
        }
        // ---- q = A z + beta q, p = z + beta p; p.q ----
        double pq_l = 0, pq;
        own_rows(L.z, a.z, nullptr, [&](int li, double w) {
            const double zi = L.z[li];
            const double qi = fresh ? w : w + beta * L.q[li];
            const double pi = fresh ? zi : zi + beta * L.p[li];
            L.q[li] = qi;
            L.p[li] = pi;
            pq_l += pi * qi;
        });
        if (!sm_sum(a, a.partA + nb, target, pq_l, sm, &s_ok, pq)) return;
        fresh = false;
        k++;
        // ---- x += alpha p, r -= alpha q (x also to global: other CTAs read it for a true residual) ----
        const double alpha = rz / pq;
        for (int li = tid; li < nr; li += kSmThreads) {
            const double xi = L.x[li] + alpha * L.p[li];
            L.x[li] = xi;
            a.x[lo + li] = xi;
            L.r[li] -= alpha * L.q[li];
        }
        recursive = true;
    }
    if (cta == 0 && tid == 0) {
        a.stats[0] = (double)k;
        a.stats[1] = rr;
        a.stats[2] = R0;
        a.stats[3] = (double)restarts;
    }
}

// Members of level-0 aggregates (chain blocks: consecutive rows).
__global__ void k_members_contig(int n, int nc, const int32_t* __restrict__ agg, int32_t* __restrict__ mptr, int32_t* __restrict__ midx) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (i == 0 || agg[i] != agg[i - 1]) mptr[agg[i]] = i;
        midx[i] = i;
        if (i == n - 1) mptr[nc] = n;
    }
}

__global__ void k_member_count(int n, const int32_t* __restrict__ agg, int32_t* __restrict__ cnt) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) atomicAdd(&cnt[agg[i]], 1);
}

__global__ void k_member_place(int n, const int32_t* __restrict__ agg, const int32_t* __restrict__ mptr, int32_t* __restrict__ cursor,
                               int32_t* __restrict__ midx) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int J = agg[i];
        midx[mptr[J] + atomicAdd(&cursor[J], 1)] = i;
    }
}

// Members of every aggregate in ascending row order (insertion sort; aggregates are small).
__global__ void k_member_sort(int nc, const int32_t* __restrict__ mptr, int32_t* __restrict__ midx) {
    for (int J = blockIdx.x * blockDim.x + threadIdx.x; J < nc; J += gridDim.x * blockDim.x) {
        const int b = mptr[J], e = mptr[J + 1];
        for (int i = b + 1; i < e; i++) {
            const int v = midx[i];
            int j = i - 1;
            while (j >= b && midx[j] > v) {
                midx[j + 1] = midx[j];
                j--;
            }
            midx[j + 1] = v;
        }
    }
}

// Length of each aggregate's restriction row P^T A_l (members' rows with their diagonals).
__global__ void k_ra_lengths(int nc, const int32_t* __restrict__ mptr, const int32_t* __restrict__ midx, const int32_t* __restrict__ rp,
                             int32_t* __restrict__ ra_len) {
    for (int J = blockIdx.x * blockDim.x + threadIdx.x; J < nc; J += gridDim.x * blockDim.x) {
        int s = mptr[J + 1] - mptr[J];
        for (int m = mptr[J]; m < mptr[J + 1]; m++) {
            const int I = midx[m];
            s += rp[I + 1] - rp[I];
        }
        ra_len[J] = s;
    }
}

// Aggregate of every entry's column.
__global__ void k_cagg(const int32_t* __restrict__ nnz, const int32_t* __restrict__ ci, const int32_t* __restrict__ agg,
                       int32_t* __restrict__ cagg) {
    const int n = *nnz;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) cagg[k] = agg[ci[k]];
}

// ---------------------------------------------------------------------------
// Smoothed level-1 prolongator (hierarchies of the grid kernel).
//
// Why: with piecewise-constant aggregates below the chain level the V-cycle is weak on
// a sparse chain graph (smoothing_pays), whose junction conductances span five orders of magnitude.  Smoothing
// the first pairwise prolongator once, Q = (I - w D^-1 A_1) P with D the l1-Jacobi
// diagonal and w = 4/3, takes a real-resistor pass of the 25k-CNT network from ~90 to
// ~35 PCG iterations and its unit pass from 54 to 39.  Then A_2 = Q^T A_1 Q, the
// restriction rows are Q^T on r_1 and -Q^T A_1 on z_1, and the prolongation-smoother rows
// are A_1 on z_1 and A_1 (Q + w P) on zc, so that the solve kernel's unchanged
//   zf = z + zc[agg] + D^-1 (r - A_1 z - A_1 (Q + w P) zc)
// equals z + Q zc + D^-1 (r - A_1 (z + Q zc)), since Q zc = zc[agg] - w D^-1 T zc with
// T = A_1 P.  Every product is a row gather: output row J sums w * (row s of B) over its
// sources (s, w); the terms are sorted by column (keys (column, gather position) are
// unique) and summed in gather order, so no result depends on thread timing.
constexpr double kSaOmega = 4.0 / 3.0;

// Row gather: output row J is the sum of w * (row s of B) over its sources (s, w), used for the
// Galerkin coarse rows (sources: an aggregate's members, columns mapped to aggregates) and for
// the products of the smoothed prolongator.  The candidate terms of a row are numbered in
// source, then entry order; their keys (column, number) are unique, so sorting them and adding
// each column's run in that order gives sums that do not depend on thread timing.
//
// What bounds it: the chains of dependent loads (source -> its row -> its entries) and, for rows
// of more than a few hundred terms, the sort.  Sources are therefore read one per thread with a
// scan of their lengths, and the terms are spread over all threads (three dependent loads per
// batch of sources, not per source); rows are dealt by length to a warp (up to kGrWarpCap
// terms), a small CTA (kGrMidCap), a large CTA (kGrBigCap, all in shared memory) or a large CTA
// sorting in global memory.  Each column's first term adds its run, so runs are summed in
// parallel.  Dense networks have mostly rows of 500-6,000 terms: on a 47.7k-CNT / 5 um
// realisation the gathers of both hierarchies took 464 ms with one thread per row above 512
// terms and serial run sums, 4.8 ms so; on 9,117 CNTs in 3.37 um 18.4 ms and 0.6 ms.
constexpr int kGrWarps = 4;
constexpr int kGrWarpCap = 512;
constexpr int kGrMidThreads = 256, kGrMidCap = 2048;
constexpr int kGrBigThreads = 1024, kGrBigCap = 8192;
constexpr int kGrTiers = 3;  // lists of the rows above kGrWarpCap: mid, big, global
constexpr uint64_t kGrNone = ~0ull;

struct RowSrc {  // sources of output row J: (J, 1) when ptr is null, else (J, diag[J]) (with diag) and row J of the CSR (val null: weight 1)
    const int32_t* ptr;
    const int32_t* idx;
    const double* val;
    const double* diag;
};
struct RowMat {  // row s of B: (s, diag[s]) (with diag), then its CSR entries; val2 / diag2: a second value set
    const int32_t* ptr;
    const int32_t* col;
    const double* val;
    const double* diag;
    const double* val2;
    const double* diag2;
    const int32_t* cmap;  // column map (null: identity)
};
struct GatherOut {
    const int32_t* seg;                 // per output row: offset of its segment (candidate terms), nrows + 1
    uint64_t* gkey;                     // terms of the rows sorted in global memory (segment layout)
    double* gv;
    double* gv2;
    int32_t* ocol;                      // summed runs (segment layout)
    double* ov;
    double* ov2;
    int32_t* ulen;                      // runs per row
    const int32_t* list;                // kGrTiers lists of nrows
    const int32_t* nlist;               // their lengths
    int skip_diag;                      // drop column J of row J
    const double* rsv;                  // with rs_out: row sum of row J = sum_t w_t rsv[s_t]
    double* rs_out;
    double* diag_out;
    double* l1_out;
};

__device__ __forceinline__ int src_count(const RowSrc& S, int J) { return S.ptr ? (S.ptr[J + 1] - S.ptr[J]) + (S.diag ? 1 : 0) : 1; }

__device__ __forceinline__ void src_get(const RowSrc& S, int J, int t, int& s, double& w) {
    if (!S.ptr) {
        s = J;
        w = 1.0;
        return;
    }
    if (S.diag) {
        if (t == 0) {
            s = J;
            w = S.diag[J];
            return;
        }
        t--;
    }
    const int k = S.ptr[J] + t;
    s = S.idx[k];
    w = S.val ? S.val[k] : 1.0;
}

__device__ __forceinline__ int mat_len(const RowMat& B, int s) { return (B.ptr[s + 1] - B.ptr[s]) + (B.diag ? 1 : 0); }

__device__ __forceinline__ void mat_get(const RowMat& B, int s, int t, int& c, double& v, double& v2) {
    if (B.diag && t == 0) {
        c = s;
        v = B.diag[s];
        v2 = B.diag2 ? B.diag2[s] : 0.0;
    } else {
        const int k = B.ptr[s] + t - (B.diag ? 1 : 0);
        c = B.col[k];
        v = B.val[k];
        v2 = B.val2 ? B.val2[k] : 0.0;
    }
    if (B.cmap) c = B.cmap[c];
}

// Candidate terms per row, and the rows too long for a warp listed by length (nlist zeroed before).
__global__ void k_gather_len(int nrows, int lanes, RowSrc S, RowMat B, int32_t* __restrict__ seg, int32_t* __restrict__ list, int32_t* nlist) {
    const RowLanes g = row_lanes(lanes);
    const unsigned mask = lanes >= 32 ? 0xffffffffu : (((1u << lanes) - 1) << ((threadIdx.x & 31) & ~(lanes - 1)));
    for (int J = g.first; J < nrows; J += g.step) {
        int c = 0;
        const int ns = src_count(S, J);
        for (int t = g.lane; t < ns; t += lanes) {
            int s;
            double w;
            src_get(S, J, t, s, w);
            c += mat_len(B, s);
        }
        for (int o = lanes / 2; o > 0; o >>= 1) c += __shfl_xor_sync(mask, c, o, lanes);
        if (g.lane != 0) continue;
        seg[J] = c;
        if (J == 0) seg[nrows] = 0;
        if (c > kGrWarpCap) {
            const int tier = c <= kGrMidCap ? 0 : c <= kGrBigCap ? 1 : 2;
            list[(size_t)tier * nrows + atomicAdd(&nlist[tier], 1)] = J;
        }
    }
}

// The T threads of one row (a warp or a CTA); sync() orders their shared or global memory accesses.
template <int T>
__device__ __forceinline__ void row_sync() {
    if constexpr (T == 32) __syncwarp();
    else __syncthreads();
}

// Ascending bitonic sort of key[0 .. n) for any n (flip-merge form: every comparison puts the
// smaller key first, so the missing keys past n act as +infinity and need no padding).
template <int T>
__device__ __forceinline__ void row_sort(uint64_t* key, int n, int tid) {
    int P = 1;
    while (P < n) P <<= 1;
    auto order = [&](int a, int b) {
        if (b >= n) return;
        const uint64_t ka = key[a], kb = key[b];
        if (ka > kb) {
            key[a] = kb;
            key[b] = ka;
        }
    };
    for (int half = 1, lg = 0; 2 * half <= P; half <<= 1, lg++) {
        for (int q = tid; q < P / 2; q += T) {
            const int base = (q >> lg) << (lg + 1), r = q & (half - 1);
            order(base + r, base + 2 * half - 1 - r);
        }
        row_sync<T>();
        for (int stride = half >> 1; stride > 0; stride >>= 1) {
            for (int q = tid; q < P / 2; q += T) {
                const int a = ((q & ~(stride - 1)) << 1) | (q & (stride - 1));
                order(a, a + stride);
            }
            row_sync<T>();
        }
    }
}

template <int T>
__device__ __forceinline__ int row_scan(int v, int tid, int* ws, int& total) {  // exclusive sum over the T threads
    const int lane = tid & 31;
    int incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += x;
    }
    if constexpr (T == 32) {
        total = __shfl_sync(0xffffffffu, incl, 31);
        return incl - v;
    } else {
        if (lane == 31) ws[tid >> 5] = incl;
        __syncthreads();
        int below = 0, all = 0;
        for (int k = 0; k < T / 32; k++) {
            if (k < (tid >> 5)) below += ws[k];
            all += ws[k];
        }
        __syncthreads();
        total = all;
        return below + incl - v;
    }
}

template <int T>
__device__ __forceinline__ double row_total(double v, int tid, double* ws) {  // sum over the T threads, fixed order
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if constexpr (T == 32) {
        return v;
    } else {
        if ((tid & 31) == 0) ws[tid >> 5] = v;
        __syncthreads();
        double s = 0;
        for (int k = 0; k < T / 32; k++) s += ws[k];
        __syncthreads();
        return s;
    }
}

// One output row by T threads: terms into key / val (/ val2), sort, run sums at segment offset o.
// ssrc, sw, spre: T shared entries each; wsi, wsd: T / 32 shared entries each.
template <int T, bool TWO>
__device__ __forceinline__ void gather_row(int J, const RowSrc& S, const RowMat& B, const GatherOut& O, uint64_t* key, double* val,
                                           double* val2, int tid, int* ssrc, double* sw, int* spre, int* wsi, double* wsd) {
    const int o = O.seg[J];
    const int ns = src_count(S, J);
    int cnt = 0;
    double rs = 0;
    for (int t0 = 0; t0 < ns; t0 += T) {
        int s = 0, L = 0, tot;
        double w = 0;
        if (t0 + tid < ns) {
            src_get(S, J, t0 + tid, s, w);
            L = mat_len(B, s);
            if (O.rsv) rs += w * O.rsv[s];
        }
        const int pre = row_scan<T>(L, tid, wsi, tot);
        ssrc[tid] = s;
        sw[tid] = w;
        spre[tid] = pre;
        row_sync<T>();
        const int nb = min(T, ns - t0);
        for (int f = tid; f < tot; f += T) {
            int lo = 0, hi = nb;  // last source whose first term is <= f (empty rows share a start; the last one holds f)
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (spre[mid] <= f) lo = mid;
                else hi = mid;
            }
            int c;
            double x, x2;
            mat_get(B, ssrc[lo], f - spre[lo], c, x, x2);
            key[cnt + f] = (O.skip_diag && c == J) ? kGrNone : (((uint64_t)(uint32_t)c << 32) | (uint32_t)(cnt + f));
            val[cnt + f] = sw[lo] * x;
            if (TWO) val2[cnt + f] = sw[lo] * x2;
        }
        cnt += tot;
        row_sync<T>();
    }
    row_sort<T>(key, cnt, tid);
    int u0 = 0;
    double off = 0, offabs = 0;
    for (int i0 = 0; i0 < cnt; i0 += T) {
        const int i = i0 + tid;
        const uint64_t k = i < cnt ? key[i] : kGrNone;
        const uint32_t c = (uint32_t)(k >> 32);
        const bool head = k != kGrNone && (i == 0 || (uint32_t)(key[i - 1] >> 32) != c);
        int nh;
        const int u = o + u0 + row_scan<T>(head ? 1 : 0, tid, wsi, nh);
        if (head) {
            double acc = 0, acc2 = 0;
            uint64_t kj = k;
            for (int j = i;;) {
                const uint32_t p = (uint32_t)kj;
                acc += val[p];
                if (TWO) acc2 += val2[p];
                if (++j >= cnt) break;
                kj = key[j];
                if ((uint32_t)(kj >> 32) != c) break;
            }
            O.ocol[u] = (int32_t)c;
            O.ov[u] = acc;
            if (TWO) O.ov2[u] = acc2;
            off += acc;
            offabs += fabs(acc);
        }
        u0 += nh;
    }
    if (tid == 0) O.ulen[J] = u0;
    if (O.rs_out) {  // the row's diagonal from its row sum (no cancellation of large entries) and its l1-Jacobi weight
        rs = row_total<T>(rs, tid, wsd);
        off = row_total<T>(off, tid, wsd);
        offabs = row_total<T>(offabs, tid, wsd);
        if (tid == 0) {
            const double d = rs - off;
            O.rs_out[J] = rs;
            O.diag_out[J] = d;
            const double l1 = fabs(d) + offabs;
            O.l1_out[J] = l1 > 0 ? 1.0 / l1 : 0.0;
        }
    }
    row_sync<T>();
}

// Rows of up to kGrWarpCap terms, one warp each.
template <bool TWO>
__global__ void __launch_bounds__(kGrWarps * 32) k_gather_rows(int nrows, RowSrc S, RowMat B, GatherOut O) {
    extern __shared__ __align__(16) unsigned char gr_sm[];
    __shared__ int ssrc[kGrWarps][32], spre[kGrWarps][32];
    __shared__ double sw[kGrWarps][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint64_t* K = reinterpret_cast<uint64_t*>(gr_sm) + warp * kGrWarpCap;
    double* V = reinterpret_cast<double*>(gr_sm) + (kGrWarps + warp) * kGrWarpCap;
    double* V2 = TWO ? reinterpret_cast<double*>(gr_sm) + (2 * kGrWarps + warp) * kGrWarpCap : nullptr;
    for (int J = blockIdx.x * kGrWarps + warp; J < nrows; J += gridDim.x * kGrWarps) {
        if (O.seg[J + 1] - O.seg[J] > kGrWarpCap) continue;
        gather_row<32, TWO>(J, S, B, O, K, V, V2, lane, ssrc[warp], sw[warp], spre[warp], nullptr, nullptr);
    }
}

// The listed rows of one tier, one CTA of T threads each: terms in shared memory (CAP > 0) or in
// the row's segment of the global scratch (CAP == 0).
template <int T, int CAP, bool TWO>
__global__ void __launch_bounds__(T) k_gather_rows_cta(int tier, int nrows, RowSrc S, RowMat B, GatherOut O) {
    extern __shared__ __align__(16) unsigned char gr_sm[];
    __shared__ int ssrc[T], spre[T], wsi[T / 32];
    __shared__ double sw[T], wsd[T / 32];
    const int n = O.nlist[tier];
    for (int q = blockIdx.x; q < n; q += gridDim.x) {
        const int J = O.list[(size_t)tier * nrows + q];
        uint64_t* K;
        double *V, *V2;
        if constexpr (CAP > 0) {
            K = reinterpret_cast<uint64_t*>(gr_sm);
            V = reinterpret_cast<double*>(K + CAP);
            V2 = TWO ? V + CAP : nullptr;
        } else {
            const int o = O.seg[J];
            K = O.gkey + o;
            V = O.gv + o;
            V2 = TWO ? O.gv2 + o : nullptr;
        }
        gather_row<T, TWO>(J, S, B, O, K, V, V2, threadIdx.x, ssrc, sw, spre, wsi, wsd);
    }
}

// Segments to compact CSR rows, `lanes` threads per row.
__global__ void k_gather_copy(int nrows, int lanes, const int32_t* __restrict__ seg, const int32_t* __restrict__ ulen,
                              const int32_t* __restrict__ rp, const int32_t* __restrict__ ocol, const double* __restrict__ ov,
                              const double* __restrict__ ov2, int32_t* __restrict__ col, double* __restrict__ val, double* __restrict__ val2) {
    const RowLanes g = row_lanes(lanes);
    for (int J = g.first; J < nrows; J += g.step) {
        const int o = seg[J], d = rp[J], n = ulen[J];
        for (int i = g.lane; i < n; i += lanes) {
            col[d + i] = ocol[o + i];
            val[d + i] = ov[o + i];
            if (val2) val2[d + i] = ov2[o + i];
        }
    }
}

// Q = P - w D^-1 T and Q + w P on T's pattern (T_i always holds column agg[i]).
__global__ void k_sa_q(int n, const int32_t* __restrict__ tp, const int32_t* __restrict__ tc, const double* __restrict__ tv,
                       const int32_t* __restrict__ agg, const double* __restrict__ l1inv, double* __restrict__ qv, double* __restrict__ qpv) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int a = agg[i];
        const double m = l1inv[i];
        for (int k = tp[i]; k < tp[i + 1]; k++) {
            const double base = tc[k] == a ? 1.0 : 0.0;
            const double q = base - kSaOmega * m * tv[k];
            qv[k] = q;
            qpv[k] = q + kSaOmega * base;
        }
    }
}

// Transpose of a CSR with unique columns per row: count, place, then each column's rows in order.
__global__ void k_col_count(int n, const int32_t* __restrict__ rp, const int32_t* __restrict__ col, int32_t* __restrict__ cnt) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        for (int k = rp[i]; k < rp[i + 1]; k++) atomicAdd(&cnt[col[k]], 1);
}

__global__ void k_col_place(int n, const int32_t* __restrict__ rp, const int32_t* __restrict__ col, const double* __restrict__ val,
                            const int32_t* __restrict__ cptr, int32_t* __restrict__ cursor, int32_t* __restrict__ ridx, double* __restrict__ rval) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        for (int k = rp[i]; k < rp[i + 1]; k++) {
            const int c = col[k];
            const int p = cptr[c] + atomicAdd(&cursor[c], 1);
            ridx[p] = i;
            rval[p] = val[k];
        }
}

// One warp per column; a column of more than kGrWarpCap rows by one thread in place.
__global__ void __launch_bounds__(kGrWarps * 32) k_seg_sort(int nc, const int32_t* __restrict__ ptr, int32_t* __restrict__ idx,
                                                            double* __restrict__ val) {
    __shared__ uint64_t sk[kGrWarps][kGrWarpCap];
    __shared__ double sv[kGrWarps][kGrWarpCap];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int J = blockIdx.x * kGrWarps + warp; J < nc; J += gridDim.x * kGrWarps) {
        const int b = ptr[J], e = ptr[J + 1], n = e - b;
        if (n <= kGrWarpCap) {
            for (int i = lane; i < n; i += 32) {
                sk[warp][i] = ((uint64_t)(uint32_t)idx[b + i] << 32) | (uint32_t)i;
                sv[warp][i] = val[b + i];
            }
            __syncwarp();
            row_sort<32>(sk[warp], n, lane);
            for (int i = lane; i < n; i += 32) {
                idx[b + i] = (int32_t)(sk[warp][i] >> 32);
                val[b + i] = sv[warp][(uint32_t)sk[warp][i]];
            }
            __syncwarp();
            continue;
        }
        if (lane != 0) continue;
        for (int i = b + 1; i < e; i++) {
            const int x = idx[i];
            const double y = val[i];
            int j = i - 1;
            while (j >= b && idx[j] > x) {
                idx[j + 1] = idx[j];
                val[j + 1] = val[j];
                j--;
            }
            idx[j + 1] = x;
            val[j + 1] = y;
        }
    }
}

// v = A_1 Q 1 for the coarse row sums: Q 1 = 1 - w D^-1 rs, so v = rs - w A_1 (D^-1 rs); rs
// is nonzero only next to prescribed nodes, so the chain conductances never cancel here.
__global__ void k_sa_y(int n, const double* __restrict__ l1inv, const double* __restrict__ rs, double* __restrict__ y) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) y[i] = l1inv[i] * rs[i];
}

__global__ void k_sa_v(int n, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci, const double* __restrict__ val,
                       const double* __restrict__ diag, const double* __restrict__ rs, const double* __restrict__ y, double* __restrict__ v) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double s = diag[i] * y[i];
        for (int k = rp[i]; k < rp[i + 1]; k++) s += val[k] * y[ci[k]];
        v[i] = rs[i] - kSaOmega * s;
    }
}

// Fused restriction rows of the smoothed level: row J = Q^T row J on r_1 (columns < n), then
// -(Q^T A_1) row J on z_1 (columns n + c).
__global__ void k_rr_fill_sa(int nc, int n, int lanes, const int32_t* __restrict__ qtp, const int32_t* __restrict__ qti, const double* __restrict__ qtv,
                             const int32_t* __restrict__ ap, const int32_t* __restrict__ ac, const double* __restrict__ av,
                             int32_t* __restrict__ rr_ptr, int32_t* __restrict__ rr_col, double* __restrict__ rr_val) {
    const RowLanes g = row_lanes(lanes);
    for (int J = g.first; J < nc; J += g.step) {
        const int q = qtp[J], nq = qtp[J + 1] - q, a = ap[J], na = ap[J + 1] - a, e = q + a;
        if (g.lane == 0) {
            rr_ptr[J] = e;
            if (J == nc - 1) rr_ptr[nc] = qtp[nc] + ap[nc];
        }
        for (int k = g.lane; k < nq; k += lanes) {
            rr_col[e + k] = qti[q + k];
            rr_val[e + k] = qtv[q + k];
        }
        for (int k = g.lane; k < na; k += lanes) {
            rr_col[e + nq + k] = n + ac[a + k];
            rr_val[e + nq + k] = -av[a + k];
        }
    }
}

// Fused prolongation-smoother rows of the smoothed level: row I = A_1 row I with its diagonal
// on z_1, then A_1 (Q + w P) row I on zc (columns n + J).
__global__ void k_pq_fill_sa(int n, int lanes, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci, const double* __restrict__ v,
                             const double* __restrict__ diag, const int32_t* __restrict__ wp, const int32_t* __restrict__ wc,
                             const double* __restrict__ wv, int32_t* __restrict__ pq_ptr, int32_t* __restrict__ pq_col,
                             double* __restrict__ pq_val) {
    const RowLanes g = row_lanes(lanes);
    for (int I = g.first; I < n; I += g.step) {
        const int b = rp[I], nb = rp[I + 1] - b, w = wp[I], nw = wp[I + 1] - w, e = b + I + w;
        if (g.lane == 0) {
            pq_ptr[I] = e;
            if (I == n - 1) pq_ptr[n] = rp[n] + n + wp[n];
            pq_col[e] = I;
            pq_val[e] = diag[I];
        }
        for (int k = g.lane; k < nb; k += lanes) {
            pq_col[e + 1 + k] = ci[b + k];
            pq_val[e + 1 + k] = v[b + k];
        }
        for (int k = g.lane; k < nw; k += lanes) {
            pq_col[e + 1 + nb + k] = n + wc[w + k];
            pq_val[e + 1 + nb + k] = wv[w + k];
        }
    }
}

template <bool TWO>
void launch_gather(MgWork& g, int nrows, const RowSrc& S, const RowMat& B, const GatherOut& O, bool global_tier, cudaStream_t s, int64_t& launches) {
    constexpr int kSets = TWO ? 3 : 2;
    constexpr int warp_sm = (int)sizeof(double) * kGrWarps * kGrWarpCap * kSets;
    constexpr int mid_sm = (int)sizeof(double) * kGrMidCap * kSets, big_sm = (int)sizeof(double) * kGrBigCap * kSets;
    if (!g.gather_attr[TWO]) {
        CICY_CUDA(cudaFuncSetAttribute(k_gather_rows<TWO>, cudaFuncAttributeMaxDynamicSharedMemorySize, warp_sm));
        CICY_CUDA(cudaFuncSetAttribute(k_gather_rows_cta<kGrMidThreads, kGrMidCap, TWO>, cudaFuncAttributeMaxDynamicSharedMemorySize, mid_sm));
        CICY_CUDA(cudaFuncSetAttribute(k_gather_rows_cta<kGrBigThreads, kGrBigCap, TWO>, cudaFuncAttributeMaxDynamicSharedMemorySize, big_sm));
        g.gather_attr[TWO] = true;
    }
    // grids: the CTAs that are resident at once (4 to 6 of the small, 1 of the large CTAs per SM); lists are shared out by stride
    k_gather_rows<TWO><<<grid_for((long long)nrows * 32, kGrWarps * 32), kGrWarps * 32, warp_sm, s>>>(nrows, S, B, O);
    k_gather_rows_cta<kGrMidThreads, kGrMidCap, TWO><<<std::min(nrows, 148 * 6), kGrMidThreads, mid_sm, s>>>(0, nrows, S, B, O);
    k_gather_rows_cta<kGrBigThreads, kGrBigCap, TWO><<<std::min(nrows, 148), kGrBigThreads, big_sm, s>>>(1, nrows, S, B, O);
    launches += 3;
    if (global_tier) {
        k_gather_rows_cta<kGrBigThreads, 0, TWO><<<std::min(nrows, 148), kGrBigThreads, 0, s>>>(2, nrows, S, B, O);
        launches++;
    }
}

// One row-gather product: the compacted CSR (optr, ocol, oval[, oval2]) of nrows rows.  Its arrays
// are sized by the number of candidate terms, which is returned (>= entries): `cand`, an upper
// bound known to the caller, or (-1) read from the device.
long long gather_product(MgWork& g, int nrows, const RowSrc& S, const RowMat& B, bool skip_diag, const double* rsv, double* rs_out,
                         double* diag_out, double* l1_out, long long cand, int lanes, DBuf<int32_t>& optr, DBuf<int32_t>& ocol,
                         DBuf<double>& oval, DBuf<double>* oval2, cudaStream_t s, int64_t& launches) {
    MgWork::Smoothed& w = g.sa;
    w.seg.ensure(nrows + 1);
    w.longr.ensure((size_t)kGrTiers * nrows + 1);
    int32_t* nlist = g.total.get() + 1;
    CICY_CUDA(cudaMemsetAsync(nlist, 0, sizeof(int32_t) * kGrTiers, s));
    k_gather_len<<<grid_for(8LL * nrows), 256, 0, s>>>(nrows, 8, S, B, w.seg.get(), w.longr.get(), nlist);
    launches++;
    exclusive_scan_i32(w.seg.get(), w.seg.get(), nrows + 1, g.total.get(), g.scan_tmp, s, launches);
    bool global_tier = cand > kGrBigCap;  // some row may have more terms than a CTA's shared memory holds
    if (cand < 0) {
        int h[1 + kGrTiers];
        CICY_CUDA(cudaMemcpyAsync(h, g.total.get(), sizeof(h), cudaMemcpyDeviceToHost, s));
        CICY_CUDA(cudaStreamSynchronize(s));
        cand = h[0];
        global_tier = h[kGrTiers] > 0;
    }
    const size_t cap = (size_t)std::max<long long>(cand, 1);
    const bool two = B.val2 != nullptr;
    w.ocol.ensure(cap);
    w.ov.ensure(cap);
    if (two) w.ov2.ensure(cap);
    if (global_tier) {
        w.gkey.ensure(cap);
        w.gv.ensure(cap);
        if (two) w.gv2.ensure(cap);
    }
    w.ulen.ensure(nrows + 1);
    const GatherOut O{w.seg.get(), w.gkey.get(), w.gv.get(), w.gv2.get(), w.ocol.get(), w.ov.get(), two ? w.ov2.get() : nullptr, w.ulen.get(),
                      w.longr.get(), nlist, skip_diag ? 1 : 0, rsv, rs_out, diag_out, l1_out};
    if (two) launch_gather<true>(g, nrows, S, B, O, global_tier, s, launches);
    else launch_gather<false>(g, nrows, S, B, O, global_tier, s, launches);
    optr.ensure(nrows + 1);
    exclusive_scan_i32(w.ulen.get(), optr.get(), nrows + 1, nullptr, g.scan_tmp, s, launches);
    ocol.ensure(cap);
    oval.ensure(cap);
    if (two) oval2->ensure(cap);
    k_gather_copy<<<grid_for((long long)nrows * lanes), 256, 0, s>>>(nrows, lanes, w.seg.get(), w.ulen.get(), optr.get(), w.ocol.get(),
                                                                     w.ov.get(), two ? w.ov2.get() : nullptr, ocol.get(), oval.get(),
                                                                     two ? oval2->get() : nullptr);
    launches++;
    CICY_LAUNCH_CHECK();
    return cand;
}

// Level 2 from level 1 through the smoothed prolongator (nc pairwise aggregates in
// g.L[1].agg), with level 1's fused restriction and prolongation-smoother rows.
void coarsen_smoothed(MgWork& g, int nc, cudaStream_t s, int64_t& launches) {
    MgWork::Lvl& F = g.L[1];
    MgWork::Lvl& G = g.L[2];
    MgWork::Smoothed& w = g.sa;
    const int n = F.n;
    const RowSrc one{nullptr, nullptr, nullptr, nullptr};
    const RowSrc a1_src{F.rp_ptr, F.ci_ptr, F.val_ptr, F.diag.get()};
    const RowMat a1{F.rp_ptr, F.ci_ptr, F.val_ptr, F.diag.get(), nullptr, nullptr, nullptr};
    const RowMat a1_agg{F.rp_ptr, F.ci_ptr, F.val_ptr, F.diag.get(), nullptr, nullptr, F.agg.get()};
    // T = A_1 P, then Q and Q + w P on its pattern
    const long long nt = gather_product(g, n, one, a1_agg, false, nullptr, nullptr, nullptr, nullptr, (long long)F.nnz + n, 8, w.tp, w.tc, w.tv,
                                        nullptr, s, launches);
    w.qv.ensure(nt);
    w.qpv.ensure(nt);
    k_sa_q<<<grid_for(n), 256, 0, s>>>(n, w.tp.get(), w.tc.get(), w.tv.get(), F.agg.get(), F.l1inv.get(), w.qv.get(), w.qpv.get());
    // Q^T: each aggregate's rows in ascending order
    w.qtp.ensure(nc + 1);
    w.qti.ensure(nt);
    w.qtv.ensure(nt);
    g.flag.ensure(nc + 1);
    CICY_CUDA(cudaMemsetAsync(g.flag.get(), 0, sizeof(int32_t) * (nc + 1), s));
    k_col_count<<<grid_for(n), 256, 0, s>>>(n, w.tp.get(), w.tc.get(), g.flag.get());
    exclusive_scan_i32(g.flag.get(), w.qtp.get(), nc + 1, nullptr, g.scan_tmp, s, launches);
    CICY_CUDA(cudaMemsetAsync(g.flag.get(), 0, sizeof(int32_t) * (nc + 1), s));
    k_col_place<<<grid_for(n), 256, 0, s>>>(n, w.tp.get(), w.tc.get(), w.qv.get(), w.qtp.get(), g.flag.get(), w.qti.get(), w.qtv.get());
    k_seg_sort<<<grid_for((long long)nc * 32, kGrWarps * 32), kGrWarps * 32, 0, s>>>(nc, w.qtp.get(), w.qti.get(), w.qtv.get());
    launches += 4;
    const RowSrc qt_src{w.qtp.get(), w.qti.get(), w.qtv.get(), nullptr};
    // W = A_1 Q and A_1 (Q + w P)
    const RowMat q{w.tp.get(), w.tc.get(), w.qv.get(), nullptr, w.qpv.get(), nullptr, nullptr};
    const long long nw = gather_product(g, n, a1_src, q, false, nullptr, nullptr, nullptr, nullptr, -1, 32, w.wp, w.wc, w.wv, &w.wpv, s, launches);
    // Q^T A_1 (the restriction rows' part on z_1)
    const long long na = gather_product(g, nc, qt_src, a1, false, nullptr, nullptr, nullptr, nullptr, -1, 32, w.ap, w.ac, w.av, nullptr, s, launches);
    // A_2 = Q^T W off the diagonal; its diagonal from the row sums Q^T A_1 Q 1
    w.y.ensure(n);
    w.v.ensure(n);
    k_sa_y<<<grid_for(n), 256, 0, s>>>(n, F.l1inv.get(), F.rs.get(), w.y.get());
    k_sa_v<<<grid_for(n), 256, 0, s>>>(n, F.rp_ptr, F.ci_ptr, F.val_ptr, F.diag.get(), F.rs.get(), w.y.get(), w.v.get());
    launches += 2;
    G.n = nc;
    G.rs.ensure(nc);
    G.diag.ensure(nc);
    G.l1inv.ensure(nc);
    const RowMat wm{w.wp.get(), w.wc.get(), w.wv.get(), nullptr, nullptr, nullptr, nullptr};
    const long long n2 = gather_product(g, nc, qt_src, wm, true, w.v.get(), G.rs.get(), G.diag.get(), G.l1inv.get(), -1, 32, G.rp, G.ci, G.val,
                                        nullptr, s, launches);
    G.nnz = (int)std::max<long long>(n2, 1);
    G.rp_ptr = G.rp.get();
    G.ci_ptr = G.ci.get();
    G.val_ptr = G.val.get();
    // level 1's fused rows
    F.rr_ptr.ensure(nc + 1);
    F.rr_col.ensure(std::max<long long>(nt + na, 1));
    F.rr_val.ensure(std::max<long long>(nt + na, 1));
    k_rr_fill_sa<<<grid_for(32LL * nc), 256, 0, s>>>(nc, n, 32, w.qtp.get(), w.qti.get(), w.qtv.get(), w.ap.get(), w.ac.get(), w.av.get(), F.rr_ptr.get(),
                                               F.rr_col.get(), F.rr_val.get());
    F.pq_ptr.ensure(n + 1);
    F.pq_col.ensure(std::max<long long>((long long)F.nnz + n + nw, 1));
    F.pq_val.ensure(std::max<long long>((long long)F.nnz + n + nw, 1));
    k_pq_fill_sa<<<grid_for(32LL * n), 256, 0, s>>>(n, 32, F.rp_ptr, F.ci_ptr, F.val_ptr, F.diag.get(), w.wp.get(), w.wc.get(), w.wpv.get(),
                                              F.pq_ptr.get(), F.pq_col.get(), F.pq_val.get());
    launches += 2;
    CICY_LAUNCH_CHECK();
}

// Galerkin coarse level l+1 from level l and its aggregates (g.L[l].agg, nc of
// them), plus level l's member lists, restriction rows (l >= 1) and column
// aggregates.  No host synchronisation here: buffers are sized by the fine level's
// non-zeros, an upper bound of the coarse level's.
void coarsen(MgWork& g, int l, int nc, cudaStream_t s, int64_t& launches) {
    if ((int)g.L.size() < l + 2) g.L.resize(l + 2);
    if (g.fused && g.smooth && l == 1) {
        coarsen_smoothed(g, nc, s, launches);
        return;
    }
    MgWork::Lvl& F = g.L[l];
    MgWork::Lvl& G = g.L[l + 1];
    const int nf = F.n, nnz = F.nnz, lf = lanes_of(nnz, nf);
    F.mptr.ensure(nc + 1);
    F.midx.ensure(std::max(nf, 1));
    if (l == 0) {
        k_members_contig<<<grid_for(nf), 256, 0, s>>>(nf, nc, F.agg.get(), F.mptr.get(), F.midx.get());
        launches++;
    } else {
        g.flag.ensure(nc + 1);
        CICY_CUDA(cudaMemsetAsync(g.flag.get(), 0, sizeof(int32_t) * (nc + 1), s));
        k_member_count<<<grid_for(nf), 256, 0, s>>>(nf, F.agg.get(), g.flag.get());
        exclusive_scan_i32(g.flag.get(), F.mptr.get(), nc + 1, nullptr, g.scan_tmp, s, launches);
        CICY_CUDA(cudaMemsetAsync(g.flag.get(), 0, sizeof(int32_t) * (nc + 1), s));
        k_member_place<<<grid_for(nf), 256, 0, s>>>(nf, F.agg.get(), F.mptr.get(), g.flag.get(), F.midx.get());
        k_member_sort<<<grid_for(nc), 256, 0, s>>>(nc, F.mptr.get(), F.midx.get());
        launches += 3;
    }
    if (l >= 1) {
        F.ra_ptr.ensure(nc + 1);
        k_ra_lengths<<<grid_for(nc), 256, 0, s>>>(nc, F.mptr.get(), F.midx.get(), F.rp_ptr, F.ra_ptr.get());
        launches++;
    }
    // coarse rows
    G.n = nc;
    G.nnz = nnz;  // upper bound (build_mg_hierarchy reads the length)
    G.rs.ensure(nc);
    G.diag.ensure(nc);
    G.l1inv.ensure(nc);
    const RowSrc members{F.mptr.get(), F.midx.get(), nullptr, nullptr};
    const RowMat fine{F.rp_ptr, F.ci_ptr, F.val_ptr, nullptr, nullptr, nullptr, F.agg.get()};
    gather_product(g, nc, members, fine, true, F.rs.get(), G.rs.get(), G.diag.get(), G.l1inv.get(), nnz, l >= 1 ? 32 : 8, G.rp, G.ci, G.val, nullptr,
                   s, launches);
    G.rp_ptr = G.rp.get();
    G.ci_ptr = G.ci.get();
    G.val_ptr = G.val.get();
    // restriction rows of level l (l >= 1) and its column aggregates; the grid kernel
    // (g.fused) reads the fused rows instead of P^T A_l and the coarse column aggregates
    if (l >= 1) {
        exclusive_scan_i32(F.ra_ptr.get(), F.ra_ptr.get(), nc + 1, nullptr, g.scan_tmp, s, launches);
        if (!g.fused) {
            F.ra_col.ensure(std::max(nnz + nf, 1));
            F.ra_val.ensure(std::max(nnz + nf, 1));
            k_ra_fill<<<grid_for((long long)nc * lf), 256, 0, s>>>(nc, lf, F.mptr.get(), F.midx.get(), F.rp_ptr, F.ci_ptr, F.val_ptr, F.diag.get(),
                                                    F.ra_ptr.get(), F.ra_col.get(), F.ra_val.get());
            launches++;
        }
    }
    if (!g.fused || l == 0) {
        F.cagg.ensure(std::max(nnz, 1));
        k_cagg<<<grid_for(nnz), 256, 0, s>>>(F.rp_ptr + nf, F.ci_ptr, F.agg.get(), F.cagg.get());
        launches++;
    }
    if (g.fused && l >= 1) {
        F.rr_ptr.ensure(nc + 1);
        F.rr_col.ensure(std::max(nnz + 2 * nf, 1));
        F.rr_val.ensure(std::max(nnz + 2 * nf, 1));
        k_rr_fill<<<grid_for((long long)nc * lf), 256, 0, s>>>(nc, nf, lf, F.mptr.get(), F.midx.get(), F.rp_ptr, F.ci_ptr, F.val_ptr, F.diag.get(), F.ra_ptr.get(),
                                                F.rr_ptr.get(), F.rr_col.get(), F.rr_val.get());
        F.pq_ptr.ensure(nf + 1);
        F.pq_col.ensure(std::max(2 * (nnz + nf), 1));
        F.pq_val.ensure(std::max(2 * (nnz + nf), 1));
        k_pq_fill<<<grid_for((long long)nf * lf), 256, 0, s>>>(nf, lf, F.rp_ptr, F.ci_ptr, F.val_ptr, F.diag.get(), F.agg.get(), F.pq_ptr.get(),
                                                F.pq_col.get(), F.pq_val.get());
        launches += 2;
    }
    CICY_LAUNCH_CHECK();
}

// Whether a chain graph of `rows` and `entries` takes the smoothed prolongator.  Smoothing a
// level whose rows have d couplings gives the next level about d^2 couplings a row, so it pays
// only on sparse chain graphs: whole path in ms, smoothed against piecewise constant, by couplings
// per chain (unit and real pass): 2.3, 2.5: 20.7 / 29.2 (48.9k CNTs, 8 um); 2.4, 2.6: 12.7 / 12.9
// (25k, 6 um); 2.8, 3.0: 11.5 / 12.5 (15.1k, 4.5 um); 3.2, 3.4: 13.7 / 12.2 (23.9k, 5 um); 3.8, 3.9:
// 42.6 / 13.4 (16.3k, 4 um); 5.3, 5.4: 28.3 / 15.9 (24.4k, 4 um); 5.7, 5.8: 60.9 / 27.5 (47.7k, 5 um).
// Small graphs are bound by the phases' latency, not by their entries: 6.3k chains of 3.5-3.7
// couplings 9.1 / 8.4, 7.2k chains 8.9 / 8.9, but 8.5k chains of 3.9-4.1 couplings 10.8 / 9.2.
bool smoothing_pays(int rows, int entries) {
    return 10LL * entries < 31LL * rows || (rows <= 8192 && 10LL * entries < 37LL * rows);
}

// Pairwise aggregates of level l; returns their number and sets the level's entry count.
int pairwise(MgWork& g, int l, cudaStream_t s, int64_t& launches) {
    MgWork::Lvl& F = g.L[l];
    const int n = F.n, ln = lanes_of(F.nnz, n), gl = grid_for((long long)n * ln);
    g.mate.ensure(n + 1);
    g.best.ensure(n + 1);
    g.rep.ensure(n + 1);
    g.flag.ensure(n + 1);
    g.pos.ensure(n + 1);
    k_fill_neg<<<grid_for(n), 256, 0, s>>>(n, g.mate.get());
    launches++;
    for (int round = 0; round < 3; round++) {
        k_strongest<<<gl, 256, 0, s>>>(n, ln, 1, F.rp_ptr, F.ci_ptr, F.val_ptr, g.mate.get(), g.best.get());
        k_handshake<<<grid_for(n), 256, 0, s>>>(n, g.best.get(), g.mate.get());
        launches += 2;
    }
    k_pair_rep<<<grid_for(n), 256, 0, s>>>(n, g.mate.get(), g.rep.get());
    k_strongest<<<gl, 256, 0, s>>>(n, ln, 0, F.rp_ptr, F.ci_ptr, F.val_ptr, g.mate.get(), g.best.get());
    k_join<<<grid_for(n), 256, 0, s>>>(n, g.mate.get(), g.best.get(), g.rep.get());
    k_is_rep<<<grid_for(n), 256, 0, s>>>(n, g.rep.get(), g.flag.get());
    launches += 4;
    exclusive_scan_i32(g.flag.get(), g.pos.get(), n, g.total.get(), g.scan_tmp, s, launches);
    F.agg.ensure(n + 1);
    k_agg_ids<<<grid_for(n), 256, 0, s>>>(n, g.rep.get(), g.pos.get(), F.agg.get());
    launches++;
    int nc = 0;
    CICY_CUDA(cudaMemcpyAsync(&nc, g.total.get(), sizeof(int), cudaMemcpyDeviceToHost, s));
    CICY_CUDA(cudaMemcpyAsync(&F.nnz, F.rp_ptr + n, sizeof(int), cudaMemcpyDeviceToHost, s));  // until here an upper bound
    CICY_CUDA(cudaStreamSynchronize(s));
    CICY_LAUNCH_CHECK();
    return nc;
}

}  // namespace

// Edge of the grid Gauss-Jordan's CTA grid: the largest square that is resident at once.
int gj_grid(int sms) {
    int P = 1;
    while ((P + 1) * (P + 1) <= sms) P++;
    return P;
}

// ---------------------------------------------------------------------------
void build_mg_hierarchy(SolverWork& w, const SolverSystem& sys, cudaStream_t s, int64_t& launches, bool fused, bool smooth, int* status) {
    MgWork& g = w.mg;
    const int n = sys.n;
    g.fused = fused;
    g.smooth = smooth;
    TraceSeq tr(s);
    g.total.ensure(1 + kGrTiers);
    if (g.L.empty()) g.L.resize(1);
    MgWork::Lvl& L0 = g.L[0];
    L0.n = n;
    L0.nnz = sys.nnz;
    L0.rp_ptr = sys.rp;
    L0.ci_ptr = sys.ci;
    L0.val_ptr = sys.val;
    L0.agg.ensure(n + 1);
    L0.rs.ensure(n + 1);
    k_block_of_row<<<grid_for(n), 256, 0, s>>>(n, w.is_start.get(), w.start_scan.get(), L0.agg.get());
    k_rowsum0<<<grid_for(n), 256, 0, s>>>(n, sys.rp, sys.ci, sys.val, L0.rs.get());
    launches += 2;
    int nc = w.n_blocks;
    int C = 0;
    // the grid kernel solves a dense coarsest of up to kMgDenseGridMax rows on all CTAs
    int dense_cap = kMgDenseMax;
    if (fused) {
        int dev = 0, sms = 0;
        CICY_CUDA(cudaGetDevice(&dev));
        CICY_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        dense_cap = std::max(kMgDenseMax, std::min(kMgDenseGridMax, gj_grid(sms) * kGjgTile));
    }
    for (int l = 0;; l++) {
        coarsen(g, l, nc, s, launches);
        tr.mark("mg.coarsen");
        C = l + 1;
        if (g.L[C].n <= dense_cap || C + 1 >= kMgMaxLevels) break;
        const int nc2 = pairwise(g, C, s, launches);
        tr.mark("mg.pairwise");
        if (C == 1) g.smooth = smooth && smoothing_pays(g.L[1].n, g.L[1].nnz);
        if (nc2 > 0.9 * g.L[C].n) break;
        nc = nc2;
    }
    g.dense = false;
    MgWork::Lvl& Lc = g.L[C];
    if (Lc.n <= kMgDenseMax) {
        g.cinv.ensure((size_t)Lc.n * Lc.n);
        CICY_CUDA(cudaMemsetAsync(g.cinv.get(), 0, sizeof(double) * Lc.n * Lc.n, s));
        k_dense_coarse<<<grid_for(32LL * Lc.n, 128), 128, 0, s>>>(Lc.n, 32, Lc.rp.get(), Lc.ci.get(), Lc.val.get(), Lc.diag.get(), g.cinv.get());
        auto bytes = [](size_t m) { return sizeof(double) * (m * m + 2 * m * kGjBlock + kGjBlock * (kGjBlock + 1) + kGjBlock); };
        const size_t smem = bytes(Lc.n);
        // always the limit of the largest level: a context in another thread may set it between this and the launch
        CICY_CUDA(cudaFuncSetAttribute(k_gauss_jordan, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes(kMgDenseMax)));
        k_gauss_jordan<<<1, kGjThreads, smem, s>>>(Lc.n, g.cinv.get());
        launches += 2;
        g.dense = true;
    } else if (Lc.n <= dense_cap) {
        // larger dense coarsest: the grid Gauss-Jordan (one cooperative launch, square tiles)
        int nC = Lc.n, dev = 0, sms = 0;
        CICY_CUDA(cudaGetDevice(&dev));
        CICY_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        g.cinv.ensure((size_t)nC * nC);
        g.gj_panel.ensure((size_t)4 * nC * kGjBlock);
        g.gj_sync.ensure(2);
        g.gj_err.ensure(1);
        CICY_CUDA(cudaMemsetAsync(g.gj_sync.get(), 0, sizeof(unsigned long long) * 2, s));
        int* err = status;
        if (!err) {
            CICY_CUDA(cudaMemsetAsync(g.gj_err.get(), 0, sizeof(int32_t), s));
            err = g.gj_err.get();
        }
        CICY_CUDA(cudaMemsetAsync(g.cinv.get(), 0, sizeof(double) * nC * nC, s));
        k_dense_coarse<<<grid_for(32LL * nC, 128), 128, 0, s>>>(nC, 32, Lc.rp.get(), Lc.ci.get(), Lc.val.get(), Lc.diag.get(), g.cinv.get());
        int P = gj_grid(sms);
        const int tile = (nC + P - 1) / P;
        if (tile > kGjgTile) throw Fail{CICY_E_INTERNAL, "multigrid: dense coarsest too large for this GPU"};
        void (*kern)(int, int, double*, double*, unsigned long long*, unsigned long long*, int*, long long) = nullptr;
        int edge[2];  // rows and columns of the kernel's tile
        if (tile <= 32) kern = k_gauss_jordan_grid<1, 2>, edge[0] = 32, edge[1] = 32;
        else if (tile <= 64) kern = k_gauss_jordan_grid<2, 4>, edge[0] = 64, edge[1] = 64;
        else if (tile <= 80) kern = k_gauss_jordan_grid<3, 5>, edge[0] = 96, edge[1] = 80;
        else if (tile <= 96) kern = k_gauss_jordan_grid<3, 6>, edge[0] = 96, edge[1] = 96;
        else kern = k_gauss_jordan_grid<4, 7>, edge[0] = 128, edge[1] = 112;
        const size_t smem = sizeof(double) * kGjBlock * (edge[0] + 2 * edge[1]);
        CICY_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        double* M = g.cinv.get();
        double* panel = g.gj_panel.get();
        unsigned long long* bar = g.gj_sync.get();
        unsigned long long* dmax = g.gj_sync.get() + 1;
        long long limit = w.spin_limit;
        void* args[] = {&nC, &P, &M, &panel, &bar, &dmax, &err, &limit};
        CICY_CUDA(cudaLaunchCooperativeKernel((void*)kern, dim3(P * P), dim3(kGjgThreads), args, smem, s));
        launches += 2;
        g.dense = true;
    }
    tr.mark("mg.coarsest");
    tr.mark("mg.restriction_rows");
    // work vectors and device descriptors
    g.host_lv.assign(C + 1, MgLevel{});
    for (int l = 0; l <= C; l++) {
        MgWork::Lvl& L = g.L[l];
        MgLevel& d = g.host_lv[l];
        d.n = L.n;
        d.rp = L.rp_ptr;
        d.ci = L.ci_ptr;
        d.val = L.val_ptr;
        d.agg = (l < C) ? L.agg.get() : nullptr;
        d.mptr = (l < C) ? L.mptr.get() : nullptr;
        d.midx = (l < C) ? L.midx.get() : nullptr;
        d.cagg = (l < C) ? L.cagg.get() : nullptr;
        d.ra_ptr = (l >= 1 && l < C) ? L.ra_ptr.get() : nullptr;
        d.ra_col = (l >= 1 && l < C) ? L.ra_col.get() : nullptr;
        d.ra_val = (l >= 1 && l < C) ? L.ra_val.get() : nullptr;
        if (l >= 1) {
            L.r.ensure(L.n + 1);
            L.z.ensure(L.n + 1);
            d.diag = L.diag.get();
            d.l1inv = L.l1inv.get();
            d.r = L.r.get();
            d.z = L.z.get();
            if (l == C && !g.dense) {
                d.zf = L.z.get();
            } else {
                L.zf.ensure(L.n + 1);
                d.zf = L.zf.get();
            }
        }
    }
    g.dev_lv.ensure(C + 1);
    CICY_CUDA(cudaMemcpyAsync(g.dev_lv.get(), g.host_lv.data(), sizeof(MgLevel) * (C + 1), cudaMemcpyHostToDevice, s));
    CICY_CUDA(cudaStreamSynchronize(s));
    g.levels = C + 1;
    CICY_LAUNCH_CHECK();
    if (trace_enabled())
        for (int l = 0; l <= C; l++) {
            int nz = 0, rr = 0, pq = 0;
            if (g.L[l].rp_ptr) cudaMemcpy(&nz, g.L[l].rp_ptr + g.L[l].n, 4, cudaMemcpyDeviceToHost);
            if (g.fused && l >= 1 && l < C) {
                cudaMemcpy(&rr, g.L[l].rr_ptr.get() + g.L[l + 1].n, 4, cudaMemcpyDeviceToHost);
                cudaMemcpy(&pq, g.L[l].pq_ptr.get() + g.L[l].n, 4, cudaMemcpyDeviceToHost);
            }
            std::fprintf(stderr, "[cicy] mg level %d rows %d entries %d restriction %d prolongation %d\n", l, g.L[l].n, nz, rr, pq);
        }
}

bool mg_fused_path(int n, bool allow_cluster) { return !(allow_cluster && n <= kMgClusterMaxRows); }

void pcg_solve_mg(SolverWork& w, const SolverSystem& sys, double tol, long long max_iter, bool allow_cluster, int num_sms, int* status,
                  cudaStream_t s, int64_t& launches, PcgStats& st) {
    const int n = sys.n;
    st = PcgStats{};
    if (n <= 0) return;
    MgWork& g = w.mg;
    w.r.ensure(n); w.z.ensure(n); w.p.ensure(n); w.q.ensure(n);
    g.z0.ensure(n);
    g.wtmp.ensure(n);
    k_residual<<<grid_for(n), 256, 0, s>>>(n, sys.rp, sys.ci, sys.val, sys.x, sys.b, w.r.get());
    launches++;
    // up to kMgClusterMaxRows one 16-CTA cluster with hardware barriers when it can be launched, else the
    // grid-wide cooperative launch
    if (g.cl_state == 0) {
        g.cl_state = cudaFuncSetAttribute(k_mg_pcg<true>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess ? 1 : -1;
        cudaGetLastError();
    }
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    bool cluster = false;
    if (allow_cluster && !g.fused && g.cl_state > 0 && n <= kMgClusterMaxRows) {
        cfg.gridDim = dim3(kMgClusterCtas);
        cfg.blockDim = dim3(kMgClusterThreads);
        cfg.dynamicSmemBytes = 0;
        cfg.stream = s;
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = kMgClusterCtas;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int nclusters = 0;
        cluster = cudaOccupancyMaxActiveClusters(&nclusters, (void*)k_mg_pcg<true>, &cfg) == cudaSuccess && nclusters >= 1;
        cudaGetLastError();
    }
    // above one cluster's size: the shared-memory-resident grid kernel, one CTA per SM
    bool sec = false;
    int nb = kMgClusterCtas;
    if (!cluster && g.fused && g.levels >= 2) {
        if (g.sm_state == 0) {
            g.sm_state = cudaFuncSetAttribute(k_mg_pcg_sm, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmBytes) == cudaSuccess ? 1 : -1;
            cudaGetLastError();
        }
        int occ = 0;
        if (g.sm_state > 0 && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_mg_pcg_sm, kSmThreads, kSmBytes) == cudaSuccess && occ >= 1) {
            nb = std::max(1, std::min({num_sms, kSmThreads, ceil_div(n, 128)}));
            sec = true;
        }
        cudaGetLastError();
    }
    if (g.fused && !sec) throw Fail{CICY_E_INTERNAL, "multigrid: the grid kernel cannot be launched for a hierarchy built for it"};
    if (!sec && !cluster) {
        int occ = 0;
        CICY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_mg_pcg<false>, kMgThreads, 0));
        const int cap = std::max(1, occ) * num_sms;
        nb = std::max(1, std::min({cap, num_sms, ceil_div(n, 2 * kMgThreads)}));
    }
    std::vector<MgSmLevel> hl;  // kept until the stream synchronisation below
    MgSmArgs sa{};
    if (sec) {
        const int C = g.levels - 1;
        hl.assign(C + 1, MgSmLevel{});
        for (int l = 0; l <= C; l++) {
            MgWork::Lvl& L = g.L[l];
            MgSmLevel& d = hl[l];
            d.n = L.n;
            if (l == 0) continue;
            if (l < C) {
                d.rr_ptr = L.rr_ptr.get();
                d.rr_col = L.rr_col.get();
                d.rr_val = L.rr_val.get();
                d.pq_ptr = L.pq_ptr.get();
                d.pq_col = L.pq_col.get();
                d.pq_val = L.pq_val.get();
                d.agg = L.agg.get();
            }
            d.l1inv = L.l1inv.get();
            d.r = L.r.get();
            d.z = L.z.get();
            d.zf = l == C && !g.dense ? d.z : L.zf.get();
        }
        g.sec_lv.ensure(sizeof(MgSmLevel) * (C + 1));
        CICY_CUDA(cudaMemcpyAsync(g.sec_lv.get(), hl.data(), sizeof(MgSmLevel) * (C + 1), cudaMemcpyHostToDevice, s));
        sa.lv = reinterpret_cast<const MgSmLevel*>(g.sec_lv.get());
        sa.mptr0 = g.L[0].mptr.get();
        sa.lfac = w.lfac.get();
        sa.ipiv = w.ipiv.get();
        sa.smem_bytes = kSmBytes;
    }
    w.cta_row.ensure(nb + 1);
    launch_cta_rows(nb, n, w.is_start.get(), w.cta_row.get(), s);
    w.part.ensure(4 * nb + 8);
    g.bar.ensure(1);
    w.stats.ensure(4);
    CICY_CUDA(cudaMemsetAsync(g.bar.get(), 0, sizeof(unsigned long long), s));
    CICY_CUDA(cudaMemsetAsync(w.stats.get(), 0, sizeof(double) * 4, s));
    MgArgs a{};
    a.n = n;
    a.rp = sys.rp; a.ci = sys.ci; a.val = sys.val; a.b = sys.b; a.x = sys.x;
    a.r = w.r.get(); a.z0 = g.z0.get(); a.z = w.z.get(); a.w = g.wtmp.get(); a.p = w.p.get(); a.q = w.q.get();
    a.tinv = w.tinv.get(); a.row_off = w.row_off.get(); a.row_base = w.row_base.get(); a.row_m = w.row_m.get();
    a.cta_row = w.cta_row.get();
    a.levels = g.levels;
    a.lv = g.dev_lv.get();
    a.cinv = g.dense ? g.cinv.get() : nullptr;
    a.omega0 = kOmega0;
    a.partA = w.part.get();
    a.partB = w.part.get() + 2 * nb;
    a.stats = w.stats.get();
    a.bar = g.bar.get();
    a.spin_limit = w.spin_limit;
    a.err = status;
    a.tol = tol;
    a.max_iter = max_iter;
    a.max_restarts = kMgMaxRestarts;
    cudaEvent_t e0, e1;
    CICY_CUDA(cudaEventCreate(&e0));
    CICY_CUDA(cudaEventCreate(&e1));
    CICY_CUDA(cudaEventRecord(e0, s));
    if (cluster) {
        CICY_CUDA(cudaLaunchKernelEx(&cfg, k_mg_pcg<true>, a));
    } else if (sec) {
        void* args[] = {&a, &sa};
        CICY_CUDA(cudaLaunchCooperativeKernel((void*)k_mg_pcg_sm, dim3(nb), dim3(kSmThreads), args, kSmBytes, s));
    } else {
        void* args[] = {&a};
        CICY_CUDA(cudaLaunchCooperativeKernel((void*)k_mg_pcg<false>, dim3(nb), dim3(kMgThreads), args, 0, s));
    }
    CICY_CUDA(cudaEventRecord(e1, s));
    launches++;
    double hs[4];
    CICY_CUDA(cudaMemcpyAsync(hs, w.stats.get(), sizeof(hs), cudaMemcpyDeviceToHost, s));
    CICY_CUDA(cudaStreamSynchronize(s));
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    st.iterations = (long long)hs[0];
    st.restarts = (int)hs[3];
    st.seconds = ms * 1e-3;
    st.ctas = nb;
    st.levels = g.levels;
    st.cluster = cluster;
}

}  // namespace cicy

namespace cicy {

// ---------------------------------------------------------------------------
// Batched MG solves (used by batch.cu): per-system hierarchies built once, all
// systems solved by k_mg_batch, one cluster per system at a time.
namespace {
__global__ void k_diag_of(int n, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci, const double* __restrict__ v,
                          double* __restrict__ d) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double x = 0;
        for (int k = rp[i]; k < rp[i + 1]; k++)
            if (ci[k] == i) x = v[k];
        d[i] = x;
    }
}
}  // namespace

struct MgBatch {
    std::vector<SolverWork*> works;
    std::vector<DBuf<double>*> diags;
    DBuf<MgArgs> args;
    DBuf<int> queue, slots;
    DBuf<double> stats;
    int count = 0, nclusters = 0, ctas = kMgClusterCtas;  // ctas: CTAs per cluster
    double tol = 0;
    ~MgBatch() {
        for (auto* w : works) delete w;
        for (auto* d : diags) {
            d->release();
            delete d;
        }
        args.release();
        queue.release();
        slots.release();
        stats.release();
    }
};

MgBatch* mg_batch_build(const std::vector<MgBatchInput>& in, double tol, long long iter_factor, cudaStream_t s, int64_t& launches) {
    if (cudaFuncSetAttribute(k_mg_batch, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        throw Fail{CICY_E_DEVICE, "batched multigrid: 16-CTA clusters are not available"};
    }
    MgBatch* B = new MgBatch;
    try {
        B->count = (int)in.size();
        B->tol = tol;
        B->stats.ensure(4 * in.size() + 4);
        auto resident = [](int ctas) {  // clusters of `ctas` CTAs that fit at once
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute attr[1];
            cfg.gridDim = dim3(ctas);
            cfg.blockDim = dim3(kMgClusterThreads);
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = ctas;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int n = 0;
            CICY_CUDA(cudaOccupancyMaxActiveClusters(&n, (void*)k_mg_batch, &cfg));
            return n;
        };
        std::vector<int> rows;
        for (const MgBatchInput& x : in) rows.push_back(x.n);
        int fits[kMgBatchShapes];
        for (int k = 0; k < kMgBatchShapes; k++) fits[k] = resident(kMgBatchCtas[k]);
        const int shape = mg_batch_shape(std::move(rows), fits);
        if (shape < 0) throw Fail{CICY_E_DEVICE, "batched multigrid: no cluster fits"};
        B->ctas = kMgBatchCtas[shape];
        const int nclusters = fits[shape];
        std::vector<MgArgs> host(in.size());
        for (size_t k = 0; k < in.size(); k++) {
            const MgBatchInput& x = in[k];
            auto* w = new SolverWork;
            B->works.push_back(w);
            auto* d = new DBuf<double>;
            B->diags.push_back(d);
            d->ensure(x.n + 1);
            k_diag_of<<<grid_for(x.n), 256, 0, s>>>(x.n, x.rp, x.ci, x.val, d->get());
            launches++;
            SolverSystem ss;
            ss.n = x.n;
            ss.nnz = x.nnz;
            ss.rp = x.rp;
            ss.ci = x.ci;
            ss.val = x.val;
            ss.diag = d->get();
            ss.b = x.b;
            ss.x = x.x;
            build_block_preconditioner(*w, ss, x.nchains, x.cs, x.cl, nullptr, nullptr, false, s, launches);
            build_mg_hierarchy(*w, ss, s, launches);
            MgWork& g = w->mg;
            w->r.ensure(x.n); w->z.ensure(x.n); w->p.ensure(x.n); w->q.ensure(x.n);
            g.z0.ensure(x.n);
            g.wtmp.ensure(x.n);
            w->cta_row.ensure(B->ctas + 1);
            launch_cta_rows(B->ctas, x.n, w->is_start.get(), w->cta_row.get(), s);
            w->part.ensure(4 * B->ctas + 8);
            MgArgs a{};
            a.n = x.n;
            a.rp = x.rp; a.ci = x.ci; a.val = x.val; a.b = x.b; a.x = x.x; a.x0 = x.x0;
            a.r = w->r.get(); a.z0 = g.z0.get(); a.z = w->z.get(); a.w = g.wtmp.get(); a.p = w->p.get(); a.q = w->q.get();
            a.tinv = w->tinv.get(); a.row_off = w->row_off.get(); a.row_base = w->row_base.get(); a.row_m = w->row_m.get();
            a.cta_row = w->cta_row.get();
            a.levels = g.levels;
            a.lv = g.dev_lv.get();
            a.cinv = g.dense ? g.cinv.get() : nullptr;
            a.omega0 = kOmega0;
            a.partA = w->part.get();
            a.partB = w->part.get() + 2 * B->ctas;
            a.stats = B->stats.get() + 4 * k;
            a.bar = nullptr;
            a.spin_limit = kSpinLimit;
            a.err = nullptr;
            a.tol = tol;
            a.max_iter = iter_factor * (long long)x.n;
            a.max_restarts = kMgMaxRestarts;
            a.cap_b = 1;
            host[k] = a;
        }
        // largest first: a cluster that takes a large system last would finish long after the others
        std::stable_sort(host.begin(), host.end(), [](const MgArgs& a, const MgArgs& b) { return a.n > b.n; });
        B->args.ensure(in.size());
        CICY_CUDA(cudaMemcpyAsync(B->args.get(), host.data(), sizeof(MgArgs) * in.size(), cudaMemcpyHostToDevice, s));
        B->queue.ensure(1);
        B->nclusters = std::min(nclusters, B->count);
        B->slots.ensure(B->nclusters + 1);
        CICY_CUDA(cudaStreamSynchronize(s));
        CICY_LAUNCH_CHECK();
    } catch (...) {
        delete B;
        throw;
    }
    return B;
}

void mg_batch_enqueue(MgBatch* B, cudaStream_t s) {
    CICY_CUDA(cudaMemsetAsync(B->queue.get(), 0, sizeof(int), s));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    cfg.gridDim = dim3(B->ctas * B->nclusters);
    cfg.blockDim = dim3(kMgClusterThreads);
    cfg.stream = s;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = B->ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    CICY_CUDA(cudaLaunchKernelEx(&cfg, k_mg_batch, (const MgArgs*)B->args.get(), B->count, B->ctas, B->queue.get(), B->slots.get()));
}

void mg_batch_stats(MgBatch* B, std::vector<double>& stats, cudaStream_t s) {
    stats.resize(4 * (size_t)B->count);
    CICY_CUDA(cudaMemcpyAsync(stats.data(), B->stats.get(), sizeof(double) * 4 * B->count, cudaMemcpyDeviceToHost, s));
    CICY_CUDA(cudaStreamSynchronize(s));
}

int mg_batch_clusters(const MgBatch* B) { return B->nclusters; }

void mg_batch_free(MgBatch* B) { delete B; }

}  // namespace cicy
