// Small dense FP64 R x R algebra: symmetric eigendecomposition (parallel
// cyclic Jacobi, one CTA per matrix) and the symmetric pseudo-inverse built
// on it.  Replaces LAPACKE_dsyev + compute_pinv_square (common.h:405-443,
// sts_cp.hpp:110-176) of the reference.
#include "dense.cuh"

#include <utility>

namespace exafac {

// Round-robin ("circle") pairing of Re = even(R) indices: in round t, pair 0
// is (0, 1 + t mod m) and pair i >= 1 is (1 + (t+i) mod m, 1 + (t-i) mod m),
// m = Re - 1.  Every unordered pair meets once per sweep of Re - 1 rounds.
__device__ __forceinline__ void rr_pair(int t, int i, int m, int& p, int& q) {
    if (i == 0) {
        p = 0;
        q = 1 + (t % m);
    } else {
        p = 1 + ((t + i) % m);
        q = 1 + ((t - i + m * 4) % m);
    }
    if (p > q) {
        int x = p;
        p = q;
        q = x;
    }
}

// Cyclic Jacobi on the symmetric matrix whose upper triangle is A (row-major
// R x R): jacobi_init, then jacobi_sweeps.
// Shared: a[Re*Re] (the working matrix), rot[Re/2] cosines and sines.
// vt (global, Re*Re) holds V^T: vt[i*Re + r] = component r of eigenvector i.
__device__ void jacobi_init(int R, const double* __restrict__ A, double* a, double* vt) {
    const int Re = R + (R & 1);
    for (int e = threadIdx.x; e < Re * Re; e += blockDim.x) {
        int i = e / Re, j = e % Re;
        double v = 0.0;
        if (i < R && j < R) v = (i <= j) ? A[i * R + j] : A[j * R + i];
        a[e] = v;
        vt[e] = (i == j && i < R) ? 1.0 : 0.0;
    }
    __syncthreads();
}

// Rotate unless a_pq is negligible relative to the diagonal (Demmel-Veselic
// criterion, tol = R * eps).  null > 0: diagonals up to it belong to eigenvalues
// that the caller drops; a pair of two such is left alone when a_pq is as small,
// a pair with one when the rotation is below R * eps.
__device__ __forceinline__ bool jacobi_rotates(int R, double apq, double app, double aqq, double null = 0.0) {
    if (fabs(apq) <= null) {
        const double lo = fmin(fabs(app), fabs(aqq)), hi = fmax(fabs(app), fabs(aqq));
        if (lo <= null && (hi <= null || fabs(apq) <= (double)R * 2.220446049250313e-16 * hi)) return false;
    }
    return apq != 0.0 && fabs(apq) > (double)R * 2.220446049250313e-16 * sqrt(fabs(app * aqq));
}

// Sweeps until no pair rotates.  A sweep starts by looking at every pair at
// once, so a matrix that is already diagonal (the end of every call, and the
// usual start of syev_finish_kernel) costs one pass instead of Re - 1 rounds.
__device__ void jacobi_sweeps(int R, double* a, double* vt, double* rc, double* rs, int* flag, double null = 0.0) {
    const int Re = R + (R & 1);
    const int m = Re - 1;
    const int npairs = Re / 2;
    const int tid = threadIdx.x, nt = blockDim.x;
    if (R == 1) return;
    for (int sweep = 0; sweep < 60; sweep++) {
        if (tid == 0) *flag = 0;
        __syncthreads();
        bool any = false;
        for (int e = tid; e < R * R && !any; e += nt) {
            const int i = e / R, j = e % R;
            any = i < j && jacobi_rotates(R, a[i * Re + j], a[i * Re + i], a[j * Re + j], null);
        }
        if (any) *flag = 1;
        __syncthreads();
        if (*flag == 0) break;
        for (int t = 0; t < m; t++) {
            // Rotation angles (Golub & Van Loan, sym.schur2).
            for (int i = tid; i < npairs; i += nt) {
                int p, q;
                rr_pair(t, i, m, p, q);
                double c = 1.0, s = 0.0;
                if (q < R) {
                    double apq = a[p * Re + q];
                    double app = a[p * Re + p], aqq = a[q * Re + q];
                    if (jacobi_rotates(R, apq, app, aqq, null)) {
                        double tau = (aqq - app) / (2.0 * apq);
                        double tt;
                        if (fabs(tau) > 1e150) {
                            tt = 0.5 / tau;
                        } else {
                            tt = (tau >= 0.0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
                        }
                        c = 1.0 / sqrt(1.0 + tt * tt);
                        s = tt * c;
                    }
                }
                rc[i] = c;
                rs[i] = s;
            }
            __syncthreads();
            // B = J^T A: rows p, q.
            for (int e = tid; e < npairs * Re; e += nt) {
                int i = e / Re, col = e % Re;
                double s = rs[i];
                if (s == 0.0) continue;
                double c = rc[i];
                int p, q;
                rr_pair(t, i, m, p, q);
                double ap = a[p * Re + col], aq = a[q * Re + col];
                a[p * Re + col] = c * ap - s * aq;
                a[q * Re + col] = s * ap + c * aq;
            }
            __syncthreads();
            // A' = B J and V' = V J: columns p, q.
            for (int e = tid; e < npairs * Re; e += nt) {
                int i = e / Re, row = e % Re;
                double s = rs[i];
                if (s == 0.0) continue;
                double c = rc[i];
                int p, q;
                rr_pair(t, i, m, p, q);
                double bp = a[row * Re + p], bq = a[row * Re + q];
                a[row * Re + p] = c * bp - s * bq;
                a[row * Re + q] = s * bp + c * bq;
                double vp = vt[p * Re + row], vq = vt[q * Re + row];
                vt[p * Re + row] = c * vp - s * vq;
                vt[q * Re + row] = s * vp + c * vq;
            }
            __syncthreads();
        }
    }
}

// Ascending order of the diagonal: rank[i] = #{j : d_j before d_i}, with
// "before" a strict total order (value, then index; NaNs after every number),
// so the ranks are a permutation of 0..R-1 whatever the values: the order[]
// built from them has no unwritten slot even when a NaN reached the matrix.
__device__ __forceinline__ bool diag_before(double dj, int j, double di, int i) {
    const bool nj = isnan(dj), ni = isnan(di);
    if (nj || ni) return nj == ni ? j < i : ni;
    return dj < di || (dj == di && j < i);
}
__device__ void ascending_ranks(int R, const double* a, int Re, int* rank) {
    for (int i = threadIdx.x; i < R; i += blockDim.x) {
        const double di = a[i * Re + i];
        int r = 0;
        for (int j = 0; j < R; j++) r += diag_before(a[j * Re + j], j, di, i);
        rank[i] = r;
    }
}

// Eigendecomposition / pseudo-inverse of one matrix by the calling CTA.
// Outputs (any may be null):
//   V[u*R + v]    eigenvector v (ascending eigenvalues), lam[v]
//   pinv          sum over lam_v > tol of v v^T / lam_v  (full symmetric)
struct SyevSmem {
    double *a, *rc, *rs;
    int *rank, *order, *flag;
};
__device__ __forceinline__ SyevSmem syev_smem(int R, double* smem) {
    const int Re = R + (R & 1);
    SyevSmem m;
    m.a = smem;
    m.rc = m.a + Re * Re;
    m.rs = m.rc + Re / 2 + 1;
    m.rank = reinterpret_cast<int*>(m.rs + Re / 2 + 1);
    m.order = m.rank + Re;
    m.flag = m.order + Re;
    return m;
}

// The outputs from the diagonalised m.a and the rows of vt.
__device__ void syev_outputs(int R, const SyevSmem& m, const double* vt, double* V, double* lam, double* pinv,
                             double tol) {
    const int Re = R + (R & 1);
    __syncthreads();
    ascending_ranks(R, m.a, Re, m.rank);
    __syncthreads();
    for (int i = threadIdx.x; i < R; i += blockDim.x) m.order[m.rank[i]] = i;
    __syncthreads();
    if (V) {
        for (int e = threadIdx.x; e < R * R; e += blockDim.x) {
            int i = e / R, u = e % R;  // eigenvector i (original slot), component u
            V[u * R + m.rank[i]] = vt[i * Re + u];
        }
    }
    if (lam) {
        for (int i = threadIdx.x; i < R; i += blockDim.x) lam[m.rank[i]] = m.a[i * Re + i];
    }
    if (pinv) {
        // Sum over eigen-pairs in ascending eigenvalue order, as
        // (V L^-1/2)(V L^-1/2)^T accumulates in the reference's dsyrk.
        for (int e = threadIdx.x; e < R * R; e += blockDim.x) {
            int r1 = e / R, r2 = e % R;
            double acc = 0.0;
            for (int k = 0; k < R; k++) {
                int i = m.order[k];
                double l = m.a[i * Re + i];
                if (l > tol) {
                    double s = 1.0 / sqrt(l);
                    acc += (vt[i * Re + r1] * s) * (vt[i * Re + r2] * s);
                }
            }
            pinv[e] = acc;
        }
    }
}

__device__ void syev_block(int R, const double* __restrict__ A, double* V, double* lam, double* pinv, double tol,
                           double* vt, double* smem) {
    const SyevSmem m = syev_smem(R, smem);
    jacobi_init(R, A, m.a, vt);
    // A pseudo-inverse alone: entries up to tol / 2R form a block whose
    // eigenvalues, at most tol / 2, are dropped whatever its basis.  The null
    // block of a singular Gram (a mode shorter than the rank) is rounding that
    // the criterion keeps rotating: 195 ms a call at R = 121, 60 sweeps, now 44.
    jacobi_sweeps(R, m.a, vt, m.rc, m.rs, m.flag, V || lam ? 0.0 : tol / (2.0 * R));
    syev_outputs(R, m, vt, V, lam, pinv, tol);
}

// One CTA per matrix (matrix b at A + b * a_stride).
__global__ void syev_kernel(int R, const double* __restrict__ A, int64_t a_stride, double* V, double* lam,
                            int64_t v_stride, double* pinv, double tol, double* vt_scratch) {
    extern __shared__ double smem[];
    const int Re = R + (R & 1);
    const int b = blockIdx.x;
    syev_block(R, A + b * a_stride, V ? V + b * v_stride : nullptr, lam ? lam + (int64_t)b * R : nullptr,
               pinv ? pinv + (int64_t)b * R * R : nullptr, tol, vt_scratch + (int64_t)b * Re * Re, smem);
}

// ---------------------------------------------------------------------------
// Eigendecomposition of the FP64 form's sampling matrices: an FP32 Jacobi
// start, refined in FP64.
//
// The FP64 Jacobi takes ~10 sweeps of ~6 R^3 FP64 operations on one SM (GB300
// retires ~1.7 of them per clock per SM): 0.85 / 5.1 / 17 ms a call at R = 25 /
// 64 / 100, which was 15 to 52 % of an FP64 STS-CP sweep.  Here
//   1. jacobi32_kernel: the sweeps in FP32 (shared memory, one CTA a matrix);
//   2. kRefineSteps refinement steps of the eigenvector matrix X in FP64
//      (Ogita and Aishima, "Iterative refinement for symmetric eigenvalue
//      decomposition", 2018): with S = X^T A X, G = X^T X, r = I - G,
//      lambda_i = S_ii / G_ii, X <- X + X E, E_ij = (S_ij + lambda_j r_ij) /
//      (lambda_j - lambda_i), or r_ij / 2 on the diagonal and where the
//      quotient is no small rotation (equal eigenvalues).  S is taken
//      symmetric (its upper triangle), which keeps E_ij + E_ji = r_ij to
//      rounding and so X orthonormal.  The error squares per step; the
//      products run on R blocks.  Eigenvalues closer than FP32 resolves
//      beside the largest get a second FP32 Jacobi in the first step, cluster
//      by cluster at the clusters' own scales (refine_first_kernel).  How
//      large a rotation counts as small falls from step to step, and the last
//      step is r / 2 alone: a pair that no step resolves leaves X orthonormal;
//   3. syev_finish_kernel: the FP64 Jacobi sweeps on S with X as the start,
//      so the result meets the same convergence criterion whatever the steps
//      left (a cluster, eigenvalues below FP32's resolution), then the sorted
//      outputs.  X that is not orthonormal to 4 R eps, or a value that is not
//      finite, starts the sweeps from A.
// Measured (GB300, one matrix, launches included), the FP64 sweeps alone ->
// this: Grams of random factors at R = 25 / 64 / 100 0.85 / 5.1 / 17 -> 0.19 /
// 0.52 / 1.6 ms, |A v - lambda v| 5e-15 .. 3e-14 -> 3e-16 |A|.  Clusters: the
// chains of converged factors at R = 25 / 58 0.86 .. 1.2 / 3.9 .. 5.9 -> 0.19 ..
// 0.28 / 0.41 .. 0.95 ms (with one mean for all clusters, rotations up to 2^-5
// in every step and no orthonormalising one X was given up: 1.1 .. 1.4 / 4.3 ..
// 6.4); 1 + 10^-u, u uniform in 0 .. 16, at R = 64 8.2 -> 2.7; half the spectrum
// null at R = 64 37 -> 4.2; I but for rounding at R = 64 0.03 -> 0.21.
// Below kRefineMinRank the FP64 sweeps alone are faster: R = 4 / 5 0.05 / 0.08
// against 0.05 / 0.065 ms.
// ---------------------------------------------------------------------------
constexpr int kRefineMinRank = 5;
constexpr int kRefineSteps = 4;
constexpr double kRefineLimit[kRefineSteps] = {0x1p-5, 0x1p-8, 0x1p-18, 0.0};
constexpr int kJacobi32MaxSweeps = 10;

// Cyclic Jacobi in FP32 on the full symmetric matrix a (Re x Re, shared; two
// buffers of it), v (Re x Re, shared) <- V^T (row i = eigenvector i).  A pair
// rotates while |a_pq| > max(2^-22 sqrt|a_pp a_qq|, floor).  A round's
// rotations act on disjoint pairs, so the two-sided update is independent 2 x
// 2 blocks J_i^T a_ij J_j: a warp per pair i, its lanes along j, then along
// the rows of V^T.  A round is latency and shared memory's bandwidth (0.97 /
// 1.06 / 2.07 us at R = 25 / 64 / 100 with the angles in one warp, a second
// barrier and IEEE divisions; 0.6 / 0.77 / 1.75 us as it is): every
// warp forms all the angles itself, a pair (kPairs of them) per lane, and the
// blocks go from one buffer to the other, so that one barrier remains.  The
// rotations need no more than FP32's approximate quotients (the refinement
// makes the vectors orthonormal).
__device__ __forceinline__ bool jacobi32_rotates(float apq, float app, float aqq, float floor) {
    return fabsf(apq) > floor && apq * apq > 0x1p-44f * fabsf(app * aqq);
}
template <int kPairs>
__device__ void jacobi32_sweeps(int R, float* cur, float* nxt, float* v, float floor, int* flag) {
    const int Re = R + (R & 1), m = Re - 1, np = Re / 2, ld = Re;
    const int tid = threadIdx.x, nt = blockDim.x, w = tid >> 5, nw = nt >> 5, lane = tid & 31;
    for (int e = tid; e < Re * Re; e += nt) v[e] = e / Re == e % Re ? 1.0f : 0.0f;
    __syncthreads();
    for (int sweep = 0; sweep < kJacobi32MaxSweeps && R > 1; sweep++) {
        if (tid == 0) *flag = 0;
        __syncthreads();
        bool any = false;  // a look at every pair: a converged matrix ends here
        for (int i = w; i < R && !any; i += nw)
            for (int j = i + 1 + lane; j < R; j += 32)
                any = any || jacobi32_rotates(cur[i * ld + j], cur[i * ld + i], cur[j * ld + j], floor);
        if (any) *flag = 1;
        __syncthreads();
        if (!*flag) break;
        for (int t = 0; t < m; t++) {
            float c[kPairs], s[kPairs];
            int p[kPairs], q[kPairs];
            bool rot = false;
#pragma unroll
            for (int h = 0; h < kPairs; h++) {
                const int j = lane + 32 * h;
                c[h] = 1.0f;
                s[h] = 0.0f;
                p[h] = q[h] = 0;
                if (j < np) {  // rr_pair without the divisions
                    const int x = t + j, y = t - j;
                    const int u = j == 0 ? 0 : 1 + (x >= m ? x - m : x), z = 1 + (y < 0 ? y + m : y);
                    p[h] = u;  // in this order: consecutive over the lanes (banks)
                    q[h] = z;
                    const float apq = cur[p[h] * ld + q[h]], app = cur[p[h] * ld + p[h]], aqq = cur[q[h] * ld + q[h]];
                    if (max(u, z) < R && jacobi32_rotates(apq, app, aqq, floor)) {
                        const float tau = fmaxf(fminf(__fdividef(0.5f * (aqq - app), apq), 0x1p40f), -0x1p40f);
                        const float k = fmaf(tau, tau, 1.0f);
                        const float tt = copysignf(__fdividef(1.0f, fabsf(tau) + k * rsqrtf(k)), tau);
                        c[h] = rsqrtf(fmaf(tt, tt, 1.0f));
                        s[h] = tt * c[h];
                        rot = true;
                    }
                }
            }
            if (!__any_sync(0xffffffffu, rot)) continue;  // the same in every warp
            for (int i = w; i < np; i += nw) {
                const int from = i & 31;
                const bool hi = kPairs > 1 && i >= 32;
                const float ci = __shfl_sync(0xffffffffu, hi ? c[kPairs - 1] : c[0], from);
                const float si = __shfl_sync(0xffffffffu, hi ? s[kPairs - 1] : s[0], from);
                const int pi = __shfl_sync(0xffffffffu, hi ? p[kPairs - 1] : p[0], from);
                const int qi = __shfl_sync(0xffffffffu, hi ? q[kPairs - 1] : q[0], from);
                const float *rp = cur + pi * ld, *rq = cur + qi * ld;
                float *wp = nxt + pi * ld, *wq = nxt + qi * ld;
#pragma unroll
                for (int h = 0; h < kPairs; h++) {
                    if (lane + 32 * h < np) {
                        const float pp = rp[p[h]], pqv = rp[q[h]], qp = rq[p[h]], qq = rq[q[h]];
                        const float l0 = ci * pp - si * qp, l1 = ci * pqv - si * qq;
                        const float m0 = si * pp + ci * qp, m1 = si * pqv + ci * qq;
                        wp[p[h]] = c[h] * l0 - s[h] * l1;
                        wp[q[h]] = s[h] * l0 + c[h] * l1;
                        wq[p[h]] = c[h] * m0 - s[h] * m1;
                        wq[q[h]] = s[h] * m0 + c[h] * m1;
                    }
                }
                if (si == 0.0f) continue;
                float *vp = v + pi * ld, *vq = v + qi * ld;
#pragma unroll
                for (int h = 0; h < 2 * kPairs; h++) {
                    const int r = lane + 32 * h;
                    if (r < Re) {
                        const float x = vp[r], y = vq[r];
                        vp[r] = ci * x - si * y;
                        vq[r] = si * x + ci * y;
                    }
                }
            }
            __syncthreads();
            float* const done = nxt;
            nxt = cur;
            cur = done;
        }
        __syncthreads();  // flag is read by everyone before the next sweep clears it
    }
    __syncthreads();
}
// a: two buffers, then v, Re x Re floats each (jacobi32_bytes).
__host__ __device__ __forceinline__ size_t jacobi32_bytes(int R) {
    const size_t Re = R + (R & 1);
    return 3 * Re * Re * sizeof(float);
}
__device__ void jacobi32_block(int R, float* a, float* v, float floor, int* flag) {
    const int Re = R + (R & 1);
    if (R <= 64) jacobi32_sweeps<1>(R, a, a + Re * Re, v, floor, flag);
    else jacobi32_sweeps<2>(R, a, a + Re * Re, v, floor, flag);
}

// The power of two that brings mx into [1, 2); 0 when there is none to speak of.
__device__ __forceinline__ double scale_of(double mx) {
    const int ex = ((__double2hiint(mx) >> 20) & 0x7ff) - 1023;
    return (mx > 0.0 && isfinite(mx) && ex > -1000) ? scalbn(1.0, -ex) : 0.0;
}
__device__ double block_sum(double x, double* red) {  // red: 32 doubles, added in warp order
    __syncthreads();
    x = warp_sum(x);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
    __syncthreads();
    x = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); q++) x += red[q];
    return x;
}
__device__ double block_max(double mx, double* red) {
    __syncthreads();
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
    __syncthreads();
    mx = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); q++) mx = fmax(mx, red[q]);
    return mx;
}

__global__ void __launch_bounds__(512) jacobi32_kernel(int R, const double* __restrict__ A, int64_t a_stride,
                                                       double* __restrict__ X, double* __restrict__ As,
                                                       int64_t scratch_stride) {
    extern __shared__ float j32[];
    __shared__ int flag;
    __shared__ double red[32];
    const int Re = R + (R & 1);
    const int tid = threadIdx.x, nt = blockDim.x;
    float* a = j32;
    float* v = a + 2 * Re * Re;
    A += blockIdx.x * a_stride;
    X += blockIdx.x * scratch_stride;
    As += blockIdx.x * scratch_stride;
    // less the mean eigenvalue: a cluster near it keeps FP32's resolution
    double tr = 0.0;
    for (int i = 0; i < R; i++) tr += A[i * R + i];
    const double mu = tr / R;
    double mx = 0.0;
    bool turns = false;
    for (int e = tid; e < R * R; e += nt) {
        const int i = e / R, j = e % R;
        const double x = i <= j ? A[i * R + j] : A[j * R + i];
        turns = turns || (i < j && jacobi_rotates(R, x, A[i * R + i], A[j * R + j]));
        As[e] = x;
        mx = fmax(mx, fabs(i == j ? x - mu : x));
    }
    // (a matrix with no pair to rotate, as of factors with orthogonal columns: X = I)
    const double sc = __syncthreads_or(turns) ? scale_of(block_max(mx, red)) : 0.0;
    for (int e = tid; e < Re * Re; e += nt) {
        const int i = e / Re, j = e % Re;
        double x = 0.0;
        if (i < R && j < R) x = (i <= j ? A[i * R + j] : A[j * R + i]) - (i == j ? mu : 0.0);
        a[e] = (float)(x * sc);
    }
    __syncthreads();
    jacobi32_block(R, a, v, 0x1p-22f, &flag);
    for (int e = tid; e < R * R; e += nt) X[e] = (double)v[(e % R) * Re + e / R];  // column j = eigenvector j
}

// Sum of x[k] y[k * stride], four chains (a dependent FP64 add takes ~64 cycles).
__device__ __forceinline__ double dot4(const double* x, const double* __restrict__ y, int stride, int n) {
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    int k = 0;
    for (; k + 3 < n; k += 4) {
        s0 = fma(x[k], y[(int64_t)k * stride], s0);
        s1 = fma(x[k + 1], y[(int64_t)(k + 1) * stride], s1);
        s2 = fma(x[k + 2], y[(int64_t)(k + 2) * stride], s2);
        s3 = fma(x[k + 3], y[(int64_t)(k + 3) * stride], s3);
    }
    for (; k < n; k++) s0 = fma(x[k], y[(int64_t)k * stride], s0);
    return (s0 + s1) + (s2 + s3);
}

// Row i (blockIdx.x) of S = X^T A X (unless null) and G = X^T X of matrix blockIdx.y.
__global__ void __launch_bounds__(128) refine_forms_kernel(int R, const double* __restrict__ As,
                                                           const double* __restrict__ X, double* __restrict__ S,
                                                           double* __restrict__ G, int64_t scratch_stride) {
    __shared__ double xi[kMaxRank], ti[kMaxRank];
    pdl_wait();
    pdl_trigger();
    const int i = blockIdx.x, j = threadIdx.x;
    const int64_t o = (int64_t)blockIdx.y * scratch_stride;
    if (j < R) xi[j] = X[o + (int64_t)j * R + i];
    __syncthreads();
    if (j < R && S) ti[j] = dot4(xi, As + o + j, R, R);
    __syncthreads();
    if (j < R) {
        if (S) S[o + (int64_t)i * R + j] = dot4(ti, X + o + j, R, R);
        G[o + (int64_t)i * R + j] = dot4(xi, X + o + j, R, R);
    }
}

// (S_ij + lambda_j r_ij, lambda_j - lambda_i) of the upper triangle's S, and
// the larger numerator of (i, j) and (j, i), so that both take the same branch.
__device__ __forceinline__ double3 refine_quotient(int R, const double* S, const double* G, int i, int j) {
    const double li = S[i * R + i] / G[i * R + i], lj = S[j * R + j] / G[j * R + j];
    const double sij = i <= j ? S[i * R + j] : S[j * R + i];
    const double g = G[i * R + j];
    return make_double3(sij - lj * g, lj - li, fmax(fabs(sij - lj * g), fabs(sij - li * g)));
}
// A quotient that is a small rotation (up to `limit`), and one that says
// something: between close eigenvalues (lmax: the largest) a numerator at the
// rounding of S would turn X by noise / gap; those pairs are left to the
// Jacobi sweeps.
__device__ __forceinline__ bool small_rotation(double3 q, double lmax, double limit) {
    return q.z < limit * fabs(q.y) && (q.z > 0x1p-48 * lmax || fabs(q.y) > 0x1p-23 * lmax);
}

// limit 0: the orthonormalising step, E = r / 2 (S is not read).
__global__ void __launch_bounds__(128) refine_e_kernel(int R, double limit, const double* __restrict__ S,
                                                       const double* __restrict__ G, double* __restrict__ E,
                                                       int64_t scratch_stride) {
    pdl_wait();
    pdl_trigger();
    __shared__ double red[32];
    const int i = blockIdx.x, j = threadIdx.x;
    const int64_t o = (int64_t)blockIdx.y * scratch_stride;
    const double lmax = limit > 0.0 ? block_max(j < R ? fabs(S[o + j * R + j]) : 0.0, red) : 0.0;
    if (j >= R) return;
    double e = 0.5 * ((i == j ? 1.0 : 0.0) - G[o + i * R + j]);
    if (i != j && limit > 0.0) {
        const double3 q = refine_quotient(R, S + o, G + o, i, j);
        if (small_rotation(q, lmax, limit)) e = q.x / q.y;
    }
    E[o + i * R + j] = e;
}

// The first step's E, a CTA per matrix.  The pairs whose rotation is not small
// link their indices to clusters; each cluster's block of X^T (A - m I) X = S -
// m G, m the mean of its eigenvalues, is diagonalised by an FP32 Jacobi at its
// own scale (so that clusters anywhere in the spectrum gain FP32's 24 bits in
// their own spread): X <- X (I + E0) V with E0 the small rotations between the
// clusters and r / 2 inside them.
__global__ void __launch_bounds__(512) refine_first_kernel(int R, double limit, const double* __restrict__ S,
                                                           const double* __restrict__ G, double* __restrict__ E,
                                                           int64_t scratch_stride) {
    extern __shared__ float j32[];
    __shared__ int flag;
    __shared__ double red[32];
    __shared__ unsigned near[kMaxRank][kMaxRank / 32];  // the pairs whose rotation is not small
    __shared__ int cluster[kMaxRank];                   // the least index of the cluster
    __shared__ double lam[kMaxRank], mean[kMaxRank];    // mean: by cluster; NaN for a cluster of one
    __shared__ int top[kMaxRank];                       // by cluster: high word of its block's largest entry
    pdl_wait();
    const int Re = R + (R & 1);
    const int tid = threadIdx.x, nt = blockDim.x;
    S += blockIdx.x * scratch_stride;
    G += blockIdx.x * scratch_stride;
    E += blockIdx.x * scratch_stride;
    for (int e = tid; e < kMaxRank * (kMaxRank / 32); e += nt) near[0][e] = 0u;
    const double lmax = block_max(tid < R ? fabs(S[tid * R + tid]) : 0.0, red);  // (its barriers: near is clear)
    bool any = false;
    for (int e = tid; e < R * R; e += nt) {
        const int i = e / R, j = e % R;
        double v = 0.5 * ((i == j ? 1.0 : 0.0) - G[e]);
        if (i != j) {
            const double3 q = refine_quotient(R, S, G, i, j);
            if (small_rotation(q, lmax, limit)) {
                v = q.x / q.y;
            } else if (jacobi_rotates(R, q.z, S[i * R + i], S[j * R + j])) {
                atomicOr(&near[i][j >> 5], 1u << (j & 31));
                any = true;
            }
        }
        E[e] = v;
    }
    if (!__syncthreads_or(any)) return;
    if (tid < R) {
        cluster[tid] = tid;
        top[tid] = 0;
        lam[tid] = S[tid * R + tid] / G[tid * R + tid];
    }
    for (bool moved = true; moved;) {  // the least index along the links
        __syncthreads();
        int c = 0;
        if (tid < R) {
            c = cluster[tid];
            for (int w = 0; w < kMaxRank / 32; w++)
                for (unsigned bits = near[tid][w]; bits; bits &= bits - 1) c = min(c, cluster[32 * w + __ffs(bits) - 1]);
            c = cluster[c];
        }
        __syncthreads();
        moved = tid < R && c != cluster[tid];
        if (moved) cluster[tid] = c;
        moved = __syncthreads_or(moved);
    }
    if (tid < R) {
        double sum = 0.0;
        int n = 0;
        for (int k = tid; k < R; k++) {
            if (cluster[k] != tid) continue;
            sum += lam[k];
            n++;
        }
        mean[tid] = n > 1 ? sum / n : __longlong_as_double(0x7ff8000000000000ll);
    }
    __syncthreads();
    auto block = [&](int i, int j) {  // of one cluster
        const int u = min(i, j) * R + max(i, j);
        return S[u] - mean[cluster[i]] * G[u];
    };
    for (int e = tid; e < R * R; e += nt) {
        const int i = e / R, j = e % R, c = cluster[i];
        if (c != cluster[j]) continue;
        const double x = fabs(block(i, j));
        if (x < 0x1p1000) atomicMax(&top[c], __double2hiint(x));  // (false for the NaN of a single index)
    }
    __syncthreads();
    float* a = j32;
    float* v = a + 2 * Re * Re;
    for (int e = tid; e < Re * Re; e += nt) {
        const int i = e / Re, j = e % Re;
        double x = 0.0;
        if (i < R && j < R && cluster[i] == cluster[j]) {
            const double sc = scale_of(__hiloint2double(top[cluster[i]], 0));
            if (sc > 0.0) x = block(i, j) * sc;
        }
        a[e] = (float)x;
    }
    __syncthreads();
    jacobi32_block(R, a, v, 0x1p-22f, &flag);
    // E = (I + E0) V - I; E0 to FP32 like V, transposed into the Jacobi's buffer
    for (int e = tid; e < R * R; e += nt) {
        const int i = e / R, k = e % R;
        a[k * Re + i] = (float)(cluster[i] == cluster[k] ? 0.5 * ((i == k ? 1.0 : 0.0) - G[e]) : E[e]);
    }
    __syncthreads();
    for (int e = tid; e < R * R; e += nt) {
        const int i = e % R, j = e / R;
        float acc = 0.0f;
        for (int k = 0; k < R; k++) acc = fmaf(a[k * Re + i], v[j * Re + k], acc);
        E[i * R + j] = (double)v[j * Re + i] - (i == j ? 1.0 : 0.0) + (double)acc;
    }
}

// Row c (blockIdx.x) of X + X E.
__global__ void __launch_bounds__(128) refine_update_kernel(int R, const double* __restrict__ X,
                                                            const double* __restrict__ E, double* __restrict__ Xn,
                                                            int64_t scratch_stride) {
    __shared__ double xr[kMaxRank];
    pdl_wait();
    pdl_trigger();
    const int c = blockIdx.x, j = threadIdx.x;
    const int64_t o = (int64_t)blockIdx.y * scratch_stride;
    if (j < R) xr[j] = X[o + (int64_t)c * R + j];
    __syncthreads();
    if (j < R) Xn[o + (int64_t)c * R + j] = xr[j] + dot4(xr, E + o + j, R, R);
}

__global__ void __launch_bounds__(512) syev_finish_kernel(int R, const double* __restrict__ A, int64_t a_stride,
                                                          const double* __restrict__ X, const double* __restrict__ S,
                                                          const double* __restrict__ G, int64_t scratch_stride,
                                                          double* V, double* lam, int64_t v_stride, double* vt) {
    extern __shared__ double smem[];
    __shared__ int bad;
    pdl_wait();
    const int Re = R + (R & 1);
    const int64_t b = blockIdx.x, o = b * scratch_stride;
    const SyevSmem m = syev_smem(R, smem);
    vt += b * Re * Re;
    if (threadIdx.x == 0) bad = 0;
    __syncthreads();
    for (int e = threadIdx.x; e < Re * Re; e += blockDim.x) {
        const int i = e / Re, j = e % Re;
        double s = 0.0, x = 0.0;
        if (i < R && j < R) {
            s = S[o + (i <= j ? i * R + j : j * R + i)];
            x = X[o + (int64_t)j * R + i];
            if (!isfinite(s) || !(fabs(G[o + i * R + j] - (i == j ? 1.0 : 0.0)) < 4.0 * R * 2.220446049250313e-16))
                bad = 1;
        }
        m.a[e] = s;
        vt[i * Re + j] = x;  // row i = eigenvector i
    }
    __syncthreads();
    const bool restart = bad != 0;
    __syncthreads();
    if (restart) jacobi_init(R, A + b * a_stride, m.a, vt);
    jacobi_sweeps(R, m.a, vt, m.rc, m.rs, m.flag);
    syev_outputs(R, m, vt, V + b * v_stride, lam + b * R, nullptr, 0.0);
}

// Symmetric pseudo-inverse, fast path: Cholesky A = L L^T, L^{-1} by
// substitution, A^{-1} = L^{-T} L^{-1}.  A^{-1} equals the thresholded
// pseudo-inverse when every eigenvalue exceeds tol; the path is taken only
// when lambda_min >= 1 / ||A^{-1}||_F > 10 tol (a guaranteed lower bound,
// with margin for rounding).  Otherwise — not positive definite, or possibly
// an eigenvalue near or below tol — the same CTA computes the Jacobi
// pseudo-inverse (compute_pinv_square semantics).
// One Newton step on an (pseudo-)inverse X of A: X <- 2X - X A X, in FP64.
// A pseudo-inverse is a fixed point of the step.  smem: 3 R^2 doubles.
__device__ void newton_refine(int R, const double* __restrict__ A, double* __restrict__ out, double* smem) {
    double* X = smem;
    double* As = smem + R * R;
    double* T = smem + 2 * R * R;
    __syncthreads();
    for (int e = threadIdx.x; e < R * R; e += blockDim.x) {
        X[e] = out[e];
        int i = e / R, j = e % R;
        As[e] = (i <= j) ? A[i * R + j] : A[j * R + i];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < R * R; e += blockDim.x) {  // T = A X
        int i = e / R, j = e % R;
        double acc = 0.0;
        for (int k = 0; k < R; k++) acc = fma(As[i * R + k], X[k * R + j], acc);
        T[e] = acc;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < R * R; e += blockDim.x) {  // out = 2X - X T
        int i = e / R, j = e % R;
        double acc = 0.0;
        for (int k = 0; k < R; k++) acc = fma(X[i * R + k], T[k * R + j], acc);
        out[e] = 2.0 * X[e] - acc;
    }
    __syncthreads();
}

__global__ void spd_pinv_kernel(int R, const double* __restrict__ A, double* __restrict__ out, double tol,
                                double* vt_scratch) {
    extern __shared__ double smem[];
    __shared__ int fail;
    __shared__ double fro;
    __shared__ double fro_w[32];  // per-warp parts, summed in warp order (no atomics: the result repeats)
    double* L = smem;
    double* Li = smem + R * R;
    const int tid = threadIdx.x, nt = blockDim.x;
    for (int e = tid; e < R * R; e += nt) {
        int i = e / R, j = e % R;
        L[e] = (i <= j) ? A[i * R + j] : A[j * R + i];
        Li[e] = 0.0;
    }
    if (tid == 0) {
        fail = 0;
        fro = 0.0;
    }
    __syncthreads();
    for (int k = 0; k < R; k++) {
        if (tid == 0) {
            double d = L[k * R + k];
            if (!(d > 0.0) || !isfinite(d)) fail = 1;
            else L[k * R + k] = sqrt(d);
        }
        __syncthreads();
        if (fail) break;
        const double lkk = L[k * R + k];
        for (int i = k + 1 + tid; i < R; i += nt) L[i * R + k] /= lkk;
        __syncthreads();
        const int m = R - k - 1;
        for (int e = tid; e < m * m; e += nt) {
            int i = k + 1 + e / m, j = k + 1 + e % m;
            if (j <= i) L[i * R + j] -= L[i * R + k] * L[j * R + k];
        }
        __syncthreads();
    }
    if (!fail) {
        for (int c = tid; c < R; c += nt) {
            for (int i = c; i < R; i++) {
                double s = (i == c) ? 1.0 : 0.0;
                for (int t = c; t < i; t++) s -= L[i * R + t] * Li[t * R + c];
                Li[i * R + c] = s / L[i * R + i];
            }
        }
        __syncthreads();
        double part = 0.0;
        for (int e = tid; e < R * R; e += nt) {
            int a = e / R, b = e % R;
            int k0 = a > b ? a : b;
            double acc = 0.0;
            for (int k = k0; k < R; k++) acc = fma(Li[k * R + a], Li[k * R + b], acc);
            out[e] = acc;
            part += acc * acc;
        }
        part = warp_sum(part);
        if ((tid & 31) == 0) fro_w[tid >> 5] = part;
        __syncthreads();
        if (tid == 0) {
            double f = 0.0;
            for (int q = 0; q < (nt + 31) / 32; q++) f += fro_w[q];
            fro = f;
        }
        __syncthreads();
        const double bound = 1.0 / sqrt(fro);
        if (isfinite(fro) && bound > 10.0 * tol) return;
        __syncthreads();
    }
    syev_block(R, A, nullptr, nullptr, out, tol, vt_scratch, smem);
}

// R <= 32: the symmetric sweep operator (Gauss-Jordan with diagonal pivots,
// stable without pivoting on a positive-definite matrix) with the upper
// triangle held in registers, kSmallPinvEpt elements per thread.  Sweeping
// every pivot leaves -A^{-1}.  A non-positive pivot means A is not positive
// definite.  The same acceptance test as the Cholesky path (lambda_min >=
// 1/||A^{-1}||_F > 10 tol) guards the result; otherwise the CTA computes the
// Jacobi pseudo-inverse.
//
// Per pivot, warp 0 forms 1/pivot and the scaled pivot row once (one FP64
// division per pivot, not one per thread: GB300 retires about two FP64
// operations per clock per SM), then every element takes one FMA.
//
// refine == 2 tries pinv_sweep_f32 first (below).  The refinement (refine
// == 1) is the Newton step written as
// X + X (I - A X): the residual I - A X is formed in FP64 (A staged in shared
// memory) and the small correction X (I - A X) in FP32 from FP32 copies of X
// and the residual, which keeps the FP64 pipe to a single R^3 product.
constexpr int kSmallPinvThreads = 128;
constexpr int kSmallPinvMaxR = 32;
constexpr int kSmallPinvEpt = (kSmallPinvMaxR * (kSmallPinvMaxR + 1) / 2 + kSmallPinvThreads - 1) / kSmallPinvThreads;

// The same sweep in FP32 (mode 2: the leverage-score pseudo-inverse of the
// mixed forms, whose scores are formed in FP32 anyway), run by warp 0 with
// the whole matrix in registers.  Lane j holds column j; the rows rotate
// through the registers so that the pivot row is always slot 0 (before pivot
// k, slot s holds row (k + s) mod 32), which keeps every register index
// static in a rolled pivot loop.  The swept matrix stays symmetric, so the
// pivot column's entry for row (k + s) is lane (k + s)'s row-k value, one
// shuffle each; no barrier per pivot.  Rows and lanes >= R hold zeros and
// stay zero.  Accepted when every pivot is positive and the FP32 error bound
// R ||A^{-1}||_F 2^-24 (A has a unit diagonal here, so R bounds ||A||) stays
// below 2^-10; otherwise the caller falls back to the FP64 sweep.  A
// dependent FP64 operation costs ~64 cycles on GB300 against ~4 for FP32, and
// this inverse sits on the step's critical path.  Returns the block-uniform
// accept flag; on acceptance out holds the inverse.
__device__ bool pinv_sweep_f32(int R, const double* __restrict__ A, double* __restrict__ out) {
    // Loads, conversions and stores run as rolled loops over the whole block:
    // a single warp's straight-line code is fetched once and pays the
    // instruction-fetch latency per line.
    __shared__ float Af[32][33];
    __shared__ int accepted;
    const int tid = threadIdx.x;
    for (int e = tid; e < 32 * 32; e += blockDim.x) {
        const int i = e >> 5, c = e & 31;
        Af[i][c] = (i < R && c < R) ? narrow_f64(A[i * R + c]) : 0.0f;
    }
    __syncthreads();
    if (tid < 32) {
        const int j = tid;
        const unsigned full = 0xffffffffu;
        float col[32];
#pragma unroll
        for (int s = 0; s < 32; s++) col[s] = Af[s][j];
        bool ok = true;
#pragma unroll 1
        for (int k = 0; k < R; k++) {
            const float akj = col[0];                     // A[k][j]
            const float piv = __shfl_sync(full, akj, k);  // A[k][k], the same in every lane
            if (!(piv > 0.0f) || !isfinite(piv)) {
                ok = false;
                break;
            }
            const float p = 1.0f / piv;
            const float akjp = akj * p;
            float nxt[32];
#pragma unroll
            for (int s = 1; s < 32; s++) {
                const float aik = __shfl_sync(full, akj, (k + s) & 31);  // A[k + s][k]
                nxt[s - 1] = (j == k) ? aik * p : fmaf(-aik, akjp, col[s]);
            }
            nxt[31] = (j == k) ? -p : akjp;  // row k moves to the last slot
#pragma unroll
            for (int s = 0; s < 32; s++) col[s] = nxt[s];
        }
        float fro = 0.0f;
#pragma unroll
        for (int s = 0; s < 32; s++) fro = fmaf(col[s], col[s], fro);
        fro = warp_sum(fro);
        ok = ok && isfinite(fro) && (float)R * sqrtf(fro) <= 0x1.0p14f;  // R ||X||_F 2^-24 <= 2^-10
        __syncwarp();
#pragma unroll
        for (int s = 0; s < 32; s++) Af[(R + s) & 31][j] = -col[s];  // after R pivots slot s holds row (R + s) mod 32
        if (j == 0) accepted = ok;
    }
    __syncthreads();
    if (!accepted) return false;
    for (int e = tid; e < R * R; e += blockDim.x) out[e] = widen_f32(Af[e / R][e % R]);
    return true;
}

__device__ void pinv_small_block(int R, const double* __restrict__ A, double* __restrict__ out, double tol,
                                 double* vt_scratch, int refine) {
    extern __shared__ double smem[];  // Jacobi fallback; in the accepted path A, X and E staged for refinement
    __shared__ double rowbuf[2][kSmallPinvMaxR];  // pivot row k (unscaled), ping-pong
    __shared__ double rp[kSmallPinvMaxR];         // pivot row k times 1/pivot
    __shared__ double pinv_k;                     // 1/pivot
    __shared__ int bad;
    __shared__ double Xs[kSmallPinvMaxR][kSmallPinvMaxR + 1];
    __shared__ double fro;
    __shared__ double fro_w[kSmallPinvThreads / 32];  // per-warp parts, summed in warp order
    if (refine == 2 && pinv_sweep_f32(R, A, out)) return;
    const int tid = threadIdx.x;
    const int P = R * (R + 1) / 2;
    int ii[kSmallPinvEpt], jj[kSmallPinvEpt];
    double a[kSmallPinvEpt];
#pragma unroll
    for (int m = 0; m < kSmallPinvEpt; m++) {
        const int e = tid + kSmallPinvThreads * m;
        int i = 0, base = 0;
        while (i < R - 1 && e >= base + (R - i)) {
            base += R - i;
            i++;
        }
        ii[m] = (e < P) ? i : -1;
        jj[m] = (e < P) ? i + (e - base) : -1;
        a[m] = (e < P) ? A[i * R + jj[m]] : 0.0;
    }
    if (tid < R) rowbuf[0][tid] = A[tid];
    if (tid == 0) {
        fro = 0.0;
        bad = 0;
    }
    __syncthreads();
    bool ok = true;
    for (int k = 0; k < R; k++) {
        const double* r = rowbuf[k & 1];
        double* nr = rowbuf[(k + 1) & 1];
        if (tid < 32) {
            const double piv = r[k];
            if (!(piv > 0.0) || !isfinite(piv)) {
                if (tid == 0) bad = 1;
            } else {
                const double p = 1.0 / piv;
                if (tid < R) rp[tid] = r[tid] * p;
                if (tid == 0) pinv_k = p;
            }
        }
        __syncthreads();
        if (bad) {  // uniform
            ok = false;
            break;
        }
        const double p = pinv_k;
#pragma unroll
        for (int m = 0; m < kSmallPinvEpt; m++) {
            const int i = ii[m], j = jj[m];
            if (i < 0) continue;
            double v;
            if (i != k && j != k) v = fma(-rp[i], r[j], a[m]);
            else if (i == k && j == k) v = -p;
            else v = rp[i == k ? j : i];
            a[m] = v;
            if (i == k + 1) nr[j] = v;
            else if (j == k + 1) nr[i] = v;
        }
        __syncthreads();
    }
    if (ok) {
        double part = 0.0;
#pragma unroll
        for (int m = 0; m < kSmallPinvEpt; m++) {
            if (ii[m] < 0) continue;
            const double x = -a[m];
            a[m] = x;
            part += (ii[m] == jj[m] ? 1.0 : 2.0) * x * x;
            Xs[ii[m]][jj[m]] = x;
            Xs[jj[m]][ii[m]] = x;
        }
        part = warp_sum(part);
        if ((tid & 31) == 0) fro_w[tid >> 5] = part;
        __syncthreads();
        if (tid == 0) {
            double f = 0.0;
            for (int q = 0; q < kSmallPinvThreads / 32; q++) f += fro_w[q];
            fro = f;
        }
        __syncthreads();
        ok = isfinite(fro) && 1.0 / sqrt(fro) > 10.0 * tol;
    }
    if (ok) {
        if (refine != 1) {
            for (int e = tid; e < R * R; e += kSmallPinvThreads) out[e] = Xs[e / R][e % R];
            return;
        }
        double* As = smem;                                        // R x R
        float* Xf = reinterpret_cast<float*>(smem + R * R);       // R x (R + 1)
        float* Ef = Xf + R * (R + 1);                             // R x (R + 1)
        for (int e = tid; e < R * R; e += kSmallPinvThreads) {
            const int i = e / R, j = e % R;
            As[e] = A[(i <= j) ? i * R + j : j * R + i];
            Xf[i * (R + 1) + j] = narrow_f64(Xs[i][j]);
        }
        __syncthreads();
        for (int e = tid; e < R * R; e += kSmallPinvThreads) {  // E = I - A X
            const int i = e / R, j = e % R;
            double acc = (i == j) ? 1.0 : 0.0;
            for (int t = 0; t < R; t++) acc = fma(-As[i * R + t], Xs[t][j], acc);
            Ef[i * (R + 1) + j] = narrow_f64(acc);
        }
        __syncthreads();
        for (int e = tid; e < R * R; e += kSmallPinvThreads) {  // out = X + X E
            const int i = e / R, j = e % R;
            float c = 0.0f;
            for (int t = 0; t < R; t++) c = fmaf(Xf[i * (R + 1) + t], Ef[t * (R + 1) + j], c);
            out[e] = Xs[i][j] + widen_f32(c);
        }
        return;
    }
    __syncthreads();
    syev_block(R, A, nullptr, nullptr, out, tol, vt_scratch, smem);
    if (refine == 1) newton_refine(R, A, out, smem);
}

__global__ void __launch_bounds__(kSmallPinvThreads)
    spd_pinv_small_kernel(int R, const double* __restrict__ A, double* __restrict__ out, double tol,
                          double* vt_scratch, int refine) {
    pinv_small_block(R, A, out, tol, vt_scratch, refine);
}

// The mixed forms' normalisation head in one block: column norms sigma_c =
// sqrt(G_cc) of the factor Gram (DistMat1D::renormalize_columns,
// distmat.hpp:85-138), the normalised Gram ngram = G_ab / (sigma_a sigma_b)
// (as products with 1 / sigma: the leverage inverse is an FP32 quantity),
// the degenerate flag, then the leverage pseudo-inverse of ngram (FP32 sweep
// first).
__global__ void __launch_bounds__(kSmallPinvThreads)
    sigma_pinv_kernel(int R, const double* __restrict__ ugram, double* __restrict__ sigma,
                      double* __restrict__ ngram, int* __restrict__ degenerate, double* __restrict__ out, double tol,
                      double* vt_scratch) {
    __shared__ double rinv[kSmallPinvMaxR];
    __shared__ int deg;
    pdl_wait();
    pdl_trigger();
    if (threadIdx.x == 0) deg = 0;
    __syncthreads();
    for (int c = threadIdx.x; c < R; c += blockDim.x) {
        const double v = sqrt(ugram[c * R + c]);
        sigma[c] = v;
        rinv[c] = 1.0 / v;
        if (!(v > 0.0)) deg = 1;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < R * R; e += blockDim.x) ngram[e] = ugram[e] * rinv[e / R] * rinv[e % R];
    if (threadIdx.x == 0) *degenerate = deg;
    __syncthreads();  // the block's writes of ngram are visible to it
    pinv_small_block(R, ngram, out, tol, vt_scratch, 2);
}

// Larger ranks (R > 92, where three full R x R matrices pass the shared
// memory cap): the same Cholesky inverse with L and L^{-1} held as packed
// lower triangles ((i, j), j <= i, at i (i + 1) / 2 + j; two times 66 KB at
// R = 128), the same acceptance test and Jacobi fallback; the Newton step,
// when asked for, runs in global scratch (2 R^2 doubles of vt_scratch: the
// sessions' scratch holds (N + 1) R^2).
__device__ __forceinline__ int tri(int i, int j) { return i * (i + 1) / 2 + j; }

// a / b from y ~ 1 / b: the quotient's exact residual, multiplied back
// (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990): the correctly rounded a / b when y is the
// rounded reciprocal, and for a y within two ulps of it unless a / b lies
// within 2^-49 ulp of a midpoint.  Three dependent FP64 operations (~64 cycles
// each) where the division itself takes some 700 cycles.
__device__ __forceinline__ double div_by(double a, double b, double y) {
    const double q = a * y;
    return fma(fma(-q, b, a), y, q);
}

// Sums with four independent FP64 accumulators (a dependent FP64 operation
// takes ~64 cycles on GB300, so one chain of R FMAs is latency-bound).
// sub_dot: s0 - sum_{t in [t0, t1)} L(i, t) Li(t, c); gram_dot: sum_{k in
// [k0, R)} Li(k, a) Li(k, b); both over packed lower triangles.
__device__ __forceinline__ double sub_dot(const double* L, const double* Li, int i, int c, int t0, int t1,
                                          double s0) {
    double s1 = 0.0, s2 = 0.0, s3 = 0.0;
    int t = t0;
    for (; t + 3 < t1; t += 4) {
        s0 -= L[tri(i, t)] * Li[tri(t, c)];
        s1 -= L[tri(i, t + 1)] * Li[tri(t + 1, c)];
        s2 -= L[tri(i, t + 2)] * Li[tri(t + 2, c)];
        s3 -= L[tri(i, t + 3)] * Li[tri(t + 3, c)];
    }
    for (; t < t1; t++) s0 -= L[tri(i, t)] * Li[tri(t, c)];
    return (s0 + s1) + (s2 + s3);
}
__device__ __forceinline__ double gram_dot(const double* Li, int a, int b, int k0, int R) {
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    int k = k0;
    for (; k + 3 < R; k += 4) {
        s0 = fma(Li[tri(k, a)], Li[tri(k, b)], s0);
        s1 = fma(Li[tri(k + 1, a)], Li[tri(k + 1, b)], s1);
        s2 = fma(Li[tri(k + 2, a)], Li[tri(k + 2, b)], s2);
        s3 = fma(Li[tri(k + 3, a)], Li[tri(k + 3, b)], s3);
    }
    for (; k < R; k++) s0 = fma(Li[tri(k, a)], Li[tri(k, b)], s0);
    return (s0 + s1) + (s2 + s3);
}

__global__ void spd_pinv_packed_kernel(int R, const double* __restrict__ A, double* __restrict__ out, double tol,
                                       double* vt_scratch) {
    extern __shared__ double smem[];
    __shared__ int fail;
    __shared__ double fro_w[32];  // per-warp parts, summed in warp order
    const int P = R * (R + 1) / 2;
    double* L = smem;
    double* Li = smem + P;
    const int tid = threadIdx.x, nt = blockDim.x;
    for (int i = tid; i < R; i += nt)
        for (int j = 0; j <= i; j++) {
            L[tri(i, j)] = A[j * R + i];  // upper triangle of A
            Li[tri(i, j)] = 0.0;
        }
    if (tid == 0) fail = 0;
    __syncthreads();
    for (int k = 0; k < R; k++) {
        if (tid == 0) {
            const double d = L[tri(k, k)];
            if (!(d > 0.0) || !isfinite(d)) fail = 1;
            else L[tri(k, k)] = sqrt(d);
        }
        __syncthreads();
        if (fail) break;
        const double lkk = L[tri(k, k)];
        for (int i = k + 1 + tid; i < R; i += nt) L[tri(i, k)] /= lkk;
        __syncthreads();
        {  // the trailing lower triangle: a warp per row, its lanes along the row
            const int wid = tid >> 5, lane = tid & 31, nw = nt >> 5;
            for (int i = k + 1 + wid; i < R; i += nw) {
                const double lik = L[tri(i, k)];
                double* row = L + tri(i, 0);
                for (int j = k + 1 + lane; j <= i; j += 32) row[j] -= lik * L[tri(j, k)];
            }
        }
        __syncthreads();
    }
    if (!fail) {
        for (int c = tid; c < R; c += nt) {
            for (int i = c; i < R; i++) {
                const double sacc = sub_dot(L, Li, i, c, c, i, (i == c) ? 1.0 : 0.0);
                Li[tri(i, c)] = sacc / L[tri(i, i)];
            }
        }
        __syncthreads();
        double part = 0.0;
        for (int e = tid; e < R * R; e += nt) {  // (a, b), a <= b, computed once and mirrored
            const int a = e / R, b = e % R;
            if (a > b) continue;
            const double acc = gram_dot(Li, a, b, b, R);
            out[a * R + b] = acc;
            out[b * R + a] = acc;
            part += (a == b ? 1.0 : 2.0) * (acc * acc);
        }
        part = warp_sum(part);
        if ((tid & 31) == 0) fro_w[tid >> 5] = part;
        __syncthreads();
        double fro = 0.0;
        for (int q = 0; q < (nt + 31) / 32; q++) fro += fro_w[q];
        const double bound = 1.0 / sqrt(fro);
        if (isfinite(fro) && bound > 10.0 * tol) return;  // the same in every thread
        __syncthreads();
    }
    syev_block(R, A, nullptr, nullptr, out, tol, vt_scratch, smem);
}

// ---------------------------------------------------------------------------
// The Cholesky inverse of one matrix over many blocks (32 < R <= 128), spread
// where its operations are independent:
//   chol_factor_kernel   one CTA: L
//   chol_columns_kernel  a block per column of L^{-1}, its rows' sums in the
//                        threads, one finished row per step
//   chol_gram_kernel     a block per row of L^{-T} L^{-1}
// then the acceptance test with the Jacobi fallback in one CTA, and the Newton
// step a block per row.  On one SM the FP64 pipe's ~1.8 operations per clock
// and the ~64 cycles of each dependent one made them 0.13 / 0.25 / 0.87 ms at
// R = 45 / 64 / 128; split, the factor takes 0.047 / 0.061 /
// 0.33 ms (twice that beside other FP64 kernels on its SM), the columns 0.013 /
// 0.027 / 0.052 and the products and the test 0.013 each.  kFour: L^{-1} and
// the products summed in four chains (sub_dot, gram_dot), as the packed
// kernels do.  At R <= 32 the small kernels' one launch is the shorter.
// ---------------------------------------------------------------------------
struct CholScratch {
    double *Lp, *Li, *T, *fro;
    int* rank;
};
__host__ __device__ inline CholScratch chol_scratch(double* p, int R) {
    CholScratch c;
    c.Lp = p;
    c.Li = c.Lp + R * (R + 1) / 2;
    c.T = c.Li + R * R;
    c.fro = c.T + R * R;
    c.rank = reinterpret_cast<int*>(c.fro + R);
    return c;
}
size_t chol_scratch_doubles(int R) { return (size_t)R * (R + 1) / 2 + 2 * (size_t)R * R + R + 8; }

constexpr int kFactorThreads = 512;

// 1 / d of a positive normal d: an FP32 reciprocal y of its mantissa (|e| <=
// 2^-22, e = 1 - m y) and one step of the third-order iteration y (1 + e +
// e^2) (Householder), three dependent FP64 operations of ~64 cycles; the
// error is e^3 and the last rounding.
__device__ __forceinline__ double pivot_reciprocal(double d) {
    const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
    const int ex = (int)((hi >> 20) & 0x7ff);
    if (ex < 3 || ex > 2040) return 1.0 / d;  // (a pivot that is not positive and finite stops the caller)
    const double m = __hiloint2double((int)((hi & 0xfffffu) | 0x3ff00000u), (int)lo);
    const float y0 = __fdividef(1.0f, __uint_as_float(0x3f800000u | ((hi & 0xfffffu) << 3) | (lo >> 29)));
    const unsigned yb = __float_as_uint(y0);  // widened in integers
    const double y = __hiloint2double((int)((yb >> 3) + (896u << 20)), (int)(yb << 29));
    const double e = fma(-m, y, 1.0);
    const double r = fma(y, fma(e, e, e), y);
    return __hiloint2double(__double2hiint(r) - ((ex - 1023) << 20), __double2loint(r));
}

// L by columns, kTpc threads per column (row i of column j: thread i % kTpc),
// every element in a register of its owner.  A step takes one barrier: the
// pivot column's owners publish it unscaled, its diagonal's owner the pivot's
// reciprocal, and the owners of the later columns take v_ij -= v_ik (v_jk /
// d_k); the square roots and the division of the columns by them follow for
// all columns at once.  With the root, its reciprocal and the division inside
// the step it took 75 / 106 / 332 us at R = 45 / 64 / 128 (now 47 / 61 / 330: a
// warp retires one FP64 instruction per 64 clocks and an SM one per 19, so at R
// > 64 the updates themselves are the bound).
template <int kTpc, int kSlots>
__global__ void __launch_bounds__(kFactorThreads) chol_factor_kernel(int R, const double* __restrict__ A,
                                                                     double* __restrict__ scr) {
    __shared__ double colv[2][kMaxRank];  // the pivot column, ping-pong
    __shared__ double rpiv[2];            // its pivot's reciprocal
    for (int i = threadIdx.x; i < 2 * kMaxRank; i += kFactorThreads) colv[0][i] = 0.0;
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    const CholScratch c = chol_scratch(scr, R);
    const int j = threadIdx.x / kTpc, g = threadIdx.x % kTpc;
    double v[kSlots];
#pragma unroll
    for (int m = 0; m < kSlots; m++) {
        const int i = kTpc * m + g;
        v[m] = j < R && i >= j && i < R ? A[j * R + i] : 0.0;  // upper triangle of A
    }
    const int m0 = (int)((threadIdx.x & ~31u) / kTpc) / kTpc, m1 = (R + kTpc - 1) / kTpc;  // the warp's live slots
    const bool diag = j < R && g == j % kTpc;
    double dj = diag ? A[j * R + j] : 0.0;  // the diagonal element, ahead of its slot
    auto publish = [&]() {
#pragma unroll
        for (int m = 0; m < kSlots; m++) {
            const int i = kTpc * m + g;
            if (i >= j && i < R) colv[j & 1][i] = v[m];
        }
    };
    if (j == 0) {
        if (diag) rpiv[0] = pivot_reciprocal(dj);
        publish();
    }
    int rank = R;
    for (int k = 0; k < R; k++) {
        const double* col = colv[k & 1];
        __syncthreads();
        const long long bits = __double_as_longlong(col[k]);
        if (!(bits > 0 && bits < 0x7ff0000000000000ll)) {  // not a positive finite number: the same in every thread
            rank = k;
            break;
        }
        if (j > k && j < R) {
            const double cj = col[j], t = cj * rpiv[k & 1];
            if (diag) {
                dj = fma(-cj, t, dj);
                if (j == k + 1) rpiv[j & 1] = pivot_reciprocal(dj);
            }
            // rows in groups of four slots from the warp's first column's on (the
            // others' are no part of L: col's slots are finite or unused)
#pragma unroll
            for (int q = 0; q < kSlots; q += 4) {
                if (q + 3 >= m0 && q < m1) {
                    double x[4];
#pragma unroll
                    for (int h = 0; h < 4; h++) x[h] = col[kTpc * (q + h) + g];
#pragma unroll
                    for (int h = 0; h < 4; h++) v[q + h] = fma(-x[h], t, v[q + h]);
                }
            }
            if (j == k + 1) publish();
        }
    }
    __syncthreads();
    double* pivots = colv[0];
    if (diag) pivots[j] = dj;
    __syncthreads();
    if (j < R) {
        const double root = sqrt(pivots[j]), y = 1.0 / root;
#pragma unroll
        for (int m = 0; m < kSlots; m++) {
            const int i = kTpc * m + g;
            if (i >= j && i < R) c.Lp[tri(i, j)] = i == j ? root : div_by(v[m], root, y);
        }
    }
    if (threadIdx.x == 0) *c.rank = rank;
}

template <bool kFour>
__global__ void __launch_bounds__(kMaxRank) chol_columns_kernel(int R, double* __restrict__ scr) {
    __shared__ double val[2];
    pdl_wait();
    pdl_trigger();
    const CholScratch s = chol_scratch(scr, R);
    if (*s.rank != R) return;
    const int c = blockIdx.x, i = threadIdx.x;
    double a0 = i == c ? 1.0 : 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    const bool row = i < R && i >= c;
    const double lii = row ? s.Lp[tri(i, i)] : 1.0, yii = 1.0 / lii;
    const int four = (i - c) & ~3;  // terms in whole groups of four
    double next = row && i > c ? s.Lp[tri(i, c)] : 0.0;  // L(i, t), one step ahead
    if (i < R && i < c) s.Li[i * R + c] = 0.0;
    for (int t = c; t < R; t++) {
        if (i == t) {
            const double x = div_by(kFour ? (a0 + a1) + (a2 + a3) : a0, lii, yii);
            val[t & 1] = x;
            s.Li[t * R + c] = x;
        }
        const double l = next;
        if (row && i > t + 1) next = s.Lp[tri(i, t + 1)];
        __syncthreads();
        if (row && i > t) {
            const double x = val[t & 1];
            const int q = kFour && t - c < four ? (t - c) & 3 : 0;
            if (q == 0) a0 -= l * x;
            else if (q == 1) a1 -= l * x;
            else if (q == 2) a2 -= l * x;
            else a3 -= l * x;
        }
    }
}

template <bool kFour>
__global__ void __launch_bounds__(kMaxRank) chol_gram_kernel(int R, double* __restrict__ scr, double* __restrict__ out) {
    __shared__ double la[kMaxRank];  // column a of L^{-1}
    __shared__ double red[4];
    pdl_wait();
    pdl_trigger();
    const CholScratch s = chol_scratch(scr, R);
    if (*s.rank != R) return;
    const int a = blockIdx.x, b = threadIdx.x;
    if (b < R) la[b] = b >= a ? s.Li[b * R + a] : 0.0;
    __syncthreads();
    double part = 0.0;
    if (b >= a && b < R) {
        double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
        int k = b;
        if (kFour) {
            for (; k + 3 < R; k += 4) {
                s0 = fma(la[k], s.Li[k * R + b], s0);
                s1 = fma(la[k + 1], s.Li[(k + 1) * R + b], s1);
                s2 = fma(la[k + 2], s.Li[(k + 2) * R + b], s2);
                s3 = fma(la[k + 3], s.Li[(k + 3) * R + b], s3);
            }
        }
        for (; k < R; k++) s0 = fma(la[k], s.Li[k * R + b], s0);
        const double acc = kFour ? (s0 + s1) + (s2 + s3) : s0;
        out[a * R + b] = acc;
        out[b * R + a] = acc;
        part = (a == b ? 1.0 : 2.0) * (acc * acc);
    }
    part = warp_sum(part);
    if ((b & 31) == 0) red[b >> 5] = part;
    __syncthreads();
    if (b == 0) s.fro[a] = (red[0] + red[1]) + (red[2] + red[3]);
}

// 1 / ||A^{-1}||_F > 10 tol, a lower bound of the smallest eigenvalue (every
// thread the same); false when the factorisation stopped.
__device__ bool chol_accepted(int R, const CholScratch& s, double tol) {
    if (*s.rank != R) return false;
    double fro = 0.0;
    for (int a = 0; a < R; a++) fro += s.fro[a];
    return isfinite(fro) && 1.0 / sqrt(fro) > 10.0 * tol;
}

// The pseudo-inverse's fallback: one CTA, which returns at once when the
// Cholesky inverse stands.
__global__ void __launch_bounds__(512) chol_accept_kernel(int R, const double* __restrict__ A, double* __restrict__ out,
                                                          double tol, double* __restrict__ scr, double* vt) {
    extern __shared__ double smem[];
    __shared__ int stands;
    pdl_wait();
    const CholScratch s = chol_scratch(scr, R);
    if (threadIdx.x < 32) {
        const bool yes = chol_accepted(R, s, tol);
        if (threadIdx.x == 0) stands = yes;
    }
    __syncthreads();
    if (stands) return;
    syev_block(R, A, nullptr, nullptr, out, tol, vt, smem);
}

// newton_refine over R blocks: T = A X, then X = 2X - X T.
__global__ void __launch_bounds__(kMaxRank) newton_ax_kernel(int R, const double* __restrict__ A,
                                                             const double* __restrict__ X, double* __restrict__ scr) {
    __shared__ double arow[kMaxRank];
    pdl_wait();
    const CholScratch s = chol_scratch(scr, R);
    const int i = blockIdx.x, j = threadIdx.x;
    if (j < R) arow[j] = i <= j ? A[i * R + j] : A[j * R + i];
    __syncthreads();
    if (j >= R) return;
    double acc = 0.0;
    for (int k = 0; k < R; k++) acc = fma(arow[k], X[k * R + j], acc);
    s.T[i * R + j] = acc;
}
__global__ void __launch_bounds__(kMaxRank) newton_out_kernel(int R, double* __restrict__ X, double* __restrict__ scr) {
    __shared__ double xrow[kMaxRank];
    pdl_wait();
    const CholScratch s = chol_scratch(scr, R);
    const int i = blockIdx.x, j = threadIdx.x;
    if (j < R) xrow[j] = X[i * R + j];
    __syncthreads();
    if (j >= R) return;
    double acc = 0.0;
    for (int k = 0; k < R; k++) acc = fma(xrow[k], s.T[k * R + j], acc);
    X[i * R + j] = 2.0 * xrow[j] - acc;
}

// The Newton step X <- X + X (I - A X) (= 2X - X A X, the fixed point a
// pseudo-inverse) for the packed path, spread over R blocks of one row each
// in FP64: T = I - A X (A's upper triangle read), then X += X T.  On one SM
// the two R^3 products took ~1.2 ms at R = 128 (GB300 retires ~1.6 FP64
// FMA per clock per SM); this form runs them on R SMs.  T: R^2 doubles.
__global__ void newton_residual_kernel(int R, const double* __restrict__ A, const double* __restrict__ X,
                                       double* __restrict__ T) {
    __shared__ double arow[kMaxRank];
    const int i = blockIdx.x;
    for (int k = threadIdx.x; k < R; k += blockDim.x) arow[k] = i <= k ? A[i * R + k] : A[k * R + i];
    __syncthreads();
    for (int j = threadIdx.x; j < R; j += blockDim.x) {
        double acc = 0.0;
        for (int k = 0; k < R; k++) acc = fma(arow[k], X[k * R + j], acc);
        T[i * R + j] = (i == j ? 1.0 : 0.0) - acc;
    }
}
__global__ void newton_update_kernel(int R, const double* __restrict__ T, double* __restrict__ X) {
    __shared__ double xrow[kMaxRank];
    const int i = blockIdx.x;
    for (int k = threadIdx.x; k < R; k += blockDim.x) xrow[k] = X[i * R + k];
    __syncthreads();
    for (int j = threadIdx.x; j < R; j += blockDim.x) {
        double acc = 0.0;
        for (int k = 0; k < R; k++) acc = fma(xrow[k], T[k * R + j], acc);
        X[i * R + j] = xrow[j] + acc;
    }
}

// Shared memory of the one-CTA Cholesky path (L, L^{-1}, and at R <= 32 the
// Newton step's third matrix).  The path in full matrices is used when three
// of them fit under kPinvSmemCap (R <= 92); larger ranks take the packed kernel.
static size_t chol_smem_bytes(int R) { return sizeof(double) * 3 * (size_t)R * R; }
static size_t chol_packed_smem_bytes(int R) { return sizeof(double) * 2 * (size_t)(R * (R + 1) / 2); }
constexpr size_t kPinvSmemCap = 200 * 1024;

// L, L^{-1} (scr) and out = A^{-1} where the factorisation goes through.
static int launch_chol_inverse(int R, const double* A, double* out, bool four, double* scr, cudaStream_t st) {
    auto factor = R <= 64 ? chol_factor_kernel<8, 8> : chol_factor_kernel<4, 32>;
    factor<<<1, kFactorThreads, 0, st>>>(R, A, scr);
    EXAFAC_CUDA_TRY(launch_dependent(four ? chol_columns_kernel<true> : chol_columns_kernel<false>, R, kMaxRank, 0, st, R,
                                     scr));
    EXAFAC_CUDA_TRY(launch_dependent(four ? chol_gram_kernel<true> : chol_gram_kernel<false>, R, kMaxRank, 0, st, R, scr,
                                     out));
    add_launches(3);
    return EXAFAC_OK;
}

// scr (chol_scratch_doubles(R)): the split kernels; null: one CTA.
static int launch_pinv_impl(int R, const double* A, double* out, double tol, double* vt_scratch, int refine,
                            cudaStream_t stream, double* scr = nullptr) {
    if (R > kSmallPinvMaxR && scr) {
        const bool four = chol_smem_bytes(R) > kPinvSmemCap;
        EXAFAC_TRY(launch_chol_inverse(R, A, out, four, scr, stream));
        const size_t smem = syev_smem_bytes(R);
        if (smem > 48 * 1024)
            EXAFAC_CUDA_TRY(allow_smem(chol_accept_kernel));
        EXAFAC_CUDA_TRY(launch_dependent(chol_accept_kernel, 1, 512, smem, stream, R, A, out, tol, scr, vt_scratch));
        count_launch();
        if (refine && four) {
            newton_residual_kernel<<<R, 128, 0, stream>>>(R, A, out, chol_scratch(scr, R).T);
            newton_update_kernel<<<R, 128, 0, stream>>>(R, chol_scratch(scr, R).T, out);
            add_launches(2);
        } else if (refine) {
            EXAFAC_CUDA_TRY(launch_dependent(newton_ax_kernel, R, kMaxRank, 0, stream, R, A, (const double*)out, scr));
            EXAFAC_CUDA_TRY(launch_dependent(newton_out_kernel, R, kMaxRank, 0, stream, R, out, scr));
            add_launches(2);
        }
        EXAFAC_CHECK_LAUNCH();
        return EXAFAC_OK;
    }
    if (R <= kSmallPinvMaxR) {
        const size_t smem = std::max(syev_smem_bytes(R), chol_smem_bytes(R));
        spd_pinv_small_kernel<<<1, kSmallPinvThreads, smem, stream>>>(R, A, out, tol, vt_scratch, refine);
        count_launch();
        EXAFAC_CHECK_LAUNCH();
        return EXAFAC_OK;
    }
    // one CTA, for the entry points without that scratch (no Newton step)
    const bool packed = chol_smem_bytes(R) > kPinvSmemCap;
    auto kernel = packed ? spd_pinv_packed_kernel : spd_pinv_kernel;
    const size_t smem = std::max(packed ? chol_packed_smem_bytes(R) : chol_smem_bytes(R), syev_smem_bytes(R));
    EXAFAC_CUDA_TRY(allow_smem(kernel));
    kernel<<<1, 512, smem, stream>>>(R, A, out, tol, vt_scratch);
    count_launch();
    EXAFAC_CHECK_LAUNCH();
    return EXAFAC_OK;
}

int launch_pinv(int R, const double* A, double* out, double tol, double* vt_scratch, cudaStream_t stream, double* scr) {
    return launch_pinv_impl(R, A, out, tol, vt_scratch, 0, stream, scr);
}

int launch_pinv_refined(int R, const double* A, double* out, double tol, double* vt_scratch, cudaStream_t stream,
                        double* scr) {
    return launch_pinv_impl(R, A, out, tol, vt_scratch, 1, stream, scr);
}

int launch_sigma_pinv_f32(int R, const double* ugram, double* sigma, double* ngram, int* degenerate, double* out,
                          double tol, double* vt_scratch, cudaStream_t stream) {
    const size_t smem = std::max(syev_smem_bytes(R), chol_smem_bytes(R));
    EXAFAC_CUDA_TRY(launch_dependent(sigma_pinv_kernel, 1, kSmallPinvThreads, smem, stream, R, ugram, sigma, ngram,
                                     degenerate, out, tol, vt_scratch));
    count_launch();
    EXAFAC_CHECK_LAUNCH();
    return EXAFAC_OK;
}

size_t syev_smem_bytes(int R) {
    int Re = R + (R & 1);
    return sizeof(double) * ((size_t)Re * Re + Re + 2) + sizeof(int) * (2 * Re + 1) + 16;
}

size_t syev_scratch_doubles(int R, int batch) {
    int Re = R + (R & 1);
    return (size_t)batch * Re * Re;
}

int launch_syev(int R, const double* A, int64_t a_stride, int batch, double* V, double* lam, int64_t v_stride,
                double* pinv, double tol, double* vt_scratch, cudaStream_t stream) {
    size_t smem = syev_smem_bytes(R);
    if (smem > 48 * 1024) {
        EXAFAC_CUDA_TRY(allow_smem(syev_kernel));
    }
    int threads = R <= 32 ? 256 : 512;
    syev_kernel<<<batch, threads, smem, stream>>>(R, A, a_stride, V, lam, v_stride, pinv, tol, vt_scratch); count_launch();
    EXAFAC_CHECK_LAUNCH();
    return EXAFAC_OK;
}

// X, its successor, A in full, S, G and E of each matrix.
size_t syev_refine_doubles(int R, int batch) { return (size_t)batch * 6 * R * R; }

int launch_syev_refined(int R, const double* A, int64_t a_stride, int batch, double* V, double* lam, int64_t v_stride,
                        double* vt_scratch, double* scratch, cudaStream_t stream) {
    if (R < kRefineMinRank) return launch_syev(R, A, a_stride, batch, V, lam, v_stride, nullptr, 0.0, vt_scratch, stream);
    const int64_t R2 = (int64_t)R * R, ss = 6 * R2;
    double *X = scratch, *Xn = X + R2, *As = Xn + R2, *S = As + R2, *G = S + R2, *E = G + R2;
    const size_t jsm = jacobi32_bytes(R);
    if (jsm > 40 * 1024) {  // (the 48 KB of a launch without it include the static part)
        EXAFAC_CUDA_TRY(allow_smem(jacobi32_kernel));
        EXAFAC_CUDA_TRY(allow_smem(refine_first_kernel));
    }
    jacobi32_kernel<<<batch, 512, jsm, stream>>>(R, A, a_stride, X, As, ss);
    count_launch();
    const dim3 grid((unsigned)R, (unsigned)batch);
    for (int it = 0; it <= kRefineSteps; it++) {
        const double limit = it < kRefineSteps ? kRefineLimit[it] : 1.0;
        EXAFAC_CUDA_TRY(launch_dependent(refine_forms_kernel, grid, 128, 0, stream, R, (const double*)As,
                                         (const double*)X, limit > 0.0 ? S : (double*)nullptr, G, ss));
        count_launch();
        if (it == kRefineSteps) break;
        if (it == 0) {
            EXAFAC_CUDA_TRY(launch_dependent(refine_first_kernel, (unsigned)batch, 512, jsm, stream, R, limit,
                                             (const double*)S, (const double*)G, E, ss));
        } else {
            EXAFAC_CUDA_TRY(launch_dependent(refine_e_kernel, grid, 128, 0, stream, R, limit, (const double*)S,
                                             (const double*)G, E, ss));
        }
        count_launch();
        EXAFAC_CUDA_TRY(launch_dependent(refine_update_kernel, grid, 128, 0, stream, R, (const double*)X,
                                         (const double*)E, Xn, ss));
        count_launch();
        std::swap(X, Xn);
    }
    const size_t smem = syev_smem_bytes(R);
    if (smem > 48 * 1024)
        EXAFAC_CUDA_TRY(allow_smem(syev_finish_kernel));
    EXAFAC_CUDA_TRY(launch_dependent(syev_finish_kernel, (unsigned)batch, R <= 32 ? 256 : 512, smem, stream, R, A,
                                     a_stride, (const double*)X, (const double*)S, (const double*)G, ss, V, lam,
                                     v_stride, vt_scratch));
    count_launch();
    EXAFAC_CHECK_LAUNCH();
    return EXAFAC_OK;
}

// ---------------------------------------------------------------------------
// STS-CP computeM of the mixed forms (sts_cp.hpp:80-188 with Cholesky factors
// in place of the two eigendecompositions).
//
// The draws use, per sampled mode, rows e_v with sum_v e_v e_v^T = M (the
// eigen tree picks v, then the row tree a row by (U_i . (h * e_v))^2): the
// row is then drawn with probability proportional to (h * U_i)^T M (h * U_i)
// whatever factor supplies the rows, so any E with E^T E = M gives the same
// distribution of rows and weights as the reference's scaled eigenvectors
// (only the intermediate leaf v differs).  The FP64 form keeps the
// eigenvectors, which reproduce the reference's draws; the mixed forms take
// Cholesky factors: about R^3 / 3 FP64 FMAs each, against some ten Jacobi
// sweeps of about 5 R^3.
//
// A = chain[first] (the Hadamard product of every Gram but mode n's) = L L^T,
// Phi = A^{-1} = L^{-T} L^{-1} (launch_chol_inverse), taken when lambda_min >=
// 1 / ||A^{-1}||_F > 10 tol (as the Cholesky pseudo-inverse above); the rows
// of L^{-1} are a factor of Phi and become E[N].  Otherwise
// sts_phi_accept_kernel (one CTA) computes the Jacobi eigendecomposition and
// the reference's W = V Lambda^{-1/2} (eigenvalues <= tol dropped).  Then
// chain[k] *= Phi for k >= 1, k != n.
//
// sts_chain_chol_kernel (one CTA per k = 1..N-1, k != n): the pivoted
// Cholesky P^T chain[k] P = L L^T (largest remaining diagonal first; stops
// once it is <= R eps times the largest diagonal, the rest of the matrix, a
// positive semidefinite remainder with entries that small, dropped): E[k]
// row v = column v of P L.
// ---------------------------------------------------------------------------

// Right-looking Cholesky of the packed lower triangle L (tri(i, j), j <= i),
// in place, with symmetric pivoting on the largest remaining diagonal (piv[j] =
// the original index at position j), stopping when it is <= stop; *rank = the
// number of columns factored.  col: R doubles of shared scratch.  Every thread
// returns the same *rank.
__device__ void chol_pivoted_block(int R, double* L, int* piv, double stop, double* col, int* rank) {
    __shared__ int s_p;
    __shared__ int s_stop;
    __shared__ double s_d, s_root[2];  // the pivot, its square root and the root's reciprocal
    const int tid = threadIdx.x, nt = blockDim.x;
    for (int i = tid; i < R; i += nt) piv[i] = i;
    if (tid == 0) s_stop = R;
    __syncthreads();
    for (int k = 0; k < R; k++) {
        if (tid < 32) {  // warp 0: the largest remaining diagonal (first index on ties)
            // positive doubles order as their bits: integer compares, off the FP64 pipe
            unsigned long long best = 0;
            int bi = k;
            for (int i = k + tid; i < R; i += 32) {
                const long long d = __double_as_longlong(L[tri(i, i)]);
                const unsigned long long v = d > 0 && d <= 0x7ff0000000000000ll ? (unsigned long long)d : 0ull;
                if (v > best) {
                    best = v;
                    bi = i;
                }
            }
            const uint32_t hi = __reduce_max_sync(0xffffffffu, (uint32_t)(best >> 32));
            const uint32_t mylo = (uint32_t)(best >> 32) == hi ? (uint32_t)best : 0u;
            const uint32_t lo = __reduce_max_sync(0xffffffffu, mylo);
            const unsigned long long top = ((unsigned long long)hi << 32) | lo;
            const int at = (int)__reduce_min_sync(0xffffffffu, best == top ? (uint32_t)bi : 0xffffu);
            if (tid == 0) {
                s_p = at;
                s_d = __longlong_as_double((long long)top);
                if (!(__longlong_as_double((long long)top) > stop)) s_stop = k;
            }
        }
        __syncthreads();
        if (s_stop == k) break;
        const int p = s_p;
        if (tid == nt - 1) {  // beside the swap (the diagonal entry to be at k moves meanwhile)
            s_root[0] = sqrt(s_d);
            s_root[1] = rsqrt(s_d);
        }
        if (p != k) {  // swap rows and columns k and p (disjoint element pairs)
            for (int j = tid; j < R; j += nt) {
                double *x = nullptr, *y = nullptr;
                if (j < k) {
                    x = &L[tri(k, j)];
                    y = &L[tri(p, j)];
                } else if (j == k) {
                    x = &L[tri(k, k)];
                    y = &L[tri(p, p)];
                } else if (j < p) {
                    x = &L[tri(j, k)];
                    y = &L[tri(p, j)];
                } else if (j > p) {
                    x = &L[tri(j, k)];
                    y = &L[tri(j, p)];
                }
                if (x) {
                    const double t = *x;
                    *x = *y;
                    *y = t;
                }
            }
            if (tid == 0) {
                const int t = piv[k];
                piv[k] = piv[p];
                piv[p] = t;
            }
        }
        __syncthreads();
        const double lkk = s_root[0], rkk = s_root[1];
        for (int i = k + 1 + tid; i < R; i += nt) col[i] = div_by(L[tri(i, k)], lkk, rkk);
        __syncthreads();
        if (tid == 0) L[tri(k, k)] = lkk;
        {  // the trailing lower triangle: a warp per row, its lanes along the row
            const int wid = tid >> 5, lane = tid & 31, nw = nt >> 5;
            for (int i = k + 1 + wid; i < R; i += nw) {
                const double ci = col[i];
                double* row = L + tri(i, 0);
                for (int j = k + 1 + lane; j < i; j += 32) row[j] -= ci * col[j];
                if (lane == 0) {
                    row[i] -= ci * ci;
                    row[k] = ci;
                }
            }
        }
        __syncthreads();
    }
    __syncthreads();
    *rank = s_stop;
}

// After launch_chol_inverse: E[N] and Phi stand, or one CTA computes them from
// the Jacobi eigendecomposition.
__global__ void __launch_bounds__(512) sts_phi_accept_kernel(int N, int R, const double* __restrict__ A, double tol,
                                                             double* __restrict__ E, double* __restrict__ Phi,
                                                             double* __restrict__ V, double* __restrict__ lam,
                                                             double* __restrict__ vt, double* __restrict__ scr) {
    extern __shared__ double smem[];
    __shared__ int stands;
    pdl_wait();
    const CholScratch s = chol_scratch(scr, R);
    const int R2 = R * R, tid = threadIdx.x, nt = blockDim.x;
    double* EN = E + (int64_t)N * R2;
    if (tid < 32) {
        const bool yes = chol_accepted(R, s, tol);
        if (tid == 0) stands = yes;
    }
    __syncthreads();
    if (stands) return;
    // Jacobi: W[:, R-1-v] = eigenvector v / sqrt(lambda_v), lambda_v > tol
    syev_block(R, A, V, lam, nullptr, tol, vt, smem);
    __syncthreads();
    for (int e = tid; e < R2; e += nt) {
        const int a = e / R, b = e % R;
        const int v = R - 1 - a;
        EN[e] = lam[v] > tol ? V[b * R + v] / sqrt(lam[v]) : 0.0;
    }
    __syncthreads();
    for (int e = tid; e < R2; e += nt) {
        const int a = e / R, b = e % R;
        double acc = 0.0;
        for (int w = 0; w < R; w++) acc = fma(EN[w * R + a], EN[w * R + b], acc);
        Phi[e] = acc;
    }
    if (tid == 0) *s.rank = -1;  // E[N] is written
}

// Row a: E[N] row a = row a of L^{-1} (when it stands), the packed Phi, and
// chain[k] *= Phi for k >= 1, k != n.
__global__ void __launch_bounds__(kMaxRank) sts_phi_rows_kernel(int N, int n, int R, double* __restrict__ chain,
                                                                double* __restrict__ E, const double* __restrict__ Phi,
                                                                double* __restrict__ PhiP, double* __restrict__ scr) {
    pdl_wait();
    const CholScratch s = chol_scratch(scr, R);
    const int R2 = R * R, a = blockIdx.x, b = threadIdx.x;
    if (b >= R) return;
    if (*s.rank != -1) E[(int64_t)N * R2 + a * R + b] = b <= a ? s.Li[a * R + b] : 0.0;
    const double p = Phi[a <= b ? a * R + b : b * R + a];
    if (a <= b) PhiP[a * R - a * (a - 1) / 2 + (b - a)] = p;  // packed upper triangle, rows in order
    for (int k = N - 1; k > 0; k--)
        if (k != n) chain[(int64_t)k * R2 + a * R + b] *= p;
}

__global__ void sts_chain_chol_kernel(int N, int n, int R, const double* __restrict__ chain, double* __restrict__ E) {
    extern __shared__ double smem[];
    __shared__ double col[kMaxRank];
    __shared__ int piv[kMaxRank];
    __shared__ double dmax_w[32];
    const int k = blockIdx.x;
    if (k == 0 || k == n || k >= N) return;
    const int R2 = R * R;
    const int tid = threadIdx.x, nt = blockDim.x;
    const double* A = chain + (int64_t)k * R2;
    double* Ek = E + (int64_t)k * R2;
    double* L = smem;
    for (int i = tid >> 5; i < R; i += nt >> 5)  // a warp per row of the packed lower triangle
        for (int j = tid & 31; j <= i; j += 32) L[tri(i, j)] = A[j * R + i];
    double dm = 0.0;
    for (int i = tid; i < R; i += nt) dm = fmax(dm, A[i * R + i]);
    for (int o = 16; o > 0; o >>= 1) dm = fmax(dm, __shfl_xor_sync(0xffffffffu, dm, o));
    if ((tid & 31) == 0) dmax_w[tid >> 5] = dm;
    __syncthreads();
    double dmax = 0.0;
    for (int q = 0; q < (nt + 31) / 32; q++) dmax = fmax(dmax, dmax_w[q]);
    int rank;
    chol_pivoted_block(R, L, piv, (double)R * 2.220446049250313e-16 * dmax, col, &rank);
    for (int e = tid; e < R2; e += nt) {  // E[k][v][piv[i]] = L[i][v]
        const int v = e / R, i = e % R;
        Ek[v * R + piv[i]] = (v < rank && i >= v) ? L[tri(i, v)] : 0.0;
    }
}

int launch_sts_factors_chol(int N, int n, int R, double tol, double* chain, double* E, double* Phi, double* PhiP,
                            double* V, double* lam, double* vt, double* scr, cudaStream_t stream) {
    const int first = (n == 0) ? 1 : 0;
    const double* A = chain + (int64_t)first * R * R;
    EXAFAC_TRY(launch_chol_inverse(R, A, Phi, true, scr, stream));
    const size_t smem = syev_smem_bytes(R);
    if (smem > 48 * 1024)
        EXAFAC_CUDA_TRY(allow_smem(sts_phi_accept_kernel));
    EXAFAC_CUDA_TRY(launch_dependent(sts_phi_accept_kernel, 1, 512, smem, stream, N, R, A, tol, E, Phi, V, lam, vt, scr));
    EXAFAC_CUDA_TRY(launch_dependent(sts_phi_rows_kernel, R, kMaxRank, 0, stream, N, n, R, chain, E, (const double*)Phi,
                                     PhiP, scr));
    add_launches(2);
    const size_t fsm = sizeof(double) * (size_t)(R * (R + 1) / 2);
    if (fsm > 48 * 1024)
        EXAFAC_CUDA_TRY(allow_smem(sts_chain_chol_kernel));
    if (N > 1) {
        sts_chain_chol_kernel<<<N, 512, fsm, stream>>>(N, n, R, chain, E);
        count_launch();
    }
    EXAFAC_CHECK_LAUNCH();
    return EXAFAC_OK;
}

}  // namespace exafac

using namespace exafac;

extern "C" size_t exafac_dense_workspace_bytes(int32_t R) {
    if (R < 1 || R > kMaxRank) return 0;
    return sizeof(double) * syev_scratch_doubles(R, 1);
}

extern "C" int exafac_syev(int32_t R, const double* A, double* V, double* lam, void* workspace, size_t workspace_bytes,
                           void* stream) {
    EXAFAC_ARG(R >= 1 && R <= kMaxRank, "exafac_syev: R out of range");
    EXAFAC_ARG(A && V && lam && workspace, "exafac_syev: null pointer");
    EXAFAC_ARG(workspace_bytes >= exafac_dense_workspace_bytes(R), "exafac_syev: workspace too small");
    return launch_syev(R, A, 0, 1, V, lam, 0, nullptr, 0.0, (double*)workspace, (cudaStream_t)stream);
}

extern "C" size_t exafac_syev_refined_workspace_bytes(int32_t R) {
    if (R < 1 || R > kMaxRank) return 0;
    return sizeof(double) * (syev_scratch_doubles(R, 1) + syev_refine_doubles(R, 1));
}

extern "C" int exafac_syev_refined(int32_t R, const double* A, double* V, double* lam, void* workspace,
                                   size_t workspace_bytes, void* stream) {
    EXAFAC_ARG(R >= 1 && R <= kMaxRank, "exafac_syev_refined: R out of range");
    EXAFAC_ARG(A && V && lam && workspace, "exafac_syev_refined: null pointer");
    EXAFAC_ARG(workspace_bytes >= exafac_syev_refined_workspace_bytes(R), "exafac_syev_refined: workspace too small");
    double* vt = (double*)workspace;
    return launch_syev_refined(R, A, 0, 1, V, lam, 0, vt, vt + syev_scratch_doubles(R, 1), (cudaStream_t)stream);
}

extern "C" int exafac_pinv_square(int32_t R, const double* A, double* out, double tol, void* workspace,
                                  size_t workspace_bytes, void* stream) {
    EXAFAC_ARG(R >= 1 && R <= kMaxRank, "exafac_pinv_square: R out of range");
    EXAFAC_ARG(A && out && workspace, "exafac_pinv_square: null pointer");
    EXAFAC_ARG(workspace_bytes >= exafac_dense_workspace_bytes(R), "exafac_pinv_square: workspace too small");
    return launch_pinv(R, A, out, tol, (double*)workspace, (cudaStream_t)stream);
}
