// Generalized CP on sampled entries: the model at sampled coordinates, its
// adjoint (the sampled MTTKRP of the loss derivatives into every factor),
// and a stratified entry sampler.  No counterpart in the reference, whose
// nearest relatives are execute_exact_mttkrp (sort_lookup.hpp:440-495) and
// the zero-sampling fit estimate of exafac/low_rank_tensor.py:110-184.
//
//   model     m_j = sum_r prod_k U_k[i_jk, r], a group of lanes per entry
//   loss      sum_j w_j f(x_j, m_j) and w_j df/dm in the model's pass
//   adjoint   G_n[i_jn, :] += g_j * prod_{k != n} U_k[i_jk, :], a group of
//             lanes per entry, every mode from one load of the entry's N
//             factor rows; the Khatri-Rao rows are recomputed here, never stored
//   sampler   J_nz nonzeros uniformly (weight nnz / J_nz) and J_z coordinates
//             uniformly (value 0, weight (prod dims - nnz) / J_z), Philox
//   adam      one Adam step over all factors in one launch, fused with the
//             projection onto nonnegative factors: 7 words of traffic per
//             parameter (parameter, moments read and written; gradient read)
//
// The adjoint accumulates with atomic adds, so its last bits depend on the
// order in which entries that share a row arrive.
#include <cmath>
#include <type_traits>

#include "common.cuh"

namespace exafac {

template <typename T>
struct PtrsT {
    T* p[kMaxModes];
};

struct Dims {
    int64_t d[kMaxModes];
};

// V consecutive elements, one 16-byte access when V * sizeof(T) == 16.
template <typename T, int V>
struct alignas(V * sizeof(T)) Pack {
    T v[V];
};

// The lanes of a warp that share an entry: a power of two, at least R / V of
// them up to the whole warp.  A factor row of 32 floats is 8 lanes' 16-byte
// loads, so a warp holds four entries in flight where a lane per column held
// one (J = 2^17 entries, R = 32, FP32, uniform coordinates in 1e6 x 1e6 x 1e4:
// model 42 -> 13 us, adjoint 70 -> 20).
static int entry_lanes(int R, int V) {
    int L = 1;
    while (L < 32 && L * V < R) L <<= 1;
    return L;
}

// The entry's coordinates, checked against the mode sizes; an entry with an
// out-of-range coordinate is skipped and flagged in *status (when given).
template <int M>
__device__ __forceinline__ bool load_entry(int N, const Dims& dims, const int32_t* __restrict__ idx, int64_t j,
                                           int32_t (&rows)[M], int* status) {
    bool ok = true;
#pragma unroll
    for (int k = 0; k < M; k++) {
        rows[k] = k < N ? __ldg(&idx[j * N + k]) : 0;
        if (k < N && (rows[k] < 0 || (int64_t)rows[k] >= dims.d[k])) ok = false;
    }
    if (!ok && status) atomicExch(status, 1);
    return ok;
}

// The kernels take the modes as a compile-time bound M (4, or 8 above four
// modes): the unrolled loops then hold no registers for modes that are not
// there (adjoint, 16-byte accesses: 40 against 80).
//
// The model value of entry j over the L lanes that share it (every lane of the
// warp calls; dead lanes pass live = false): the same sum on each of them.
template <typename T, int V, int M>
__device__ __forceinline__ T entry_model(int N, int R, const Dims& dims, int64_t j, bool live, int L, int gl,
                                         const int32_t* __restrict__ idx, const PtrsT<const T>& f, int* status) {
    int32_t rows[M];
    T acc = 0;
    if (live && load_entry(N, dims, idx, j, rows, status)) {
        for (int c = gl * V; c < R; c += L * V) {
            Pack<T, V> p;
#pragma unroll
            for (int v = 0; v < V; v++) p.v[v] = T(1);
#pragma unroll
            for (int k = 0; k < M; k++)
                if (k < N) {
                    const Pack<T, V> u = *reinterpret_cast<const Pack<T, V>*>(&f.p[k][(int64_t)rows[k] * R + c]);
#pragma unroll
                    for (int v = 0; v < V; v++) p.v[v] *= u.v[v];
                }
            if constexpr (V == 4)  // the pairwise order of a lane per column
                acc += (p.v[0] + p.v[1]) + (p.v[2] + p.v[3]);
            else if constexpr (V == 2)
                acc += p.v[0] + p.v[1];
            else
                acc += p.v[0];
        }
    }
    for (int o = L >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    return acc;
}

template <typename T, int V, int M>
__global__ void __launch_bounds__(256) cp_model_kernel(int N, int R, int L, Dims dims, int64_t J,
                                                       const int32_t* __restrict__ idx, PtrsT<const T> f,
                                                       T* __restrict__ m, int* status) {
    const int lane = threadIdx.x & 31, G = 32 / L, gl = lane & (L - 1);
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t j0 = warp * G; j0 < J; j0 += nwarps * G) {
        const int64_t j = j0 + lane / L;
        const T v = entry_model<T, V, M>(N, R, dims, j, j < J, L, gl, idx, f, status);
        if (gl == 0 && j < J) m[j] = v;
    }
}

// The losses f(x, m) and their derivatives in m (Hong, Kolda, Duersch, Table
// 2.1), the operations torch's autograd does on the same expressions.
constexpr double kLossEps = 1e-10;
template <typename T>
__device__ __forceinline__ void loss_term(int kind, T x, T w, T m, T& term, T& d) {
    if (kind == EXAFAC_LOSS_GAUSSIAN) {
        const T r = x - m;
        term = w * (r * r);
        d = -(w * (T(2) * r));
        return;
    }
    const T me = m + (T)kLossEps;
    const T lg = log(me);
    if (kind == EXAFAC_LOSS_POISSON) {
        term = w * (m - x * lg);
        d = w - (w * x) / me;
    } else {
        const T m1 = m + T(1);
        term = w * (log(m1) - x * lg);
        d = w / m1 - (w * x) / me;
    }
}

// The weighted loss over the sampled entries and its derivative in each model
// value, in one pass: no model values, loss values or derivatives of the steps
// between go through memory, where torch's elementwise kernels took ten
// launches (FP32, J = 2^17, Zipf coordinates: model 40 us and 45 us of those; 29
// us together).  Terms are summed in FP64: each thread its own, the block's in a
// fixed tree, and the last block to finish (partial[0 .. grid) written, a
// ticket taken) adds the blocks' sums in order, so the sum does not depend on
// the schedule.
template <typename T, int V, int M>
__global__ void __launch_bounds__(256) cp_loss_kernel(int kind, int N, int R, int L, Dims dims, int64_t J,
                                                      const int32_t* __restrict__ idx, const T* __restrict__ x,
                                                      const T* __restrict__ w, PtrsT<const T> f, T* __restrict__ d,
                                                      T* __restrict__ loss, double* __restrict__ partial, int* ticket,
                                                      int* status) {
    __shared__ double red[8];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, G = 32 / L, gl = lane & (L - 1);
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    double sum = 0.0;
    for (int64_t j0 = warp * G; j0 < J; j0 += nwarps * G) {
        const int64_t j = j0 + lane / L;
        const bool own = gl == 0 && j < J;
        const T xj = own ? x[j] : T(0), wj = own ? w[j] : T(0);
        const T m = entry_model<T, V, M>(N, R, dims, j, j < J, L, gl, idx, f, status);
        if (own) {
            T term, dj;
            loss_term<T>(kind, xj, wj, m, term, dj);
            d[j] = dj;
            sum += (double)term;
        }
    }
    sum = warp_sum(sum);
    if (lane == 0) red[wid] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int i = 0; i < 8; i++) s += red[i];
        partial[blockIdx.x] = s;
        __threadfence();
        last = atomicAdd(ticket, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double s = 0.0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += 256) s += __ldcg(&partial[i]);
    s = warp_sum(s);
    if (lane == 0) red[wid] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int i = 0; i < 8; i++) t += red[i];
        *loss = (T)t;
    }
}

// Adds V consecutive elements to device memory: one 16-byte reduction for four
// floats, an element at a time otherwise (there is no wider FP64 form).
template <typename T, int V>
__device__ __forceinline__ void add_pack(T* at, const Pack<T, V>& p) {
    if constexpr (std::is_same<T, float>::value && V == 4) {
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(__cvta_generic_to_global(at)), "f"(p.v[0]),
                     "f"(p.v[1]), "f"(p.v[2]), "f"(p.v[3])
                     : "memory");
    } else {
#pragma unroll
        for (int v = 0; v < V; v++) atomicAdd(at + v, p.v[v]);
    }
}

// scale: a device scalar multiplied into every gm[j], or null.
template <typename T, int V, int M>
__global__ void __launch_bounds__(256) cp_adjoint_kernel(int N, int R, int L, Dims dims, int64_t J,
                                                         const int32_t* __restrict__ idx, const T* __restrict__ gm,
                                                         const T* __restrict__ scale, PtrsT<const T> f, PtrsT<T> g,
                                                         int* status) {
    const int lane = threadIdx.x & 31, G = 32 / L, gl = lane & (L - 1);
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const T sc = scale ? *scale : T(1);
    for (int64_t j = warp * G + lane / L; j < J; j += nwarps * G) {
        const T gj = scale ? gm[j] * sc : gm[j];
        if (gj == T(0)) continue;
        int32_t rows[M];
        if (!load_entry(N, dims, idx, j, rows, status)) continue;
        for (int c = gl * V; c < R; c += L * V) {
            Pack<T, V> v[M];
#pragma unroll
            for (int k = 0; k < M; k++)
                if (k < N) v[k] = *reinterpret_cast<const Pack<T, V>*>(&f.p[k][(int64_t)rows[k] * R + c]);
#pragma unroll
            for (int n = 0; n < M; n++) {
                if (n < N && g.p[n]) {
                    Pack<T, V> p;
#pragma unroll
                    for (int e = 0; e < V; e++) p.v[e] = gj;
#pragma unroll
                    for (int k = 0; k < M; k++)
                        if (k < N && k != n)
#pragma unroll
                            for (int e = 0; e < V; e++) p.v[e] *= v[k].v[e];
                    add_pack<T, V>(&g.p[n][(int64_t)rows[n] * R + c], p);
                }
            }
        }
    }
}

// Zeroes up to kMaxModes device arrays in one launch (16-byte stores where the
// array starts on a 16-byte boundary); lengths in 4-byte words.
struct ZeroList {
    uint32_t* p[kMaxModes];
    int64_t words[kMaxModes];
};
__global__ void __launch_bounds__(256) zero_list_kernel(int count, ZeroList z) {
    const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int t = 0; t < count; t++) {
        const int64_t nv = ((uintptr_t)z.p[t] & 15u) ? 0 : z.words[t] >> 2;
        for (int64_t i = tid; i < nv; i += stride) reinterpret_cast<uint4*>(z.p[t])[i] = make_uint4(0, 0, 0, 0);
        for (int64_t i = nv * 4 + tid; i < z.words[t]; i += stride) z.p[t][i] = 0u;
    }
}

template <typename T>
__global__ void gcp_sample_kernel(int N, Dims dims, int64_t nnz, const int32_t* __restrict__ nz_idx,
                                  const T* __restrict__ nz_vals, int64_t Jnz, int64_t Jz, uint64_t seed, uint64_t ctr,
                                  T wnz, T wz, int32_t* __restrict__ idx_out, T* __restrict__ x_out,
                                  T* __restrict__ w_out) {
    const int64_t J = Jnz + Jz;
    const uint2 key = make_uint2((unsigned)seed, (unsigned)(seed >> 32));
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < J; j += (int64_t)gridDim.x * blockDim.x) {
        const uint4 r0 = philox4x32_10(make_uint4((unsigned)j, (unsigned)(j >> 32), (unsigned)ctr,
                                                  (unsigned)(ctr >> 32) ^ 0x9E3779B9u), key);
        if (j < Jnz) {
            // uniform nonzero: 64 random bits reduced modulo nnz (bias < nnz / 2^64)
            const uint64_t b = ((uint64_t)r0.x << 32) | r0.y;
            const int64_t e = (int64_t)(b % (uint64_t)nnz);
            for (int k = 0; k < N; k++) idx_out[j * N + k] = nz_idx[e * N + k];
            x_out[j] = nz_vals[e];
            w_out[j] = wnz;
        } else {
            // uniform coordinate, taken as a zero (a hit on a nonzero has
            // probability nnz / prod dims)
            const uint4 r1 = philox4x32_10(make_uint4((unsigned)j, (unsigned)(j >> 32), (unsigned)ctr,
                                                      (unsigned)(ctr >> 32) ^ 0x7F4A7C15u), key);
            const unsigned w8[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
            for (int k = 0; k < N; k++) {
                const uint64_t b = ((uint64_t)w8[k] << 21) ^ (uint64_t)w8[(k + 4) & 7];
                idx_out[j * N + k] = (int32_t)(b % (uint64_t)dims.d[k]);
            }
            x_out[j] = T(0);
            w_out[j] = wz;
        }
    }
}

// Adam (Kingma and Ba; torch.optim.Adam's update without weight decay or
// amsgrad), per element in the parameter's own precision:
//   m = m + (1 - b1) (g - m);  v = b2 v + (1 - b2) g^2;
//   p = p - step_size m / (sqrt(v) / sqrt(1 - b2^t) + eps),  step_size = lr / (1 - b1^t)
// then p = max(p, lower) when projecting (a NaN stays NaN).  A null gradient
// counts as zero (the moments still decay and the parameter still moves).
struct AdamTensors {
    void* p[kMaxModes];
    const void* g[kMaxModes];
    void* m[kMaxModes];
    void* v[kMaxModes];
    int64_t n[kMaxModes];
};

template <typename T>
struct AdamCoef {
    T step_size, omb1, b2, omb2, bc2_sqrt, eps, lower;
    int project;
};

template <typename T>
__device__ __forceinline__ void adam_elem(T& p, T g, T& m, T& v, const AdamCoef<T>& c) {
    m = m + c.omb1 * (g - m);
    v = c.b2 * v + c.omb2 * (g * g);
    const T denom = sqrt(v) / c.bc2_sqrt + c.eps;
    p = p - c.step_size * (m / denom);
    if (c.project && p < c.lower) p = c.lower;
}

// V elements per access (16 bytes when every base is 16-byte aligned); bound by
// DRAM: 64 million FP32 parameters in 0.29 ms, 6.3 TB/s.  A block per
// contiguous tile instead of the grid-stride loop was slower (0.32 ms).
template <typename T, int V>
__global__ void __launch_bounds__(256) adam_step_kernel(int count, AdamTensors ts, AdamCoef<T> c) {
    using P = Pack<T, V>;
    const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int t = 0; t < count; t++) {
        T* __restrict__ p = static_cast<T*>(ts.p[t]);
        const T* __restrict__ g = static_cast<const T*>(ts.g[t]);
        T* __restrict__ m = static_cast<T*>(ts.m[t]);
        T* __restrict__ v = static_cast<T*>(ts.v[t]);
        const int64_t n = ts.n[t], nv = n / V;
        for (int64_t i = tid; i < nv; i += stride) {
            P a = reinterpret_cast<P*>(p)[i], b = reinterpret_cast<P*>(m)[i], d = reinterpret_cast<P*>(v)[i], e;
            if (g)
                e = reinterpret_cast<const P*>(g)[i];
            else
#pragma unroll
                for (int u = 0; u < V; u++) e.v[u] = T(0);
#pragma unroll
            for (int u = 0; u < V; u++) adam_elem(a.v[u], e.v[u], b.v[u], d.v[u], c);
            reinterpret_cast<P*>(p)[i] = a;
            reinterpret_cast<P*>(m)[i] = b;
            reinterpret_cast<P*>(v)[i] = d;
        }
        for (int64_t i = nv * V + tid; i < n; i += stride) adam_elem(p[i], g ? g[i] : T(0), m[i], v[i], c);
    }
}

static int grid_for(int64_t work, int per_block) {
    int64_t b = (work + per_block - 1) / per_block;
    return (int)std::max<int64_t>(1, std::min<int64_t>(b, 152 * 16));
}

}  // namespace exafac

using namespace exafac;

#define GCP_DTYPE_ARG(dtype) \
    EXAFAC_ARG((dtype) == EXAFAC_DTYPE_F32 || (dtype) == EXAFAC_DTYPE_F64, "dtype must be EXAFAC_DTYPE_F32 or F64")

static int dims_arg(int N, const int64_t* dims, Dims* d) {
    EXAFAC_ARG(dims != nullptr, "null dims");
    for (int k = 0; k < kMaxModes; k++) d->d[k] = 0;
    for (int k = 0; k < N; k++) {
        EXAFAC_ARG(dims[k] >= 1 && dims[k] <= 0x7fffffffll, "mode sizes must be in [1, 2^31)");
        d->d[k] = dims[k];
    }
    return EXAFAC_OK;
}

// 16-byte accesses need rows that are a multiple of 16 bytes and bases on a
// 16-byte boundary.
static bool packable(int R, int N, const void* const* a, const void* const* b, int dtype) {
    if ((int64_t)R * (dtype == EXAFAC_DTYPE_F32 ? 4 : 8) % 16) return false;
    for (int k = 0; k < N; k++) {
        if ((uintptr_t)a[k] & 15u) return false;
        if (b && ((uintptr_t)b[k] & 15u)) return false;
    }
    return true;
}

template <typename T>
static PtrsT<T> ptrs_of(int N, const void* const* a) {
    PtrsT<T> f{};
    for (int k = 0; k < N; k++) f.p[k] = static_cast<T*>(const_cast<void*>(a[k]));
    return f;
}

template <typename T, int V, int M>
static void launch_model(int N, int R, const Dims& d, int64_t J, const int32_t* idx, const void* const* factors,
                         void* m, int* status, cudaStream_t st) {
    const int L = entry_lanes(R, V);
    cp_model_kernel<T, V, M><<<grid_for(J, 8 * (32 / L)), 256, 0, st>>>(N, R, L, d, J, idx, ptrs_of<const T>(N, factors),
                                                                    static_cast<T*>(m), status);
}

template <typename T, int V, int M>
static void launch_adjoint(int N, int R, const Dims& d, int64_t J, const int32_t* idx, const void* gm,
                           const void* scale, const void* const* factors, void* const* grads, int* status,
                           cudaStream_t st) {
    const int L = entry_lanes(R, V);
    cp_adjoint_kernel<T, V, M><<<grid_for(J, 8 * (32 / L)), 256, 0, st>>>(
        N, R, L, d, J, idx, static_cast<const T*>(gm), static_cast<const T*>(scale), ptrs_of<const T>(N, factors),
        ptrs_of<T>(N, grads), status);
}

template <typename T, int V, int M>
static void launch_loss(int kind, int N, int R, const Dims& d, int64_t J, const int32_t* idx, const void* x,
                        const void* w, const void* const* factors, void* deriv, void* loss, double* partial,
                        int* ticket, int* status, cudaStream_t st) {
    const int L = entry_lanes(R, V);
    cp_loss_kernel<T, V, M><<<std::min<int>(grid_for(J, 8 * (32 / L)), EXAFAC_LOSS_BLOCKS), 256, 0, st>>>(
        kind, N, R, L, d, J, idx, static_cast<const T*>(x), static_cast<const T*>(w), ptrs_of<const T>(N, factors),
        static_cast<T*>(deriv), static_cast<T*>(loss), partial, ticket, status);
}

#define GCP_DISPATCH_MODES(fn, T, V, ...) (N <= 4 ? fn<T, V, 4> : fn<T, V, kMaxModes>)(__VA_ARGS__)
#define GCP_DISPATCH(fn, pack, ...)                           \
    do {                                                      \
        const bool p_ = (pack);                               \
        if (dtype == EXAFAC_DTYPE_F32) {                      \
            if (p_)                                           \
                GCP_DISPATCH_MODES(fn, float, 4, __VA_ARGS__); \
            else                                              \
                GCP_DISPATCH_MODES(fn, float, 1, __VA_ARGS__); \
        } else if (p_) {                                      \
            GCP_DISPATCH_MODES(fn, double, 2, __VA_ARGS__);   \
        } else {                                              \
            GCP_DISPATCH_MODES(fn, double, 1, __VA_ARGS__);   \
        }                                                     \
    } while (0)

extern "C" int exafac_cp_sampled_model(int32_t N, int32_t R, const int64_t* dims, int64_t J, const int32_t* idx,
                                       const void* const* factors, void* m_out, int32_t dtype, int32_t* status,
                                       void* stream) {
    EXAFAC_ARG(N >= 1 && N <= kMaxModes, "N must be in [1, 8]");
    EXAFAC_ARG(R >= 1, "R must be >= 1");
    EXAFAC_ARG(J >= 0, "J must be >= 0");
    GCP_DTYPE_ARG(dtype);
    Dims d;
    EXAFAC_TRY(dims_arg(N, dims, &d));
    if (J == 0) return EXAFAC_OK;
    EXAFAC_ARG(idx && factors && m_out, "null argument");
    for (int k = 0; k < N; k++) EXAFAC_ARG(factors[k] != nullptr, "null factor matrix");
    cudaStream_t st = (cudaStream_t)stream;
    GCP_DISPATCH(launch_model, packable(R, N, factors, nullptr, dtype), N, R, d, J, idx, factors, m_out, status, st);
    count_launch();
    EXAFAC_CHECK_LAUNCH();
    return EXAFAC_OK;
}

extern "C" int exafac_cp_sampled_adjoint(int32_t N, int32_t R, const int64_t* dims, int64_t J, const int32_t* idx,
                                         const void* grad_m, const void* const* factors, void* const* grads,
                                         int32_t dtype, int32_t* status, void* stream) {
    EXAFAC_ARG(N >= 1 && N <= kMaxModes, "N must be in [1, 8]");
    EXAFAC_ARG(R >= 1, "R must be >= 1");
    EXAFAC_ARG(J >= 0, "J must be >= 0");
    GCP_DTYPE_ARG(dtype);
    Dims d;
    EXAFAC_TRY(dims_arg(N, dims, &d));
    if (J == 0) return EXAFAC_OK;
    EXAFAC_ARG(idx && grad_m && factors && grads, "null argument");
    for (int k = 0; k < N; k++) EXAFAC_ARG(factors[k] != nullptr, "null factor matrix");
    cudaStream_t st = (cudaStream_t)stream;
    GCP_DISPATCH(launch_adjoint, packable(R, N, factors, grads, dtype), N, R, d, J, idx, grad_m, nullptr, factors,
                 grads, status, st);
    count_launch();
    EXAFAC_CHECK_LAUNCH();
    return EXAFAC_OK;
}

extern "C" int exafac_cp_sampled_loss(int32_t kind, int32_t N, int32_t R, const int64_t* dims, int64_t J,
                                      const int32_t* idx, const void* x, const void* w, const void* const* factors,
                                      void* deriv_out, void* loss_out, void* scratch, int32_t dtype, int32_t* status,
                                      void* stream) {
    EXAFAC_ARG(kind >= EXAFAC_LOSS_POISSON && kind <= EXAFAC_LOSS_GAUSSIAN, "unknown loss");
    EXAFAC_ARG(N >= 1 && N <= kMaxModes, "N must be in [1, 8]");
    EXAFAC_ARG(R >= 1, "R must be >= 1");
    EXAFAC_ARG(J >= 1, "J must be >= 1");
    GCP_DTYPE_ARG(dtype);
    Dims d;
    EXAFAC_TRY(dims_arg(N, dims, &d));
    EXAFAC_ARG(idx && x && w && factors && deriv_out && loss_out && scratch, "null argument");
    EXAFAC_ARG(((uintptr_t)scratch & 7u) == 0, "scratch must be 8-byte aligned");
    for (int k = 0; k < N; k++) EXAFAC_ARG(factors[k] != nullptr, "null factor matrix");
    cudaStream_t st = (cudaStream_t)stream;
    double* partial = static_cast<double*>(scratch) + 1;
    int* ticket = static_cast<int*>(scratch);
    EXAFAC_CUDA_TRY(cudaMemsetAsync(ticket, 0, sizeof(int), st));
    GCP_DISPATCH(launch_loss, packable(R, N, factors, nullptr, dtype), kind, N, R, d, J, idx, x, w, factors,
                 deriv_out, loss_out, partial, ticket, status, st);
    count_launch();
    EXAFAC_CHECK_LAUNCH();
    return EXAFAC_OK;
}

extern "C" int exafac_cp_sampled_gradient(int32_t N, int32_t R, const int64_t* dims, int64_t J, const int32_t* idx,
                                          const void* grad_m, const void* scale, const void* const* factors,
                                          void* const* grads, int32_t dtype, int32_t* status, void* stream) {
    EXAFAC_ARG(N >= 1 && N <= kMaxModes, "N must be in [1, 8]");
    EXAFAC_ARG(R >= 1, "R must be >= 1");
    EXAFAC_ARG(J >= 1, "J must be >= 1");
    GCP_DTYPE_ARG(dtype);
    Dims d;
    EXAFAC_TRY(dims_arg(N, dims, &d));
    EXAFAC_ARG(idx && grad_m && factors && grads, "null argument");
    for (int k = 0; k < N; k++) EXAFAC_ARG(factors[k] != nullptr, "null factor matrix");
    cudaStream_t st = (cudaStream_t)stream;
    ZeroList z{};
    int count = 0;
    int64_t most = 0;
    for (int k = 0; k < N; k++)
        if (grads[k]) {
            z.p[count] = static_cast<uint32_t*>(grads[k]);
            z.words[count] = dims[k] * R * (dtype == EXAFAC_DTYPE_F32 ? 1 : 2);
            most = std::max(most, z.words[count++]);
        }
    if (count == 0) return EXAFAC_OK;
    zero_list_kernel<<<grid_for(most / 4 + 1, 256), 256, 0, st>>>(count, z);
    count_launch();
    GCP_DISPATCH(launch_adjoint, packable(R, N, factors, grads, dtype), N, R, d, J, idx, grad_m, scale, factors,
                 grads, status, st);
    count_launch();
    EXAFAC_CHECK_LAUNCH();
    return EXAFAC_OK;
}

extern "C" int exafac_gcp_sample_entries(int32_t N, const int64_t* dims, int64_t nnz, const int32_t* nz_idx,
                                         const void* nz_vals, int64_t J_nz, int64_t J_z, uint64_t seed,
                                         uint64_t counter, int32_t* idx_out, void* x_out, void* w_out,
                                         int32_t dtype, void* stream) {
    EXAFAC_ARG(N >= 1 && N <= kMaxModes, "N must be in [1, 8]");
    EXAFAC_ARG(J_nz >= 0 && J_z >= 0, "sample counts must be >= 0");
    EXAFAC_ARG(J_nz == 0 || (nnz >= 1 && nz_idx && nz_vals), "nonzero samples need the nonzeros");
    GCP_DTYPE_ARG(dtype);
    Dims d;
    EXAFAC_TRY(dims_arg(N, dims, &d));
    if (J_nz + J_z == 0) return EXAFAC_OK;
    EXAFAC_ARG(idx_out && x_out && w_out, "null output");
    double total = 1.0;
    for (int k = 0; k < N; k++) total *= (double)dims[k];
    const double wnz = J_nz ? (double)nnz / (double)J_nz : 0.0;
    const double wz = J_z ? std::max(total - (double)nnz, 0.0) / (double)J_z : 0.0;
    cudaStream_t st = (cudaStream_t)stream;
    const int grid = grid_for(J_nz + J_z, 256);
    if (dtype == EXAFAC_DTYPE_F32)
        gcp_sample_kernel<float><<<grid, 256, 0, st>>>(N, d, nnz, nz_idx, static_cast<const float*>(nz_vals), J_nz,
                                                       J_z, seed, counter, (float)wnz, (float)wz, idx_out,
                                                       static_cast<float*>(x_out), static_cast<float*>(w_out));
    else
        gcp_sample_kernel<double><<<grid, 256, 0, st>>>(N, d, nnz, nz_idx, static_cast<const double*>(nz_vals), J_nz,
                                                        J_z, seed, counter, wnz, wz, idx_out,
                                                        static_cast<double*>(x_out), static_cast<double*>(w_out));
    count_launch();
    EXAFAC_CHECK_LAUNCH();
    return EXAFAC_OK;
}

template <typename T>
static void launch_adam(int count, const AdamTensors& ts, int64_t total, double lr, double b1, double b2, double eps,
                        int64_t step, int project, double lower, bool vec, cudaStream_t st) {
    AdamCoef<T> c;
    c.step_size = (T)(lr / (1.0 - std::pow(b1, (double)step)));
    c.omb1 = (T)(1.0 - b1);
    c.b2 = (T)b2;
    c.omb2 = (T)(1.0 - b2);
    c.bc2_sqrt = (T)std::sqrt(1.0 - std::pow(b2, (double)step));
    c.eps = (T)eps;
    c.lower = (T)lower;
    c.project = project;
    constexpr int V = 16 / sizeof(T);
    const int grid = grid_for(vec ? (total + V - 1) / V : total, 256);
    if (vec)
        adam_step_kernel<T, V><<<grid, 256, 0, st>>>(count, ts, c);
    else
        adam_step_kernel<T, 1><<<grid, 256, 0, st>>>(count, ts, c);
}

extern "C" int exafac_adam_step(int32_t count, void* const* params, const void* const* grads, void* const* exp_avg,
                                void* const* exp_avg_sq, const int64_t* numel, int32_t dtype, double lr,
                                double beta1, double beta2, double eps, int64_t step, int32_t project, double lower,
                                void* stream) {
    EXAFAC_ARG(count >= 0 && count <= kMaxModes, "count must be in [0, 8]");
    GCP_DTYPE_ARG(dtype);
    EXAFAC_ARG(step >= 1, "step must be >= 1 (the step count after this update)");
    EXAFAC_ARG(beta1 >= 0.0 && beta1 < 1.0 && beta2 >= 0.0 && beta2 < 1.0, "betas must be in [0, 1)");
    EXAFAC_ARG(eps >= 0.0 && lr >= 0.0, "lr and eps must be >= 0");
    if (count == 0) return EXAFAC_OK;
    EXAFAC_ARG(params && exp_avg && exp_avg_sq && numel, "null argument");
    AdamTensors ts{};
    int64_t total = 0;
    bool vec = true;  // 16-byte accesses
    for (int t = 0; t < count; t++) {
        EXAFAC_ARG(numel[t] >= 0, "element counts must be >= 0");
        EXAFAC_ARG(numel[t] == 0 || (params[t] && exp_avg[t] && exp_avg_sq[t]), "null parameter or moment");
        ts.p[t] = params[t];
        ts.g[t] = grads ? grads[t] : nullptr;
        ts.m[t] = exp_avg[t];
        ts.v[t] = exp_avg_sq[t];
        ts.n[t] = numel[t];
        total = std::max<int64_t>(total, numel[t]);
        const uintptr_t a = (uintptr_t)ts.p[t] | (uintptr_t)ts.g[t] | (uintptr_t)ts.m[t] | (uintptr_t)ts.v[t];
        if (a & 15u) vec = false;
    }
    if (total == 0) return EXAFAC_OK;
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == EXAFAC_DTYPE_F32)
        launch_adam<float>(count, ts, total, lr, beta1, beta2, eps, step, project, lower, vec, st);
    else
        launch_adam<double>(count, ts, total, lr, beta1, beta2, eps, step, project, lower, vec, st);
    count_launch();
    EXAFAC_CHECK_LAUNCH();
    return EXAFAC_OK;
}

