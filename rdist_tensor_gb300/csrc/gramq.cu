// The design rows of the FP64 form and their Gram matrix sum_j x_j x_j^T
// (accumulator_stationary.hpp:212-249) from exact digit products on the tensor
// cores.
//
// An SM retires an FP64 instruction of a warp per 19 clocks, R (R + 1) / 64 of
// them per row: 1.27 ms for the design Gram at R = 64, J = 2^18.  Here the rows go
// in tiles of 64, each column scaled by a power of two to |x'| < 2^6 within
// the tile and cut into eight balanced base-256 digits (units of 2^-56, so that
// a value down to 2^-9 of its column's largest keeps all its bits); the products
// of the digits i and j with i + j <= 7 accumulate by weight i + j in tensor
// memory, at most 8 x 64 products of below 2^14, exact integers.  The eight
// weights are put together in 64-bit integers, scaled back and added to an
// FP64 total per entry, once per tile.
//
// Error of an entry and tile, in the scaled units (the columns' largest values
// are 2^5 to 2^6): the cut of x' to 2^-56 on both sides 64 x 2 x 2^6 x 2^-56 =
// 2^-43, the dropped weights (i + j >= 8) 64 x 7.1 x 2^14 x 2^-64 = 2^-41.2, the
// cut of the sum 2^-44: together below 2^-40.6, that is 2^-50.6 of the product of
// the two columns' largest values in the tile.  64 FMAs may lose 64^2 / 2 x
// 2^-53 = 2^-42 of it.  An entry all of whose products are far smaller than that
// (columns that are large in different rows) keeps fewer bits than an FMA sum
// would; the inverse takes no harm, since a Cholesky factor's own error is a
// rounding of sqrt(G_aa G_bb) in every entry.
//
// A tile with a value above 2^877, infinite or NaN, or with values below 2^-895
// (a group of eight rows of a column, not all zero), is summed in FP64: products
// would overflow on the way, infinities have no digits, and a column of
// subnormals does not scale to 2^5.
// Measured (GB300): R = 64, J = 2^18: 1270 -> 436 us; R = 100, J = 100003, four modes:
// 970 -> 180 us (and their partial sums' reduction 65 -> 10 us).
#include "digits.cuh"
#include "engine.cuh"

namespace exafac {

constexpr int kGqRows = 64;     // rows of a tile (the products' K)
constexpr int kGqDigits = 8;
constexpr int kGqThreads = 512;
constexpr int kGqCols = 64;     // columns per pass: 8 weights of them fill tensor memory
constexpr int kGqMinExp = 128, kGqMaxExp = 1900;  // biased exponents between which a tile goes by digits

struct GqShape {
    int Rp, nb, passes;   // R padded to 16, columns per pass, passes
    uint32_t digit;       // bytes of one digit's slice, Rp x 64 bf16
};
__host__ __device__ inline GqShape gq_shape(int R) {
    GqShape g;
    g.Rp = (R + 15) & ~15;
    g.nb = g.Rp < kGqCols ? g.Rp : kGqCols;
    g.passes = (g.Rp + g.nb - 1) / g.nb;
    g.digit = (uint32_t)g.Rp * kGqRows * 2u;
    return g;
}
// The products read 128 rows of the first operand from every digit's start (and
// a whole pass of columns): what lies past R belongs to the next digit or to the
// padding, finite or not, and lands in accumulators that nobody reads.
static size_t gq_smem(int R) {
    const GqShape g = gq_shape(R);
    return (size_t)kGqDigits * g.digit + (size_t)(128 - std::min(128, g.Rp)) * kGqRows * 2 + 128;
}

__global__ void __launch_bounds__(kGqThreads, 1)
    design_digits_kernel(int N, int n, int R, const int64_t* __restrict__ ju_dev, const uint32_t* __restrict__ sd,
                         const double* __restrict__ wd, FactorPtrs f, double* __restrict__ D, double* __restrict__ part,
                         DeviceStatus* status, uint32_t wait_polls, int64_t withhold) {
    extern __shared__ __align__(128) unsigned char gq_raw[];
    __shared__ uint32_t at[kMaxModes][kGqRows];  // the rows' indices
    __shared__ double sw[kGqRows];
    __shared__ double scale[kMaxRank];
    __shared__ int ecol[2][kMaxRank];  // the columns' largest exponents, ping-pong
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_base;
    const GqShape g = gq_shape(R);
    unsigned char* X = gq_raw + ((128u - (smem_u32(gq_raw) & 127u)) & 127u);
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    if (w == 0) tmem_alloc(&tmem_base, 512);
    if (tid == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    for (int a = tid; a < 2 * kMaxRank; a += kGqThreads) ecol[0][a] = 0;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    const int64_t live = *ju_dev;
    const int64_t ntiles = (live + kGqRows - 1) / kGqRows;
    uint32_t phase = 0;
    bool lost = false, dead = false;
    bool flight = false;  // thread 0: products on their way
    // entry (a, b): a = tensor memory lane, b in this thread's 16 columns of each pass
    const int a = (w & 3) * 32 + lane, grp = w >> 2;
    const int cpt = g.nb / 4;
    double total[2][16];
#pragma unroll
    for (int q = 0; q < 16; q++) total[0][q] = total[1][q] = 0.0;
    int buf = 0;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, buf ^= 1) {
        const int64_t j0 = tile * kGqRows;
        const int nr = (int)min((int64_t)kGqRows, live - j0);
        for (int e = tid; e < kGqRows * N; e += kGqThreads) {
            const int r = e / N, k = e - r * N;
            at[k][r] = r >= nr ? 0u : sd[(j0 + r) * N + k];
        }
        if (tid >= kGqThreads - kGqRows) {
            const int r = tid - (kGqThreads - kGqRows);
            sw[r] = r < nr ? sqrt(wd[j0 + r]) : 0.0;
        }
        __syncthreads();
        // column a, rows 8 kc .. + 7 per item, the column fastest
        double v[2][8];
        bool fp64 = false;
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int e = tid + u * kGqThreads, kc = e / g.Rp, c = e - kc * g.Rp;
            int top = 0;
#pragma unroll
            for (int q = 0; q < 8; q++) v[u][q] = 1.0;
            if (kc < 8 && c < R) {
                bool first = true;
                for (int k = 0; k < N; k++) {  // eight loads in flight per mode
                    if (k == n) continue;
                    const double* U = f.U[k] + c;
                    double y[8];
#pragma unroll
                    for (int q = 0; q < 8; q++) y[q] = __ldg(U + (int64_t)at[k][8 * kc + q] * R);
#pragma unroll
                    for (int q = 0; q < 8; q++) v[u][q] = first ? y[q] : v[u][q] * y[q];
                    first = false;
                }
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const int r = 8 * kc + q;
                    v[u][q] *= sw[r];
                    if (r < nr) D[(j0 + r) * R + c] = v[u][q] * sw[r];
                    else v[u][q] = 0.0;
                    top = max(top, bexp(v[u][q]));
                }
            }
            if (kc >= 8 || c >= R) {
#pragma unroll
                for (int q = 0; q < 8; q++) v[u][q] = 0.0;
            }
            if (top > 0) atomicMax(&ecol[buf][c], top);  // (c < R here)
            long long bits = 0;
#pragma unroll
            for (int q = 0; q < 8; q++) bits |= __double_as_longlong(v[u][q]);
            fp64 = fp64 || top > kGqMaxExp || (top < kGqMinExp && bits << 1 != 0);
        }
        fp64 = __syncthreads_or(fp64);
        if (tid < kMaxRank) {
            // the accumulators' integers are in units of 2^-44 of the scaled columns' products
            scale[tid] = scalbn(1.0, ecol[buf][tid] - 1028 - 22);
            ecol[buf ^ 1][tid] = 0;
        }
        if (fp64) {  // in FP64, the rows in shared memory where the digits go
            double* x = reinterpret_cast<double*>(X);
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int e = tid + u * kGqThreads, kc = e / g.Rp, c = e - kc * g.Rp;
                if (kc >= 8) continue;
#pragma unroll
                for (int q = 0; q < 8; q++) x[(8 * kc + q) * g.Rp + c] = v[u][q];
            }
            __syncthreads();
#pragma unroll
            for (int pass = 0; pass < 2; pass++)
#pragma unroll
                for (int q = 0; q < 16; q++) {
                    const int b = pass * kGqCols + grp * cpt + q;
                    if (pass < g.passes && q < cpt && a < R && b <= a) {
                        // the smaller column 2^600 larger where its products would be subnormal
                        const int lo = ecol[buf][a] <= ecol[buf][b] ? a : b, hi = a + b - lo;
                        const bool up = ecol[buf][lo] < 400;
                        double sum = 0.0;
                        for (int r = 0; r < nr; r++)
                            sum = fma(x[r * g.Rp + lo] * (up ? 0x1p600 : 1.0), x[r * g.Rp + hi], sum);
                        total[pass][q] = fma(sum, up ? 0x1p-600 : 1.0, total[pass][q]);
                    }
                }
            __syncthreads();
            continue;
        }
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int e = tid + u * kGqThreads, kc = e / g.Rp, c = e - kc * g.Rp;
            if (kc >= 8) continue;
            const int emax = ecol[buf][c];  // |x| < 2^(emax - 1022)
            uint32_t lo[8], hi[8];
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const long long t = fix56(v[u][q], emax) + 0x80808080808080ll;
                lo[q] = (uint32_t)t;
                hi[q] = (uint32_t)(t >> 32);
            }
            uint32_t o[kGqDigits][4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const uint32_t p = lo[2 * q], s = lo[2 * q + 1], ph = hi[2 * q], sh = hi[2 * q + 1];
                o[0][q] = pack_bf16(lead_f((int)ph >> 24), lead_f((int)sh >> 24));
                o[1][q] = pack_bf16(digit_f<0>(ph, 2), digit_f<0>(sh, 2));
                o[2][q] = pack_bf16(digit_f<0>(ph, 1), digit_f<0>(sh, 1));
                o[3][q] = pack_bf16(digit_f<0>(ph, 0), digit_f<0>(sh, 0));
                o[4][q] = pack_bf16(digit_f<0>(p, 3), digit_f<0>(s, 3));
                o[5][q] = pack_bf16(digit_f<0>(p, 2), digit_f<0>(s, 2));
                o[6][q] = pack_bf16(digit_f<0>(p, 1), digit_f<0>(s, 1));
                o[7][q] = pack_bf16(digit_f<0>(p, 0), digit_f<0>(s, 0));
            }
            unsigned char* dst = X + (uint32_t)(c >> 3) * 1024u + (uint32_t)kc * 128u + (uint32_t)(c & 7) * 16u;
#pragma unroll
            for (int d = 0; d < kGqDigits; d++)
                *reinterpret_cast<uint4*>(dst + d * g.digit) = make_uint4(o[d][0], o[d][1], o[d][2], o[d][3]);
        }
        fence_proxy_async_smem();
        tc_fence_before();
        __syncthreads();
#pragma unroll
        for (int pass = 0; pass < 2; pass++) {
            if (pass >= g.passes) break;
            const int b0 = pass * kGqCols, nb = min(g.nb, g.Rp - b0);
            if (tid == 0 && tile != withhold) {
                flight = true;
                tc_fence_after();
                const uint32_t idesc = umma_idesc_bf16(128, nb);
                for (int i = 0; i < kGqDigits; i++)
                    for (int d = 0; i + d < kGqDigits; d++)
                        for (int ks = 0; ks < kGqRows / 16; ks++)
                            umma_bf16(tmem + (uint32_t)((i + d) * kGqCols), umma_desc(X + i * g.digit + ks * 256, 128u, 1024u),
                                      umma_desc(X + d * g.digit + (uint32_t)(b0 >> 3) * 1024u + ks * 256, 128u, 1024u),
                                      idesc, (i > 0 || ks > 0) ? 1u : 0u);
                umma_commit(&bar);
            }
            if (mbar_wait_limited(&bar, phase, wait_polls)) {
                phase ^= 1u;
                flight = false;
            } else {
                lost = true;
            }
            tc_fence_after();
            const double sa = scale[a];
#pragma unroll
            for (int h = 0; h < 4; h++) {
                const int c0 = grp * cpt + 4 * h;  // four columns of this thread
                // only b <= a is kept (the same in a warp)
                if (4 * h < cpt && c0 < nb && (w & 3) * 32 < R && b0 + c0 <= (w & 3) * 32 + 31) {
                    uint32_t m[kGqDigits][4];
#pragma unroll
                    for (int s = 0; s < kGqDigits; s++)
                        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                                     : "=r"(m[s][0]), "=r"(m[s][1]), "=r"(m[s][2]), "=r"(m[s][3])
                                     : "r"(tmem + ((uint32_t)((w & 3) * 32) << 16) + (uint32_t)(s * kGqCols + c0))
                                     : "memory");
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int s = 0; s < kGqDigits; s++)
                        asm volatile("" : "+r"(m[s][0]), "+r"(m[s][1]), "+r"(m[s][2]), "+r"(m[s][3]));
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        int z[kGqDigits];
#pragma unroll
                        for (int s = 0; s < kGqDigits; s++) z[s] = __float2int_rn(__uint_as_float(m[s][q]));
                        const long long high = ((long long)z[0] * 65536 + ((long long)z[1] * 256 + z[2])) * 256 + z[3];
                        const long long low = ((long long)z[4] * 65536 + ((long long)z[5] * 256 + z[6])) * 256 + z[7];
                        const long long V = (high << 20) + (low >> 12);
                        total[pass][4 * h + q] = fma((double)V * sa, scale[b0 + c0 + q], total[pass][4 * h + q]);
                    }
                }
            }
            tc_fence_before();
            dead = __syncthreads_or(lost);  // the accumulators, the digits and the scales are read
            if (dead) break;
        }
        if (dead) break;
    }
    if (dead) {
        if (tid == 0) {
            report(status, EXAFAC_ERR_TIMEOUT, 26, blockIdx.x, 0);
            if (flight) mbar_wait_limited(&bar, phase, kSpinLimit);
        }
    }
#pragma unroll
    for (int pass = 0; pass < 2; pass++)
#pragma unroll
        for (int q = 0; q < 16; q++) {
            const int b = pass * kGqCols + grp * cpt + q;
            if (pass < g.passes && q < cpt && a < R && b <= a)
                part[(int64_t)blockIdx.x * packed_size(R) + packed_index(R, b, a)] = total[pass][q];
        }
    tc_fence_before();
    __syncthreads();
    if (w == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

// A tile takes ~12 us whatever its columns (the latencies of its phases, one
// after the other); in FP64 its 64 rows take R (R + 1) / 2 FMAs each.  R = 25, J =
// 65536: 88 us either way; R = 45, J = 50001: 155 -> 78 us.
bool design_digits_wanted(int R, int64_t J) { return R > 32 && J * (int64_t)packed_size(R) >= (1ll << 22); }

// *nblk partial sums in s.part for gram_reduce_kernel.
int design_gram_digits(Session& s, int n, int64_t J, int64_t* nblk, cudaStream_t st) {
    FactorPtrs f;
    for (int k = 0; k < kMaxModes; k++) f.U[k] = k < s.N ? s.F.U[k] : nullptr;
    const size_t smem = gq_smem(s.R);
    EXAFAC_CUDA_TRY(allow_smem(design_digits_kernel));
    *nblk = std::max<int64_t>(1, std::min<int64_t>(ceil_div(J, kGqRows), 152));
    design_digits_kernel<<<(unsigned)*nblk, kGqThreads, smem, st>>>(s.N, n, s.R, s.counters + 0, s.sd, s.wd, f, s.D, s.part,
                                                                    s.status, s.wait_polls ? s.wait_polls : kSpinLimit,
                                                                    s.withheld(26));
    count_launch();
    EXAFAC_CHECK_LAUNCH();
    return EXAFAC_OK;
}

}  // namespace exafac
