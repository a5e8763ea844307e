// STS-CP draws of the FP64 form, breadth first on the tensor cores
// (STS_CP::KRPDrawSamples, sts_cp.hpp:203-300, and PartitionTree::PTSample,
// partition_tree.hpp:204-380, at one rank), with the decisions of the
// depth-first FP64 kernel (sts_draw_kernel<double>).
//
// The depth-first kernel evaluates every node mass x^T G x in FP64, about
// R^2 / 2 FMAs each on a pipe that retires ~1.7 of them per clock per SM: 66 to
// 82 % of an FP64 sweep.  A descent only uses a mass to decide d <= low + m_L
// / m, so here the masses are formed from bf16 digits on the tensor cores
// with an error that is bounded in advance, every decision whose distance
// from its cutoff is within the bound (of both evaluations) marks its sample,
// and the marked samples are drawn again, whole, by the depth-first kernel.
// The others took the same branch at every node, so their rows are the same.
// Their weights come from the same kind of products with enough digits to be
// below FP64's rounding (zq_weight_kernel).
//
// Digits.  A vector x (scaled by a power of two to |x'| < 2^6) is held in
// fixed point (units of 2^-47, int64) and cut into balanced base-256 digits:
// x' = x0 + xr, x0 = d0 + d1 2^-8 + d2 2^-16 + d3 2^-24, |xr| <= 2^-25; a node
// (scaled by its tree's root diagonal, |A'| < 2^6) into six digits, the
// remainder |Ar| <= 2^-41.  A digit has at most 8 significant bits, so d_i
// 2^-8i is a bf16 value, a product of two digits and a sum of R <= 128 of
// them per weight 2^-8s, s = i + j, are integers below 2^24 in that unit: the
// FP32 accumulators of the tensor core hold every weight's sum exactly.  Per
// 32 columns of the node and digit i of x, one MMA multiplies the stacked
// node digits 0 .. 5 - i, whose results land on the accumulators of the
// weights s = i .. 5.  With Y = x0 A (weights <= 5) the mass is
//   q = sum_c Y_c (x0 + 2 xr)_c = x'^T A' x' - xr^T A' xr - (dropped weights),
// the dot product in integers (GB300's FP64 pipe would take longer over it
// than the tensor cores over the products).
//
// Error, in the scaled units (n1 = sum |x'_c|):
//   dropped digits and remainders: |Y_c| error <= R 3.7 2^-34
//   FP32 add of the weights 4 and 5 and its rounding to 2^-31: <= 1.5 2^-32
//   xr^T A' xr <= R^2 2^-44
//   the depth-first kernel's own rounding: <= 40 2^-53 |x'|^T |A'| |x'|
//                                         <= n1 R 0.31 2^-34
//   E = n1 (R 4.6 2^-34 + 1.7 2^-32) + R^2 2^-44
// A cutoff low + q / m is then off by at most E / m for the root mass, E / m
// for its own mass and E / m per earlier right turn.  The leaf's row is picked
// from FP32 squares of dots with 30-bit x, with its own bound (zq_leaf_kernel),
// and from FP64 dots where that bound leaves it open (zq_place_kernel).
//
// Measured (GB300), draws of a step: R = 64, J = 2^18, three 2000-row modes:
// 55.8 -> 4.1 ms; R = 25, J = 65536: 4.3 -> 0.8 ms.
#include "digits.cuh"
#include "engine.cuh"
#include "prims.cuh"
#include "umma.cuh"
#include "zq.cuh"

namespace exafac {

constexpr int kZTile = 128;  // slots per tile (the MMA's M)
constexpr int kZx = 4;       // digits of x
constexpr int kZa = 6;       // digits of a node entry
constexpr int kZu = 4;       // digits of a leaf row's entry
constexpr int kZCols = 32;   // node columns (leaf rows) per chunk
constexpr int64_t kZPrefSmem = 16384;  // tiles whose prefix fits in shared memory

struct ZShape {
    int Rk, nch;                 // K padded to 16, chunks of kZCols columns
    uint32_t sbo, xs, bs;        // bytes of 8 rows, of one x digit (128 rows), of one chunk digit (32 rows)
};
__host__ __device__ inline ZShape z_shape(int R) {
    ZShape z;
    z.Rk = (R + 15) & ~15;
    z.nch = (R + kZCols - 1) / kZCols;
    z.sbo = (uint32_t)z.Rk * 16u;
    z.xs = 16u * z.sbo;
    z.bs = 4u * z.sbo;
    return z;
}
static size_t z_smem(int R, int digits) {
    const ZShape z = z_shape(R);
    return (size_t)kZx * z.xs + (size_t)digits * z.bs + 128;
}

// Waits for the loads above; the registers pass through so that no use of
// them moves before the wait.
template <int S>
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[S][8]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int s = 0; s < S; s++)
        asm volatile("" : "+r"(r[s][0]), "+r"(r[s][1]), "+r"(r[s][2]), "+r"(r[s][3]), "+r"(r[s][4]), "+r"(r[s][5]),
                     "+r"(r[s][6]), "+r"(r[s][7]));
}

// v 2^(52 - (emax - 1023)) cut to an integer (toward zero): with |v| < 2^(emax
// - 1022) this is v', scaled to below 2^6, in units of 2^-47.
__device__ __forceinline__ long long fix47(double v, int emax) {
    const long long b = __double_as_longlong(v);
    const int e = (int)((b >> 52) & 0x7ff);
    unsigned long long m = (unsigned long long)b & 0xfffffffffffffull;
    if (e) m |= 1ull << 52;
    const int s = max(max(emax, 1) - max(e, 1), 0);
    m = s > 63 ? 0ull : m >> s;
    return b < 0 ? -(long long)m : (long long)m;
}

// The same rounded to nearest (the vectors: their weights take the mass to
// FP64's own accuracy).
__device__ __forceinline__ long long fix47_rn(double v, int emax) {
    const long long b = __double_as_longlong(v);
    const int e = (int)((b >> 52) & 0x7ff);
    unsigned long long m = (unsigned long long)b & 0xfffffffffffffull;
    if (e) m |= 1ull << 52;
    const int s = max(max(emax, 1) - max(e, 1), 0);
    m = s > 60 ? 0ull : (s > 0 ? (m + (1ull << (s - 1))) >> s : m);
    return b < 0 ? -(long long)m : (long long)m;
}

// What fix47_rn leaves off v, in 256ths of its unit: the eight bits below the
// last one, as a signed number where they rounded it up (rounded themselves).
__device__ __forceinline__ int fix47_rest(double v, int emax) {
    const long long b = __double_as_longlong(v);
    const int e = (int)((b >> 52) & 0x7ff);
    unsigned long long m = (unsigned long long)b & 0xfffffffffffffull;
    if (e) m |= 1ull << 52;
    const int s = max(max(emax, 1) - max(e, 1), 0);
    const uint32_t f = s >= 32 ? (s < 96 ? (uint32_t)(m >> (s - 32)) : 0u) : (uint32_t)(m << (32 - s));
    const int r = min(((int)f >> 24) + (int)((f >> 23) & 1u), 127);
    return b < 0 ? -r : r;
}

// Rows of the fixed-point vectors are padded with zeros to a multiple of 4
// (32 bytes), so that a thread's eight values are two 32-byte loads: with
// 8-byte loads of 32 different rows the level kernel took 3.3 times the
// sectors from L2.
__host__ __device__ __forceinline__ int z_row(int R) { return (R + 3) & ~3; }
__device__ __forceinline__ void load_x4(const long long* p, long long (&v)[8], int at) {
    asm volatile("ld.global.v4.b64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(v[at]), "=l"(v[at + 1]), "=l"(v[at + 2]), "=l"(v[at + 3])
                 : "l"(p));
}
__device__ __forceinline__ void load_x8(const long long* row, int k, int Rx, bool live, long long (&v)[8]) {
#pragma unroll
    for (int h = 0; h < 8; h += 4) {
        if (live && k + h < Rx) {
            load_x4(row + k + h, v, h);
        } else {
#pragma unroll
            for (int q = 0; q < 4; q++) v[h + q] = 0ll;
        }
    }
}

// A fixed-point entry X is kept as its rounding z4 to multiples of 2^23 (low
// word; the four digits) and the rest, |xr| <= 2^22 (high word): X = 2^23 z4 +
// xr.  Every level reads the entries and none needs 64-bit arithmetic.
__device__ __forceinline__ long long pack_x(long long X) {
    const int z4 = (int)((X + (1ll << 22)) >> 23);
    const int xr = (int)((unsigned)X - ((unsigned)z4 << 23));
    return (long long)(((unsigned long long)(unsigned)xr << 32) | (unsigned)z4);
}
__device__ __forceinline__ int x_z4(long long x) { return (int)x; }
__device__ __forceinline__ int x_rest(long long x) { return (int)(x >> 32); }

// The four digits of eight x values into the slices of the operand, 16 bytes
// each.
__device__ __forceinline__ void store_x_digits(unsigned char* dst, uint32_t xs, const long long (&X)[8]) {
    uint32_t t[8];
#pragma unroll
    for (int q = 0; q < 8; q++) t[q] = (uint32_t)x_z4(X[q]) + 0x808080u;
    uint32_t o[kZx][4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const uint32_t a = t[2 * q], b = t[2 * q + 1];
        o[0][q] = pack_bf16(lead_f((int)a >> 24), lead_f((int)b >> 24));
        o[1][q] = pack_bf16(digit_f<1>(a, 2), digit_f<1>(b, 2));
        o[2][q] = pack_bf16(digit_f<2>(a, 1), digit_f<2>(b, 1));
        o[3][q] = pack_bf16(digit_f<3>(a, 0), digit_f<3>(b, 0));
    }
#pragma unroll
    for (int d = 0; d < kZx; d++)
        *reinterpret_cast<uint4*>(dst + d * xs) = make_uint4(o[d][0], o[d][1], o[d][2], o[d][3]);
}

// The digits of eight node entries (DG = 6: units down to 2^-40; 4: 2^-24).
template <int DG>
__device__ __forceinline__ void store_a_digits(unsigned char* dst, uint32_t bs, const double (&v)[8], int emax) {
    uint32_t lo[8];
    int hi[8];  // DG = 6: byte 4 of the biased value and the leading digit above it
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const long long f = fix47(v[q], emax);
        if (DG == 6) {
            const long long t = ((f + 64) >> 7) + 0x8080808080ll;
            lo[q] = (uint32_t)t;
            hi[q] = (int)(t >> 32);
        } else {
            lo[q] = (uint32_t)(int)((f + (1ll << 22)) >> 23) + 0x808080u;
            hi[q] = 0;
        }
    }
    uint32_t o[DG][4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const uint32_t a = lo[2 * q], b = lo[2 * q + 1];
        const int ah = hi[2 * q], bh = hi[2 * q + 1];
        if (DG == 6) {
            o[0][q] = pack_bf16(lead_f(ah >> 8), lead_f(bh >> 8));
            o[1][q] = pack_bf16(digit_f<1>((uint32_t)ah, 0), digit_f<1>((uint32_t)bh, 0));
            o[2][q] = pack_bf16(digit_f<2>(a, 3), digit_f<2>(b, 3));
            o[3][q] = pack_bf16(digit_f<3>(a, 2), digit_f<3>(b, 2));
            o[DG - 2][q] = pack_bf16(digit_f<4>(a, 1), digit_f<4>(b, 1));
            o[DG - 1][q] = pack_bf16(digit_f<5>(a, 0), digit_f<5>(b, 0));
        } else {
            o[0][q] = pack_bf16(lead_f((int)a >> 24), lead_f((int)b >> 24));
            o[1][q] = pack_bf16(digit_f<1>(a, 2), digit_f<1>(b, 2));
            o[2][q] = pack_bf16(digit_f<2>(a, 1), digit_f<2>(b, 1));
            o[3][q] = pack_bf16(digit_f<3>(a, 0), digit_f<3>(b, 0));
        }
    }
#pragma unroll
    for (int d = 0; d < DG; d++)
        *reinterpret_cast<uint4*>(dst + d * bs) = make_uint4(o[d][0], o[d][1], o[d][2], o[d][3]);
}

// The tile's vectors xi[js[r]] as the A operand: rows past n and columns past
// R zero.  The row runs fastest over the threads (conflict-free stores).
__device__ __forceinline__ void stage_x(unsigned char* A, const long long* __restrict__ xi, const int32_t* js, int n,
                                        int R, const ZShape& z) {
    // lanes: eight rows, four 64-byte pieces of each (half the cache lines per
    // load of a row per lane, the same conflict-free stores)
    const int k8s = z.Rk / 8, quads = (k8s + 3) / 4, lane = threadIdx.x & 31;
    for (int q = threadIdx.x >> 5; q < (kZTile / 8) * quads; q += blockDim.x >> 5) {
        const int r = 8 * (q & (kZTile / 8 - 1)) + (lane & 7), k8 = 4 * (q / (kZTile / 8)) + (lane >> 3);
        if (k8 >= k8s) continue;
        long long X[8];
        load_x8(xi + (int64_t)js[r < n ? r : 0] * z_row(R), 8 * k8, z_row(R), r < n, X);
        store_x_digits(A + (uint32_t)(r >> 3) * z.sbo + (uint32_t)k8 * 128u + (uint32_t)(r & 7) * 16u, z.xs, X);
    }
}

// Columns 32 ch .. + 31 of the packed node g as the B operand (digit j of
// column c in row 32 j + c).
__device__ __forceinline__ void expand_node(unsigned char* B, const double* __restrict__ g, const int* rs, int ch,
                                            int R, int emax, const ZShape& z) {
    const int total = kZCols * (z.Rk / 8);
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
        const int c = e & (kZCols - 1), k = 8 * (e / kZCols);
        const int col = ch * kZCols + c;
        double v[8];
        const int rc = col < R ? rs[col] : 0;
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const int kk = k + q;
            v[q] = (col < R && kk < R) ? __ldg(g + (kk >= col ? rc + (kk - col) : rs[kk] + (col - kk))) : 0.0;
        }
        store_a_digits<kZa>(B + (uint32_t)(c >> 3) * z.sbo + (uint32_t)(k >> 3) * 128u + (uint32_t)(c & 7) * 16u, z.bs,
                            v, emax);
    }
}

// One chunk of a node's B operand in global memory, for bulk copies: eight
// entries per item.
__host__ __device__ __forceinline__ uint32_t z_chunk_bytes(const ZShape& z) { return kZa * z.bs; }
__device__ __forceinline__ void expand_item(unsigned char* B, const double* __restrict__ g, int ch, int item, int R,
                                            int emax, const ZShape& z) {
    const int c = item & (kZCols - 1), k = 8 * (item / kZCols);
    const int col = ch * kZCols + c;
    double v[8];
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const int kk = k + q;
        v[q] = (col < R && kk < R) ? __ldg(g + packed_index(R, min(kk, col), max(kk, col))) : 0.0;
    }
    store_a_digits<kZa>(B + (uint32_t)(c >> 3) * z.sbo + (uint32_t)(k >> 3) * 128u + (uint32_t)(c & 7) * 16u, z.bs, v,
                        emax);
}

// Rows 32 ch .. + 31 of a leaf (its first rows live, else zero) as the B operand.
__device__ __forceinline__ void expand_rows(unsigned char* B, const double* __restrict__ Ub, int ch, int rows, int R,
                                            int emax, const ZShape& z) {
    const int total = kZCols * (z.Rk / 8);
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
        const int c = e & (kZCols - 1), k = 8 * (e / kZCols);
        const int r = ch * kZCols + c;
        double v[8];
#pragma unroll
        for (int q = 0; q < 8; q++) v[q] = (r < rows && k + q < R) ? __ldg(Ub + (int64_t)r * R + k + q) : 0.0;
        store_a_digits<kZu>(B + (uint32_t)(c >> 3) * z.sbo + (uint32_t)(k >> 3) * 128u + (uint32_t)(c & 7) * 16u, z.bs,
                            v, emax);
    }
}

// One chunk's products, by one thread: weights s = i + j < DG in the TMEM
// columns 32 s ..
template <int DG>
__device__ __forceinline__ void issue_chunk(uint32_t tmem, const unsigned char* A, const unsigned char* B,
                                            const ZShape& z, uint64_t* bar) {
    tc_fence_after();
#pragma unroll
    for (int i = 0; i < kZx; i++) {
        const uint32_t idesc = umma_idesc_bf16(kZTile, kZCols * (DG - i));
        for (int ks = 0; ks < z.Rk / 16; ks++)
            umma_bf16(tmem + (uint32_t)(kZCols * i), umma_desc(A + i * z.xs + ks * 256, 128u, z.sbo),
                      umma_desc(B + ks * 256, 128u, z.sbo), idesc, (i > 0 || ks > 0) ? 1u : 0u);
    }
    umma_commit(bar);
}

// Marks sample j for the depth-first kernel (once).
__device__ __forceinline__ void z_mark(int32_t* redo, int32_t* list, int32_t* count, int32_t j) {
    if (atomicExch(redo + j, 1) == 0) list[atomicAdd(count, 1)] = j;
}

// A wait of this draw ran out (ZState::lost): the draw's later kernels return
// at once, every sample that is not drawn yet takes row 0 and no weight.  The
// caller sees EXAFAC_ERR_TIMEOUT.  Every thread of the block calls.
__device__ __forceinline__ bool z_lost(const ZState& b) {
    return __syncthreads_or(threadIdx.x == 0 && *reinterpret_cast<volatile int32_t*>(b.lost) != 0);
}

// E of the header, in the scaled units.
__device__ __forceinline__ double z_bound(float n1, int R) {
    return (double)n1 * ((double)R * 4.6 * 0x1p-34 + 1.7 * 0x1p-32) + (double)R * (double)R * 0x1p-44;
}

// The block's share of a level's runs.  A run (consecutive slots of one tile
// at the same node) costs its node's expansion and products whatever its
// length, and the runs are spread unevenly over the tiles (skewed modes: the
// tiles of the rare rows hold up to 128), so every block takes the same number
// of runs: runs [first, first + count) in slot order, found from the tiles'
// run starts (a bit per slot, ZState::runs).  With equal numbers of tiles the
// slowest block took 3.9 ms on a tail level of a Zipf mode, with equal numbers
// of runs 0.2 ms.  A tile's runs may belong to several blocks, in any order of
// time: a block takes the starts from the bits, which no level changes, and
// reads and writes the nodes of its own slots only.
struct ZShare {
    int64_t tile;   // first tile
    int run;        // first run within it
    int64_t count;  // runs
};
template <int NT>
__device__ __forceinline__ ZShare z_share(const uint32_t* __restrict__ runs, int64_t ntiles) {
    __shared__ long long wsum[NT / 32];
    __shared__ long long found[2];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int64_t per = (ntiles + NT - 1) / NT;
    const int64_t a = min(ntiles, per * tid), e = min(ntiles, a + per);
    auto count = [&](int64_t q) {
        const uint4 m = __ldg(reinterpret_cast<const uint4*>(runs) + q);
        return 1 + (__popc(m.x) + __popc(m.y)) + (__popc(m.z) + __popc(m.w));
    };
    long long sum = 0;
    for (int64_t q = a; q < e; q++) sum += count(q);
    long long inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
    }
    if (lane == 31) wsum[w] = inc;
    if (tid == 0) {
        found[0] = ntiles;
        found[1] = 0;
    }
    __syncthreads();
    long long before = inc - sum, total = 0;
    for (int q = 0; q < NT / 32; q++) {
        if (q < w) before += wsum[q];
        total += wsum[q];
    }
    const long long first = total * blockIdx.x / gridDim.x, last = total * (blockIdx.x + 1) / gridDim.x;
    if (first >= before && first < before + sum) {
        long long at = before;
        for (int64_t q = a; q < e; q++) {
            const long long r = count(q);
            if (first < at + r) {
                found[0] = q;
                found[1] = first - at;
                break;
            }
            at += r;
        }
    }
    __syncthreads();
    ZShare s;
    s.tile = found[0];
    s.run = (int)found[1];
    s.count = last - first;
    return s;
}

// The end of the run that slot i0 belongs to, from the tile's run starts.
__device__ __forceinline__ int z_run_end(const uint32_t* rmask, int i0, int n) {
    for (int q = (i0 + 1) >> 5; q < 4; q++) {
        uint32_t bits = rmask[q];
        if (q == ((i0 + 1) >> 5)) bits &= ~0u << ((i0 + 1) & 31);
        if (bits) return min(n, (q << 5) + __ffs(bits) - 1);
    }
    return n;
}
// The block's slots [first, last) of the tile: `count` runs from run `run` on.
__device__ __forceinline__ int2 z_run_slots(const uint32_t* rmask, int run, int64_t count, int n) {
    int first = 0;
    for (int q = 0; q < run && first < n; q++) first = z_run_end(rmask, first, n);
    const int all = 1 + (__popc(rmask[0]) + __popc(rmask[1])) + (__popc(rmask[2]) + __popc(rmask[3]));
    int last = n;
    if (count < all - run) {
        last = first;
        for (int64_t q = 0; q < count; q++) last = z_run_end(rmask, last, n);
    }
    return make_int2(first, last);
}

// One chunk's read-back, columns c0 .. c0 + 7 of the node: the five integer
// sums of Y_c (x0 + 2 xr)_c.
struct ZSums {
    long long Ph, Pl, Qh, Ql, V;
};
__device__ __forceinline__ void z_dot8(uint32_t taddr, const long long* xrow, int c0, int Rx, ZSums& s) {
    uint32_t a[kZa][8];
#pragma unroll
    for (int q = 0; q < kZa; q++) tmem_ld8_nowait(taddr + (uint32_t)(kZCols * q), a[q]);
    long long X[8];
    load_x8(xrow, c0, Rx, true, X);
    tmem_ld_wait<kZa>(a);
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const float a0 = __uint_as_float(a[0][q]), a1 = __uint_as_float(a[1][q]), a2 = __uint_as_float(a[2][q]),
                    a3 = __uint_as_float(a[3][q]), a4 = __uint_as_float(a[4][q]), a5 = __uint_as_float(a[5][q]);
        // the weights' integers, by adding a power of two whose ulp is the
        // unit: n0 (1), n1 (2^-8), n2 (2^-16), and weight 3 (2^-24) as a
        // multiple of 2^-23 and a rest
        const int m0 = __float_as_int(a0 + 12582912.0f) - 0x4B400000;
        const int m1 = __float_as_int(a1 + 49152.0f) - 0x47400000;
        const int m2 = __float_as_int(a2 + 192.0f) - 0x43400000;
        const float f3 = a3 + 1.5f;
        const int m3 = __float_as_int(f3) - 0x3FC00000;
        const float v = (a3 - (f3 - 1.5f)) + (a4 + a5);
        const int V = __float_as_int(v + 0.005859375f) - 0x3BC00000;  // units of 2^-31
        const int Pn = m0 * 256 + m1;                                  // units of 2^-8
        const int Qn = m2 * 128 + m3;                                  // units of 2^-23
        // x0 + 2 xr = 2^27 wh + wl
        const int z4 = x_z4(X[q]), wh = z4 >> 4, wl = ((z4 & 15) << 23) + 2 * x_rest(X[q]);
        s.Ph += (long long)Pn * wh;
        s.Pl += (long long)Pn * wl;
        s.Qh += (long long)Qn * wh;
        s.Ql += (long long)Qn * wl;
        s.V += (long long)V * wh;
    }
}

// MODE 0: the root's mass of every sample (slot s holds sample s).
// MODE 1: a level: the left child's mass and the branch.
// MODE 2: the tail level: as MODE 1; samples already at a leaf stay.
// The branch flags of a tile's slots are set in mask[p], their count added to
// tcount[p] (both zero before); runs[p] holds the tiles' run starts, runs[p ^ 1]
// is cleared for the partition that follows.
// NT = 512 (R > 64, one block per SM): a chunk's products run beside the
// previous chunk's read-back (two accumulator sets), and beside the next
// chunk's expansion when a second node buffer fits (nb = 2).
// nodes != null (R > 32, two chunks or more): the operands of the level's left
// children (of the root: MODE 0), node by node in z_chunk_bytes chunks
// (zq_partition_kernel has expanded them; lb the parents' first index), brought
// by bulk copies, the first one of a run ahead of its use; null: each run
// expands its node here.
// A run's sums are kept and a tile's masses and branches formed together: an
// SM takes an FP64 instruction per 19 clocks whatever its active lanes, and
// the ~14 of them per run cost as much as the products on levels with short
// runs.
template <int MODE, int NT>
__global__ void __launch_bounds__(NT, NT == 256 ? 2 : 1)
    zq_level_kernel(int R, int nb, TreeShape t, const double* __restrict__ G, const unsigned char* __restrict__ nodes,
                    int64_t lb, const int32_t* __restrict__ tree_exp, int64_t J, ZState b, int p,
                    const int32_t* __restrict__ order, const double* __restrict__ dv, DeviceStatus* status,
                    uint32_t wait_polls, int64_t withhold) {
    extern __shared__ __align__(128) unsigned char z_raw[];
    if (z_lost(b)) return;
    constexpr int NG = NT / 128;        // threads per slot in the read-back
    constexpr int CPT = kZCols / NG;    // columns of a chunk per thread
    constexpr bool kPipe = NT == 512;
    constexpr uint32_t kTmem = kPipe ? 512 : 256;
    __shared__ int32_t cs[kZTile], js[kZTile];
    __shared__ uint32_t rmask[4];
    __shared__ long long part[NG][5][kZTile];
    __shared__ int rs[kMaxRank];
    __shared__ __align__(8) uint64_t bars[2];    // products
    __shared__ __align__(8) uint64_t copied[2];  // node buffers
    __shared__ uint32_t tmem_base;
    const ZShape z = z_shape(R);
    const int Rx = z_row(R);
    unsigned char* A = z_raw + ((128u - (smem_u32(z_raw) & 127u)) & 127u);
    unsigned char* Bb[2] = {A + kZx * z.xs, A + kZx * z.xs + (nb - 1) * kZa * z.bs};
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const int P = packed_size(R);
    const bool pre = nodes != nullptr;
    const uint32_t cbytes = z_chunk_bytes(z);
    if (w == 0) tmem_alloc(&tmem_base, kTmem);
    for (int a = tid; a < R; a += NT) rs[a] = packed_index(R, a, a);
    if (tid == 0) {
        for (int q = 0; q < 2; q++) {
            mbar_init(&bars[q], 1);
            mbar_init(&copied[q], 1);
        }
        fence_mbar_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    const int emax = *tree_exp;
    uint32_t phase[2] = {0, 0}, cphase[2] = {0, 0};
    bool lost = false;     // a wait of this thread ran out
    uint32_t flight = 0;   // thread 0: bit q a copy into buffer q, bit 2 + q products of set q
    int64_t resident = -1; // the node B holds (one-chunk ranks)
    bool aborted = false;
    const int row = (w & 3) * 32 + lane, grp = w >> 2;
    const uint32_t lane_base = tmem + ((uint32_t)((w & 3) * 32) << 16);
    const int64_t ntiles = (J + kZTile - 1) / kZTile;
    ZShare sh;
    if (MODE == 0) {
        sh.tile = ntiles * blockIdx.x / gridDim.x;
        sh.run = 0;
        sh.count = ntiles * (blockIdx.x + 1) / gridDim.x - sh.tile;
    } else {
        sh = z_share<NT>(b.runs[p], ntiles);
        for (int64_t q = (int64_t)blockIdx.x * NT + tid; q < ntiles; q += (int64_t)gridDim.x * NT)
            reinterpret_cast<uint4*>(b.runs[p ^ 1])[q] = make_uint4(0u, 0u, 0u, 0u);
    }
    const bool ok = emax < 2047;  // a tree with a non-finite root: every sample is marked at the root
    // the chunk's products are done (every thread)
    auto wait = [&](int q) {
        if (mbar_wait_limited(&bars[q], phase[q], wait_polls)) {
            phase[q] ^= 1u;
            flight &= ~(4u << q);
        } else {
            lost = true;
        }
        tc_fence_after();
    };
    // thread 0: chunk ch of the left child of parent c into buffer q; the products of buffer q's
    // chunk into accumulator set `set`, after its copy (fresh).  Nothing more once a wait ran out
    // (the others' waits run out as well), nor for the tile of the wait-limit test hook.
    auto fetch = [&](int q, int32_t c, int ch) {
        if (lost) return;
        flight |= 1u << q;
        const int64_t slot = MODE == 0 ? 0 : (int64_t)c - lb;
        mbar_arrive_expect_tx(&copied[q], cbytes);
        bulk_g2s(Bb[q], nodes + (slot * z.nch + ch) * cbytes, cbytes, &copied[q]);
    };
    auto issue = [&](int q, int set, bool fresh) {
        if (lost) return;
        if (fresh) {
            if (!mbar_wait_limited(&copied[q], cphase[q], wait_polls)) {
                lost = true;
                return;
            }
            cphase[q] ^= 1u;
            flight &= ~(1u << q);
        }
        if (sh.tile == withhold) return;
        flight |= 4u << set;
        issue_chunk<kZa>(tmem + (uint32_t)(set * 256), A, Bb[q], z, &bars[set]);
    };
    // the chunk's columns of this thread
    auto dots = [&](uint32_t acc, const long long* xrow, int ch, ZSums& sum) {
#pragma unroll
        for (int h = 0; h < CPT / 8; h++) z_dot8(acc + 8 * h, xrow, ch * kZCols + grp * CPT + 8 * h, Rx, sum);
    };
    auto stays = [&](int32_t c) { return MODE == 2 && tree_is_leaf(t, c); };
    for (; sh.count > 0 && sh.tile < ntiles; sh.tile++, sh.run = 0) {
        const int64_t s0 = sh.tile * kZTile;
        const int n = (int)min((int64_t)kZTile, J - s0);
        double low = 0.0, rinv = 0.0, d = 0.0;
        float2 er = make_float2(0.f, 0.f);
        float e0 = 0.f, n1 = 0.f;
        int ex = 0;
        int flag = -1;  // -1: not this block's, 0 right, 1 left (or stays), 2 summed
        if (tid < 4) rmask[tid] = MODE == 0 ? 0u : b.runs[p][4 * sh.tile + tid];
        __syncthreads();
        const int2 own = z_run_slots(rmask, sh.run, sh.count, n);
        int i0 = own.x;
        if (tid < kZTile) {
            int32_t j = 0, c = -1;
            if (tid < n) j = order ? order[s0 + tid] : (int32_t)(s0 + tid);
            if (tid >= own.x && tid < own.y) {
                c = MODE == 0 ? 0 : (int32_t)b.node[j];
                ex = b.ex[j];
                n1 = b.n1[j];
                if (MODE != 0) {
                    low = b.lh[j].x;
                    rinv = b.rinv[j];
                    er = b.err[j];
                    e0 = b.e0[j];
                    d = dv[j];
                }
            }
            js[tid] = j;
            cs[tid] = c;
        }
        __syncthreads();
        bool ahead = false;  // the next run's first chunk is on its way
        if (pre && i0 < own.y && !stays(cs[i0])) {
            if (tid == 0) fetch(0, cs[i0], 0);
            ahead = true;
        }
        stage_x(A, reinterpret_cast<const long long*>(b.xi), js, n, R, z);
        fence_proxy_async_smem();
        tc_fence_before();
        __syncthreads();
        for (; i0 < own.y; sh.count--) {  // runs of equal node (uniform over the block)
            const int32_t c = cs[i0];
            const int i1 = z_run_end(rmask, i0, n);
            if (stays(c)) {
                if (tid >= i0 && tid < i1) flag = 1;
                i0 = i1;
                continue;
            }
            ZSums sum = {0, 0, 0, 0, 0};
            const long long* xrow = reinterpret_cast<const long long*>(b.xi) + (int64_t)js[row < n ? row : 0] * Rx;
            if (pre) {
                if (tid == 0) {
                    if (!ahead) fetch(0, c, 0);
                    if (nb == 2) fetch(1, c, 1);
                    issue(0, 0, true);
                }
                ahead = false;
                for (int ch = 0; ch < z.nch; ch++) {
                    const int cur = kPipe ? ch & 1 : 0;
                    const bool more = ch + 1 < z.nch;
                    const uint32_t acc = lane_base + (uint32_t)(cur * 256 + grp * CPT);
                    if (kPipe && nb == 2 && more && tid == 0) issue((ch + 1) & 1, cur ^ 1, true);
                    wait(cur);
                    if (more) {
                        if (tid == 0) {
                            if (kPipe && nb == 2) {
                                if (ch + 2 < z.nch) fetch(ch & 1, c, ch + 2);
                            } else {
                                fetch(0, c, ch + 1);
                                if (kPipe) issue(0, cur ^ 1, true);
                            }
                        }
                    } else if (i1 < own.y && !stays(cs[i1])) {
                        if (tid == 0) fetch(0, cs[i1], 0);
                        ahead = true;
                    }
                    dots(acc, xrow, ch, sum);
                    if (more) {  // the accumulators are read
                        tc_fence_before();
                        __syncthreads();
                        if (!kPipe && tid == 0) issue(0, 0, true);
                    }
                }
            } else {
                const int64_t g = MODE == 0 ? 0 : 2 * (int64_t)c + 1;
                if (resident != c || z.nch > 1) expand_node(Bb[0], G + g * P, rs, 0, R, emax, z);
                resident = c;
                fence_proxy_async_smem();
                tc_fence_before();
                __syncthreads();
                if (tid == 0) issue(0, 0, false);
                for (int ch = 0; ch < z.nch; ch++) {
                    const int cur = kPipe ? ch & 1 : 0;
                    const bool more = ch + 1 < z.nch;
                    const uint32_t acc = lane_base + (uint32_t)(cur * 256 + grp * CPT);
                    if (kPipe) {
                        if (more) {
                            if (nb == 1) wait(cur);
                            expand_node(Bb[(ch + 1) & (nb - 1)], G + g * P, rs, ch + 1, R, emax, z);
                            fence_proxy_async_smem();
                            tc_fence_before();
                            __syncthreads();
                            if (tid == 0) issue((ch + 1) & (nb - 1), cur ^ 1, false);
                        }
                        if (nb == 2 || !more) wait(cur);
                        dots(acc, xrow, ch, sum);
                    } else {
                        wait(0);
                        dots(acc, xrow, ch, sum);
                        if (more) {
                            expand_node(Bb[0], G + g * P, rs, ch + 1, R, emax, z);
                            fence_proxy_async_smem();
                            tc_fence_before();
                            __syncthreads();
                            if (tid == 0) issue(0, 0, false);
                        }
                    }
                }
            }
            if (row >= i0 && row < i1) {
                part[grp][0][row] = sum.Ph;
                part[grp][1][row] = sum.Pl;
                part[grp][2][row] = sum.Qh;
                part[grp][3][row] = sum.Ql;
                part[grp][4][row] = sum.V;
            }
            if (tid >= i0 && tid < i1) flag = 2;
            tc_fence_before();
            // part, and the accumulators and node buffers for the next run
            if (__syncthreads_or(lost)) {
                aborted = true;
                break;
            }
            i0 = i1;
        }
        if (aborted) break;
        // runs that stay take no barrier: everyone is done with cs before the next tile's replaces it
        if (MODE == 2) __syncthreads();
        if (tid < kZTile && flag == 2) {
            long long s5[5];
#pragma unroll
            for (int u = 0; u < 5; u++) {
                s5[u] = part[0][u][tid];
#pragma unroll
                for (int gq = 1; gq < NG; gq++) s5[u] += part[gq][u][tid];
            }
            // weights: P 2^-8, Q 2^-23, V 2^-31; wh 2^-20, wl 2^-47
            const double q = (double)s5[0] * 0x1p-28 + (double)s5[1] * 0x1p-55 + (double)s5[2] * 0x1p-43 +
                             (double)s5[3] * 0x1p-70 + (double)s5[4] * 0x1p-51;
            const int32_t j = js[tid], c = cs[tid];
            if (MODE == 0) {
                const double E = z_bound(n1, R);
                const double e = E / q;
                const bool good = ok && ex < 2047 && q > 0.0 && e < 0x1p-10;
                b.rinv[j] = good ? 1.0 / q : 0.0;
                const float ef = __double2float_ru(e + 0x1p-50);
                b.e0[j] = good ? ef : 1.0f;
                b.err[j] = make_float2(good ? ef : 1.0f, good ? ef : 1.0f);
                if (!good) z_mark(b.redo, b.redo_list, b.redo_count, j);
            } else {
                const double cutoff = low + q * rinv;
                const float ec = (er.x + e0) * 1.0001f + 0x1p-50f;
                const bool left = d <= cutoff;
                if (!(fabs(d - cutoff) > (double)ec)) z_mark(b.redo, b.redo_list, b.redo_count, j);
                b.node[j] = left ? 2 * (int64_t)c + 1 : 2 * (int64_t)c + 2;
                if (left) {
                    b.lh[j].y = cutoff;
                    b.err[j].y = ec;
                } else {
                    b.lh[j].x = cutoff;
                    b.err[j].x = ec;
                }
                flag = left ? 1 : 0;
            }
        }
        if (MODE != 0 && tid < kZTile) {
            const uint32_t bits = __ballot_sync(0xffffffffu, flag > 0);
            if (lane == 0 && bits) {
                atomicOr(b.mask[p] + 4 * sh.tile + w, bits);
                atomicAdd(b.tcount[p] + sh.tile, __popc(bits));
            }
        }
    }
    __syncthreads();
    if (tid == 0) {
        if (aborted) {
            report(status, EXAFAC_ERR_TIMEOUT, 23, blockIdx.x, 0);
            *b.lost = 1;
        }
        // the copies and products in flight (after a wait that ran out only)
        for (int q = 0; q < 2; q++) {
            if (flight & (1u << q)) mbar_wait_limited(&copied[q], cphase[q], kSpinLimit);
            if (flight & (4u << q)) mbar_wait_limited(&bars[q], phase[q], kSpinLimit);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (w == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmem);
    }
}

// The common exponent of a leaf's rows from the largest of its Gram's diagonal
// exponents: max G_jj < 2^(e - 1022), |U| < 2^ceil((e - 1022) / 2); one more
// for rounding.
__device__ __forceinline__ int z_leaf_exp(int e) { return e >= 2047 ? 2047 : ((e - 1022 + 2047) >> 1) - 1023 + 1 + 1022; }

// The leaf stage: dots v_r = U_r . x of the leaf's rows from four digits of
// each (weights <= 3), their FP32 squares' prefix in row order, and the row
// whose range (before, before + v_r^2] holds frac x total, frac = (d - low) /
// (high - low), when frac x total keeps a distance from both ends that
// covers every error; otherwise the sample is listed for zq_place_kernel.  In scaled units
// (|x'|, |U'| < 2^6): a dot is off by at most e0 = R 5.2 2^-18 plus 2^-24 of
// itself, so a prefix by 2 e0 sqrt(F total) + F e0^2 + 70 2^-24 total, and
// frac by (err_low + err_high) / (high - low).
template <int NT>
__global__ void __launch_bounds__(NT, NT == 256 ? 2 : 1)
    zq_leaf_kernel(int R, TreeShape t, const double* __restrict__ G, const double* __restrict__ U, int64_t J, ZState b,
                   int p, const int32_t* __restrict__ order, const double* __restrict__ dv, int N, int col,
                   uint32_t* __restrict__ samples, DeviceStatus* status, uint32_t wait_polls, int64_t withhold) {
    extern __shared__ __align__(128) unsigned char z_raw[];
    if (z_lost(b)) return;
    constexpr int NG = NT / 128;
    constexpr int CPT = kZCols / NG;
    constexpr int NS = (NT == 256 ? 2 : 4);  // chunks (leaf rows / 32) at most
    __shared__ int32_t cs[kZTile], js[kZTile];
    __shared__ uint32_t rmask[4];
    __shared__ float psum[NS * NG][kZTile];
    __shared__ int diag_exp;
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_base;
    __shared__ int abort_flag;
    const ZShape z = z_shape(R);
    unsigned char* A = z_raw + ((128u - (smem_u32(z_raw) & 127u)) & 127u);
    unsigned char* B = A + kZx * z.xs;
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const int P = packed_size(R), F = (int)t.F;
    const int nch = (F + kZCols - 1) / kZCols;
    if (w == 0) tmem_alloc(&tmem_base, 128);
    if (tid == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
        abort_flag = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    uint32_t phase = 0;
    bool flight = false;  // thread 0: products on their way
    const int row = (w & 3) * 32 + lane, grp = w >> 2;
    const int64_t ntiles = (J + kZTile - 1) / kZTile;
    ZShare sh = z_share<NT>(b.runs[p], ntiles);
    for (; sh.count > 0 && sh.tile < ntiles; sh.tile++, sh.run = 0) {
        const int64_t s0 = sh.tile * kZTile;
        const int n = (int)min((int64_t)kZTile, J - s0);
        if (tid < kZTile) {
            const int32_t j = tid < n ? (order ? order[s0 + tid] : (int32_t)(s0 + tid)) : 0;
            js[tid] = j;
            cs[tid] = tid < n ? (int32_t)b.node[j] : -1;
        }
        if (tid < 4) rmask[tid] = b.runs[p][4 * sh.tile + tid];
        __syncthreads();
        stage_x(A, reinterpret_cast<const long long*>(b.xi), js, n, R, z);
        const int2 own = z_run_slots(rmask, sh.run, sh.count, n);
        for (int i0 = own.x; i0 < own.y; sh.count--) {
            const int32_t c = cs[i0];
            const int i1 = z_run_end(rmask, i0, n);
            const int64_t leaf = tree_leaf_idx(t, c);
            const int rows = (int)min((int64_t)F, t.n - leaf * F);
            const double* Ub = U + leaf * F * R;
            // |U_rj| <= sqrt(G_jj) of the leaf's Gram: the rows' common exponent
            if (tid < 32) {
                int e = 0;
                for (int a = lane; a < R; a += 32) e = max(e, bexp(__ldg(G + (int64_t)c * P + packed_index(R, a, a))));
                e = __reduce_max_sync(0xffffffffu, e);
                if (lane == 0) diag_exp = z_leaf_exp(e);
            }
            __syncthreads();
            const int emax = diag_exp;
            float y[NS][CPT];
#pragma unroll
            for (int ch = 0; ch < NS; ch++) {
                if (ch < nch) {
                    expand_rows(B, Ub, ch, rows, R, emax, z);
                    fence_proxy_async_smem();
                    tc_fence_before();
                    __syncthreads();
                    if (tid == 0 && sh.tile != withhold) {
                        issue_chunk<kZu>(tmem, A, B, z, &bar);
                        flight = true;
                    }
                    if (mbar_wait_limited(&bar, phase, wait_polls)) {
                        phase ^= 1u;
                        flight = false;
                    } else {
                        abort_flag = 1;
                    }
                    tc_fence_after();
                    float ps = 0.0f;
#pragma unroll
                    for (int h = 0; h < CPT / 8; h++) {
                        uint32_t a[kZu][8];
#pragma unroll
                        for (int s = 0; s < kZu; s++)
                            tmem_ld8_nowait(tmem + ((uint32_t)((w & 3) * 32) << 16) +
                                                (uint32_t)(kZCols * s + grp * CPT + 8 * h), a[s]);
                        tmem_ld_wait<kZu>(a);
#pragma unroll
                        for (int q = 0; q < 8; q++) {
                            const float v = __uint_as_float(a[0][q]) +
                                            (__uint_as_float(a[1][q]) +
                                             (__uint_as_float(a[2][q]) + __uint_as_float(a[3][q])));
                            y[ch][8 * h + q] = v * v;
                            ps += v * v;
                        }
                    }
                    psum[ch * NG + grp][row] = ps;
                    tc_fence_before();
                    __syncthreads();
                    if (abort_flag) break;
                } else {
#pragma unroll
                    for (int q = 0; q < CPT; q++) y[ch][q] = 0.0f;
                }
            }
            if (abort_flag) break;
            if (row >= i0 && row < i1) {
                const int32_t j = js[row];
                float total = 0.0f;
                for (int s = 0; s < nch * NG; s++) total += psum[s][row];
                const double2 lh = b.lh[j];
                const float2 er = b.err[j];
                const double width = lh.y - lh.x;
                const float rw = (float)(1.0 / width);
                const float frac = (float)((dv[j] - lh.x) / width);
                const float thr = frac * total;
                const float de = (er.x + er.y + 0x1p-49f) * rw * total * 1.001f;
                const float ev = (float)R * 5.2f * 0x1p-18f;
                const float delta = 1.01f * (de + 2.0f * ev * sqrtf((float)F * total) + (float)F * ev * ev +
                                             70.0f * 0x1p-24f * total);
                // every thread of the slot looks for the row in its slices
                bool found = false;
                float before = 0.0f;
                int at = 0;
#pragma unroll
                for (int ch = 0; ch < NS; ch++) {
                    if (ch < nch) {
                        for (int gq = 0; gq < NG; gq++) {
                            const float ps = psum[ch * NG + gq][row];
                            if (gq == grp) {
                                float pre = before;
#pragma unroll
                                for (int q = 0; q < CPT; q++) {
                                    const float nx = pre + y[ch][q];
                                    const int r = ch * kZCols + grp * CPT + q;
                                    if (!found && r < rows && thr < nx - delta && (r == 0 || thr > pre + delta)) {
                                        found = true;
                                        at = r;
                                    }
                                    pre = nx;
                                }
                            }
                            before += ps;
                        }
                    }
                }
                // delta is a finite number only if every input was; a sample
                // that no thread places is left to zq_place_kernel
                if (found && width > 0.0 && total > 0.0f && delta < total && emax < 2047)
                    b.pick[j] = at;
            }
            __syncthreads();
            if (tid >= i0 && tid < i1) {
                const int32_t j = js[tid];
                const int at = b.pick[j];
                if (at < 0) b.near_list[atomicAdd(b.near_count, 1)] = j;  // zq_place_kernel
                samples[(int64_t)j * N + col] = (uint32_t)(leaf * F + max(at, 0));
            }
            i0 = i1;
        }
        __syncthreads();
        if (abort_flag) break;
    }
    __syncthreads();
    if (abort_flag) {
        if (tid == 0) {
            report(status, EXAFAC_ERR_TIMEOUT, 24, blockIdx.x, 0);
            *b.lost = 1;
            if (flight) mbar_wait_limited(&bar, phase, kSpinLimit);
        }
        tc_fence_before();
        __syncthreads();
    }
    if (w == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 128);
    }
}

// The listed samples' rows (three to twelve in a thousand: the FP32 squares'
// rounding), a block per sample in turn: the leaf's dots, squares and prefix
// in FP64 from the fixed-point vector, eight lanes per row.  In scaled units a
// dot, and the depth-first kernel's own, is off by at most e1 = R (2^-42 +
// 2^-45 n1) (the vector's rounding, the two sums'), a prefix by 2 e1 sqrt(F
// total) + F e1^2 + F 2^-50 total, frac as in zq_leaf_kernel.  A sample that
// is still within the bound is marked.  Drawing the listed samples again depth
// first took 0.46 ms a step at R = 64, J = 2^18 and 1.8 ms at R = 100, J =
// 100003, four modes.
constexpr int kPlaceThreads = 256;
__global__ void __launch_bounds__(kPlaceThreads)
    zq_place_kernel(int R, TreeShape t, const double* __restrict__ G, const double* __restrict__ U, ZState b,
                    const double* __restrict__ dv, int N, int col, uint32_t* __restrict__ samples) {
    __shared__ double xs[kMaxRank], sq[kMaxLeafRows];
    __shared__ int diag_exp;
    const int tid = threadIdx.x, lane = tid & 31, P = packed_size(R), F = (int)t.F;
    if (z_lost(b)) return;
    const int count = *b.near_count;
    for (int q = blockIdx.x; q < count; q += gridDim.x) {
        const int32_t j = b.near_list[q];
        const int64_t c = b.node[j];
        const int64_t leaf = tree_leaf_idx(t, c);
        const int rows = (int)min((int64_t)F, t.n - leaf * F);
        const double* Ub = U + leaf * F * R;
        if (tid < 32) {
            int e = 0;
            for (int a = lane; a < R; a += 32) e = max(e, bexp(__ldg(G + c * P + packed_index(R, a, a))));
            e = __reduce_max_sync(0xffffffffu, e);
            if (lane == 0) diag_exp = z_leaf_exp(e);
        }
        const long long* X = reinterpret_cast<const long long*>(b.xi) + (int64_t)j * z_row(R);
        for (int a = tid; a < R; a += kPlaceThreads) xs[a] = (double)(((long long)x_z4(X[a]) << 23) + x_rest(X[a])) * 0x1p-47;
        __syncthreads();
        const int emax = diag_exp;
        const double scale = scalbn(1.0, max(min(1028 - emax, 1000), -1000));
        for (int r0 = 0; r0 < F; r0 += kPlaceThreads / 8) {
            const int r = r0 + (tid >> 3);
            double v = 0.0;
            if (r < rows)
                for (int a = tid & 7; a < R; a += 8) v = fma(__ldg(Ub + (int64_t)r * R + a), xs[a], v);
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            v *= scale;
            if ((tid & 7) == 0 && r < F) sq[r] = v * v;
        }
        __syncthreads();
        if (tid < 32) {
            double incl[4], own[4], total = 0.0;
#pragma unroll
            for (int blk = 0; blk < 4; blk++) {
                const int r = 32 * blk + lane;
                double v = r < F ? sq[r] : 0.0;
                own[blk] = v;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const double u = __shfl_up_sync(0xffffffffu, v, o);
                    if (lane >= o) v += u;
                }
                incl[blk] = total + v;
                total += __shfl_sync(0xffffffffu, v, 31);
            }
            const double2 lh = b.lh[j];
            const float2 er = b.err[j];
            const double width = lh.y - lh.x;
            const double thr = (dv[j] - lh.x) / width * total;
            const double de = 1.001 * ((double)er.x + (double)er.y + 0x1p-49) / width * total;
            const double e1 = (double)R * (0x1p-42 + (double)b.n1[j] * 0x1p-45);
            const double delta =
                1.01 * (de + 2.0 * e1 * sqrt((double)F * total) + (double)F * e1 * e1 + (double)F * 0x1p-50 * total);
            const bool usable = width > 0.0 && total > 0.0 && delta < total && emax < 2047 && emax > 28;
            int at = -1;
#pragma unroll
            for (int blk = 0; blk < 4; blk++) {
                const int r = 32 * blk + lane;
                const bool hit = usable && r < rows && thr < incl[blk] - delta &&
                                 (r == 0 || thr > (incl[blk] - own[blk]) + delta);
                const unsigned mask = __ballot_sync(0xffffffffu, hit);
                if (at < 0 && mask) at = 32 * blk + __ffs(mask) - 1;
            }
            if (lane == 0) {
                if (at < 0) z_mark(b.redo, b.redo_list, b.redo_count, j);
                else samples[(int64_t)j * N + col] = (uint32_t)(leaf * F + at);
            }
        }
        __syncthreads();
    }
}

// Exclusive prefix of the tiles' counts in a block's shared memory.
__device__ __forceinline__ void tile_prefix(const int32_t* __restrict__ tcount, int ntiles, int32_t* pref) {
    __shared__ int32_t wsum[32];
    const int nt = blockDim.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int32_t carry = 0;
    for (int base = 0; base < ntiles; base += 4 * nt) {
        int32_t v[4], s = 0;
        const int i = base + 4 * threadIdx.x;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            v[q] = i + q < ntiles ? __ldg(tcount + i + q) : 0;
            s += v[q];
        }
        int32_t inc = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t u = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += u;
        }
        if (lane == 31) wsum[w] = inc;
        __syncthreads();
        int32_t pre = carry + inc - s, all = 0;
        for (int q = 0; q < (nt >> 5); q++) {
            if (q < w) pre += wsum[q];
            all += wsum[q];
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (i + q < ntiles) pref[i + q] = pre;
            pre += v[q];
        }
        carry += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) pref[ntiles] = carry;
    __syncthreads();
}

// The stable partition after a level in one launch: SL(s), the flags set
// before slot s, is the tile's prefix plus the bits below s of its mask.
// Within its parent's slot range a slot whose flag is set (went left, or
// stayed at a leaf) keeps its order among those, before the others; the
// children's slot ranges (coff) and their run starts follow, and the next
// level's flags are cleared, and the next level's left children are expanded
// into `nodes` (where it takes them: nx_nl > 0).  Every block
// forms the tiles' prefix in shared memory (up to kZPrefSmem tiles), or reads
// pref64 (more).  lb: the parents' first node index, nl their number.
__global__ void __launch_bounds__(512)
    zq_partition_kernel(int64_t J, int ntiles, const uint32_t* __restrict__ mask, const int32_t* __restrict__ tcount,
                        uint32_t* __restrict__ mask_next, int32_t* __restrict__ tcount_next,
                        uint32_t* __restrict__ runs_next, const int64_t* __restrict__ pref64, int64_t lb, int64_t nl, const int32_t* __restrict__ order,
                        const int64_t* __restrict__ node, const int64_t* __restrict__ off,
                        int32_t* __restrict__ order2, int64_t* __restrict__ coff, int R, const double* __restrict__ G,
                        const int32_t* __restrict__ tree_exp, int64_t node_count, int64_t nx_lb, int64_t nx_nl,
                        unsigned char* __restrict__ nodes, const int32_t* __restrict__ lost) {
    extern __shared__ int32_t z_pref[];
    if (*lost) return;  // (no level runs beside this kernel: the same in every thread)
    if (nx_nl > 0) {
        const ZShape z = z_shape(R);
        const int emax = *tree_exp, items = kZCols * (z.Rk / 8);
        const int64_t all = nx_nl * z.nch * items;
        for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < all; q += (int64_t)gridDim.x * blockDim.x) {
            const int64_t at = q / items;  // node and chunk
            const int64_t g = 2 * (nx_lb + at / z.nch) + 1;
            if (g < node_count)
                expand_item(nodes + at * z_chunk_bytes(z), G + g * packed_size(R), (int)(at % z.nch), (int)(q - at * items),
                            R, emax, z);
        }
    }
    if (!pref64) tile_prefix(tcount, ntiles, z_pref);
    auto SL = [&](int64_t s) -> int64_t {
        const int64_t tile = s >> 7;
        int64_t v = pref64 ? pref64[tile] : (int64_t)z_pref[tile];
        const int in = (int)(s & 127);
        if (in) {
            const uint32_t* m = mask + 4 * tile;
            for (int q = 0; q < (in >> 5); q++) v += __popc(__ldg(m + q));
            if (in & 31) v += __popc(__ldg(m + (in >> 5)) & ((1u << (in & 31)) - 1u));
        }
        return v;
    };
    const int64_t step = (int64_t)gridDim.x * blockDim.x, first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (int64_t s = first; s < J; s += step) {
        const int32_t j = order ? order[s] : (int32_t)s;
        const int64_t c = node[j];
        const int64_t i = (c >= lb + nl ? (c - 1) / 2 : c) - lb;
        const int64_t start = off[i], end = off[i + 1];
        const int64_t at0 = SL(start), at = SL(s);
        const bool fl = (__ldg(mask + 4 * (s >> 7) + ((s & 127) >> 5)) >> (s & 31)) & 1u;
        const int64_t before = at - at0;
        const int64_t pos = fl ? start + before : start + (SL(end) - at0) + ((s - start) - before);
        order2[pos] = j;
    }
    for (int64_t i = first; i < nl; i += step) {
        const int64_t start = off[i], end = off[i + 1];
        const int64_t mid = start + (SL(end) - SL(start));
        coff[2 * i] = start;
        coff[2 * i + 1] = mid;
        if (i == 0) coff[2 * nl] = J;
        // a child that begins inside a tile begins one more run there
        if (mid > start && (start & 127)) atomicOr(runs_next + (start >> 5), 1u << (start & 31));
        if (end > mid && (mid & 127)) atomicOr(runs_next + (mid >> 5), 1u << (mid & 31));
    }
    for (int64_t q = first; q < ntiles; q += step) {
        reinterpret_cast<uint4*>(mask_next)[q] = make_uint4(0u, 0u, 0u, 0u);
        tcount_next[q] = 0;
    }
}

// Largest diagonal exponent of a tree's root, plus one (the entries of the
// tree's nodes are bounded by their diagonals, those by the root's; one more
// bit for rounding).  nodes != null: blockIdx.x = node and chunk of the root
// and its left child, which the block expands.
__global__ void __launch_bounds__(256) zq_tree_exp_kernel(int R, const double* __restrict__ root,
                                                          int32_t* __restrict__ out, int64_t node_count,
                                                          unsigned char* __restrict__ nodes) {
    __shared__ int top;
    if (threadIdx.x < 32) {
        int e = 0;
        for (int a = threadIdx.x; a < R; a += 32) e = max(e, bexp(root[packed_index(R, a, a)]));
        e = __reduce_max_sync(0xffffffffu, e);
        if (threadIdx.x == 0) {
            top = e >= 2047 ? 2047 : e + 1;
            if (blockIdx.x == 0) *out = top;
        }
    }
    __syncthreads();
    if (!nodes) return;
    const ZShape z = z_shape(R);
    const int64_t g = blockIdx.x / z.nch;
    if (g >= node_count) return;
    for (int q = threadIdx.x; q < kZCols * (z.Rk / 8); q += blockDim.x)
        expand_item(nodes + (int64_t)blockIdx.x * z_chunk_bytes(z), root + g * packed_size(R), blockIdx.x % z.nch, q, R,
                    top, z);
}

// The vector of the next descent in fixed point, a warp per sample, and the
// sample's state at the root.
// KIND 0: h = 1.  KIND 1: x = h * E[v].  KIND 2: h *= U[row], x = h.
template <int KIND>
__global__ void zq_vector_kernel(int R, int64_t J, double* __restrict__ h, const double* __restrict__ M,
                                 uint32_t* __restrict__ samples, int N, int col, int64_t rows, ZState b,
                                 DeviceStatus* status) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const bool lost = KIND != 0 && *b.lost != 0;
    for (int64_t j = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; j < J; j += nw) {
        if (lost) {
            if (lane == 0) samples[j * N + col] = 0u;
            if (j == 0 && lane == 0) *b.near_count = 0;
            continue;
        }
        double x[4];
        int64_t r = 0;
        if (KIND != 0) {
            r = KIND == 1 ? (int64_t)b.v[j] : (int64_t)samples[j * N + col];
            if (r < 0 || r >= rows) {  // as the depth-first kernel: report, take the last row
                if (lane == 0) report(status, EXAFAC_ERR_DEVICE, KIND, r, rows);
                r = rows - 1;
            }
        }
        int e = 0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int c = lane + 32 * q;
            x[q] = 0.0;
            if (c < R) {
                if (KIND == 0) x[q] = 1.0;
                else x[q] = h[j * R + c] * __ldg(M + r * R + c);
                if (KIND != 1) h[j * R + c] = x[q];
                e = max(e, bexp(x[q]));
            }
        }
        e = __reduce_max_sync(0xffffffffu, e);
        float n1 = 0.0f;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int c = lane + 32 * q;
            if (c < z_row(R)) {  // (x is zero past R)
                const long long f = e < 2047 ? fix47_rn(x[q], e) : 0ll;
                reinterpret_cast<long long*>(b.xi)[j * z_row(R) + c] = pack_x(f);
                if (KIND == 2) b.rest[j * z_row(R) + c] = (int8_t)(e < 2047 ? fix47_rest(x[q], e) : 0);
                n1 += (float)((int)(llabs(f) >> 24) + 1) * 0x1p-23f;
            }
        }
        n1 = warp_sum(n1);
        if (lane == 0) {
            b.ex[j] = e;
            b.n1[j] = 1.001f * n1;
            b.node[j] = 0;
            b.lh[j] = make_double2(0.0, 1.0);
            b.pick[j] = -1;
            if (KIND == 0) b.redo[j] = 0;
            if (KIND == 0 && j == 0) *b.redo_count = 0;
            if (KIND == 0 && j == 0) *b.lost = 0;
            if (j == 0) *b.near_count = 0;
            if ((j & 127) == 0) {
                const int64_t tile = j >> 7;
                reinterpret_cast<uint4*>(b.mask[0])[tile] = make_uint4(0u, 0u, 0u, 0u);
                b.tcount[0][tile] = 0;
                reinterpret_cast<uint4*>(b.runs[0])[tile] = make_uint4(0u, 0u, 0u, 0u);
            }
            if (j == 0) {
                b.off[0][0] = 0;
                b.off[0][1] = J;
            }
        }
    }
}

// The eigen tree's leaves: the leaf's index (F = 1).
__global__ void zq_leaf1_kernel(TreeShape t, int64_t J, ZState b, int N, int col, uint32_t* __restrict__ samples) {
    if (*b.lost) return;
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < J; j += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = tree_leaf_idx(t, b.node[j]);
        samples[j * N + col] = (uint32_t)v;
        b.v[j] = (int32_t)v;
    }
}

// ---- the weights R / (J h^T Phi h)
//
// The same products with five digits of h and eight of Phi (weights <= 7, in
// chunks of 16 columns), in place of R^2 / 2 FP64 products and sums per sample,
// which took 3.1 ms at R = 64, J = 2^18.  What the fixed point of h leaves off
// (up to 2^-48 of the scaled units, more than FP64 where the entries of h differ
// by decades) is kept to 256ths of its unit (ZState::rest) and added in FP32 to
// first order, 2 sum_c Y_c (h - x)_c.  The digits and the cut of Phi that are
// dropped are below R 4 2^-50 of n1; an FP64 sum's own rounding is some 2^-53 of
// sum |h_a Phi_ab h_b|, of which sum_c Phi_cc h_c^2 is a part.  A sample whose
// bound is above 2^-42 of its form or above 2^-46 of that diagonal part gets the
// depth-first kernel's own sum from h (sts_weight_list_kernel); one whose form
// is not positive or not finite is marked.  Against exact arithmetic, the
// largest error of a dozen samples, FP64 sums -> digits: Grams of random
// factors at R = 64 3e-16 -> 2e-17, nearly collinear columns (Phi_cc to 170) at
// R = 100 9e-15 -> 2.4e-15, small h where Phi is large (three decades) 2.2e-16
// -> 2.2e-16 (6e-15 without the diagonal's test). As a decomposition converges
// up to a tenth of the samples go to FP64; drawing them again whole took 1.1 ms
// a step at R = 100 with four modes, 6 ms at R = 66 with three.
constexpr int kWx = 5, kWa = 8, kWCols = 16;

static size_t zw_smem(int R) {
    const ZShape z = z_shape(R);
    return (size_t)kWx * z.xs + (size_t)kWa * 2 * z.sbo + 128;
}

__device__ __forceinline__ void tmem_ld4_nowait(uint32_t taddr, uint32_t (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr)
                 : "memory");
}

constexpr int kWThreads = 512;
__global__ void __launch_bounds__(kWThreads, 1)
    zq_weight_kernel(int R, int64_t J, ZState b, const double* __restrict__ PhiP, const int32_t* __restrict__ phi_exp,
                     double* __restrict__ weights, DeviceStatus* status, uint32_t wait_polls, int64_t withhold) {
    extern __shared__ __align__(128) unsigned char z_raw[];
    if (z_lost(b)) {
        for (int64_t j = (int64_t)blockIdx.x * kWThreads + threadIdx.x; j < J; j += (int64_t)gridDim.x * kWThreads)
            weights[j] = 0.0;
        return;
    }
    constexpr int NG = kWThreads / 128;  // threads per slot in the read-back, four columns each
    __shared__ long long part[NG][7][kZTile];
    __shared__ float2 fpart[NG][kZTile];
    __shared__ int rs[kMaxRank];
    __shared__ float diag[kMaxRank];  // Phi_cc in the scaled units
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_base;
    __shared__ int abort_flag;
    const ZShape z = z_shape(R);
    const int Rx = z_row(R);
    const uint32_t bs = 2u * z.sbo;  // one digit of 16 columns
    unsigned char* A = z_raw + ((128u - (smem_u32(z_raw) & 127u)) & 127u);
    unsigned char* B = A + kWx * z.xs;
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    if (w == 0) tmem_alloc(&tmem_base, 128);
    for (int a = tid; a < R; a += kWThreads) rs[a] = packed_index(R, a, a);
    if (tid == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
        abort_flag = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    const int emax = *phi_exp;
    for (int c = tid; c < kMaxRank; c += kWThreads)  // (read after the barriers of the first chunk)
        diag[c] = c < R ? (float)scalbn(PhiP[packed_index(R, c, c)], 1028 - emax) : 0.0f;
    uint32_t phase = 0;
    bool flight = false;  // thread 0: products on their way
    const int row = (w & 3) * 32 + lane, grp = w >> 2;
    const int nch = (R + kWCols - 1) / kWCols;
    const int64_t ntiles = (J + kZTile - 1) / kZTile;
    const long long* xi = reinterpret_cast<const long long*>(b.xi);
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int64_t s0 = tile * kZTile;
        const int n = (int)min((int64_t)kZTile, J - s0);
        for (int e = tid; e < kZTile * (z.Rk / 8); e += kWThreads) {  // h, the row fastest
            const int r = e & (kZTile - 1), k = 8 * (e / kZTile);
            long long X[8];
            load_x8(xi + (s0 + (r < n ? r : 0)) * Rx, k, Rx, r < n, X);
            uint32_t lo[8];
            int hi[8];
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const long long t = (long long)x_z4(X[q]) * 256 + ((x_rest(X[q]) + (1 << 14)) >> 15) +
                                    0x80808080ll;  // units of 2^-32
                lo[q] = (uint32_t)t;
                hi[q] = (int)(t >> 32);
            }
            uint32_t o[kWx][4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const uint32_t u = lo[2 * q], v = lo[2 * q + 1];
                o[0][q] = pack_bf16(lead_f(hi[2 * q]), lead_f(hi[2 * q + 1]));
                o[1][q] = pack_bf16(digit_f<1>(u, 3), digit_f<1>(v, 3));
                o[2][q] = pack_bf16(digit_f<2>(u, 2), digit_f<2>(v, 2));
                o[3][q] = pack_bf16(digit_f<3>(u, 1), digit_f<3>(v, 1));
                o[4][q] = pack_bf16(digit_f<4>(u, 0), digit_f<4>(v, 0));
            }
            unsigned char* dst = A + (uint32_t)(r >> 3) * z.sbo + (uint32_t)(k >> 3) * 128u + (uint32_t)(r & 7) * 16u;
#pragma unroll
            for (int d = 0; d < kWx; d++)
                *reinterpret_cast<uint4*>(dst + d * z.xs) = make_uint4(o[d][0], o[d][1], o[d][2], o[d][3]);
        }
        long long sum[7] = {0, 0, 0, 0, 0, 0, 0};  // P, Q, T times the high and low parts of x0 + 2 xr, W times the high
        float rest = 0.0f, dsum = 0.0f;  // sum_c Y_c (h - x)_c in units of 2^-55, sum_c Phi_cc x_c^2
        const int64_t jrow = s0 + (row < n ? row : 0);
        const long long* xrow = xi + jrow * Rx;
        const uint32_t* rrow = reinterpret_cast<const uint32_t*>(b.rest + jrow * Rx);
        for (int ch = 0; ch < nch; ch++) {
            for (int e = tid; e < kWCols * (z.Rk / 8); e += kWThreads) {  // Phi's columns, the column fastest
                const int c = e & (kWCols - 1), k = 8 * (e / kWCols);
                const int col = ch * kWCols + c;
                const int rc = col < R ? rs[col] : 0;
                uint32_t lo[8], hi[8];
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const int kk = k + q;
                    const double v =
                        (col < R && kk < R) ? __ldg(PhiP + (kk >= col ? rc + (kk - col) : rs[kk] + (col - kk))) : 0.0;
                    const long long t = fix56(v, emax) + 0x80808080808080ll;  // eight digits
                    lo[q] = (uint32_t)t;
                    hi[q] = (uint32_t)(t >> 32);
                }
                uint32_t o[kWa][4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const uint32_t u = lo[2 * q], v = lo[2 * q + 1], uh = hi[2 * q], vh = hi[2 * q + 1];
                    o[0][q] = pack_bf16(lead_f((int)uh >> 24), lead_f((int)vh >> 24));
                    o[1][q] = pack_bf16(digit_f<1>(uh, 2), digit_f<1>(vh, 2));
                    o[2][q] = pack_bf16(digit_f<2>(uh, 1), digit_f<2>(vh, 1));
                    o[3][q] = pack_bf16(digit_f<3>(uh, 0), digit_f<3>(vh, 0));
                    o[4][q] = pack_bf16(digit_f<4>(u, 3), digit_f<4>(v, 3));
                    o[5][q] = pack_bf16(digit_f<5>(u, 2), digit_f<5>(v, 2));
                    o[6][q] = pack_bf16(digit_f<6>(u, 1), digit_f<6>(v, 1));
                    o[7][q] = pack_bf16(digit_f<7>(u, 0), digit_f<7>(v, 0));
                }
                unsigned char* dst = B + (uint32_t)(c >> 3) * z.sbo + (uint32_t)(k >> 3) * 128u + (uint32_t)(c & 7) * 16u;
#pragma unroll
                for (int d = 0; d < kWa; d++)
                    *reinterpret_cast<uint4*>(dst + d * bs) = make_uint4(o[d][0], o[d][1], o[d][2], o[d][3]);
            }
            fence_proxy_async_smem();
            tc_fence_before();
            __syncthreads();
            if (tid == 0 && tile != withhold) {
                flight = true;
                tc_fence_after();
#pragma unroll
                for (int i = 0; i < kWx; i++) {
                    const uint32_t idesc = umma_idesc_bf16(kZTile, kWCols * (kWa - i));
                    for (int ks = 0; ks < z.Rk / 16; ks++)
                        umma_bf16(tmem + (uint32_t)(kWCols * i), umma_desc(A + i * z.xs + ks * 256, 128u, z.sbo),
                                  umma_desc(B + ks * 256, 128u, z.sbo), idesc, (i > 0 || ks > 0) ? 1u : 0u);
                }
                umma_commit(&bar);
            }
            if (mbar_wait_limited(&bar, phase, wait_polls)) {
                phase ^= 1u;
                flight = false;
            } else {
                abort_flag = 1;
            }
            tc_fence_after();
            const int cc = 4 * grp;
            uint32_t a[kWa][4];
#pragma unroll
            for (int q = 0; q < kWa; q++)
                tmem_ld4_nowait(tmem + ((uint32_t)((w & 3) * 32) << 16) + (uint32_t)(kWCols * q + cc), a[q]);
            long long X[4] = {0, 0, 0, 0};
            uint32_t r4 = 0x80808080u;  // the four rests, plus 128 each
            if (ch * kWCols + cc < Rx) {
                asm volatile("ld.global.v4.b64 {%0, %1, %2, %3}, [%4];"
                             : "=l"(X[0]), "=l"(X[1]), "=l"(X[2]), "=l"(X[3])
                             : "l"(xrow + ch * kWCols + cc));
                r4 ^= __ldg(rrow + (ch * kWCols + cc) / 4);
            }
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int q = 0; q < kWa; q++)
                asm volatile("" : "+r"(a[q][0]), "+r"(a[q][1]), "+r"(a[q][2]), "+r"(a[q][3]));
#pragma unroll
            for (int q = 0; q < 4; q++) {
                float f[kWa];
#pragma unroll
                for (int u = 0; u < kWa; u++) f[u] = __uint_as_float(a[u][q]);
                // integers of the weights 0, 1, 2; weight 3 to 2^-23, weight
                // 4 to 2^-30; their (exact) rests with weight 5 to 2^-38;
                // that rest with the weights 6 and 7 to 2^-46
                const int m0 = __float_as_int(f[0] + 12582912.0f) - 0x4B400000;
                const int m1 = __float_as_int(f[1] + 49152.0f) - 0x47400000;
                const int m2 = __float_as_int(f[2] + 192.0f) - 0x43400000;
                const float t3 = f[3] + 1.5f;
                const int m3 = __float_as_int(t3) - 0x3FC00000;
                const float t4 = f[4] + 0x1.8p-7f;
                const int m4 = __float_as_int(t4) - 0x3C400000;
                const float g5 = ((f[3] - (t3 - 1.5f)) + (f[4] - (t4 - 0x1.8p-7f))) + f[5];
                const float t5 = g5 + 0x1.8p-15f;
                const int m5 = __float_as_int(t5) - 0x38400000;
                const float g6 = (g5 - (t5 - 0x1.8p-15f)) + (f[6] + f[7]);
                const int W = __float_as_int(g6 + 0x1.8p-23f) - 0x34400000;
                const int Pn = m0 * 256 + m1, Qn = m2 * 128 + m3, Tn = m4 * 256 + m5;
                const int z4 = x_z4(X[q]), xr = x_rest(X[q]), k5 = (xr + (1 << 14)) >> 15;
                const int wh = z4 >> 4, wl = ((z4 & 15) << 23) + 2 * xr - (k5 << 15);
                sum[0] += (long long)Pn * wh;
                sum[1] += (long long)Pn * wl;
                sum[2] += (long long)Qn * wh;
                sum[3] += (long long)Qn * wl;
                sum[4] += (long long)Tn * wh;
                sum[5] += (long long)Tn * wl;
                sum[6] += (long long)W * wh;
                const float x = (float)z4 * 0x1p-24f;
                rest = fmaf((f[0] + f[1]) + f[2], digit_f<0>(r4, q), rest);
                dsum = fmaf(diag[ch * kWCols + cc + q] * x, x, dsum);
            }
            tc_fence_before();
            __syncthreads();  // the accumulators and B are free for the next chunk
            if (abort_flag) break;
        }
        if (abort_flag) {  // this tile and the block's later ones
            for (int64_t q = tile; q < ntiles; q += gridDim.x)
                if (tid < kZTile && q * kZTile + tid < J) weights[q * kZTile + tid] = 0.0;
            break;
        }
#pragma unroll
        for (int u = 0; u < 7; u++) part[grp][u][row] = sum[u];
        fpart[grp][row] = make_float2(rest, dsum);
        __syncthreads();
        if (tid < n) {
            long long s6[7];
            float2 fs = fpart[0][tid];
#pragma unroll
            for (int gq = 1; gq < NG; gq++) {
                fs.x += fpart[gq][tid].x;
                fs.y += fpart[gq][tid].y;
            }
#pragma unroll
            for (int u = 0; u < 7; u++) {
                s6[u] = part[0][u][tid];
#pragma unroll
                for (int gq = 1; gq < NG; gq++) s6[u] += part[gq][u][tid];
            }
            // P 2^-8, Q 2^-23, T 2^-38, W 2^-46; the parts of x0 + 2 xr 2^-20, 2^-47
            const double q = ((((double)fs.x * 0x1p-54 + (double)s6[5] * 0x1p-85) + (double)s6[6] * 0x1p-66) +
                              (double)s6[4] * 0x1p-58) +
                             (((double)s6[3] * 0x1p-70 + (double)s6[1] * 0x1p-55) +
                              ((double)s6[2] * 0x1p-43 + (double)s6[0] * 0x1p-28));
            const int64_t j = s0 + tid;
            const int ex = b.ex[j];
            const bool usable = q > 0.0 && ex < 2047 && emax < 2047;
            const double err = (double)b.n1[j] * (double)R * 0x1p-48 + (double)R * (double)R * 0x1p-57;
            const bool good = usable && err < q * 0x1p-42 && err < (double)fs.y * 0x1p-46;
            const double hq = scalbn(q, 2 * ex + emax - 3084);
            weights[j] = good ? (double)R / (hq * (double)J) : 0.0;
            if (!usable) z_mark(b.redo, b.redo_list, b.redo_count, (int32_t)j);
            else if (!good) b.near_list[atomicAdd(b.near_count, 1)] = (int32_t)j;
        }
        __syncthreads();
    }
    __syncthreads();
    if (abort_flag) {
        if (tid == 0) {
            report(status, EXAFAC_ERR_TIMEOUT, 25, blockIdx.x, 0);
            if (flight) mbar_wait_limited(&bar, phase, kSpinLimit);
        }
        tc_fence_before();
        __syncthreads();
    }
    if (w == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 128);
    }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

// A level of the breadth-first form is two launches whatever J (about 8 us),
// and the marked samples' pass takes the latency of one depth-first draw; the
// depth-first kernel takes J R (R + 1) / 2 FMAs per level over the whole chip.
// 2^22 of them is the size from which the breadth-first form was no slower.
bool sts_zq_wanted(int R, int64_t J) { return J * (int64_t)packed_size(R) >= (1ll << 22); }

// The levels whose nodes are expanded once into global memory: those with at
// most half as many parents as tiles (each is then read twice or more), within
// 32 MB.  R = 64, J = 2^18: a level 135 -> 114 us (the runs' scattered reads of
// the packed node were half of its L1 wavefronts).  A node of one chunk (R <=
// 32) is expanded by one item per thread and kept from tile to tile: there the
// partition's extra work was the larger (a sweep at R = 25 4.65 against 4.71 ms).
constexpr size_t kZNodeBytes = 32u << 20;
static bool z_expands(int R) { return R > kZCols; }
static int64_t z_node_cap(int R, int64_t J) {
    const ZShape z = z_shape(R);
    const int64_t fit = (int64_t)(kZNodeBytes / ((size_t)z.nch * z_chunk_bytes(z)));
    return std::max<int64_t>(2, std::min<int64_t>(ceil_div(J, kZTile) / 2, fit));
}

void zq_carve(Arena& a, ZState& b, int R, int64_t J, int64_t widest, int trees) {
    b.xi = a.take<int64_t>(J * z_row(R));
    b.rest = a.take<int8_t>(J * z_row(R));
    b.lh = a.take<double2>(J);
    b.rinv = a.take<double>(J);
    b.err = a.take<float2>(J);
    b.e0 = a.take<float>(J);
    b.n1 = a.take<float>(J);
    b.ex = a.take<int32_t>(J);
    b.node = a.take<int64_t>(J);
    b.order[0] = a.take<int32_t>(J);
    b.order[1] = a.take<int32_t>(J);
    b.v = a.take<int32_t>(J);
    b.pick = a.take<int32_t>(J);
    b.redo = a.take<int32_t>(J);
    b.redo_list = a.take<int32_t>(J);
    b.redo_count = a.take<int32_t>(1);
    b.near_list = a.take<int32_t>(J);
    b.near_count = a.take<int32_t>(1);
    b.lost = a.take<int32_t>(1);
    for (int q = 0; q < 2; q++) {
        b.mask[q] = a.take<uint32_t>(4 * ceil_div(J, kZTile));
        b.tcount[q] = a.take<int32_t>(ceil_div(J, kZTile) + 4);
        b.runs[q] = a.take<uint32_t>(4 * ceil_div(J, kZTile));
    }
    b.pref64 = a.take<int64_t>(ceil_div(J, kZTile) + 1);
    b.off[0] = a.take<int64_t>(2 * widest + 2);
    b.off[1] = a.take<int64_t>(2 * widest + 2);
    b.tree_exp = a.take<int32_t>(trees + 1);
    const ZShape z = z_shape(R);
    if (z_expands(R)) b.nodes = a.take<uint4>(z_node_cap(R, J) * z.nch * z_chunk_bytes(z) / sizeof(uint4));
}

static unsigned z_grid(int64_t work) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(work, 256), 152 * 16));
}

// One wave of the chip (or the test hook's number of blocks: the draws are the
// same for any).
static unsigned z_blocks(const Session& s, int64_t J, int64_t wave) {
    return (unsigned)(s.draw_blocks > 0 ? s.draw_blocks : std::min(ceil_div(J, kZTile), wave));
}

template <int MODE, int NT>
static int z_level(Session& s, const TreeShape& t, const double* G, const unsigned char* nodes, int64_t lb,
                   const int32_t* ex, int64_t J, int p, const int32_t* order, const double* dv, cudaStream_t st) {
    // a second node buffer where one block per SM runs and it fits beside the
    // 22 KB of static shared memory
    const size_t two = z_smem(s.R, 2 * kZa);
    const int nb = NT == 512 && two <= 200 * 1024 ? 2 : 1;
    const size_t smem = nb == 2 ? two : z_smem(s.R, kZa);
    EXAFAC_CUDA_TRY(allow_smem(zq_level_kernel<MODE, NT>));
    const unsigned blocks = z_blocks(s, J, NT == 256 ? 304 : 152);
    zq_level_kernel<MODE, NT><<<blocks, NT, smem, st>>>(s.R, nb, t, G, nodes, lb, ex, J, s.zq, p, order, dv,
                                                        s.status, s.wait_polls ? s.wait_polls : kSpinLimit,
                                                        MODE == 0 ? -1 : s.withheld(23));
    count_launch();
    return EXAFAC_OK;
}
template <int MODE>
static int z_level_any(Session& s, const TreeShape& t, const double* G, const unsigned char* nodes, int64_t lb,
                       const int32_t* ex, int64_t J, int p, const int32_t* order, const double* dv, cudaStream_t st) {
    return s.R <= 64 ? z_level<MODE, 256>(s, t, G, nodes, lb, ex, J, p, order, dv, st)
                     : z_level<MODE, 512>(s, t, G, nodes, lb, ex, J, p, order, dv, st);
}
template <int NT>
static int z_leaf(Session& s, const TreeShape& t, const double* G, const double* U, int64_t J, int p,
                  const int32_t* order, const double* dv, int col, cudaStream_t st) {
    const size_t smem = z_smem(s.R, kZu);
    EXAFAC_CUDA_TRY(allow_smem(zq_leaf_kernel<NT>));
    const unsigned blocks = z_blocks(s, J, NT == 256 ? 304 : 152);
    zq_leaf_kernel<NT><<<blocks, NT, smem, st>>>(s.R, t, G, U, J, s.zq, p, order, dv, s.N, col, s.samples, s.status,
                                                 s.wait_polls ? s.wait_polls : kSpinLimit, s.withheld(24));
    count_launch();
    return EXAFAC_OK;
}

// One descent of every sample; the vectors and the root state are in place.
static int z_descend(Session& s, const TreeShape& t, const double* G, const double* U, const double* dv, int64_t J,
                     int col, int tree, cudaStream_t st) {
    ZState& b = s.zq;
    int32_t* ex = b.tree_exp + tree;
    const ZShape z = z_shape(s.R);
    unsigned char* nodes = z_expands(s.R) ? reinterpret_cast<unsigned char*>(b.nodes) : nullptr;
    const int64_t cap = nodes ? z_node_cap(s.R, J) : 0;
    zq_tree_exp_kernel<<<nodes ? (unsigned)(2 * z.nch) : 1u, 256, 0, st>>>(s.R, G, ex, t.node_count, nodes);
    count_launch();
    EXAFAC_TRY(z_level_any<0>(s, t, G, nodes, 0, ex, J, 0, nullptr, dv, st));
    const int64_t ntiles = ceil_div(J, kZTile);
    const bool in_smem = ntiles <= kZPrefSmem;
    const size_t psm = in_smem ? sizeof(int32_t) * (ntiles + 1) : 0;
    if (psm > 40 * 1024)  // (the 48 KB of a launch without it include the static part)
        EXAFAC_CUDA_TRY(allow_smem(zq_partition_kernel));
    const bool tail = t.node_count > t.nodes_upto_lfill;
    const int32_t* order = nullptr;
    int p = 0;  // parity of the level
    int64_t lb = 0, nl = 1;
    for (int64_t lvl = 0; lvl <= t.lfill_level; lvl++) {
        const bool is_tail = lvl == t.lfill_level;
        if (is_tail && !tail) break;
        // the root's left child lies after the root in `nodes`
        const unsigned char* at = nl > cap || !nodes ? nullptr : nodes + (lvl == 0 ? (size_t)z.nch * z_chunk_bytes(z) : 0);
        if (is_tail) EXAFAC_TRY(z_level_any<2>(s, t, G, at, lb, ex, J, p, order, dv, st));
        else EXAFAC_TRY(z_level_any<1>(s, t, G, at, lb, ex, J, p, order, dv, st));
        if (is_tail && t.F <= 1) break;  // the leaf index needs no order
        if (!in_smem)
            EXAFAC_TRY(scan_exclusive_u32_to_i64(reinterpret_cast<const uint32_t*>(b.tcount[p]), b.pref64, ntiles,
                                                 b.pref64 + ntiles, s.scan_sc, st));
        zq_partition_kernel<<<(unsigned)std::min<int64_t>(ceil_div(J, 512), 152 * 2), 512, psm, st>>>(
            J, (int)ntiles, b.mask[p], b.tcount[p], b.mask[p ^ 1], b.tcount[p ^ 1], b.runs[p ^ 1],
            in_smem ? nullptr : b.pref64, lb, nl, order, b.node, b.off[p], b.order[p], b.off[p ^ 1], s.R, G, ex,
            t.node_count, 2 * lb + 1, lvl + 1 < t.lfill_level + (tail ? 1 : 0) && 2 * nl <= cap ? 2 * nl : 0, nodes,
            b.lost);
        count_launch();
        order = b.order[p];
        p ^= 1;
        lb = 2 * lb + 1;
        nl *= 2;
    }
    if (t.F <= 1) {
        zq_leaf1_kernel<<<z_grid(J), 256, 0, st>>>(t, J, b, s.N, col, s.samples);
        count_launch();
    } else if (s.R <= 64) {
        EXAFAC_TRY(z_leaf<256>(s, t, G, U, J, p, order, dv, col, st));
    } else {
        EXAFAC_TRY(z_leaf<512>(s, t, G, U, J, p, order, dv, col, st));
    }
    if (t.F > 1) {
        zq_place_kernel<<<(unsigned)std::min<int64_t>(J, 152 * 4), kPlaceThreads, 0, st>>>(s.R, t, G, U, b, dv, s.N, col,
                                                                                         s.samples);
        count_launch();
    }
    EXAFAC_CHECK_LAUNCH();
    return EXAFAC_OK;
}

int sts_draw_zq(Session& s, int n, int64_t J, const double* uni, cudaStream_t st) {
    const int N = s.N, R = s.R, P = s.P;
    ZState& b = s.zq;
    double* h = s.D;  // J x R; the design rows are formed after the draw
    const unsigned vgrid = z_grid(J * 32);
    zq_vector_kernel<0><<<vgrid, 256, 0, st>>>(R, J, h, nullptr, nullptr, N, 0, 0, b, s.status);
    count_launch();
    for (int k = 0; k < N; k++) {
        if (k == n) continue;
        int nx = k + 1;
        if (nx == n) nx++;
        if (nx > N) nx = N;
        // eigen tree of mode k, driven by h: v, then x = h * E_next[v]
        EXAFAC_TRY(z_descend(s, s.etree, s.eigG + (int64_t)k * s.etree.node_count * P, nullptr,
                             uni + ((int64_t)k * 2 + 0) * J, J, n, 2 * k, st));
        zq_vector_kernel<1><<<vgrid, 256, 0, st>>>(R, J, h, s.Emat + (int64_t)nx * R * R, s.samples, N, n, R, b,
                                                   s.status);
        count_launch();
        // row tree of mode k, driven by x: the row, then h *= U_k[row]
        EXAFAC_TRY(z_descend(s, s.rtree[k], s.treeG[k], s.F.U[k], uni + ((int64_t)k * 2 + 1) * J, J, k, 2 * k + 1, st));
        zq_vector_kernel<2><<<vgrid, 256, 0, st>>>(R, J, h, s.F.U[k], s.samples, N, k, s.dims[k], b, s.status);
        count_launch();
    }
    zq_tree_exp_kernel<<<1, 256, 0, st>>>(R, s.PhiP, b.tree_exp + 2 * N, 0, nullptr);
    count_launch();
    const size_t smem = zw_smem(R);
    const unsigned blocks = (unsigned)std::min<int64_t>(ceil_div(J, kZTile), 152);
    EXAFAC_CUDA_TRY(allow_smem(zq_weight_kernel));
    zq_weight_kernel<<<blocks, kWThreads, smem, st>>>(R, J, b, s.PhiP, b.tree_exp + 2 * N, s.weights, s.status,
                                                     s.wait_polls ? s.wait_polls : kSpinLimit, s.withheld(25));
    count_launch();
    EXAFAC_CHECK_LAUNCH();
    return EXAFAC_OK;
}

}  // namespace exafac
