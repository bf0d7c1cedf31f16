// gemm_sliced.cu -- FP64 products on the tcgen05 tensor cores.
//
// GB300 issues 2 FP64 FMAs per SM per clock (1.25 TFLOP/s on the device) and
// 4096 BF16 FMAs.  The product is therefore taken apart into exact integer
// products (the error-free splitting of Ozaki, Ogita, Oishi and Rump, "Error-
// free transformations of matrix multiplication", Numer. Algorithms 2012):
// every row of A and every column of B is scaled by a power of two and cut
// into kSlices = 8 signed digits of 8 bits, |digit| <= 128, stored as BF16
// (exact).  Digit products are integers up to 2^14, so an FP32 accumulator in
// tensor memory holds the sum of up to 1024 of them exactly: the (at most 8)
// digit pairs (i, j) with i + j = d over a chunk of 128 in K share one
// accumulator, d = 0..7, and pairs with i + j > 7 (below 2^-64 of the largest
// product) are left out: 36 of 64.  The epilogue adds the eight accumulators
// into a 96-bit integer per element of C and rounds to FP64 once.
//
// Accuracy: an element's error is about 2^-64 sqrt(K) times (row maximum of A
// x column maximum of B), against 2^-54 of sum |a||b| for a chain of FMAs.
// That is smaller unless the row's and the column's large entries do not
// meet, i.e. unless sum |a||b| < 2^-9 sqrt(K) of that product of maxima.  Two
// looks decide that before a tile is multiplied: the slicing kernel counts,
// per vector, the entries within 2^-4 of the largest, and where the fewest of
// the tile's rows and columns must overlap in 1.75 sqrt(K) places (pigeonhole)
// the tile is good; otherwise the CTA sums the products of the leading digits'
// moduli, which ends as soon as every element has passed.  A tile that fails
// both, or has an entry that is not finite or a vector of extreme scale, is put
// on a list and multiplied by a kernel of its own on the FP64 pipe, from the
// unsliced operands and with the FMA chain of gemm_simt_kernel (the second look
// keeps tiles of ordinary data, of which one in some thousand fails the first,
// off that list).
//
// Data flow per CTA (persistent over 128 x 64 tiles of C): one thread loads
// stages of K = 32 (8 digits x (128 + 64) rows x 64 bytes = 96 KB, two
// stages) by TMA into 64-byte-swizzled shared memory; one thread multiplies
// digit i of A with digits 0..7-i of B at once (they lie behind one another
// in shared memory, and so do their accumulators in the 512 TMEM columns:
// N = 64 (8 - i), in pieces of up to 256, so that A is read once per 256
// columns); sixteen warps drain the accumulators after every K = 128.  Short K
// takes tiles of 128 x 32: two sets of accumulators fit, and one tile is
// multiplied while another is drained.
// All waits are bounded; on a timeout the kernel records kDevTimeout.
#include <cuda.h>
#include <cudaTypedefs.h>

#include "async.cuh"
#include "gemm_sliced.cuh"

#include <algorithm>
#include <climits>
#include <cmath>

namespace tmvg {

constexpr int kSlices = 8;
constexpr int kSlM = 128, kSlN = 64;    // tile of C (short K: 128 x 32)
constexpr int kSlK = 32;                // K per stage: 64 bytes of BF16
constexpr int kSlChunk = 4;             // stages per accumulation chunk (K = 128)
constexpr int kSlStages = 2;
constexpr int kSlABytes = kSlices * kSlM * kSlK * 2;
constexpr int kSlEpiWarps = 16;  // 4 per scheduler: the epilogue is bound by latencies
constexpr int kSlThreads = 32 * (kSlEpiWarps + 2);
static_assert(kSlM / 16 * kSlN == 32 * kSlEpiWarps, "a prefetch per epilogue thread");
constexpr int kSlCols = kSlN / (kSlEpiWarps / 4);  // columns of C per epilogue thread
constexpr int kFillBad = -(1 << 29);    // fill count of a group that cannot be sliced
constexpr int kFillRange = 4;           // entries within 2^-4 of the vector's largest count
constexpr int kZeroExp = -(1 << 20);    // scale exponent of a zero vector
constexpr int kMaxTilesPerCta = 16384;
constexpr int kExpLimit = 450;          // |scale exponent| beyond this takes the FP64 pipe

size_t sliced_bytes(int64_t rows, int64_t K)
{
    const int64_t Kp = ceil_div(K, (int64_t)kSlK) * kSlK;
    return (size_t)kSlices * rows * Kp * 2 + 8 * ((size_t)rows + 64) + 512;
}

SlicedOperand sliced_layout(void* buf, int64_t rows, int64_t K)
{
    SlicedOperand s;
    s.rows = rows;
    s.Kp = ceil_div(K, (int64_t)kSlK) * kSlK;
    s.group = K <= kSlK ? 64 : 16;
    s.digits = static_cast<uint16_t*>(buf);
    s.exps = reinterpret_cast<int*>(s.digits + (size_t)kSlices * rows * s.Kp);
    s.fill = s.exps + rows;
    return s;
}

// ---------------------------------------------------------------------
// Slicing.  A CTA takes R vectors; the first pass over them finds the largest
// exponent, the second (from L2) cuts the digits with integer operations
// only (the FP64 pipe would take 2 elements per SM per clock).  Bound: 8
// bytes read and 16 written per element.
// ---------------------------------------------------------------------
constexpr int kSplitThreads = 256;

// Element (r, k) of an operand; Z: of a complex matrix's real form.
template <bool Z>
__device__ __forceinline__ double sl_at(const double* __restrict__ p, int64_t sr, int64_t sk, int64_t r, int64_t k)
{
    if constexpr (!Z) return __ldg(p + r * sr + k * sk);
    const double v = __ldg(p + 2 * ((r >> 1) * sr + (k >> 1) * sk) + ((r ^ k) & 1));
    return (r & 1) < (k & 1) ? -v : v;
}

struct SplitSide {
    const double* p;
    int64_t sr, sk;   // element (vector r, place k) at p[r*sr + k*sk]
    uint16_t* digits;
    int* exps;
    int* fill;
    int64_t rows, Kp;
};

// value = (-1)^s X 2^(E - 63) with E the vector's scale, as 8 balanced bytes
__device__ __forceinline__ unsigned long long fixed63(double v, int emax)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const int ef = (int)((b >> 52) & 0x7ff);
    unsigned long long x = (b & 0x000fffffffffffffull) | 0x0010000000000000ull;
    const int sh = 10 - (emax - ef);
    if (ef == 0 || sh < -53) x = 0;  // zero, subnormal, or below the last digit
    else if (sh >= 0) x <<= sh;
    else x = (x + (1ull << (-sh - 1))) >> (-sh);
    return (b >> 63) ? 0ull - x : x;
}

template <int R, bool Z>
__device__ __forceinline__ void split_vectors(const SplitSide& s, int64_t grp, int64_t K)
{
    constexpr int G = kSplitThreads / R;  // threads sharing a vector
    __shared__ int s_emax[R], s_big[R];
    __shared__ int s_min;
    const int tid = threadIdx.x;
    const bool kc = s.sk == 1;  // K contiguous: neighbouring threads take neighbouring k
    const int r = kc ? tid / G : tid % R;
    const int g = kc ? tid % G : tid / R;
    const int64_t row = grp * R + r;
    const bool have = row < s.rows;
    const double* p = Z ? s.p : s.p + row * s.sr;
    const int64_t zr = Z ? row : 0;
    if (tid < R) {
        s_emax[tid] = 0;
        s_big[tid] = 0;
    }
    if (tid == 0) s_min = INT_MAX;
    __syncthreads();
    if (have) {
        int e = 0;
#pragma unroll 8
        for (int64_t k = g; k < K; k += G)
            e = max(e, (int)((unsigned)__double2hiint(sl_at<Z>(p, s.sr, s.sk, zr, k)) >> 20 & 0x7ff));
        atomicMax(&s_emax[r], e);
    }
    __syncthreads();
    const int emax = s_emax[r];
    int big = 0;
    if (have) {
        const size_t slice = (size_t)s.rows * s.Kp;
        for (int64_t k0 = (int64_t)g * 8; k0 < s.Kp; k0 += G * 8) {
            double v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = k0 + q < K ? sl_at<Z>(p, s.sr, s.sk, zr, k0 + q) : 0.0;
            uint32_t w[kSlices][4];
#pragma unroll
            for (int q = 0; q < 8; q += 2) {
                uint32_t lo[2], hi[2], top[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int ef = (int)((unsigned)__double2hiint(v[q + h]) >> 20 & 0x7ff);
                    big += ef != 0 && ef >= emax - kFillRange;
                    const unsigned long long x = fixed63(v[q + h], emax);
                    // adding 128 to every byte below the top one makes each an
                    // unsigned digit + 128, with the carries resolved
                    const unsigned long long y = (x & 0x00ffffffffffffffull) + 0x0080808080808080ull;
                    lo[h] = (uint32_t)y;
                    hi[h] = (uint32_t)(y >> 32);
                    top[h] = (uint32_t)((int)((long long)x >> 56) + (int)(hi[h] >> 24) + 128);
                }
                // byte b -> the BF16 of b - 128: 2^23 + b, less 2^23 + 128, is exact
                auto bf = [](uint32_t byte) {
                    return __float_as_uint(__uint_as_float(0x4b000000u | byte) - 8388736.0f);
                };
                w[0][q / 2] = __byte_perm(bf(top[0]), bf(top[1]), 0x7632);
#pragma unroll
                for (int d = 1; d < kSlices; ++d) {
                    const int at = 7 - d;  // byte of y
                    const uint32_t b0 = ((at < 4 ? lo[0] : hi[0]) >> (8 * (at & 3))) & 0xff;
                    const uint32_t b1 = ((at < 4 ? lo[1] : hi[1]) >> (8 * (at & 3))) & 0xff;
                    w[d][q / 2] = __byte_perm(bf(b0), bf(b1), 0x7632);
                }
            }
            uint16_t* dst = s.digits + (size_t)row * s.Kp + k0;
#pragma unroll
            for (int d = 0; d < kSlices; ++d)
                *reinterpret_cast<uint4*>(dst + d * slice) = make_uint4(w[d][0], w[d][1], w[d][2], w[d][3]);
        }
        atomicAdd(&s_big[r], big);
    }
    __syncthreads();
    if (tid < R && grp * R + tid < s.rows) {
        const int ee = s_emax[tid];  // exponent field: |entries| < 2^(ee - 1022)
        int b = s_big[tid];
        const int sc = ee == 0 ? kZeroExp : ee - 1022;
        if (ee == 0) b = INT_MAX / 4;  // a zero vector: every product is exactly zero (but see below)
        else if (ee == 0x7ff || sc > kExpLimit || sc < -kExpLimit) b = kFillBad;
        s.exps[grp * R + tid] = sc;
        atomicMin(&s_min, b);
    }
    // a vector of subnormals only would be sliced as zero: it takes the FP64 pipe
    if (have && s_emax[r] == 0) {
        bool sub = false;
        for (int64_t k = g; k < K; k += G) sub |= (__double_as_longlong(sl_at<Z>(p, s.sr, s.sk, zr, k)) << 1) != 0;
        if (sub) atomicMin(&s_min, kFillBad);
    }
    __syncthreads();
    if (tid == 0) s.fill[grp] = s_min;
}

// Both operands in one launch: groups_a CTAs for A, the rest for B.
// `listed`: the count of the product's list, cleared here.
template <int R, bool ZLEFT>
__global__ void __launch_bounds__(kSplitThreads)
sliced_split_kernel(SplitSide sa, SplitSide sb, int64_t groups_a, int64_t K, int* listed)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) *listed = 0;
    if ((int64_t)blockIdx.x < groups_a) split_vectors<R, ZLEFT>(sa, blockIdx.x, K);
    else split_vectors<R, false>(sb, blockIdx.x - groups_a, K);
}

static tmvg_status sliced_split(Context* c, int64_t K, Mat<const double> A, const SlicedOperand& sa,
                                Mat<const double> B, const SlicedOperand& sb, int* listed, bool zleft)
{
    const int R = sa.rows ? sa.group : sb.group;
    const SplitSide a{A.p, A.si, A.sj, sa.digits, sa.exps, sa.fill, sa.rows, sa.Kp};
    const SplitSide b{B.p, B.sj, B.si, sb.digits, sb.exps, sb.fill, sb.rows, sb.Kp};
    const int64_t ga = ceil_div(sa.rows, (int64_t)R), gb = ceil_div(sb.rows, (int64_t)R);
    auto kern = R == 64 ? (zleft ? sliced_split_kernel<64, true> : sliced_split_kernel<64, false>)
                        : (zleft ? sliced_split_kernel<16, true> : sliced_split_kernel<16, false>);
    kern<<<(unsigned)(ga + gb), kSplitThreads, 0, c->stream>>>(a, b, ga, K, listed);
    ++c->launches;
    return check_cuda(c, cudaGetLastError(), "sliced split launch");
}

// ---------------------------------------------------------------------
// The product.
// ---------------------------------------------------------------------
__device__ __forceinline__ void sl_tma_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
            smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(0)
        : "memory");
}

__device__ __forceinline__ void sl_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void sl_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor: K-major, 64-byte swizzle, rows of 64 bytes
// in 8-row (512-byte) groups.
__device__ __forceinline__ uint64_t sw64_desc(uint32_t addr)
{
    uint64_t d = (addr >> 4) & 0x3FFFull;
    d |= 1ull << 16;
    d |= (uint64_t)(512 >> 4) << 32;
    d |= 1ull << 46;
    d |= 4ull << 61;
    return d;
}

// Instruction descriptor: D FP32, A and B BF16, both K-major, M = 128.
__device__ __forceinline__ uint32_t bf16_idesc(int n)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kSlM >> 4) << 24);
}

__device__ __forceinline__ void sl_umma(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

__device__ __forceinline__ void sl_commit(uint64_t* bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void sl_ld4(uint32_t taddr, uint32_t (&v)[4])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                 : "r"(taddr)
                 : "memory");
}

__device__ __forceinline__ void sl_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// One chunk's eight accumulators of an element as p 2^32 + q in units of
// 2^-62: p = a0 2^16 + a1 2^8 + a2, q = a3 2^24 + a4 2^16 + a5 2^8 + a6 +
// a7 2^-8.  The accumulators are integers: |a_d| <= (d + 1) 2^21, so a0 and
// a1 (up to 2^22) convert by one FP32 addition of 1.5 2^23, whose mantissa
// then holds the integer; a2..a5 take the converter (16 per SM per clock);
// a6 + a7 2^-8 is rounded to a multiple of 4 (2^-60) by the same addition.
__device__ __forceinline__ void sl_combine(const uint32_t (&a)[kSlices], long long& p, long long& q)
{
    constexpr float kMagic = 12582912.0f;  // 1.5 2^23
    constexpr uint32_t kBits = 0x4b400000u;
    const uint32_t b0 = __float_as_uint(__uint_as_float(a[0]) + kMagic);
    const uint32_t b1 = __float_as_uint(__uint_as_float(a[1]) + kMagic);
    const int s = (int)(b0 * 256u + b1 - (kBits * 257u));
    const int i2 = __float2int_rn(__uint_as_float(a[2]));
    const int i3 = __float2int_rn(__uint_as_float(a[3]));
    const int i4 = __float2int_rn(__uint_as_float(a[4]));
    const int i5 = __float2int_rn(__uint_as_float(a[5]));
    const float f = fmaf(__uint_as_float(a[7]), 0.00390625f, __uint_as_float(a[6]));
    const int i6 = (int)(__float_as_uint(fmaf(f, 0.25f, kMagic)) - kBits);
    p = (long long)s * 256 + i2;
    q = (long long)i3 * 16777216 + ((long long)i4 * 65536 + ((long long)i5 * 256 + (long long)i6 * 4));
}

// A chunk's eight accumulators of one element into its 96-bit sum: q + (p << 32).
__device__ __forceinline__ void sl_add(const uint32_t (&a)[kSlices], uint32_t& t0, uint32_t& t1, uint32_t& t2)
{
    long long p, q;
    sl_combine(a, p, q);
    const uint32_t q0 = (uint32_t)q, q1 = (uint32_t)((unsigned long long)q >> 32);
    const uint32_t p0 = (uint32_t)p, p1 = (uint32_t)((unsigned long long)p >> 32);
    asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %5;"
        : "+r"(t0), "+r"(t1), "+r"(t2)
        : "r"(q0), "r"(q1), "r"((uint32_t)((int)q1 >> 31)));
    asm("add.cc.u32 %0, %0, %2;\n\taddc.u32 %1, %1, %3;" : "+r"(t1), "+r"(t2) : "r"(p0), "r"(p1));
}

// The 96-bit integer (w2:w1:w0) 2^(e - 62) rounded to FP64 (nearest; a tie
// goes away from zero), on the integer pipe and without branches.
__device__ __forceinline__ double sl_to_double(uint32_t w0, uint32_t w1, uint32_t w2, int e)
{
    const uint32_t sgn = (uint32_t)((int)w2 >> 31);
    uint32_t a, m, l;  // |w|
    asm("sub.cc.u32 %0, %3, %6;\n\tsubc.cc.u32 %1, %4, %6;\n\tsubc.u32 %2, %5, %6;"
        : "=r"(l), "=r"(m), "=r"(a)
        : "r"(w0 ^ sgn), "r"(w1 ^ sgn), "r"(w2 ^ sgn), "r"(sgn));
    int msb = 95;
#pragma unroll
    for (int q = 0; q < 2; ++q) {  // the leading word into a
        const bool z = a == 0u;
        a = z ? m : a;
        m = z ? l : m;
        l = z ? 0u : l;
        msb -= z ? 32 : 0;
    }
    const int lz = __clz((int)a);
    const uint32_t hi = __funnelshift_l(m, a, lz), lo = __funnelshift_l(l, m, lz);
    msb -= lz;
    const unsigned long long top = ((unsigned long long)hi << 32) | lo;
    const unsigned long long mant = (top >> 11) + ((lo >> 10) & 1u);
    const unsigned long long bits = ((unsigned long long)(uint32_t)(msb + e - 62 + 1023 - 1) << 52) + mant;
    const unsigned long long r = bits | ((unsigned long long)(sgn & 0x80000000u) << 32);
    return __longlong_as_double((long long)(a ? r : 0ull));
}

struct SlicedArgs {
    int64_t M, N, K;
    double alpha;
    int add;                         // beta
    int unit;                        // alpha: 1 or -1, or 0 for any other value
    const double *A, *B;             // the operands themselves (listed tiles)
    int64_t asi, asj, bsi, bsj;
    bool zleft;
    const int *ea, *eb, *fa, *fb;
    int ga, gb;                      // vectors per fill group
    int need;                        // first look: overlap that a sliced tile needs
    float need_sum;                  // second look: sum of leading digits' products
    const uint16_t *da, *db;         // leading digits, K contiguous (stride Kp)
    int64_t Kp;
    double* C;
    int64_t ldc;
    int64_t mt, nt;                  // tiles
    int silent;                      // the CTA that loads nothing (failure-path test; -1: none)
    int* listed;                     // the tiles for the FP64 pipe: their count, then their numbers
};

// Tile t of the persistent order: columns of 16 tile rows, so that the tiles
// in flight together share their operands in L2.
__device__ __forceinline__ void sl_tile(const SlicedArgs& g, int64_t t, int64_t& mi, int64_t& ni)
{
    constexpr int64_t GM = 16;
    const int64_t per = GM * g.nt, band = t / per, rem = t - band * per;
    const int64_t h = min(GM, g.mt - band * GM);
    mi = band * GM + rem % h;
    ni = rem / h;
}

// First look at a tile: 1 good, 0 undecided, -1 for the FP64 pipe.
template <int TN>
__device__ __forceinline__ int sl_look(const SlicedArgs& g, int64_t mi, int64_t ni)
{
    int a = INT_MAX / 4, b = INT_MAX / 4;
    const int64_t a1 = min((g.M - 1) / g.ga, (mi * kSlM + kSlM - 1) / g.ga);
    const int64_t b1 = min((g.N - 1) / g.gb, (ni * TN + TN - 1) / g.gb);
    for (int64_t i = mi * kSlM / g.ga; i <= a1; ++i) a = min(a, __ldg(&g.fa[i]));
    for (int64_t i = ni * TN / g.gb; i <= b1; ++i) b = min(b, __ldg(&g.fb[i]));
    if (a < 0 || b < 0) return -1;
    return (int64_t)a + b - g.K >= g.need ? 1 : 0;
}

// Second look (the whole CTA): the sum of |leading digit of a| |leading digit
// of b| over K reaches need_sum for every element, or the element's row or
// column is zero.  A warp's 32 x 16 elements as 2 x 2 BF16 tiles of the warp-wide
// tensor instruction (a tile that fails looks at all of K: by FMAs that took 3 us
// per 32 places, 640 us of a product of K = 2048).
template <int TN>
__device__ __noinline__ bool sl_look_again(const SlicedArgs& g, int64_t mi, int64_t ni)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q = lane >> 2, t = lane & 3;
    const bool work = warp < kSlEpiWarps / (kSlN / TN);
    const int64_t r0 = mi * kSlM + (warp & 3) * 32 + q;                 // rows r0 + 8 (0..3)
    const int64_t c0 = ni * TN + (int64_t)(warp >> 2) * kSlCols;        // columns
    // (rows and columns outside read the last one's digits; they do not vote.  A
    // lane reads eight neighbouring places, which stand for the places the
    // instruction would have it hold: the order of the sum is free)
    const uint4 *pa[4], *pb[2];
#pragma unroll
    for (int u = 0; u < 4; ++u) pa[u] = reinterpret_cast<const uint4*>(g.da + min(r0 + 8 * u, g.M - 1) * g.Kp) + t;
#pragma unroll
    for (int u = 0; u < 2; ++u) pb[u] = reinterpret_cast<const uint4*>(g.db + min(c0 + 8 * u + q, g.N - 1) * g.Kp) + t;
    constexpr uint32_t kAbs = 0x7fff7fffu;
    float sum[2][2][4] = {};
    // which of sum's elements need no more: bit 8 i + 4 j + e
    unsigned done = work ? 0u : 0xffffu;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int64_t r = r0 + 16 * i + 8 * (e >> 1), c = c0 + 8 * j + 2 * t + (e & 1);
                if (r >= g.M || c >= g.N || __ldg(&g.ea[min(r, g.M - 1)]) == kZeroExp ||
                    __ldg(&g.eb[min(c, g.N - 1)]) == kZeroExp)
                    done |= 1u << (8 * i + 4 * j + e);
            }
    const int64_t steps = g.Kp / kSlK;
    for (int64_t s0 = 0; s0 < steps; s0 += 2) {  // a vote every two
        if (__any_sync(0xffffffffu, done != 0xffffu)) {
            uint4 av[2][4], bv[2][2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int64_t at = 4 * min(s0 + h, steps - 1);
#pragma unroll
                for (int u = 0; u < 4; ++u) av[h][u] = __ldg(pa[u] + at);
#pragma unroll
                for (int u = 0; u < 2; ++u) bv[h][u] = __ldg(pb[u] + at);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (s0 + h >= steps) break;
#pragma unroll
                for (int x = 0; x < 2; ++x)  // words x, y and then z, w: 16 places each
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const uint4 &lo = av[h][2 * i], &hi = av[h][2 * i + 1];
                        const uint32_t a[4] = {(x ? lo.z : lo.x) & kAbs, (x ? hi.z : hi.x) & kAbs,
                                               (x ? lo.w : lo.y) & kAbs, (x ? hi.w : hi.y) & kAbs};
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            const uint32_t b0 = (x ? bv[h][j].z : bv[h][j].x) & kAbs;
                            const uint32_t b1 = (x ? bv[h][j].w : bv[h][j].y) & kAbs;
                            asm volatile(
                                "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, "
                                "%7}, {%8, %9}, {%0, %1, %2, %3};"
                                : "+f"(sum[i][j][0]), "+f"(sum[i][j][1]), "+f"(sum[i][j][2]), "+f"(sum[i][j][3])
                                : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
                        }
                    }
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (sum[i][j][e] >= g.need_sum) done |= 1u << (8 * i + 4 * j + e);
        }
        if (__syncthreads_and(done == 0xffffu)) return true;
    }
    return false;
}

template <int TN>
__host__ __device__ constexpr int sl_stage_bytes() { return kSlABytes + kSlices * TN * kSlK * 2; }

template <int TN>
__global__ void __launch_bounds__(kSlThreads, 1)
sliced_gemm_kernel(const __grid_constant__ CUtensorMap mA, const __grid_constant__ CUtensorMap mB,
                   const __grid_constant__ SlicedArgs g, int* err)
{
    // TN = 64: the accumulators of a tile take all 512 TMEM columns, and all
    // sixteen epilogue warps drain them.  TN = 32: two tiles' accumulators, and
    // eight warps for each, so that one tile is multiplied while the other is
    // drained, rounded and stored.
    constexpr int GR = kSlN / TN, GW = kSlEpiWarps / GR;
    constexpr int kStageBytes = sl_stage_bytes<TN>();
    extern __shared__ uint8_t sl_smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(sl_smem_raw) + 1023) &
                                               ~static_cast<uintptr_t>(1023));
    __shared__ __align__(8) uint64_t full[kSlStages], empty[kSlStages], acc_full[GR], acc_empty[GR], drained;
    __shared__ uint32_t s_tmem;
    __shared__ uint32_t s_ok[kMaxTilesPerCta / 32];
    __shared__ int s_open;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    if (warp == kSlEpiWarps) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int s = 0; s < kSlStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        s_open = 0;
        for (int s = 0; s < GR; ++s) {
            mbar_init(&acc_full[s], 1);
            mbar_init(&acc_empty[s], GW);
        }
        mbar_init(&drained, 1);
        mbar_fence_init();
    }
    sl_fence_before();
    __syncthreads();
    sl_fence_after();
    const uint32_t tmem = s_tmem;
    const int nst = (int)((g.K + kSlK - 1) / kSlK);
    const int64_t tiles = g.mt * g.nt;

    // which of this CTA's tiles are sliced, before the warps part
    const int mine = (int)((tiles - blockIdx.x + gridDim.x - 1) / gridDim.x);
    for (int i0 = warp * 32; i0 < mine; i0 += kSlThreads) {
        int64_t mi, ni;
        int look = 1;
        if (i0 + lane < mine) {
            sl_tile(g, blockIdx.x + (int64_t)(i0 + lane) * gridDim.x, mi, ni);
            look = sl_look<TN>(g, mi, ni);
        }
        const unsigned good = __ballot_sync(0xffffffffu, look == 1);
        if (lane == 0) {
            s_ok[i0 >> 5] = good;
            if (good != 0xffffffffu) s_open = 1;
        }
    }
    __syncthreads();
    if (s_open) {
        for (int i = 0; i < mine; ++i) {
            if ((s_ok[i >> 5] >> (i & 31)) & 1u) continue;
            int64_t mi, ni;
            const int64_t t = blockIdx.x + (int64_t)i * gridDim.x;
            sl_tile(g, t, mi, ni);
            const bool again = sl_look<TN>(g, mi, ni) == 0 && sl_look_again<TN>(g, mi, ni);
            __syncthreads();  // every thread has read the word
            if (tid == 0) {
                if (again) s_ok[i >> 5] |= 1u << (i & 31);
                else g.listed[1 + atomicAdd(g.listed, 1)] = (int)t;
            }
            __syncthreads();
        }
    }
    auto sliced = [&](int i) { return ((s_ok[i >> 5] >> (i & 31)) & 1u) != 0u; };

    if (warp == kSlEpiWarps) {
        // operands by TMA
        if (lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            for (int i = 0; i < mine && ok && (int)blockIdx.x != g.silent; ++i) {
                if (!sliced(i)) continue;
                int64_t mi, ni;
                sl_tile(g, blockIdx.x + (int64_t)i * gridDim.x, mi, ni);
                for (int s = 0; s < nst; ++s, ++it) {
                    const uint32_t slot = it % kSlStages;
                    if (it >= kSlStages && !mbar_wait(&empty[slot], (it / kSlStages - 1) & 1)) {
                        ok = false;
                        break;
                    }
                    uint8_t* st = base + slot * kStageBytes;
                    mbar_expect_tx(&full[slot], (uint32_t)kStageBytes);
                    sl_tma_3d(st, &mA, &full[slot], s * kSlK, (int)(mi * kSlM));
                    sl_tma_3d(st + kSlABytes, &mB, &full[slot], s * kSlK, (int)(ni * TN));
                }
            }
            if (!ok) atomicCAS(err, (int)kDevOk, (int)kDevTimeout);
            // the last loads must have landed before the CTA leaves
            for (uint32_t q = it > kSlStages ? it - kSlStages : 0; q < it; ++q)
                mbar_wait(&full[q % kSlStages], (q / kSlStages) & 1);
        }
    } else if (warp == kSlEpiWarps + 1) {
        // products
        if (lane == 0) {
            uint32_t it = 0, ch[GR] = {};
            bool ok = true;
            for (int i = 0; i < mine && ok; ++i) {
                if (!sliced(i)) continue;
                const int gr = i % GR;
                const uint32_t acc0 = tmem + (uint32_t)(gr * kSlices * TN);
                for (int s = 0; s < nst && ok; ++s, ++it) {
                    const bool first = s % kSlChunk == 0;
                    if (first && ch[gr] > 0) ok = mbar_wait(&acc_empty[gr], (ch[gr] - 1) & 1);
                    const uint32_t slot = it % kSlStages;
                    ok = ok && mbar_wait(&full[slot], (it / kSlStages) & 1);
                    if (!ok) break;
                    sl_fence_after();
                    const uint32_t a0 = smem_u32(base + slot * kStageBytes), b0 = a0 + kSlABytes;
#pragma unroll
                    for (int kk = 0; kk < kSlK / 16; ++kk) {
                        const uint64_t bd = sw64_desc(b0 + kk * 32);
#pragma unroll
                        for (int d = 0; d < kSlices; ++d) {
                            const uint64_t ad = sw64_desc(a0 + d * (kSlM * kSlK * 2) + kk * 32);
                            const int cols = TN * (kSlices - d);
                            const uint32_t acc = (first && kk == 0 && d == 0) ? 0u : 1u;
                            const int n0 = cols < 256 ? cols : 256;
                            sl_umma(acc0 + TN * d, ad, bd, bf16_idesc(n0), acc);
                            if (cols > 256)
                                sl_umma(acc0 + TN * d + 256, ad, bd + ((256 * kSlK * 2) >> 4),
                                        bf16_idesc(cols - 256), acc);
                        }
                    }
                    sl_commit(&empty[slot]);
                    if (s % kSlChunk == kSlChunk - 1 || s == nst - 1) {
                        sl_commit(&acc_full[gr]);
                        ++ch[gr];
                    }
                }
            }
            if (!ok) atomicCAS(err, (int)kDevOk, (int)kDevTimeout);
            // every product must be done before the tensor memory goes back
            sl_commit(&drained);
            mbar_wait(&drained, 0);
        }
    } else {
        // the warps of a tile: warp w of them drains lanes 32 (w % 4).. (rows of
        // the tile) and columns 16 (w / 4).. of every accumulator
        const int gr = warp / GW, tg = tid - gr * GW * 32;
        const int rl = (warp & 3) * 32 + lane, ch0 = (tg >> 7) * kSlCols;
        const uint32_t tb = tmem + ((uint32_t)((warp & 3) * 32) << 16) + ch0 + gr * kSlices * TN;
        uint32_t ch = 0;
        bool ok = true;
        for (int i = gr; i < mine && ok; i += GR) {
            int64_t mi, ni;
            sl_tile(g, blockIdx.x + (int64_t)i * gridDim.x, mi, ni);
            const int64_t r = mi * kSlM + rl, col0 = ni * TN + ch0;
            const bool in = r < g.M;
            const int nc = (int)max((int64_t)0, min((int64_t)kSlCols, g.N - col0));
            double* Cp = g.C + r + col0 * g.ldc;
            if (!sliced(i)) continue;
            // this row's scale, and a column's per lane; C's first columns on
            // their way while the products run
            const int ea = in ? __ldg(&g.ea[r]) : 0;
            const int ebl = lane < nc ? __ldg(&g.eb[col0 + lane]) : 0;
            const bool add = g.add != 0;
            if (add && i + GR < mine) {
                // the next tile of C into L2: a line of 16 rows per thread
                int64_t mx, nx;
                sl_tile(g, blockIdx.x + (int64_t)(i + GR) * gridDim.x, mx, nx);
                const int64_t rx = mx * kSlM + 16 * (tg & 7), cx = nx * TN + (tg >> 3);
                if (rx < g.M && cx < g.N)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(g.C + rx + cx * g.ldc));
            }
            // one element rounded and into C (alpha +-1 by the sign bit)
            const auto store = [&](int j, uint32_t w0, uint32_t w1, uint32_t w2, double cold) {
                double v = sl_to_double(w0, w1, w2, ea + __shfl_sync(0xffffffffu, ebl, j));
                if (g.unit != 0) {
                    v = __hiloint2double(__double2hiint(v) ^ (g.unit & (int)0x80000000u), __double2loint(v));
                    if (add) v = cold + v;
                } else {
                    v = add ? fma(g.alpha, v, cold) : g.alpha * v;
                }
                if (in && j < nc) Cp[j * g.ldc] = v;
            };
            const auto load_c = [&](auto& cold, int j) {
#pragma unroll
                for (int e = 0; e < (int)(sizeof(cold) / sizeof(double)); ++e) cold[e] = (add && in && j + e < nc) ? Cp[(j + e) * g.ldc] : 0.0;
            };
            if constexpr (GR > 1) {
                // a single chunk: four columns at a time from the accumulators
                // into C, the next four on their way
                uint32_t v[2][kSlices][4];
                double cold[2][4];
                load_c(cold[0], 0);
                ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[gr], ch & 1));
                ++ch;
                if (!ok) break;
                sl_fence_after();
                __syncwarp();
#pragma unroll
                for (int d = 0; d < kSlices; ++d) sl_ld4(tb + d * TN, v[0][d]);
#pragma unroll
                for (int j = 0; j < kSlCols; j += 4) {
                    const int cur = (j >> 2) & 1;
                    __syncwarp();
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (j + 4 < kSlCols) {
#pragma unroll
                        for (int d = 0; d < kSlices; ++d) sl_ld4(tb + d * TN + j + 4, v[cur ^ 1][d]);
                        load_c(cold[cur ^ 1], j + 4);
                    } else {
                        // drained: the next products may start
                        sl_fence_before();
                        __syncwarp();
                        if (lane == 0) sl_arrive(&acc_empty[gr]);
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        uint32_t a[kSlices];
#pragma unroll
                        for (int d = 0; d < kSlices; ++d) a[d] = v[cur][d][e];
                        uint32_t t0 = 0u, t1 = 0u, t2 = 0u;
                        sl_add(a, t0, t1, t2);
                        store(j + e, t0, t1, t2, cold[cur][e]);
                    }
                }
            } else {
                constexpr int CB = 8;
                double cold[CB];
                load_c(cold, 0);
                uint32_t t0[kSlCols], t1[kSlCols], t2[kSlCols];
#pragma unroll
                for (int j = 0; j < kSlCols; ++j) t0[j] = t1[j] = t2[j] = 0u;
                for (int s = 0; s < nst; s += kSlChunk, ++ch) {
                    ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[gr], ch & 1));
                    if (!ok) break;
                    sl_fence_after();
#pragma unroll
                    for (int j = 0; j < kSlCols; j += 4) {
                        uint32_t v[kSlices][4];
                        __syncwarp();
#pragma unroll
                        for (int d = 0; d < kSlices; ++d) sl_ld4(tb + d * TN + j, v[d]);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                        if (j + 4 == kSlCols) {
                            // drained: the next products may start
                            sl_fence_before();
                            __syncwarp();
                            if (lane == 0) sl_arrive(&acc_empty[gr]);
                        }
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            uint32_t a[kSlices];
#pragma unroll
                            for (int d = 0; d < kSlices; ++d) a[d] = v[d][e];
                            sl_add(a, t0[j + e], t1[j + e], t2[j + e]);
                        }
                    }
                }
                if (!ok) break;
                // rounded and into C, the next columns of C loaded ahead
#pragma unroll
                for (int j0 = 0; j0 < kSlCols; j0 += CB) {
                    double next[CB];
                    if (j0 + CB < kSlCols) load_c(next, j0 + CB);
#pragma unroll
                    for (int q = 0; q < CB; ++q) store(j0 + q, t0[j0 + q], t1[j0 + q], t2[j0 + q], cold[q]);
#pragma unroll
                    for (int q = 0; q < CB; ++q) cold[q] = next[q];
                }
            }
            __syncwarp();
        }
        if (!ok && lane == 0) atomicCAS(err, (int)kDevOk, (int)kDevTimeout);
    }
    sl_fence_before();
    __syncthreads();
    // (at the end: the listed tiles' CTAs would hold the SMs that a smaller grid
    // leaves to others while they wait)
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (warp == kSlEpiWarps) {
        sl_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// ---------------------------------------------------------------------
// The listed tiles on the FP64 pipe, 8 x 8 entries of C at a time, one per
// thread, over all of this launch's CTAs: sixteen groups of two warps each.  The
// same chain of FMAs per entry as gemm_simt_kernel.  Bound: 2 FMAs per SM per
// clock; a single tile takes 128 groups K x 64 clocks.  In the kernel above, where
// a CTA multiplied its own, one tile took K x 4096 clocks, and the loader and the
// multiplier waited for it.  One CTA per SM (by its shared memory), so that a
// grid smaller than the device leaves the other SMs free.  Launched as a
// dependent of the kernel above, so that an empty list costs little
// (0.8 us at 1024 x 1024 x 1024; as a plain launch 4).  1024 x 1024 x 1024 with a NaN in A:
// 2.1 ms -> 0.33, A lower triangular 2.6 -> 0.33, 300 x 300 x 300 with such an A 0.79 -> 0.08.
// ---------------------------------------------------------------------
constexpr int kRestGroups = 16;  // (named barriers 0..15)
constexpr int kRestB = 8, kRestK = 32;
constexpr int kRestThreads = kRestGroups * kRestB * kRestB;
struct RestBlock {
    double a[kRestK][kRestB + 1], b[kRestK][kRestB + 1];
};
constexpr int kRestSmem = 120 * 1024;
static_assert(kRestGroups * sizeof(RestBlock) <= kRestSmem && kRestSmem > 114 * 1024, "one CTA per SM");

template <int TN, bool Z>
__global__ void __launch_bounds__(kRestThreads)
sliced_rest_kernel(const __grid_constant__ SlicedArgs g)
{
    constexpr int kSub = (kSlM / kRestB) * (TN / kRestB);  // per tile
    constexpr int kLoads = kRestK / kRestB;
    extern __shared__ __align__(16) unsigned char rest_smem[];
    const int group = threadIdx.x / (kRestB * kRestB), gt = threadIdx.x % (kRestB * kRestB);
    RestBlock& sh = reinterpret_cast<RestBlock*>(rest_smem)[group];
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int listed = g.listed[0];
    const int64_t items = (int64_t)listed * kSub;
    const int tx = gt % kRestB, ty = gt / kRestB;
    const bool ak = !Z && g.asj == 1, bk = g.bsi == 1;  // K contiguous
    auto a_at = [&](int t, int& r, int& k) { r = ak ? t / kRestK : t % kRestB, k = ak ? t % kRestK : t / kRestB; };
    auto b_at = [&](int t, int& q, int& k) { q = bk ? t / kRestK : t % kRestB, k = bk ? t % kRestK : t / kRestB; };
    auto sync = [&] { asm volatile("bar.sync %0, 64;" ::"r"(group) : "memory"); };
    for (int64_t it = (int64_t)group * gridDim.x + blockIdx.x; it < items; it += (int64_t)kRestGroups * gridDim.x) {
        int64_t mi, ni;
        // (one block of every tile after the other, the blocks in C first: they fall
        // evenly on the CTAs)
        sl_tile(g, g.listed[1 + it % listed], mi, ni);
        const int sub = (int)(it / listed);
        const int hb = (int)min((int64_t)(kSlM / kRestB), (g.M - mi * kSlM + kRestB - 1) / kRestB);
        const int wb = (int)min((int64_t)(TN / kRestB), (g.N - ni * TN + kRestB - 1) / kRestB);
        if (sub >= hb * wb) continue;
        const int64_t r0 = mi * kSlM + (sub % hb) * kRestB, c0 = ni * TN + (sub / hb) * kRestB;
        double pa[kLoads], pb[kLoads], acc = 0.0;
        auto load = [&](int64_t k0) {
#pragma unroll
            for (int u = 0; u < kLoads; ++u) {
                int r, q, k;
                a_at(gt + u * kRestB * kRestB, r, k);
                pa[u] = r0 + r < g.M && k0 + k < g.K ? sl_at<Z>(g.A, g.asi, g.asj, r0 + r, k0 + k) : 0.0;
                b_at(gt + u * kRestB * kRestB, q, k);
                pb[u] = c0 + q < g.N && k0 + k < g.K ? __ldg(&g.B[(k0 + k) * g.bsi + (c0 + q) * g.bsj]) : 0.0;
            }
        };
        load(0);
        for (int64_t k0 = 0; k0 < g.K; k0 += kRestK) {
            sync();  // the group is done with the last block
#pragma unroll
            for (int u = 0; u < kLoads; ++u) {
                int r, q, k;
                a_at(gt + u * kRestB * kRestB, r, k);
                sh.a[k][r] = pa[u];
                b_at(gt + u * kRestB * kRestB, q, k);
                sh.b[k][q] = pb[u];
            }
            sync();
            if (k0 + kRestK < g.K) load(k0 + kRestK);
            const int kn = (int)min((int64_t)kRestK, g.K - k0);
#pragma unroll 8
            for (int k = 0; k < kn; ++k) acc = fma(sh.a[k][tx], sh.b[k][ty], acc);
        }
        if (r0 + tx < g.M && c0 + ty < g.N) {
            double* cp = g.C + (r0 + tx) + (c0 + ty) * g.ldc;
            const double v = g.alpha * acc;
            *cp = g.add ? v + *cp : v;
        }
    }
}

static PFN_cuTensorMapEncodeTiled_v12000 sl_encode_fn()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
        cudaGetLastError();
        return (PFN_cuTensorMapEncodeTiled_v12000) nullptr;
    }();
    return fn;
}

static bool sl_map(CUtensorMap* map, const SlicedOperand& s, int box_rows)
{
    auto fn = sl_encode_fn();
    if (!fn) return false;
    cuuint64_t dims[3] = {(cuuint64_t)s.Kp, (cuuint64_t)s.rows, (cuuint64_t)kSlices};
    cuuint64_t strides[2] = {(cuuint64_t)s.Kp * 2, (cuuint64_t)s.rows * s.Kp * 2};
    cuuint32_t box[3] = {(cuuint32_t)kSlK, (cuuint32_t)box_rows, (cuuint32_t)kSlices};
    cuuint32_t estr[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, s.digits, dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// C (M x N, column-major) = alpha A B + beta C (beta 0 or 1) from the slices; A
// and B themselves are read only for listed tiles.  `max_ctas` bounds the
// persistent grid (0: one per SM).
static tmvg_status sliced_apply(Context* c, int64_t M, int64_t N, int64_t K, double alpha, Mat<const double> A,
                                const SlicedOperand& sa, Mat<const double> B, const SlicedOperand& sb, double beta,
                                double* C, int64_t ldc, int* listed, int max_ctas, bool zleft)
{
    if (M <= 0 || N <= 0 || K <= 0) return TMVG_OK;
    CUtensorMap mA, mB;
    // a single chunk takes tiles of 32 columns, whose epilogues overlap (alpha
    // A B + C, normal data, 64 against 32 columns: 4096 x 4096 x 32 139 -> 123
    // us, 8192 x 8192 x 32 496 -> 435, 2048 x 2048 x 64 52 -> 43.5, 700 x 700 x 32
    // 31 -> 19), except a full one over many tiles, where reading A's digits
    // twice as often costs more (4096 x 4096 x 128: 156 -> 167; 2048 x 2048 x 128:
    // 56 -> 54)
    const int64_t cap = max_ctas > 0 ? max_ctas : c->num_sms;
    const bool narrow = K <= (kSlChunk - 1) * kSlK ||
                        (K <= kSlChunk * kSlK && ceil_div(M, (int64_t)kSlM) * ceil_div(N, (int64_t)kSlN) <= 4 * cap);
    const int tn = narrow ? 32 : kSlN;
    if (!sl_map(&mA, sa, kSlM) || !sl_map(&mB, sb, tn))
        return set_error(c, TMVG_CUDA_ERROR, "sliced product: tensor map encoding failed");
    SlicedArgs g;
    g.M = M, g.N = N, g.K = K, g.alpha = alpha, g.add = beta != 0.0, g.unit = alpha == 1.0 ? 1 : alpha == -1.0 ? -1 : 0;
    g.A = A.p, g.asi = A.si, g.asj = A.sj, g.zleft = zleft;
    g.B = B.p, g.bsi = B.si, g.bsj = B.sj;
    g.ea = sa.exps, g.eb = sb.exps, g.fa = sa.fill, g.fb = sb.fill, g.ga = sa.group, g.gb = sb.group;
    // sum |a||b| of at least 2^-9.2 sqrt(K) of the product of the scales: an
    // entry within 2^-4 of its vector's largest is at least 2^-5 of the scale;
    // a leading digit d (of 2^7) stands for at least d / 2
    g.need = (int)std::ceil(1.75 * std::sqrt((double)K));
    g.need_sum = (float)(112.0 * std::sqrt((double)K));
    g.da = sa.digits, g.db = sb.digits, g.Kp = sa.Kp;
    g.C = C, g.ldc = ldc;
    g.mt = ceil_div(M, (int64_t)kSlM), g.nt = ceil_div(N, (int64_t)tn);
    g.listed = listed, g.silent = c->silenced(TMVG_SILENT_PRODUCT) ? 0 : -1;
    const unsigned grid = (unsigned)std::min<int64_t>(g.mt * g.nt, cap);
    auto kern = tn == 32 ? sliced_gemm_kernel<32> : sliced_gemm_kernel<kSlN>;
    const size_t smem = (size_t)kSlStages * (tn == 32 ? sl_stage_bytes<32>() : sl_stage_bytes<kSlN>()) + 1024;
    tmvg_status st = check_cuda(
        c, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "sliced product");
    if (st) return st;
    kern<<<grid, kSlThreads, smem, c->stream>>>(mA, mB, g, c->dflags);
    ++c->launches;
    if ((st = check_cuda(c, cudaGetLastError(), "sliced product launch"))) return st;
    auto rest = tn == 32 ? (zleft ? sliced_rest_kernel<32, true> : sliced_rest_kernel<32, false>)
                         : (zleft ? sliced_rest_kernel<kSlN, true> : sliced_rest_kernel<kSlN, false>);
    st = check_cuda(c, cudaFuncSetAttribute(rest, cudaFuncAttributeMaxDynamicSharedMemorySize, kRestSmem),
                    "sliced product");
    if (st) return st;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3((unsigned)cap);
    cfg.blockDim = dim3(kRestThreads);
    cfg.dynamicSmemBytes = kRestSmem;
    cfg.stream = c->stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    ++c->launches;
    return check_cuda(c, cudaLaunchKernelEx(&cfg, rest, g), "sliced product, listed tiles");
}

void* scratch_alloc(Context* c, size_t bytes, cudaStream_t s)
{
    if (!c->pool) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = c->device;
        if (cudaMemPoolCreate(&c->pool, &props) != cudaSuccess) {
            cudaGetLastError();
            c->pool = nullptr;
            return nullptr;
        }
        uint64_t keep = 1ull << 30;
        cudaMemPoolSetAttribute(c->pool, cudaMemPoolAttrReleaseThreshold, &keep);
    }
    void* p = nullptr;
    if (c->refuse & TMVG_BUFFER_POOL) return nullptr;
    if (cudaMallocFromPoolAsync(&p, bytes, c->pool, s) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return p;
}

void scratch_free(void* p, cudaStream_t s)
{
    if (p && cudaFreeAsync(p, s) != cudaSuccess) cudaGetLastError();
}

bool sliced_wanted(Context* c, int64_t M, int64_t N, int64_t K)
{
    if (M < 64 || N < 48 || K < 24 || M > INT_MAX / 2 || N > INT_MAX / 2) return false;
    if ((double)M * (double)N * (double)K < 1.2e7) return false;
    if (!c->may_pool) return false;
    if (!sl_encode_fn()) return false;
    // a captured stream keeps the FP64 pipe: its graph would hold scratch of
    // the pool
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(c->stream, &cap) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return cap == cudaStreamCaptureStatusNone;
}

tmvg_status sliced_gemm(Context* c, int64_t M, int64_t N, int64_t K, double alpha, Mat<const double> A,
                        Mat<const double> B, double beta, double* C, int64_t ldc, int max_ctas,
                        bool zleft)
{
    // blocks of at most 256 MiB of digits per operand
    constexpr int64_t kMaxK = 16384;
    // (blocks of K are added into C one after the other, each times alpha: an
    // infinite alpha, or one that takes a partial sum out of range, would not give
    // alpha times the sum)
    if (K > kMaxK && !(std::fabs(alpha) <= 0x1p60)) return TMVG_UNSUPPORTED;
    const int64_t kb = std::min(K, kMaxK);
    const int64_t cap = std::max<int64_t>(kSlM, (((int64_t)1 << 28) / (2 * kSlices * (kb + kSlK))) / kSlM * kSlM);
    const int64_t mb = std::min(M, cap);
    const int64_t nb = std::min(std::min(N, cap), std::max<int64_t>(1, kMaxTilesPerCta / ceil_div(mb, (int64_t)kSlM)) *
                                                      32 * (max_ctas > 0 ? max_ctas : c->num_sms));
    auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
    const size_t ba = al(sliced_bytes(mb, kb)), bb = al(sliced_bytes(nb, kb));
    const size_t bl = sizeof(int) * (size_t)(1 + ceil_div(mb, (int64_t)kSlM) * ceil_div(nb, (int64_t)32));
    unsigned char* ws = (unsigned char*)scratch_alloc(c, ba + bb + bl, c->stream);
    if (!ws) return TMVG_UNSUPPORTED;
    int* listed = reinterpret_cast<int*>(ws + ba + bb);
    tmvg_status st = TMVG_OK;
    for (int64_t k0 = 0; k0 < K && !st; k0 += kb) {
        const int64_t k = std::min(kb, K - k0);
        for (int64_t i0 = 0; i0 < M && !st; i0 += mb) {
            const int64_t m = std::min(mb, M - i0);
            // (i0 and k0 are even: the real form's offsets are the same)
            const Mat<const double> a{A.p + i0 * A.si + k0 * A.sj, A.si, A.sj};
            const SlicedOperand sa = sliced_layout(ws, m, k);
            for (int64_t j0 = 0; j0 < N && !st; j0 += nb) {
                const int64_t n = std::min(nb, N - j0);
                const Mat<const double> b{B.p + k0 * B.si + j0 * B.sj, B.si, B.sj};
                const SlicedOperand sb = sliced_layout(ws + ba, n, k);
                SlicedOperand one = sa;
                if (j0 > 0) one.rows = 0;  // A's block is sliced already
                st = sliced_split(c, k, a, one, b, sb, listed, zleft);
                if (!st)
                    st = sliced_apply(c, m, n, k, alpha, a, sa, b, sb, k0 > 0 ? 1.0 : beta, C + i0 + j0 * ldc, ldc,
                                      listed, max_ctas, zleft);
            }
        }
    }
    scratch_free(ws, c->stream);
    return st;
}

}  // namespace tmvg
