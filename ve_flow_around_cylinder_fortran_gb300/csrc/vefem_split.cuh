// FP64 matrix product on the bf16 tensor cores: a 128 x 48 tile of A B from
// 64-bit fixed-point operands cut into eight digits.
//
// The FP64 pipe of this GPU does 2 multiply-adds per clock and SM, its tensor
// cores 4,096 in bf16.  An entry of A becomes an integer of 63 bits relative to
// the largest entry of its row (of B: of its column), written in eight balanced
// digits of base 256, d in [-128, 127]: exact in bf16.  Digit a of A times digit
// b of B has weight 256^(14-a-b); the products of equal a + b go to one FP32
// accumulator, where sums over up to 128 k are at most 2^24 and therefore exact
// integers.  The 43 pairs a + b <= 8 are kept.  The accumulators are added up in
// 64-bit integers, so a result is rounded once, at the end.  (The error-free
// splitting is that of Ozaki, Ogita, Oishi and Rump, "Error-free transformations
// of matrix multiplication", Numer. Algorithms 59, 2012.)
//
// Error: quantisation and dropped pairs are below 2^-60 of (largest entry of the
// row) x (largest entry of the column) per k.  The inner index is first scaled by
// powers of two, exactly, so that every row of B has the same largest exponent
// (inner_exponent): neither the units of the unknowns (stresses, velocities,
// pressures) nor the size of a pivot then cost digits.  On the Schur
// complements of a 2,000-quad Jacobian the error against extended precision is a
// quarter of an FP64 product's (all its fronts and rows no larger); with the
// pairs a + b <= 7 alone, or A's columns evened too, single rows were 2 to 14
// times worse and the residual of a solve grew by 40%.  FP64 is the better one
// for entries that spread inside a row or column by more than powers of two of
// rows, columns and inner indices even: an entry 2^-10 of the largest in the
// scaled row keeps fewer than 53 bits, one below 2^-62 of it none.  What that does
// to a solve stands at the elimination (vefem_tree.cu).
//
// One tcgen05.mma takes a digit of A (128 x 16) against several digits of B,
// laid out as one operand of up to 256 columns: 13 instructions per 16 k with 48
// columns, 9 with 32.
// Operands are cut by the CTA's 16 warps straight into the core-matrix layout
// (8 rows x 16 bytes, no swizzle), 32 k a stage; the nine accumulators take 432 of the SM's 512
// tensor memory columns, which is why a tile has 48 columns and not 64.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace split {

constexpr int TM = 128, TN = 48;       // tile
constexpr int KS = 32;                 // k per stage
constexpr int EXACT_K = 128;           // k per exact FP32 sum: 8 pairs x 128 x 2^14 = 2^24
constexpr int ND = 8;                  // digits
constexpr int NA = 9;                  // accumulators: sums of digit numbers kept
constexpr int TMEM = 512;              // columns taken (a power of two)
static_assert(NA * TN <= TMEM, "tensor memory");
constexpr int THREADS = 512;
constexpr int LBO_A = ND * TM * 16;    // bytes between k-neighbouring core matrices
constexpr int LBO_B = ND * TN * 16;
constexpr int STAGE_A = (KS / 8) * LBO_A, STAGE_B = (KS / 8) * LBO_B;
constexpr int STAGE = STAGE_A + STAGE_B;
constexpr int OUT_LD = TN + 1;         // the result tile, in the stages' place
static_assert(TM * OUT_LD * 8 <= STAGE, "result tile");
constexpr int NOT_FINITE = 1 << 20;    // exponent of a row or column with an infinity or NaN
constexpr int EMPTY = -(1 << 20);      // ... of one with zeros only

// exponent field of the high word of |x|: 1 for subnormal numbers too
__device__ __forceinline__ int field_of(int hi) { return max((hi >> 20) & 0x7ff, 1); }

// high word of |x|, 0 for infinities and NaN
__device__ __forceinline__ int finite_high(double x)
{
    const int hi = __double2hiint(x) & 0x7fffffff;
    return hi < 0x7ff00000 ? hi : 0;
}

// power of two applied to column k of A (its inverse to row k of B) from the
// largest high word of |B[k,:]|
__device__ __forceinline__ int inner_exponent(int hi_b) { return hi_b ? field_of(hi_b) - 1023 : 0; }

// exponent of x 2^s for a row's or column's largest
__device__ __forceinline__ int scaled_exponent(double x, int s)
{
    const int hi = __double2hiint(x) & 0x7fffffff;
    if (hi >= 0x7ff00000) return NOT_FINITE;
    return (hi | __double2loint(x)) == 0 ? EMPTY : field_of(hi) + s;
}

// x 2^s 2^(1084 - top) to the nearest integer, biased by 128 in every byte
__device__ __forceinline__ uint64_t fixed_point(double x, int s, int top)
{
    const int hi = __double2hiint(x);
    const uint64_t m = ((uint64_t)((hi & 0xfffff) | ((hi & 0x7ff00000) ? 0x100000 : 0)) << 32) |
                       (uint32_t)__double2loint(x);
    const int sh = min(max(top - (field_of(hi) + s), 0), 63);
    const uint64_t v = (((m << 10) >> sh) + 1) >> 1;
    return hi < 0 ? 0x8080808080808080ull - v : 0x8080808080808080ull + v;
}

// the digits of eight k of one row, 16 bytes per digit, digits a stride apart
__device__ __forceinline__ void put_digits(char *dst, int stride, const uint64_t (&w)[8])
{
#pragma unroll
    for (int a = 0; a < ND; a++) {
        uint32_t r[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint32_t w0 = (uint32_t)(w[2 * u] >> (a < 4 ? 32 : 0)), w1 = (uint32_t)(w[2 * u + 1] >> (a < 4 ? 32 : 0));
            // 2^23 + byte, less 2^23 + 128: a small integer, its bf16 the upper half
            const float f0 = __uint_as_float(__byte_perm(w0, 0x4b000000u, 0x7440u | (3 - (a & 3)))) - 8388736.0f;
            const float f1 = __uint_as_float(__byte_perm(w1, 0x4b000000u, 0x7440u | (3 - (a & 3)))) - 8388736.0f;
            r[u] = __byte_perm(__float_as_uint(f0), __float_as_uint(f1), 0x7632);
        }
        *reinterpret_cast<uint4 *>(dst + a * stride) = make_uint4(r[0], r[1], r[2], r[3]);
    }
}

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// K-major operand without swizzle: leading offset along k, stride offset along rows
__device__ __forceinline__ uint64_t operand(uint32_t addr, int lbo)
{
    return (uint64_t)((addr >> 4) & 0x3fff) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(128 >> 4) << 32) | (1ull << 46);
}

__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, int n, uint32_t accumulate)
{
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n / 8) << 17) | ((uint32_t)(TM / 16) << 24);
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                 " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d), "l"(a), "l"(b), "r"(idesc),
                 "r"(accumulate)
                 : "memory");
}

// bounded: the products of a stage take microseconds
__device__ __forceinline__ bool wait(uint32_t bar, uint32_t parity)
{
    for (int i = 0; i < (1 << 20); i++) {
        uint32_t ok;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                     : "=r"(ok)
                     : "r"(bar), "r"(parity)
                     : "memory");
        if (ok) return true;
    }
    return false;
}

// four columns of a warp's 32 rows; the values are there after tmem_wait
__device__ __forceinline__ void tmem_load(uint32_t addr, uint32_t (&r)[4])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
__device__ __forceinline__ void tmem_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// hi 2^40 + lo += four columns of the nine accumulators, N columns apart (the
// one of a + b = d is at most (d + 1) 2^21 in size, and 2^24).  Five and four
// loads in flight: a wait after each made a tile's rounding wait 27 times.
template <int N>
__device__ __forceinline__ void add_sums(uint32_t addr, int64_t *hi, int64_t *lo)
{
    uint32_t r[5][4];
    auto at = [&](int d, int i) { return __float2int_rn(__uint_as_float(r[d][i])); };
#pragma unroll
    for (int d = 0; d < 4; d++) tmem_load(addr + d * N, r[d]);
    tmem_wait();
#pragma unroll
    for (int d = 0; d < 4; d++)
#pragma unroll
        for (int i = 0; i < 4; i++) asm volatile("" : "+r"(r[d][i]));  // not read before the wait
#pragma unroll
    for (int i = 0; i < 4; i++)
        hi[i] += (int64_t)(at(0, i) * 256 + at(1, i)) * 65536 + (at(2, i) * 256 + at(3, i));
#pragma unroll
    for (int d = 0; d < 5; d++) tmem_load(addr + (d + 4) * N, r[d]);
    tmem_wait();
#pragma unroll
    for (int d = 0; d < 5; d++)
#pragma unroll
        for (int i = 0; i < 4; i++) asm volatile("" : "+r"(r[d][i]));
#pragma unroll
    for (int i = 0; i < 4; i++)
        lo[i] += ((int64_t)at(0, i) * 256 + at(1, i)) * 16777216 + ((int64_t)at(2, i) * 256 + at(3, i)) * 256 + at(4, i);
}

// (hi 2^40 + lo) 2^e rounded to a double, e from the largest exponents of row
// and column.  In integers: two conversions, a multiply-add and a scaling would
// be 64 clocks each per warp on the FP64 pipe, two thirds of a short tile.
__device__ __forceinline__ double rounded(int64_t hi, int64_t lo, int ta, int tb)
{
    if (max(ta, tb) >= NOT_FINITE / 2) return __longlong_as_double(0x7ff8000000000000ll);
    const int e = ta + tb - (2 * 1084 - 48);
    int64_t top = hi + (lo >> 40);                                 // with rem, a fraction of 64 bits
    uint64_t rem = (uint64_t)lo << 24;
    const uint64_t neg = (uint64_t)(top >> 63);
    top ^= neg;                                                    // less 2^-64 if negative: rounded away
    rem ^= neg;
    // the leading 64 bits, from words
    uint32_t w2 = (uint32_t)((uint64_t)top >> 32), w1 = (uint32_t)top, w0 = (uint32_t)(rem >> 32);
    int n = 0;
    if (w2 == 0) {
        w2 = w1;
        w1 = w0;
        w0 = (uint32_t)rem;
        n = 32;
        if (w2 == 0) {                                             // 2^46 below the largest possible
            if ((w1 | w0) == 0) return 0.0;
            if (w1 == 0) {
                w1 = w0;
                w0 = 0;
                n = 64;
            }
            w2 = w1;
            w1 = w0;
            w0 = 0;
            n += 32;
        }
    }
    const int z = __clz((int)w2);
    n += z;
    const uint32_t y1 = __funnelshift_l(w1, w2, z), y0 = __funnelshift_l(w0, w1, z);
    const uint64_t y = ((uint64_t)y1 << 32) | y0;
    const uint64_t mant = (y >> 11) + ((y0 >> 10) & 1);            // 2^52 .. 2^53, times 2^(51 - n + e)
    const int be = e + 51 - n + 52 + 1023;
    if (be < 1 || be >= 2046) {
        const double v = ldexp((double)mant, e + 51 - n);
        return neg ? -v : v;
    }
    return __longlong_as_double((long long)((((uint64_t)(be - 1) << 52) + mant) | (neg << 63)));
}

// count columns (a multiple of 4) of a warp's rows, from c0, rounded into out
template <int N, class TB>
__device__ __forceinline__ void round_columns(uint32_t tmem, int c0, int count, bool in, int ta, TB tb, double *out)
{
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
    for (int c = c0; c < c0 + count; c += 4) {
        int64_t hi[4], lo[4];
#pragma unroll
        for (int i = 0; i < 4; i++) hi[i] = lo[i] = 0;
        add_sums<N>(tmem + c, hi, lo);
        if (in)
#pragma unroll
            for (int i = 0; i < 4; i++) out[c + i] = rounded(hi[i], lo[i], ta, tb(c + i));
        __syncwarp();
    }
}

// 16 k: every digit of A with the digits of B it meets, N columns per digit.
// accumulate = 0 starts the sums: digit 0 of A writes a + b = 0 .. 7, digit 1
// with digit 7 of B writes a + b = 8.
template <int N>
__device__ __forceinline__ void mma_step(uint32_t tmem, uint32_t sa, uint32_t sb, int lbo_a, int lbo_b, uint32_t accumulate)
{
    constexpr int PER = 256 / N;                       // digits of B in one instruction
    const uint64_t da = operand(sa, lbo_a), db = operand(sb, lbo_b);
    auto go = [&](int a, int b, int count, uint32_t acc) { mma(tmem + (a + b) * N, da + a * TM, db + b * N, count * N, acc); };
#pragma unroll
    for (int a = 0; a < ND; a++) {
        const int digits = a == 1 ? ND - 1 : a == 0 ? ND : NA - a;
#pragma unroll
        for (int b = 0; b < digits; b += PER) go(a, b, digits - b < PER ? digits - b : PER, a == 0 ? accumulate : 1u);
        if (a == 1) go(a, ND - 1, 1, accumulate);
    }
}

__device__ __forceinline__ void tmem_alloc(uint32_t *slot)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(slot)), "n"(TMEM) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_free(uint32_t tmem)
{
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(TMEM) : "memory");
}

struct Operands {
    const double *a;        // rows of A, k contiguous, 16-byte aligned rows
    const double *b;        // rows k of B
    int64_t lda, ldb;
    int m, n, k;            // rows and columns left from the tile's corner, inner length
    const int32_t *s;       // inner exponents
    const int32_t *ta, *tb; // largest exponents of the tile's rows and columns
};

// out[row * OUT_LD + column] (shared) = the tile of A B; false (to all threads)
// if a wait ran out.  All THREADS threads call; smem: BUFFERS * STAGE bytes.
//
// Two stages, one CTA on an SM, for long products: the tensor core multiplies
// one stage while the next is cut.  One stage, two CTAs on an SM, for k <=
// EXACT_K: most of such a tile is its loads, its rounding and its update of the
// result, which the other CTA's share then covers; the tensor memory is taken
// after the first stage is cut.  512 threads (16 warps a CTA at 64 registers):
// with 256 at 128 a scheduler issued every fourth clock, 44.5 ms for 40.3.
template <int BUFFERS>
__device__ __forceinline__ bool product(char *smem, const Operands &o)
{
    __shared__ uint32_t s_tmem;
    __shared__ __align__(8) uint64_t s_bar[BUFFERS];
    constexpr int GROUPS = THREADS / TM;               // 8-k groups of A in one go
    constexpr int PART = TN / GROUPS;                  // columns of a warp's share
    constexpr bool LONG = BUFFERS > 1;
    const int t = threadIdx.x, warp = t >> 5;
    const uint32_t bar0 = smem_addr(&s_bar[0]);
    if (LONG && warp == 0) tmem_alloc(&s_tmem);
    if (t == 0) {
#pragma unroll
        for (int i = 0; i < BUFFERS; i++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8 * i) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    uint32_t tmem = LONG ? s_tmem : 0;

    const int ra = t & (TM - 1), g0 = t / TM;          // row and first 8-k group of A
    const int cb = t % TN, gb = t / TN;                // column and group of B (the first threads)
    const int top_a = ra < o.m ? o.ta[ra] : EMPTY, top_b = cb < o.n ? o.tb[cb] : EMPTY;
    const double *pa = o.a + (int64_t)min(ra, o.m - 1) * o.lda;
    int64_t hi[LONG ? PART : 1], lo[LONG ? PART : 1];
#pragma unroll
    for (int i = 0; i < (LONG ? PART : 1); i++) hi[i] = lo[i] = 0;
    auto drain = [&]() {
        const uint32_t mine = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((warp >> 2) * PART);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int c = 0; c < PART; c += 4) add_sums<TN>(mine + c, hi + c, lo + c);
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    };
    auto buffer = [&](int st) { return LONG ? st & 1 : 0; };
    auto parity = [&](int st) { return (uint32_t)((LONG ? st >> 1 : st) & 1); };

    const int steps = (o.k + KS - 1) / KS;
    bool ok = true;
    int sent = 0;                                      // stages handed to the tensor core
    for (int st = 0; st < steps; st++) {
        char *const stage = smem + buffer(st) * STAGE;
        if (st >= BUFFERS) ok = wait(bar0 + 8 * buffer(st), parity(st - BUFFERS));
        // the thread's groups of A and then its group of B, by one copy of the
        // code: unrolled, a tile streamed 90 KB of instructions through their
        // cache and waited for them half of the time.  Rows beyond m and
        // columns beyond n stay undefined, and unread.
#pragma unroll 1
        for (int i = 0; i <= KS / 8 / GROUPS; i++) {
            const bool is_b = i == KS / 8 / GROUPS;
            if (is_b ? t >= TN * (KS / 8) || cb >= o.n : ra >= o.m) continue;
            const int g = is_b ? gb : g0 + i * GROUPS, k0 = st * KS + g * 8;
            const double *from = is_b ? o.b + (int64_t)k0 * o.ldb + cb : pa + k0;
            const int64_t step = is_b ? o.ldb : 1;
            double x[8];
            int e[8];
            if (!is_b && k0 + 8 <= o.k) {
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const double2 v = __ldg(reinterpret_cast<const double2 *>(from) + u);
                    x[2 * u] = v.x;
                    x[2 * u + 1] = v.y;
                }
            } else {
#pragma unroll
                for (int u = 0; u < 8; u++) x[u] = k0 + u < o.k ? __ldg(from + u * step) : 0.0;
            }
#pragma unroll
            for (int u = 0; u < 8; u++) e[u] = k0 + u < o.k ? __ldg(o.s + k0 + u) : 0;
            uint64_t w[8];
            const int top = is_b ? top_b : top_a;
#pragma unroll
            for (int u = 0; u < 8; u++) w[u] = fixed_point(x[u], is_b ? -e[u] : e[u], top);
            put_digits(stage + (is_b ? STAGE_A + g * LBO_B + cb * 16 : g * LBO_A + ra * 16), is_b ? TN * 16 : TM * 16, w);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if constexpr (LONG) if (st > 0 && st % (EXACT_K / KS) == 0) {  // the exact sums are full
            ok = wait(bar0 + 8 * buffer(st - 1), parity(st - 1)) && ok;
            __syncwarp();
            if (__all_sync(0xffffffffu, ok)) drain();
        }
        if (!LONG && st == 0) {
            if (warp == 0) tmem_alloc(&s_tmem);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        }
        if (__syncthreads_or(!ok)) {
            ok = false;
            break;
        }
        if (!LONG) tmem = s_tmem;
        if (t == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t sa = smem_addr(stage), sb = sa + STAGE_A;
            const int halves = min(KS / 16, (o.k - st * KS + 15) / 16);
            for (int h = 0; h < halves; h++)
                mma_step<TN>(tmem, sa + h * 2 * LBO_A, sb + h * 2 * LBO_B, LBO_A, LBO_B,
                             (st % (EXACT_K / KS) != 0 || h > 0) ? 1u : 0u);
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             bar0 + 8 * buffer(st))
                         : "memory");
        }
        __syncwarp();
        sent = st + 1;
    }
    // the last stages' products (also after a failed wait, again bounded)
    bool done = true;
    if (LONG && sent > 1) done = wait(bar0 + 8 * buffer(sent - 2), parity(sent - 2));
    if (sent > 0) done = wait(bar0 + 8 * buffer(sent - 1), parity(sent - 1)) && done;
    ok = !__syncthreads_or(!(ok && done));
    double *out = reinterpret_cast<double *>(smem);
    const int row = (warp & 3) * 32 + (t & 31), col = (warp >> 2) * PART;
    const int ta = row < o.m ? o.ta[row] : EMPTY;
    if constexpr (LONG) {
        if (ok) drain();
        if (ok && row < o.m)
#pragma unroll
            for (int i = 0; i < PART; i++)
                out[row * OUT_LD + col + i] = rounded(hi[i], lo[i], ta, col + i < o.n ? o.tb[col + i] : EMPTY);
    } else if (ok) {
        round_columns<TN>(tmem + ((uint32_t)((warp & 3) * 32) << 16), col, PART, row < o.m, ta,
                          [&](int c) { return c < o.n ? __ldg(o.tb + c) : EMPTY; }, out + row * OUT_LD);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) tmem_free(tmem);
    return ok;
}

// programmatic launches: let the next kernel of the stream start, wait for the
// one before
__device__ __forceinline__ void launch_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ---- products of up to 32 inner indices: one stage, exponents found by the CTA

template <int N>
constexpr int SHORT_SMEM = (KS / 8) * ND * (TM + N) * 16;

// out[row * (N + 1) + column] (shared) = sum over k < 32 of A[row, k] B[k, column]
// for m rows and n columns; fa(row, k, x) and fb(column, k, x) give eight
// entries from k on, 0 for k outside.  EVEN_A: the columns of A, not the rows of
// B, are the ones evened (the transpose of a product evens its right factor so),
// and A is cut before b_ready() is called and B read.  The tensor memory is
// taken after the operands are cut: with two CTAs on an SM one cuts while the
// other multiplies.
template <int N, bool EVEN_A, class FA, class FB, class Ready>
__device__ __forceinline__ bool short_product(char *smem, int m, int n, FA fa, FB fb, Ready b_ready)
{
    constexpr int LA = ND * TM * 16, LB = ND * N * 16;
    static_assert(TM * (N + 1) * 8 <= SHORT_SMEM<N>, "result tile");
    static_assert(THREADS == TM * (KS / 8), "a group of A per thread");
    __shared__ uint32_t s_tmem;
    __shared__ __align__(8) uint64_t s_bar;
    __shared__ int s_k[KS], s_ta[TM], s_tb[N];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const uint32_t bar = smem_addr(&s_bar);
    if (t < KS) s_k[t] = 0;
    if (t < TM) s_ta[t] = EMPTY;
    if (t < N) s_tb[t] = EMPTY;
    if (t == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const int ra = t & (TM - 1), ga = t / TM;          // row and 8-k group of A
    // columns 16 to a half warp, so that one maximum per half warp is one k's
    const int hw = t / 16, gb = hw / (N / 16), cb = hw % (N / 16) * 16 + (t & 15);
    const bool in_a = ra < m, in_b = gb < KS / 8 && cb < n;
    double x[8], y[8];
    auto inner = [&](int k) { return EVEN_A ? -inner_exponent(s_k[k]) : inner_exponent(s_k[k]); };
    auto load_a = [&]() {
#pragma unroll
        for (int u = 0; u < 8; u++) x[u] = 0.0;
        if (in_a) fa(ra, ga * 8, x);
    };
    auto load_b = [&]() {
#pragma unroll
        for (int u = 0; u < 8; u++) y[u] = 0.0;
        if (in_b) fb(cb, gb * 8, y);
    };
    auto top_a = [&]() {
        int top = EMPTY;
#pragma unroll
        for (int u = 0; u < 8; u++) top = max(top, scaled_exponent(x[u], inner(ga * 8 + u)));
        if (in_a) atomicMax(&s_ta[ra], top);
    };
    auto top_b = [&]() {
        int top = EMPTY;
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (in_b) top = max(top, scaled_exponent(y[u], -inner(gb * 8 + u)));
        if (in_b) atomicMax(&s_tb[cb], top);
    };
    // one copy of the code cuts both operands
    auto cut = [&](int first, int last) {
#pragma unroll 1
        for (int i = first; i <= last; i++) {
            if (i ? in_b : in_a) {
                const int g = i ? gb : ga, top = i ? s_tb[cb] : s_ta[ra];
                uint64_t w[8];
#pragma unroll
                for (int u = 0; u < 8; u++) w[u] = fixed_point(i ? y[u] : x[u], i ? -inner(g * 8 + u) : inner(g * 8 + u), top);
                put_digits(smem + (i ? (KS / 8) * LA + g * LB + cb * 16 : g * LA + ra * 16), i ? N * 16 : TM * 16, w);
            }
        }
    };
    if constexpr (EVEN_A) {
        load_a();
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int r = __reduce_max_sync(0xffffffffu, finite_high(x[u]));
            if (lane == 0) atomicMax(&s_k[ga * 8 + u], r);
        }
        __syncthreads();
        top_a();
        __syncthreads();
        cut(0, 0);
        b_ready();
        load_b();
        top_b();
        __syncthreads();
        cut(1, 1);
    } else {
        b_ready();
        load_a();
        load_b();
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int r = __reduce_max_sync(0xffffu << (lane & 16), finite_high(y[u]));
            if ((t & 15) == 0 && gb < KS / 8) atomicMax(&s_k[gb * 8 + u], r);
        }
        __syncthreads();
        top_a();
        top_b();
        __syncthreads();
        cut(0, 1);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (warp == 0) tmem_alloc(&s_tmem);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    if (t == 0) {
        const uint32_t sa = smem_addr(smem), sb = sa + (KS / 8) * LA;
        for (int h = 0; h < KS / 16; h++) mma_step<N>(tmem, sa + h * 2 * LA, sb + h * 2 * LB, LA, LB, h > 0 ? 1u : 0u);
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
    }
    __syncwarp();
    bool ok = wait(bar, 0);
    if (!ok) ok = wait(bar, 0);
    ok = !__syncthreads_or(!ok);
    if (ok) {
        const int row = (warp & 3) * 32 + lane;
        round_columns<N>(tmem + ((uint32_t)((warp & 3) * 32) << 16), (warp >> 2) * (N / 4), N / 4, row < m, s_ta[row],
                         [&](int c) { return s_tb[c]; }, reinterpret_cast<double *>(smem) + row * (N + 1));
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) tmem_free(tmem);
    return ok;
}

}  // namespace split
