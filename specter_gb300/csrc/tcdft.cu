// FP64 column transforms as exact integer-digit products on the tensor cores.
//
// FP64 arithmetic runs at 1/70 of the FP32 rate on this chip (503 GFMA/s), the tensor cores at
// 1970 TFLOP/s in bf16.  A transform of length n = 2m splits by parity of the frequency (inputs
// x[k] +- x[k+m]) and folds k <-> m-k, which leaves four real matrix products of about n/4 x n/4 per
// column: cosines and sines of the even and of the odd frequencies, the same for real and imaginary
// parts.  Inputs become 62-bit integers against their column's largest value, folded exactly, and
// split into seven signed 9-bit digits (|d| <= 256, exact in bf16); the matrices are held as seven
// digits too.  Products of digit i of the data and digit j of the matrix, i + j <= 6, accumulate in
// FP32 in tensor memory, one accumulator per level i + j (levels 5 and 6 share one).  The sums of levels
// 0 to 2 are integers below 2^24 for any data (checked for every matrix when its table is built), so they are
// exact whatever the order; those of levels 3 and 4 are, but for data whose digits are in step with the
// matrix's at lengths above about 400, and such sums are found by their size and made again in integers
// (mend_outputs).  What is rounded or dropped beyond is below 2^-58 of the column's largest value an input.  The
// levels are put together as a 64-bit integer and rounded once to FP64.  (Products of floating-point matrices by
// splitting into parts whose products are exact: Ozaki, Ogita, Oishi and Rump, 2012.)
//
// Error against long double, relative L2 (n = 58 .. 538): 5e-17 .. 1.7e-16, a double-precision FFT
// 1.4e-16 .. 5e-16.
#include <cmath>
#include <complex>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include <cuda_bf16.h>

#include "chain.h"
#include "fast.h"
#include "ops.h"
#include "smem.h"
#include "tcdft.h"
#include "tcranges.h"
#include "tctables.h"

namespace sg {

#define SG_TRY(x)                  \
    do {                           \
        int _st = (x);             \
        if (_st != OK) return _st; \
    } while (0)

namespace {

constexpr int kLev = 6;             // accumulators (levels 0..4, 5 + 6)
constexpr int kLanes = 128;         // rows of an MMA: 64 columns, real and imaginary parts
constexpr int kAStage = kDig * kLanes * 16 * 2;  // bytes of one 16-deep step of data digits
constexpr int kDigThreads = 256;
// Outputs as integers in units of 2^-kSh of the level-0 unit: results are below (n + 2) * sqrt(2) * 2^14
// level-0 units (each input is below 2^14 of them, twice that in a half spectrum), 2^62.7 at n = 550.
constexpr int kSh = 39;
constexpr int kNaN = 0x40000000;    // exponent of a column that holds a non-finite value

// what a launch transforms: complex columns; real rows to half spectra; half spectra to real rows
enum { kCol = 0, kR2C = 1, kC2R = 2 };

}  // namespace

struct TcSet {
    unsigned char *mat = nullptr;
    int expo = 0;
    double post = 1.0;
    float top[2] = {0.f, 0.f};
};

struct TcState {
    std::map<std::pair<int, double>, TcSet> sets;  // by length (negative: half spectrum to real) and factor
    unsigned char *ws = nullptr;  // digits
    size_t ws_bytes = 0;
    int ws_jobs = 0;              // of launches of that many transforms
    int *expo = nullptr;          // column exponents of the digits in ws (behind them)
    size_t expo_count = 0;
    double *phys = nullptr;       // physical rows in tiles, of one range of tiles of the x passes
    size_t phys_count = 0, phys_asked = 0;
    std::vector<void *> kept;     // tables; and smaller buffers from before, which captured graphs may hold
    size_t kept_bytes = 0;
    unsigned char *slab = nullptr;  // what is left of the tables' latest block (in kept)
    size_t slab_left = 0;
    size_t tiles(int n) const { return std::min(ws_bytes / ((size_t)dims(n).ks.all() * kAStage), expo_count / kLanes); }
};

namespace {

// ------------------------------------------------------------------ device helpers
__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Waits for the phase, at most about two seconds; false when it gave up or the block is aborting.
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, volatile int *abort_flag) {
    if (mbar_try(bar, parity)) return true;
    const long long t0 = clock64();
    for (;;) {
        for (int i = 0; i < 64; i++)
            if (mbar_try(bar, parity)) return true;
        if (*abort_flag) return false;
        if (clock64() - t0 > 4000000000ll) {
            *abort_flag = 1;
            return false;
        }
    }
}
__device__ __forceinline__ void bulk_load(unsigned dst, const void *src, unsigned bytes, unsigned bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
// shared-memory operand descriptor, K-major without swizzle: 8-row x 16-byte core matrices, lbo
// bytes apart along K and sbo bytes apart along the rows
__device__ __forceinline__ unsigned long long smem_desc(unsigned addr, unsigned lbo, unsigned sbo) {
    return (unsigned long long)((addr & 0x3FFFF) >> 4) | ((unsigned long long)(lbo >> 4) << 16) |
           ((unsigned long long)(sbo >> 4) << 32) | (1ull << 46);
}
// Issued by the lane with lead != 0 of a converged warp: operands that are the same in all lanes stay in
// uniform registers (39 clocks an instruction at most, against 60 from a branch that one lane takes).
__device__ __forceinline__ void mma_bf16(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc,
                                         unsigned acc, unsigned lead) {
    asm volatile(
        "{\n.reg .pred p, e;\nsetp.ne.u32 p, %4, 0;\nsetp.ne.u32 e, %5, 0;\n"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(lead)
        : "memory");
}
__device__ __forceinline__ void mma_commit(unsigned bar, unsigned lead) {
    asm volatile(
        "{\n.reg .pred e;\nsetp.ne.u32 e, %1, 0;\n"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(bar),
        "r"(lead)
        : "memory");
}
__device__ __forceinline__ unsigned elect_one() {
    unsigned r;
    asm volatile("{\n.reg .pred e;\nelect.sync _|e, 0xffffffff;\nselp.u32 %0, 1, 0, e;\n}\n" : "=r"(r));
    return r;
}
// four columns of every level, asynchronously; the values are there after tmem_wait
__device__ __forceinline__ void tmem_ld4(unsigned (&r)[4], unsigned addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
// waits for this thread's loads; the operands keep their uses behind it
__device__ __forceinline__ void tmem_wait(unsigned (&r)[kLev][4]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0][0]), "+r"(r[0][1]), "+r"(r[0][2]), "+r"(r[0][3]), "+r"(r[1][0]), "+r"(r[1][1]), "+r"(r[1][2]),
                   "+r"(r[1][3]), "+r"(r[2][0]), "+r"(r[2][1]), "+r"(r[2][2]), "+r"(r[2][3]), "+r"(r[3][0]), "+r"(r[3][1]),
                   "+r"(r[3][2]), "+r"(r[3][3]), "+r"(r[4][0]), "+r"(r[4][1]), "+r"(r[4][2]), "+r"(r[4][3]), "+r"(r[5][0]),
                   "+r"(r[5][1]), "+r"(r[5][2]), "+r"(r[5][3])::"memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ size_t col_offset(const TcShape &s, unsigned c) {
    const unsigned q = c / s.w;
    return (size_t)q * s.s + (c - q * s.w);
}

// Epilogue warps per quarter of the lanes: the more there are, the better they hide one another's latencies,
// until the registers of a thread (80 with five) no longer hold its sine products.  z transform of 512^2 x 538
// and half spectra to rows of 512 x 512 x 538, ms, with three, four, five, six, seven:
// 1.15 1.13 1.10 1.13 1.13 and 1.03 1.13 0.97 1.03 1.00.
constexpr int kEpiQ = 5;
constexpr int kEpiThreads = 128 * kEpiQ, kLoadWarp = kEpiThreads / 32, kMmaWarp = kLoadWarp + 1;
constexpr int kGemmBlock = kEpiThreads + 64;
constexpr int kGemmSmem = 221 * 1024;  // dynamic shared memory: what the static arrays leave of 227 KB
constexpr int kGroups = (kMaxNc / 4 + kEpiQ - 1) / kEpiQ;  // groups of 4 outputs per epilogue warp

// Outputs of a thread that its epilogue has left for mend_outputs, by parity: bit 16 * (sine list) + 4 * (group of
// the warp) + (output of the group).
__shared__ unsigned s_marks[2][kEpiThreads];

// The levels of four outputs as integers, sum over v of l[v] * 2^kSh.  A level times 2^9v (level 5 times
// 2^kSh, rounded) is an integer that an addition of 1.5 * 2^23 leaves in the low mantissa bits while it
// is below 2^22, as sums of signed digits nearly always are; level 0 goes up to 2^24 and hands what is
// below its multiples of 4 down to level 1.  False where a level was too large.  (Conversion instructions
// would run at 16 a clock: six a value are 3800 clocks a list of 80 outputs, as long as a product of n = 256.)
__device__ __forceinline__ bool join_levels(const unsigned (&l)[kLev][4], long long (&u)[4]) {
    constexpr unsigned kB4 = 0x4C400000u, kB = 0x4B400000u;  // 1.5 * 2^25, 1.5 * 2^23
    constexpr unsigned long long kOff = ((unsigned long long)kB4 << (kSh + 2)) + ((unsigned long long)kB << (kSh - 9)) +
                                        ((unsigned long long)kB << (kSh - 18)) + ((unsigned long long)kB << (kSh - 27)) +
                                        ((unsigned long long)kB << (kSh - 36)) + kB;
    unsigned bad = 0;
#pragma unroll
    for (int t = 0; t < 4; t++) {
        auto f = [&](int v) { return __uint_as_float(l[v][t]); };
        const float m4 = __uint_as_float(kB4), m = __uint_as_float(kB);
        const float r0 = f(0) + m4, rem = f(0) - (r0 - m4);
        const unsigned b0 = __float_as_uint(r0), b1 = __float_as_uint(fmaf(f(1) + rem, 512.f, m)),
                       b2 = __float_as_uint(fmaf(f(2), 262144.f, m)), b3 = __float_as_uint(fmaf(f(3), 134217728.f, m)),
                       b4 = __float_as_uint(fmaf(f(4), 68719476736.f, m)),
                       b5 = __float_as_uint(fmaf(f(5), (float)(1ull << kSh), m));
        bad |= (b1 ^ kB) | (b2 ^ kB) | (b3 ^ kB) | (b4 ^ kB) | (b5 ^ kB);
        unsigned long long y = (unsigned long long)b3 * (1u << (kSh - 27)) - kOff;
        y = (unsigned long long)b4 * (1u << (kSh - 36)) + y;
        y = (unsigned long long)b2 * (1u << (kSh - 18)) + y;
        y = (unsigned long long)b1 * (1u << (kSh - 9)) + y;
        y += b5;
        u[t] = (long long)(y + ((unsigned long long)(b0 << (kSh + 2 - 32)) << 32));
    }
    return (bad & 0xFF800000u) == 0;
}

// The same for levels of any size, read again from tensor memory.  An output whose level 3 or 4 may have passed 2^24
// in FP32 (at or above TcJob::top: digits in step with the matrix's; random data is far below) leaves these two
// out and is marked, from bit `at` on: mend_outputs adds them.
struct Four {
    long long u[4];
};
template <bool MARK>
__device__ __noinline__ Four join_levels_wide(unsigned tm, int nc, float top3, float top4, int par, int at) {
    unsigned l[kLev][4];
#pragma unroll
    for (int v = 0; v < kLev; v++) tmem_ld4(l[v], tm + v * nc);
    tmem_wait(l);
    Four r;
#pragma unroll
    for (int t = 0; t < 4; t++) {
        auto level = [&](int v, float w) { return (long long)__float2int_rn(__uint_as_float(l[v][t]) * w); };
        if (MARK && (fabsf(__uint_as_float(l[3][t])) * 134217728.f >= top3 || fabsf(__uint_as_float(l[4][t])) * 68719476736.f >= top4)) {
            s_marks[par][threadIdx.x] |= 1u << (at + t);
            l[3][t] = l[4][t] = 0;
        }
        r.u[t] = (level(0, 1.f) << kSh) + (level(1, 512.f) << (kSh - 9)) + (level(2, 262144.f) << (kSh - 18)) +
                 (level(3, 134217728.f) << (kSh - 27)) + (level(4, 68719476736.f) << (kSh - 36)) +
                 level(5, (float)(1ull << kSh));
    }
    return r;
}

// t * 2^q as a double, rounded to nearest, for |t| < 2^63 and a result whose exponent is a normal
// number's.  The leading bit goes to bit 62, the rounding addend cannot overflow, and the implicit bit
// carries into the exponent field, as does rounding up to the next power of two.
__device__ __forceinline__ double scaled_double(long long t, int q) {
    const long long sg = t >> 63;
    const unsigned long long u = (unsigned long long)((t ^ sg) - sg);
    const unsigned uh = (unsigned)(u >> 32), ul = (unsigned)u;
    const int lz = __clz((int)(uh ? uh : ul)) + (uh ? 0 : 32);
    const unsigned long long mant = ((u << (lz - 1)) + 0x200) >> 10;
    const unsigned hi = (unsigned)(mant >> 32) + ((unsigned)(1085 + q - lz) << 20);
    // zero has a zero mantissa: its exponent goes as well
    return __hiloint2double((int)(lz == 64 ? 0u : hi | ((unsigned)(sg >> 32) & 0x80000000u)), (int)(unsigned)mant);
}

// ------------------------------------------------------------------ digits
struct DigArgs {
    TcShape s;
    TcJob job[kTcMaxJobs];
    const double *dir;      // FC-Gram matrix (s.next rows, column-major) and its matching points
    int oz;
    int m, K;
    Steps ks;
    unsigned tile0, ntile;  // tiles [tile0, tile0 + ntile) of every job
    unsigned char *ws;
    int *expo;              // [job][ntile][128 lanes]
};

// Columns are split into digits of the four folded lists.  Bound by memory traffic (8 bytes read and 14
// written a value, 5.3 TB/s) and beside it by the ALU pipe (84 % active in columns), hence no shift where a digit
// can become a float as it stands (3 % of the kernels' time).
//
// A value (times k for the derivative) as an integer in units of 2^-60 of 2^(emax - 1022).
template <bool DERIV>
__device__ __forceinline__ long long fixed_point(double x, int k, int emax) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const unsigned hi = (unsigned)(b >> 32);
    int e = (hi >> 20) & 0x7ff;
    unsigned long long M = b & 0xfffffffffffffull;
    if (e) M |= 1ull << 52;
    else e = 1;
    bool neg = (int)hi < 0;
    int sh;
    if (DERIV) {
        if (k < 0) { k = -k; neg = !neg; }
        M *= (unsigned)k;
        sh = emax - e - 7;
        if (sh < 0) { M <<= -sh; sh = 0; }
    } else {
        M <<= 7;
        sh = emax - e;
    }
    M = sh < 64 ? M >> sh : 0;
    return neg ? -(long long)M : (long long)M;
}

__device__ __forceinline__ void put_digits(unsigned char *dst, const long long (&v)[8]) {
    unsigned long long w[8];
    unsigned long long bias = 0;
#pragma unroll
    for (int i = 0; i < kDig; i++) bias += 256ull << (54 - 9 * i);
#pragma unroll
    for (int t = 0; t < 8; t++) w[t] = (unsigned long long)v[t] + bias;
#pragma unroll
    for (int i = 0; i < kDig; i++) {
        unsigned r[4];
        // bit of digit i in a word whose bits 0..22 hold it whole: of the upper word (moved down for digit 0),
        // of bits 18..49, of the lower word
        constexpr int kAt[kDig] = {0, 13, 4, 9, 0, 9, 0};
        const int at = kAt[i];
#pragma unroll
        for (int t = 0; t < 8; t += 2) {
            float f[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                // (2^23 + u * 2^at) * 2^(-9i - at) through the exponent field, minus the same of the bias:
                // d * 2^-9i exactly, with the digit left where it stands
                const unsigned lo = (unsigned)w[t + h], hi = (unsigned)(w[t + h] >> 32);
                const unsigned u = i == 0 ? hi >> 22 : (i <= 2 ? hi : i <= 4 ? __funnelshift_r(lo, hi, 18) : lo) & (511u << at);
                const float off = (float)((1 << (23 - at)) + 256) / (float)(1ull << (9 * i));
                f[h] = __uint_as_float(0x4B000000u - ((unsigned)(9 * i + at) << 23) | u) - off;
            }
            const __nv_bfloat162 p = __floats2bfloat162_rn(f[0], f[1]);
            r[t / 2] = *reinterpret_cast<const unsigned *>(&p);
        }
        *reinterpret_cast<uint4 *>(dst + (size_t)i * kLanes * 32) = make_uint4(r[0], r[1], r[2], r[3]);
    }
}

// the exponent field e of a bound: |x| (times k) < 2^(e - 1022); 0 for zero
template <bool DERIV>
__device__ __forceinline__ int value_exponent(double v, int k) {
    const unsigned hi = (unsigned)__double2hiint(v) & 0x7fffffffu;
    int e = hi >> 20;
    if (e == 0x7ff) return kNaN;
    if (!hi && !__double2loint(v)) return 0;
    const unsigned top = ((hi & 0xfffffu) | (e ? 0x100000u : 0u)) + 1u;
    e = max(e, 1);
    if (DERIV) e = k ? max(e + 31 - __clz((int)(top * (unsigned)abs(k))) - 20, 1) : 0;
    return e;
}

// Digits of LW lanes staged in shared memory (x[row * LW + l]), so that the largest value and the
// digits cost one read of the field.  A thread owns one lane and eight consecutive k of the lists, so
// that it writes whole 16-byte rows of core matrices.  REAL: lanes are real rows; else lanes are the
// real and imaginary parts of columns.
template <bool DERIV, bool REAL, int LW>
__device__ __forceinline__ void digits_body(const DigArgs &a, int job, double *tile_s, int *s_e, unsigned lt,
                                            int lane0) {
    const int n = a.s.n, m = a.m;
    const int l = threadIdx.x % LW, part = REAL ? 0 : l & 1, lane = lane0 + l;
    double *xd = tile_s + l;
    long long *x = (long long *)xd;
    int emax = 0;
    // rows as wavenumbers: r for r < m, r - n above
    for (int row = threadIdx.x / LW; row < n; row += kDigThreads / LW)
        emax = max(emax, value_exponent<DERIV>(xd[row * LW], row < m ? row : row - n));
    atomicMax(&s_e[REAL ? l : l & ~1], emax);
    __syncthreads();
    emax = s_e[REAL ? l : l & ~1];
    if (emax == 0) emax = 1023;  // a column of zeros: any exponent
    if (blockIdx.y == 0 && threadIdx.x < LW) a.expo[((size_t)job * a.ntile + lt) * kLanes + lane] = emax;
    if (emax >= kNaN) emax = 0x7ff;  // a non-finite column's digits are not used
    // to integers in place, each value once (both parities of the frequency read it)
    for (int row = threadIdx.x / LW; row < n; row += kDigThreads / LW)
        x[row * LW] = fixed_point<DERIV>(xd[row * LW], row < m ? row : row - n, emax);
    __syncthreads();
    unsigned char *tb = a.ws + ((size_t)job * a.ntile + lt) * a.ks.all() * kAStage;
    // effective part: multiplying by i moves real data to imaginary lanes and imaginary data, negated,
    // to real lanes; so does the sine list of a complex transform
    const int epart = DERIV ? part ^ 1 : part;
    const int row0 = DERIV ? lane ^ 1 : lane, row1 = REAL ? lane : row0 ^ 1;
    const bool flip = DERIV && part == 1;
    for (int g = blockIdx.y * (kDigThreads / LW) + threadIdx.x / LW; g < 2 * a.ks.first; g += gridDim.y * (kDigThreads / LW)) {
        unsigned char *d = tb + (size_t)(g >> 1) * kAStage + (size_t)(g & 1) * kLanes * 16;
        const bool rest = g < 2 * a.ks.rest;  // else the first list alone goes on
#pragma unroll 1
        for (int par = 0; par < (rest ? 2 : 1); par++) {  // even frequencies: x[k] + x[k+m]; odd: x[k] - x[k+m]
            long long c[8], w[8];
#pragma unroll
            for (int t = 0; t < 8; t++) {
                const int k = 8 * g + t;
                c[t] = w[t] = 0;
                if (k >= a.K) continue;
                const bool self = k == 0 || 2 * k == m;
                const long long x0 = x[k * LW], x1 = x[(k + m) * LW];
                const long long x2 = self ? 0 : x[(m - k) * LW], x3 = self ? 0 : x[(n - k) * LW];
                long long E = par ? x0 - x1 : x0 + x1, E2 = par ? x2 - x3 : x2 + x3;
                if (flip) { E = -E; E2 = -E2; }
                // even: cos gets E + E', sin E - E'; odd: cos O - O', sin O + O'
                if (par) E2 = -E2;
                c[t] = E + E2;
                w[t] = E - E2;
                if (self) w[t] = 0;
                if (par && 2 * k == m) c[t] = 0;
                if (epart == 1) w[t] = -w[t];
            }
            // the last of the odd sine list (k = m/2) takes the place of k = 0, which has no sine
            if (par && g == 0 && m % 2 == 0) {
                const long long O = x[m / 2 * LW] - x[(m / 2 + m) * LW];
                w[0] = flip != (epart == 1) ? -O : O;
            }
            put_digits(d + (size_t)a.ks.before(2 * par) * kAStage + row0 * 16, c);
            if (rest) put_digits(d + (size_t)a.ks.before(2 * par + 1) * kAStage + row1 * 16, w);
        }
    }
}

// Columns: LW = 16 keeps three blocks on an SM at n = 538 (69 KB), LW = 32 at up to half of that.
template <int LW>
__global__ void __launch_bounds__(kDigThreads, 4) k_digits(DigArgs a) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ int s_e[LW];
    const TcShape &s = a.s;
    const int job = blockIdx.z;
    const TcJob &J = a.job[job];
    constexpr int kParts = kLanes / LW, kCols = LW / 2;
    const unsigned lt = blockIdx.x / kParts;
    const int lane0 = (blockIdx.x % kParts) * LW;
    const int n0 = s.n - s.next;  // rows below n0 come from the field, the others from the continuation
    if (threadIdx.x < LW) s_e[threadIdx.x] = 0;
    chain_wait();
    {
        const int cc = threadIdx.x % kCols;
        const unsigned c = (a.tile0 + lt) * 64 + lane0 / 2 + cc;
        const bool live = c < s.ncol;
        const double2 *in = J.in + (live ? col_offset(s, c) : 0);
        double2 *dst = (double2 *)smem + cc;
        for (int row = threadIdx.x / kCols; row < n0; row += kDigThreads / kCols) {
            if (live) cp_async<16>(dst + row * kCols, in + (size_t)row * s.rs);
            else dst[row * kCols] = make_double2(0.0, 0.0);
        }
        async_commit();
        async_wait();
    }
    __syncthreads();
    if (s.next) {  // FC-Gram continuation (src/fftp/fftp.fpp:755-773), FP64, beside other blocks' integer work
        const int C = s.next, d = a.oz, l = threadIdx.x % LW;
        double *x = (double *)smem + l;
        for (int i = threadIdx.x / LW; i < C; i += kDigThreads / LW) {
            double v = __ldg(a.dir + i) * x[(n0 - d) * LW] + __ldg(a.dir + (C - 1 - i)) * x[(d - 1) * LW];
            for (int j = 1; j < d; j++)
                v = v + __ldg(a.dir + i + C * j) * x[(n0 - d + j) * LW] + __ldg(a.dir + (C - 1 - i) + C * j) * x[(d - 1 - j) * LW];
            x[(n0 + i) * LW] = v;
        }
        __syncthreads();
    }
    if (J.deriv) digits_body<true, false, LW>(a, job, (double *)smem, s_e, lt, lane0);
    else digits_body<false, false, LW>(a, job, (double *)smem, s_e, lt, lane0);
}

// Real rows.  PROD: the rows are sums of products of physical rows in tiles [k][128 lanes] (the
// nonlinear term: sum over i of phys[i] * phys[J.prod + i], times scale); else they come from a
// field's rows.
template <int LW, bool PROD>
__global__ void __launch_bounds__(kDigThreads, 4) k_digits_real(DigArgs a, const double *phys, size_t fstride, double scale) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ int s_e[LW];
    const TcShape &s = a.s;
    const int job = blockIdx.z;
    const TcJob &J = a.job[job];
    constexpr int kParts = kLanes / LW;
    const unsigned lt = blockIdx.x / kParts;
    const int lane0 = (blockIdx.x % kParts) * LW;
    if (threadIdx.x < LW) s_e[threadIdx.x] = 0;
    chain_wait();
    double *dst = (double *)smem;
    if (PROD) {
        const int l = threadIdx.x % LW;
        const double *u = phys + (size_t)lt * s.n * kLanes + lane0 + l, *d = u + J.prod * fstride;
#pragma unroll 2
        for (int k = threadIdx.x / LW; k < s.n; k += kDigThreads / LW) {
            const size_t o = (size_t)k * kLanes;
            const double u0 = u[o], u1 = u[o + fstride], u2 = u[o + 2 * fstride];
            const double d0 = d[o], d1 = d[o + fstride], d2 = d[o + 2 * fstride];
            dst[k * LW + l] = (u0 * d0 + u1 * d1 + u2 * d2) * scale;
        }
    } else {
        // neighbouring threads read neighbouring rows (whose lines the next k find in L1), so that the writes
        // to shared memory stay off one bank
        const int l = threadIdx.x % LW;
        const unsigned row = (a.tile0 + lt) * kLanes + lane0 + l;
        const bool live = row < s.ncol;
        const double *in = (const double *)J.in + (live ? (size_t)row * s.n : 0);
#pragma unroll 4
        for (int k = threadIdx.x / LW; k < s.n; k += kDigThreads / LW) dst[k * LW + l] = live ? in[k] : 0.0;
    }
    __syncthreads();
    digits_body<false, true, LW>(a, job, dst, s_e, lt, lane0);
}

// Half spectra (rows of n/2 + 1 complex values, row stride s.rs): the lists are the real and imaginary
// parts of the even and of the odd frequencies, doubled but for frequencies 0 and n/2, whose imaginary
// parts do not count.
template <bool DERIV, int LW>
__device__ __forceinline__ void half_digits(const DigArgs &a, int job, const double2 *tile_s, int *s_e, unsigned lt,
                                            int lane0) {
    const int m = a.m, l = threadIdx.x % LW, lane = lane0 + l;
    const double2 *x = tile_s + l;
    int emax = 0;
    for (int f = threadIdx.x / LW; f <= m; f += kDigThreads / LW) {
        const double2 v = x[f * (LW + 1)];
        emax = max(emax, max(value_exponent<DERIV>(v.x, f), value_exponent<DERIV>(v.y, f)));
    }
    atomicMax(&s_e[l], emax);
    __syncthreads();
    emax = s_e[l];
    if (emax == 0) emax = 1023;
    if (blockIdx.y == 0 && threadIdx.x < LW) a.expo[((size_t)job * a.ntile + lt) * kLanes + lane] = emax;
    if (emax >= kNaN) emax = 0x7ff;
    unsigned char *tb = a.ws + ((size_t)job * a.ntile + lt) * a.ks.all() * kAStage + lane * 16;
    for (int g = blockIdx.y * (kDigThreads / LW) + threadIdx.x / LW; g < 2 * a.ks.first; g += gridDim.y * (kDigThreads / LW)) {
        unsigned char *d = tb + (size_t)(g >> 1) * kAStage + (size_t)(g & 1) * kLanes * 16;
        const bool rest = g < 2 * a.ks.rest;  // else the first list alone goes on
#pragma unroll 1
        for (int par = 0; par < (rest ? 2 : 1); par++) {
            long long c[8], w[8];
#pragma unroll
            for (int t = 0; t < 8; t++) {
                const int f = 2 * (8 * g + t) + par;
                c[t] = w[t] = 0;
                if (f > m) continue;
                const double2 v = x[f * (LW + 1)];
                const bool end = f == 0 || f == m;
                // frequency n/2 is the wavenumber -n/2; i k (re, im) = (-k im, k re)
                const int k = f == m ? -m : f;
                long long re = fixed_point<DERIV>(DERIV ? v.y : v.x, DERIV ? -k : k, emax);
                long long im = fixed_point<DERIV>(DERIV ? v.x : v.y, k, emax);
                c[t] = end ? re : 2 * re;
                w[t] = end ? 0 : 2 * im;
            }
            put_digits(d + (size_t)a.ks.before(2 * par) * kAStage, c);
            if (rest) put_digits(d + (size_t)a.ks.before(2 * par + 1) * kAStage, w);
        }
    }
}

template <int LW>
__global__ void __launch_bounds__(kDigThreads, 3) k_digits_half(DigArgs a) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ int s_e[LW];
    const TcShape &s = a.s;
    const int job = blockIdx.z, H = a.m + 1;
    const TcJob &J = a.job[job];
    constexpr int kParts = kLanes / LW;
    const unsigned lt = blockIdx.x / kParts;
    const int lane0 = (blockIdx.x % kParts) * LW;
    const unsigned r0 = (a.tile0 + lt) * kLanes + lane0;
    if (threadIdx.x < LW) s_e[threadIdx.x] = 0;
    chain_wait();
    double2 *dst = (double2 *)smem;  // [frequency][LW + 1]: the odd stride keeps the row writes off one bank
    for (int i = threadIdx.x; i < H * LW; i += kDigThreads) {
        const int l = i / H, f = i - l * H;
        if (r0 + l < s.ncol) cp_async<16>(dst + f * (LW + 1) + l, J.in + (size_t)(r0 + l) * s.rs + f);
        else dst[f * (LW + 1) + l] = make_double2(0.0, 0.0);
    }
    async_commit();
    async_wait();
    __syncthreads();
    if (J.deriv) half_digits<true, LW>(a, job, dst, s_e, lt, lane0);
    else half_digits<false, LW>(a, job, dst, s_e, lt, lane0);
}

// ------------------------------------------------------------------ products
struct GemmArgs {
    TcShape s;
    TcJob job[kTcMaxJobs];
    int m, nq[2], nchunk, nc, nstage;  // m = n / 2
    Steps ks;
    unsigned tile0, ntile, units;
    const unsigned char *ws;
    const int *expo;
    int *err;
};

// A unit of work: one tile of 64 columns, one parity of the frequency, one chunk of nc outputs.  The
// data digits are the M = 128 rows (64 columns x real, imaginary), the matrix digits the N = nc columns
// of the MMAs; a pipeline of bulk copies feeds 28 MMAs a 16-deep step.  One block per SM walks over
// units: the cosine product moves from tensor memory to shared memory as integers, the sine product to
// registers, and while the next unit's MMAs run, their sum and difference (the frequencies f and n - f)
// become doubles.  Half spectra to real rows (kC2R): a unit holds both parities; with A the even and B
// the odd frequencies' sum, x[k] = A + B and x[k + n/2] = A - B, and the integers A wait in the output
// until the same thread has B.  The MMAs (operand reads from shared memory: (128 + nc) * 32 bytes each) and the
// integer work of the epilogue bound it.
struct Unit {
    int job, par, chunk, cols;  // cols: outputs of the chunk that exist
    unsigned lt;
};
template <int MODE>
__device__ __forceinline__ Unit unit_of(const GemmArgs &a, unsigned u) {
    Unit w;
    w.par = 0;
    if (MODE != kC2R) {
        w.par = u % 2;
        u /= 2;
    }
    w.chunk = u % a.nchunk;
    w.cols = min(a.nc, a.nq[MODE == kC2R ? 0 : w.par] - w.chunk * a.nc);
    u /= a.nchunk;
    w.lt = u % a.ntile;
    w.job = u / a.ntile;
    return w;
}

// Adds levels 3 and 4 to the outputs of this thread that join_levels_wide has left without them: summed in integers
// from the digits, which are exact whatever their size.  Beside the epilogue, whose registers it would cost 4 % of
// every launch from within.
template <int MODE>
__device__ __noinline__ void mend_outputs(const GemmArgs &a, unsigned u, double *out) {
    const Unit w = unit_of<MODE>(a, u);
    const TcJob &J = a.job[w.job];
    const TcShape &s = a.s;
    const int lane = threadIdx.x & 127, g0 = threadIdx.x >> 7, nc = a.nc;
    const int e = a.expo[((size_t)w.job * a.ntile + w.lt) * kLanes + lane], q = e - 1022 - 14 - kSh + J.expo;
    unsigned long long marks = s_marks[0][threadIdx.x] | (unsigned long long)s_marks[1][threadIdx.x] << 32;
    s_marks[0][threadIdx.x] = s_marks[1][threadIdx.x] = 0;
    if (e >= kNaN) return;
    for (; marks; marks &= marks - 1) {
        const int bit = __ffsll(marks) - 1, par = bit >> 5, sine = bit >> 4 & 1, list = 2 * par + sine;
        const int col = (g0 + kEpiQ * (bit >> 2 & 3)) * 4 + (bit & 3), j = w.chunk * nc + col;
        if (col >= w.cols) continue;
        const unsigned char *data = a.ws + (((size_t)w.job * a.ntile + w.lt) * a.ks.all() + a.ks.before(list)) * kAStage + lane * 16;
        const unsigned char *mat = J.mat + (size_t)(a.ks.before(list) * a.nchunk + w.chunk * a.ks.of(list)) * (kDig * 32 * nc) + col * 16;
        long long e3 = 0, e4 = 0;
        for (int k = 0; k < 16 * a.ks.of(list); k++) {
            const unsigned step = k / 16, half = k / 8 % 2;  // eight values side by side, two such groups a step
            const unsigned char *pd = data + (size_t)step * kAStage + half * kLanes * 16 + k % 8 * 2;
            const unsigned char *pm = mat + (size_t)step * (kDig * 32 * nc) + half * nc * 16 + k % 8 * 2;
            auto digit = [](const unsigned char *p, int i) {  // bf16 in units of 2^-9i
                const float v = __uint_as_float((unsigned)*(const unsigned short *)p << 16);
                return __float2int_rn(v * __uint_as_float((unsigned)(127 + 9 * i) << 23));
            };
            int x[5], y[5];
#pragma unroll
            for (int i = 0; i < 5; i++) {
                x[i] = digit(pd + i * (kLanes * 32), i);
                y[i] = digit(pm + i * (nc * 32), i);
            }
            e3 += x[0] * y[3] + x[1] * y[2] + x[2] * y[1] + x[3] * y[0];
            e4 += x[0] * y[4] + x[1] * y[3] + x[2] * y[2] + x[3] * y[1] + x[4] * y[0];
        }
        long long t = (e3 << (kSh - 27)) + (e4 << (kSh - 36));
        if (sine && (MODE == kR2C || (MODE == kCol && s.sign < 0))) t = -t;
        const double v = scalbn((double)t, q) * J.post;
        if (MODE == kCol) {
            const int f = 2 * j + par, f2 = s.n - f;
            if (f < s.nrows) out[2 * (size_t)f * s.rs] += v;
            if (f && f != f2 && f2 < s.nrows) out[2 * (size_t)f2 * s.rs] += sine ? -v : v;
        } else if (MODE == kR2C) {
            const int f = 2 * j + par;
            if (f <= a.m) out[2 * f + sine] += v;
        } else {
            const bool two = j && 2 * j != a.m;
            // x[k] = A + B and x[k + n/2] = A - B
            const size_t h = (size_t)a.m * s.rs;
            const double d0 = sine ? -v : v, d1 = par ? -v : v;  // of A[j] or B[j], and of A or B[n/2 - j]
            double *o0 = out + (size_t)j * s.rs, *o1 = out + (size_t)(a.m - j) * s.rs;
            o0[0] += d0;
            o0[h] += par ? -d0 : d0;
            if (two) {
                o1[0] += d1;
                o1[h] += par ? -d1 : d1;
            }
        }
    }
}

// ADD: jobs may have a field to add (each value's branch costs 5 to 12 %, so launches without one do without).
// NACC: sets of accumulators in tensor memory, used by the lists in turn.  With two, a list's MMAs run while
// the sums of the one before are read; lengths below 128 leave room for it (2 * kLev * 32 columns), and their
// lists are as short as that read: half spectra to rows of 96 x 96 x 122, 91 -> 80 us, of 64 x 64 x 90, 45 -> 40 us.
// (As a run-time choice it costs longer lengths 5 to 14 %.)
// MARK: some job has sums that FP32 may not hold (TcJob::top), so outputs may be left to mend_outputs.  At lengths
// below about 300 hardly any has, and their launches do without the registers for it (with marks in every kernel a
// step at 256^2 x 257 took 25.3 instead of 24.7 ms).
template <int MODE, bool ADD, int NACC, bool MARK>
__global__ void __launch_bounds__(kGemmBlock, 1) k_gemm(const __grid_constant__ GemmArgs a) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ unsigned long long bars[2 * 8 + 4];
    __shared__ unsigned s_tmem;
    __shared__ int s_abort;
    const TcShape &s = a.s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nc = a.nc;
    const unsigned b_bytes = kDig * nc * 32, stage_bytes = kAStage + b_bytes;
    const unsigned full = smem_u32(bars), empty = full + 8 * 8, accfull = full + 16 * 8, accempty = accfull + 16;
    unsigned tcols = 32;
    while (tcols < (unsigned)(NACC * kLev * nc)) tcols *= 2;
    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int i = 0; i < a.nstage; i++) {
            mbar_init(full + 8 * i, 1);
            mbar_init(empty + 8 * i, 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(accfull + 8 * i, 1);
            mbar_init(accempty + 8 * i, kEpiThreads);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(tcols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    fence_before();
    __syncthreads();
    fence_after();
    chain_wait();
    const unsigned tmem = s_tmem;
    volatile int *ab = &s_abort;
    constexpr int kLists = MODE == kC2R ? 4 : 2;  // of a unit: cosine list, sine list (of each parity)
    if (warp == kLoadWarp) {
        if (lane == 0) {
            int it = 0, st = 0, ph = 1;  // steps issued so far, their stage and the phase its buffer is free after
            bool ok = true;
            for (unsigned u = blockIdx.x; u < a.units && ok; u += gridDim.x) {
                const Unit w = unit_of<MODE>(a, u);
                int list = 2 * w.par, left = a.ks.of(list);
                const unsigned char *A = a.ws + (((size_t)w.job * a.ntile + w.lt) * a.ks.all() + a.ks.before(list)) * kAStage;
                auto matrix = [&] {
                    return a.job[w.job].mat + (size_t)(a.ks.before(list) * a.nchunk + w.chunk * a.ks.of(list)) * b_bytes;
                };
                const unsigned char *B = matrix();
                const int nit = a.ks.before(list + kLists) - a.ks.before(list);
                for (int i = 0; i < nit; i++, it++) {
                    if (it >= a.nstage && !mbar_wait(empty + 8 * st, ph, ab)) { ok = false; break; }
                    const unsigned dst = smem_u32(smem) + st * stage_bytes;
                    mbar_expect(full + 8 * st, stage_bytes);
                    bulk_load(dst, A + (size_t)i * kAStage, kAStage, full + 8 * st);
                    bulk_load(dst + kAStage, B, b_bytes, full + 8 * st);
                    B += b_bytes;
                    if (--left == 0) {  // the next list's matrix of the same chunk
                        left = a.ks.of(++list);
                        B = matrix();
                    }
                    if (++st == a.nstage) { st = 0; ph ^= 1; }
                }
            }
            if (!ok)  // giving up: this block's own copies land before it ends
                for (int i = max(0, it - a.nstage); i < it; i++) {
                    const long long t0 = clock64();
                    while (!mbar_try(full + 8 * (i % a.nstage), (i / a.nstage) & 1) && clock64() - t0 < 2000000000ll) {}
                }
        }
    } else if (warp == kMmaWarp) {
        // D FP32, A and B bf16, both K-major, N = nc, M = 128
        const unsigned idesc0 = (1u << 4) | (1u << 7) | (1u << 10) | (8u << 24);
        // sine lists of forward transforms with A negated (bit 13)
        const unsigned neg = MODE == kR2C || (MODE == kCol && s.sign < 0) ? 1u << 13 : 0u;
        const unsigned lead = elect_one();
        int st = 0, ph = 0, lists = 0;
        bool ok = true;
        for (unsigned u = blockIdx.x; u < a.units && ok; u += gridDim.x) {
            const Unit w = unit_of<MODE>(a, u);
            const unsigned idesc = idesc0 | ((unsigned)((w.cols + 15) / 16 * 2) << 17);  // N / 8
            for (int list = 0; list < kLists && ok; list++, lists++) {
                const int ks = a.ks.of(2 * w.par + list);
                const unsigned id = idesc | (lists & 1 ? neg : 0u);
                const int set = lists % NACC;
                if (lists >= NACC) {  // the set's previous sums have left tensor memory
                    ok = __all_sync(~0u, mbar_wait(accempty + 8 * set, ((lists / NACC) - 1) & 1, ab));
                    if (!ok) break;
                    fence_after();
                }
                const unsigned tm = tmem + set * kLev * nc;
                for (int i = 0; i < ks; i++) {
                    ok = __all_sync(~0u, mbar_wait(full + 8 * st, ph, ab));
                    if (!ok) break;
                    fence_after();
                    const unsigned sa = smem_u32(smem) + st * stage_bytes;
                    const unsigned long long da = smem_desc(sa, kLanes * 16, 128), db = smem_desc(sa + kAStage, nc * 16, 128);
                    const unsigned keep = i != 0;
                    // neighbours in this order add to different accumulators; address fields count 16 bytes
#pragma unroll
                    for (int d = 0; d < kDig; d++)
#pragma unroll
                        for (int j = 0; j < kDig - d; j++) {
                            const int acc = d + j < kLev ? d + j : kLev - 1;
                            mma_bf16(tm + acc * nc, da + d * (kLanes * 2), db + j * (nc * 2), id,
                                     d == 0 && j < kLev ? keep : 1u, lead);
                        }
                    mma_commit(empty + 8 * st, lead);
                    if (i == ks - 1) mma_commit(accfull + 8 * set, lead);
                    if (++st == a.nstage) { st = 0; ph ^= 1; }
                }
            }
        }
    } else {
        // a warp holds a quarter of the lanes and every kEpiQ-th group of 4 outputs
        const int quad = warp & 3, g0 = warp >> 2;
        const int r = quad * 32 + lane;
        const unsigned taddr = tmem + ((unsigned)(quad * 32) << 16);
        // [nc][128], and at least 4 kEpiQ outputs: every warp's first group has a place.  (Tensor memory has it
        // too: 5 nc + 4 kEpiQ columns are fewer than 6 nc, or than the 128 of nc = 16.)
        long long *Ps = (long long *)(smem + a.nstage * stage_bytes) + r;
        // the levels of 4 outputs, and those as integers
        unsigned tset = taddr;  // of the list's set of accumulators
        auto fetch = [&](int gi, unsigned (&l)[kLev][4]) {
            const unsigned at = tset + (g0 + kEpiQ * gi) * 4;
#pragma unroll
            for (int v = 0; v < kLev; v++) tmem_ld4(l[v], at + v * nc);
        };
        auto gather = [&](const TcJob &J, int par, int sine, int gi, const unsigned (&l)[kLev][4], long long (&u)[4]) {
            if (__any_sync(~0u, !join_levels(l, u))) {
                const unsigned at = tset + (g0 + kEpiQ * gi) * 4;
                const Four w = MARK ? join_levels_wide<true>(at, nc, J.top[0], J.top[1], par, 16 * sine + 4 * gi)
                                    : join_levels_wide<false>(at, nc, 0.f, 0.f, 0, 0);
#pragma unroll
                for (int t = 0; t < 4; t++) u[t] = w.u[t];
            }
        };
        if (MARK) s_marks[0][threadIdx.x] = s_marks[1][threadIdx.x] = 0;
        int lists = 0;
        auto take = [&] {  // the next list's sums are there
            const int set = lists % NACC;
            tset = taddr + set * kLev * nc;
            if (!__all_sync(~0u, mbar_wait(accfull + 8 * set, (lists / NACC) & 1, ab))) return false;
            fence_after();
            return true;
        };
        auto give = [&] {  // and have been read
            fence_before();
            mbar_arrive(accempty + 8 * (lists % NACC));
            lists++;
        };
        bool ok = true;
        for (unsigned u = blockIdx.x; u < a.units && ok; u += gridDim.x) {
            const Unit w = unit_of<MODE>(a, u);
            const TcJob &J = a.job[w.job];
            // this warp's groups (at least one: what it reads beyond the outputs is not stored)
            const int ngr = max(1, ((w.cols + 3) / 4 - g0 + kEpiQ - 1) / kEpiQ);
            bool live;
            size_t off;  // of this lane's column or row in the output
            if (MODE == kCol) {
                const unsigned c = (a.tile0 + w.lt) * 64 + (r >> 1);
                live = c < s.ncol;
                off = live ? 2 * col_offset(s, c) + (r & 1) : 0;
            } else {
                live = (a.tile0 + w.lt) * kLanes + r < s.ncol;
                off = (size_t)w.lt * s.ts + (size_t)r * s.ls;
            }
            const int e = a.expo[((size_t)w.job * a.ntile + w.lt) * kLanes + r];
            // results are t * 2^q: with an exponent 1086 + q - lz, 0 <= lz < 64, that could leave the normal
            // numbers' a further power of two, times the job's own factor; NaN for a non-finite column
            const int q = e - 1022 - 14 - kSh + J.expo, qc = max(-1000, min(q, 900));
            const double fac = e >= kNaN ? __longlong_as_double(0x7ff8000000000000ll) : scalbn(J.post, q - qc);
            const bool more = __any_sync(~0u, !(fac == 1.0));
            double *out = (double *)J.out + off;
            auto value = [&](long long t) { return scaled_double(t, qc); };
            const double *add = ADD && J.add ? (const double *)J.add + off : nullptr;  // may be the output itself
            auto plus = [&](double v, double b) {
                // behind a branch: a multiplication of every value would bind the loop to the FP64 pipe
                if (more) asm volatile("mul.rn.f64 %0, %0, %1;" : "+d"(v) : "d"(fac));
                return v + b;
            };
            for (int par = w.par; par < (MODE == kC2R ? 2 : w.par + 1); par++) {
                __syncwarp();  // lanes without a column skip the output below
                ok = take();
                if (!ok) break;
                unsigned l[kLev][4];
#pragma unroll
                for (int gi = 0; gi < kGroups; gi++)
                    if (gi < ngr) {
                        fetch(gi, l);
                        tmem_wait(l);
                        long long P[4];
                        gather(J, par, 0, gi, l, P);
#pragma unroll
                        for (int t = 0; t < 4; t++) Ps[((g0 + kEpiQ * gi) * 4 + t) * kLanes] = P[t];
                    }
                give();
                ok = take();
                if (!ok) break;
                long long Q[kGroups][4];
#pragma unroll
                for (int gi = 0; gi < kGroups; gi++)
                    if (gi < ngr) {
                        fetch(gi, l);
                        tmem_wait(l);
                        gather(J, par, 1, gi, l, Q[gi]);
                    }
                give();
                if (!live) continue;
                // a group's loads, conversions and stores one after another: loads do not move across stores
#pragma unroll
                for (int gi = 0; gi < kGroups; gi++)
                    if (gi < ngr) {
                        const int col = (g0 + kEpiQ * gi) * 4, j0 = w.chunk * nc + col;
                        const int left = a.nq[MODE == kC2R ? 0 : par] - j0;  // outputs of this group that exist
                        long long p[4];
#pragma unroll
                        for (int t = 0; t < 4; t++) p[t] = Ps[(col + t) * kLanes];
                        if (MODE == kCol) {
                            // fields hold fewer than 2^32 elements: 32-bit row offsets
                            double v[4], v2[4];
                            const int f0 = 2 * j0 + par;
                            unsigned o = (unsigned)f0 * s.rs, o2 = (unsigned)(s.n - f0) * s.rs;
#pragma unroll
                            for (int t = 0; t < 4; t++) {
                                v[t] = value(p[t] + Q[gi][t]);
                                v2[t] = value(p[t] - Q[gi][t]);
                            }
#pragma unroll
                            for (int t = 0; t < 4; t++, o += 2 * s.rs, o2 -= 2 * s.rs) {
                                const int f = f0 + 2 * t, f2 = s.n - f;
                                if (t < left && f < s.nrows) {
                                    if (ADD && add) v[t] = plus(v[t], add[2 * (size_t)o]);
                                    out[2 * (size_t)o] = v[t];
                                }
                                if (t < left && f && f != f2 && f2 < s.nrows) {
                                    if (ADD && add) v2[t] = plus(v2[t], add[2 * (size_t)o2]);
                                    out[2 * (size_t)o2] = v2[t];
                                }
                            }
                        } else if (MODE == kR2C) {
                            double2 v[4];
#pragma unroll
                            for (int t = 0; t < 4; t++) v[t] = make_double2(value(p[t]), value(Q[gi][t]));
#pragma unroll
                            for (int t = 0; t < 4; t++) {
                                const int f = 2 * (j0 + t) + par;
                                if (t < left && f <= a.m) *(double2 *)(out + 2 * f) = v[t];
                            }
                        } else {
                            // even: A[k] = p - d, A[n/2 - k] = p + d; odd: B[k] = p - d, B[n/2 - k] = -p - d
                            double *o0 = out + (size_t)j0 * s.rs, *o1 = out + (size_t)(a.m - j0) * s.rs;
                            const size_t h = (size_t)a.m * s.rs;
                            if (par == 0) {
#pragma unroll
                                for (int t = 0; t < 4; t++) {
                                    const int j = j0 + t;
                                    const long long d = Q[gi][t];
                                    if (t < left) *(long long *)(o0 + (size_t)t * s.rs) = p[t] - d;
                                    if (t < left && j && 2 * j != a.m) *(long long *)(o1 - (size_t)t * s.rs) = p[t] + d;
                                }
                            } else {
                                long long A[4], A1[4];
#pragma unroll
                                for (int t = 0; t < 4; t++) {
                                    const int j = j0 + t;
                                    A[t] = t < left ? *(const long long *)(o0 + (size_t)t * s.rs) : 0;
                                    A1[t] = t < left && j && 2 * j != a.m ? *(const long long *)(o1 - (size_t)t * s.rs) : 0;
                                }
#pragma unroll
                                for (int t = 0; t < 4; t++) {
                                    const int j = j0 + t;
                                    const long long d = Q[gi][t], B = p[t] - d, B1 = -p[t] - d;
                                    const double v0 = value(A[t] + B), v1 = value(A[t] - B);
                                    const double v2 = value(A1[t] + B1), v3 = value(A1[t] - B1);
                                    double *q0 = o0 + (size_t)t * s.rs, *q1 = o1 - (size_t)t * s.rs;
                                    if (t < left) {
                                        q0[0] = v0;
                                        q0[h] = v1;
                                    }
                                    if (t < left && j && 2 * j != a.m) {
                                        q1[0] = v2;
                                        q1[h] = v3;
                                    }
                                }
                            }
                        }
                    }
                if (more && !(ADD && add) && (MODE != kC2R || par == 1)) {
                    // a factor that is no power of two, results beyond the normal numbers, non-finite columns: in a
                    // pass of its own over this thread's outputs (a branch at each value costs every launch 5 to 12 %)
                    auto finish = [&](size_t o) { out[o] *= fac; };
                    for (int gi = 0; gi < ngr; gi++)
#pragma unroll
                        for (int t = 0; t < 4; t++) {
                            const int j = w.chunk * nc + (g0 + kEpiQ * gi) * 4 + t, f = 2 * j + par, f2 = s.n - f;
                            if (j >= a.nq[MODE == kC2R ? 0 : par]) break;
                            if (MODE == kCol) {
                                if (f < s.nrows) finish(2 * ((size_t)f * s.rs));
                                if (f && f != f2 && f2 < s.nrows) finish(2 * ((size_t)f2 * s.rs));
                            } else if (MODE == kR2C) {
                                if (f <= a.m) {
                                    finish(2 * f);
                                    finish(2 * f + 1);
                                }
                            } else {
                                finish((size_t)j * s.rs);
                                finish((size_t)(a.m + j) * s.rs);
                                if (j && 2 * j != a.m) {
                                    finish((size_t)(a.m - j) * s.rs);
                                    finish((size_t)(2 * a.m - j) * s.rs);
                                }
                            }
                        }
                }
            }
            if (MARK && (s_marks[0][threadIdx.x] | s_marks[1][threadIdx.x])) {
                if (live) mend_outputs<MODE>(a, u, out);
                else s_marks[0][threadIdx.x] = s_marks[1][threadIdx.x] = 0;  // of what lies beyond the outputs
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_abort) {
        *(volatile int *)a.err = 1;
        __threadfence_system();
    }
    if (warp == kMmaWarp) {
        if (s_abort) {  // issued MMAs end before their tensor memory is given back
            const long long t0 = clock64();
            while (clock64() - t0 < 2000000ll) {}
        }
        __syncwarp();
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tcols));
    }
}

// physical rows from tiles [tile][x][128 rows] to a field [row][x]
__global__ void __launch_bounds__(256) k_untile(const double *tiles, double *out, int n, unsigned rows) {
    __shared__ double t[32][33];
    chain_wait();
    const unsigned r0 = blockIdx.x * 32, x0 = blockIdx.y * 32;
    const double *src = tiles + (size_t)(r0 / kLanes) * n * kLanes + r0 % kLanes;
    for (unsigned i = threadIdx.y; i < 32; i += 8)
        if (x0 + i < (unsigned)n) t[i][threadIdx.x] = src[(size_t)(x0 + i) * kLanes + threadIdx.x];
    __syncthreads();
    for (unsigned i = threadIdx.y; i < 32; i += 8)
        if (r0 + i < rows && x0 + threadIdx.x < (unsigned)n) out[(size_t)(r0 + i) * n + x0 + threadIdx.x] = t[threadIdx.x][i];
}

// ------------------------------------------------------------------ tables
// The first quadrant's cosines and sines of one set (MatrixDigits), as an argument of the kernel: a copy would have to
// wait for the stream or for the host's memory.
struct QuadrantArg {
    long long v[2][kMaxLen / 4 + 1];
};
// -> the matrices of the set
__global__ void k_fill_mat(__nv_bfloat16 *mat, const __grid_constant__ QuadrantArg quad, int n, int K, Steps ks, int nq0, int nq1, int nchunk,
                           int nc, int half) {
    const long long total = (long long)nchunk * ks.all() * 16 * nc;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total; q += (long long)gridDim.x * blockDim.x) {
        const int kk = (int)(q % 16), col = (int)(q / 16 % nc), t = (int)(q / 16 / nc);  // [list][chunk][step][col][kk]
        const int set = t < nchunk * ks.first ? 0 : 1 + (t - nchunk * ks.first) / (nchunk * ks.rest);
        const int r = t - nchunk * ks.before(set), chunk = r / ks.of(set), step = r % ks.of(set);
        const int list = set % 2, par = set / 2;
        int k = 16 * step + kk;
        const int j = chunk * nc + col;
        if (!half && set == 3 && n % 4 == 0) k = k == 0 ? n / 4 : k == n / 4 ? K : k;  // as the digits have it
        // the K side runs over points and the N side over frequencies, the other way about for half spectra
        const int pt = half ? j : k, fq = half ? k : j;
        const bool on = pt < K && fq < (par ? nq1 : nq0);
        const Folded f = fold_angle(n, on ? (int)((long long)(2 * fq + par) * pt % n) : 0);
        const long long v = !on ? 0 : list ? f.ss * quad.v[1][f.t] : f.cs * quad.v[0][f.t];
        __nv_bfloat16 *dst = mat + (long long)t * (kDig * 16 * nc) + (kk / 8) * (nc * 8) + col * 8 + kk % 8;
#pragma unroll
        for (int i = 0; i < kDig; i++)
            dst[(long long)i * nc * 16] = __float2bfloat16((float)matrix_digit(v, i) * __uint_as_float((unsigned)(127 - 9 * i) << 23));
    }
}

TcState *state(Plan &P) {
    if (!P.tc) P.tc = new TcState();
    return P.tc;
}

}  // namespace

static bool capturing(const Plan &P) {
    cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(P.stream, &c) != cudaSuccess || c != cudaStreamCaptureStatusNone;
}

bool tc_length_ok(int n) { return n >= 32 && n <= kMaxLen && n % 2 == 0; }

void tc_job_set(TcJob &j, const TcSet *s) {
    j.mat = s->mat;
    j.expo = s->expo;
    j.post = s->post;
    j.top[0] = s->top[0];
    j.top[1] = s->top[1];
}

// Device memory of tables, cut from blocks: an allocation takes as long as a short transform.
static unsigned char *table_memory(TcState *S, size_t bytes) {
    bytes = (bytes + 255) / 256 * 256;
    if (S->slab_left < bytes) {
        const size_t block = std::max<size_t>(bytes, 256 * 1024);
        void *m = nullptr;
        if (cudaMalloc(&m, block) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        S->kept.push_back(m);
        S->kept_bytes += block;
        S->slab = (unsigned char *)m;
        S->slab_left = block;
    }
    unsigned char *p = S->slab;
    S->slab += bytes;
    S->slab_left -= bytes;
    return p;
}

const TcSet *tc_set(Plan &P, int n, double factor, int *status, bool half) {
    *status = OK;
    TcState *S = state(P);
    const std::pair<int, double> key(half ? -n : n, factor);
    auto it = S->sets.find(key);
    if (it != S->sets.end()) return &it->second;
    *status = kNoFast;  // without memory for the tables, or where none may be allocated
    if (capturing(P)) return nullptr;
    *status = OK;
    const Dims D = dims(n);
    TcSet set;
    MatrixDigits M;
    if (!matrix_digits_for(D, factor, half, M)) { set_error("digit tables: exactness bound"); *status = ERR_SHAPE; return nullptr; }
    set.expo = M.expo;
    set.post = M.post;
    set.top[0] = M.top[0];
    set.top[1] = M.top[1];
    QuadrantArg h;
    std::copy(M.c.begin(), M.c.end(), h.v[0]);
    std::copy(M.s.begin(), M.s.end(), h.v[1]);
    set.mat = table_memory(S, (size_t)D.nchunk * D.ks.all() * kDig * 32 * D.nc);
    if (!set.mat) {
        *status = kNoFast;
        return nullptr;
    }
    k_fill_mat<<<2 * kSMs, 256, 0, P.stream>>>((__nv_bfloat16 *)set.mat, h, n, D.K, D.ks, D.nq[0], D.nq[1], D.nchunk, D.nc,
                                            half ? 1 : 0);
    if ((*status = check_launch("digit tables"))) return nullptr;
    return &(S->sets[key] = set);
}

// Room for digits, sized for what the plan's calls use: plans that run single transforms (conversions, output) hold the
// digits of one, those that run the nonlinear term those of its launches, both up to a limit beyond which launches
// run in ranges of tiles.  Buffers keep their addresses: one that has become too small stays until the plan's
// end, for graphs that hold it.
// The limit, MiB, against an RK2 step of convection, ms: 512^2 x 513 2048: 235, 1024: 240, 512: 249, 128: 312; 256^2 x 257
// 25.1, 25.7, 27.9, 35.4; 128^2 x 129 (701 MB at most) 4.08, 4.08, 4.09, 4.86.
constexpr size_t kRoomMiB = 2048;
constexpr size_t kSpareMiB = 64;  // beyond this, at most an eighth of the free memory

// bytes and lanes of digits for launches of up to `jobs` transforms (1 or more), in `most` bytes if 16 tiles fit them
static void room_for(const Plan &P, int jobs, size_t most, size_t *bytes, size_t *lanes) {
    const int len[3] = {P.nz, P.ny, P.nx}, many[3] = {8, 8, 15};  // of the z and y passes and of the nonlinear x pass
    const size_t cols[3] = {((size_t)P.ny * P.ldx + 63) / 64, ((size_t)P.nz * P.ldx + 63) / 64,
                            ((size_t)P.nz * P.ny + kLanes - 1) / kLanes};
    *bytes = *lanes = 0;
    for (int i = 0; i < 3; i++) {
        if (!tc_length_ok(len[i])) continue;
        const size_t per = (size_t)dims(len[i]).ks.all() * kAStage;
        const size_t t = std::min(cols[i] * (jobs > 1 ? many[i] : 1), std::max<size_t>(most / per, kTcMaxJobs));
        *bytes = std::max(*bytes, t * per);
        *lanes = std::max(*lanes, t * kLanes);
    }
}

// kNoFast: there is no memory for it, or it would have to be allocated during a capture (the general engine needs
// none)
static int room(Plan &P, int jobs) {
    TcState *S = state(P);
    jobs = jobs > 1 ? kTcMaxJobs : 1;
    if (P.digit_room_mb < 0) return kNoFast;
    if (S->ws_jobs >= jobs) return OK;
    if (capturing(P)) return S->ws ? OK : kNoFast;
    size_t last = 0, most = (size_t)(P.digit_room_mb ? P.digit_room_mb : kRoomMiB) << 20, bytes, lanes;
    room_for(P, jobs, most, &bytes, &lanes);
    if (bytes > kSpareMiB << 20) {  // the fields that a solver allocates after it need the rest
        size_t free = 0, total = 0;
        if (cudaMemGetInfo(&free, &total) == cudaSuccess) most = std::min(most, std::max(free / 8, kSpareMiB << 20));
        else cudaGetLastError();
    }
    for (;; most /= 2) {
        room_for(P, jobs, most, &bytes, &lanes);
        if (bytes == last || (bytes <= S->ws_bytes && lanes <= S->expo_count)) break;  // no smaller, or no gain
        last = bytes;
        void *ws = nullptr;
        if (cudaMalloc(&ws, bytes + lanes * sizeof(int)) == cudaSuccess) {
            if (S->ws) {
                S->kept.push_back(S->ws);
                S->kept_bytes += S->ws_bytes + S->expo_count * sizeof(int);
            }
            S->ws = (unsigned char *)ws;
            S->ws_bytes = bytes;
            S->expo = (int *)(S->ws + bytes);
            S->expo_count = lanes;
            break;
        }
        cudaGetLastError();
    }
    if (!S->ws) return kNoFast;
    S->ws_jobs = jobs;  // as much of it as there is
    return OK;
}

int tc_status(const Plan &P) {
    if (!*(volatile int *)P.gave_up) return OK;
    set_error("a transform kernel gave up a wait");
    return ERR_CUDA;
}

namespace {

// One range of tiles of one set of jobs: arguments of the digit and of the product kernels.
int fill_args(Plan &P, const Dims &D, const TcShape &s, const TcJob *jobs, int nj, unsigned t0, unsigned nt, DigArgs &d,
               GemmArgs &g) {
    TcState *S = P.tc;
    if ((size_t)nj * nt * D.ks.all() * kAStage > S->ws_bytes || (size_t)nj * nt * kLanes > S->expo_count) {
        set_error("digit workspace too small for a launch");
        return ERR_STATE;
    }
    d.s = g.s = s;
    for (int j = 0; j < nj; j++) d.job[j] = g.job[j] = jobs[j];
    d.m = g.m = D.m;
    d.K = D.K;
    d.ks = g.ks = D.ks;
    d.dir = P.geo.dir;
    d.oz = P.oz;
    d.tile0 = g.tile0 = t0;
    d.ntile = g.ntile = nt;
    d.ws = S->ws;
    g.ws = S->ws;
    d.expo = S->expo;
    g.expo = S->expo;
    g.nq[0] = D.nq[0];
    g.nq[1] = D.nq[1];
    g.nchunk = D.nchunk;
    g.nc = D.nc;
    g.err = P.gave_up_dev;
    return OK;
}

// lanes per digit block: three blocks on an SM
int digit_lanes(int n) { return n <= 300 ? 32 : 16; }

// Small launches split a tile's lists over blocks (each reads its columns itself) until there are two
// blocks per SM.
int digit_split(const Dims &D, int lw, size_t blocks) {
    const int rounds = (2 * D.ks.first * lw + kDigThreads - 1) / kDigThreads;
    int split = 1;
    while (split < rounds && blocks * split < 2 * kSMs) split++;
    return split;
}

template <int MODE>
void launch_gemm(Plan &P, const Dims &D, GemmArgs &g, int nj) {
    const unsigned stage = kAStage + kDig * D.nc * 32, psize = (unsigned)std::max(D.nc, 4 * kEpiQ) * kLanes * 8;
    g.nstage = std::min(8, (int)((kGemmSmem - psize) / stage));
    g.units = g.ntile * (MODE == kC2R ? 1 : 2) * D.nchunk * nj;
    const size_t smem = (size_t)g.nstage * stage + psize;
    bool add = false, mark = false;
    for (int j = 0; j < nj; j++) {
        add = add || g.job[j].add;
        mark = mark || !(std::isinf(g.job[j].top[0]) && std::isinf(g.job[j].top[1]));
    }
    const bool two = 2 * kLev * D.nc <= 512;  // lengths below 128, whose sums are always exact
    constexpr bool kAdd = MODE == kCol;
    const auto k = kAdd && add ? (two ? k_gemm<MODE, kAdd, 2, false> : mark ? k_gemm<MODE, kAdd, 1, true> : k_gemm<MODE, kAdd, 1, false>)
                               : (two ? k_gemm<MODE, false, 2, false> : mark ? k_gemm<MODE, false, 1, true> : k_gemm<MODE, false, 1, false>);
    allow_smem(k, smem);
    if (g.units <= kSMs) chain(k, g.units, kGemmBlock, smem, P.stream, g);  // one unit a block
    else k<<<kSMs, kGemmBlock, smem, P.stream>>>(g);
}

template <typename K>
K with_smem(K k, size_t bytes) {
    allow_smem(k, bytes);
    return k;
}

}  // namespace

int tc_run(Plan &P, const TcShape &s, const TcJob *jobs, int njobs, const char *name, double bytes) {
    SG_TRY(room(P, njobs));
    SG_TRY(tc_status(P));
    const Dims D = dims(s.n);
    const size_t per = (size_t)D.ks.all() * kAStage;
    const unsigned tiles = (s.ncol + 63) / 64;
    const TcRange range = tc_range(njobs, tiles, P.tc->tiles(s.n));
    const int lw = digit_lanes(s.n);
    const size_t dsm = (size_t)s.n * lw * 8;
    for (int j0 = 0; j0 < njobs; j0 += range.jobs)
        for (unsigned t0 = 0; t0 < tiles; t0 += range.tiles) {
            const int nj = std::min(range.jobs, njobs - j0);
            const unsigned nt = std::min(range.tiles, tiles - t0);
            DigArgs d{};
            GemmArgs g{};
            SG_TRY(fill_args(P, D, s, jobs + j0, nj, t0, nt, d, g));
            const size_t blocks = (size_t)nt * (kLanes / lw);
            const dim3 grid((unsigned)blocks, digit_split(D, lw, blocks * nj), nj);
            const double share = (double)nt * nj / ((double)tiles * njobs);
            {
                Launch L(P, "digits", share * bytes * 0.5 + (double)nt * nj * per);
                chain(with_smem(lw == 32 ? k_digits<32> : k_digits<16>, dsm), grid, kDigThreads, dsm, P.stream, d);
            }
            {
                Launch L(P, name, share * bytes);
                launch_gemm<kCol>(P, D, g, nj);
            }
        }
    return check_launch(name);
}

// Buffer of physical rows in tiles ([field][tile][x][128 rows]) for one range of tiles: one field's, or the 15 of the
// nonlinear term's x pass.
static int phys_rows(Plan &P, int fields) {
    TcState *S = P.tc;
    const size_t cap = S->tiles(P.nx), all = ((size_t)P.nz * P.ny + kLanes - 1) / kLanes;
    const size_t t = std::min(all, std::max<size_t>(fields > 1 ? cap / kTcMaxJobs : cap, 1));
    const size_t one = (size_t)fields * P.nx * kLanes, want = t * one;
    if (want <= S->phys_asked || capturing(P)) return S->phys_count >= one ? OK : kNoFast;
    S->phys_asked = want;
    double *m = nullptr;
    size_t n = want;
    while (n > S->phys_count && n >= one && cudaMalloc(&m, n * sizeof(double)) != cudaSuccess) {
        cudaGetLastError();
        m = nullptr;
        n = n / 2 / one * one;
    }
    if (m) {
        if (S->phys) {
            S->kept.push_back(S->phys);
            S->kept_bytes += S->phys_count * sizeof(double);
        }
        S->phys = m;
        S->phys_count = n;
    }
    return S->phys_count >= one ? OK : kNoFast;
}

// gradre / advect between the y passes (pseudospec_hd.f90:209-319, pseudospec_phd.f90:23-113): the
// velocity and the derivatives of components [c0, c1) to physical rows, the products, and back, in
// ranges of tiles whose physical rows ([field][tile][x][128 rows]) stay in a buffer of the plan.
int tc_x_nonlinear(Plan &P, const XNLArgs &x, double bytes) {
    if (!tc_length_ok(P.nx)) return kNoFast;
    const void *const *u = x.u, *const *dy = x.dy, *const *dz = x.dz;
    void *const *out = x.out;
    const int c0 = x.c0, c1 = x.c1, nrows = x.nrows;
    const double scale = x.tmp;
    const int n = P.nx, nc = c1 - c0, nin = 3 + 3 * nc;
    SG_TRY(room(P, nin));
    SG_TRY(phys_rows(P, 15));
    SG_TRY(tc_status(P));
    TcState *S = P.tc;
    int st = OK;
    const TcSet *inv = tc_set(P, n, 1.0, &st, true), *dinv = inv ? tc_set(P, n, P.Dkx, &st, true) : nullptr;
    const TcSet *fwd = dinv ? tc_set(P, n, 1.0, &st, false) : nullptr;
    if (!fwd) return st;
    const Dims D = dims(n);
    const size_t per = (size_t)D.ks.all() * kAStage, ptile = (size_t)n * kLanes;
    const unsigned rows = (unsigned)nrows * P.ny, tiles = (rows + kLanes - 1) / kLanes;
    const size_t fit = std::min(S->tiles(n) / kTcMaxJobs, S->phys_count / (15 * ptile));
    if (!fit) return kNoFast;
    const unsigned tstep = tc_range(1, tiles, fit).tiles;
    const size_t fstride = tstep * ptile;
    const int lw = digit_lanes(n);
    for (unsigned t0 = 0; t0 < tiles; t0 += tstep) {
        const unsigned nt = std::min(tstep, tiles - t0);
        const double share = (double)nt / tiles * bytes;
        const size_t blocks = (size_t)nt * (kLanes / lw);
        TcJob jobs[kTcMaxJobs];
        // physical fields: u, v, w, then d/dx, d/dy, d/dz of each component
        for (int j = 0; j < nin; j++) {
            const int c = c0 + (j - 3) / 3, dir = (j - 3) % 3;
            TcJob &J = jobs[j];
            J = TcJob{};
            J.in = (const double2 *)(j < 3 ? u[j] : dir == 0 ? u[c] : dir == 1 ? dy[c] : dz[c]);
            J.out = (double2 *)(S->phys + j * fstride);
            J.deriv = j >= 3 && dir == 0;
            tc_job_set(J, J.deriv ? dinv : inv);
        }
        TcShape s{};
        s.n = n;
        s.ncol = rows;
        s.rs = P.ldx;
        DigArgs d{};
        GemmArgs g{};
        SG_TRY(fill_args(P, D, s, jobs, nin, t0, nt, d, g));
        {
            const size_t sm = (size_t)(D.m + 1) * (lw + 1) * sizeof(double2);
            Launch L(P, "digits", share * nin / (nin + nc) + (double)nt * nin * per);
            chain(with_smem(lw == 32 ? k_digits_half<32> : k_digits_half<16>, sm),
                  dim3((unsigned)blocks, digit_split(D, lw, blocks * nin), nin), kDigThreads, sm, P.stream, d);
        }
        g.s.rs = kLanes;
        g.s.ls = 1;
        g.s.ts = ptile;
        {
            Launch L(P, "x_inverse", (double)nt * nin * (per + ptile * 8.0));
            launch_gemm<kC2R>(P, D, g, nin);
        }
        for (int c = 0; c < nc; c++) {
            TcJob &J = jobs[c];
            J = TcJob{};
            J.out = (double2 *)out[c0 + c] + (size_t)t0 * kLanes * P.ldx;
            J.prod = 3 + 3 * c;
            tc_job_set(J, fwd);
        }
        s.ls = 2 * P.ldx;
        s.ts = (size_t)kLanes * s.ls;
        DigArgs d2{};
        GemmArgs g2{};
        SG_TRY(fill_args(P, D, s, jobs, nc, t0, nt, d2, g2));
        {
            const size_t sm = (size_t)n * lw * sizeof(double);
            Launch L(P, "products", (double)nt * (nin * ptile * 8.0 + nc * per));
            chain(with_smem(lw == 32 ? k_digits_real<32, true> : k_digits_real<16, true>, sm),
                  dim3((unsigned)blocks, digit_split(D, lw, blocks * nc), nc), kDigThreads, sm, P.stream, d2, S->phys, fstride,
                  scale);
        }
        {
            Launch L(P, "x_forward", share * nc / (nin + nc) + (double)nt * nc * per);
            launch_gemm<kR2C>(P, D, g2, nc);
        }
    }
    return check_launch("x_nonlinear");
}

// FP64 passes over the digit-product transforms (tcdft.cu).  They serve every even length of 32 to
// 550: nearly everywhere they are faster than the FP64 Stockham engine, which the FP64 pipe bounds (z passes
// 1.0 to 8 times, on grids of 4 x 2 to 64 x 32 columns; y passes at lengths 32 and 36 with a few columns 0.9 times).
// kNoFast: a form that they do not take (another length, a scale on part of the rows).
static int tc_add(Plan &P, TcJob *jobs, int *nj, int n, double factor, const void *in, void *out, const void *add,
                  int deriv) {
    int st = OK;
    const TcSet *set = tc_set(P, n, factor, &st);
    if (!set) return st;
    TcJob &j = jobs[(*nj)++];
    j = TcJob{};
    j.in = (const double2 *)in;
    j.out = (double2 *)out;
    j.add = (const double2 *)add;
    j.deriv = deriv;
    tc_job_set(j, set);
    return OK;
}

static TcShape tc_z_shape(const Plan &P, int sign, int nrows) {
    TcShape s{};
    s.n = P.nz;
    s.sign = sign;
    s.nrows = nrows;
    s.ncol = s.w = s.s = s.rs = (unsigned)P.ny * P.ldx;
    return s;
}

int tc_z_inverse(Plan &P, const ZInvArgs &a, int nf, double bytes) {
    if (!tc_length_ok(P.nz) || (a.scale_rows > 0 && a.scale_rows < a.nrows)) return kNoFast;
    const double sc = a.scale_rows > 0 ? a.scale : 1.0;
    TcJob jobs[kTcMaxJobs];
    int nj = 0;
    // derivatives first: out0 may alias in
    for (int f = 0; f < nf; f++)
        if (a.out1[f]) SG_TRY(tc_add(P, jobs, &nj, P.nz, P.Dkz * sc, a.in[f], a.out1[f], nullptr, 1));
    for (int f = 0; f < nf; f++)
        if (a.out0[f]) SG_TRY(tc_add(P, jobs, &nj, P.nz, sc, a.in[f], a.out0[f], a.add[f], 0));
    return tc_run(P, tc_z_shape(P, +1, a.nrows), jobs, nj, "z_inverse", bytes);
}

int tc_z_forward(Plan &P, const ZFwdArgs &a, int nf, double bytes) {
    if (!tc_length_ok(P.nz) || a.in_scale != 1.0) return kNoFast;
    TcJob jobs[kTcMaxJobs];
    int nj = 0;
    for (int f = 0; f < nf; f++) SG_TRY(tc_add(P, jobs, &nj, P.nz, 1.0, a.in[f], a.out[f], nullptr, 0));
    TcShape s = tc_z_shape(P, -1, P.nz);
    s.next = P.cz;
    return tc_run(P, s, jobs, nj, "z_forward", bytes);
}

// Rows of fields: real rows to half spectra (r2c) and back.  Back they go through tiles whose writes are
// coalesced (written row by row, 256^2 x 282 took 439 us instead of 251 and 61 for the copy).  A few short
// rows stay with the Stockham engine, one launch instead of two or three (whole transforms to physical
// space, Stockham against digits, us: 32 x 32 x 58 33 and 38, 64 x 64 x 90 60 and 51, 32 x 128 x 154 107 and 78,
// 64 x 192 x 282 338 and 195).  Longer rows are digit products whatever their number, for half the error: up to 2432
// rows, one wave of the Stockham kernel's blocks, that costs up to a third of a c2r pass and a tenth of an r2c pass at
// lengths of 96 to 256 (rows of 128, 1080 of them, to physical space 34.5 and 45.1 us, from it 34.9 and 38.3; 3000
// and more 1.03 and 1.15 times faster).
constexpr unsigned kFewRows = 16 * kLanes;
int tc_x(Plan &P, const XArgs &a, int nf, bool r2c, double bytes) {
    if (!tc_length_ok(P.nx) || (P.nx < 96 && (unsigned)a.nrows * P.ny < kFewRows)) return kNoFast;
    SG_TRY(room(P, 1));
    if (!r2c) SG_TRY(phys_rows(P, 1));
    SG_TRY(tc_status(P));
    TcState *S = P.tc;
    int st = OK;
    const TcSet *set = tc_set(P, P.nx, a.scale, &st, !r2c);
    if (!set) return st;
    const Dims D = dims(P.nx);
    const size_t per = (size_t)D.ks.all() * kAStage, cap = S->tiles(P.nx);
    const unsigned rows = (unsigned)a.nrows * P.ny, tiles = (rows + kLanes - 1) / kLanes;
    const unsigned tstep = tc_range(1, tiles, r2c ? cap : std::min(cap, S->phys_count / ((size_t)P.nx * kLanes))).tiles;
    const int lw = digit_lanes(P.nx);
    const char *name = r2c ? "x_r2c" : "x_c2r";
    for (int f = 0; f < nf; f++)
        for (unsigned t0 = 0; t0 < tiles; t0 += tstep) {
            const unsigned nt = std::min(tstep, tiles - t0);
            TcShape s{};
            s.n = P.nx;
            s.ncol = rows;
            s.rs = r2c ? 1 : P.ldx;
            s.ls = r2c ? 2 * P.ldx : 1;
            s.ts = (size_t)kLanes * (r2c ? s.ls : P.nx);
            TcJob J{};
            J.in = (const double2 *)a.in[f];
            J.out = r2c ? (double2 *)((double *)a.out[f] + t0 * s.ts) : (double2 *)S->phys;
            tc_job_set(J, set);
            DigArgs d{};
            GemmArgs g{};
            SG_TRY(fill_args(P, D, s, &J, 1, t0, nt, d, g));
            const size_t blocks = (size_t)nt * (kLanes / lw);
            const dim3 grid((unsigned)blocks, digit_split(D, lw, blocks), 1);
            const double share = bytes * nt / ((double)tiles * nf);
            {
                Launch L(P, "digits", share * 0.5 + (double)nt * per);
                if (r2c) {
                    const size_t sm = (size_t)P.nx * lw * sizeof(double);
                    chain(with_smem(lw == 32 ? k_digits_real<32, false> : k_digits_real<16, false>, sm), grid, kDigThreads, sm,
                          P.stream, d, nullptr, 0, 1.0);
                } else {
                    const size_t sm = (size_t)(D.m + 1) * (lw + 1) * sizeof(double2);
                    chain(with_smem(lw == 32 ? k_digits_half<32> : k_digits_half<16>, sm), grid, kDigThreads, sm, P.stream, d);
                }
            }
            g.s.rs = r2c ? 1 : kLanes;
            {
                Launch L(P, name, share);
                if (r2c) launch_gemm<kR2C>(P, D, g, 1);
                else launch_gemm<kC2R>(P, D, g, 1);
            }
            if (!r2c) {
                const unsigned left = std::min(rows - t0 * kLanes, nt * kLanes);
                Launch L(P, "untile", 16.0 * left * P.nx);
                chain(k_untile, dim3((left + 31) / 32, (P.nx + 31) / 32), dim3(32, 8), 0, P.stream, S->phys, (double *)a.out[f] + (size_t)t0 * kLanes * P.nx, P.nx, left);
            }
        }
    return check_launch(name);
}

int tc_y(Plan &P, const YArgs &a, int nf, int nplanes, double bytes) {
    if (!tc_length_ok(P.ny)) return kNoFast;
    TcJob jobs[kTcMaxJobs];
    int nj = 0;
    for (int f = 0; f < nf; f++)
        if (a.out1[f]) SG_TRY(tc_add(P, jobs, &nj, P.ny, P.Dky * a.scale, a.in[f], a.out1[f], nullptr, 1));
    for (int f = 0; f < nf; f++)
        if (a.out0[f]) SG_TRY(tc_add(P, jobs, &nj, P.ny, a.scale, a.in[f], a.out0[f], nullptr, 0));
    TcShape s{};
    s.n = P.ny;
    s.sign = a.sign;
    s.nrows = P.ny;
    s.w = s.rs = P.ldx;
    s.s = (unsigned)P.ny * P.ldx;
    s.ncol = (unsigned)nplanes * P.ldx;
    return tc_run(P, s, jobs, nj, a.sign < 0 ? "y_forward" : "y_inverse", bytes);
}

int tc_reserve(Plan &P) {
    SG_TRY(room(P, kTcMaxJobs));
    return tc_length_ok(P.nx) ? phys_rows(P, 15) : OK;
}

void tc_free(Plan &P) {
    if (!P.tc) return;
    for (void *m : P.tc->kept) cudaFree(m);
    if (P.tc->ws) cudaFree(P.tc->ws);
    if (P.tc->phys) cudaFree(P.tc->phys);
    delete P.tc;
    P.tc = nullptr;
}

unsigned long long tc_bytes(const Plan &P) {
    if (!P.tc) return 0;
    unsigned long long b = P.tc->ws_bytes + P.tc->expo_count * sizeof(int);
    b += P.tc->kept_bytes + P.tc->phys_count * sizeof(double);
    return b;
}

}  // namespace sg
