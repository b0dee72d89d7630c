// Lengths, matrix digits and exactness bounds of the digit products (tcdft.cu); host code without CUDA.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <utility>
#include <vector>

#ifdef __CUDACC__
#define SG_BOTH __host__ __device__
#else
#define SG_BOTH
#endif

namespace sg {

constexpr int kDig = 7;       // digits of data and matrix
constexpr int kMaxNc = 80;    // outputs per block: six accumulators of 80 are 480 of 512 tensor-memory columns
constexpr int kMaxLen = 550;  // every even length up to here holds the bounds of matrix_digits_for

// Steps of 16 values in the four lists: `first` for the cosine list of the even frequencies (K = m/2 + 1
// values), `rest` for each of the others, one step less where m is a multiple of 32 (they hold m/2 values;
// 64^3: 5 steps instead of 8, 128^3: 9 of 12, 512^3: 33 of 36).
struct Steps {
    int first, rest;
    SG_BOTH int of(int list) const { return list ? rest : first; }
    SG_BOTH int before(int list) const { return list ? first + (list - 1) * rest : 0; }
    SG_BOTH int all() const { return first + 3 * rest; }
};
struct Dims {
    int n, m, K, nq[2], nchunk, nc;
    Steps ks;
};
inline Dims dims(int n) {
    Dims d;
    d.n = n;
    d.m = n / 2;
    d.K = d.m / 2 + 1;
    d.nq[0] = d.m / 2 + 1;
    d.nq[1] = (d.m + 1) / 2;
    d.ks.first = (d.nq[0] + 15) / 16;
    d.ks.rest = (d.nq[1] + 15) / 16;
    const int np = (d.nq[0] + 15) / 16 * 16;
    d.nchunk = (np + kMaxNc - 1) / kMaxNc;
    d.nc = ((np + d.nchunk - 1) / d.nchunk + 15) / 16 * 16;
    return d;
}

// cos and sin of 2 pi t / n for the first quadrant, t = 0 .. n / 4, in long double
inline void quadrant(int n, std::vector<long double> &c, std::vector<long double> &s) {
    const long double pi = 3.14159265358979323846264338327950288L;
    c.resize(n / 4 + 1);
    s.resize(n / 4 + 1);
    for (int t = 0; t <= n / 4; t++) {
        const bool first = 8 * t <= n;  // octant; the second from the angle's complement
        const long double x = pi * (long double)(first ? 4 * t : n - 4 * t) / (2.0L * (long double)n);
        c[t] = first ? cosl(x) : sinl(x);
        s[t] = first ? sinl(x) : cosl(x);
    }
}

// the angle t of 0 .. n - 1 by one of the first quadrant (n even): cos = cs * cos, sin = ss * sin
struct Folded {
    int t, cs, ss;
};
SG_BOTH inline Folded fold_angle(int n, int t) {
    Folded f = {t, 1, 1};
    if (2 * f.t > n) f = {n - f.t, 1, -1};
    if (4 * f.t > n) f = {n / 2 - f.t, -1, f.ss};
    return f;
}

// digit i of a number in units of 2^-62: signed, in -256 .. 255 but for digit 0
SG_BOTH inline int matrix_digit(long long v, int i) {
    unsigned long long bias = 0;
    for (int k = 1; k < kDig; k++) bias += 256ull << (54 - 9 * k);
    const unsigned long long w = (unsigned long long)v + bias;
    return i ? (int)((w >> (54 - 9 * i)) & 511) - 256 : (int)((long long)w >> 54);
}

// The matrices of one set: cosines and sines times a scale, in units of 2^-62 ...
struct MatrixDigits {
    std::vector<long long> c, s;  // of the first quadrant
    int expo = 0;                 // ... times 2^expo
    double post = 1.0;            // and times this after the products (1: none)
    // A sum of level 3 or 4 whose result is below this is exact in FP32, whatever the order of its terms:
    // had a partial sum passed 2^24, what is left of the bound could not have brought it back below.
    float top[2] = {0.f, 0.f};
    int digit(int n, bool sine, int t, int i) const {
        const Folded f = fold_angle(n, t);
        return matrix_digit(sine ? f.ss * s[f.t] : f.cs * c[f.t], i);
    }
};

// Level v of an output is the sum over the list of the products of digit i of the data and digit v - i of the
// matrix.  The largest absolute sum of the products, over the outputs, that any data digits (|d| <= 256) can make:
// every partial sum in any order is below it.  For levels 2, 3 and 4 (those above are in all of them).
inline void level_bounds(const Dims &D, bool half, const MatrixDigits &m, long long b[3]) {
    struct Sums {
        int v[3];
    };
    std::vector<Sums> a(D.n);
    long long most[3] = {0, 0, 0};
    for (int sine = 0; sine < 2; sine++) {
        for (int t = 0; t < D.n; t++) {
            int sum = 0;
            for (int i = 0; i < 5; i++) {
                sum += std::abs(m.digit(D.n, sine, t, i));
                if (i >= 2) a[t].v[i - 2] = sum;
            }
        }
        for (int par = 0; par < 2; par++) {
            const int no = half ? D.K : D.nq[par], ni = half ? D.nq[par] : D.K;
            for (int o = 0; o < no; o++) {
                // angles (2 f + par) * point: advance by a fixed step from one input to the next
                const int step = half ? 2 * o % D.n : (2 * o + par) % D.n;
                int ang = half ? par * o % D.n : 0, s0 = 0, s1 = 0, s2 = 0;
                for (int i = 0; i < ni; i++) {
                    s0 += a[ang].v[0];
                    s1 += a[ang].v[1];
                    s2 += a[ang].v[2];
                    ang += step;
                    if (ang >= D.n) ang -= D.n;
                }
                most[0] = std::max<long long>(most[0], s0);
                most[1] = std::max<long long>(most[1], s1);
                most[2] = std::max<long long>(most[2], s2);
            }
        }
    }
    for (int v = 0; v < 3; v++) b[v] = 256 * most[v];
}

// factor = scale * 2^expo with scale in (1/2, 1]: the matrices hold cosines and sines times scale.  A smaller scale
// where those digits miss the bounds, and the plain matrices with a multiplication after them where all do.
// Bounds: level 2 (and so 0 and 1) exact for any data; levels 3 and 4 trusted up to 2^22 at least, the size from
// which the epilogue looks at them (join_levels).
inline bool matrix_digits_for(const Dims &D, double factor, bool half, MatrixDigits &m) {
    std::vector<long double> c, s;
    quadrant(D.n, c, s);
    m.c.resize(c.size());
    m.s.resize(s.size());
    int ex = 0;
    double fr = std::frexp(factor, &ex);
    if (fr == 0.5) { fr = 1.0; ex -= 1; }
    for (int t = 0; t < 5; t++) {
        const long double sc = t < 4 ? (long double)fr / (long double)(1 << t) : 1.0L;
        for (size_t k = 0; k < c.size(); k++) {
            m.c[k] = llrintl(c[k] * sc * 4611686018427387904.0L);  // 2^62
            m.s[k] = llrintl(s[k] * sc * 4611686018427387904.0L);
        }
        m.expo = t < 4 ? ex + t : 0;
        m.post = t < 4 ? 1.0 : factor;
        // no digits pass 2^24 in short lists
        const long long any = 256 * 256 * (long long)D.K;
        long long b[3] = {3 * any, 4 * any, 5 * any};
        if (b[2] > 1 << 24) level_bounds(D, half, m, b);
        if (b[0] > 1 << 24) continue;
        bool ok = true;
        for (int v = 0; v < 2; v++) {
            const long long top = (1ll << 25) - b[v + 1];
            if (top < 1 << 22) ok = false;
            m.top[v] = b[v + 1] <= 1 << 24 ? INFINITY : (float)top;
        }
        if (ok) return true;
    }
    return false;
}

}  // namespace sg
