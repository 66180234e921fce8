// Lined-up overlaps <n l m | n' l' m> of Slater functions on two centres, l <= 1,
// by SOLAP's method (overlap_D.f:701-962): basic integrals <n00|n'00> from a 1F1
// table (Fernandez-Rico), then the recurrences in l, l' and m.
//
// Written for GB300's FP64 unit, which takes a warp instruction 64-76 cycles: what
// does not depend on the distance is a table or a closed form.
//   - basic integral of the indices n (larger exponent z) and n' (smaller z'),
//     N = n + n':
//       <n|n'> = 4 pi e^{-zR} (z + z')^{-(N+1)} sum_k ((z + z') R)^k D_k,
//       D_k = sum_j 1F1[j+1, k+2] c(n, n', k, j),
//       c = n! n'! (N - k)! / ((k + 1)! (n + j - k)! (n' - j)!),
//     with c from a table: one FMA per term and one multiplication per k, where
//     SOLAP's loops take two and four.
//   - for l <= 1 the recurrences reduce to
//       <s|s>  = B(n, n')
//       <p|s>  =  P(n, n')   with P(n, n') = (B(n+1, n') + R^2 B(n-1, n') - B(n-1, n'+2)) / 2R
//       <s|p>  = -(B(n, n'+1) + R^2 B(n, n'-1) - B(n+2, n'-1)) / 2R
//       <p|p>0 = -(P(n, n'+1) + R^2 P(n, n'-1) - P(n+2, n'-1)) / 2R
//       <p|p>1 = (2 (B(n+1, n'+1) + R^2 (B(n+1, n'-1) + B(n-1, n'+1))) - B(n+3, n'-1)
//                 - B(n-1, n'+3) - R^4 B(n-1, n'-1)) / 8R^2
//     (n, n' now of atoms A and B), which read 13 cells B for the four shell pairs of
//     two atoms with s and p shells, where the tabulated recurrences filled 49-entry
//     arrays three times per shell pair.
// The 1F1 table starts at the highest column these cells read.
#pragma once

#include <cmath>
#include <cstring>

namespace elhl {
namespace sto {

constexpr int kMaxN = 3, kMaxL = 1;
constexpr int kIdx = kMaxN + 4;             // cell indices 0 .. 6
constexpr int kKs = 2 * (kMaxN + 1) + 1;    // k = 0 .. N, N <= 8
constexpr int kRows = kIdx + 2;             // 1F1 rows 1 .. 7 (and one beyond)
constexpr int kCols = kKs + 2;              // 1F1 columns 2 .. 10
constexpr int kCellTable = kIdx * kIdx * kKs * kIdx;
constexpr int kSeries = 1024;               // terms of the 1F1 series
constexpr int kSeriesTable = kCols * kSeries;
constexpr int kTableMax = kCellTable > kSeriesTable ? kCellTable : kSeriesTable;

struct Tables {
    const double *cell, *series;
};

__host__ __device__ inline double factorial(int n) {
    double f = 1.0;
    for (int i = 2; i <= n; ++i) f *= (double)i;
    return f;
}
// c(n, n', k, j), 0 outside the sum
__host__ __device__ inline double cell_constant(int i) {
    const int j = i % kIdx, k = i / kIdx % kKs, np = i / (kIdx * kKs) % kIdx, n = i / (kIdx * kKs * kIdx);
    if (k > n + np || j > np || j > k || n + j - k < 0) return 0.0;
    return factorial(n) * factorial(np) * factorial(n + np - k) /
           (factorial(k + 1) * factorial(n + j - k) * factorial(np - j));
}
// 1 / ((g + i) (i + 1)) for the series of column g; row g = 0: the reciprocals 1 / (i + 1)
__host__ __device__ inline double series_constant(int q) {
    const int g = q / kSeries, i = q % kSeries;
    return 1.0 / ((double)(g > 0 ? g + i : 1) * (double)(i + 1));
}

__host__ __device__ inline bool supported(int n, int l) { return n >= 1 && n <= kMaxN && l >= 0 && l <= kMaxL; }

// the largest index on A and on B and the largest index sum of a shell pair's cells
struct Reach {
    int a, b, sum;
};
__host__ __device__ inline Reach reach(int na, int la, int nb, int lb) {
    return Reach{na + la + 2 * lb, nb + lb + 2 * la, na + nb + la + lb};
}
__host__ __device__ inline Reach widest(const Reach &x, const Reach &y) {
    return Reach{x.a > y.a ? x.a : y.a, x.b > y.b ? x.b : y.b, x.sum > y.sum ? x.sum : y.sum};
}

// per-AO normalisation of one exponent: sqrt((2 zeta)^(2n+1) (2l+1) / (2n)!) / sqrt(4 pi),
// so that the product of two AOs' factors is GET_ANOR's (overlap_D.f:464-517)
inline double norm(double zeta, int n, int l) {
    double a = 1.0;
    for (int e = 0; e < 2 * n + 1; ++e) a *= zeta * 2.0;
    return std::sqrt(a * (2.0 * l + 1.0) / factorial(2 * n)) / std::sqrt(4.0 * 3.141592653589793);
}

struct PairTable {
    const double *cell;
    double R, Rinv, zzpR;
    bool a_big;
    double scale[kKs + 1];         // 4 pi e^{-zR} (z + z')^{-(N+1)} by N
    double f[kRows][kCols];        // 1F1[i, j, (z - z') R]
};

__host__ __device__ inline int exponent_of(double x) {
#ifdef __CUDA_ARCH__
    return (__double2hiint(x) >> 20) & 0x7ff;
#else
    unsigned long long b;
    std::memcpy(&b, &x, 8);
    return (int)((b >> 52) & 0x7ff);
#endif
}

// The table of exponents za (A) and zb (B) at distance R for cells within `need`.
// 1F1[i, j] for i <= min(rows, j - 1) as SOLAP builds it (overlap_D.f:766-819): the
// top column from its series at ia and ia + 1 and the three-term recursion in i, the
// lower columns by the contiguous relations.  The series of ia + 1 has the terms of
// ia's times (ia + i) / ia, so one loop sums both.
__host__ __device__ inline void pair_table(const Tables &T, double za, double zb, double R, const Reach &need,
                                           PairTable &t) {
    const bool a_big = za >= zb;
    const double z = a_big ? za : zb, zp = a_big ? zb : za;
    const int g = need.sum + 2;                          // top column
    const int rows = (a_big ? need.b : need.a) + 1;      // rows 1 .. rows
    t.cell = T.cell;
    t.a_big = a_big;
    t.R = R;
    t.Rinv = 1.0 / R;
    t.zzpR = (z + zp) * R;
    const double zi = 1.0 / (z + zp);
    double sc = 12.566370614359172953850573533118012 * exp(-z * R) * zi;
    for (int n = 0; n <= need.sum; ++n) {
        t.scale[n] = sc;
        sc *= zi;
    }
    const double arg = (z - zp) * R;
    int ia = (g - (int)z) / 2;
    if (ia < 1) ia = 1;
    if (ia >= rows) ia = rows - 1;

    const double *ser = T.series + (size_t)g * kSeries, *rcp = T.series - 1;  // rcp[i] = 1 / i
    double term = 1.0, fa = 1.0, fw = (double)ia, d = (double)ia;  // fw: sum of term_i (ia + i)
    for (int i = 0; i < kSeries - 1; ++i) {
        term = term * (ser[i] * d) * arg;                // term_{i+1}
        d += 1.0;
        fa += term;
        fw = fma(term, d, fw);
        if (exponent_of(term) + 80 < exponent_of(fa)) break;  // below 2^-79 of the sum, and falling
    }
    t.f[ia][g] = fa;
    t.f[ia + 1][g] = fw * rcp[ia];
    double aux = arg - (double)g;
    for (int i = ia + 1; i <= rows - 1; ++i)
        t.f[i + 1][g] = ((aux + (double)(i + i)) * t.f[i][g] + (double)(g - i) * t.f[i - 1][g]) * rcp[i];
    for (int i = ia; i >= 2; --i)
        t.f[i - 1][g] = ((double)i * t.f[i + 1][g] - (aux + (double)(i + i)) * t.f[i][g]) * rcp[g - i];
    for (int j = g - 1; j >= 2; --j) {
        const double ji = rcp[j];
        t.f[1][j] = (t.f[2][j + 1] + (double)(j - 1) * t.f[1][j + 1]) * ji;
        aux = arg * ji;
        const int itop = rows - 1 < j - 2 ? rows - 1 : j - 2;
        for (int i = 1; i <= itop; ++i) t.f[i + 1][j] = fma(aux, t.f[i + 1][j + 1], t.f[i][j]);
    }
}

// basic integral of indices ka (A) and kb (B)
__host__ __device__ inline double cell(const PairTable &t, int ka, int kb) {
    const int n = t.a_big ? ka : kb, np = t.a_big ? kb : ka, N = n + np;
    const double *c = t.cell + (size_t)(n * kIdx + np) * kKs * kIdx;
    double sum = 0.0;
    for (int k = N; k >= 0; --k) {
        double v = sum * t.zzpR;
        const int j0 = k - n > 0 ? k - n : 0, j1 = k < np ? k : np;
        for (int j = j0; j <= j1; ++j) v = fma(t.f[j + 1][k + 2], c[k * kIdx + j], v);
        sum = v;
    }
    return t.scale[N] * sum;
}

// <na la m | nb lb m>, m = 0 .. min(la, lb), unnormalised (sol[1] = 0 unless both are p)
__host__ __device__ inline void lined_up(const PairTable &t, int na, int la, int nb, int lb, double *sol) {
    const double R2 = t.R * t.R, h = 0.5 * t.Rinv;
    sol[1] = 0.0;
    if (!la && !lb) {
        sol[0] = cell(t, na, nb);
    } else if (!lb) {
        sol[0] = h * (cell(t, na + 1, nb) + R2 * cell(t, na - 1, nb) - cell(t, na - 1, nb + 2));
    } else if (!la) {
        sol[0] = -h * (cell(t, na, nb + 1) + R2 * cell(t, na, nb - 1) - cell(t, na + 2, nb - 1));
    } else {
        const double pp = cell(t, na + 1, nb + 1), pm = cell(t, na + 1, nb - 1), mp = cell(t, na - 1, nb + 1);
        const double mm = cell(t, na - 1, nb - 1), p3 = cell(t, na + 3, nb - 1), m3 = cell(t, na - 1, nb + 3);
        const double Ppp = h * (pp + R2 * mp - m3), Ppm = h * (pm + R2 * mm - mp), P3m = h * (p3 + R2 * pm - pp);
        sol[0] = -h * (Ppp + R2 * Ppm - P3m);
        sol[1] = 0.5 * h * h * (2.0 * (pp + R2 * (pm + mp)) - p3 - m3 - R2 * R2 * mm);
    }
}

}  // namespace sto
}  // namespace elhl
