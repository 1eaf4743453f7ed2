// dft.cuh -- R-point DFTs in one thread's registers, R = 2..16 with factors 2,
// 3, 5, 7, for the pair-packed step kernels (pair.cuh).
//
//   Reg<T, R, SIGN>::run(v):  v[k] <- sum_n v[n] exp(SIGN * 2 pi i n k / R)
//
// Composite lengths with coprime factors use the Good-Thomas index maps, which
// need no twiddle factors; 4, 8, 9 and 16 are Cooley-Tukey with constant ones.
#pragma once
#include "common.cuh"

namespace scft {

// multiply by SIGN * i
template <typename T, int SIGN>
__device__ __forceinline__ cplx<T> rot(cplx<T> a)
{
    return SIGN > 0 ? cplx<T>{-a.y, a.x} : cplx<T>{a.y, -a.x};
}

// multiply by c + SIGN * i * s
template <typename T, int SIGN>
__device__ __forceinline__ cplx<T> turn(cplx<T> a, T c, T s)
{
    return SIGN > 0 ? cplx<T>{a.x * c - a.y * s, a.x * s + a.y * c} : cplx<T>{a.x * c + a.y * s, a.y * c - a.x * s};
}

template <typename T, int R, int SIGN>
struct Reg;

template <typename T, int SIGN>
struct Reg<T, 1, SIGN> {
    static __device__ __forceinline__ void run(cplx<T> *) {}
};

template <typename T, int SIGN>
struct Reg<T, 2, SIGN> {
    static __device__ __forceinline__ void run(cplx<T> *v)
    {
        const cplx<T> a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    }
};

template <typename T, int SIGN>
struct Reg<T, 3, SIGN> {
    static __device__ __forceinline__ void run(cplx<T> *v)
    {
        const T h = (T)0.86602540378443864676;  // sqrt(3)/2
        const cplx<T> t = cadd(v[1], v[2]), u = rot<T, SIGN>(csub(v[1], v[2]));
        const cplx<T> m = {v[0].x - (T)0.5 * t.x, v[0].y - (T)0.5 * t.y};
        v[0] = cadd(v[0], t);
        v[1] = {m.x + h * u.x, m.y + h * u.y};
        v[2] = {m.x - h * u.x, m.y - h * u.y};
    }
};

template <typename T, int SIGN>
struct Reg<T, 4, SIGN> {
    static __device__ __forceinline__ void run(cplx<T> *v)
    {
        const cplx<T> a = cadd(v[0], v[2]), b = csub(v[0], v[2]);
        const cplx<T> c = cadd(v[1], v[3]), d = rot<T, SIGN>(csub(v[1], v[3]));
        v[0] = cadd(a, c);
        v[1] = cadd(b, d);
        v[2] = csub(a, c);
        v[3] = csub(b, d);
    }
};

template <typename T, int SIGN>
struct Reg<T, 5, SIGN> {
    static __device__ __forceinline__ void run(cplx<T> *v)
    {
        const T c1 = (T)0.30901699437494742410, c2 = (T)-0.80901699437494742410;  // cos(2 pi/5), cos(4 pi/5)
        const T s1 = (T)0.95105651629515357212, s2 = (T)0.58778525229247312917;   // sin(2 pi/5), sin(4 pi/5)
        const cplx<T> a1 = cadd(v[1], v[4]), a2 = cadd(v[2], v[3]);
        const cplx<T> b1 = rot<T, SIGN>(csub(v[1], v[4])), b2 = rot<T, SIGN>(csub(v[2], v[3]));
        const cplx<T> r1 = {v[0].x + c1 * a1.x + c2 * a2.x, v[0].y + c1 * a1.y + c2 * a2.y};
        const cplx<T> r2 = {v[0].x + c2 * a1.x + c1 * a2.x, v[0].y + c2 * a1.y + c1 * a2.y};
        const cplx<T> i1 = {s1 * b1.x + s2 * b2.x, s1 * b1.y + s2 * b2.y};
        const cplx<T> i2 = {s2 * b1.x - s1 * b2.x, s2 * b1.y - s1 * b2.y};
        v[0] = {v[0].x + a1.x + a2.x, v[0].y + a1.y + a2.y};
        v[1] = cadd(r1, i1);
        v[4] = csub(r1, i1);
        v[2] = cadd(r2, i2);
        v[3] = csub(r2, i2);
    }
};

template <typename T, int SIGN>
struct Reg<T, 7, SIGN> {
    static __device__ __forceinline__ void run(cplx<T> *v)
    {
        // cos and sin of 2 pi/7, 4 pi/7, 6 pi/7
        const T c[3] = {(T)0.62348980185873353053, (T)-0.22252093395631440429, (T)-0.90096886790241912624};
        const T s[3] = {(T)0.78183148246802980871, (T)0.97492791218182360702, (T)0.43388373911755812048};
        cplx<T> a[3], b[3];
#pragma unroll
        for (int j = 0; j < 3; j++) {
            a[j] = cadd(v[j + 1], v[6 - j]);
            b[j] = rot<T, SIGN>(csub(v[j + 1], v[6 - j]));
        }
        const cplx<T> v0 = v[0];
        v[0] = {v0.x + a[0].x + a[1].x + a[2].x, v0.y + a[0].y + a[1].y + a[2].y};
#pragma unroll
        for (int k = 1; k <= 3; k++) {
            cplx<T> r = v0, i = {(T)0, (T)0};
#pragma unroll
            for (int j = 1; j <= 3; j++) {
                const int p = (j * k) % 7, q = p <= 3 ? p : 7 - p;
                r.x += c[q - 1] * a[j - 1].x;
                r.y += c[q - 1] * a[j - 1].y;
                const T sj = p <= 3 ? s[q - 1] : -s[q - 1];
                i.x += sj * b[j - 1].x;
                i.y += sj * b[j - 1].y;
            }
            v[k] = cadd(r, i);
            v[7 - k] = csub(r, i);
        }
    }
};

template <typename T, int SIGN>
struct Reg<T, 8, SIGN> {
    static __device__ __forceinline__ void run(cplx<T> *v)
    {
        const T h = (T)0.70710678118654752440;  // sqrt(1/2)
        cplx<T> e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
        Reg<T, 4, SIGN>::run(e);
        Reg<T, 4, SIGN>::run(o);
        const cplx<T> r1 = rot<T, SIGN>(o[1]), r3 = rot<T, SIGN>(o[3]);
        o[1] = {h * (o[1].x + r1.x), h * (o[1].y + r1.y)};
        o[2] = rot<T, SIGN>(o[2]);
        o[3] = {h * (r3.x - o[3].x), h * (r3.y - o[3].y)};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            v[k] = cadd(e[k], o[k]);
            v[k + 4] = csub(e[k], o[k]);
        }
    }
};

template <typename T, int SIGN>
struct Reg<T, 9, SIGN> {
    static __device__ __forceinline__ void run(cplx<T> *v)
    {
        // cos and sin of 2 pi/9, 4 pi/9, 8 pi/9
        const T c1 = (T)0.76604444311897803520, s1 = (T)0.64278760968653932632;
        const T c2 = (T)0.17364817766693034885, s2 = (T)0.98480775301220805937;
        const T c4 = (T)-0.93969262078590838405, s4 = (T)0.34202014332566873304;
        cplx<T> t[3][3];
#pragma unroll
        for (int j = 0; j < 3; j++) {
#pragma unroll
            for (int r = 0; r < 3; r++) t[j][r] = v[j + 3 * r];
            Reg<T, 3, SIGN>::run(t[j]);
        }
        t[1][1] = turn<T, SIGN>(t[1][1], c1, s1);
        t[1][2] = turn<T, SIGN>(t[1][2], c2, s2);
        t[2][1] = turn<T, SIGN>(t[2][1], c2, s2);
        t[2][2] = turn<T, SIGN>(t[2][2], c4, s4);
#pragma unroll
        for (int k = 0; k < 3; k++) {
            cplx<T> u[3] = {t[0][k], t[1][k], t[2][k]};
            Reg<T, 3, SIGN>::run(u);
#pragma unroll
            for (int q = 0; q < 3; q++) v[k + 3 * q] = u[q];
        }
    }
};

template <typename T, int SIGN>
struct Reg<T, 16, SIGN> {
    static __device__ __forceinline__ void run(cplx<T> *v)
    {
        const T c = (T)0.92387953251128675613, s = (T)0.38268343236508977173;  // cos, sin of pi/8
        const T h = (T)0.70710678118654752440;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            cplx<T> t[4] = {v[j], v[j + 4], v[j + 8], v[j + 12]};
            Reg<T, 4, SIGN>::run(t);
            if (j == 1) {
                t[1] = turn<T, SIGN>(t[1], c, s);
                t[2] = turn<T, SIGN>(t[2], h, h);
                t[3] = turn<T, SIGN>(t[3], s, c);
            } else if (j == 2) {
                t[1] = turn<T, SIGN>(t[1], h, h);
                t[2] = rot<T, SIGN>(t[2]);
                t[3] = turn<T, SIGN>(t[3], -h, h);
            } else if (j == 3) {
                t[1] = turn<T, SIGN>(t[1], s, c);
                t[2] = turn<T, SIGN>(t[2], -h, h);
                t[3] = turn<T, SIGN>(t[3], -c, -s);
            }
#pragma unroll
            for (int k = 0; k < 4; k++) v[j + 4 * k] = t[k];
        }
        cplx<T> o[16];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            cplx<T> t[4] = {v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]};
            Reg<T, 4, SIGN>::run(t);
#pragma unroll
            for (int q = 0; q < 4; q++) o[k + 4 * q] = t[q];
        }
#pragma unroll
        for (int k = 0; k < 16; k++) v[k] = o[k];
    }
};

// R = A B with coprime A, B: n = (B n1 + A n2) mod R, and output k with
// k = k1 mod A, k = k2 mod B holds the (k1, k2) term
template <typename T, int A, int B, int SIGN>
struct RegCoprime {
    static constexpr int R = A * B;
    static __device__ __forceinline__ void run(cplx<T> *v)
    {
        cplx<T> t[A][B];
#pragma unroll
        for (int n1 = 0; n1 < A; n1++) {
#pragma unroll
            for (int n2 = 0; n2 < B; n2++) t[n1][n2] = v[(B * n1 + A * n2) % R];
            Reg<T, B, SIGN>::run(t[n1]);
        }
#pragma unroll
        for (int j = 0; j < B; j++) {
            cplx<T> u[A];
#pragma unroll
            for (int n1 = 0; n1 < A; n1++) u[n1] = t[n1][j];
            Reg<T, A, SIGN>::run(u);
#pragma unroll
            for (int i = 0; i < A; i++) t[i][j] = u[i];
        }
        // x[(B n1 + A n2) mod R] pairs with exp(2 pi i (n1 k/A + n2 k/B)), so k1 = k mod A, k2 = k mod B
#pragma unroll
        for (int k = 0; k < R; k++) v[k] = t[k % A][k % B];
    }
};

template <typename T, int SIGN>
struct Reg<T, 6, SIGN> : RegCoprime<T, 2, 3, SIGN> {};
template <typename T, int SIGN>
struct Reg<T, 10, SIGN> : RegCoprime<T, 2, 5, SIGN> {};
template <typename T, int SIGN>
struct Reg<T, 12, SIGN> : RegCoprime<T, 4, 3, SIGN> {};
template <typename T, int SIGN>
struct Reg<T, 14, SIGN> : RegCoprime<T, 2, 7, SIGN> {};
template <typename T, int SIGN>
struct Reg<T, 15, SIGN> : RegCoprime<T, 3, 5, SIGN> {};
template <typename T, int SIGN>
struct Reg<T, 20, SIGN> : RegCoprime<T, 4, 5, SIGN> {};
template <typename T, int SIGN>
struct Reg<T, 24, SIGN> : RegCoprime<T, 8, 3, SIGN> {};

// x / 3, correctly rounded but for double rounding below the normal range: the
// residual of x * (1/3) by a fused multiply-add, added back once (P. Markstein, IBM J.
// Res. Dev. 34, 1990); five operations instead of a divide's subroutine; infinities
// stay infinite
__device__ __forceinline__ double third(double x)
{
    const double c = 1.0 / 3.0, big = 1.7976931348623157e308;
    const double q = x * c;
    const double r = fma(fma(-3.0, q, x), c, q);
    return fabs(q) <= big ? r : q;
}

}  // namespace scft
