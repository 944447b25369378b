// Register-resident DFT building blocks of the spectral Poisson solve
// (nova_spec.cuh, nova_pois_i.cu, nova_pois_dct.cu, nova_fft2d.cu): complex
// products, and R-point DFTs (R = 4, 5, 6, 8, 9, 10, 12, 15, 16) in natural order with
// twiddles W_R^m read from a table of W_N^m (N a multiple of R) at
// compile-time indices.
#pragma once

#include <cuda_runtime.h>

namespace nova {

__device__ __forceinline__ double2 cmul(double2 a, double2 w)
{
    return make_double2(fma(a.x, w.x, -a.y * w.y), fma(a.x, w.y, a.y * w.x));
}

__device__ __forceinline__ double2 conj2(double2 w) { return make_double2(w.x, -w.y); }

// 1/a for a >= 1e-16 (normal in FP32 for every mesh the Poisson scales meet):
// the correctly rounded FP32 reciprocal refined by two Newton-Raphson steps
// y <- y + y (1 - a y) in FP64 (relative error about 2^-23 -> 2^-46 -> below
// an ulp of FP64, up to the rounding of the last step)
__device__ __forceinline__ double recip(double a)
{
    double y = (double)__frcp_rn((float)a);
    y = fma(y, fma(-a, y, 1.0), y);
    return fma(y, fma(-a, y, 1.0), y);
}

__host__ __device__ constexpr int bitrev(int x, int bits)
{
    int r = 0;
    for (int b = 0; b < bits; b++) r |= ((x >> b) & 1) << (bits - 1 - b);
    return r;
}

// in-place R-point DFT of v in natural order: v[k] = sum_n v[n] W_R^(+-n k)
// (- forward, + inverse); W_R^m = tw[m * (N / R)] (tw: the W_N table in
// shared memory, read at compile-time indices, i.e. broadcast).
// R = 8: radix-2 decimation in time.
template <int R, int N, bool INV> __device__ __forceinline__ void dft_radix2(double2 (&v)[R], const double2 *tw)
{
    constexpr int bits = R == 8 ? 3 : 4;
#pragma unroll
    for (int x = 0; x < R; x++) {
        const int y = bitrev(x, bits);
        if (y > x) {
            const double2 t = v[x];
            v[x] = v[y];
            v[y] = t;
        }
    }
#pragma unroll
    for (int len = 2; len <= R; len *= 2) {
        const int half = len / 2;
#pragma unroll
        for (int b = 0; b < R; b += len) {
#pragma unroll
            for (int j = 0; j < half; j++) {
                const double2 a = v[b + j];
                double2 c = v[b + j + half];
                if (j != 0) {
                    const double2 w = tw[j * (R / len) * (N / R)];
                    c = cmul(c, INV ? conj2(w) : w);
                }
                v[b + j] = make_double2(a.x + c.x, a.y + c.y);
                v[b + j + half] = make_double2(a.x - c.x, a.y - c.y);
            }
        }
    }
}

// 4-point DFT in place; W_4 = -i forward, +i inverse (no multiplications)
template <bool INV> __device__ __forceinline__ void dft4(double2 &a0, double2 &a1, double2 &a2, double2 &a3)
{
    const double2 t0 = make_double2(a0.x + a2.x, a0.y + a2.y), t1 = make_double2(a0.x - a2.x, a0.y - a2.y);
    const double2 t2 = make_double2(a1.x + a3.x, a1.y + a3.y), d = make_double2(a1.x - a3.x, a1.y - a3.y);
    const double2 t3 = INV ? make_double2(-d.y, d.x) : make_double2(d.y, -d.x);
    a0 = make_double2(t0.x + t2.x, t0.y + t2.y);
    a2 = make_double2(t0.x - t2.x, t0.y - t2.y);
    a1 = make_double2(t1.x + t3.x, t1.y + t3.y);
    a3 = make_double2(t1.x - t3.x, t1.y - t3.y);
}

// R = 16 as 4 x 4 (n = 4 n1 + n2, k = k1 + 4 k2): 4-point DFTs over n1, the
// twiddles W_16^(n2 k1) (W_16^4 = -+i free), 4-point DFTs over n2, then the
// 4 x 4 index transpose, which is a renaming of registers
template <int N, bool INV> __device__ __forceinline__ void dft16(double2 (&v)[16], const double2 *tw)
{
#pragma unroll
    for (int n2 = 0; n2 < 4; n2++) dft4<INV>(v[n2], v[4 + n2], v[8 + n2], v[12 + n2]);
#pragma unroll
    for (int n2 = 1; n2 < 4; n2++)
#pragma unroll
        for (int k1 = 1; k1 < 4; k1++) {
            double2 &x = v[4 * k1 + n2];
            if (n2 * k1 == 4)
                x = INV ? make_double2(-x.y, x.x) : make_double2(x.y, -x.x);
            else
                x = cmul(x, INV ? conj2(tw[n2 * k1 * (N / 16)]) : tw[n2 * k1 * (N / 16)]);
        }
#pragma unroll
    for (int k1 = 0; k1 < 4; k1++) dft4<INV>(v[4 * k1], v[4 * k1 + 1], v[4 * k1 + 2], v[4 * k1 + 3]);
    double2 o[16];
#pragma unroll
    for (int k1 = 0; k1 < 4; k1++)
#pragma unroll
        for (int k2 = 0; k2 < 4; k2++) o[k1 + 4 * k2] = v[4 * k1 + k2];
#pragma unroll
    for (int k = 0; k < 16; k++) v[k] = o[k];
}

// 2-, 3- and 5-point DFTs in place (strided registers a[0], a[S], a[2 S], ...)
template <int S> __device__ __forceinline__ void dft2s(double2 *a)
{
    const double2 t = a[S];
    a[S] = make_double2(a[0].x - t.x, a[0].y - t.y);
    a[0] = make_double2(a[0].x + t.x, a[0].y + t.y);
}

template <int S, bool INV> __device__ __forceinline__ void dft3s(double2 *a)
{
    const double h = 0.86602540378443864676;  // sqrt(3)/2
    const double2 t = make_double2(a[S].x + a[2 * S].x, a[S].y + a[2 * S].y);
    const double2 d = make_double2(h * (a[S].x - a[2 * S].x), h * (a[S].y - a[2 * S].y));
    const double2 u = make_double2(fma(-0.5, t.x, a[0].x), fma(-0.5, t.y, a[0].y));
    a[0] = make_double2(a[0].x + t.x, a[0].y + t.y);
    // u -+ i d
    a[S] = INV ? make_double2(u.x - d.y, u.y + d.x) : make_double2(u.x + d.y, u.y - d.x);
    a[2 * S] = INV ? make_double2(u.x + d.y, u.y - d.x) : make_double2(u.x - d.y, u.y + d.x);
}

template <int S, bool INV> __device__ __forceinline__ void dft5s(double2 *a)
{
    // cos and sin of 2 pi / 5 and 4 pi / 5
    const double c1 = 0.30901699437494742410, c2 = -0.80901699437494742410;
    const double s1 = 0.95105651629515357212, s2 = 0.58778525229247312917;
    const double2 p1 = make_double2(a[S].x + a[4 * S].x, a[S].y + a[4 * S].y);
    const double2 p2 = make_double2(a[2 * S].x + a[3 * S].x, a[2 * S].y + a[3 * S].y);
    const double2 m1 = make_double2(a[S].x - a[4 * S].x, a[S].y - a[4 * S].y);
    const double2 m2 = make_double2(a[2 * S].x - a[3 * S].x, a[2 * S].y - a[3 * S].y);
    const double2 e1 = make_double2(fma(c1, p1.x, fma(c2, p2.x, a[0].x)), fma(c1, p1.y, fma(c2, p2.y, a[0].y)));
    const double2 e2 = make_double2(fma(c2, p1.x, fma(c1, p2.x, a[0].x)), fma(c2, p1.y, fma(c1, p2.y, a[0].y)));
    const double2 o1 = make_double2(fma(s1, m1.x, s2 * m2.x), fma(s1, m1.y, s2 * m2.y));
    const double2 o2 = make_double2(fma(s2, m1.x, -s1 * m2.x), fma(s2, m1.y, -s1 * m2.y));
    a[0] = make_double2(a[0].x + p1.x + p2.x, a[0].y + p1.y + p2.y);
    const double g = INV ? -1.0 : 1.0;  // X_k = e - i o (forward)
    a[S] = make_double2(fma(g, o1.y, e1.x), fma(-g, o1.x, e1.y));
    a[4 * S] = make_double2(fma(-g, o1.y, e1.x), fma(g, o1.x, e1.y));
    a[2 * S] = make_double2(fma(g, o2.y, e2.x), fma(-g, o2.x, e2.y));
    a[3 * S] = make_double2(fma(-g, o2.y, e2.x), fma(g, o2.x, e2.y));
}

template <int P, int S, bool INV> __device__ __forceinline__ void dft_prime(double2 *a)
{
    if constexpr (P == 2)
        dft2s<S>(a);
    else if constexpr (P == 3)
        dft3s<S, INV>(a);
    else if constexpr (P == 4)
        dft4<INV>(a[0], a[S], a[2 * S], a[3 * S]);
    else
        dft5s<S, INV>(a);
}

// R = A x B (n = B n1 + n2, k = k1 + A k2), A and B in 2..5: A-point DFTs over
// n1, the twiddles W_R^(n2 k1), B-point DFTs over n2, then the index transpose
template <int A, int B, int N, bool INV> __device__ __forceinline__ void dft_ab(double2 (&v)[A * B], const double2 *tw)
{
    constexpr int R = A * B;
#pragma unroll
    for (int n2 = 0; n2 < B; n2++) dft_prime<A, B, INV>(&v[n2]);
#pragma unroll
    for (int n2 = 1; n2 < B; n2++)
#pragma unroll
        for (int k1 = 1; k1 < A; k1++) {
            double2 &x = v[B * k1 + n2];
            if (4 * n2 * k1 == R)
                x = INV ? make_double2(-x.y, x.x) : make_double2(x.y, -x.x);
            else
                x = cmul(x, INV ? conj2(tw[n2 * k1 * (N / R)]) : tw[n2 * k1 * (N / R)]);
        }
#pragma unroll
    for (int k1 = 0; k1 < A; k1++) dft_prime<B, 1, INV>(&v[B * k1]);
    double2 o[R];
#pragma unroll
    for (int k1 = 0; k1 < A; k1++)
#pragma unroll
        for (int k2 = 0; k2 < B; k2++) o[k1 + A * k2] = v[B * k1 + k2];
#pragma unroll
    for (int k = 0; k < R; k++) v[k] = o[k];
}

template <int R, int N, bool INV> __device__ __forceinline__ void dft(double2 (&v)[R], const double2 *tw)
{
    static_assert(R == 4 || R == 5 || R == 6 || R == 8 || R == 9 || R == 10 || R == 12 || R == 15 || R == 16,
                  "register DFT lengths");
    if constexpr (R == 16)
        dft16<N, INV>(v, tw);
    else if constexpr (R == 4)
        dft4<INV>(v[0], v[1], v[2], v[3]);
    else if constexpr (R == 5)
        dft5s<1, INV>(&v[0]);
    else if constexpr (R == 6)
        dft_ab<2, 3, N, INV>(v, tw);
    else if constexpr (R == 9)
        dft_ab<3, 3, N, INV>(v, tw);
    else if constexpr (R == 15)
        dft_ab<3, 5, N, INV>(v, tw);
    else if constexpr (R == 10)
        dft_ab<2, 5, N, INV>(v, tw);
    else if constexpr (R == 12)
        dft_ab<4, 3, N, INV>(v, tw);
    else
        dft_radix2<R, N, INV>(v, tw);
}

}  // namespace nova
