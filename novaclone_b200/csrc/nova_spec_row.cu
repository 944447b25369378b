// Real transforms along k of the spectral Poisson solve: rows of N2 = 2 m
// reals <-> m + 1 half-spectrum values (unnormalised, as cuFFT's D2Z and Z2D;
// the imaginary parts of the first and last value are ignored on the way
// back).  A row is an m-point complex transform of z[n] = x[2n] + i x[2n + 1]
// (nova_spec.cuh), with
//   X[k] = e - i W^k o,  X[m - k] = conj(e + i W^k o),  W = W_N2,
//   e, o = (Z[k] +- conj Z[m - k]) / 2
// afterwards, and before the inverse
//   Z[k] = E + i O,  Z[m - k] = conj(E) + i conj(O),
//   E = X[k] + conj X[m - k],  O = (X[k] - conj X[m - k]) W^-k.
// Bound by HBM (16 B per real value moved); every load of a block is in flight
// before its first barrier.  Against cuFFT's real
// kernels: 256^3 55 us (68), rows of 384 of the 192 x 192 x 384 mesh 50 us (120),
// rows of 128 of the 256 x 257 x 128 wall mesh 27 us (53), 128^3 9 us (11).
#include "nova_ops.cuh"
#include "nova_spec.cuh"

namespace nova {

// rows r = 0..rows-1: real row (r / ny) plane + (r % ny) N2, spectrum row r (m + 1)
struct Rows {
    long long rows, plane;
    int ny;
};

// the half lengths m = N2 / 2 of group G: false where m is none of them
template <int G>
bool rows_group(int m, const Rows &R, bool inv, const double *x, double2 *spec, double *p, const double2 *tw,
                cudaStream_t st);

#ifdef NOVA_FFT_GROUP
namespace {

template <int R1, int R2> struct RowCfg {
    static constexpr int m = R1 * R2, T = Line<R1, R2>::T, U = Line<R1, R2>::U;
    static constexpr int B = 128 / T;  // rows per block
    static constexpr int threads = B * T;
    static constexpr int LD = R1 * (R2 + 1);  // transposed rows padded: 16-byte accesses without bank conflicts
    static constexpr size_t smem = sizeof(double2) * (2 * m + B * LD);
    static constexpr int minb = R2 >= 12 || U * R1 >= 12 ? 4 : 5;
};

// step 1 and 2 of a row in shared memory: v0 (step-1 order) -> natural order in s
template <int R1, int R2, bool INV>
__device__ __forceinline__ void row_fft(double2 (&v0)[Line<R1, R2>::U][R1], double2 (&w)[R2], double2 *s,
                                        const double2 *tw, int t)
{
    constexpr int m = R1 * R2, T = Line<R1, R2>::T, U = Line<R1, R2>::U;
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int n2 = t + T * u;
        dft<R1, 2 * m, INV>(v0[u], tw);
#pragma unroll
        for (int k1 = 0; k1 < R1; k1++) {
            const double2 f = tw[2 * n2 * k1];
            s[k1 * (R2 + 1) + n2] = k1 == 0 ? v0[u][0] : cmul(v0[u][k1], INV ? conj2(f) : f);
        }
    }
    __syncthreads();
    if (T == R1 || t < R1) {
#pragma unroll
        for (int n2 = 0; n2 < R2; n2++) w[n2] = s[t * (R2 + 1) + n2];
        dft<R2, 2 * m, INV>(w, tw);
    }
}

template <int R1, int R2>
__global__ void __launch_bounds__(RowCfg<R1, R2>::threads, RowCfg<R1, R2>::minb)
    k_row_fwd(Rows R, const double *__restrict__ x, double2 *__restrict__ spec, const double2 *__restrict__ twN)
{
    using C = RowCfg<R1, R2>;
    constexpr int m = C::m, T = C::T, U = C::U;
    extern __shared__ __align__(16) unsigned char smraw[];
    double2 *tw = reinterpret_cast<double2 *>(smraw);  // W_N2^k, k < N2
    const int row = threadIdx.x / T, t = threadIdx.x % T;
    double2 *s = tw + 2 * m + row * C::LD;
    const long long r = blockIdx.x * (long long)C::B + row;
    const bool on = r < R.rows;
    const double2 *z = reinterpret_cast<const double2 *>(x + (on ? (r / R.ny) * R.plane + (r % R.ny) * (2 * m) : 0));
    double2 v[U][R1], w[R2];
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
        for (int n1 = 0; n1 < R1; n1++) v[u][n1] = on ? z[R2 * n1 + t + T * u] : make_double2(0.0, 0.0);
    for (int k = threadIdx.x; k < 2 * m; k += C::threads) tw[k] = twN[k];
    __syncthreads();
    row_fft<R1, R2, false>(v, w, s, tw, t);
    __syncthreads();  // s is rewritten in natural order
    if (T == R1 || t < R1)
#pragma unroll
        for (int k2 = 0; k2 < R2; k2++) s[t + R1 * k2] = w[k2];
    __syncthreads();
    if (!on) return;
    double2 *X = spec + r * (m + 1);
#pragma unroll 4
    for (int k = t; k <= m / 2; k += T) {
        const double2 a = s[k], b = s[k == 0 ? 0 : m - k];
        const double2 e = make_double2(0.5 * (a.x + b.x), 0.5 * (a.y - b.y));
        const double2 o = cmul(make_double2(0.5 * (a.x - b.x), 0.5 * (a.y + b.y)), tw[k]);
        X[k] = make_double2(e.x + o.y, e.y - o.x);
        X[m - k] = make_double2(e.x - o.y, -(e.y + o.x));
    }
}

template <int R1, int R2>
__global__ void __launch_bounds__(RowCfg<R1, R2>::threads, RowCfg<R1, R2>::minb)
    k_row_inv(Rows R, const double2 *__restrict__ spec, double *__restrict__ x, const double2 *__restrict__ twN)
{
    using C = RowCfg<R1, R2>;
    constexpr int m = C::m, T = C::T, U = C::U, P = (m / 2 + T) / T;  // pairs (k, m - k) per thread
    extern __shared__ __align__(16) unsigned char smraw[];
    double2 *tw = reinterpret_cast<double2 *>(smraw);
    const int row = threadIdx.x / T, t = threadIdx.x % T;
    double2 *s = tw + 2 * m + row * C::LD;
    const long long r = blockIdx.x * (long long)C::B + row;
    const bool on = r < R.rows;
    const double2 *X = spec + (on ? r * (m + 1) : 0);
    double2 a[P], b[P];
#pragma unroll
    for (int q = 0; q < P; q++) {
        const int k = t + T * q;
        const bool in = on && k <= m / 2;
        a[q] = in ? X[k] : make_double2(0.0, 0.0);
        b[q] = in ? X[m - k] : make_double2(0.0, 0.0);
    }
    for (int k = threadIdx.x; k < 2 * m; k += C::threads) tw[k] = twN[k];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < P; q++) {
        const int k = t + T * q;
        if (k > m / 2) break;
        if (k == 0) a[q].y = b[q].y = 0.0;
        const double2 E = make_double2(a[q].x + b[q].x, a[q].y - b[q].y);
        const double2 O = cmul(make_double2(a[q].x - b[q].x, a[q].y + b[q].y), conj2(tw[k]));
        s[k] = make_double2(E.x - O.y, E.y + O.x);
        if (k != 0 && 2 * k != m) s[m - k] = make_double2(E.x + O.y, O.x - E.y);
    }
    __syncthreads();
    double2 v[U][R1], w[R2];
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
        for (int n1 = 0; n1 < R1; n1++) v[u][n1] = s[R2 * n1 + t + T * u];
    __syncthreads();
    row_fft<R1, R2, true>(v, w, s, tw, t);
    if (on && (T == R1 || t < R1)) {
        double2 *z = reinterpret_cast<double2 *>(x + (r / R.ny) * R.plane + (r % R.ny) * (2 * m));
#pragma unroll
        for (int k2 = 0; k2 < R2; k2++) z[t + R1 * k2] = w[k2];
    }
}

template <int R1, int R2>
void row(const Rows &R, bool inv, const double *x, double2 *spec, double *p, const double2 *tw, cudaStream_t st)
{
    using C = RowCfg<R1, R2>;
    const unsigned nb = (unsigned)((R.rows + C::B - 1) / C::B);
    if (inv) {
        NOVA_SPEC_SMEM((k_row_inv<R1, R2>), C::smem);
        k_row_inv<R1, R2><<<nb, C::threads, C::smem, st>>>(R, spec, p, tw);
    } else {
        NOVA_SPEC_SMEM((k_row_fwd<R1, R2>), C::smem);
        k_row_fwd<R1, R2><<<nb, C::threads, C::smem, st>>>(R, x, spec, tw);
    }
}

}  // namespace

template <int G>
bool rows_group(int m, const Rows &R, bool inv, const double *x, double2 *spec, double *p, const double2 *tw,
                cudaStream_t st)
{
    switch (m) {
#define NOVA_X(l, r1, r2) \
    case l: row<r1, r2>(R, inv, x, spec, p, tw, st); return true;
        NOVA_FFT_GROUP(NOVA_X)
#undef NOVA_X
    default: return false;
    }
}

template bool rows_group<NOVA_PART>(int, const Rows &, bool, const double *, double2 *, double *, const double2 *,
                                    cudaStream_t);
#else
namespace {

void rows_any(const Rows &R, int n2, bool inv, const double *x, void *spec, double *p, const double *tw,
              cudaStream_t st)
{
    const int m = n2 / 2;
    double2 *s = (double2 *)spec;
    const double2 *w = reinterpret_cast<const double2 *>(tw);
    (void)(rows_group<0>(m, R, inv, x, s, p, w, st) || rows_group<1>(m, R, inv, x, s, p, w, st) ||
           rows_group<2>(m, R, inv, x, s, p, w, st) || rows_group<3>(m, R, inv, x, s, p, w, st) ||
           rows_group<4>(m, R, inv, x, s, p, w, st) || rows_group<5>(m, R, inv, x, s, p, w, st));
}

}  // namespace

bool spec_rows_fit(int n2) { return n2 % 2 == 0 && fft_length(n2 / 2); }

void launch_rows_fwd(int planes, int ny, long long plane, int n2, const double *x, void *spec, const double *twN,
                     cudaStream_t st)
{
    rows_any(Rows{(long long)planes * ny, plane, ny}, n2, false, x, spec, nullptr, twN, st);
}

void launch_rows_inv(int planes, int ny, long long plane, int n2, const void *spec, double *x, const double *twN,
                     cudaStream_t st)
{
    rows_any(Rows{(long long)planes * ny, plane, ny}, n2, true, nullptr, const_cast<void *>(spec), x, twN, st);
}
#endif

}  // namespace nova
