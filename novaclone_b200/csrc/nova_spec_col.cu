// Complex line transforms of the spectral Poisson solve along j (or i): in
// place on the half spectrum [i][j][kz], kSpecCols adjacent columns per block
// (nova_spec.cuh), unnormalised.  Bound by HBM (32 B per value); a block's
// loads are all in flight before its first barrier.  256^3: 50 us (cuFFT 48, byte
// floor 41), 192 x 192 x 384: 40 us (50), 128^3: 7.4 us (8.2).
#include "nova_ops.cuh"
#include "nova_spec.cuh"

namespace nova {

// the lengths of group G: false where L is none of them
template <int G> bool cols_group(int L, const Columns &C, bool inv, double2 *spec, const double2 *tw, cudaStream_t st);

#ifdef NOVA_FFT_GROUP
namespace {

template <int R1, int R2, bool INV>
__global__ void __launch_bounds__(column_threads<R1, R2>(), column_blocks<R1, R2>())
    k_col(Columns C, double2 *__restrict__ spec, const double2 *__restrict__ twL)
{
    constexpr int L = R1 * R2, T = Line<R1, R2>::T, U = Line<R1, R2>::U;
    extern __shared__ __align__(16) unsigned char smraw[];
    double2 *tw = reinterpret_cast<double2 *>(smraw), *S = tw + L;
    const int col = threadIdx.x % kSpecCols, t = threadIdx.x / kSpecCols;
    const long long c = blockIdx.x * (long long)kSpecCols + col;
    const bool on = c < C.total;
    double2 *p = spec + column_base(C, on ? c : 0);
    double2 v[U][R1], w[R2];
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
        for (int n1 = 0; n1 < R1; n1++) v[u][n1] = on ? p[(R2 * n1 + t + T * u) * C.step] : make_double2(0.0, 0.0);
    for (int k = threadIdx.x; k < L; k += column_threads<R1, R2>()) tw[k] = twL[k];
    __syncthreads();
    column_fft<R1, R2, INV>(v, w, S, tw, t, col);
    if (on && (T == R1 || t < R1))
#pragma unroll
        for (int k2 = 0; k2 < R2; k2++) p[(t + R1 * k2) * C.step] = w[k2];
}

template <int R1, int R2> void col(const Columns &C, bool inv, double2 *spec, const double2 *tw, cudaStream_t st)
{
    constexpr size_t smem = column_smem<R1, R2>();
    const unsigned nb = (unsigned)((C.total + kSpecCols - 1) / kSpecCols);
    if (inv) {
        NOVA_SPEC_SMEM((k_col<R1, R2, true>), smem);
        k_col<R1, R2, true><<<nb, column_threads<R1, R2>(), smem, st>>>(C, spec, tw);
    } else {
        NOVA_SPEC_SMEM((k_col<R1, R2, false>), smem);
        k_col<R1, R2, false><<<nb, column_threads<R1, R2>(), smem, st>>>(C, spec, tw);
    }
}

}  // namespace

template <int G> bool cols_group(int L, const Columns &C, bool inv, double2 *spec, const double2 *tw, cudaStream_t st)
{
    switch (L) {
#define NOVA_X(l, r1, r2) \
    case l: col<r1, r2>(C, inv, spec, tw, st); return true;
        NOVA_FFT_GROUP(NOVA_X)
#undef NOVA_X
    default: return false;
    }
}

template bool cols_group<NOVA_PART>(int, const Columns &, bool, double2 *, const double2 *, cudaStream_t);
#else
namespace {

void cols_any(int L, const Columns &C, bool inv, void *spec, const double *tw, cudaStream_t st)
{
    double2 *s = (double2 *)spec;
    const double2 *w = reinterpret_cast<const double2 *>(tw);
    (void)(cols_group<0>(L, C, inv, s, w, st) || cols_group<1>(L, C, inv, s, w, st) ||
           cols_group<2>(L, C, inv, s, w, st) || cols_group<3>(L, C, inv, s, w, st) ||
           cols_group<4>(L, C, inv, s, w, st) || cols_group<5>(L, C, inv, s, w, st));
}

}  // namespace

bool spec_cols_fit(int L) { return fft_length(L); }

void launch_cols_j(int n0, int ny, int nzh, bool inv, void *spec, const double *twL, cudaStream_t st)
{
    cols_any(ny, Columns{nzh, (long long)ny * nzh, (long long)n0 * nzh, nzh}, inv, spec, twL, st);
}

void launch_cols_i(int n0, long long per_plane, bool inv, void *spec, const double *twL, cudaStream_t st)
{
    cols_any(n0, Columns{per_plane, 0, per_plane, (int)per_plane}, inv, spec, twL, st);
}
#endif

}  // namespace nova
