// The i direction of the periodic spectral Poisson solve, fused with the
// spectral scale (src/poisson/poisson.cpp:223-265):
//
//   rhs^ = FFT_i FFT_j FFT_k rhs,  rhs^ = -rhs^ / k'^2 / (N0 N1 N2)  (0 where k'^2 < 1e-16),
//   p = IFFT_k IFFT_j IFFT_i rhs^
//
// The (j, k) planes are transformed before and after (nova_spec_row.cu and
// nova_spec_col.cu, or cuFFT's batched 2-D D2Z and Z2D); this kernel does
// FFT_i, the scale and IFFT_i of every (j, kz) column of the half spectrum
// [i][j][kz] in one pass over HBM, where a 3-D cuFFT plan needs an i pass on
// either side and the scale a pass of its own.
//
// Length N0 = R1 R2 (nova_spec.cuh).  A block owns kSpecCols consecutive
// (j, kz) columns; a thread loads its values straight from HBM, runs the
// forward steps, the scale and the inverse steps with the indices' roles
// exchanged.  The twiddles W_N^m are a host-computed table; the scale is
// k_scale's up to the rounding of one reciprocal (within an ulp or two of its
// two divisions).
//
// N0 = 256 with N2 % 16 == 0 and N1 % 8 == 0 runs k_pois_tma instead: the
// same arithmetic on tiles of 8 columns, fed by bulk tensor loads into a
// double-buffered shared-memory tile (the next tile lands while the block
// transforms the current one), in a persistent grid: 70 us at 256^3, k_pois_i 96
// us, byte floor 41 us (k_pois_i loads, computes and stores in turn, so with two
// blocks per SM the memory pipe idles while both compute).
#include "nova_fft.cuh"
#include "nova_internal.cuh"
#include "nova_ops.cuh"
#include "nova_spec.cuh"
#include "nova_tma.cuh"

#include <algorithm>
#include <cstring>

namespace nova {

// N0 of group G: false where N0 is none of its lengths
template <int G>
bool pois_group(const Geo &g, int ny, void *spec, const double *twN, const double *kx2, const double *ky2,
                const double *kz2, double invN3, cudaStream_t st);

#ifdef NOVA_FFT_GROUP
namespace {

template <int R1, int R2>
__global__ void __launch_bounds__(column_threads<R1, R2>(), column_blocks<R1, R2>())
    k_pois_i(int nzh, long long ncol, double2 *__restrict__ spec, const double2 *__restrict__ twN,
             const double *__restrict__ kx2, const double *__restrict__ ky2, const double *__restrict__ kz2,
             double invN3)
{
    constexpr int N = R1 * R2, T = Line<R1, R2>::T, U = Line<R1, R2>::U;
    extern __shared__ __align__(16) unsigned char smraw[];
    double2 *tw = reinterpret_cast<double2 *>(smraw);  // W_N^m, m = 0..N-1
    double2 *S = tw + N;                               // transpose buffer [R1][R2][kSpecCols]
    const int tid = threadIdx.x;
    const int col = tid % kSpecCols, t = tid / kSpecCols;
    // column j nzh + kz in 32 bits (2^31 columns of 16 or more nodes exceed any
    // memory): the two 64-bit divisions cost 2 us at 256 x 256 x 250
    const unsigned c = blockIdx.x * kSpecCols + col;
    const bool valid = c < ncol;
    double2 *p = spec + (valid ? c : 0);  // element i at p[i ncol]
    // one address and two strides (as products per element the addresses spilled: 98
    // -> 89 us at 256 x 250 x 256, 240 x 250 x 260 91 -> 80, 75 x 77 x 79 8.1 -> 8.3)
    p += t * ncol;
    const long long step = R2 * ncol, ustep = T * ncol;
    double2 v[U][R1], w[R2];
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
        for (int n1 = 0; n1 < R1; n1++) v[u][n1] = valid ? p[n1 * step + u * ustep] : make_double2(0.0, 0.0);
    for (int m = tid; m < N; m += column_threads<R1, R2>()) tw[m] = twN[m];
    __syncthreads();
    column_fft<R1, R2, false>(v, w, S, tw, t, col);
    // S is rewritten below: for R1 = R2 every thread holds its values by now, and the
    // barrier here keeps the scale's operands out of the registers of the forward
    // step (256 x 250 x 256 88.6 -> 83.9 us, 64 x 64 x 62 5.1 -> 4.9); else it waits for
    // threads without a second step (240 x 250 x 260 79.8 us, here 104)
    if (R1 == R2) __syncthreads();
    // scale: -1 / k'^2 / (N0 N1 N2), 0 where k'^2 < 1e-16 (k'^2 summed in
    // k_scale's order; one reciprocal per element instead of two divisions)
    if (T == R1 || t < R1) {
        const double kyz = ky2[valid ? c / (unsigned)nzh : 0u], kzz = kz2[valid ? c % (unsigned)nzh : 0u];
#pragma unroll
        for (int k2 = 0; k2 < R2; k2++) {
            const double k2v = (kx2[t + R1 * k2] + kyz) + kzz;
            const double f = k2v < 1.0e-16 ? 0.0 : -invN3 * recip(k2v);
            w[k2] = make_double2(w[k2].x * f, w[k2].y * f);
        }
        // inverse, step 1 (thread = k1 = t): DFT over k2, twiddle W_N^-(n2 t)
        dft<R2, N, true>(w, tw);
    }
    if (R1 != R2) __syncthreads();
    if (T == R1 || t < R1)
#pragma unroll
        for (int n2 = 0; n2 < R2; n2++)
            S[(t * R2 + n2) * kSpecCols + col] = n2 == 0 ? w[0] : cmul(w[n2], conj2(tw[t * n2]));
    __syncthreads();
    // inverse, step 2 (thread = n2): DFT over k1 -> x[n2 + R2 n1]
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int n2 = t + T * u;
#pragma unroll
        for (int k1 = 0; k1 < R1; k1++) v[u][k1] = S[(k1 * R2 + n2) * kSpecCols + col];
        dft<R1, N, true>(v[u], tw);
        if (valid)
#pragma unroll
            for (int n1 = 0; n1 < R1; n1++) p[n1 * step + u * ustep] = v[u][n1];
    }
}

template <int R1, int R2>
void launch_r(const Geo &g, int ny, void *spec, const double *twN, const double *kx2, const double *ky2,
              const double *kz2, double invN3, cudaStream_t st)
{
    constexpr size_t smem = column_smem<R1, R2>();
    NOVA_SPEC_SMEM((k_pois_i<R1, R2>), smem);
    const int nzh = g.N2 / 2 + 1;
    const long long ncol = (long long)ny * nzh;
    k_pois_i<R1, R2><<<(unsigned)((ncol + kSpecCols - 1) / kSpecCols), column_threads<R1, R2>(), smem, st>>>(
        nzh, ncol, (double2 *)spec, (const double2 *)twN, kx2, ky2, kz2, invN3);
}

}  // namespace

template <int G>
bool pois_group(const Geo &g, int ny, void *spec, const double *twN, const double *kx2, const double *ky2,
                const double *kz2, double invN3, cudaStream_t st)
{
    switch (g.N0) {
#define NOVA_X(l, r1, r2) \
    case l: launch_r<r1, r2>(g, ny, spec, twN, kx2, ky2, kz2, invN3, st); return true;
        NOVA_FFT_GROUP(NOVA_X)
#undef NOVA_X
    default: return false;
    }
}

template bool pois_group<NOVA_PART>(const Geo &, int, void *, const double *, const double *, const double *,
                                    const double *, double, cudaStream_t);
#else
namespace {

// ---- N0 = 256 on a TMA-fed, double-buffered tile ----
constexpr int kTR = 16, kTN = kTR * kTR;  // 256 = 16 x 16
constexpr int kTC = 8;                    // columns per tile
constexpr int kTThreads = kTC * kTR;      // thread (col, t): col = tid % 8, t = tid / 8
constexpr uint32_t kTileBytes = kTN * kTC * sizeof(double2);  // 32 KB
constexpr size_t kTSmem =
    2 * (size_t)kTileBytes + kTN * sizeof(double2) + kTN * sizeof(double) + 2 * sizeof(unsigned long long);

// the half spectrum as FP64 [i][j][2 nzh]: `col` boxes 16 x 1 x 256 (8 kz of
// one j, every i), `rem` boxes 2 x 8 x 256 (the last kz of 8 consecutive j);
// both land as [i][8 columns] complex
struct PoisMaps {
    CUtensorMap col, rem;
};

// Tasks t < nmain: j = t / nch, kz = 8 (t % nch) + col (nch = (nzh - 1) / 8);
// tasks t >= nmain: j = 8 (t - nmain) + col, kz = nzh - 1.  Block b takes
// tasks b, b + gridDim.x, ...; the load of the next one is issued when the
// current one starts.  Arithmetic, order and twiddles are k_pois_i<16, 16>'s.
__global__ void __launch_bounds__(kTThreads, 3)
    k_pois_tma(int ny, int nzh, double2 *__restrict__ spec, const double2 *__restrict__ twN,
               const double *__restrict__ kx2, const double *__restrict__ ky2, const double *__restrict__ kz2,
               double invN3, const __grid_constant__ PoisMaps maps, int nmain, int ntask, int *err)
{
    extern __shared__ __align__(128) unsigned char smtile[];
    double2 *tiles = reinterpret_cast<double2 *>(smtile);  // [2][kTN][kTC]
    double2 *tw = tiles + 2 * kTN * kTC;                   // W_256^m
    double *kx2s = reinterpret_cast<double *>(tw + kTN);   // kx'^2 (the scale's i wavenumbers)
    const uint32_t bar0 = smem_addr(kx2s + kTN);           // one mbarrier per tile
    const int tid = threadIdx.x, col = tid % kTC, t = tid / kTC;
    const int nch = (nzh - 1) / kTC;
    for (int m = tid; m < kTN; m += kTThreads) {
        tw[m] = twN[m];
        kx2s[m] = kx2[m];
    }
    if (tid == 0) {
        mbar_init(bar0, 1);
        mbar_init(bar0 + 8, 1);
        mbar_init_fence();
    }
    __syncthreads();
    auto issue = [&](int task, int b) {  // thread 0
        const uint32_t dst = smem_addr(tiles + b * kTN * kTC), bar = bar0 + 8u * b;
        mbar_expect_tx(bar, kTileBytes);
        if (task < nmain)
            tma_load_3d(dst, &maps.col, bar, 2 * kTC * (task % nch), task / nch, 0);
        else
            tma_load_3d(dst, &maps.rem, bar, 2 * (nzh - 1), kTC * (task - nmain), 0);
    };
    const long long rowstride = (long long)ny * nzh;
    int task = blockIdx.x;
    if (tid == 0 && task < ntask) issue(task, 0);
    for (int n = 0; task < ntask; n++, task += gridDim.x) {
        const int b = n & 1;
        const bool more = task + (int)gridDim.x < ntask;
        if (tid == 0 && more) issue(task + gridDim.x, b ^ 1);  // that tile was released at the end of step n - 1
        if (!__syncthreads_and(mbar_wait(bar0 + 8u * b, (n >> 1) & 1, err))) {
            // timed out: the loads still in flight land before the block leaves
            if (tid == 0) {
                mbar_wait(bar0 + 8u * b, (n >> 1) & 1, err, true);
                if (more) mbar_wait(bar0 + 8u * (b ^ 1), ((n + 1) >> 1) & 1, err, true);
            }
            return;
        }
        double2 *S = tiles + b * kTN * kTC;
        int jc, kzc;
        if (task < nmain) {
            jc = task / nch;
            kzc = kTC * (task % nch) + col;
        } else {
            jc = kTC * (task - nmain) + col;
            kzc = nzh - 1;
        }
        const double kyz = ky2[jc], kzz = kz2[kzc];  // issued early: used after the forward DFT
        double2 v[kTR];
#pragma unroll
        for (int n1 = 0; n1 < kTR; n1++) v[n1] = S[(t + kTR * n1) * kTC + col];
        __syncthreads();  // the tile is rewritten below
        // forward, step 1 (thread = n2 = t): DFT over n1, twiddle W_N^(t k1)
        dft<kTR, kTN, false>(v, tw);
#pragma unroll
        for (int k1 = 0; k1 < kTR; k1++) S[(k1 * kTR + t) * kTC + col] = k1 == 0 ? v[0] : cmul(v[k1], tw[(t * k1) % kTN]);
        __syncthreads();
        // forward, step 2 (thread = k1 = t): DFT over n2 -> X[t + R k2]
#pragma unroll
        for (int n2 = 0; n2 < kTR; n2++) v[n2] = S[(t * kTR + n2) * kTC + col];
        __syncthreads();
        dft<kTR, kTN, false>(v, tw);
#pragma unroll
        for (int k2 = 0; k2 < kTR; k2++) {
            const double k2v = (kx2s[t + kTR * k2] + kyz) + kzz;
            const double f = k2v < 1.0e-16 ? 0.0 : -invN3 * recip(k2v);
            v[k2] = make_double2(v[k2].x * f, v[k2].y * f);
        }
        // inverse, step 1 (thread = k1 = t): DFT over k2, twiddle W_N^-(n1 t)
        dft<kTR, kTN, true>(v, tw);
#pragma unroll
        for (int n1 = 0; n1 < kTR; n1++)
            S[(n1 * kTR + t) * kTC + col] = n1 == 0 ? v[0] : cmul(v[n1], conj2(tw[(t * n1) % kTN]));
        __syncthreads();
        // inverse, step 2 (thread = n1 = t): DFT over k1 -> x[t + R n2]
#pragma unroll
        for (int k1 = 0; k1 < kTR; k1++) v[k1] = S[(t * kTR + k1) * kTC + col];
        dft<kTR, kTN, true>(v, tw);
        double2 *dst = spec + (long long)t * rowstride + (long long)jc * nzh + kzc;
#pragma unroll
        for (int n2 = 0; n2 < kTR; n2++) dst[(long long)n2 * kTR * rowstride] = v[n2];
        // the transposes wrote the tile through the generic proxy; order those
        // writes before the bulk copy (async proxy) that refills it
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();  // the tile is free for the load of step n + 2
    }
}

bool encode_spec(CUtensorMap *m, const void *spec, int n0, int ny, int nzh, unsigned bx, unsigned by)
{
    PFN_cuTensorMapEncodeTiled_v12000 fn = tma_encode_tiled();
    if (!fn) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)2 * nzh, (cuuint64_t)ny, (cuuint64_t)n0};
    const cuuint64_t strides[2] = {(cuuint64_t)2 * nzh * sizeof(double), (cuuint64_t)2 * nzh * ny * sizeof(double)};
    const cuuint32_t box[3] = {bx, by, (cuuint32_t)n0}, estr[3] = {1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<void *>(spec), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool pois_tma_fits(const Geo &g, int ny)
{
    const int nzh = g.N2 / 2 + 1;
    return g.N0 == kTN && (nzh - 1) % kTC == 0 && ny % kTC == 0;
}

bool launch_pois_tma(const Geo &g, int ny, void *spec, const double *twN, const double *kx2, const double *ky2,
                     const double *kz2, double invN3, int *err, cudaStream_t st)
{
    const int nzh = g.N2 / 2 + 1;
    PoisMaps maps;
    std::memset(&maps, 0, sizeof maps);
    if (!encode_spec(&maps.col, spec, g.N0, ny, nzh, 2 * kTC, 1) || !encode_spec(&maps.rem, spec, g.N0, ny, nzh, 2, kTC))
        return false;
    static int nsm = 0;
    static bool attr = false;
    if (!attr) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        cudaFuncSetAttribute(k_pois_tma, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTSmem);
        attr = true;
    }
    const int nmain = ny * ((nzh - 1) / kTC), ntask = nmain + ny / kTC;
    const int grid = std::min(ntask, 3 * std::max(nsm, 1));
    k_pois_tma<<<grid, kTThreads, kTSmem, st>>>(ny, nzh, (double2 *)spec, (const double2 *)twN, kx2, ky2, kz2, invN3,
                                                maps, nmain, ntask, err);
    return true;
}

}  // namespace

bool pois_i_fits(const Geo &g) { return fft_length(g.N0); }

void launch_pois_i(const Geo &g, int ny, void *spec, const double *twN, const double *kx2, const double *ky2,
                   const double *kz2, double invN3, int *err, cudaStream_t st)
{
    if (g.N0 == 256 && err && pois_tma_fits(g, ny) &&
        launch_pois_tma(g, ny, spec, twN, kx2, ky2, kz2, invN3, err, st))
        return;
    (void)(pois_group<0>(g, ny, spec, twN, kx2, ky2, kz2, invN3, st) ||
           pois_group<1>(g, ny, spec, twN, kx2, ky2, kz2, invN3, st) ||
           pois_group<2>(g, ny, spec, twN, kx2, ky2, kz2, invN3, st) ||
           pois_group<3>(g, ny, spec, twN, kx2, ky2, kz2, invN3, st) ||
           pois_group<4>(g, ny, spec, twN, kx2, ky2, kz2, invN3, st) ||
           pois_group<5>(g, ny, spec, twN, kx2, ky2, kz2, invN3, st));
}
#endif

}  // namespace nova
