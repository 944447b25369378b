// Line transforms of the spectral Poisson solve for lengths L = R1 R2 that two
// register DFTs cover (NOVA_FFT_LENGTHS): n = R2 n1 + n2, k = k1 + R1 k2,
//   X[k1 + R1 k2] = sum_n2 W_R2^(n2 k2) W_L^(n2 k1) sum_n1 x[R2 n1 + n2] W_R1^(n1 k1),
// T threads per line (T = R1 where R1 divides R2, else R2), each with R2/T
// DFTs of R1 points in the first step (loads of all of them in flight) and, on
// the first R1 threads, one DFT of R2 points in the second; one shared-memory
// transpose between the steps.
#pragma once

#include "nova_fft.cuh"
#include "nova_internal.cuh"
#include "nova_parts.h"

namespace nova {

// (L, R1, R2), R1 <= R2: the composites of the register DFTs that a mesh extent is
// likely to be; 81, 135 and 225 are left to cuFFT.  Along k L is N2 / 2, so that rows
// of 32 to 512 reals are covered; along i and j the extent itself, 16 to 256.
// In six groups: a part of nova_spec_row.cu, nova_spec_col.cu and nova_pois_i.cu each.
#define NOVA_FFT_G0(X) X(16, 4, 4) X(20, 4, 5) X(24, 4, 6) X(25, 5, 5) X(30, 5, 6)
#define NOVA_FFT_G1(X) X(32, 4, 8) X(36, 6, 6) X(40, 4, 10) X(45, 5, 9) X(48, 6, 8)
#define NOVA_FFT_G2(X) X(50, 5, 10) X(54, 6, 9) X(60, 6, 10) X(64, 8, 8) X(72, 6, 12)
#define NOVA_FFT_G3(X) X(75, 5, 15) X(80, 8, 10) X(90, 9, 10) X(96, 8, 12) X(100, 10, 10)
#define NOVA_FFT_G4(X) X(108, 9, 12) X(120, 10, 12) X(128, 8, 16) X(144, 12, 12) X(150, 10, 15)
#define NOVA_FFT_G5(X) X(160, 10, 16) X(180, 12, 15) X(192, 12, 16) X(240, 15, 16) X(256, 16, 16)
#define NOVA_FFT_LENGTHS(X) \
    NOVA_FFT_G0(X) NOVA_FFT_G1(X) NOVA_FFT_G2(X) NOVA_FFT_G3(X) NOVA_FFT_G4(X) NOVA_FFT_G5(X)

// the group of this part (the dispatch, part 6, has none)
#if NOVA_PART == 0
#define NOVA_FFT_GROUP NOVA_FFT_G0
#elif NOVA_PART == 1
#define NOVA_FFT_GROUP NOVA_FFT_G1
#elif NOVA_PART == 2
#define NOVA_FFT_GROUP NOVA_FFT_G2
#elif NOVA_PART == 3
#define NOVA_FFT_GROUP NOVA_FFT_G3
#elif NOVA_PART == 4
#define NOVA_FFT_GROUP NOVA_FFT_G4
#elif NOVA_PART == 5
#define NOVA_FFT_GROUP NOVA_FFT_G5
#endif

inline bool fft_length(int L)
{
    switch (L) {
#define NOVA_X(l, r1, r2) case l:
        NOVA_FFT_LENGTHS(NOVA_X)
#undef NOVA_X
        return true;
    default: return false;
    }
}

template <int R1, int R2> struct Line {
    static constexpr int L = R1 * R2;
    static constexpr int T = R2 % R1 == 0 ? R1 : R2;  // threads per line
    static constexpr int U = R2 / T;                  // R1-point DFTs per thread in step 1
};

// ---- columns: element n of column c at base(c) + n step ----
// Columns are numbered contiguously over (outer, inner) with `per` inner
// columns: base = (c / per) outer + c % per.
struct Columns {
    long long step, outer, total;  // elements (double2); number of columns
    int per;
};

// the two steps on the columns of a block: thread (col, t) of kCols columns;
// S is the transpose buffer [R1][R2][kCols].  v0 (step-1 order) -> v1
// (thread t < R1: element t + R1 k2 of the result in v1[k2])
constexpr int kSpecCols = 16;  // 16 columns x 16 B = 256 contiguous bytes per row

template <int R1, int R2, bool INV>
__device__ __forceinline__ void column_fft(double2 (&v0)[Line<R1, R2>::U][R1], double2 (&v1)[R2], double2 *S,
                                           const double2 *tw, int t, int col)
{
    constexpr int L = R1 * R2, T = Line<R1, R2>::T, U = Line<R1, R2>::U;
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int n2 = t + T * u;
        dft<R1, L, INV>(v0[u], tw);
#pragma unroll
        for (int k1 = 0; k1 < R1; k1++) {
            const double2 w = tw[n2 * k1];
            S[(k1 * R2 + n2) * kSpecCols + col] = k1 == 0 ? v0[u][0] : cmul(v0[u][k1], INV ? conj2(w) : w);
        }
    }
    __syncthreads();
    if (T == R1 || t < R1) {
#pragma unroll
        for (int n2 = 0; n2 < R2; n2++) v1[n2] = S[(t * R2 + n2) * kSpecCols + col];
        dft<R2, L, INV>(v1, tw);
    }
}

template <int R1, int R2> constexpr size_t column_smem() { return sizeof(double2) * R1 * R2 * (1 + kSpecCols); }
template <int R1, int R2> __host__ __device__ constexpr int column_threads() { return kSpecCols * Line<R1, R2>::T; }

// resident blocks per SM the column kernels ask for: registers for the values
// a thread holds (four each) and the DFTs' temporaries
template <int R1, int R2> __host__ __device__ constexpr int column_blocks()
{
    constexpr int held = Line<R1, R2>::U * R1 > R2 ? Line<R1, R2>::U * R1 : R2;
    constexpr int regs = held >= 16 ? 128 : (held >= 12 ? 104 : (held >= 10 ? 88 : 72));
    constexpr int b = 65536 / (regs * column_threads<R1, R2>());
    return b > 8 ? 8 : b;
}

inline __device__ long long column_base(const Columns &C, long long c)
{
    return (c / C.per) * C.outer + c % C.per;
}

// sets a kernel's dynamic shared memory limit once per call site
#define NOVA_SPEC_SMEM(kern, bytes)                                                                \
    do {                                                                                           \
        static bool done = false;                                                                  \
        if ((bytes) > 48 * 1024 && !done) {                                                        \
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(bytes)); \
            done = true;                                                                           \
        }                                                                                          \
    } while (0)

}  // namespace nova
