// The explicit operators ex:: (src/ex) as drop-in calls: one sweep each.
//
// Bound by HBM at large sizes and by L1 wavefronts in between: a derivative
// along j or k reads its 2H neighbours through L1, one along i costs one load
// per node (the register queue of nova_dmarch.cuh).  Before this the kernels
// took one thread per node, recomputed (i, j, k) and each neighbour's wrap by
// integer divisions and read the i neighbours from L2.
//
// Components whose outputs are independent (grad of a vector, laplacian, div
// of a tensor) are separate blocks (grid.y), so that small meshes still fill
// the device; the i range is cut into chunks by march_chunk.
#include "nova_dmarch.cuh"
#include "nova_ops.cuh"
#include "nova_tile.cuh"

namespace nova {

namespace {

struct OpArgs {
    Geo g;
    Walls<double> wa, wb;
    Coef<double> co;
    const double *ia, *corr2, *a, *b;
    double nu, *out;
    int ngrp, ichunk;  // component groups in grid.y, planes per chunk
    int symm;
};

// sum_l w[l] (v(l + 1) - v(-l - 1))
template <int H, class V> __device__ __forceinline__ double cd(const V &v, const double *w)
{
    double r = 0.0;
#pragma unroll
    for (int l = 0; l < H; l++) r = fma(w[l], v(l + 1) - v(-l - 1), r);
    return r;
}

// the stencil of ex::grad(Field<vector>), c_l/(l+1)/delta (f(+l) - f(-1-l)) (src/ex/grad/grad.cpp:82-94), w = 2 a
template <int H, class V> __device__ __forceinline__ double q1(const V &v, const double *w)
{
    double r = 0.0;
#pragma unroll
    for (int l = 0; l < H; l++) r = fma(w[l], v(l) - v(-1 - l), r);
    return r;
}

// OP: an OpKind; NF: components of f that a thread takes (OP_DIV_VF), else 1
template <int OP, int H, int NF, bool WALLS>
__global__ void __launch_bounds__(kThreads, (OP == OP_DIV_VF || H == 4) ? 2 : 3) k_ex(const __grid_constant__ OpArgs A)
{
    const Geo &g = A.g;
    const int ktiles = (g.N2 + kTK - 1) / kTK;
    const int k = (blockIdx.x % ktiles) * kTK + threadIdx.x, j = (blockIdx.x / ktiles) * kTJ + threadIdx.y;
    if (k >= g.N2 || j >= g.N1) return;
    const int grp = blockIdx.y % A.ngrp, ib = (blockIdx.y / A.ngrp) * A.ichunk, ie = min(ib + A.ichunk, g.N0);
    const Nbr<H, WALLS> nb(g, j, k);
    const long long N3 = g.N3, col = (long long)j * g.N2 + k;
    const double *a = A.a + col, *b = A.b + col;
    double *out = A.out + col;
    const double iak = A.ia[k];
    double ax[H], ay[H], az[H];
#pragma unroll
    for (int l = 0; l < H; l++) {
        ax[l] = A.co.a[0][l];
        ay[l] = A.co.a[1][l];
        az[l] = A.co.a[2][l] * iak;
    }

    if constexpr (OP == OP_GRAD_S) {
        const double *const p[1] = {a};
        dmarch<H>(g, p, ib, ie, [&](long long o, const auto &q) {
            out[o] = cd<H>([&](int s) { return q[0][H + s]; }, ax);
            out[N3 + o] = cd<H>([&](int s) { return nb.y(a + o, s, A.wa, 0); }, ay);
            out[2 * N3 + o] = cd<H>([&](int s) { return nb.z(a + o, s); }, az);
        });
    } else if constexpr (OP == OP_GRAD_V) {
        const double *f = a + grp * N3;
        double *r = out + 3 * grp * N3;
        double wz[H];
#pragma unroll
        for (int l = 0; l < H; l++) {
            ax[l] *= 2.0;
            ay[l] *= 2.0;
            wz[l] = 2.0 * A.co.a[2][l] * iak;
        }
        const double *const p[1] = {f};
        dmarch<H>(g, p, ib, ie, [&](long long o, const auto &q) {
            r[o] = q1<H>([&](int s) { return q[0][H + s]; }, ax);
            r[N3 + o] = q1<H>([&](int s) { return s ? nb.y(f + o, s, A.wa, grp) : q[0][H]; }, ay);
            r[2 * N3 + o] = q1<H>([&](int s) { return s ? nb.z(f + o, s) : q[0][H]; }, wz);
        });
    } else if constexpr (OP == OP_CURL) {
        // antisymmetric part of ex::grad(vector) (src/ex/curl/curl.cpp:44-50)
        double wz[H];
#pragma unroll
        for (int l = 0; l < H; l++) {
            ax[l] *= 2.0;
            ay[l] *= 2.0;
            wz[l] = 2.0 * A.co.a[2][l] * iak;
        }
        const double *u = a, *v = a + N3, *w = a + 2 * N3;
        const double *const p[2] = {v, w};
        dmarch<H>(g, p, ib, ie, [&](long long o, const auto &q) {
            const double wy = q1<H>([&](int s) { return s ? nb.y(w + o, s, A.wa, 2) : q[1][H]; }, ay);
            const double vz = q1<H>([&](int s) { return s ? nb.z(v + o, s) : q[0][H]; }, wz);
            const double uz = q1<H>([&](int s) { return nb.z(u + o, s); }, wz);
            const double wx = q1<H>([&](int s) { return q[1][H + s]; }, ax);
            const double vx = q1<H>([&](int s) { return q[0][H + s]; }, ax);
            const double uy = q1<H>([&](int s) { return nb.y(u + o, s, A.wa, 0); }, ay);
            out[o] = wy - vz;
            out[N3 + o] = uz - wx;
            out[2 * N3 + o] = vx - uy;
        });
    } else if constexpr (OP == OP_DIV_V) {
        const double *const p[1] = {a};
        dmarch<H>(g, p, ib, ie, [&](long long o, const auto &q) {
            const double dx = cd<H>([&](int s) { return q[0][H + s]; }, ax);
            const double dy = cd<H>([&](int s) { return nb.y(a + N3 + o, s, A.wa, 1); }, ay);
            const double dz = cd<H>([&](int s) { return nb.z(a + 2 * N3 + o, s); }, az);
            out[o] = dx + dy + dz;
        });
    } else if constexpr (OP == OP_DIV_VF) {
        // skew div(V, f) = 1/2 [ f div V + sum_d D_d(V_d f) + V_d D_d f ] (src/ex/div/div.hxx:84-172)
        const int c0 = grp * NF;
        const double *f = b + c0 * N3;
        const double *p[1 + NF];
        p[0] = a;
#pragma unroll
        for (int c = 0; c < NF; c++) p[1 + c] = f + c * N3;
        dmarch<H, 1 + NF>(g, p, ib, ie, [&](long long o, const auto &q) {
            double acc[NF], dv = 0.0;
#pragma unroll
            for (int c = 0; c < NF; c++) acc[c] = 0.0;
#pragma unroll
            for (int d = 0; d < 3; d++) {
                const double *w = d == 0 ? ax : (d == 1 ? ay : az);
                auto V = [&](int s) {
                    return d == 0 ? q[0][H + s] : (d == 1 ? nb.y(a + N3 + o, s, A.wa, 1) : nb.z(a + 2 * N3 + o, s));
                };
                double vp[H], vm[H], dd = 0.0;
#pragma unroll
                for (int l = 0; l < H; l++) {
                    vp[l] = V(l + 1);
                    vm[l] = V(-l - 1);
                    dd = fma(w[l], vp[l] - vm[l], dd);
                }
                dv += dd;
                const double v0 = d == 0 ? q[0][H] : a[d * N3 + o];
#pragma unroll
                for (int c = 0; c < NF; c++) {
                    double dq = 0.0, df = 0.0;
#pragma unroll
                    for (int l = 0; l < H; l++) {
                        const double fp = d == 0 ? q[1 + c][H + l + 1]
                                                 : (d == 1 ? nb.y(p[1 + c] + o, l + 1, A.wb, c0 + c)
                                                           : nb.z(p[1 + c] + o, l + 1));
                        const double fm = d == 0 ? q[1 + c][H - l - 1]
                                                 : (d == 1 ? nb.y(p[1 + c] + o, -l - 1, A.wb, c0 + c)
                                                           : nb.z(p[1 + c] + o, -l - 1));
                        dq = fma(w[l], vp[l] * fp - vm[l] * fm, dq);
                        df = fma(w[l], fp - fm, df);
                    }
                    acc[c] += fma(v0, df, dq);
                }
            }
#pragma unroll
            for (int c = 0; c < NF; c++) out[(c0 + c) * N3 + o] = 0.5 * fma(q[1 + c][H], dv, acc[c]);
        });
    } else if constexpr (OP == OP_LAP) {
        // laplacian(nu, f) with the stretched-z term (src/ex/laplacian/laplacian.hxx:130-191)
        const double *f = a + grp * N3;
        const double i2 = iak * iak, cr = A.corr2[k];
        double bz[H];
#pragma unroll
        for (int l = 0; l < H; l++) bz[l] = A.co.b[2][l] * i2;
        const double *const p[1] = {f};
        dmarch<H>(g, p, ib, ie, [&](long long o, const auto &q) {
            const double f0 = q[0][H];
            double r = 0.0, sx = 0.0, sy = 0.0, sz = 0.0, dz = 0.0;
#pragma unroll
            for (int l = 0; l < H; l++) {
                sx = fma(A.co.b[0][l], q[0][H + l + 1] + q[0][H - l - 1], sx);
                sy = fma(A.co.b[1][l], nb.y(f + o, l + 1, A.wa, grp) + nb.y(f + o, -l - 1, A.wa, grp), sy);
                const double zp = nb.z(f + o, l + 1), zm = nb.z(f + o, -l - 1);
                sz = fma(bz[l], zp + zm, sz);
                dz = fma(az[l], zp - zm, dz);
            }
            r += fma(-A.co.b2[0], f0, sx);
            r += fma(-A.co.b2[1], f0, sy);
            r += fma(-A.co.b2[2] * i2, f0, sz);
            out[grp * N3 + o] = A.nu * fma(-cr, dz, r);
        });
    } else if constexpr (OP == OP_DIV_T) {
        // div(tensor) and div(symmTensor; xx xy xz yy yz zz) (src/ex/div/div.hxx:222-285): out_c =
        // sum_d D_d T[3c + d], without the z metric, as in the reference
        const int S[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
        int t[3];
#pragma unroll
        for (int d = 0; d < 3; d++) t[d] = A.symm ? S[3 * grp + d] : 3 * grp + d;
        const double *f0 = a + t[0] * N3, *f1 = a + t[1] * N3, *f2 = a + t[2] * N3;
        const double *const p[1] = {f0};
        dmarch<H>(g, p, ib, ie, [&](long long o, const auto &q) {
            double r = cd<H>([&](int s) { return q[0][H + s]; }, ax);
            r += cd<H>([&](int s) { return nb.y(f1 + o, s, A.wa, t[1]); }, ay);
            r += cd<H>([&](int s) { return nb.z(f2 + o, s); }, A.co.a[2]);
            out[grp * N3 + o] = r;
        });
    } else if constexpr (OP == OP_DIV_ST) {
        // div(scalar s, tensor T) (src/ex/div/div.hxx:173-207): sum_d D_d (s T[3c + d])
        const double *f0 = b + 3 * grp * N3, *f1 = f0 + N3, *f2 = f1 + N3;
        const double *const p[2] = {a, f0};
        dmarch<H>(g, p, ib, ie, [&](long long o, const auto &q) {
            double r = cd<H>([&](int s) { return q[0][H + s] * q[1][H + s]; }, ax);
            r += cd<H>([&](int s) { return nb.y(a + o, s, A.wa, 0) * nb.y(f1 + o, s, A.wb, 3 * grp + 1); }, ay);
            r += cd<H>([&](int s) { return nb.z(a + o, s) * nb.z(f2 + o, s); }, A.co.a[2]);
            out[grp * N3 + o] = r;
        });
    } else {
        // laplacian(Field<scalar> nu, Field<T>) (src/ex/laplacian/laplacian.hxx:64-127): the + neighbour at
        // 1+l weighted by nu at offset l, the - neighbour at -1-l by nu at -1-l, both against the centre;
        // z terms over dzdxi^2 and the stretched-z term -nu(0) D_z f d2zdxi2/dzdxi^3
        const double *f = b + grp * N3;
        const double i2 = iak * iak, cr = A.corr2[k];
        const double *const p[2] = {a, f};
        dmarch<H>(g, p, ib, ie, [&](long long o, const auto &q) {
            const double n0 = q[0][H], f0 = q[1][H];
            double r = 0.0, dz = 0.0;
#pragma unroll
            for (int d = 0; d < 3; d++) {
                const double m = d == 2 ? i2 : 1.0;
#pragma unroll
                for (int l = 0; l < H; l++) {
                    auto NU = [&](int s) {
                        return s == 0 ? n0 : (d == 0 ? q[0][H + s] : (d == 1 ? nb.y(a + o, s, A.wa, 0) : nb.z(a + o, s)));
                    };
                    auto F = [&](int s) {
                        return d == 0 ? q[1][H + s] : (d == 1 ? nb.y(f + o, s, A.wb, grp) : nb.z(f + o, s));
                    };
                    const double fp = F(l + 1), fm = F(-l - 1);
                    r = fma(A.co.b[d][l] * m, fma(NU(l), fp - f0, NU(-l - 1) * (fm - f0)), r);
                    if (d == 2) dz = fma(az[l], fp - fm, dz);
                }
            }
            out[grp * N3 + o] = fma(-n0 * cr, dz, r);
        });
    }
}

template <int OP, int H, int NF> void launch_h(OpArgs &A, cudaStream_t st)
{
    constexpr int bps = (OP == OP_DIV_VF || H == 4) ? 2 : 3;
    const Geo &g = A.g;
    const long long tiles = (long long)((g.N2 + kTK - 1) / kTK) * ((g.N1 + kTJ - 1) / kTJ);
    A.ichunk = march_chunk(g.N0, tiles * A.ngrp, bps, 2.0);
    const dim3 grid((unsigned)tiles, (unsigned)(A.ngrp * ((g.N0 + A.ichunk - 1) / A.ichunk)));
    if (g.wallY)
        k_ex<OP, H, NF, true><<<grid, dim3(kTK, kTJ), 0, st>>>(A);
    else
        k_ex<OP, H, NF, false><<<grid, dim3(kTK, kTJ), 0, st>>>(A);
}

template <int OP, int NF = 1> void launch_nf(int h, OpArgs &A, cudaStream_t st)
{
    switch (h) {
    case 1: launch_h<OP, 1, NF>(A, st); break;
    case 2: launch_h<OP, 2, NF>(A, st); break;
    case 3: launch_h<OP, 3, NF>(A, st); break;
    default: launch_h<OP, 4, NF>(A, st); break;
    }
}

}  // namespace

void launch_op(int op, int h, const Geo &g, const Walls<double> &wa, const Walls<double> &wb, const Coef<double> &co,
               const double *ia, const double *corr2, const double *a, const double *b, int nc, double nu, double *out,
               cudaStream_t st)
{
    OpArgs A{};
    A.g = g;
    A.wa = wa;
    A.wb = wb;
    A.co = co;
    A.ia = ia;
    A.corr2 = corr2;
    A.a = a;
    A.b = b ? b : a;
    A.nu = nu;
    A.out = out;
    A.ngrp = 1;
    switch (op) {
    case OP_GRAD_S: launch_nf<OP_GRAD_S>(h, A, st); break;
    case OP_DIV_V: launch_nf<OP_DIV_V>(h, A, st); break;
    case OP_CURL: launch_nf<OP_CURL>(h, A, st); break;
    case OP_GRAD_V:
        A.ngrp = 3;
        launch_nf<OP_GRAD_V>(h, A, st);
        break;
    case OP_DIV_VF:
        // three components of f per thread share V's loads (72 loads a node against 108)
        A.ngrp = nc % 3 ? nc : nc / 3;
        if (nc % 3)
            launch_nf<OP_DIV_VF, 1>(h, A, st);
        else
            launch_nf<OP_DIV_VF, 3>(h, A, st);
        break;
    case OP_DIV_T:
        A.ngrp = 3;
        A.symm = nc == 6;
        launch_nf<OP_DIV_T>(h, A, st);
        break;
    case OP_DIV_ST:
        A.ngrp = 3;
        launch_nf<OP_DIV_ST>(h, A, st);
        break;
    case OP_LAP_F:
        A.ngrp = nc;
        launch_nf<OP_LAP_F>(h, A, st);
        break;
    default:
        A.ngrp = nc;
        launch_nf<OP_LAP>(h, A, st);
        break;
    }
}

}  // namespace nova
