// Direct march: a thread owns one (j, k) column of the grid and walks it along
// i.  The i stencil lives in a register queue (each plane loaded once, one
// plane ahead); the j and k neighbours are read from global memory at offsets
// that are computed once per thread, so that they hit L1 (the block's own rows
// passed through it as queue heads H planes earlier) or L2 (the rows beside
// the tile).  No shared memory and no barriers: every warp runs at its own
// pace and all loads of a plane are independent of one another.  Any mesh:
// periodic axes wrap in the offsets, y walls mirror (Walls<double>).
#pragma once

#include "nova_internal.cuh"

namespace nova {

// row and column offsets of the j and k neighbours of a thread's column
template <int H, bool WALLS> struct Nbr {
    int j, n1, rowb;  // rowb: bytes of a row (a plane may hold more than 2^31 nodes)
    int jo[2 * H + 1], ko[2 * H + 1];
    __device__ __forceinline__ Nbr(const Geo &g, int jj, int k) : j(jj), n1(g.N1), rowb(g.N2 * (int)sizeof(double))
    {
#pragma unroll
        for (int s = -H; s <= H; s++) {
            int jn = j + s;
            if (WALLS)
                jn = jn < 0 ? -jn : (jn >= n1 ? 2 * (n1 - 1) - jn : jn);
            else
                jn = wrapi(jn, n1);
            jo[H + s] = jn - j;
            ko[H + s] = wrapi(k + s, g.N2) - k;
        }
    }
    // f at offset s along j (component c of its wall BCs) and along k; f points at the column's current plane
    __device__ __forceinline__ double y(const double *f, int s, const Walls<double> &wl, int c) const
    {
        const double v = *reinterpret_cast<const double *>(reinterpret_cast<const char *>(f) + (long long)jo[H + s] * rowb);
        if constexpr (WALLS) {
            const int jn = j + s;
            if (jn < 0) return wall_ghost(wl, 0, c, -jn, v);
            if (jn >= n1) return wall_ghost(wl, 1, c, jn - (n1 - 1), v);
        }
        return v;
    }
    __device__ __forceinline__ double z(const double *f, int s) const { return f[ko[H + s]]; }
};

// Walks planes ib .. ie - 1.  p[c]: the queued components at node (0, j, k) of
// the thread's column.  body(off, q): off = i N12, the plane's offset from
// those pointers; q[c][H + s] the queued values at i + s.
template <int H, int NC, class Body>
__device__ __forceinline__ void dmarch(const Geo &g, const double *const (&p)[NC], int ib, int ie, Body &&body)
{
    double q[NC][2 * H + 1];
#pragma unroll
    for (int s = 0; s < 2 * H; s++) {
        const long long o = (long long)wrapi(ib - H + s, g.N0) * g.N12;
#pragma unroll
        for (int c = 0; c < NC; c++) q[c][s + 1] = p[c][o];
    }
    int lead = wrapi(ib + H, g.N0);
    double qn[NC];
#pragma unroll
    for (int c = 0; c < NC; c++) qn[c] = p[c][(long long)lead * g.N12];
    for (int i = ib; i < ie; i++) {
#pragma unroll
        for (int c = 0; c < NC; c++) {
#pragma unroll
            for (int s = 0; s < 2 * H; s++) q[c][s] = q[c][s + 1];
            q[c][2 * H] = qn[c];
        }
        if (i + 1 < ie) {  // the next head, in flight during this plane's arithmetic
            lead = lead + 1 == g.N0 ? 0 : lead + 1;
#pragma unroll
            for (int c = 0; c < NC; c++) qn[c] = p[c][(long long)lead * g.N12];
        }
        body((long long)i * g.N12, q);
    }
}

}  // namespace nova
