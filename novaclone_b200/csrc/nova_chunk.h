// Chunk length of the marching kernels.  Host code only.
#pragma once

namespace nova {

// i-chunk of a kernel whose blocks walk (j, k) tiles along i: `tiles` tiles,
// bps resident blocks per SM, `warm` the cost of a block's start (launch,
// queue fill) in planes.  The chunk of least estimated time: full waves of
// resident blocks, then the last one, in which a block that has its SM to
// itself takes half the time of one that shares it with bps - 1 others, and
// `tail`, the last block's lateness as a share of a block's time (walls: the
// tiles next to a wall take longer, and short chunks spread them).
// The rule before (halve the chunk from N0 to 16 until there are four waves)
// left small meshes on a few SMs.  FP64 stage at 64^3: 16 planes, 32 blocks,
// 23.7 us; 4 planes, 128 blocks, 10.0 us; divergence 12.9 -> 5.9 us (2
// planes).  At 128^3: FP64 stage 50 -> 46 us, MHD stage 99 -> 92 us.  At 256^3
// both rules are within 2%.
// Every launch asks, so only the distinct chunks are looked at (about 2 sqrt(n0) of
// the n0 counts, the same result): 64 planes 0.9 -> 0.3 us on the host, 256 4.6 -> 0.7,
// 4096 39 -> 2.1.
inline int march_chunk(int n0, long long tiles, int bps, double warm, double tail = 0.15)
{
    int best = n0;
    double cost = 1e300;
    for (int n = 1, ch; n <= n0 && n <= 4096; n = (n0 + ch - 2) / (ch - 1)) {  // the next count with a shorter chunk
        ch = (n0 + n - 1) / n;
        const long long blocks = tiles * ((n0 + ch - 1) / ch), wave = 148LL * bps, rest = blocks % wave;
        const double share = rest ? 0.5 + 0.5 * (double)((rest + 147) / 148) / bps : 0.0;
        const double c = (ch + warm) * ((double)(blocks / wave) + share + tail);
        if (c < cost) {
            cost = c;
            best = ch;
        }
        if (ch == 1) break;
    }
    return best;
}

}  // namespace nova
