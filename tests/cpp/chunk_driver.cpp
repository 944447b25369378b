// march_chunk (nova_chunk.h) against the rule spelled out over every count of
// chunks; prints the time of a call of either at argv[1] planes.
#include "nova_chunk.h"

#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <initializer_list>

static int every_count(int n0, long long tiles, int bps, double warm, double tail)
{
    int best = n0;
    double cost = 1e300;
    for (int n = 1; n <= n0 && n <= 4096; n++) {
        const int ch = (n0 + n - 1) / n;
        const long long blocks = tiles * ((n0 + ch - 1) / ch), wave = 148LL * bps, rest = blocks % wave;
        const double share = rest ? 0.5 + 0.5 * (double)((rest + 147) / 148) / bps : 0.0;
        const double c = (ch + warm) * ((double)(blocks / wave) + share + tail);
        if (c < cost) cost = c, best = ch;
    }
    return best;
}

template <class F> static double us(F f, int n0)
{
    const int calls = 400;
    volatile int sink = 0;
    double best = 1e300;
    for (int rep = 0; rep < 5; rep++) {
        const auto t = std::chrono::steady_clock::now();
        for (int q = 0; q < calls; q++) sink = sink + f(n0, 8 + q, 1, 2.5, 0.15);
        const std::chrono::duration<double, std::micro> d = std::chrono::steady_clock::now() - t;
        best = d.count() / calls < best ? d.count() / calls : best;
    }
    return best;
}

int main(int, char **argv)
{
    for (int n0 = 1; n0 < 700; n0 += n0 < 300 ? 1 : 37)
        for (long long tiles : {1, 2, 5, 16, 37, 128, 592, 4096})
            for (int bps = 1; bps <= 4; bps++)
                for (double tail : {0.15, 0.3, 0.45})
                    if (nova::march_chunk(n0, tiles, bps, 2.5, tail) != every_count(n0, tiles, bps, 2.5, tail)) {
                        std::printf("n0 %d tiles %lld bps %d tail %g\n", n0, tiles, bps, tail);
                        return 1;
                    }
    for (int n0 : {4095, 4096, 4097, 5000, 9001})
        for (long long tiles : {1, 4, 150})
            if (nova::march_chunk(n0, tiles, 2, 3.0, 0.15) != every_count(n0, tiles, 2, 3.0, 0.15)) return 1;
    const int n0 = std::atoi(argv[1]);
    std::printf("%g %g\n", us(nova::march_chunk, n0), us(every_count, n0));
    return 0;
}
