// Rules that choose lanes per chain and warps per SM (host only).
#pragma once
#include <stddef.h>

#include <algorithm>
#include <vector>

namespace cuo_host {

// Launch shape of a file batch: lanes per chain and warps per SM.  More lanes
// decode a chain faster, fewer lanes put more chains on the GPU, and more warps
// on an SM slow each other down, because each of them fetches its own part of a
// program larger than the SM's instruction caches.  Speeds are per group,
// relative to 32 lanes at 4 warps per SM, from files of 300 to 5400 one-second
// chains (ms at 32 lanes / 16 / 8):
//   speech, 300 chains 19 / 26 / 42, 1800 58 / 42 / 50, 5400 160 / 113 / 81;
//   mono and stereo mixed, 1085 chains 92 / 116 / 188 (105 at 5 warps per SM,
//   138 at 8), 2070 165 / 140 / 230, 3100 248 / 207 / 272;
//   voice, 600 chains 18 at 4 warps per SM (two rounds), 11.5 at 5;
//   at 8 lanes, speech of 7200 chains 106 at 8 warps per SM and 112 at 12, voice
//   of 5400 53 and 36 (two rounds at 8).
struct LaunchShape {
    int width, warps_per_sm;   // 0 warps: every resident group
    double speed;
};
const LaunchShape SHAPES[] = {{32, 4, 1.0}, {32, 5, 0.8}, {16, 4, 0.62}, {16, 6, 0.55}, {8, 8, 0.37}, {8, 0, 0.33}};

// The shape (of want_width lanes, when that is not 0) with the least estimate
// max(longest chain, total work / groups, what a group with a second chain has
// to do) / speed for chains of the given costs, the longest first; groups(shape)
// is how many decoder groups the GPU gives it.  The last term is taken at 0.7,
// since chains speed up as groups run dry.  Null when no shape has that width.
template <class Groups>
const LaunchShape *choose_shape(const std::vector<double> &cost, int want_width, Groups &&groups)
{
    double sum = 0.0, best = -1.0;
    for (double c : cost) sum += c;
    const LaunchShape *chosen = nullptr;
    for (const LaunchShape &s : SHAPES) {
        if (want_width && s.width != want_width) continue;
        const long long g = groups(s);
        double t = cost.empty() ? 0.0 : std::max(cost[0], sum / (double)g);
        if ((long long)cost.size() > g) t = std::max(t, 0.7 * (cost[g - 1] + cost[g]));
        t /= s.speed;
        if (best >= 0.0 && t >= best) continue;
        best = t;
        chosen = &s;
    }
    return chosen;
}

// Lanes per chain of a server wave, from the chains in flight with it (the
// wave's own and those of the waves still decoding).  A wave launches a group
// for every chain, with no limit of warps per SM: up to eight warps an SM at 32
// and 16 lanes, twelve at 8.  Wide groups decode a chain faster, narrow ones keep
// more chains on the GPU.  Milliseconds from the first submit to the last result
// of 30 s files sent together (mixed and stereo in turn; speech), by chains per
// SM, with every wave at 32 lanes, 16 and 8:
//     2    55   89  196
//     4    80  102  204;    30   33   45
//     6   108  112  193
//     7   117  113  203;    47   39   49
//    10   152  155  219;    66   50   55
//    16   208  225  234;    92   74   63
//    24   301  286  320;   123  114   94
//    36   454  394  455;   198  136  129
//    48   591  575  620;   237  202  170
// So 32 lanes up to six chains an SM.  Beyond that 16 lanes lose little on mixed
// files and win on speech.  From 16 on speech asks for 8 lanes and stereo for 16;
// the line at 24 lies between (8 lanes from 16 on: 365 and 95 ms at 24 chains an
// SM, now 308 and 114; 16 lanes throughout: 425 and 154 at 36, now 549 and 135).
inline int server_wave_width(size_t load, int sms, int narrow)
{
    return load <= 6 * (size_t)sms ? 32 : load <= 24 * (size_t)sms ? 16 : narrow;
}

} // namespace cuo_host
