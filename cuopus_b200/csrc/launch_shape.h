// Rules that choose lanes per chain and warps per SM (host only).
#pragma once
#include <stddef.h>

namespace cuo_host {

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
