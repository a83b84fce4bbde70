// The probability tables of the symbols that a SILK frame decodes by the
// hundred (shell splits, pulse counts, NLSF residuals), as rows of four
// entries a word, padded with zeros: rdi_icdf_row (rangedec.cuh) reads four
// candidates with one load and stops at the row's end by itself.  Each block
// keeps a copy in shared memory (1.8 KB), filled when the kernel starts: a
// dependent load there takes 29 cycles, from the constant bank 51 and from L1
// 63, and every symbol waits for one.
#pragma once
#include "common.cuh"

namespace cuo {

struct HotTabs {
    uint32_t shell[4][17][5];   // level, pulses in the node (0 unused)
    uint32_t pulses[11][5];     // rate level; 9: after a count of 17; 10: after ten of those
    uint32_t rate[2][3];        // signalType >> 1
    uint32_t nlsf[2][8][3];     // NB / MB, WB; codebook selector
};

#ifdef __CUDACC__
static __shared__ HotTabs s_hot_tabs;
DFN const HotTabs &hot_tabs() { return s_hot_tabs; }
#endif

// Words of `row` from the n byte entries of t, zeros after them.
DFN void hot_row(uint32_t *row, int words, const uint8_t *t, int n)
{
    ROLLED for (int w = 0; w < words; w++) {
        uint32_t v = 0;
        ROLLED for (int k = 0; k < 4; k++)
            if (4 * w + k < n) v |= (uint32_t)t[4 * w + k] << (8 * k);
        row[w] = v;
    }
}

// Fill T: rows id, id + n, ... of all of them (the threads of a block).
DFN void hot_fill(HotTabs *T, int id, int n)
{
    ROLLED for (int q = id; q < 4 * 17 + 11 + 2 + 16; q += n) {
        int r = q;
        if (r < 4 * 17) {
            const int lvl = r / 17, p = r - 17 * lvl;
            const uint8_t *t = lvl == 3 ? T_silk_shell_code_table3
                             : lvl == 2 ? T_silk_shell_code_table2
                             : lvl == 1 ? T_silk_shell_code_table1 : T_silk_shell_code_table0;
            hot_row(T->shell[lvl][p], 5, p ? t + T_silk_shell_code_table_offsets[p] : t, p ? p + 1 : 0);
        } else if ((r -= 4 * 17) < 11) {
            const int skip = r == 10;
            hot_row(T->pulses[r], 5, &T_silk_pulses_per_block_iCDF[(r - skip) * 18 + skip], 18 - skip);
        } else if ((r -= 11) < 2) {
            hot_row(T->rate[r], 3, &T_silk_rate_levels_iCDF[r * 9], 9);
        } else {
            r -= 2;
            hot_row(T->nlsf[r >> 3][r & 7], 3, (r < 8 ? T_NLSF_NB_MB_ec_iCDF : T_NLSF_WB_ec_iCDF) + (r & 7) * 9, 9);
        }
    }
}

#ifndef __CUDACC__
struct HotTabsHost : HotTabs {
    HotTabsHost() { hot_fill(this, 0, 1); }
};
static const HotTabsHost g_hot_tabs;
DFN const HotTabs &hot_tabs() { return g_hot_tabs; }
#endif

} // namespace cuo
