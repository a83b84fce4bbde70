// CELT decoder (RFC 6716 section 4.3), fixed point, static 48 kHz / 960 mode.
//
// Restates libopus 1.5.2:
//   celt/celt_decoder.c   celt_decode_with_ec_dred, celt_decode_lost,
//                         prefilter_and_fold, celt_plc_pitch_search,
//                         tf_decode, celt_synthesis, deemphasis, reset
//   celt/quant_bands.c    unquant_coarse/fine_energy, unquant_energy_finalise
//   celt/rate.c           clt_compute_allocation, interp_bits2pulses
//   celt/rate.h           get_pulses, bits2pulses, pulses2bits
//   celt/bands.c          quant_all_bands (decode), quant_band(_stereo),
//                         quant_partition, compute_theta, anti_collapse,
//                         denormalise_bands, haar1, (de)interleave_hadamard,
//                         stereo_merge, special_hybrid_folding
//   celt/vq.c             alg_unquant, exp_rotation, renormalise_vector
//   celt/cwrs.c           cwrsi / decode_pulses (non-SMALL_FOOTPRINT)
//   celt/celt.c           comb_filter, init_caps
//   celt/mdct.c           clt_mdct_backward_c
//   celt/kiss_fft.c       opus_fft_impl, kf_bfly2/3/4/5
//   celt/pitch.c          pitch_downsample, pitch_search
//   celt/celt_lpc.c       _celt_lpc, celt_fir, celt_iir, _celt_autocorr
// The recursive band split (quant_partition) is one loop with a small explicit
// stack (at most LM + 1 <= 4 splits).  Every lane decodes the band's symbols,
// each with a range decoder of its own in step with the others, and the lanes
// share out the vector work (normalisation, rotations, Haar and Hadamard
// steps, folding, IMDCT, denormalisation, windowing, the searches and filters
// of concealment).
#pragma once
#include "rangedec.cuh"

namespace cuo {

enum { CELT_NB = 21, CELT_OVERLAP = 120, CELT_DEC_BUF = 2048, CELT_LPC_ORDER = 24, CELT_MAX_PERIOD = 1024 };
enum { SPREAD_NONE = 0, SPREAD_LIGHT = 1, SPREAD_NORMAL = 2, SPREAD_AGGRESSIVE = 3 };
static const int CELT_SIG_SAT = 300000000;

struct CeltDec {
    int32_t channels, stream_channels, start, end, disable_inv;
    // reset region (DECODER_RESET_START = rng)
    uint32_t rng;
    int32_t error, last_pitch_index, loss_duration, skip_plc;
    int32_t postfilter_period, postfilter_period_old;
    int32_t postfilter_gain, postfilter_gain_old;
    int32_t postfilter_tapset, postfilter_tapset_old;
    int32_t prefilter_and_fold;
    int32_t preemph_memD[2];
    alignas(16) int32_t decode_mem[2][CELT_DEC_BUF + CELT_OVERLAP];
    int16_t lpc[2][CELT_LPC_ORDER];
    int16_t oldBandE[2 * CELT_NB], oldLogE[2 * CELT_NB], oldLogE2[2 * CELT_NB], backgroundLogE[2 * CELT_NB];
};

// A split of quant_partition: what its second half needs.
struct QPSplit {
    int16_t *X, *lowband;
    int32_t bits, first_bits, rebalance, N, B, B0, LM, fill, mid_first, fixed;
    int16_t gain;
};

// Per lane group, in the decoder slot.  Besides the frame buffers it holds
// what would otherwise be function-local arrays of the serial stages: every
// lane of a group computes the same values, so one copy per group serves all
// of them (a per-lane stack copy would multiply the memory these stages touch
// by the group width).
struct CeltScratch {
    QPSplit qp[4];                    // quant_partition's splits, outermost first
    int32_t bits1[CELT_NB], bits2[CELT_NB], thresh[CELT_NB], trim_offset[CELT_NB];   // allocation
    union {
        int16_t X[2 * 960];
        alignas(16) int32_t deemph[960];   // the second channel of deemphasis, when X is done with
    };
    alignas(16) int32_t freq[960];
    int16_t norm[2 * 8 * 78];
    int16_t tmp[176];                 // (de)interleave staging
    int32_t iy[176];                  // PVQ pulses of one partition
    int32_t tf_res[CELT_NB], cap[CELT_NB], offsets[CELT_NB], fine_quant[CELT_NB], pulses[CELT_NB],
        fine_priority[CELT_NB];
    uint8_t collapse_masks[2 * CELT_NB];
    // PLC
    int16_t lp_pitch_buf[CELT_DEC_BUF >> 1];
    int16_t exc[CELT_MAX_PERIOD + CELT_LPC_ORDER];
    int16_t fir_tmp[CELT_MAX_PERIOD];
    int16_t x_lp4[(CELT_DEC_BUF - 720) >> 2];          // len >> 2, len = DEC_BUF - PLC_PITCH_LAG_MAX
    int16_t y_lp4[(CELT_DEC_BUF - 720 + 620) >> 2];    // (len + max_pitch) >> 2
    int32_t xcorr[CELT_MAX_PERIOD >> 1];
    int16_t ac_xx[CELT_MAX_PERIOD];
    int32_t etmp[CELT_OVERLAP];
};

// ------------------------------------------------------------------ init / reset

DNI void celt_reset(CeltDec *st)
{
    st->rng = 0;
    st->error = 0;
    st->last_pitch_index = 0;
    st->loss_duration = 0;
    st->skip_plc = 0;
    st->postfilter_period = st->postfilter_period_old = 0;
    st->postfilter_gain = st->postfilter_gain_old = 0;
    st->postfilter_tapset = st->postfilter_tapset_old = 0;
    st->prefilter_and_fold = 0;
    st->preemph_memD[0] = st->preemph_memD[1] = 0;
    memset(st->decode_mem, 0, sizeof(st->decode_mem));
    memset(st->lpc, 0, sizeof(st->lpc));
    memset(st->oldBandE, 0, sizeof(st->oldBandE));
    memset(st->backgroundLogE, 0, sizeof(st->backgroundLogE));
    ROLLED for (int i = 0; i < 2 * CELT_NB; i++) st->oldLogE[i] = st->oldLogE2[i] = -28672;   // -QCONST16(28.f, DB_SHIFT)
    st->skip_plc = 1;
}

// celt_decoder_init + CELT_SET_SIGNALLING(0) as done by opus_decoder_init
DFN void celt_init(CeltDec *st, int channels)
{
    st->channels = st->stream_channels = channels;
    st->start = 0;
    st->end = T_CELT_EFFEBANDS;
    st->disable_inv = channels == 1;
    celt_reset(st);
}

// ------------------------------------------------------------------ FFT / IMDCT

struct Cpx { int32_t r, i; };

DFN Cpx cmul(Cpx a, int16_t br, int16_t bi)
{
    Cpx m;
    m.r = wsub(c_mul16_32_q15(br, a.r), c_mul16_32_q15(bi, a.i));
    m.i = wadd(c_mul16_32_q15(bi, a.r), c_mul16_32_q15(br, a.i));
    return m;
}

// One radix-p stage of opus_fft_impl: N groups of m butterflies, group stride mm.
// Every butterfly touches its own p outputs, so the N*m of them are spread over lanes.
DNI void fft_stage(Lanes L, Cpx *F, int p, int fstride, int m, int N, int mm)
{
    const int inv = (int)((65536u + m - 1) / (unsigned)m);   // q / m == q * inv >> 16 for q < 480, m <= 120
    const int16_t *tw = T_fft_twiddles;
    if (p == 2) {
        // kf_bfly2 (m == 4 in the static mode)
        const int16_t k = 23170;   // QCONST16(0.7071067812, 15)
        LFOR(L, i, 0, N) {
            Cpx *Fo = F + 8 * i, *F2 = Fo + 4, t;
            t = F2[0];
            F2[0].r = wsub(Fo[0].r, t.r); F2[0].i = wsub(Fo[0].i, t.i);
            Fo[0].r = wadd(Fo[0].r, t.r); Fo[0].i = wadd(Fo[0].i, t.i);
            t.r = c_mul16_32_q15(k, wadd(F2[1].r, F2[1].i));
            t.i = c_mul16_32_q15(k, wsub(F2[1].i, F2[1].r));
            F2[1].r = wsub(Fo[1].r, t.r); F2[1].i = wsub(Fo[1].i, t.i);
            Fo[1].r = wadd(Fo[1].r, t.r); Fo[1].i = wadd(Fo[1].i, t.i);
            t.r = F2[2].i; t.i = -F2[2].r;
            F2[2].r = wsub(Fo[2].r, t.r); F2[2].i = wsub(Fo[2].i, t.i);
            Fo[2].r = wadd(Fo[2].r, t.r); Fo[2].i = wadd(Fo[2].i, t.i);
            t.r = c_mul16_32_q15(k, wsub(F2[3].i, F2[3].r));
            t.i = c_mul16_32_q15(k, (int32_t)(0u - (uint32_t)wadd(F2[3].i, F2[3].r)));
            F2[3].r = wsub(Fo[3].r, t.r); F2[3].i = wsub(Fo[3].i, t.i);
            Fo[3].r = wadd(Fo[3].r, t.r); Fo[3].i = wadd(Fo[3].i, t.i);
        }
    } else if (p == 4) {
        if (m == 1) {
            LFOR(L, i, 0, N) {
                Cpx *Fo = F + 4 * i, s0, s1;
                s0.r = wsub(Fo[0].r, Fo[2].r); s0.i = wsub(Fo[0].i, Fo[2].i);
                Fo[0].r = wadd(Fo[0].r, Fo[2].r); Fo[0].i = wadd(Fo[0].i, Fo[2].i);
                s1.r = wadd(Fo[1].r, Fo[3].r); s1.i = wadd(Fo[1].i, Fo[3].i);
                Fo[2].r = wsub(Fo[0].r, s1.r); Fo[2].i = wsub(Fo[0].i, s1.i);
                Fo[0].r = wadd(Fo[0].r, s1.r); Fo[0].i = wadd(Fo[0].i, s1.i);
                s1.r = wsub(Fo[1].r, Fo[3].r); s1.i = wsub(Fo[1].i, Fo[3].i);
                Fo[1].r = wadd(s0.r, s1.i); Fo[1].i = wsub(s0.i, s1.r);
                Fo[3].r = wsub(s0.r, s1.i); Fo[3].i = wadd(s0.i, s1.r);
            }
        } else {
            LFOR(L, q, 0, N * m) {
                int i = q * inv >> 16, j = q - i * m;
                Cpx *Fo = F + i * mm + j, s[6];
                s[0] = cmul(Fo[m], tw[2 * (j * fstride)], tw[2 * (j * fstride) + 1]);
                s[1] = cmul(Fo[2 * m], tw[2 * (2 * j * fstride)], tw[2 * (2 * j * fstride) + 1]);
                s[2] = cmul(Fo[3 * m], tw[2 * (3 * j * fstride)], tw[2 * (3 * j * fstride) + 1]);
                s[5].r = wsub(Fo[0].r, s[1].r); s[5].i = wsub(Fo[0].i, s[1].i);
                Fo[0].r = wadd(Fo[0].r, s[1].r); Fo[0].i = wadd(Fo[0].i, s[1].i);
                s[3].r = wadd(s[0].r, s[2].r); s[3].i = wadd(s[0].i, s[2].i);
                s[4].r = wsub(s[0].r, s[2].r); s[4].i = wsub(s[0].i, s[2].i);
                Fo[2 * m].r = wsub(Fo[0].r, s[3].r); Fo[2 * m].i = wsub(Fo[0].i, s[3].i);
                Fo[0].r = wadd(Fo[0].r, s[3].r); Fo[0].i = wadd(Fo[0].i, s[3].i);
                Fo[m].r = wadd(s[5].r, s[4].i); Fo[m].i = wsub(s[5].i, s[4].r);
                Fo[3 * m].r = wsub(s[5].r, s[4].i); Fo[3 * m].i = wadd(s[5].i, s[4].r);
            }
        }
    } else if (p == 3) {
        const int16_t epi3i = -28378;
        LFOR(L, q, 0, N * m) {
            int i = q * inv >> 16, j = q - i * m;
            Cpx *Fo = F + i * mm + j, s[4];
            s[1] = cmul(Fo[m], tw[2 * (j * fstride)], tw[2 * (j * fstride) + 1]);
            s[2] = cmul(Fo[2 * m], tw[2 * (2 * j * fstride)], tw[2 * (2 * j * fstride) + 1]);
            s[3].r = wadd(s[1].r, s[2].r); s[3].i = wadd(s[1].i, s[2].i);
            s[0].r = wsub(s[1].r, s[2].r); s[0].i = wsub(s[1].i, s[2].i);
            Fo[m].r = wsub(Fo[0].r, s[3].r >> 1);
            Fo[m].i = wsub(Fo[0].i, s[3].i >> 1);
            s[0].r = c_mul16_32_q15(epi3i, s[0].r);
            s[0].i = c_mul16_32_q15(epi3i, s[0].i);
            Fo[0].r = wadd(Fo[0].r, s[3].r); Fo[0].i = wadd(Fo[0].i, s[3].i);
            Fo[2 * m].r = wadd(Fo[m].r, s[0].i);
            Fo[2 * m].i = wsub(Fo[m].i, s[0].r);
            Fo[m].r = wsub(Fo[m].r, s[0].i);
            Fo[m].i = wadd(Fo[m].i, s[0].r);
        }
    } else {
        // kf_bfly5
        const int16_t yar = 10126, yai = -31164, ybr = -26510, ybi = -19261;
        LFOR(L, q, 0, N * m) {
            int i = q * inv >> 16, u = q - i * m;
            Cpx *F0 = F + i * mm + u, *F1 = F0 + m, *F2 = F0 + 2 * m, *F3 = F0 + 3 * m, *F4 = F0 + 4 * m;
            Cpx s[13];
            s[0] = *F0;
            s[1] = cmul(*F1, tw[2 * (u * fstride)], tw[2 * (u * fstride) + 1]);
            s[2] = cmul(*F2, tw[2 * (2 * u * fstride)], tw[2 * (2 * u * fstride) + 1]);
            s[3] = cmul(*F3, tw[2 * (3 * u * fstride)], tw[2 * (3 * u * fstride) + 1]);
            s[4] = cmul(*F4, tw[2 * (4 * u * fstride)], tw[2 * (4 * u * fstride) + 1]);
            s[7].r = wadd(s[1].r, s[4].r); s[7].i = wadd(s[1].i, s[4].i);
            s[10].r = wsub(s[1].r, s[4].r); s[10].i = wsub(s[1].i, s[4].i);
            s[8].r = wadd(s[2].r, s[3].r); s[8].i = wadd(s[2].i, s[3].i);
            s[9].r = wsub(s[2].r, s[3].r); s[9].i = wsub(s[2].i, s[3].i);
            F0->r = wadd(F0->r, wadd(s[7].r, s[8].r));
            F0->i = wadd(F0->i, wadd(s[7].i, s[8].i));
            s[5].r = wadd(s[0].r, wadd(c_mul16_32_q15(yar, s[7].r), c_mul16_32_q15(ybr, s[8].r)));
            s[5].i = wadd(s[0].i, wadd(c_mul16_32_q15(yar, s[7].i), c_mul16_32_q15(ybr, s[8].i)));
            s[6].r = wadd(c_mul16_32_q15(yai, s[10].i), c_mul16_32_q15(ybi, s[9].i));
            s[6].i = (int32_t)(0u - (uint32_t)wadd(c_mul16_32_q15(yai, s[10].r), c_mul16_32_q15(ybi, s[9].r)));
            F1->r = wsub(s[5].r, s[6].r); F1->i = wsub(s[5].i, s[6].i);
            F4->r = wadd(s[5].r, s[6].r); F4->i = wadd(s[5].i, s[6].i);
            s[11].r = wadd(s[0].r, wadd(c_mul16_32_q15(ybr, s[7].r), c_mul16_32_q15(yar, s[8].r)));
            s[11].i = wadd(s[0].i, wadd(c_mul16_32_q15(ybr, s[7].i), c_mul16_32_q15(yar, s[8].i)));
            s[12].r = wsub(c_mul16_32_q15(yai, s[9].i), c_mul16_32_q15(ybi, s[10].i));
            s[12].i = wsub(c_mul16_32_q15(ybi, s[10].r), c_mul16_32_q15(yai, s[9].r));
            F2->r = wadd(s[11].r, s[12].r); F2->i = wadd(s[11].i, s[12].i);
            F3->r = wsub(s[11].r, s[12].r); F3->i = wsub(s[11].i, s[12].i);
        }
    }
    lsync(L);
}

DNI void celt_fft(Lanes L, int shift_idx, Cpx *fout)
{
    const int16_t *factors;
    int sh;
    switch (shift_idx) {
    case 0: factors = T_fft0_factors; sh = T_FFT0_SHIFT; break;
    case 1: factors = T_fft1_factors; sh = T_FFT1_SHIFT; break;
    case 2: factors = T_fft2_factors; sh = T_FFT2_SHIFT; break;
    default: factors = T_fft3_factors; sh = T_FFT3_SHIFT; break;
    }
    int shift = sh > 0 ? sh : 0;
    int fstride[8];
    fstride[0] = 1;
    int Lf = 0, p, m;
    ROLLED do {
        p = factors[2 * Lf];
        m = factors[2 * Lf + 1];
        fstride[Lf + 1] = fstride[Lf] * p;
        Lf++;
    } while (m != 1);
    m = factors[2 * Lf - 1];
    ROLLED for (int i = Lf - 1; i >= 0; i--) {
        int m2 = i != 0 ? factors[2 * i - 1] : 1;
        fft_stage(L, fout, factors[2 * i], fstride[i] << shift, m, fstride[i], m2);
        m = m2;
    }
}

DFN const int16_t *fft_bitrev(int shift)
{
    return shift == 0 ? T_fft0_bitrev : shift == 1 ? T_fft1_bitrev : shift == 2 ? T_fft2_bitrev : T_fft3_bitrev;
}

// celt/mdct.c clt_mdct_backward_c.  With `twin`, a second output buffer gets the
// same transform (a mono frame in a stereo stream): what precedes the
// overlap-add is done once and copied.
DNI void mdct_backward(Lanes L, const int32_t *in, int32_t *out, int shift, int stride, int32_t *twin = nullptr)
{
    int N = T_CELT_MDCT_N;
    const int16_t *trig = T_celt_mdct_trig;
    ROLLED for (int i = 0; i < shift; i++) { N >>= 1; trig += N; }
    int N2 = N >> 1, N4 = N >> 2;
    const int16_t *bitrev = fft_bitrev(shift);
    int32_t *yp = out + (CELT_OVERLAP >> 1);
    LFOR(L, i, 0, N4) {
        int rev = bitrev[i];
        int32_t x1 = in[2 * i * stride], x2 = in[stride * (N2 - 1) - 2 * i * stride];
        int32_t yr = wadd(c_mul16_32_q15(trig[i], x2), c_mul16_32_q15(trig[N4 + i], x1));
        int32_t yi = wsub(c_mul16_32_q15(trig[i], x1), c_mul16_32_q15(trig[N4 + i], x2));
        yp[2 * rev + 1] = yr;
        yp[2 * rev] = yi;
    }
    lsync(L);
    celt_fft(L, shift, (Cpx *)yp);
    LFOR(L, i, 0, (N4 + 1) >> 1) {
        int32_t *yp0 = yp + 2 * i, *yp1 = yp + N2 - 2 - 2 * i;
        int32_t re = yp0[1], im = yp0[0];
        int16_t t0 = trig[i], t1 = trig[N4 + i];
        int32_t yr = wadd(c_mul16_32_q15(t0, re), c_mul16_32_q15(t1, im));
        int32_t yi = wsub(c_mul16_32_q15(t1, re), c_mul16_32_q15(t0, im));
        re = yp1[1];
        im = yp1[0];
        yp0[0] = yr;
        yp1[1] = yi;
        t0 = trig[N4 - i - 1];
        t1 = trig[N2 - i - 1];
        yr = wadd(c_mul16_32_q15(t0, re), c_mul16_32_q15(t1, im));
        yi = wsub(c_mul16_32_q15(t1, re), c_mul16_32_q15(t0, im));
        yp1[0] = yr;
        yp0[1] = yi;
    }
    lsync(L);
    if (twin) {
        LFOR(L, i, 0, N2) twin[CELT_OVERLAP / 2 + i] = yp[i];
        lsync(L);
    }
    const int16_t *w = T_celt_window;
    LFOR(L, q, 0, twin ? CELT_OVERLAP : CELT_OVERLAP / 2) {
        const int i = q < CELT_OVERLAP / 2 ? q : q - CELT_OVERLAP / 2;
        int32_t *o = q < CELT_OVERLAP / 2 ? out : twin;
        int32_t *xp1 = o + CELT_OVERLAP - 1 - i, *yp1 = o + i;
        int32_t x1 = *xp1, x2 = *yp1;
        int16_t w1 = w[i], w2 = w[CELT_OVERLAP - 1 - i];
        *yp1 = wsub(c_mul16_32_q15(w2, x2), c_mul16_32_q15(w1, x1));
        *xp1 = wadd(c_mul16_32_q15(w1, x2), c_mul16_32_q15(w2, x1));
    }
    lsync(L);
}

// ------------------------------------------------------------------ synthesis helpers

// Band of a bin of the shortest frame (eBands inverted).
struct BandOf {
    uint8_t b[101];
    constexpr BandOf() : b()
    {
        const int e[22] = {0, 1, 2, 3, 4, 5, 6, 7, 8, 10, 12, 14, 16, 20, 24, 28, 34, 40, 48, 60, 78, 100};
        for (int k = 0; k < 21; k++)
            for (int u = e[k]; u < e[k + 1]; u++) b[u] = (uint8_t)k;
        b[100] = 21;
    }
};
TABC(BandOf, T_band_of) = BandOf();
TABG(BandOf, T_band_of_lanes) = BandOf();   // for lookups that differ between the lanes

// celt/bands.c denormalise_bands (downsample 1).  The lanes work out the bands'
// gains and shifts first (gain << 8 | shift + 2, in band_gain), then scale the
// bins, four in flight each.
DNI void denormalise_bands(Lanes L, const int16_t *X, int32_t *freq, const int16_t *bandLogE, int start,
                           int end, int LM, int silence, int32_t *band_gain)
{
    const int16_t *eB = T_celt_eBands;
    const int N = T_CELT_SHORTMDCT << LM;
    int bound = eB[end] << LM, low = eB[start] << LM;
    if (silence) bound = low = 0;
    LFOR(L, b, start, end) {
        int16_t lg = c_sat16(wadd(bandLogE[b], shl32((int32_t)T_celt_eMeans[b], 6)));
        int shift = 16 - (lg >> 10);
        int16_t g;
        if (shift > 31) { shift = 0; g = 0; }
        else g = (int16_t)c_exp2_frac((int16_t)(lg & 1023));
        if (shift <= -2) { g = 16384; shift = -2; }
        band_gain[b] = shl32((int32_t)g, 8) | (shift + 2);
    }
    lsync(L);
    ROLLED for (int j0 = L.id; j0 < N; j0 += 4 * L.n) {
        int32_t x[4], g[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int j = j0 + k * L.n;
            x[k] = 0;
            g[k] = 2;
            if (j >= low && j < bound) {
                x[k] = X[j];
                g[k] = band_gain[T_band_of_lanes.b[j >> LM]];
            }
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int j = j0 + k * L.n, shift = (g[k] & 0xff) - 2;
            const int32_t v = c_mul16(x[k], g[k] >> 8);
            if (j < N) freq[j] = shift < 0 ? shl32(v, -shift) : v >> shift;
        }
    }
    lsync(L);
}

// gains[3][3] of celt/celt.c (comb filter taps per tapset)
TABC(int16_t, T_comb_gains[3][3]) = {{10048, 7112, 4248}, {15200, 8784, 0}, {26208, 3280, 0}};

// celt/celt.c comb_filter split across the lanes.  In place (y == x) output i reads the
// input at i and outputs at i - T - 2 .. i - T + 2 (T >= 15), so a block of
// min(T0, T1) - 2 consecutive outputs depends only on earlier blocks: the
// blocks run in order with a barrier between them and the outputs of a block
// in parallel, each with the serial code's exact arithmetic.  Out of place
// every output depends on the input only and one block covers the frame.
DNI void comb_filter_lanes(Lanes L, int32_t *y, int32_t *x, int T0, int T1, int N, int16_t g0, int16_t g1,
                           int tapset0, int tapset1, const int16_t *window, int overlap)
{
    const int16_t (*gains)[3] = T_comb_gains;
    lsync(L);
    if (g0 == 0 && g1 == 0) {
        if (x != y) {
            LFOR(L, i, 0, N) y[i] = x[i];
            lsync(L);
        }
        return;
    }
    T0 = imax(T0, 15);
    T1 = imax(T1, 15);
    int16_t g00 = (int16_t)c_mul16_p15(g0, gains[tapset0][0]);
    int16_t g01 = (int16_t)c_mul16_p15(g0, gains[tapset0][1]);
    int16_t g02 = (int16_t)c_mul16_p15(g0, gains[tapset0][2]);
    int16_t g10 = (int16_t)c_mul16_p15(g1, gains[tapset1][0]);
    int16_t g11 = (int16_t)c_mul16_p15(g1, gains[tapset1][1]);
    int16_t g12 = (int16_t)c_mul16_p15(g1, gains[tapset1][2]);
    if (g0 == g1 && T0 == T1 && tapset0 == tapset1) overlap = 0;
    const int B = x == y ? imin(T0, T1) - 2 : imax(N, 1);
    ROLLED for (int s = 0; s < overlap; s += B) {
        int e = imin(s + B, overlap);
        LFOR(L, i, s, e) {
            int16_t f = (int16_t)c_mul16_q15(window[i], window[i]);
            int32_t v = x[i];
            v = wadd(v, c_mul16_32_q15((int16_t)c_mul16_q15(32767 - f, g00), x[i - T0]));
            v = wadd(v, c_mul16_32_q15((int16_t)c_mul16_q15(32767 - f, g01), wadd(x[i - T0 + 1], x[i - T0 - 1])));
            v = wadd(v, c_mul16_32_q15((int16_t)c_mul16_q15(32767 - f, g02), wadd(x[i - T0 + 2], x[i - T0 - 2])));
            v = wadd(v, c_mul16_32_q15((int16_t)c_mul16_q15(f, g10), x[i - T1]));
            v = wadd(v, c_mul16_32_q15((int16_t)c_mul16_q15(f, g11), wadd(x[i - T1 + 1], x[i - T1 - 1])));
            v = wadd(v, c_mul16_32_q15((int16_t)c_mul16_q15(f, g12), wadd(x[i - T1 + 2], x[i - T1 - 2])));
            y[i] = c_sat(v, CELT_SIG_SAT);
        }
        lsync(L);
    }
    if (g1 == 0) {
        if (x != y) {
            LFOR(L, k, overlap, N) y[k] = x[k];
            lsync(L);
        }
        return;
    }
    ROLLED for (int s = overlap; s < N; s += B) {
        int e = imin(s + B, N);
        LFOR(L, k, s, e) {
            int32_t v = wadd(wadd(wadd(x[k], c_mul16_32_q15(g10, x[k - T1])),
                                  c_mul16_32_q15(g11, wadd(x[k - T1 + 1], x[k - T1 - 1]))),
                             c_mul16_32_q15(g12, wadd(x[k - T1 + 2], x[k - T1 - 2])));
            y[k] = c_sat(v, CELT_SIG_SAT);
        }
        lsync(L);
    }
}

// Four samples moved as one 16-byte word.
struct alignas(16) Quad { int32_t v[4]; };

// celt/celt_decoder.c deemphasis (downsample 1): a one-pole recursion, serial.
// One step is m = (coef0 (x + m)) >> 15: with c the 32-bit value of coef0 * 2^17
// less 2^32, tmp + (tmp c >> 32) is that product exactly, so a step waits for one
// add and one mad.hi, and a lone warp pays for every other instruction beside
// them: lane c runs channel c's recursion and nothing else (a single lane one
// after the other), eight samples a step, loaded a step ahead and stored as
// 16-byte words, and all lanes then scale, saturate and place the samples.
// t0 and t1 receive the recursions' outputs.  A second of audio, with the
// scaling and the stores in the recursion's loop and now: stereo frames 5.0 and
// 2.2 M cycles, mono 2.7 and 0.95 (a 94 s file 18.8 and 17.5 ms a call).
DNI void deemphasis(Lanes L, const int32_t *in0, const int32_t *in1, int16_t *pcm, int N, int C, int32_t *mem,
                    int accum, int32_t *t0, int32_t *t1)
{
    const int32_t cm = (int32_t)(((uint32_t)T_CELT_PREEMPH0 << 17));
    lsync(L);
    int c0 = 0, c1 = C;
    if (L.n > 1) {
        c0 = L.id;
        c1 = L.id < C ? L.id + 1 : L.id;
    }
    ROLLED for (int c = c0; c < c1; c++) {
        const Quad *x = (const Quad *)(c == 0 ? in0 : in1);
        Quad *t = (Quad *)(c == 0 ? t0 : t1);
        int32_t m = mem[c];
        Quad a0 = x[0], a1 = x[1];   // N is a multiple of 8
        ROLLED for (int j = 0; j < N / 4; j += 2) {
            Quad b0 = a0, b1 = a1;
            const int nx = j + 2 < N / 4 ? j + 2 : j;
            a0 = x[nx];
            a1 = x[nx + 1];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                b0.v[k] = wadd(b0.v[k], m);
                m = s_smlawh(b0.v[k], b0.v[k], cm);
            }
            t[j] = b0;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                b1.v[k] = wadd(b1.v[k], m);
                m = s_smlawh(b1.v[k], b1.v[k], cm);
            }
            t[j + 1] = b1;
        }
        mem[c] = m;
    }
    lsync(L);
    const int total = N * C;
    ROLLED for (int b = L.id; b < total; b += 4 * L.n) {
        int32_t v[4], add[4] = {0, 0, 0, 0};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int q = b + k * L.n;
            if (q < total) {
                v[k] = (C == 2 && (q & 1) ? t1 : t0)[C == 2 ? q >> 1 : q];
                if (accum) add[k] = pcm[q];
            }
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int q = b + k * L.n;
            if (q < total) pcm[q] = (int16_t)c_sat16(add[k] + c_sig2word16(v[k]));
        }
    }
    lsync(L);
}

// celt/celt_decoder.c celt_synthesis (downsample 1)
DNI void celt_synthesis(Lanes L, CeltScratch *w, const int16_t *X, int32_t **out_syn,
                        const int16_t *oldBandE, int start, int effEnd, int C, int CC, int isTransient, int LM,
                        int silence)
{
    int M = 1 << LM;
    int N = T_CELT_SHORTMDCT << LM;
    int B, NB, shift;
    if (isTransient) { B = M; NB = T_CELT_SHORTMDCT; shift = T_CELT_MAXLM; }
    else { B = 1; NB = T_CELT_SHORTMDCT << LM; shift = T_CELT_MAXLM - LM; }
    int32_t *freq = w->freq;
    if (CC == 2 && C == 1) {
        denormalise_bands(L, X, freq, oldBandE, start, effEnd, LM, silence, w->bits1);
        ROLLED for (int b = 0; b < B; b++)
            mdct_backward(L, &freq[b], out_syn[0] + NB * b, shift, B, out_syn[1] + NB * b);
    } else if (CC == 1 && C == 2) {
        int32_t *freq2 = out_syn[0] + CELT_OVERLAP / 2;
        denormalise_bands(L, X, freq, oldBandE, start, effEnd, LM, silence, w->bits1);
        denormalise_bands(L, X + N, freq2, oldBandE + CELT_NB, start, effEnd, LM, silence, w->bits1);
        LFOR(L, i, 0, N) freq[i] = wadd(freq[i] >> 1, freq2[i] >> 1);
        lsync(L);
        ROLLED for (int b = 0; b < B; b++) mdct_backward(L, &freq[b], out_syn[0] + NB * b, shift, B);
    } else {
        ROLLED for (int c = 0; c < CC; c++) {
            denormalise_bands(L, X + c * N, freq, oldBandE + c * CELT_NB, start, effEnd, LM, silence, w->bits1);
            ROLLED for (int b = 0; b < B; b++) mdct_backward(L, &freq[b], out_syn[c] + NB * b, shift, B);
        }
    }
    ROLLED for (int c = 0; c < CC; c++) {
        int32_t *o = out_syn[c];
        LFOR(L, i, 0, N) o[i] = c_sat(o[i], CELT_SIG_SAT);
    }
    lsync(L);
}

// ------------------------------------------------------------------ energy

DNI void unquant_coarse_energy(int start, int end, int16_t *oldEBands, int intra, RangeDec *rd, int C, int LM)
{
    RangeDec dd = *rd, *dec = &dd;   // in registers
    const uint8_t *prob = &T_celt_e_prob_model[(LM * 2 + intra) * 42];
    int32_t prev[2] = {0, 0};
    int16_t coef, beta;
    if (intra) { coef = 0; beta = T_CELT_BETA_INTRA; }
    else { beta = T_celt_beta_coef[LM]; coef = T_celt_pred_coef[LM]; }
    int32_t budget = dec->storage * 8;
    ROLLED for (int i = start; i < end; i++) {
        ROLLED for (int c = 0; c < C; c++) {
            int qi;
            int32_t tell = rd_tell(dec);
            if (budget - tell >= 15) {
                int pi = 2 * imin(i, 20);
                qi = rdi_laplace(dec, prob[pi] << 7, prob[pi + 1] << 6);
            } else if (budget - tell >= 2) {
                qi = rdi_icdf(dec, T_celt_small_energy_icdf, 2);
                qi = (qi >> 1) ^ -(qi & 1);
            } else if (budget - tell >= 1) {
                qi = -rdi_bit_logp(dec, 1);
            } else {
                qi = -1;
            }
            int32_t q = shl32(qi, 10);
            int16_t *e = &oldEBands[i + c * CELT_NB];
            *e = (int16_t)max32(-9216, *e);   // -QCONST16(9, DB_SHIFT)
            int32_t tmp = wadd(wadd(c_pshr(c_mul16(coef, *e), 8), prev[c]), shl32(q, 7));
            tmp = max32(-3670016, tmp);       // -QCONST32(28, DB_SHIFT + 7)
            *e = (int16_t)c_pshr(tmp, 7);
            prev[c] = wsub(wadd(prev[c], shl32(q, 7)), c_mul16(beta, c_pshr(q, 8)));
        }
    }
    *rd = dd;
}

DNI void unquant_fine_energy(int start, int end, int16_t *oldEBands, const int32_t *fine_quant, RangeDec *rd,
                             int C)
{
    RangeDec dd = *rd, *dec = &dd;   // in registers
    ROLLED for (int i = start; i < end; i++) {
        if (fine_quant[i] <= 0) continue;
        ROLLED for (int c = 0; c < C; c++) {
            int q2 = (int)rdi_bits(dec, fine_quant[i]);
            int16_t offset = (int16_t)(((shl32(q2, 10) + 512) >> fine_quant[i]) - 512);
            oldEBands[i + c * CELT_NB] = (int16_t)(oldEBands[i + c * CELT_NB] + offset);
        }
    }
    *rd = dd;
}

DNI void unquant_energy_finalise(int start, int end, int16_t *oldEBands, const int32_t *fine_quant,
                                 const int32_t *fine_priority, int bits_left, RangeDec *rd, int C)
{
    RangeDec dd = *rd, *dec = &dd;   // in registers
    ROLLED for (int prio = 0; prio < 2; prio++) {
        ROLLED for (int i = start; i < end && bits_left >= C; i++) {
            if (fine_quant[i] >= 8 || fine_priority[i] != prio) continue;
            ROLLED for (int c = 0; c < C; c++) {
                int q2 = (int)rdi_bits(dec, 1);
                int16_t offset = (int16_t)((int16_t)((uint16_t)q2 << 10) - 512) >> (fine_quant[i] + 1);
                oldEBands[i + c * CELT_NB] = (int16_t)(oldEBands[i + c * CELT_NB] + offset);
                bits_left--;
            }
        }
    }
    *rd = dd;
}

// ------------------------------------------------------------------ allocation

DFN int get_pulses(int i) { return i < 8 ? i : (8 + (i & 7)) << ((i >> 3) - 1); }

DFN const uint8_t *pulse_cache(int band, int LM)
{
    return T_celt_cache_bits + T_celt_cache_index[(LM + 1) * CELT_NB + band];
}

DFN int bits2pulses(int band, int LM, int bits)
{
    const uint8_t *cache = pulse_cache(band, LM);
    int lo = 0, hi = cache[0];
    bits--;
    ROLLED for (int i = 0; i < 6; i++) {
        int mid = (lo + hi + 1) >> 1;
        if ((int)cache[mid] >= bits) hi = mid;
        else lo = mid;
    }
    if (bits - (lo == 0 ? -1 : (int)cache[lo]) <= (int)cache[hi] - bits) return lo;
    return hi;
}

DFN int pulses2bits(int band, int LM, int pulses)
{
    const uint8_t *cache = pulse_cache(band, LM);
    return pulses == 0 ? 0 : cache[pulses] + 1;
}

DFN void init_caps(const Lanes &L, int32_t *cap, int LM, int C)
{
    LFOR(L, i, 0, CELT_NB) {
        int N = (T_celt_eBands[i + 1] - T_celt_eBands[i]) << LM;
        cap[i] = (T_celt_cache_caps[CELT_NB * (2 * LM + C - 1) + i] + 64) * C * N >> 2;
    }
}

// Bit allocation.  It runs on every lane of the group: the lanes split the
// bands (band j of a search step adds its own share to the total, up to the
// highest band that reaches its threshold), and the symbols between the
// searches are decoded by all of them from a range decoder in registers.  One
// lane walking the bands took 52 k cycles a full-band frame, this 16 k.

// Sum over the bands of what each takes when it asks for want(j) bits: bands up
// to the highest that reaches its threshold take what they ask for, at most
// their cap; the ones above take the floor when they reach that.
template <class F>
DFN int32_t alloc_sum(const Lanes &L, int start, int end, const int32_t *thresh, const int32_t *cap, int alloc_floor,
                      F want)
{
    int top = -1;
    LFOR(L, j, start, end) if (want(j) >= thresh[j]) top = imax(top, j);
    top = lmax(L, top);
    int32_t sum = 0;
    LFOR(L, j, start, end) {
        const int bits = want(j);
        sum += j <= top ? imin(bits, cap[j]) : bits >= alloc_floor ? alloc_floor : 0;
    }
    return lsum(L, sum);
}

DFN int interp_bits2pulses(const Lanes &L, int start, int end, int skip_start, const int32_t *bits1,
                           const int32_t *bits2, const int32_t *thresh, const int32_t *cap, int32_t total,
                           int32_t *_balance, int skip_rsv, int *intensity, int intensity_rsv, int *dual_stereo,
                           int dual_stereo_rsv, int32_t *bits, int32_t *ebits, int32_t *fine_priority, int C,
                           int LM, RangeDec *ec)
{
    const int16_t *eB = T_celt_eBands;
    int alloc_floor = C << 3;
    int stereo = C > 1;
    int logM = LM << 3;
    int lo = 0, hi = 1 << 6;
    ROLLED for (int i = 0; i < 6; i++) {
        int mid = (lo + hi) >> 1;
        const int32_t psum = alloc_sum(L, start, end, thresh, cap, alloc_floor,
                                       [&](int j) CUO_INLINE { return bits1[j] + (mid * bits2[j] >> 6); });
        if (psum > total) hi = mid;
        else lo = mid;
    }
    int top = -1;
    LFOR(L, j, start, end) if (bits1[j] + (lo * bits2[j] >> 6) >= thresh[j]) top = imax(top, j);
    top = lmax(L, top);
    int32_t psum = 0;
    LFOR(L, j, start, end) {
        int tmp = bits1[j] + (lo * bits2[j] >> 6);
        if (j > top) tmp = tmp >= alloc_floor ? alloc_floor : 0;
        tmp = imin(tmp, cap[j]);
        bits[j] = tmp;
        psum += tmp;
    }
    psum = lsum(L, psum);
    lsync(L);
    // which of the highest bands are skipped: every lane reads the bands' bits
    // as they are; the skipped bands' new ones are written after the loop
    unsigned floored = 0;
    int codedBands;
    ROLLED for (codedBands = end;; codedBands--) {
        int j = codedBands - 1;
        if (j <= skip_start) {
            total += skip_rsv;
            break;
        }
        int32_t left = total - psum;
        int32_t percoeff = (int32_t)((uint32_t)left / (uint32_t)(eB[codedBands] - eB[start]));
        left -= (eB[codedBands] - eB[start]) * percoeff;
        int rem = imax(left - (eB[j] - eB[start]), 0);
        int band_width = eB[codedBands] - eB[j];
        int band_bits = (int)(bits[j] + percoeff * band_width + rem);
        if (band_bits >= imax(thresh[j], alloc_floor + (1 << 3))) {
            if (rdi_bit_logp(ec, 1)) break;
            psum += 1 << 3;
            band_bits -= 1 << 3;
        }
        psum -= bits[j] + intensity_rsv;
        if (intensity_rsv > 0) intensity_rsv = T_celt_log2_frac_table[j - start];
        psum += intensity_rsv;
        if (band_bits >= alloc_floor) {
            psum += alloc_floor;
            floored |= 1u << j;
        }
    }
    if (intensity_rsv > 0) *intensity = start + (int)rdi_uint(ec, codedBands + 1 - start);
    else *intensity = 0;
    if (*intensity <= start) {
        total += dual_stereo_rsv;
        dual_stereo_rsv = 0;
    }
    if (dual_stereo_rsv > 0) *dual_stereo = rdi_bit_logp(ec, 1);
    else *dual_stereo = 0;
    int32_t left = total - psum;
    int32_t percoeff = (int32_t)((uint32_t)left / (uint32_t)(eB[codedBands] - eB[start]));
    left -= (eB[codedBands] - eB[start]) * percoeff;
    lsync(L);
    LFOR(L, j, start, end) {
        if (j >= codedBands) {
            bits[j] = floored >> j & 1 ? alloc_floor : 0;
        } else {
            const int width = eB[j + 1] - eB[j];
            bits[j] += percoeff * width + imax(0, imin(left - (eB[j] - eB[start]), width));
        }
    }
    // fine energy against shapes, band after band: what a band cannot use goes
    // to the next
    int32_t balance = 0;
    lead(L, [&]() CUO_INLINE {
        int j;
        ROLLED for (j = start; j < codedBands; j++) {
            int N0 = eB[j + 1] - eB[j];
            int N = N0 << LM;
            int32_t bit = (int32_t)bits[j] + balance;
            int32_t excess;
            int32_t bj, ej, fp;
            if (N > 1) {
                excess = max32(bit - cap[j], 0);
                bj = bit - excess;
                int den = C * N + ((C == 2 && N > 2 && !*dual_stereo && j < *intensity) ? 1 : 0);
                int NClogN = den * (T_celt_logN[j] + logM);
                int offset = (NClogN >> 1) - den * 21;   // FINE_OFFSET
                if (N == 2) offset += den << 3 >> 2;
                if (bj + offset < den * 2 << 3) offset += NClogN >> 2;
                else if (bj + offset < den * 3 << 3) offset += NClogN >> 3;
                ej = imax(0, bj + offset + (den << 2));
                ej = (int32_t)((uint32_t)ej / (uint32_t)den) >> 3;
                if (C * ej > (bj >> 3)) ej = bj >> stereo >> 3;
                ej = imin(ej, 8);
                fp = ej * (den << 3) >= bj + offset;
                bj -= C * ej << 3;
            } else {
                excess = max32(0, bit - (C << 3));
                bj = bit - excess;
                ej = 0;
                fp = 1;
            }
            if (excess > 0) {
                int extra_fine = imin(excess >> (stereo + 3), 8 - ej);
                ej += extra_fine;
                int extra_bits = extra_fine * C << 3;
                fp = extra_bits >= excess - balance;
                excess -= extra_bits;
            }
            bits[j] = bj;
            ebits[j] = ej;
            fine_priority[j] = fp;
            balance = excess;
        }
        ROLLED for (; j < end; j++) {
            ebits[j] = bits[j] >> stereo >> 3;
            bits[j] = 0;
            fine_priority[j] = ebits[j] < 1;
        }
    });
    *_balance = lbcast(L, balance);
    return codedBands;
}

DNI int clt_compute_allocation(Lanes L, int start, int end, const int32_t *offsets, const int32_t *cap,
                               int alloc_trim, int *intensity, int *dual_stereo, int32_t total, int32_t *balance,
                               int32_t *pulses, int32_t *ebits, int32_t *fine_priority, int C, int LM,
                               RangeDec *rd, CeltScratch *w)
{
    const int16_t *eB = T_celt_eBands;
    int32_t *bits1 = w->bits1, *bits2 = w->bits2, *thresh = w->thresh, *trim_offset = w->trim_offset;
    RangeDec d = *rd;
    total = max32(total, 0);
    int skip_rsv = total >= 1 << 3 ? 1 << 3 : 0;
    total -= skip_rsv;
    int intensity_rsv = 0, dual_stereo_rsv = 0;
    if (C == 2) {
        intensity_rsv = T_celt_log2_frac_table[end - start];
        if (intensity_rsv > total) {
            intensity_rsv = 0;
        } else {
            total -= intensity_rsv;
            dual_stereo_rsv = total >= 1 << 3 ? 1 << 3 : 0;
            total -= dual_stereo_rsv;
        }
    }
    LFOR(L, j, start, end) {
        thresh[j] = imax(C << 3, (3 * (eB[j + 1] - eB[j]) << LM << 3) >> 4);
        trim_offset[j] = C * (eB[j + 1] - eB[j]) * (alloc_trim - 5 - LM) * (end - j - 1) * (1 << (LM + 3)) >> 6;
        if ((eB[j + 1] - eB[j]) << LM == 1) trim_offset[j] -= C << 3;
    }
    lsync(L);
    int lo = 1, hi = T_CELT_NBALLOCV - 1;
    ROLLED do {
        int mid = (lo + hi) >> 1;
        const int32_t psum = alloc_sum(L, start, end, thresh, cap, C << 3, [&](int j) CUO_INLINE {
            int bitsj = C * (eB[j + 1] - eB[j]) * T_celt_allocVectors[mid * CELT_NB + j] << LM >> 2;
            if (bitsj > 0) bitsj = imax(0, bitsj + trim_offset[j]);
            return bitsj + offsets[j];
        });
        if (psum > total) hi = mid - 1;
        else lo = mid + 1;
    } while (lo <= hi);
    hi = lo--;
    int boosted = -1;
    LFOR(L, j, start, end) {
        int N = eB[j + 1] - eB[j];
        int bits1j = C * N * T_celt_allocVectors[lo * CELT_NB + j] << LM >> 2;
        int bits2j = hi >= T_CELT_NBALLOCV ? cap[j] : C * N * T_celt_allocVectors[hi * CELT_NB + j] << LM >> 2;
        if (bits1j > 0) bits1j = imax(0, bits1j + trim_offset[j]);
        if (bits2j > 0) bits2j = imax(0, bits2j + trim_offset[j]);
        if (lo > 0) bits1j += offsets[j];
        bits2j += offsets[j];
        if (offsets[j] > 0) boosted = imax(boosted, j);
        bits2j = imax(0, bits2j - bits1j);
        bits1[j] = bits1j;
        bits2[j] = bits2j;
    }
    const int skip_start = imax(start, lmax(L, boosted));
    lsync(L);
    const int coded = interp_bits2pulses(L, start, end, skip_start, bits1, bits2, thresh, cap, total, balance,
                                         skip_rsv, intensity, intensity_rsv, dual_stereo, dual_stereo_rsv, pulses,
                                         ebits, fine_priority, C, LM, &d);
    *rd = d;
    return coded;
}

// ------------------------------------------------------------------ PVQ

DFN uint32_t pvq_u(int n, int k)
{
    int a = imin(n, k), b = imax(n, k);
    return T_celt_pvq_u_data[T_celt_pvq_u_row[a] + b];
}
DFN uint32_t pvq_v(int n, int k) { return pvq_u(n, k) + pvq_u(n, k + 1); }
DFN uint32_t pvq_row(int r, int c) { return T_celt_pvq_u_data[T_celt_pvq_u_row[r] + c]; }

// celt/cwrs.c cwrsi: combinatorial index -> pulse vector; returns sum of squares.
// With fewer pulses than positions most positions stay empty, so the two counts
// that decide the next position are loaded while this one is decided, for the
// case that it stays empty; with no pulse left (idx is 0 then) zeros follow.
DNI int32_t cwrsi(int n, int k, uint32_t idx, int32_t *y)
{
    uint32_t p, q;
    int s, k0, rows = -1;   // rows: the k that row and row1 are for
    int16_t val;
    int32_t yy = 0;
    const uint32_t *row = T_celt_pvq_u_data, *row1 = row;
    uint32_t pn = 0, qn = 0;
    ROLLED while (n > 2) {
        if (k >= n) {
            const uint32_t *rn = T_celt_pvq_u_data + T_celt_pvq_u_row[n];
            p = rn[k + 1];
            s = -(idx >= p);
            idx -= p & s;
            k0 = k;
            if (rn[n] > idx) {
                k = n;
                ROLLED do p = pvq_row(--k, n);
                while (p > idx);
            } else {
                ROLLED for (p = rn[k]; p > idx; p = rn[k]) k--;
            }
            idx -= p;
            val = (int16_t)((k0 - k + s) ^ s);
            *y++ = val;
            yy = c_mac16(yy, val, val);
        } else {
            if (k == 0) {
                ROLLED for (; n > 0; n--) *y++ = 0;
                return yy;
            }
            if (rows != k) {
                rows = k;
                row = T_celt_pvq_u_data + T_celt_pvq_u_row[k];
                row1 = T_celt_pvq_u_data + T_celt_pvq_u_row[k + 1];
                pn = row[n];
                qn = row1[n];
            }
            p = pn;
            q = qn;
            pn = row[n - 1];
            qn = row1[n - 1];   // not a count when n - 1 == k, and not used then
            if (p <= idx && idx < q) {
                idx -= p;
                *y++ = 0;
            } else {
                s = -(idx >= q);
                idx -= q & s;
                k0 = k;
                ROLLED do p = pvq_row(--k, n);
                while (p > idx);
                idx -= p;
                val = (int16_t)((k0 - k + s) ^ s);
                *y++ = val;
                yy = c_mac16(yy, val, val);
            }
        }
        n--;
    }
    p = 2 * k + 1;
    s = -(idx >= p);
    idx -= p & s;
    k0 = k;
    k = (idx + 1) >> 1;
    if (k) idx -= 2 * k - 1;
    val = (int16_t)((k0 - k + s) ^ s);
    *y++ = val;
    yy = c_mac16(yy, val, val);
    s = -(int)idx;
    val = (int16_t)((k + s) ^ s);
    *y = val;
    yy = c_mac16(yy, val, val);
    return yy;
}

// celt/vq.c exp_rotation1 on one residue class.  Each pass rotates the pairs
// (X[i], X[i + stride]) in order, and pair i + stride reads the element pair i
// has just written: the pass is `stride` independent recurrences, one per
// residue class r of i mod stride, which the lanes share out.  A class's
// carried element stays in a register; its other inputs are loaded four
// ahead.  The coefficients come doubled: the rounded product sums are then the
// high halves of wrap-around 32-bit sums ((v << 1) >> 16 is (int16_t)(v >> 15)),
// so a step waits for one multiply-add and one shift.
DFN void exp_rotation_class(int16_t *X, int len, int stride, int32_t c, int32_t s, int r)
{
    const int32_t c2 = 2 * c, s2 = 2 * s, rnd = 32768;
    const int n = (len - r + stride - 1) / stride - 1;   // pairs of the class
    if (n <= 0) return;
    int16_t *x = X + r;
    // forward: pairs 0 .. n - 1
    auto fwd = [&](int i, int32_t x2, int32_t &x1) CUO_INLINE {
        x[i * stride] = (int16_t)(wadd(wadd(wmul(c2, x1), rnd), -wmul(s2, x2)) >> 16);
        x1 = wadd(wadd(wmul(c2, x2), rnd), wmul(s2, x1)) >> 16;
    };
    int32_t x1 = x[0], v[4];
#pragma unroll
    for (int j = 0; j < 4; j++) v[j] = x[imin(j + 1, n) * stride];
    int i = 0;
    ROLLED for (; i + 4 <= n; i += 4) {
        int32_t u[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            u[j] = v[j];
            v[j] = x[imin(i + j + 5, n) * stride];
        }
#pragma unroll
        for (int j = 0; j < 4; j++) fwd(i + j, u[j], x1);
    }
    if (i < n) fwd(i, v[0], x1);
    if (i + 1 < n) fwd(i + 1, v[1], x1);
    if (i + 2 < n) fwd(i + 2, v[2], x1);
    x[n * stride] = (int16_t)x1;
    // backward: pairs n - 2 .. 0 (libopus's second pass starts at len - 2 stride - 1)
    if (n < 2) return;
    auto bwd = [&](int i, int32_t w, int32_t &x2) CUO_INLINE {
        x[(i + 1) * stride] = (int16_t)(wadd(wadd(wmul(c2, x2), rnd), wmul(s2, w)) >> 16);
        x2 = wadd(wadd(wmul(c2, w), rnd), -wmul(s2, x2)) >> 16;
    };
    int32_t x2 = x[(n - 1) * stride];
    i = n - 2;
#pragma unroll
    for (int j = 0; j < 4; j++) v[j] = x[imax(i - j, 0) * stride];
    ROLLED for (; i >= 3; i -= 4) {
        int32_t u[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            u[j] = v[j];
            v[j] = x[imax(i - j - 4, 0) * stride];
        }
#pragma unroll
        for (int j = 0; j < 4; j++) bwd(i - j, u[j], x2);
    }
    if (i >= 0) bwd(i, v[0], x2);
    if (i >= 1) bwd(i - 1, v[1], x2);
    if (i >= 2) bwd(i - 2, v[2], x2);
    x[0] = (int16_t)x2;
}

// celt/vq.c exp_rotation, dir = -1 (decoder)
DNI void exp_rotation_dec(Lanes L, int16_t *X, int len, int stride, int K, int spread)
{
    if (2 * K >= len || spread == SPREAD_NONE) return;
    int factor = spread == 1 ? 15 : spread == 2 ? 10 : 5;   // SPREAD_FACTOR[spread - 1] = {15, 10, 5}
    int16_t gain = (int16_t)c_mul32_q31(c_mul16(32767, len), c_rcp(len + factor * K));
    int16_t theta = (int16_t)(c_mul16_q15(gain, gain) >> 1);
    int16_t c = c_cos_norm(theta);
    int16_t s = c_cos_norm((int16_t)(32767 - theta));
    int stride2 = 0;
    if (len >= 8 * stride) {
        stride2 = 1;
        ROLLED while ((stride2 * stride2 + stride2) * stride + (stride >> 2) < len) stride2++;
    }
    len = (int)((unsigned)len / (unsigned)stride);
    // first the residue classes of stride2 with the coefficients swapped, then
    // the whole blocks
    ROLLED for (int pass = stride2 ? 0 : 1; pass < 2; pass++) {
        const int st = pass ? 1 : stride2;
        ROLLED for (int q = L.id; q < stride * st; q += L.n) {
            const int i = pass ? q : (int)((unsigned)q / (unsigned)st);
            exp_rotation_class(X + i * len, len, st, pass ? c : s, pass ? s : c, q - i * st);
        }
        lsync(L);
    }
}

// celt/vq.c renormalise_vector
// (the energy is a wrap-around sum, so the lanes' partial sums give the serial
// value; every element is scaled on its own)
DNI void renormalise_vector(Lanes L, int16_t *X, int N, int16_t gain)
{
    PHASE_BEGIN(t_rn);
    int32_t E = 0;
    LFOR(L, i, 0, N) E = c_mac16(E, X[i], X[i]);
    E = wadd(lsum(L, E), 1);
    int k = c_ilog2(E) >> 1;
    int32_t t = c_vshr(E, 2 * (k - 7));
    int16_t g = (int16_t)c_mul16_p15(c_rsqrt_norm(t), gain);
    LFOR(L, i, 0, N) X[i] = (int16_t)c_pshr(c_mul16(g, X[i]), k + 1);
    lsync(L);
    PHASE_END(PH_PVQ_RENORM, t_rn, L.id);
}

// celt/vq.c alg_unquant.  Every lane decodes the codeword (same index, same
// pulses) and the lanes share out the vector work.
DFN unsigned alg_unquant(const Lanes &L, int16_t *X, int N, int K, int spread, int B, RangeDec *dec, int16_t gain,
                         int32_t *iy)
{
    PHASE_BEGIN(t_cw);
    const uint32_t idx = rd_uint(dec, pvq_v(N, K));
    lsync(L);   // every lane is done with the last partition's pulses
    int32_t Ryy = cwrsi(N, K, idx, iy);
    PHASE_END(PH_PVQ_CWRSI, t_cw, L.id);
    // normalise_residual (every element on its own)
    int k = c_ilog2(Ryy) >> 1;
    int32_t t = c_vshr(Ryy, 2 * (k - 7));
    int16_t g = (int16_t)c_mul16_p15(c_rsqrt_norm(t), gain);
    lsync(L);
    LFOR(L, i, 0, N) X[i] = (int16_t)c_pshr(c_mul16(g, iy[i]), k + 1);
    lsync(L);
    PHASE_BEGIN(t_rt);
    exp_rotation_dec(L, X, N, B, K, spread);
    PHASE_END(PH_PVQ_ROT, t_rt, L.id);
    // extract_collapse_mask
    if (B <= 1) return 1;
    const int N0 = (int)((unsigned)N / (unsigned)B);
    unsigned mask = 0;
    LFOR(L, i, 0, N) if (iy[i]) mask |= 1u << (i / N0);
    return lor(L, mask);
}

// ------------------------------------------------------------------ bands

DFN int16_t bitexact_cos(int16_t x)
{
    int32_t tmp = (4096 + (int32_t)x * x) >> 13;
    int16_t x2 = (int16_t)tmp;
    x2 = (int16_t)((32767 - x2) + c_frac_mul16(x2, (-7651 + c_frac_mul16(x2, (8277 + c_frac_mul16(-626, x2))))));
    return (int16_t)(1 + x2);
}

DFN int bitexact_log2tan(int isin, int icos)
{
    int lc = ilog((uint32_t)icos), ls = ilog((uint32_t)isin);
    icos <<= 15 - lc;
    isin <<= 15 - ls;
    return (ls - lc) * (1 << 11) + c_frac_mul16(isin, c_frac_mul16(isin, -2597) + 7932) -
           c_frac_mul16(icos, c_frac_mul16(icos, -2597) + 7932);
}

// In place over independent pairs: the lanes split them.
DNI void haar1(Lanes L, int16_t *X, int N0, int stride)
{
    LFOR(L, q, 0, (N0 >> 1) * stride) {
        const int j = q / stride, i = q - j * stride;
        int16_t *x = X + stride * 2 * j + i;
        int32_t t1 = c_mul16(23170, x[0]);
        int32_t t2 = c_mul16(23170, x[stride]);
        x[0] = (int16_t)c_pshr(wadd(t1, t2), 15);
        x[stride] = (int16_t)c_pshr(wsub(t1, t2), 15);
    }
    lsync(L);
}

// celt/bands.c deinterleave_hadamard (to = 1) and interleave_hadamard (to = 0)
DNI void hadamard_order(Lanes L, int16_t *X, int N0, int stride, int hadamard, int to, int16_t *tmp)
{
    const int32_t *ordery = T_celt_ordery_table + stride - 2;
    const int N = N0 * stride;
    LFOR(L, q, 0, N) {
        const int j = q / stride, i = q - j * stride;       // element i of group j, interleaved at q
        const int at = (hadamard ? ordery[i] : i) * N0 + j;   // its place with the blocks apart
        tmp[to ? at : q] = X[to ? q : at];
    }
    lsync(L);
    LFOR(L, i, 0, N) X[i] = tmp[i];
    lsync(L);
}

// Band decoding runs on every lane of the group: each lane decodes the same
// symbols from its own copy of the range decoder and the lanes share out the
// work on the band vectors.  The loop over the bands is the kernel's largest
// and what it costs above all is instruction fetch (an SM's first instruction
// cache holds a part of it), so everything a band does once or twice is a call
// and every inlined piece has one call site: 29 KB of code, where everything
// inlined came to 53 KB and decoded no faster (12 stereo files 60.3 ms against
// 58.5 now, 30 files to int16 115 against 108).
struct BandCtx {
    Lanes L;
    RangeDec *d;
    int i;
    int intensity;
    int spread;
    int tf_change;
    int32_t remaining_bits;
    uint32_t seed;
    int disable_inv;
    CeltScratch *w;
};

struct SplitCtx {
    int inv, imid, iside, delta, itheta, qalloc;
};

// exp2_table8 of celt/bands.c compute_qn
TABC(int16_t, T_exp2_table8[8]) = {16384, 17866, 19483, 21247, 23170, 25267, 27554, 30048};

DFN int compute_qn(int N, int b, int offset, int pulse_cap, int stereo)
{
    const int16_t *exp2_table8 = T_exp2_table8;
    int N2 = 2 * N - 1;
    if (stereo && N == 2) N2--;
    int qb = (b + N2 * offset) / N2;
    qb = imin(b - pulse_cap - (4 << 3), qb);
    qb = imin(8 << 3, qb);
    int qn;
    if (qb < (1 << 3 >> 1)) {
        qn = 1;
    } else {
        qn = exp2_table8[qb & 0x7] >> (14 - (qb >> 3));
        qn = (qn + 1) >> 1 << 1;
    }
    return qn;
}

// celt/bands.c compute_theta (decoder side).  may_invert: bit 0, there are bits
// left for the inversion flag; bit 1, the flag counts.
DNI void compute_theta(RangeDec *ec, SplitCtx *sctx, int i, int intensity, int may_invert, int N, int *b, int B,
                       int B0, int LM, int stereo, int *fill)
{
    int itheta = 0, delta, imid, iside, inv = 0;
    int pulse_cap = T_celt_logN[i] + LM * (1 << 3);
    int offset = (pulse_cap >> 1) - (stereo && N == 2 ? 16 : 4);
    int qn = compute_qn(N, *b, offset, pulse_cap, stereo);
    if (stereo && i >= intensity) qn = 1;
    int32_t tell = (int32_t)rd_tell_frac(ec);
    if (qn != 1) {
        // the three models of the angle: a step, uniform, a triangle; each is
        // one decode of a total and one update with the range it falls in
        const int step = stereo && N > 2, uniform = !step && (B0 > 1 || stereo);
        const int x0 = qn / 2, half = qn >> 1;
        if (uniform && qn + 1 > 256) {   // more than eight bits: part of them raw
            itheta = (int)rd_uint(ec, qn + 1);
        } else {
            const unsigned ft = step ? (unsigned)(3 * (x0 + 1) + x0) : uniform ? (unsigned)(qn + 1)
                                                                               : (unsigned)((half + 1) * (half + 1));
            const int fm = (int)rd_decode(ec, ft);
            unsigned fl, fh;
            if (step) {
                const int p0 = 3;
                itheta = fm < (x0 + 1) * p0 ? fm / p0 : x0 + 1 + (fm - (x0 + 1) * p0);
                fl = itheta <= x0 ? p0 * itheta : (itheta - 1 - x0) + (x0 + 1) * p0;
                fh = itheta <= x0 ? p0 * (itheta + 1) : (itheta - x0) + (x0 + 1) * p0;
            } else if (uniform) {
                itheta = fm;
                fl = fm;
                fh = fm + 1;
            } else {
                const int low = fm < (half * (half + 1) >> 1);
                const int root = (int)c_isqrt32(8 * (uint32_t)(low ? fm : (int)ft - fm - 1) + 1);
                int fs;
                if (low) {
                    itheta = (root - 1) >> 1;
                    fs = itheta + 1;
                    fl = itheta * (itheta + 1) >> 1;
                } else {
                    itheta = (2 * (qn + 1) - root) >> 1;
                    fs = qn + 1 - itheta;
                    fl = ft - ((qn + 1 - itheta) * (qn + 2 - itheta) >> 1);
                }
                fh = fl + fs;
            }
            rd_update(ec, fl, fh, ft);
        }
        itheta = (int)((uint32_t)((int32_t)itheta * 16384) / (uint32_t)qn);
    } else if (stereo) {
        if (*b > 2 << 3 && (may_invert & 1)) inv = rd_bit_logp(ec, 2);
        if (!(may_invert & 2)) inv = 0;
        itheta = 0;
    }
    int qalloc = (int)rd_tell_frac(ec) - tell;
    *b -= qalloc;
    if (itheta == 0) {
        imid = 32767; iside = 0;
        *fill &= (1 << B) - 1;
        delta = -16384;
    } else if (itheta == 16384) {
        imid = 0; iside = 32767;
        *fill &= ((1 << B) - 1) << B;
        delta = 16384;
    } else {
        imid = bitexact_cos((int16_t)itheta);
        iside = bitexact_cos((int16_t)(16384 - itheta));
        delta = c_frac_mul16((N - 1) << 7, bitexact_log2tan(iside, imid));
    }
    sctx->inv = inv; sctx->imid = imid; sctx->iside = iside;
    sctx->delta = delta; sctx->itheta = itheta; sctx->qalloc = qalloc;
}

// celt/bands.c quant_band_n1; returns the bits left.  Ends with a barrier: the
// group's lanes may read X, Y and lowband_out.
DNI int quant_band_n1(Lanes L, RangeDec *d, int remaining_bits, int16_t *X, int16_t *Y, int16_t *lowband_out)
{
    int sign[2] = {0, 0};
    ROLLED for (int c = 0; c < 1 + (Y != 0); c++) {
        if (remaining_bits >= 1 << 3) {
            const int v = (int)rd_bits(d, 1);
            if (c) sign[1] = v;
            else sign[0] = v;
            remaining_bits -= 1 << 3;
        }
    }
    lead(L, [&]() CUO_INLINE {
        X[0] = sign[0] ? -16384 : 16384;
        if (Y) Y[0] = sign[1] ? -16384 : 16384;
        if (lowband_out) lowband_out[0] = (int16_t)(X[0] >> 4);
    });
    return remaining_bits;
}

// celt/bands.c celt_lcg_rand k steps on is the affine map seed -> a[k] seed +
// c[k] mod 2^32; k up to the longest band.
struct LcgPowers {
    uint32_t a[177], c[177];
    constexpr LcgPowers() : a(), c()
    {
        a[0] = 1;
        c[0] = 0;
        for (int k = 1; k < 177; k++) {
            a[k] = 1664525u * a[k - 1];
            c[k] = 1664525u * c[k - 1] + 1013904223u;
        }
    }
};
TABG(LcgPowers, T_lcg) = LcgPowers();

// celt/bands.c quant_partition, leaf: pulses for the band piece (PVQ) or,
// with none, folding / noise fill.
DFN unsigned quant_partition_leaf(BandCtx &ctx, int16_t *X, int N, int b, int B, int16_t *lowband, int LM,
                                  int16_t gain, int fill)
{
    const int i = ctx.i;
    unsigned cm = 0;
    int q = bits2pulses(i, LM, b);
    int curr_bits = pulses2bits(i, LM, q);
    ctx.remaining_bits -= curr_bits;
    ROLLED while (ctx.remaining_bits < 0 && q > 0) {
        ctx.remaining_bits += curr_bits;
        q--;
        curr_bits = pulses2bits(i, LM, q);
        ctx.remaining_bits -= curr_bits;
    }
    if (q != 0) {
        int K = get_pulses(q);
        cm = alg_unquant(ctx.L, X, N, K, ctx.spread, B, ctx.d, gain, ctx.w->iy);
    } else {
        unsigned cm_mask = (unsigned)(1UL << B) - 1;
        fill &= cm_mask;
        if (!fill) {
            LFOR(ctx.L, j, 0, N) X[j] = 0;
            lsync(ctx.L);
        } else {
            // sample j takes the seed j + 1 steps on
            LFOR(ctx.L, j, 0, N) {
                const uint32_t seed = T_lcg.a[j + 1] * ctx.seed + T_lcg.c[j + 1];
                if (lowband == 0) {
                    X[j] = (int16_t)((int32_t)seed >> 20);
                } else {
                    int16_t tmp = (seed & 0x8000) ? 4 : -4;   // QCONST16(1.0f/256, 10)
                    X[j] = (int16_t)(lowband[j] + tmp);
                }
            }
            ctx.seed = T_lcg.a[N] * ctx.seed + T_lcg.c[N];
            cm = lowband == 0 ? cm_mask : fill;
            lsync(ctx.L);
            renormalise_vector(ctx.L, X, N, gain);
        }
    }
    return cm;
}

// celt/bands.c quant_partition.  libopus recurses into the two halves of a
// split band; here one loop walks down to a leaf and back up, so a single copy
// of the code serves every depth (the split depth is bounded by LM + 1 <= 4).
// What the second half of a split needs is kept in the group's memory, written
// once when the band splits; the collapse mask of the first half (8 bits per
// depth) and which halves are done are registers.  The bit rebalancing between
// the halves and the collapse-mask combination happen in libopus's order.
DFN unsigned quant_partition(BandCtx &ctx, int16_t *X, int N, int b, int B, int16_t *lowband, int LM,
                             int16_t gain, int fill)
{
    QPSplit *st = ctx.w->qp;
    const Lanes &L = ctx.L;
    const int i = ctx.i;
    int sp = 0;                          // splits above the current piece
    unsigned second = 0, cms = 0;        // bit d: split d is in its second half; byte d: first half's mask
    ROLLED while (1) {
        // down: split while the piece has more bits than one codeword takes
        const uint8_t *cache = pulse_cache(i, LM);
        if (LM != -1 && b > cache[cache[0]] + 12 && N > 2 && sp < 4) {
            SplitCtx sctx;
            const int B0 = B, n2 = N >> 1, parent_gain = gain;
            N = n2;
            if (B == 1) fill = (fill & 1) | (fill << 1);
            B = (B + 1) >> 1;
            LM--;
            PHASE_BEGIN(t_th);
            compute_theta(ctx.d, &sctx, i, ctx.intensity, 0, N, &b, B, B0, LM, 0, &fill);
            PHASE_END(PH_PVQ_THETA, t_th, L.id);
            int delta = sctx.delta;
            const int itheta = sctx.itheta;
            if (B0 > 1 && (itheta & 0x3fff)) {
                if (itheta > 8192) delta -= delta >> (4 - LM);
                else delta = imin(0, delta + (N << 3 >> (5 - LM)));
            }
            const int mbits = imax(0, imin(b, (b - delta) / 2));
            const int sbits = b - mbits;
            ctx.remaining_bits -= sctx.qalloc;
            const int mid_first = mbits >= sbits;
            const int16_t gmid = (int16_t)c_mul16_p15(parent_gain, (int16_t)sctx.imid);
            const int16_t gside = (int16_t)c_mul16_p15(parent_gain, (int16_t)sctx.iside);
            int16_t *const Y = X + N, *const lowband2 = lowband ? lowband + N : 0;
            QPSplit *f = &st[sp];
            lsync(L);   // every lane has read what an earlier split left here
            f->X = mid_first ? Y : X;
            f->lowband = mid_first ? lowband2 : lowband;
            f->bits = mid_first ? sbits : mbits;
            f->first_bits = mid_first ? mbits : sbits;
            f->rebalance = ctx.remaining_bits;
            f->N = N;
            f->B = B;
            f->B0 = B0;
            f->LM = LM;
            f->fill = mid_first ? fill >> B : fill;
            f->gain = mid_first ? gside : gmid;
            f->mid_first = mid_first;
            // no rebalancing towards a half that gets no energy
            f->fixed = mid_first ? itheta == 0 : itheta == 16384;
            lsync(L);
            if (!mid_first) {
                X = Y;
                lowband = lowband2;
                fill >>= B;
            }
            b = mid_first ? mbits : sbits;
            gain = mid_first ? gmid : gside;
            second &= ~(1u << sp);
            sp++;
            continue;
        }
        unsigned cm = quant_partition_leaf(ctx, X, N, b, B, lowband, LM, gain, fill);
        // up: to the nearest split whose second half is still to come
        ROLLED while (sp > 0 && (second >> (sp - 1) & 1)) {
            sp--;
            const unsigned first = cms >> (8 * sp) & 0xff;
            const int shift = st[sp].B0 >> 1;
            cm = st[sp].mid_first ? first | cm << shift : first << shift | cm;
        }
        if (sp == 0) return cm;
        const QPSplit *f = &st[sp - 1];
        X = f->X;
        lowband = f->lowband;
        N = f->N;
        B = f->B;
        LM = f->LM;
        fill = f->fill;
        gain = f->gain;
        b = f->bits;
        const int32_t rebalance = f->first_bits - (f->rebalance - ctx.remaining_bits);
        if (rebalance > 3 << 3 && !f->fixed) b += rebalance - (3 << 3);
        cms = (cms & ~(0xffu << (8 * (sp - 1)))) | (cm & 0xff) << (8 * (sp - 1));
        second |= 1u << (sp - 1);
    }
}

// bit_interleave_table / bit_deinterleave_table of celt/bands.c quant_band
TABC(uint8_t, T_bit_interleave[16]) = {0, 1, 1, 1, 2, 3, 3, 3, 2, 3, 3, 3, 2, 3, 3, 3};
TABC(uint8_t, T_bit_deinterleave[16]) = {0x00, 0x03, 0x0C, 0x0F, 0x30, 0x33, 0x3C, 0x3F,
                                         0xC0, 0xC3, 0xCC, 0xCF, 0xF0, 0xF3, 0xFC, 0xFF};

// celt/bands.c quant_band (decoder, resynth always on).  Ends with a barrier.
DFN unsigned quant_band(BandCtx &ctx, int16_t *X, int N, int b, int B, int16_t *lowband, int LM,
                        int16_t *lowband_out, int16_t gain, int16_t *lowband_scratch, int fill)
{
    const Lanes &L = ctx.L;
    const uint8_t *bit_interleave_table = T_bit_interleave;
    const uint8_t *bit_deinterleave_table = T_bit_deinterleave;
    int N0 = N, N_B = N, N_B0, B0 = B, time_divide = 0, recombine = 0;
    int longBlocks = B0 == 1;
    unsigned cm = 0;
    int tf_change = ctx.tf_change;
    N_B = (int)((unsigned)N_B / (unsigned)B);
    if (N == 1) {
        ctx.remaining_bits = quant_band_n1(L, ctx.d, ctx.remaining_bits, X, 0, lowband_out);
        return 1;
    }
    if (tf_change > 0) recombine = tf_change;
    PHASE_BEGIN(t_tf);
    if (lowband_scratch && lowband && (recombine || ((N_B & 1) == 0 && tf_change < 0) || B0 > 1)) {
        LFOR(L, j, 0, N) lowband_scratch[j] = lowband[j];
        lsync(L);
        lowband = lowband_scratch;
    }
    ROLLED for (int k = 0; k < recombine; k++) {
        if (lowband) haar1(L, lowband, N >> k, 1 << k);
        fill = bit_interleave_table[fill & 0xF] | bit_interleave_table[fill >> 4] << 2;
    }
    B >>= recombine;
    N_B <<= recombine;
    ROLLED while ((N_B & 1) == 0 && tf_change < 0) {
        if (lowband) haar1(L, lowband, N_B, B);
        fill |= fill << B;
        B <<= 1;
        N_B >>= 1;
        time_divide++;
        tf_change++;
    }
    B0 = B;
    N_B0 = N_B;
    if (B0 > 1 && lowband)
        hadamard_order(L, lowband, N_B >> recombine, B0 << recombine, longBlocks, 1, ctx.w->tmp);
    PHASE_END(PH_PVQ_TF, t_tf, L.id);
    cm = quant_partition(ctx, X, N, b, B, lowband, LM, gain, fill);
    PHASE_BEGIN(t_tf2);
    if (B0 > 1) hadamard_order(L, X, N_B >> recombine, B0 << recombine, longBlocks, 0, ctx.w->tmp);
    N_B = N_B0;
    B = B0;
    ROLLED for (int k = 0; k < time_divide; k++) {
        B >>= 1;
        N_B <<= 1;
        cm |= cm >> B;
        haar1(L, X, N_B, B);
    }
    ROLLED for (int k = 0; k < recombine; k++) {
        cm = bit_deinterleave_table[cm];
        haar1(L, X, N0 >> k, 1 << k);
    }
    PHASE_END(PH_PVQ_TF, t_tf2, L.id);
    B <<= recombine;
    if (lowband_out) {
        int16_t n = (int16_t)c_sqrt(shl32(N0, 22));
        LFOR(L, j, 0, N0) lowband_out[j] = (int16_t)c_mul16_q15(n, X[j]);
        lsync(L);
    }
    cm &= (1 << B) - 1;
    return cm;
}

// (the two dot products are wrap-around sums, so the lanes' partial sums give
// the serial values; every element is mixed on its own)
DNI void stereo_merge(Lanes L, int16_t *X, int16_t *Y, int16_t mid, int N)
{
    int32_t xp = 0, side = 0;
    LFOR(L, j, 0, N) {
        xp = c_mac16(xp, Y[j], X[j]);
        side = c_mac16(side, Y[j], Y[j]);
    }
    xp = lsum(L, xp);
    side = lsum(L, side);
    xp = c_mul16_32_q15(mid, xp);
    int16_t mid2 = (int16_t)(mid >> 1);
    int32_t El = wsub(wadd(c_mul16(mid2, mid2), side), 2 * xp);
    int32_t Er = wadd(wadd(c_mul16(mid2, mid2), side), 2 * xp);
    if (Er < 161061 || El < 161061) {   // QCONST32(6e-4f, 28)
        LFOR(L, j, 0, N) Y[j] = X[j];
        lsync(L);
        return;
    }
    int kl = c_ilog2(El) >> 1, kr = c_ilog2(Er) >> 1;
    int32_t t = c_vshr(El, (kl - 7) << 1);
    int16_t lgain = c_rsqrt_norm(t);
    t = c_vshr(Er, (kr - 7) << 1);
    int16_t rgain = c_rsqrt_norm(t);
    if (kl < 7) kl = 7;
    if (kr < 7) kr = 7;
    LFOR(L, j, 0, N) {
        int16_t l = (int16_t)c_mul16_p15(mid, X[j]);
        int16_t r = Y[j];
        X[j] = (int16_t)c_pshr(c_mul16(lgain, (int16_t)(l - r)), kl + 1);
        Y[j] = (int16_t)c_pshr(c_mul16(rgain, (int16_t)(l + r)), kr + 1);
    }
    lsync(L);
}

// celt/bands.c quant_all_bands, decoder path (encode = 0, resynth = 1, no theta
// RDO), with quant_band_stereo.  A band takes one pass through quant_band or
// two: mono, stereo of two samples and a band coded mid only: X; dual stereo: X
// then Y; mid / side stereo: whichever half has more bits, then the other.
// One call site serves them all.
DNI void quant_all_bands_dec(Lanes L, int start, int end, int16_t *X_, int16_t *Y_, uint8_t *collapse_masks,
                             const int32_t *pulses, int shortBlocks, int spread, int dual_stereo, int intensity,
                             const int32_t *tf_res, int32_t total_bits, int32_t balance, RangeDec *ec, int LM,
                             int codedBands, uint32_t *seed, int disable_inv, CeltScratch *w)
{
    const int16_t *eB = T_celt_eBands;
    int M = 1 << LM;
    int B = shortBlocks ? M : 1;
    int norm_offset = M * eB[start];
    int C = Y_ != 0 ? 2 : 1;
    int16_t *norm = w->norm;
    int16_t *norm2 = norm + M * eB[CELT_NB - 1] - norm_offset;
    int16_t *lowband_scratch = X_ + M * eB[T_CELT_EFFEBANDS - 1];
    int lowband_offset = 0, update_lowband = 1;
    BandCtx ctx;
    ctx.L = L;
    ctx.d = ec;
    ctx.intensity = intensity;
    ctx.seed = *seed;
    ctx.spread = spread;
    ctx.disable_inv = disable_inv;
    ctx.w = w;
    ROLLED for (int i = start; i < end; i++) {
        int effective_lowband = -1;
        unsigned x_cm, y_cm;
        ctx.i = i;
        int last = i == end - 1;
        int16_t *X = X_ + M * eB[i];
        int16_t *Y = Y_ != 0 ? Y_ + M * eB[i] : 0;
        int N = M * eB[i + 1] - M * eB[i];
        int32_t tell = (int32_t)rd_tell_frac(ec);
        if (i != start) balance -= tell;
        int32_t remaining_bits = total_bits - tell - 1;
        ctx.remaining_bits = remaining_bits;
        int b;
        if (i <= codedBands - 1) {
            const int share = codedBands - i;
            int32_t curr_balance = share >= 3 ? balance / 3 : share == 2 ? balance / 2 : balance;
            b = imax(0, imin(16383, imin(remaining_bits + 1, pulses[i] + curr_balance)));
        } else {
            b = 0;
        }
        if ((M * eB[i] - N >= M * eB[start] || i == start + 1) && (update_lowband || lowband_offset == 0))
            lowband_offset = i;
        if (i == start + 1) {
            // special_hybrid_folding
            int n1 = M * (eB[start + 1] - eB[start]);
            int n2 = M * (eB[start + 2] - eB[start + 1]);
            // the copied range starts where the copy's source ends or later
            LFOR(L, j, 0, n2 - n1) {
                norm[n1 + j] = norm[2 * n1 - n2 + j];
                if (dual_stereo) norm2[n1 + j] = norm2[2 * n1 - n2 + j];
            }
            lsync(L);
        }
        int tf_change = tf_res[i];
        ctx.tf_change = tf_change;
        if (i >= T_CELT_EFFEBANDS) {
            X = norm;
            if (Y_ != 0) Y = norm;
            lowband_scratch = 0;
        }
        if (last) lowband_scratch = 0;
        // (a band of one bin takes a sign and neither folds nor looks at the masks)
        if (N > 1 && lowband_offset != 0 && (spread != SPREAD_AGGRESSIVE || B > 1 || tf_change < 0)) {
            effective_lowband = imax(0, M * eB[lowband_offset] - norm_offset - N);
            // the bands the folding source covers, from the lowest at or below its
            // first bin to the one its last bin is in (of the bands decoded)
            const int first = effective_lowband + norm_offset;
            const int fold_start = imin(lowband_offset - 1, T_band_of.b[first >> LM]);
            const int fold_end = imin(i, imax(lowband_offset, T_band_of.b[(first + N - 1) >> LM] + 1));
            x_cm = y_cm = 0;
            int fold_i = fold_start;
            ROLLED do {
                x_cm |= collapse_masks[fold_i * C + 0];
                y_cm |= collapse_masks[fold_i * C + C - 1];
            } while (++fold_i < fold_end);
        } else {
            x_cm = y_cm = (1 << B) - 1;
        }
        if (dual_stereo && i == intensity) {
            dual_stereo = 0;
            lsync(L);
            LFOR(L, j, 0, M * eB[i] - norm_offset) norm[j] = (int16_t)((norm[j] + norm2[j]) >> 1);
            lsync(L);
        }
        int16_t *const lowband = effective_lowband != -1 ? norm + effective_lowband : 0;
        int16_t *const lowband_out = last ? 0 : norm + M * eB[i] - norm_offset;
        const int orig_fill = (int)(x_cm | y_cm);
        if (Y != 0 && !dual_stereo && N == 1) {
            ctx.remaining_bits = quant_band_n1(L, ctx.d, ctx.remaining_bits, X, Y, lowband_out);
            x_cm = y_cm = 1;
        } else {
            // the passes: vector, bits, folding source and target, gain, fill
            int16_t *px = X, *plow = lowband, *pout = lowband_out, *pscratch = lowband_scratch;
            int pb = b, pfill = orig_fill, passes = 1, mid_first = 1, second_bits = 0;
            int16_t pgain = 32767;
            SplitCtx sctx = {0, 0, 0, 0, 0, 0};
            int sign = 0, fill = orig_fill;
            int32_t rebalance = 0;
            if (dual_stereo) {
                pb = b / 2;
                pfill = (int)x_cm;
                passes = 2;
            } else if (Y != 0) {
                int left = b;   // without the angle's bits
                PHASE_BEGIN(t_th);
                compute_theta(ctx.d, &sctx, i, ctx.intensity, (ctx.remaining_bits > 2 << 3) | (ctx.disable_inv ? 0 : 2), N,
                              &left, B, B, LM, 1, &fill);
                PHASE_END(PH_PVQ_THETA, t_th, L.id);
                if (N == 2) {
                    int sbits = 0;
                    if (sctx.itheta != 0 && sctx.itheta != 16384) sbits = 1 << 3;
                    pb = left - sbits;
                    ctx.remaining_bits -= sctx.qalloc + sbits;
                    px = sctx.itheta > 8192 ? Y : X;
                    if (sbits) sign = (int)rd_bits(ctx.d, 1);
                    sign = 1 - 2 * sign;
                } else {
                    const int mbits = imax(0, imin(left, (left - sctx.delta) / 2)), sbits = left - mbits;
                    ctx.remaining_bits -= sctx.qalloc;
                    rebalance = ctx.remaining_bits;
                    passes = 2;
                    mid_first = mbits >= sbits;
                    pb = mid_first ? mbits : sbits;
                    second_bits = mid_first ? sbits : mbits;
                    pfill = fill;
                    if (!mid_first) {
                        px = Y;
                        plow = pout = pscratch = 0;
                        pgain = (int16_t)sctx.iside;
                        pfill = fill >> B;
                    }
                }
            }
            unsigned cm[2] = {0, 0};
            ROLLED for (int pass = 0; pass < passes; pass++) {
                const unsigned m = quant_band(ctx, px, N, pb, B, plow, LM, pout, pgain, pscratch, pfill);
                if (pass) cm[1] = m;
                else cm[0] = m;
                // the second pass
                const int first_bits = pb;
                px = dual_stereo || mid_first ? Y : X;
                if (dual_stereo) {
                    plow = effective_lowband != -1 ? norm2 + effective_lowband : 0;
                    pout = last ? 0 : norm2 + M * eB[i] - norm_offset;
                    pfill = (int)y_cm;
                } else {
                    const int32_t gained = first_bits - (rebalance - ctx.remaining_bits);
                    pb = second_bits;
                    if (gained > 3 << 3 && sctx.itheta != (mid_first ? 0 : 16384)) pb += gained - (3 << 3);
                    plow = mid_first ? 0 : lowband;
                    pout = mid_first ? 0 : lowband_out;
                    pscratch = mid_first ? 0 : lowband_scratch;
                    pgain = mid_first ? (int16_t)sctx.iside : (int16_t)32767;
                    pfill = mid_first ? fill >> B : fill;
                }
            }
            x_cm = cm[0];
            y_cm = cm[1];
            if (!dual_stereo) {
                x_cm = y_cm = cm[0] | cm[1];
                if (Y != 0) {
                    const int16_t mid = (int16_t)sctx.imid, side = (int16_t)sctx.iside;
                    if (N == 2) {
                        lead(L, [&]() CUO_INLINE {
                            int16_t *x2 = sctx.itheta > 8192 ? Y : X, *y2 = sctx.itheta > 8192 ? X : Y;
                            y2[0] = (int16_t)(-sign * x2[1]);
                            y2[1] = (int16_t)(sign * x2[0]);
                            X[0] = (int16_t)c_mul16_q15(mid, X[0]);
                            X[1] = (int16_t)c_mul16_q15(mid, X[1]);
                            Y[0] = (int16_t)c_mul16_q15(side, Y[0]);
                            Y[1] = (int16_t)c_mul16_q15(side, Y[1]);
                            int16_t tmp = X[0];
                            X[0] = (int16_t)(tmp - Y[0]);
                            Y[0] = (int16_t)(tmp + Y[0]);
                            tmp = X[1];
                            X[1] = (int16_t)(tmp - Y[1]);
                            Y[1] = (int16_t)(tmp + Y[1]);
                        });
                    } else {
                        stereo_merge(L, X, Y, mid, N);
                    }
                    if (sctx.inv) {
                        LFOR(L, j, 0, N) Y[j] = (int16_t)-Y[j];
                        lsync(L);
                    }
                }
            }
        }
        collapse_masks[i * C + 0] = (uint8_t)x_cm;
        collapse_masks[i * C + C - 1] = (uint8_t)y_cm;
        balance += pulses[i] + tell;
        update_lowband = b > (N << 3);
    }
    lsync(L);
    *seed = ctx.seed;
    lsync(L);
}

// celt/bands.c anti_collapse
DNI void anti_collapse(Lanes L, int16_t *X_, const uint8_t *collapse_masks, int LM, int C, int size, int start,
                       int end,
                       const int16_t *logE, const int16_t *prev1logE, const int16_t *prev2logE,
                       const int32_t *pulses, uint32_t seed)
{
    const int16_t *eB = T_celt_eBands;
    ROLLED for (int i = start; i < end; i++) {
        int N0 = eB[i + 1] - eB[i];
        int depth = (int)((uint32_t)(1 + pulses[i]) / (uint32_t)N0) >> LM;
        int32_t thresh32 = c_exp2((int16_t)-(int16_t)((uint16_t)depth << 7)) >> 1;
        int16_t thresh = (int16_t)c_mul16_32_q15(16384, min32(32767, thresh32));
        int32_t t = N0 << LM;
        int shift = c_ilog2(t) >> 1;
        t = shl32(t, (7 - shift) << 1);
        int16_t sqrt_1 = c_rsqrt_norm(t);
        ROLLED for (int c = 0; c < C; c++) {
            int renormalize = 0;
            int16_t prev1 = prev1logE[c * CELT_NB + i], prev2 = prev2logE[c * CELT_NB + i];
            if (C == 1) {
                prev1 = prev1 > prev1logE[CELT_NB + i] ? prev1 : prev1logE[CELT_NB + i];
                prev2 = prev2 > prev2logE[CELT_NB + i] ? prev2 : prev2logE[CELT_NB + i];
            }
            int32_t Ediff = (int32_t)logE[c * CELT_NB + i] - (int32_t)(prev1 < prev2 ? prev1 : prev2);
            Ediff = max32(0, Ediff);
            int16_t r;
            if (Ediff < 16384) {
                int32_t r32 = c_exp2((int16_t)-(int16_t)Ediff) >> 1;
                r = (int16_t)(2 * (r32 < 16383 ? r32 : 16383));
            } else {
                r = 0;
            }
            if (LM == 3) r = (int16_t)c_mul16_q14(23170, min32(23169, r));
            r = (int16_t)((thresh < r ? thresh : r) >> 1);
            r = (int16_t)(c_mul16_q15(sqrt_1, r) >> shift);
            int16_t *X = X_ + c * size + (eB[i] << LM);
            ROLLED for (int k = 0; k < 1 << LM; k++) {
                if (!(collapse_masks[i * C + c] & 1 << k)) {
                    ROLLED for (int j = 0; j < N0; j++) {
                        seed = c_lcg_rand(seed);
                        X[(j << LM) + k] = (seed & 0x8000) ? r : (int16_t)-r;
                    }
                    renormalize = 1;
                }
            }
            if (renormalize) renormalise_vector(L, X, N0 << LM, 32767);
        }
    }
}

DNI void tf_decode(int start, int end, int isTransient, int32_t *tf_res, int LM, RangeDec *rd)
{
    RangeDec dd = *rd, *dec = &dd;   // in registers
    uint32_t budget = dec->storage * 8;
    uint32_t tell = (uint32_t)rd_tell(dec);
    int logp = isTransient ? 2 : 4;
    int tf_select_rsv = LM > 0 && tell + logp + 1 <= budget;
    budget -= tf_select_rsv;
    int tf_changed = 0, curr = 0;
    ROLLED for (int i = start; i < end; i++) {
        if (tell + logp <= budget) {
            curr ^= rdi_bit_logp(dec, logp);
            tell = (uint32_t)rd_tell(dec);
            tf_changed |= curr;
        }
        tf_res[i] = curr;
        logp = isTransient ? 4 : 5;
    }
    int tf_select = 0;
    const int8_t *tt = &T_celt_tf_select_table[LM * 8];
    if (tf_select_rsv && tt[4 * isTransient + 0 + tf_changed] != tt[4 * isTransient + 2 + tf_changed])
        tf_select = rdi_bit_logp(dec, 1);
    ROLLED for (int i = start; i < end; i++) tf_res[i] = tt[4 * isTransient + 2 * tf_select + tf_res[i]];
    *rd = dd;
}

// ------------------------------------------------------------------ PLC (pitch / LPC)
//
// Concealment runs on every lane: sums that wrap are split over the lanes, and
// so are the sample loops; recursions keep their window in registers.  (On the
// first lane alone a lost 20 ms CELT frame took several million cycles: the
// correlations, the FIR and the IIR are 25 k multiply-adds each, one load pair
// at a time.)

// celt/mathops.h celt_maxabs16 / celt_maxabs32 over the lanes
template <class T> DFN int32_t c_maxabs_lanes(const Lanes &L, const T *x, int len)
{
    int32_t mx = 0, mn = 0;
    LFOR(L, i, 0, len) {
        const int32_t v = x[i];
        mx = max32(mx, v);
        mn = min32(mn, v);
    }
    return lmax(L, max32(mx, -mn));
}

// sum of x[i] y[i], n a multiple of 4, this lane alone
DFN int32_t c_dot4(const int16_t *x, const int16_t *y, int n)
{
    int32_t s0 = 0, s1 = 0, s2 = 0, s3 = 0;
    ROLLED for (int j = 0; j < n; j += 4) {
        s0 = c_mac16(s0, x[j], y[j]);
        s1 = c_mac16(s1, x[j + 1], y[j + 1]);
        s2 = c_mac16(s2, x[j + 2], y[j + 2]);
        s3 = c_mac16(s3, x[j + 3], y[j + 3]);
    }
    return wadd(wadd(s0, s1), wadd(s2, s3));
}

// Writes ac[0 .. lag] (the group's memory) and ends with a barrier.
DNI void celt_autocorr(Lanes L, const int16_t *x, int32_t *ac, const int16_t *window, int overlap, int lag, int n,
                       int16_t *xx)
{
    const int16_t *xptr = x;
    int shift;
    if (overlap) {
        LFOR(L, i, 0, n) {
            int16_t v = x[i];
            if (i < overlap) v = (int16_t)c_mul16_q15(v, window[i]);
            if (n - 1 - i < overlap) v = (int16_t)c_mul16_q15(x[i], window[n - 1 - i]);
            xx[i] = v;
        }
        lsync(L);
        xptr = xx;
    }
    int32_t ac0 = 0;
    LFOR(L, i, 0, n) ac0 = wadd(ac0, c_mul16(xptr[i], xptr[i]) >> 9);
    ac0 = wadd(lsum(L, ac0), 1 + (n << 7));
    shift = c_ilog2(ac0) - 30 + 10;
    shift = shift / 2;
    if (shift > 0) {
        lsync(L);
        LFOR(L, i, 0, n) xx[i] = (int16_t)c_pshr(xptr[i], shift);
        lsync(L);
        xptr = xx;
    } else {
        shift = 0;
    }
    LFOR(L, k, 0, lag + 1) {
        const int len = n - k, main = len & ~3;
        int32_t s = c_dot4(xptr, xptr + k, main);
        ROLLED for (int j = main; j < len; j++) s = c_mac16(s, xptr[j], xptr[j + k]);
        ac[k] = s;
    }
    lead(L, [&]() CUO_INLINE {
        shift = 2 * shift;
        if (shift <= 0) ac[0] = wadd(ac[0], shl32(1, -shift));
        if (ac[0] < 268435456) {
            int shift2 = 29 - ilog((uint32_t)ac[0]);
            ROLLED for (int i = 0; i <= lag; i++) ac[i] = shl32(ac[i], shift2);
        } else if (ac[0] >= 536870912) {
            int shift2 = 1;
            if (ac[0] >= 1073741824) shift2++;
            ROLLED for (int i = 0; i <= lag; i++) ac[i] = ac[i] >> shift2;
        }
    });
}

DNI void celt_lpc(int16_t *_lpc, const int32_t *ac, int p)
{
    int32_t error = ac[0];
    int32_t lpc[CELT_LPC_ORDER];
    ROLLED for (int i = 0; i < p; i++) lpc[i] = 0;
    if (ac[0] != 0) {
        ROLLED for (int i = 0; i < p; i++) {
            int32_t rr = 0;
            ROLLED for (int j = 0; j < i; j++) rr = wadd(rr, c_mul32_q31(lpc[j], ac[i - j]));
            rr = wadd(rr, ac[i + 1] >> 6);
            int32_t r = -c_frac_div32(shl32(rr, 6), error);
            lpc[i] = r >> 6;
            ROLLED for (int j = 0; j < (i + 1) >> 1; j++) {
                int32_t t1 = lpc[j], t2 = lpc[i - 1 - j];
                lpc[j] = wadd(t1, c_mul32_q31(r, t2));
                lpc[i - 1 - j] = wadd(t2, c_mul32_q31(r, t1));
            }
            error = wsub(error, c_mul32_q31(c_mul32_q31(r, r), error));
            if (error <= (ac[0] >> 10)) break;
        }
    }
    int iter, idx = 0;
    ROLLED for (iter = 0; iter < 10; iter++) {
        int32_t maxabs = 0;
        ROLLED for (int i = 0; i < p; i++) {
            int32_t a = lpc[i] < 0 ? -lpc[i] : lpc[i];
            if (a > maxabs) { maxabs = a; idx = i; }
        }
        maxabs = c_pshr(maxabs, 13);
        if (maxabs > 32767) {
            maxabs = min32(maxabs, 163838);
            int32_t chirp_Q16 = 65470 - shl32(maxabs - 32767, 14) / (wmul(maxabs, idx + 1) >> 2);
            int32_t cm1 = chirp_Q16 - 65536;
            ROLLED for (int i = 0; i < p - 1; i++) {
                lpc[i] = c_mul32_q16(chirp_Q16, lpc[i]);
                chirp_Q16 += c_pshr(wmul(chirp_Q16, cm1), 16);
            }
            lpc[p - 1] = c_mul32_q16(chirp_Q16, lpc[p - 1]);
        } else {
            break;
        }
    }
    if (iter == 10) {
        _lpc[0] = 4096;   // the remaining outputs keep their previous values, as in libopus
    } else {
        ROLLED for (int i = 0; i < p; i++) _lpc[i] = (int16_t)c_pshr(lpc[i], 13);
    }
}

// every output on its own: the lanes split them
DNI void celt_fir(Lanes L, const int16_t *x, const int16_t *num, int16_t *y, int N)
{
    int32_t a[CELT_LPC_ORDER];
#pragma unroll
    for (int j = 0; j < CELT_LPC_ORDER; j++) a[j] = num[j];
    LFOR(L, i, 0, N) {
        int32_t sum = shl32((int32_t)x[i], 12), sum1 = 0;
#pragma unroll
        for (int j = 0; j < CELT_LPC_ORDER; j += 2) {
            sum = c_mac16(sum, a[j], x[i - j - 1]);
            sum1 = c_mac16(sum1, a[j + 1], x[i - j - 2]);
        }
        y[i] = c_sround16(wadd(sum, sum1), 12);
    }
    lsync(L);
}

// celt/celt_lpc.c celt_iir, in place on x (the 4-way unrolled form computes the
// same values), with the saturation of the extrapolated signal.  Four samples
// at a time with the filter memory (y, negated and rounded outputs) in
// registers, as in silk_lpc_synth; every lane runs it and the first one stores.
DNI void celt_iir(Lanes L, int32_t *x, const int16_t *den, int N, const int16_t *mem)
{
    int32_t a[CELT_LPC_ORDER], y[CELT_LPC_ORDER];   // y[0] oldest
#pragma unroll
    for (int j = 0; j < CELT_LPC_ORDER; j++) {
        a[j] = den[j];
        y[j] = (int16_t)-mem[CELT_LPC_ORDER - 1 - j];
    }
    int32_t ahead[4];
#pragma unroll
    for (int s = 0; s < 4; s++) ahead[s] = x[s];
    ROLLED for (int i = 0; i < N; i += 4) {
        int32_t v[4], o[4];
        const int nx = i + 4 < N ? i + 4 : i;
#pragma unroll
        for (int s = 0; s < 4; s++) {
            v[s] = ahead[s];
            ahead[s] = x[nx + s];
        }
        lsync(L);   // every lane has read what the first lane overwrites below
#pragma unroll
        for (int j = CELT_LPC_ORDER - 1; j >= 0; j--) {
#pragma unroll
            for (int s = 0; s < 4; s++)
                if (j >= s) v[s] = c_mac16(v[s], a[j], y[CELT_LPC_ORDER - 1 + s - j]);
        }
#pragma unroll
        for (int s = 0; s < 4; s++) {
#pragma unroll
            for (int t = 0; t < s; t++) v[s] = c_mac16(v[s], a[s - 1 - t], o[t]);
            o[s] = (int16_t)-c_sround16(v[s], 12);
        }
#pragma unroll
        for (int j = 0; j < CELT_LPC_ORDER - 4; j++) y[j] = y[j + 4];
#pragma unroll
        for (int s = 0; s < 4; s++) {
            y[CELT_LPC_ORDER - 4 + s] = o[s];
            if (L.id == 0) x[i + s] = c_sat(v[s], CELT_SIG_SAT);
        }
    }
    lsync(L);
}

// Syy: 1 plus the energy of the first len samples of y.
DNI void find_best_pitch(const int32_t *xcorr, const int16_t *y, int len, int max_pitch, int *best_pitch,
                         int yshift, int32_t maxcorr, int32_t Syy)
{
    int16_t best_num[2] = {-1, -1};
    int32_t best_den[2] = {0, 0};
    int xshift = c_ilog2(maxcorr) - 14;
    best_pitch[0] = 0;
    best_pitch[1] = 1;
    ROLLED for (int i = 0; i < max_pitch; i++) {
        if (xcorr[i] > 0) {
            int16_t xcorr16 = (int16_t)c_vshr(xcorr[i], xshift);
            int16_t num = (int16_t)c_mul16_q15(xcorr16, xcorr16);
            if (c_mul16_32_q15(num, best_den[1]) > c_mul16_32_q15(best_num[1], Syy)) {
                if (c_mul16_32_q15(num, best_den[0]) > c_mul16_32_q15(best_num[0], Syy)) {
                    best_num[1] = best_num[0];
                    best_den[1] = best_den[0];
                    best_pitch[1] = best_pitch[0];
                    best_num[0] = num;
                    best_den[0] = Syy;
                    best_pitch[0] = i;
                } else {
                    best_num[1] = num;
                    best_den[1] = Syy;
                    best_pitch[1] = i;
                }
            }
        }
        Syy = wadd(Syy, wsub(c_mul16(y[i + len], y[i + len]) >> yshift, c_mul16(y[i], y[i]) >> yshift));
        Syy = max32(1, Syy);
    }
}

DNI void pitch_downsample(Lanes L, int32_t *x0, int32_t *x1, int16_t *x_lp, int len, int C, int16_t *xx, int32_t *ac)
{
    int16_t tmp = 32767, lpc[4], lpc2[5];
    const int16_t c1 = 26214;   // QCONST16(.8f, 15)
    int32_t maxabs = c_maxabs_lanes(L, x0, len);
    if (C == 2) maxabs = max32(maxabs, c_maxabs_lanes(L, x1, len));
    if (maxabs < 1) maxabs = 1;
    int shift = c_ilog2(maxabs) - 10;
    if (shift < 0) shift = 0;
    if (C == 2) shift++;
    LFOR(L, i, 0, len >> 1) {
        int32_t v = (x0[2 * i + 1] >> (shift + 2)) + (x0[2 * i] >> (shift + 1));
        if (i) v += x0[2 * i - 1] >> (shift + 2);
        if (C == 2) {
            v += (x1[2 * i + 1] >> (shift + 2)) + (x1[2 * i] >> (shift + 1));
            if (i) v += x1[2 * i - 1] >> (shift + 2);
        }
        x_lp[i] = (int16_t)v;
    }
    lsync(L);
    celt_autocorr(L, x_lp, ac, 0, 0, 4, len >> 1, xx);
    int32_t acl[5];
#pragma unroll
    for (int i = 0; i < 5; i++) acl[i] = ac[i];
    acl[0] = wadd(acl[0], acl[0] >> 13);
#pragma unroll
    for (int i = 1; i <= 4; i++) acl[i] = wsub(acl[i], c_mul16_32_q15(2 * i * i, acl[i]));
    lpc[0] = lpc[1] = lpc[2] = lpc[3] = 0;
    celt_lpc(lpc, acl, 4);
    ROLLED for (int i = 0; i < 4; i++) {
        tmp = (int16_t)c_mul16_q15(29491, tmp);   // QCONST16(.9f, 15)
        lpc[i] = (int16_t)c_mul16_q15(lpc[i], tmp);
    }
    lpc2[0] = (int16_t)(lpc[0] + 3277);   // QCONST16(.8f, SIG_SHIFT)
    lpc2[1] = (int16_t)(lpc[1] + c_mul16_q15(c1, lpc[0]));
    lpc2[2] = (int16_t)(lpc[2] + c_mul16_q15(c1, lpc[1]));
    lpc2[3] = (int16_t)(lpc[3] + c_mul16_q15(c1, lpc[2]));
    lpc2[4] = (int16_t)c_mul16_q15(c1, lpc[3]);
    // celt_fir5 of the unfiltered samples, through xx
    lsync(L);
    LFOR(L, i, 0, len >> 1) {
        int32_t sum = shl32((int32_t)x_lp[i], 12);
#pragma unroll
        for (int j = 0; j < 5; j++)
            if (i > j) sum = c_mac16(sum, lpc2[j], x_lp[i - 1 - j]);
        xx[i] = (int16_t)c_pshr(sum, 12);
    }
    lsync(L);
    LFOR(L, i, 0, len >> 1) x_lp[i] = xx[i];
    lsync(L);
}

// Sum of squares of y[0 .. len), each shifted, plus 1 (find_best_pitch's Syy).
DFN int32_t c_energy_lanes(const Lanes &L, const int16_t *y, int len, int shift)
{
    int32_t s = 0;
    LFOR(L, j, 0, len) s = wadd(s, c_mul16(y[j], y[j]) >> shift);
    return wadd(1, lsum(L, s));
}

// The pitch, on every lane.  (len >> 2 and len >> 1 are multiples of 4.)
DNI int pitch_search(Lanes L, const int16_t *x_lp, int16_t *y, int len, int max_pitch, CeltScratch *w)
{
    int lag = len + max_pitch;
    int best_pitch[2] = {0, 0};
    int16_t *x_lp4 = w->x_lp4, *y_lp4 = w->y_lp4;
    int32_t *xcorr = w->xcorr;
    LFOR(L, j, 0, len >> 2) x_lp4[j] = x_lp[2 * j];
    LFOR(L, j, 0, lag >> 2) y_lp4[j] = y[2 * j];
    lsync(L);
    int32_t xmax = c_maxabs_lanes(L, x_lp4, len >> 2), ymax = c_maxabs_lanes(L, y_lp4, lag >> 2);
    int shift = c_ilog2(max32(1, max32(xmax, ymax))) - 11;
    if (shift > 0) {
        lsync(L);
        LFOR(L, j, 0, len >> 2) x_lp4[j] = (int16_t)(x_lp4[j] >> shift);
        LFOR(L, j, 0, lag >> 2) y_lp4[j] = (int16_t)(y_lp4[j] >> shift);
        shift *= 2;
    } else {
        shift = 0;
    }
    lsync(L);
    // celt_pitch_xcorr: every lag is an independent dot product
    int32_t maxcorr = 1;
    LFOR(L, i, 0, max_pitch >> 2) {
        xcorr[i] = c_dot4(x_lp4, y_lp4 + i, len >> 2);
        maxcorr = max32(maxcorr, xcorr[i]);
    }
    maxcorr = lmax(L, maxcorr);
    int32_t Syy = c_energy_lanes(L, y_lp4, len >> 2, 0);
    lead(L, [&]() CUO_INLINE { find_best_pitch(xcorr, y_lp4, len >> 2, max_pitch >> 2, best_pitch, 0, maxcorr, Syy); });
    best_pitch[0] = lbcast(L, best_pitch[0]);
    best_pitch[1] = lbcast(L, best_pitch[1]);
    // libopus tracks max(1, raw sums); the -1 floor and the zeroed lags cannot exceed 1
    maxcorr = 1;
    LFOR(L, i, 0, max_pitch >> 1) {
        int32_t v = 0;
        int d0 = i - 2 * best_pitch[0], d1 = i - 2 * best_pitch[1];
        if (!((d0 < 0 ? -d0 : d0) > 2 && (d1 < 0 ? -d1 : d1) > 2)) {
            int32_t s0 = 0, s1 = 0;
            ROLLED for (int j = 0; j < len >> 1; j += 4) {
                s0 = wadd(s0, c_mul16(x_lp[j], y[i + j]) >> shift);
                s1 = wadd(s1, c_mul16(x_lp[j + 1], y[i + j + 1]) >> shift);
                s0 = wadd(s0, c_mul16(x_lp[j + 2], y[i + j + 2]) >> shift);
                s1 = wadd(s1, c_mul16(x_lp[j + 3], y[i + j + 3]) >> shift);
            }
            v = max32(-1, wadd(s0, s1));
        }
        xcorr[i] = v;
        maxcorr = max32(maxcorr, v);
    }
    maxcorr = lmax(L, maxcorr);
    Syy = c_energy_lanes(L, y, len >> 1, shift + 1);
    int pitch = 0;
    lead(L, [&]() CUO_INLINE {
        find_best_pitch(xcorr, y, len >> 1, max_pitch >> 1, best_pitch, shift + 1, maxcorr, Syy);
        int offset;
        if (best_pitch[0] > 0 && best_pitch[0] < (max_pitch >> 1) - 1) {
            int32_t a = xcorr[best_pitch[0] - 1], b = xcorr[best_pitch[0]], c = xcorr[best_pitch[0] + 1];
            if ((c - a) > c_mul16_32_q15(22938, b - a)) offset = 1;          // QCONST16(.7f, 15)
            else if ((a - c) > c_mul16_32_q15(22938, b - c)) offset = -1;
            else offset = 0;
        } else {
            offset = 0;
        }
        pitch = 2 * best_pitch[0] - offset;
    });
    return lbcast(L, pitch);
}

DNI void prefilter_and_fold(Lanes L, CeltDec *st, int N, CeltScratch *w)
{
    ROLLED for (int c = 0; c < st->channels; c++) {
        int32_t *dm = st->decode_mem[c];
        comb_filter_lanes(L, w->etmp, dm + CELT_DEC_BUF - N, st->postfilter_period_old, st->postfilter_period,
                          CELT_OVERLAP, (int16_t)-st->postfilter_gain_old, (int16_t)-st->postfilter_gain,
                          st->postfilter_tapset_old, st->postfilter_tapset, 0, 0);
        lsync(L);
        LFOR(L, i, 0, CELT_OVERLAP / 2)
            dm[CELT_DEC_BUF - N + i] = wadd(c_mul16_32_q15(T_celt_window[i], w->etmp[CELT_OVERLAP - 1 - i]),
                                            c_mul16_32_q15(T_celt_window[CELT_OVERLAP - i - 1], w->etmp[i]));
        lsync(L);
    }
}

// celt/celt_decoder.c celt_decode_lost (no deep PLC)
DNI void celt_decode_lost(Lanes L, CeltDec *st, int N, int LM, CeltScratch *w)
{
    const int C = st->channels;
    const int16_t *eB = T_celt_eBands;
    int32_t *out_syn[2];
    ROLLED for (int c = 0; c < C; c++) out_syn[c] = st->decode_mem[c] + CELT_DEC_BUF - N;
    const int loss_duration = st->loss_duration;
    const int start = st->start;
    const int noise_based = loss_duration >= 40 || start != 0 || st->skip_plc;
    if (noise_based) {
        const int end = st->end;
        const int effEnd = imax(start, imin(end, T_CELT_EFFEBANDS));
        int16_t *X = w->X;
        ROLLED for (int c = 0; c < C; c++) lshift_copy(L, st->decode_mem[c], CELT_DEC_BUF - N + CELT_OVERLAP, N);
        if (st->prefilter_and_fold) prefilter_and_fold(L, st, N, w);
        int16_t decay = loss_duration == 0 ? 1536 : 512;   // QCONST16(1.5f / .5f, DB_SHIFT)
        ROLLED for (int c = 0; c < C; c++)
            LFOR(L, i, start, end) {
                int32_t a = st->backgroundLogE[c * CELT_NB + i];
                int32_t b = st->oldBandE[c * CELT_NB + i] - decay;
                st->oldBandE[c * CELT_NB + i] = (int16_t)(a > b ? a : b);
            }
        uint32_t seed = st->rng;
        ROLLED for (int c = 0; c < C; c++) {
            ROLLED for (int i = start; i < effEnd; i++) {
                const int boffs = N * c + (eB[i] << LM);
                const int blen = (eB[i + 1] - eB[i]) << LM;
                LFOR(L, j, 0, blen) X[boffs + j] = (int16_t)((int32_t)(T_lcg.a[j + 1] * seed + T_lcg.c[j + 1]) >> 20);
                seed = T_lcg.a[blen] * seed + T_lcg.c[blen];
                lsync(L);
                renormalise_vector(L, X + boffs, blen, 32767);
            }
        }
        celt_synthesis(L, w, X, out_syn, st->oldBandE, start, effEnd, C, C, 0, LM, 0);
        lead(L, [&]() CUO_INLINE {
            st->rng = seed;
            st->prefilter_and_fold = 0;
            st->skip_plc = 1;
        });
    } else {
        int16_t fade = 32767;
        int pitch_index;
        if (loss_duration == 0) {
            pitch_downsample(L, st->decode_mem[0], st->decode_mem[1], w->lp_pitch_buf, CELT_DEC_BUF, C, w->ac_xx, w->etmp);
            pitch_index = 720 - pitch_search(L, w->lp_pitch_buf + (720 >> 1), w->lp_pitch_buf, CELT_DEC_BUF - 720,
                                             720 - 100, w);
        } else {
            pitch_index = st->last_pitch_index;
            fade = 26214;   // QCONST16(.8f, 15)
        }
        const int exc_length = imin(2 * pitch_index, CELT_MAX_PERIOD);
        int16_t *exc = w->exc + CELT_LPC_ORDER;
        const int16_t *window = T_celt_window;
        ROLLED for (int c = 0; c < C; c++) {
            int32_t *buf = st->decode_mem[c];
            int16_t *lpc = st->lpc[c];
            lsync(L);
            LFOR(L, i, 0, CELT_MAX_PERIOD + CELT_LPC_ORDER)
                exc[i - CELT_LPC_ORDER] = c_sround16(buf[CELT_DEC_BUF - CELT_MAX_PERIOD - CELT_LPC_ORDER + i], 12);
            lsync(L);
            if (loss_duration == 0) {
                int32_t *ac = w->etmp;
                celt_autocorr(L, exc, ac, window, CELT_OVERLAP, CELT_LPC_ORDER, CELT_MAX_PERIOD, w->ac_xx);
                lead(L, [&]() CUO_INLINE {
                    ac[0] = wadd(ac[0], ac[0] >> 13);
                    ROLLED for (int i = 1; i <= CELT_LPC_ORDER; i++) ac[i] = wsub(ac[i], c_mul16_32_q15(2 * i * i, ac[i]));
                    celt_lpc(lpc, ac, CELT_LPC_ORDER);
                    ROLLED while (1) {
                        int16_t tmp = 32767;
                        int32_t sum = 4096;   // QCONST16(1., SIG_SHIFT)
                        ROLLED for (int i = 0; i < CELT_LPC_ORDER; i++) sum += lpc[i] < 0 ? -lpc[i] : lpc[i];
                        if (sum < 65535) break;
                        ROLLED for (int i = 0; i < CELT_LPC_ORDER; i++) {
                            tmp = (int16_t)c_mul16_q15(32440, tmp);   // QCONST16(.99f, 15)
                            lpc[i] = (int16_t)c_mul16_q15(lpc[i], tmp);
                        }
                    }
                });
            }
            celt_fir(L, exc + CELT_MAX_PERIOD - exc_length, lpc, w->fir_tmp, exc_length);
            LFOR(L, i, 0, exc_length) exc[CELT_MAX_PERIOD - exc_length + i] = w->fir_tmp[i];
            lsync(L);
            int16_t decay;
            {
                int shift = imax(0, 2 * c_zlog2(c_maxabs_lanes(L, &exc[CELT_MAX_PERIOD - exc_length], exc_length)) - 20);
                const int decay_length = exc_length >> 1;
                int32_t E1 = 0, E2 = 0;
                LFOR(L, i, 0, decay_length) {
                    int16_t e = exc[CELT_MAX_PERIOD - decay_length + i];
                    E1 = wadd(E1, c_mul16(e, e) >> shift);
                    e = exc[CELT_MAX_PERIOD - 2 * decay_length + i];
                    E2 = wadd(E2, c_mul16(e, e) >> shift);
                }
                E1 = wadd(1, lsum(L, E1));
                E2 = wadd(1, lsum(L, E2));
                E1 = min32(E1, E2);
                decay = (int16_t)c_sqrt(c_frac_div32(E1 >> 1, E2));
            }
            lshift_copy(L, buf, CELT_DEC_BUF - N, N);
            const int extrapolation_offset = CELT_MAX_PERIOD - pitch_index;
            const int extrapolation_len = N + CELT_OVERLAP;
            int16_t attenuation = (int16_t)c_mul16_q15(fade, decay);
            // period after period of the excitation, each weaker than the last
            int32_t S1 = 0;
            ROLLED for (int b = 0; b < extrapolation_len; b += pitch_index) {
                LFOR(L, j, 0, imin(pitch_index, extrapolation_len - b)) {
                    buf[CELT_DEC_BUF - N + b + j] = shl32((int32_t)(int16_t)c_mul16_q15(attenuation,
                                                          exc[extrapolation_offset + j]), 12);
                    int16_t tmp = c_sround16(buf[CELT_DEC_BUF - CELT_MAX_PERIOD - N + extrapolation_offset + j], 12);
                    S1 = wadd(S1, c_mul16(tmp, tmp) >> 10);
                }
                attenuation = (int16_t)c_mul16_q15(attenuation, decay);
            }
            S1 = lsum(L, S1);
            lsync(L);
            int16_t lpc_mem[CELT_LPC_ORDER];
#pragma unroll
            for (int i = 0; i < CELT_LPC_ORDER; i++) lpc_mem[i] = c_sround16(buf[CELT_DEC_BUF - N - 1 - i], 12);
            celt_iir(L, buf + CELT_DEC_BUF - N, lpc, extrapolation_len, lpc_mem);
            int32_t S2 = 0;
            LFOR(L, i, 0, extrapolation_len) {
                int16_t tmp = c_sround16(buf[CELT_DEC_BUF - N + i], 12);
                S2 = wadd(S2, c_mul16(tmp, tmp) >> 10);
            }
            S2 = lsum(L, S2);
            lsync(L);
            if (!(S1 > (S2 >> 2))) {
                LFOR(L, i, 0, extrapolation_len) buf[CELT_DEC_BUF - N + i] = 0;
            } else if (S1 < S2) {
                const int16_t ratio = (int16_t)c_sqrt(c_frac_div32((S1 >> 1) + 1, S2 + 1));
                LFOR(L, i, 0, extrapolation_len) {
                    const int16_t tmp_g = i < CELT_OVERLAP
                        ? (int16_t)(32767 - c_mul16_q15(window[i], (int16_t)(32767 - ratio))) : ratio;
                    buf[CELT_DEC_BUF - N + i] = c_mul16_32_q15(tmp_g, buf[CELT_DEC_BUF - N + i]);
                }
            }
            lsync(L);
        }
        lead(L, [&]() CUO_INLINE {
            st->last_pitch_index = pitch_index;
            st->prefilter_and_fold = 1;
        });
    }
    lead(L, [&]() CUO_INLINE { st->loss_duration = imin(10000, loss_duration + (1 << LM)); });
}

// ------------------------------------------------------------------ frame decode

// The band energies of the first frame after a loss that is not intra coded
// (celt/celt_decoder.c, in celt_decode_with_ec_dred before unquant_coarse_energy):
// each energy may rise at most as the previous two frames did, less a safety
// margin.  Its own function, so the code of the lossless path stays small.
DNI void energy_after_loss(CeltDec *st, int start, int end, int LM)
{
    int16_t *oldBandE = st->oldBandE, *oldLogE = st->oldLogE, *oldLogE2 = st->oldLogE2;
    ROLLED for (int c = 0; c < 2; c++) {
        int16_t safety = 0;
        int missing = imin(10, st->loss_duration >> LM);
        if (LM == 0) safety = 1536;
        else if (LM == 1) safety = 512;
        ROLLED for (int i = start; i < end; i++) {
            int16_t *e0 = &oldBandE[c * CELT_NB + i];
            int16_t e1 = oldLogE[c * CELT_NB + i], e2 = oldLogE2[c * CELT_NB + i];
            if (*e0 < (e1 > e2 ? e1 : e2)) {
                int32_t E0 = *e0, E1 = e1, E2 = e2;
                int32_t slope = max32(E1 - E0, (E2 - E0) >> 1);
                E0 -= max32(0, (1 + missing) * slope);
                *e0 = (int16_t)max32(-20480, E0);   // -QCONST16(20.f, DB_SHIFT)
            } else {
                int16_t m = *e0 < e1 ? *e0 : e1;
                *e0 = m < e2 ? m : e2;
            }
            *e0 = (int16_t)(*e0 - safety);
        }
    }
}

// celt/celt_decoder.c celt_decode_with_ec_dred (downsample 1, no deep PLC).
// data == 0 or len <= 1 runs the concealment.  Returns samples or < 0.
DNI int celt_decode(Lanes L, CeltDec *st, const uint8_t *data, int len, int16_t *pcm, int frame_size,
                    RangeDec *dec, int accum, CeltScratch *w)
{
    const int16_t *eB = T_celt_eBands;
    const int CC = st->channels;
    int C = st->stream_channels;
    int start = st->start, end = st->end;
    int LM;
    ROLLED for (LM = 0; LM <= T_CELT_MAXLM; LM++)
        if (T_CELT_SHORTMDCT << LM == frame_size) break;
    if (LM > T_CELT_MAXLM) return -1;   // OPUS_BAD_ARG
    int M = 1 << LM;
    if (len < 0 || len > 1275 || pcm == 0) return -1;
    int N = M * T_CELT_SHORTMDCT;
    int32_t *out_syn[2];
    ROLLED for (int c = 0; c < CC; c++) out_syn[c] = st->decode_mem[c] + CELT_DEC_BUF - N;
    if (CC == 1) out_syn[1] = out_syn[0];
    int effEnd = end;
    if (effEnd > T_CELT_EFFEBANDS) effEnd = T_CELT_EFFEBANDS;
    if (data == 0 || len <= 1) {
        // concealment (mode transitions, lost packets)
        celt_decode_lost(L, st, N, LM, w);
        deemphasis(L, out_syn[0], out_syn[1], pcm, N, CC, st->preemph_memD, accum, w->freq, w->deemph);
        return frame_size;
    }
    RangeDec _dec;
    if (dec == 0) {
        rd_init(&_dec, data, len);
        dec = &_dec;
    }
    int16_t *oldBandE = st->oldBandE, *oldLogE = st->oldLogE, *oldLogE2 = st->oldLogE2,
            *backgroundLogE = st->backgroundLogE;
    if (C == 1) {
        LFOR(L, i, 0, CELT_NB) oldBandE[i] = oldBandE[i] > oldBandE[CELT_NB + i] ? oldBandE[i] : oldBandE[CELT_NB + i];
    }
    int32_t *tf_res = w->tf_res;
    int32_t *pulses = w->pulses, *fine_quant = w->fine_quant, *fine_priority = w->fine_priority;
    // The frame header and the energies: entropy decoding and state updates in
    // place, on the first lane; every lane gets the outcome (the per-band tables
    // stay in the scratch).
    enum { H_SILENCE, H_PF_GAIN, H_PF_PITCH, H_PF_TAPSET, H_TRANSIENT, H_SPREAD, H_AC_RSV, H_TRIM, H_BITS, H_N };
    int32_t hv[H_N] = {0};
    init_caps(L, w->cap, LM, C);
    lead_rd(L, dec, [&]() CUO_INLINE {
        if (st->loss_duration == 0) st->skip_plc = 0;
        int32_t total_bits = len * 8;
        int32_t tell = rd_tell(dec);
        int silence;
        if (tell >= total_bits) silence = 1;
        else if (tell == 1) silence = rd_bit_logp(dec, 15);
        else silence = 0;
        if (silence) {
            tell = len * 8;
            dec->nbits_total += tell - rd_tell(dec);
        }
        int16_t postfilter_gain = 0;
        int postfilter_pitch = 0, postfilter_tapset = 0;
        if (start == 0 && tell + 16 <= total_bits) {
            if (rd_bit_logp(dec, 1)) {
                int octave = (int)rd_uint(dec, 6);
                postfilter_pitch = (16 << octave) + (int)rd_bits(dec, 4 + octave) - 1;
                int qg = (int)rd_bits(dec, 3);
                if (rd_tell(dec) + 2 <= total_bits) postfilter_tapset = rd_icdf(dec, T_celt_tapset_icdf, 2);
                postfilter_gain = (int16_t)(3072 * (qg + 1));   // QCONST16(.09375f, 15)
            }
            tell = rd_tell(dec);
        }
        int isTransient;
        if (LM > 0 && tell + 3 <= total_bits) {
            isTransient = rd_bit_logp(dec, 3);
            tell = rd_tell(dec);
        } else {
            isTransient = 0;
        }
        int intra_ener = tell + 3 <= total_bits ? rd_bit_logp(dec, 3) : 0;
        if (!intra_ener && st->loss_duration != 0) energy_after_loss(st, start, end, LM);
        PHASE_BEGIN(t_ce);
        unquant_coarse_energy(start, end, oldBandE, intra_ener, dec, C, LM);
        PHASE_END(PH_CELT_COARSE, t_ce, L.id);
        tf_decode(start, end, isTransient, tf_res, LM, dec);
        tell = rd_tell(dec);
        int spread_decision = SPREAD_NORMAL;
        if (tell + 4 <= total_bits) spread_decision = rd_icdf(dec, T_celt_spread_icdf, 5);
        int32_t *cap = w->cap, *offsets = w->offsets;
        int dynalloc_logp = 6;
        total_bits <<= 3;
        RangeDec d = *dec;   // in registers for the boosts
        tell = (int32_t)rd_tell_frac(&d);
        ROLLED for (int i = start; i < end; i++) {
            int width = C * (eB[i + 1] - eB[i]) << LM;
            int quanta = imin(width << 3, imax(6 << 3, width));
            int dll = dynalloc_logp, boost = 0;
            ROLLED while (tell + (dll << 3) < total_bits && boost < cap[i]) {
                int flag = rdi_bit_logp(&d, dll);
                tell = (int32_t)rd_tell_frac(&d);
                if (!flag) break;
                boost += quanta;
                total_bits -= quanta;
                dll = 1;
            }
            offsets[i] = boost;
            if (boost > 0) dynalloc_logp = imax(2, dynalloc_logp - 1);
        }
        *dec = d;
        int alloc_trim = tell + (6 << 3) <= total_bits ? rd_icdf(dec, T_celt_trim_icdf, 7) : 5;
        int32_t bits = (((int32_t)len * 8) << 3) - (int32_t)rd_tell_frac(dec) - 1;
        int anti_collapse_rsv = isTransient && LM >= 2 && bits >= ((LM + 2) << 3) ? (1 << 3) : 0;
        bits -= anti_collapse_rsv;
        hv[H_SILENCE] = silence;
        hv[H_PF_GAIN] = postfilter_gain;
        hv[H_PF_PITCH] = postfilter_pitch;
        hv[H_PF_TAPSET] = postfilter_tapset;
        hv[H_TRANSIENT] = isTransient;
        hv[H_SPREAD] = spread_decision;
        hv[H_AC_RSV] = anti_collapse_rsv;
        hv[H_TRIM] = alloc_trim;
        hv[H_BITS] = bits;
    });
    for (int k = 0; k < H_N; k++) hv[k] = lbcast(L, hv[k]);
    int intensity = 0, dual_stereo = 0;
    int32_t balance;
    PHASE_BEGIN(t_al);
    const int codedBands = clt_compute_allocation(L, start, end, w->offsets, w->cap, hv[H_TRIM], &intensity,
                                                  &dual_stereo, hv[H_BITS], &balance, pulses, fine_quant,
                                                  fine_priority, C, LM, dec, w);
    PHASE_END(PH_CELT_ALLOC, t_al, L.id);
    lead_rd(L, dec, [&]() CUO_INLINE { unquant_fine_energy(start, end, oldBandE, fine_quant, dec, C); });
    const int silence = hv[H_SILENCE];
    const int16_t postfilter_gain = (int16_t)hv[H_PF_GAIN];
    const int postfilter_pitch = hv[H_PF_PITCH], postfilter_tapset = hv[H_PF_TAPSET];
    const int isTransient = hv[H_TRANSIENT], shortBlocks = isTransient ? M : 0;
    const int spread_decision = hv[H_SPREAD], anti_collapse_rsv = hv[H_AC_RSV];
    PHASE_BEGIN(t_sh);
    ROLLED for (int c = 0; c < CC; c++) lshift_copy(L, st->decode_mem[c], CELT_DEC_BUF - N + CELT_OVERLAP, N);
    PHASE_END(PH_CELT_SHIFT, t_sh, L.id);
    int16_t *X = w->X;
    // the band shapes
    PHASE_BEGIN(t_qb);
    {
        quant_all_bands_dec(L, start, end, X, C == 2 ? X + N : 0, w->collapse_masks, pulses, shortBlocks,
                            spread_decision, dual_stereo, intensity, tf_res, len * (8 << 3) - anti_collapse_rsv,
                            balance, dec, LM, codedBands, &st->rng, st->disable_inv, w);
    }
    PHASE_END(PH_CELT_BANDS, t_qb, L.id);
    int anti_collapse_on = 0;
    lead_rd(L, dec, [&]() CUO_INLINE {
        if (anti_collapse_rsv > 0) anti_collapse_on = (int)rd_bits(dec, 1);
        unquant_energy_finalise(start, end, oldBandE, fine_quant, fine_priority, len * 8 - rd_tell(dec), dec, C);
    });
    anti_collapse_on = lbcast(L, anti_collapse_on);
    lead(L, [&]() CUO_INLINE {
        if (anti_collapse_on)
            anti_collapse(lone(L), X, w->collapse_masks, LM, C, N, start, end, oldBandE, oldLogE, oldLogE2, pulses,
                          st->rng);
        if (silence)
            ROLLED for (int i = 0; i < C * CELT_NB; i++) oldBandE[i] = -28672;   // -QCONST16(28.f, DB_SHIFT)
    });
    if (st->prefilter_and_fold) prefilter_and_fold(L, st, N, w);
    PHASE_BEGIN(t_sy);
    celt_synthesis(L, w, X, out_syn, oldBandE, start, effEnd, C, CC, isTransient, LM, silence);
    PHASE_END(PH_CELT_SYNTH, t_sy, L.id);
    PHASE_BEGIN(t_cb);
    // the post-filter state is read once into registers here and written back
    // on the first lane after the filter, both with the period floored at 15
    const int pf_period = imax(st->postfilter_period, 15), pf_period_old = imax(st->postfilter_period_old, 15);
    const int16_t pf_gain = (int16_t)st->postfilter_gain, pf_gain_old = (int16_t)st->postfilter_gain_old;
    const int pf_tapset = st->postfilter_tapset, pf_tapset_old = st->postfilter_tapset_old;
    ROLLED for (int c = 0; c < CC; c++) {
        comb_filter_lanes(L, out_syn[c], out_syn[c], pf_period_old, pf_period, T_CELT_SHORTMDCT, pf_gain_old,
                          pf_gain, pf_tapset_old, pf_tapset, T_celt_window, CELT_OVERLAP);
        if (LM != 0)
            comb_filter_lanes(L, out_syn[c] + T_CELT_SHORTMDCT, out_syn[c] + T_CELT_SHORTMDCT, pf_period,
                              postfilter_pitch, N - T_CELT_SHORTMDCT, pf_gain, postfilter_gain, pf_tapset,
                              postfilter_tapset, T_celt_window, CELT_OVERLAP);
    }
    PHASE_END(PH_CELT_COMB, t_cb, L.id);
    lead(L, [&]() CUO_INLINE {
        st->postfilter_period_old = pf_period;
        st->postfilter_gain_old = pf_gain;
        st->postfilter_tapset_old = pf_tapset;
        st->postfilter_period = postfilter_pitch;
        st->postfilter_gain = postfilter_gain;
        st->postfilter_tapset = postfilter_tapset;
        if (LM != 0) {
            st->postfilter_period_old = st->postfilter_period;
            st->postfilter_gain_old = st->postfilter_gain;
            st->postfilter_tapset_old = st->postfilter_tapset;
        }
    });
    // energy history: every band of both channels on its own, so lanes split them
    if (C == 1) {
        LFOR(L, i, 0, CELT_NB) oldBandE[CELT_NB + i] = oldBandE[i];
        lsync(L);
    }
    int32_t mbi = imin(160, st->loss_duration + M) * 1;   // QCONST16(0.001f, DB_SHIFT) == 1
    LFOR(L, j, 0, 2 * CELT_NB) {
        int16_t e = oldBandE[j];
        if (!isTransient) {
            oldLogE2[j] = oldLogE[j];
            oldLogE[j] = e;
        } else {
            oldLogE[j] = oldLogE[j] < e ? oldLogE[j] : e;
        }
        int32_t v = backgroundLogE[j] + mbi;
        backgroundLogE[j] = (int16_t)(v < e ? v : e);
        int i = j < CELT_NB ? j : j - CELT_NB;
        if (i < start || i >= end) {
            oldBandE[j] = 0;
            oldLogE[j] = oldLogE2[j] = -28672;
        }
    }
    PHASE_BEGIN(t_de);
    deemphasis(L, out_syn[0], out_syn[1], pcm, N, CC, st->preemph_memD, accum, w->freq, w->deemph);
    PHASE_END(PH_CELT_DEEMPH, t_de, L.id);
    lead(L, [&]() CUO_INLINE {
        st->rng = dec->rng;
        st->loss_duration = 0;
        st->prefilter_and_fold = 0;
        if (rd_tell(dec) <= 8 * len && dec->error) st->error = 1;
    });
    if (rd_tell(dec) > 8 * len) return -3;   // OPUS_INTERNAL_ERROR
    return frame_size;
}

} // namespace cuo
