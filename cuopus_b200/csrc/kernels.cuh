// Device kernels of libcuopus (sm_100a).
//
//   k_decode_chains   one decoder per group of `width` lanes; the groups of a
//                     launch are resident decoder slots.  Two schedules:
//                       plain      chain c goes to group c % ngroups (static)
//                       queue      groups pull chain indices from a device
//                                  counter in the order given by `order`
//                                  (longest first when the host sorts it);
//                                  the loop is bounded by the chain count
//   k_resample48to16  49-tap Kaiser-windowed sinc, 3:1 decimation of the
//                     compacted int16 48 kHz stream into fp32 16 kHz: input
//                     tiles staged in shared memory, packed FP32 multiply-adds,
//                     outputs staged back and stored as float4.
//
// Arithmetic of the resampler follows the reference kernel
// (cuopus_kernels.cuh:96-111): acc starts at 0 and adds taps[t] * x/32768
// for t = 0..48 in order with a fused multiply-add, samples outside the
// stream read as zero.
#pragma once
#include "dec/chain.cuh"

namespace cuo {

struct DecodeArgs {
    const uint8_t *data;        // packet bytes
    const uint64_t *off;        // per packet offset
    const uint32_t *len;        // per packet length
    const uint32_t *first;      // per chain first packet
    const uint32_t *npkts;      // per chain packet count
    const uint8_t *channels;    // per chain channel count (1 or 2)
    const uint64_t *trim;       // per chain samples to drop (per channel)
    const uint64_t *keep;       // per chain samples to keep (per channel)
    const uint64_t *out_off;    // per chain int16 element offset into out
    int16_t *out;               // kept PCM, interleaved
    const uint32_t *order;      // queue schedule: chain visiting order (may be null)
    const uint64_t *rec_off;    // per chain first per-packet record (may be null)
    uint32_t *pkt_nsamp;        // per-packet records (may be null)
    uint32_t *pkt_rng;
    ChainResult *res;           // per chain result
    ChainSlot *slots;           // one per group of the launch
    unsigned *queue_head;       // queue schedule: next position in `order`
    int nchains;
    int width;                  // lanes per chain: 1, 2, 4, 8, 16 or 32
    int use_queue;
    int stage;                  // packets staged in shared memory (STAGE_BYTES per group)
    int scalar;                 // one active lane per group (the reference kernel's slot layout)
    int fec;                    // in-band FEC for lost packets (decode_chain)
    // Tail scheduling (queue schedule, light_sms > 0): the warps of SMs whose id
    // is below light_sms keep only light_warps of themselves and take the
    // first long_chains positions of the order first; every other SM keeps
    // heavy_warps.  queue_head[0] counts the long positions, queue_head[1] the
    // rest; sm_rank[smid] counts the warps that arrived on each SM.
    unsigned *sm_rank;
    int light_sms, light_warps, heavy_warps, long_chains;
};

// Number of SM ids sm_rank covers (%smid is masked to it).
enum { SM_RANK_SLOTS = 256 };

// Shared memory a block of `block` threads at `width` lanes per chain uses for
// packet staging; 0 (no staging) when it would exceed 48 KB per block.
// Packet staging takes shared memory from the SM's unified L1 / shared
// storage; CUOPUS_STAGE=0 turns it off (all of that storage stays L1).
inline int stage_smem_bytes(int block, int width)
{
    const char *e = getenv("CUOPUS_STAGE");
    if (e && e[0] == '0' && e[1] == 0) return 0;
    int bytes = (block / width) * (int)STAGE_BYTES;
    return bytes <= 48 * 1024 ? bytes : 0;
}

// Decoder kernel: defined in decode_kernel.cu, which is compiled on its own
// (see the note there); the host side reaches it through these calls.  The
// launch decides packet staging from block and width (stage_smem_bytes).
cudaError_t decode_kernel_occupancy(int block, int width, int *blocks_per_sm);
cudaError_t decode_kernel_launch(const DecodeArgs &a, int blocks, int block, cudaStream_t st);

// The 48 -> 16 kHz resampler of libcuopus.cu for other host translation units:
// uploads the taps to the current device on first use, then launches on st.
cudaError_t resample_into(const int16_t *in, long long avail, long long n_out, float *out, cudaStream_t st);

#ifdef CUO_DECODE_KERNEL_TU
// The device's global nanosecond timer (PTX %globaltimer).
__device__ __forceinline__ unsigned long long globaltimer_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Next queue position under tail scheduling: light groups take the long
// positions [0, long_chains) first, the others the rest; each takes from the
// other part when its own is used up.  nchains when nothing is left.
__device__ __forceinline__ unsigned queue_next(const DecodeArgs &a, int light)
{
    const unsigned K = (unsigned)a.long_chains, n = (unsigned)a.nchains;
    if (light) {
        unsigned v = atomicAdd(&a.queue_head[0], 1u);
        if (v < K) return v;
        v = K + atomicAdd(&a.queue_head[1], 1u);
        return v < n ? v : n;
    }
    unsigned v = K + atomicAdd(&a.queue_head[1], 1u);
    if (v < n) return v;
    v = atomicAdd(&a.queue_head[0], 1u);
    return v < K ? v : n;
}

// MIN_BLOCKS: resident 128-thread blocks per SM the register allocation is
// sized for (decode_kernel.cu instantiates 1 and 3 and says which runs when).
template <int MIN_BLOCKS>
__global__ void __launch_bounds__(128, MIN_BLOCKS) k_decode_chains(DecodeArgs a)
{
    hot_fill(&s_hot_tabs, threadIdx.x, blockDim.x);
    __syncthreads();
    const int W = a.width;
    const int lane = threadIdx.x & 31;
    const int sub = lane / W;
    Lanes L;
    L.id = lane - sub * W;
    L.n = W;
    L.mask = W == 32 ? 0xffffffffu : (((1u << W) - 1u) << (sub * W));
    if (a.scalar) {            // the group's first lane decodes alone; the others idle
        if (L.id != 0) return;
        L.n = 1;
        L.mask = 1u << lane;
    }
    const long long gtid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int group = (int)(gtid / W);
    const int ngroups = (int)((long long)gridDim.x * blockDim.x / W);
    ChainSlot *slot = a.slots + group;
    extern __shared__ __align__(16) uint8_t s_stage[];
    PacketStage S;
    PacketStage *stage = nullptr;
    if (a.stage) {
        stage_init(L, S, s_stage + (size_t)(threadIdx.x / W) * STAGE_BYTES);
        stage = &S;
    }
    int light = 0;
    if (a.light_sms > 0) {   // tail scheduling: keep this warp or leave (whole warps, before any decoding)
        unsigned smid, r = 0;
        asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
        if (lane == 0) r = atomicAdd(&a.sm_rank[smid % SM_RANK_SLOTS], 1u);
        r = __shfl_sync(0xffffffffu, r, 0);
        light = smid < (unsigned)a.light_sms;
        if ((int)r >= (light ? a.light_warps : a.heavy_warps)) {
            if (stage) stage_drain(L, *stage);
            return;
        }
    }
    for (int it = 0; it < a.nchains; it++) {
        int pos;
        if (a.use_queue) {
            unsigned v = 0;
            if (L.id == 0) v = a.long_chains > 0 ? queue_next(a, light) : atomicAdd(a.queue_head, 1u);
            v = __shfl_sync(L.mask, v, sub * W);
            pos = (int)v;
        } else {
            pos = group + it * ngroups;
        }
        if (pos >= a.nchains) break;
        int c = a.order ? (int)a.order[pos] : pos;
        unsigned long long t0 = globaltimer_ns();
        decode_chain(L, slot, a.data, a.off, a.len, a.first[c], a.npkts[c], a.channels[c],
                     a.out ? a.out + a.out_off[c] : nullptr, a.trim[c], a.keep[c],
                     a.pkt_nsamp ? a.pkt_nsamp + a.rec_off[c] : nullptr,
                     a.pkt_rng ? a.pkt_rng + a.rec_off[c] : nullptr, &a.res[c], stage, a.fec);
        unsigned long long us = (globaltimer_ns() - t0) / 1000ull;
        if (L.id == 0) a.res[c].time_us = (uint32_t)(us < 1 ? 1 : us > 0xffffffffull ? 0xffffffffull : us);
    }
}
#endif

// The resampler kernel and its taps belong to libcuopus.cu; other host
// translation units define CUO_NO_RESAMPLE_KERNEL and use resample_into.
#if !defined(CUO_DECODE_KERNEL_TU) && !defined(CUO_NO_RESAMPLE_KERNEL)
// Bounds: 10 bytes an output sample against HBM, 49 multiply-adds an output
// against the FP32 pipe; an hour of audio costs 88 us of HBM and 78 us of FMA,
// so both have to be near their rates at once, and shared memory, which every
// operand comes from, is the third (80 % of its rate now).
//   * Packed fma.rn.f32x2 halves the FMA instructions: a thread's outputs come
//     in pairs (i, i + HALF), the tile's inputs are staged as pairs (x[n],
//     x[n + 3 HALF]), and the taps are constants, twice each.  Every output
//     still adds its taps 0..48 in order, one fused multiply-add each, so the
//     sums are the scalar kernel's.
//   * RUN outputs of a half per thread: each staged pair is read once (73
//     8-byte reads for 18 outputs at RUN = 9) and the threads' stride of
//     3 RUN pairs is odd, so the reads do not conflict in the banks.  RUN = 9
//     once four of the five blocks that an SM holds have a tile (rs_run), 3
//     below: a short input is over in one block's latency, which the run sets,
//     and few blocks of nine leave SMs idle.  Microseconds a call with RUN = 3
//     and 9: 0.1 to 2 M samples 13.9-15.5 and 15.7-17.4, 2.1 M 15.0 and 16.6,
//     3 M 15.5 and 15.8, 4 M 16.6 and 17.5, 4.5 M 17.5 and 16.8, 6 M 18.8 and
//     18.4, 10 M 24.0 and 23.4, 20 M 34.7 and 32.1.
//   * Interior tiles read the input as aligned words, neighbouring lanes
//     neighbouring words, whose pairs go to shared memory without conflicts (a
//     16-byte vector per lane stored them 16 to a bank), and a block loads the
//     next tile's words before it computes this one's.
//   * Every mono tile whose output is 16-byte aligned leaves as float4 through
//     shared memory.
// 172,800,001 samples: 395 us as four outputs per thread with scalar FMAs on
// shared reads that conflicted 4 ways; 266 us packed, 200 us with the staging
// stores free of conflicts, 158 us with the next tile's loads in flight (158-169
// a call, by box).
enum { RS_TAPS = 49, RS_PAD = 24, RS_THREADS = 128, RS_BLOCKS = 5 };
constexpr int rs_tile(int run) { return 2 * RS_THREADS * run; }   // outputs per block
inline int rs_run(long long n_out, int sms) { return n_out >= 4ll * sms * rs_tile(9) ? 9 : 3; }

__constant__ uint64_t c_rs_taps[RS_TAPS];   // each tap twice, a pair of floats

__device__ __forceinline__ uint64_t rs_pack(float lo, float hi)
{
    uint64_t v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}

// Two samples / 32768, exactly: the 16 bits as the low mantissa of
// 2^23 + (x + 2^15), then one packed multiply-add.
__device__ __forceinline__ uint64_t rs_pair(uint32_t a16, uint32_t b16)
{
    uint64_t v = rs_pack(__uint_as_float(a16 ^ 0x4B008000u), __uint_as_float(b16 ^ 0x4B008000u));
    const uint64_t scale = rs_pack(1.0f / 32768.0f, 1.0f / 32768.0f);
    const uint64_t shift = rs_pack(-8421376.0f / 32768.0f, -8421376.0f / 32768.0f);
    asm("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(v) : "l"(scale), "l"(shift));
    return v;
}

// out[i * chans] for i in [0, n_out): taps over in[(3 i - 24 + t) * chans], the
// input valid for sample indices [0, avail); chans > 1 resamples one channel of
// an interleaved stream into one channel of an interleaved output.
template <int RUN>
__global__ void __launch_bounds__(RS_THREADS, RS_BLOCKS) k_resample48to16(const int16_t *__restrict__ in, long long avail,
                                                                          long long n_out, float *__restrict__ out,
                                                                          int chans)
{
    constexpr int HALF = RS_THREADS * RUN, TILE = 2 * HALF, PAIRS = 3 * HALF + RS_TAPS - 1;
    constexpr int WORDS = PAIRS / 2, PER = (WORDS + RS_THREADS - 1) / RS_THREADS;
    static_assert(RUN % 2 == 1 && PAIRS % 2 == 0, "odd shared-memory stride, whole words");
    __shared__ __align__(16) uint64_t xs[PAIRS];   // pairs of floats
    __shared__ __align__(16) float ys[TILE];
    const long long tiles = (n_out + TILE - 1) / TILE;
    // elements from the 4-byte boundary below in[0]; every tile's base is even
    const int skew = (int)(((uintptr_t)in & 3) >> 1);
    // an interior mono tile is read as words: word v holds samples 2 v - skew
    // and 2 v - skew + 1 of each half, so lanes take neighbouring words and
    // store their pairs without conflicts
    auto interior = [&](long long tile) {
        const long long base = 3 * tile * TILE - RS_PAD;
        return chans == 1 && base - skew >= 0 && base + 3 * HALF + PAIRS + 2 <= avail;
    };
    uint32_t wa[PER], wb[PER];
    auto load = [&](long long tile) {
        const uint32_t *a = reinterpret_cast<const uint32_t *>(in + 3 * tile * TILE - RS_PAD - skew);
        const uint32_t *b = reinterpret_cast<const uint32_t *>(in + 3 * (tile * TILE + HALF) - RS_PAD - skew);
#pragma unroll
        for (int i = 0; i < PER; i++) {
            const int v = threadIdx.x + i * RS_THREADS;
            if (v < WORDS) {
                wa[i] = a[v];
                wb[i] = b[v];
            }
        }
    };
    long long tile = blockIdx.x;
    if (tile < tiles && interior(tile)) load(tile);
    for (; tile < tiles; tile += gridDim.x) {
        const long long o0 = tile * TILE, base = 3 * o0 - RS_PAD;
        if (interior(tile)) {
#pragma unroll
            for (int i = 0; i < PER; i++) {
                const int v = threadIdx.x + i * RS_THREADS;
                if (v < WORDS) {
                    const uint64_t p0 = rs_pair(wa[i] & 0xffffu, wb[i] & 0xffffu), p1 = rs_pair(wa[i] >> 16, wb[i] >> 16);
                    if (skew == 0) {
                        reinterpret_cast<ulonglong2 *>(xs)[v] = make_ulonglong2(p0, p1);
                    } else {
                        if (v > 0) xs[2 * v - 1] = p0;
                        xs[2 * v] = p1;
                    }
                }
            }
            if (skew && threadIdx.x == 0)
                xs[PAIRS - 1] = rs_pair((uint16_t)in[base + PAIRS - 1], (uint16_t)in[base + 3 * HALF + PAIRS - 1]);
        } else {
            for (int i = threadIdx.x; i < PAIRS; i += RS_THREADS) {
                const long long g = base + i, h = g + 3 * HALF;
                xs[i] = rs_pack((g >= 0 && g < avail) ? (float)in[g * chans] * (1.0f / 32768.0f) : 0.0f,
                                (h >= 0 && h < avail) ? (float)in[h * chans] * (1.0f / 32768.0f) : 0.0f);
            }
        }
        __syncthreads();
        if (tile + gridDim.x < tiles && interior(tile + gridDim.x)) load(tile + gridDim.x);
        uint64_t acc[RUN];
#pragma unroll
        for (int k = 0; k < RUN; k++) acc[k] = 0;
        const uint64_t *x = xs + 3 * RUN * threadIdx.x;
#pragma unroll
        for (int n = 0; n < 3 * (RUN - 1) + RS_TAPS; n++) {
            const uint64_t xn = x[n];
#pragma unroll
            for (int k = 0; k < RUN; k++)
                if (n - 3 * k >= 0 && n - 3 * k < RS_TAPS)
                    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[k]) : "l"(c_rs_taps[n - 3 * k]), "l"(xn));
        }
#pragma unroll
        for (int k = 0; k < RUN; k++) {
            float lo, hi;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(acc[k]));
            ys[RUN * threadIdx.x + k] = lo;
            ys[HALF + RUN * threadIdx.x + k] = hi;
        }
        __syncthreads();
        const long long left = n_out - o0;
        const int cnt = left < TILE ? (int)left : TILE;
        float *o = out + o0 * chans;
        if (chans == 1 && cnt == TILE && ((uintptr_t)o & 15) == 0) {
#pragma unroll
            for (int i = threadIdx.x; i < TILE / 4; i += RS_THREADS)
                reinterpret_cast<float4 *>(o)[i] = reinterpret_cast<const float4 *>(ys)[i];
        } else {
            for (int i = threadIdx.x; i < cnt; i += RS_THREADS) o[(long long)i * chans] = ys[i];
        }
    }
}
#endif

} // namespace cuo
