// IncoherentDedisperser on the B200
// (cpp/skyweaver/src/IncoherentDedisperser.cu:66-125, a host OpenMP loop in
// the reference).
//
// out[t', d, b] = clamp(sum_{tau < ts} sum_f in[t + tau - delay[d,f], f, b]
//                       / scale_factor),   t = max_delay + t' * ts
// with truncation toward zero (types.cuh:211-221).  The int8 sums are exact
// integers (the reference accumulates them in float, exact below 2^24), so
// the kernels sum bytes in int32 with dp4a: dp4a(word, 1 << 8b, acc) adds
// beam b of a 32-bit word of 4 beams, and on byte-transposed words one dp4a
// adds two or four channels of one beam.  (Biasing each word to unsigned and
// adding pairs of 16-bit lanes, two per instruction, measured 8 % slower
// than one dp4a per addition: it needs a xor and two byte permutes per word
// on the pipe that also issues the adds.)  The final float divide is the
// reference's single IEEE division.
#include "sw_common.cuh"

namespace swb {
namespace {

// One CTA = (trial DM, output sample, block of 128 beam quads).  The linear
// block index runs over the DMs of a group of `group` DMs fastest, then
// output samples, then beam-quad blocks, then DM groups, so the CTAs resident
// at any moment are neighbouring DMs at neighbouring times of one 512-beam
// block: they read nearly the same (time - delay) rows of every channel, a
// window that fits in L2, instead of streaming the rows from HBM once per DM.
__global__ void __launch_bounds__(128)
idd_k(const uint32_t* __restrict__ tfb, int nchans, int nquads,
      const int* __restrict__ delays, int max_delay, int tscrunch,
      float scale_factor, uint32_t* __restrict__ tdb, int ndms, int nout,
      int nqb, int group, long long blk0)
{
    long long blk = blk0 + blockIdx.x;
    const int dl = (int)(blk % group);
    blk /= group;
    const int to = (int)(blk % nout);
    blk /= nout;
    const int qb = (int)(blk % nqb);
    const int d  = (int)(blk / nqb) * group + dl;
    const int q  = qb * blockDim.x + threadIdx.x;
    if(d >= ndms || q >= nquads) return;
    const int t = max_delay + to * tscrunch;
    const int* dl_f = delays + (size_t)d * nchans;
    int acc[4] = {0, 0, 0, 0};
    for(int tau = 0; tau < tscrunch; ++tau) {
#pragma unroll 4
        for(int f = 0; f < nchans; ++f) {
            const size_t row = (size_t)(t + tau - dl_f[f]) * nchans + f;
            const int w = (int)tfb[row * nquads + q];
#pragma unroll
            for(int b = 0; b < 4; ++b) acc[b] = __dp4a(w, 1 << (8 * b), acc[b]);
        }
    }
    uint32_t packed = 0;
#pragma unroll
    for(int k = 0; k < 4; ++k) {
        const float v = fdiv((float)acc[k], scale_factor);
        packed |= ((uint32_t)(uint8_t)clamp_i8(v)) << (8 * k);
    }
    tdb[((size_t)to * ndms + d) * nquads + q] = packed;
}

// 16 sums -> clamp(trunc(sum / scale)) bytes, bit for bit the division's, in
// most cases without one.  q = sum * (1 / scale) lies within 2^-22.4 |q| of the
// rounded quotient, 2.4e-5 inside the clamp.  Away from whole numbers by more
// than 2^-15, trunc(q) is therefore the quotient's; next to a whole n, an FMA
// tells whether sum = n scale exactly, where the quotient is n.  If any of the
// 16 is next to a whole number without being one (1 in 10^4), or the scale's
// reciprocal is no ordinary number, all are divided.  (q -+ 0.5) + 1.5 2^23
// leaves the truncated integer in the low byte.  Clamping to [-128.5, 127.5]
// gives saturated sums the truncated integers 127 and -128 without their lying
// next to a whole number: clamped to the integers themselves they all passed
// for such and were divided (512 beams x 32 trials x 2000 outputs x 24 channels,
// 5 % of the beams saturated: 85 us, 68 us so).  (With 32-bit row offsets, read four at a time:
// 1024 beams x 32 trials x 3968 outputs x 64 channels 605 -> 509 us on their own
// and 596 -> 546 us back to back, 512 x 128 x 4096 x 256 3.78 -> 3.61 ms.)
__device__ __forceinline__ void quantise16(const int* acc, float scale, uint32_t* packed)
{
    const float kMagic = 12582912.0f, kNear = 3.0517578125e-5f;
    const float r = __frcp_rn(scale);
    bool divide = !(fabsf(scale) > 1e-30f && fabsf(scale) < 1e30f);
#pragma unroll
    for(int k = 0; k < 4; ++k) {
        packed[k] = 0;
#pragma unroll
        for(int b = 0; b < 4; ++b) {
            const float x = (float)acc[4 * k + b];
            const float c = fmaxf(-128.5f, fminf(127.5f, fmul(x, r)));
            const float m = fadd(c, kMagic), n = fsub(m, kMagic);
            const bool near = fabsf(fsub(c, n)) < kNear;
            divide |= near && __fmaf_rn(-n, scale, x) != 0.0f;
            const float half = __uint_as_float((__float_as_uint(c) & 0x80000000u) | 0x3f000000u);
            const uint32_t v = __float_as_uint(near ? m : fadd(fsub(c, half), kMagic));
            packed[k] |= (v & 0xffu) << (8 * b);
        }
    }
    if(divide) {
#pragma unroll
        for(int k = 0; k < 4; ++k) {
            packed[k] = 0;
            for(int b = 0; b < 4; ++b)
                packed[k] |= ((uint32_t)(uint8_t)clamp_i8(fdiv((float)acc[4 * k + b], scale)))
                             << (8 * b);
        }
    }
}

// Same sums, 16 beams per thread (one 16-byte load per row): the per-load
// address work is shared by 16 beams and each channel's row offset comes
// from a per-CTA table in shared memory.  A CTA is 128 threads = `tpc` consecutive output samples
// x `lw` lanes of 16 beams (lw <= 32: at most 512 beams), one trial DM.
// Block order as idd_k (DMs of a group fastest, then output chunks, then
// beam blocks, then DM groups), so the CTAs resident at any moment read the
// (time - delay) rows of one 512-beam block, a working set that mostly stays
// in L2.  (All 2048 beams per CTA measured a 38 % L2 hit rate and HBM reads
// of 22x the input; on 4096 samples x 128 DMs x 2048 beams x 256 channels,
// 64/128/256/512/1024/2048 beams per CTA took 44/31/21/20/24/29 ms, and two
// 16-byte loads per thread instead of one 129 -> 154 ms.)
//
// Fewer multiply-add instructions than one dp4a per addition: the words of
// four channels for the same four beams are byte-transposed with PRMT
// (integer ALU pipe) so that one dp4a adds two or four channels of a beam.
// Pair form (words of channels f, f+1 -> [a0 b0 a1 b1], [a2 b2 a3 b3]): 2
// PRMT + 4 dp4a per 8 additions; full form (a second PRMT stage -> [a0 b0 c0
// d0] ...): 8 PRMT + 4 dp4a per 16.  The first NT of the four words of each
// 16-byte load take the full form, the rest the pair form, which splits the
// work between the ALU and the multiply-add pipes.  Channels past the last
// multiple of 4 take one dp4a per addition.  On the case above: one dp4a
// per addition (12 CTAs per SM) 17.3 ms; NT = 0..4 with 8 CTAs per SM 16.3,
// 15.4, 14.9, 15.6, 15.3 ms; NT = 2 with 10 CTAs per SM 14.8 ms, with 12
// (register spills) 23.6 ms.  L2 bandwidth then bounds it: every addition
// reads its byte from L2.
// Beams that are no multiple of 16, or buffers off the 16-byte grid, take the
// same kernel with each lane's 16 beams loaded as 8- or 4-byte words (ALIGN)
// and the words past the last beam left out: 200 beams x 24 trials x 2000
// outputs x 64 channels at tscrunch 2 took 387 us in idd_k, whose CTAs of 128
// quads were 39 % full, and take 138 us.  Row offsets are kept in units of
// ALIGN bytes and in 32 bits where the block of beams allows (OFF).
template <int ALIGN>
__device__ __forceinline__ uint4 load16(const uint8_t* p, int nwords)
{
    if constexpr(ALIGN == 16) {
        return *reinterpret_cast<const uint4*>(p);
    } else if constexpr(ALIGN == 8) {
        const uint2 lo = *reinterpret_cast<const uint2*>(p);
        const uint2 hi = nwords > 2 ? *reinterpret_cast<const uint2*>(p + 8) : make_uint2(0, 0);
        return make_uint4(lo.x, lo.y, hi.x, hi.y);
    } else {
        const uint32_t* w = reinterpret_cast<const uint32_t*>(p);
        return make_uint4(w[0], nwords > 1 ? w[1] : 0, nwords > 2 ? w[2] : 0,
                          nwords > 3 ? w[3] : 0);
    }
}

template <int NT, int MINB, int ALIGN, typename OFF>
__global__ void __launch_bounds__(128, MINB)
idd16q_k(const uint8_t* __restrict__ tfb, int nchans, int nbeams, int nlanes,
         const int* __restrict__ delays, int max_delay, int tscrunch,
         float scale_factor, uint8_t* __restrict__ tdb, int ndms, int nout,
         int nqb, int group, int lw, int ntc, long long blk0)
{
    extern __shared__ __align__(16) uint8_t s_raw[];
    OFF* const s_off = reinterpret_cast<OFF*>(s_raw);  // [nchans] row offsets in ALIGN bytes
    long long blk = blk0 + blockIdx.x;
    const int dl = (int)(blk % group);
    blk /= group;
    const int tc = (int)(blk % ntc);
    blk /= ntc;
    const int qb = (int)(blk % nqb);
    const int d  = (int)(blk / nqb) * group + dl;
    if(d >= ndms) return;  // uniform across the CTA
    const int tpc = blockDim.x / lw;
    const int to = tc * tpc + (int)threadIdx.x / lw;
    const int* dl_f = delays + (size_t)d * nchans;
    const long long row = (long long)nchans * nbeams;  // bytes per time sample
    for(int f = threadIdx.x; f < nchans; f += blockDim.x)
        s_off[f] = (OFF)(((long long)f * nbeams - (long long)dl_f[f] * row) / ALIGN);
    __syncthreads();
    const int q = qb * lw + (int)threadIdx.x % lw;  // 16 beams of this thread
    if((int)threadIdx.x >= tpc * lw || q >= nlanes || to >= nout) return;
    const int nwords = ALIGN == 16 ? 4 : min(4, (nbeams - 16 * q) / 4);
    const int t = max_delay + to * tscrunch;
    int acc[16];
#pragma unroll
    for(int k = 0; k < 16; ++k) acc[k] = 0;
    const int nc4 = nchans & ~3;
    for(int tau = 0; tau < tscrunch; ++tau) {
        const uint8_t* bt = tfb + (long long)(t + tau) * row + 16 * q;
#pragma unroll 2
        for(int f = 0; f < nc4; f += 4) {
            OFF o[4];
            if constexpr(sizeof(OFF) == 4) {
                const int4 v = *reinterpret_cast<const int4*>(s_off + f);
                o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
            } else {
#pragma unroll
                for(int c = 0; c < 4; ++c) o[c] = s_off[f + c];
            }
            const uint4 va = load16<ALIGN>(bt + (long long)o[0] * ALIGN, nwords);
            const uint4 vb = load16<ALIGN>(bt + (long long)o[1] * ALIGN, nwords);
            const uint4 vc = load16<ALIGN>(bt + (long long)o[2] * ALIGN, nwords);
            const uint4 vd = load16<ALIGN>(bt + (long long)o[3] * ALIGN, nwords);
            const uint32_t wa[4] = {va.x, va.y, va.z, va.w};
            const uint32_t wb[4] = {vb.x, vb.y, vb.z, vb.w};
            const uint32_t wc[4] = {vc.x, vc.y, vc.z, vc.w};
            const uint32_t wd[4] = {vd.x, vd.y, vd.z, vd.w};
#pragma unroll
            for(int k = 0; k < 4; ++k) {
                const int t0 = (int)__byte_perm(wa[k], wb[k], 0x5140);  // a0 b0 a1 b1
                const int t1 = (int)__byte_perm(wa[k], wb[k], 0x7362);  // a2 b2 a3 b3
                const int t2 = (int)__byte_perm(wc[k], wd[k], 0x5140);  // c0 d0 c1 d1
                const int t3 = (int)__byte_perm(wc[k], wd[k], 0x7362);  // c2 d2 c3 d3
                int* a = acc + 4 * k;
                if(k < NT) {
                    a[0] = __dp4a((int)__byte_perm(t0, t2, 0x5410), 0x01010101, a[0]);
                    a[1] = __dp4a((int)__byte_perm(t0, t2, 0x7632), 0x01010101, a[1]);
                    a[2] = __dp4a((int)__byte_perm(t1, t3, 0x5410), 0x01010101, a[2]);
                    a[3] = __dp4a((int)__byte_perm(t1, t3, 0x7632), 0x01010101, a[3]);
                } else {
                    a[0] = __dp4a(t2, 0x00000101, __dp4a(t0, 0x00000101, a[0]));
                    a[1] = __dp4a(t2, 0x01010000, __dp4a(t0, 0x01010000, a[1]));
                    a[2] = __dp4a(t3, 0x00000101, __dp4a(t1, 0x00000101, a[2]));
                    a[3] = __dp4a(t3, 0x01010000, __dp4a(t1, 0x01010000, a[3]));
                }
            }
        }
        for(int f = nc4; f < nchans; ++f) {
            const uint4 v = load16<ALIGN>(bt + (long long)s_off[f] * ALIGN, nwords);
            const int w[4] = {(int)v.x, (int)v.y, (int)v.z, (int)v.w};
#pragma unroll
            for(int k = 0; k < 4; ++k)
#pragma unroll
                for(int b = 0; b < 4; ++b)
                    acc[4 * k + b] = __dp4a(w[k], 1 << (8 * b), acc[4 * k + b]);
        }
    }
    uint32_t packed[4];
    quantise16(acc, scale_factor, packed);
    uint8_t* out = tdb + ((size_t)to * ndms + d) * nbeams + 16 * q;
    if constexpr(ALIGN == 16) {
        *reinterpret_cast<uint4*>(out) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
    } else {
#pragma unroll
        for(int k = 0; k < 4; ++k)
            if(k < nwords) reinterpret_cast<uint32_t*>(out)[k] = packed[k];
    }
}

}  // namespace
}  // namespace swb

extern "C" int sw_incoherent_dedisperse(const int8_t* d_tfb, int nsamples,
                                        int nchans, int nbeams,
                                        const int* d_delays, int ndms,
                                        int max_delay, int tscrunch,
                                        float scale_factor, int8_t* d_tdb,
                                        sw_stream_t stream)
{
    SW_REQUIRE(d_tfb && d_delays && d_tdb, "sw_incoherent_dedisperse: null pointer");
    SW_REQUIRE(nsamples > max_delay,
               "Fewer than max_sample_delay samples passed to dedisperse method");
    SW_REQUIRE(tscrunch > 0 && (nsamples - max_delay) % tscrunch == 0,
               "(nsamples - max_sample_delay) must be a multiple of tscrunch;");
    SW_REQUIRE(nbeams % 4 == 0, "sw_incoherent_dedisperse: nbeams must be a multiple of 4");
    SW_REQUIRE(ndms > 0 && ndms <= 65535, "sw_incoherent_dedisperse: bad DM count");
    // what the beams and both buffers allow a lane of 16 beams to load at a time
    const uintptr_t grid = reinterpret_cast<uintptr_t>(d_tfb) | reinterpret_cast<uintptr_t>(d_tdb) |
                           (uintptr_t)nbeams;
    SW_REQUIRE(grid % 4 == 0, "sw_incoherent_dedisperse: the TFB and TDB must be aligned to 4 bytes");
    const int nout = (nsamples - max_delay) / tscrunch;
    const int align = grid % 16 == 0 ? 16 : grid % 8 == 0 ? 8 : 4;
    // idd_k only where a CTA's table of 64-bit row offsets outgrows 48 KB of
    // shared memory (above 6144 channels)
    const bool wide = (size_t)nchans * sizeof(long long) <= 48 * 1024;
    const int nlanes = swb::cdiv(nbeams, wide ? 16 : 4);  // threads per (DM, sample)
    // wide: CTAs of (128 / lw) output samples x lw lanes of 16 beams
    const int lw = wide ? (nlanes < 32 ? nlanes : 32) : 128;
    const int nqb = swb::cdiv(nlanes, lw);
    const int ntc = wide ? swb::cdiv(nout, 128 / lw) : nout;
    const int group = ndms < 16 ? ndms : 16;
    const long long ngroups = swb::cdiv(ndms, group);
    const long long total = ngroups * ntc * nqb * group;
    const long long chunk = 1ll << 30;  // blocks per launch (grid.x limit 2^31 - 1)
    const bool off32 = wide && (long long)nsamples * nchans * nbeams / align < (1ll << 31);
    for(long long b0 = 0; b0 < total; b0 += chunk) {
        const long long n = total - b0 < chunk ? total - b0 : chunk;
        const cudaStream_t s = swb::as_cuda(stream);
        auto launch = [&](auto kernel, size_t off_bytes) {  // two of four words transposed in full
            kernel<<<(unsigned)n, 128, nchans * off_bytes, s>>>(
                reinterpret_cast<const uint8_t*>(d_tfb), nchans, nbeams, nlanes, d_delays, max_delay,
                tscrunch, scale_factor, reinterpret_cast<uint8_t*>(d_tdb), ndms, nout, nqb, group,
                lw, ntc, b0);
        };
        if(align == 16 && off32) launch(swb::idd16q_k<2, 10, 16, int>, 4);
        else if(align == 16 && wide) launch(swb::idd16q_k<2, 10, 16, long long>, 8);
        else if(align == 8 && off32) launch(swb::idd16q_k<2, 10, 8, int>, 4);
        else if(align == 4 && off32) launch(swb::idd16q_k<2, 10, 4, int>, 4);
        else if(wide) launch(swb::idd16q_k<2, 10, 4, long long>, 8);
        else
            swb::idd_k<<<(unsigned)n, 128, 0, s>>>(
                reinterpret_cast<const uint32_t*>(d_tfb), nchans, nlanes, d_delays, max_delay,
                tscrunch, scale_factor, reinterpret_cast<uint32_t*>(d_tdb), ndms, nout, nqb,
                group, b0);
        SW_LAUNCH_CHECK();
    }
    return SW_OK;
}
