// WeightsManager on the B200 (cpp/skyweaver/src/WeightsManager.cu:16-87).
//
// w = clamp(rn(127 * a * cos(2 pi phi))), clamp(rn(-127 * a * sin(2 pi phi)))
// with phi = ((t - t0) * rate + offset) * f in FP64, exactly the reference
// formula.  Besides the reference [F][B][A] char2 layout the kernel emits the
// A operand of the tensor-core beamformer: for each channel a "re" block of
// rows (w_re, -w_im) and an "im" block of rows (w_im, w_re) per antenna, so
// that D_re = sum(w_re v_re - w_im v_im) and D_im = sum(w_im v_re + w_re v_im)
// are plain int8 GEMMs against the (v_re, v_im) interleaved K dimension.
#include "sw_common.cuh"

namespace swb {
namespace {

constexpr double kTwoPi = 6.283185307179586;  // TWOPI in WeightsManager.cu:9

__device__ __forceinline__ int8_t clamp_int(int v)
{
    // clamp<int8_t, int> (types.cuh:211-221)
    return static_cast<int8_t>(fmaxf(-128.0f, fminf(127.0f, static_cast<float>(v))));
}

__device__ __forceinline__ int8_t neg_sat(int8_t v)
{
    // -(-128) is not representable; it only arises for |antenna weight| > 1.
    return v == -128 ? (int8_t)127 : (int8_t)(-v);
}

// The weight from a single-precision sine and cosine of the phase's fraction
// of a turn (split off exactly in FP64), where that must round to the same
// integer as the FP64 formula.  Errors of 127 a cos: the fraction's rounding
// to float 2 pi 127 a 2^-26, the angle's (factor and product) pi 127 a 2^-23,
// __sincosf's 2^-21.19 on [-pi, pi] 127 a, two products 127 a 2^-23 and, below
// 10^7 turns, the FP64 formula's own 2 pi 10^7 127 a 2^-52: together under
// 1.4e-4 a.  Within 2e-4 a of a half-integer (1 value in 1250), beyond 10^7
// turns and for numbers that are none: false, and the caller takes the formula.
// 2048 beams x 64 antennas x 256 channels: 272 us with the FP64 sine and cosine
// and a flat index per element, 96 us so.
__device__ __forceinline__ bool fast_weight(double phase, float a, int8_t& wr, int8_t& wi)
{
    const double turns = rint(phase);
    float sn, cs;
    __sincosf(6.283185307f * (float)(phase - turns), &sn, &cs);
    const float re = 127.0f * cs * a, im = -127.0f * sn * a;
    const float nr = rintf(re), ni = rintf(im);
    const float limit = 0.5f - 2e-4f * fabsf(a);
    if(!(fabs(turns) < 1e7 && fabsf(re - nr) < limit && fabsf(im - ni) < limit)) return false;
    wr = clamp_int(__float2int_rn(nr));
    wi = clamp_int(__float2int_rn(ni));
    return true;
}

// Both rows of one antenna: `at` is its element in the re block of a channel,
// `block` = nbeams * nant the distance to the im block.
__device__ __forceinline__ void store_gemm(char2* gemm, size_t at, size_t block, int8_t wr,
                                           int8_t wi)
{
    gemm[at]         = make_char2(wr, neg_sat(wi));
    gemm[at + block] = make_char2(wi, wr);
}

// One thread per (beam, antenna) and every gridDim.y-th channel: the delay is
// read and brought to the epoch once, and every index is a sum (the divisions
// that took a flat index apart cost more than the sine and cosine).
__global__ void __launch_bounds__(256)
generate_weights_k(const float3* __restrict__ delays, const double* __restrict__ freqs,
                   size_t block, int nchans, double current_epoch, double delay_epoch,
                   const double* __restrict__ d_epochs, char2* __restrict__ fba,
                   char2* __restrict__ gemm)
{
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if(i >= block) return;
    const float3 dm = delays[i];
    // d_epochs (optional) = {current, delay} on the device, so a captured
    // graph can follow the epoch without re-instantiation
    const double t = d_epochs ? (d_epochs[0] - d_epochs[1]) : (current_epoch - delay_epoch);
    const double delay = t * (double)dm.z + (double)dm.y;
    for(int f = blockIdx.y; f < nchans; f += gridDim.y) {
        const double phase = delay * freqs[f];
        int8_t wr, wi;
        if(!fast_weight(phase, dm.x, wr, wi)) {
            double sn, cs;
            sincos(kTwoPi * phase, &sn, &cs);
            wr = clamp_int(__double2int_rn(cs * 127.0 * (double)dm.x));
            wi = clamp_int(__double2int_rn(-1.0 * sn * 127.0 * (double)dm.x));
        }
        if(fba) fba[f * block + i] = make_char2(wr, wi);
        if(gemm) store_gemm(gemm, 2 * f * block + i, block, wr, wi);
    }
}

__global__ void __launch_bounds__(256)
pack_weights_k(const char2* __restrict__ fba, char2* __restrict__ gemm, size_t block, int nchans)
{
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if(i >= block) return;
    for(int f = blockIdx.y; f < nchans; f += gridDim.y) {
        const char2 w = fba[f * block + i];
        store_gemm(gemm, 2 * f * block + i, block, w.x, w.y);
    }
}

// (beam, antenna) blocks x enough channel slices for 16 CTAs per SM
dim3 weights_grid(size_t block, int nchans)
{
    const size_t x = (block + 255) / 256;
    size_t y = (148 * 16 + x - 1) / x;
    if(y > (size_t)nchans) y = nchans;
    if(y > 65535) y = 65535;
    return dim3((unsigned)x, (unsigned)y);
}

}  // namespace

int launch_weights(const float* d_delays, const double* d_freqs, int nant,
                   int nbeams, int nchans, double current_epoch, double delay_epoch,
                   const double* d_epochs, void* d_fba, void* d_gemm,
                   cudaStream_t stream)
{
    SW_REQUIRE(d_delays && d_freqs, "sw_generate_weights: null input");
    SW_REQUIRE(d_fba || d_gemm, "sw_generate_weights: no output");
    SW_REQUIRE(nant > 0 && nbeams > 0 && nchans > 0, "sw_generate_weights: empty shape");
    const size_t block = (size_t)nbeams * nant;
    generate_weights_k<<<weights_grid(block, nchans), 256, 0, stream>>>(
        reinterpret_cast<const float3*>(d_delays), d_freqs, block, nchans, current_epoch,
        delay_epoch, d_epochs, static_cast<char2*>(d_fba), static_cast<char2*>(d_gemm));
    SW_LAUNCH_CHECK();
    return SW_OK;
}

}  // namespace swb

using namespace swb;

extern "C" {

int sw_generate_weights(const float* d_delays, const double* d_freqs,
                        int nant, int nbeams, int nchans, double current_epoch,
                        double delay_epoch, void* d_weights_fba,
                        void* d_weights_gemm, sw_stream_t stream)
{
    return launch_weights(d_delays, d_freqs, nant, nbeams, nchans, current_epoch,
                          delay_epoch, nullptr, d_weights_fba, d_weights_gemm,
                          as_cuda(stream));
}

int sw_pack_weights(const void* d_weights_fba, void* d_weights_gemm,
                    int nchans, int nbeams, int nant, sw_stream_t stream)
{
    SW_REQUIRE(d_weights_fba && d_weights_gemm, "sw_pack_weights: null pointer");
    if(nchans <= 0 || nbeams <= 0 || nant <= 0) return SW_OK;
    const size_t block = (size_t)nbeams * nant;
    pack_weights_k<<<weights_grid(block, nchans), 256, 0, as_cuda(stream)>>>(
        static_cast<const char2*>(d_weights_fba), static_cast<char2*>(d_weights_gemm), block,
        nchans);
    SW_LAUNCH_CHECK();
    return SW_OK;
}

}  // extern "C"
