// Voltage layout kernels: the TAFTP -> FTPA transpose of the reference
// Transposer (cpp/skyweaver/src/Transposer.cu:13-104,117-184), the B200
// TAFTP -> FPACT (planar stream-major) transpose used by the pipeline,
// converters between FTPA and FPACT, and the overlap-save history copy.
//
// Both transposes are pure HBM streaming: every input byte is read once with
// 16-byte loads and every output byte written once with 16- or 4-byte
// stores, so their roofline is the HBM copy bandwidth.
#include "sw_common.cuh"

namespace swb {
namespace {

constexpr int kHeap = 256;  // SKYWEAVER_NSAMPLES_PER_HEAP
constexpr int kPol  = 2;    // SKYWEAVER_NPOL

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel)
{
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}

// ---------------------------------------------------------------------------
// TAFTP -> FTPA.  One CTA per (1 / PARTS heap, channel).  Its A_in x S x P char2
// block (S = 256 / PARTS samples) is staged in shared memory as 32-bit words
// w[a][s] = (p0.re, p0.im, p1.re, p1.im); the word index within a row is
// XOR-swizzled by the antenna group so that the column reads below are
// bank-conflict free.  Each thread then emits 16-byte output chunks
// (8 antennas x char2 of one (t, pol) row), fully coalesced.
// Half heaps (29 KiB for 57 antennas) let several CTAs per SM overlap their
// loads and stores: 57 of 64 antennas x 64 channels x 67 heaps 104 us, whole
// heaps 133 us.  With few antennas whole heaps fit as many CTAs and are ahead
// once these fill several waves: 9 heaps x 600 channels of 16 antennas 35.1
// against 37.6 us, of 24 52.5 against 54.4, of 32 71 against 69; 512 CTAs of 24
// antennas 5.7 against 5.3.
// ---------------------------------------------------------------------------
constexpr int kWholeHeapAnt = 24, kWholeHeapCtas = 2048;

template <int S>
__device__ __forceinline__ int swz_word(int a, int s)
{
    return a * S + (s ^ (((a >> 3) & 7) << 2));
}

template <int PARTS>
__global__ void __launch_bounds__(256)
transpose_ftpa_k(const uint4* __restrict__ taftp, uint4* __restrict__ ftpa,
                 int in_nant, int out_nant, int nchans, int nheaps)
{
    constexpr int S = kHeap / PARTS, C = S / 4;  // samples, 16-byte chunks of an antenna
    extern __shared__ uint32_t sm_words[];
    const int h = blockIdx.x;
    const int f = blockIdx.y;
    const int z = blockIdx.z;  // part of the heap
    // stage: A_in x C chunks of 16 bytes (4 samples x 2 pols x char2)
    for(int idx = threadIdx.x; idx < in_nant * C; idx += blockDim.x) {
        const int a = (unsigned)idx / C, c = idx & (C - 1);
        const size_t src = (((size_t)h * in_nant + a) * nchans + f) * 64 + C * z + c;
        uint4 v = taftp[src];
        uint4* dst = reinterpret_cast<uint4*>(&sm_words[swz_word<S>(a, c * 4)]);
        *dst = v;
    }
    __syncthreads();
    const int groups = out_nant >> 3;  // 8 antennas -> 16 bytes per row
    const size_t nsamp = (size_t)nheaps * kHeap;
    for(int idx = threadIdx.x; idx < groups * S; idx += blockDim.x) {
        const int g = idx % groups;
        const int s = idx / groups;
        uint32_t w[8];
#pragma unroll
        for(int i = 0; i < 8; ++i) {
            const int a = g * 8 + i;
            w[i] = (a < in_nant) ? sm_words[swz_word<S>(a, s)] : 0u;
        }
        uint4 o0, o1;
        o0.x = prmt(w[0], w[1], 0x5410); o1.x = prmt(w[0], w[1], 0x7632);
        o0.y = prmt(w[2], w[3], 0x5410); o1.y = prmt(w[2], w[3], 0x7632);
        o0.z = prmt(w[4], w[5], 0x5410); o1.z = prmt(w[4], w[5], 0x7632);
        o0.w = prmt(w[6], w[7], 0x5410); o1.w = prmt(w[6], w[7], 0x7632);
        const size_t t   = (size_t)h * kHeap + z * S + s;
        const size_t row = ((size_t)f * nsamp + t) * kPol;  // (f, t, p=0)
        // row of out_nant char2 = out_nant/8 uint4
        ftpa[row * groups + g]           = o0;
        ftpa[(row + 1) * groups + g]     = o1;
    }
}

// ---------------------------------------------------------------------------
// TAFTP -> FPACT.  One CTA per (heap, channel); 64 threads per antenna, each
// turning 16 input bytes (4 samples x 2 pols x re/im) into one 32-bit word
// in each of the four planar rows (p0.re, p0.im, p1.re, p1.im).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
transpose_fpact_k(const uint4* __restrict__ taftp, uint8_t* __restrict__ fpact,
                  int in_nant, int out_nant, int nchans, size_t row_stride,
                  size_t sample_offset)
{
    const int h = blockIdx.x;
    const int f = blockIdx.y;
    for(int idx = threadIdx.x; idx < out_nant * 64; idx += blockDim.x) {
        const int a = idx >> 6, c = idx & 63;
        uint32_t r0 = 0, r1 = 0, r2 = 0, r3 = 0;
        if(a < in_nant) {
            const size_t src = (((size_t)h * in_nant + a) * nchans + f) * 64 + c;
            uint4 v = taftp[src];
            uint32_t t0 = prmt(v.x, v.y, 0x5140), t1 = prmt(v.z, v.w, 0x5140);
            uint32_t t2 = prmt(v.x, v.y, 0x7362), t3 = prmt(v.z, v.w, 0x7362);
            r0 = prmt(t0, t1, 0x5410);  // p0 re
            r1 = prmt(t0, t1, 0x7632);  // p0 im
            r2 = prmt(t2, t3, 0x5410);  // p1 re
            r3 = prmt(t2, t3, 0x7632);  // p1 im
        }
        const size_t s = sample_offset + (size_t)h * kHeap + c * 4;
        const size_t base0 = ((((size_t)f * kPol + 0) * out_nant + a) * 2) * row_stride + s;
        const size_t base1 = ((((size_t)f * kPol + 1) * out_nant + a) * 2) * row_stride + s;
        *reinterpret_cast<uint32_t*>(fpact + base0)              = r0;
        *reinterpret_cast<uint32_t*>(fpact + base0 + row_stride) = r1;
        *reinterpret_cast<uint32_t*>(fpact + base1)              = r2;
        *reinterpret_cast<uint32_t*>(fpact + base1 + row_stride) = r3;
    }
}

// FTPA <-> FPACT converters (reference-layout stage wrappers and tests).  Both
// layouts number the 4 nant bytes of a sample the same way (pol, antenna,
// re|im), so per channel this is a byte transpose of [nsamples][4 nant] to
// [4 nant][row_stride].  A CTA takes 128 samples x 64 words (64 antennas): it
// reads words along the contiguous side of the source, passes them through
// shared memory and writes words along the contiguous side of the
// destination, four 32-bit words byte-transposed by PRMT per thread.  Word
// (sample t, column w) lies at column w ^ (t / 4 mod 32), which keeps both
// the accesses along w and those along t (4 samples apart) free of bank
// conflicts.  64 antennas x 16 channels x 8192 samples took 287 us with a byte
// access per value and takes 13 us so (67 MB, 5.1 TB/s, back to back in L2).
// Bases, strides or offsets off the 4-byte grid take the byte accesses of
// `row_words` = 0, as does a last group of fewer than 4 samples.
constexpr int kConvT = 128, kConvW = 64;
constexpr int kDirectAnt = 6, kDirectTiles = 24, kDirectTilesOff = 148;  // see convert_direct_k

// up to four bytes of p as a word, loaded as one where `word`
__device__ __forceinline__ uint32_t load_bytes(const uint8_t* p, int n, bool word)
{
    if(word) return *reinterpret_cast<const uint32_t*>(p);
    uint32_t v = 0;
#pragma unroll
    for(int k = 0; k < 4; ++k)
        if(k < n) v |= (uint32_t)p[k] << (8 * k);
    return v;
}
__device__ __forceinline__ void store_bytes(uint8_t* p, uint32_t v, int n, bool word)
{
    if(word) {
        *reinterpret_cast<uint32_t*>(p) = v;
        return;
    }
#pragma unroll
    for(int k = 0; k < 4; ++k)
        if(k < n) p[k] = (uint8_t)(v >> (8 * k));
}
// byte i of x[j] to byte j of y[i]
__device__ __forceinline__ void transpose4(const uint32_t* x, uint32_t* y)
{
    const uint32_t a = prmt(x[0], x[1], 0x5140), b = prmt(x[2], x[3], 0x5140);
    const uint32_t c = prmt(x[0], x[1], 0x7362), d = prmt(x[2], x[3], 0x7362);
    y[0] = prmt(a, b, 0x5410);
    y[1] = prmt(a, b, 0x7632);
    y[2] = prmt(c, d, 0x5410);
    y[3] = prmt(c, d, 0x7632);
}

template <bool TO_FPACT>
__global__ void __launch_bounds__(256)
convert_k(uint8_t* __restrict__ ftpa, uint8_t* __restrict__ fpact, int nsamples, int nant,
          size_t row_stride, size_t sample_offset, int row_words, int ftpa_words)
{
    __shared__ uint32_t sm[kConvT][kConvW];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t0 = blockIdx.x * kConvT, w0 = blockIdx.y * kConvW, f = blockIdx.z;
    const int nt = min(kConvT, nsamples - t0), nw = min(kConvW, nant - w0);
    uint8_t* const samples = ftpa + ((size_t)f * nsamples + t0) * 4 * nant + 4 * (size_t)w0;
    uint8_t* const rows = fpact + ((size_t)f * 4 * nant + 4 * (size_t)w0) * row_stride +
                          sample_offset + t0;
    // Both sides issue a batch of loads before the first is used: one at a time
    // took 142 us (back 126) for 64 antennas x 64 channels x 16384 samples, and
    // takes 100 (106) so.
    // the FTPA side: one warp per sample, 32 words at a time
    auto ftpa_side = [&] {
        for(int tb = warp; tb < nt; tb += 32) {
            uint32_t v[4][2];
#pragma unroll
            for(int i = 0; i < 8; ++i) {
                const int t = tb + 8 * (i / 2), w = lane + 32 * (i & 1);
                if(t >= nt || w >= nw) continue;
                uint32_t& s = sm[t][w ^ ((t >> 2) & 31)];
                uint8_t* g = samples + (size_t)t * 4 * nant + 4 * w;
                if(TO_FPACT) v[i / 2][i & 1] = load_bytes(g, 4, ftpa_words);
                else store_bytes(g, s, 4, ftpa_words);
            }
            if constexpr(TO_FPACT) {
#pragma unroll
                for(int i = 0; i < 8; ++i) {
                    const int t = tb + 8 * (i / 2), w = lane + 32 * (i & 1);
                    if(t < nt && w < nw) sm[t][w ^ ((t >> 2) & 31)] = v[i / 2][i & 1];
                }
            }
        }
    };
    // the FPACT side: one warp per word (4 rows), 4 samples per lane
    auto fpact_side = [&] {
        const int t = 4 * lane, n = min(4, nt - t);
        if(n <= 0) return;
        const bool word = row_words && n == 4;
        for(int wb = warp; wb < nw; wb += 16) {
            uint32_t x[2][4], y[4];
#pragma unroll
            for(int i = 0; i < 2; ++i) {
                const int w = wb + 8 * i;
                if(w >= nw) break;
                const uint8_t* g = rows + (size_t)(4 * w) * row_stride + t;
#pragma unroll
                for(int k = 0; k < 4; ++k)  // TO_FPACT: samples past nt are not stored
                    x[i][k] = TO_FPACT ? sm[t + k][w ^ lane] : load_bytes(g + k * row_stride, n, word);
            }
#pragma unroll
            for(int i = 0; i < 2; ++i) {
                const int w = wb + 8 * i;
                if(w >= nw) break;
                uint8_t* g = rows + (size_t)(4 * w) * row_stride + t;
                transpose4(x[i], y);
#pragma unroll
                for(int k = 0; k < 4; ++k) {
                    if(TO_FPACT) store_bytes(g + k * row_stride, y[k], n, word);
                    else sm[t + k][w ^ lane] = y[k];
                }
            }
        }
    };
    if(TO_FPACT) ftpa_side(); else fpact_side();
    __syncthreads();
    if(TO_FPACT) fpact_side(); else ftpa_side();
}

// The same for launches whose tiles would be mostly empty (up to kDirectAnt
// antennas) or too few to fill the SMs: a thread per (4 samples, antenna) with
// its four words in registers.  Its accesses on the FTPA side are 4 nant bytes
// apart, which the L1 gathers as long as there are few.  Tiles / direct, to
// FPACT and back: 64 channels x 16384 samples of 1 antenna 48, 35 / 2.9, 3.3 us, of
// 6 51, 38 / 18, 30 us, of 8 53, 39 / 36, 46 us; 64 antennas in 8 tiles 4.5, 5.1 /
// 2.5, 2.9 us, in 32 4.5, 5.3 / 4.5, 5.8 us.  Rows off the 4-byte grid cost the
// tiles more: 99 of them back 10.3 / 7.4 us.
template <bool TO_FPACT>
__global__ void __launch_bounds__(256)
convert_direct_k(uint8_t* __restrict__ ftpa, uint8_t* __restrict__ fpact, int nsamples, int nant,
                 size_t row_stride, size_t sample_offset, int row_words, int ftpa_words)
{
    const int t = 4 * (blockIdx.x * 256 + threadIdx.x), a = blockIdx.y, f = blockIdx.z;
    if(t >= nsamples) return;
    const int n = min(4, nsamples - t);
    uint8_t* s = ftpa + (((size_t)f * nsamples + t) * nant + a) * 4;
    uint8_t* r = fpact + ((size_t)f * nant + a) * 4 * row_stride + sample_offset + t;
    const bool word = row_words && n == 4;
    uint32_t x[4] = {0, 0, 0, 0}, y[4];
#pragma unroll
    for(int k = 0; k < 4; ++k) {
        if(!TO_FPACT) x[k] = load_bytes(r + k * row_stride, n, word);
        else if(k < n) x[k] = load_bytes(s + (size_t)k * 4 * nant, 4, ftpa_words);
    }
    transpose4(x, y);
#pragma unroll
    for(int k = 0; k < 4; ++k) {
        if(TO_FPACT) store_bytes(r + k * row_stride, y[k], n, word);
        else if(k < n) store_bytes(s + (size_t)k * 4 * nant, y[k], 4, ftpa_words);
    }
}

// the last history16 16-byte chunks of every row of `src` to the front of
// the same row of `dst` (src == dst: in place)
__global__ void keep_history_k(const uint4* src, uint4* dst, size_t nrows,
                               size_t row_stride16, size_t history16,
                               size_t nsamples16)
{
    const size_t total = nrows * history16;
    for(size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total;
        i += (size_t)gridDim.x * blockDim.x) {
        const size_t row = i / history16, k = i % history16;
        dst[row * row_stride16 + k] = src[row * row_stride16 + nsamples16 + k];
    }
}

int grid_for(size_t work, int block)
{
    size_t g = (work + block - 1) / block;
    if(g > 148 * 32) g = 148 * 32;
    return (int)(g ? g : 1);
}

}  // namespace
}  // namespace swb

using namespace swb;

extern "C" {

int sw_transpose_ftpa(const void* d_taftp, void* d_ftpa, int nheaps,
                      int input_nantennas, int output_nantennas, int nchans,
                      sw_stream_t stream)
{
    SW_REQUIRE(d_taftp && d_ftpa, "sw_transpose_ftpa: null pointer");
    SW_REQUIRE(nheaps > 0 && nchans > 0, "sw_transpose_ftpa: empty input");
    SW_REQUIRE(input_nantennas > 0 && input_nantennas <= output_nantennas,
               "Input number of antennas must be <= to the maximum nantennas");
    SW_REQUIRE(output_nantennas % 8 == 0 && output_nantennas <= 256,
               "sw_transpose_ftpa: output antennas must be a multiple of 8 and <= 256");
    SW_REQUIRE(nheaps <= 65535 && nchans <= 65535, "sw_transpose_ftpa: grid too large");
    auto launch = [&](auto kernel, int parts) {
        const size_t smem = (size_t)input_nantennas * (kHeap / parts) * 4;
        SW_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem));
        kernel<<<dim3(nheaps, nchans, parts), 256, smem, as_cuda(stream)>>>(
            static_cast<const uint4*>(d_taftp), static_cast<uint4*>(d_ftpa), input_nantennas,
            output_nantennas, nchans, nheaps);
        SW_LAUNCH_CHECK();
        return SW_OK;
    };
    const bool whole = input_nantennas <= kWholeHeapAnt && (long)nheaps * nchans >= kWholeHeapCtas;
    return whole ? launch(transpose_ftpa_k<1>, 1) : launch(transpose_ftpa_k<2>, 2);
}

int sw_transpose_fpact(const void* d_taftp, void* d_fpact, int nheaps,
                       int input_nantennas, int output_nantennas, int nchans,
                       size_t row_stride, size_t sample_offset,
                       sw_stream_t stream)
{
    SW_REQUIRE(d_taftp && d_fpact, "sw_transpose_fpact: null pointer");
    SW_REQUIRE(nheaps > 0 && nchans > 0, "sw_transpose_fpact: empty input");
    SW_REQUIRE(input_nantennas > 0 && input_nantennas <= output_nantennas,
               "Input number of antennas must be <= to the maximum nantennas");
    SW_REQUIRE(row_stride % 16 == 0 && sample_offset % 16 == 0,
               "sw_transpose_fpact: row stride and offset must be multiples of 16");
    SW_REQUIRE(sample_offset + (size_t)nheaps * kHeap <= row_stride,
               "sw_transpose_fpact: rows too short for the gulp");
    SW_REQUIRE(nheaps <= 65535 && nchans <= 65535, "sw_transpose_fpact: grid too large");
    dim3 grid(nheaps, nchans);
    transpose_fpact_k<<<grid, 256, 0, as_cuda(stream)>>>(
        static_cast<const uint4*>(d_taftp), static_cast<uint8_t*>(d_fpact),
        input_nantennas, output_nantennas, nchans, row_stride, sample_offset);
    SW_LAUNCH_CHECK();
    return SW_OK;
}

static int convert(const void* ftpa, void* fpact, int nchans, int nsamples,
                   int nant, size_t row_stride, size_t off, sw_stream_t stream,
                   int to_fpact)
{
    SW_REQUIRE(ftpa && fpact, "FTPA/FPACT conversion: null pointer");
    SW_REQUIRE(nsamples > 0 && nchans > 0 && nant > 0, "FTPA/FPACT conversion: empty shape");
    SW_REQUIRE(off + nsamples <= row_stride, "FTPA/FPACT conversion: rows too short");
    const int row_words = row_stride % 4 == 0 && off % 4 == 0 &&
                          (reinterpret_cast<uintptr_t>(fpact) & 3) == 0;
    const int ftpa_words = (reinterpret_cast<uintptr_t>(ftpa) & 3) == 0;
    uint8_t* fp = static_cast<uint8_t*>(fpact);
    uint8_t* ft = static_cast<uint8_t*>(const_cast<void*>(ftpa));
    // grid.y and grid.z end at 65535: 64 antennas and one channel apiece
    const long tiles = (long)cdiv(nsamples, kConvT) * cdiv(nant, kConvW) * nchans;
    const bool direct = nant <= kDirectAnt ||
                        (tiles < (row_words ? kDirectTiles : kDirectTilesOff) && nant <= 65535);
    for(int f0 = 0; f0 < nchans; f0 += 65535) {
        const int nf = nchans - f0 < 65535 ? nchans - f0 : 65535;
        const dim3 grid = direct ? dim3(cdiv(cdiv(nsamples, 4), 256), nant, nf)
                                 : dim3(cdiv(nsamples, kConvT), cdiv(nant, kConvW), nf);
        auto* kernel = direct ? (to_fpact ? convert_direct_k<true> : convert_direct_k<false>)
                              : (to_fpact ? convert_k<true> : convert_k<false>);
        kernel<<<grid, 256, 0, as_cuda(stream)>>>(ft + (size_t)f0 * nsamples * 4 * nant,
                                                  fp + (size_t)f0 * 4 * nant * row_stride,
                                                  nsamples, nant, row_stride, off, row_words,
                                                  ftpa_words);
        SW_LAUNCH_CHECK();
    }
    return SW_OK;
}

int sw_ftpa_to_fpact(const void* d_ftpa, void* d_fpact, int nchans,
                     int nsamples, int nantennas, size_t row_stride,
                     size_t sample_offset, sw_stream_t stream)
{
    return convert(d_ftpa, d_fpact, nchans, nsamples, nantennas, row_stride,
                   sample_offset, stream, 1);
}

int sw_fpact_to_ftpa(const void* d_fpact, void* d_ftpa, int nchans,
                     int nsamples, int nantennas, size_t row_stride,
                     size_t sample_offset, sw_stream_t stream)
{
    return convert(d_ftpa, const_cast<void*>(d_fpact), nchans, nsamples,
                   nantennas, row_stride, sample_offset, stream, 0);
}

int sw_fpact_keep_history(void* d_fpact, size_t nrows, size_t row_stride,
                          size_t history, sw_stream_t stream)
{
    SW_REQUIRE(d_fpact, "sw_fpact_keep_history: null pointer");
    SW_REQUIRE(row_stride % 16 == 0 && history % 16 == 0,
               "sw_fpact_keep_history: stride and history must be multiples of 16");
    if(history == 0 || nrows == 0) return SW_OK;
    SW_REQUIRE(row_stride >= 2 * history,
               "sw_fpact_keep_history: rows must hold at least twice the history");
    // rows hold [history | nsamples] with nsamples = row_stride - history
    const size_t nsamples = row_stride - history;
    const size_t work = nrows * (history / 16);
    keep_history_k<<<grid_for(work, 256), 256, 0, as_cuda(stream)>>>(
        static_cast<const uint4*>(d_fpact), static_cast<uint4*>(d_fpact), nrows,
        row_stride / 16, history / 16, nsamples / 16);
    SW_LAUNCH_CHECK();
    return SW_OK;
}

int sw_fpact_copy_history(const void* d_prev, void* d_next, size_t nrows, size_t row_stride,
                          size_t history, sw_stream_t stream)
{
    SW_REQUIRE(d_prev && d_next, "sw_fpact_copy_history: null pointer");
    SW_REQUIRE(row_stride % 16 == 0 && history % 16 == 0 &&
                   (reinterpret_cast<uintptr_t>(d_prev) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(d_next) & 15) == 0,
               "sw_fpact_copy_history: pointers, stride and history must be multiples of 16");
    if(history == 0 || nrows == 0) return SW_OK;
    SW_REQUIRE(row_stride >= 2 * history,
               "sw_fpact_copy_history: rows must hold at least twice the history");
    const size_t nsamples = row_stride - history;
    const size_t work = nrows * (history / 16);
    keep_history_k<<<grid_for(work, 256), 256, 0, as_cuda(stream)>>>(
        static_cast<const uint4*>(d_prev), static_cast<uint4*>(d_next), nrows,
        row_stride / 16, history / 16, nsamples / 16);
    SW_LAUNCH_CHECK();
    return SW_OK;
}

}  // extern "C"
