// IncoherentBeamformer on the B200
// (cpp/skyweaver/src/IncoherentBeamformer.cu:15-91; CPU form
//  cpp/skyweaver/test/src/IncoherentBeamformerTester.cu:41-103).
//
// P[s,t',f] = sum_{t in t'} sum_a w[s,a] * Stokes(v_p0, v_p1)  (float, in the
// reference's (t outer, a inner) order), then int8 = clamp(rint(rescale)).
//
// Every Stokes term of int8 voltages is an exact integer, so when the
// antenna weights are integers the float chain is exact as long as the sum
// of |terms| stays below 2^24.  The kernel therefore sums the terms with
// dp4a in integers, checks that bound, and only walks the float chain in the
// reference order (slow path) for outputs that fail it.  The result is
// bit-identical to the reference's CPU implementation in both cases.
//
// ib_k: one thread per (channel, output sample); the planar FPACT rows make
// each thread's tscrunch samples a contiguous 4/8/16-byte load, coalesced across
// the warp.  ib_run_k, for tscrunch 4 to 32 on aligned rows: 16-byte runs of
// every row, the antennas over four warps.  Both are HBM bound (one read of the
// voltages).
#include "sw_common.cuh"

namespace swb {
namespace {

constexpr int kMaxBs = 8;          // beamsets per pass (registers)
constexpr int kMaxAnt = 256;
constexpr int kTableAnt = 64;  // antennas of the float-chain product table (4 KB a thread)

// signed byte k (0..15, unrolled) of a 16-byte load
__device__ __forceinline__ int sbyte(const uint4& v, int k)
{
    const uint32_t w = k < 4 ? v.x : k < 8 ? v.y : k < 12 ? v.z : v.w;
    return (int)(int8_t)(w >> (8 * (k & 3)));
}

struct IbArgs {
    const uint8_t* fpact;
    size_t row_stride, offset;
    int nchans, nsamples, nant, tscrunch, nbeamsets, stokes;
    const float *scale, *offset_v, *weights;
    float* raw;
    int8_t* out;
    const int* chan_order;  // CTA row -> channel (nullptr: identity)
};

__device__ __forceinline__ float stokes_f(int stokes, float r0, float i0,
                                          float r1, float i1)
{
    // beamformer_utils.cuh:125-140 with the reference's op order
    switch(stokes) {
    case 0: return fadd(fadd(fmul(r0, r0), fmul(i0, i0)), fadd(fmul(r1, r1), fmul(i1, i1)));
    case 1: return fsub(fadd(fmul(r0, r0), fmul(i0, i0)), fadd(fmul(r1, r1), fmul(i1, i1)));
    case 2: return fmul(2.0f, fsub(fmul(r0, r1), fmul(i0, -i1)));
    default: return fmul(2.0f, fadd(fmul(r0, -i1), fmul(i0, r1)));
    }
}

// NC = 1: one Stokes parameter (args.stokes); NC = 4: I, Q, U, V
// (FullStokesBeamformerTraits, beamformer_utils.cuh:198-278: float4 raw power,
// char4 output, component c computed exactly like single-Stokes mode c).
template <int NC>
__global__ void __launch_bounds__(128)
ib_k(IbArgs args, int bs0)
{
    constexpr int kBs = kMaxBs / NC;  // beamsets per pass
    __shared__ float sw[kBs][kMaxAnt];
    __shared__ int s_intw[kBs];
    const int nbs = min(kBs, args.nbeamsets - bs0);
    for(int i = threadIdx.x; i < kBs * args.nant; i += blockDim.x) {
        const int s = i / args.nant, a = i % args.nant;
        sw[s][a] = (s < nbs) ? args.weights[(size_t)(bs0 + s) * args.nant + a] : 0.0f;
    }
    __syncthreads();
    if(threadIdx.x < kBs) {
        int ok = 1;
        for(int a = 0; a < args.nant; ++a) {
            const float w = sw[threadIdx.x][a];
            ok &= (w == rintf(w)) && fabsf(w) <= 1024.0f;
        }
        s_intw[threadIdx.x] = ok;
    }
    __syncthreads();

    const int nout = args.nsamples / args.tscrunch;
    const int tp = blockIdx.x * blockDim.x + threadIdx.x;
    const int f  = args.chan_order ? args.chan_order[blockIdx.y] : (int)blockIdx.y;
    if(tp >= nout) return;
    const int t0 = tp * args.tscrunch;
    const size_t P = 2;
    long long S[kBs * NC], B[kBs];
#pragma unroll
    for(int s = 0; s < kBs; ++s) {
        B[s] = 0;
#pragma unroll
        for(int c = 0; c < NC; ++c) S[s * NC + c] = 0;
    }

    const bool words = (args.tscrunch % 4) == 0;
    // 16-byte loads when each thread's samples are whole aligned 16-byte runs
    const bool quads = (args.tscrunch % 16) == 0 && (args.row_stride % 16) == 0 &&
                       (args.offset % 16) == 0 &&
                       (reinterpret_cast<uintptr_t>(args.fpact) & 15) == 0;
#pragma unroll 2  // two antennas' loads in flight: 3 % faster on 64 channels
    for(int a = 0; a < args.nant; ++a) {
        const uint8_t* r0 = args.fpact + (((size_t)f * P + 0) * args.nant + a) * 2 * args.row_stride + args.offset + t0;
        const uint8_t* r1 = args.fpact + (((size_t)f * P + 1) * args.nant + a) * 2 * args.row_stride + args.offset + t0;
        int pI = 0, pQ = 0, pU = 0, pV = 0;
        if(quads) {
            for(int k = 0; k < args.tscrunch; k += 16) {
                const uint4 R0 = *reinterpret_cast<const uint4*>(r0 + k);
                const uint4 I0 = *reinterpret_cast<const uint4*>(r0 + args.row_stride + k);
                const uint4 R1 = *reinterpret_cast<const uint4*>(r1 + k);
                const uint4 I1 = *reinterpret_cast<const uint4*>(r1 + args.row_stride + k);
                const int xr0[4] = {(int)R0.x, (int)R0.y, (int)R0.z, (int)R0.w};
                const int xi0[4] = {(int)I0.x, (int)I0.y, (int)I0.z, (int)I0.w};
                const int xr1[4] = {(int)R1.x, (int)R1.y, (int)R1.z, (int)R1.w};
                const int xi1[4] = {(int)I1.x, (int)I1.y, (int)I1.z, (int)I1.w};
#pragma unroll
                for(int q = 0; q < 4; ++q) {
                    const int e0 = __dp4a(xi0[q], xi0[q], __dp4a(xr0[q], xr0[q], 0));
                    const int e1 = __dp4a(xi1[q], xi1[q], __dp4a(xr1[q], xr1[q], 0));
                    pI += e0 + e1;
                    pQ += e0 - e1;
                    pU += __dp4a(xi0[q], xi1[q], __dp4a(xr0[q], xr1[q], 0));
                    pV += __dp4a(xi0[q], xr1[q], 0) - __dp4a(xr0[q], xi1[q], 0);
                }
            }
        } else if(words) {
            for(int k = 0; k < args.tscrunch; k += 4) {
                const int xr0 = *reinterpret_cast<const int*>(r0 + k);
                const int xi0 = *reinterpret_cast<const int*>(r0 + args.row_stride + k);
                const int xr1 = *reinterpret_cast<const int*>(r1 + k);
                const int xi1 = *reinterpret_cast<const int*>(r1 + args.row_stride + k);
                const int e0 = __dp4a(xi0, xi0, __dp4a(xr0, xr0, 0));
                const int e1 = __dp4a(xi1, xi1, __dp4a(xr1, xr1, 0));
                pI += e0 + e1;
                pQ += e0 - e1;
                pU += __dp4a(xi0, xi1, __dp4a(xr0, xr1, 0));
                pV += __dp4a(xi0, xr1, 0) - __dp4a(xr0, xi1, 0);
            }
        } else {
            for(int k = 0; k < args.tscrunch; ++k) {
                const int xr0 = (int8_t)r0[k], xi0 = (int8_t)r0[args.row_stride + k];
                const int xr1 = (int8_t)r1[k], xi1 = (int8_t)r1[args.row_stride + k];
                const int e0 = xr0 * xr0 + xi0 * xi0, e1 = xr1 * xr1 + xi1 * xi1;
                pI += e0 + e1;
                pQ += e0 - e1;
                pU += xr0 * xr1 + xi0 * xi1;
                pV += xi0 * xr1 - xr0 * xi1;
            }
        }
        int pv[NC];
        if constexpr(NC == 4) {
            pv[0] = pI; pv[1] = pQ; pv[2] = 2 * pU; pv[3] = 2 * pV;
        } else {
            pv[0] = args.stokes == 0 ? pI : args.stokes == 1 ? pQ
                  : args.stokes == 2 ? 2 * pU : 2 * pV;
        }
#pragma unroll
        for(int s = 0; s < kBs; ++s) {
            const int wi = (int)sw[s][a];
#pragma unroll
            for(int c = 0; c < NC; ++c) S[s * NC + c] += (long long)wi * pv[c];
            B[s] += (long long)abs(wi) * pI;  // |Q|,|U|,|V| <= I per sample
        }
    }

    for(int s = 0; s < nbs; ++s) {
        const int bs = bs0 + s;
        const size_t o  = ((size_t)bs * nout + tp) * args.nchans + f;
        const size_t so = (size_t)bs * args.nchans + f;
        for(int c = 0; c < NC; ++c) {
            const int stokes = NC == 4 ? c : args.stokes;
            float power;
            if(s_intw[s] && B[s] <= (1ll << 24)) {
                power = (float)S[s * NC + c];  // the float chain is exact
            } else if(quads && args.nant <= kTableAnt) {
                // reference order (t outer, a inner) from a table of the
                // products: each antenna's four 16-sample rows are read once
                // with 16-byte loads, the 16 x nant products go to a
                // per-thread table in local memory (lane-interleaved, so
                // coalesced and mostly L1/L2 resident), and the chain then
                // walks the table.  Walking the rows byte by byte in chain
                // order instead re-reads every row once per sample, because
                // the warp's 4 rows x nant windows do not stay in L1.
                power = 0.0f;
                for(int tc = 0; tc < args.tscrunch; tc += 16) {
                    float x[16][kTableAnt];
#pragma unroll 4
                    for(int a = 0; a < args.nant; ++a) {
                        const uint8_t* q0 = args.fpact + (((size_t)f * P + 0) * args.nant + a) * 2 * args.row_stride + args.offset + t0 + tc;
                        const uint8_t* q1 = args.fpact + (((size_t)f * P + 1) * args.nant + a) * 2 * args.row_stride + args.offset + t0 + tc;
                        const uint4 R0 = *reinterpret_cast<const uint4*>(q0);
                        const uint4 I0 = *reinterpret_cast<const uint4*>(q0 + args.row_stride);
                        const uint4 R1 = *reinterpret_cast<const uint4*>(q1);
                        const uint4 I1 = *reinterpret_cast<const uint4*>(q1 + args.row_stride);
                        const float w = sw[s][a];
#pragma unroll
                        for(int k = 0; k < 16; ++k)
                            x[k][a] = fmul(stokes_f(stokes, (float)sbyte(R0, k), (float)sbyte(I0, k),
                                                    (float)sbyte(R1, k), (float)sbyte(I1, k)),
                                           w);
                    }
                    for(int k = 0; k < 16; ++k)
                        for(int a = 0; a < args.nant; ++a) power = fadd(power, x[k][a]);
                }
            } else {
                // reference order: t outer, a inner, float multiply and add
                power = 0.0f;
                for(int t = t0; t < t0 + args.tscrunch; ++t)
                    for(int a = 0; a < args.nant; ++a) {
                        const uint8_t* q0 = args.fpact + (((size_t)f * P + 0) * args.nant + a) * 2 * args.row_stride + args.offset + t;
                        const uint8_t* q1 = args.fpact + (((size_t)f * P + 1) * args.nant + a) * 2 * args.row_stride + args.offset + t;
                        const float st = stokes_f(stokes, (float)(int8_t)q0[0],
                                                  (float)(int8_t)q0[args.row_stride],
                                                  (float)(int8_t)q1[0],
                                                  (float)(int8_t)q1[args.row_stride]);
                        power = fadd(power, fmul(st, sw[s][a]));
                    }
            }
            args.raw[o * NC + c] = power;
            const float sc = stokes == 0
                                 ? rintf(fdiv(fsub(power, args.offset_v[so]), args.scale[so]))
                                 : rintf(fdiv(power, args.scale[so]));
            args.out[o * NC + c] = clamp_i8(sc);
        }
    }
}

// tscrunch 4, 8, 16 and 32 on rows aligned to 16 bytes: every thread takes one
// 16-byte run of samples (two for 32) of a channel, that is 16 / TS outputs,
// for a quarter of the antennas; the four warps of a CTA share 32 runs and add
// their exact integer sums in shared memory.
//
// ib_k gives a thread all antennas of one output: 4-byte loads below tscrunch
// 16, sums of all four Stokes parameters for 8 beamsets in 64 bits whatever is
// asked for, and too few threads on short gulps.  Here the Stokes parameter
// and the number of beamsets are compile-time choices and sums stay in 32
// bits: the bound sum(max |w| I) that decides whether they are exact saturates
// at 2^29, and a sum can only wrap where that bound is far above 2^24.  Bound
// by HBM (one read of the voltages).  64 antennas: 8 beamsets on 64 channels x
// 32768 samples at tscrunch 8 214 -> 115 us (537 MB, 4.7 TB/s), one beamset on
// 256 channels x 16384 samples 386 -> 163 us (6.6 TB/s); 8 channels x 4096
// samples of 16 antennas at tscrunch 4 18 -> 5.6 us.
constexpr int kIbWarps = 4;

// Four samples of one antenna as words (p0.re, p0.im, p1.re, p1.im) from the
// words of its four rows (a byte transpose).
__device__ __forceinline__ void sample_words(const uint32_t* v, uint32_t* s)
{
    const uint32_t t0 = __byte_perm(v[0], v[1], 0x5140), t1 = __byte_perm(v[2], v[3], 0x5140);
    const uint32_t t2 = __byte_perm(v[0], v[1], 0x7362), t3 = __byte_perm(v[2], v[3], 0x7362);
    s[0] = __byte_perm(t0, t1, 0x5410);
    s[1] = __byte_perm(t0, t1, 0x7632);
    s[2] = __byte_perm(t2, t3, 0x5410);
    s[3] = __byte_perm(t2, t3, 0x7632);
}

// The Stokes parameter of one sample word: every term of the reference's float
// formula is a whole number of at most 2^17, exact in float, so the sum is the
// integer one.
template <int STOKES>
__device__ __forceinline__ int stokes_word(uint32_t s)
{
    const int lo = (int)(s & 0xffffu), hi = (int)(s >> 16);  // pol 0 / pol 1: (re, im, 0, 0)
    if constexpr(STOKES == 0) return __dp4a((int)s, (int)s, 0);
    else if constexpr(STOKES == 1) return 2 * __dp4a(lo, lo, 0) - __dp4a((int)s, (int)s, 0);
    else if constexpr(STOKES == 2) return 2 * __dp4a(lo, hi, 0);
    else {
        const int x = (int)__byte_perm((uint32_t)hi, 0, 0x4401);  // (im1, re1, 0, 0)
        return 2 * (__dp4a(lo & 0xff00, x, 0) - __dp4a(lo & 0xff, x, 0));
    }
}

// L samples of a row, in one load, as words v[.][r].
template <int L>
__device__ __forceinline__ void load_run(const uint8_t* p, uint32_t (*v)[4], int r)
{
    if constexpr(L == 16) {
        const uint4 x = *reinterpret_cast<const uint4*>(p);
        v[0][r] = x.x; v[1][r] = x.y; v[2][r] = x.z; v[3][r] = x.w;
    } else if constexpr(L == 8) {
        const uint2 x = *reinterpret_cast<const uint2*>(p);
        v[0][r] = x.x; v[1][r] = x.y;
    } else {
        v[0][r] = *reinterpret_cast<const uint32_t*>(p);
    }
}

// The four rows of antenna a from sample t on.
template <int L>
__device__ __forceinline__ void load_rows(const uint8_t* p0, const uint8_t* p1, size_t rs, int a,
                                          int t, uint32_t (*v)[4])
{
    load_run<L>(p0 + 2 * a * rs + t, v, 0);
    load_run<L>(p0 + (2 * a + 1) * rs + t, v, 1);
    load_run<L>(p1 + 2 * a * rs + t, v, 2);
    load_run<L>(p1 + (2 * a + 1) * rs + t, v, 3);
}

// The chain of one output over TS samples, L at a time: the products of L
// samples and all antennas go to a table of rows of LDA, which is then walked
// in order.
template <int TS, int L, int LDA, int STOKES>
__device__ __forceinline__ float chain_walk(const uint8_t* p0, const uint8_t* p1, size_t rs,
                                            int nant, const float* w, float* x)
{
    float power = 0.0f;
    for(int tc = 0; tc < TS; tc += L) {
#pragma unroll 2
        for(int a = 0; a < nant; ++a) {
            uint32_t v[L / 4][4];
            load_rows<L>(p0, p1, rs, a, tc, v);
#pragma unroll
            for(int k = 0; k < L / 4; ++k) {
                uint32_t s[4];
                sample_words(v[k], s);
#pragma unroll
                for(int i = 0; i < 4; ++i)
                    x[(4 * k + i) * LDA + a] = fmul((float)stokes_word<STOKES>(s[i]), w[a]);
            }
        }
        for(int k = 0; k < L; ++k) {  // 16 entries in flight
            const float* y = x + k * LDA;
            int a = 0;
            for(; a + 16 <= nant; a += 16) {
                float v[16];
#pragma unroll
                for(int i = 0; i < 16; ++i) v[i] = y[a + i];
#pragma unroll
                for(int i = 0; i < 16; ++i) power = fadd(power, v[i]);
            }
            for(; a < nant; ++a) power = fadd(power, y[a]);
        }
    }
    return power;
}

template <int TS, int L, int LDA>
__device__ __forceinline__ float chain_stokes(int stokes, const uint8_t* p0, const uint8_t* p1,
                                              size_t rs, int nant, const float* w, float* x)
{
    switch(stokes) {
    case 0: return chain_walk<TS, L, LDA, 0>(p0, p1, rs, nant, w, x);
    case 1: return chain_walk<TS, L, LDA, 1>(p0, p1, rs, nant, w, x);
    case 2: return chain_walk<TS, L, LDA, 2>(p0, p1, rs, nant, w, x);
    default: return chain_walk<TS, L, LDA, 3>(p0, p1, rs, nant, w, x);
    }
}

// The reference's float chain (t outer, a inner, float multiply and add) of
// one output, from a table of its products in local memory (see ib_k): 16
// samples of up to kTableAnt antennas, 4 samples of more.  Where several
// beamsets share the bound (`recheck`), first decides in 64 bits whether this
// beamset's own sum is exact after all (`sum` holds it).
// Whole products on sample words and a compile-time Stokes parameter take the
// place of four conversions and up to seven float operations a product, one
// load a row the place of four, and 16 table entries are in flight: 64 antennas
// x 16 channels x 8192 samples at tscrunch 16 with fractional weights 52 -> 41 us
// for I, 83 -> 42 us for Q and, with the components on four warps, 323 -> 92 us
// for IQUV; two beamsets of I over 100 antennas, which were walked sample by
// sample, 400 -> 149 us.  On 64 channels x 65536 samples, where the tables live
// in L2, 853 -> 822 us for I and 2.87 -> 2.07 ms for IQUV.
template <int TS>
__device__ __noinline__ float ib_chain(const IbArgs& args, int f, int t0, const float* w,
                                       bool recheck, int stokes, int sum)
{
    constexpr int L = TS < 16 ? TS : 16;
    const size_t rs = args.row_stride;
    const uint8_t* p0 = args.fpact + ((size_t)f * 2 * args.nant) * 2 * rs + args.offset + t0;
    const uint8_t* p1 = p0 + (size_t)args.nant * 2 * rs;
    if(recheck) {
        long long bound = 0;
        for(int a = 0; a < args.nant; ++a) {
            int e = 0;
            for(int k = 0; k < TS; k += L) {
                uint32_t v[L / 4][4];
                load_rows<L>(p0, p1, rs, a, k, v);
#pragma unroll
                for(int i = 0; i < L; ++i) {
                    const int x = (int)v[i / 4][i & 3];
                    e = __dp4a(x, x, e);
                }
            }
            bound += (long long)fabsf(w[a]) * e;
        }
        if(bound <= (1ll << 24)) return (float)sum;
    }
    static_assert(4 * kMaxAnt == 16 * kTableAnt, "one table serves both forms");
    float x[16 * kTableAnt];
    if(args.nant <= kTableAnt)
        return chain_stokes<TS, L, kTableAnt>(stokes, p0, p1, rs, args.nant, w, x);
    return chain_stokes<TS, 4, kMaxAnt>(stokes, p0, p1, rs, args.nant, w, x);
}

// NC components (4: I, Q, U, V), NBS beamsets per pass; I_ONLY: NC = 1 and
// Stokes I.  Up to tscrunch 16 the bounds name one CTA per SM: without that
// the compiler holds a kernel that calls the chain to few registers, and its
// row loads to fewer in flight (64 channels x 65536 samples, Stokes I: one
// beamset at tscrunch 16 159 -> 149 us, eight at 8 206 -> 182 us); at 32 its own
// choice is 5-10 % ahead on half that many channels.
template <int TS, int NC, int NBS, bool I_ONLY>
__global__ void __launch_bounds__(32 * kIbWarps, TS < 32 ? 1 : 0)
ib_run_k(const __grid_constant__ IbArgs args, int bs0)
{
    constexpr int NO = TS < 16 ? 16 / TS : 1;   // outputs per thread
    constexpr int RUN = TS < 16 ? 16 : TS;      // samples per thread
    constexpr int NV = NO * (NBS * NC + 1);     // sums per thread, the bounds last
    __shared__ float sw[NBS][kMaxAnt];
    __shared__ int s_max[kMaxAnt];              // max |w| over the beamsets of whole weights
    __shared__ int s_int[NBS];                  // whole weights of at most 1024
    __shared__ uint32_t red[kIbWarps][NV][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nbs = min(NBS, args.nbeamsets - bs0);
    if(threadIdx.x < NBS) s_int[threadIdx.x] = 1;
    __syncthreads();
    for(int a = threadIdx.x; a < args.nant; a += blockDim.x) {
        int m = 0;
#pragma unroll
        for(int s = 0; s < NBS; ++s) {
            const float w = s < nbs ? args.weights[(size_t)(bs0 + s) * args.nant + a] : 0.0f;
            sw[s][a] = w;
            const bool ok = (w == rintf(w)) && fabsf(w) <= 1024.0f;
            if(!ok) s_int[s] = 0;
            else m = max(m, abs((int)w));
        }
        s_max[a] = m;
    }
    __syncthreads();

    const int f  = args.chan_order ? args.chan_order[blockIdx.y] : (int)blockIdx.y;
    const int t0 = (blockIdx.x * 32 + lane) * RUN;
    uint32_t S[NO][NBS * NC], B[NO];
#pragma unroll
    for(int o = 0; o < NO; ++o) {
        B[o] = 0;
#pragma unroll
        for(int i = 0; i < NBS * NC; ++i) S[o][i] = 0;
    }
    if(t0 < args.nsamples) {
        const size_t rs = args.row_stride;
        const uint8_t* p0 = args.fpact + ((size_t)f * 2 * args.nant) * 2 * rs + args.offset + t0;
        const uint8_t* p1 = p0 + (size_t)args.nant * 2 * rs;
#pragma unroll 4
        for(int a = warp; a < args.nant; a += kIbWarps) {
            uint32_t pI[NO], p[NO][NC];
#pragma unroll
            for(int o = 0; o < NO; ++o) {
                pI[o] = 0;
#pragma unroll
                for(int c = 0; c < NC; ++c) p[o][c] = 0;
            }
#pragma unroll
            for(int k = 0; k < RUN; k += 16) {
                const uint4 R0 = *reinterpret_cast<const uint4*>(p0 + 2 * a * rs + k);
                const uint4 I0 = *reinterpret_cast<const uint4*>(p0 + (2 * a + 1) * rs + k);
                const uint4 R1 = *reinterpret_cast<const uint4*>(p1 + 2 * a * rs + k);
                const uint4 I1 = *reinterpret_cast<const uint4*>(p1 + (2 * a + 1) * rs + k);
                const int r0[4] = {(int)R0.x, (int)R0.y, (int)R0.z, (int)R0.w};
                const int i0[4] = {(int)I0.x, (int)I0.y, (int)I0.z, (int)I0.w};
                const int r1[4] = {(int)R1.x, (int)R1.y, (int)R1.z, (int)R1.w};
                const int i1[4] = {(int)I1.x, (int)I1.y, (int)I1.z, (int)I1.w};
#pragma unroll
                for(int q = 0; q < 4; ++q) {
                    const int o = NO == 1 ? 0 : q * 4 / TS;
                    if constexpr(I_ONLY) {
                        pI[o] = __dp4a(r0[q], r0[q], __dp4a(i0[q], i0[q], __dp4a(r1[q], r1[q],
                                       __dp4a(i1[q], i1[q], (int)pI[o]))));
                    } else {
                        const int e0 = __dp4a(r0[q], r0[q], __dp4a(i0[q], i0[q], 0));
                        const int e1 = __dp4a(r1[q], r1[q], __dp4a(i1[q], i1[q], 0));
                        const int u = 2 * __dp4a(r0[q], r1[q], __dp4a(i0[q], i1[q], 0));
                        const int v = 2 * (__dp4a(i0[q], r1[q], 0) - __dp4a(r0[q], i1[q], 0));
                        pI[o] += e0 + e1;
                        if constexpr(NC == 4) {
                            p[o][0] += e0 + e1;
                            p[o][1] += e0 - e1;
                            p[o][2] += u;
                            p[o][3] += v;
                        } else {
                            p[o][0] += args.stokes == 0 ? e0 + e1 : args.stokes == 1 ? e0 - e1
                                     : args.stokes == 2 ? u : v;
                        }
                    }
                }
            }
            const uint32_t m = s_max[a];
#pragma unroll
            for(int o = 0; o < NO; ++o) {
                // |w| I <= 2^10 2^21 per antenna, four warps: no wrap
                B[o] = min(B[o] + m * pI[o], 1u << 29);
#pragma unroll
                for(int s = 0; s < NBS; ++s) {
                    const uint32_t wi = (uint32_t)(int)sw[s][a];
#pragma unroll
                    for(int c = 0; c < NC; ++c)
                        S[o][s * NC + c] += wi * (I_ONLY ? pI[o] : p[o][c]);
                }
            }
        }
    }
#pragma unroll
    for(int o = 0; o < NO; ++o) {
#pragma unroll
        for(int i = 0; i < NBS * NC; ++i) red[warp][o * NBS * NC + i][lane] = S[o][i];
        red[warp][NO * NBS * NC + o][lane] = B[o];
    }
    __syncthreads();
    // A warp per (32 consecutive outputs, component, beamset), as each may have
    // to walk the chain: neighbouring lanes then read neighbouring samples.
    const int nout = args.nsamples / TS;
    for(int i = warp; i < NO * NC * nbs; i += kIbWarps) {
        const int q = i % NO * 32 + lane, c = i / NO % NC, s = i / (NO * NC), bs = bs0 + s;
        const int o = q % NO, run = q / NO;
        const int tp = blockIdx.x * 32 * NO + q;
        if(tp >= nout) continue;
        uint32_t bound = 0;
        for(int k = 0; k < kIbWarps; ++k) bound += red[k][NO * NBS * NC + o][run];
        const size_t at = ((size_t)bs * nout + tp) * args.nchans + f;
        const size_t so = (size_t)bs * args.nchans + f;
        const int stokes = NC == 4 ? c : args.stokes;
        uint32_t sum = 0;
        for(int k = 0; k < kIbWarps; ++k) sum += red[k][(o * NBS + s) * NC + c][run];
        const float power = s_int[s] && bound <= (1u << 24)
                                ? (float)(int)sum  // the float chain is exact
                                : ib_chain<TS>(args, f, tp * TS, sw[s], s_int[s] && nbs > 1,
                                               stokes, (int)sum);
        args.raw[at * NC + c] = power;
        const float sc = stokes == 0
                             ? rintf(fdiv(fsub(power, args.offset_v[so]), args.scale[so]))
                             : rintf(fdiv(power, args.scale[so]));
        args.out[at * NC + c] = clamp_i8(sc);
    }
}

template <int TS, int NC, int NBS, bool I_ONLY>
int launch_runs(const IbArgs& args, cudaStream_t stream)
{
    const dim3 grid(cdiv(args.nsamples / (TS < 16 ? 16 : TS), 32), args.nchans);
    for(int bs0 = 0; bs0 < args.nbeamsets; bs0 += NBS) {
        ib_run_k<TS, NC, NBS, I_ONLY><<<grid, 32 * kIbWarps, 0, stream>>>(args, bs0);
        SW_LAUNCH_CHECK();
    }
    return SW_OK;
}

template <int TS>
int launch_ts(const IbArgs& args, cudaStream_t stream)
{
    if(args.stokes == 4)
        return args.nbeamsets == 1 ? launch_runs<TS, 4, 1, false>(args, stream)
                                   : launch_runs<TS, 4, 2, false>(args, stream);
    if(args.stokes == 0)
        return args.nbeamsets == 1 ? launch_runs<TS, 1, 1, true>(args, stream)
                                   : launch_runs<TS, 1, 8, true>(args, stream);
    return args.nbeamsets == 1 ? launch_runs<TS, 1, 1, false>(args, stream)
                               : launch_runs<TS, 1, 8, false>(args, stream);
}

}  // namespace

int launch_incoherent_beamform(const void* d_fpact, size_t row_stride,
                               size_t sample_offset, int nchans, int nsamples,
                               int nant, int tscrunch, const float* d_scale,
                               const float* d_offset,
                               const float* d_beamset_weights, int nbeamsets,
                               int stokes, float* d_raw, int8_t* d_out,
                               cudaStream_t stream, const int* d_chan_order)
{
    SW_REQUIRE(d_fpact && d_scale && d_offset && d_beamset_weights && d_raw && d_out,
               "sw_incoherent_beamform: null pointer");
    SW_REQUIRE(nbeamsets > 0, "Number of beamsets must be greater than zero");
    SW_REQUIRE(nant > 0 && nant <= kMaxAnt, "sw_incoherent_beamform: bad antenna count");
    SW_REQUIRE(tscrunch > 0 && nsamples % tscrunch == 0,
               "sw_incoherent_beamform: nsamples must be a multiple of tscrunch");
    SW_REQUIRE(stokes >= 0 && stokes <= 4, "sw_incoherent_beamform: bad Stokes mode");
    SW_REQUIRE(tscrunch % 4 != 0 || (row_stride % 4 == 0 && sample_offset % 4 == 0 &&
                                     (reinterpret_cast<uintptr_t>(d_fpact) & 3) == 0),
               "sw_incoherent_beamform: with tscrunch a multiple of 4 the voltage pointer, "
               "row stride and sample offset must be multiples of 4 bytes");
    SW_REQUIRE(nchans > 0 && nchans <= 65535, "sw_incoherent_beamform: bad channel count");
    IbArgs args{static_cast<const uint8_t*>(d_fpact), row_stride, sample_offset,
                nchans, nsamples, nant, tscrunch, nbeamsets, stokes, d_scale,
                d_offset, d_beamset_weights, d_raw, d_out, d_chan_order};
    // whole aligned 16-byte runs of samples per thread
    if(nsamples % 16 == 0 && row_stride % 16 == 0 && sample_offset % 16 == 0 &&
       (reinterpret_cast<uintptr_t>(d_fpact) & 15) == 0) {
        switch(tscrunch) {
        case 4: return launch_ts<4>(args, stream);
        case 8: return launch_ts<8>(args, stream);
        case 16: return launch_ts<16>(args, stream);
        case 32: return launch_ts<32>(args, stream);
        }
    }
    const int nout = nsamples / tscrunch;
    dim3 grid(cdiv(nout, 128), nchans);
    if(stokes == 4) {
        for(int bs0 = 0; bs0 < nbeamsets; bs0 += kMaxBs / 4) {
            ib_k<4><<<grid, 128, 0, stream>>>(args, bs0);
            SW_LAUNCH_CHECK();
        }
    } else {
        for(int bs0 = 0; bs0 < nbeamsets; bs0 += kMaxBs) {
            ib_k<1><<<grid, 128, 0, stream>>>(args, bs0);
            SW_LAUNCH_CHECK();
        }
    }
    return SW_OK;
}

namespace {

// Channels in descending order of voltage power (sum over pols and antennas
// of mean^2 + std^2, from the statistics stage).  The incoherent beam maps
// its CTA rows through this order, so the channels most likely to need the
// float chain (RFI-saturated ones, whose CTAs take longest) start first and
// overlap the others instead of trailing behind them.  Ties go by channel
// index and a NaN power counts as lowest, so the order is a permutation.
__global__ void ib_channel_order_k(const float4* __restrict__ stats, int nchans, int npa,
                                   int* __restrict__ order)
{
    extern __shared__ float pw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    for(int c = warp; c < nchans; c += nwarps) {  // one warp per channel
        float s = 0.0f;
        for(int i = lane; i < npa; i += 32) {
            const float4 v = stats[(size_t)c * npa + i];
            s += v.x * v.x + v.y * v.y;
        }
#pragma unroll
        for(int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if(lane == 0) pw[c] = isnan(s) ? -1.0f : s;
    }
    __syncthreads();
    for(int c = threadIdx.x; c < nchans; c += blockDim.x) {
        int r = 0;
        for(int k = 0; k < nchans; ++k) r += (pw[k] > pw[c]) || (pw[k] == pw[c] && k < c);
        order[r] = c;
    }
}

}  // namespace

int launch_ib_channel_order(const float* d_stats, int nchans, int npol, int nant,
                            int* d_order, cudaStream_t stream)
{
    SW_REQUIRE(d_stats && d_order, "ib channel order: null pointer");
    SW_REQUIRE(nchans > 0 && nchans <= kIbOrderMaxChans, "ib channel order: bad channel count");
    // one CTA: the ranks need every channel's power (8 warps took 28 us for 256
    // channels of 64 antennas, 32 warps 11 us)
    ib_channel_order_k<<<1, 1024, nchans * sizeof(float), stream>>>(
        reinterpret_cast<const float4*>(d_stats), nchans, npol * nant, d_order);
    SW_LAUNCH_CHECK();
    return SW_OK;
}

}  // namespace swb

extern "C" int sw_incoherent_beamform(const void* d_fpact, size_t row_stride,
                                      size_t sample_offset, int nchans,
                                      int nsamples, int nant, int tscrunch,
                                      const float* d_scale, const float* d_offset,
                                      const float* d_beamset_weights,
                                      int nbeamsets, int stokes, float* d_raw,
                                      int8_t* d_out, sw_stream_t stream)
{
    return swb::launch_incoherent_beamform(
        d_fpact, row_stride, sample_offset, nchans, nsamples, nant, tscrunch,
        d_scale, d_offset, d_beamset_weights, nbeamsets, stokes, d_raw, d_out,
        swb::as_cuda(stream), nullptr);
}
