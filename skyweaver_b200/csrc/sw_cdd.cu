// CoherentDedisperser on the B200.
//
// Reference: cpp/skyweaver/src/CoherentDedisperser.cu:142-225 (per channel:
// int8 -> complex64, cuFFT forward, chirp multiply, cuFFT inverse, trim
// overlap/2 each side, /N, round, int8 wrap) with the chirp of
// DMResponse (:293-336) and the golden-vector generator
// python/skyweaver_test_utils/dedisperse.py:58-80,143-173.
//
// B200 design: one overlap-save window of one (channel, pol, antenna) stream is
// transformed entirely on chip, for 1024 to 8192 points by a group of N / 32
// threads in packed pairs (sw_cdd_pk.cuh, cdd_pk_kernel), for 256 and 512 points
// by a CTA of N / 16 threads (cdd_kernel); longer windows are split into
// 8192-point sub-transforms (cdd_split_kernel):
//   * the forward FFT is in place, decimation in frequency, its first pass read
//     straight from the staged planar int8 rows, its last pass leaving each
//     thread's spectral bins in digit-reversed order, in registers (256 and 512
//     points) or in tensor memory (longer windows);
//   * for every coherent DM the thread multiplies its bins by the chirp (FP64
//     phases, stored as complex float in the order the threads load it), runs
//     the exact inverse passes (decimation in time, conjugate twiddles), and
//     the last pass writes the trimmed, scaled, rounded and int8-wrapped
//     samples straight to the planar output rows.
// So the forward transform is done once per window for all DMs, there is no
// spectrum in HBM (up to 8192 points), and all global traffic is coalesced.
//
// Trim.  The reference trims overlap/2 samples at each end of a window.  Its
// chirp's impulse response is one-sided (nearly all of it at lags 0 .. the
// intra-channel smear), so a window here trims `overlap - lag` samples at its
// start (the causal part) and `lag` at its end (the short anti-causal part);
// output sample m is the dedispersed voltage at gulp position m - lag.
// lag = overlap / 2 is the reference's own per-window trim.
// Twiddles come from FP64-computed tables; FFT arithmetic is FP32.
#include <algorithm>

#include "sw_cdd_pk.cuh"
#include "sw_common.cuh"

namespace swb {
namespace cdd {

constexpr int kMaxDms = 64;

// ---------------------------------------------------------------- plan
struct Plan {
    int logn, n, r0, npass;
    int radix[8];
    int span[8];    // G_p
    int stride[8];  // s_p = G_p / R_p
    int tw_off[8];  // offset (complex entries) of pass p's table
    int tw_total;
};

__host__ __device__ constexpr Plan make_plan(int logn)
{
    Plan P{};
    P.logn = logn;
    P.n    = 1 << logn;
    const int rem = logn % 4;
    P.r0 = rem ? (1 << rem) : 16;
    int g = P.n, off = 0, p = 0;
    int r = P.r0;
    while(g > 1) {
        P.radix[p]  = r;
        P.span[p]   = g;
        P.stride[p] = g / r;
        P.tw_off[p] = off;
        // radix-16 tables hold twiddle pairs (w1,w2),(w3,w4),..,(w15,0) per j,
        // read with one 16-byte load per pair; other radices hold w1..w(R-1)
        if(P.stride[p] > 1) off += (r == 16 ? 16 : r - 1) * P.stride[p];
        g /= r;
        r = 16;
        ++p;
    }
    P.npass    = p;
    P.tw_total = off;
    return P;
}

// DIF output position -> natural frequency bin
__host__ __device__ inline int digit_reverse(const Plan& P, int pos)
{
    int k = 0, mult = 1;
    for(int p = 0; p < P.npass; ++p) {
        const int q = (pos / P.stride[p]) % P.radix[p];
        k += q * mult;
        mult *= P.radix[p];
    }
    return k;
}

// ------------------------------------------------------- complex helpers
struct c32 {
    float x, y;
};
__device__ __forceinline__ c32 cadd(c32 a, c32 b) { return {a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ c32 csub(c32 a, c32 b) { return {a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ c32 cmul(c32 a, c32 b)
{
    return {a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x};
}
__device__ __forceinline__ c32 cmulc(c32 a, c32 b)  // a * conj(b)
{
    return {a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y};
}
// multiply by -i (forward) or +i (inverse)
template <bool INV>
__device__ __forceinline__ c32 rot90(c32 a)
{
    return INV ? c32{-a.y, a.x} : c32{a.y, -a.x};
}

template <bool INV>
__device__ __forceinline__ void dft2(c32* x)
{
    c32 a = x[0], b = x[1];
    x[0] = cadd(a, b);
    x[1] = csub(a, b);
}

template <bool INV>
__device__ __forceinline__ void dft4(c32& x0, c32& x1, c32& x2, c32& x3)
{
    const c32 t0 = cadd(x0, x2), t1 = csub(x0, x2);
    const c32 t2 = cadd(x1, x3), t3 = rot90<INV>(csub(x1, x3));
    x0 = cadd(t0, t2);
    x2 = csub(t0, t2);
    x1 = cadd(t1, t3);
    x3 = csub(t1, t3);
}

// W_16^k for k = 0..9 (forward sign); constants rounded once by the compiler
__device__ __forceinline__ c32 w16(int k)
{
    const float c1 = 0.92387953251128675613f, s1 = 0.38268343236508977173f;
    const float c2 = 0.70710678118654752440f;
    switch(k) {
    case 0: return {1.0f, 0.0f};
    case 1: return {c1, -s1};
    case 2: return {c2, -c2};
    case 3: return {s1, -c1};
    case 4: return {0.0f, -1.0f};
    case 5: return {-s1, -c1};
    case 6: return {-c2, -c2};
    case 7: return {-c1, -s1};
    case 8: return {-1.0f, 0.0f};
    default: return {-c1, s1};  // k == 9
    }
}

// In-register DFT of size 16, natural order in and out.
template <bool INV>
__device__ __forceinline__ void dft16(c32* x)
{
#pragma unroll
    for(int r2 = 0; r2 < 4; ++r2) dft4<INV>(x[r2], x[4 + r2], x[8 + r2], x[12 + r2]);
    // now x[4*q1 + r2] holds A[r2][q1]; twiddle by W16^(r2*q1)
#pragma unroll
    for(int r2 = 1; r2 < 4; ++r2)
#pragma unroll
        for(int q1 = 1; q1 < 4; ++q1) {
            c32 w = w16(r2 * q1);
            if(INV) w.y = -w.y;
            x[4 * q1 + r2] = cmul(x[4 * q1 + r2], w);
        }
#pragma unroll
    for(int q1 = 0; q1 < 4; ++q1) dft4<INV>(x[4 * q1], x[4 * q1 + 1], x[4 * q1 + 2], x[4 * q1 + 3]);
    // x[4*q1 + q2] holds X[q1 + 4*q2]; transpose to natural order
    c32 t[16];
#pragma unroll
    for(int q1 = 0; q1 < 4; ++q1)
#pragma unroll
        for(int q2 = 0; q2 < 4; ++q2) t[q1 + 4 * q2] = x[4 * q1 + q2];
#pragma unroll
    for(int i = 0; i < 16; ++i) x[i] = t[i];
}

template <int R, bool INV>
__device__ __forceinline__ void dft(c32* x)
{
    static_assert(R == 16 || R == 2, "256 = 16 x 16, 512 = 2 x 16 x 16");
    if constexpr(R == 16) dft16<INV>(x);
    else dft2<INV>(x);
}

// one padding slot per 16 complex values keeps the strided radix-16 passes
// free of shared-memory bank conflicts
__host__ __device__ constexpr int pad(int i) { return i + (i >> 4); }
// pad(b + q * s) for a stride s that is a multiple of 16: the padding of
// b + q s is pad(b) + q (s + s / 16), i.e. one base plus constant offsets
// (the compiler folds them into the shared-memory instructions).
__device__ __forceinline__ int pad_at(int b, int pb, int q, int s)
{
    return (s & 15) == 0 ? pb + q * (s + (s >> 4)) : pad(b + q * s);
}

struct Args {
    const uint8_t* in;
    size_t row_stride;
    int nstreams;      // F * P * A
    int nsamples;      // T
    int overlap;       // O: samples of history in front of the gulp
    int lag;           // trimmed at the end of each window (output delay)
    int nseg;
    int ndms;
    int ndmg, dm_group;  // cdd_pk_kernel: DM groups of a window, DMs of a group
    const c32* tw;     // twiddle tables
    const c32* chirp;  // [ndms][F][N] in per-thread load order (chirp_k)
    size_t chirp_dm_stride;    // complex entries between two DMs' tables
    const uint32_t* zero_flags;  // [ndms]: non-zero if the DM is 0 (chirp exactly 1)
    int npa;           // P * A (streams per channel)
    uint8_t* out[kMaxDms];
    size_t out_stride;
    float2* dbg;  // optional [ndms][nstreams][nsamples] scaled values before rounding
};

// Twiddles w[1..R-1] of butterfly column j for a pass with stride s.
template <int R>
__device__ __forceinline__ void load_tw(const c32* tw_s, int tw_off, int s, int j, c32* w)
{
    if constexpr(R == 16) {
        const float4* p = reinterpret_cast<const float4*>(tw_s + tw_off);
#pragma unroll
        for(int k = 0; k < 8; ++k) {
            const float4 v = p[k * s + j];
            w[2 * k + 1] = c32{v.x, v.y};
            if(k < 7) w[2 * k + 2] = c32{v.z, v.w};
        }
    } else {
#pragma unroll
        for(int q = 1; q < R; ++q) w[q] = tw_s[tw_off + (q - 1) * s + j];
    }
}

// One radix-R pass of the inverse (DIT) on shared memory.
template <int LOGN, int R>
__device__ __forceinline__ void inv_pass(c32* buf, const c32* tw_s, int G, int s,
                                         int tw_off)
{
    constexpr int N   = 1 << LOGN;
    constexpr int NT  = N / 16;
    constexpr int BPT = 16 / R;  // butterflies per thread
#pragma unroll
    for(int u = 0; u < BPT; ++u) {
        const int beta = threadIdx.x + u * NT;
        const int g = beta / s, j = beta - g * s;
        const int base = g * G + j;
        const int pb = pad(base);
        c32 z[R];
#pragma unroll
        for(int q = 0; q < R; ++q) z[q] = buf[pad_at(base, pb, q, s)];
        if(s > 1) {
{
                c32 w[R];
                load_tw<R>(tw_s, tw_off, s, j, w);
#pragma unroll
                for(int q = 1; q < R; ++q) z[q] = cmulc(z[q], w[q]);
            }
        }
        dft<R, true>(z);
#pragma unroll
        for(int r = 0; r < R; ++r) buf[pad_at(base, pb, r, s)] = z[r];
    }
}

template <int LOGN, int R>
__device__ __forceinline__ void fwd_pass(c32* buf, const c32* tw_s, int G, int s,
                                         int tw_off)
{
    constexpr int N   = 1 << LOGN;
    constexpr int NT  = N / 16;
    constexpr int BPT = 16 / R;
#pragma unroll
    for(int u = 0; u < BPT; ++u) {
        const int beta = threadIdx.x + u * NT;
        const int g = beta / s, j = beta - g * s;
        const int base = g * G + j;
        const int pb = pad(base);
        c32 x[R];
#pragma unroll
        for(int r = 0; r < R; ++r) x[r] = buf[pad_at(base, pb, r, s)];
        dft<R, false>(x);
        if(s > 1) {
{
                c32 w[R];
                load_tw<R>(tw_s, tw_off, s, j, w);
#pragma unroll
                for(int q = 1; q < R; ++q) x[q] = cmul(x[q], w[q]);
            }
        }
#pragma unroll
        for(int q = 0; q < R; ++q) buf[pad_at(base, pb, q, s)] = x[q];
    }
}

__device__ __forceinline__ uint32_t smem_addr(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Stage the int8 window of one work item (re row then im row, N bytes each)
// into shared memory: asynchronously with 16-byte cp.async (zero-filled past
// the end of the rows) when the rows and segment starts are 16-byte aligned,
// otherwise with plain byte copies.
template <int N, int NT>
__device__ __forceinline__ void stage_input(uint8_t* st, const Args& A, int item, int L,
                                            bool aligned, int tid)
{
    const int stream = item / A.nseg;
    const int seg    = item - stream * A.nseg;
    const uint8_t* row_re = A.in + (size_t)stream * 2 * A.row_stride;
    const uint8_t* row_im = row_re + A.row_stride;
    const int start = seg * L;
    const int avail = A.overlap + A.nsamples;
    if(aligned) {
        constexpr int kChunks = N / 16;
        for(int c = tid; c < 2 * kChunks; c += NT) {
            const int plane = c >= kChunks;
            const int k     = (c - plane * kChunks) * 16;
            const int left  = avail - (start + k);
            const int bytes = left <= 0 ? 0 : (left >= 16 ? 16 : left);
            const uint8_t* src = bytes > 0 ? (plane ? row_im : row_re) + start + k : row_re;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                             smem_addr(st + plane * N + k)),
                         "l"(src), "r"(bytes)
                         : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    } else {
        for(int i = tid; i < N; i += NT) {
            const int idx = start + i;
            st[i]     = idx < avail ? row_re[idx] : 0;
            st[N + i] = idx < avail ? row_im[idx] : 0;
        }
    }
}

// The DMs of exactly 0 (bits of zero_dms): their output is the staged window
// itself, trimmed like the others.
template <int N, int NT>
__device__ __forceinline__ void copy_zero_dms(const uint8_t* stage, const Args& A,
                                              uint32_t zero_dms, int stream, int start, int L,
                                              int head, bool copy16, int tid)
{
    for(uint32_t zm = zero_dms; zm; zm &= zm - 1) {
        const int d = __ffs(zm) - 1;
        uint8_t* o_re = A.out[d] + (size_t)stream * 2 * A.out_stride;
        const int n = min(L, A.nsamples - start);  // kept samples of this window
        if(copy16 && ((reinterpret_cast<uintptr_t>(A.out[d]) & 15) == 0)) {
            const int chunks = (n + 15) / 16;
            for(int c = tid; c < 2 * chunks; c += NT) {
                const int plane = c >= chunks;
                const int k = (c - plane * chunks) * 16;
                const uint8_t* src = stage + plane * N + head + k;
                uint8_t* dst = o_re + plane * A.out_stride + start + k;
                if(k + 16 <= n) {
                    *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(src);
                } else {
                    for(int b = 0; b < n - k; ++b) dst[b] = src[b];
                }
            }
        } else {
            for(int i = tid; i < 2 * n; i += NT) {
                const int plane = i >= n, k = i - plane * n;
                o_re[plane * A.out_stride + start + k] = stage[plane * N + head + k];
            }
        }
    }
}

// Windows of 256 and 512 points, one per CTA of 16 points a thread; several
// CTAs per SM hide the latency across the per-pass barriers.
template <int LOGN, bool DBG>
__global__ void __launch_bounds__((1 << LOGN) / 16, 4)
cdd_kernel(const __grid_constant__ Args A)
{
    constexpr int N  = 1 << LOGN;
    constexpr int NT = N / 16;
    constexpr Plan P = make_plan(LOGN);
    constexpr int R0 = P.r0;
    constexpr int B0 = 16 / R0;  // first-pass butterflies per thread
    extern __shared__ __align__(16) uint8_t smem[];
    c32* buf  = reinterpret_cast<c32*>(smem);
    c32* tw_s = buf + pad(N) + 16;
    uint8_t* stage = reinterpret_cast<uint8_t*>(tw_s + ((P.tw_total + 1) & ~1));
    for(int i = threadIdx.x; i < P.tw_total; i += NT) tw_s[i] = A.tw[i];

    const int L = N - A.overlap;
    const int head = A.overlap - A.lag;  // trimmed at the start of each window
    const float inv_n = 1.0f / (float)N;  // exact (power of two)
    const int nitems = A.nstreams * A.nseg;
    const bool aligned = (A.row_stride % 16 == 0) && (L % 16 == 0) &&
                         ((reinterpret_cast<uintptr_t>(A.in) & 15) == 0);
    // DMs of exactly 0 (chirp 1): the dedispersed window is the input itself
    // (the FP32 round trip of int8 samples rounds back to them exactly), so
    // they are copied from the staged window instead of transformed.  The
    // debug instance transforms them to report the float round trip.
    uint32_t zero_dms = 0;
    if constexpr(!DBG)
        for(int d = 0; d < A.ndms && d < 32; ++d) zero_dms |= (A.zero_flags[d] ? 1u : 0u) << d;
    const bool copy16 = aligned && (head % 16) == 0 && (A.out_stride % 16) == 0;
    if(blockIdx.x < nitems) stage_input<N, NT>(stage, A, blockIdx.x, L, aligned, threadIdx.x);
    for(int item = blockIdx.x; item < nitems; item += gridDim.x) {
        const int stream = item / A.nseg;
        const int seg    = item - stream * A.nseg;
        const int f      = stream / A.npa;
        const int start  = seg * L;  // first input sample of the window
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();

        // ---- forward pass 0 (radix R0, span N) from the staged int8 window
        {
            constexpr int s0 = N / R0;
#pragma unroll
            for(int u = 0; u < B0; ++u) {
                const int j = threadIdx.x + u * NT;
                c32 x[R0];
#pragma unroll
                for(int r = 0; r < R0; ++r) {
                    const int i = j + r * s0;
                    x[r] = c32{(float)(int8_t)stage[i], (float)(int8_t)stage[N + i]};
                }
                dft<R0, false>(x);
{
                    c32 w[R0];
                    load_tw<R0>(tw_s, P.tw_off[0], s0, j, w);
#pragma unroll
                    for(int q = 1; q < R0; ++q) x[q] = cmul(x[q], w[q]);
                }
#pragma unroll
                for(int q = 0; q < R0; ++q) buf[pad_at(j, pad(j), q, s0)] = x[q];
            }
        }
        copy_zero_dms<N, NT>(stage, A, zero_dms, stream, start, L, head, copy16, threadIdx.x);
        __syncthreads();
        // the staging buffer is free: fetch the next work item's window now so
        // that its global-memory latency hides behind this item's transforms
        if(item + (int)gridDim.x < nitems)
            stage_input<N, NT>(stage, A, item + gridDim.x, L, aligned, threadIdx.x);
        // ---- forward radix-16 passes except the last
#pragma unroll
        for(int p = 1; p < P.npass - 1; ++p) {
            fwd_pass<LOGN, 16>(buf, tw_s, P.span[p], P.stride[p], P.tw_off[p]);
            __syncthreads();
        }
        // ---- last forward pass (span 16, no twiddles): spectrum -> registers
        c32 spec[16];
#pragma unroll
        for(int r = 0; r < 16; ++r) spec[r] = buf[pad(threadIdx.x * 16 + r)];
        dft16<false>(spec);

        const size_t chirp_stride = A.chirp_dm_stride;  // complex entries per DM
        const float4* chp = reinterpret_cast<const float4*>(A.chirp + (size_t)f * N) + threadIdx.x;
        // the transformed DMs in order; chn holds the chirp of DM `d`
        int d = 0;
        while(d < A.ndms && d < 32 && ((zero_dms >> d) & 1u)) ++d;
        float4 chn[8];
        if(d < A.ndms) {
            const float4* cur = chp + (size_t)d * chirp_stride / 2;
#pragma unroll
            for(int k = 0; k < 8; ++k) chn[k] = cur[k * NT];
        }
        __syncthreads();
        for(; d < A.ndms;) {
            int dn = d + 1;
            while(dn < A.ndms && dn < 32 && ((zero_dms >> dn) & 1u)) ++dn;
            c32 y[16];
#pragma unroll
            for(int k = 0; k < 8; ++k) {
                y[2 * k]     = cmul(spec[2 * k], c32{chn[k].x, chn[k].y});
                y[2 * k + 1] = cmul(spec[2 * k + 1], c32{chn[k].z, chn[k].w});
            }
            if(dn < A.ndms) {  // next DM's chirp, in flight during this inverse
                const float4* nxt = chp + (size_t)dn * chirp_stride / 2;
#pragma unroll
                for(int k = 0; k < 8; ++k) chn[k] = nxt[k * NT];
            }
            dft16<true>(y);
#pragma unroll
            for(int r = 0; r < 16; ++r) buf[pad(threadIdx.x * 16 + r)] = y[r];
            __syncthreads();
#pragma unroll
            for(int p = P.npass - 2; p >= 1; --p) {
                inv_pass<LOGN, 16>(buf, tw_s, P.span[p], P.stride[p], P.tw_off[p]);
                __syncthreads();
            }
            // ---- inverse pass 0 (radix R0, span N): natural-order output
            uint8_t* o_re = A.out[d] + (size_t)stream * 2 * A.out_stride;
            uint8_t* o_im = o_re + A.out_stride;
            constexpr int s0 = N / R0;
#pragma unroll
            for(int u = 0; u < B0; ++u) {
                const int j = threadIdx.x + u * NT;
                c32 z[R0];
#pragma unroll
                for(int q = 0; q < R0; ++q) z[q] = buf[pad_at(j, pad(j), q, s0)];
{
                    c32 w[R0];
                    load_tw<R0>(tw_s, P.tw_off[0], s0, j, w);
#pragma unroll
                    for(int q = 1; q < R0; ++q) z[q] = cmulc(z[q], w[q]);
                }
                dft<R0, true>(z);
#pragma unroll
                for(int r = 0; r < R0; ++r) {
                    const int i = j + r * s0;           // index within the window
                    const int m = start + i - head;     // output sample in the gulp
                    if(i >= head && i < head + L && m < A.nsamples) {
                        const float fr = z[r].x * inv_n, fi = z[r].y * inv_n;
                        o_re[m] = (uint8_t)__float2int_rn(fr);  // int8 wrap, like static_cast<char>
                        o_im[m] = (uint8_t)__float2int_rn(fi);
                        if constexpr(DBG)
                            A.dbg[((size_t)d * A.nstreams + stream) * A.nsamples + m] =
                                make_float2(fr, fi);
                    }
                }
            }
            __syncthreads();
            d = dn;
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// A chirp with a bin that is no number (a DM that is none, or a channel with a
// bin at 0 Hz) makes every sample of its windows none, and their bytes 0: one
// sample tells.
__device__ __forceinline__ bool no_number(const Pk& x)
{
    float lo, hi;
    unpk2(x.re, lo, hi);
    return isnan(lo);
}

// bits d0 .. d1 - 1 of a mask of the first 32 DMs
__device__ __forceinline__ uint32_t dm_bits(int d0, int d1)
{
    return (d1 < 32 ? (1u << d1) - 1u : ~0u) & ~(d0 < 32 ? (1u << d0) - 1u : ~0u);
}

// Windows of 1024 .. 8192 points: 16384 / N windows per CTA, each by a group of
// N / 32 threads with its own barrier and staging buffer (sw_cdd_pk.cuh).
//
// One window per CTA at 16 points a thread (scalar arithmetic, one more pass,
// twiddles in shared memory, spectrum in registers: cdd_kernel) was bound by
// shared-memory wavefronts (63 %), issue (61 %) and its CTA-wide barriers:
// 64 antennas x 64 channels x 65536 samples at DMs 50, 150 and 500 took 9.21 ms
// that way with 8192 points and take 5.48 ms here; 32 channels x 32768 samples
// with 4096 points 2.10 -> 1.33 ms; 48 antennas x 32 channels x 16384 samples,
// one DM, with 2048 points 0.285 -> 0.204 ms.  With 16 warps of 126 registers per
// SM no unit is saturated: FMA pipe and shared-memory wavefronts 54 %, issue
// 48 %.  (Barriers for the whole group after every pass: 5.81 ms.)
template <int LOGN, bool DBG, bool SPLIT>
__global__ void __launch_bounds__(kPkThreads, 1)
cdd_pk_kernel(const __grid_constant__ Args A)
{
    using G = PkGeo<LOGN>;
    constexpr int N = G::N, NT = G::T;
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ uint32_t s_tmem;
    PkGroup g;
    const uint32_t tmem =
        pk_setup<LOGN, true>(g, smem, &s_tmem, reinterpret_cast<const float*>(A.tw));
    const int t = g.t;
    uint8_t* stage = smem + kPkBufBytes + g.window * 2 * N;

    const int L = N - A.overlap;
    const int head = A.overlap - A.lag;  // trimmed at the start of each window
    const float inv_n = 1.0f / (float)N;  // exact (power of two)
    // a unit of work: a window, or (SPLIT) one group of its DMs
    const int ngroups = SPLIT ? A.ndmg : 1;
    const int nunits = A.nstreams * A.nseg * ngroups, step = G::W * gridDim.x;
    const bool aligned = (A.row_stride % 16 == 0) && (L % 16 == 0) &&
                         ((reinterpret_cast<uintptr_t>(A.in) & 15) == 0);
    // DMs of exactly 0: copied from the staged window (see cdd_kernel)
    uint32_t zero_dms = 0;
    if constexpr(!DBG)
        for(int d = 0; d < A.ndms && d < 32; ++d) zero_dms |= (A.zero_flags[d] ? 1u : 0u) << d;
    const bool copy16 = aligned && (head % 16) == 0 && (A.out_stride % 16) == 0;
    // both samples of a pair are kept or trimmed together and their bytes may
    // be stored as one 16-bit word
    const bool even = ((head | L | A.nsamples) & 1) == 0 && (A.out_stride & 1) == 0;
    // v / N rounded to the nearest even integer in the low mantissa bits (v / N
    // is below 2^14 in magnitude): the low byte is the int8-wrapped sample
    const uint64_t scale = pk2(inv_n, inv_n), magic = pk2(12582912.0f, 12582912.0f);
    int unit = g.window * gridDim.x + blockIdx.x;
    if(unit < nunits) stage_input<N, NT>(stage, A, unit / ngroups, L, aligned, t);
    for(; unit < nunits; unit += step) {
        // window `item`, DMs d0 .. d1 - 1
        const int item = unit / ngroups;
        const int d0 = SPLIT ? (unit - item * ngroups) * A.dm_group : 0;
        const int d1 = SPLIT ? min(A.ndms, d0 + A.dm_group) : A.ndms;
        const int stream = item / A.nseg;
        const int seg    = item - stream * A.nseg;
        const int f      = stream / A.npa;
        const int start  = seg * L;  // first input sample of the window
        asm volatile("cp.async.wait_all;" ::: "memory");
        pk_sync<LOGN>(g);
        copy_zero_dms<N, NT>(stage, A, SPLIT ? zero_dms & dm_bits(d0, d1) : zero_dms, stream,
                             start, L, head, copy16, t);
        __syncwarp();  // lanes leave the copy at different lengths; see pk_sync
        Pk x[16];
#pragma unroll
        for(int r = 0; r < 16; ++r) {
            const uint32_t re = *reinterpret_cast<const uint16_t*>(stage + 2 * t + (N / 16) * r);
            const uint32_t im = *reinterpret_cast<const uint16_t*>(stage + N + 2 * t + (N / 16) * r);
            x[r] = {pk2((float)(int8_t)re, (float)(int8_t)(re >> 8)),
                    pk2((float)(int8_t)im, (float)(int8_t)(im >> 8))};
        }
        // the next window's bytes are fetched behind this one's transforms
        pk_forward<LOGN>(g, x, [&] {
            if(unit + step < nunits)
                stage_input<N, NT>(stage, A, (unit + step) / ngroups, L, aligned, t);
        });
        const float4* chp = reinterpret_cast<const float4*>(A.chirp + (size_t)f * N) + t;
        // samples of this window that the output holds: window index head + u,
        // output sample start + u, u < kept
        const unsigned kept = (unsigned)max(0, min(L, A.nsamples - start));
        const size_t out_at = (size_t)stream * 2 * A.out_stride + start;
        for(int d = d0; d < d1; ++d) {
            if(d < 32 && ((zero_dms >> d) & 1u)) continue;
            pk_inverse<LOGN>(g, chp + (size_t)d * A.chirp_dm_stride / 2, x);
            uint8_t* o_re = A.out[d] + out_at;
            uint8_t* o_im = o_re + A.out_stride;
            const bool words = even && (reinterpret_cast<uintptr_t>(A.out[d]) & 1) == 0;
            const bool none = no_number(x[0]);
            if constexpr(!DBG) {
                if(none) {
#pragma unroll
                    for(int r = 0; r < 16; ++r) x[r] = {0, 0};
                }
            }
#pragma unroll
            for(int r = 0; r < 16; ++r) {
                const int u = 2 * t + (N / 16) * r - head;
                uint32_t ra, rb, ia, ib;
                unpk2u(pfma(x[r].re, scale, magic), ra, rb);
                unpk2u(pfma(x[r].im, scale, magic), ia, ib);
                if constexpr(DBG)
                    if(none) ra = rb = ia = ib = 0;
                if(words) {
                    if((unsigned)u < kept) {
                        *reinterpret_cast<uint16_t*>(o_re + u) =
                            (uint16_t)__byte_perm(ra, rb, 0x0040);
                        *reinterpret_cast<uint16_t*>(o_im + u) =
                            (uint16_t)__byte_perm(ia, ib, 0x0040);
                    }
                } else {
                    if((unsigned)u < kept) {
                        o_re[u] = (uint8_t)ra;
                        o_im[u] = (uint8_t)ia;
                    }
                    if((unsigned)(u + 1) < kept) {
                        o_re[u + 1] = (uint8_t)rb;
                        o_im[u + 1] = (uint8_t)ib;
                    }
                }
                if constexpr(DBG) {
                    float fr[2], fi[2];
                    unpk2(pmul(x[r].re, scale), fr[0], fr[1]);
                    unpk2(pmul(x[r].im, scale), fi[0], fi[1]);
                    for(int e = 0; e < 2; ++e)
                        if((unsigned)(u + e) < kept)
                            A.dbg[((size_t)d * A.nstreams + stream) * A.nsamples + start + u + e] =
                                make_float2(fr[e], fi[e]);
                }
            }
            pk_sync<LOGN>(g);  // the next store of this group waits for these loads
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    pk_tmem_free(tmem);
}

// ------------------------------------------------- long FFTs (N = S x 8192)
// Overlap-save windows longer than one CTA's shared memory are split four-step
// style into S = N / 8192 sub-transforms of M = 8192 points:
//   n = M n1 + n2, k = k1 + S k2 (n1, k1 < S; n2, k2 < M)
//   forward:  X[k1 + S k2] = DFT_M over n2 of
//                 W_N^(n2 k1) * sum_n1 x[M n1 + n2] W_S^(n1 k1)
//   inverse:  x[n2 + M n1] = sum_k1 W_S^(-n1 k1) *
//                 W_N^(-n2 k1) * IDFT_M over k2 of Y[k1 + S k2]
// cdd_split_kernel runs one (segment, k1) per group of 256 threads: the S-point
// partial DFT straight from the int8 rows into pass 0's registers, the M-point
// forward FFT, and for every DM the chirp of bins k1 + S k2 and the M-point
// inverse FFT (sw_cdd_pk.cuh), leaving W_N^(-n2 k1) * z in a workspace of pairs
// (8-byte accesses: the caller's workspace need not be aligned further);
// cdd_split_combine then does the S-point inverse DFT over k1, the overlap-save
// trim, /N, rint and int8 wrap.  DMs of exactly 0 are copied from the rows by
// the combine step.
// 64 antennas x 8 channels x 65536 samples at 65536 points and DMs 0, 50, 150
// and 500: 7.46 ms with 16 points a thread in scalar arithmetic, 4.12 ms with
// these sub-transforms, 2.72 ms with the rows loaded without a branch between
// the loads (before, each waited for the last), 2.64 ms with pairs stored
// whole.  A cluster of S CTAs that combines from each other's shared memory
// instead of through the workspace took 3.58 ms: 15 clusters of 8 run at once,
// and its barriers tie both windows of a CTA together.
constexpr int kSplitLog = 13;
constexpr int kSplitM   = 1 << kSplitLog;

struct SplitArgs {
    const uint8_t* in;
    size_t row_stride;
    int nstreams, nsamples, overlap, lag, nseg, ndms, npa;
    size_t chirp_dm_stride;  // complex entries between two DMs' tables
    int item0, nitems;  // work items [item0, item0 + nitems) of this chunk
    const c32* tw;      // M-point plan tables
    const c32* chirp;   // [ndms][F][S][M]: bin k1 + S k2 at k1's per-thread load order
    const float4* tws;  // [S][M / 2] pair quads: W_N^(n2 k1)
    float2* z;          // [ndms][nitems][S][re|im][M / 2] pairs
    const uint32_t* zero_flags;  // [ndms]: non-zero if the DM is 0 (chirp exactly 1)
    uint8_t* out[kMaxDms];
    size_t out_stride;
    float2* dbg;
};

// W_S^m (forward sign) for S in {2, 4, 8}
template <int S>
__device__ __forceinline__ c32 wsm(int m)
{
    const float c2 = 0.70710678118654752440f;
    switch((m % S) * (8 / S)) {
    case 0: return {1.0f, 0.0f};
    case 1: return {c2, -c2};
    case 2: return {0.0f, -1.0f};
    case 3: return {-c2, -c2};
    case 4: return {-1.0f, 0.0f};
    case 5: return {-c2, c2};
    case 6: return {0.0f, 1.0f};
    default: return {c2, c2};
    }
}

template <int S>
__global__ void __launch_bounds__(kPkThreads, 1)
cdd_split_kernel(const __grid_constant__ SplitArgs A)
{
    constexpr int LOGN = kSplitLog, M = kSplitM, N = S * M;
    using G = PkGeo<LOGN>;
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ uint32_t s_tmem;
    PkGroup g;
    const uint32_t tmem =
        pk_setup<LOGN, false>(g, smem, &s_tmem, reinterpret_cast<const float*>(A.tw));
    const int t = g.t;
    const int L = N - A.overlap;
    const int avail = A.overlap + A.nsamples;
    // pairs of samples are aligned, and inside the rows or past them together
    const bool even = ((L | avail | (int)(A.row_stride & 1)) & 1) == 0 &&
                      (reinterpret_cast<uintptr_t>(A.in) & 1) == 0;

    const int nunits = A.nitems * S;
    for(int u = g.window * gridDim.x + blockIdx.x; u < nunits; u += G::W * gridDim.x) {
        const int il = u / S, k1 = u - il * S;
        const int item   = A.item0 + il;
        const int stream = item / A.nseg;
        const int seg    = item - stream * A.nseg;
        const int f      = stream / A.npa;
        const int start  = seg * L;
        const uint8_t* row_re = A.in + (size_t)stream * 2 * A.row_stride + start + 2 * t;
        const uint8_t* row_im = row_re + A.row_stride;
        // ---- S-point partial DFT for this k1, times W_N^(n2 k1), n2 = 2 t + 512 r
        Pk x[16];
#pragma unroll
        for(int r = 0; r < 16; ++r) x[r] = {0, 0};
#pragma unroll 1
        for(int n1 = 0; n1 < S; ++n1) {
            const c32 w = wsm<S>(n1 * k1);
            const Pk wp = {pk2(w.x, w.x), pk2(w.y, w.y)};
            const int left = avail - (start + n1 * M + 2 * t);  // samples from this thread's first
            if(avail - (start + n1 * M) <= 0) break;            // zero padding from here on
            // all loads of 8 pairs in flight at once: no branch between them (pairs
            // past the end read the row's first samples and count as zeros)
#pragma unroll
            for(int h = 0; h < 16; h += 8) {
                uint32_t re[8], im[8];
                if(even) {
#pragma unroll
                    for(int i = 0; i < 8; ++i) {
                        const bool in = 512 * (h + i) < left;
                        const int at  = in ? n1 * M + 512 * (h + i) : -2 * t;
                        const uint32_t a = *reinterpret_cast<const uint16_t*>(row_re + at);
                        const uint32_t b = *reinterpret_cast<const uint16_t*>(row_im + at);
                        re[i] = in ? a : 0;
                        im[i] = in ? b : 0;
                    }
                } else {
                    for(int i = 0; i < 8; ++i) {
                        const int at = n1 * M + 512 * (h + i);
                        re[i] = im[i] = 0;
                        if(512 * (h + i) < left) { re[i] = row_re[at]; im[i] = row_im[at]; }
                        if(512 * (h + i) + 1 < left) {
                            re[i] |= (uint32_t)row_re[at + 1] << 8;
                            im[i] |= (uint32_t)row_im[at + 1] << 8;
                        }
                    }
                }
#pragma unroll
                for(int i = 0; i < 8; ++i) {
                    const uint64_t xr = pk2((float)(int8_t)re[i], (float)(int8_t)(re[i] >> 8));
                    const uint64_t xi = pk2((float)(int8_t)im[i], (float)(int8_t)(im[i] >> 8));
                    Pk& v = x[h + i];
                    v.re = psub(pfma(xr, wp.re, v.re), pmul(xi, wp.im));
                    v.im = pfma(xi, wp.re, pfma(xr, wp.im, v.im));
                }
            }
        }
        const float4* tws = A.tws + (size_t)k1 * (M / 2) + t;
        if(k1 > 0) {
#pragma unroll
            for(int r = 0; r < 16; ++r) {
                const float4 w = tws[256 * r];
                x[r] = pcmul<false>(x[r], Pk{pk2(w.x, w.y), pk2(w.z, w.w)});
            }
        }
        pk_sync<LOGN>(g);  // the previous unit's last reads of shared memory are done
        pk_forward<LOGN>(g, x, [] {});
        const float4* chp =
            reinterpret_cast<const float4*>(A.chirp + (size_t)f * N + (size_t)k1 * M) + t;
        for(int d = 0; d < A.ndms; ++d) {
            if(A.zero_flags[d] && !A.dbg) continue;
            pk_inverse<LOGN>(g, chp + (size_t)d * A.chirp_dm_stride / 2, x);
            float2* zo = A.z + (((size_t)d * A.nitems + il) * S + k1) * M + t;
#pragma unroll
            for(int r = 0; r < 16; ++r) {
                const float4 w = tws[256 * r];
                const Pk z = pcmul<true>(x[r], Pk{pk2(w.x, w.y), pk2(w.z, w.w)});
                float2 re, im;
                unpk2(z.re, re.x, re.y);
                unpk2(z.im, im.x, im.y);
                zo[256 * r]         = re;
                zo[M / 2 + 256 * r] = im;
            }
            pk_sync<LOGN>(g);
        }
    }
    pk_tmem_free(tmem);
}

template <int S>
__global__ void __launch_bounds__(256)
cdd_split_combine(const __grid_constant__ SplitArgs A)
{
    constexpr int M = kSplitM, N = S * M;
    const int L = N - A.overlap, head = A.overlap - A.lag;
    const float inv_n = 1.0f / (float)N;  // exact (power of two)
    // as in cdd_pk_kernel: the low byte of v / N + 1.5 2^23 is the sample
    const uint64_t scale = pk2(inv_n, inv_n), magic = pk2(12582912.0f, 12582912.0f);
    // both samples of a pair are kept or trimmed together, at even places
    const bool even = ((L | head | A.nsamples) & 1) == 0 && (A.out_stride & 1) == 0;
    const bool even_in = even && (A.row_stride & 1) == 0 &&
                         (reinterpret_cast<uintptr_t>(A.in) & 1) == 0;
    const size_t total = (size_t)A.ndms * A.nitems * (M / 2);
    for(size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
        idx += (size_t)gridDim.x * blockDim.x) {
        const int n2 = 2 * (int)(idx % (M / 2));
        const size_t rest = idx / (M / 2);
        const int il = (int)(rest % A.nitems);
        const int d  = (int)(rest / A.nitems);
        const int item   = A.item0 + il;
        const int stream = item / A.nseg;
        const int seg    = item - stream * A.nseg;
        const int start  = seg * L;
        const unsigned kept = (unsigned)max(0, min(L, A.nsamples - start));
        uint8_t* o_re = A.out[d] + (size_t)stream * 2 * A.out_stride + start;
        uint8_t* o_im = o_re + A.out_stride;
        if(A.zero_flags[d] && !A.dbg) {
            const uint8_t* i_re = A.in + (size_t)stream * 2 * A.row_stride + start + head;
            if(even_in && (reinterpret_cast<uintptr_t>(A.out[d]) & 1) == 0) {
#pragma unroll
                for(int n1 = 0; n1 < S; ++n1) {
                    const int v = n2 + n1 * M - head;
                    if((unsigned)v < kept) {
                        *reinterpret_cast<uint16_t*>(o_re + v) =
                            *reinterpret_cast<const uint16_t*>(i_re + v);
                        *reinterpret_cast<uint16_t*>(o_im + v) =
                            *reinterpret_cast<const uint16_t*>(i_re + A.row_stride + v);
                    }
                }
                continue;
            }
            for(int n1 = 0; n1 < S; ++n1)
                for(int e = 0; e < 2; ++e) {
                    const int v = n2 + e + n1 * M - head;
                    if((unsigned)v < kept) {
                        o_re[v] = i_re[v];
                        o_im[v] = i_re[A.row_stride + v];
                    }
                }
            continue;
        }
        const float2* zi = A.z + ((size_t)d * A.nitems + il) * S * M + n2 / 2;
        Pk z[S];
#pragma unroll
        for(int k1 = 0; k1 < S; ++k1) {
            const float2 re = zi[(size_t)k1 * M], im = zi[(size_t)k1 * M + M / 2];
            z[k1] = {pk2(re.x, re.y), pk2(im.x, im.y)};
        }
        pdft<S, true>(z);  // z[n1] = sum_k1 W_S^(-n1 k1) z'[k1]
        const bool none = no_number(z[0]);
        const bool words = even && !A.dbg && (reinterpret_cast<uintptr_t>(A.out[d]) & 1) == 0;
#pragma unroll
        for(int n1 = 0; n1 < S; ++n1) {
            const int v = n2 + n1 * M - head;
            uint32_t re[2], im[2];
            unpk2u(pfma(z[n1].re, scale, magic), re[0], re[1]);
            unpk2u(pfma(z[n1].im, scale, magic), im[0], im[1]);
            if(none) re[0] = re[1] = im[0] = im[1] = 0;
            if(words) {
                if((unsigned)v < kept) {
                    *reinterpret_cast<uint16_t*>(o_re + v) =
                        (uint16_t)__byte_perm(re[0], re[1], 0x0040);
                    *reinterpret_cast<uint16_t*>(o_im + v) =
                        (uint16_t)__byte_perm(im[0], im[1], 0x0040);
                }
                continue;
            }
            float fr[2], fi[2];
            unpk2(pmul(z[n1].re, scale), fr[0], fr[1]);
            unpk2(pmul(z[n1].im, scale), fi[0], fi[1]);
#pragma unroll
            for(int e = 0; e < 2; ++e)
                if((unsigned)(v + e) < kept) {
                    o_re[v + e] = (uint8_t)re[e];
                    o_im[v + e] = (uint8_t)im[e];
                    if(A.dbg)
                        A.dbg[((size_t)d * A.nstreams + stream) * A.nsamples + start + v + e] =
                            make_float2(fr[e], fi[e]);
                }
        }
    }
}

template <int S>
int launch_split(SplitArgs a, int total_items, size_t ws_items, cudaStream_t stream)
{
    const size_t smem = kPkBufBytes;
    SW_CUDA_CHECK(cudaFuncSetAttribute(cdd_split_kernel<S>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    for(int i0 = 0; i0 < total_items; i0 += (int)ws_items) {
        a.item0  = i0;
        a.nitems = (int)std::min<size_t>(ws_items, (size_t)(total_items - i0));
        const long units = (long)a.nitems * S;
        cdd_split_kernel<S><<<(int)std::min<long>(units, nsm), kPkThreads, smem, stream>>>(a);
        SW_LAUNCH_CHECK();
        const size_t total = (size_t)a.ndms * a.nitems * (kSplitM / 2);
        const size_t blocks = std::min<size_t>(cdiv(total, (size_t)256), (size_t)nsm * 16);
        cdd_split_combine<S><<<(int)blocks, 256, 0, stream>>>(a);
        SW_LAUNCH_CHECK();
    }
    return SW_OK;
}

// ------------------------------------------------------------- setup
struct SetupArgs {
    int logn, ndms, nchans;
    double low_freq, coarse_bw, fine_bw;
    double prefactor[kMaxDms];
};

struct ZeroFlags {
    uint32_t f[kMaxDms];
};
__global__ void set_flags_k(uint32_t* p, ZeroFlags z) { p[threadIdx.x] = z.f[threadIdx.x]; }

__global__ void twiddle_k(c32* tw, int logn)
{
    const Plan P = make_plan(logn);
    for(int p = 0; p < P.npass; ++p) {
        const int s = P.stride[p], R = P.radix[p], G = P.span[p];
        if(s <= 1) continue;
        const int entries = (R == 16 ? 16 : R - 1) * s;
        for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < entries;
            i += gridDim.x * blockDim.x) {
            int q, j;
            if(R == 16) {  // c32 index i = 2*(k*s + j) + h holds w_(2k+1+h)
                const int m = i >> 1, h = i & 1;
                q = 2 * (m / s) + 1 + h;
                j = m % s;
            } else {
                q = i / s + 1;
                j = i % s;
            }
            double sn = 0.0, cs = 0.0;
            // exp(-2 pi i j q / G) in FP64
            if(q < R) sincospi(-2.0 * (double)(j * q) / (double)G, &sn, &cs);
            tw[P.tw_off[p] + i] = c32{(float)cs, (float)sn};
        }
    }
}

// Twiddles of the packed transform (PkGeo: pass 0's quads, then pass 1's).
__global__ void twiddle_pk_k(float4* tw, int logn)
{
    const int n = 1 << logn, cols0 = n / 32, cols1 = n / 512;
    for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < 15 * (cols0 + cols1);
        i += gridDim.x * blockDim.x) {
        const bool first = i < 15 * cols0;
        const int k = first ? i : i - 15 * cols0, cols = first ? cols0 : cols1;
        const int q = 1 + k / cols, j = 2 * (k % cols), span = first ? n : n / 16;
        double s0, c0, s1, c1;
        sincospi(-2.0 * (double)(j * q) / (double)span, &s0, &c0);
        sincospi(-2.0 * (double)((j + 1) * q) / (double)span, &s1, &c1);
        tw[i] = make_float4((float)c0, (float)c1, (float)s0, (float)s1);
    }
}
template <int LOGN>
constexpr bool pk_twiddles_fit()
{
    return (PkGeo<LOGN>::TW0 + PkGeo<LOGN>::TW1) * 2 <= make_plan(LOGN).tw_total;
}
static_assert(pk_twiddles_fit<10>() && pk_twiddles_fit<11>() && pk_twiddles_fit<12>() &&
                  pk_twiddles_fit<13>(),
              "setup block layout");

// Entry q of an N-point chirp table in the packed transform's order: quad
// (i, t) at i * (N / 32) + t holds the two bins of pair i of thread t as
// (re, re, im, im).
struct PkBin {
    int bin;
    int word;  // of the table: the real part; the imaginary part is 2 words on
};
__device__ __forceinline__ PkBin pk_bin(int logn, int q)
{
    const int n = 1 << logn, r2 = n / 256, cols = n / 32;
    const int h = q & 1, quad = q >> 1, t = quad % cols, i = quad / cols;
    const int block = t * (32 / r2) + i / (r2 / 2);  // transform of pass 2
    const int k = i % (r2 / 2) + h * (r2 / 2);
    return {block / 16 + 16 * (block % 16) + 256 * k, 4 * quad + h};
}

// DMResponse (CoherentDedisperser.cu:313-335) in FP64.  The transform
// leaves bin digit_reverse(16 t + r) in register r of thread t; the table
// stores the chirp of that bin at ((r / 2) * (N / 16) + t) * 2 + r % 2, so
// that the k-th 16-byte load of every thread (registers 2k and 2k+1) reads
// one contiguous 512-byte span per warp.
__global__ void chirp_k(c32* chirp, SetupArgs S)
{
    const Plan P = make_plan(S.logn);
    const int nt = P.n / 16;
    const size_t total = (size_t)S.ndms * S.nchans * P.n;
    for(size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total;
        i += (size_t)gridDim.x * blockDim.x) {
        const int q   = (int)(i % P.n);
        const int c   = (int)((i / P.n) % S.nchans);
        const int d   = (int)(i / ((size_t)P.n * S.nchans));
        const int t   = (q >> 1) % nt;
        const int r   = 2 * ((q >> 1) / nt) + (q & 1);
        const bool pk = S.logn >= kPkMinLog;
        const PkBin b = pk ? pk_bin(S.logn, q) : PkBin{};
        const int k   = pk ? b.bin : digit_reverse(P, 16 * t + r);
        const double nu0   = S.low_freq + c * S.coarse_bw - 0.5 * S.coarse_bw;
        const double nu    = k * S.fine_bw;
        const double phase = (nu * nu * S.prefactor[d]) / ((nu0 + nu) * nu0 * nu0);
        double sn, cs;
        sincos(phase, &sn, &cs);
        if(pk) {
            float* w = reinterpret_cast<float*>(chirp + (i - q)) + b.word;
            w[0] = (float)cs;
            w[2] = (float)sn;
        } else {
            chirp[i] = c32{(float)cs, (float)sn};
        }
    }
}

// Chirp tables for the split transform: bin k1 + S k2 of sub-transform k1
// at k1 * M + (the M-point per-thread load order of k2).
__global__ void chirp_split_k(c32* chirp, SetupArgs S, int split)
{
    const int n  = split * kSplitM;
    const size_t total = (size_t)S.ndms * S.nchans * n;
    for(size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total;
        i += (size_t)gridDim.x * blockDim.x) {
        const int q  = (int)(i % n);
        const int c  = (int)((i / n) % S.nchans);
        const int d  = (int)(i / ((size_t)n * S.nchans));
        const int k1 = q / kSplitM, qq = q % kSplitM;
        const PkBin b = pk_bin(kSplitLog, qq);
        const int k  = k1 + split * b.bin;
        const double nu0   = S.low_freq + c * S.coarse_bw - 0.5 * S.coarse_bw;
        const double nu    = k * S.fine_bw;
        const double phase = (nu * nu * S.prefactor[d]) / ((nu0 + nu) * nu0 * nu0);
        double sn, cs;
        sincos(phase, &sn, &cs);
        float* w = reinterpret_cast<float*>(chirp + (i - qq)) + b.word;
        w[0] = (float)cs;
        w[2] = (float)sn;
    }
}

// W_N^(n2 k1) = exp(-2 pi i n2 k1 / N) in FP64, [k1][n2 / 2] pair quads
__global__ void split_twiddle_k(float* tws, int split)
{
    const int n = split * kSplitM;
    for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int k1 = i / kSplitM, n2 = i % kSplitM;
        double sn, cs;
        sincospi(-2.0 * (double)((long long)n2 * k1) / (double)n, &sn, &cs);
        float* w = tws + 4 * (i / 2) + (i & 1);  // n2 = i mod M: pairs stay together
        w[0] = (float)cs;
        w[2] = (float)sn;
    }
}

template <int LOGN, bool DBG>
int launch_logn_dbg(const Args& a, cudaStream_t stream)
{
    constexpr int N = 1 << LOGN;
    constexpr Plan P = make_plan(LOGN);
    const size_t smem = (size_t)(pad(N) + 16 + ((P.tw_total + 1) & ~1)) * sizeof(c32) + 2 * N;
    SW_CUDA_CHECK(cudaFuncSetAttribute(cdd_kernel<LOGN, DBG>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int dev = 0, nsm = 148, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    SW_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cdd_kernel<LOGN, DBG>,
                                                                 N / 16, smem));
    if(per_sm < 1) per_sm = 1;
    const long items = (long)a.nstreams * a.nseg;
    const long grid  = items < (long)nsm * per_sm ? items : (long)nsm * per_sm;
    cdd_kernel<LOGN, DBG><<<(int)grid, N / 16, smem, stream>>>(a);
    SW_LAUNCH_CHECK();
    return SW_OK;
}

template <int LOGN, bool DBG, bool SPLIT>
int launch_pk_instance(const Args& a, long units, int nsm, cudaStream_t stream)
{
    const size_t smem = kPkBufBytes + kPkStageBytes;
    SW_CUDA_CHECK(cudaFuncSetAttribute(cdd_pk_kernel<LOGN, DBG, SPLIT>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    // the first window of every SM before the second of any
    const int ctas = (int)std::min<long>(units, nsm);
    cdd_pk_kernel<LOGN, DBG, SPLIT><<<ctas, kPkThreads, smem, stream>>>(a);
    SW_LAUNCH_CHECK();
    return SW_OK;
}

template <int LOGN>
int launch_pk(Args a, cudaStream_t stream)
{
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const long items = (long)a.nstreams * a.nseg;
    if(a.dbg) return launch_pk_instance<LOGN, true, false>(a, items, nsm, stream);
    // A window's DMs are one group's serial chain, 1.9 us apiece for a lone
    // warp of 1024 points.  Launches with fewer windows than the SMs can run
    // side by side (groups of up to four warps, one per scheduler) share the
    // DMs between groups, each with its own forward transform: 64 windows and 8
    // DMs 21.7 -> 8.6 us at 1024 points, 22.9 -> 11.1 at 2048, 34.7 -> 21.7 at 8192.
    const long groups = (long)nsm * std::max(1, 128 / PkGeo<LOGN>::T);
    const int share = (int)std::max(1l, std::min<long>(a.ndms, groups / items));
    if(share == 1) return launch_pk_instance<LOGN, false, false>(a, items, nsm, stream);
    a.dm_group = cdiv(a.ndms, share);
    a.ndmg     = cdiv(a.ndms, a.dm_group);
    return launch_pk_instance<LOGN, false, true>(a, items * a.ndmg, nsm, stream);
}

// the float output for precision studies is a separate instance, so the
// production kernel carries none of its registers
template <int LOGN>
int launch_logn(const Args& a, cudaStream_t stream)
{
    return a.dbg ? launch_logn_dbg<LOGN, true>(a, stream) : launch_logn_dbg<LOGN, false>(a, stream);
}

int log2_exact(int n)
{
    int l = 0;
    while((1 << l) < n) ++l;
    return (1 << l) == n ? l : -1;
}

// Setup block: per-pass twiddles, a gap of kSetupGap complex entries whose
// first words flag the DMs of exactly 0, the chirp tables [ndms][nchans][N]
// and, for split transforms, the W_N^(n2 k1) table.
constexpr int kSetupGap = 64;  // >= kMaxDms 32-bit flags

// Dedisperse `nchans` channels (of a setup built for setup_nchans channels
// and setup_ndms DMs, starting at channel chan0) for `ndms` DMs starting at
// dm0 of the setup.
int launch_cdd(const void* d_fpact_in, size_t row_stride, int nchans, int npol, int nant,
               int nsamples, int fft_len, int overlap, int lag, const void* d_setup,
               int setup_ndms, int setup_nchans, int chan0, int dm0, int ndms,
               void* const* h_d_out, size_t out_row_stride, void* d_workspace,
               size_t workspace_bytes, float* d_debug_f32, sw_stream_t stream)
{
    const int logn = log2_exact(fft_len);
    SW_REQUIRE(logn >= 8 && logn <= 16,
               "coherent dedispersion: fft_len must be a power of two in [256, 65536]");
    SW_REQUIRE(d_fpact_in && d_setup && h_d_out, "coherent dedispersion: null pointer");
    SW_REQUIRE(ndms > 0 && ndms <= kMaxDms, "coherent dedispersion: 1..%d DMs", kMaxDms);
    SW_REQUIRE(overlap >= 0 && overlap < fft_len,
               "coherent dedispersion: overlap must be smaller than the FFT");
    SW_REQUIRE(lag >= 0 && lag <= overlap,
               "coherent dedispersion: the lag (%d) must lie in [0, overlap = %d]", lag, overlap);
    SW_REQUIRE(nsamples > 0 && (size_t)overlap + nsamples <= row_stride,
               "coherent dedispersion: input rows must hold history + gulp");
    SW_REQUIRE((size_t)nsamples <= out_row_stride, "coherent dedispersion: output rows too short");
    SW_REQUIRE(nchans > 0 && npol > 0 && nant > 0, "coherent dedispersion: empty shape");
    const int plog = logn > kSplitLog ? kSplitLog : logn;
    const Plan P = make_plan(plog);
    const c32* tw = static_cast<const c32*>(d_setup);
    const c32* ch_all = tw + P.tw_total + kSetupGap;
    const c32* ch = ch_all + ((size_t)dm0 * setup_nchans + chan0) * fft_len;
    const uint32_t* zero_flags = reinterpret_cast<const uint32_t*>(tw + P.tw_total) + dm0;
    const int nstreams = nchans * npol * nant;
    const int nseg = cdiv(nsamples, fft_len - overlap);
    cudaStream_t s = as_cuda(stream);
    if(logn > kSplitLog) {
        const size_t per_item = (size_t)ndms * fft_len * sizeof(c32);
        SW_REQUIRE(d_workspace && workspace_bytes >= per_item,
                   "coherent dedispersion: fft_len %d needs a workspace of at least %zu bytes "
                   "(sw_cdd_workspace_bytes)", fft_len, per_item);
        SplitArgs a{};
        a.in = static_cast<const uint8_t*>(d_fpact_in);
        a.row_stride = row_stride;
        a.nstreams = nstreams;
        a.nsamples = nsamples;
        a.overlap = overlap;
        a.lag = lag;
        a.nseg = nseg;
        a.ndms = ndms;
        a.npa = npol * nant;
        a.chirp_dm_stride = (size_t)setup_nchans * fft_len;
        a.tw = tw;
        a.chirp = ch;
        a.tws = reinterpret_cast<const float4*>(ch_all + (size_t)setup_ndms * setup_nchans * fft_len);
        a.z = static_cast<float2*>(d_workspace);
        a.zero_flags = zero_flags;
        for(int d = 0; d < ndms; ++d) {
            SW_REQUIRE(h_d_out[d], "coherent dedispersion: null output for DM %d", d);
            a.out[d] = static_cast<uint8_t*>(h_d_out[d]);
        }
        a.out_stride = out_row_stride;
        a.dbg = reinterpret_cast<float2*>(d_debug_f32);
        const int items = nstreams * nseg;
        const size_t ws_items = std::min<size_t>(workspace_bytes / per_item, (size_t)items);
        switch(fft_len / kSplitM) {
        case 2: return launch_split<2>(a, items, ws_items, s);
        case 4: return launch_split<4>(a, items, ws_items, s);
        default: return launch_split<8>(a, items, ws_items, s);
        }
    }
    Args a{};
    a.in         = static_cast<const uint8_t*>(d_fpact_in);
    a.row_stride = row_stride;
    a.npa        = npol * nant;
    a.nstreams   = nstreams;
    a.nsamples   = nsamples;
    a.overlap    = overlap;
    a.lag        = lag;
    a.nseg       = nseg;
    a.ndms       = ndms;
    a.chirp_dm_stride = (size_t)setup_nchans * fft_len;
    a.tw         = tw;
    a.chirp      = ch;
    a.zero_flags = zero_flags;
    for(int d = 0; d < ndms; ++d) {
        SW_REQUIRE(h_d_out[d], "coherent dedispersion: null output for DM %d", d);
        a.out[d] = static_cast<uint8_t*>(h_d_out[d]);
    }
    a.out_stride = out_row_stride;
    a.dbg        = reinterpret_cast<float2*>(d_debug_f32);
    switch(logn) {
    case 8: return launch_logn<8>(a, s);
    case 9: return launch_logn<9>(a, s);
    case 10: return launch_pk<10>(a, s);
    case 11: return launch_pk<11>(a, s);
    case 12: return launch_pk<12>(a, s);
    default: return launch_pk<13>(a, s);
    }
}

}  // namespace cdd
}  // namespace swb

using namespace swb;
using namespace swb::cdd;

extern "C" {

size_t sw_cdd_setup_bytes(int ndms, int nchans, int fft_len)
{
    const int logn = log2_exact(fft_len);
    if(logn < 8 || logn > 16 || ndms <= 0 || nchans <= 0) return 0;
    const Plan P = make_plan(logn > kSplitLog ? kSplitLog : logn);
    const size_t split_tw = logn > kSplitLog ? (size_t)fft_len : 0;
    return ((size_t)P.tw_total + kSetupGap + (size_t)ndms * nchans * fft_len + split_tw) *
           sizeof(c32);
}

int sw_cdd_chirps(const float* h_dms, int ndms, int nchans, int fft_len,
                  double low_freq, double bw, void* d_setup, sw_stream_t stream)
{
    const int logn = log2_exact(fft_len);
    SW_REQUIRE(logn >= 8 && logn <= 16,
               "coherent dedispersion: fft_len must be a power of two in [256, 65536]");
    SW_REQUIRE(h_dms && ndms > 0 && ndms <= kMaxDms, "coherent dedispersion: 1..%d DMs", kMaxDms);
    SW_REQUIRE(d_setup && nchans > 0, "coherent dedispersion: bad setup arguments");
    const int plog = logn > kSplitLog ? kSplitLog : logn;
    const Plan P = make_plan(plog);
    c32* tw = static_cast<c32*>(d_setup);
    c32* ch = tw + P.tw_total + kSetupGap;
    if(plog >= kPkMinLog)
        twiddle_pk_k<<<32, 128, 0, as_cuda(stream)>>>(reinterpret_cast<float4*>(tw), plog);
    else twiddle_k<<<64, 256, 0, as_cuda(stream)>>>(tw, plog);
    SW_LAUNCH_CHECK();
    // the words after the twiddle tables flag the DMs of exactly 0
    ZeroFlags zf{};
    for(int d = 0; d < ndms; ++d) zf.f[d] = h_dms[d] == 0.0f ? 1u : 0u;
    set_flags_k<<<1, kMaxDms, 0, as_cuda(stream)>>>(reinterpret_cast<uint32_t*>(tw + P.tw_total),
                                                     zf);
    SW_LAUNCH_CHECK();
    SetupArgs S{};
    S.logn      = logn;
    S.ndms      = ndms;
    S.nchans    = nchans;
    S.low_freq  = low_freq;
    S.coarse_bw = bw / nchans;
    S.fine_bw   = S.coarse_bw / fft_len;
    for(int d = 0; d < ndms; ++d)
        S.prefactor[d] = -1.0 * (2.0 * 3.1415926535897932385) * 4.148806423e15 * (double)h_dms[d];
    if(logn > kSplitLog) {
        const int split = fft_len / kSplitM;
        chirp_split_k<<<148 * 4, 256, 0, as_cuda(stream)>>>(ch, S, split);
        SW_LAUNCH_CHECK();
        split_twiddle_k<<<64, 256, 0, as_cuda(stream)>>>(
            reinterpret_cast<float*>(ch + (size_t)ndms * nchans * fft_len), split);
        SW_LAUNCH_CHECK();
    } else {
        chirp_k<<<148 * 4, 256, 0, as_cuda(stream)>>>(ch, S);
        SW_LAUNCH_CHECK();
    }
    return SW_OK;
}

size_t sw_cdd_workspace_bytes(int nchans, int npol, int nant, int nsamples, int fft_len,
                              int overlap, int ndms)
{
    const int logn = log2_exact(fft_len);
    if(logn <= kSplitLog) return 0;
    if(logn > 16 || overlap < 0 || overlap >= fft_len || nsamples <= 0 || ndms <= 0) return 0;
    const size_t items = (size_t)nchans * npol * nant * cdiv(nsamples, fft_len - overlap);
    return items * ndms * fft_len * sizeof(c32);
}

int sw_coherent_dedisperse_ws(const void* d_fpact_in, size_t row_stride, int nchans, int npol,
                              int nant, int nsamples, int fft_len, int overlap, int lag,
                              const void* d_setup, int ndms, void* const* h_d_out,
                              size_t out_row_stride, void* d_workspace,
                              size_t workspace_bytes, float* d_debug_f32,
                              sw_stream_t stream)
{
    SW_REQUIRE(d_setup, "coherent dedispersion: null setup");
    return launch_cdd(d_fpact_in, row_stride, nchans, npol, nant, nsamples, fft_len, overlap,
                      lag, d_setup, ndms, nchans, 0, 0, ndms, h_d_out, out_row_stride,
                      d_workspace, workspace_bytes, d_debug_f32, stream);
}

int sw_coherent_dedisperse_channel(const void* d_fpact_in, size_t row_stride, int npol,
                                   int nant, int nsamples, int fft_len, int overlap, int lag,
                                   const void* d_setup, int setup_ndms, int setup_nchans,
                                   int freq_idx, int dm_idx, void* d_out,
                                   size_t out_row_stride, void* d_workspace,
                                   size_t workspace_bytes, sw_stream_t stream)
{
    SW_REQUIRE(d_setup && d_out, "coherent dedispersion: null pointer");
    SW_REQUIRE(setup_ndms > 0 && setup_nchans > 0 && freq_idx >= 0 && freq_idx < setup_nchans &&
                   dm_idx >= 0 && dm_idx < setup_ndms,
               "coherent dedispersion: channel %d / DM %d outside the setup (%d channels, %d DMs)",
               freq_idx, dm_idx, setup_nchans, setup_ndms);
    void* outs[1] = {d_out};
    return launch_cdd(d_fpact_in, row_stride, 1, npol, nant, nsamples, fft_len, overlap, lag,
                      d_setup, setup_ndms, setup_nchans, freq_idx, dm_idx, 1, outs,
                      out_row_stride, d_workspace, workspace_bytes, nullptr, stream);
}

int sw_coherent_dedisperse(const void* d_fpact_in, size_t row_stride,
                           int nchans, int npol, int nant, int nsamples,
                           int fft_len, int overlap, int lag, const void* d_setup,
                           int ndms, void* const* h_d_out,
                           size_t out_row_stride, sw_stream_t stream)
{
    SW_REQUIRE(fft_len <= kSplitM,
               "coherent dedispersion: fft_len %d > %d needs sw_coherent_dedisperse_ws", fft_len,
               kSplitM);
    return sw_coherent_dedisperse_ws(d_fpact_in, row_stride, nchans, npol, nant, nsamples,
                                     fft_len, overlap, lag, d_setup, ndms, h_d_out, out_row_stride,
                                     nullptr, 0, nullptr, stream);
}

}  // extern "C"
