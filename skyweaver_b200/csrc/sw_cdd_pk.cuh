// Transforms of the coherent dedisperser in packed pairs: N = 1024 .. 8192
// points as 16 x 16 x R2, R2 = N / 256.
//
// A window is transformed by a group of N / 32 threads, 32 points a thread, in
// shared memory, which it crosses twice.  Points are kept in pairs of
// neighbours (2 i, 2 i + 1) as (re0, re1, im0, im1): one 16-byte access, and
// both butterflies of a pair run in packed f32x2 instructions.
//   pass 0 (span N):      butterflies j = 2 t, 2 t + 1, points j + (N / 16) r
//   pass 1 (span 16 R2):  butterflies b = 2 t, 2 t + 1 (block b / R2, column
//                         b % R2), points R2 apart
//   pass 2 (span R2):     points 32 t .. 32 t + 31 as 32 / R2 transforms of R2
//                         points, each as R2 / 2 points of its even and of its
//                         odd points in the two lanes, combined across the
//                         lanes
// Passes 1 and 2 exchange points inside R2 / 2 neighbouring threads of one
// warp only, so just pass 0 needs the group's barrier.  Pair beta (R2 / 2) + k
// of thread t ends the forward with bins q0 + 16 q1 + 256 k of transform
// 16 q0 + q1 = t (32 / R2) + beta and with the bin 128 R2 above.
//
// What never changes between windows stays in tensor memory, whose loads go
// past the shared-memory pipe: the twiddles of passes 0 and 1 (each thread
// always needs the same 60 floats of each) and, between the DMs, the window's
// spectrum.
//
// Shared memory holds rows of 32 points padded by one 16-byte quad, which
// keeps the three passes' 16-byte accesses free of bank conflicts for every R2.
#pragma once

#include "sw_common.cuh"

namespace swb {
namespace cdd {

constexpr int kPkMinLog  = 10, kPkMaxLog = 13;
constexpr int kPkThreads = 512;                   // per CTA
constexpr int kPkRow     = 34;                    // points per padded row of 32
constexpr int kPkBufBytes = kPkThreads * kPkRow * 8;  // all windows of a CTA
constexpr int kPkStageBytes = 2 * 32 * kPkThreads;    // their int8 inputs

// Geometry of N = 2^LOGN.
template <int LOGN>
struct PkGeo {
    static constexpr int N = 1 << LOGN, R2 = N / 256;
    static constexpr int T = N / 32;              // threads per window
    static constexpr int W = kPkThreads / T;      // windows per CTA
    // twiddle table (quads): pass 0 as [15][N / 32] and pass 1 as [15][R2 / 2]
    // quads (wr_j, wr_j+1, wi_j, wi_j+1), w = exp(-2 pi i j q / span), q = 1 .. 15
    static constexpr int TW0 = 15 * T, TW1 = 15 * (R2 / 2);
    static constexpr int STEP0 = N / 16 / 32 * kPkRow * 8;  // bytes between pass 0's quads
    // byte offset of pass 1's quad q from its first (R2 q points on)
    static __device__ __forceinline__ constexpr int off1(int q)
    {
        return ((R2 * q / 32) * kPkRow + R2 * q % 32) * 8;
    }
};

struct Pk {
    uint64_t re, im;
};

__device__ __forceinline__ uint64_t pk2(float lo, float hi)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ uint64_t pk2u(uint32_t lo, uint32_t hi)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ void unpk2(uint64_t v, float& lo, float& hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ void unpk2u(uint64_t v, uint32_t& lo, uint32_t& hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t padd(uint64_t a, uint64_t b)
{
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t psub(uint64_t a, uint64_t b)
{
    uint64_t d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t pmul(uint64_t a, uint64_t b)
{
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t pfma(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// a * w, or a * conj(w)
template <bool CONJ>
__device__ __forceinline__ Pk pcmul(const Pk& a, const Pk& w)
{
    if constexpr(CONJ)
        return {pfma(a.re, w.re, pmul(a.im, w.im)), psub(pmul(a.im, w.re), pmul(a.re, w.im))};
    else
        return {psub(pmul(a.re, w.re), pmul(a.im, w.im)), pfma(a.re, w.im, pmul(a.im, w.re))};
}

// 4-point DFT of each lane; ROT2: x2 still lacks its factor -i (inverse: +i)
template <bool INV, bool ROT2>
__device__ __forceinline__ void pdft4(Pk& x0, Pk& x1, Pk& x2, Pk& x3)
{
    Pk t0, t1;
    if constexpr(!ROT2) {
        t0 = {padd(x0.re, x2.re), padd(x0.im, x2.im)};
        t1 = {psub(x0.re, x2.re), psub(x0.im, x2.im)};
    } else if constexpr(!INV) {  // x2 -> (im, -re)
        t0 = {padd(x0.re, x2.im), psub(x0.im, x2.re)};
        t1 = {psub(x0.re, x2.im), padd(x0.im, x2.re)};
    } else {  // x2 -> (-im, re)
        t0 = {psub(x0.re, x2.im), padd(x0.im, x2.re)};
        t1 = {padd(x0.re, x2.im), psub(x0.im, x2.re)};
    }
    const Pk t2 = {padd(x1.re, x3.re), padd(x1.im, x3.im)};
    const Pk t3 = {psub(x1.re, x3.re), psub(x1.im, x3.im)};
    x0 = {padd(t0.re, t2.re), padd(t0.im, t2.im)};
    x2 = {psub(t0.re, t2.re), psub(t0.im, t2.im)};
    if constexpr(!INV) {
        x1 = {padd(t1.re, t3.im), psub(t1.im, t3.re)};
        x3 = {psub(t1.re, t3.im), padd(t1.im, t3.re)};
    } else {
        x1 = {psub(t1.re, t3.im), padd(t1.im, t3.re)};
        x3 = {padd(t1.re, t3.im), psub(t1.im, t3.re)};
    }
}

// 16-point DFT of each lane, natural order in and out
template <bool INV>
__device__ __forceinline__ void pdft16(Pk* x)
{
    const float c1 = 0.92387953251128675613f, s1 = 0.38268343236508977173f;
    const float c2 = 0.70710678118654752440f;
#pragma unroll
    for(int r = 0; r < 4; ++r) pdft4<INV, false>(x[r], x[4 + r], x[8 + r], x[12 + r]);
    // x[4 q + r] times W_16^(r q); W_16^4 = -i is left to the second pdft4
    auto mulc = [](Pk& a, float wr, float wi) {  // wi of the forward sign
        a = pcmul<INV>(a, Pk{pk2(wr, wr), pk2(wi, wi)});
    };
    mulc(x[5], c1, -s1);
    mulc(x[7], s1, -c1);
    mulc(x[13], s1, -c1);
    mulc(x[15], -c1, s1);
    const uint64_t C = pk2(c2, c2), NC = pk2(-c2, -c2);
    auto mul2 = [&](Pk& a) {  // W_16^2 = c2 (1 - i)
        const uint64_t s = padd(a.re, a.im);
        const uint64_t d = INV ? psub(a.re, a.im) : psub(a.im, a.re);
        a = INV ? Pk{pmul(d, C), pmul(s, C)} : Pk{pmul(s, C), pmul(d, C)};
    };
    auto mul6 = [&](Pk& a) {  // W_16^6 = -c2 (1 + i)
        const uint64_t s = padd(a.re, a.im);
        const uint64_t d = INV ? psub(a.re, a.im) : psub(a.im, a.re);
        a = INV ? Pk{pmul(s, NC), pmul(d, C)} : Pk{pmul(d, C), pmul(s, NC)};
    };
    mul2(x[6]);
    mul2(x[9]);
    mul6(x[11]);
    mul6(x[14]);
    pdft4<INV, false>(x[0], x[1], x[2], x[3]);
    pdft4<INV, false>(x[4], x[5], x[6], x[7]);
    pdft4<INV, true>(x[8], x[9], x[10], x[11]);
    pdft4<INV, false>(x[12], x[13], x[14], x[15]);
    // x[4 q1 + q2] holds X[q1 + 4 q2]
    Pk t[16];
#pragma unroll
    for(int q1 = 0; q1 < 4; ++q1)
#pragma unroll
        for(int q2 = 0; q2 < 4; ++q2) t[q1 + 4 * q2] = x[4 * q1 + q2];
#pragma unroll
    for(int i = 0; i < 16; ++i) x[i] = t[i];
}

// 8-point DFT of each lane, natural order in and out
template <bool INV>
__device__ __forceinline__ void pdft8(Pk* x)
{
#pragma unroll
    for(int r = 0; r < 4; ++r) {
        const Pk a = x[r], b = x[4 + r];
        x[r]     = {padd(a.re, b.re), padd(a.im, b.im)};
        x[4 + r] = {psub(a.re, b.re), psub(a.im, b.im)};
    }
    const float c2 = 0.70710678118654752440f;
    const uint64_t C = pk2(c2, c2), NC = pk2(-c2, -c2);
    {  // x[5] *= W_8, x[7] *= W_8^3; W_8^2 = -i of x[6] is left to pdft4
        Pk &a = x[5], &b = x[7];
        const uint64_t s5 = padd(a.re, a.im), d5 = INV ? psub(a.re, a.im) : psub(a.im, a.re);
        a = INV ? Pk{pmul(d5, C), pmul(s5, C)} : Pk{pmul(s5, C), pmul(d5, C)};
        const uint64_t s7 = padd(b.re, b.im), d7 = INV ? psub(b.re, b.im) : psub(b.im, b.re);
        b = INV ? Pk{pmul(s7, NC), pmul(d7, C)} : Pk{pmul(d7, C), pmul(s7, NC)};
    }
    pdft4<INV, false>(x[0], x[1], x[2], x[3]);
    pdft4<INV, true>(x[4], x[5], x[6], x[7]);
    // x[q2] = X[2 q2], x[4 + q2] = X[2 q2 + 1]
    Pk t[8];
#pragma unroll
    for(int q = 0; q < 4; ++q) {
        t[2 * q]     = x[q];
        t[2 * q + 1] = x[4 + q];
    }
#pragma unroll
    for(int i = 0; i < 8; ++i) x[i] = t[i];
}

template <int R, bool INV>
__device__ __forceinline__ void pdft(Pk* x)
{
    if constexpr(R == 16) {
        pdft16<INV>(x);
    } else if constexpr(R == 8) {
        pdft8<INV>(x);
    } else if constexpr(R == 4) {
        pdft4<INV, false>(x[0], x[1], x[2], x[3]);
    } else {
        const Pk a = x[0], b = x[1];
        x[0] = {padd(a.re, b.re), padd(a.im, b.im)};
        x[1] = {psub(a.re, b.re), psub(a.im, b.im)};
    }
}

// cos and sin of pi k / 16, rounded once by the compiler
__device__ __forceinline__ float cos32(int k)
{
    constexpr float c[17] = {1.0f, 0.98078528040323044913f, 0.92387953251128675613f,
                             0.83146961230254523708f, 0.70710678118654752440f,
                             0.55557023301960222474f, 0.38268343236508977173f,
                             0.19509032201612826785f, 0.0f, -0.19509032201612826785f,
                             -0.38268343236508977173f, -0.55557023301960222474f,
                             -0.70710678118654752440f, -0.83146961230254523708f,
                             -0.92387953251128675613f, -0.98078528040323044913f, -1.0f};
    return c[k];
}
__device__ __forceinline__ float sin32(int k) { return k <= 8 ? cos32(8 - k) : cos32(k - 8); }

// Pass 2 on a thread's 16 pairs: 32 / R2 transforms of R2 points.  In, pair m
// of a transform = points (2 m, 2 m + 1); out, pair k = bins (k, k + R2 / 2).
// Inverse: the other way round.
template <int R2>
__device__ __forceinline__ void pass2_fwd(Pk* x)
{
    constexpr int H = R2 / 2;
#pragma unroll
    for(int b = 0; b < 16; b += H) pdft<H, false>(x + b);
#pragma unroll
    for(int i = 0; i < 16; ++i) {
        const int k = (i % H) * (32 / R2);  // W_R2^(i % H) = W_32^k
        float er, orr, ei, oi;
        unpk2(x[i].re, er, orr);
        unpk2(x[i].im, ei, oi);
        const float c = cos32(k), s = sin32(k);  // W_32^k = c - i s
        const float pr = k == 0 ? orr : k == 8 ? oi : orr * c + oi * s;
        const float pi = k == 0 ? oi : k == 8 ? -orr : oi * c - orr * s;
        x[i] = {pk2(er + pr, er - pr), pk2(ei + pi, ei - pi)};
    }
}
template <int R2>
__device__ __forceinline__ void pass2_inv(Pk* x)
{
    constexpr int H = R2 / 2;
#pragma unroll
    for(int i = 0; i < 16; ++i) {
        const int k = (i % H) * (32 / R2);
        float ar, br, ai, bi;
        unpk2(x[i].re, ar, br);
        unpk2(x[i].im, ai, bi);
        const float dr = ar - br, di = ai - bi;
        const float c = cos32(k), s = sin32(k);  // W_32^-k = c + i s
        const float pr = k == 0 ? dr : k == 8 ? -di : dr * c - di * s;
        const float pi = k == 0 ? di : k == 8 ? dr : di * c + dr * s;
        x[i] = {pk2(ar + br, pr), pk2(ai + bi, pi)};
    }
#pragma unroll
    for(int b = 0; b < 16; b += H) pdft<H, true>(x + b);
}

// ---------------------------------------------------------- tensor memory
__device__ __forceinline__ void tm_ld16(uint32_t addr, uint32_t* r)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                   "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
                   "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(addr));
}
// Waits for this thread's loads; the registers pass through so that no use of
// them can be moved above the wait.
__device__ __forceinline__ void tm_wait_ld16(uint32_t* r)
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]),
                   "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                   "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :
                 : "memory");
}
__device__ __forceinline__ void tm_st16(uint32_t addr, const uint32_t* r)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
                 "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(addr),
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
                 "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
                 "r"(r[14]), "r"(r[15])
                 : "memory");
}
__device__ __forceinline__ void tm_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// x[q] *= w_q (conjugated for the inverse), q = 1 .. 15, w from tensor memory;
// the caller has started the load of the first 16 registers into w[0], as long
// before as its registers allow
template <bool INV>
__device__ __forceinline__ void ptwiddle(Pk* x, uint32_t tw, uint32_t (*w)[16])
{
#pragma unroll
    for(int c = 0; c < 4; ++c) {
        uint32_t* v = w[c & 1];
        tm_wait_ld16(v);
        if(c < 3) tm_ld16(tw + 16 * (c + 1), w[(c + 1) & 1]);
#pragma unroll
        for(int i = 0; i < 4; ++i) {
            const int q = 4 * c + i + 1;
            if(q < 16)
                x[q] = pcmul<INV>(x[q], Pk{pk2u(v[4 * i], v[4 * i + 1]),
                                           pk2u(v[4 * i + 2], v[4 * i + 3])});
        }
    }
}

// A window group's place: thread number, its first quad of each pass in shared
// memory and its columns of tensor memory (lane quarter included).
struct PkGroup {
    int t;            // thread of the group, 0 .. N / 32 - 1
    int window;       // window of the CTA
    uint8_t *p0, *p1, *p2;
    uint32_t tm_spec, tm_tw0, tm_tw1;
};

// Barrier of one window's threads (named barriers 1 .. W; a warp for N = 1024).
// bar.sync and the tensor memory instructions need a converged warp, and the
// stores and copies before them leave lanes on different sides of their bounds:
// __syncwarp joins them wherever such code ends.
template <int LOGN>
__device__ __forceinline__ void pk_sync(const PkGroup& g)
{
    constexpr int T = PkGeo<LOGN>::T;
    __syncwarp();
    if constexpr(T > 32) asm volatile("bar.sync %0, %1;" ::"r"(1 + g.window), "n"(T) : "memory");
}

__device__ __forceinline__ Pk pk_load(const uint8_t* p)
{
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
    return {v.x, v.y};
}
__device__ __forceinline__ void pk_store(uint8_t* p, const Pk& x)
{
    *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(x.re, x.im);
}

// Twiddles of thread t to tensor memory, Q quads in flight at a time.
template <int LOGN, int Q>
__device__ __forceinline__ void pk_fill(const float4* t0, int t, uint32_t tm)
{
    using G = PkGeo<LOGN>;
#pragma unroll 1
    for(int c = 0; c < 32; c += Q) {
        float4 w[Q];
#pragma unroll
        for(int i = 0; i < Q; ++i) {
            const int q = (c & 15) + i;
            w[i] = q >= 15  ? make_float4(0.0f, 0.0f, 0.0f, 0.0f)
                   : c < 16 ? t0[q * G::T + t]
                            : t0[G::TW0 + q * (G::R2 / 2) + t % (G::R2 / 2)];
        }
#pragma unroll
        for(int i = 0; i < Q; i += 4) {
            uint32_t v[16];
#pragma unroll
            for(int k = 0; k < 4; ++k) {
                v[4 * k]     = __float_as_uint(w[i + k].x);
                v[4 * k + 1] = __float_as_uint(w[i + k].y);
                v[4 * k + 2] = __float_as_uint(w[i + k].z);
                v[4 * k + 3] = __float_as_uint(w[i + k].w);
            }
            tm_st16(tm + (c < 16 ? 0 : 128 - 64) + 4 * (c + i), v);
        }
    }
    tm_wait_st();
}
// All of a pass in flight (72 windows of 1024 points: 7.8 us, 4 at a time 9.0),
// out of line so that its registers are the set-up's alone: inline the transforms
// spill (2-4 % slower at 8192 points).  The split kernel spills around the call
// (5 % slower), and fills 4 at a time.
template <int LOGN>
__device__ __noinline__ void pk_fill_fast(const float4* t0, int t, uint32_t tm)
{
    pk_fill<LOGN, 16>(t0, t, tm);
}

// Tensor memory of one CTA: 512 columns = spectra of the 4 warps that share a
// lane quarter (64 columns each), then the pass 0 and pass 1 twiddles of the
// (at most two) warps of a window that share it, common to all windows.
// Called by all threads; the first window's threads (the first four warps
// where a window is shorter) fill the twiddles.  Returns the base for
// pk_tmem_free.
template <int LOGN, bool FAST>
__device__ __forceinline__ uint32_t pk_setup(PkGroup& g, uint8_t* bufs, uint32_t* s_tmem,
                                             const float* tw)
{
    using G = PkGeo<LOGN>;
    const int warp = threadIdx.x >> 5;
    if(warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
            static_cast<uint32_t>(__cvta_generic_to_shared(s_tmem))));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t base = *s_tmem;
    const uint32_t mine = base + ((uint32_t)(32 * (warp & 3)) << 16);
    g.window = threadIdx.x / G::T;
    g.t      = threadIdx.x - g.window * G::T;
    // the window's rows follow those of the windows before: row = CTA thread
    uint8_t* buf = bufs + g.window * G::T * kPkRow * 8;
    const int b = 2 * g.t, i1 = b / G::R2 * 16 * G::R2 + b % G::R2;  // pass 1's first point
    g.p0 = buf + (b / 32 * kPkRow + b % 32) * 8;
    g.p1 = buf + (i1 / 32 * kPkRow + i1 % 32) * 8;
    g.p2 = buf + g.t * kPkRow * 8;
    g.tm_spec = mine + 64 * (warp >> 2);
    g.tm_tw0  = mine + 256 + (G::T > 128 ? 64 * ((warp >> 2) & 1) : 0);
    g.tm_tw1  = g.tm_tw0 + 128;
    if(threadIdx.x < (G::T > 128 ? G::T : 128)) {  // whole warps
        const float4* quads = reinterpret_cast<const float4*>(tw);
        if constexpr(FAST) pk_fill_fast<LOGN>(quads, g.t, g.tm_tw0);
        else pk_fill<LOGN, 4>(quads, g.t, g.tm_tw0);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return base;
}

__device__ __forceinline__ void pk_tmem_free(uint32_t base)
{
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if(threadIdx.x < 32) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(base));
    }
}

// Forward transform of x (pass 0's pairs: points 2 t + (N / 16) r and the
// next); the spectrum goes to tensor memory.  `after_p0` runs once the group's
// threads have all passed their pass 0 (the staged input is free then).
template <int LOGN, typename F>
__device__ __forceinline__ void pk_forward(const PkGroup& g, Pk* x, F after_p0)
{
    using G = PkGeo<LOGN>;
    uint32_t w[2][16];
    tm_ld16(g.tm_tw0, w[0]);
    pdft16<false>(x);
    ptwiddle<false>(x, g.tm_tw0, w);
#pragma unroll
    for(int q = 0; q < 16; ++q) pk_store(g.p0 + q * G::STEP0, x[q]);
    pk_sync<LOGN>(g);
    after_p0();
    __syncwarp();
    tm_ld16(g.tm_tw1, w[0]);
#pragma unroll
    for(int q = 0; q < 16; ++q) x[q] = pk_load(g.p1 + G::off1(q));
    pdft16<false>(x);
    ptwiddle<false>(x, g.tm_tw1, w);
#pragma unroll
    for(int q = 0; q < 16; ++q) pk_store(g.p1 + G::off1(q), x[q]);
    __syncwarp();
#pragma unroll
    for(int q = 0; q < 16; ++q) x[q] = pk_load(g.p2 + 16 * q);
    pass2_fwd<G::R2>(x);
#pragma unroll
    for(int c = 0; c < 4; ++c) {
        uint32_t v[16];
#pragma unroll
        for(int i = 0; i < 4; ++i) {
            unpk2u(x[4 * c + i].re, v[4 * i], v[4 * i + 1]);
            unpk2u(x[4 * c + i].im, v[4 * i + 2], v[4 * i + 3]);
        }
        tm_st16(g.tm_spec + 16 * c, v);
    }
    tm_wait_st();
}

// Inverse transform of spectrum x chirp; x ends as pass 0's pairs.  chirp:
// this thread's column of the [16][N / 32] quads of one channel and DM.  The
// caller puts a pk_sync between this and the next pass 0 or pass 2 store.
template <int LOGN>
__device__ __forceinline__ void pk_inverse(const PkGroup& g, const float4* chirp, Pk* x)
{
    using G = PkGeo<LOGN>;
    // all 16 chirp quads in flight at once, in the registers that become x
#pragma unroll
    for(int k = 0; k < 16; ++k) {
        const float4 c = chirp[k * G::T];
        x[k] = {pk2(c.x, c.y), pk2(c.z, c.w)};
    }
    uint32_t w[2][16];
    tm_ld16(g.tm_spec, w[0]);
#pragma unroll
    for(int c = 0; c < 4; ++c) {
        uint32_t* v = w[c & 1];
        tm_wait_ld16(v);
        if(c < 3) tm_ld16(g.tm_spec + 16 * (c + 1), w[(c + 1) & 1]);
#pragma unroll
        for(int i = 0; i < 4; ++i)
            x[4 * c + i] = pcmul<false>(x[4 * c + i], Pk{pk2u(v[4 * i], v[4 * i + 1]),
                                                         pk2u(v[4 * i + 2], v[4 * i + 3])});
    }
    pass2_inv<G::R2>(x);
    tm_ld16(g.tm_tw1, w[0]);
#pragma unroll
    for(int q = 0; q < 16; ++q) pk_store(g.p2 + 16 * q, x[q]);
    __syncwarp();
#pragma unroll
    for(int q = 0; q < 16; ++q) x[q] = pk_load(g.p1 + G::off1(q));
    ptwiddle<true>(x, g.tm_tw1, w);
    pdft16<true>(x);
    tm_ld16(g.tm_tw0, w[0]);
#pragma unroll
    for(int q = 0; q < 16; ++q) pk_store(g.p1 + G::off1(q), x[q]);
    pk_sync<LOGN>(g);
#pragma unroll
    for(int q = 0; q < 16; ++q) x[q] = pk_load(g.p0 + q * G::STEP0);
    ptwiddle<true>(x, g.tm_tw0, w);
    pdft16<true>(x);
}

}  // namespace cdd
}  // namespace swb
