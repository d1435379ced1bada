// Resampling FFT kernels: one transform per CTA at a time, the whole transform
// resident in shared memory, persistent grids (one CTA per SM looping over
// transforms, twiddle tables loaded into shared memory once per CTA).
//
// Reference: the three cuFFT plans of vdif_inout_gpu_thread.cu:271-333 run by
// SwarmC2R / SwarmR2C / R2dbeC2R (:589-709) on each 143-snapshot batch.
//   stage A  C2R 32768 per snapshot  = 16384-point complex inverse FFT plus
//            Hermitian pre-processing, fed straight from the packed 2-bit
//            spectrum (beng_int8_to_cufftComplex and the Nyquist memset fused);
//            the spectra of the next two snapshots are bulk-copied ahead.
//   stage BC R2C 36608 per chunk = 18304-point complex FFT + post-processing,
//            bins [skip, skip+16384] selected in registers, C2R 32768 through
//            a 16384-point inverse FFT, then quantize2bit in the epilogue.
// All scaling is cuFFT's unnormalised convention.
#include <cmath>
#include <vector>

#include "fft_core.cuh"
#include "launchers.cuh"
#include "sdbe_internal.cuh"
#include "tcgen05.cuh"

namespace sdbe {

constexpr int kNTA = 512;   // stage A threads: 512 radix-32 butterflies per pass
constexpr int kNTB = 512;   // stage BC threads: 4 warps per SM sub-partition -> 128 registers
// The 18304-point data (stage BC) is padded one float2 per 16, so that the
// first pass's digit-reversed stores, 16 lanes at a time, land in 16
// distinct bank pairs (see fft18304_from_global); the 16384-point transforms
// keep one per 32 (their layouts are built on it).
__host__ __device__ constexpr int padb(int a) { return a + (a >> 4); }
// One of the 16 sub-transforms of the inverse 16384: 32 rows of 33 slots, and
// one more so that 16 consecutive columns' stores land in 16 bank pairs.
constexpr int kSub = 1057;
constexpr int kPadB = padb(kMB) + 1;

// Shared-memory twiddle tables (float2).  The per-pass tables are laid out
// [r][k] so that the 16 lanes of a half-warp, which hold consecutive k, read
// consecutive words; the two-level tables are padded with tp().
constexpr int kT32 = 10 * 32;          // W_1024^{j s}, s = 1..7, then W_1024^{8 j a}, a = 1..3 (16384-point pass 2)
constexpr int kT128 = tp_len(128);     // two-level halves
constexpr int kT13 = 12 * 16;          // W_208^{k r}, r = 1..12, k = 0..15   (18304-point radix-13 pass)
constexpr int kH18304 = tp_len(143);   // W_18304^{128 a}
constexpr int kTwA = kT32 + 2 * kT128;               // stage A tables
constexpr int kTwB = kTwA + kT13 + kH18304 + kT128;  // stage BC tables
constexpr size_t kSmemA = 2 * kGroups * sizeof(uint32_t) + (24 * kSub + kTwA) * sizeof(float2);
constexpr size_t kSmemB = (kPadB + kTwB) * sizeof(float2);
// The standalone R2C and C2R kernels fit the 164 KB shared-memory carveout.
// Above it k_swarm_r2c's plain loads, as stage BC's did, have too little L1 for
// their lines in flight (9% of stage BC at the 228 KB carveout).
static_assert(kSmemB + 512 + 1024 <= 164 * 1024, "standalone kernels' shared memory above the 164 KB carveout");

// ---- table loading --------------------------------------------------------
struct TabsA {  // inverse-16384 tables
    float2 *t32, *h16384, *l16384;
};
struct TabsB {  // forward-18304 tables in shared memory; W_36608^q in global memory
    float2 *t13, *h18304, *l18304;
    const float2 *w36608;
};

__device__ __forceinline__ TabsA tabs_a_at(float2 *p) {
    return TabsA{p, p + kT32, p + kT32 + kT128};
}

// For a launch of an item or two per CTA, whose tables are a visible part of
// it: their entries numbered through and dealt out evenly to the 512 threads,
// every thread's loads issued before its first store.  One trip to L2 (about
// 1.5k cycles) instead of one per table in the low warps (5.5k).  The packing
// stage BC keeps the loops below: it measured 0.8% slower per chunk with this,
// from registers given out differently.
constexpr int kEntA = kT32 + 256, kEntB = kT13 + 143 + 128;
struct TabEntry {
    const float2 *src;
    float2 *dst;
};
__device__ __forceinline__ TabEntry tab_entry_a(const TabsA &t, const Twiddles &tw, int m) {
    if (m < kT32) {
        const int j = m & 31, g = m >> 5;                       // g < 7: s = g + 1; else a = g - 6
        const int e = g < 7 ? j * (g + 1) : 8 * j * (g - 6);   // exponent of W_1024
        return {tw.w16384 + 16 * e, t.t32 + m};
    }
    const int q = (m - kT32) & 127;
    return m < kT32 + 128 ? TabEntry{tw.w16384 + 128 * q, t.h16384 + tp(q)} : TabEntry{tw.w16384 + q, t.l16384 + tp(q)};
}
__device__ __forceinline__ TabEntry tab_entry_b(const TabsB &t, const Twiddles &tw, int m) {
    if (m < kT13) {
        const int r = (m >> 4) + 1, k = m & 15;
        return {tw.w18304 + 88 * k * r, t.t13 + m};
    }
    const int q = m - kT13;
    return q < 143 ? TabEntry{tw.w18304 + 128 * q, t.h18304 + tp(q)} : TabEntry{tw.w18304 + q - 143, t.l18304 + tp(q - 143)};
}
template <int N, class F>
__device__ __forceinline__ void load_tabs(F entry) {
    constexpr int R = (N + 511) / 512;
    TabEntry e[R];
    float2 v[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int m = threadIdx.x + 512 * i;
        if (m < N) {
            e[i] = entry(m);
            v[i] = __ldg(e[i].src);
        }
    }
#pragma unroll
    for (int i = 0; i < R; ++i)
        if (static_cast<int>(threadIdx.x) + 512 * i < N) *e[i].dst = v[i];
}
__device__ __forceinline__ void load_tabs_ab(const TabsA &ta, const TabsB &tb, const Twiddles &tw) {
    load_tabs<kEntA + kEntB>([&](int m) { return m < kEntA ? tab_entry_a(ta, tw, m) : tab_entry_b(tb, tw, m - kEntA); });
}
__device__ __forceinline__ void load_tabs_a(TabsA t, const Twiddles &tw) {
    for (int m = threadIdx.x; m < kT32; m += blockDim.x) {
        const int j = m & 31, g = m >> 5;                       // g < 7: s = g + 1; else a = g - 6
        const int e = g < 7 ? j * (g + 1) : 8 * j * (g - 6);   // exponent of W_1024
        t.t32[m] = __ldg(tw.w16384 + 16 * e);
    }
    for (int m = threadIdx.x; m < 128; m += blockDim.x) {
        t.h16384[tp(m)] = __ldg(tw.w16384 + 128 * m);
        t.l16384[tp(m)] = __ldg(tw.w16384 + m);
    }
}

__device__ __forceinline__ void load_tabs_b(TabsB t, const Twiddles &tw) {
    for (int m = threadIdx.x; m < kT13; m += blockDim.x) {
        const int r = (m >> 4) + 1, k = m & 15;
        t.t13[m] = __ldg(tw.w18304 + 88 * k * r);
    }
    for (int m = threadIdx.x; m < 143; m += blockDim.x) t.h18304[tp(m)] = __ldg(tw.w18304 + 128 * m);
    for (int m = threadIdx.x; m < 128; m += blockDim.x) t.l18304[tp(m)] = __ldg(tw.w18304 + m);
}

__device__ __forceinline__ TabsB tabs_b_at(float2 *tb, const Twiddles &tw) {
    float2 *p = tb + kTwA;
    return TabsB{p, p + kT13, p + kT13 + kH18304, tw.w36608};
}

// First-pass lane order of the 18304-point transform: half-warp h takes the
// groups of 8 consecutive inputs g0 = kFirstPassGroups[2h], g1 = [2h+1]
// (inputs j = 8g + c, c = 0..7; 255 = none).  Output slot 16*rho(j) + r has
// rho(8g + c) = rho(8g) - c (mod 16); the pairs are chosen with rho(8 g1) =
// rho(8 g0) + 8 (mod 16), so the 16 lanes' padded slots cover all 16 bank
// pairs and every store is one wavefront.
__constant__ uint8_t kFirstPassGroups[144] = {
    0,   8,   28,  14,  34,  42,  62,  48,  68,  76,  96,  82,  102, 88,  130, 116, 136, 122, 5,   19,  11,  25,
    39,  53,  45,  59,  73,  87,  79,  93,  107, 99,  113, 127, 141, 133, 10,  2,   16,  30,  22,  36,  50,  64,
    56,  70,  84,  98,  90,  104, 118, 110, 124, 138, 21,  7,   27,  13,  33,  41,  61,  47,  67,  75,  95,  81,
    101, 109, 129, 115, 135, 121, 4,   18,  32,  24,  38,  52,  44,  58,  72,  86,  78,  92,  106, 120, 112, 126,
    140, 132, 9,   1,   15,  29,  43,  35,  49,  63,  55,  69,  83,  97,  89,  103, 117, 131, 123, 137, 20,  6,
    26,  12,  54,  40,  60,  46,  66,  74,  94,  80,  100, 108, 128, 114, 134, 142, 3,   17,  31,  23,  37,  51,
    65,  57,  71,  85,  77,  91,  105, 119, 111, 125, 139, 255};

// ---------------------------------------------------------------------------
// Inverse 16384-point FFT, radices 32 x 32 x 16 (Stockham).  zin(v) gives
// input elements col + 512 r, r < 32, of this thread's first-pass column
// `col` (a permutation of the thread index); epi(jj, u) receives outputs
// z[jj + 1024 r], r < 16.  blockDim.x is 512.
// The last pass's per-thread twiddle bases W_16384^(tid s), s = 1..3, and
// W_16384^(4 tid a), a = 1..3: they depend on the thread only, so a
// persistent kernel can form them once.
struct LastTw {
    float2 S0[4], A0[4];
};
__device__ __forceinline__ LastTw last_tw(const TabsA &T) {
    LastTw t;
    const int tid = threadIdx.x;
#pragma unroll
    for (int s = 1; s < 4; ++s) t.S0[s] = tw2(T.h16384, T.l16384, tid * s);
#pragma unroll
    for (int a = 1; a < 4; ++a) t.A0[a] = tw2(T.h16384, T.l16384, tid * 4 * a);
    return t;
}

// The transform is 16 transforms of 1024 points (first-pass columns col = w
// mod 16, radices 32 x 32), each in its own kSub slots of `sm`, and a last
// radix-16 pass across them.  Column w + 16 i leaves its 32 outputs in row i
// of sub-transform w; the second pass, one warp per sub-transform, reads
// column l of those rows (lane l) and writes its outputs to the very slots it
// read, so no barrier separates its loads from its stores, and a warp that
// takes its own sub-transform's columns needs no block barrier between the
// first two passes at all.

// First pass: the DFT-32 outputs v of column `col`, its sub-transform's slots at `slots`.
__device__ __forceinline__ void inv_store1(float2 *slots, int col, const float2 *v) {
    float2 *dst = slots + 33 * (col >> 4);
#pragma unroll
    for (int r = 0; r < 32; ++r) dst[r] = v[r];
}

// The second pass's twiddles W_1024^{l r} = A[r/8] * S[r%8] of lane l, r = 1..31 (w[0] unused).
__device__ __forceinline__ void pass2_twiddles(const TabsA &T, float2 *w) {
    const float2 *tj = T.t32 + (threadIdx.x & 31);
    float2 S[8], A[4];
#pragma unroll
    for (int s = 1; s < 8; ++s) S[s] = tj[32 * (s - 1)];
#pragma unroll
    for (int a = 1; a < 4; ++a) A[a] = tj[32 * (6 + a)];
    w[0] = make_float2(1.f, 0.f);
#pragma unroll
    for (int r = 1; r < 32; ++r) {
        const int a = r >> 3, s = r & 7;
        w[r] = a == 0 ? S[s] : (s == 0 ? A[a] : cmul(A[a], S[s]));
    }
}

// Second pass of the sub-transform at `slots`, in place; apply(v) multiplies
// v[r] by conj W_1024^{l r}.
template <class Apply>
__device__ __forceinline__ void inv_pass2(float2 *slots, Apply apply) {
    float2 v[32];
    float2 *p = slots + (threadIdx.x & 31);
#pragma unroll
    for (int r = 0; r < 32; ++r) v[r] = p[33 * r];
    apply(v);
    dft<32, true>(v);
#pragma unroll
    for (int r = 0; r < 32; ++r) p[33 * r] = v[r];
}

// Last pass: jj = tid + 512 i, i = 0, 1; W_16384^(jj s) = W^(tid s) W^(512 i s).
// at(r) is where sub-transform r's slots begin (r a compile-time index);
// read_done() runs after this thread's last loads.
// ROLL: a loop, its factors from constant memory (1 for i = 0) with the same
// rounding.  A CTA's first item runs at half speed while its straight-line code
// (100 KB of stage BC) comes from L2: with this and the R2C pass rolled and the
// tables loaded at once, a first batch takes 82 us for 90.  The loop itself
// costs 0.6% per chunk (17.14 for 17.02 us) once the code is there, and 3.5% in
// stage A, so the kernels for many items don't take it.
#define SDBE_W(N, E) {TwC<N, E>::c, TwC<N, E>::s}
__constant__ float2 kLastStep[2][6] = {{{1.f, 0.f}, {1.f, 0.f}, {1.f, 0.f}, {1.f, 0.f}, {1.f, 0.f}, {1.f, 0.f}},
                                       {SDBE_W(kMA, 512), SDBE_W(kMA, 1024), SDBE_W(kMA, 1536), SDBE_W(kMA, 2048),
                                        SDBE_W(kMA, 4096), SDBE_W(kMA, 6144)}};
template <bool ROLL, class At, class Epi, class Done>
__device__ __forceinline__ void inv_pass3(At at, const LastTw &lt, Epi epi, Done read_done) {
    const int tid = threadIdx.x;
    const float2 *S0 = lt.S0, *A0 = lt.A0;
    auto half = [&](int i, auto cst) {
        const int jj = tid + 512 * i;
        float2 u[16];
        const int o = pad(jj);
#pragma unroll
        for (int r = 0; r < 16; ++r) u[r] = at(r)[o];
        if (i == 1) read_done();
        // W_16384^{jj r} = A[r/4] * S[r%4]
        float2 S[4], A[4];
        if constexpr (decltype(cst)::value) {
            S[1] = i ? mul_tc<kMA, 512, false>(S0[1]) : S0[1];
            S[2] = i ? mul_tc<kMA, 1024, false>(S0[2]) : S0[2];
            S[3] = i ? mul_tc<kMA, 1536, false>(S0[3]) : S0[3];
            A[1] = i ? mul_tc<kMA, 2048, false>(A0[1]) : A0[1];
            A[2] = i ? mul_tc<kMA, 4096, false>(A0[2]) : A0[2];
            A[3] = i ? mul_tc<kMA, 6144, false>(A0[3]) : A0[3];
        } else {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                S[k + 1] = cmul_rn<0, 1>(S0[k + 1], kLastStep[i][k]);
                A[k + 1] = cmul_rn<0, 0>(A0[k + 1], kLastStep[i][3 + k]);
            }
        }
#pragma unroll
        for (int r = 1; r < 16; ++r) {
            const int a = r >> 2, s = r & 3;
            const float2 w = a == 0 ? S[s] : (s == 0 ? A[a] : cmul(A[a], S[s]));
            u[r] = cmulc(u[r], w);
        }
        dft<16, true>(u);
        epi(jj, u);
    };
    if constexpr (ROLL) {
#pragma unroll 1
        for (int i = 0; i < 2; ++i) half(i, std::false_type{});
    } else {
        half(0, std::true_type{});
        half(1, std::true_type{});
    }
}

template <int... R, class F>
__device__ __forceinline__ void for_r(std::integer_sequence<int, R...>, F f) {
    (f(std::integral_constant<int, R>{}), ...);
}

// Radix 13, Ns = 16: twiddles W_208^{k r}, k = 0..15, the same for every
// butterfly of a thread that keeps its k; butterfly k of block b (208 slots).
__device__ __forceinline__ void pass13_twiddles(const TabsB &T, int k, float2 *w13) {
#pragma unroll
    for (int r = 1; r < 13; ++r) w13[r] = T.t13[16 * (r - 1) + k];
}
__device__ __forceinline__ void fwd_pass13(float2 *sm, const float2 *w13, int b, int k) {
    float2 *p = sm + padb(b * 208 + k);  // padb(base + 16 r) = padb(base) + 17 r
    float2 v[13];
#pragma unroll
    for (int r = 0; r < 13; ++r) v[r] = p[17 * r];
#pragma unroll
    for (int r = 1; r < 13; ++r) v[r] = cmul(v[r], w13[r]);
    dft<13, false>(v);
#pragma unroll
    for (int r = 0; r < 13; ++r) p[17 * r] = v[r];
}

// Radix 11, Ns = 208: twiddles W_2288^{k r}.  Butterfly (m, k) is at base
// 2288 m + k, m < 8, k < 208; thread t takes k = t % 208 and m = t / 208
// + j nk, nk = the threads sharing its k, so its ten twiddles are formed
// once per transform, from the two-level W_18304 tables (at most 4
// butterflies a thread, as with b = t + 512 j).
__device__ __forceinline__ void fwd_pass11(float2 *sm, const TabsB &T) {
    static_assert(kNTB == 512, "512 threads share 208 x 8 butterflies");
    const int t = threadIdx.x, k = t % 208, nk = k < 512 - 2 * 208 ? 3 : 2;
    float2 w11[11];
#pragma unroll
    for (int r = 1; r < 11; ++r) w11[r] = tw2(T.h18304, T.l18304, 8 * k * r);  // W_2288^(k r), 8 k r < 18304
    for (int m = t / 208; m < 8; m += nk) {
        float2 *p = sm + padb(2288 * m + k);  // padb(base + 208 r) = padb(base) + 221 r
        float2 v[11];
#pragma unroll
        for (int r = 0; r < 11; ++r) v[r] = p[221 * r];
#pragma unroll
        for (int r = 1; r < 11; ++r) v[r] = cmul(v[r], w11[r]);
        dft<11, false>(v);
#pragma unroll
        for (int r = 0; r < 11; ++r) p[221 * r] = v[r];
    }
}

// Radix 8, Ns = 2288, the last pass: twiddles W_18304^{k r}.  With R2C it also applies the R2C pairing, leaving X[q] (q <= 18304,
// X[18304] in the spare slot padb(18304)) instead of Z.  Its butterfly k
// holds Z[k + 2288 r] and butterfly 2288 - k holds their mirrors Z[18304 - q]
// at r' = 7 - r, so one thread takes both (k = 0 and k = 1144 are their own
// mirrors) and pairs in registers: one pass and one barrier fewer.
//
// W_36608^(u + 2288 r) = wu W_16^r with its rounding pinned (MID: the unit u = 1144).
template <int R, bool MID = false>
__device__ __forceinline__ float2 r2c_tw(float2 wu) {
    if constexpr (R == 0) return wu;
    constexpr int X = MID ? (R == 3 ? 1 : 0) : (R >= 5 ? 2 : 0), Y = MID ? (R == 3 ? 0 : 1) : (R >= 5 ? 2 : 1);
    return cmul_rn<X, Y>(wu, make_float2(TwC<16, R>::c, TwC<16, R>::s));
}
// ROLL: units in a loop (see inv_pass3); kUnitStep: W_18304^(512 i q), q = 1..4, and W_36608^(512 i).
__constant__ float2 kUnitStep[3][5] = {
    {{1.f, 0.f}, {1.f, 0.f}, {1.f, 0.f}, {1.f, 0.f}, {1.f, 0.f}},
    {SDBE_W(kMB, 512), SDBE_W(kMB, 1024), SDBE_W(kMB, 1536), SDBE_W(kMB, 2048), SDBE_W(kNB, 512)},
    {SDBE_W(kMB, 1024), SDBE_W(kMB, 2048), SDBE_W(kMB, 3072), SDBE_W(kMB, 4096), SDBE_W(kNB, 1024)}};
template <bool R2C, bool ROLL = false>
__device__ __forceinline__ void fwd_pass8(float2 *sm, const TabsB &T) {
    // twiddles W_18304^{k r} = A[r/4] * S[r%4]
    // butterfly k with its twiddles S[q] = W^(k q), q = 1..3, and A1 = W^(4 k)
    auto bfly8w = [&](int k, float2 *v, const float2 *S, float2 A1) {
        const float2 *p = sm + padb(k);  // padb(k + 2288 r) = padb(k) + 2431 r
#pragma unroll
        for (int r = 0; r < 8; ++r) v[r] = p[2431 * r];
#pragma unroll
        for (int r = 1; r < 8; ++r) {
            const float2 w = r < 4 ? S[r] : (r == 4 ? A1 : cmul(A1, S[r - 4]));
            v[r] = cmul(v[r], w);
        }
        dft<8, false>(v);
    };
    auto bfly8 = [&](int k, float2 *v) {
        float2 S[4];
#pragma unroll
        for (int q = 1; q < 4; ++q) S[q] = tw2(T.h18304, T.l18304, k * q);
        bfly8w(k, v, S, tw2(T.h18304, T.l18304, 4 * k));
    };
    if constexpr (!R2C) {
        for (int k = threadIdx.x; k < kMB / 8; k += blockDim.x) {
            float2 v[8];
            bfly8(k, v);
            float2 *p = sm + padb(k);
#pragma unroll
            for (int r = 0; r < 8; ++r) p[2431 * r] = v[r];
        }
    } else {
        constexpr int K = kMB / 8;  // 2288
        // Units u = tid + 512 i (i < 3, u <= 1144).  Twiddles from per-thread
        // bases and compile-time factors: W_18304^(u q) = W^(tid q) W^(512 i q);
        // the mirror butterfly's W^((2288 - u) q) = W^(2288 q) conj(W^(u q));
        // W_36608^(u + 2288 r) = W_36608^u W_16^r.
        static_assert(kNTB == 512, "units u = tid + 512 i");
        const int tid = threadIdx.x;
        float2 B[5];
#pragma unroll
        for (int q = 1; q <= 4; ++q) B[q] = tw2(T.h18304, T.l18304, tid * q);
        const float2 wt = __ldg(T.w36608 + tid);  // W_36608^tid
        auto unit = [&](int u, const float2 (&S)[4], float2 A1, auto wu_at) {
            float2 a[8];
            bfly8w(u, a, S, A1);
            float2 *pa = sm + padb(u);
            const float2 wu = wu_at();
            if (u == 0) {  // q = 2288 r pairs with 2288 (8 - r); X[0], X[18304] from Z[0]
                pa[0] = make_float2(a[0].x + a[0].y, 0.f);
                sm[padb(kMB)] = make_float2(a[0].x - a[0].y, 0.f);
                for_r(std::integer_sequence<int, 1, 2, 3, 4>{}, [&](auto rc) {
                    constexpr int r = decltype(rc)::value;
                    float2 xq, xmq;
                    r2c_pair(a[r], a[8 - r], mul_tc<16, r, false>(make_float2(1.f, 0.f)), xq, xmq);
                    pa[2431 * r] = xq;
                    if (r != 4) pa[2431 * (8 - r)] = xmq;
                });
            } else if (u == K / 2) {  // q = 1144 + 2288 r pairs with r' = 7 - r
                for_r(std::make_integer_sequence<int, 4>{}, [&](auto rc) {
                    constexpr int r = decltype(rc)::value;
                    float2 xq, xmq;
                    r2c_pair(a[r], a[7 - r], r2c_tw<r, true>(wu), xq, xmq);
                    pa[2431 * r] = xq;
                    pa[2431 * (7 - r)] = xmq;
                });
            } else {  // butterflies u and 2288 - u
                float2 Sm[4];
                Sm[1] = mul_tc<kMB, K, false>(conjf2(S[1]));
                Sm[2] = mul_tc<kMB, 2 * K, false>(conjf2(S[2]));
                Sm[3] = mul_tc<kMB, 3 * K, false>(conjf2(S[3]));
                float2 b[8];
                bfly8w(K - u, b, Sm, mul_tc<kMB, 4 * K, false>(conjf2(A1)));
                float2 *pb = sm + padb(K - u);
                for_r(std::make_integer_sequence<int, 8>{}, [&](auto rc) {
                    constexpr int r = decltype(rc)::value;
                    float2 xq, xmq;
                    r2c_pair(a[r], b[7 - r], r2c_tw<r>(wu), xq, xmq);
                    pa[2431 * r] = xq;
                    pb[2431 * (7 - r)] = xmq;
                });
            }
        };
        if constexpr (ROLL) {
#pragma unroll 1
            for (int i = 0; i < 3; ++i) {
                const int u = tid + 512 * i;
                if (u > K / 2) break;
                float2 S[4];
#pragma unroll
                for (int q = 1; q < 4; ++q) S[q] = cmul_rn<0, 1>(B[q], kUnitStep[i][q - 1]);
                unit(u, S, cmul_rn<0, 1>(B[4], kUnitStep[i][3]), [&] { return cmul_rn<0, 1>(wt, kUnitStep[i][4]); });
            }
        } else {
            for_r(std::make_integer_sequence<int, 3>{}, [&](auto ic) {
                constexpr int i = decltype(ic)::value;
                const int u = tid + 512 * i;
                if (u > K / 2) return;
                float2 S[4];
                S[1] = mul_tc<kMB, 512 * i, false>(B[1]);
                S[2] = mul_tc<kMB, 1024 * i, false>(B[2]);
                S[3] = mul_tc<kMB, 1536 * i, false>(B[3]);
                unit(u, S, mul_tc<kMB, 2048 * i, false>(B[4]), [&] { return mul_tc<kNB, 512 * i, false>(wt); });
            });
        }
    }
}

// Forward 18304-point FFT of z[m] = x[2m] + i x[2m+1] read from global memory;
// result Z in natural order in `sm` (padded with padb).  In-place decimation
// in time, radices 16 (from global) x 13 x 11 x 8: the first pass reads
// z[j + 1144 r] (8 consecutive j per 8 lanes: 64-B segments) and writes its 16
// outputs to slots 16*rho(j) + r, rho = digit reversal of j over (8, 11, 13);
// every later butterfly reads and writes the same slots g*Ns*R + k + Ns*r
// with twiddles W_{Ns*R}^{k r}, so passes need no staging.  R2C: see fwd_pass8.
template <bool R2C>
__device__ __forceinline__ void fft18304_from_global(float2 *sm, const float2 *__restrict__ z, const TabsB &T) {
    constexpr int NB1 = kMB / 16;  // 1144 = 143 groups of 8
    for (int h = threadIdx.x >> 4; h < 72; h += blockDim.x >> 4) {
        const int g = kFirstPassGroups[2 * h + ((threadIdx.x >> 3) & 1)];
        if (g == 255) continue;
        const int c = threadIdx.x & 7, j = 8 * g + c;
        float2 v[16];
        // read-only loads (ld.global.nc), not streaming ones (ld.global.cs):
        // measured 2% faster for the kernel, though L1 hits stay rare (7% of
        // sectors), so the gain is not from reuse of the other half of each
        // 128-byte line
#pragma unroll
        for (int r = 0; r < 16; ++r) v[r] = __ldg(z + j + NB1 * r);
        dft<16, false>(v);
        // rho(8g + c) = g/11 + 13 (g%11) + 143 c; padb(16 rho + r) = 17 rho + r (r < 16)
        float2 *d = sm + 17 * (g / 11 + 13 * (g % 11) + 143 * c);
#pragma unroll
        for (int r = 0; r < 16; ++r) d[r] = v[r];
    }
    __syncthreads();
    {
        const int k = threadIdx.x & 15;
        float2 w13[13];
        pass13_twiddles(T, k, w13);
        for (int b = threadIdx.x; b < kMB / 13; b += blockDim.x) fwd_pass13(sm, w13, b >> 4, k);
    }
    __syncthreads();
    fwd_pass11(sm, T);
    __syncthreads();
    fwd_pass8<R2C, R2C>(sm, T);
    __syncthreads();
}

// Unnormalised R2C bin q (0 <= q <= 18304) of the 36608 real samples from the
// half-length complex transform Z in `sm`, given w = e^{-2 pi i q/36608}:
//   X[q] = (Z[q] + conj Z[M-q])/2 - i w (Z[q] - conj Z[M-q])/2.
__device__ __forceinline__ float2 r2c_bin(const float2 *sm, int q, float2 w) {
    const int qa = q == kMB ? 0 : q;
    const int qb = q == 0 ? 0 : kMB - q;
    const float2 za = sm[padb(qa)];
    const float2 zb = conjf2(sm[padb(qb)]);
    const float2 s = cadd(za, zb), d = csub(za, zb);
    const float2 wd = cmul(w, d);
    return make_float2(0.5f * (s.x + wd.y), 0.5f * (s.y - wd.x));
}

// Hermitian pre-processing of a C2R of length 32768 from bins Y[0..16384],
// given we = e^{+2 pi i k/32768}:
//   Z[k] = (Y[k] + conj Y[M-k]) + i we (Y[k] - conj Y[M-k]),
// imaginary parts of Y[0] and Y[16384] ignored (as cuFFT / numpy do).  X, Y:
// the product's rounding (cmul_rn), X < 0 leaves it to the compiler.
template <int X = -1, int Y = -1>
__device__ __forceinline__ float2 c2r_pre(float2 y, float2 ym, int k, float2 we) {
    if (k == 0) {
        y.y = 0.f;
        ym.y = 0.f;
    }
    const float2 e = make_float2(y.x + ym.x, y.y - ym.y);
    const float2 d = make_float2(y.x - ym.x, y.y + ym.y);
    float2 o;
    if constexpr (X < 0) {
        o = cmul(d, we);
    } else {
        o = cmul_rn<X, Y>(d, we);
    }
    return make_float2(e.x - o.y, e.y + o.x);
}

// e^{+2 pi i (tid + 512 r)/32768} for r = 0..31 from one table value.
template <int R>
__device__ __forceinline__ float2 c2r_tw(float2 base) {
    return mul_tc<64, R, true>(base);
}

// The same with each product's rounding pinned, for stage BC.
template <int R>
__device__ __forceinline__ float2 c2r_tw_rn(float2 base) {
    if constexpr (R == 0) return base;
    constexpr bool both = R == 1 || (R >= 7 && R <= 9) || R == 15;
    constexpr int X = both || R <= 6 ? (R <= 15 ? 2 : 0) : 0;
    constexpr int Y = both || (R >= 10 && R <= 14) ? 2 : ((R >= 17 && R <= 25) || R == 31 ? 1 : 0);
    return cmul_rn<X, Y>(base, make_float2(TwC<64, R>::c, -TwC<64, R>::s));
}

// First-pass columns for the paired C2R input below, numbered so that slots
// l and l ^ 16 hold mirror columns (b + b' = 512); slot 16 takes 256.
__device__ __forceinline__ int c2r_col(int t) {
    const int w = t >> 5, l = t & 31;
    if (l < 16) return 16 * w + l;
    return (w == 0 && l == 16) ? 256 : 512 - 16 * w - (l - 16);
}
// The slot of c2r_col that thread t takes.  Columns w + 16 i and their mirrors
// 512 - w - 16 i = (16 - w) + 16 (31 - i) belong to sub-transforms w and
// 16 - w, so two warps take both between them: warps 2w and 2w + 1 the halves
// i < 16 and i >= 16 of sub-transform w in lanes l < 16 and the mirrors in
// lanes l ^ 16 (w = 1..7); then warp 2w runs the second pass of sub-transform
// w, warp 2w + 1 of 16 - w, and only the two of them wait for each other.
// Sub-transforms 0 and 8 are their own mirrors: warps 0 and 1 (warp 0's lane
// 16 takes column 256, the other column, besides lane 0's column 0, that is
// its own mirror).
__device__ __forceinline__ int c2r_slot(int t) {
    const int w = t >> 6, s = (t >> 5) & 1, l = t & 31;
    const int b = (w == 0 ? 8 * s : w + 256 * s) + 16 * (l & 15);  // column of lane l & 15
    const int lo = b < 256 ? b : 512 - b;
    return 32 * (lo >> 4) + (lo & 15) + 16 * ((l >> 4) ^ (b > 256 ? 1 : 0));
}
__device__ __forceinline__ int c2r_sub(int t) {
    const int w = t >> 6, s = (t >> 5) & 1;
    return w == 0 ? 8 * s : (s ? 16 - w : w);
}

// The inverse's first-pass inputs Z'[j], j = col + 512 r, of the window Y[j] =
// X[skip + j], j = 0..16384, by the C2R pairing on the fly (no pass of its own),
// with W_32768^-j = wc e^{2 pi i r/64} (wc per thread, the rest compile-time);
// Im Y[0] and Im Y[16384] are dropped.  A warp's columns are 16 apart, one
// padded row of `sm` each: both runs, up from Y[col] and down from
// Y[16384 - col], are conflict-free.
__device__ __forceinline__ void c2r_window(float2 *v, const float2 *sm, int skip, int col, float2 wc) {
    const float2 *lo = sm + padb(skip + col);        // Y[col + 512 r] = lo[544 r]
    const float2 *hi = sm + padb(skip + kMA - col);  // Y[16384 - col - 512 r] = hi[-544 r]
    for_r(std::make_integer_sequence<int, 32>{}, [&](auto rc) {
        constexpr int r = decltype(rc)::value;
        v[r] = c2r_pre<0, r == 0 ? 1 : 0>(lo[544 * r], hi[-544 * r], col + 512 * r, c2r_tw_rn<r>(wc));
    });
}

// The C2R 32768 input Z[col + 512 r], r < 32, from the bins Y[0..16384]
// (M = 16384): Z[k] = (Y[k] + conj Y[M-k]) + i e^{2 pi i k/32768}
// (Y[k] - conj Y[M-k]), Im Y[0] and Im Y[M] dropped (Y[M] = 0 if NYQ_ZERO).
// Each pair (k, M - k) is formed once: for p < 16 the thread pairs its
// k = col + 512 p with M - k, which is element 31 - p of the mirror column
// 512 - col, held by lane l ^ 16; one shuffle swaps the halves.  Columns 0
// and 256 are their own mirrors (M - 512 p = 512 (32 - p); M - 256 - 512 p
// = 256 + 512 (31 - p)) and keep both halves; column 0 forms Z[8192] alone.
// lo(p) = Y[col + 512 p] (p <= 16), hi(p) = Y[M - col - 512 p] (p < 16);
// we[p] = e^{2 pi i (col + 512 p)/32768}, w16 its value at p = 16.
template <bool NYQ_ZERO, class Lo, class Hi>
__device__ __forceinline__ void c2r_paired(float2 *v, int col, const float2 *we, float2 w16, Lo lo, Hi hi) {
    const int lane = threadIdx.x & 31;
    // Every warp runs the same code (a second copy for warp 0 would be fetched
    // beside the others').  Lane 16 of warp 0 (column 256) keeps its own mirror
    // halves; lane 0 (column 0) its own too, one element on.
    const bool w0 = threadIdx.x < 32, c0 = threadIdx.x == 0;
    const int src = w0 && lane == 16 ? lane : lane ^ 16;
    for_r(std::make_integer_sequence<int, 16>{}, [&](auto pc) {
        constexpr int p = decltype(pc)::value;
        float2 y = lo(pc), ym = hi(pc);
        if (p == 0 && col == 0) {
            y.y = 0.f;
            ym = NYQ_ZERO ? make_float2(0.f, 0.f) : make_float2(ym.x, 0.f);
        }
        float2 zk, zmk;
        c2r_pair_rn<p == 0 ? 1 : 0, 1>(y, ym, we[p], zk, zmk);
        v[p] = zk;
        v[31 - p] = make_float2(__shfl_sync(0xffffffffu, zmk.x, src), __shfl_sync(0xffffffffu, zmk.y, src));
        if constexpr (p >= 1) v[32 - p] = make_float2(c0 ? zmk.x : v[32 - p].x, c0 ? zmk.y : v[32 - p].y);
    });
    if (w0) {
        // column 0: Z[8192] = Y[8192] + conj Y[8192] + i e^{i pi/2} (Y[8192] - conj Y[8192]);
        // the other lanes' lo(16) is in range and discarded
        const float2 y = lo(std::integral_constant<int, 16>{});
        const float2 z = c2r_pre(y, y, 8192, w16);
        v[16] = make_float2(c0 ? z.x : v[16].x, c0 ? z.y : v[16].y);
    }
}

// Barrier `id` (1..15; 0 is __syncthreads) of n threads.
__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }

// ---------------------------------------------------------------------------
// Stage A (persistent): items = n_snaps x n_pols.  Packed spectrum of snapshot
// s of pol p at spec + p*spec_pol_stride + (snap0 + s)*2048; time series to
// out + p*out_pol_stride + s*32768.
template <class Segs>
__device__ __forceinline__ int seg_of(const Segs &S, int64_t item) {
    int j = 0;
    while (j + 1 < S.n && item >= S.s[j + 1].item0) ++j;
    return j;
}

// The stage-A pipeline of one CTA.  A warp's work on an item is its input
// columns (pairing and DFT-32), the first two passes of one sub-transform and
// its share of the last pass.  Only the last pass needs every warp's earlier
// work, and only the first pass's stores overwrite what every warp has read,
// so each of these two dependencies is an mbarrier (one arrival per warp) with
// other work between the arrival and the wait: a warp that has finished its
// second pass forms the NEXT item's input columns before it waits for the
// others, parking the 64 registers in tensor memory.  In a plain barrier
// form, warps that ran in step competed for the shared-memory pipe in one
// phase and for the FMA pipe in the next, and each was idle a third of the
// time.
struct PipeA {
    uint64_t full[2];  // spectrum of an even / odd item landed
    uint64_t read;     // a warp's last-pass loads are done
    uint64_t second;   // a warp's second pass is stored
    uint32_t tmem;
    int err;
};
// Tensor memory columns: parked registers, 64 for each of the four warps of a
// lane quarter, and the second pass's twiddles, 64, the same for the four
// (forming them anew costs 84 instructions and 10 loads a thread and item).
constexpr uint32_t kColPark = 0, kColTw2 = 256, kColsA = 512;

// Shared memory holds the sub-transforms of an item and a half: three blocks
// of eight, item k in blocks 2k and 2k + 1 (mod 3).  Its first block is never
// one that item k - 1 is still read from, so the eight warps whose columns go
// there (warps 0-7: sub-transforms 0, 8, 1, 15, 2, 14, 3, 13) store without
// waiting, half an item ahead of the other eight: one half's shared-memory
// phases meet the other half's arithmetic.
constexpr int kBlkA = 8 * kSub;
__host__ __device__ constexpr bool blk_second(int sub) { return (sub >= 4 && sub <= 7) || (sub >= 9 && sub <= 12); }
__host__ __device__ constexpr int blk_index(int sub) {  // warps 2 p and 2 p + 1 hold sub-transforms p and 16 - p
    const int p = sub == 8 ? 0 : (sub > 8 ? 16 - sub : sub);
    return 2 * (p & 3) + (sub >= 8 ? 1 : 0);
}

__global__ void __launch_bounds__(kNTA, 1) k_swarm_c2r(const __grid_constant__ SegsA S, Twiddles tw) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint32_t *sp = reinterpret_cast<uint32_t *>(smem_raw);  // [2][2048] double buffer
    float2 *sm = reinterpret_cast<float2 *>(smem_raw + 2 * kGroups * sizeof(uint32_t));
    __shared__ PipeA P;
    TabsA T = tabs_a_at(sm + 3 * kBlkA);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t n_items = S.n_items;
    const int64_t G = gridDim.x;
    auto fetch = [&](int64_t item, int buf) {  // one thread
        const SegA &g = S.s[seg_of(S, item)];
        const int64_t local = item - g.item0;
        const int64_t pol = local >= g.n_snaps, s = local - pol * g.n_snaps;  // n_pols <= 2: no division
        tc5::bulk_g2s(sp + buf * kGroups, g.spec + pol * g.spec_pol_stride + (g.snap0 + s) * kGroups,
                      kGroups * sizeof(uint32_t), &P.full[buf]);
    };
    if (threadIdx.x == 0) {
        tc5::mbar_init(&P.full[0], 1);
        tc5::mbar_init(&P.full[1], 1);
        tc5::mbar_init(&P.read, kNTA / 32);
        tc5::mbar_init(&P.second, kNTA / 32 + (tw.withhold == 1 ? 1 : 0));
        tc5::fence_mbar_init();
        P.err = 0;
        // the first spectra on their way while the tables load
        if (blockIdx.x < n_items) fetch(blockIdx.x, 0);
        if (blockIdx.x + G < n_items) fetch(blockIdx.x + G, 1);
    }
    if (warp == 0) tc5::tmem_alloc(&P.tmem, kColsA);
    load_tabs<kEntA>([&](int m) { return tab_entry_a(T, tw, m); });
    const int col = c2r_col(c2r_slot(threadIdx.x)), sub = c2r_sub(threadIdx.x);
    const float2 wc = conjf2(__ldg(tw.w32768 + col));  // W_32768^-col
    tc5::fence_before();
    __syncthreads();  // tables loaded, barriers and tensor memory ready
    tc5::fence_after();
    const uint32_t quarter = P.tmem + (static_cast<uint32_t>(warp & 3) << 21);
    const uint32_t park = quarter + kColPark + 64u * (warp >> 2), tw2nd = quarter + kColTw2;
    if (warp < 4) {
        float2 w[32];
        pass2_twiddles(T, w);
        tc5::tmem_park<32>(tw2nd, w);
    }
    tc5::fence_before();
    __syncthreads();  // the four warps of a quarter read one table
    tc5::fence_after();
    const LastTw lt = last_tw(T);  // once per CTA
    auto wait = [&](uint64_t *bar, uint32_t parity) { return tc5::wait_or_flag(bar, parity, &P.err); };
    // The first item whose spectrum this thread did not see land (after a
    // wait has run out); none is asked for after that.
    uint32_t lost = ~0u;
    // Input columns of the k-th item (its spectrum in buffer k & 1), DFT-32,
    // parked.  The first pass takes Z[col + 512 r] from the packed bins X[k]
    // (k < 16384; the Nyquist bin X[16384] = 0, Im X[0] dropped), each
    // Hermitian pair once with its mirror half from lane ^ 16.
    auto input = [&](uint32_t k) {
        if (!wait(&P.full[k & 1], k >> 1) && lost == ~0u) lost = k;
        const uint32_t *cur = sp + (k & 1) * kGroups;
        float2 v[32], w[16];
        for_r(std::make_integer_sequence<int, 16>{}, [&](auto pc) { w[decltype(pc)::value] = c2r_tw<decltype(pc)::value>(wc); });
        c2r_paired<true>(
            v, col, w, c2r_tw<16>(wc), [&](auto pc) { return nib_value(cur, col + kNTA * decltype(pc)::value); },
            [&](auto pc) {
                constexpr int p = decltype(pc)::value;
                const int j = kMA - col - kNTA * p;  // 16384 only for col = 0, p = 0 (replaced by 0)
                return nib_value(cur, p == 0 ? (j & (kMA - 1)) : j);
            });
        dft<32, true>(v);
        tc5::tmem_park<32>(park, v);
    };
    int64_t item = blockIdx.x;
    if (item < n_items) input(0);
    float2 *first = sm, *second = sm + kBlkA, *spare = sm + 2 * kBlkA;
    for (uint32_t k = 0; item < n_items; item += G, ++k) {
        float2 *mine = warp < 8 ? first : second;
        {
            float2 v[32];
            tc5::tmem_unpark<32>(park, v);
            if (warp >= 8 && k > 0) wait(&P.read, k - 1);
            inv_store1(mine + kSub * blk_index(col & 15), col, v);
        }
        bar_sync(1 + (threadIdx.x >> 6), 64);
        inv_pass2(mine + kSub * blk_index(sub), [&](float2 *v) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float2 w[16];
                tc5::tmem_unpark<16>(tw2nd + 32 * h, w);
#pragma unroll
                for (int r = 0; r < 16; ++r)
                    if (16 * h + r > 0) v[16 * h + r] = cmulc(v[16 * h + r], w[r]);
            }
        });
        __syncwarp();
        if (lane == 0) tc5::mbar_arrive(&P.second);
        if (item + G < n_items) input(k + 1);
        wait(&P.second, k);
        // every warp is done with this item's spectrum (its input columns
        // came before its second pass): the buffer takes the item after next,
        // unless a copy's wait ran out
        if (threadIdx.x == 0 && item + 2 * G < n_items && lost == ~0u) fetch(item + 2 * G, k & 1);
        const SegA &g = S.s[seg_of(S, item)];
        const int64_t local = item - g.item0;
        const int64_t pol = local >= g.n_snaps, s = local - pol * g.n_snaps;
        float2 *dst = reinterpret_cast<float2 *>(g.out + pol * g.out_pol_stride + s * kNA);
        inv_pass3<false>(
            [&](int r) { return (blk_second(r) ? second : first) + kSub * blk_index(r); }, lt,
            [&](int jj, const float2 *u) {
#pragma unroll
                for (int r = 0; r < 16; ++r) __stcs(dst + jj + 1024 * r, u[r]);
            },
            [&] {
                __syncwarp();
                if (lane == 0) tc5::mbar_arrive(&P.read);
            });
        float2 *t = first;
        first = spare;
        spare = second;
        second = t;
    }
    // no copy outlives the CTA: one more bounded wait for the lost item's, and
    // for item 1's, asked for together with item 0's
    if (threadIdx.x == 0 && lost != ~0u) {
        tc5::mbar_wait(&P.full[lost & 1], lost >> 1);
        if (lost == 0 && blockIdx.x + G < n_items) tc5::mbar_wait(&P.full[1], 0);
    }
    tc5::fence_before();
    __syncthreads();
    if (warp == 0) tc5::tmem_free(P.tmem, kColsA);
    if (threadIdx.x == 0 && tc5::flag_set(&P.err)) S.status.raise();
}

// ---------------------------------------------------------------------------
// Stage BC (persistent): items = n_chunks x n_pols.  Chunk c of pol p: 36608
// floats at in + p*in_pol_stride + c*36608.
//   MODE 0: quantize with thr[p] / thr[2+p] into the u32 payload at
//           out + p*out_pol_stride + (pkt0 + c)*pkt_stride + payload_off.
//   MODE 1: floats to fout + p*fout_pol_stride + c*32768 and per-chunk
//           (n, mean, M2) in FP64 to partials[(p*n_chunks + c)*3].
//   MODE 2: floats only.
//   MODE 3: MODE 0, plus the (n, sum, sum of squares) of each chunk's
//           floats (FP32 per thread and warp, FP64 across warps) to partials
//           when the segment has them (windowed thresholds).
//
// The CTA's pipeline.  Each pass needs every warp's work of the pass before,
// and the transform's buffer is rewritten while the next chunk waits for it;
// every one of these dependencies is an mbarrier with one arrival per warp,
// and the next chunk's first pass (radix 16), whose inputs come from global
// memory and whose outputs wait in tensor memory, is done in three rounds
// between the arrivals at and the waits for three of them.  Four teams of
// four warps each take every fourth of eleven groups of 1664 elements through
// passes 1 and 2: group m holds the first-pass butterflies j = 8 (m + 11 t) +
// c (t < 13, c < 8) and the radix-13 blocks m + 11 c, so the two passes need
// a team's barrier only.  A round's inputs (16 rows of 13 x 8 complex values
// per team) are copied to shared memory by cp.async one round ahead: no
// registers and, bypassing L1, none of its lines are held by loads in flight
// (reading them with plain loads cost 9% of the kernel once L1 is small, as
// beside stage A's shared memory).
struct PipeB {
    uint64_t xfree;   // the inverse's last-pass loads are done
    uint64_t pass2, pass3, pass4;  // forward passes stored
    uint64_t taken;   // the inverse has read X
    uint64_t inv2;    // the inverse's second pass is stored
    uint32_t tmem;
    int err;
};
// Tensor memory columns: three parked rounds (32 columns for each of the four
// warps of a lane quarter), the inverse's second-pass twiddles (the same for
// the four), its last pass's bases (12 values, for each).
constexpr uint32_t kColRound = 0, kColTw2B = 384, kColLast = 448, kColsB = 512;
// One staged round of a team: row r (16) holds inputs t < 8 then, eight slots
// further on, t >= 8, so that a half-warp (t and t + 8, c = 0..7) reads 16
// bank pairs.
constexpr int kStageRow = 13 * 8 + 8;
constexpr int kStage = 16 * kStageRow;
constexpr size_t kSmemPipeB = kSmemB + 4 * kStage * sizeof(float2);
static_assert(kSmemPipeB <= 232448 - 1024, "stage BC shared memory above 227 KB");

template <int MODE>
__global__ void __launch_bounds__(kNTB, 1) k_resample(const __grid_constant__ SegsB S, Twiddles tw) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2 *stages = reinterpret_cast<float2 *>(smem_raw);  // 16-byte aligned rows
    float2 *sm = stages + 4 * kStage;
    float2 *tb = sm + kPadB;
    TabsA TA = tabs_a_at(tb);
    TabsB TB = tabs_b_at(tb, tw);
    __shared__ double red[64];
    __shared__ PipeB P;
    // the first batch runs a chunk or two per CTA (6000 chunks of floats alone: 687 us rolled, 676 not)
    constexpr bool ROLL = MODE == 1;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        uint64_t *bars[6] = {&P.xfree, &P.pass2, &P.pass3, &P.pass4, &P.taken, &P.inv2};
        for (uint64_t *b : bars) tc5::mbar_init(b, kNTB / 32 + (b == &P.pass2 && tw.withhold == 2 ? 1 : 0));
        tc5::fence_mbar_init();
        P.err = 0;
    }
    const int64_t n_items = S.n_items, G = gridDim.x;
    auto wait = [&](uint64_t *bar, uint32_t parity) { tc5::wait_or_flag(bar, parity, &P.err); };
    auto arrive = [&](uint64_t *bar) {
        __syncwarp();
        if (lane == 0) tc5::mbar_arrive(bar);
    };
    auto src_of = [&](int64_t item) {
        const SegB &g = S.s[seg_of(S, item)];
        const int64_t local = item - g.item0;
        const int64_t pol = local >= g.n_chunks;  // n_pols <= 2: no division
        return reinterpret_cast<const float2 *>(g.in + pol * g.in_pol_stride + (local - pol * g.n_chunks) * kNB);
    };
    // first two forward passes: this thread's team, its butterfly (c, t) of a
    // group in pass 1 and its radix-13 column (block m + 11 c13, k13) in pass 2
    const int team = warp >> 2, tt = tid & 127;
    const int c1 = tt & 7, t1 = (tt >> 4) + (tt & 8), c13 = tt >> 4, k13 = tt & 15;
    float2 *stg = stages + team * kStage;
    auto team_sync = [&] { bar_sync(1 + team, 128); };
    // Groups of this team, round by round.  Team 0 has one fewer: its warps
    // have one more unit of the last forward pass than the others.
    const int m0 = (team + 3) & 3;
    // The inputs of round r (group m0 + 4 r) to the team's stage: 16 rows of
    // 13 runs of 64 bytes, eight threads a row.
    const int frow = tt >> 3, fpart = 2 * (tt & 3), ft = (tt >> 2) & 1;
    float2 *fdst = stg + frow * kStageRow + 8 * ft + fpart;
    const int fsrc = 1144 * frow + 8 * (m0 + 11 * ft) + fpart;
    auto fetch = [&](const float2 *z, int r) {
        if (m0 + 4 * r < 11) {
            const float2 *src = z + fsrc + 32 * r;
#pragma unroll
            for (int j = 0; j < 7; ++j)  // runs t = ft + 2 j < 13
                if (j < 6 || ft == 0) tc5::cp_async16(fdst + 16 * j + (j < 4 ? 0 : 8), src + 176 * j);
        }
        tc5::cp_async_commit();
    };
    int64_t item = blockIdx.x;
    if (item < n_items) fetch(src_of(item), 0);  // on its way while the tables load
    if (warp == 0) tc5::tmem_alloc(&P.tmem, kColsB);
    if constexpr (ROLL) {
        load_tabs_ab(TA, TB, tw);
    } else {
        load_tabs_a(TA, tw);
        load_tabs_b(TB, tw);
    }
    // the inverse's first-pass column: warp w takes those of sub-transform w,
    // so its first two passes need no barrier but the warp's own
    const int sub = warp, col = sub + 16 * lane;
    const float2 wc = conjf2(__ldg(tw.w32768 + col));  // W_32768^-col
    tc5::fence_before();
    __syncthreads();  // tables loaded, barriers and tensor memory ready
    tc5::fence_after();
    const uint32_t quarter = P.tmem + (static_cast<uint32_t>(warp & 3) << 21);
    const uint32_t tw2nd = quarter + kColTw2B, twlast = quarter + kColLast + 16u * (warp >> 2);
    {
        float2 w[32];
        if (warp < 4) {
            pass2_twiddles(TA, w);
            tc5::tmem_park<32>(tw2nd, w);
        }
        const LastTw lt = last_tw(TA);
        float2 l[8];
        l[0] = l[7] = make_float2(0.f, 0.f);
#pragma unroll
        for (int j = 1; j < 4; ++j) {
            l[j] = lt.S0[j];
            l[3 + j] = lt.A0[j];
        }
        tc5::tmem_park<8>(twlast, l);
    }
    tc5::fence_before();
    __syncthreads();  // the four warps of a quarter read one table
    tc5::fence_after();
    // Round r of the first pass from the stage, parked; then the next fetch.
    auto first_pass = [&](int r, const float2 *znext, int rnext) {
        tc5::cp_async_wait_all();
        team_sync();  // the whole team's copies landed
        if (m0 + 4 * r < 11) {
            float2 v[16];
            const float2 *p = stg + (t1 < 13 ? 8 * t1 + (t1 < 8 ? 0 : 8) : 0) + c1;
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = p[kStageRow * i];
            dft<16, false>(v);
            tc5::tmem_park<16>(quarter + kColRound + 96u * (warp >> 2) + 32u * r, v);
        }
        team_sync();  // the stage has been read
        if (znext) fetch(znext, rnext);
    };
    if (item < n_items) {
        // rounds 1 and 2 of the first chunk straight to registers, beside round 0
        const float2 *z = src_of(item);
        float2 early[2][16];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int i = 0; i < 16; ++i)
                early[h][i] = t1 < 13 && m0 + 4 * (h + 1) < 11 ? __ldg(z + 8 * (m0 + 4 * (h + 1) + 11 * t1) + c1 + 1144 * i)
                                                               : make_float2(0.f, 0.f);
        first_pass(0, item + G < n_items ? src_of(item + G) : nullptr, 0);
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (m0 + 4 * (h + 1) < 11) {
                dft<16, false>(early[h]);
                tc5::tmem_park<16>(quarter + kColRound + 96u * (warp >> 2) + 32u * (h + 1), early[h]);
            }
    }
    for (uint32_t k = 0; item < n_items; item += G, ++k) {
        const SegB &g = S.s[seg_of(S, item)];
        const ResampleOut &o = g.o;
        const int n_chunks = g.n_chunks, skip = g.skip;
        const int64_t local = item - g.item0;
        const int pol = local >= n_chunks;  // n_pols <= 2: no division
        const int64_t c = local - pol * n_chunks;
        const bool more = item + G < n_items;
        const float2 *zn = more ? src_of(item + G) : nullptr;
        // forward 18304: the parked first pass into X, then radix 13
        if (k > 0) wait(&P.xfree, k - 1);
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const int m = m0 + 4 * r;
            if (m < 11) {
                float2 v[16];
                tc5::tmem_unpark<16>(quarter + kColRound + 96u * (warp >> 2) + 32u * r, v);
                // rho(8g + c) = g/11 + 13 (g%11) + 143 c; padb(16 rho + r) = 17 rho + r (r < 16)
                float2 *d = sm + 17 * (t1 + 13 * m + 143 * c1);
                if (t1 < 13) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) d[i] = v[i];
                }
            }
        }
        team_sync();
        {
            float2 w13[13];
            pass13_twiddles(TB, k13, w13);
            for (int m = m0; m < 11; m += 4) fwd_pass13(sm, w13, m + 11 * c13, k13);
        }
        arrive(&P.pass2);
        if (more) first_pass(0, zn, 1);
        wait(&P.pass2, k);
        fwd_pass11(sm, TB);
        arrive(&P.pass3);
        if (more) first_pass(1, zn, 2);
        wait(&P.pass3, k);
        // the last forward pass with the R2C pairing: X[q], q <= 18304
        fwd_pass8<true, ROLL>(sm, TB);
        arrive(&P.pass4);
        // The chunk after next, 146 KB, to L2 as nine bulk prefetches from nine
        // threads of a warp that waits here for those with a third unit
        if (warp == 12 && lane < 9 && item + 2 * G < n_items) {  // 146432 B = 8 x 16384 + 15360, 16-byte aligned pieces
            const uint32_t bytes = lane < 8 ? 16384u : static_cast<uint32_t>(kNB * 4 - 8 * 16384);
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(
                             reinterpret_cast<const char *>(src_of(item + 2 * G)) + 16384 * lane),
                         "r"(bytes)
                         : "memory");
        }
        wait(&P.pass4, k);
        auto inverse = [&](auto epi) {
            {
                float2 v[32];
                c2r_window(v, sm, skip, col, wc);
                arrive(&P.taken);
                dft<32, true>(v);
                wait(&P.taken, k);  // every read of X ends before the first stores over it
                inv_store1(sm + kSub * sub, col, v);
            }
            __syncwarp();
            inv_pass2(sm + kSub * sub, [&](float2 *v) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float2 w[16];
                    tc5::tmem_unpark<16>(tw2nd + 32 * h, w);
#pragma unroll
                    for (int r = 0; r < 16; ++r)
                        if (16 * h + r > 0) v[16 * h + r] = cmulc(v[16 * h + r], w[r]);
                }
            });
            arrive(&P.inv2);
            if (more) first_pass(2, item + 2 * G < n_items ? src_of(item + 2 * G) : nullptr, 0);
            LastTw lt;
            {
                float2 l[8];
                tc5::tmem_unpark<8>(twlast, l);
#pragma unroll
                for (int j = 1; j < 4; ++j) {
                    lt.S0[j] = l[j];
                    lt.A0[j] = l[3 + j];
                }
            }
            wait(&P.inv2, k);
            inv_pass3<ROLL>([&](int r) { return sm + kSub * r; }, lt, epi, [&] { arrive(&P.xfree); });
        };
        if constexpr (MODE == 0 || MODE == 3) {
            uint32_t *words = reinterpret_cast<uint32_t *>(o.out + pol * o.out_pol_stride +
                                                           (o.pkt0 + c) * o.pkt_stride + o.payload_off);
            const Coder2 cd = coder2(o.thr[pol], o.thr[2 + pol]);
            float f1 = 0.f, f2 = 0.f;
            // Word (jj >> 3) + 128 r holds the 4-bit codes of outputs jj + 1024 r
            // of the 8 lanes jj & 7 = c (lane c at bits 4c).  Each lane builds
            // its codes of rows r < 8 and 8 <= r < 16 as two words (row r at
            // bits 4 (r % 8)); an 8 x 8 nibble transpose over the 8 lanes then
            // leaves lane c with the output words of rows c and 8 + c.
            auto epi = [&](int jj, const float2 *u) {
                uint32_t wl = 0, wh = 0;
#pragma unroll
                for (int r = 7; r >= 0; --r) {
                    push2(wl, u[r].y, cd);
                    push2(wl, u[r].x, cd);
                    push2(wh, u[8 + r].y, cd);
                    push2(wh, u[8 + r].x, cd);
                }
                wl = codes2(wl);
                wh = codes2(wh);
                if constexpr (MODE == 3) {
#pragma unroll
                    for (int r = 0; r < 16; ++r) {
                        f1 += u[r].x + u[r].y;
                        f2 = fmaf(u[r].x, u[r].x, fmaf(u[r].y, u[r].y, f2));
                    }
                }
                const int c = jj & 7;
                wl = nib_transpose8(wl, c);
                wh = nib_transpose8(wh, c);
                words[(jj >> 3) + 128 * c] = wl;
                words[(jj >> 3) + 128 * (8 + c)] = wh;
            };
            inverse(epi);
            if constexpr (MODE == 3) {
                if (o.partials != nullptr) {  // uniform over the block
                    double s1, s2;
                    block_sum2_f(f1, f2, s1, s2, red);
                    if (tid == 0) {
                        double *pp = o.partials + (static_cast<int64_t>(pol) * n_chunks + c) * 3;
                        pp[0] = static_cast<double>(kNC);
                        pp[1] = s1;
                        pp[2] = s2;
                    }
                }
            }
        } else {
            float2 *fo = reinterpret_cast<float2 *>(o.fout + pol * o.fout_pol_stride + c * kNC);
            Moments2 mo;
            auto epi = [&](int jj, const float2 *u) {
#pragma unroll
                for (int r = 0; r < 16; ++r) {
                    fo[jj + 1024 * r] = u[r];
                    if constexpr (MODE == 1) {
                        mo.add(u[r].x);
                        mo.add(u[r].y);
                    }
                }
            };
            inverse(epi);
            if constexpr (MODE == 1) {
                double s1, s2;
                block_moments<kNTB / 32>(mo, s1, s2, reinterpret_cast<float *>(red));
                if (tid == 0) {
                    const double n = static_cast<double>(kNC);
                    const double mean = s1 * (1.0 / kNC);  // a power of two: exact
                    double *pp = o.partials + (static_cast<int64_t>(pol) * n_chunks + c) * 3;
                    pp[0] = n;
                    pp[1] = mean;
                    pp[2] = s2 - s1 * mean;
                }
            }
        }
    }
    tc5::fence_before();
    __syncthreads();
    if (warp == 0) tc5::tmem_free(P.tmem, kColsB);
    if (tid == 0 && tc5::flag_set(&P.err)) S.status.raise();
}

// k_resample<2> for at most two chunks per SM, one CTA each: little to overlap,
// so no pipeline to set up (tensor memory, stages, barriers), block barriers
// between the passes.  A call of 1 to 152 chunks takes 24.8 us (bound by the
// latency of each pass, 16 warps an SM), 29 through the pipeline, 153 to 304
// take 42 to 43 (46 to 48), 456 would take 69.4 (68.3).
__global__ void __launch_bounds__(kNTB, 1)
    k_resample_once(const float *__restrict__ in, int skip, float *__restrict__ out, Twiddles tw) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2 *sm = reinterpret_cast<float2 *>(smem_raw);
    float2 *tb = sm + kPadB;
    TabsA TA = tabs_a_at(tb);
    TabsB TB = tabs_b_at(tb, tw);
    load_tabs_ab(TA, TB, tw);
    const int sub = threadIdx.x >> 5, col = sub + 16 * (threadIdx.x & 31);
    const float2 wc = conjf2(__ldg(tw.w32768 + col));  // W_32768^-col
    fft18304_from_global<true>(sm, reinterpret_cast<const float2 *>(in + static_cast<int64_t>(blockIdx.x) * kNB), TB);
    float2 v[32];
    c2r_window(v, sm, skip, col, wc);
    dft<32, true>(v);
    __syncthreads();  // every read of X ends before the first stores over it
    inv_store1(sm + kSub * sub, col, v);
    __syncwarp();
    inv_pass2(sm + kSub * sub, [&](float2 *u) {
        float2 w[32];
        pass2_twiddles(TA, w);
#pragma unroll
        for (int r = 1; r < 32; ++r) u[r] = cmulc(u[r], w[r]);
    });
    __syncthreads();
    float2 *dst = reinterpret_cast<float2 *>(out + static_cast<int64_t>(blockIdx.x) * kNC);
    inv_pass3<true>([&](int r) { return sm + kSub * r; }, last_tw(TA), [&](int jj, const float2 *u) {
#pragma unroll
        for (int r = 0; r < 16; ++r) dst[jj + 1024 * r] = u[r];
    }, [] {});
}

// SwarmR2C alone: complex64 [n][18305] spectra (persistent over chunks).
__global__ void __launch_bounds__(kNTB, 1)
    k_swarm_r2c(const float *__restrict__ in, int64_t n_chunks, float2 *__restrict__ out, Twiddles tw) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2 *sm = reinterpret_cast<float2 *>(smem_raw);
    float2 *tb = sm + kPadB;
    TabsB TB = tabs_b_at(tb, tw);
    load_tabs_b(TB, tw);
    for (int64_t c = blockIdx.x; c < n_chunks; c += gridDim.x) {
        __syncthreads();
        fft18304_from_global<false>(sm, reinterpret_cast<const float2 *>(in + c * kNB), TB);
        float2 *dst = out + c * (kMB + 1);
        for (int q = threadIdx.x; q <= kMB; q += kNTB) dst[q] = r2c_bin(sm, q, __ldg(tw.w36608 + q));
    }
}

// R2dbeC2R alone: complex64 [n][18305] from bin skip -> float [n][32768].
__global__ void __launch_bounds__(kNTB, 1)
    k_r2dbe_c2r(const float2 *__restrict__ in, int64_t in_stride, int64_t n_chunks, int skip, float *__restrict__ out,
                Twiddles tw) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2 *sm = reinterpret_cast<float2 *>(smem_raw);
    float2 *tb = sm + kPadB;
    TabsA TA = tabs_a_at(tb);
    load_tabs_a(TA, tw);
    const int tid = threadIdx.x;
    const float2 wc = conjf2(__ldg(tw.w32768 + tid));
    for (int64_t c = blockIdx.x; c < n_chunks; c += gridDim.x) {
        const float2 *y = in + c * in_stride + skip;
        auto zin = [&](float2 *v) {
            for_r(std::make_integer_sequence<int, 32>{}, [&](auto rc) {
                constexpr int r = decltype(rc)::value;
                const int k = tid + 512 * r;
                v[r] = c2r_pre(__ldg(y + k), __ldg(y + kMA - k), k, c2r_tw<r>(wc));
            });
        };
        float2 *dst = reinterpret_cast<float2 *>(out + c * kNC);
        auto epi = [&](int jj, const float2 *u) {
#pragma unroll
            for (int r = 0; r < 16; ++r) dst[jj + 1024 * r] = u[r];
        };
        float2 v[32];
        zin(v);
        dft<32, true>(v);
        __syncthreads();  // the previous chunk's last reads of `sm` (and the table loads) are done
        // consecutive columns (coalesced reads): a sub-transform's first two
        // passes span all warps
        inv_store1(sm + kSub * (tid & 15), tid, v);
        __syncthreads();
        inv_pass2(sm + kSub * (tid >> 5), [&](float2 *v) {
            float2 w[32];
            pass2_twiddles(TA, w);
#pragma unroll
            for (int r = 1; r < 32; ++r) v[r] = cmulc(v[r], w[r]);
        });
        __syncthreads();
        inv_pass3<true>([&](int r) { return sm + kSub * r; }, last_tw(TA), epi, [] {});
    }
}

// ---------------------------------------------------------------------------
struct Moments {
    double n, mean, m2;
};

// Chan et al. pairwise merge of (n, mean, M2) for equal counts.
__device__ __forceinline__ Moments merge_equal(Moments a, Moments b) {
    const double delta = b.mean - a.mean;
    return Moments{a.n + b.n, a.mean + 0.5 * delta, a.m2 + b.m2 + delta * delta * (0.5 * a.n)};
}

// Threshold from the per-chunk partials, FP64, one warp per pol: each lane
// merges its four chunks, then a fixed butterfly tree merges the lanes
// (deterministic).  thr_state: [0..1] effective threshold, [2..3] effective
// offset, [4..5] own threshold, [6..7] own offset.
__global__ void k_finalize_thresholds(const double *__restrict__ partials, int pol1_uses_pol0,
                                      float *__restrict__ thr_state) {
    __shared__ float th_s[2], off_s[2];
    const int pol = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (pol < 2) {
        // pairs of equal counts (every chunk has kNC samples): the merge's
        // n_b / n is 1/2 and its n_a n_b / n is n_a / 2, no division (FP64
        // divisions, 18 of them, took 9 us)
        static_assert(kChunks == 128, "four chunks a lane");
        auto at = [&](int c) {
            const double *pp = partials + (static_cast<int64_t>(pol) * kChunks + c) * 3;
            return Moments{pp[0], pp[1], pp[2]};
        };
        Moments m = merge_equal(merge_equal(at(lane), at(lane + 32)), merge_equal(at(lane + 64), at(lane + 96)));
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            Moments other{__shfl_xor_sync(0xffffffffu, m.n, o), __shfl_xor_sync(0xffffffffu, m.mean, o),
                          __shfl_xor_sync(0xffffffffu, m.m2, o)};
            m = (lane & o) ? merge_equal(other, m) : merge_equal(m, other);
        }
        if (lane == 0) {
            th_s[pol] = static_cast<float>(sqrt(m.m2 / (m.n - 1.0)));
            off_s[pol] = static_cast<float>(m.mean);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        thr_state[4] = th_s[0];
        thr_state[5] = th_s[1];
        thr_state[6] = off_s[0];
        thr_state[7] = off_s[1];
        thr_state[0] = th_s[0];
        thr_state[1] = pol1_uses_pol0 ? th_s[0] : th_s[1];
        thr_state[2] = off_s[0];
        thr_state[3] = pol1_uses_pol0 ? off_s[0] : off_s[1];
    }
}

// Windowed thresholds: one CTA per handle, warps 0-3 pol 0 and 4-7 pol 1.
// Pushes the (n, sum, sum of squares) of each of the nb batches just
// quantized (128 chunk partials each, [pol][nb*128][3]; the first batch's
// partials are (n, mean, M2) and are converted) into the handle's FP64 ring
// (slot t mod W), then, if `update`, sets the thresholds from the sums over
// batches [max(0, T-W), T), T = t0 + nb.  Plain FP64 sums in a fixed order:
// no division but the final mean and variance.
__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__global__ void __launch_bounds__(256) k_window_update(const __grid_constant__ WinUpds U) {
    const WinUpd &u = U.u[blockIdx.x];
    __shared__ float th_s[2], off_s[2];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pol = warp >> 2, wq = warp & 3;
    const int64_t n_chunks = static_cast<int64_t>(u.nb) * kChunks;
    for (int b = wq; b < u.nb; b += 4) {
        double n = 0.0, s1 = 0.0, s2 = 0.0;
        for (int c = lane; c < kChunks; c += 32) {
            const double *pp = u.partials + (pol * n_chunks + static_cast<int64_t>(b) * kChunks + c) * 3;
            if (u.moments) {  // (n, mean, M2)
                const double cn = pp[0], cm = pp[1];
                n += cn;
                s1 += cn * cm;
                s2 += pp[2] + cn * cm * cm;
            } else {
                n += pp[0];
                s1 += pp[1];
                s2 += pp[2];
            }
        }
        n = warp_sum_d(n);
        s1 = warp_sum_d(s1);
        s2 = warp_sum_d(s2);
        if (lane == 0) {
            double *slot = u.ring + (static_cast<int64_t>(pol) * u.W + (u.t0 + b) % u.W) * 3;
            slot[0] = n;
            slot[1] = s1;
            slot[2] = s2;
        }
    }
    __syncthreads();
    if (!u.update) return;  // uniform over the CTA
    if (wq == 0) {
        const int64_t T = u.t0 + u.nb, lo = T - u.W > 0 ? T - u.W : 0;
        double n = 0.0, s1 = 0.0, s2 = 0.0;
        for (int64_t t = lo + lane; t < T; t += 32) {
            const double *slot = u.ring + (static_cast<int64_t>(pol) * u.W + t % u.W) * 3;
            n += slot[0];
            s1 += slot[1];
            s2 += slot[2];
        }
        n = warp_sum_d(n);
        s1 = warp_sum_d(s1);
        s2 = warp_sum_d(s2);
        if (lane == 0) {
            const double mean = s1 / n;
            th_s[pol] = static_cast<float>(sqrt((s2 - s1 * mean) / (n - 1.0)));
            off_s[pol] = static_cast<float>(mean);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float *t = u.thr;
        t[4] = th_s[0];
        t[5] = th_s[1];
        t[6] = off_s[0];
        t[7] = off_s[1];
        t[0] = th_s[0];
        t[1] = u.pol1 ? th_s[0] : th_s[1];
        t[2] = off_s[0];
        t[3] = u.pol1 ? off_s[0] : off_s[1];
    }
}

// quantize2bit over float chunks: each thread packs 16 samples into one word.
// grid (n_chunks*2048/256, 2 pols).
__global__ void k_quantize_chunks(const float *__restrict__ fin, int64_t fin_pol_stride, int64_t n_words,
                                  const float *__restrict__ thr, uint8_t *__restrict__ out, int64_t out_pol_stride,
                                  int64_t pkt_stride, int64_t payload_off, int64_t pkt0) {
    const int64_t w = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (w >= n_words) return;
    const int pol = blockIdx.y;
    const float th = thr[pol], off = thr[2 + pol];
    const float4 *src = reinterpret_cast<const float4 *>(fin + pol * fin_pol_stride + w * 16);
    uint32_t word = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 v = __ldcs(src + i);
        word |= code2(v.x, th, off) << (8 * i);
        word |= code2(v.y, th, off) << (8 * i + 2);
        word |= code2(v.z, th, off) << (8 * i + 4);
        word |= code2(v.w, th, off) << (8 * i + 6);
    }
    const int64_t c = w / kOutWords, k = w % kOutWords;
    uint32_t *dst = reinterpret_cast<uint32_t *>(out + pol * out_pol_stride + (pkt0 + c) * pkt_stride + payload_off);
    dst[k] = word;
}

// Reference-signature quantize2bit: contiguous in/out, scalar threshold.
__global__ void k_quantize_flat(const float *__restrict__ in, uint32_t *__restrict__ out, int64_t n_words, float th,
                                float off) {
    const int64_t w = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (w >= n_words) return;
    const float4 *src = reinterpret_cast<const float4 *>(in + w * 16);
    uint32_t word = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 v = __ldg(src + i);
        word |= code2(v.x, th, off) << (8 * i);
        word |= code2(v.y, th, off) << (8 * i + 2);
        word |= code2(v.z, th, off) << (8 * i + 4);
        word |= code2(v.w, th, off) << (8 * i + 6);
    }
    out[w] = word;
}

// Per-block FP64 sums for summary statistics over n floats, of the samples
// shifted by the first one (x - in[0]): a large common offset then cancels
// before the sums, not in the variance (the shifted-data algorithm; the
// finalizers add in[0] back to the mean).  A thread's sums are unevaluated
// FP32 ones (Shifted2; FP64 every 1024 samples): with four FP64 instructions a sample the kernel took
// 27 us for 2^22 samples that 3 us would read.  A batch of 1.1 million samples
// is 14 a thread: all loaded at once, and the block's sums turned into FP64
// once (block_moments), took another 4 us off a call.
// shift (optional) receives in[0].
__global__ void __launch_bounds__(256) k_stats_partial(const float *__restrict__ in, int64_t n,
                                                       double *__restrict__ partials, double *__restrict__ shift) {
    __shared__ double red[64];
    const float c = __ldg(in);
    Shifted2 m;
    const int64_t step = static_cast<int64_t>(gridDim.x) * blockDim.x;
    constexpr int U = 16;
    int group = 0;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += U * step) {
        float v[U];
        if (++group % 64 == 0) m.flush();  // at most 1024 samples in FP32 sums
        const int left = static_cast<int>(min(static_cast<int64_t>(U), (n - i + step - 1) / step));
#pragma unroll
        for (int k = 0; k < U; ++k)
            if (k < left) v[k] = __ldg(in + i + k * step);
#pragma unroll
        for (int k = 0; k < U; ++k)
            if (k < left) m.add(v[k], c);
    }
    double s1, s2;
    block_moments<8>(m.m, s1, s2, reinterpret_cast<float *>(red));
    if (__syncthreads_or(m.wide)) {
        block_sum2(m.fs, m.fq, red);
        s1 += m.fs;
        s2 += m.fq;
    }
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x] = s1;
        partials[2 * blockIdx.x + 1] = s2;
        if (shift != nullptr && blockIdx.x == 0) *shift = static_cast<double>(c);
    }
}

// ---------------------------------------------------------------------------
// Twiddle tables, FP64 on the host then rounded to FP32.
cudaError_t build_twiddles(Twiddles &tw, float2 **storage) {
    const int sizes[4] = {kMA, kMB, kMA, kMB + 1};
    const double periods[4] = {double(kMA), double(kMB), double(kNA), double(kNB)};
    size_t total = 0;
    for (int i = 0; i < 4; ++i) total += sizes[i];
    std::vector<float2> host(total);
    size_t off = 0;
    size_t offs[4];
    for (int t = 0; t < 4; ++t) {
        offs[t] = off;
        for (int k = 0; k < sizes[t]; ++k) {
            const double a = -2.0 * M_PI * static_cast<double>(k) / periods[t];
            host[off + k] = make_float2(static_cast<float>(std::cos(a)), static_cast<float>(std::sin(a)));
        }
        off += sizes[t];
    }
    float2 *d = nullptr;
    cudaError_t e = cudaMalloc(&d, total * sizeof(float2));
    if (e != cudaSuccess) return e;
    e = cudaMemcpy(d, host.data(), total * sizeof(float2), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        cudaFree(d);
        return e;
    }
    tw.w16384 = d + offs[0];
    tw.w18304 = d + offs[1];
    tw.w32768 = d + offs[2];
    tw.w36608 = d + offs[3];
    *storage = d;
    return cudaSuccess;
}

cudaError_t configure_fft_kernels() {
    cudaError_t e;
    if ((e = cudaFuncSetAttribute(k_swarm_c2r, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemA))) != cudaSuccess)
        return e;
    if ((e = cudaFuncSetAttribute(k_resample<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemPipeB))) != cudaSuccess)
        return e;
    if ((e = cudaFuncSetAttribute(k_resample<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemPipeB))) != cudaSuccess)
        return e;
    if ((e = cudaFuncSetAttribute(k_resample<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemPipeB))) != cudaSuccess)
        return e;
    if ((e = cudaFuncSetAttribute(k_resample<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemPipeB))) != cudaSuccess)
        return e;
    if ((e = cudaFuncSetAttribute(k_resample_once, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemB))) != cudaSuccess)
        return e;
    if ((e = cudaFuncSetAttribute(k_swarm_r2c, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemB))) != cudaSuccess)
        return e;
    if ((e = cudaFuncSetAttribute(k_r2dbe_c2r, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemB))) != cudaSuccess)
        return e;
    return cudaSuccess;
}

// Persistent grid size: one CTA per SM, at most `items`.
static unsigned persistent_grid(int64_t items) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) {
        cudaGetLastError();
        sms = 1;
    }
    return static_cast<unsigned>(items < sms ? items : sms);
}

// ---- launchers ----------------------------------------------------------------
cudaError_t launch_swarm_c2r_segs(const SegsA &S, const Twiddles &tw, cudaStream_t st) {
    if (S.n_items <= 0) return cudaSuccess;
    if (S.n < 1 || S.n > kMaxSegs) return cudaErrorInvalidValue;
    k_swarm_c2r<<<persistent_grid(S.n_items), kNTA, kSmemA, st>>>(S, tw);
    return cudaGetLastError();
}

cudaError_t launch_resample_segs(int mode, const SegsB &S, const Twiddles &tw, cudaStream_t st) {
    if (S.n_items <= 0) return cudaSuccess;
    if (S.n < 1 || S.n > kMaxSegs) return cudaErrorInvalidValue;
    const unsigned grid = persistent_grid(S.n_items);
    if (mode == 0)
        k_resample<0><<<grid, kNTB, kSmemPipeB, st>>>(S, tw);
    else if (mode == 3)
        k_resample<3><<<grid, kNTB, kSmemPipeB, st>>>(S, tw);
    else if (mode == 1)
        k_resample<1><<<grid, kNTB, kSmemPipeB, st>>>(S, tw);
    else if (S.n == 1 && S.n_items <= 2 * static_cast<int64_t>(grid) && S.s[0].n_chunks == S.n_items)
        k_resample_once<<<static_cast<unsigned>(S.n_items), kNTB, kSmemB, st>>>(S.s[0].in, S.s[0].skip, S.s[0].o.fout, tw);
    else
        k_resample<2><<<grid, kNTB, kSmemPipeB, st>>>(S, tw);
    return cudaGetLastError();
}

cudaError_t launch_swarm_c2r(const uint32_t *spec, int64_t spec_pol_stride, int64_t snap0, int64_t n_snaps, int n_pols,
                             float *out, int64_t out_pol_stride, const Twiddles &tw, cudaStream_t st) {
    if (n_snaps <= 0) return cudaSuccess;
    SegsA S{};
    S.n = 1;
    S.n_items = n_snaps * n_pols;
    S.s[0] = SegA{spec, out, spec_pol_stride, snap0, n_snaps, out_pol_stride, 0};
    S.status.add(tw.status);
    return launch_swarm_c2r_segs(S, tw, st);
}

cudaError_t launch_resample(int mode, const float *in, int64_t in_pol_stride, int skip, int64_t n_chunks, int n_pols,
                            const ResampleOut &o, const Twiddles &tw, cudaStream_t st) {
    if (n_chunks <= 0) return cudaSuccess;
    SegsB S{};
    S.n = 1;
    S.n_items = n_chunks * n_pols;
    S.s[0] = SegB{in, in_pol_stride, 0, static_cast<int>(n_chunks), skip, o};
    S.status.add(tw.status);
    return launch_resample_segs(mode, S, tw, st);
}

cudaError_t launch_swarm_r2c(const float *in, int64_t n_chunks, void *out, const Twiddles &tw, cudaStream_t st) {
    if (n_chunks <= 0) return cudaSuccess;
    k_swarm_r2c<<<persistent_grid(n_chunks), kNTB, kSmemB, st>>>(in, n_chunks, static_cast<float2 *>(out), tw);
    return cudaGetLastError();
}

cudaError_t launch_r2dbe_c2r(const void *in, int64_t in_stride, int64_t n_chunks, int skip, float *out,
                             const Twiddles &tw, cudaStream_t st) {
    if (n_chunks <= 0) return cudaSuccess;
    k_r2dbe_c2r<<<persistent_grid(n_chunks), kNTB, kSmemB, st>>>(static_cast<const float2 *>(in), in_stride, n_chunks,
                                                                  skip, out, tw);
    return cudaGetLastError();
}

cudaError_t launch_window_update(const WinUpds &U, cudaStream_t st) {
    if (U.n <= 0) return cudaSuccess;
    if (U.n > kMaxSegs) return cudaErrorInvalidValue;
    k_window_update<<<U.n, 256, 0, st>>>(U);
    return cudaGetLastError();
}

cudaError_t launch_finalize_thresholds(const double *partials, int pol1_uses_pol0, float *thr_state,
                                       cudaStream_t st) {
    k_finalize_thresholds<<<1, 64, 0, st>>>(partials, pol1_uses_pol0, thr_state);
    return cudaGetLastError();
}

cudaError_t launch_quantize_chunks(const float *fin, int64_t fin_pol_stride, int64_t n_chunks, const float *thr,
                                   uint8_t *out, int64_t out_pol_stride, int64_t pkt_stride, int64_t payload_off,
                                   int64_t pkt0, cudaStream_t st) {
    const int64_t n_words = n_chunks * kOutWords;
    if (n_words <= 0) return cudaSuccess;
    dim3 grid(static_cast<unsigned>((n_words + 255) / 256), 2);
    k_quantize_chunks<<<grid, 256, 0, st>>>(fin, fin_pol_stride, n_words, thr, out, out_pol_stride, pkt_stride,
                                            payload_off, pkt0);
    return cudaGetLastError();
}

cudaError_t launch_quantize_flat(const float *in, uint32_t *out, int64_t n, float th, float off, cudaStream_t st) {
    const int64_t n_words = n / 16;
    if (n_words <= 0) return cudaSuccess;
    k_quantize_flat<<<static_cast<unsigned>((n_words + 255) / 256), 256, 0, st>>>(in, out, n_words, th, off);
    return cudaGetLastError();
}

int stats_partial_blocks(int64_t n) {
    int64_t b = (n + 255) / 256;
    return static_cast<int>(b < 304 ? (b < 1 ? 1 : b) : 304);  // two a SM: few FP64 sums at the end
}

cudaError_t launch_stats_partial(const float *in, int64_t n, double *partials, double *shift, int blocks,
                                 cudaStream_t st) {
    k_stats_partial<<<blocks, 256, 0, st>>>(in, n, partials, shift);
    return cudaGetLastError();
}

}  // namespace sdbe
