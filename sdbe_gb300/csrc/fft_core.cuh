// Register-resident DFT codelets and shared-memory helpers for the
// Stockham FFT passes of the resampling kernels.
//
// A pass of radix R over an N-point sequence held in shared memory
// (Stockham autosort, natural order in and out):
//   for butterfly j < N/R:  v[r] = x[j + r*N/R]
//                           v[r] *= W_{Ns*R}^{(j mod Ns)*r}
//                           v = DFT_R(v)
//                           y[(j/Ns)*Ns*R + (j mod Ns) + r*Ns] = v[r]
// with Ns the product of the radices of the earlier passes.  The first pass
// therefore reads with stride N/R (coalesced straight from global memory)
// and the last pass writes with stride N/R (coalesced straight to global).
#pragma once

#include "sdbe_internal.cuh"

namespace sdbe {

// Padded shared-memory index: one float2 of padding per 32 elements keeps
// the stride-16/32 accesses of the passes free of bank conflicts.
__device__ __forceinline__ int pad(int a) { return a + (a >> 5); }
constexpr int padded_len(int n) { return n + (n >> 5) + 1; }

// cos(2 pi m / 32) for integer m; constant-folds when m is a compile-time value.
__device__ __forceinline__ float cos32(int m) {
    m &= 31;
    constexpr float t[9] = {1.0f, 0.98078528040323043f, 0.92387953251128674f,
                            0.83146961230254524f, 0.70710678118654757f, 0.55557023301960229f,
                            0.38268343236508984f, 0.19509032201612833f, 0.0f};
    if (m <= 8) return t[m];
    if (m <= 16) return -t[16 - m];
    if (m <= 24) return -t[m - 16];
    return t[32 - m];
}
__device__ __forceinline__ float sin32(int m) { return cos32(m - 8); }

// a * W_32^m, W_32 = exp(-2 pi i / 32) (forward) or its conjugate (inverse).
template <bool INV>
__device__ __forceinline__ float2 mul_w32(float2 a, int m) {
    m &= 31;
    if (m == 0) return a;
    if (m == 16) return make_float2(-a.x, -a.y);
    if (m == 8) return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
    if (m == 24) return INV ? make_float2(a.y, -a.x) : make_float2(-a.y, a.x);
    const float c = cos32(m);
    const float s = INV ? sin32(m) : -sin32(m);
    return make_float2(a.x * c - a.y * s, a.x * s + a.y * c);
}

__host__ __device__ constexpr int ilog2c(int n) { return n <= 1 ? 0 : 1 + ilog2c(n >> 1); }
__host__ __device__ constexpr int bitrev(int x, int bits) {
    int r = 0;
    for (int b = 0; b < bits; ++b) r |= ((x >> b) & 1) << (bits - 1 - b);
    return r;
}

// In-register power-of-two DFT (R <= 32), natural order in and out:
// bit-reversal by register renaming, then radix-2 decimation-in-time stages.
template <int R, bool INV>
__device__ __forceinline__ void dft_pow2(float2 *v) {
    constexpr int B = ilog2c(R);
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int j = bitrev(i, B);
        if (i < j) {
            const float2 t = v[i];
            v[i] = v[j];
            v[j] = t;
        }
    }
#pragma unroll
    for (int half = 1; half < R; half <<= 1) {
#pragma unroll
        for (int i = 0; i < R; i += 2 * half) {
#pragma unroll
            for (int k = 0; k < half; ++k) {
                const float2 b = mul_w32<INV>(v[i + k + half], k * (32 / (2 * half)));
                const float2 a = v[i + k];
                v[i + k] = cadd(a, b);
                v[i + k + half] = csub(a, b);
            }
        }
    }
}

// cos/sin(2 pi m / P) tables for the odd prime radices.
template <int P>
struct OddConst;
template <>
struct OddConst<11> {
    __device__ static __forceinline__ float c(int m) {
        constexpr float t[6] = {1.0f, 0.84125353283118121f, 0.41541501300188644f, -0.142314838273285f,
                                -0.65486073394528499f, -0.95949297361449737f};
        return t[m];
    }
    __device__ static __forceinline__ float s(int m) {
        constexpr float t[6] = {0.0f, 0.54064081745559756f, 0.90963199535451833f, 0.9898214418809328f,
                                0.75574957435425827f, 0.28173255684142967f};
        return t[m];
    }
};
template <>
struct OddConst<13> {
    __device__ static __forceinline__ float c(int m) {
        constexpr float t[7] = {1.0f, 0.88545602565320991f, 0.56806474673115592f, 0.12053668025532301f,
                                -0.35460488704253545f, -0.74851074817110119f, -0.97094181742605201f};
        return t[m];
    }
    __device__ static __forceinline__ float s(int m) {
        constexpr float t[7] = {0.0f, 0.46472317204376851f, 0.82298386589365635f, 0.99270887409805397f,
                                0.93501624268541483f, 0.66312265824079519f, 0.23931566428755768f};
        return t[m];
    }
};

// Odd prime DFT by conjugate-pair symmetry: with s_j = v_j + v_{P-j},
// d_j = v_j - v_{P-j}, A_k = v_0 + sum s_j cos(2 pi jk/P),
// B_k = sum d_j sin(2 pi jk/P):  y_k = A_k -+ i B_k, y_{P-k} = A_k +- i B_k.
template <int P, bool INV>
__device__ __forceinline__ void dft_odd(float2 *v) {
    constexpr int H = (P - 1) / 2;
    float2 s[H + 1], d[H + 1];
#pragma unroll
    for (int j = 1; j <= H; ++j) {
        s[j] = cadd(v[j], v[P - j]);
        d[j] = csub(v[j], v[P - j]);
    }
    float2 y0 = v[0];
#pragma unroll
    for (int j = 1; j <= H; ++j) y0 = cadd(y0, s[j]);
    float2 out[P];
    out[0] = y0;
#pragma unroll
    for (int k = 1; k <= H; ++k) {
        float2 A = v[0];
        float2 Bv = make_float2(0.f, 0.f);
#pragma unroll
        for (int j = 1; j <= H; ++j) {
            int m = (j * k) % P;
            float cs, sn;
            if (m <= H) {
                cs = OddConst<P>::c(m);
                sn = OddConst<P>::s(m);
            } else {
                cs = OddConst<P>::c(P - m);
                sn = -OddConst<P>::s(P - m);
            }
            A.x = fmaf(s[j].x, cs, A.x);
            A.y = fmaf(s[j].y, cs, A.y);
            Bv.x = fmaf(d[j].x, sn, Bv.x);
            Bv.y = fmaf(d[j].y, sn, Bv.y);
        }
        // forward: y_k = A - i B = (A.x + B.y, A.y - B.x)
        if (!INV) {
            out[k] = make_float2(A.x + Bv.y, A.y - Bv.x);
            out[P - k] = make_float2(A.x - Bv.y, A.y + Bv.x);
        } else {
            out[k] = make_float2(A.x - Bv.y, A.y + Bv.x);
            out[P - k] = make_float2(A.x + Bv.y, A.y - Bv.x);
        }
    }
#pragma unroll
    for (int k = 0; k < P; ++k) v[k] = out[k];
}

template <int R, bool INV>
__device__ __forceinline__ void dft(float2 *v) {
    if constexpr (R == 11 || R == 13) {
        dft_odd<R, INV>(v);
    } else {
        dft_pow2<R, INV>(v);
    }
}

// ---- compile-time twiddle constants ---------------------------------------
// sin/cos of 2*pi*num/den in double at compile time: exact integer reduction
// to a quadrant, then Taylor series on |x| <= pi/4 (error < 1e-16).
constexpr double kPi = 3.141592653589793238462643383279502884;
__host__ __device__ constexpr double cx_sin_small(double x) {
    double x2 = x * x, term = x, sum = x;
    for (int k = 1; k < 14; ++k) {
        term *= -x2 / ((2.0 * k) * (2.0 * k + 1.0));
        sum += term;
    }
    return sum;
}
__host__ __device__ constexpr double cx_cos_small(double x) {
    double x2 = x * x, term = 1.0, sum = 1.0;
    for (int k = 1; k < 14; ++k) {
        term *= -x2 / ((2.0 * k - 1.0) * (2.0 * k));
        sum += term;
    }
    return sum;
}
// Returns {cos, sin} of 2*pi*num/den.
struct CS {
    double c, s;
};
__host__ __device__ constexpr CS cx_cossin_2pi(long long num, long long den) {
    long long m = num % den;
    if (m < 0) m += den;
    // 8m/den in [0, 8): octant index q = round(4m/den) in [0, 4], remainder t in [-1/2, 1/2]
    const long long q4 = (8 * m + den) / (2 * den);       // nearest quarter-turn
    const double t = (4.0 * static_cast<double>(m) - static_cast<double>(q4) * static_cast<double>(den)) /
                     static_cast<double>(den);          // fraction of a quarter-turn
    const double x = t * (kPi / 2.0);
    const double sx = cx_sin_small(x), cxv = cx_cos_small(x);
    switch (q4 & 3) {
        case 0: return CS{cxv, sx};
        case 1: return CS{-sx, cxv};
        case 2: return CS{-cxv, -sx};
        default: return CS{sx, -cxv};
    }
}
// W_N^E = exp(-2 pi i E/N) rounded to float, usable as device constants.
template <long long N, long long E>
struct TwC {
    static constexpr CS v = cx_cossin_2pi(E, N);
    static constexpr float c = static_cast<float>(v.c);
    static constexpr float s = static_cast<float>(-v.s);
};
// a * W_N^E (or a * conj(W_N^E) when CONJ) with E a compile-time value.
template <long long N, long long E, bool CONJ>
__device__ __forceinline__ float2 mul_tc(float2 a) {
    constexpr float c = TwC<N, E>::c;
    constexpr float s = CONJ ? -TwC<N, E>::s : TwC<N, E>::s;
    if constexpr (E % N == 0) {
        return a;
    } else {
        return make_float2(a.x * c - a.y * s, a.x * s + a.y * c);
    }
}

// Padded index of the small shared-memory twiddle tables.
__device__ __forceinline__ int tp(int m) { return m + (m >> 4); }
constexpr int tp_len(int n) { return n + ((n - 1) >> 4) + 1; }

// W_N^e from the two-level tables H[a] = W_N^{128 a}, L[b] = W_N^b.
__device__ __forceinline__ float2 tw2(const float2 *H, const float2 *L, int e) {
    return cmul(H[tp(e >> 7)], L[tp(e & 127)]);
}

// Table twiddle W_N^e (forward) or its conjugate (inverse).
template <bool INV>
__device__ __forceinline__ float2 twiddle(const float2 *__restrict__ tab, int e) {
    const float2 w = __ldg(tab + e);
    return INV ? make_float2(w.x, -w.y) : w;
}

// ---- 2-bit requantization (quantize2bit, vdif_inout_gpu_thread.cu:577) ----
__device__ __forceinline__ uint32_t code2(float x, float th, float off) {
    const float v = x - off;
    return ((static_cast<uint32_t>(fabsf(v) >= th) | 2u) ^ (3u * static_cast<uint32_t>(v < 0.f))) & 3u;
}

// code2 for many samples into packed words, with two shifts a sample instead
// of comparisons, selects and logic (the pipe that runs these has half the
// FMA pipe's rate, which the rest of a transform keeps busy).  With v = x -
// off and d = |v| - th, the code's high bit is v >= 0 and its low bit (d >= 0)
// ^ (v < 0); push2 shifts the two sign bits into the word from below, so the
// sample pushed last ends up lowest, and codes2 turns the 16 pairs of a full
// word into codes.  Adding +0 makes v = -0 count as v >= 0; coder2 stands in
// finite values for a NaN threshold (no sample reaches it) or offset (v >= 0
// and below the threshold), so that no NaN reaches a sign bit.
struct Coder2 {
    float th, off;
};
__device__ __forceinline__ Coder2 coder2(float th, float off) {
    constexpr float kBig = 3.402823466e38f;
    const bool nan_off = off != off;
    if (th != th || nan_off) {
        th = __int_as_float(0x7F800000);
        off = nan_off ? -kBig : fminf(fmaxf(off, -kBig), kBig);
    }
    return Coder2{th, off};
}
__device__ __forceinline__ void push2(uint32_t &w, float x, Coder2 c) {
    const float v = (x - c.off) + 0.f;
    w = __funnelshift_l(__float_as_uint(v), w, 1);
    w = __funnelshift_l(__float_as_uint(fabsf(v) - c.th), w, 1);
}
__device__ __forceinline__ uint32_t codes2(uint32_t w) { return ~(w ^ ((w >> 1) & 0x55555555u)); }

// 8 x 8 transpose of 4-bit nibbles over the aligned groups of 8 lanes: on
// return, nibble r of lane c is nibble c of lane r (c = lane & 7).  Step m
// (1, 2, 4) swaps, between lanes c and c ^ m, the nibbles whose index bit m
// differs from the lane's own bit m.
__device__ __forceinline__ uint32_t nib_transpose8(uint32_t x, int c) {
    constexpr uint32_t kKeep[3] = {0x0F0F0F0Fu, 0x00FF00FFu, 0x0000FFFFu};  // nibbles with index bit m clear
#pragma unroll
    for (int s = 0; s < 3; ++s) {
        const int m = 1 << s, sh = 4 << s;
        const uint32_t y = __shfl_xor_sync(0xffffffffu, x, m);
        x = (c & m) ? ((x & ~kKeep[s]) | ((y >> sh) & kKeep[s])) : ((x & kKeep[s]) | ((y << sh) & ~kKeep[s]));
    }
    return x;
}

// ---- block reductions -------------------------------------------------------
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Per-thread FP32 sums a, b reduced in FP32 within each warp and in FP64
// across warps; results valid in thread 0.  scratch >= 2*32 doubles.
__device__ __forceinline__ void block_sum2_f(float a, float b, double &sa, double &sb, double *scratch) {
    a = warp_sum_f(a);
    b = warp_sum_f(b);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nw = (blockDim.x + 31) >> 5;
    __syncthreads();
    if (lane == 0) {
        scratch[warp] = a;
        scratch[32 + warp] = b;
    }
    __syncthreads();
    sa = 0.0;
    sb = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < nw; ++w) {
            sa += scratch[w];
            sb += scratch[32 + w];
        }
}

// Sums a and b over the block; result valid in thread 0.  scratch >= 2*32 doubles.
__device__ __forceinline__ void block_sum2(double &a, double &b, double *scratch) {
    a = warp_sum(a);
    b = warp_sum(b);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nw = (blockDim.x + 31) >> 5;
    __syncthreads();
    if (lane == 0) {
        scratch[warp] = a;
        scratch[32 + warp] = b;
    }
    __syncthreads();
    if (warp == 0) {
        a = warp_sum(lane < nw ? scratch[lane] : 0.0);
        b = warp_sum(lane < nw ? scratch[32 + lane] : 0.0);
    }
}

// One thread's sum and sum of squares of FP32 samples as unevaluated sums of
// FP32 values (Knuth's two-sum; a square is its rounded value plus the exact
// fma remainder), handed on in FP64: FP64 instructions, conversions included,
// run at 1/64 of the FP32 rate, and seven of them for two samples took 28k of
// a first-batch chunk's 65k cycles.  Three levels each (72 bits) leave
// every sum of up to 1024 samples nearer to the exact one than FP64 sums do:
// emulated over constants, uniform, Gaussian (offset by 1000 spreads too) and
// log-normal samples, 64 to 1024 of them, no error in FP64's last place against
// 5e-15 for FP64 sums.  Two levels for the sum, the form before, were off by
// 5e-14 (64 log-normal samples) to 1.5e-12 (1024).  Past some thousand samples
// the last level's own rounding shows (a constant's squares: 1e-13 at 14,000).
struct Moments2 {
    float s = 0.f, se = 0.f, sf = 0.f, q = 0.f, qe = 0.f, qf = 0.f;
    static __device__ __forceinline__ float two_sum(float &a, float x) {  // a += x, returns the rounding error
        const float t = __fadd_rn(a, x), z = __fsub_rn(t, a);
        const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(t, z)), __fsub_rn(x, z));
        a = t;
        return e;
    }
    __device__ __forceinline__ void add(float x) {
        sf = __fadd_rn(sf, two_sum(se, two_sum(s, x)));
        const float p = __fmul_rn(x, x);
        const float e = two_sum(q, p);
        qf = __fadd_rn(qf, two_sum(qe, e));
        qf = __fadd_rn(qf, two_sum(qe, __fmaf_rn(x, x, -p)));
    }
    __device__ __forceinline__ double sum() const {
        return static_cast<double>(s) + (static_cast<double>(se) + static_cast<double>(sf));
    }
    __device__ __forceinline__ double squares() const {
        return static_cast<double>(q) + (static_cast<double>(qe) + static_cast<double>(qf));
    }
};

// The same of samples less c.  x - c is its rounded value dh plus the exact
// remainder dl, and (dh + dl)^2 = dh^2 + 2 dh dl + dl^2 with the products'
// remainders.  Samples whose squares would leave FP32's range one way or the
// other (and infinities and NaN) go to FP64 sums directly; flush() moves the
// FP32 sums there, which a thread does every 1024 samples.
struct Shifted2 {
    Moments2 m;
    double fs = 0.0, fq = 0.0;
    bool wide = false;  // fs and fq hold something
    __device__ __forceinline__ void flush() {
        fs += m.sum();
        fq += m.squares();
        m = Moments2{};
        wide = true;
    }
    __device__ __forceinline__ void add(float x, float c) {
        const float dh0 = __fsub_rn(x, c);
        if (!(fabsf(dh0) < 1e12f) || (fabsf(dh0) < 1e-10f && dh0 != 0.f)) {
            const double v = static_cast<double>(x) - static_cast<double>(c);
            fs += v;
            fq += v * v;
            wide = true;
            return;
        }
        float dh = x;
        const float dl = Moments2::two_sum(dh, -c);
        const float g = Moments2::two_sum(m.se, Moments2::two_sum(m.s, dh));
        m.sf = __fadd_rn(m.sf, __fadd_rn(g, Moments2::two_sum(m.se, dl)));
        const float p = __fmul_rn(dh, dh), cr = __fmul_rn(2.f * dh, dl);
        const float e = Moments2::two_sum(m.q, p);
        float f = __fadd_rn(Moments2::two_sum(m.qe, e), Moments2::two_sum(m.qe, __fmaf_rn(dh, dh, -p)));
        f = __fadd_rn(f, Moments2::two_sum(m.qe, cr));
        f = __fadd_rn(f, __fmaf_rn(dl, dl, __fmaf_rn(2.f * dh, dl, -cr)));
        m.qf = __fadd_rn(m.qf, f);
    }
};

// An unevaluated sum a + b + c of FP32 values, merged across lanes and warps
// before it is turned into FP64: the conversions and the shuffle trees of all
// warps in FP64 took 20 instructions a warp at 76 cycles each.
struct Sum3 {
    float a, b, c;
    __device__ __forceinline__ void merge(float oa, float ob, float oc) {
        const float e = Moments2::two_sum(a, oa);
        const float f = Moments2::two_sum(b, ob);
        c = __fadd_rn(__fadd_rn(c, oc), __fadd_rn(f, Moments2::two_sum(b, e)));
    }
    template <int N>
    __device__ __forceinline__ void merge_lanes() {  // over N lanes
#pragma unroll
        for (int m = N / 2; m > 0; m >>= 1) {
            const float oa = __shfl_xor_sync(0xffffffffu, a, m), ob = __shfl_xor_sync(0xffffffffu, b, m),
                        oc = __shfl_xor_sync(0xffffffffu, c, m);
            merge(oa, ob, oc);
        }
    }
    __device__ __forceinline__ double value() const {
        return static_cast<double>(a) + (static_cast<double>(b) + static_cast<double>(c));
    }
};

// The sums of m over a block of NW full warps (a power of two <= 16); result
// valid in warp 0.  scratch: 6 * 16 floats.
template <int NW>
__device__ __forceinline__ void block_moments(const Moments2 &m, double &s1, double &s2, float *scratch) {
    Sum3 s{m.s, m.se, m.sf}, q{m.q, m.qe, m.qf};
    s.merge_lanes<32>();
    q.merge_lanes<32>();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) {
        const float v[6] = {s.a, s.b, s.c, q.a, q.b, q.c};
#pragma unroll
        for (int k = 0; k < 6; ++k) scratch[16 * k + warp] = v[k];
    }
    __syncthreads();
    if (warp == 0) {
        const float *p = scratch + (lane & (NW - 1));
        s = Sum3{p[0], p[16], p[32]};
        q = Sum3{p[48], p[64], p[80]};
        s.merge_lanes<NW>();
        q.merge_lanes<NW>();
        s1 = s.value();
        s2 = q.value();
    }
}

// Packed nibble k -> (real, imag) = codes - 2.  A 2-bit code c placed in the
// mantissa of 1.5 * 2^23 gives the float 12582912 + c exactly; subtracting
// 12582914 leaves c - 2 (one logic op and one add, no int-to-float convert).
// The real code stays where it is, at bits 2-3, under the exponent that gives
// those bits the weights 1 and 2 (1.5 * 2^21): one shift fewer, on a pipe that
// runs at half the FMA pipe's rate (stage A 6.81 -> 6.54 us a snapshot and SM).
__device__ __forceinline__ float2 nib_value(const uint32_t *sp, int k) {
    const uint32_t w = sp[k >> 3] >> ((k & 7) * 4);
    const float re = __uint_as_float(0x4A400000u | (w & 12u)) - 3145730.0f;
    const float im = __uint_as_float(0x4B400000u | (w & 3u)) - 12582914.0f;
    return make_float2(re, im);
}

// Hermitian pair of a length-32768 C2R input: from Y[k], Y[M-k] (M = 16384)
// and we = e^{+2 pi i k/32768},
//   Z[k]   = (Y[k] + conj Y[M-k]) + i we (Y[k] - conj Y[M-k]) =: e + i t
//   Z[M-k] = conj(e) + i conj(t),
// so one complex multiply serves both.
__device__ __forceinline__ void c2r_pair(float2 y, float2 ym, float2 we, float2 &zk, float2 &zmk) {
    const float2 e = make_float2(y.x + ym.x, y.y - ym.y);
    const float2 t = cmul(make_float2(y.x - ym.x, y.y + ym.y), we);
    zk = make_float2(e.x - t.y, e.y + t.x);
    zmk = make_float2(e.x + t.y, t.x - e.y);
}

// c2r_pair with the product's rounding pinned (cmul_rn).
template <int X, int Y>
__device__ __forceinline__ void c2r_pair_rn(float2 y, float2 ym, float2 we, float2 &zk, float2 &zmk) {
    const float2 e = make_float2(y.x + ym.x, y.y - ym.y);
    const float2 t = cmul_rn<X, Y>(make_float2(y.x - ym.x, y.y + ym.y), we);
    zk = make_float2(e.x - t.y, e.y + t.x);
    zmk = make_float2(e.x + t.y, t.x - e.y);
}

// Hermitian pair of a length-36608 R2C output: from Z[q], Z[M'-q] (M' = 18304)
// and w = e^{-2 pi i q/36608}, with s = Z[q] + conj Z[M'-q], t = w (Z[q] - conj Z[M'-q]):
//   X[q] = (s - i t)/2,   X[M'-q] = (conj(s) - i conj(t))/2.
__device__ __forceinline__ void r2c_pair(float2 za, float2 zb, float2 w, float2 &xq, float2 &xmq) {
    const float2 s = make_float2(za.x + zb.x, za.y - zb.y);
    const float2 t = cmul(w, make_float2(za.x - zb.x, za.y + zb.y));
    xq = make_float2(0.5f * (s.x + t.y), 0.5f * (s.y - t.x));
    xmq = make_float2(0.5f * (s.x - t.y), -0.5f * (s.y + t.x));
}


}  // namespace sdbe
