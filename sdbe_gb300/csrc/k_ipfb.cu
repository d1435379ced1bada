// Inverse polyphase filter bank for PFB-mode SWARM spectra: Shaw's
// least-squares inversion, the method of
// software/prototyping/cuda/pfb_inverse.cu:213-488.
//
// The forward PFB (pfb_inverse.cu:173-207) maps ntap consecutive time blocks
// x_i..x_{i+ntap-1} of L = 32768 samples to the spectrum S_i whose C2R is
// y_i[p] = sum_t w[t*L + p] x_{i+t}[p] (w: Hamming over ntap*L, :51-53).  For
// each phase p that is y[:, p] = P_p x[:, p] with P_p banded (nblock x
// nblock+ntap-1); the inverse is x = P^T (P P^T)^-1 y, P P^T symmetric banded
// Toeplitz with a[d] = sum_k w[(k+d)L + p] w[kL + p].
//
// GB300 layout: the pseudo time stream comes from the complex-input C2R
// kernel (one CTA per snapshot, smem-resident 16384-point transform); the
// solve runs one thread per phase p, all of a block's phases reading
// consecutive words of each row (coalesced), walking the rows in FP64: the
// matrices are ill-conditioned (condition ~3e5 at 128 blocks, growing with
// the square of the block count), so FP32 elimination would lose the answer.
// LDL^T factor rows are formed on the fly in the forward sweep (no division
// but one per row) and streamed to scratch with the forward-substituted
// values; the backward sweep reads them once, and emits x_{m+ntap-1} as soon
// as z_m is known (the projection P^T z fused in).
//
// The factor depends on ntap and the row only, not on the spectra, and row m
// is the same for any number of blocks above m.  FP64 instructions (64 cycles
// a warp here) bound the solve, and forming the factor anew was two thirds of
// them, so the handle keeps it, as it keeps the window's table: k_ipfb_factor
// forms it once for the largest call so far (up to kPlanBlocks rows), and
// k_ipfb_apply does the two substitutions.  Calls of more blocks, or without room
// for it, form the factor as they go.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "handle.cuh"

namespace sdbe {

// scr layout: [nblock][NT][L]: entries 0..NT-2 = L[m][m-1-k], entry NT-1 = v_m.
template <int NT>
__global__ void __launch_bounds__(128) k_ipfb_solve(const float *__restrict__ y, int64_t nblock, double scale,
                                                    const double *__restrict__ tab, double *__restrict__ scr,
                                                    float *__restrict__ out) {
    constexpr int B = NT - 1;
    constexpr int L = kNA;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= L) return;
    double a[NT], w[NT];
#pragma unroll
    for (int d = 0; d < NT; ++d) {
        a[d] = tab[d * L + p];
        w[d] = tab[(NT + d) * L + p];
    }
    // rows m-1..m-B of the factorisation: pl[k-1][q-1] = L[m-k][m-k-q], pd = d, pdi = 1/d, pw = forward values
    double pl[B][B], pd[B], pdi[B], pw[B];
#pragma unroll
    for (int k = 0; k < B; ++k) {
        pd[k] = 1.0;
        pdi[k] = 0.0;
        pw[k] = 0.0;
#pragma unroll
        for (int q = 0; q < B; ++q) pl[k][q] = 0.0;
    }
    for (int64_t m = 0; m < nblock; ++m) {
        double l[B];  // l[k-1] = L[m][m-k]
#pragma unroll
        for (int k = B; k >= 1; --k) {
            double s = a[k];
#pragma unroll
            for (int q = k + 1; q <= B; ++q) s -= l[q - 1] * pd[q - 1] * pl[k - 1][q - k - 1];
            l[k - 1] = m - k >= 0 ? s * pdi[k - 1] : 0.0;
        }
        double dm = a[0], wm = static_cast<double>(__ldg(y + m * L + p)) * scale;
#pragma unroll
        for (int k = 1; k <= B; ++k) {
            dm -= l[k - 1] * l[k - 1] * pd[k - 1];
            wm -= l[k - 1] * pw[k - 1];
        }
        const double dinv = 1.0 / dm;
        double *row = scr + m * NT * L + p;
#pragma unroll
        for (int k = 0; k < B; ++k) row[k * L] = l[k];
        row[B * L] = wm * dinv;
#pragma unroll
        for (int k = B - 1; k >= 1; --k) {
            pd[k] = pd[k - 1];
            pdi[k] = pdi[k - 1];
            pw[k] = pw[k - 1];
#pragma unroll
            for (int q = 0; q < B; ++q) pl[k][q] = pl[k - 1][q];
        }
        pd[0] = dm;
        pdi[0] = dinv;
        pw[0] = wm;
#pragma unroll
        for (int q = 0; q < B; ++q) pl[0][q] = l[q];
    }
    // backward sweep: z_m = v_m - sum_k L[m+k][m] z_{m+k}; rows m+1..m+B held in nl/nz
    double nl[B][B], nz[B];  // nl[k-1][q-1] = L[m+k][m+k-q]
#pragma unroll
    for (int k = 0; k < B; ++k) {
        nz[k] = 0.0;
#pragma unroll
        for (int q = 0; q < B; ++q) nl[k][q] = 0.0;
    }
    for (int64_t m = nblock - 1; m >= 0; --m) {
        const double *row = scr + m * NT * L + p;
        double z = row[B * L];
#pragma unroll
        for (int k = 1; k <= B; ++k) z -= nl[k - 1][k - 1] * nz[k - 1];
        // x_{m+B} = sum_t w[t] z_{m+B-t}, t = 0..B  (z_{m..m+B} known)
        double x = w[B] * z;
#pragma unroll
        for (int t = 0; t < B; ++t) x += w[t] * nz[B - 1 - t];
        out[(m + B) * L + p] = static_cast<float>(x);
#pragma unroll
        for (int k = B - 1; k >= 1; --k) {
            nz[k] = nz[k - 1];
#pragma unroll
            for (int q = 0; q < B; ++q) nl[k][q] = nl[k - 1][q];
        }
        nz[0] = z;
#pragma unroll
        for (int q = 0; q < B; ++q) nl[0][q] = row[q * L];
    }
    // x_j for j = B-1 .. 0: z_0..z_{B-1} are nz[0..B-1]
#pragma unroll
    for (int j = B - 1; j >= 0; --j) {
        double x = 0.0;
#pragma unroll
        for (int t = 0; t <= j; ++t) x += w[t] * nz[j - t];
        out[j * L + p] = static_cast<float>(x);
    }
}

// fac layout: [nblock][NT][L]: entries 0..NT-2 = L[m][m-1-k], entry NT-1 = 1/d_m.
template <int NT>
__global__ void __launch_bounds__(128) k_ipfb_factor(int64_t nblock, double *__restrict__ tab,
                                                     double *__restrict__ fac) {
    constexpr int B = NT - 1;
    constexpr int L = kNA;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    double a[NT];
#pragma unroll
    for (int d = 0; d < NT; ++d) a[d] = tab[d * L + p];
    // The backward sweep runs on z w_c, c the middle tap (0.5 and above, but for
    // two taps' 0.08): scaled in the factor's 1/d, and the projection's tap c is 1.
    const double wc = tab[(NT + NT / 2) * L + p], wci = 1.0 / wc;
#pragma unroll
    for (int d = 0; d < NT; ++d) tab[(2 * NT + d) * L + p] = tab[(NT + d) * L + p] * wci;
    double pl[B][B], pd[B], pdi[B];  // as in k_ipfb_solve
#pragma unroll
    for (int k = 0; k < B; ++k) {
        pd[k] = 1.0;
        pdi[k] = 0.0;
#pragma unroll
        for (int q = 0; q < B; ++q) pl[k][q] = 0.0;
    }
    for (int64_t m = 0; m < nblock; ++m) {
        double l[B];
#pragma unroll
        for (int k = B; k >= 1; --k) {
            double s = a[k];
#pragma unroll
            for (int q = k + 1; q <= B; ++q) s -= l[q - 1] * pd[q - 1] * pl[k - 1][q - k - 1];
            l[k - 1] = m - k >= 0 ? s * pdi[k - 1] : 0.0;
        }
        double dm = a[0];
#pragma unroll
        for (int k = 1; k <= B; ++k) dm -= l[k - 1] * l[k - 1] * pd[k - 1];
        const double dinv = 1.0 / dm;
        double *row = fac + m * NT * L + p;
#pragma unroll
        for (int k = 0; k < B; ++k) row[k * L] = l[k];
        row[B * L] = dinv * wc;
#pragma unroll
        for (int k = B - 1; k >= 1; --k) {
            pd[k] = pd[k - 1];
            pdi[k] = pdi[k - 1];
#pragma unroll
            for (int q = 0; q < B; ++q) pl[k][q] = pl[k - 1][q];
        }
        pd[0] = dm;
        pdi[0] = dinv;
#pragma unroll
        for (int q = 0; q < B; ++q) pl[0][q] = l[q];
    }
}

// The conversions as instructions; functions, so that no FP64 instruction of
// theirs is issued, predicated off, in the ordinary case (three of 14 a row).
__device__ __noinline__ double scaled_f64_instr(float y) { return static_cast<double>(y) * (1.0 / kNA); }
__device__ __noinline__ float rounded_f32_instr(double x) { return static_cast<float>(x); }

// y / 32768 in FP64, exactly; the conversion by integer operations (a
// conversion instruction takes as long as an FP64 one) but for zeros,
// denormals, infinities and NaN.
__device__ __forceinline__ double scaled_f64(float y) {
    const uint32_t u = __float_as_uint(y), e = (u >> 23) & 255u;
    if (e == 0u || e == 255u) return scaled_f64_instr(y);
    const uint32_t hi = (u & 0x80000000u) | (((u & 0x7FFFFFFFu) >> 3) + ((896u - 15u) << 20));
    return __hiloint2double(static_cast<int>(hi), static_cast<int>(u << 29));
}

// x in FP32, rounded to nearest even by integer operations where the result is
// a normal number (as scaled_f64).
__device__ __forceinline__ float rounded_f32(double x) {
    const uint32_t hi = static_cast<uint32_t>(__double2hiint(x)), lo = static_cast<uint32_t>(__double2loint(x));
    const uint32_t e = (hi >> 20) & 2047u;
    if (e - 897u > 252u) return rounded_f32_instr(x);  // below FP32's normal numbers, or at its last binade or above
    const uint32_t mag = ((hi & 0x7FFFFFFFu) - (896u << 20)) << 3 | lo >> 29;
    const uint32_t up = (lo & 0x1FFFFFFFu) + 0x0FFFFFFFu + (mag & 1u);  // carries into bit 29 where it rounds up
    return __uint_as_float((hi & 0x80000000u) | (mag + (up >> 29)));
}

// Rows of k_ipfb_apply in flight (a power of two): two rows 72.7, four 67.7,
// eight 68.3, sixteen 71.8 us a call of 48 blocks, caches cold.
constexpr int kRing = 4;
// Asynchronous copies to shared memory that only the issuing thread reads.
__device__ __forceinline__ void copy_async8(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy_async4(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() {  // all but the last N groups have landed
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Forward and backward substitution with a kept factor; v: [nblock][L] scratch.
// One warp per CTA, so that 1024 warps leave no sub-partition with more than
// two.  FP64 issue (64 cycles a warp instruction, 10 for a row of four taps) is
// the bound, if a row's values are there: four instructions of the forward
// sweep are a fraction of a trip to DRAM, so kRing rows are on their way.  48
// blocks, four taps: 60.8 us with one row ahead and 14 FP64 instructions a row,
// 38.0 with 11 (two warps' instructions take 33.4); a tap of 1 in the
// projection takes one more away (the call 50.1 -> 48.2 us).
template <int NT>
__global__ void __launch_bounds__(32) k_ipfb_apply(const float *__restrict__ y, int64_t nblock,
                                                   const double *__restrict__ tab, const double *__restrict__ fac,
                                                   double *__restrict__ v, float *__restrict__ out) {
    static_assert(kNA == 1 << 15, "scaled_f64 divides by 2^15");
    constexpr int B = NT - 1;
    constexpr int L = kNA;
    __shared__ double ring[kRing][NT][32];
    __shared__ float yring[kRing][32];
    const int lane = threadIdx.x, p = blockIdx.x * 32 + lane;
    double w[NT];
#pragma unroll
    for (int d = 0; d < NT; ++d) w[d] = d == NT / 2 ? 1.0 : tab[(2 * NT + d) * L + p];
    double pw[B];
#pragma unroll
    for (int k = 0; k < B; ++k) pw[k] = 0.0;
    auto forward_row = [&](int64_t m) {
        if (m < nblock) {
            const int s = static_cast<int>(m) & (kRing - 1);
            copy_async4(&yring[s][lane], y + m * L + p);
#pragma unroll
            for (int k = 0; k < NT; ++k) copy_async8(&ring[s][k][lane], fac + (m * NT + k) * L + p);
        }
        copy_commit();
    };
    for (int i = 0; i < kRing; ++i) forward_row(i);
    for (int64_t m = 0; m < nblock; ++m) {
        copy_wait<kRing - 1>();
        const int s = static_cast<int>(m) & (kRing - 1);
        double wm = scaled_f64(yring[s][lane]), l[NT];
#pragma unroll
        for (int k = 0; k < NT; ++k) l[k] = ring[s][k][lane];
        forward_row(m + kRing);
#pragma unroll
        for (int k = 1; k <= B; ++k) wm -= l[k - 1] * pw[k - 1];
        v[m * L + p] = wm * l[B];
#pragma unroll
        for (int k = B - 1; k >= 1; --k) pw[k] = pw[k - 1];
        pw[0] = wm;
    }
    double nl[B][B], nz[B];  // as in k_ipfb_solve
#pragma unroll
    for (int k = 0; k < B; ++k) {
        nz[k] = 0.0;
#pragma unroll
        for (int q = 0; q < B; ++q) nl[k][q] = 0.0;
    }
    auto backward_row = [&](int64_t m) {
        if (m >= 0) {
            const int s = static_cast<int>(m) & (kRing - 1);
#pragma unroll
            for (int k = 0; k < B; ++k) copy_async8(&ring[s][k][lane], fac + (m * NT + k) * L + p);
        }
        copy_commit();
    };
    for (int i = 1; i <= kRing; ++i) backward_row(nblock - i);
    double vm = v[(nblock - 1) * L + p];
    for (int64_t m = nblock - 1; m >= 0; --m) {
        copy_wait<kRing - 1>();
        const int s = static_cast<int>(m) & (kRing - 1);
        double z = vm, l[B];
#pragma unroll
        for (int k = 0; k < B; ++k) l[k] = ring[s][k][lane];
        backward_row(m - kRing);
        if (m > 0) vm = v[(m - 1) * L + p];
#pragma unroll
        for (int k = 1; k <= B; ++k) z -= nl[k - 1][k - 1] * nz[k - 1];
        // x_{m+B} = sum_t w[t] z_{m+B-t}, t = 0..B  (z_{m..m+B} known)
        // (w[NT / 2] is 1, and z_m itself for two taps)
        constexpr int c = NT / 2;
        double x = c == B ? z : nz[B - 1 - c];
#pragma unroll
        for (int t = 0; t < B; ++t)
            if (t != c) x += w[t] * nz[B - 1 - t];
        if constexpr (c != B) x += w[B] * z;
        out[(m + B) * L + p] = rounded_f32(x);
#pragma unroll
        for (int k = B - 1; k >= 1; --k) {
            nz[k] = nz[k - 1];
#pragma unroll
            for (int q = 0; q < B; ++q) nl[k][q] = nl[k - 1][q];
        }
        nz[0] = z;
#pragma unroll
        for (int q = 0; q < B; ++q) nl[0][q] = l[q];
    }
    // x_j for j = B-1 .. 0: z_0..z_{B-1} are nz[0..B-1]
#pragma unroll
    for (int j = B - 1; j >= 0; --j) {
        double x = 0.0;
#pragma unroll
        for (int t = 0; t <= j; ++t) x += w[t] * nz[j - t];
        out[j * L + p] = static_cast<float>(x);
    }
}

namespace {

// Host table per ntap: a[d][p] (band of P P^T) and w[t][p] (P taps), FP64.
std::vector<double> ipfb_table(int ntap) {
    const int L = kNA;
    const double m = static_cast<double>(ntap) * L;
    std::vector<double> win(static_cast<size_t>(ntap) * L);
    for (int64_t n = 0; n < static_cast<int64_t>(win.size()); ++n)
        win[n] = 0.54 - 0.46 * std::cos(2.0 * 3.14159265358979323846 * static_cast<double>(n) / (m - 1.0));
    std::vector<double> tab(static_cast<size_t>(2) * ntap * L);
    for (int d = 0; d < ntap; ++d)
        for (int p = 0; p < L; ++p) {
            double s = 0.0;
            for (int k = 0; k < ntap - d; ++k) s += win[static_cast<size_t>(k + d) * L + p] * win[static_cast<size_t>(k) * L + p];
            tab[static_cast<size_t>(d) * L + p] = s;
            tab[static_cast<size_t>(ntap + d) * L + p] = win[static_cast<size_t>(d) * L + p];
        }
    return tab;
}

// Calls of more blocks than this form the factor as they go (k_ipfb_solve):
// their factor would hold over 4 GB beside the scratch, and is read from HBM.
constexpr int64_t kPlanBlocks = 4096;

template <int NT>
cudaError_t launch_solve(const float *y, int64_t nblock, const double *tab, double *scr, float *out, cudaStream_t st) {
    k_ipfb_solve<NT><<<kNA / 128, 128, 0, st>>>(y, nblock, 1.0 / kNA, tab, scr, out);
    return cudaGetLastError();
}
template <int NT>
cudaError_t launch_factor(int64_t nblock, double *tab, double *fac, cudaStream_t st) {
    k_ipfb_factor<NT><<<kNA / 128, 128, 0, st>>>(nblock, tab, fac);
    return cudaGetLastError();
}
template <int NT>
cudaError_t launch_apply(const float *y, int64_t nblock, const double *tab, const double *fac, double *v, float *out,
                         cudaStream_t st) {
    k_ipfb_apply<NT><<<kNA / 32, 32, 0, st>>>(y, nblock, tab, fac, v, out);
    return cudaGetLastError();
}

// f(integral_constant<int, ntap>) for 2 <= ntap <= 8.
template <class F>
cudaError_t with_taps(int ntap, F f) {
    switch (ntap) {
        case 2: return f(std::integral_constant<int, 2>{});
        case 3: return f(std::integral_constant<int, 3>{});
        case 4: return f(std::integral_constant<int, 4>{});
        case 5: return f(std::integral_constant<int, 5>{});
        case 6: return f(std::integral_constant<int, 6>{});
        case 7: return f(std::integral_constant<int, 7>{});
        default: return f(std::integral_constant<int, 8>{});
    }
}

// Room for at least `need` bytes, `want` if there is so much; a larger buffer
// replaces the old one after all work on the device.
bool make_room(uint8_t **buf, int64_t *cap, int64_t want, int64_t need) {
    if (*cap >= need) return true;
    if (*buf && cudaDeviceSynchronize() != cudaSuccess) return false;
    cudaFree(*buf);
    *buf = nullptr;
    *cap = 0;
    for (const int64_t bytes : {want > need ? want : need, need}) {
        if (cudaMalloc(buf, static_cast<size_t>(bytes)) == cudaSuccess) {
            *cap = bytes;
            return true;
        }
        cudaGetLastError();
        *buf = nullptr;
    }
    return false;
}

void drop_factor(sdbe_resampler *h) {
    if (h->ipfb_fac || h->ipfb_v) cudaDeviceSynchronize();
    cudaFree(h->ipfb_fac);
    cudaFree(h->ipfb_v);
    h->ipfb_fac = h->ipfb_v = nullptr;
    h->ipfb_fac_bytes = h->ipfb_v_bytes = 0;
    h->ipfb_rows = 0;
}

}  // namespace
}  // namespace sdbe

using namespace sdbe;

extern "C" int sdbe_inverse_pfb(sdbe_resampler *h, const void *spec_c64, int64_t nblock, int32_t ntap, float *out,
                                void *stream) {
    if (!h || nblock < 1 || ntap < 2 || ntap > 8 || !spec_c64 || !out) return fail(h, SDBE_ERR_ARG, "bad argument");
    if (reinterpret_cast<uintptr_t>(spec_c64) & 7u)  // read as float2
        return fail(h, SDBE_ERR_ARG, "complex spectra must be 8-byte aligned");
    if (nblock > (int64_t(1) << 20)) return fail(h, SDBE_ERR_CAPACITY, "at most 2^20 blocks per call");
    DeviceGuard g(h->cfg.device);
    if (!g.ok) return fail(h, SDBE_ERR_CUDA, "cudaSetDevice failed");
    if (int rc = check_status(h)) return rc;
    cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : h->stream;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    SDBE_CK(h, cudaStreamIsCapturing(st, &cap));
    const bool capturing = cap != cudaStreamCaptureStatusNone;
    constexpr int64_t kRowF = kNA * static_cast<int64_t>(sizeof(float)), kRowD = 2 * kRowF;
    if (h->ipfb_ntap != ntap) {
        const std::vector<double> tab = ipfb_table(ntap);
        if (h->ipfb_tab) SDBE_CK(h, cudaDeviceSynchronize());
        h->ipfb_ntap = 0;
        h->ipfb_rows = 0;
        if (!h->ipfb_tab) SDBE_CK(h, cudaMalloc(&h->ipfb_tab, 3 * 8 * kRowD));  // of eight taps
        SDBE_CK(h, cudaMemcpyAsync(h->ipfb_tab, tab.data(), tab.size() * sizeof(double), cudaMemcpyHostToDevice, st));
        SDBE_CK(h, cudaStreamSynchronize(st));  // tab is freed on return
        h->ipfb_ntap = ntap;
    }
    // Scratch owned by the handle, grown to the largest call so far and by
    // doubling.  What a captured call uses is replaced only where its y is (a
    // larger call) or its table (other taps): the factor and the substituted
    // values are laid out for as many rows as y has, and calls without the
    // factor have scratch of their own.  Where memory is short, or the stream
    // is being captured and there is no room yet, a call forms its factor as it
    // goes, which takes 8 nblock rows less.
    const int64_t have = h->ipfb_y_bytes / kRowF;
    const int64_t twice = nblock > kPlanBlocks ? nblock : std::min(2 * have, kPlanBlocks);
    bool room = make_room(&h->ipfb_y, &h->ipfb_y_bytes, twice * kRowF, nblock * kRowF);
    if (!room) {
        if (!capturing) drop_factor(h);
        if (int rc = grow(h, &h->ipfb_y, &h->ipfb_y_bytes, nblock * kRowF, "the inverse PFB scratch")) return rc;
    }
    float *y = reinterpret_cast<float *>(h->ipfb_y);
    const int64_t rows = std::min(h->ipfb_y_bytes / kRowF, kPlanBlocks);
    bool plan = nblock <= kPlanBlocks;
    if (plan && capturing) {
        plan = h->ipfb_v_bytes >= nblock * kRowD && h->ipfb_fac_bytes >= nblock * ntap * kRowD;
    } else if (plan) {
        if (h->ipfb_fac_bytes < nblock * ntap * kRowD) h->ipfb_rows = 0;
        plan = make_room(&h->ipfb_v, &h->ipfb_v_bytes, rows * kRowD, nblock * kRowD) &&
               make_room(&h->ipfb_fac, &h->ipfb_fac_bytes, rows * ntap * kRowD, nblock * ntap * kRowD);
        if (!plan) drop_factor(h);
    }
    double *fac = reinterpret_cast<double *>(h->ipfb_fac), *v = reinterpret_cast<double *>(h->ipfb_v);
    if (!plan) {
        const int64_t need = nblock * ntap * kRowD;
        if (!make_room(&h->ipfb_scr, &h->ipfb_scr_bytes, need, need)) {
            if (!capturing) drop_factor(h);
            if (int rc = grow(h, &h->ipfb_scr, &h->ipfb_scr_bytes, need, "the inverse PFB scratch")) return rc;
        }
        fac = v = reinterpret_cast<double *>(h->ipfb_scr);
    } else if (h->ipfb_rows < nblock) {
        // rows formed before are formed again, with the same values
        const int64_t form = capturing ? nblock
                                       : std::max(nblock, std::min(2 * h->ipfb_rows, h->ipfb_fac_bytes / (ntap * kRowD)));
        SDBE_CK(h, with_taps(ntap, [&](auto nt) { return launch_factor<decltype(nt)::value>(form, h->ipfb_tab, fac, st); }));
        h->launches += 1;
        if (!capturing) {  // (a captured call forms its rows in each replay)
            SDBE_CK(h, cudaStreamSynchronize(st));  // later calls, on any stream, find them complete
            h->ipfb_rows = form;
        }
    }
    cudaError_t e = cudaSuccess;
    if (h->cfg.precision != SDBE_PRECISION_FP32) {
        // the pseudo time stream on the tensor cores
        if (int rc = tc_c2r_spectra(h, static_cast<const float2 *>(spec_c64), kMA + 1, nblock,
                                    reinterpret_cast<float2 *>(v), y, st))
            return rc;
    } else {
        e = launch_r2dbe_c2r(spec_c64, kMA + 1, nblock, 0, y, h->tw, st);
    }
    if (e == cudaSuccess)
        e = with_taps(ntap, [&](auto nt) {
            constexpr int NT = decltype(nt)::value;
            return plan ? launch_apply<NT>(y, nblock, h->ipfb_tab, fac, v, out, st)
                        : launch_solve<NT>(y, nblock, h->ipfb_tab, fac, out, st);
        });
    if (e != cudaSuccess) return fail(h, SDBE_ERR_CUDA, std::string("inverse_pfb: ") + cudaGetErrorString(e));
    h->launches += 2;
    return SDBE_OK;
}
