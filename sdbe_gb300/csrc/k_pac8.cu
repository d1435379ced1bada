// Ingest transforms on the device: 8pac unpack (software/aphids/vdif_8pac.c)
// and the B-engine header reform (software/aphids/beng_reform.c), the
// receive-side pre-pass of vdif_in_net_thread.c:291-298.
#include <cuda_runtime.h>

#include "handle.cuh"

namespace sdbe {

constexpr int kPktU64 = kPktBytes / 8;                        // 132
constexpr int32_t kClkPerSec = 286000000;                     // SWARM_CLK_PER_SEC
constexpr int32_t kBframeClk = 262144;                        // SWARM_BFRAME_CLK
constexpr int32_t kClkTol = 1024;                             // BFRAME_CLK_TOL
constexpr int64_t kMaxOffset = 1000;                          // MAX_COUNTABLE_BFRAME_OFFSET
constexpr int kReformThreads = 1024;

static_assert(sizeof(sdbe_reform_state) == 48, "reform state layout");

// ---------------------------------------------------------------------------
// 8pac unpack: one warp per output packet, 8-byte words (the packets inside a
// unit sit at 8-byte but not 16-byte offsets: 0, then 1064*k).  The header
// words the reference rewrites (vdif_8pac.c:5-41) are fixed in registers.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_unpack_8pac(const uint8_t *__restrict__ src, int64_t n_units,
                                                     uint8_t *__restrict__ dst) {
    const int64_t pkt = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (pkt >= n_units * 8) return;
    const int64_t unit = pkt >> 3;
    const int k = static_cast<int>(pkt & 7);
    const uint8_t *u = src + unit * kPac8Bytes;
    const uint64_t *s = reinterpret_cast<const uint64_t *>(u + 1064 * k);
    uint64_t *d = reinterpret_cast<uint64_t *>(dst + pkt * kPktBytes);
    for (int i = lane; i < kPktU64; i += 32) {
        uint64_t v = __ldcs(s + i);
        if (i < 4) {
            const uint32_t *h1 = reinterpret_cast<const uint32_t *>(u);
            uint32_t lo = static_cast<uint32_t>(v), hi = static_cast<uint32_t>(v >> 32);
            if (i == 0) {
                if (k) lo = (lo & 0x7FFFFFFFu) | (__ldg(h1) & 0x80000000u);                  // fix_8pac_flags
                hi = (hi & 0xFF000000u) | ((8u * (__ldg(h1 + 1) & 0xFFFFFFu) + k) & 0xFFFFFFu);  // data frame
            } else if (i == 1) {
                const int len = static_cast<int>(__ldg(h1 + 2) & 0xFFFFFFu) - 7;               // reset_8pac_size
                lo = (lo & 0xFF000000u) | (static_cast<uint32_t>(len / 8) & 0xFFFFFFu);
            } else if (i == 3) {
                const uint64_t psn = (static_cast<uint64_t>(__ldg(h1 + 7)) << 32) | __ldg(h1 + 6);
                const uint64_t p = 8ull * psn + static_cast<uint64_t>(k);                     // fix_8pac_psn
                lo = static_cast<uint32_t>(p);
                hi = static_cast<uint32_t>(p >> 32);
            }
            v = (static_cast<uint64_t>(hi) << 32) | lo;
        }
        __stcs(d + i, v);
    }
}

// ---------------------------------------------------------------------------
// Header reform.  The reference walks the packets in order with a state of
// T0, TPREV and BPREV; each valid packet's count is BPREV plus the B-frames
// from TPREV to its timestamp, found by stepping one frame at a time with a
// 1024-clock tolerance (beng_reform.c:34-104, 137-186).
//
// One CTA walks tiles of 1024 packets.  When every valid packet of a tile and
// its predecessor have clk < 286e6 and lie a whole number k of frames apart
// with |k| <= 1000, stepping returns exactly k (each step adds 262144 clocks
// to the absolute time and lands on the other timestamp), so the counts are
// BPREV plus a prefix sum: computed with block scans.  Any other pair (jitter,
// corrupt clocks) is stepped by its own thread, bounded by the cap.  A packet
// beyond the cap becomes invalid, which changes its successor's predecessor:
// such a tile is summed by one thread, which steps that pair anew.  So results
// match the reference in all cases.  (With one thread stepping every pair of a
// tile with jitter, 2048 packets took 218 us; 44 now, 155 with a jump.)
//
// Walking the tiles one after another takes 3.9 us a tile, most of it latency
// (1122 us for the 292,864 packets of a group).  The usual batch is regular
// throughout, and then each count is simply BPREV plus the B-frames from TPREV
// to the packet's own timestamp: k_reform_check looks at every pair of
// neighbouring valid packets, all tiles at once, and k_beng_reform then
// rewrites the headers a tile per CTA; one CTA walks only if a pair was
// irregular (or the batch is shorter than kReformWalk packets, where the other
// launch costs as much as two tiles).  Whole calls by the walk /
// with the check: 4096 packets 46.0 / 44.4 us, 8192 59.2 / 44.2, a group 1188 /
// 143; the check costs an irregular batch 12 us.
// ---------------------------------------------------------------------------
struct Ts {
    int32_t sec, clk;
};

__device__ __forceinline__ Ts read_ts(uint32_t w4, uint32_t w5) {
    const int64_t b = (static_cast<int64_t>(w4) << 21) | static_cast<int64_t>((w5 >> 11) & 0x1FFFFFu);
    return Ts{static_cast<int32_t>((b & 0x001FFFFFE0000000ll) >> 29), static_cast<int32_t>(b & 0x1FFFFFFFll)};
}

__device__ int ts_compare(Ts then, Ts now) {  // _beng_timestamp_compare_then_now, as written
    if (then.sec < now.sec) {
        if (then.sec == now.sec - 1 && then.clk + kClkTol > kClkPerSec && (then.clk + kClkTol) % kClkPerSec >= now.clk)
            return 0;
        return -1;
    }
    if (then.sec > now.sec) {
        if (now.clk + kClkTol > kClkPerSec && (now.clk + kClkTol) % kClkPerSec >= then.clk) return 0;
        return 1;
    }
    if (then.clk + kClkTol < now.clk) return -1;
    if (now.clk + kClkTol < then.clk) return 1;
    return 0;
}

__device__ Ts ts_increment(Ts t) {
    t.clk += kBframeClk;
    if (t.clk > kClkPerSec) {
        t.sec += 1;
        t.clk %= kClkPerSec;
    }
    return t;
}

__device__ int64_t ts_offset(Ts then, Ts now) {  // at most kMaxOffset + 1 steps
    const int cmp = ts_compare(then, now);
    if (cmp == 0) return 0;
    Ts start = cmp < 0 ? then : now;
    const Ts end = cmp < 0 ? now : then;
    const int64_t step = cmp < 0 ? 1 : -1;
    int64_t off = 0;
    while (ts_compare(start, end) < 0) {
        start = ts_increment(start);
        off += step;
        if (off > kMaxOffset || -off > kMaxOffset) break;
    }
    return off;
}

__device__ __forceinline__ void write_old_header(uint32_t *w, uint32_t w5, int32_t off) {
    const uint32_t c = w5 & 0xFFu, f = (w5 >> 8) & 7u, o = static_cast<uint32_t>(off);
    w[5] = (w5 & 0x0000FF00u) | c | (f << 16) | ((o & 0xFFu) << 24);
    w[4] = (o & 0x7FFFFF00u) >> 8;
}

template <class T, class Op>
__device__ T block_scan_inclusive(T v, T *warp_tot, Op op, T identity) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T u = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o) v = op(u, v);
    }
    if (lane == 31) warp_tot[warp] = v;
    __syncthreads();
    if (warp == 0) {
        T t = warp_tot[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const T u = __shfl_up_sync(0xFFFFFFFFu, t, o);
            if (lane >= o) t = op(u, t);
        }
        warp_tot[lane] = t;
    }
    __syncthreads();
    const T before = warp ? warp_tot[warp - 1] : identity;
    const T r = op(before, v);
    __syncthreads();  // warp_tot reusable
    return r;
}

struct MaxOp {
    __device__ int operator()(int a, int b) const { return a > b ? a : b; }
};
struct SumOp {
    __device__ long long operator()(long long a, long long b) const { return a + b; }
};

// What k_reform_check found besides the tiles with irregular pairs (a byte
// each, behind this): the timestamps of the batch's first and last valid
// packets, if there are none of those.
struct ReformInfo {
    Ts first, last;
};
constexpr int64_t kReformWalk = 4 * kReformThreads;
__host__ __device__ constexpr int64_t reform_tiles(int64_t n) { return (n + kReformThreads - 1) / kReformThreads; }

// Whole frames from p to ts within the stepping cap, both clocks in range.
__device__ __forceinline__ bool regular_step(Ts p, Ts ts) {
    const long long delta = static_cast<long long>(ts.sec - p.sec) * kClkPerSec + (ts.clk - p.clk);
    return ts.clk < kClkPerSec && p.clk < kClkPerSec && ts.clk >= 0 && p.clk >= 0 && delta % kBframeClk == 0 &&
           delta <= kMaxOffset * kBframeClk && -delta <= kMaxOffset * kBframeClk;
}

// One tile per CTA.  A valid packet's predecessor is the valid packet before
// it in the tile, or for the tile's first one the last valid packet of the
// 1024 before the tile, or the stream's state; where there is none of these
// (over 1024 invalid packets in a row) the batch counts as irregular.
__global__ void __launch_bounds__(kReformThreads) k_reform_check(const uint8_t *__restrict__ pkts, int64_t n,
                                                                 sdbe_reform_state in, ReformInfo *info) {
    uint8_t *bad = reinterpret_cast<uint8_t *>(info + 1);
    __shared__ Ts s_ts[kReformThreads];
    __shared__ int s_pv[kReformThreads];
    __shared__ int s_scan_i[32];
    __shared__ int s_back;
    __shared__ Ts s_prev;
    const int tid = threadIdx.x;
    const int64_t base = static_cast<int64_t>(blockIdx.x) * kReformThreads, i = base + tid;
    auto header = [&](int64_t j, Ts *ts) {
        const uint32_t *w = reinterpret_cast<const uint32_t *>(pkts + j * kPktBytes);
        *ts = read_ts(__ldg(w + 4), __ldg(w + 5));
        return (__ldg(w) >> 31) == 0u;
    };
    if (tid == 0) s_back = -1;
    Ts ts{0, 0}, bts{0, 0};
    const bool valid = i < n && header(i, &ts);
    const int64_t j = base - 1 - tid;  // the tile before, newest first
    const bool bvalid = j >= 0 && header(j, &bts);
    s_ts[tid] = ts;
    s_pv[tid] = block_scan_inclusive<int>(valid ? tid : -1, s_scan_i, MaxOp(), -1);
    // the newest valid packet of the tile before: the largest 1023 - tid
    if (bvalid) atomicMax(&s_back, kReformThreads - 1 - tid);
    __syncthreads();
    const int before = tid ? s_pv[tid - 1] : -1;
    const int last = s_pv[kReformThreads - 1];
    if (bvalid && s_back == kReformThreads - 1 - tid) s_prev = bts;
    __syncthreads();
    const bool unset = in.t0_sec == -1 && in.t0_clk == -1;
    bool ok = true;
    if (valid) {
        Ts p = ts;  // the stream's first valid packet is its own predecessor
        if (before >= 0)
            p = s_ts[before];
        else if (s_back >= 0)
            p = s_prev;
        else if (base >= kReformThreads)
            ok = false;  // nothing valid in the tile before: not looked at further
        else if (!unset)
            p = Ts{in.tprev_sec, in.tprev_clk};
        ok = ok && regular_step(p, ts);
        if (base == 0 && before < 0) info->first = ts;
    }
    // the batch's first and last valid packets lie in its first and last tiles
    if (tid == 0 && last < 0 && (base == 0 || base + kReformThreads >= n)) ok = false;
    if (base + kReformThreads >= n && tid == last) info->last = ts;
    const int irregular = __syncthreads_or(!ok);
    if (tid == 0) bad[blockIdx.x] = irregular != 0;
}

// This CTA's tile of a batch that is regular throughout.
__device__ __forceinline__ void reform_tile(uint8_t *pkts, int64_t n, const sdbe_reform_state &in,
                                            sdbe_reform_state *out, uint32_t *hdr, const ReformInfo *info) {
    const bool unset = in.t0_sec == -1 && in.t0_clk == -1;
    const Ts p = unset ? info->first : Ts{in.tprev_sec, in.tprev_clk};
    const long long bprev = unset ? 0 : in.bprev;
    auto count = [&](Ts ts) {
        const long long d = (static_cast<long long>(ts.sec - p.sec) * kClkPerSec + (ts.clk - p.clk)) / kBframeClk;
        return static_cast<int32_t>(static_cast<uint32_t>(static_cast<unsigned long long>(bprev + d)));
    };
    const int64_t i = static_cast<int64_t>(blockIdx.x) * kReformThreads + threadIdx.x;
    if (i < n) {
        uint32_t *w = reinterpret_cast<uint32_t *>(pkts + i * kPktBytes);
        const uint32_t w0 = w[0], w5 = w[5];
        if ((w0 >> 31) == 0u) write_old_header(w, w5, count(read_ts(w[4], w5)));
        if (hdr != nullptr) {
            hdr[3 * i] = w0;
            hdr[3 * i + 1] = w[4];
            hdr[3 * i + 2] = w[5];
        }
    }
    if (i == 0) {
        sdbe_reform_state s = in;
        if (unset) {
            s.t0_sec = info->first.sec;
            s.t0_clk = info->first.clk;
        }
        s.tprev_sec = info->last.sec;
        s.tprev_clk = info->last.clk;
        s.bprev = count(info->last);
        *out = s;
    }
}

__global__ void __launch_bounds__(kReformThreads) k_beng_reform(uint8_t *__restrict__ pkts, int64_t n,
                                                                sdbe_reform_state in, sdbe_reform_state *out,
                                                                uint32_t *__restrict__ hdr,
                                                                const ReformInfo *__restrict__ info) {
    if (info != nullptr) {
        const uint8_t *bad = reinterpret_cast<const uint8_t *>(info + 1);
        bool irregular = false;
        for (int64_t t = threadIdx.x; t < reform_tiles(n); t += kReformThreads) irregular |= bad[t] != 0;
        if (!__syncthreads_or(irregular)) {
            reform_tile(pkts, n, in, out, hdr, info);
            return;
        }
        if (blockIdx.x > 0) return;
    }
    __shared__ sdbe_reform_state s;
    __shared__ Ts s_ts[kReformThreads];
    __shared__ int s_pv[kReformThreads];
    __shared__ int32_t s_off[kReformThreads];
    __shared__ int s_first;
    __shared__ int s_scan_i[32];
    __shared__ long long s_scan_l[32];
    const int tid = threadIdx.x;
    if (tid == 0) s = in;
    for (int64_t base = 0; base < n; base += kReformThreads) {
        if (tid == 0) s_first = kReformThreads;
        __syncthreads();
        const int64_t i = base + tid;
        uint32_t *w = reinterpret_cast<uint32_t *>(pkts + i * kPktBytes);
        bool valid = false;
        uint32_t w5 = 0;
        Ts ts{0, 0};
        if (i < n) {
            valid = (w[0] >> 31) == 0u;
            w5 = w[5];
            ts = read_ts(w[4], w5);
        }
        s_ts[tid] = ts;
        if (valid) atomicMin(&s_first, tid);
        __syncthreads();
        if (tid == s_first && s.t0_sec == -1 && s.t0_clk == -1) {  // first valid packet of the stream
            s.t0_sec = s.tprev_sec = ts.sec;
            s.t0_clk = s.tprev_clk = ts.clk;
            s.bprev = 0;
        }
        // index of the previous valid packet in the tile (exclusive max scan)
        s_pv[tid] = block_scan_inclusive<int>(valid ? tid : -1, s_scan_i, MaxOp(), -1);
        __syncthreads();
        const int before = tid ? s_pv[tid - 1] : -1;
        const int last = s_pv[kReformThreads - 1];
        const Ts p = before >= 0 ? s_ts[before] : Ts{s.tprev_sec, s.tprev_clk};
        bool ok = true;
        long long d = 0;
        if (valid) {
            const long long delta = static_cast<long long>(ts.sec - p.sec) * kClkPerSec + (ts.clk - p.clk);
            const long long apart = delta < 0 ? -delta : delta;
            const bool clocks = ts.clk < kClkPerSec && p.clk < kClkPerSec && ts.clk >= 0 && p.clk >= 0;
            ok = clocks && delta % kBframeClk == 0 && apart <= kMaxOffset * kBframeClk;
            d = delta / kBframeClk;
            // an irregular pair is stepped by its own thread, unless it is surely
            // beyond the cap (which a pair that compares equal never is)
            if (!ok)
                d = clocks && apart > (kMaxOffset + 2) * kBframeClk && ts_compare(p, ts) != 0 ? kMaxOffset + 1
                                                                                             : ts_offset(p, ts);
        }
        // A valid packet's predecessor is the valid one before it, unless that
        // lies beyond the cap and becomes invalid: only then the tile is counted
        // packet by packet.
        const bool stepped = __syncthreads_or(valid && !ok) != 0;
        const bool slow = stepped && __syncthreads_or(valid && (d > kMaxOffset || -d > kMaxOffset)) != 0;
        if (!slow) {
            const long long sum = block_scan_inclusive<long long>(valid ? d : 0, s_scan_l, SumOp(), 0);
            const int32_t off = static_cast<int32_t>(static_cast<uint32_t>(static_cast<unsigned long long>(s.bprev + sum)));
            if (valid) write_old_header(w, w5, off);
            __syncthreads();  // everyone has read s.bprev
            if (tid == last) {
                s.tprev_sec = ts.sec;
                s.tprev_clk = ts.clk;
                s.bprev = off;
            }
            if (stepped && tid == 0) s.slow_tiles += 1;
        } else {
            s_off[tid] = static_cast<int32_t>(d);  // |d| <= kMaxOffset + 1
            __syncthreads();
            if (tid == 0) {
                const int end = static_cast<int>(n - base < kReformThreads ? n - base : kReformThreads);
                Ts prev{s.tprev_sec, s.tprev_clk};
                long long bprev = s.bprev;
                bool marked = false;  // the valid packet before
                for (int j = 0; j < end; ++j) {
                    if (s_pv[j] != j) continue;
                    const Ts now = s_ts[j];
                    int32_t off = marked ? static_cast<int32_t>(ts_offset(prev, now)) : s_off[j];
                    marked = off > kMaxOffset || off < -kMaxOffset;
                    if (marked) {
                        s_pv[j] = -1;
                        off = -1;
                        s.marked_invalid += 1;
                    } else {
                        off = static_cast<int32_t>(static_cast<uint32_t>(static_cast<unsigned long long>(off + bprev)));
                        prev = now;
                        bprev = off;
                    }
                    s_off[j] = off;
                }
                s.tprev_sec = prev.sec;
                s.tprev_clk = prev.clk;
                s.bprev = bprev;
                s.slow_tiles += 1;
            }
            __syncthreads();
            if (valid) {
                if (s_pv[tid] != tid) w[0] |= 0x80000000u;
                write_old_header(w, w5, s_off[tid]);
            }
        }
        __syncthreads();
        if (hdr != nullptr && i < n) {
            hdr[3 * i] = w[0];
            hdr[3 * i + 1] = w[4];
            hdr[3 * i + 2] = w[5];
        }
    }
    __syncthreads();
    if (tid == 0) *out = s;
}

// Header words (w0, w4, w5) of plain packets, for the host-side ingest policy.
__global__ void k_gather_headers(const uint8_t *__restrict__ pkts, int64_t n, uint32_t *__restrict__ hdr) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t *w = reinterpret_cast<const uint32_t *>(pkts + i * kPktBytes);
    hdr[3 * i] = __ldg(w);
    hdr[3 * i + 1] = __ldg(w + 4);
    hdr[3 * i + 2] = __ldg(w + 5);
}

cudaError_t launch_unpack_8pac(const void *src, int64_t n_units, void *dst, cudaStream_t st) {
    if (n_units <= 0) return cudaSuccess;
    const int64_t threads = n_units * 8 * 32;
    k_unpack_8pac<<<static_cast<unsigned>((threads + 255) / 256), 256, 0, st>>>(static_cast<const uint8_t *>(src),
                                                                               n_units, static_cast<uint8_t *>(dst));
    return cudaGetLastError();
}

// Device bytes: the state after a batch of n packets, then the check's findings.
int64_t reform_scratch(int64_t n) {
    return static_cast<int64_t>(sizeof(sdbe_reform_state) + sizeof(ReformInfo)) + reform_tiles(n);
}

// out_dev: reform_scratch(n) bytes.
cudaError_t launch_beng_reform(void *pkts, int64_t n, const sdbe_reform_state &in, sdbe_reform_state *out_dev,
                               uint32_t *hdr, cudaStream_t st) {
    uint8_t *p = static_cast<uint8_t *>(pkts);
    ReformInfo *info = nullptr;
    unsigned grid = 1;
    if (n >= kReformWalk) {
        info = reinterpret_cast<ReformInfo *>(out_dev + 1);
        grid = static_cast<unsigned>(reform_tiles(n));
        k_reform_check<<<grid, kReformThreads, 0, st>>>(p, n, in, info);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    k_beng_reform<<<grid, kReformThreads, 0, st>>>(p, n, in, out_dev, hdr, info);
    return cudaGetLastError();
}

cudaError_t launch_gather_headers(const void *pkts, int64_t n, uint32_t *hdr, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_gather_headers<<<static_cast<unsigned>((n + 255) / 256), 256, 0, st>>>(static_cast<const uint8_t *>(pkts), n,
                                                                            hdr);
    return cudaGetLastError();
}

}  // namespace sdbe

using namespace sdbe;

extern "C" {

int sdbe_reform_init(sdbe_reform_state *st) {
    if (!st) return SDBE_ERR_ARG;
    *st = sdbe_reform_state{};
    st->t0_sec = st->t0_clk = st->tprev_sec = st->tprev_clk = -1;
    st->bprev = -1;
    return SDBE_OK;
}

int sdbe_unpack_8pac(const void *src, int64_t n_units, void *dst, void *stream) {
    if (n_units < 0 || (n_units > 0 && (!src || !dst))) return fail(nullptr, SDBE_ERR_ARG, "bad argument");
    if ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 7u)
        return fail(nullptr, SDBE_ERR_ARG, "8pac buffers must be 8-byte aligned");
    SDBE_CK(nullptr, launch_unpack_8pac(src, n_units, dst, static_cast<cudaStream_t>(stream)));
    return SDBE_OK;
}

int sdbe_beng_reform(sdbe_reform_state *st, void *pkts, int64_t n_pkts, void *stream) {
    if (!st || n_pkts < 0 || (n_pkts > 0 && !pkts)) return fail(nullptr, SDBE_ERR_ARG, "bad argument");
    if (reinterpret_cast<uintptr_t>(pkts) & 3u) return fail(nullptr, SDBE_ERR_ARG, "packets must be 4-byte aligned");
    if (n_pkts == 0) return SDBE_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    void *scr = nullptr;  // this thread's reusable scratch: the call waits for its stream below
    SDBE_CK(nullptr, thread_scratch(static_cast<size_t>(reform_scratch(n_pkts)), &scr));
    sdbe_reform_state *dev = static_cast<sdbe_reform_state *>(scr);
    cudaError_t e = launch_beng_reform(pkts, n_pkts, *st, dev, nullptr, s);
    sdbe_reform_state out{};
    if (e == cudaSuccess) e = cudaMemcpyAsync(&out, dev, sizeof(out), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return fail(nullptr, SDBE_ERR_CUDA, std::string("beng_reform: ") + cudaGetErrorString(e));
    *st = out;
    return SDBE_OK;
}

}  // extern "C"
