// Internal declarations of libibs: error plumbing, the handle structs behind
// the C-ABI, and the device-side table lookup shared by every scan kernel.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/ibs.h"
#include "ibs_core.cuh"
#include "mz_core.cuh"
#include "wide_core.cuh"

namespace ibs {

// ---- errors ---------------------------------------------------------------
void set_error(const std::string &msg);
void clear_error();
std::atomic<uint64_t> &launch_counter();

// "CUDA error in <what>: <text>", the reference's message shape
// (src/gpu/EncodeProbe.cu:15-20).
ibs_status cuda_fail(cudaError_t e, const char *what);

#define IBS_CUDA(call, what)                                  \
    do {                                                      \
        cudaError_t e_ = (call);                              \
        if (e_ != cudaSuccess)                                \
            return ::ibs::cuda_fail(e_, what);                \
    } while (0)

// Device count check shared by the entry points.
ibs_status check_device_ordinal(int dev);
// Rows carry 32-bit window coordinates (ibs_window.start / end, the
// reference's int Window::start / end, src/Window.hpp:11-12), so a contig
// longer than INT32_MAX bases would print wrapped, negative coordinates:
// IBS_ERR_ARG with a message naming the contig instead.
ibs_status check_contig_lengths(const uint64_t *lens, uint32_t n, const char *what);
constexpr uint64_t kMaxContigLen = 2147483647ull;
// Decodes a KMC 3 database into canonical codes in device memory (caller
// frees). decode_kmc takes k <= 32 (one word per code); decode_kmc_any also
// takes 33 <= k <= 64, whose codes are two words each ({lo, hi}).
ibs_status decode_kmc(const char *prefix, int dev, uint64_t **dCodes, uint64_t *n, uint32_t *k);
ibs_status decode_kmc_any(const char *prefix, int dev, uint64_t **dCodes, uint64_t *n, uint32_t *k);
// Wide-key tables (ibs_wide.cu): the build from device codes ({lo, hi} per
// key; the device must be current), membership counts, and the release of
// the levels.
ibs_status build_wide(ibs_table *t, const ulonglong2 *dCodes, uint64_t n, uint32_t k, const ibs_table_opts *o);
ibs_status count_present_wide(ibs_table *t, const ulonglong2 *dCodes, uint64_t n, uint64_t *count);
void free_wide(ibs_table *t);
constexpr uint32_t kMaxWideK = 64;
// Packed base offset of each contig (roundup64 of the lengths before it) and
// the seq / mask word counts with their tail padding.
void packed_offsets(const uint64_t *lens, uint32_t n, std::vector<uint64_t> &off, uint64_t &seqWords,
                    uint64_t &maskWords);
// A reference around device arrays already in the packed layout; it takes
// ownership of dSeq / dMask (freed by ibs_reference_free, also on failure).
ibs_status reference_adopt(const std::vector<uint64_t> &lens, int device, uint64_t *dSeq, uint64_t *dMask,
                           ibs_reference **out);

#define IBS_LAUNCHED() (::ibs::launch_counter().fetch_add(1, std::memory_order_relaxed))

// RAII guard that makes `dev` current and restores the previous device.
struct DeviceGuard {
    int prev = -1;
    bool ok = false;
    explicit DeviceGuard(int dev)
    {
        if (cudaGetDevice(&prev) != cudaSuccess)
            prev = -1;
        ok = cudaSetDevice(dev) == cudaSuccess;
    }
    ~DeviceGuard()
    {
        if (prev >= 0)
            cudaSetDevice(prev);
    }
};

// ---- tuning -----------------------------------------------------------------
const ibs_tuning &tuning();

// ---- device table view ----------------------------------------------------
struct TableView {
    TableGeom g;
    const uint4 *buckets; // 2 x uint4 per bucket
    const uint64_t *stash;
};

#if defined(__CUDACC__)
__device__ __forceinline__ bool stash_lookup(const TableView &t, uint64_t code)
{
    if (t.g.stashBuckets == 0)
        return false;
    uint64_t b = stash_home(code, t.g.stashBuckets);
    for (uint64_t i = 0; i < t.g.stashBuckets; ++i) {
        const ulonglong2 *p = reinterpret_cast<const ulonglong2 *>(t.stash + 4 * b);
        const ulonglong2 a = __ldg(p), c = __ldg(p + 1);
        if (a.x == code || a.y == code || c.x == code || c.y == code)
            return true;
        if (a.x == STASH_EMPTY || a.y == STASH_EMPTY || c.x == STASH_EMPTY || c.y == STASH_EMPTY)
            return false;
        b = (b + 1) & (t.g.stashBuckets - 1);
    }
    return false;
}

// One bucket compare, given the bucket's two 16-byte halves. Returns 1 on a
// hit, 0 on a sure miss, 2 when the bucket overflowed into the stash.
template <uint32_t FMT>
__device__ __forceinline__ uint32_t bucket_match(const uint4 &v0, const uint4 &v1, uint64_t fp)
{
    if (FMT == FMT_B8X32) {
        const uint32_t f = (uint32_t)fp;
        const bool hit = (v0.x == f) | (v0.y == f) | (v0.z == f) | (v0.w == f) | (v1.x == f) |
                         (v1.y == f) | (v1.z == f) | (v1.w == f);
        return hit ? 1u : (v1.w == B8_OVERFLOW ? 2u : 0u);
    } else {
        const uint32_t qhi = (uint32_t)(fp >> 8), qlo = (uint32_t)(fp & 0xff);
        const uint32_t cnt = (v1.w >> 16) & 0xff;
        bool hit = false;
        hit |= (0 < cnt) & (v0.x == qhi) & ((v1.z & 0xff) == qlo);
        hit |= (1 < cnt) & (v0.y == qhi) & (((v1.z >> 8) & 0xff) == qlo);
        hit |= (2 < cnt) & (v0.z == qhi) & (((v1.z >> 16) & 0xff) == qlo);
        hit |= (3 < cnt) & (v0.w == qhi) & ((v1.z >> 24) == qlo);
        hit |= (4 < cnt) & (v1.x == qhi) & ((v1.w & 0xff) == qlo);
        hit |= (5 < cnt) & (v1.y == qhi) & (((v1.w >> 8) & 0xff) == qlo);
        return hit ? 1u : ((v1.w >> 24) & 1u ? 2u : 0u);
    }
}

// Whether a minimizer line's sector holds a slot value. B6x40: each slot's
// 32-bit half by one comparison and its byte by one masked difference; the
// slots past the count hold zeros, which only a slot value of zero can match.
template <uint32_t SEC>
__device__ __forceinline__ bool mz_sector_holds(const uint4 &v0, const uint4 &v1, uint32_t slot, uint32_t high)
{
    if (SEC == FMT_B8X32)
        return (v0.x == slot) | (v0.y == slot) | (v0.z == slot) | (v0.w == slot) | (v1.x == slot) | (v1.y == slot) |
               (v1.z == slot) | (v1.w == slot);
    const uint32_t qhi = __funnelshift_r(slot, high, 8), qlo = slot & 0xffu;
    const uint32_t rep = qlo * 0x01010101u, d0 = v1.z ^ rep, d1 = v1.w ^ rep;
    bool hit = v0.x == qhi && !(d0 & 0x000000ffu);
    hit |= v0.y == qhi && !(d0 & 0x0000ff00u);
    hit |= v0.z == qhi && !(d0 & 0x00ff0000u);
    hit |= v0.w == qhi && !(d0 & 0xff000000u);
    hit |= v1.x == qhi && !(d1 & 0x000000ffu);
    hit |= v1.y == qhi && !(d1 & 0x0000ff00u);
    if ((qhi | qlo) == 0)
        hit = bucket_match<FMT_B6X40>(v0, v1, 0) == 1u;
    return hit;
}

template <uint32_t SEC> __device__ __forceinline__ uint32_t mz_reach(const uint4 &v1)
{
    return SEC == FMT_B8X32 ? mz8_reach(v1.w) : mz6_reach(v1.w);
}

// The rest of a minimizer-line probe that its sector r (of reach > 0) does
// not hold: sectors r ^ 1, then r ^ 2 and r ^ 3 of the same line (the stash
// is next). 16-byte loads: ptxas 12.9 crashes on 32-byte ones in the
// functions kept out of line that this goes into.
template <uint32_t SEC>
__device__ __forceinline__ bool mz_line_holds(const TableView &t, uint64_t r, uint32_t reach, uint32_t slot,
                                              uint32_t high)
{
    auto holds = [&](uint64_t x) {
        return mz_sector_holds<SEC>(__ldg(t.buckets + 2 * x), __ldg(t.buckets + 2 * x + 1), slot, high);
    };
    return holds(r ^ 1) || (reach > 1u && (holds(r ^ 2) || holds(r ^ 3)));
}

template <uint32_t FMT>
__device__ __forceinline__ bool table_lookup(const TableView &t, uint64_t code)
{
    if constexpr (FMT == FMT_MZ8 || FMT == FMT_MZ6) {
        constexpr uint32_t SEC = FMT == FMT_MZ8 ? FMT_B8X32 : FMT_B6X40;
        uint64_t r, slot;
        if (!mz::locate(code, t.g, r, slot))
            return stash_lookup(t, code);
        const uint32_t lo = (uint32_t)slot, hi = (uint32_t)(slot >> 32);
        uint4 v0, v1;
        load_sector(t.buckets + 2 * r, v0, v1);
        if (mz_sector_holds<SEC>(v0, v1, lo, hi))
            return true;
        const uint32_t reach = mz_reach<SEC>(v1);
        if (!reach)
            return false;
        return mz_line_holds<SEC>(t, r, reach, lo, hi) || (reach == 3u && stash_lookup(t, code));
    }
    const uint64_t h = perm_hash(code, t.g.bits);
    const uint64_t r = bucket_of(h, t.g);
    uint4 v0, v1;
    load_sector(t.buckets + 2 * r, v0, v1);
    const uint32_t m = bucket_match<FMT>(v0, v1, fp_of(h, t.g));
    return m == 1u || (m == 2u && stash_lookup(t, code));
}
#endif

} // namespace ibs

// ---- handles ----------------------------------------------------------------
struct ibs_table {
    int device = 0;
    ibs::TableGeom geom{};
    uint4 *buckets = nullptr;
    uint64_t *stash = nullptr;
    uint64_t nKeys = 0, stashKeys = 0;
    double buildSeconds = 0;
    uint64_t deviceBytes = 0;
    ibs::wide::View wide{}; // the levels of a wide-key table (geom.format == FMT_WIDE)
    std::mutex countMu;     // held by a membership count: its total lies behind the buckets
    ibs::TableView view() const { return ibs::TableView{geom, buckets, stash}; }
};

namespace ibs {
// Per-window descriptor on the device.
struct WinDesc {
    uint64_t base; // packed base offset of the window's first base
    uint32_t nPos; // k-mer positions
    int32_t start, end;
    uint32_t pad;
};

#if defined(__CUDACC__)
namespace dev {
// A window's row from its n span summaries, by a group of 2^log2 lanes (lane
// `at` of the group calls it, every lane of the warp does; n = 0 and no row for
// a group without a window): each lane combines a run of consecutive summaries,
// and a shuffle tree the group's runs in order. The group is as wide as a
// window has spans (finish_lanes): one thread a window took 20 us for the 25
// spans of a 50 kbp window, each load waiting for the one before, and a warp
// for each of the one-span windows of a small W cost more than the scan itself
// (8 samples at W = 64, k = 25: 3.2 ms against 1.4).
__device__ __forceinline__ void finish_window(const WinDesc *w, const SegStats *__restrict__ spans, uint32_t n, int k,
                                              uint32_t at, uint32_t log2, ibs_window *__restrict__ out)
{
    const uint32_t run = (n + (1u << log2) - 1) >> log2, a = min(at * run, n), b = min(a + run, n);
    SegStats acc = seg_empty();
    for (uint32_t s = a; s < b; ++s)
        acc = seg_combine(acc, spans[s], k);
    for (uint32_t off = 1; off < 1u << log2; off <<= 1) {
        SegStats o;
        o.total = __shfl_down_sync(0xffffffffu, acc.total, off);
        o.obs = __shfl_down_sync(0xffffffffu, acc.obs, off);
        o.lead = __shfl_down_sync(0xffffffffu, acc.lead, off);
        o.trail = __shfl_down_sync(0xffffffffu, acc.trail, off);
        o.gaps = __shfl_down_sync(0xffffffffu, acc.gaps, off);
        o.dist = __shfl_down_sync(0xffffffffu, acc.dist, off);
        o.pad = 0;
        acc = seg_combine(acc, o, k); // right for lanes that are multiples of 2 off in their group
    }
    if (at == 0 && out) {
        WindowRow row;
        seg_finish(acc, k, row);
        ibs_window o;
        o.start = w->start;
        o.end = w->end;
        o.total_kmers = row.total_kmers;
        o.observed_kmers = row.observed_kmers;
        o.variations = row.variations;
        o.kmer_distance = row.kmer_distance;
        *out = o;
    }
}
} // namespace dev
#endif

// Windows, spans and scratch of one (reference, W, k, span length) plan.
struct ScanPlan {
    uint32_t W = 0, k = 0, spanLen = 0;
    uint64_t nWin = 0, nSpans = 0;
    uint32_t maxSpans = 0;        // of one window
    std::vector<WinDesc> win;     // host copy
    std::vector<uint32_t> span0;  // host copy, nWin + 1
    WinDesc *dWin = nullptr;
    uint32_t *dSpan0 = nullptr;
    SegStats *dSpans = nullptr;   // scratch: one summary per span
    void release();
};

// log2 of the lanes that finish each of `windows` windows of the plan: as many
// as a window has spans, up to a warp. As many as the largest one has while
// that leaves lanes of the GPU idle (a few long contigs among many short ones),
// as many as there are on average otherwise.
uint32_t finish_lanes(const ScanPlan &p, uint64_t windows);

// Expected fraction of keys beyond a bucket's slots when the keys per bucket are
// Poisson(lam).
inline double overflow_fraction(double lam, int slots)
{
    if (lam <= 0)
        return 0;
    double p = std::exp(-lam), over = 0;
    for (int x = 0; x < 400; ++x) {
        if (x > slots)
            over += (x - slots) * p;
        p *= lam / (x + 1);
    }
    return over / lam;
}

// Positions per span for a reference (or a group of its windows) of `bases`:
// the tuned length, or less where that would leave the GPU's warps without a
// span (1 Mbp in spans of 2048 is 490 warps on 32 of 148 SMs, 51 us; in spans
// of 128, 7800 warps), and cutting full windows evenly. hash: the scan of a
// hash-bucket table.
uint32_t span_length(uint64_t bases, uint32_t tuned, uint32_t W, uint32_t k, bool hash);
inline bool is_hash(uint32_t format) { return format == FMT_B8X32 || format == FMT_B6X40; }

// Build the plan's host arrays for contigs `lens` starting at packed
// offsets `baseOff`.
void plan_windows(ScanPlan &p, const std::vector<uint64_t> &lens,
                  const std::vector<uint64_t> &baseOff, uint32_t W, uint32_t k, uint32_t spanLen);

// Launch the span kernel over spans [s0, s1) and, when fin, the window
// finalizer over every window of the plan.
ibs_status launch_scan(const ibs_table *t, const uint64_t *dSeq, const uint64_t *dMask,
                       const ScanPlan &p, uint64_t s0, uint64_t s1, cudaStream_t st);
ibs_status launch_finalize(const ScanPlan &p, uint32_t k, ibs_window *dRows, cudaStream_t st);
ibs_status launch_panel(ibs_table *const *tables, uint32_t nTables, const uint64_t *dSeq,
                        const uint64_t *dMask, const ScanPlan &p, ibs_window *dRows,
                        SegStats *dSpans, cudaStream_t st);
} // namespace ibs

struct ibs_reference {
    int device = 0;
    std::vector<uint64_t> lens, baseOff;
    std::vector<std::string> ids;       // contig ids when parsed from FASTA by the library
    uint64_t seqWords = 0, maskWords = 0;
    uint64_t *dSeq = nullptr, *dMask = nullptr;
    ibs::ScanPlan plans[2];             // cached for the last (W, k); [1]: spans of the hash-bucket scan
    ibs_window *dRows = nullptr;        // cached row buffer for ibs_scan
    uint64_t dRowsCap = 0;
    ibs::SegStats *dPanelSpans = nullptr; // panel scratch
    uint64_t dPanelSpansCap = 0;
    cudaStream_t stream = nullptr;
};
