// Panel scan: one reference pass against up to 16 samples through ONE joint
// table whose slots carry a sample-membership mask.
//
// The reference's panel mode encodes each batch once and probes every
// resident database separately (encodeProbeMultiKernel + MultiBsProbe,
// src/gpu/EncodeProbe.cu:82-108, :175-193; MAX_DBS = 16,
// src/gpu/EncodeProbeCore.hpp:291), so a position costs one index search
// per sample. Here the samples' k-mer sets are merged into one table: a
// position costs one random 32-byte bucket load whatever the panel size,
// and the mask in the matching slot says which samples hold the k-mer.
// Every sample's rows are still exactly its single-sample rows.
//
// Bucket format P5x48 (one 32-byte sector): u32 fingerprints of slots 0-4
// (words 0-4), u16 sample masks of slots 0-4 (bytes 20-29), slot count
// (byte 30), flags (byte 31, bit 0 = some key of this bucket is in the
// stash). The fingerprint is the same quotient of the bijective k-mer hash
// as in the single-sample table, so it needs nBuckets >= 2^(2k-32).
// Stash: {code, mask} pairs, two per 32-byte bucket, linear probing.
//
// Format PM (FMT_PANEL_MZ, 16 <= k <= 27): the same sectors laid out as the
// minimizer lines of the single-sample MZ tables (mz_core.cuh): the line is
// the k-mer's minimizer's, one of its four sectors is picked by the k-mer
// itself, and the 32-bit slot value identifies the k-mer within its line
// (at least 2^(2k-28) lines). Consecutive reference positions mostly share a
// minimizer, so a warp's probes fall in few 128-byte lines instead of 32
// random ones. A full sector keeps further keys in its partner sector (index
// ^ 1, the same line; flag bit 25 of byte 31's word), then in the line's
// other two (bit 26) and then in the stash (bit 24).
//
// Format PM6 (FMT_PANEL_MZ6, 28 <= k <= 31): the same lines for 40-bit slot
// values, four slots a sector: their high 32 bits in words 0-3, low bytes in
// word 4, masks in words 5-6, count and flags in word 7 as above (at least
// 2^(2k-37) lines).
#pragma once

#include "ibs_internal.cuh"
#include "mz_scan.cuh"

#include <vector>

namespace ibs {
namespace panel {

constexpr uint32_t kMaxSamples = IBS_PANEL_MAX_SAMPLES;
constexpr uint32_t kSlots = 5, kSlots6 = 4;
// The minimizer-line layout of a k, and the sector layout whose slot values it has.
IBS_HD bool is_joint_mz(uint32_t fmt) { return fmt == FMT_PANEL_MZ || fmt == FMT_PANEL_MZ6; }
constexpr uint32_t joint_mz_format(uint32_t k) { return k <= 27 ? FMT_PANEL_MZ : FMT_PANEL_MZ6; }
constexpr uint32_t joint_mz_slots(uint32_t k) { return k <= 27 ? FMT_B8X32 : FMT_B6X40; }
constexpr uint64_t kStashEmpty = ~0ull;
constexpr uint32_t kStashFlag = 1u << 24;   // word 7: some key of this sector is in the stash
constexpr uint32_t kPartnerFlag = 1u << 25; // word 7 (PM): some key of this sector is in its partner sector
constexpr uint32_t kLineFlag = 1u << 26;    // word 7 (PM): ... or in one of the line's other two

struct View {
    TableGeom g;
    const uint4 *buckets;
    const ulonglong2 *stash; // {code, mask}
    uint64_t stashBuckets;   // power of two; two entries each
};

__device__ __forceinline__ uint32_t stash_mask(const View &t, uint64_t code)
{
    uint64_t b = stash_home(code, t.stashBuckets);
    for (uint64_t i = 0; i < t.stashBuckets; ++i) {
        const ulonglong2 e0 = __ldg(t.stash + 2 * b), e1 = __ldg(t.stash + 2 * b + 1);
        if (e0.x == code)
            return (uint32_t)e0.y;
        if (e1.x == code)
            return (uint32_t)e1.y;
        if (e0.x == kStashEmpty || e1.x == kStashEmpty)
            return 0;
        b = (b + 1) & (t.stashBuckets - 1);
    }
    return 0;
}

// Sample mask of fingerprint (or slot value) fp in a sector's halves; 0
// when no slot holds it (a slot past the sector's count has an empty mask).
__device__ __forceinline__ uint32_t sector_mask(const uint4 &v0, const uint4 &v1, uint32_t fp)
{
    uint32_t m = v0.x == fp ? v1.y & 0xffffu : 0u;
    m |= v0.y == fp ? v1.y >> 16 : 0u;
    m |= v0.z == fp ? v1.z & 0xffffu : 0u;
    m |= v0.w == fp ? v1.z >> 16 : 0u;
    m |= v1.x == fp ? v1.w & 0xffffu : 0u;
    return m;
}

// The same of a minimizer line's sector, for a slot value of 32 (PM) or 40
// bits (PM6: high holds its top byte).
template <bool WIDE>
__device__ __forceinline__ uint32_t line_sector_mask(const uint4 &v0, const uint4 &v1, uint32_t slot, uint32_t high)
{
    if (!WIDE)
        return sector_mask(v0, v1, slot);
    const uint32_t hi = __funnelshift_r(slot, high, 8), d = v1.x ^ ((slot & 0xffu) * 0x01010101u);
    uint32_t m = v0.x == hi && !(d & 0x000000ffu) ? v1.y & 0xffffu : 0u;
    m |= v0.y == hi && !(d & 0x0000ff00u) ? v1.y >> 16 : 0u;
    m |= v0.z == hi && !(d & 0x00ff0000u) ? v1.z & 0xffffu : 0u;
    m |= v0.w == hi && !(d & 0xff000000u) ? v1.z >> 16 : 0u;
    return m;
}

// Sample mask of a k-mer given its bucket halves and fingerprint; bit 31
// set = look in the stash.
__device__ __forceinline__ uint32_t bucket_mask(const uint4 &v0, const uint4 &v1, uint32_t fp)
{
    uint32_t m = sector_mask(v0, v1, fp);
    if (!m && (v1.w & kStashFlag))
        m = 0x80000000u;
    return m;
}

// Minimizer lines: the mask of a k-mer that its home sector r does not hold,
// from the line's other sectors as the home sector's flags say (the stash is
// next).
template <bool WIDE>
__device__ __forceinline__ uint32_t pm_line_mask(const View &t, uint32_t flags, uint64_t r, uint32_t slot,
                                                 uint32_t high)
{
    uint32_t m = 0;
    auto look = [&](uint64_t x) {
        return line_sector_mask<WIDE>(__ldg(t.buckets + 2 * x), __ldg(t.buckets + 2 * x + 1), slot, high);
    };
    if (flags & kPartnerFlag) {
        m = look(r ^ 1);
        if (!m && (flags & kLineFlag))
            m = look(r ^ 2) | look(r ^ 3);
    }
    return m;
}

// Home sectors and stored fingerprints (P5x48) or slot values of a key;
// returns how many places it has (mz::placements; none: the stash only).
__device__ __forceinline__ uint32_t joint_places(const View &t, uint64_t code, uint64_t r[2], uint64_t fp[2])
{
    if (is_joint_mz(t.g.format))
        return mz::placements(code, t.g, r, fp);
    const uint64_t h = perm_hash(code, t.g.bits);
    r[0] = bucket_of(h, t.g);
    fp[0] = fp_of(h, t.g);
    return 1;
}

template <bool WIDE>
__device__ __forceinline__ uint32_t lookup_line_mask(const View &t, uint64_t code, uint64_t r, uint64_t fp)
{
    uint4 v0, v1;
    load_sector(t.buckets + 2 * r, v0, v1);
    uint32_t m = line_sector_mask<WIDE>(v0, v1, (uint32_t)fp, (uint32_t)(fp >> 32));
    if (!m)
        m = pm_line_mask<WIDE>(t, v1.w, r, (uint32_t)fp, (uint32_t)(fp >> 32));
    return !m && (v1.w & kStashFlag) ? stash_mask(t, code) : m;
}

__device__ __forceinline__ uint32_t lookup_mask(const View &t, uint64_t code)
{
    uint64_t r[2], fp[2];
    if (!joint_places(t, code, r, fp))
        return stash_mask(t, code);
    if (t.g.format == FMT_PANEL_MZ)
        return lookup_line_mask<false>(t, code, r[0], fp[0]);
    if (t.g.format == FMT_PANEL_MZ6)
        return lookup_line_mask<true>(t, code, r[0], fp[0]);
    uint4 v0, v1;
    load_sector(t.buckets + 2 * r[0], v0, v1);
    const uint32_t m = bucket_mask(v0, v1, (uint32_t)fp[0]);
    return m & 0x80000000u ? stash_mask(t, code) : m;
}

// The same of the k-mer at packed base G, out of line (see dev::mz_elsewhere);
// flags is the home sector's flag byte.
template <bool WIDE>
__device__ __noinline__ uint32_t elsewhere_mask(const View *t, const uint64_t *__restrict__ seq,
                                                const uint64_t *__restrict__ mask, uint64_t G, uint32_t k,
                                                uint32_t line, uint32_t slot, uint32_t high, uint32_t flags)
{
    const uint32_t m = pm_line_mask<WIDE>(
        *t, flags << 24, (uint64_t)line * mz::kSectorsPerLine + mz::sector_of(slot, high), slot, high);
    if (m || !((flags << 24) & kStashFlag))
        return m;
    bool acgt;
    return stash_mask(*t, dev::canonical_at(seq, mask, G, k, key_mask(2 * k), key_mask(k), acgt));
}

// The sample masks of a block's positions (MzWarp::block has located it): m[i]
// is position 32 i + lane's, valid[i] whether it has a k-mer. RANGE: sectors
// outside [bLo, bHi) count as empty (they read sector bLo).
template <uint32_t K, bool RANGE>
__device__ __forceinline__ void mz_masks(const dev::MzShared<joint_mz_slots(K)> *sh, const View &t,
                                         const uint64_t *__restrict__ seq, const uint64_t *__restrict__ mask,
                                         uint64_t blockBase, uint32_t lane, uint64_t bLo, uint64_t bHi,
                                         uint32_t (&m)[4], bool (&valid)[4])
{
    constexpr bool kWide = K > 27;
    uint32_t more = 0; // 3 bits a position: the flags of a full sector that does not hold it
    {
        dev::MzSectors s;
        bool mine[4];
        if (RANGE) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                s.record(sh, i, 32 * i + lane);
                const uint64_t r = s.sector(i);
                mine[i] = s.valid(i) && r >= bLo && r < bHi;
                load_sector(t.buckets + 2 * (mine[i] ? r : bLo), s.v0[i], s.v1[i]);
            }
        } else {
            s.load(sh, t.buckets, lane);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            valid[i] = s.valid(i);
            if (!RANGE)
                mine[i] = valid[i];
            m[i] = mine[i] ? line_sector_mask<kWide>(s.v0[i], s.v1[i], s.slot[i], s.high[i]) : 0u;
            if (mine[i] && !m[i])
                more |= ((s.v1[i].w >> 24) & 7u) << (3 * i);
        }
    }
    while (more) {
        const int i = (__ffs(more) - 1) / 3;
        dev::MzSectors s;
        s.record(sh, 0, 32 * i + lane);
        const uint32_t x = elsewhere_mask<kWide>(&t, seq, mask, blockBase + 32 * i + lane, K, s.line[0], s.slot[0],
                                                 s.high[0], (more >> (3 * i)) & 7u);
        m[0] = i == 0 ? x : m[0];
        m[1] = i == 1 ? x : m[1];
        m[2] = i == 2 ? x : m[2];
        m[3] = i == 3 ? x : m[3];
        more &= ~(7u << (3 * i));
    }
}

// Statistics of up to 16 samples over a span's blocks of 128 positions, from
// the last block to the first. A block's four 16-bit masks a lane are two
// 32 x 32 bit matrices (positions by samples), transposed by five shuffles
// each: lane j then has sample j's hits of the block's first 64 positions and
// lane 16 + j those of its last 64, so that all 32 lanes summarise
// (16 ballots and a select each gave the words to 16 lanes only).
struct JointFold {
    Seg32 acc{0, 0, 0, 0, 0, 0}; // lane j < 16: sample j, the blocks so far
    uint32_t amount[5], keep[5];

    __device__ __forceinline__ explicit JointFold(uint32_t lane)
    {
        const uint32_t M[5] = {0x0000ffffu, 0x00ff00ffu, 0x0f0f0f0fu, 0x33333333u, 0x55555555u};
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            const uint32_t s = 16u >> i;
            amount[i] = lane & s ? 32 - s : s;
            keep[i] = lane & s ? ~M[i] : M[i];
        }
    }

    // Bit i of lane l's result is bit l of lane i's x.
    __device__ __forceinline__ uint32_t transpose(uint32_t x) const
    {
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            const uint32_t y = __shfl_xor_sync(dev::FULL_MASK, x, 16 >> i);
            x = (x & keep[i]) | (__funnelshift_l(y, y, amount[i]) & ~keep[i]);
        }
        return x;
    }

    // m: the lane's masks of positions 32 i + lane; valid: whether they count.
    __device__ __forceinline__ void push(const uint32_t (&m)[4], const bool (&valid)[4], uint32_t lane, int k)
    {
        const uint32_t V0 = __ballot_sync(dev::FULL_MASK, valid[0]), V1 = __ballot_sync(dev::FULL_MASK, valid[1]),
                       V2 = __ballot_sync(dev::FULL_MASK, valid[2]), V3 = __ballot_sync(dev::FULL_MASK, valid[3]);
        const uint32_t Ha = transpose(m[0] | m[2] << 16), Hb = transpose(m[1] | m[3] << 16);
        Seg32 s = seg32_combine(block_seg32(lane < 16 ? V0 : V2, Ha, k), block_seg32(lane < 16 ? V1 : V3, Hb, k), k);
        Seg32 o;
        o.total = __shfl_down_sync(dev::FULL_MASK, s.total, 16);
        o.obs = __shfl_down_sync(dev::FULL_MASK, s.obs, 16);
        o.lead = __shfl_down_sync(dev::FULL_MASK, s.lead, 16);
        o.trail = __shfl_down_sync(dev::FULL_MASK, s.trail, 16);
        o.gaps = __shfl_down_sync(dev::FULL_MASK, s.gaps, 16);
        o.dist = __shfl_down_sync(dev::FULL_MASK, s.dist, 16);
        acc = seg32_combine(seg32_combine(s, o, k), acc, k);
    }
};

// Block statistics of one sample from its valid (V) and hit (H) masks,
// computed by one lane with bit operations: the gaps between hits are the
// runs of valid misses, visited one run at a time.
__device__ __forceinline__ SegStats block_stats_serial(uint32_t V, uint32_t H, int k)
{
    SegStats b;
    b.pad = 0;
    b.total = __popc(V);
    b.obs = __popc(H);
    b.gaps = 0;
    b.dist = 0;
    if (H == 0) {
        b.lead = b.trail = b.total;
        return b;
    }
    const uint32_t first = __ffs(H) - 1;
    const uint32_t last = 31 - __clz(H);
    b.lead = __popc(V & ((1u << first) - 1u));
    b.trail = last == 31 ? 0u : __popc(V >> (last + 1));
    // valid misses strictly between the first and the last hit
    const uint64_t inner = ((2ull << last) - 1ull) & ~((2ull << first) - 1ull);
    uint32_t m = V & ~H & (uint32_t)inner;
    while (m) {
        const uint32_t start = __ffs(m) - 1;
        const uint32_t next = H & ~((2u << start) - 1u); // hits after the run starts (nonzero)
        const uint32_t j = __ffs(next) - 1;
        const uint32_t g = __popc(m & ((1u << j) - 1u));
        b.gaps += 1;
        b.dist += gap_distance(g, k);
        m &= ~((1u << j) - 1u);
    }
    return b;
}

} // namespace panel
} // namespace ibs

// A joint table and its scan state (the handle behind the ibs_panel_table_* calls).
struct ibs_panel_table {
    using View = ibs::panel::View;
    int device = 0;
    ibs::TableGeom geom{};
    uint4 *buckets = nullptr;
    ulonglong2 *stash = nullptr;
    uint64_t stashBuckets = 0;
    uint32_t nSamples = 0;
    uint64_t keysAdded = 0; // sum of the samples' key counts
    uint64_t deviceBytes = 0;
    double buildSeconds = 0;
    int *dErr = nullptr;
    unsigned long long *dCounters = nullptr; // [0] pending count, [1] scan work counter, [2] failed
    uint32_t stashGrowths = 0;
    // scan plan and scratch
    const ibs_reference *planRef = nullptr;
    std::vector<uint64_t> planLens;
    ibs::ScanPlan plan;
    ibs::SegStats *dSpans = nullptr;
    uint16_t *dMasks = nullptr; // per-position masks of a multi-pass scan
    uint64_t spansCap = 0;
    // captured scan graph for (reference, W, rows, stream)
    cudaGraphExec_t graph = nullptr;
    const void *graphKey[3] = {nullptr, nullptr, nullptr};
    uint32_t graphShape[3] = {0, 0, 0}; // what it was captured with: CTAs per SM, blocks in flight, passes
    uint32_t graphW = 0;
    View view() const { return View{geom, buckets, stash, stashBuckets}; }
};

namespace ibs {
void panel_release_table(ibs_panel_table *p);
} // namespace ibs
