// The minimizer-line scan of one span of positions, shared by the window
// scan (ibs_scan.cu), the joint-table scan (ibs_panel.cu) and the serving
// kernels (ibs_serve.cu).
#pragma once

#include "ibs_internal.cuh"
#include "scan_device.cuh"

#include <type_traits>

namespace ibs {
namespace dev {

// ---------------------------------------------------------------------------
// The span scan's locator: a warp finds the lines and slot values of 128
// consecutive positions at a time.
//
// Each lane takes 4 neighbouring positions: their k-mers and m-mers are
// funnel shifts by compile-time amounts of one pair of 64-bit windows (the
// bases, and the bases reversed), read and reversed once, and the window
// minimum over the w m-mers is a suffix minimum of the lane's own keys and
// prefix minima of the two lanes after it: 4 shuffles and about 12 minima for
// 4 positions, where one position a lane costs w shuffles, w selects and 2 w
// integer operations each. The minimizer's hash comes from shared memory,
// where every m-mer's hash lies by position. The (line, slot value) pairs go
// through shared memory too, so that the lookups that follow have one
// position a lane in position order again: neighbouring lanes then read one
// line (with 4 positions a lane every lane of a load would touch a line of
// its own, and the load would cost 32 L1 lookups instead of about 9).
//
// Blocks run from the span's last to its first: the keys right of a block's
// last position, which its last windows need, are then those of the block
// done before, kept in a few registers and in the other half of the hash ring.
//
// Bound: instruction issue, and DRAM lines (about 4 positions share one).
// ---------------------------------------------------------------------------
constexpr uint32_t kMzBlock = 128;              // positions a block
constexpr uint32_t kMzNone = 0xffffffffu;       // line of a position without a k-mer (nLines < 2^31)

// A warp's shared memory: the m-mer hashes of two blocks ({lo, slot bits}),
// and the block's (line, low 32 bits of the slot value) pairs with, for
// 40-bit slots, the high bits.
template <uint32_t SEC> struct alignas(16) MzShared {
    uint4 g[2 * kMzBlock / 2];
    uint4 rec[kMzBlock / 2];
    uint32_t high[SEC == FMT_B6X40 ? kMzBlock / 4 : 4];
};

// Reverses the 16 two-bit symbols of a word.
__device__ __forceinline__ uint32_t rev2_32(uint32_t x)
{
    const uint32_t y = __brev(x);
    return ((y >> 1) & 0x55555555u) | ((y << 1) & 0xaaaaaaaau);
}

// Bits [at, at + 32) of a word array (little-endian, zeros around it), at a
// compile-time `at`.
template <int N> __device__ __forceinline__ uint32_t bits_at(const uint32_t (&v)[N], int at)
{
    if (at < 0)
        return at > -32 ? v[0] << (-at & 31) : 0u;
    const int i = at >> 5, s = at & 31;
    const uint32_t a = i < N ? v[i < N ? i : 0] : 0u, b = i + 1 < N ? v[i + 1 < N ? i + 1 : 0] : 0u;
    return s ? __funnelshift_r(a, b, s) : a;
}

// (ahi, alo) < (bhi, blo) as 64-bit numbers.
__device__ __forceinline__ bool less64(uint32_t alo, uint32_t ahi, uint32_t blo, uint32_t bhi)
{
    return (((uint64_t)ahi << 32) | alo) < (((uint64_t)bhi << 32) | blo);
}

// This lane's number, in a register (computed again from the thread index at
// every use otherwise).
__device__ __forceinline__ uint32_t lane_id()
{
    uint32_t l;
    asm volatile("mov.u32 %0, %%laneid;" : "=r"(l));
    return l;
}

template <uint32_t K, uint32_t SEC> class MzWarp
{
    static constexpr uint32_t M = K >= 23 ? K - 7 : 16, W = K - M + 1;
    static constexpr uint32_t HB = 2 * M - 32, KB = 2 * K - 32; // bits of an m-mer, a k-mer past the top 32
    static constexpr bool kWide = SEC == FMT_B6X40;
    static_assert(W <= 8 && K <= 31 && K >= 16, "minimizer windows of at most 8 m-mers");

    // 32-bit words that the K + 3 bases (N bits) of a lane's positions lie in
    static constexpr int kWords = K + 3 + 15 > 48 ? 4 : 3, kMasks = K + 3 + 31 > 64 ? 3 : 2;

    const uint32_t *sp, *mp; // words holding the span's first base and its N bit
    uint32_t word[kWords], nbits[kMasks]; // of the block to do next
    int wordOff, maskOff, lastWord, lastMask;
    uint32_t shift, mshift, lane;
    int len; // positions of the span
    uint32_t nLines, hmul, hmask, hbits;
    uint32_t q1, q2, q3, q4; // prefix minima of the block to the right
    MzShared<SEC> *sh;

  public:
    // Positions [0, n) from packed base `first`; the last base that any of
    // their k-mers has is `lastBase` (words past its word are not read).
    __device__ __forceinline__ MzWarp(MzShared<SEC> *shared, const TableGeom &g, const uint64_t *seq,
                                      const uint64_t *mask, uint64_t first, uint32_t n, uint64_t lastBase,
                                      uint32_t lane_)
        : lane(lane_), len((int)n), q1(~0u), q2(~0u), q3(~0u), q4(~0u), sh(shared)
    {
        const uint64_t w0 = first >> 4, m0 = first >> 5;
        sp = reinterpret_cast<const uint32_t *>(seq) + w0;
        mp = reinterpret_cast<const uint32_t *>(mask) + m0;
        const uint32_t a = ((uint32_t)first & 15) + 4 * lane, c = ((uint32_t)first & 31) + 4 * lane;
        wordOff = (int)(a >> 4);
        shift = 2 * (a & 15);
        maskOff = (int)(c >> 5);
        mshift = c & 31;
        lastWord = (int)((lastBase >> 4) - w0);
        lastMask = (int)((lastBase >> 5) - m0);
        nLines = (uint32_t)(g.nBuckets / mz::kSectorsPerLine);
        hbits = g.fpBits;
        hmask = hbits >= 32 ? 0xffffffffu : (1u << hbits) - 1u;
        hmul = hbits >= 32 ? 0u : 1u << hbits;
    }

    __device__ __forceinline__ int blocks() const { return (len + (int)kMzBlock - 1) / (int)kMzBlock; }

    // Block b: its positions' lines and slot values in sh->rec (and
    // sh->high), in position order. Blocks are done from blocks() - 1 down
    // to 0, after start(). The writes are visible to the warp on return; a
    // lane's reads of block b + 1 may come right up to the call.
    __device__ __forceinline__ void block(int b)
    {
        uint32_t N[3], Y[3], key[4];
        streams(N, Y);
        keys(b, N, Y, key);
        const uint32_t p2 = min(key[0], key[1]), p3 = min(p2, key[2]), p4 = min(p3, key[3]);
        const uint32_t s2 = min(key[2], key[3]), s1 = min(key[1], s2);
        const uint32_t pre[5] = {0, key[0], p2, p3, p4}, old[5] = {0, q1, q2, q3, q4};
        const uint32_t suf[4] = {p4, s1, s2, key[3]};
        uint32_t n1[5], n2[5];
#pragma unroll
        for (int n = 1; n <= 4; ++n) {
            // prefix minima that some window of the four ends in, of the next
            // lane (its windows' ends run from W - 4 to W - 1) and the one
            // after; tags count twice the position from the lane's first
            n1[n] = n2[n] = ~0u;
            if ((n < 4 && n >= (int)W - 4 && n <= (int)W - 1) || (n == 4 && (int)W - 1 >= 4))
                n1[n] = __shfl_sync(FULL_MASK, lane == 0 ? old[n] : pre[n], lane + 1) + 8u;
            if (n >= (int)W - 8 && n <= (int)W - 5 && W >= 6)
                n2[n] = __shfl_sync(FULL_MASK, lane < 2 ? old[n] : pre[n], lane + 2) + 16u;
        }
        q1 = key[0];
        q2 = p2;
        q3 = p3;
        q4 = p4;
        __syncwarp(); // the block's hashes are in the ring, and the records before are read
        const uint32_t ok = valid(b);
        if (b > 0)
            fetch(b - 1);
        const uint8_t *ring = reinterpret_cast<const uint8_t *>(sh->g);
        const uint32_t at = ((uint32_t)(b & 1) * kMzBlock + 4 * lane) * 8;
        uint2 rec[4];
        uint32_t high = 0;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int end = t + (int)W - 1; // the window's last m-mer, from the lane's first position
            uint32_t v;
            if (end < 3) {
                v = key[t];
#pragma unroll
                for (int i = t + 1; i <= end; ++i)
                    v = min(v, key[i < 4 ? i : 3]);
            } else {
                v = suf[t];
                if (end >= 4)
                    v = min(v, n1[end - 3 < 4 ? end - 3 : 4]);
                if (end >= 8)
                    v = min(v, n2[end - 7 < 4 ? end - 7 : 4]);
            }
            const uint2 g = *reinterpret_cast<const uint2 *>(ring + ((at + 4 * (v & 30u)) & (16 * kMzBlock - 1)));
            // the k-mer on the strand that holds the minimizer itself, at the
            // top of 64 bits (its 2K bits and other bases below), and twice
            // the minimizer's offset in it
            const bool rev = v & 1u;
            const uint32_t fhi = bits_at(Y, 64 - 2 * t), flo = bits_at(Y, 32 - 2 * t);
            const uint32_t rhi = bits_at(N, 2 * t + (int)KB), rlo = bits_at(N, 2 * t + (int)KB - 32);
            const uint32_t hi = rev ? rhi : fhi, lo = KB ? (rev ? rlo : flo) >> (KB ? 32 - KB : 0) : 0u;
            const uint32_t d2 = (v & 30u) - 2 * t, o2 = rev ? 2 * (W - 1) - d2 : d2;
            // the other K - M bases, and the slot value (mz::slot_high, mz::place)
            const uint32_t rest = K > M ? __funnelshift_l(hi, lo, o2) & ((1u << (2 * (K - M))) - 1u) : 0u;
            const uint32_t top = K > M ? o2 * (1u << (K > M ? 2 * (K - M) - 1 : 0)) + rest : 0u;
            const uint32_t low = HB ? g.y : g.x & hmask;
            rec[t] = make_uint2(__umulhi(g.x, nLines), top * hmul + low);
            if (kWide) // bits 32 .. 39 of (top << hbits)
                high |= (top >> (32 - hbits)) << (8 * t);
        }
        if (ok != 15u) { // N runs and the span's end
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (!((ok >> t) & 1u))
                    rec[t].x = kMzNone;
        }
        sh->rec[2 * lane] = make_uint4(rec[0].x, rec[0].y, rec[1].x, rec[1].y);
        sh->rec[2 * lane + 1] = make_uint4(rec[2].x, rec[2].y, rec[3].x, rec[3].y);
        if (kWide)
            sh->high[lane] = high;
        __syncwarp();
    }

    // Before the first block: the keys right of the span's last block, where
    // its last windows reach past it, and the last block's words.
    __device__ __forceinline__ void start()
    {
        const int nb = blocks();
        if (len + (int)W - 1 > nb * (int)kMzBlock) {
            uint32_t N[3], Y[3], key[4];
            fetch(nb);
            streams(N, Y);
            keys(nb, N, Y, key);
            q1 = key[0];
            q2 = min(q1, key[1]);
            q3 = min(q2, key[2]);
            q4 = min(q3, key[3]);
        }
        fetch(nb - 1);
    }

  private:
    // Reads block b's sequence and N words, one block ahead of their use.
    __device__ __forceinline__ void fetch(int b)
    {
        const int at = wordOff + 8 * b, mt = maskOff + 4 * b;
#pragma unroll
        for (int i = 0; i < kWords; ++i)
            word[i] = __ldg(sp + min(at + i, lastWord));
#pragma unroll
        for (int i = 0; i < kMasks; ++i)
            nbits[i] = __ldg(mp + min(mt + i, lastMask));
    }

    // The 48 bases from the lane's first position: complemented (N, base t at
    // bits 2t) and reversed (Y, base t at bits 94 - 2t); only the K + 3 first
    // ones are used.
    __device__ __forceinline__ void streams(uint32_t (&N)[3], uint32_t (&Y)[3]) const
    {
        const uint32_t x0 = __funnelshift_r(word[0], word[1], shift), x1 = __funnelshift_r(word[1], word[2], shift);
        const uint32_t x2 = K + 3 > 32 ? (kWords > 3 ? __funnelshift_r(word[2], word[kWords - 1], shift)
                                                     : word[2] >> shift)
                                       : 0u;
        N[0] = ~x0;
        N[1] = ~x1;
        N[2] = ~x2;
        Y[2] = rev2_32(x0);
        Y[1] = rev2_32(x1);
        Y[0] = K + 3 > 32 ? rev2_32(x2) : 0;
    }

    // Rank keys of the m-mers at the lane's 4 positions, with twice the
    // position and, in the lowest bit, whether the reverse complement is the
    // canonical one; their hashes go into the ring: lo, and the low bits of
    // the line hash that the slot value takes.
    __device__ __forceinline__ void keys(int b, const uint32_t (&N)[3], const uint32_t (&Y)[3], uint32_t (&key)[4])
    {
        uint2 g[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const uint32_t fhi = bits_at(Y, 64 - 2 * t), flo = bits_at(Y, 32 - 2 * t);
            const uint32_t rhi = bits_at(N, 2 * t + (int)HB), rlo = bits_at(N, 2 * t + (int)HB - 32);
            bool rLess;
            uint32_t low = 0; // the m-mer's bits past its top 32
            if (!HB) {
                rLess = rhi < fhi;
            } else if (M & 1) { // never its own reverse complement: the bits below decide nothing
                rLess = less64(rlo, rhi, flo, fhi);
                low = (rLess ? rlo : flo) >> (HB ? 32 - HB : 0);
            } else {
                const uint32_t fl = flo >> (HB ? 32 - HB : 0), rl = rlo >> (HB ? 32 - HB : 0);
                rLess = less64(rl, rhi, fl, fhi);
                low = rLess ? rl : fl;
            }
            const mz::Mixed x = mz::mix(rLess ? rhi : fhi, low);
            key[t] = mz::rank_key_of(x) + (rLess ? 2u * t + 1u : 2u * t);
            g[t] = make_uint2(x.lo, HB ? ((x.lo << HB) | low) & hmask : 0u);
        }
        uint4 *to = sh->g + (b & 1) * (kMzBlock / 2) + 2 * lane;
        to[0] = make_uint4(g[0].x, g[0].y, g[1].x, g[1].y);
        to[1] = make_uint4(g[2].x, g[2].y, g[3].x, g[3].y);
    }

    // Bit t: position t of the lane's four lies in the span and its K bases
    // are ACGT.
    __device__ __forceinline__ uint32_t valid(int b) const
    {
        const uint32_t lo = __funnelshift_r(nbits[0], nbits[1], mshift);
        const uint32_t hi = K + 3 > 32 ? (kMasks > 2 ? __funnelshift_r(nbits[1], nbits[kMasks - 1], mshift)
                                                     : nbits[1] >> mshift)
                                       : 0u;
        const int left = len - b * (int)kMzBlock - 4 * (int)lane;
        uint32_t ok = left >= 4 ? 15u : (left > 0 ? (1u << left) - 1u : 0u);
        if (lo | hi) { // N runs are few
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (__funnelshift_r(lo, hi, t) & ((1u << K) - 1u))
                    ok &= ~(1u << t);
        }
        return ok;
    }
};

// A lane's four sectors of a block (32 bytes each), all in flight together.
// (Locating the next block while they are in flight was slower: the 32
// registers they hold cost a third of the warps, which hide more.)
struct MzSectors {
    uint4 v0[4], v1[4];
    uint32_t line[4], slot[4], high[4]; // the records of positions 32 i + lane

    template <uint32_t SEC> __device__ __forceinline__ void record(const MzShared<SEC> *sh, int i, uint32_t at)
    {
        const uint2 r = reinterpret_cast<const uint2 *>(sh->rec)[at];
        line[i] = r.x;
        slot[i] = r.y;
        high[i] = SEC == FMT_B6X40 ? reinterpret_cast<const uint8_t *>(sh->high)[at] : 0u;
    }

    __device__ __forceinline__ uint64_t sector(int i) const
    {
        return (uint64_t)line[i] * mz::kSectorsPerLine + mz::sector_of(slot[i], high[i]);
    }

    __device__ __forceinline__ bool valid(int i) const { return line[i] != kMzNone; }

    template <uint32_t SEC>
    __device__ __forceinline__ void load(const MzShared<SEC> *sh, const uint4 *buckets, uint32_t lane)
    {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            record(sh, i, 32 * i + lane);
            // a position without a k-mer reads sector 0 .. 3 of line 0
            load_sector(buckets + (uint64_t)(valid(i) ? line[i] : 0u) * 8 + 2 * mz::sector_of(slot[i], high[i]), v0[i],
                        v1[i]);
        }
    }
};

// The rest of a probe that its full sector does not hold: the line's other
// sectors, then the stash, which is keyed by the canonical k-mer, read again
// from packed base G. Out of line: inlined, it costs the scan's main path
// registers (104 bytes of spills, 15% of its time).
template <uint32_t K, uint32_t SEC>
__device__ __noinline__ bool mz_elsewhere(const TableView *t, const uint64_t *__restrict__ seq,
                                          const uint64_t *__restrict__ mask, uint64_t G, uint32_t line, uint32_t slot,
                                          uint32_t high, uint32_t reach)
{
    const uint64_t r = (uint64_t)line * mz::kSectorsPerLine + mz::sector_of(slot, high);
    if (mz_line_holds<SEC>(*t, r, reach, slot, high))
        return true;
    bool acgt;
    return reach == 3u && stash_lookup(*t, canonical_at(seq, mask, G, K, key_mask(2 * K), key_mask(K), acgt));
}

// The hits of a block's positions (MzWarp::block has located it), from its
// last 32 positions to its first: use(V, H) gets their valid and hit ballots.
template <uint32_t K, uint32_t SEC, typename Use>
__device__ __forceinline__ void mz_hits(const MzShared<SEC> *sh, const TableView &t, const uint64_t *__restrict__ seq,
                                        const uint64_t *__restrict__ mask, uint64_t blockBase, uint32_t lane,
                                        Use &&use)
{
    uint32_t hit = 0, valid = 0; // a bit a position
    uint32_t more = 0;           // two bits a position: the reach of a full sector that does not hold it
    {
        MzSectors s;
        s.load(sh, t.buckets, lane);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (s.valid(i)) {
                valid |= 1u << i;
                if (mz_sector_holds<SEC>(s.v0[i], s.v1[i], s.slot[i], s.high[i]))
                    hit |= 1u << i;
                else
                    more |= mz_reach<SEC>(s.v1[i]) << (2 * i);
            }
        }
    }
    while (more) { // about 1% of the positions
        const int i = (__ffs(more) - 1) >> 1;
        MzSectors s;
        s.record(sh, 0, 32 * i + lane);
        if (mz_elsewhere<K, SEC>(&t, seq, mask, blockBase + 32 * i + lane, s.line[0], s.slot[0], s.high[0],
                                 (more >> (2 * i)) & 3u))
            hit |= 1u << i;
        more &= ~(3u << (2 * i));
    }
#pragma unroll
    for (int i = 3; i >= 0; --i)
        use(__ballot_sync(FULL_MASK, valid & (1u << i)), __ballot_sync(FULL_MASK, hit & (1u << i)));
}

// Statistics of the n positions from packed base `first` against a
// minimizer-line table; the last base of their window's k-mers is
// `lastBase`. The result is in lane 0. SEC: FMT_B8X32 sectors (format MZ8) or
// FMT_B6X40 (MZ6).
template <uint32_t K, uint32_t SEC>
__device__ __forceinline__ SegStats mz_span_stats(MzShared<SEC> *sh, const TableView &t,
                                                  const uint64_t *__restrict__ seq,
                                                  const uint64_t *__restrict__ mask, uint64_t first, uint32_t n,
                                                  uint64_t lastBase, uint32_t lane)
{
    LaneFold<true> fold;
    MzWarp<K, SEC> warp(sh, t.g, seq, mask, first, n, lastBase, lane);
    warp.start();
    for (int b = warp.blocks() - 1; b >= 0; --b) {
        warp.block(b);
        mz_hits<K, SEC>(sh, t, seq, mask, first + kMzBlock * b, lane,
                        [&](uint32_t V, uint32_t H) { fold.push(V, H, lane, (int)K); });
    }
    return fold.finish((int)K);
}

} // namespace dev

// Calls f with a minimizer table's k (16 <= k <= last) as a compile-time
// constant.
template <uint32_t K, uint32_t LAST, typename F> void with_mz_k(uint32_t k, F &&f)
{
    if (k == K)
        f(std::integral_constant<uint32_t, K>{});
    else if constexpr (K < LAST)
        with_mz_k<K + 1, LAST>(k, f);
}

// The same with the sector layout of a table's format: f(K, SEC).
template <typename F> void with_mz_table(const TableGeom &g, F &&f)
{
    if (g.format == FMT_MZ8)
        with_mz_k<16, 27>(g.k, [&](auto K) { f(K, std::integral_constant<uint32_t, FMT_B8X32>{}); });
    else
        with_mz_k<16, 31>(g.k, [&](auto K) { f(K, std::integral_constant<uint32_t, FMT_B6X40>{}); });
}
} // namespace ibs
