// Wide-key tables and codes: k-mers of 33 <= k <= 64 bases.
//
// The reference takes such k through its string path (k > 32 routes every
// database to getStatsFromSequenceLegacy, src/KmerDatabase.hpp:100-124 and
// :675-708): canonical k-mers as strings, each looked up in the KMC
// database. Here the canonical k-mer is a 2k-bit code held in two 64-bit
// words (lo = bits 0..63, hi = the rest; first base most significant, so
// the integer order is the string order of ACGT), and the table holds whole
// keys: no quotienting, since a 128-bit key space has no cheap bijection
// whose remainder fits a slot.
//
// Layout (format FMT_WIDE): 128-byte lines of eight 16-byte slots
// {lo, hi}; an empty slot is all ones in both words (never a canonical
// code: all ones is the all-T k-mer, whose reverse complement all-A is
// smaller; the build leaves out a key equal to it, which no scan asks for).
// The lines form up to kMaxLevels levels, each with its own line hash: level
// 0 holds the keys at about 4 per line; the keys of lines that got more than
// 8 go to level 1, sized at about 2 per line, and so on until none is left.
// A line's two 64-byte halves fill one after the other: a key takes the next
// slot of its home half (a bit of its hash), then of the other half. A probe
// therefore reads its home half; a hit or an empty last slot ends it there
// (86% of the absent keys at 4 keys a line), a full half sends it to the other
// one and a full line to the next level.
#pragma once

#include <cuda_runtime.h>

#include "ibs_core.cuh"

namespace ibs {
namespace wide {

constexpr uint32_t kSlots = 8;
constexpr uint32_t kMaxLevels = 12;
constexpr uint64_t kEmpty = ~0ull;

// A table's levels: each its own device array of lines[L] lines of kSlots
// {lo, hi} slots.
struct View {
    uint32_t k, nLevels;
    uint64_t lines[kMaxLevels];
    const ulonglong2 *slots[kMaxLevels];
};

// A 64-bit mix of both words of a key, its own in every level; scaled to the
// level's line count it is the key's line, and its lowest bit the home half.
IBS_HD uint64_t hash_of(uint64_t lo, uint64_t hi, uint32_t level)
{
    return fmix64(lo ^ fmix64(hi + 0x9e3779b97f4a7c15ull * (level + 1)));
}

IBS_HD uint64_t line_of(uint64_t lo, uint64_t hi, uint32_t level, uint64_t nLines)
{
    return mulhi64(hash_of(lo, hi, level), nLines);
}

// The slot a key's home half starts at.
IBS_HD uint64_t home_of(uint64_t lo, uint64_t hi, uint32_t level, uint64_t nLines)
{
    const uint64_t h = hash_of(lo, hi, level);
    return mulhi64(h, nLines) * kSlots + (h & 1) * (kSlots / 2);
}

// 2-bit symbols of x in reverse order.
IBS_HD uint64_t rev2(uint64_t x)
{
#if defined(__CUDA_ARCH__)
    uint64_t y = __brevll(x);
#else
    uint64_t y = x;
    y = ((y >> 1) & 0x5555555555555555ull) | ((y & 0x5555555555555555ull) << 1);
    y = ((y >> 2) & 0x3333333333333333ull) | ((y & 0x3333333333333333ull) << 2);
    y = ((y >> 4) & 0x0f0f0f0f0f0f0f0full) | ((y & 0x0f0f0f0f0f0f0f0full) << 4);
    y = ((y >> 8) & 0x00ff00ff00ff00ffull) | ((y & 0x00ff00ff00ff00ffull) << 8);
    y = ((y >> 16) & 0x0000ffff0000ffffull) | ((y & 0x0000ffff0000ffffull) << 16);
    y = (y >> 32) | (y << 32);
#endif
    return ((y >> 1) & 0x5555555555555555ull) | ((y & 0x5555555555555555ull) << 1);
}

// Canonical code of the 2k-bit little-endian base stream (xlo, xhi) (base 0
// in bits 0-1 of xlo; bits of xhi above 2k - 64 are ignored): the forward
// code is the stream with its symbols reversed, the reverse complement is
// the complemented stream; the smaller one, compared as 128-bit integers.
IBS_HD void canonical_of_stream(uint64_t xlo, uint64_t xhi, uint32_t k, uint64_t &clo, uint64_t &chi)
{
    const uint32_t d = 128 - 2 * k; // 0 <= d < 64
    const uint64_t ylo = rev2(xhi), yhi = rev2(xlo);
    const uint64_t fhi = yhi >> d;
    const uint64_t flo = d ? ((ylo >> d) | (yhi << (64 - d))) : ylo;
    const uint64_t rlo = ~xlo, rhi = ~xhi & key_mask(2 * k - 64);
    const bool fwd = fhi < rhi || (fhi == rhi && flo <= rlo);
    clo = fwd ? flo : rlo;
    chi = fwd ? fhi : rhi;
}

// Canonical code of the k-mer whose first base is packed base G, and
// whether its k bases are all ACGT, from the sequence words G / 32 .. + 2
// (w0..w2: the k-mer spans at most three) and the mask words G / 64 .. + 1.
IBS_HD void canonical_from_words(uint64_t w0, uint64_t w1, uint64_t w2, uint64_t m0, uint64_t m1, uint64_t G,
                                 uint32_t k, bool &acgt, uint64_t &clo, uint64_t &chi)
{
    const uint32_t sh = (uint32_t)(G & 31) * 2;
    const uint64_t xlo = (w0 >> sh) | ((w1 << (63 - sh)) << 1);
    const uint64_t xhi = (w1 >> sh) | ((w2 << (63 - sh)) << 1);
    const uint32_t ms = (uint32_t)(G & 63);
    const uint64_t mm = (m0 >> ms) | ((m1 << (63 - ms)) << 1);
    acgt = (mm & key_mask(k)) == 0;
    canonical_of_stream(xlo, xhi, k, clo, chi);
}

#if defined(__CUDACC__)
// The same reading the packed reference (the packed layout's tail padding
// covers the word after a contig's last).
__device__ __forceinline__ void canonical_at(const uint64_t *__restrict__ seq, const uint64_t *__restrict__ mask,
                                             uint64_t G, uint32_t k, bool &acgt, uint64_t &clo, uint64_t &chi)
{
    const uint64_t wi = G >> 5, mi = G >> 6;
    canonical_from_words(__ldg(seq + wi), __ldg(seq + wi + 1), __ldg(seq + wi + 2), __ldg(mask + mi),
                         __ldg(mask + mi + 1), G, k, acgt, clo, chi);
}

// A half line's four slots.
struct Half {
    uint4 v[4];
    __device__ __forceinline__ void load(const ulonglong2 *p)
    {
        load_sector(reinterpret_cast<const uint4 *>(p), v[0], v[1]);
        load_sector(reinterpret_cast<const uint4 *>(p) + 2, v[2], v[3]);
    }
    __device__ __forceinline__ bool holds(uint64_t lo, uint64_t hi) const
    {
        bool hit = false;
#pragma unroll
        for (int s = 0; s < 4; ++s)
            hit |= (v[s].x == (uint32_t)lo) & (v[s].y == (uint32_t)(lo >> 32)) & (v[s].z == (uint32_t)hi) &
                   (v[s].w == (uint32_t)(hi >> 32));
        return hit;
    }
    __device__ __forceinline__ bool full() const { return (v[3].x & v[3].y & v[3].z & v[3].w) != 0xffffffffu; }
};

// Membership of one wide key whose home half in level 0, starting at slot
// `home`, is full without it: the line's other half, then the next levels.
__device__ __forceinline__ bool lookup_rest(const View &t, uint64_t lo, uint64_t hi, uint64_t home)
{
    for (uint32_t L = 0;;) {
        Half x;
        x.load(t.slots[L] + (home ^ (kSlots / 2)));
        if (x.holds(lo, hi))
            return true;
        if (!x.full() || ++L == t.nLevels)
            return false;
        home = home_of(lo, hi, L, t.lines[L]);
        x.load(t.slots[L] + home);
        if (x.holds(lo, hi))
            return true;
        if (!x.full())
            return false;
    }
}

// The level-0 home halves of a warp's 32 keys, one per lane, read by pairs of
// lanes: each lane reads half of its pair's two halves, so a key's 64 bytes
// come by one load of two lanes. (By two loads of its own lane they are two
// requests, which fetch a line from DRAM twice when both are in flight: 17 G
// probes/s over 2 GB.) Every lane of the warp calls both functions.
struct PairProbe {
    uint4 a[2], b[2];        // this lane's share of the even and the odd lane's half
    uint64_t lo, hi, oLo, oHi; // this lane's key and its pair's

    __device__ __forceinline__ void load(const View &t, uint64_t lo_, uint64_t hi_, uint64_t home, uint32_t lane)
    {
        lo = lo_;
        hi = hi_;
        oLo = __shfl_xor_sync(0xffffffffu, lo, 1);
        oHi = __shfl_xor_sync(0xffffffffu, hi, 1);
        const uint64_t oHome = __shfl_xor_sync(0xffffffffu, home, 1);
        const bool odd = lane & 1;
        const ulonglong2 *base = t.slots[0] + (odd ? 2 : 0);
        load_sector(reinterpret_cast<const uint4 *>(base + (odd ? oHome : home)), a[0], a[1]);
        load_sector(reinterpret_cast<const uint4 *>(base + (odd ? home : oHome)), b[0], b[1]);
    }

    static __device__ __forceinline__ bool holds(const uint4 &v, uint64_t lo, uint64_t hi)
    {
        return (v.x == (uint32_t)lo) & (v.y == (uint32_t)(lo >> 32)) & (v.z == (uint32_t)hi) &
               (v.w == (uint32_t)(hi >> 32));
    }
    static __device__ __forceinline__ bool taken(const uint4 &v) { return (v.x & v.y & v.z & v.w) != 0xffffffffu; }

    // Whether this lane's half holds its key, and whether the half is full.
    __device__ __forceinline__ void result(uint32_t lane, bool &hit, bool &full) const
    {
        const bool odd = lane & 1;
        const uint64_t aLo = odd ? oLo : lo, aHi = odd ? oHi : hi, bLo = odd ? lo : oLo, bHi = odd ? hi : oHi;
        const uint32_t ha = __ballot_sync(0xffffffffu, holds(a[0], aLo, aHi) || holds(a[1], aLo, aHi));
        const uint32_t hb = __ballot_sync(0xffffffffu, holds(b[0], bLo, bHi) || holds(b[1], bLo, bHi));
        const uint32_t fa = __ballot_sync(0xffffffffu, taken(a[1])), fb = __ballot_sync(0xffffffffu, taken(b[1]));
        const uint32_t pair = lane & ~1u;
        hit = ((odd ? hb : ha) >> pair) & 3u;
        full = ((odd ? fb : fa) >> (pair + 1)) & 1u; // the odd lane has the last slot
    }
};

// Membership of one wide key.
__device__ __forceinline__ bool lookup(const View &t, uint64_t lo, uint64_t hi)
{
    const uint64_t home = home_of(lo, hi, 0, t.lines[0]);
    Half x;
    x.load(t.slots[0] + home);
    return x.holds(lo, hi) || (x.full() && lookup_rest(t, lo, hi, home));
}
#endif

} // namespace wide
} // namespace ibs
