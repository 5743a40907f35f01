// Minimizer-bucketed table (format MZ8): the key -> (bucket, slot) map.
//
// A k-mer is filed under its minimizer: among its w = k - m + 1 m-mers (m =
// k - 7 from k = 23, else 16), the one whose canonical form has the smallest
// rank key (27 bits derived from the m-mer's hash, below), ties going to the
// leftmost (placements() below has what that means on either strand).
// Consecutive reference positions mostly share their minimizer: the scan
// touches a new line every (w + 1) / 2 = 4.5 positions on average, and the
// random lines of a table beyond a few GB come at 36.4 G/s at most on a B200
// (one 32-byte load each; measured), which bounds the scan. m grows with k so
// that a minimizer rarely occurs at two loci of a large genome (4^18 18-mers
// against 2e9 positions), which would pile two runs into one place.
//
// The table is an array of 128-byte lines of four 32-byte sectors; a sector
// is a B8x32 bucket (format MZ8) or a B6x40 bucket (format MZ6). The
// minimizer picks the line and the slot value one of its four sectors, so a
// minimizer's k-mers spread over the line and a warp's loads for a run of
// positions touch one DRAM line.
//
// The slot value identifies the k-mer exactly inside its line: with g =
// line_hash(M) (a bijection of the 2m-bit canonical minimizer M), line = the
// top 32 bits of g scaled to [0, nLines), so the low hbits = 2m -
// floor(log2(nLines)) bits of g single out g, hence M, among the line's
// interval; the k-mer, on the strand where it holds M itself, is then M at
// offset o (< w <= 8) with the other k - m bases around it:
//   slot = (o << 2(k-m) | k-mer-without-the-m-mer) << hbits | (g mod 2^hbits)
// which has 2k + 3 - floor(log2(nLines)) bits and must fit the sector's slots:
// 31 bits in B8x32 sectors (format MZ8, the sentinels above), nLines >=
// 2^(2k-28); 40 bits in B6x40 sectors (format MZ6, for k up to 31), nLines
// >= 2^(2k-37).
#pragma once

#include "ibs_core.cuh"

namespace ibs {
namespace mz {

constexpr uint32_t kSectorsPerLine = 4;
// Flags of a key in the builds' lists of keys without a slot (2k <= 62 bits):
// its second place is meant, or it has none (not canonical).
constexpr uint64_t kSecondPlace = 1ull << 63, kNoPlace = 1ull << 62;

IBS_HD uint32_t m_of(uint32_t k) { return k >= 23 ? k - 7 : 16; }
IBS_HD uint32_t w_of(uint32_t k) { return k - m_of(k) + 1; }

IBS_HD uint64_t brev64(uint64_t x)
{
#if defined(__CUDA_ARCH__)
    return __brevll(x);
#else
    x = ((x >> 1) & 0x5555555555555555ull) | ((x & 0x5555555555555555ull) << 1);
    x = ((x >> 2) & 0x3333333333333333ull) | ((x & 0x3333333333333333ull) << 2);
    x = ((x >> 4) & 0x0f0f0f0f0f0f0f0full) | ((x & 0x0f0f0f0f0f0f0f0full) << 4);
    x = ((x >> 8) & 0x00ff00ff00ff00ffull) | ((x & 0x00ff00ff00ff00ffull) << 8);
    x = ((x >> 16) & 0x0000ffff0000ffffull) | ((x & 0x0000ffff0000ffffull) << 16);
    return (x >> 32) | (x << 32);
#endif
}

// Reverse complement of an m-mer code (first base in the high bits).
IBS_HD uint64_t rc_m(uint64_t v, uint32_t m)
{
    uint64_t y = brev64(v);
    y = ((y >> 1) & 0x5555555555555555ull) | ((y & 0x5555555555555555ull) << 1);
    return ~y >> (64 - 2 * m);
}

IBS_HD uint64_t canon_m(uint64_t v, uint32_t m)
{
    const uint64_t r = rc_m(v, m);
    return v < r ? v : r;
}

// A canonical m-mer's hash, a bijection of its 2m bits (32 <= 2m <= 50) on two
// 32-bit words (lo from the m-mer's top 32 bits, hi its 2m - 32 low bits,
// which stay as they are): the scan computes one per reference position, so
// it is five instructions; the 64-bit multiply-xorshift rounds it replaces
// were about 18. Given hi, each step is a bijection of lo.
struct Mixed {
    uint32_t lo, hi;
};

IBS_HD Mixed mix(uint32_t top, uint32_t rest)
{
    uint32_t y = top * 0xd6e8feb9u + rest * 0x85ebca6bu;
    y ^= y >> 15;
    return Mixed{y * 0xbf58476du, rest};
}

IBS_HD Mixed mix_m(uint64_t canonical, uint32_t m)
{
    const uint32_t hb = 2 * m - 32;
    return mix((uint32_t)(canonical >> hb), (uint32_t)canonical & ((1u << hb) - 1u));
}

// The line hash of a canonical m-mer: its hash as one 2m-bit number.
IBS_HD uint64_t line_hash_of(const Mixed &x, uint32_t m) { return ((uint64_t)x.lo << (2 * m - 32)) | x.hi; }

IBS_HD uint64_t line_hash(uint64_t canonical, uint32_t m) { return line_hash_of(mix_m(canonical, m), m); }

// The key minimizers are chosen by: a multiple of the hash's words with its
// low 5 bits clear, where the scan keeps a window offset and an orientation,
// so that one integer minimum per step finds the leftmost smallest key. The
// line index comes from lo's high bits; for every fixed line the multiples of
// lo's low bits and of hi are spread evenly over the key range (golden-ratio
// multipliers), so picking small keys does not crowd lines.
IBS_HD uint32_t rank_key_of(const Mixed &x) { return x.lo * (0x9e3779b1u << 5) + x.hi * (0x94d049bbu << 5); }

IBS_HD uint32_t rank_key(uint64_t canonical, uint32_t m) { return rank_key_of(mix_m(canonical, m)); }

// The m-mer of C (2k-bit code, first base high) at offset o.
IBS_HD uint64_t mmer_at(uint64_t C, uint32_t k, uint32_t o, uint32_t m)
{
    return (C >> (2 * (k - m - o))) & key_mask(2 * m);
}

// (o, D without the m-mer) part of the slot value, D being the k-mer on the
// strand where its minimizer reads as its canonical form and o the
// minimizer's offset there: the k - m other bases are taken by rotating D
// left by 2o bits inside its 2k, which puts the m-mer on top and below it the
// bases right of the m-mer followed by the o bases left of it. 2(k - m) + 3
// <= 17 bits; m >= 16 and o <= k - m keep both shifts below 32.
IBS_HD uint32_t slot_high(uint64_t D, uint32_t k, uint32_t o)
{
    const uint32_t m = m_of(k);
    const uint32_t lo = (uint32_t)D, hi = (uint32_t)(D >> 32);
    const uint32_t rest = ((lo << (2 * o)) | (hi >> (2 * k - 32 - 2 * o))) & (uint32_t)key_mask(2 * (k - m));
    return (o << (2 * (k - m))) | rest;
}

// Sector of a k-mer inside its line: the top two bits of a golden-ratio
// multiple of its slot value's two halves folded together. The slot value
// names the k-mer within its line, so it spreads the line's k-mers, and a
// probe that has the slot value needs nothing else.
IBS_HD uint32_t sector_of(uint32_t slotLo, uint32_t slotHi) { return ((slotLo ^ slotHi) * 0x9e3779b1u) >> 30; }

// Line of a minimizer with line hash g (2m >= 32 bits) among nLines < 2^32:
// the top 32 bits of g scaled to [0, nLines). Those of one line form an
// interval of at most ceil(2^32 / nLines) values, so the g of a line form an
// interval of at most 2^(2m - floor(log2 nLines)) = 2^hbits values and
// g mod 2^hbits singles g out in its line.
IBS_HD uint64_t line_of(uint64_t g, uint32_t m, uint64_t nLines)
{
    const uint32_t top = (uint32_t)(g >> (2 * m - 32));
#if defined(__CUDA_ARCH__)
    return __umulhi(top, (uint32_t)nLines);
#else
    return ((uint64_t)top * (uint32_t)nLines) >> 32;
#endif
}

// Bucket (32-byte sector index) and slot value of the k-mer D (either strand)
// whose minimizer sits at offset o, with line hash g; s is 1 when D holds the
// minimizer's reverse complement there: the k-mer then goes by its other
// strand. hbits = 2m - floor(log2(nLines)).
IBS_HD void place(uint64_t D, uint32_t k, uint32_t o, uint32_t s, uint64_t g, uint64_t nBuckets,
                  uint32_t hbits, uint64_t &bucket, uint64_t &slot)
{
    if (s) {
        D = rc_m(D, k);
        o = w_of(k) - 1 - o;
    }
    slot = ((uint64_t)slot_high(D, k, o) << hbits) | (g & key_mask(hbits));
    bucket = line_of(g, m_of(k), nBuckets / kSectorsPerLine) * kSectorsPerLine +
             sector_of((uint32_t)slot, (uint32_t)(slot >> 32));
}

// Offsets of the leftmost and the rightmost smallest rank key among the w (<= 8)
// m-mers of C; R is C's reverse complement. The m-mers come as words by shifts
// of a known amount each from C at the top of 64 bits and from R, and the
// offsets ride in the keys' low bits.
IBS_HD void minimizer_offsets(uint64_t C, uint64_t R, uint32_t k, uint32_t &left, uint32_t &right)
{
    const uint32_t m = m_of(k), w = w_of(k), hb = 2 * m - 32, restMask = (1u << hb) - 1u;
    const uint64_t X = C << (64 - 2 * k), R1 = R >> hb;
    uint32_t bestL = 0xffffffffu, bestR = 0xffffffffu;
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (uint32_t j = 0; j < 8; ++j) {
        if (j >= w)
            break;
        const uint32_t fh = (uint32_t)((X << (2 * j)) >> 32), fl = (uint32_t)X << (2 * j);
        const uint32_t fr = hb ? fl >> (32 - hb) : 0u;
        const uint32_t rh = (uint32_t)(R1 >> (2 * j)), rr = (uint32_t)(R >> (2 * j)) & restMask;
        const bool rLess = rh < fh || (rh == fh && rr < fr);
        const uint32_t key = rank_key_of(mix(rLess ? rh : fh, rLess ? rr : fr));
        bestL = bestL < key + j ? bestL : key + j;
        bestR = bestR < key + (7 - j) ? bestR : key + (7 - j);
    }
    left = bestL & 7u;
    right = 7u - (bestR & 7u);
}

// The place of k-mer D (D2 its reverse complement) by its minimizer at offset o.
IBS_HD void place_at(uint64_t D, uint64_t D2, uint32_t o, const TableGeom &g, uint64_t &bucket, uint64_t &slot)
{
    const uint32_t k = g.k, m = m_of(k);
    const uint64_t mmask = key_mask(2 * m);
    const uint64_t f = (D >> (2 * (k - m - o))) & mmask, r = (D2 >> (2 * o)) & mmask;
    const bool rev = r < f;
    const uint64_t h = line_hash(rev ? r : f, m);
    const uint64_t own = rev ? D2 : D; // the strand that holds the minimizer itself
    const uint32_t at = rev ? w_of(k) - 1 - o : o;
    slot = ((uint64_t)slot_high(own, k, at) << g.fpBits) | (h & key_mask(g.fpBits));
    bucket = line_of(h, m, g.nBuckets / kSectorsPerLine) * kSectorsPerLine +
             sector_of((uint32_t)slot, (uint32_t)(slot >> 32));
}

// The places of canonical k-mer C: where a scan that reads C looks (by C's
// leftmost smallest rank key), and where one that reads the other strand
// does. They are one place but for a k-mer whose smallest key occurs at
// several offsets (a short tandem repeat: leftmost on one strand is rightmost
// on the other), or whose minimizer is its own reverse complement; such a
// k-mer is filed under both, so that a scan needs no look at which strand is
// canonical. Returns how many (1 or 2; [0] is C's), and 0 for a code that is
// not canonical: no scan asks for it, and a table keeps it in the stash, by
// the code itself.
IBS_HD uint32_t placements(uint64_t C, const TableGeom &g, uint64_t bucket[2], uint64_t slot[2])
{
    const uint64_t R = rc_m(C, g.k);
    if (R < C)
        return 0;
    const uint32_t m = m_of(g.k);
    uint32_t left, right;
    minimizer_offsets(C, R, g.k, left, right);
    place_at(C, R, left, g, bucket[0], slot[0]);
    if (left == right) {
        if (m & 1) // never its own reverse complement
            return 1;
        const uint64_t f = (C >> (2 * (g.k - m - left))) & key_mask(2 * m);
        if (f != ((R >> (2 * left)) & key_mask(2 * m)))
            return 1;
    }
    place_at(R, C, w_of(g.k) - 1 - right, g, bucket[1], slot[1]);
    return bucket[0] == bucket[1] && slot[0] == slot[1] ? 1 : 2;
}

// The place where a probe for the k-mer's code looks; false for a code that is
// not canonical.
IBS_HD bool locate(uint64_t C, const TableGeom &g, uint64_t &bucket, uint64_t &slot)
{
    const uint64_t R = rc_m(C, g.k);
    bucket = slot = 0;
    if (R < C)
        return false;
    uint32_t left, right;
    minimizer_offsets(C, R, g.k, left, right);
    place_at(C, R, left, g, bucket, slot);
    return true;
}

} // namespace mz
} // namespace ibs
