// Host build of the minimizer tables' key map, as the scan kernel's located
// blocks use it (gpu-ibs_b200/csrc/mz_scan.cuh) and as the build files keys
// (mz::placements, gpu-ibs_b200/csrc/mz_core.cuh).
#include <cstdint>

#include "mz_core.cuh"

using namespace ibs;

// Of the positions of `bases` (values 0-3): how many look, by the leftmost
// smallest rank key on the strand read and with the k-mer on its minimizer's
// strand, at a place that the build does not file the canonical k-mer under.
extern "C" uint64_t mz_unfiled(const uint8_t *bases, uint64_t n, uint32_t k, uint64_t nBuckets)
{
    TableGeom g{};
    g.k = k;
    g.bits = 2 * k;
    g.format = FMT_MZ8;
    g.nBuckets = nBuckets;
    const uint32_t m = mz::m_of(k), w = mz::w_of(k);
    g.fpBits = 2 * m - (63 - __builtin_clzll(nBuckets / mz::kSectorsPerLine));
    uint64_t bad = 0;
    for (uint64_t q = 0; q + k <= n; ++q) {
        uint64_t F = 0;
        for (uint32_t t = 0; t < k; ++t)
            F = (F << 2) | bases[q + t];
        const uint64_t R = mz::rc_m(F, k);
        uint32_t best = 0, o = 0;
        for (uint32_t j = 0; j < w; ++j) {
            const uint32_t key = mz::rank_key(mz::canon_m(mz::mmer_at(F, k, j, m), m), m);
            if (j == 0 || key < best) {
                best = key;
                o = j;
            }
        }
        const uint64_t f = mz::mmer_at(F, k, o, m), r = mz::rc_m(f, m);
        uint64_t bucket, slot, b[2], s[2];
        mz::place(F, k, o, r < f, mz::line_hash(mz::canon_m(f, m), m), nBuckets, g.fpBits, bucket, slot);
        const uint32_t places = mz::placements(F < R ? F : R, g, b, s);
        bool found = false;
        for (uint32_t a = 0; a < places; ++a)
            found |= b[a] == bucket && s[a] == slot;
        bad += found ? 0 : 1;
    }
    return bad;
}
