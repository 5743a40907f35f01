// Device table: KMC 3 decode and the sector-bucket build.
//
// ibs_open reads the KMC 3 random-access files with the same layout rules as
// the reference's KmcRaIndex (src/gpu/KmcRaIndex.hpp:497-708): header fields
// and version from the end of .kmc_pre, the bin-major prefix LUT with KMC's
// total+1 guard, and big-endian suffix records followed by counter bytes in
// .kmc_suf. Records are decoded on the device (prefix from the LUT bucket,
// suffix bytes to an integer, counters dropped) straight into canonical
// codes, which the build then hashes into 32-byte buckets.
#include "ibs_internal.cuh"

#include <cooperative_groups.h>

#include <chrono>
#include <cstdio>
#include <cstring>
#include <memory>
#include <condition_variable>
#include <mutex>
#include <thread>
#include <unistd.h>

namespace ibs {

// ---------------------------------------------------------------------------
// errors
// ---------------------------------------------------------------------------
static thread_local std::string g_error;

void set_error(const std::string &msg) { g_error = msg; }
void clear_error() { g_error.clear(); }

std::atomic<uint64_t> &launch_counter()
{
    static std::atomic<uint64_t> c{0};
    return c;
}

ibs_status cuda_fail(cudaError_t e, const char *what)
{
    set_error(std::string("CUDA error in ") + what + ": " + cudaGetErrorString(e));
    cudaGetLastError(); // clear a sticky-free error so the next call starts clean
    return e == cudaErrorMemoryAllocation ? IBS_ERR_NOMEM : IBS_ERR_CUDA;
}

// ---------------------------------------------------------------------------
// geometry
// ---------------------------------------------------------------------------
static uint32_t floor_log2(uint64_t x) { return 63u - (uint32_t)__builtin_clzll(x); }

static uint64_t next_pow2(uint64_t x)
{
    uint64_t p = 1;
    while (p < x)
        p <<= 1;
    return p;
}

static TableGeom choose_geometry(uint64_t nKeys, uint32_t k, const ibs_table_opts *o)
{
    TableGeom g{};
    g.k = k;
    g.bits = 2 * k;
    uint32_t fmt = o ? o->force_format : 0;
    const bool tunedMz = tuning().table_format == FMT_MZ8;
    // minimum line count of a minimizer table: its slot values must fit 31
    // bits (B8x32 sectors, k <= 27) or 40 bits (B6x40 sectors, k <= 31)
    auto mzMinLog2 = [&](uint32_t f) { return (int)(2 * k) - (f == FMT_MZ8 ? 28 : 37); };
    if (fmt == 0 && tunedMz && k >= 16 && k <= 31) {
        // the tuned default, from twice the layout's minimum line count on.
        // Between the two a table fits minimizer lines as well, and scans of it
        // are twice as fast (250 Mbp at k = 31: 2.0 ms on 7.8 GB of lines, 5.5
        // on 3.1 GB of hash sectors), but it takes 2.6 times the memory, which
        // callers who keep many tables have planned: force_format asks for it.
        const uint32_t f = k <= 27 ? FMT_MZ8 : FMT_MZ6;
        const int from = mzMinLog2(f) + 1;
        const double want = (double)nKeys / tuning().keys_per_bucket / mz::kSectorsPerLine;
        if (from <= 0 || want >= (double)(1ull << from))
            fmt = f;
    }
    if (fmt == FMT_AUTO_HASH)
        fmt = 0;
    // the tuned load belongs to the tuned layout; hash tables under a tuned
    // minimizer default keep the hash layout's default of 4 keys per bucket
    double lam = tuning().keys_per_bucket;
    if (tunedMz && !is_mz(fmt))
        lam = 4.0;
    if (o && o->keys_per_bucket > 0)
        lam = o->keys_per_bucket;
    const uint64_t space = g.bits >= 64 ? ~0ull : (1ull << g.bits);
    auto clampN = [&](uint64_t n) {
        if (n < 1)
            n = 1;
        if (g.bits < 64 && n > space)
            n = space;
        return n;
    };
    const uint64_t n8 = clampN((uint64_t)((double)nKeys / lam) + 1);
    const uint64_t min8 = g.bits > 31 ? (1ull << (g.bits - 31)) : 1;
    const uint64_t n6 = clampN((uint64_t)((double)nKeys / (lam * 6.0 / 8.0)) + 1);
    const uint64_t min6 = g.bits > 40 ? (1ull << (g.bits - 40)) : 1;
    if (is_mz(fmt)) {
        // minimizer lines of four sectors, at least 2^mzMinLog2 of them
        g.format = fmt;
        const uint32_t m = mz::m_of(k);
        const uint64_t minLines = mzMinLog2(fmt) > 0 ? (1ull << mzMinLog2(fmt)) : 1;
        const uint64_t want = fmt == FMT_MZ8 ? n8 : n6; // sectors at the load
        const uint64_t nLines =
            std::min<uint64_t>(std::max((want + mz::kSectorsPerLine - 1) / mz::kSectorsPerLine, minLines),
                               1ull << 31); // line_of needs nLines < 2^32
        g.nBuckets = nLines * mz::kSectorsPerLine;
        g.fpBits = 2 * m - floor_log2(nLines);
        g.stashBuckets = 0;
        return g;
    }
    if (fmt == 0)
        fmt = (std::max(n8, min8) <= 2 * n8) ? FMT_B8X32 : FMT_B6X40;
    g.format = fmt;
    g.nBuckets = fmt == FMT_B8X32 ? std::max(n8, min8) : std::max(n6, min6);
    g.nBuckets = clampN(g.nBuckets);
    int fpb = (int)g.bits - (int)floor_log2(g.nBuckets);
    g.fpBits = (uint32_t)std::max(fpb, 1);
    g.stashBuckets = 0;
    return g;
}

// ---------------------------------------------------------------------------
// build kernels
// ---------------------------------------------------------------------------
// Buckets and stored fingerprints of a key in either table family; returns how
// many places it has (a minimizer table files a k-mer whose leftmost and
// rightmost minimizers differ under both: mz::placements).
__device__ __forceinline__ uint32_t locate_key(uint64_t code, const TableGeom &g, uint64_t r[2], uint64_t fp[2])
{
    if (is_mz(g.format))
        return mz::placements(code, g, r, fp);
    const uint64_t h = perm_hash(code, g.bits);
    r[0] = bucket_of(h, g);
    fp[0] = fp_of(h, g);
    return 1;
}

__device__ __forceinline__ bool stash_insert(uint64_t *stash, uint64_t stashBuckets, uint64_t code)
{
    uint64_t b = stash_home(code, stashBuckets);
    for (uint64_t i = 0; i < stashBuckets; ++i) {
        for (int s = 0; s < 4; ++s) {
            unsigned long long *slot = reinterpret_cast<unsigned long long *>(stash + 4 * b + s);
            const unsigned long long old = atomicCAS(slot, (unsigned long long)STASH_EMPTY,
                                                     (unsigned long long)code);
            if (old == STASH_EMPTY || old == code)
                return true;
        }
        b = (b + 1) & (stashBuckets - 1);
    }
    return false;
}

// ---- placement ---------------------------------------------------------------
// Every key takes a free slot of its bucket in one pass over the keys
// (k_fill): the bucket is read and the slot claimed by a compare-and-swap on
// the same line, so a key costs one random line. (Counting the keys of every
// bucket first and placing them in a second pass touched three: 14 ms against
// 7 for 220M keys.) Keys that find no slot go to a list, and a second, small
// pass (k_spill) settles those.

// Claims one of 32-bit slots [0, last) of a B8x32 bucket for fp, the first free
// one; true when it is there (an equal value there already counts: a duplicate
// key). (Starting each search at a slot of the value's own, so that the keys of
// one minimizer, which come together, do not all try the same one, took 12.9
// ms against 7.1 for 220M keys.)
__device__ __forceinline__ bool claim8(uint32_t *w, uint32_t fp, uint32_t last)
{
    const uint4 a = __ldcg(reinterpret_cast<const uint4 *>(w)), b = __ldcg(reinterpret_cast<const uint4 *>(w) + 1);
    const uint32_t v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (uint32_t j = 0; j < 8; ++j) {
        if (j >= last)
            break;
        if (v[j] == fp)
            return true;
        if (v[j] == B8_EMPTY) {
            const uint32_t old = atomicCAS(w + j, B8_EMPTY, fp);
            if (old == B8_EMPTY || old == fp)
                return true;
        }
    }
    return false;
}

// The same for a B6x40 bucket, whose count byte says which slots are taken.
__device__ __forceinline__ bool claim6(uint32_t *w, uint64_t fp)
{
    uint32_t old = __ldcg(w + 7);
    for (int tries = 0; tries < 1 << 20; ++tries) {
        const uint32_t s = (old >> 16) & 0xffu;
        if (s >= 6)
            return false;
        const uint32_t seen = atomicCAS(w + 7, old, old + (1u << 16));
        if (seen == old) {
            w[s] = (uint32_t)(fp >> 8);
            // bytes 24 .. 29: two of them share word 7 with the count
            atomicOr(w + 6 + s / 4, (uint32_t)(fp & 0xff) << (8 * (s & 3)));
            return true;
        }
        old = seen;
    }
    return false;
}

// A place in a list for each lane that calls it, one atomic for all of them
// (with one each, 66M keys at 8 a bucket took 7.7 ms to build, so 6.2).
__device__ __forceinline__ unsigned long long list_place(unsigned long long *listN)
{
    const auto lanes = cooperative_groups::coalesced_threads();
    unsigned long long at = 0;
    if (lanes.thread_rank() == 0)
        at = atomicAdd(listN, (unsigned long long)lanes.size());
    return lanes.shfl(at, 0) + lanes.thread_rank();
}

// Slot 7 of a B8x32 bucket stays free in this pass: it becomes a key's when
// one key is left over, or the marker when there are more.
__global__ void k_fill(const uint64_t *__restrict__ codes, uint64_t n, TableGeom g, uint32_t *__restrict__ words,
                       uint64_t *__restrict__ list, unsigned long long *__restrict__ listN, uint64_t listCap)
{
    const bool b8 = g.format == FMT_B8X32 || g.format == FMT_MZ8;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t code = codes[i];
        uint64_t rr[2], ff[2];
        const uint32_t places = locate_key(code, g, rr, ff);
        for (uint32_t a = 0; a < places || a == 0; ++a) {
            const uint64_t r = a ? rr[1] : rr[0], fp = a ? ff[1] : ff[0];
            if (places && (b8 ? claim8(words + r * 8, (uint32_t)fp, 7) : claim6(words + r * 8, fp)))
                continue;
            const unsigned long long j = list_place(listN);
            if (j < listCap)
                list[j] = code | (!places ? mz::kNoPlace : a ? mz::kSecondPlace : 0ull);
        }
    }
}

// B8x32 sectors: the number of listed keys of each bucket, up to 3, two bits a
// bucket.
__global__ void k_count_left(const uint64_t *__restrict__ list, const unsigned long long *__restrict__ listN,
                             uint64_t listCap, TableGeom g, uint32_t *__restrict__ left)
{
    const uint64_t n = *listN <= listCap ? *listN : 0; // a list that overran is filled again
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const bool mz = is_mz(g.format);
        if (mz && (list[i] & mz::kNoPlace))
            continue;
        uint64_t rr[2], ff[2];
        locate_key(mz ? list[i] & ~mz::kSecondPlace : list[i], g, rr, ff);
        const uint64_t r = mz && (list[i] & mz::kSecondPlace) ? rr[1] : rr[0];
        // the first key sets the low bit, any further one the high bit
        const uint32_t one = 1u << (2 * (r & 15));
        if (atomicOr(left + (r >> 4), one) & one)
            atomicOr(left + (r >> 4), one << 1);
    }
}

// Settles the listed keys: a B8x32 bucket's only one takes slot 7; otherwise
// a minimizer line's go to the line's free slots, the partner sector's first
// (a sector's slot 7 only where that sector has no listed keys of its own),
// and what is left, as every listed key of a hash bucket, stays in the list for
// the stash (the others' entries become STASH_EMPTY, which is no key). The home
// bucket's marker says how far.
__global__ void k_spill(uint64_t *__restrict__ list, const unsigned long long *__restrict__ listN, uint64_t listCap,
                        TableGeom g, const uint32_t *__restrict__ left, uint32_t *__restrict__ words,
                        unsigned long long *__restrict__ stashN)
{
    const uint64_t n = *listN <= listCap ? *listN : 0;
    const bool b8 = g.format == FMT_B8X32 || g.format == FMT_MZ8, mz = is_mz(g.format);
    uint32_t stashed = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t entry = list[i], code = mz ? entry & ~(mz::kSecondPlace | mz::kNoPlace) : entry;
        if (mz && (entry & mz::kNoPlace)) {
            list[i] = code;
            ++stashed;
            continue;
        }
        uint64_t rr[2], ff[2];
        locate_key(code, g, rr, ff);
        const uint32_t a = mz ? (uint32_t)(entry >> 63) : 0; // which of its places
        const uint64_t r = a ? rr[1] : rr[0], fp = a ? ff[1] : ff[0];
        uint32_t *home = words + r * 8;
        auto left_of = [&](uint64_t x) { return (left[x >> 4] >> (2 * (x & 15))) & 3u; };
        if (b8 && left_of(r) == 1u) {
            home[7] = (uint32_t)fp;
            list[i] = STASH_EMPTY;
            continue;
        }
        uint32_t reach = 3;
        for (uint32_t d = 1; d < 4 && mz && reach == 3; ++d) {
            uint32_t *w = words + (r ^ d) * 8;
            if (b8 ? claim8(w, (uint32_t)fp, left_of(r ^ d) ? 7 : 8) : claim6(w, fp))
                reach = d == 1 ? 1 : 2;
        }
        list[i] = reach == 3 ? code : STASH_EMPTY;
        stashed += reach == 3;
        if (!mz)
            reach = 1; // hash buckets: the marker (B8_OVERFLOW, flag bit 0) means the stash
        if (b8)
            atomicMin(home + 7, 0xffffffffu - reach); // EMPTY, then the markers downwards
        else
            atomicOr(home + 7, reach << 24); // 1 | 2 reads as 3: one place more is looked at
    }
    stashed = __reduce_add_sync(0xffffffffu, stashed);
    if ((threadIdx.x & 31) == 0 && stashed)
        atomicAdd(stashN, (unsigned long long)stashed);
}

__global__ void k_stash(const uint64_t *__restrict__ list, uint64_t n, uint64_t *__restrict__ stash,
                        uint64_t stashBuckets, int *__restrict__ err)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x)
        if (list[i] != STASH_EMPTY && !stash_insert(stash, stashBuckets, list[i]))
            atomicExch(err, 1);
}

// Record r of a .kmc_suf chunk -> canonical code. The LUT bucket j holding
// record r is the last j with lut[j] <= r (empty buckets repeat a value and
// are skipped by taking the last); j mod 4^p is the prefix.
__global__ void k_decode(const uint8_t *__restrict__ raw, uint64_t r0, uint64_t nRec,
                         uint32_t recBytes, uint32_t sufBytes, const uint64_t *__restrict__ lut,
                         uint64_t lutN, uint64_t prefixMask, uint32_t sufBits,
                         uint64_t *__restrict__ out)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nRec;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t r = r0 + i;
        uint64_t lo = 0, hi = lutN - 1;
        while (lo < hi) {
            const uint64_t mid = (lo + hi + 1) >> 1;
            if (__ldg(lut + mid) <= r)
                lo = mid;
            else
                hi = mid - 1;
        }
        const uint8_t *q = raw + i * recBytes;
        uint64_t suf = 0;
        for (uint32_t b = 0; b < sufBytes; ++b)
            suf = (suf << 8) | q[b];
        const uint64_t prefix = lo & prefixMask;
        out[r] = sufBits >= 64 ? suf : ((prefix << sufBits) | suf);
    }
}

// The same for 33 <= k <= 64: the suffix (up to 16 bytes) and the prefix
// shifted above it as a 128-bit code {lo, hi}; sufBits = 2 (k - p) > 0.
__global__ void k_decode_wide(const uint8_t *__restrict__ raw, uint64_t r0, uint64_t nRec, uint32_t recBytes,
                              uint32_t sufBytes, const uint64_t *__restrict__ lut, uint64_t lutN,
                              uint64_t prefixMask, uint32_t sufBits, ulonglong2 *__restrict__ out)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nRec;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t r = r0 + i;
        uint64_t lo = 0, hi = lutN - 1;
        while (lo < hi) {
            const uint64_t mid = (lo + hi + 1) >> 1;
            if (__ldg(lut + mid) <= r)
                lo = mid;
            else
                hi = mid - 1;
        }
        const uint8_t *q = raw + i * recBytes;
        uint64_t slo = 0, shi = 0;
        for (uint32_t b = 0; b < sufBytes; ++b) {
            shi = (shi << 8) | (slo >> 56);
            slo = (slo << 8) | q[b];
        }
        const uint64_t prefix = lo & prefixMask;
        if (sufBits >= 64) {
            shi |= prefix << (sufBits - 64);
        } else {
            slo |= prefix << sufBits;
            shi |= prefix >> (64 - sufBits);
        }
        out[r] = make_ulonglong2(slo, shi);
    }
}

template <uint32_t FMT>
__global__ void k_probe(TableView t, const uint64_t *__restrict__ codes, uint64_t n,
                        uint8_t *__restrict__ hits)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x)
        hits[i] = table_lookup<FMT>(t, codes[i]) ? 1 : 0;
}

// Number of codes present in the table: each thread counts its share, each
// warp adds its lanes' counts and one lane adds the warp's to the total.
template <uint32_t FMT>
__global__ void k_count_present(TableView t, const uint64_t *__restrict__ codes, uint64_t n,
                                unsigned long long *__restrict__ count)
{
    unsigned long long local = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x)
        local += table_lookup<FMT>(t, codes[i]) ? 1 : 0;
    for (int o = 16; o; o >>= 1)
        local += __shfl_xor_sync(0xffffffffu, local, o);
    if ((threadIdx.x & 31) == 0 && local)
        atomicAdd(count, local);
}

static int grid_for(uint64_t n, int threads)
{
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const uint64_t want = (n + threads - 1) / threads;
    const uint64_t cap = (uint64_t)sms * 16;
    return (int)std::max<uint64_t>(1, std::min(want, cap));
}

// Builds the table from device codes. The caller has set the device.
static ibs_status build_from_device_codes(ibs_table *t, const uint64_t *dCodes, uint64_t n,
                                          uint32_t k, const ibs_table_opts *o)
{
    t->geom = choose_geometry(n, k, o);
    t->nKeys = n;
    TableGeom &g = t->geom;
    const uint64_t nb = g.nBuckets;
    const bool b8 = g.format == FMT_B8X32 || g.format == FMT_MZ8;
    // 32 bytes past the buckets hold the membership counts' total: an 8-byte
    // allocation of their own cost up to 0.6 ms a call
    IBS_CUDA(cudaMalloc(&t->buckets, nb * 32 + 32), "table alloc");
    t->deviceBytes = nb * 32;
    uint32_t *words = reinterpret_cast<uint32_t *>(t->buckets);
    // scratch in one allocation: counts (listed keys, keys for the stash, error),
    // the list, and two bits a bucket
    const uint64_t leftBytes = b8 ? (nb + 15) / 16 * 4 : 0;
    std::unique_ptr<uint8_t, cudaError_t (*)(void *)> scratch(nullptr, cudaFree);
    unsigned long long *dCounts = nullptr;
    uint64_t *list = nullptr;
    uint32_t *left = nullptr;
    unsigned long long counts[2] = {0, 0};
    // The list has room for the keys that hash buckets leave (2.4% at the default
    // load, 40% at 12 keys a bucket), and a little more; minimizer lines leave
    // about 2% at theirs. A table that leaves more (a forced load of lines, many
    // duplicates) is filled again with a list of the size that it then needs
    // (which of several equal keys are listed can differ from pass to pass), at
    // most of every place of every key. (Filled twice, 66M keys
    // at 8 a bucket took 11.6 ms, filled once 7.7.)
    const double share = is_mz(g.format) ? 1.0 / 16 : overflow_fraction((double)n / (double)nb, b8 ? 7 : 6) * 1.02 + 1.0 / 64;
    uint64_t listCap = (uint64_t)((double)n * share) + 4096;
    const uint64_t most = n * (is_mz(g.format) ? 2 : 1) + 4096;
    for (int attempt = 0;; ++attempt) {
        void *mem = nullptr;
        IBS_CUDA(cudaMalloc(&mem, 32 + listCap * 8 + leftBytes), "table build scratch");
        scratch.reset(static_cast<uint8_t *>(mem));
        dCounts = static_cast<unsigned long long *>(mem);
        list = reinterpret_cast<uint64_t *>(dCounts + 4);
        left = reinterpret_cast<uint32_t *>(list + listCap);
        IBS_CUDA(cudaMemsetAsync(t->buckets, b8 ? 0xff : 0x00, nb * 32, 0), "table init");
        IBS_CUDA(cudaMemsetAsync(dCounts, 0, 32, 0), "table build scratch");
        if (n) {
            k_fill<<<grid_for(n, 256), 256>>>(dCodes, n, g, words, list, dCounts, listCap);
            IBS_LAUNCHED();
            if (b8) {
                IBS_CUDA(cudaMemsetAsync(left, 0, leftBytes, 0), "table build scratch");
                k_count_left<<<grid_for(listCap, 256), 256>>>(list, dCounts, listCap, g, left);
                IBS_LAUNCHED();
            }
            k_spill<<<grid_for(listCap, 256), 256>>>(list, dCounts, listCap, g, left, words, dCounts + 1);
            IBS_LAUNCHED();
        }
        IBS_CUDA(cudaMemcpy(counts, dCounts, 16, cudaMemcpyDeviceToHost), "table build");
        if (counts[0] <= listCap)
            break;
        scratch.reset();
        listCap = std::min<uint64_t>(attempt ? 2 * counts[0] : counts[0] + counts[0] / 16 + 4096, most);
    }
    t->stashKeys = counts[1];
    if (!counts[1])
        return IBS_OK;
    const uint64_t stashBuckets = next_pow2((counts[1] * 2 + 3) / 4);
    IBS_CUDA(cudaMalloc(&t->stash, stashBuckets * 32), "stash alloc");
    g.stashBuckets = stashBuckets;
    t->deviceBytes += stashBuckets * 32;
    IBS_CUDA(cudaMemsetAsync(t->stash, 0xff, stashBuckets * 32, 0), "stash alloc");
    k_stash<<<grid_for(counts[0], 256), 256>>>(list, counts[0], t->stash, stashBuckets,
                                               reinterpret_cast<int *>(dCounts + 2));
    IBS_LAUNCHED();
    int herr = 0;
    IBS_CUDA(cudaMemcpy(&herr, dCounts + 2, sizeof herr, cudaMemcpyDeviceToHost), "table build stash");
    if (herr) {
        set_error("table build: stash full");
        return IBS_ERR_CAPACITY;
    }
    return IBS_OK;
}

// ---------------------------------------------------------------------------
// KMC 3 files (layout as read by src/gpu/KmcRaIndex.hpp:497-708)
// ---------------------------------------------------------------------------
struct KmcHeader {
    uint32_t version = 0, k = 0, mode = 0, counterSize = 0, p = 0, sigLen = 0;
    uint64_t total = 0, headerOffset = 0, fileBytes = 0;
};

struct File {
    FILE *f = nullptr;
    explicit File(const std::string &path) { f = fopen(path.c_str(), "rb"); }
    ~File()
    {
        if (f)
            fclose(f);
    }
};

static bool read_at(FILE *f, long long off, void *dst, size_t n)
{
    if (fseeko(f, off, SEEK_SET) != 0)
        return false;
    return fread(dst, 1, n, f) == n;
}

static uint64_t file_size(FILE *f)
{
    fseeko(f, 0, SEEK_END);
    return (uint64_t)ftello(f);
}

static ibs_status check_markers(FILE *f, uint64_t size, const char *marker, const std::string &path)
{
    char head[4], tail[4];
    if (size < 8 || !read_at(f, 0, head, 4) || !read_at(f, (long long)size - 4, tail, 4)) {
        set_error("KMC: short read of markers in " + path);
        return IBS_ERR_IO;
    }
    if (memcmp(head, marker, 4) || memcmp(tail, marker, 4)) {
        set_error("KMC: bad marker in " + path);
        return IBS_ERR_FORMAT;
    }
    return IBS_OK;
}

// maxK: 32 for the callers that take one-word codes, 64 for those that also
// take wide-key codes.
static ibs_status read_kmc_header(FILE *f, const std::string &path, KmcHeader &h, uint32_t maxK = 32)
{
    h.fileBytes = file_size(f);
    ibs_status s = check_markers(f, h.fileBytes, "KMCP", path);
    if (s != IBS_OK)
        return s;
    if (h.fileBytes < 20 || !read_at(f, (long long)h.fileBytes - 12, &h.version, 4)) {
        set_error("KMC: short read of version in " + path);
        return IBS_ERR_IO;
    }
    if (h.version != 0 && h.version != 0x200) {
        set_error("KMC: unsupported KMC format version in " + path);
        return IBS_ERR_FORMAT;
    }
    unsigned char off = 0; // only the first byte of header_offset is read, as KMC does
    if (!read_at(f, (long long)h.fileBytes - 8, &off, 1)) {
        set_error("KMC: short read of header offset in " + path);
        return IBS_ERR_IO;
    }
    h.headerOffset = off;
    const long long pos = (long long)h.fileBytes - (long long)(h.headerOffset + 8);
    if (pos < 4) {
        set_error("KMC: header offset out of range in " + path);
        return IBS_ERR_FORMAT;
    }
    if (h.version == 0x200) {
        uint32_t w[5];
        if (!read_at(f, pos, w, sizeof w) || !read_at(f, pos + 28, &h.total, 8)) {
            set_error("KMC: short read of header in " + path);
            return IBS_ERR_IO;
        }
        h.k = w[0], h.mode = w[1], h.counterSize = w[2], h.p = w[3], h.sigLen = w[4];
    } else {
        uint32_t w[4];
        if (!read_at(f, pos, w, sizeof w) || !read_at(f, pos + 24, &h.total, 8)) {
            set_error("KMC: short read of header in " + path);
            return IBS_ERR_IO;
        }
        h.k = w[0], h.mode = w[1], h.counterSize = w[2], h.p = w[3];
    }
    if (h.mode != 0) {
        set_error("KMC: Quake-compatible counters are not supported");
        return IBS_ERR_UNSUPPORTED;
    }
    if (h.k == 0 || h.k > maxK) {
        set_error("KMC: k=" + std::to_string(h.k) + " is not supported (k must be 1.." + std::to_string(maxK) +
                  (maxK < kMaxWideK ? " here; wide-key tables take k up to 64)" : ")"));
        return IBS_ERR_UNSUPPORTED;
    }
    if (h.p > h.k || (h.k - h.p) % 4 != 0 || h.k - h.p > maxK || h.p > 31) {
        set_error("KMC: unexpected suffix geometry");
        return IBS_ERR_FORMAT;
    }
    return IBS_OK;
}

// Reads the prefix LUT (bin-major for 0x200) with the guard set to
// total + 1 as KMC sets it (src/gpu/KmcRaIndex.hpp:564-591).
static ibs_status read_kmc_lut(FILE *f, const std::string &path, const KmcHeader &h,
                               std::vector<uint64_t> &lut)
{
    uint64_t entries;
    if (h.version == 0x200) {
        const uint64_t sigEntries = (1ull << (2 * h.sigLen)) + 1;
        const uint64_t fixed = sigEntries * 4 + h.headerOffset + 8 + 12;
        if (h.fileBytes < fixed) {
            set_error("KMC: .kmc_pre too small in " + path);
            return IBS_ERR_FORMAT;
        }
        const uint64_t lutArea = h.fileBytes - 12 - (sigEntries * 4 + h.headerOffset + 8);
        entries = (lutArea + 8) / 8;
    } else {
        entries = (1ull << (2 * h.p)) + 1;
    }
    const uint64_t single = 1ull << (2 * h.p);
    if (entries < 2 || (entries - 1) % single != 0) {
        set_error("KMC: LUT size is not a whole number of bins in " + path);
        return IBS_ERR_FORMAT;
    }
    lut.resize(entries);
    if (!read_at(f, 4, lut.data(), entries * 8)) {
        set_error("KMC: short read of prefix LUT in " + path);
        return IBS_ERR_IO;
    }
    lut[entries - 1] = h.total + 1;
    return IBS_OK;
}

} // namespace ibs

using namespace ibs;

// ---------------------------------------------------------------------------
// C-ABI
// ---------------------------------------------------------------------------
extern "C" const char *ibs_last_error(void) { return ibs::g_error.c_str(); }

extern "C" int ibs_device_count(void)
{
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

extern "C" uint64_t ibs_launch_count(void) { return launch_counter().load(); }


static ibs_status check_format(uint32_t k, const ibs_table_opts *o)
{
    if (o && o->force_format == FMT_WIDE && k <= 32) {
        set_error("wide-key tables (format 8) need 33 <= k <= 64");
        return IBS_ERR_UNSUPPORTED;
    }
    if (k > 32) {
        if (o && o->force_format && o->force_format != FMT_WIDE) {
            set_error("k=" + std::to_string(k) + " > 32 takes only the wide-key table layout (format 8)");
            return IBS_ERR_UNSUPPORTED;
        }
        return IBS_OK;
    }
    if (o && o->force_format == FMT_MZ8 && (k < 16 || k > 27)) {
        set_error("minimizer-bucketed tables (format 4) need 16 <= k <= 27");
        return IBS_ERR_UNSUPPORTED;
    }
    if (o && o->force_format == FMT_MZ6 && (k < 16 || k > 31)) {
        set_error("minimizer-bucketed tables with 40-bit slots (format 6) need 16 <= k <= 31");
        return IBS_ERR_UNSUPPORTED;
    }
    if (o && ((o->force_format > FMT_MZ6 && o->force_format != FMT_WIDE) || o->force_format == FMT_PANEL)) {
        set_error("unknown table format " + std::to_string(o->force_format));
        return IBS_ERR_ARG;
    }
    return IBS_OK;
}

extern "C" ibs_status ibs_table_from_codes(const uint64_t *codes, uint64_t n, uint32_t k,
                                           int codes_on_device, const ibs_table_opts *opts,
                                           ibs_table **out)
{
    clear_error();
    if (!out || (!codes && n) || k == 0 || k > 32) {
        set_error(k > 32 ? "ibs_table_from_codes: k > 32 codes take two words (ibs_table_from_codes128)"
                         : "ibs_table_from_codes: bad argument");
        return IBS_ERR_ARG;
    }
    *out = nullptr;
    const int dev = opts ? opts->device : 0;
    ibs_status s = check_format(k, opts);
    if (s != IBS_OK)
        return s;
    s = check_device_ordinal(dev);
    if (s != IBS_OK)
        return s;
    DeviceGuard guard(dev);
    const auto t0 = std::chrono::steady_clock::now();
    std::unique_ptr<ibs_table> t(new ibs_table);
    t->device = dev;
    uint64_t *dCodes = nullptr;
    const uint64_t *src = codes;
    if (!codes_on_device && n) {
        IBS_CUDA(cudaMalloc(&dCodes, n * 8), "codes alloc");
        cudaError_t e = cudaMemcpy(dCodes, codes, n * 8, cudaMemcpyHostToDevice);
        if (e != cudaSuccess) {
            cudaFree(dCodes);
            return cuda_fail(e, "codes upload");
        }
        src = dCodes;
    }
    s = build_from_device_codes(t.get(), src, n, k, opts);
    cudaFree(dCodes);
    if (s != IBS_OK) {
        ibs_close(t.release());
        return s;
    }
    t->buildSeconds =
        std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    *out = t.release();
    return IBS_OK;
}

ibs_status ibs::check_device_ordinal(int dev)
{
    const int n = ibs_device_count();
    if (n == 0) {
        set_error("no usable CUDA device (the scan has no CPU fallback)");
        return IBS_ERR_CUDA;
    }
    if (dev < 0 || dev >= n) {
        set_error("device " + std::to_string(dev) + " out of range");
        return IBS_ERR_ARG;
    }
    return IBS_OK;
}

namespace ibs {
// Decodes <prefix>.kmc_pre/.kmc_suf into canonical codes in device memory
// (cudaMalloc'd; the caller frees *dCodes): one word per code for k <= 32,
// {lo, hi} for 33 <= k <= maxK. The device must be current.
static ibs_status decode_kmc_impl(const char *prefix, int dev, uint64_t **dCodesOut, uint64_t *nOut,
                                  uint32_t *kOut, uint32_t maxK)
{
    *dCodesOut = nullptr;
    const std::string pre = std::string(prefix) + ".kmc_pre";
    const std::string suf = std::string(prefix) + ".kmc_suf";
    KmcHeader h;
    std::vector<uint64_t> lut;
    {
        File f(pre);
        if (!f.f) {
            set_error("KMC: cannot open " + pre);
            return IBS_ERR_IO;
        }
        ibs_status s = read_kmc_header(f.f, pre, h, maxK);
        if (s != IBS_OK)
            return s;
        s = read_kmc_lut(f.f, pre, h, lut);
        if (s != IBS_OK)
            return s;
    }
    File sf(suf);
    if (!sf.f) {
        set_error("KMC: cannot open " + suf);
        return IBS_ERR_IO;
    }
    const uint64_t sufSize = file_size(sf.f);
    {
        ibs_status s = check_markers(sf.f, sufSize, "KMCS", suf);
        if (s != IBS_OK)
            return s;
    }
    const uint32_t sufBytes = (h.k - h.p) / 4;
    const uint32_t recBytes = sufBytes + h.counterSize;
    if (recBytes == 0 || sufSize - 8 < h.total * (uint64_t)recBytes) {
        set_error("KMC: suffix file smaller than expected: " + suf);
        return IBS_ERR_FORMAT;
    }
    ibs_status s = check_device_ordinal(dev);
    if (s != IBS_OK)
        return s;
    // The records go up in chunks through a ring of kSlots pinned buffers:
    // kReaders host threads read chunks ahead (pread, in parallel), and this
    // thread uploads and decodes them in order; a buffer is read into again
    // once the upload of its previous chunk has finished.
    constexpr int kSlots = 8, kReaders = 4;
    uint64_t *dCodes = nullptr, *dLut = nullptr;
    uint8_t *dRaw[kSlots] = {};
    uint8_t *hRaw[kSlots] = {};
    cudaEvent_t done[kSlots] = {};
    cudaStream_t st = nullptr;
    const uint64_t total = h.total;
    const uint64_t chunkRecs = std::max<uint64_t>(1, (128ull << 20) / recBytes);
    const uint64_t chunkBytes = chunkRecs * recBytes;
    const uint64_t nChunks = (total + chunkRecs - 1) / chunkRecs;
    const int nSlots = (int)std::min<uint64_t>(kSlots, std::max<uint64_t>(nChunks, 1));
    // ring state: chunk filled[i] is in slot i ready for upload; consumed[i]
    // is the last chunk whose upload from slot i was enqueued
    std::mutex mu;
    std::condition_variable cv;
    std::vector<int64_t> filled(nSlots, -1), consumed(nSlots, -1);
    bool readFailed = false, stopReading = false;
    std::vector<std::thread> readers;
    auto cleanup = [&]() {
        {
            std::lock_guard<std::mutex> lock(mu);
            stopReading = true;
        }
        cv.notify_all();
        for (auto &t : readers)
            t.join();
        readers.clear();
        if (st)
            cudaStreamSynchronize(st);
        cudaFree(dCodes);
        cudaFree(dLut);
        for (int i = 0; i < nSlots; i++) {
            cudaFree(dRaw[i]);
            cudaFreeHost(hRaw[i]);
            if (done[i])
                cudaEventDestroy(done[i]);
        }
        if (st)
            cudaStreamDestroy(st);
    };
    const uint32_t codeWords = h.k > 32 ? 2 : 1;
    cudaError_t e = cudaMalloc(&dCodes, std::max<uint64_t>(total, 1) * 8 * codeWords);
    if (e == cudaSuccess)
        e = cudaMalloc(&dLut, lut.size() * 8);
    if (e == cudaSuccess)
        e = cudaMemcpy(dLut, lut.data(), lut.size() * 8, cudaMemcpyHostToDevice);
    for (int i = 0; i < nSlots && e == cudaSuccess; i++) {
        e = cudaMalloc(&dRaw[i], chunkBytes);
        if (e == cudaSuccess)
            e = cudaMallocHost(&hRaw[i], chunkBytes);
        if (e == cudaSuccess)
            e = cudaEventCreateWithFlags(&done[i], cudaEventDisableTiming);
    }
    if (e == cudaSuccess)
        e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
        cleanup();
        return cuda_fail(e, "KMC decode buffers");
    }
    const int fd = fileno(sf.f);
    int device = 0;
    cudaGetDevice(&device);
    auto reader = [&](int r) {
        cudaSetDevice(device);
        for (uint64_t c = r; c < nChunks; c += kReaders) {
            const int slot = (int)(c % nSlots);
            {
                // the slot's previous chunk (c - nSlots) must have been enqueued
                std::unique_lock<std::mutex> lock(mu);
                cv.wait(lock, [&] {
                    return stopReading || (c < (uint64_t)nSlots ? true : consumed[slot] == (int64_t)(c - nSlots));
                });
                if (stopReading)
                    return;
            }
            if (c >= (uint64_t)nSlots && cudaEventSynchronize(done[slot]) != cudaSuccess) {
                std::lock_guard<std::mutex> lock(mu);
                readFailed = true;
                cv.notify_all();
                return;
            }
            const uint64_t r0 = c * chunkRecs;
            const uint64_t bytes = std::min(chunkRecs, total - r0) * recBytes;
            uint64_t got = 0;
            while (got < bytes) {
                const ssize_t n = pread(fd, hRaw[slot] + got, bytes - got, (off_t)(4 + r0 * recBytes + got));
                if (n <= 0)
                    break;
                got += (uint64_t)n;
            }
            std::lock_guard<std::mutex> lock(mu);
            if (got != bytes)
                readFailed = true;
            else
                filled[slot] = (int64_t)c;
            cv.notify_all();
            if (got != bytes)
                return;
        }
    };
    for (int r = 0; r < kReaders && (uint64_t)r < nChunks; ++r)
        readers.emplace_back(reader, r);
    const uint64_t lutN = lut.size() - 1;
    const uint64_t prefixMask = (1ull << (2 * h.p)) - 1;
    for (uint64_t c = 0; c < nChunks && e == cudaSuccess; ++c) {
        const int slot = (int)(c % nSlots);
        {
            std::unique_lock<std::mutex> lock(mu);
            cv.wait(lock, [&] { return readFailed || filled[slot] == (int64_t)c; });
            if (readFailed) {
                lock.unlock();
                cleanup();
                set_error("KMC: short read of suffix records in " + suf);
                return IBS_ERR_IO;
            }
        }
        const uint64_t r0 = c * chunkRecs;
        const uint64_t nRec = std::min(chunkRecs, total - r0);
        e = cudaMemcpyAsync(dRaw[slot], hRaw[slot], nRec * recBytes, cudaMemcpyHostToDevice, st);
        if (e != cudaSuccess)
            break;
        if (codeWords == 2)
            k_decode_wide<<<grid_for(nRec, 256), 256, 0, st>>>(dRaw[slot], r0, nRec, recBytes, sufBytes, dLut, lutN,
                                                               prefixMask, 2 * (h.k - h.p),
                                                               reinterpret_cast<ulonglong2 *>(dCodes));
        else
            k_decode<<<grid_for(nRec, 256), 256, 0, st>>>(dRaw[slot], r0, nRec, recBytes, sufBytes, dLut, lutN,
                                                          prefixMask, 2 * (h.k - h.p), dCodes);
        IBS_LAUNCHED();
        e = cudaEventRecord(done[slot], st);
        {
            std::lock_guard<std::mutex> lock(mu);
            consumed[slot] = (int64_t)c;
        }
        cv.notify_all();
    }
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(st);
    if (e == cudaSuccess)
        e = cudaGetLastError();
    if (e != cudaSuccess) {
        cleanup();
        return cuda_fail(e, "KMC decode");
    }
    *dCodesOut = dCodes;
    dCodes = nullptr;
    *nOut = total;
    *kOut = h.k;
    cleanup();
    return IBS_OK;
}

ibs_status decode_kmc(const char *prefix, int dev, uint64_t **dCodes, uint64_t *n, uint32_t *k)
{
    return decode_kmc_impl(prefix, dev, dCodes, n, k, 32);
}

ibs_status decode_kmc_any(const char *prefix, int dev, uint64_t **dCodes, uint64_t *n, uint32_t *k)
{
    return decode_kmc_impl(prefix, dev, dCodes, n, k, kMaxWideK);
}
} // namespace ibs

extern "C" ibs_status ibs_open(const char *prefix, const ibs_table_opts *opts, ibs_table **out)
{
    clear_error();
    if (!prefix || !out) {
        set_error("ibs_open: bad argument");
        return IBS_ERR_ARG;
    }
    *out = nullptr;
    const auto t0 = std::chrono::steady_clock::now();
    const int dev = opts ? opts->device : 0;
    {
        // read the header first so a bad file is reported before any device check
        KmcHeader h;
        File f(std::string(prefix) + ".kmc_pre");
        if (!f.f) {
            set_error(std::string("KMC: cannot open ") + prefix + ".kmc_pre");
            return IBS_ERR_IO;
        }
        ibs_status s = read_kmc_header(f.f, std::string(prefix) + ".kmc_pre", h, kMaxWideK);
        if (s != IBS_OK)
            return s;
        s = check_format(h.k, opts);
        if (s != IBS_OK)
            return s;
    }
    ibs_status s = check_device_ordinal(dev);
    if (s != IBS_OK)
        return s;
    DeviceGuard guard(dev);
    uint64_t *dCodes = nullptr, total = 0;
    uint32_t k = 0;
    s = decode_kmc_any(prefix, dev, &dCodes, &total, &k);
    if (s != IBS_OK)
        return s;
    std::unique_ptr<ibs_table> t(new ibs_table);
    t->device = dev;
    if (k > 32)
        s = build_wide(t.get(), reinterpret_cast<const ulonglong2 *>(dCodes), total, k, opts);
    else
        s = build_from_device_codes(t.get(), dCodes, total, k, opts);
    cudaFree(dCodes);
    if (s != IBS_OK) {
        ibs_close(t.release());
        return s;
    }
    t->buildSeconds =
        std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    *out = t.release();
    return IBS_OK;
}

extern "C" ibs_status ibs_table_info_get(const ibs_table *t, ibs_table_info *info)
{
    clear_error();
    if (!t || !info) {
        set_error("ibs_table_info_get: bad argument");
        return IBS_ERR_ARG;
    }
    memset(info, 0, sizeof *info);
    info->k = t->geom.k;
    info->format = t->geom.format;
    info->fp_bits = t->geom.fpBits;
    info->n_keys = t->nKeys;
    info->n_buckets = t->geom.nBuckets;
    info->stash_keys = t->stashKeys;
    info->stash_buckets = t->geom.stashBuckets;
    info->device_bytes = t->deviceBytes;
    info->build_seconds = t->buildSeconds;
    return IBS_OK;
}

extern "C" ibs_status ibs_probe(ibs_table *t, const uint64_t *codes, uint64_t n, uint8_t *hits)
{
    clear_error();
    if (!t || (n && (!codes || !hits))) {
        set_error("ibs_probe: bad argument");
        return IBS_ERR_ARG;
    }
    if (t->geom.format == FMT_WIDE) {
        set_error("ibs_probe: a wide-key table (k > 32) takes ibs_probe128");
        return IBS_ERR_ARG;
    }
    if (!n)
        return IBS_OK;
    DeviceGuard guard(t->device);
    uint64_t *dCodes = nullptr;
    uint8_t *dHits = nullptr;
    cudaError_t e = cudaMalloc(&dCodes, n * 8);
    if (e == cudaSuccess)
        e = cudaMalloc(&dHits, n);
    if (e == cudaSuccess)
        e = cudaMemcpy(dCodes, codes, n * 8, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        if (t->geom.format == FMT_B8X32)
            k_probe<FMT_B8X32><<<grid_for(n, 256), 256>>>(t->view(), dCodes, n, dHits);
        else if (t->geom.format == FMT_MZ8)
            k_probe<FMT_MZ8><<<grid_for(n, 256), 256>>>(t->view(), dCodes, n, dHits);
        else if (t->geom.format == FMT_MZ6)
            k_probe<FMT_MZ6><<<grid_for(n, 256), 256>>>(t->view(), dCodes, n, dHits);
        else
            k_probe<FMT_B6X40><<<grid_for(n, 256), 256>>>(t->view(), dCodes, n, dHits);
        IBS_LAUNCHED();
        e = cudaGetLastError();
    }
    if (e == cudaSuccess)
        e = cudaMemcpy(hits, dHits, n, cudaMemcpyDeviceToHost);
    cudaFree(dCodes);
    cudaFree(dHits);
    if (e != cudaSuccess)
        return cuda_fail(e, "probe");
    return IBS_OK;
}

// Codes on the device -> how many the table holds.
static ibs_status count_present_device(ibs_table *t, const uint64_t *dCodes, uint64_t n, uint64_t *count)
{
    *count = 0;
    if (!n)
        return IBS_OK;
    std::lock_guard<std::mutex> lock(t->countMu);
    unsigned long long *dCount = reinterpret_cast<unsigned long long *>(t->buckets + 2 * t->geom.nBuckets);
    IBS_CUDA(cudaMemsetAsync(dCount, 0, sizeof *dCount, 0), "count init");
    const int grid = grid_for(n, 256);
    if (t->geom.format == FMT_B8X32)
        k_count_present<FMT_B8X32><<<grid, 256>>>(t->view(), dCodes, n, dCount);
    else if (t->geom.format == FMT_MZ8)
        k_count_present<FMT_MZ8><<<grid, 256>>>(t->view(), dCodes, n, dCount);
    else if (t->geom.format == FMT_MZ6)
        k_count_present<FMT_MZ6><<<grid, 256>>>(t->view(), dCodes, n, dCount);
    else
        k_count_present<FMT_B6X40><<<grid, 256>>>(t->view(), dCodes, n, dCount);
    IBS_LAUNCHED();
    IBS_CUDA(cudaGetLastError(), "count launch");
    unsigned long long c = 0;
    IBS_CUDA(cudaMemcpy(&c, dCount, sizeof c, cudaMemcpyDeviceToHost), "count read");
    *count = c;
    return IBS_OK;
}

extern "C" ibs_status ibs_count_present(ibs_table *t, const uint64_t *codes, uint64_t n, int codes_on_device,
                                        uint64_t *count)
{
    clear_error();
    if (!t || !count || (n && !codes)) {
        set_error("ibs_count_present: bad argument");
        return IBS_ERR_ARG;
    }
    if (t->geom.format == FMT_WIDE) {
        set_error("ibs_count_present: takes the 64-bit codes of k <= 32 tables (a wide-key table counts "
                  "through ibs_count_present_kmc)");
        return IBS_ERR_ARG;
    }
    DeviceGuard guard(t->device);
    if (codes_on_device || !n)
        return count_present_device(t, codes, n, count);
    uint64_t *d = nullptr;
    IBS_CUDA(cudaMalloc(&d, n * 8), "codes alloc");
    std::unique_ptr<uint64_t, cudaError_t (*)(void *)> guard2(d, cudaFree);
    IBS_CUDA(cudaMemcpy(d, codes, n * 8, cudaMemcpyHostToDevice), "codes upload");
    return count_present_device(t, d, n, count);
}

extern "C" ibs_status ibs_count_present_kmc(ibs_table *t, const char *kmc_prefix, uint64_t *count)
{
    clear_error();
    if (!t || !kmc_prefix || !count) {
        set_error("ibs_count_present_kmc: bad argument");
        return IBS_ERR_ARG;
    }
    DeviceGuard guard(t->device);
    uint64_t *d = nullptr, n = 0;
    uint32_t k = 0;
    ibs_status s = decode_kmc_any(kmc_prefix, t->device, &d, &n, &k);
    if (s != IBS_OK)
        return s;
    std::unique_ptr<uint64_t, cudaError_t (*)(void *)> guard2(d, cudaFree);
    if (k != t->geom.k) {
        set_error("K-mer lengths do not match");
        return IBS_ERR_ARG;
    }
    if (t->geom.format == FMT_WIDE)
        return count_present_wide(t, reinterpret_cast<const ulonglong2 *>(d), n, count);
    return count_present_device(t, d, n, count);
}

extern "C" uint64_t ibs_table_bytes_for(uint64_t n_keys, uint32_t k, const ibs_table_opts *opts)
{
    if (k == 0 || k > kMaxWideK)
        return 0;
    if (k > 32) {
        // level 0 at the load, plus about 1% for the later levels
        const double lam = (opts && opts->keys_per_bucket > 0) ? opts->keys_per_bucket : 4.0;
        const uint64_t lines = (uint64_t)((double)n_keys / lam) + 1;
        return (lines + lines / 100 + 1) * wide::kSlots * 16;
    }
    return choose_geometry(n_keys, k, opts).nBuckets * 32;
}

extern "C" ibs_status ibs_device_memory(int device, uint64_t *free_bytes, uint64_t *total_bytes)
{
    clear_error();
    ibs_status s = check_device_ordinal(device);
    if (s != IBS_OK)
        return s;
    DeviceGuard guard(device);
    size_t f = 0, t = 0;
    IBS_CUDA(cudaMemGetInfo(&f, &t), "cudaMemGetInfo");
    if (free_bytes)
        *free_bytes = f;
    if (total_bytes)
        *total_bytes = t;
    return IBS_OK;
}

extern "C" void ibs_close(ibs_table *t)
{
    if (!t)
        return;
    {
        DeviceGuard guard(t->device);
        cudaFree(t->buckets);
        cudaFree(t->stash);
        free_wide(t);
    }
    delete t;
}
