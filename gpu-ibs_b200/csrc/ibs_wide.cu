// Wide-key tables (33 <= k <= 64): the level-by-level build, membership
// probes and counts. Layout and lookup rule in wide_core.cuh.
//
// The reference has no device table for these k: its string path looks each
// canonical k-mer string up in the KMC database on the host
// (getStatsFromSequenceLegacy, src/KmerDatabase.hpp:675-708; CKmerAPI::
// from_string + CKMCFile::IsKmer). The build here is one pass a level: every
// key claims the next free slot of its home half line, then of the line's
// other half (a 128-bit compare-and-swap), and a key whose line is full goes
// to the next level's input (which 8 stay does not matter to membership).
#include "ibs_internal.cuh"

#include <algorithm>
#include <chrono>
#include <cstring>
#include <memory>
#include <vector>

namespace ibs {
namespace {

using wide::kEmpty;
using wide::kSlots;

__device__ __forceinline__ bool is_empty_key(const ulonglong2 &v) { return v.x == kEmpty && v.y == kEmpty; }

// Puts v in an empty slot; false when another key has it.
__device__ __forceinline__ bool claim_slot(ulonglong2 *slot, const ulonglong2 &v)
{
    unsigned long long lo, hi;
    asm volatile("{\n\t"
                 ".reg .b128 old, cmp, val;\n\t"
                 "mov.b128 cmp, {%4, %4};\n\t"
                 "mov.b128 val, {%2, %3};\n\t"
                 "atom.global.cas.b128 old, [%5], cmp, val;\n\t"
                 "mov.b128 {%0, %1}, old;\n\t"
                 "}"
                 : "=l"(lo), "=l"(hi)
                 : "l"(v.x), "l"(v.y), "l"(kEmpty), "l"(slot)
                 : "memory");
    return lo == kEmpty && hi == kEmpty;
}

__global__ void k_wplace(const ulonglong2 *__restrict__ keys, uint64_t n, uint32_t level, uint64_t lines,
                         ulonglong2 *__restrict__ slots, ulonglong2 *__restrict__ next,
                         unsigned long long *__restrict__ nextN, uint64_t nextCap)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const ulonglong2 v = keys[i];
        if (is_empty_key(v))
            continue;
        const uint64_t home = wide::home_of(v.x, v.y, level, lines);
        bool placed = false;
        for (uint32_t j = 0; j < kSlots && !placed; ++j) { // the home half's slots, then the other's
            ulonglong2 *slot = slots + (j < kSlots / 2 ? home + j : (home ^ (kSlots / 2)) + (j - kSlots / 2));
            const ulonglong2 old = __ldcg(slot);
            placed = is_empty_key(old) && claim_slot(slot, v);
        }
        if (!placed) {
            const unsigned long long j = atomicAdd(nextN, 1ull);
            if (j < nextCap)
                next[j] = v;
        }
    }
}

__global__ void k_wprobe(wide::View t, const ulonglong2 *__restrict__ keys, uint64_t n, uint8_t *__restrict__ hits)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const ulonglong2 v = keys[i];
        hits[i] = wide::lookup(t, v.x, v.y) ? 1 : 0;
    }
}

__global__ void k_wcount_present(wide::View t, const ulonglong2 *__restrict__ keys, uint64_t n,
                                 unsigned long long *__restrict__ count)
{
    unsigned long long local = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const ulonglong2 v = keys[i];
        local += wide::lookup(t, v.x, v.y) ? 1 : 0;
    }
    for (int o = 16; o; o >>= 1)
        local += __shfl_xor_sync(0xffffffffu, local, o);
    if ((threadIdx.x & 31) == 0 && local)
        atomicAdd(count, local);
}

int grid_of(uint64_t n, int threads)
{
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const uint64_t want = (n + threads - 1) / threads;
    return (int)std::max<uint64_t>(1, std::min<uint64_t>(want, (uint64_t)sms * 16));
}

template <typename T> struct DevPtr {
    T *p = nullptr;
    DevPtr() = default;
    DevPtr(const DevPtr &) = delete;
    DevPtr &operator=(const DevPtr &) = delete;
    ~DevPtr() { cudaFree(p); }
    cudaError_t alloc(uint64_t n) { return cudaMalloc(&p, std::max<uint64_t>(n, 1) * sizeof(T)); }
};

bool key_less(const ibs_code128 &a, const ibs_code128 &b) { return a.hi != b.hi ? a.hi < b.hi : a.lo < b.lo; }
bool key_eq(const ibs_code128 &a, const ibs_code128 &b) { return a.hi == b.hi && a.lo == b.lo; }

ibs_status check_wide_k(uint32_t k, const char *what)
{
    if (k <= 32 || k > kMaxWideK) {
        set_error(std::string(what) + ": wide-key tables need 33 <= k <= 64 (k=" + std::to_string(k) + ")");
        return k > kMaxWideK ? IBS_ERR_UNSUPPORTED : IBS_ERR_ARG;
    }
    return IBS_OK;
}

} // namespace

void free_wide(ibs_table *t)
{
    for (uint32_t L = 0; L < wide::kMaxLevels; ++L) {
        cudaFree(const_cast<ulonglong2 *>(t->wide.slots[L]));
        t->wide.slots[L] = nullptr;
    }
    t->wide.nLevels = 0;
}

ibs_status build_wide(ibs_table *t, const ulonglong2 *dCodes, uint64_t n, uint32_t k, const ibs_table_opts *o)
{
    ibs_status s = check_wide_k(k, "wide-key table");
    if (s != IBS_OK)
        return s;
    if (o && o->force_format && o->force_format != FMT_WIDE) {
        set_error("k=" + std::to_string(k) + " > 32 takes only the wide-key table layout (format 8)");
        return IBS_ERR_UNSUPPORTED;
    }
    const double lam = (o && o->keys_per_bucket > 0) ? o->keys_per_bucket : 4.0; // keys per 128-byte line
    t->geom = TableGeom{};
    t->geom.k = k;
    t->geom.bits = 2 * k;
    t->geom.format = FMT_WIDE;
    t->nKeys = n;
    t->wide = wide::View{};
    t->wide.k = k;
    const uint64_t lines0 = std::max<uint64_t>(1, (uint64_t)((double)n / lam) + 1);
    DevPtr<unsigned long long> dOver; // keys for the next level
    IBS_CUDA(dOver.alloc(1), "wide table scratch");
    // cur: this level's input (the caller's codes, then the surplus of the
    // previous level, held by owned)
    const ulonglong2 *cur = dCodes;
    uint64_t nCur = n;
    std::unique_ptr<DevPtr<ulonglong2>> owned;
    uint64_t bytes = 0, stashKeys = 0;
    for (uint32_t L = 0;; ++L) {
        if (L == wide::kMaxLevels) {
            set_error("wide-key table: keys left after " + std::to_string(wide::kMaxLevels) +
                      " levels (duplicate keys in the input?)");
            return IBS_ERR_CAPACITY;
        }
        const uint64_t lines = L == 0 ? lines0 : std::max<uint64_t>(1, (nCur + 1) / 2);
        ulonglong2 *slots = nullptr;
        IBS_CUDA(cudaMalloc(&slots, lines * kSlots * sizeof(ulonglong2)), "wide table alloc");
        t->wide.slots[L] = slots;
        t->wide.lines[L] = lines;
        t->wide.nLevels = L + 1;
        bytes += lines * kSlots * sizeof(ulonglong2);
        // about 1% of the keys find their line full at the default load; a level
        // that leaves more is filled again with room for as many (a line of c keys
        // leaves c - 8, whichever they are)
        std::unique_ptr<DevPtr<ulonglong2>> next(new DevPtr<ulonglong2>);
        unsigned long long over = 0;
        for (uint64_t cap = nCur / 16 + 4096;;) {
            IBS_CUDA(next->alloc(cap), "wide table level input");
            IBS_CUDA(cudaMemset(slots, 0xff, lines * kSlots * sizeof(ulonglong2)), "wide table init");
            IBS_CUDA(cudaMemset(dOver.p, 0, sizeof(unsigned long long)), "wide table counts");
            if (nCur) {
                k_wplace<<<grid_of(nCur, 256), 256>>>(cur, nCur, L, lines, slots, next->p, dOver.p, cap);
                IBS_LAUNCHED();
            }
            IBS_CUDA(cudaMemcpy(&over, dOver.p, sizeof over, cudaMemcpyDeviceToHost), "wide table place");
            if (over <= cap)
                break;
            cap = over;
            next.reset(new DevPtr<ulonglong2>);
        }
        if (L == 0)
            stashKeys = over; // every key past level 0 stays in a later level
        owned = std::move(next);
        cur = owned->p;
        nCur = over;
        if (!over)
            break;
    }
    t->geom.nBuckets = 0;
    for (uint32_t L = 0; L < t->wide.nLevels; ++L)
        t->geom.nBuckets += t->wide.lines[L] * 4; // in 32-byte units, as the other formats report
    t->stashKeys = stashKeys;                     // keys held by levels past the first
    t->deviceBytes = bytes;
    return IBS_OK;
}

ibs_status count_present_wide(ibs_table *t, const ulonglong2 *dCodes, uint64_t n, uint64_t *count)
{
    *count = 0;
    if (!n)
        return IBS_OK;
    DevPtr<unsigned long long> dCount;
    IBS_CUDA(dCount.alloc(1), "count alloc");
    IBS_CUDA(cudaMemset(dCount.p, 0, sizeof(unsigned long long)), "count init");
    k_wcount_present<<<grid_of(n, 256), 256>>>(t->wide, dCodes, n, dCount.p);
    IBS_LAUNCHED();
    IBS_CUDA(cudaGetLastError(), "count launch");
    unsigned long long c = 0;
    IBS_CUDA(cudaMemcpy(&c, dCount.p, sizeof c, cudaMemcpyDeviceToHost), "count read");
    *count = c;
    return IBS_OK;
}

} // namespace ibs

using namespace ibs;

extern "C" ibs_status ibs_table_from_codes128(const ibs_code128 *codes, uint64_t n, uint32_t k, int codes_on_device,
                                              const ibs_table_opts *opts, ibs_table **out)
{
    clear_error();
    if (!out || (!codes && n)) {
        set_error("ibs_table_from_codes128: bad argument");
        return IBS_ERR_ARG;
    }
    *out = nullptr;
    ibs_status s = check_wide_k(k, "ibs_table_from_codes128");
    if (s != IBS_OK)
        return s;
    const int dev = opts ? opts->device : 0;
    s = check_device_ordinal(dev);
    if (s != IBS_OK)
        return s;
    DeviceGuard guard(dev);
    const auto t0 = std::chrono::steady_clock::now();
    // duplicates removed on the host (a key repeated more than 8 times per
    // level would never leave the level chain)
    std::vector<ibs_code128> keys(n);
    if (n) {
        if (codes_on_device)
            IBS_CUDA(cudaMemcpy(keys.data(), codes, n * sizeof(ibs_code128), cudaMemcpyDeviceToHost), "codes download");
        else
            memcpy(keys.data(), codes, n * sizeof(ibs_code128));
    }
    std::sort(keys.begin(), keys.end(), key_less);
    keys.erase(std::unique(keys.begin(), keys.end(), key_eq), keys.end());
    const uint64_t m = keys.size();
    DevPtr<ulonglong2> d;
    IBS_CUDA(d.alloc(m), "codes alloc");
    if (m)
        IBS_CUDA(cudaMemcpy(d.p, keys.data(), m * sizeof(ibs_code128), cudaMemcpyHostToDevice), "codes upload");
    std::unique_ptr<ibs_table> t(new ibs_table);
    t->device = dev;
    s = build_wide(t.get(), d.p, m, k, opts);
    if (s != IBS_OK) {
        ibs_close(t.release());
        return s;
    }
    t->buildSeconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    *out = t.release();
    return IBS_OK;
}

extern "C" ibs_status ibs_probe128(ibs_table *t, const ibs_code128 *codes, uint64_t n, uint8_t *hits)
{
    clear_error();
    if (!t || (n && (!codes || !hits))) {
        set_error("ibs_probe128: bad argument");
        return IBS_ERR_ARG;
    }
    if (t->geom.format != FMT_WIDE) {
        set_error("ibs_probe128: the table is not a wide-key table (k <= 32 tables take ibs_probe)");
        return IBS_ERR_ARG;
    }
    if (!n)
        return IBS_OK;
    DeviceGuard guard(t->device);
    DevPtr<ulonglong2> dCodes;
    DevPtr<uint8_t> dHits;
    IBS_CUDA(dCodes.alloc(n), "probe alloc");
    IBS_CUDA(dHits.alloc(n), "probe alloc");
    IBS_CUDA(cudaMemcpy(dCodes.p, codes, n * sizeof(ibs_code128), cudaMemcpyHostToDevice), "probe upload");
    k_wprobe<<<grid_of(n, 256), 256>>>(t->wide, dCodes.p, n, dHits.p);
    IBS_LAUNCHED();
    IBS_CUDA(cudaGetLastError(), "probe launch");
    IBS_CUDA(cudaMemcpy(hits, dHits.p, n, cudaMemcpyDeviceToHost), "probe");
    return IBS_OK;
}
