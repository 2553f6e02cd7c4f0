// Stable LSD radix sort of (u64 key, u32 value) pairs and the reference's
// z-order sort products (emerald/sph_common/neighborhood.cpp:10-106).
//
// The step itself never needs a global z-sorted order: cells are found
// through the per-scene hash tables. The sorted (z, index) pairs, block
// indices and block ranges are produced here when a caller asks for them,
// by sorting the occupied cells by z and expanding each cell's (already
// index-ordered) member list.
#include "engine_types.cuh"
#include "kernels.cuh"
#include "sph_math.cuh"

#include <algorithm>
#include <cstddef>

namespace emerald {

namespace {

constexpr int kThreads = 256;
constexpr int kRounds = 8;
constexpr int kItems = kThreads * kRounds;  // keys per block and pass
constexpr int kDigits = 256;

__global__ void k_hist(uint64_t const* keys, uint32_t n, int shift, uint32_t* hist, uint32_t nblocks) {
    __shared__ uint32_t cnt[kDigits];
    cnt[threadIdx.x] = 0;
    __syncthreads();
    size_t const base = static_cast<size_t>(blockIdx.x) * kItems;
    for (int r = 0; r < kRounds; ++r) {
        size_t const e = base + static_cast<size_t>(r) * kThreads + threadIdx.x;
        if (e < n) atomicAdd(&cnt[(keys[e] >> shift) & 0xffu], 1u);
    }
    __syncthreads();
    hist[static_cast<size_t>(threadIdx.x) * nblocks + blockIdx.x] = cnt[threadIdx.x];
}

__global__ void k_rank_scatter(uint64_t const* kin, uint32_t const* vin, uint64_t* kout,
                               uint32_t* vout, uint32_t n, int shift, uint32_t const* offsets,
                               uint32_t nblocks) {
    __shared__ uint32_t base[kDigits];
    __shared__ uint32_t wcnt[kThreads / 32][kDigits];
    base[threadIdx.x] = offsets[static_cast<size_t>(threadIdx.x) * nblocks + blockIdx.x];
    int const lane = threadIdx.x & 31;
    int const warp = threadIdx.x >> 5;
    uint32_t const lt = (1u << lane) - 1u;
    size_t const blk = static_cast<size_t>(blockIdx.x) * kItems;
    for (int r = 0; r < kRounds; ++r) {
        for (int w = 0; w < kThreads / 32; ++w) wcnt[w][threadIdx.x] = 0;
        __syncthreads();
        size_t const e = blk + static_cast<size_t>(r) * kThreads + threadIdx.x;
        bool const live = e < n;
        uint64_t const key = live ? kin[e] : 0ull;
        uint32_t const dg = live ? static_cast<uint32_t>((key >> shift) & 0xffu) : 0xffffffffu;
        uint32_t const peers = __match_any_sync(0xffffffffu, dg);
        uint32_t const rank = __popc(peers & lt);
        if (live && rank == 0) wcnt[warp][dg] = __popc(peers);
        __syncthreads();
        uint32_t run = 0;
        for (int w = 0; w < kThreads / 32; ++w) {
            uint32_t const t = wcnt[w][threadIdx.x];
            wcnt[w][threadIdx.x] = base[threadIdx.x] + run;
            run += t;
        }
        base[threadIdx.x] += run;
        __syncthreads();
        if (live) {
            uint32_t const pos = wcnt[warp][dg] + rank;
            kout[pos] = key;
            vout[pos] = vin[e];
        }
        __syncthreads();
    }
}

// Words of the resident sort, zero at launch.
struct SortControl {
    unsigned long long any;      // OR of the keys
    unsigned long long any_not;  // OR of their complements
    uint32_t arrived;            // blocks at the grid barriers so far
    // a barrier ran out of polls: every block returns (last: a second sort of
    // the same scratch leaves it as it is)
    uint32_t stalled;
};

constexpr int kSortThreads = 1024;
constexpr int kSortWarps = kSortThreads / 32;
constexpr uint32_t kSortPolls = 1u << 22;

// False when a block did not come within `limit` polls (0: none does): the
// launch is cooperative, so all are resident and this only bounds the wait.
__device__ __forceinline__ bool sort_barrier(SortControl* c, uint32_t target, uint32_t limit) {
    __syncthreads();
    uint32_t bad = 0;
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&c->arrived, 1u);
        uint32_t polls = 0;
        while (!limit || *reinterpret_cast<uint32_t volatile*>(&c->arrived) < target) {
            bad = *reinterpret_cast<uint32_t volatile*>(&c->stalled);
            if (bad) break;
            if (++polls > limit) {
                atomicExch(&c->stalled, 1u);
                bad = 1;
                break;
            }
        }
        __threadfence();
    }
    return __syncthreads_or(static_cast<int>(bad)) == 0;
}

// All passes of the sort in one cooperative launch, block b on a contiguous
// run of the kItems-key tiles. What bounds these sizes is not the keys' traffic
// but the chain of launches (histogram, three of a scan, scatter: 30 us a pass
// at 100k keys), and most passes move nothing: a sweep first finds the bits in
// which the keys differ, and a digit that is the same in all of them is left
// out. Each block adds up the other blocks' histograms itself, so a pass has
// two barriers. The result is put in buffer `out`.
__global__ void __launch_bounds__(kSortThreads, 1)
  k_sort_resident(uint64_t* k0, uint64_t* k1, uint32_t* v0, uint32_t* v1, uint32_t n, int bits,
                  uint32_t tiles, uint32_t* hist, SortControl* ctl, uint32_t polls, int out) {
    __shared__ uint32_t wcnt[kSortWarps][kDigits];  // also the partial sums of the offsets
    __shared__ uint32_t base[kDigits];
    __shared__ uint32_t wsum[kDigits / 32];
    uint32_t const t = threadIdx.x, lane = t & 31u, warp = t >> 5, b = blockIdx.x, nb = gridDim.x;
    size_t const lo = static_cast<size_t>(static_cast<uint64_t>(tiles) * b / nb) * kItems;
    size_t const end = static_cast<size_t>(static_cast<uint64_t>(tiles) * (b + 1) / nb) * kItems;
    size_t const hi = end < n ? end : n;
    uint64_t any = 0, any_not = 0;
    for (size_t e = lo + t; e < hi; e += kSortThreads) {
        uint64_t const k = __ldcg(k0 + e);
        any |= k;
        any_not |= ~k;
    }
    for (int d = 16; d; d >>= 1) {
        any |= __shfl_xor_sync(0xffffffffu, any, d);
        any_not |= __shfl_xor_sync(0xffffffffu, any_not, d);
    }
    if (lane == 0) {
        if (any) atomicOr(&ctl->any, static_cast<unsigned long long>(any));
        if (any_not) atomicOr(&ctl->any_not, static_cast<unsigned long long>(any_not));
    }
    uint32_t target = nb;
    if (!sort_barrier(ctl, target, polls)) return;
    uint64_t const differ = __ldcg(&ctl->any) & __ldcg(&ctl->any_not);
    int cur = 0;
    for (int shift = 0; shift < bits; shift += 8) {
        if (((differ >> shift) & 0xffu) == 0) continue;
        uint64_t const* const kin = cur ? k1 : k0;
        uint32_t const* const vin = cur ? v1 : v0;
        uint64_t* const kout = cur ? k0 : k1;
        uint32_t* const vout = cur ? v0 : v1;
        if (t < kDigits) base[t] = 0;
        __syncthreads();
        for (size_t e = lo + t; e < hi; e += kSortThreads) {
            atomicAdd(&base[(__ldcg(kin + e) >> shift) & 0xffu], 1u);
        }
        __syncthreads();
        if (t < kDigits) __stcg(hist + static_cast<size_t>(b) * kDigits + t, base[t]);
        target += nb;
        if (!sort_barrier(ctl, target, polls)) return;
        // digit d over all blocks, and over the blocks before this one
        {
            uint32_t const d = t % kDigits, part = t / kDigits, parts = kSortThreads / kDigits;
            uint32_t total = 0, before = 0;
#pragma unroll 8
            for (uint32_t q = part; q < nb; q += parts) {
                uint32_t const c = __ldcg(hist + static_cast<size_t>(q) * kDigits + d);
                total += c;
                before += q < b ? c : 0u;
            }
            wcnt[2 * part][d] = total;
            wcnt[2 * part + 1][d] = before;
        }
        __syncthreads();
        uint32_t total = 0, before = 0, run = 0;
        if (t < kDigits) {
            for (int part = 0; part < kSortThreads / kDigits; ++part) {
                total += wcnt[2 * part][t];
                before += wcnt[2 * part + 1][t];
            }
            run = total;
            for (uint32_t d = 1; d < 32; d <<= 1) {
                uint32_t const o = __shfl_up_sync(0xffffffffu, run, d);
                if (lane >= d) run += o;
            }
            if (lane == 31) wsum[warp] = run;
        }
        __syncthreads();
        if (t < kDigits) {
            uint32_t first = run - total + before;
            for (uint32_t w = 0; w < warp; ++w) first += wsum[w];
            base[t] = first;
        }
        for (size_t e0 = lo; e0 < hi; e0 += kSortThreads) {
            __syncthreads();
            for (uint32_t q = t; q < kSortWarps * kDigits; q += kSortThreads) (&wcnt[0][0])[q] = 0;
            __syncthreads();
            size_t const e = e0 + t;
            bool const live = e < hi;
            uint64_t const key = live ? __ldcg(kin + e) : 0ull;
            uint32_t const val = live ? __ldcg(vin + e) : 0u;
            uint32_t const dg = live ? static_cast<uint32_t>((key >> shift) & 0xffu) : 0xffffffffu;
            uint32_t const peers = __match_any_sync(0xffffffffu, dg);
            uint32_t const rank = __popc(peers & ((1u << lane) - 1u));
            if (live && rank == 0) wcnt[warp][dg] = __popc(peers);
            __syncthreads();
            if (t < kDigits) {
                uint32_t at = base[t];
#pragma unroll 8
                for (int w = 0; w < kSortWarps; ++w) {
                    uint32_t const c = wcnt[w][t];
                    wcnt[w][t] = at;
                    at += c;
                }
                base[t] = at;
            }
            __syncthreads();
            if (live) {
                uint32_t const pos = wcnt[warp][dg] + rank;
                __stcg(kout + pos, key);
                __stcg(vout + pos, val);
            }
        }
        target += nb;
        if (!sort_barrier(ctl, target, polls)) return;
        cur ^= 1;
    }
    if (cur != out) {
        for (size_t e = lo + t; e < hi; e += kSortThreads) {
            __stcg((out ? k1 : k0) + e, __ldcg((cur ? k1 : k0) + e));
            __stcg((out ? v1 : v0) + e, __ldcg((cur ? v1 : v0) + e));
        }
    }
}

__global__ void k_occupied_flags(uint32_t const* count, uint32_t total, uint32_t* flags) {
    uint32_t const e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < total) flags[e] = count[e] ? 1u : 0u;
}

__global__ void k_compact_cells(uint64_t const* keys, uint32_t const* count, uint32_t const* flags,
                                uint32_t const* offsets, uint32_t total, uint32_t cap,
                                uint64_t* kout, uint32_t* vout, uint32_t* ncells) {
    uint32_t const e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= total) return;
    if (flags[e]) {
        uint32_t const o = offsets[e];
        kout[o] = (e == cap) ? kEmptyKey : keys[e];
        vout[o] = e;
    }
    if (e == total - 1) *ncells = offsets[e] + flags[e];
}

__global__ void k_fill_tail(uint64_t* keys, uint32_t* vals, uint32_t const* ncells, uint32_t limit) {
    uint32_t const k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= limit || k < *ncells) return;
    keys[k] = kEmptyKey;
    vals[k] = UINT32_MAX;
}

__global__ void k_cell_counts(uint32_t const* sorted_slots, uint32_t const* count,
                              uint32_t const* ncells, uint32_t limit, uint32_t* cell_count,
                              uint32_t const* gave_up) {
    uint32_t const c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= limit) return;
    cell_count[c] = c < *ncells && !sort_gave_up(gave_up) ? count[sorted_slots[c]] : 0u;
}

__global__ void k_expand_pairs(uint64_t const* sorted_z, uint32_t const* sorted_slots,
                               uint32_t const* cell_start, uint32_t const* count,
                               uint32_t const* start, uint32_t const* members,
                               uint32_t const* oid, uint32_t const* ncells, uint32_t limit,
                               uint32_t first, uint64_t* pair_z, uint32_t* pair_index,
                               uint32_t* block_indices, uint32_t* blocks,
                               uint32_t const* gave_up) {
    uint32_t const c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= limit || c >= *ncells || sort_gave_up(gave_up)) return;
    uint32_t const slot = sorted_slots[c];
    uint32_t const n = count[slot];
    uint32_t const b = cell_start[c];
    uint32_t const* m = members + start[slot];
    for (uint32_t k = 0; k < n; ++k) {
        pair_z[b + k] = sorted_z[c];
        pair_index[b + k] = oid ? oid[m[k]] : m[k] - first;
        block_indices[b + k] = c;
    }
    blocks[2 * c] = b;
    blocks[2 * c + 1] = b + n;
}

__device__ __forceinline__ uint32_t compact_bits(uint64_t x) {
    x &= 0x5555555555555555ull;
    x = (x | (x >> 1)) & 0x3333333333333333ull;
    x = (x | (x >> 2)) & 0x0F0F0F0F0F0F0F0Full;
    x = (x | (x >> 4)) & 0x00FF00FF00FF00FFull;
    x = (x | (x >> 8)) & 0x0000FFFF0000FFFFull;
    x = (x | (x >> 16)) & 0x00000000FFFFFFFFull;
    return static_cast<uint32_t>(x);
}

// Grid coords and z keys of the last build per original index, recovered
// from the stored keys.
__global__ void k_keys_of(uint64_t const* zkey, uint32_t const* slot_of, uint32_t begin,
                          uint32_t count, int2* gc, uint64_t* z) {
    uint32_t const k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    uint64_t const key = zkey[slot_of ? slot_of[begin + k] : begin + k];
    gc[k] = make_int2(static_cast<int32_t>(compact_bits(key)),
                      static_cast<int32_t>(compact_bits(key >> 1)));
    z[k] = key;
}

}  // namespace

// Lays out the scratch regions for n keys; with base == nullptr it only
// measures. Sizing and placement share this code so they cannot disagree.
static size_t carve(char* base, uint32_t n, SortScratch* s) {
    size_t const nb = (n + kItems - 1) / kItems + 1;
    size_t const words = static_cast<size_t>(n) + 1;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char* r = base ? base + off : nullptr;
        off += (bytes + 255) & ~size_t(255);
        return r;
    };
    char* k0 = take(words * 8);
    char* k1 = take(words * 8);
    char* v0 = take(words * 4);
    char* v1 = take(words * 4);
    char* fl = take(words * 4);
    char* of = take(words * 4);
    char* hi = take(kDigits * nb * 8);
    // the scan's words, then (from a multiple of eight) the sort's control words
    size_t const scan = scan_scratch_words(static_cast<uint32_t>(kDigits * nb + words));
    char* sc = take((scan + 16) * 4);
    static_assert(sizeof(SortControl) <= 4 * 8, "seven words to the next multiple, eight for it");
    if (s) {
        s->keys[0] = reinterpret_cast<uint64_t*>(k0);
        s->keys[1] = reinterpret_cast<uint64_t*>(k1);
        s->vals[0] = reinterpret_cast<uint32_t*>(v0);
        s->vals[1] = reinterpret_cast<uint32_t*>(v1);
        s->flags = reinterpret_cast<uint32_t*>(fl);
        s->offsets = reinterpret_cast<uint32_t*>(of);
        s->hist = reinterpret_cast<uint32_t*>(hi);
        s->scan = reinterpret_cast<uint32_t*>(sc);
        s->control = sc + (scan + 7) / 8 * 8 * 4;
        s->polls = kSortPolls;
        s->capacity = n;
    }
    return off;
}

size_t sort_scratch_bytes(uint32_t n) { return carve(nullptr, n, nullptr); }

void sort_scratch_carve(void* base, uint32_t n, SortScratch& s) {
    carve(static_cast<char*>(base), n, &s);
}

// Keys up to which the passes run in one launch. A pass of a few hundred tiles
// costs the chain of launches about 30 us whatever its size, the resident sort
// 17 us at 100k keys and 23 us at 300k, but 43 us to 35 us at 1M, where the
// chain has more warps in flight: keys of few digits, which all differ, change
// over at 2^19. Of 64-bit keys some digits are the same in all keys as a rule,
// and those passes are left out: a pair sort (index, then z) takes 450 -> 114
// us at 100k, 527 -> 261 us at 1M and 1232 -> 754 us at 4M pairs. At 2^22 it
// still breaks even when all of z's digits differ.
constexpr uint32_t kResidentKeysShort = 1u << 19;
constexpr uint32_t kResidentKeysLong = 1u << 22;

static bool launch_sort_resident(SortScratch& s, uint32_t n, int bits, int out, bool again,
                                 cudaStream_t st) {
    int dev = 0, coop = 0, sms = 0;
    if (n > (bits > 40 ? kResidentKeysLong : kResidentKeysShort) ||
        cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    uint32_t const tiles = (n + kItems - 1) / kItems;
    uint32_t const blocks = std::min<uint32_t>(tiles, static_cast<uint32_t>(sms));
    SortControl* const ctl = static_cast<SortControl*>(s.control);
    cudaMemsetAsync(ctl, 0, again ? offsetof(SortControl, stalled) : sizeof(SortControl), st);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kSortThreads);
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, k_sort_resident, s.keys[0], s.keys[1], s.vals[0], s.vals[1], n,
                           bits, tiles, s.hist, ctl, s.polls, out) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return true;
}

SortResult launch_radix_sort(SortScratch& s, uint32_t n, int bits, cudaStream_t st, bool again) {
    int cur = 0;
    if (n <= 1) return {cur, nullptr, 0};
    int const out = ((bits + 7) / 8) & 1;
    if (launch_sort_resident(s, n, bits, out, again, st)) {
        return {out, &static_cast<SortControl*>(s.control)->stalled, 1};
    }
    uint32_t const nb = (n + kItems - 1) / kItems;
    uint32_t* offsets = s.hist + static_cast<size_t>(kDigits) * nb;
    int kernels = 0;
    for (int shift = 0; shift < bits; shift += 8) {
        k_hist<<<nb, kThreads, 0, st>>>(s.keys[cur], n, shift, s.hist, nb);
        launch_exclusive_scan(s.hist, kDigits * nb, offsets, s.scan, st);
        k_rank_scatter<<<nb, kThreads, 0, st>>>(s.keys[cur], s.vals[cur], s.keys[cur ^ 1],
                                                s.vals[cur ^ 1], n, shift, offsets, nb);
        kernels += 5;  // three of them the scan
        cur ^= 1;
    }
    return {cur, nullptr, kernels};
}

uint32_t const* launch_sort_products(Arena const& a, bool solid, int scene, uint32_t begin, uint32_t count,
                          uint32_t tab_begin, uint32_t tab_size, float cell, SortScratch& s,
                          int2* grid_coords, uint64_t* z, uint64_t* pair_z, uint32_t* pair_index,
                          uint32_t* block_indices, uint32_t* blocks, uint32_t* nblocks,
                          cudaStream_t st) {
    (void)scene;
    uint32_t const* cnt = (solid ? a.scount : a.fcount) + tab_begin;
    uint32_t const* start = (solid ? a.sstart : a.fstart) + tab_begin;
    uint64_t const* keys = (solid ? a.skeys : a.fkeys) + tab_begin;
    uint32_t const* members = solid ? a.smembers : a.members;
    (void)cell;
    if (count) {
        k_keys_of<<<(count + 255) / 256, 256, 0, st>>>(solid ? a.szkey : a.zkey,
                                                      solid ? nullptr : a.slot_of, begin, count,
                                                      grid_coords, z);
    }
    uint32_t const total = tab_size;
    k_occupied_flags<<<(total + 255) / 256, 256, 0, st>>>(cnt, total, s.flags);
    launch_exclusive_scan(s.flags, total, s.offsets, s.scan, st);
    k_compact_cells<<<(total + 255) / 256, 256, 0, st>>>(keys, cnt, s.flags, s.offsets, total,
                                                        total - 1, s.keys[0], s.vals[0], nblocks);
    // Every occupied cell holds at least one particle, so count bounds the
    // number of cells; unused tail keys sort last.
    uint32_t const limit = count;
    // The tail [ncells, limit) gets the largest key; the stable sort keeps it
    // behind every real cell, including a real cell with that key.
    k_fill_tail<<<(limit + 255) / 256, 256, 0, st>>>(s.keys[0], s.vals[0], nblocks, limit);
    SortResult const sorted = launch_radix_sort(s, limit, 64, st);
    int const cur = sorted.cur;
    uint32_t* cell_count = s.flags;
    uint32_t* cell_start = s.offsets;
    k_cell_counts<<<(limit + 255) / 256, 256, 0, st>>>(s.vals[cur], cnt, nblocks, limit, cell_count,
                                                     sorted.gave_up);
    launch_exclusive_scan(cell_count, limit, cell_start, s.scan, st);
    k_expand_pairs<<<(limit + 255) / 256, 256, 0, st>>>(s.keys[cur], s.vals[cur], cell_start, cnt,
                                                       start, members, solid ? nullptr : a.oid,
                                                       nblocks, limit, begin, pair_z, pair_index,
                                                       block_indices, blocks, sorted.gave_up);
    return sorted.gave_up;
}

}  // namespace emerald
