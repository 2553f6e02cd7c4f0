// The solve of a sub-step (everything after the neighbour lists: densities,
// coefficients, warm starts, the pressure loops and the integration) as one
// cooperative launch of resident blocks.
//
// What bounds it: the loops run tens of iterations over the same lists, and
// the launch-per-phase kernels read every list from L2 or HBM in each phase
// (12 bytes an entry, two phases an iteration) behind three launches an
// iteration, each phase a chain of dependent L2 reads (count, index,
// neighbour's value, coefficients). Here a scene is split over a gang of
// blocks, one block per multiprocessor, each with a contiguous run of the
// scene's warp tiles (32 particles, one warp). A block holds for the whole
// solve, in shared memory, the lists of its particles (10 bytes an entry: a
// 16-bit code of the neighbour and the kernel gradient; boundary entries with
// their mass and velocity) and the values its folds gather, for its own
// particles and for the neighbours it has in other blocks (its halo). What a
// particle alone needs (counts, rho, alpha, ...) stays in the arena, where the
// L1 keeps it.
// A phase is then folds from shared memory and one exchange of the halo's
// values. An exchange has no barrier: a particle with neighbours in other
// blocks publishes its value together with the exchange's number (its tag) in
// one 8-byte word per 4 bytes of value, and the blocks that need it read the
// word until it carries that tag, so the value's own way through L2 is all the
// wait there is (a barrier adds a fence, an atomic and a poll before the first
// value can be read). Two exchanges of different arrays alternate, and lists
// are symmetric, so a value is read before it is overwritten: its owner writes
// the next one only after an exchange that the reader joined after reading.
// Lists that are not symmetric (cut at 64 entries) or have a neighbour without
// a code make the scene's blocks use barriers and plain arrays instead.
// The exit test needs no launch either: every block writes its error sums as a
// tagged record, and one warp of each block reads them all, behind the next
// phase's folds.
//
// Every sum runs the functions of solve_math.cuh in list order, so the
// results are the launch-per-phase kernels' bit for bit.
//
// Measured on B200, per pass of three frames of a DFSPH_P dam break in motion
// (12 sub-steps, 240 to 420 density iterations), launch-per-phase against
// resident: 36,503 particles 5.30 / 2.49 ms, 262,144 particles 12.2 / 8.4 ms.
// An exchange (half an iteration) takes 1.9 us at 2,000 to 37,000 particles
// (one tile a warp: 1,600 cycles of folds and division, 850 for the halo's
// values, the rest waiting for the slowest block), 7.3 us at 262,144 (two tiles
// a warp, 28 warps).
#pragma once

#include <algorithm>

#include "engine_types.cuh"
#include "kernels.cuh"
#include "solve_math.cuh"
#include "sph_math.cuh"

namespace emerald {

namespace {

constexpr uint32_t kRowBytes = 320;      // a list row: 32 16-bit codes, 32 gradients
constexpr uint32_t kCodeRowBytes = 64;   // without gradients (PCISPH)
constexpr uint32_t kBoundaryUnits = 2;   // rows of space per boundary row: 32 masses,
                                         // gradients and velocities (640 bytes)
constexpr uint32_t kMaxTiles = 256;      // warp tiles of a share at most
constexpr uint32_t kNoKey = 0xffffffffu;
// Polls of a wait before it gives up: about a second, where a sub-step's solve
// takes milliseconds. (A constant: as a parameter it costs spills in the loops.)
constexpr uint32_t kMaxPolls = 1u << 20;
constexpr uint32_t kFar = 0xffffu;       // a neighbour without a code

// A particle's published values and the codes of its list that do not fit in
// shared memory live in the upper half of its own column of the boundary lists
// (64 entries a particle; a particle has at most a dozen boundary neighbours).
// One with more than kBoundaryRows of them sends its scene to the barrier form
// and its list to the arena.
constexpr uint32_t kBoundaryRows = 32;
constexpr uint32_t kWords = 6;  // published 64-bit words a particle has at most

// Published word w of particle i: 32 bits of value and the tag above them.
__device__ __forceinline__ unsigned long long* published(Arena const& a, uint32_t w, uint32_t i) {
    return reinterpret_cast<unsigned long long*>(a.ns_gw) +
           static_cast<size_t>(uint32_t(kMaxNeighbors) - 1u - w) * a.stride + i;
}
// The code of entry k of particle i's list.
__device__ __forceinline__ uint16_t* arena_code(Arena const& a, int k, uint32_t i) {
    return reinterpret_cast<uint16_t*>(
             a.ns_idx + static_cast<size_t>(kBoundaryRows + (uint32_t(k) >> 1)) * a.stride + i) +
           (k & 1);
}

struct Shared {
    GangPart part;
    SceneParams P;
    float dt;
    int new_frame;
    uint32_t ticket;
    uint32_t used;    // rows handed out
    uint32_t wanted;  // rows the share's lists have
    uint32_t halo_n;
    uint32_t target;  // arrivals the gang's next barrier waits for
    int ok;           // no wait has given up
    int plain;        // this block cannot use tagged exchanges
    int tagged;       // the gang uses tagged exchanges
    int ends;         // the loop ends after this iteration
    unsigned long long w_sum[32];
    double w_exact[32];
    uint32_t w_max[32];
    // per tile: first staged row, staged rows << 16, flags << 24 (kTail: there
    // are more rows in the arena; kFarList: some neighbour has no code and the
    // list stays there); first staged row and rows of its boundary lists
    uint32_t list[kMaxTiles];
    uint32_t blist[kMaxTiles];
};

extern __shared__ __align__(16) unsigned char mem[];

// Offsets into the dynamic shared memory, the same for every block of a
// launch: the gathered values (`locals` slots), the halo's arena slots, then
// the staged rows. While the lists are staged, the values' place holds the
// hash table that finds the halo.
struct Layout {
    uint32_t locals;      // value slots: own particles, then the halo
    uint32_t halo_max;
    uint32_t hash_log2;
    uint32_t halo_at, rows_at;
    uint32_t row_bytes, capacity;
};

// A thread's view of its block's share.
struct Share {
    uint32_t first;   // first arena slot of the share
    uint32_t tiles;   // its warp tiles
    uint32_t end;     // end of the scene's slots
    uint32_t epoch;   // tag of the last exchange
    uint32_t exports; // bit r: the particle of the warp's tile r has neighbours in other blocks
    bool tagged;
    __device__ __forceinline__ uint32_t own() const { return tiles * 32u; }  // its slots
};

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }

// ------------------------------------------------------------- list views

// A particle's fluid list: entries [0, rows) staged, the rest read from the
// arena (codes by arena_code), neighbours' values by code from shared
// memory. A code is 4 times the neighbour's local slot. `rows` is the same for
// the whole warp and rows past a lane's count hold its own code and a zero
// gradient, so nothing needs a guard but the additions. A far list is read from
// the arena, values included (and has no staged rows).
constexpr uint32_t kTail = 1u, kFarList = 2u;  // flags of a tile's list
template <uint32_t ROW>
struct StagedList {
    static constexpr int kUnroll = 4;
    Arena const& a;
    uint32_t i;
    unsigned char const* row0;  // this lane's code in the tile's first row
    int rows;
    uint32_t flags;

    __device__ __forceinline__ uint32_t tail_code(int k) const {
        return *arena_code(a, k, i);
    }
    static __device__ __forceinline__ uint32_t staged_code(unsigned char const* row) {
        return *reinterpret_cast<uint16_t const*>(row);
    }
    // a lane's gradient lies this far behind its code
    static __device__ __forceinline__ uint32_t gradient_at() { return 64u + lane_id() * 6u; }
    static __device__ __forceinline__ float2 staged_gradient(unsigned char const* row) {
        return *reinterpret_cast<float2 const*>(row);
    }
    __device__ __forceinline__ float2 gradient(int k) const {
        return k < rows ? staged_gradient(row0 + gradient_at() + uint32_t(k) * ROW)
                        : ArenaList{a, i}.gradient(k);
    }
    // N staged rows; left: entries of this lane from here on
    template <int N, class Source, class Fold>
    static __device__ __forceinline__ void fold_rows(unsigned char const*& row,
                                                     unsigned char const*& grad, int& left,
                                                     Source const& src, Fold& f) {
        using T = decltype(src.local(0u));
        uint32_t code[N];
        T val[N];
        float2 gw[N];
#pragma unroll
        for (int u = 0; u < N; ++u) {
            code[u] = staged_code(row + u * ROW);
            gw[u] = staged_gradient(grad + u * ROW);
        }
#pragma unroll
        for (int u = 0; u < N; ++u) val[u] = src.local(code[u]);
#pragma unroll
        for (int u = 0; u < N; ++u) f(val[u], gw[u], u < left);
        row += N * ROW;
        grad += N * ROW;
        left -= N;
    }
    template <int CH, class Source, class Fold>
    __device__ __forceinline__ void fold(int c, Source const& src, Fold f) const {
        unsigned char const* row = row0;
        unsigned char const* grad = row0 + gradient_at();
        int left = c;
        int n = rows;
#pragma unroll 1
        for (; n >= CH; n -= CH) fold_rows<CH>(row, grad, left, src, f);
        static_assert(CH == 2 || CH == 4 || CH == 8, "the remainder's steps below");
        if (CH > 4 && (n & 4)) fold_rows<4>(row, grad, left, src, f);
        if (CH > 2 && (n & 2)) fold_rows<2>(row, grad, left, src, f);
        if (n & 1) fold_rows<1>(row, grad, left, src, f);
        if (!flags) return;
        ArenaList const arena{a, i};
        if (flags & kFarList) {
            arena.template fold<1>(c, src, f);
            return;
        }
        // (asking for these before the staged rows would hide their way, but
        // the registers it takes spill: slower at every size)
#pragma unroll 1
        for (int k = rows; k < c; k += 2) {
            bool const two = k + 1 < c;
            uint32_t const c0 = tail_code(k);
            float2 const g0 = arena.gradient(k);
            uint32_t const c1 = two ? tail_code(k + 1) : c0;
            float2 const g1 = two ? arena.gradient(k + 1) : g0;
            f(src.local(c0), g0, true);
            f(src.local(c1), g1, two);
        }
    }
    template <int N, class Source, class Fold>
    static __device__ __forceinline__ void fold_row_values(unsigned char const*& row, int& left,
                                                           Source const& src, Fold& f) {
        using T = decltype(src.local(0u));
        T val[N];
#pragma unroll
        for (int u = 0; u < N; ++u) val[u] = src.local(staged_code(row + u * ROW));
#pragma unroll
        for (int u = 0; u < N; ++u) f(val[u], u < left);
        row += N * ROW;
        left -= N;
    }
    template <int CH, class Source, class Fold>
    __device__ __forceinline__ void fold_values(int c, Source const& src, Fold f) const {
        unsigned char const* row = row0;
        int left = c;
        int n = rows;
#pragma unroll 1
        for (; n >= CH; n -= CH) fold_row_values<CH>(row, left, src, f);
#pragma unroll 1
        for (; n > 0; --n) fold_row_values<1>(row, left, src, f);
        if (!flags) return;
        if (flags & kFarList) {
            ArenaList{a, i}.template fold_values<1>(c, src, f);
            return;
        }
#pragma unroll 1
        for (int k = rows; k < c; ++k) f(src.local(tail_code(k)), true);
    }
};

// A particle's boundary list: entries [0, rows) staged, the rest in the arena.
struct StagedBoundary {
    static constexpr int kUnroll = 1;
    ArenaBoundary arena;
    uint32_t at;  // of this lane's mass in the tile's first boundary row
    int rows;
    __device__ __forceinline__ uint32_t entry(int k) const {
        return at + uint32_t(k) * (kBoundaryUnits * kRowBytes);
    }
    __device__ __forceinline__ float mass(int k) const {
        return k < rows ? *reinterpret_cast<float const*>(mem + entry(k)) : arena.mass(k);
    }
    __device__ __forceinline__ float2 gradient(int k) const {
        return k < rows ? *reinterpret_cast<float2 const*>(mem + entry(k) + 128u + lane_id() * 4u)
                        : arena.gradient(k);
    }
    __device__ __forceinline__ float2 velocity(int k) const {
        return k < rows ? *reinterpret_cast<float2 const*>(mem + entry(k) + 384u + lane_id() * 4u)
                        : arena.velocity(k);
    }
};

template <uint32_t ROW>
__device__ __forceinline__ StagedList<ROW> staged_rows(Arena const& a, Layout const& l,
                                                       Shared const& s, uint32_t t, uint32_t i) {
    uint32_t const m = s.list[t];
    return StagedList<ROW>{a, i, mem + l.rows_at + (m & 0xffffu) * ROW + lane_id() * 2u,
                           int(m >> 16 & 0xffu), m >> 24};
}
__device__ __forceinline__ StagedList<kRowBytes> staged_list(Arena const& a, Layout const& l,
                                                             Shared const& s, uint32_t t,
                                                             uint32_t i) {
    return staged_rows<kRowBytes>(a, l, s, t, i);
}
__device__ __forceinline__ StagedBoundary staged_boundary(Arena const& a, Layout const& l,
                                                          Shared const& s, uint32_t t, uint32_t i) {
    uint32_t const m = s.blist[t];
    return StagedBoundary{ArenaBoundary{a, i, s.P.rho0},
                          l.rows_at + (m & 0xffffu) * kRowBytes + lane_id() * 4u, int(m >> 16)};
}

// The value a code (4 times a local slot) stands for in the shared array at
// offset `off`.
template <class T>
__device__ __forceinline__ T value_of(uint32_t off, uint32_t code) {
    return *reinterpret_cast<T const*>(mem + off + code * uint32_t(sizeof(T) / 4));
}

// Values of neighbours: by code from the shared array at offset `off`, by
// arena slot from `p`.
template <class T>
struct Values {
    uint32_t off;
    T const* p;
    __device__ __forceinline__ T local(uint32_t code) const { return value_of<T>(off, code); }
    __device__ __forceinline__ T at(uint32_t j) const { return p[j]; }
};
template <class T>
__device__ __forceinline__ T* values_at(uint32_t off) {
    return reinterpret_cast<T*>(mem + off);
}

// -------------------------------------------------------------- the share

// The block's last warp has no tiles: it keeps the exit test. It runs code of
// its own between the block's barriers (the other warps need the registers).
__device__ __forceinline__ uint32_t worker_warps() { return (blockDim.x >> 5) - 1u; }
__device__ __forceinline__ uint32_t workers() { return blockDim.x - 32u; }
__device__ __forceinline__ bool keeps_exit() { return threadIdx.x >= workers(); }

// The block's barrier, which its warps reach from different places.
__device__ __forceinline__ void block_sync() {
    __syncwarp();
    asm volatile("bar.sync 0;" ::: "memory");
}

// Runs f(r, t, li, i, live) for the warp's tiles t = warp + r * warps: li the
// particle's local slot, i its arena slot. R: the warp has at most R tiles
// (0: any number).
template <int R = 0, class F>
__device__ __forceinline__ void for_tiles(Share const& sh, F f) {
    if (keeps_exit()) return;
    uint32_t const warps = worker_warps();
    auto tile = [&](uint32_t r, uint32_t t) {
        uint32_t const li = t * 32u + lane_id();
        uint32_t const i = sh.first + li;
        f(r, t, li, i, i < sh.end);
    };
    if constexpr (R > 0) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            uint32_t const t = (threadIdx.x >> 5) + uint32_t(r) * warps;
            if (t < sh.tiles) tile(uint32_t(r), t);
        }
    } else {
        uint32_t r = 0u;
#pragma unroll 1
        for (uint32_t t = threadIdx.x >> 5; t < sh.tiles; t += warps, ++r) tile(r, t);
    }
}

// What the loops read of a particle in every phase: with R > 0 kept in
// registers (an L2 read each, once, instead of at the start of every phase).
template <int N>
struct Kept {
    float f[N];
    int c, cs;
};
template <int R, int N>
struct KeptTiles {
    Kept<N> k[R > 0 ? R : 1];
    // read(i) loads a particle's
    template <class Read>
    __device__ __forceinline__ void load(Share const& sh, Read read) {
        if constexpr (R > 0) {
            for_tiles<R>(sh, [&](uint32_t r, uint32_t, uint32_t, uint32_t i, bool live) {
                if (live) k[r] = read(i);
            });
        }
    }
    template <class Read>
    __device__ __forceinline__ Kept<N> get(uint32_t r, uint32_t i, Read read) const {
        if constexpr (R > 0) {
            return k[r];
        } else {
            return read(i);
        }
    }
};

// Takes n rows of shared memory; returns how many there are and the first.
__device__ __forceinline__ uint32_t take_rows(Layout const& l, Shared& s, uint32_t n,
                                              uint32_t& at) {
    at = 0u;
    if (n && lane_id() == 0) at = atomicAdd(&s.used, n);
    at = __shfl_sync(0xffffffffu, at, 0);
    uint32_t const left = at < l.capacity ? l.capacity - at : 0u;
    if (!left) at = 0u;
    return min(n, left);
}

__device__ __forceinline__ uint32_t* hash_keys() { return reinterpret_cast<uint32_t*>(mem); }
__device__ __forceinline__ uint16_t* hash_codes(Layout const& l) {
    return reinterpret_cast<uint16_t*>(mem + (4u << l.hash_log2));
}

// The hash slot of halo neighbour j (kFar: the table is full).
__device__ __forceinline__ uint32_t halo_slot(Layout const& l, uint32_t j) {
    uint32_t const mask = (1u << l.hash_log2) - 1u;
    uint32_t h = (j * 0x9E3779B1u) >> (32u - l.hash_log2);
    uint32_t* const keys = hash_keys();
#pragma unroll 1
    for (int probe = 0; probe < 64; ++probe) {
        uint32_t const k = keys[h];
        if (k == j) return h;
        if (k == kNoKey) {
            uint32_t const prev = atomicCAS(&keys[h], kNoKey, j);
            if (prev == kNoKey || prev == j) return h;
        }
        h = (h + 1u) & mask;
    }
    return kFar;
}

// Copies the lists of the share into shared memory and finds its halo. Each
// lane copies, and later reads, its own column. Entries of neighbours in the
// share get their local slot as code; the others go through a hash table that
// is then numbered. Where the rows do not fit, the last rows of every tile
// keep their gradients in the arena and their codes go there too (arena_code). A tile
// with a neighbour that finds no code (the table or the halo is full) keeps
// its fluid list in the arena.
template <bool GRADIENTS>
__device__ __forceinline__ void stage_lists(Arena const& a, Layout const& l, Share& sh,
                                            Shared& s) {
    constexpr uint32_t ROW = GRADIENTS ? kRowBytes : kCodeRowBytes;
    uint32_t const lane = lane_id();
#pragma unroll 1
    for (uint32_t h = threadIdx.x; h < (1u << l.hash_log2); h += blockDim.x) {
        hash_keys()[h] = kNoKey;
    }
    for_tiles(sh, [&](uint32_t, uint32_t, uint32_t, uint32_t i, bool live) {
        uint32_t const rows = __reduce_max_sync(0xffffffffu, live ? uint32_t(a.nf_cnt[i]) : 0u);
        uint32_t const brows = __reduce_max_sync(0xffffffffu, live ? uint32_t(a.ns_cnt[i]) : 0u);
        if (lane == 0) {
            atomicAdd(&s.wanted, rows + (GRADIENTS ? kBoundaryUnits * brows : 0u));
            if (rows >= uint32_t(kMaxNeighbors) || brows > kBoundaryRows) s.plain = 1;
        }
    });
    block_sync();
    uint32_t const wanted = s.wanted;
    sh.exports = 0u;
    for_tiles(sh, [&](uint32_t r, uint32_t t, uint32_t li, uint32_t i, bool live) {
        int const c = live ? int(a.nf_cnt[i]) : 0;
        int const cs = live ? int(a.ns_cnt[i]) : 0;
        uint32_t const want = __reduce_max_sync(0xffffffffu, uint32_t(c));
        uint32_t const bmost = __reduce_max_sync(0xffffffffu, uint32_t(cs));
        uint32_t const bwant = GRADIENTS ? bmost : 0u;
        uint32_t at;
        // boundary rows whole (few tiles have any), fluid rows in proportion
        uint32_t const brows = take_rows(l, s, kBoundaryUnits * bwant, at) / kBoundaryUnits;
        if (lane == 0) s.blist[t] = at | brows << 16;
        ArenaBoundary const bnd{a, i, s.P.rho0};
#pragma unroll 1
        for (int k = 0; k < int(brows); ++k) {
            if (k < cs) {
                unsigned char* const row =
                  mem + l.rows_at + (at + uint32_t(k) * kBoundaryUnits) * ROW;
                reinterpret_cast<float*>(row)[lane] = bnd.mass(k);
                reinterpret_cast<float2*>(row + 128)[lane] = bnd.gradient(k);
                reinterpret_cast<float2*>(row + 384)[lane] = bnd.velocity(k);
            }
        }
        uint32_t const fit = wanted <= l.capacity
                               ? want
                               : uint32_t(uint64_t(want) * l.capacity / wanted);
        int const rows = int(take_rows(l, s, fit, at));
        if (uint32_t(rows) < want && bmost > kBoundaryRows) {
            // no room for the other rows' codes either
            if (lane == 0) s.list[t] = kFarList << 24;
            return;
        }
        ArenaList const list{a, i};
        unsigned char* const row0 = mem + l.rows_at + at * ROW;
        bool far = false, out = false;
#pragma unroll 4
        for (int k = 0; k < int(want); ++k) {
            uint32_t code = li * 4u;
            float2 g = mk2(0.0f, 0.0f);
            if (k < c) {
                uint32_t const j = list.index(k);
                if (GRADIENTS && k < rows) g = list.gradient(k);
                code = (j - sh.first) * 4u;
                if (j - sh.first >= sh.own()) {
                    // an odd code: the halo's numbers come below
                    uint32_t const h = halo_slot(l, j);
                    far = far || h == kFar;
                    out = true;
                    code = h * 4u | 1u;
                }
            }
            if (k < rows) {
                reinterpret_cast<uint16_t*>(row0 + k * ROW)[lane] = uint16_t(code);
                if (GRADIENTS) reinterpret_cast<float2*>(row0 + k * ROW + 64)[lane] = g;
            } else if (k < c) {
                *arena_code(a, k, i) = uint16_t(code);
            }
        }
        if (out) {
            sh.exports |= 1u << r;
            // no word of an earlier launch can carry one of this one's tags
            if (bmost <= kBoundaryRows) {
#pragma unroll
                for (uint32_t w = 0; w < kWords; ++w) *published(a, w, i) = 0ull;
            }
        }
        far = __any_sync(0xffffffffu, far);
        if (lane == 0) {
            uint32_t const flags = far ? kFarList : uint32_t(rows) < want ? kTail : 0u;
            s.list[t] = at | (far ? 0u : uint32_t(rows)) << 16 | flags << 24;
            if (far) s.plain = 1;
        }
    });
    block_sync();
    // number the halo
#pragma unroll 1
    for (uint32_t h = threadIdx.x; h < (1u << l.hash_log2); h += blockDim.x) {
        uint32_t const j = hash_keys()[h];
        if (j == kNoKey) continue;
        uint32_t const n = atomicAdd(&s.halo_n, 1u);
        bool const fits = n < l.halo_max;
        if (fits) reinterpret_cast<uint32_t*>(mem + l.halo_at)[n] = j;
        hash_codes(l)[h] = uint16_t(fits ? (sh.own() + n) * 4u : kFar);
    }
    block_sync();
    for_tiles(sh, [&](uint32_t, uint32_t t, uint32_t, uint32_t i, bool live) {
        uint32_t const m = s.list[t];
        if (m >> 24 & kFarList) return;
        int const rows = int(m >> 16 & 0xffu);
        int const c = live ? int(a.nf_cnt[i]) : 0;
        unsigned char* const row0 = mem + l.rows_at + (m & 0xffffu) * ROW;
        bool far = false;
        auto number = [&](uint16_t* p) {
            if (*p & 1u) {
                uint32_t const code = hash_codes(l)[*p >> 2];
                far = far || code == kFar;
                *p = uint16_t(code);
            }
        };
#pragma unroll 2
        for (int k = 0; k < rows; ++k) number(reinterpret_cast<uint16_t*>(row0 + k * ROW) + lane);
#pragma unroll 2
        for (int k = rows; k < c; ++k) number(arena_code(a, k, i));
        if (__any_sync(0xffffffffu, far) && lane == 0) {
            s.list[t] = kFarList << 24;
            s.plain = 1;
        }
    });
    block_sync();
    if (threadIdx.x == 0) {
        s.halo_n = min(s.halo_n, l.halo_max);
        // how far the storage order has drifted, for the choice of path
        uint32_t const drift = static_cast<uint32_t>(
          16.0f * static_cast<float>(s.halo_n) / sqrtf(static_cast<float>(max(sh.own(), 1u))));
        atomicMax(&a.control->drift, s.plain ? kPlainForm : min(drift, kPlainForm - 1u));
    }
}

// ---------------------------------------------------------------- barriers

// Waits until every block of the gang has arrived, making their writes before
// it visible after it. Returns false when the others did not arrive within the
// poll limit: the caller leaves.
__device__ __forceinline__ bool gang_sync(Arena const& a, Shared& s) {
    block_sync();
    if (threadIdx.x == 0 && s.part.size > 1) {
        uint32_t* const arrive = &a.gangs[s.part.scene].arrive;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(arrive) : "memory");
        uint32_t const target = s.target + s.part.size;
        s.target = target;
        uint32_t polls = 0;
        uint32_t seen;
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(arrive) : "memory");
            if (seen >= target) break;
            if (++polls > kMaxPolls) {
                s.ok = 0;
                break;
            }
        }
    }
    block_sync();
    return s.ok != 0;
}

// Record `slot` (0 or 1) of the gang's block `rank`.
__device__ __forceinline__ GangRecord* record_of(Arena const& a, Shared const& s, uint32_t rank,
                                                 uint32_t slot) {
    return a.records + 2u * (s.part.base + rank) + slot;
}

// The gang's first barrier, after the lists are staged: agrees on tagged
// exchanges or barriers.
__device__ __forceinline__ bool agree(Arena const& a, Share& sh, Shared& s) {
    GangState& g = a.gangs[s.part.scene];
    if (threadIdx.x == 0 && s.plain) atomicOr(&g.plain, 1u);
    if (threadIdx.x < 12) {
        // the block's two records carry no tag yet
        record_of(a, s, s.part.rank, threadIdx.x / 6)->w[threadIdx.x % 6] = 0ull;
    }
    bool const ok = gang_sync(a, s);
    // (injected: one block on its own in the other form, whose values never come)
    bool const astray = a.inject == 2u && s.part.rank == 0u;
    if (threadIdx.x == 0) s.tagged = __ldcg(&g.plain) || astray ? 0 : 1;
    block_sync();
    sh.tagged = s.tagged != 0;
    return ok;
}

// --------------------------------------------------------------- exchanges

__device__ __forceinline__ unsigned long long tag_word(float v, uint32_t tag) {
    return (static_cast<unsigned long long>(tag) << 32) | __float_as_uint(v);
}
__device__ __forceinline__ float word_value(unsigned long long w) {
    return __uint_as_float(static_cast<uint32_t>(w));
}
__device__ __forceinline__ uint32_t word_tag(unsigned long long w) {
    return static_cast<uint32_t>(w >> 32);
}
__device__ __forceinline__ void put(unsigned long long* p, float v, uint32_t tag) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(tag_word(v, tag)) : "memory");
}
__device__ __forceinline__ unsigned long long get(unsigned long long const* p) {
    unsigned long long w;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
    return w;
}

// An array of per-particle values that blocks exchange: plain for the barrier
// form, published words from `word` on for the other.
template <class T>
struct Field {
    T* plain;
    uint32_t word;
};
__device__ __forceinline__ void put_value(Arena const& a, Field<float> const& f, uint32_t i,
                                          float v, uint32_t tag) {
    put(published(a, f.word, i), v, tag);
}
__device__ __forceinline__ void put_value(Arena const& a, Field<float2> const& f, uint32_t i,
                                          float2 v, uint32_t tag) {
    put(published(a, f.word, i), v.x, tag);
    put(published(a, f.word + 1u, i), v.y, tag);
}
__device__ __forceinline__ bool get_value(Arena const& a, Field<float> const& f, uint32_t i,
                                          uint32_t tag, float& v) {
    unsigned long long const w = get(published(a, f.word, i));
    v = word_value(w);
    return word_tag(w) == tag;
}
__device__ __forceinline__ bool get_value(Arena const& a, Field<float2> const& f, uint32_t i,
                                          uint32_t tag, float2& v) {
    unsigned long long const w0 = get(published(a, f.word, i));
    unsigned long long const w1 = get(published(a, f.word + 1u, i));
    v = mk2(word_value(w0), word_value(w1));
    return word_tag(w0) == tag && word_tag(w1) == tag;
}

// Publishes the value of the particle of the warp's tile r for the next
// exchange.
template <class T>
__device__ __forceinline__ void publish(Arena const& a, Share const& sh, Field<T> const& f,
                                        uint32_t r, uint32_t i, T v) {
    if (!sh.tagged) {
        f.plain[i] = v;
    } else if (sh.exports >> r & 1u) {
        put_value(a, f, i, v, sh.epoch + 1u);
    }
}

// Calls store(local slot, value) with the halo's published values (by the
// workers; a share has about as many as it has workers). One that has not
// arrived is read again.
template <class T, class Store>
__device__ __forceinline__ void receive(Arena const& a, Layout const& l, Share const& sh,
                                        Shared& s, Field<T> const& f, Store store) {
    uint32_t const* const halo = reinterpret_cast<uint32_t const*>(mem + l.halo_at);
    uint32_t const n = s.halo_n;
    uint32_t const own = sh.own();
    if (!sh.tagged) {
#pragma unroll 1
        for (uint32_t h = threadIdx.x; h < n; h += workers()) {
            store(own + h, __ldcg(f.plain + halo[h]));
        }
        return;
    }
#pragma unroll 1
    for (uint32_t h = threadIdx.x; h < n; h += workers()) {
        T v;
        uint32_t polls = 0;
        while (!get_value(a, f, halo[h], sh.epoch, v)) {
            if (++polls > kMaxPolls) {
                s.ok = 0;
                return;
            }
        }
        store(own + h, v);
    }
}

// One exchange: everything published since the last one becomes readable.
// fill() receives the halo's values where the next folds read them (beside the
// block's own, stored when they were computed). Returns false when a wait gave
// up.
template <class Fill>
__device__ __forceinline__ bool exchange(Arena const& a, Share& sh, Shared& s, Fill fill) {
    if (!sh.tagged && !gang_sync(a, s)) return false;
    ++sh.epoch;
    fill();
    block_sync();
    return s.ok != 0;
}

// The exit test's warp in an exchange of the others.
__device__ __forceinline__ bool attend_exchange(Share& sh, Shared const& s) {
    if (!sh.tagged) {
        block_sync();
        block_sync();
        if (!s.ok) return false;
    }
    ++sh.epoch;
    block_sync();
    return s.ok != 0;
}

// --------------------------------------------------------------- exit test

// A thread's error contributions of one phase.
struct PhaseErr {
    unsigned long long sum;
    uint32_t max;
    __device__ __forceinline__ void add(unsigned long long v, float m) {
        sum += v;
        if (m == m && m > 0.0f) {
            uint32_t const b = __float_as_uint(m);
            max = b > max ? b : max;
        }
    }
};

__device__ __forceinline__ void reduce_warp(PhaseErr& e) {
    // the integer sums are small unless the flow has blown up
    if (__any_sync(0xffffffffu, (e.sum >> 26) != 0ull)) {
        for (int o = 16; o; o >>= 1) e.sum += __shfl_xor_sync(0xffffffffu, e.sum, o);
    } else {
        e.sum = __reduce_add_sync(0xffffffffu, static_cast<uint32_t>(e.sum));
    }
    e.max = __reduce_max_sync(0xffffffffu, e.max);
}

// Leaves the warp's error sums for post_errors, which runs after the next
// block barrier.
__device__ __forceinline__ void stash_errors(Shared& s, PhaseErr e) {
    reduce_warp(e);
    if (lane_id() == 0) {
        uint32_t const warp = threadIdx.x >> 5;
        s.w_sum[warp] = e.sum;
        s.w_max[warp] = e.max;
    }
}

__device__ __forceinline__ void put_record(unsigned long long* p, uint32_t lo, uint32_t hi,
                                           uint32_t tag) {
    unsigned long long const t = static_cast<unsigned long long>(tag) << 32;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(t | lo), "l"(t | hi)
                 : "memory");
}

// The block's error sums as a tagged record (by the exit test's warp). Two
// records take turns: a block writes an iteration's after it has read all of
// the previous iteration's, whose writers had read the one before that.
__device__ __forceinline__ void post_errors(Arena const& a, Shared const& s, uint32_t slot,
                                            uint32_t tag) {
    PhaseErr t{0ull, 0u};
    uint32_t const lane = lane_id();
    if (lane < worker_warps()) t = PhaseErr{s.w_sum[lane], s.w_max[lane]};
    reduce_warp(t);
    if (lane == 0) {
        // a sum of 2^32 - 1 and more is marked so, and in words 2 and 3
        bool const large = t.sum >= 0xffffffffull;
        unsigned long long* const p = record_of(a, s, s.part.rank, slot)->w;
        put_record(p, large ? 0xffffffffu : static_cast<uint32_t>(t.sum), t.max, tag);
        if (large) {
            put_record(p + 2, static_cast<uint32_t>(t.sum), static_cast<uint32_t>(t.sum >> 32),
                       tag);
        }
    }
}

// The two words from word k of a record, waited for until they carry the tag.
__device__ __forceinline__ void record_words(GangRecord const* r, int k, uint32_t tag, Shared& s,
                                             uint32_t& lo, uint32_t& hi) {
    unsigned long long w0, w1;
    uint32_t polls = 0;
    for (;;) {
        asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                     : "=l"(w0), "=l"(w1)
                     : "l"(r->w + k)
                     : "memory");
        if (word_tag(w0) == tag && word_tag(w1) == tag) break;
        if (++polls > kMaxPolls) {
            s.ok = 0;
            break;
        }
    }
    lo = static_cast<uint32_t>(w0);
    hi = static_cast<uint32_t>(w1);
}

// Reads the gang's records of the iteration and applies the exit test; all of
// a lane's records in flight together. The scene's statistics are written by
// the gang's first block.
__device__ __forceinline__ void decide_exit(Arena const& a, Shared& s, int kind, int iter,
                                            uint32_t slot, uint32_t tag) {
    PhaseErr t{0ull, 0u};
    uint32_t const lane = lane_id();
    uint32_t const size = s.part.size;
#pragma unroll 1
    for (uint32_t k0 = 0u; k0 < size; k0 += 160u) {
        unsigned long long w0[5], w1[5];
        bool ready;
        uint32_t polls = 0;
        do {
            ready = true;
#pragma unroll
            for (int u = 0; u < 5; ++u) {
                uint32_t const k = k0 + u * 32u + lane;
                if (k < size) {
                    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                                 : "=l"(w0[u]), "=l"(w1[u])
                                 : "l"(record_of(a, s, k, slot)->w)
                                 : "memory");
                }
            }
#pragma unroll
            for (int u = 0; u < 5; ++u) {
                ready = ready && (k0 + u * 32u + lane >= size ||
                                  (word_tag(w0[u]) == tag && word_tag(w1[u]) == tag));
            }
            if (++polls > kMaxPolls) {
                s.ok = 0;
                break;
            }
        } while (!ready);
#pragma unroll
        for (int u = 0; u < 5; ++u) {
            uint32_t const k = k0 + u * 32u + lane;
            if (k >= size) break;
            uint32_t lo = static_cast<uint32_t>(w0[u]), hi = static_cast<uint32_t>(w1[u]);
            t.max = hi > t.max ? hi : t.max;
            unsigned long long sum = lo;
            if (lo == 0xffffffffu) {
                record_words(record_of(a, s, k, slot), 2, tag, s, lo, hi);
                sum = (static_cast<unsigned long long>(hi) << 32) | lo;
            }
            t.sum += sum;
        }
    }
    reduce_warp(t);
    bool const ends = loop_ends(s.P, kind, iter, t.sum, t.max);
    if (lane == 0) s.ends = ends ? 1 : 0;
    // (only the last iteration's statistics can be seen)
    if (ends && lane == 0 && s.part.rank == 0) {
        report_loop(s.P, a.ss[s.part.scene], kind, iter, t.sum, t.max, true);
    }
    __syncwarp();
}

// The mean of the errors of a finished loop's last iteration, in double and
// with nothing dropped (the exit test's metric drops what is below 0.1%):
// every block adds up its threads' sums and posts the total, and the gang's
// first block adds those up in order and reports the mean where the loop's
// statistics are.
__device__ __forceinline__ void sum_exact(Shared& s, double sum) {
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane_id() == 0) s.w_exact[threadIdx.x >> 5] = sum;
    block_sync();
}
__device__ __forceinline__ void report_exact(Arena const& a, Share& sh, Shared& s, int kind,
                                             int iters, uint32_t slot) {
    block_sync();
    uint32_t const lane = lane_id();
    double t = lane < worker_warps() ? s.w_exact[lane] : 0.0;
    for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) {
        unsigned long long const w = static_cast<unsigned long long>(__double_as_longlong(t));
        put_record(record_of(a, s, s.part.rank, slot)->w + 4, static_cast<uint32_t>(w),
                   static_cast<uint32_t>(w >> 32), sh.epoch);
    }
    if (s.part.rank != 0) return;
    t = 0.0;
#pragma unroll 1
    for (uint32_t k = lane; k < s.part.size && s.ok; k += 32u) {
        uint32_t lo, hi;
        record_words(record_of(a, s, k, slot), 4, sh.epoch, s, lo, hi);
        t += __longlong_as_double(
          static_cast<long long>((static_cast<unsigned long long>(hi) << 32) | lo));
    }
    for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) {
        report_exact_mean(s.P, a.ss[s.part.scene], kind, iters - 1, t);
    }
}

// Before a pressure loop whose coefficients read neighbours' velocities from
// the arena: the loop's first exchange comes after those reads in every block,
// and the velocities are overwritten after the loop. A loop that runs no
// iteration has no exchange, so the gang waits here instead.
__device__ __forceinline__ bool start_loop(Arena const& a, Shared& s) {
    if (iteration_cap(s.P, 0) <= 0) return gang_sync(a, s);
    block_sync();
    return true;
}

// One solver loop of the reference: body(iter) runs an iteration, during which
// the exit test's warp sets s.ends, and ends in a block barrier. Returns the
// iterations run, or -1 when a wait gave up.
template <class Body>
__device__ __forceinline__ int solver_loop(Shared const& s, int kind, Body body) {
    if (iteration_cap(s.P, kind) <= 0) return 0;
#pragma unroll 1
    for (int iter = 0;; ++iter) {
        if (!body(iter)) return -1;
        if (s.ends) return iter + 1;
    }
}

// The exit test's warp during a solver loop of two exchanges an iteration: the
// error sums are stashed before the first (and the second ends the iteration),
// or before the second (and a block barrier ends it). Two records take turns
// (slot).
__device__ __forceinline__ int attend_loop(Arena const& a, Share& sh, Shared& s, int kind,
                                           bool errors_first, uint32_t& slot) {
    return solver_loop(s, kind, [&](int iter) {
        if (!errors_first && !attend_exchange(sh, s)) return false;
        if (!attend_exchange(sh, s)) return false;
        post_errors(a, s, slot, sh.epoch);
        decide_exit(a, s, kind, iter, slot, sh.epoch);
        slot ^= 1u;
        if (errors_first) return attend_exchange(sh, s);
        block_sync();
        return s.ok != 0;
    });
}

// Loop bookkeeping the launch-per-phase path leaves in the scene's state.
__device__ __forceinline__ void finish_loop(Arena const& a, Shared const& s, int iters) {
    if (s.part.rank == 0 && threadIdx.x == 0) {
        SceneState& S = a.ss[s.part.scene];
        S.iter = iters;
        S.done = 1;
    }
}

// ----------------------------------------------------------------- solvers

// dfsph_p.cpp:265-374 after the neighbour lists. The shared values are the
// velocities (from offset 0), gathered by the divergence sums, and p / rho^2
// (behind them), gathered by the pressure sums.
template <bool K, int R, int CH>
__device__ __forceinline__ bool solve_dfsph(Arena const& a, Layout const& l, Share& sh, Shared& s) {
    SceneParams const& P = s.P;
    float const dt = s.dt;
    uint32_t const at_q = l.locals * 8u;
    float2* const V = values_at<float2>(0u);
    float* const Q = values_at<float>(at_q);
    Field<float2> const vels{a.v, 0u};
    Field<float> const qs{a.qdens, 2u};
    stage_lists<true>(a, l, sh, s);
    if (!agree(a, sh, s)) return false;
    for_tiles(sh, [&](uint32_t, uint32_t t, uint32_t li, uint32_t i, bool live) {
        if (!live) return;
        float rho, alpha;
        dfsph_density_alpha<K>(a, P, i, a.nf_cnt[i], a.ns_cnt[i], staged_list(a, l, s, t, i), rho,
                               alpha);
        a.rho[i] = rho;
        a.alpha[i] = alpha;
        if (s.new_frame) {
            a.kdiv[i] = 0.0f;
            a.kdens[i] = 0.0f;
        }
        V[li] = a.v[i];
    });
    if (keeps_exit()) {
        uint32_t slot = 0u;
#pragma unroll 1
        for (int kind = 2; kind >= 1; --kind) {
            if (!attend_exchange(sh, s) || !attend_exchange(sh, s)) return false;
            int const n = attend_loop(a, sh, s, kind, true, slot);
            if (n < 0) return false;
            if (n > 0) report_exact(a, sh, s, kind, n, slot);
        }
        return true;
    }
    auto exchange_q = [&] {
        return exchange(a, sh, s, [&] {
            receive(a, l, sh, s, qs, [&](uint32_t li, float x) { Q[li] = x; });
        });
    };
    auto exchange_v = [&] {
        return exchange(a, sh, s, [&] {
            receive(a, l, sh, s, vels, [&](uint32_t li, float2 x) { V[li] = x; });
        });
    };
    auto read = [&](uint32_t i) {
        return Kept<2>{{a.rho[i], a.alpha[i]}, a.nf_cnt[i], a.ns_cnt[i]};
    };
    KeptTiles<R, 2> kept;
    kept.load(sh, read);
    auto apply = [&](bool external) {
        for_tiles<R>(sh, [&](uint32_t r, uint32_t t, uint32_t li, uint32_t i, bool live) {
            if (!live) return;
            auto const k = kept.get(r, i, read);
            float2 v = V[li];
            if (external) v = integrate_external(a, P, i, v, dt);
            v = apply_pressure_of<K, CH>(P, k.c, k.cs, v, Q[li], Values<float>{at_q, a.qdens}, dt,
                                         staged_list(a, l, s, t, i), staged_boundary(a, l, s, t, i));
            V[li] = v;
            publish(a, sh, vels, r, i, v);
        });
    };
    int iters = 0;
    // the divergence solve (kind 2), then the density solve (kind 1), each
    // after its warm start
#pragma unroll 1
    for (int kind = 2; kind >= 1; --kind) {
        float* const kappas = kind == 2 ? a.kdiv : a.kdens;
        for_tiles(sh, [&](uint32_t r, uint32_t, uint32_t li, uint32_t i, bool live) {
            if (!live) return;
            float const q = p_over_rho2(kappas[i], a.rho[i]);
            Q[li] = q;
            publish(a, sh, qs, r, i, q);
        });
        if (!exchange_q()) return false;
        apply(kind == 1);
        if (!exchange_v()) return false;
        iters = solver_loop(s, kind, [&](int) {
            PhaseErr e{0ull, 0u};
            for_tiles<R>(sh, [&](uint32_t r, uint32_t t, uint32_t li, uint32_t i, bool live) {
                if (!live) return;
                auto const k = kept.get(r, i, read);
                float const div = divergence_of<K, CH>(
                  P, k.c, k.cs, V[li], Values<float2>{0u, a.v}, staged_list(a, l, s, t, i),
                  staged_boundary(a, l, s, t, i));
                DfsphStep const d = kind == 2 ? dfsph_divergence_step(P, dt, k.f[0], k.f[1], div)
                                              : dfsph_density_step(P, dt, k.f[0], k.f[1], div);
                Q[li] = d.q;
                publish(a, sh, qs, r, i, d.q);
                kappas[i] = d.kappa;
                a.rho_star[i] = d.star;
                e.add(static_cast<unsigned long long>(static_cast<long long>(d.err * 1000.0f)),
                      d.err);
            });
            stash_errors(s, e);
            if (!exchange_q()) return false;
            apply(false);
            return exchange_v();
        });
        if (iters < 0) return false;
        if (iters > 0) {
            double exact = 0.0;
            for_tiles(sh, [&](uint32_t, uint32_t, uint32_t, uint32_t i, bool live) {
                if (!live) return;
                float const star = a.rho_star[i];
                float const err = kind == 2 ? dfsph_divergence_error(P, dt, star)
                                            : dfsph_density_error(P, star);
                if (err == err && err > 0.0f) exact += static_cast<double>(err);
            });
            sum_exact(s, exact);
        }
    }
    finish_loop(a, s, iters);
    for_tiles(sh, [&](uint32_t, uint32_t, uint32_t li, uint32_t i, bool live) {
        if (!live) return;
        float2 const v = V[li];
        a.v[i] = v;
        advance_position(a, P, i, dt, v);
    });
    return true;
}

// Sources of the IISPH sums. The shared values are rho, the current and the
// next pressures, the sums of d_ij p_j (the velocities until the first
// iteration) and d_ii.
struct IisphValues {
    uint32_t rho, p[2], sdp, dii;
};
struct IisphRhoV {
    Arena const& a;
    IisphValues o;
    __device__ __forceinline__ RhoV local(uint32_t k) const {
        return RhoV{value_of<float>(o.rho, k), value_of<float2>(o.sdp, k)};
    }
    __device__ __forceinline__ RhoV at(uint32_t j) const { return RhoV{a.rho[j], a.v[j]}; }
};
struct IisphPRho {
    Arena const& a;
    float const* p;
    uint32_t at_p, at_rho;
    __device__ __forceinline__ float2 local(uint32_t k) const {
        return mk2(value_of<float>(at_p, k), value_of<float>(at_rho, k));
    }
    __device__ __forceinline__ float2 at(uint32_t j) const { return mk2(p[j], a.rho[j]); }
};
struct IisphAll {
    Arena const& a;
    float const* p;
    uint32_t at_p, at_rho, sdp, dii;
    __device__ __forceinline__ IisphNeighbor local(uint32_t k) const {
        return IisphNeighbor{value_of<float>(at_rho, k), value_of<float>(at_p, k),
                             value_of<float2>(sdp, k), value_of<float2>(dii, k)};
    }
    __device__ __forceinline__ IisphNeighbor at(uint32_t j) const {
        return IisphNeighbor{a.rho[j], p[j], a.sdp[j], a.dii[j]};
    }
};
struct IisphQ {
    Arena const& a;
    float const* p;
    uint32_t off;
    __device__ __forceinline__ float local(uint32_t k) const { return value_of<float>(off, k); }
    __device__ __forceinline__ float at(uint32_t j) const { return p_over_rho2(p[j], a.rho[j]); }
};

// iisph.cpp:23-151 after the neighbour lists.
template <bool K, int R, int CH>
__device__ __forceinline__ bool solve_iisph(Arena const& a, Layout const& l, Share& sh, Shared& s) {
    SceneParams const& P = s.P;
    float const dt = s.dt;
    IisphValues const o{0u, {l.locals * 4u, l.locals * 8u}, l.locals * 12u, l.locals * 20u};
    float* const RHO = values_at<float>(o.rho);
    float2* const S = values_at<float2>(o.sdp);
    float2* const D = values_at<float2>(o.dii);
    stage_lists<true>(a, l, sh, s);
    for_tiles(sh, [&](uint32_t, uint32_t t, uint32_t, uint32_t i, bool live) {
        if (!live) return;
        float const rho = density_of<K>(a, P, i);
        a.rho[i] = rho;
        a.v[i] = integrate_external(a, P, i, a.v[i], dt);
        a.dii[i] = iisph_dii<K>(P, dt, rho, a.nf_cnt[i], a.ns_cnt[i], staged_list(a, l, s, t, i),
                                staged_boundary(a, l, s, t, i));
        a.pbuf0[i] = 0.0f;
    });
    if (!agree(a, sh, s)) return false;
    {
        uint32_t const* const halo = reinterpret_cast<uint32_t const*>(mem + l.halo_at);
#pragma unroll 1
        for (uint32_t h = threadIdx.x; h < s.halo_n; h += blockDim.x) {
            uint32_t const j = halo[h], li = sh.own() + h;
            RHO[li] = __ldcg(a.rho + j);
            values_at<float>(o.p[0])[li] = 0.0f;
            S[li] = __ldcg(a.v + j);
            D[li] = __ldcg(a.dii + j);
        }
    }
    for_tiles(sh, [&](uint32_t, uint32_t, uint32_t li, uint32_t i, bool live) {
        if (!live) return;
        RHO[li] = a.rho[i];
        values_at<float>(o.p[0])[li] = 0.0f;
        S[li] = a.v[i];
        D[li] = a.dii[i];
    });
    block_sync();
    for_tiles(sh, [&](uint32_t, uint32_t t, uint32_t li, uint32_t i, bool live) {
        if (!live) return;
        float aii, star;
        iisph_aii<K, 2>(P, dt, RHO[li], S[li], D[li], a.nf_cnt[i], a.ns_cnt[i], IisphRhoV{a, o},
                        staged_list(a, l, s, t, i), staged_boundary(a, l, s, t, i), aii, star);
        a.aii[i] = aii;
        a.rho_star[i] = star;
    });
    if (!start_loop(a, s)) return false;
    if (keeps_exit()) {
        uint32_t slot = 0u;
        if (attend_loop(a, sh, s, 0, false, slot) < 0) return false;
        block_sync();
        block_sync();
        return true;
    }
    auto read = [&](uint32_t i) {
        return Kept<2>{{a.aii[i], a.rho_star[i]}, a.nf_cnt[i], a.ns_cnt[i]};
    };
    KeptTiles<R, 2> kept;
    kept.load(sh, read);
    // sums of d_ij p_j of the pressures of iteration `iter`
    auto sum_dij = [&](int iter) {
        float const* const pc = (iter & 1) ? a.pbuf1 : a.pbuf0;
        for_tiles<R>(sh, [&](uint32_t r, uint32_t t, uint32_t li, uint32_t i, bool live) {
            if (!live) return;
            S[li] = iisph_sum_dij<K, CH>(P, dt, kept.get(r, i, read).c,
                                         IisphPRho{a, pc, o.p[iter & 1], o.rho},
                                         staged_list(a, l, s, t, i));
        });
    };
    Field<float2> const sums{a.sdp, 0u};
    sum_dij(0);
    int const iters = solver_loop(s, 0, [&](int iter) {
        float const* pc = (iter & 1) ? a.pbuf1 : a.pbuf0;
        float* pn = (iter & 1) ? a.pbuf0 : a.pbuf1;
        uint32_t const at_p = o.p[iter & 1];
        float* const PC = values_at<float>(at_p);
        float* const PN = values_at<float>(o.p[(iter & 1) ^ 1]);
        Field<float> const ps{pn, 2u};
        for_tiles(sh, [&](uint32_t r, uint32_t, uint32_t li, uint32_t i, bool live) {
            if (!live) return;
            a.sdp[i] = S[li];
            if (sh.tagged) publish(a, sh, sums, r, i, S[li]);
        });
        if (!exchange(a, sh, s, [&] {
                receive(a, l, sh, s, sums, [&](uint32_t li, float2 x) { S[li] = x; });
            })) {
            return false;
        }
        PhaseErr e{0ull, 0u};
        for_tiles<R>(sh, [&](uint32_t r, uint32_t t, uint32_t li, uint32_t i, bool live) {
            if (!live) return;
            auto const k = kept.get(r, i, read);
            float const p = PC[li];
            float const beta =
              iisph_beta<K, 2>(P, dt, p, S[li], k.c, k.cs,
                               IisphAll{a, pc, at_p, o.rho, o.sdp, o.dii},
                               staged_list(a, l, s, t, i), staged_boundary(a, l, s, t, i));
            float err = 0.0f;
            bool counted;
            float const q = iisph_new_pressure(P, &a.ss[s.part.scene], p, k.f[0], k.f[1], beta,
                                               err, counted);
            PN[li] = q;
            publish(a, sh, ps, r, i, q);
            if (counted) e.add(static_cast<unsigned long long>(err * 1000.0f), err);
        });
        stash_errors(s, e);
        if (!exchange(a, sh, s, [&] {
                receive(a, l, sh, s, ps, [&](uint32_t li, float x) { PN[li] = x; });
            })) {
            return false;
        }
        // the next iteration's sums while the exit test's records travel
        // (a.sdp keeps the last iteration's for the accessors)
        sum_dij(iter + 1);
        block_sync();
        return s.ok != 0;
    });
    if (iters < 0) return false;
    finish_loop(a, s, iters);
    // p / rho^2 of the final pressures, the halo's too, in the sums' place
    float* const pc = (iters & 1) ? a.pbuf1 : a.pbuf0;
    float const* const PC = values_at<float>(o.p[iters & 1]);
    float* const Q = values_at<float>(o.sdp);
    block_sync();
#pragma unroll 1
    for (uint32_t h = threadIdx.x; h < s.halo_n; h += workers()) {
        uint32_t const li = sh.own() + h;
        Q[li] = p_over_rho2(PC[li], RHO[li]);
    }
    for_tiles(sh, [&](uint32_t, uint32_t, uint32_t li, uint32_t i, bool live) {
        if (!live) return;
        pc[i] = PC[li];
        Q[li] = p_over_rho2(PC[li], RHO[li]);
    });
    block_sync();
    for_tiles(sh, [&](uint32_t, uint32_t t, uint32_t li, uint32_t i, bool live) {
        if (!live) return;
        float2 const u = apply_pressure_of<K, 4>(
          P, a.nf_cnt[i], a.ns_cnt[i], a.v[i], Q[li], IisphQ{a, pc, o.sdp}, dt,
          staged_list(a, l, s, t, i), staged_boundary(a, l, s, t, i));
        a.v[i] = u;
        advance_position(a, P, i, dt, u);
    });
    return true;
}

// iisph_ap.cpp and iisph_pseudo_ap.cpp after the neighbour lists. The shared
// values are the velocities, then the pressure accelerations (from offset 0),
// and p / rho^2 (behind them).
template <bool K, int R, int CH>
__device__ __forceinline__ bool solve_iisph_ap(Arena const& a, Layout const& l, Share& sh,
                                               Shared& s, int pseudo) {
    SceneParams const& P = s.P;
    float const dt = s.dt;
    uint32_t const at_q = l.locals * 8u;
    float2* const A = values_at<float2>(0u);
    float* const Q = values_at<float>(at_q);
    Field<float2> const accs{a.acc, 0u};
    Field<float> const qs{a.qdens, 2u};
    stage_lists<true>(a, l, sh, s);
    for_tiles(sh, [&](uint32_t, uint32_t, uint32_t, uint32_t i, bool live) {
        if (!live) return;
        a.rho[i] = density_of<K>(a, P, i);
        a.v[i] = integrate_external(a, P, i, a.v[i], dt);
        a.pbuf0[i] = 0.0f;
        a.qdens[i] = 0.0f;
    });
    if (!agree(a, sh, s)) return false;
    {
        uint32_t const* const halo = reinterpret_cast<uint32_t const*>(mem + l.halo_at);
#pragma unroll 1
        for (uint32_t h = threadIdx.x; h < s.halo_n; h += blockDim.x) {
            A[sh.own() + h] = __ldcg(a.v + halo[h]);
            Q[sh.own() + h] = 0.0f;
        }
    }
    for_tiles(sh, [&](uint32_t, uint32_t, uint32_t li, uint32_t i, bool live) {
        if (!live) return;
        A[li] = a.v[i];
        Q[li] = 0.0f;
    });
    block_sync();
    for_tiles(sh, [&](uint32_t, uint32_t t, uint32_t li, uint32_t i, bool live) {
        if (!live) return;
        float aii, star;
        ap_diag<K>(P, dt, a.rho[i], A[li], a.nf_cnt[i], a.ns_cnt[i], pseudo,
                   Values<float2>{0u, a.v}, staged_list(a, l, s, t, i),
                   staged_boundary(a, l, s, t, i), aii, star);
        a.aii[i] = aii;
        a.rho_star[i] = star;
    });
    if (!start_loop(a, s)) return false;
    if (keeps_exit()) {
        uint32_t slot = 0u;
        return attend_loop(a, sh, s, 0, false, slot) >= 0;
    }
    auto read = [&](uint32_t i) {
        return Kept<3>{{a.rho[i], a.aii[i], a.rho_star[i]}, a.nf_cnt[i], a.ns_cnt[i]};
    };
    KeptTiles<R, 3> kept;
    kept.load(sh, read);
    // pressure accelerations (displacements) of the current pressures
    auto accelerate = [&] {
        for_tiles<R>(sh, [&](uint32_t r, uint32_t t, uint32_t li, uint32_t i, bool live) {
            if (!live) return;
            auto const k = kept.get(r, i, read);
            A[li] = pressure_accel_of<K, CH>(P, k.c, k.cs, Q[li], Values<float>{at_q, a.qdens},
                                             staged_list(a, l, s, t, i),
                                             staged_boundary(a, l, s, t, i));
        });
    };
    accelerate();
    int const iters = solver_loop(s, 0, [&](int iter) {
        for_tiles(sh, [&](uint32_t r, uint32_t, uint32_t li, uint32_t i, bool live) {
            if (live) publish(a, sh, accs, r, i, A[li]);
        });
        if (!exchange(a, sh, s, [&] {
                receive(a, l, sh, s, accs, [&](uint32_t li, float2 x) { A[li] = x; });
            })) {
            return false;
        }
        PhaseErr e{0ull, 0u};
        for_tiles<R>(sh, [&](uint32_t r, uint32_t t, uint32_t li, uint32_t i, bool live) {
            if (!live) return;
            auto const k = kept.get(r, i, read);
            float const old = a.pbuf0[i];
            float err = 0.0f;
            bool counted;
            float const p = ap_iterate<K, CH>(P, dt, k.c, k.cs, pseudo, k.f[1], k.f[2], old, A[li],
                                              Values<float2>{0u, a.acc}, staged_list(a, l, s, t, i),
                                              staged_boundary(a, l, s, t, i), err, counted);
            a.pbuf0[i] = p;
            float const q = p_over_rho2(p, k.f[0]);
            Q[li] = q;
            publish(a, sh, qs, r, i, q);
            if (counted) e.add(static_cast<unsigned long long>(err * 1000.0f), err);
        });
        stash_errors(s, e);
        if (!exchange(a, sh, s, [&] {
                receive(a, l, sh, s, qs, [&](uint32_t li, float x) { Q[li] = x; });
            })) {
            return false;
        }
        // the new pressures' accelerations (the next iteration's, or the
        // final ones) while the exit test's records travel
        accelerate();
        block_sync();
        return s.ok != 0;
    });
    if (iters < 0) return false;
    finish_loop(a, s, iters);
    for_tiles(sh, [&](uint32_t, uint32_t, uint32_t li, uint32_t i, bool live) {
        if (!live) return;
        float2 const acc = A[li];
        a.acc[i] = acc;
        ap_integrate(a, P, i, dt, a.v[i], acc, pseudo);
    });
    return true;
}

// Source of the PCISPH forces: predicted positions from offset 0, predicted
// velocities from v, (rho, p / rho^2) from r.
struct PcAll {
    Arena const& a;
    float2 const* xs;
    float2 const* vs;
    uint32_t v, r;
    __device__ __forceinline__ PcNeighbor local(uint32_t k) const {
        float2 const f = value_of<float2>(r, k);
        return PcNeighbor{value_of<float2>(0u, k), value_of<float2>(v, k), f.x, f.y};
    }
    __device__ __forceinline__ PcNeighbor at(uint32_t j) const {
        return PcNeighbor{xs[j], vs[j], a.rho[j], a.qdens[j]};
    }
};

// pcisph.cpp:36-164 after the neighbour lists. In the barrier form the
// predicted positions and velocities alternate between two arena buffers: a
// block may predict the next pass while another still reads this one's where
// its lists are in the arena.
template <bool K, int R, int CH>
__device__ __forceinline__ bool solve_pcisph(Arena const& a, Layout const& l, Share& sh,
                                             Shared& s) {
    SceneParams const& P = s.P;
    float const dt = s.dt;
    uint32_t const at_v = l.locals * 8u, at_r = l.locals * 16u;
    float2* const X = values_at<float2>(0u);
    float2* const V = values_at<float2>(at_v);
    float2* const RQ = values_at<float2>(at_r);
    auto codes = [&](uint32_t t, uint32_t i) {
        return staged_rows<kCodeRowBytes>(a, l, s, t, i);
    };
    stage_lists<false>(a, l, sh, s);
    if (!agree(a, sh, s)) return false;
    for_tiles(sh, [&](uint32_t, uint32_t, uint32_t, uint32_t i, bool live) {
        if (!live) return;
        a.vext[i] = pc_external_velocity(a, P, i, dt, a.v[i]);
        a.pbuf0[i] = 0.0f;
    });
    if (keeps_exit()) {
        uint32_t slot = 0u;
        return attend_loop(a, sh, s, 3, false, slot) >= 0;
    }
    auto read = [&](uint32_t i) { return Kept<1>{{0.0f}, a.nf_cnt[i], a.ns_cnt[i]}; };
    KeptTiles<R, 1> kept;
    kept.load(sh, read);
    int const iters = solver_loop(s, 3, [&](int iter) {
        bool const alt = iter & 1;
        Field<float2> const fx{alt ? a.tx : a.xstar, 0u};
        Field<float2> const fv{alt ? a.tv : a.vstar, 2u};
        Field<float> const frho{a.rho, 4u};
        Field<float> const fq{a.qdens, 5u};
        for_tiles(sh, [&](uint32_t r, uint32_t, uint32_t li, uint32_t i, bool live) {
            if (!live) return;
            float2 const vs = pc_predicted_velocity(P, dt, iter, a.vext[i],
                                                    iter > 0 ? a.fp[i] : mk2(0.0f, 0.0f));
            float2 const xs = add2(a.x[i], scl2(dt, vs));
            X[li] = xs;
            V[li] = vs;
            publish(a, sh, fx, r, i, xs);
            publish(a, sh, fv, r, i, vs);
        });
        if (!exchange(a, sh, s, [&] {
                receive(a, l, sh, s, fx, [&](uint32_t li, float2 y) { X[li] = y; });
                receive(a, l, sh, s, fv, [&](uint32_t li, float2 y) { V[li] = y; });
            })) {
            return false;
        }
        PhaseErr e{0ull, 0u};
        for_tiles<R>(sh, [&](uint32_t r, uint32_t t, uint32_t li, uint32_t i, bool live) {
            if (!live) return;
            auto const k = kept.get(r, i, read);
            float const old = a.pbuf0[i];
            float const d = pc_density_of<K, CH>(a, P, i, X[li], k.c, k.cs,
                                                 Values<float2>{0u, fx.plain}, codes(t, i));
            float const p = pc_pressure(P, old, d);
            float const q = p / sqrf(d);
            a.pbuf0[i] = p;
            a.rho[i] = d;
            RQ[li] = mk2(d, q);
            if (sh.tagged) publish(a, sh, frho, r, i, d);
            publish(a, sh, fq, r, i, q);
            e.add(0ull, max_0x(d - P.rho0));
        });
        stash_errors(s, e);
        if (!exchange(a, sh, s, [&] {
                receive(a, l, sh, s, frho, [&](uint32_t li, float y) { RQ[li].x = y; });
                receive(a, l, sh, s, fq, [&](uint32_t li, float y) { RQ[li].y = y; });
            })) {
            return false;
        }
        for_tiles<R>(sh, [&](uint32_t r, uint32_t t, uint32_t li, uint32_t i, bool live) {
            if (!live) return;
            auto const k = kept.get(r, i, read);
            float2 const rq = RQ[li];
            a.fp[i] = pc_forces<K, 2>(a, P, i, PcNeighbor{X[li], V[li], rq.x, rq.y}, a.pbuf0[i],
                                      k.c, k.cs,
                                      PcAll{a, fx.plain, fv.plain, at_v, at_r}, codes(t, i));
        });
        block_sync();
        return s.ok != 0;
    });
    if (iters < 0) return false;
    finish_loop(a, s, iters);
    for_tiles(sh, [&](uint32_t, uint32_t, uint32_t li, uint32_t i, bool live) {
        if (!live) return;
        // (in the barrier form other blocks may still read the last pass's
        // buffers: these get the values they hold, or the other buffer does)
        a.xstar[i] = X[li];
        a.vstar[i] = V[li];
        float2 const u = add2(a.vext[i], scl2(dt / P.mass, a.fp[i]));
        a.v[i] = u;
        advance_position(a, P, i, dt, u);
    });
    return true;
}

// The forms of a method's kernel: threads of a block at most, tiles of a warp
// (0: any number), and list rows loaded together.
template <int METHOD, int MODE, int FORM>
struct Form {
    // (needs registers: IISPH's and PCISPH's terms, compensated sums)
    static constexpr bool kWide = METHOD == kIisph || METHOD == kPcisph || MODE == 1;
    static constexpr int kThreads = (FORM == 0 || kWide) ? 512 : 1024;
    static constexpr int kTiles = FORM == 0 ? 1 : FORM == 1 ? (kWide ? 2 : 1)
                                : FORM == 2 ? (kWide ? 4 : 2) : 0;
    static constexpr int kRows = FORM == 0 ? 8 : 4;
};

template <int METHOD, bool K, int R, int CH>
__device__ __forceinline__ bool solve(Arena const& a, Layout const& l, Share& sh, Shared& s) {
    if constexpr (METHOD == kDfsph) return solve_dfsph<K, R, CH>(a, l, sh, s);
    if constexpr (METHOD == kIisph) return solve_iisph<K, R, CH>(a, l, sh, s);
    if constexpr (METHOD == kIisphAp) return solve_iisph_ap<K, R, CH>(a, l, sh, s, 0);
    if constexpr (METHOD == kIisphPseudoAp) return solve_iisph_ap<K, R, CH>(a, l, sh, s, 1);
    if constexpr (METHOD == kPcisph) return solve_pcisph<K, R, CH>(a, l, sh, s);
    return false;
}

// Between two shares of a block (one thread): the share before is done, and
// its scene when it was the last of them, unless a wait gave up after the
// threads' last look.
__device__ __forceinline__ void next_share(Arena const& a, Shared& s) {
    if (s.part.size) {
        if (!s.ok) {
            s.ticket = kNoKey;
            *reinterpret_cast<uint32_t volatile*>(a.gave_up) = 1u;
            return;
        }
        // (both atomics on their way together)
        uint32_t const done = atomicAdd(&a.gangs[s.part.scene].done, 1u);
        s.ticket = atomicAdd(&a.control->ticket, 1u);
        if (done + 1u == s.part.size) atomicAnd(&a.ss[s.part.scene].error, ~kErrUnsolved);
        s.part.size = 0u;
    } else {
        s.ticket = atomicAdd(&a.control->ticket, 1u);
    }
    s.used = 0u;
    s.wanted = 0u;
    s.halo_n = 0u;
    s.ok = 1;
    s.plain = 0;
    s.target = 0u;
}

// Every block takes shares in order until none is left. A gang's blocks wait
// for each other only: shares are taken in order, so when a block waits, every
// earlier gang is fully staffed and finishes, and its blocks go on to staff
// this one. The launch is cooperative: all its blocks are resident. A block
// whose wait gives up leaves the launch; every scene that is not solved to the
// end, of that gang or of one that found no blocks any more, keeps the
// kErrUnsolved that k_begin_substep gave it.
template <int METHOD, int MODE, int FORM>
__global__ void __launch_bounds__(Form<METHOD, MODE, FORM>::kThreads, 1)
  k_resident_solve(Arena a, GangPart const* parts, uint32_t const* nparts, Layout l, int watched) {
    __shared__ Shared s;
    if (watched && a.control->drifted) return;
    if (threadIdx.x == 0) s.part.size = 0u;
    for (;;) {
        block_sync();
        if (threadIdx.x == 0) next_share(a, s);
        block_sync();
        uint32_t const ticket = s.ticket;
        if (ticket >= *nparts) return;
        GangPart const part = parts[ticket];
        if (!a.ss[part.scene].active) continue;
        {
            uint32_t const* const from = reinterpret_cast<uint32_t const*>(a.sp + part.scene);
            uint32_t* const to = reinterpret_cast<uint32_t*>(&s.P);
#pragma unroll 1
            for (uint32_t k = threadIdx.x; k < sizeof(SceneParams) / 4; k += blockDim.x) {
                to[k] = from[k];
            }
            if (threadIdx.x == 0) {
                s.part = part;
                s.dt = a.ss[part.scene].dt;
                s.new_frame = a.ss[part.scene].new_frame;
                if (a.inject == 1u && part.rank == 0u) s.target = 1u;  // waits for one too many
            }
        }
        block_sync();
        Share sh{s.P.fluid_begin + part.tile * 32u, part.tiles, s.P.fluid_begin + s.P.fluid_count,
                 0u, 0u, false};
        constexpr int R = Form<METHOD, MODE, FORM>::kTiles, CH = Form<METHOD, MODE, FORM>::kRows;
        bool const ok = (MODE && s.P.precision) ? solve<METHOD, true, R, CH>(a, l, sh, s)
                                                : solve<METHOD, false, R, CH>(a, l, sh, s);
        // A thread whose wait gave up, or that saw another's give up, leaves; the
        // block's barriers then count the threads that are left, and no share is
        // taken any more.
        if (!ok) {
            s.ticket = kNoKey;
            *reinterpret_cast<uint32_t volatile*>(a.gave_up) = 1u;
            return;
        }
    }
}

// Bytes of the gathered values per local slot.
constexpr uint32_t value_bytes(int method) {
    return method == kIisph ? 28u : method == kPcisph ? 24u : 12u;
}

// Halo slots of a share of n particles: a compact share of the storage order
// has 8 to 12 sqrt(n) neighbours outside (two rings at support = dx); up to
// 16 sqrt(n) leaves room for ragged shares and moved particles.
uint32_t halo_slots(uint32_t n) {
    uint32_t root = 1;
    while (root * root < n) ++root;
    return std::min<uint32_t>(2048u, 64u + 16u * root) / 32u * 32u;
}

// The shared-memory layout for shares of at most `tiles` warp tiles.
Layout layout_for(int method, uint32_t tiles, uint32_t smem) {
    Layout l{};
    l.halo_max = halo_slots(tiles * 32u);
    l.locals = tiles * 32u + l.halo_max;
    while ((1u << l.hash_log2) < 2u * l.halo_max) ++l.hash_log2;
    uint32_t const values = std::max(l.locals * value_bytes(method), 6u << l.hash_log2);
    l.halo_at = (values + 15u) / 16u * 16u;
    l.rows_at = l.halo_at + (4u * l.halo_max + 15u) / 16u * 16u;
    l.row_bytes = method == kPcisph ? kCodeRowBytes : kRowBytes;
    l.capacity = smem > l.rows_at ? (smem - l.rows_at) / l.row_bytes : 0u;
    l.capacity = std::min<uint32_t>(l.capacity, 65535u);
    return l;
}

// The largest share (warp tiles of a block) that is faster here than in the
// launch-per-phase kernels; those keep 2,048 threads of a multiprocessor busy,
// this one a tenth of a phase's latency. Measured on B200, two frames of an
// n x n dam break (sub-steps of 3 to 100 iterations), launch-per-phase against
// resident, in us:
//   DFSPH_P  512^2 12,091 / 7,811 (56 tiles), 800^2 20,408 / 13,619 (136),
//            1024^2 45,581 / 53,415 (222: the lists stream from HBM, and two
//            entries in flight per thread do not keep up)
//   AP       256^2 1,337 / 1,098 (14), 512^2 2,417 / 2,196 (56)
//   IISPH    256^2 2,058 / 1,818 (14), 360^2 2,597 / 2,570 (28), 512^2
//            4,051 / 4,880 (56: two divisions an entry, 16 warps)
//   PCISPH   256^2 1,514 / 1,328 (14), 360^2 1,918 / 2,043 (28)
constexpr uint32_t best_share(int method) {
    return method == kDfsph ? 144u : method == kIisph ? 24u : method == kPcisph ? 16u : 64u;
}

template <int METHOD, int MODE, int FORM>
cudaError_t launch_form(Arena const& a, ResidentPlan const& p, bool watched, cudaStream_t st) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(p.grid);
    cfg.blockDim = dim3(p.threads);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_resident_solve<METHOD, MODE, FORM>, a, p.parts, p.nparts,
                              layout_for(METHOD, p.share, p.smem), watched ? 1 : 0);
}

template <int METHOD, int MODE>
cudaError_t launch_one(Arena const& a, ResidentPlan const& p, bool watched, cudaStream_t st) {
    switch (p.form) {
    case 0: return launch_form<METHOD, MODE, 0>(a, p, watched, st);
    case 1: return launch_form<METHOD, MODE, 1>(a, p, watched, st);
    case 2: return launch_form<METHOD, MODE, 2>(a, p, watched, st);
    default: return launch_form<METHOD, MODE, 3>(a, p, watched, st);
    }
}

template <int METHOD, int MODE, int FORM>
bool prepare_form(ResidentLimits& l) {
    auto* const kernel = k_resident_solve<METHOD, MODE, FORM>;
    constexpr int threads = Form<METHOD, MODE, FORM>::kThreads;
    cudaFuncAttributes fa{};
    int dev = 0, optin = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaFuncGetAttributes(&fa, kernel) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) !=
          cudaSuccess) {
        return false;
    }
    uint32_t const smem = (uint32_t(optin) - uint32_t(fa.sharedSizeBytes)) / 16u * 16u;
    l.smem = std::min(l.smem, smem);
    l.warps[FORM] = uint32_t(threads) / 32u - 1u;  // one keeps the exit test
    l.tiles[FORM] = uint32_t(Form<METHOD, MODE, FORM>::kTiles);
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) ==
             cudaSuccess &&
           cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) ==
             cudaSuccess &&
           per_sm > 0;
}

template <int METHOD, int MODE>
bool prepare_one(ResidentLimits& l) {
    int dev = 0, sms = 0, coop = 0;
    l = ResidentLimits{};
    l.smem = 0xffffffffu;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
        !prepare_form<METHOD, MODE, 0>(l) || !prepare_form<METHOD, MODE, 1>(l) ||
        !prepare_form<METHOD, MODE, 2>(l) || !prepare_form<METHOD, MODE, 3>(l)) {
        return false;
    }
    l.share = std::min(kMaxTiles, best_share(METHOD));
    // the values and the halo of a share have to fit whole
    while (l.share && layout_for(METHOD, l.share, l.smem).rows_at > l.smem) --l.share;
    l.blocks = l.share ? uint32_t(sms) : 0u;
    return l.blocks > 0u;
}

}  // namespace

// One method's entries, instantiated in its own source file.
template <int METHOD>
bool resident_limits_of(bool comp, ResidentLimits& l) {
    return comp ? prepare_one<METHOD, 1>(l) : prepare_one<METHOD, 0>(l);
}
template <int METHOD>
uint32_t resident_smem_of(uint32_t tiles, uint32_t most) {
    Layout const l = layout_for(METHOD, tiles, 0xffffffu);
    return uint32_t(std::min<uint64_t>(most, l.rows_at + uint64_t(tiles) * 24u * l.row_bytes));
}
template <int METHOD>
cudaError_t launch_resident_of(Arena const& a, ResidentPlan const& p, bool comp, bool watched,
                               cudaStream_t st) {
    return comp ? launch_one<METHOD, 1>(a, p, watched, st)
                : launch_one<METHOD, 0>(a, p, watched, st);
}

}  // namespace emerald
