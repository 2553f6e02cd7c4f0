// Neighbour build on the GPU: Morton keys, cell binning, cell ranges and the
// per-particle neighbour lists of emerald/sph_common/neighborhood.{h,cpp}.
//
// The reference sorts (z, index) pairs and keeps a hash map from z to the
// [begin, end) range of each cell (neighborhood.cpp:10-124). Here each scene
// has an open-addressing table keyed by z; binning counts the members of
// every cell, and an exclusive scan turns the counts into ranges. The
// neighbour search then walks the 3x3 cells in the reference's row-major
// order, keeps the first 64 accepted candidates and orders them by (distance,
// index) (neighborhood.h:199-282), so the lists are bit-identical. Inside a
// cell the reference's sorted pairs are in index order; here a fluid cell's
// members are in no order, which shows only where the cap cuts a cell (and
// there the search takes them by index) and in the exported cell maps (which
// order them first).
#include "engine_types.cuh"
#include "kernels.cuh"
#include "short_list.cuh"
#include "sph_math.cuh"

namespace emerald {

namespace {

__device__ __forceinline__ uint32_t cell_hash(uint64_t z, uint32_t log2cap) {
    return static_cast<uint32_t>((z * 0x9E3779B97F4A7C15ull) >> (64u - log2cap));
}

// Inserts z into the table (capacity 2^log2cap plus one extra slot reserved
// for z == kEmptyKey, the key of cell (-1, -1)). Returns the slot or
// UINT32_MAX when the table is full; the probe loop is bounded.
__device__ uint32_t table_insert(uint64_t* keys, uint32_t log2cap, uint64_t z) {
    uint32_t const cap = 1u << log2cap;
    if (z == kEmptyKey) return cap;
    uint32_t h = cell_hash(z, log2cap);
    for (uint32_t probe = 0; probe < cap; ++probe) {
        unsigned long long const prev = atomicCAS(
          reinterpret_cast<unsigned long long*>(keys + h), kEmptyKey, z);
        if (prev == kEmptyKey || prev == z) return h;
        h = (h + 1u) & (cap - 1u);
    }
    return UINT32_MAX;
}

__device__ __forceinline__ bool table_find(uint64_t const* keys,
                                           uint32_t log2cap,
                                           uint64_t z,
                                           uint32_t& slot) {
    uint32_t const cap = 1u << log2cap;
    if (z == kEmptyKey) {
        slot = cap;
        return true;
    }
    uint32_t h = cell_hash(z, log2cap);
    for (uint32_t probe = 0; probe < cap; ++probe) {
        uint64_t const k = keys[h];
        if (k == z) {
            slot = h;
            return true;
        }
        if (k == kEmptyKey) return false;
        h = (h + 1u) & (cap - 1u);
    }
    return false;
}

struct OtherSet {
    float2 const* x;
    uint64_t const* keys;
    uint32_t const* count;
    uint32_t const* start;
    uint32_t const* members;
    float2 const* member_x;  // positions in member order (nullptr: by x[members])
    uint32_t log2cap;
    uint32_t begin;
    uint32_t const* oid;      // original index of a stored slot (nullptr: slot - begin)
    uint32_t const* slot_of;  // stored slot of an original index (nullptr: begin + oid)
};

__device__ __forceinline__ uint32_t original_index(OtherSet const& o, uint32_t slot) {
    return o.oid ? o.oid[slot] : slot - o.begin;
}
__device__ __forceinline__ uint32_t stored_slot(OtherSet const& o, uint32_t oid) {
    return o.slot_of ? o.slot_of[o.begin + oid] : o.begin + oid;
}

// The member of [b, e) that comes next by original index after `after`.
__device__ __noinline__ uint32_t next_by_index(uint32_t const* members, uint32_t const* oid,
                                               uint32_t first, uint32_t b, uint32_t e,
                                               int64_t after) {
    uint32_t best = 0;
    int64_t best_index = INT64_MAX;
#pragma unroll 1
    for (uint32_t m = b; m != e; ++m) {
        uint32_t const other = members[m];
        int64_t const index = oid ? oid[other] : other - first;
        if (index > after && index < best_index) {
            best = other;
            best_index = index;
        }
    }
    return best;
}

// The neighbour search of create_neighborhoods
// (emerald/sph_common/neighborhood.h:199-282). Accepted candidates are kept
// in `list` as (distance bits << 32 | scene-local index), sorted ascending,
// which is the reference's (distance, index) order for non-negative
// distances. Returns the count. by_index takes each cell's members by index
// from lists that are in no order, which matters only where the 64-entry cap
// cuts the candidates.
__device__ __forceinline__ int find_neighbors(float2 pos,
                              uint32_t self,
                              bool same_set,
                              float cell,
                              float max_distance,
                              OtherSet const& o,
                              bool by_index,
                              uint64_t (&list)[kMaxNeighbors]) {
    int32_t gx, gy;
    grid_coord(pos, cell, gx, gy);
    int cnt = 0;
    // (offsets, and cells as their bit patterns: a position too far out is in
    // the last cell of an int32, whose neighbour wraps)
    for (uint32_t j = 0; cnt < kMaxNeighbors && j < 3; ++j) {
        for (uint32_t k = 0; cnt < kMaxNeighbors && k < 3; ++k) {
            uint32_t slot;
            uint64_t const z = morton2(static_cast<uint32_t>(gx) + k - 1u,
                                       static_cast<uint32_t>(gy) + j - 1u);
            if (!table_find(o.keys, o.log2cap, z, slot)) continue;
            uint32_t const b = o.start[slot];
            uint32_t const e = b + o.count[slot];
            int64_t last = -1;
            for (uint32_t m = b; cnt < kMaxNeighbors && m != e; ++m) {
                uint32_t const other =
                  by_index ? next_by_index(o.members, o.oid, o.begin, b, e, last) : o.members[m];
                if (by_index) last = original_index(o, other);
                if (same_set && other == self) continue;
                float2 const vec = sub2(o.x[other], pos);
                float const dist = length2f(vec);
                if (dist >= max_distance) continue;
                uint64_t const key = (static_cast<uint64_t>(__float_as_uint(dist)) << 32) |
                                     static_cast<uint64_t>(original_index(o, other));
                int p = cnt;
                while (p > 0 && list[p - 1] > key) {
                    list[p] = list[p - 1];
                    --p;
                }
                list[p] = key;
                ++cnt;
            }
        }
    }
    return cnt;
}

template <bool SOLID>
__global__ void k_bin(Arena a) {
    int32_t const s = (SOLID ? a.stile_scene : a.tile_scene)[blockIdx.x];
    if (s < 0) return;
    SceneParams const& P = a.sp[s];
    if (!SOLID && !a.ss[s].active) return;
    uint32_t const i = blockIdx.x * kTile + threadIdx.x;
    uint32_t const begin = SOLID ? P.solid_begin : P.fluid_begin;
    uint32_t const count = SOLID ? P.solid_count : P.fluid_count;
    if (i - begin >= count) return;
    float2 const p = SOLID ? a.xs[i] : a.x[i];
    int32_t gx, gy;
    grid_coord(p, P.cell_size, gx, gy);
    uint64_t const z = morton2(static_cast<uint32_t>(gx), static_cast<uint32_t>(gy));
    (SOLID ? a.szkey : a.zkey)[i] = z;
    uint32_t const tb = SOLID ? P.stab_begin : P.ftab_begin;
    uint32_t const lg = SOLID ? P.stab_log2 : P.ftab_log2;
    uint32_t const slot = table_insert((SOLID ? a.skeys : a.fkeys) + tb, lg, z);
    uint32_t* out_slot = SOLID ? a.sslot : a.slot;
    if (slot == UINT32_MAX) {
        atomicOr(&a.ss[s].error, kErrTableFull);
        out_slot[i] = UINT32_MAX;
        return;
    }
    uint32_t const r = atomicAdd((SOLID ? a.scount : a.fcount) + tb + slot, 1u);
    out_slot[i] = tb + slot;
    (SOLID ? a.srank : a.rank)[i] = r;
}

template <bool SOLID>
__global__ void k_scatter(Arena a) {
    int32_t const s = (SOLID ? a.stile_scene : a.tile_scene)[blockIdx.x];
    if (s < 0) return;
    SceneParams const& P = a.sp[s];
    if (!SOLID && !a.ss[s].active) return;
    uint32_t const i = blockIdx.x * kTile + threadIdx.x;
    uint32_t const begin = SOLID ? P.solid_begin : P.fluid_begin;
    uint32_t const count = SOLID ? P.solid_count : P.fluid_count;
    if (i - begin >= count) return;
    uint32_t const slot = (SOLID ? a.sslot : a.slot)[i];
    if (slot == UINT32_MAX) return;
    uint32_t const pos = (SOLID ? a.sstart : a.fstart)[slot] + (SOLID ? a.srank : a.rank)[i];
    (SOLID ? a.smembers : a.members)[pos] = i;
    if (!SOLID) {
        // for the search: the cells' positions side by side, and where the
        // particle itself stands among them
        a.member_x[pos] = a.x[i];
        a.rank[i] = pos;
    }
}

// Orders every cell's members by original index (the within-cell order of
// the reference's sorted (z, index) pairs). oid may be nullptr (storage order
// is the original order).
__global__ void k_sort_cells(uint32_t const* count,
                             uint32_t const* start,
                             uint32_t* members,
                             uint32_t const* oid,
                             uint32_t total) {
    uint32_t const e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= total) return;
    uint32_t const c = count[e];
    if (c < 2) return;
    uint32_t* m = members + start[e];
    for (uint32_t q = 1; q < c; ++q) {
        uint32_t const v = m[q];
        uint32_t const kv = oid ? oid[v] : v;
        uint32_t p = q;
        while (p > 0 && (oid ? oid[m[p - 1]] : m[p - 1]) > kv) {
            m[p] = m[p - 1];
            --p;
        }
        m[p] = v;
    }
}

// kSearchBatch of a row's candidates in flight together (a row
// holds about twelve at one particle per support squared).
constexpr int kSearchBatch = 6;

// The first members and the counts of the nine cells around (gx, gy), in the
// reference's row-major order: nine first probes in flight together, then
// nine ranges. Linear probing from the first probe is bounded by the
// capacity, as in table_find.
__device__ __forceinline__ void cell_ranges(OtherSet const& o, int32_t gx, int32_t gy,
                                            uint32_t (&b)[9], uint32_t (&n)[9]) {
    uint32_t const cap = 1u << o.log2cap;
    uint64_t zx[3], zy[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        zx[q] = spread_bits(static_cast<uint32_t>(gx) + static_cast<uint32_t>(q) - 1u);
        zy[q] = spread_bits(static_cast<uint32_t>(gy) + static_cast<uint32_t>(q) - 1u) << 1;
    }
    uint32_t slot[9];
    uint64_t k[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        // the reserved slot of cell (-1, -1) is read through the same load
        uint64_t const z = zx[q % 3] | zy[q / 3];
        slot[q] = z == kEmptyKey ? cap : cell_hash(z, o.log2cap);
        k[q] = z == kEmptyKey ? z : o.keys[slot[q]];
    }
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        uint64_t const z = zx[q % 3] | zy[q / 3];
#pragma unroll 1
        for (uint32_t probe = 1; k[q] != z && k[q] != kEmptyKey && probe < cap; ++probe) {
            slot[q] = (slot[q] + 1u) & (cap - 1u);
            k[q] = o.keys[slot[q]];
        }
        bool const found = k[q] == z;
        b[q] = found ? o.start[slot[q]] : 0u;
        n[q] = found ? o.count[slot[q]] : 0u;
    }
}

// One thread's column of the block's short lists.
struct ShortList {
    float* x;       // vector to the candidate
    float* y;
    uint32_t* who;  // its place among the members, then its slot
};

// Appends the candidates of row r's three cells (first members b, counts n)
// that are closer than the search distance to the list and returns the new
// count; what is past kShortList is counted only, and past the cap not even
// that. The three cells are one run of candidates, so that lanes with
// differently filled cells stay together. low: the smallest squared distance
// listed.
template <bool BY_PLACE>
__device__ __forceinline__ int search_row(OtherSet const& o, float2 pos, uint32_t self,
                                          float reject_l2, uint32_t const (&b)[9],
                                          uint32_t const (&n)[9], int r, ShortList const& list,
                                          int cnt, float& low) {
    uint32_t const n0 = n[3 * r];
    uint32_t const n01 = n0 + n[3 * r + 1];
    uint32_t const all = n01 + n[3 * r + 2];
    uint32_t const off0 = b[3 * r];
    uint32_t const off1 = b[3 * r + 1] - n0;
    uint32_t const off2 = b[3 * r + 2] - n01;
#pragma unroll 1
    for (uint32_t m0 = 0; m0 < all && cnt <= kMaxNeighbors; m0 += kSearchBatch) {
        uint32_t at[kSearchBatch];
        float2 xo[kSearchBatch];
#pragma unroll
        for (int u = 0; u < kSearchBatch; ++u) {
            uint32_t const m = m0 + u;
            at[u] = m + (m < n0 ? off0 : (m < n01 ? off1 : off2));
            // past the end of the row: the particle's own place, not taken
            if (m >= all) at[u] = self;
        }
        if (!BY_PLACE) {
#pragma unroll
            for (int u = 0; u < kSearchBatch; ++u) {
                if (at[u] != self) at[u] = o.members[at[u]];
            }
        }
#pragma unroll
        for (int u = 0; u < kSearchBatch; ++u) {
            if (BY_PLACE) {
                xo[u] = o.member_x[at[u]];
            } else {
                xo[u] = pos;
                if (at[u] != self) xo[u] = o.x[at[u]];
            }
        }
#pragma unroll
        for (int u = 0; u < kSearchBatch; ++u) {
            float2 const vec = sub2(xo[u], pos);
            float const l2 = vec.x * vec.x + vec.y * vec.y;
            bool const take = at[u] != self && !(l2 >= reject_l2);
            if (take && cnt < kShortList) {
                list.x[cnt * kTile] = vec.x;
                list.y[cnt * kTile] = vec.y;
                list.who[cnt * kTile] = at[u];
            }
            low = take ? fminf(low, l2) : low;
            cnt += take ? 1 : 0;
        }
    }
    return cnt;
}

// The order of the cnt <= kShortList listed candidates by (distance, index).
template <bool BY_PLACE>
__device__ __forceinline__ uint64_t sort_short_list(OtherSet const& o, ShortList const& list,
                                                    int cnt) {
    uint32_t d[kShortList];
#pragma unroll
    for (int q = 0; q < kShortList; ++q) {
        d[q] = unused_key(q);
        if (q < cnt) {
            float const vx = list.x[q * kTile], vy = list.y[q * kTile];
            d[q] = (__float_as_uint(sqrtf(vx * vx + vy * vy)) & ~15u) | q;
            if (BY_PLACE) list.who[q * kTile] = o.members[list.who[q * kTile]];
        }
    }
    return order_short_list(d, cnt, [&](int q) {
        uint32_t const at = static_cast<uint32_t>(q) * kTile;
        float const dist = sqrtf(list.x[at] * list.x[at] + list.y[at] * list.y[at]);
        return ShortKey{__float_as_uint(dist), original_index(o, list.who[at])};
    });
}

// Writes list entry k of particle i: index, W and GradW(-vector_to)
// (compute_neighbor_kernels / compute_neighbor_kernel_gradients,
// emerald/sph_common/neighborhood.cpp:178-210) from the vector to the
// neighbour and its length.
__device__ __forceinline__ void write_entry(uint32_t* idx_out, float* w_out, float2* gw_out,
                                            size_t e, uint32_t j, float dist, float2 vec,
                                            float h, bool kernels) {
    idx_out[e] = j;
    if (!kernels) return;
    float w, dw;
    kernel_w_dw(dist, h, w, dw);
    w_out[e] = w;
    float2 const dp = neg2(vec);
    float2 g = mk2(0.0f, 0.0f);
    if (safe_v(dp, dist)) {
        float2 const u = div2(dp, dist);
        g = mk2(u.x * dw, u.y * dw);
    }
    gw_out[e] = g;
}

// Compensated mode: the entry's vector and distance come from the double
// positions (x_i - x_j in double, rounded once), so that the rounding of
// large coordinates does not enter the kernel values.
__device__ __noinline__ void write_entry_precise(uint32_t* idx_out, float* w_out, float2* gw_out,
                                                 size_t e, uint32_t j, double2 pos64,
                                                 double2 const* x64o, float2 const* xo, float h) {
    idx_out[e] = j;
    double2 const xj = x64o ? x64o[j] : make_double2(double(xo[j].x), double(xo[j].y));
    double const ddx = pos64.x - xj.x;
    double const ddy = pos64.y - xj.y;
    float2 const dp = mk2(static_cast<float>(ddx), static_cast<float>(ddy));
    float const dist = static_cast<float>(sqrt(ddx * ddx + ddy * ddy));
    float w, dw;
    kernel_w_dw(dist, h, w, dw);
    w_out[e] = w;
    float2 g = mk2(0.0f, 0.0f);
    if (safe_v(dp, dist)) {
        float2 const u = div2(dp, dist);
        g = mk2(u.x * dw, u.y * dw);
    }
    gw_out[e] = g;
}

// What the search of a particle without a short list needs.
struct LongSearch {
    OtherSet o;
    float2 pos;
    uint32_t i, self;
    int cnt;      // accepted candidates, or any number past the cap
    bool normal;  // every vector's length is the root of its dot product
    float cell, reject_l2, h;
    uint8_t* cnt_out;
    uint32_t* idx_out;
    float* w_out;
    float2* gw_out;
    size_t stride;
    bool kernels, precise;
    double2 pos64;
    double2 const* x64o;
    ShortList list;
};

// Particles with 17 to 64 neighbours: runs of sixteen are sorted by the network
// and merged as they are written. Where a vector is too short for its dot
// product the one-at-a-time search decides.
// Out of line, so that k_neighbors keeps its registers. A 256 x 256 frame at a
// support of two spacings (45 neighbours) took 5.3 ms with PCISPH when every
// long list was made by insertion, 2.1 ms now; 1.5 spacings (26 neighbours)
// with IISPH 3.5 and 1.9 ms.
template <bool SOLID_OTHER>
__device__ __noinline__ void neighbors_long(LongSearch s) {
    OtherSet const& o = s.o;
    ShortList const& list = s.list;
    float2 const pos = s.pos;
    int cnt = s.cnt;
    uint64_t full[kMaxNeighbors];
    int ends[4];  // of the sorted runs of `full`
    // the places of the first kMaxNeighbors accepted, in any order
    int found = 0;
    float low = s.normal ? 1.0f : 0.0f;
    if (s.normal) {
        uint32_t b[9], n[9];
        int32_t gx, gy;
        grid_coord(pos, s.cell, gx, gy);
        cell_ranges(o, gx, gy, b, n);
#pragma unroll 1
        for (int q = 0; q < 9 && found < kMaxNeighbors; ++q) {
            uint32_t const e = b[q] + n[q];
            int const before = found;
            auto test = [&](uint32_t m, uint32_t& place, float& l2) {
                place = SOLID_OTHER ? o.members[m] : m;
                float2 const vec = sub2(SOLID_OTHER ? o.x[place] : o.member_x[place], pos);
                l2 = vec.x * vec.x + vec.y * vec.y;
                return place != s.self && !(l2 >= s.reject_l2);
            };
            uint32_t place;
            float l2;
#pragma unroll 1
            for (uint32_t m = b[q]; m != e; ++m) {
                if (!test(m, place, l2)) continue;
                low = fminf(low, l2);
                if (found < kMaxNeighbors) full[found] = place;
                ++found;
            }
            if (found <= kMaxNeighbors) continue;
            found = kMaxNeighbors;
            if (SOLID_OTHER) continue;
            // the cap cuts this cell, whose members are in no order: those of
            // the lowest indices stay
            int c = before;
#pragma unroll 1
            for (uint32_t m = b[q]; m != e; ++m) {
                if (!test(m, place, l2)) continue;
                uint64_t const key =
                  (static_cast<uint64_t>(original_index(o, o.members[place])) << 32) | place;
                if (c == kMaxNeighbors && key >= full[c - 1]) continue;
                int p = c < kMaxNeighbors ? c++ : c - 1;
                for (; p > before && full[p - 1] > key; --p) full[p] = full[p - 1];
                full[p] = key;
            }
        }
    }
    if (low >= 2.0f * kFltMin) {
        // sixteen at a time through the short list, then merged
        cnt = found;
#pragma unroll
        for (int run = 0; run < 4; ++run) {
            int const first = run * kShortList;
            int const c = max(0, min(cnt - first, kShortList));
            ends[run] = first + c;
            if (c == 0) continue;
#pragma unroll
            for (int q = 0; q < kShortList; ++q) {
                if (q < c) {
                    uint32_t const place = static_cast<uint32_t>(full[first + q]);
                    float2 const vec =
                      sub2(SOLID_OTHER ? o.x[place] : o.member_x[place], pos);
                    list.x[q * kTile] = vec.x;
                    list.y[q * kTile] = vec.y;
                    list.who[q * kTile] = place;
                }
            }
            uint64_t order = sort_short_list<!SOLID_OTHER>(o, list, c);
#pragma unroll 1
            for (int q = 0; q < c; ++q, order >>= 4) {
                uint32_t const at = (static_cast<uint32_t>(order) & 15u) * kTile;
                float const dist = sqrtf(list.x[at] * list.x[at] + list.y[at] * list.y[at]);
                full[first + q] = (static_cast<uint64_t>(__float_as_uint(dist)) << 32) |
                                  original_index(o, list.who[at]);
            }
        }
    } else {
        cnt = find_neighbors(pos, s.i, !SOLID_OTHER, s.cell, s.cell, o,
                             !SOLID_OTHER && cnt > kMaxNeighbors, full);
        ends[0] = cnt;
        ends[1] = kShortList;
        ends[2] = 2 * kShortList;
        ends[3] = 3 * kShortList;
    }
    s.cnt_out[s.i] = static_cast<uint8_t>(cnt);
    int at[4] = {0, kShortList, 2 * kShortList, 3 * kShortList};
    uint64_t head[4];
#pragma unroll
    for (int run = 0; run < 4; ++run) head[run] = at[run] < ends[run] ? full[at[run]] : ~0ull;
#pragma unroll 1
    for (int k = 0; k < cnt; ++k) {
        uint64_t const lo = head[0] < head[1] ? head[0] : head[1];
        uint64_t const hi = head[2] < head[3] ? head[2] : head[3];
        uint64_t const key = lo < hi ? lo : hi;
#pragma unroll
        for (int run = 0; run < 4; ++run) {
            if (head[run] == key) {
                ++at[run];
                head[run] = at[run] < ends[run] ? full[at[run]] : ~0ull;
            }
        }
        size_t const e = static_cast<size_t>(k) * s.stride + s.i;
        uint32_t const j = stored_slot(o, static_cast<uint32_t>(key & 0xffffffffu));
        if (s.precise) {
            write_entry_precise(s.idx_out, s.w_out, s.gw_out, e, j, s.pos64, s.x64o, o.x, s.h);
        } else {
            write_entry(s.idx_out, s.w_out, s.gw_out, e, j,
                        __uint_as_float(static_cast<uint32_t>(key >> 32)), sub2(o.x[j], pos), s.h,
                        s.kernels);
        }
    }
}

// kernel_w_dw's quotients by what depends on the support alone, with the same
// bits from five multiply-adds each: for y = RN(1 / b) and a q within one ulp
// of a / b whose remainder r = a - b q is exact, RN(q + r y) is the correctly
// rounded quotient (P. Markstein, "Computation of elementary functions on the
// IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990). The first
// correction makes q that close. Supports in [2^-16, 2^10] keep every
// quotient and remainder in the normal range for 2^-62 <= r < 2 h (what the
// short lists hold): the smallest numerators are 2^-71 (W), 2^-46 and 2^-61
// (GradW), the divisors lie in 2^-46..2^32, and no numerator is zero because
// r / h cannot round to 2 for r < 2 h.
struct KernelDivisors {
    float h, hh, h4, hhh, k;
    float y_h, y_hh, y_h4, y_hhh, y_k;
    bool quick;
    __device__ __forceinline__ explicit KernelDivisors(float support)
        : h(support), hh(h * h), h4(4.0f * h), hhh(h * h * h), k(h * h * h * kPi),
          y_h(1.0f / h), y_hh(1.0f / hh), y_h4(1.0f / h4), y_hhh(1.0f / hhh), y_k(1.0f / k),
          quick(h >= 0x1p-16f && h <= 0x1p10f) {}
    static __device__ __forceinline__ float quotient(float a, float b, float y) {
        float q = a * y;
        q = __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
        return __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
    }
    __device__ __forceinline__ void kernel_w_dw(float r, float& w, float& dw) const {
        float const q = quotient(r, h, y_h);
        bool const inner = q <= 1.0f;
        float const t = 2.0f - q;
        float d = quotient(inner ? -3.0f * r : -3.0f * sqrf(t), inner ? hh : h4,
                           inner ? y_hh : y_h4);
        if (inner) d = d + quotient(2.25f * r * r, hhh, y_hhh);
        w = quotient(inner ? 1.0f + q * q * (q * 0.75f - 1.5f) : (t * t * t) / 4.0f, k, y_k);
        dw = quotient(d, k, y_k);
        // past the support; a distance in a list is below 2 h or a NaN, which
        // counts as outside, as in kernel_w_dw
        if (!(q <= 2.0f)) {
            w = 0.0f;
            dw = 0.0f;
        }
    }
};

// One thread a particle, 62 registers (eight blocks an SM; left alone the
// compiler takes 56 and spills). What bounds it is instruction issue and, below
// a wave of blocks, one warp's chain of dependent reads: cell keys, cell
// ranges, then per row two batches of positions that the cell build has laid
// side by side (an index in between would double the chain and the loads).
// Kernel time on one B200 with cold caches, before -> after the short lists
// moved from an insertion sort to the fixed network, the positions to member
// order and W's divisions to multiply-adds: 2k particles 28 -> 15.7 us, 37k
// 30 -> 17.8 us, 262k 70 -> 50 us, 1M 232 -> 171 us. Batches of four measured
// 16.8 / 18.6 / 50.6 / 173 us, with the next batch in flight 17.3 / 19.2 /
// 51.8 / 178 us; four lanes a particle 17.6 / 38 / 158 / 629 us.
template <bool SOLID_OTHER, bool COMP>
__global__ void __launch_bounds__(kTile, 8) k_neighbors(Arena a, int write_kernels) {
    int32_t const s = a.tile_scene[blockIdx.x];
    if (s < 0) return;
    SceneParams const& P = a.sp[s];
    if (!a.ss[s].active) return;
    uint32_t const i = blockIdx.x * kTile + threadIdx.x;
    if (i - P.fluid_begin >= P.fluid_count) return;
    float const h = P.support;
    float const cell = P.cell_size;
    OtherSet o;
    if (SOLID_OTHER) {
        o = OtherSet{a.xs, a.skeys + P.stab_begin, a.scount + P.stab_begin, a.sstart + P.stab_begin,
                     a.smembers, nullptr, P.stab_log2, P.solid_begin, nullptr, nullptr};
    } else {
        o = OtherSet{a.x, a.fkeys + P.ftab_begin, a.fcount + P.ftab_begin, a.fstart + P.ftab_begin,
                     a.members, a.member_x, P.ftab_log2, P.fluid_begin, a.oid, a.slot_of};
    }
    uint8_t* cnt_out = SOLID_OTHER ? a.ns_cnt : a.nf_cnt;
    uint32_t* idx_out = SOLID_OTHER ? a.ns_idx : a.nf_idx;
    float* w_out = SOLID_OTHER ? a.ns_w : a.nf_w;
    float2* gw_out = SOLID_OTHER ? a.ns_gw : a.nf_gw;
    size_t const stride = a.stride;
    if (SOLID_OTHER && P.solid_count == 0) {
        cnt_out[i] = 0;
        return;
    }
    bool const kernels = write_kernels != 0;
    float2 const pos = a.x[i];
    int32_t gx, gy;
    grid_coord(pos, cell, gx, gy);
    if (SOLID_OTHER && P.near_w) {
        int64_t const ix = int64_t(gx) - P.near_x0;
        int64_t const iy = int64_t(gy) - P.near_y0;
        bool near = false;
        if (ix >= 0 && iy >= 0 && ix < int64_t(P.near_w) && iy < int64_t(P.near_h)) {
            uint64_t const bit = uint64_t(iy) * P.near_w + uint64_t(ix);
            near = (a.near_bits[P.near_begin + (bit >> 5)] >> (bit & 31u)) & 1u;
        }
        if (!near) {
            cnt_out[i] = 0;
            return;
        }
    }
    __shared__ uint32_t s_list[3 * kShortList * kTile];
    ShortList const list{reinterpret_cast<float*>(s_list) + threadIdx.x,
                         reinterpret_cast<float*>(s_list) + kShortList * kTile + threadIdx.x,
                         s_list + 2 * kShortList * kTile + threadIdx.x};
    int cnt = 0;
    float low = 1.0f;
    uint32_t const self = SOLID_OTHER ? UINT32_MAX : a.rank[i];
    {
        uint32_t b[9], n[9];
        cell_ranges(o, gx, gy, b, n);
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            cnt = search_row<!SOLID_OTHER>(o, pos, self, P.reject_l2, b, n, r, list, cnt, low);
        }
    }
    bool const precise = COMP && P.precision && kernels;
    double2 const pos64 = precise ? a.x64[i] : make_double2(0.0, 0.0);
    double2 const* const x64o = SOLID_OTHER ? nullptr : a.x64;
    KernelDivisors const div(h);
    // From 2*FLT_MIN on a vector's length is the root of its dot product, which
    // is below max_distance exactly when the product is below reject_l2.
    if (cnt <= kShortList && low >= 2.0f * kFltMin) {
        uint64_t order = sort_short_list<!SOLID_OTHER>(o, list, cnt);
        cnt_out[i] = static_cast<uint8_t>(cnt);
#pragma unroll 1
        for (int k = 0; k < cnt; ++k, order >>= 4) {
            uint32_t const at = (static_cast<uint32_t>(order) & 15u) * kTile;
            size_t const e = static_cast<size_t>(k) * stride + i;
            if (precise) {
                write_entry_precise(idx_out, w_out, gw_out, e, list.who[at], pos64, x64o, o.x, h);
                continue;
            }
            idx_out[e] = list.who[at];
            if (!kernels) continue;
            float2 const dp = mk2(-list.x[at], -list.y[at]);
            float const dist = sqrtf(dp.x * dp.x + dp.y * dp.y);
            float w, dw;
            if (div.quick) {
                div.kernel_w_dw(dist, w, dw);
            } else {
                kernel_w_dw(dist, h, w, dw);
            }
            w_out[e] = w;
            // safe_v: dist is not zero, so only a NaN fails it
            float2 g = mk2(0.0f, 0.0f);
            if (dist > 0.0f) {
                float2 const u = div2(dp, dist);
                g = mk2(u.x * dw, u.y * dw);
            }
            gw_out[e] = g;
        }
        return;
    }
    neighbors_long<SOLID_OTHER>(LongSearch{o, pos, i, self, cnt, low >= 2.0f * kFltMin, cell,
                                           P.reject_l2, h, cnt_out, idx_out, w_out, gw_out, stride,
                                           kernels, precise, pos64, x64o, list});
}

// compute_volumes (emerald/sph2d_box/solids.cpp:52-74) over the solid-solid
// neighbourhood of compute_neighbor_data_and_volumes (:76-137):
// V = numer / (W(0) + sum W) in list order, 1/W(0) without neighbours.
__global__ void k_solid_volumes(Arena a, float numer, int only_scene) {
    int32_t const s = a.stile_scene[blockIdx.x];
    if (s < 0 || s != only_scene) return;
    SceneParams const& P = a.sp[s];
    uint32_t const i = blockIdx.x * kTile + threadIdx.x;
    if (i - P.solid_begin >= P.solid_count) return;
    OtherSet const o{a.xs, a.skeys + P.stab_begin, a.scount + P.stab_begin, a.sstart + P.stab_begin,
                     a.smembers, nullptr, P.stab_log2, P.solid_begin, nullptr, nullptr};
    uint64_t list[kMaxNeighbors];
    int const cnt = find_neighbors(a.xs[i], i, true, P.cell_size, P.cell_size, o, false, list);
    float const w0 = kernel_w(0.0f, P.support);
    if (!cnt) {
        a.vols[i] = 1.0f / w0;
        return;
    }
    float m = w0;
    for (int k = 0; k < cnt; ++k) {
        m += kernel_w(__uint_as_float(static_cast<uint32_t>(list[k] >> 32)), P.support);
    }
    a.vols[i] = numer / m;
}

// Exclusive scan of uint32 counts: per-block sums, a single-block scan of
// the sums, then per-block scans offset by the scanned sums.
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanBlock = kScanThreads * kScanItems;

__device__ __forceinline__ uint32_t warp_inclusive_scan(uint32_t v) {
    int const lane = threadIdx.x & 31;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t const t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Block-wide exclusive scan of one value per thread; returns the block total.
__device__ uint32_t block_exclusive_scan(uint32_t v, uint32_t& excl) {
    __shared__ uint32_t warp_sums[kScanThreads / 32];
    int const lane = threadIdx.x & 31;
    int const warp = threadIdx.x >> 5;
    uint32_t const incl = warp_inclusive_scan(v);
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < kScanThreads / 32 ? warp_sums[lane] : 0u;
        w = warp_inclusive_scan(w);
        if (lane < kScanThreads / 32) warp_sums[lane] = w;
    }
    __syncthreads();
    uint32_t const warp_off = warp ? warp_sums[warp - 1] : 0u;
    excl = warp_off + incl - v;
    uint32_t const total = warp_sums[kScanThreads / 32 - 1];
    __syncthreads();
    return total;
}

__global__ void k_scan_reduce(uint32_t const* in, uint32_t n, uint32_t* sums) {
    size_t const base = static_cast<size_t>(blockIdx.x) * kScanBlock + threadIdx.x * kScanItems;
    uint32_t t = 0;
    for (int k = 0; k < kScanItems; ++k) {
        size_t const e = base + k;
        if (e < n) t += in[e];
    }
    uint32_t excl;
    uint32_t const total = block_exclusive_scan(t, excl);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void k_scan_sums(uint32_t* sums, uint32_t nblocks) {
    uint32_t carry = 0;
    for (uint32_t base = 0; base < nblocks; base += kScanThreads) {
        uint32_t const e = base + threadIdx.x;
        uint32_t const v = e < nblocks ? sums[e] : 0u;
        uint32_t excl;
        uint32_t const total = block_exclusive_scan(v, excl);
        if (e < nblocks) sums[e] = carry + excl;
        carry += total;
    }
}

__global__ void k_scan_apply(uint32_t const* in, uint32_t n, uint32_t const* sums, uint32_t* out) {
    size_t const base = static_cast<size_t>(blockIdx.x) * kScanBlock + threadIdx.x * kScanItems;
    uint32_t vals[kScanItems];
    uint32_t t = 0;
    for (int k = 0; k < kScanItems; ++k) {
        size_t const e = base + k;
        vals[k] = e < n ? in[e] : 0u;
        t += vals[k];
    }
    uint32_t excl;
    block_exclusive_scan(t, excl);
    uint32_t run = sums[blockIdx.x] + excl;
    for (int k = 0; k < kScanItems; ++k) {
        size_t const e = base + k;
        if (e < n) out[e] = run;
        run += vals[k];
    }
}

// Cell ranges in one pass: every block scans its slots' counts and takes its
// range of the members array with one atomic on the cursor count[n], which
// the caller cleared with the counts. Cells land in block order, not slot
// order; each cell's members stay contiguous, which is all the searches and
// the sort products read (start[cell], count[cell]).
__global__ void k_cell_ranges(uint32_t const* count, uint32_t n, uint32_t* start) {
    size_t const base = static_cast<size_t>(blockIdx.x) * kScanBlock + threadIdx.x * kScanItems;
    uint32_t vals[kScanItems];
    uint32_t t = 0;
    for (int k = 0; k < kScanItems; ++k) {
        size_t const e = base + k;
        vals[k] = e < n ? count[e] : 0u;
        t += vals[k];
    }
    uint32_t excl;
    uint32_t const total = block_exclusive_scan(t, excl);
    __shared__ uint32_t block_base;
    if (threadIdx.x == 0) {
        block_base = total ? atomicAdd(const_cast<uint32_t*>(count) + n, total) : 0u;
    }
    __syncthreads();
    uint32_t run = block_base + excl;
    for (int k = 0; k < kScanItems; ++k) {
        size_t const e = base + k;
        if (e < n) start[e] = run;
        run += vals[k];
    }
}

}  // namespace

uint32_t scan_scratch_words(uint32_t n) { return (n + kScanBlock - 1) / kScanBlock + 1; }

void launch_exclusive_scan(uint32_t const* in, uint32_t n, uint32_t* out, uint32_t* scratch,
                           cudaStream_t st) {
    if (n == 0) return;
    uint32_t const nb = (n + kScanBlock - 1) / kScanBlock;
    k_scan_reduce<<<nb, kScanThreads, 0, st>>>(in, n, scratch);
    k_scan_sums<<<1, kScanThreads, 0, st>>>(scratch, nb);
    k_scan_apply<<<nb, kScanThreads, 0, st>>>(in, n, scratch, out);
}

// The count arrays hold one word more than the table: the cursor of
// k_cell_ranges, cleared with the counts.
void launch_build_cells(Arena const& a, bool solid, uint32_t tiles, uint32_t* scan_scratch,
                        cudaStream_t st) {
    (void)scan_scratch;
    if (solid) {
        cudaMemsetAsync(a.skeys, 0xff, sizeof(uint64_t) * a.stab_total, st);
        cudaMemsetAsync(a.scount, 0, sizeof(uint32_t) * (a.stab_total + 1), st);
        k_bin<true><<<tiles, kTile, 0, st>>>(a);
        k_cell_ranges<<<(a.stab_total + kScanBlock - 1) / kScanBlock, kScanThreads, 0, st>>>(
          a.scount, a.stab_total, a.sstart);
        k_scatter<true><<<tiles, kTile, 0, st>>>(a);
        k_sort_cells<<<(a.stab_total + 255) / 256, 256, 0, st>>>(a.scount, a.sstart, a.smembers,
                                                                 nullptr, a.stab_total);
    } else {
        cudaMemsetAsync(a.fkeys, 0xff, sizeof(uint64_t) * a.ftab_total, st);
        cudaMemsetAsync(a.fcount, 0, sizeof(uint32_t) * (a.ftab_total + 1), st);
        k_bin<false><<<tiles, kTile, 0, st>>>(a);
        k_cell_ranges<<<(a.ftab_total + kScanBlock - 1) / kScanBlock, kScanThreads, 0, st>>>(
          a.fcount, a.ftab_total, a.fstart);
        k_scatter<false><<<tiles, kTile, 0, st>>>(a);
    }
}

void launch_order_members(Arena const& a, uint32_t tab_begin, uint32_t tab_size, cudaStream_t st) {
    k_sort_cells<<<(tab_size + 255) / 256, 256, 0, st>>>(a.fcount + tab_begin, a.fstart + tab_begin,
                                                         a.members, a.oid, tab_size);
}

void launch_neighbors(Arena const& a, uint32_t tiles, bool solid_other, bool write_kernels,
                      cudaStream_t st, bool comp) {
    int const wk = write_kernels ? 1 : 0;
    if (solid_other) {
        if (comp) {
            k_neighbors<true, true><<<tiles, kTile, 0, st>>>(a, wk);
        } else {
            k_neighbors<true, false><<<tiles, kTile, 0, st>>>(a, wk);
        }
    } else {
        if (comp) {
            k_neighbors<false, true><<<tiles, kTile, 0, st>>>(a, wk);
        } else {
            k_neighbors<false, false><<<tiles, kTile, 0, st>>>(a, wk);
        }
    }
}

void launch_solid_volumes(Arena const& a, uint32_t solid_tiles, float numer, int scene,
                          cudaStream_t st) {
    k_solid_volumes<<<solid_tiles, kTile, 0, st>>>(a, numer, scene);
}

}  // namespace emerald
