// Patterns of a search that ran in another item order, put into the
// reference's insertion order on the device.
//
// The deep levels extend patterns by items of increasing support (few
// candidates fail that way: 9.8 M intersections instead of 139.6 M on
// 1,000,000 x 20,000 Zipf baskets), so a pattern's parent in the emitted tree
// is the pattern without its most frequent item.  The reference's order
// (cuEclat.py:183-245) needs the prefix tree of the column order, where the
// parent is the pattern without its largest column.  That subset is frequent
// too, hence among the patterns; it is found by a hash of its set of items --
// the sum of one 64-bit value per item, so that leaving an item out is a
// subtraction -- and every hit is checked item by item.
//
// With the canonical parents, the children of every pattern sorted by column
// (one radix sort) and the number of descendants of each, a pattern's place
// follows from its parent's: the reference lists a pair's children, then each
// child's subtree in the same way.  Levels are walked deepest first for the
// descendants and shallowest first for the places, one small launch each.
//
// Everything here is bound by random 4-byte accesses that mostly stay in L2:
// 6.27 M patterns take about 5 ms, where the host walk took 130 ms.
#pragma once
#include "common.cuh"

namespace cpm {

constexpr uint32_t ORD_NONE = 0xffffffffu;

struct OrdParams {
    const uint32_t *parent, *item, *sup, *db;  // the emitted tree (db null: one database)
    uint32_t n, base;                          // patterns; singletons and pairs come first, per database
    uint64_t *hash;                            // of pairs and deeper patterns
    uint32_t *top;                             // largest column
    uint16_t *depth;
    uint32_t *table, mask;                     // open addressing: pattern ids
    uint32_t *cpar;                            // canonical parent (patterns from base on)
    uint64_t *key;                             // cpar << col_bits | top, and the pattern, from base on
    uint32_t *val;
    uint32_t col_bits;
    const uint64_t *skey;                      // sorted by key
    const uint32_t *sval;
    uint32_t *cbeg, *cend;                     // a pattern's children: sval[cbeg, cend)
    uint32_t *at;                              // a deep pattern's position in sval
    uint32_t *desc;                            // descendants
    uint32_t *sdesc;                           // desc in the order of sval, then its exclusive sum
    uint32_t *dbase;                           // exclusive sum of desc over the patterns before base
    uint32_t *reg, *pos;                       // a deep pattern's descendants start at reg, itself at pos
    const uint64_t *pat_base;                  // per database: its first pattern id (n_db + 1 entries)
    uint32_t n_db;
    unsigned long long *info;                  // [0] longest pattern, [1] item slots, [2] nonzero: a parent is missing
    // in final order
    uint32_t *inv, *o_sup, *o_par;
    uint16_t *o_depth;
    unsigned long long *db_first;              // per database: its first pattern in the final order
};

// The value of an item (database d): the SplitMix64 output function (Steele,
// Lea, Flood, "Fast splittable pseudorandom number generators", 2014).
__host__ __device__ __forceinline__ uint64_t ord_value(uint32_t item, uint32_t d) {
    uint64_t z = (((uint64_t)d << 32) | item) + 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}

// Hash, largest column and length of every pattern; pairs and deeper ones enter the table.
__global__ void k_ord_hash(OrdParams P) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t d = 0, top = 0;
    if (k < P.n) {
        const uint32_t db = P.db ? P.db[k] : 0u;
        uint64_t h = 0;
        for (uint32_t v = k; v != ORD_NONE; v = P.parent[v]) {
            const uint32_t it = P.item[v];
            h += ord_value(it, db);
            top = max(top, it);
            ++d;
        }
        P.top[k] = top;
        P.depth[k] = (uint16_t)min(d, 65535u);
        P.hash[k] = h;
        if (d > 1) {
            // The table has twice as many slots as patterns: a free one is met.
            for (uint32_t s = (uint32_t)h & P.mask; atomicCAS(P.table + s, ORD_NONE, k) != ORD_NONE; s = (s + 1) & P.mask) {
            }
        }
    }
    const unsigned long long slots = warp_sum_u64(d);
    const uint32_t most = warp_max_u32(d);
    if ((threadIdx.x & 31) == 0 && most) {
        atomicMax(P.info, (unsigned long long)most);
        atomicAdd(P.info + 1, slots);
    }
}

// The canonical parent of every deep pattern, and its sort key.
__global__ void k_ord_parent(OrdParams P) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.n - P.base) return;
    const uint32_t k = P.base + i, d = P.depth[k], top = P.top[k];
    const uint64_t want = P.hash[k] - ord_value(top, P.db ? P.db[k] : 0u);
    constexpr uint32_t KEPT = 24;
    uint32_t x[KEPT];
    if (d <= KEPT) {
        uint32_t v = k;
        for (uint32_t j = 0; j < d; ++j, v = P.parent[v]) x[j] = P.item[v];
    }
    uint32_t q = ORD_NONE;
    for (uint32_t s = (uint32_t)want & P.mask;; s = (s + 1) & P.mask) {
        q = P.table[s];
        if (q == ORD_NONE) break;
        if (P.hash[q] != want || P.depth[q] + 1u != d) continue;
        bool same = !P.db || P.db[q] == P.db[k];
        for (uint32_t v = q; same && v != ORD_NONE; v = P.parent[v]) {
            const uint32_t it = P.item[v];
            bool found = false;
            if (d <= KEPT) {
                for (uint32_t j = 0; j < d; ++j) found |= x[j] == it;
            } else {
                for (uint32_t u = k; u != ORD_NONE && !found; u = P.parent[u]) found = P.item[u] == it;
            }
            same = found && it != top;
        }
        if (same) break;
    }
    if (q == ORD_NONE) {
        P.info[2] = 1;
        q = 0;
    }
    P.cpar[k] = q;
    P.key[i] = ((uint64_t)q << P.col_bits) | top;
    P.val[i] = k;
}

// ---- the steps after the sort, each for one index ----

__device__ __forceinline__ void ord_children(const OrdParams &P, uint32_t s) {
    const uint32_t nd = P.n - P.base, p = (uint32_t)(P.skey[s] >> P.col_bits);
    if (s == 0 || (uint32_t)(P.skey[s - 1] >> P.col_bits) != p) P.cbeg[p] = s;
    if (s + 1 == nd || (uint32_t)(P.skey[s + 1] >> P.col_bits) != p) P.cend[p] = s + 1;
    P.at[P.sval[s]] = s;
}

// Descendants of a pattern of length d, once those of length d + 1 are known.
__device__ __forceinline__ void ord_desc(const OrdParams &P, uint32_t k, uint32_t d) {
    if (P.depth[k] != d) return;
    const uint32_t a = P.cbeg[k], b = P.cend[k];
    uint32_t sum = b - a;
    for (uint32_t s = a; s < b; ++s) sum += P.desc[P.sval[s]];
    P.desc[k] = sum;
}

// Place of a deep pattern of length d, once those of length d - 1 have theirs.
// (sdesc may wrap around 2^32: only differences below n are taken.)
__device__ __forceinline__ void ord_place(const OrdParams &P, uint32_t k, uint32_t d) {
    if (P.depth[k] != d) return;
    const uint32_t p = P.cpar[k], s = P.at[k], a = P.cbeg[p];
    const uint32_t r = p < P.base ? P.dbase[p] : P.reg[p];
    P.pos[k] = r + (s - a);
    P.reg[k] = r + (P.cend[p] - a) + (P.sdesc[s] - P.sdesc[a]);
}

// Deep patterns before database d's; final place of a pattern of database d.
__device__ __forceinline__ uint64_t ord_deep_before(const OrdParams &P, uint32_t d) {
    const uint64_t b = P.pat_base[d];
    return b < P.base ? P.dbase[b] : P.n - P.base;
}
__device__ __forceinline__ uint64_t ord_final(const OrdParams &P, uint32_t k, uint32_t d) {
    return k < P.base ? k + ord_deep_before(P, d) : P.pat_base[d + 1] + P.pos[k];
}

// Supports, lengths and parents (within their database) in final order.
__device__ __forceinline__ void ord_out(const OrdParams &P, uint32_t k) {
    if (k <= P.n_db) P.db_first[k] = k < P.n_db ? P.pat_base[k] + ord_deep_before(P, k) : P.n;
    if (k >= P.n) return;
    const uint32_t d = P.db ? P.db[k] : 0u;
    const uint64_t g = ord_final(P, k, d);
    const uint32_t p = k < P.base ? P.parent[k] : P.cpar[k];
    P.inv[g] = k;
    P.o_sup[g] = P.sup[k];
    P.o_depth[g] = P.depth[k];
    P.o_par[g] = p == ORD_NONE ? ORD_NONE
                               : (uint32_t)(ord_final(P, p, d) - (P.pat_base[d] + ord_deep_before(P, d)));
}

// The items of pattern g of the final order, columns ascending, at its offset;
// slot_first[g] = the first item slot of database g.
template <class Item>
__device__ __forceinline__ void ord_items(const OrdParams &P, uint32_t g, const uint64_t *off, Item *items,
                                          unsigned long long *slot_first) {
    if (g <= P.n_db) {
        const unsigned long long f = P.db_first[g];
        slot_first[g] = f < P.n ? off[f] : P.info[1];
    }
    if (g >= P.n) return;
    uint32_t v = P.inv[g];
    Item *o = items + off[g];
    for (uint32_t j = P.depth[v]; j-- > 0;) {
        const bool deep = v >= P.base;
        o[j] = (Item)(deep ? P.top[v] : P.item[v]);
        v = deep ? P.cpar[v] : P.parent[v];
    }
}

__global__ void k_ord_children(OrdParams P) {
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < P.n - P.base) ord_children(P, s);
}
__global__ void k_ord_desc(OrdParams P, uint32_t d) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < P.n) ord_desc(P, k, d);
}
__global__ void k_ord_gather(OrdParams P) {
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < P.n - P.base) P.sdesc[s] = P.desc[P.sval[s]];
}
__global__ void k_ord_place(OrdParams P, uint32_t d) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < P.n - P.base) ord_place(P, P.base + i, d);
}
__global__ void k_ord_out(OrdParams P) { ord_out(P, blockIdx.x * blockDim.x + threadIdx.x); }
template <class Item>
__global__ void k_ord_items(OrdParams P, const uint64_t *__restrict__ off, Item *__restrict__ items,
                            unsigned long long *__restrict__ slot_first) {
    ord_items(P, blockIdx.x * blockDim.x + threadIdx.x, off, items, slot_first);
}

// All of these steps, and the sums between them, in one CTA: for up to
// ORD_SMALL patterns, where two dozen launches cost more than their work
// (4,837 patterns: about 85 us of launches, 30 us in one).
constexpr uint32_t ORD_SMALL = 16384;

// Exclusive sum of n values read by get(i), put(i, sum); s_w holds 32 partial sums.
template <class Get, class Put>
__device__ __forceinline__ void ord_cta_sum(uint32_t n, uint64_t *s_w, Get get, Put put) {
    const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint64_t run = 0;
    for (uint32_t i0 = 0; i0 < n; i0 += blockDim.x) {
        const uint32_t i = i0 + threadIdx.x;
        const uint64_t v = i < n ? get(i) : 0;
        uint64_t incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t y = __shfl_up_sync(CPM_FULL, incl, o);
            if (lane >= (unsigned)o) incl += y;
        }
        if (lane == 31) s_w[wid] = incl;
        __syncthreads();
        uint64_t before = 0, tot = 0;
        for (unsigned w = 0; w < blockDim.x >> 5; ++w) {
            if (w < wid) before += s_w[w];
            tot += s_w[w];
        }
        if (i < n) put(i, run + before + incl - v);
        run += tot;
        __syncthreads();
    }
}

template <class Item>
__global__ void __launch_bounds__(1024) k_ord_tail(OrdParams P, uint32_t longest, uint64_t *off, Item *items,
                                                   unsigned long long *slot_first) {
    __shared__ uint64_t s_w[32];
    const uint32_t t = threadIdx.x, T = blockDim.x, nd = P.n - P.base;
    for (uint32_t s = t; s < nd; s += T) ord_children(P, s);
    __syncthreads();
    for (uint32_t d = longest - 1; nd && d >= 2; --d) {
        for (uint32_t k = t; k < P.n; k += T) ord_desc(P, k, d);
        __syncthreads();
    }
    ord_cta_sum(nd, s_w, [&](uint32_t s) { return P.desc[P.sval[s]]; },
                [&](uint32_t s, uint64_t v) { P.sdesc[s] = (uint32_t)v; });
    ord_cta_sum(P.base, s_w, [&](uint32_t k) { return P.desc[k]; },
                [&](uint32_t k, uint64_t v) { P.dbase[k] = (uint32_t)v; });
    __syncthreads();
    for (uint32_t d = 3; nd && d <= longest; ++d) {
        for (uint32_t i = t; i < nd; i += T) ord_place(P, P.base + i, d);
        __syncthreads();
    }
    for (uint32_t k = t; k < max(P.n, P.n_db + 1u); k += T) ord_out(P, k);
    __syncthreads();
    ord_cta_sum(P.n, s_w, [&](uint32_t g) { return (uint32_t)P.o_depth[g]; },
                [&](uint32_t g, uint64_t v) { off[g] = v; });
    __syncthreads();
    for (uint32_t g = t; g < max(P.n, P.n_db + 1u); g += T) ord_items(P, g, off, items, slot_first);
}

}  // namespace cpm
