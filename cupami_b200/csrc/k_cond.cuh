// Deep levels over conditional rows: sparse databases mined from the transactions' side.
//
// Reference: the same step as k_deep -- cuEclat._searchClass
// (cuEclat.py:211-245) with intersect_extensions (_bitsets.py:55-77): unit
// (F, p) needs the support of every later member q of frame F together with
// member p, keeps those that pass and recurses into them when two or more do.
//
// A frame here is a conditional database.  Row r of frame F (prefix P) is one
// transaction that holds P: the ascending indices (uint16) of the members of
// F it holds; next to the rows, every member has the list of its occurrences
// (position in the row array, elements after it in the row).  The supports of unit (F, p)
// come from walking, for each occurrence of p, the rest of its row: every
// element met is a later member, so every load ends in one count, and the
// work is the sum of the siblings' supports (P, p, q) -- not the siblings'
// tidsets, and not the whole transactions.  Survivors' rows become the child
// frame's rows (members renumbered 0 .. ns - 1), with two cuts that keep the
// search exact: a row with fewer than two survivors, and the occurrence of a
// row's last survivor, can meet no further pair.  A child frame of R kept
// rows with R below the threshold has no children at all.
//
// The top frame of a database is its rows of frequent indices (k_cond_top);
// its units build the classes of the pair level, whose supports the Gram
// already holds (or which k_cond_count itself counted).  Child frames whose bitsets are small (ns members of
// ceil(R / 128) 16-byte words each, at most bitset_work in all) are written as
// bitsets over the kept rows and mined by k_local, a warp per unit; larger
// ones stay rows.  Few do: below the classes of rare items everything is
// small, and frequent items have few members after them in the mining order.
//
// Units run level by level over the whole grid, a chunk of occurrences per
// CTA: a class can hold most of the transactions (one CTA took 50 ms over the
// class of an item held by 1.5 of 2 million), and every level has enough
// chunks or little work.  Counts go to shared memory, in up to 32 copies so
// that the lanes of a warp meet different banks.
//
// Capacity overflows set the error bits of k_deep, after which the host grows
// the buffers and reruns; nothing here waits.
//
// Measured (deep phase, k_local included; before: k_deep over tidsets in column
// order): 1M x 20k 347 -> 23.5 ms, 250k x 20k 37 -> 3.5 ms, 512 databases of 200
// items 15.2 -> 7.1 ms, planted 100k x 1,000 0.227 -> 0.143 ms.  Long tidsets over
// few items are left to k_deep, in order of support (cond_plan): a mine of 2.4M
// x 500 takes 4.3 ms in column order, 3.2 over rows and 1.5 so.
#pragma once
#include "k_batch.cuh"
#include "k_deep.cuh"
#include "k_local.cuh"

namespace cpm {

constexpr uint32_t COND_NONE = 0xffffffffu;   // a sibling that did not survive
constexpr int COND_BLOCK = 512;
constexpr uint32_t COND_COPY_WORDS = 8192;    // shared words for copies of the counters
constexpr uint32_t COND_CHUNK = 8192;         // occurrences per CTA and task (small searches: fewer)

struct CFrame {
    const uint16_t *idx;  // rows
    const uint2 *occ;     // occurrences, grouped by member: (position in idx, elements after it in its row)
    uint64_t mem_off;     // first member entry (top frames: global index of the first frequent row)
    uint32_t m;           // members
    uint32_t db;
    uint32_t root;        // as in DFrame
    uint32_t lg;          // log2 of the lanes that read a row together
    uint32_t top, pad;    // top 1: a database's top frame
    long long minsup;
};

// A unit.  Member q of a frame of rows has its occurrence
// list's start (high) and length (low half) in mem_bits[mem_off + q].
struct CBig {
    uint32_t fid, p, start, n;
    uint64_t pool;         // its counters, then its survivors' ranks (not for top frames)
    uint64_t mb, ab, idx_words, frame;
    uint32_t ns;           // survivors
    uint32_t next;         // next free row position (rows) or row number (bitsets)
    uint32_t rows;         // kept rows (rows)
    uint32_t form;         // 0 no child frame, 1 rows, 2 bitsets
};

// One level's units and their chunks (chunk c of the level is chunk
// chunk_part[c] of unit chunk_unit[c]).
struct CLevel {
    CBig *units;
    uint32_t *chunk_unit, *chunk_part;
    unsigned long long *n;  // [0] units, [1] chunks, [2] pool words
};

struct CondParams {
    DeepParams d;  // patterns, members, arena, state; d.frames and d.lq take the bitset frames
    CFrame *cframes;
    uint64_t cframes_cap;
    const DbDesc *dbs;
    uint32_t *cur;       // per member entry: cursor of its occurrence list while rows are written
    uint32_t *pool;      // the level's counters, then ranks
    uint32_t chunk;      // occurrences per CTA and task
    uint64_t units_cap, chunks_cap, pool_cap;
    CLevel now, next;    // the level being run, and the one it fills
    unsigned long long bitset_work;
};

// The 32 x 32 bit matrix with row l in lane l, transposed.
__device__ __forceinline__ uint32_t transpose32(uint32_t x, unsigned lane) {
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const int s = 16 >> k;
        const uint32_t m = s == 16 ? 0x0000ffffu : s == 8 ? 0x00ff00ffu : s == 4 ? 0x0f0f0f0fu : s == 2 ? 0x33333333u
                                                                                                       : 0x55555555u;
        const uint32_t y = __shfl_xor_sync(CPM_FULL, x, s);
        x = (lane & s) ? (x & ~m) | ((y >> s) & m) : (x & m) | ((y << s) & ~m);
    }
    return x;
}

// Top frames: the transpose of the frequent tidsets, in mining order.  A CTA
// takes 128 transactions of a database (group g; every tidset row gives it 16
// bytes) and each of its eight warps a contiguous share of the frequent items,
// 32 at a time, one per lane, transposed in registers.  WRITE = false: len[row]
// = items held, and part[] the items before each warp's share; true: the rows
// at idx[off[row] ..] and every occurrence at its item's cursor (the order
// within an item's list is arbitrary).  Rows are numbered 128 * group +
// transaction; a database's last group is padded with empty rows.
constexpr unsigned COND_TOP_WARPS = 8;
template <bool WRITE>
__global__ void __launch_bounds__(32 * COND_TOP_WARPS)
    k_cond_top(const DbDesc *__restrict__ dbs, uint32_t n_db, const uint64_t *__restrict__ group_base,
               uint32_t *__restrict__ len, uint16_t *__restrict__ part, const uint64_t *__restrict__ off,
               uint16_t *__restrict__ idx, uint32_t *__restrict__ cursor, uint2 *__restrict__ occ) {
    __shared__ uint32_t s_word[COND_TOP_WARPS][4][32], s_at[COND_TOP_WARPS][4][32];
    const uint64_t gg = blockIdx.x;
    const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t lo = 0, hi = n_db;  // last database with group_base <= gg
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (group_base[mid] <= gg) lo = mid; else hi = mid;
    }
    const DbDesc D = dbs[lo];
    const uint64_t g = gg - group_base[lo];
    const uint32_t blocks = (D.F + 31) / 32;
    const uint32_t fa = blocks * wid / COND_TOP_WARPS * 32, fb = min(D.F, blocks * (wid + 1) / COND_TOP_WARPS * 32);
    uint16_t *const my_part = part + (gg * COND_TOP_WARPS + wid) * 128;
    uint32_t n[4] = {0, 0, 0, 0};
    uint64_t at[4];
    if (WRITE)
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const uint32_t before = my_part[w * 32 + lane];
            at[w] = off[gg * 128 + w * 32 + lane] + before;
            n[w] = len[gg * 128 + w * 32 + lane] - before;  // elements from this share on
        }
    for (uint32_t f0 = fa; f0 < fb; f0 += 32) {
        const uint32_t f = f0 + lane;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (f < fb) v = __ldg(reinterpret_cast<const uint4 *>(D.bits + (uint64_t)D.freq[D.ord[f]] * D.stride) + g);
        const uint32_t x[4] = {v.x, v.y, v.z, v.w};
        if (WRITE) {
            const uint32_t c = __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
            uint32_t a = c ? atomicAdd(cursor + D.row_base + f, c) : 0u;
            __syncwarp();
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                s_word[wid][w][lane] = x[w];
                s_at[wid][w][lane] = a;
                a += __popc(x[w]);
            }
            __syncwarp();
        }
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            uint32_t b = transpose32(x[w], lane);
            if (!WRITE) {
                n[w] += __popc(b);
            } else {
                for (; b; b &= b - 1) {
                    const uint32_t i = __ffs(b) - 1;
                    idx[at[w]] = (uint16_t)(f0 + i);
                    const uint32_t o = s_at[wid][w][i] + __popc(s_word[wid][w][i] & ((1u << lane) - 1u));
                    occ[o] = make_uint2((uint32_t)at[w], --n[w]);
                    ++at[w];
                }
            }
        }
    }
    if (!WRITE) {
#pragma unroll
        for (int w = 0; w < 4; ++w) s_word[wid][w][lane] = n[w];
        __syncthreads();
        if (wid < 4) {
            uint32_t run = 0;
            for (unsigned k = 0; k < COND_TOP_WARPS; ++k) {
                part[(gg * COND_TOP_WARPS + k) * 128 + wid * 32 + lane] = (uint16_t)run;
                run += s_word[k][wid][lane];
            }
            len[gg * 128 + wid * 32 + lane] = run;
        }
    }
}

// ---- rows read by groups of lanes ----
// 1 << lg lanes take a row together, 16 bytes (eight elements) each per step,
// so that a row of up to 8 << lg elements is one coalesced load, and 32 >> lg
// rows go side by side in a warp.

__device__ __forceinline__ uint32_t cond_elem(const uint4 &v, int u) {
    const uint32_t w = u < 2 ? v.x : u < 4 ? v.y : u < 6 ? v.z : v.w;
    return (u & 1) ? w >> 16 : w & 0xffffu;
}

// log2 of the lanes for rows of this many elements: walks start at a random
// element, so half of a row is left on average.
__host__ __device__ __forceinline__ uint32_t cond_group_lg(unsigned long long elems, unsigned long long rows) {
    const unsigned long long avg = rows ? elems / rows : 0;
    return avg <= 10 ? 0u : avg <= 20 ? 1u : avg <= 40 ? 2u : 3u;
}

// The elements after an occurrence, as a lane of its group sees them.
struct CRow {
    const uint4 *w;  // this lane's next 16 bytes
    uint4 v;         // the first of them (loaded where the row reaches them)
    uint32_t skip;   // elements of v before the row's
    int left;        // elements from v's first to the row's end; none left: <= 0
    int turn;        // of the whole group: elements after this step
};

// f(v, valid) per step: bit u of valid marks element u of this lane's v as one
// of its row.  Every lane of the warp calls f the same number of times.
template <class F>
__device__ __forceinline__ void cond_steps(CRow r, bool act, unsigned lg, F f) {
    uint32_t cut = 0xffu << r.skip;
    if (!act) r.left = r.turn = 0;
    for (;;) {
        f(r.v, r.left > 0 ? (0xffu >> (8 - min(r.left, 8))) & cut : 0u);
        if (!__any_sync(CPM_FULL, r.turn > 0)) break;
        cut = 0xffu;
        r.left -= 8 << lg;
        r.turn -= 8 << lg;
        r.w += 1u << lg;
        if (r.left > 0) r.v = *r.w;
    }
}

// body(act, o, row) for the occurrences o = src[0, n), 32 >> lg per warp and
// turn, `warp` of `warps` warps; the next turn's occurrences and first words
// are loaded before the body runs.
template <class Body>
__device__ __forceinline__ void cond_rows(const uint16_t *idx, const uint2 *src, uint32_t n, unsigned lg,
                                          uint32_t warp, uint32_t warps, unsigned lane, Body body) {
    const uint32_t per = 32u >> lg, stride = warps * per, gj = lane >> lg;
    const int gl = (int)(lane & ((1u << lg) - 1u));
    uint32_t j0 = warp * per;
    auto first = [&](const uint2 &o) {
        CRow r;
        const unsigned long long a = reinterpret_cast<unsigned long long>(idx + (uint64_t)o.x + 1);
        const uint32_t s = (uint32_t)(a & 15ull) >> 1;
        r.w = reinterpret_cast<const uint4 *>(a & ~15ull) + gl;
        r.skip = gl ? 0u : s;
        r.left = o.y ? (int)(o.y + s) - 8 * gl : 0;
        r.turn = o.y ? (int)(o.y + s) - (8 << lg) : 0;
        if (r.left > 0) r.v = *r.w;
        return r;
    };
    const uint2 none = make_uint2(0, 0);
    uint2 o = j0 + gj < n ? src[j0 + gj] : none;
    uint2 o1 = j0 + stride + gj < n ? src[j0 + stride + gj] : none;
    CRow r = first(o);
    for (; j0 < n; j0 += stride) {
        const uint32_t jn = j0 + stride + gj;
        const CRow r1 = first(o1);
        const uint2 o2 = jn + stride < n ? src[jn + stride] : none;
        body(j0 + gj < n, o, r);
        o = o1;
        r = r1;
        o1 = o2;
    }
}

// ---- the walks of a unit ----

// Supports: sm[((x - p1) << lc) + copy] counts the elements x met.
__device__ __forceinline__ void cond_count(const uint16_t *idx, const uint2 *occ, uint32_t n, unsigned lg,
                                           uint32_t p1, uint32_t *sm, unsigned lc) {
    const unsigned lane = threadIdx.x & 31;
    uint32_t *const mine = sm + (lane & ((1u << lc) - 1u)) - (p1 << lc);
    cond_rows(idx, occ, n, lg, threadIdx.x >> 5, blockDim.x >> 5, lane, [&](bool act, const uint2 &, const CRow &row) {
        cond_steps(row, act, lg, [&](const uint4 &x, uint32_t valid) {
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if ((valid >> u) & 1u) atomicAdd(mine + (cond_elem(x, u) << lc), 1u);
        });
    });
}

// The survivors among the valid elements of x (map[x - p1] != COND_NONE).
__device__ __forceinline__ uint32_t cond_alive(const uint4 &x, uint32_t valid, uint32_t p1, const uint32_t *map) {
    uint32_t m = 0;
#pragma unroll
    for (int u = 0; u < 8; ++u)
        if ((valid >> u) & 1u) m |= map[cond_elem(x, u) - p1] != COND_NONE ? 1u << u : 0u;
    return m;
}

// Rows in turn: go(kept, o, c) with the row's survivors c (on every lane of its
// group; kept: two or more), then, where go says so (the same on the whole
// warp), each(r, i) for the kept rows' survivors, the i-th of its row having rank r.
template <class Go, class Each>
__device__ __forceinline__ void cond_kept(const uint16_t *idx, const uint2 *src, uint32_t n, unsigned lg, uint32_t p1,
                                          const uint32_t *map, Go go, Each each) {
    const unsigned lane = threadIdx.x & 31, G = 1u << lg, gl = lane & (G - 1u);
    cond_rows(idx, src, n, lg, threadIdx.x >> 5, blockDim.x >> 5, lane, [&](bool act, const uint2 &o, const CRow &row) {
        uint32_t c = 0, first = 0;
        bool at0 = true;
        cond_steps(row, act, lg, [&](const uint4 &x, uint32_t valid) {
            const uint32_t m = cond_alive(x, valid, p1, map);
            if (at0) first = m;  // kept for the second pass
            at0 = false;
            c += __popc(m);
        });
        c = group_sum(c, G);
        const bool kept = act && c >= 2u;
        if (!go(kept, o, c)) return;
        uint32_t i = 0;
        at0 = true;
        cond_steps(row, kept, lg, [&](const uint4 &x, uint32_t valid) {
            uint32_t m = first;
            if (!at0) m = cond_alive(x, valid, p1, map);
            if (!kept) m = 0;
            at0 = false;
            const uint32_t k = __popc(m);
            uint32_t before = k;
            for (unsigned s = 1; s < G; s <<= 1) {
                const uint32_t y = __shfl_up_sync(CPM_FULL, before, s);
                if (gl >= s) before += y;
            }
            const uint32_t step = __shfl_sync(CPM_FULL, before, lane | (G - 1u));
            uint32_t at = i + before - k;
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if ((m >> u) & 1u) each(map[cond_elem(x, u) - p1], at++);
            i += step;
        });
    });
}

// Kept rows written as rows: reserve(total) gives a warp that many positions
// of o_idx, cursor(r) the next slot of survivor r's occurrence list.
template <class Reserve, class Cursor>
__device__ __forceinline__ void cond_write_rows(const uint16_t *idx, const uint2 *src, uint32_t n, unsigned lg,
                                                uint32_t p1, const uint32_t *map, uint16_t *o_idx, uint2 *o_occ,
                                                Reserve reserve, Cursor cursor) {
    const unsigned lane = threadIdx.x & 31, G = 1u << lg;
    uint32_t pos = 0, len = 0;
    cond_kept(idx, src, n, lg, p1, map,
              [&](bool kept, const uint2 &, uint32_t c) {
                  len = c;
                  const uint32_t need = kept && (lane & (G - 1u)) == 0 ? c : 0u;
                  uint32_t incl = need;
#pragma unroll
                  for (int o = 1; o < 32; o <<= 1) {
                      const uint32_t y = __shfl_up_sync(CPM_FULL, incl, o);
                      if (lane >= (unsigned)o) incl += y;
                  }
                  const uint32_t total = __shfl_sync(CPM_FULL, incl, 31);
                  if (!total) return false;
                  uint32_t base = 0;
                  if (lane == 0) base = reserve(total);
                  base = __shfl_sync(CPM_FULL, base, 0);
                  pos = __shfl_sync(CPM_FULL, base + incl - need, lane & ~(G - 1u));
                  return true;
              },
              [&](uint32_t r, uint32_t i) {
                  o_idx[pos + i] = (uint16_t)r;
                  // (the last survivor of a row meets nothing further)
                  if (i + 1u != len) o_occ[cursor(r)] = make_uint2(pos + i, len - 1u - i);
              });
}

// Rank of this thread's item among those of the CTA's chunk that keep theirs;
// *total the chunk's count.  s_w holds a count per warp.
__device__ __forceinline__ uint32_t cond_rank(bool keep, uint32_t *s_w, uint32_t *total) {
    const unsigned lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned bal = __ballot_sync(CPM_FULL, keep);
    if (lane == 0) s_w[wid] = __popc(bal);
    __syncthreads();
    uint32_t before = 0, tot = 0;
#pragma unroll
    for (unsigned w = 0; w < COND_BLOCK / 32; ++w) {
        const uint32_t c = s_w[w];
        before += w < wid ? c : 0u;
        tot += c;
    }
    __syncthreads();
    *total = tot;
    return before + __popc(bal & ((1u << lane) - 1u));
}

// Survivors of a unit, in member order: their patterns and member entries, and
// over the supports in sup[0, cnt) their ranks; on_rank(r, s) per survivor.
template <class OnRank>
__device__ __forceinline__ void cond_survivors(const DeepParams &D, const CFrame &f, uint32_t p1, uint32_t cnt,
                                               uint32_t *sup, uint32_t parent_pat, unsigned long long pid0,
                                               unsigned long long mb, uint32_t *s_w, OnRank on_rank) {
    uint32_t run = 0;
    for (uint32_t q0 = 0; q0 < cnt; q0 += COND_BLOCK) {
        const uint32_t q = q0 + threadIdx.x;
        const uint32_t s = q < cnt ? sup[q] : 0u;
        const bool keep = q < cnt && (long long)s >= f.minsup;
        uint32_t tot;
        const uint32_t r = run + cond_rank(keep, s_w, &tot);
        if (q < cnt) sup[q] = keep ? r : COND_NONE;
        if (keep) {
            if (!f.top) {
                const unsigned long long pid = pid0 + r;
                const uint32_t item = D.mem_item[f.mem_off + p1 + q];
                D.pat_parent[pid] = parent_pat;
                D.pat_item[pid] = item;
                D.pat_sup[pid] = s;
                if (D.pat_db) D.pat_db[pid] = f.db;
                D.mem_pat[mb + r] = (uint32_t)pid;
                D.mem_item[mb + r] = item;
            }
            on_rank(r, s);
        }
        run += tot;
    }
}

// Whether the frame of ns members over at most R rows is written as bitsets.
__host__ __device__ __forceinline__ bool cond_bits(uint32_t ns, uint32_t R, unsigned long long bitset_work) {
    const uint32_t W2 = (R + 127u) / 128u;
    return R <= LOCAL_MAX_BITS && (unsigned long long)ns * (W2 ? W2 : 1u) <= bitset_work;
}

// Form and size (64-bit words) of the child frame of ns survivors, at most R
// rows of K elements and `listed` occurrence slots.
struct CForm {
    bool bits;
    uint32_t W2;
    unsigned long long idx_words, words;
};
__device__ __forceinline__ CForm cond_form(uint32_t ns, uint32_t R, unsigned long long K, unsigned long long listed,
                                           unsigned long long bitset_work) {
    CForm c;
    c.W2 = max(1u, (R + 127u) / 128u);
    c.bits = cond_bits(ns, R, bitset_work);
    c.idx_words = (K * 2 + 15) / 16 * 2 + 2;  // (rows are read in aligned 16-byte words)
    c.words = c.bits ? 2ull * c.W2 * ns : (c.idx_words + listed + 15) / 16 * 16;
    return c;
}

__device__ __forceinline__ void cond_frame(const CondParams &P, const CFrame &f, bool bits, uint64_t fid, uint64_t mb,
                                           uint32_t ns, uint64_t ab, uint64_t idx_words, uint32_t W2, uint32_t R,
                                           unsigned long long K) {  // bits: R rows of the 128 * W2 that a member has room for
    if (bits) {
        DFrame c;
        c.mask = nullptr;
        c.mem_off = mb;
        c.m = ns;
        c.root = f.root;
        c.stride = 2u * W2;
        c.db = f.db;
        c.minsup = f.minsup;
        c.bits = P.d.arena + ab;
        c.used = max(1u, (R + 127u) / 128u);
        P.d.frames[fid] = c;
    } else {
        CFrame c;
        c.idx = reinterpret_cast<const uint16_t *>(P.d.arena + ab);
        c.occ = reinterpret_cast<const uint2 *>(P.d.arena + ab + idx_words);
        c.mem_off = mb;
        c.m = ns;
        c.db = f.db;
        c.root = f.root;
        c.lg = cond_group_lg(K, R);
        c.top = c.pad = 0;
        c.minsup = f.minsup;
        P.cframes[fid] = c;
    }
}

// Copies of the counters of cnt siblings for a walk of n occurrences: as many
// as shared memory and the walk's length pay for (they are zeroed and summed).
__device__ __forceinline__ unsigned cond_copies_lg(uint32_t cnt, uint32_t n) {
    unsigned lc = 0;
    while (lc < 5 && ((uint64_t)cnt << (lc + 1)) <= COND_COPY_WORDS && ((uint64_t)cnt << (lc + 1)) <= 2ull * n) ++lc;
    return lc;
}

__device__ __forceinline__ uint32_t cond_copies_sum(const uint32_t *sm, uint32_t q, unsigned lc) {
    uint32_t s = 0;
    for (uint32_t c = 0; c < (1u << lc); ++c) s += sm[(q << lc) + ((c + q) & ((1u << lc) - 1u))];
    return s;
}

// ---- units, level by level ----
// k_cond_count (chunks), k_cond_emit (units), k_cond_write (chunks),
// k_cond_publish (units); the level of the classes has its supports from
// the Gram.  What one of them writes the next reads: the kernels' ends order
// them.  A child frame is sized by bounds -- its unit's occurrences and its
// survivors' supports -- and filled by the rows kept, in one walk per chunk to
// count what the chunk writes and one to write it at places reserved by one
// atomic per chunk and survivor.  (With an atomic per element on each
// survivor's cursor the write took 3 to 4 times the count walk: 28 against
// 6.4 ms on a level of 6,720 units and 285 M occurrences.)

// The survivors' ranks of unit u: from the pool, or for a class from its member table.
__device__ __forceinline__ void cond_map(const CondParams &P, const CBig &u, const CFrame &f, uint32_t p1,
                                         uint32_t cnt, uint32_t *sm) {
    if (!f.top) {
        for (uint32_t q = threadIdx.x; q < cnt; q += COND_BLOCK) sm[q] = P.pool[u.pool + q];
        return;
    }
    const uint32_t *crank = P.dbs[f.db].crank;
    for (uint32_t q = threadIdx.x; q < cnt; q += COND_BLOCK) sm[q] = COND_NONE;
    __syncthreads();
    for (uint32_t r = threadIdx.x; r < u.ns; r += COND_BLOCK) sm[crank[P.d.mem_item[u.mb + r]] - p1] = r;
}

// Supports of every unit's later members, into the pool -- or, for units of a
// top frame, the pairs of their item, into the Gram matrix (zeroed): sparse
// databases count their pairs this way instead of multiplying tidsets
// (1M x 20k, 4,612 frequent items: pair level 3.0 ms, 1.1 of it the rows that the
// deep levels need anyway, against 13.5 ms on the tensor cores).
__global__ void __launch_bounds__(COND_BLOCK, 3) k_cond_count(CondParams P) {
    extern __shared__ uint32_t sm[];
    const unsigned long long chunks = min(P.now.n[1], (unsigned long long)P.chunks_cap);
    for (unsigned long long t = blockIdx.x; t < chunks; t += gridDim.x) {
        const CBig &u = P.now.units[P.now.chunk_unit[t]];
        const CFrame f = P.cframes[u.fid];
        const uint32_t p1 = u.p + 1, cnt = f.m - p1;
        const uint32_t a = P.now.chunk_part[t] * P.chunk, n = min(u.n - a, P.chunk);
        const unsigned lc = cond_copies_lg(cnt, n);
        for (uint32_t i = threadIdx.x; i < cnt << lc; i += COND_BLOCK) sm[i] = 0u;
        __syncthreads();
        cond_count(f.idx, f.occ + u.start + a, n, f.lg, p1, sm, lc);
        __syncthreads();
        if (f.top) {
            const DbDesc &d = P.dbs[f.db];
            const uint64_t i = d.ord[u.p];
            for (uint32_t q = threadIdx.x; q < cnt; q += COND_BLOCK) {
                const uint32_t s = cond_copies_sum(sm, q, lc);
                const uint64_t j = d.ord[p1 + q];
                if (s) atomicAdd(d.C + min(i, j) * d.F + max(i, j), s);
            }
        } else {
            for (uint32_t q = threadIdx.x; q < cnt; q += COND_BLOCK) {
                const uint32_t s = cond_copies_sum(sm, q, lc);
                if (s) atomicAdd(P.pool + u.pool + q, s);
            }
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(COND_BLOCK) k_cond_emit(CondParams P) {
    __shared__ unsigned long long s_pid0, s_mb, s_ab, s_fid;
    __shared__ int s_ok;
    __shared__ uint32_t s_w[32];
    __shared__ uint64_t s_w64[32];
    const DeepParams &D = P.d;
    DeepState *st = D.st;
    const unsigned tid = threadIdx.x;
    const unsigned long long units = min(P.now.n[0], (unsigned long long)P.units_cap);
    for (unsigned long long i = blockIdx.x; i < units; i += gridDim.x) {
        CBig &u = P.now.units[i];
        const CFrame f = P.cframes[u.fid];
        const uint32_t p1 = u.p + 1, cnt = f.m - p1;
        uint32_t ns = u.ns;
        uint64_t mb = u.mb;
        if (!f.top) {
            uint32_t *sup = P.pool + u.pool;
            unsigned long long visits = 0;
            ns = 0;
            for (uint32_t q0 = 0; q0 < cnt; q0 += COND_BLOCK) {
                const uint32_t q = q0 + tid;
                const uint32_t s = q < cnt ? sup[q] : 0u;
                visits += s;
                ns += __syncthreads_count(q < cnt && (long long)s >= f.minsup);
            }
            visits = warp_sum_u64(visits);
            if ((tid & 31) == 0 && visits) atomicAdd(&st->bytes_alg, 2ull * visits);
            if (tid == 0) {
                s_ok = ns > 0;
                s_mb = s_pid0 = 0;
                if (ns) {
                    s_pid0 = atomicAdd(&st->n_patterns, (unsigned long long)ns);
                    s_mb = atomicAdd(&st->n_members, (unsigned long long)ns);
                    if (s_pid0 + ns > D.pat_cap) { deep_fail(st, DEEP_ERR_PATTERNS); s_ok = 0; }
                    if (s_mb + ns > D.members_cap) { deep_fail(st, DEEP_ERR_MEMBERS); s_ok = 0; }
                }
                u.ns = s_ok ? ns : 0u;
                u.mb = s_mb;
                atomicAdd(&st->intersections, (unsigned long long)cnt);
                atomicAdd(&st->bytes_alg, 8ull * u.n);
                atomicAdd(&st->work_items, 1ull);
                atomicAdd(&st->h_units, 1ull);
                atomicAdd(&st->survivors, (unsigned long long)ns);
            }
            __syncthreads();
            const bool ok = s_ok;
            mb = s_mb;
            if (ok)
                cond_survivors(D, f, p1, cnt, sup, D.mem_pat[f.mem_off + u.p], s_pid0, mb, s_w,
                               [](uint32_t, uint32_t) {});
            __syncthreads();  // the patterns and members are written (and s_ok read)
            if (!ok) ns = 0;
        }
        if (ns < 2) continue;  // u.form stays 0
        // The child frame: room for every occurrence's row, and a list of each survivor's support.
        uint64_t S = 0;
        for (uint32_t r0 = 0; r0 < ns; r0 += COND_BLOCK) {
            const uint32_t r = r0 + tid;
            uint64_t tot = 0;
            const uint64_t s = S + block_excl_scan_u64(r < ns ? D.pat_sup[D.mem_pat[mb + r]] : 0u, s_w64, &tot);
            if (r < ns) {
                P.cur[mb + r] = (uint32_t)s;
                D.mem_bits[mb + r] = reinterpret_cast<const uint64_t *>((unsigned long long)s << 32);
            }
            S += tot;
        }
        const CForm form = cond_form(ns, u.n, S, S, P.bitset_work);
        if (tid == 0) {
            s_ab = atomicAdd(&st->arena_next, form.words);
            s_fid = atomicAdd(form.bits ? &st->n_frames : &st->n_cframes, 1ull);
            s_ok = 0;
            if (s_ab + form.words > D.arena_words || S > 0xffffffffull) deep_fail(st, DEEP_ERR_ARENA);
            else if (s_fid >= (form.bits ? D.frames_cap : P.cframes_cap)) deep_fail(st, DEEP_ERR_FRAMES);
            else s_ok = 1;
            if (s_ok) {
                u.form = form.bits ? 2u : 1u;
                u.ab = s_ab;
                u.idx_words = form.idx_words;
                u.frame = s_fid;
            }
        }
        __syncthreads();
        if (s_ok && form.bits)
            for (uint64_t k = tid; k < form.words; k += COND_BLOCK) D.arena[s_ab + k] = 0ull;
        __syncthreads();
    }
}

// Bound by instruction issue: 74% of the issue slots busy at the classes of 250k
// x 20k (0.85 ms; L2 29%, DRAM 2% of peak), 63% of the warps active.
__global__ void __launch_bounds__(COND_BLOCK, 3) k_cond_write(CondParams P) {
    extern __shared__ uint32_t sm[];
    __shared__ uint32_t s_len, s_rows;
    const DeepParams &D = P.d;
    const unsigned tid = threadIdx.x, lane = tid & 31;
    const unsigned long long chunks = min(P.now.n[1], (unsigned long long)P.chunks_cap);
    for (unsigned long long t = blockIdx.x; t < chunks; t += gridDim.x) {
        CBig &u = P.now.units[P.now.chunk_unit[t]];
        if (!u.form) continue;  // the same for the whole CTA
        const CFrame f = P.cframes[u.fid];
        const uint32_t p1 = u.p + 1, cnt = f.m - p1;
        const uint32_t a = P.now.chunk_part[t] * P.chunk, n = min(u.n - a, P.chunk);
        cond_map(P, u, f, p1, cnt, sm);
        const uint2 *occ = f.occ + u.start + a;
        const unsigned G = 1u << f.lg;
        const bool leader = (lane & (G - 1u)) == 0;
        if (u.form == 1) {
            uint32_t *const cur = sm + cnt;
            const uint32_t ns = u.ns;
            for (uint32_t r = tid; r < ns; r += COND_BLOCK) cur[r] = 0u;
            if (tid == 0) s_len = s_rows = 0;
            __syncthreads();
            // What this chunk writes: row elements, rows, occurrences of each survivor.
            uint32_t len = 0, rows = 0, c_row = 0;
            cond_kept(
                f.idx, occ, n, f.lg, p1, sm,
                [&](bool kept, const uint2 &, uint32_t c) {
                    c_row = c;
                    if (kept && leader) {
                        len += c;
                        ++rows;
                    }
                    return __any_sync(CPM_FULL, kept) != 0;
                },
                [&](uint32_t r, uint32_t i) {
                    if (i + 1u != c_row) atomicAdd(cur + r, 1u);
                });
            len = warp_sum_u32(len);
            rows = warp_sum_u32(rows);
            if (lane == 0 && rows) {
                atomicAdd(&s_len, len);
                atomicAdd(&s_rows, rows);
            }
            __syncthreads();
            for (uint32_t r = tid; r < ns; r += COND_BLOCK) {
                const uint32_t c = cur[r];
                if (c) cur[r] = atomicAdd(P.cur + u.mb + r, c);
            }
            if (tid == 0 && s_rows) {
                atomicAdd(&u.rows, s_rows);
                s_len = atomicAdd(&u.next, s_len);  // now the chunk's next position
            }
            __syncthreads();
            cond_write_rows(f.idx, occ, n, f.lg, p1, sm, reinterpret_cast<uint16_t *>(D.arena + u.ab),
                            reinterpret_cast<uint2 *>(D.arena + u.ab + u.idx_words),
                            [&](uint32_t k) { return atomicAdd(&s_len, k); },
                            [&](uint32_t r) { return atomicAdd(cur + r, 1u); });
        } else {
            __syncthreads();
            // Bitsets: the kept rows take numbers as they come, every survivor's bit an atomic OR.
            uint32_t *const blk = reinterpret_cast<uint32_t *>(D.arena + u.ab);
            const uint32_t nw32 = 4u * max(1u, (u.n + 127u) / 128u);
            uint32_t row = 0;
            cond_kept(
                f.idx, occ, n, f.lg, p1, sm,
                [&](bool kept, const uint2 &, uint32_t) {
                    const unsigned bal = __ballot_sync(CPM_FULL, kept && leader);
                    if (!bal) return false;
                    uint32_t base = 0;
                    if (lane == 0) base = atomicAdd(&u.next, (uint32_t)__popc(bal));
                    base = __shfl_sync(CPM_FULL, base, 0);
                    row = base + __popc(bal & ((1u << (lane & ~(G - 1u))) - 1u));
                    return true;
                },
                [&](uint32_t r, uint32_t) {
                    atomicOr(blk + (uint64_t)r * nw32 + (row >> 5), 1u << (row & 31u));
                });
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(COND_BLOCK) k_cond_publish(CondParams P) {
    __shared__ unsigned long long s_qb;
    __shared__ uint32_t s_w[32];
    const DeepParams &D = P.d;
    DeepState *st = D.st;
    const unsigned tid = threadIdx.x;
    const unsigned long long units = min(P.now.n[0], (unsigned long long)P.units_cap);
    for (unsigned long long i = blockIdx.x; i < units; i += gridDim.x) {
        const CBig &u = P.now.units[i];
        if (!u.form) continue;
        const CFrame f = P.cframes[u.fid];
        const uint32_t ns = u.ns;
        const bool bits = u.form == 2;
        const uint32_t R = bits ? u.next : u.rows;
        if ((long long)R < f.minsup) continue;  // no two survivors meet often enough
        if (tid == 0) {
            cond_frame(P, f, bits, u.frame, u.mb, ns, u.ab, u.idx_words, max(1u, (u.n + 127u) / 128u), R, u.next);
            // What the child frame holds: its bitsets, or row elements and an occurrence for each but a row's last.
            atomicAdd(&st->bytes_alg, bits ? 16ull * ns * max(1u, (R + 127u) / 128u) : 2ull * u.next + 8ull * (u.next - R));
        }
        // Chunks of members: occurrences, then a unit for each that has enough for a child.
        for (uint32_t r0 = 0; r0 < ns; r0 += COND_BLOCK) {
            const uint32_t r = r0 + tid;
            uint32_t c = 0, start = 0;
            if (r < ns && bits) {
                c = D.pat_sup[D.mem_pat[u.mb + r]];
            } else if (r < ns) {
                const unsigned long long s = reinterpret_cast<unsigned long long>(D.mem_bits[u.mb + r]);
                start = (uint32_t)(s >> 32);
                c = P.cur[u.mb + r] - start;
                D.mem_bits[u.mb + r] = reinterpret_cast<const uint64_t *>(s | c);
            }
            bool push = r + 1 < ns && (long long)c >= f.minsup;
            if (push && !bits) {
                const uint32_t cnt = ns - r - 1, parts = (c + P.chunk - 1) / P.chunk;
                const unsigned long long k = atomicAdd(P.next.n, 1ull), pc = atomicAdd(P.next.n + 1, (unsigned long long)parts),
                                         pw = atomicAdd(P.next.n + 2, (unsigned long long)cnt);
                if (k >= P.units_cap || pc + parts > P.chunks_cap || pw + cnt > P.pool_cap) {
                    deep_fail(st, DEEP_ERR_LEVEL);
                } else {
                    CBig b;
                    b.fid = (uint32_t)u.frame;
                    b.p = r;
                    b.start = start;
                    b.n = c;
                    b.pool = pw;
                    b.mb = b.ab = b.idx_words = b.frame = 0;
                    b.ns = b.next = b.rows = b.form = 0;
                    P.next.units[k] = b;
                    for (uint32_t x = 0; x < parts; ++x) {
                        P.next.chunk_unit[pc + x] = (uint32_t)k;
                        P.next.chunk_part[pc + x] = x;
                    }
                }
            }
            if (!bits) continue;
            uint32_t tot;
            const uint32_t k = cond_rank(push, s_w, &tot);
            if (tid == 0) {
                s_qb = atomicAdd(&st->lq_tail, (unsigned long long)tot);
                if (s_qb + tot > D.lq_cap) {
                    deep_fail(st, DEEP_ERR_QUEUE);
                    s_qb = ~0ull;
                } else {
                    atomicAdd(&st->lq_pending, (unsigned long long)tot);
                }
            }
            __syncthreads();
            if (push && s_qb != ~0ull) D.lq[s_qb + k] = ((unsigned long long)u.frame << 32) | r;
            __syncthreads();
        }
    }
}

}  // namespace cpm
