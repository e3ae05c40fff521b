// Projected deep levels: a persistent kernel with one warp per unit.
//
// Reference: the same step as k_deep -- cuEclat._searchClass
// (cuEclat.py:211-245) with intersect_extensions (_bitsets.py:55-77): unit
// (F, p) intersects member p of frame F with every later member, keeps the
// children whose support reaches the threshold and recurses into them when
// two or more pass.
//
// k_deep hands over every frame whose prefix held at most LOCAL_MAX_BITS
// transactions, with its members written as bitsets of that many bits,
// numbered by rank within the prefix (k_deep.cuh, build_rank_dir).  A
// descendant of such a frame only loses transactions, so it keeps the same
// numbering and size: every tidset of the subtree is at most 8 KB, the
// members of a frame lie side by side in one arena block (member q at bits +
// q * stride), and no unit needs more.  One warp runs a unit without a block
// barrier.
//
// A unit: the prefix stays in registers, the later members are streamed, G
// lanes per member (G the power of two covering a tidset, up to 32), several
// members in flight; AND, popcount and a group sum give each support, and a
// survivor's child tidset is written from the registers that counted it, at
// the end of the warp's own chunk of the arena.  A child frame is then mined
// by the same warp, depth first, from a stack in shared memory, and its chunk
// space is taken back when it is done (one of two members, half of all
// frames, is counted on the spot): most tidsets live in L2 for a few
// microseconds and never meet the queue or DRAM.  While fewer units are
// queued or running than keep the grid busy, child frames and what is left on
// the stack go to the queue instead, for any warp.
//
// What bounds it: the latency of L2 and DRAM under load (250k x 20k: long
// scoreboard the first stall, 41% of the issue slots busy, L2 34% and DRAM 22%
// of peak, all 16 warps per SM that the registers allow).  More warps lose
// more to each other's evictions than they hide: 1M x 20,000 sparse rows
// (3.2M units, tidsets of 2.7 KB on average) take 7.5 ms with 16 warps per SM
// (128 registers), 8.8 with 12, 8.6 with 20, 9.9 with 24 and 11.5 with 32;
// prefixes in shared memory, which leave L1 less room for loads in flight,
// 8.8 at best.  One queued unit per claim, as before, read each member twice,
// wrote every child to DRAM and read it back: 13.6 ms.  250,000 x 20,000:
// 3.9 -> 1.95 ms; 512 databases 0.76 -> 0.68.
//
// Where the arena has no room for chunks or a unit has more later members
// than the survivor list holds, the unit is counted first and written by a
// second pass into a block of exactly its survivors.
//
// Waits are bounded by spin_limit, and capacity overflows set the same error
// bits as k_deep, after which the host reruns.
#pragma once
#include "k_deep.cuh"

namespace cpm {

// Largest projected prefix, in transactions: ranks (and the rank directory
// of k_deep) are 16-bit, and a tidset is at most 511 16-byte words.
constexpr uint32_t LOCAL_MAX_BITS = 65536 - 128;
constexpr uint32_t LOCAL_BLOCK = 128;
constexpr uint32_t LOCAL_WARPS = LOCAL_BLOCK / 32;
constexpr uint32_t LOCAL_LIST = 128;  // survivors a warp holds before it writes their records
constexpr uint32_t LOCAL_DEPTH = 24;  // frames on a warp's stack; deeper ones are queued

// One frame being mined: members' tidsets from base, entries from mem, next unit p.
struct LocalLevel {
    const ulonglong2 *base;
    unsigned long long mem;
    uint32_t m, p;
};

// A warp's state in shared memory.
struct LocalWarp {
    uint2 list[LOCAL_LIST];  // survivors: later member, support
    LocalLevel lv[LOCAL_DEPTH];
    // The chunk: arena words [low, end), used below at; nothing below floor is taken back.
    unsigned long long low, at, end, floor;
    long long minsup;
    unsigned long long pid0, mb, items;  // the unit's first pattern id and member entry, its later members' entries
    uint32_t w2, pitch, root, db;  // tidsets: w2 16-byte words (pitch apart in the claimed frame)
    unsigned long long inter, bytes, units, surv, frames;  // statistics
};

constexpr size_t LOCAL_SMEM = sizeof(LocalWarp) * LOCAL_WARPS;

// Sum over an aligned group of G lanes (G a power of two, the same on every lane).
__device__ __forceinline__ uint32_t group_sum(uint32_t c, uint32_t G) {
    for (uint32_t o = G >> 1; o; o >>= 1) c += __shfl_xor_sync(CPM_FULL, c, o);
    return c;
}

// Lane 0 claims the next projected unit: a ticket, then a bounded wait for
// its queue entry, or until no projected unit is queued or running, or an
// error.  Returns 0 with *item set, or 1 to stop.
__device__ int local_claim(const DeepParams &P, unsigned long long *item) {
    DeepState *st = P.st;
    const unsigned long long h = atomicAdd(&st->lq_head, 1ull);
    unsigned backoff = 32;
    for (unsigned long long it = 0; it < P.spin_limit; ++it) {
        if (h < P.lq_cap) {
            const unsigned long long v = ld_acquire_u64(P.lq + h);
            if (v != QUEUE_EMPTY) {
                *item = v;
                return 0;
            }
        }
        if ((it & 7) == 0) {
            if (ld_acquire_u32(&st->error)) return 1;
            if (ld_acquire_u64(&st->lq_pending) == 0) return 1;
        }
        __nanosleep(backoff);
        backoff = min(backoff * 2, 2048u);
    }
    deep_fail(st, DEEP_ERR_SPIN);
    return 1;
}

// Records of survivors [first, first + k) of the unit, from the list: their
// patterns (below `parent`) and, when the unit has a child frame, member
// entries.  Lane q holds later member q's item in `item` (q < 32).
__device__ __forceinline__ void local_records(const DeepParams &P, const LocalWarp &w, unsigned lane, uint32_t parent,
                                              uint32_t item, bool members, uint32_t first, uint32_t k) {
    __syncwarp();
    for (uint32_t i0 = 0; i0 < k; i0 += 32) {
        const uint32_t i = i0 + lane;
        const uint2 e = i < k ? w.list[i] : make_uint2(0, 0);
        uint32_t it = __shfl_sync(CPM_FULL, item, e.x & 31);
        if (i < k) {
            if (e.x >= 32) it = __ldcg(P.mem_item + w.items + e.x);
            const unsigned long long pid = w.pid0 + first + i;
            P.pat_parent[pid] = parent;
            P.pat_item[pid] = it;
            P.pat_sup[pid] = e.y;
            if (P.pat_db) P.pat_db[pid] = w.db;
            if (members) {
                P.mem_pat[w.mb + first + i] = (uint32_t)pid;
                P.mem_item[w.mb + first + i] = it;
            }
        }
    }
    __syncwarp();
}

// What a pass over a unit's later members leaves besides its count.
struct LocalScan {
    bool write;      // child tidsets to out, survivor i at out + i * w2, i < cap
    bool records;    // records written whenever the list fills
    uint32_t cap;
    uint32_t done;   // survivors whose records are written
    uint32_t parent, item;
    ulonglong2 *out;
};

// One pass: survivors are listed in member order (from scan.done), their
// child tidsets written if asked.  K 16-byte words of a tidset per lane in
// registers (K = 1: each tidset over a group of G lanes; else G = 32), U steps
// of NG = 32 / G members loaded before they are reduced.  Tidsets of more than
// 256 words: the words from there on are counted first, and written before the
// member is known to survive (the next one takes the place if it does not).
// (Three forms: more of them, closer to a tidset's length, cost more in
// instruction fetches than they save: 2.0 -> 2.3 ms with five at 250,000 rows.)
template <int K, int U>
__device__ __forceinline__ uint32_t local_scan(const DeepParams &P, LocalWarp &w, unsigned lane,
                                               const ulonglong2 *pre2, uint32_t pitch, uint32_t cnt, LocalScan &scan) {
    const uint32_t W2 = w.w2;
    const uint32_t lg = W2 >= 32 ? 5u : (W2 <= 1 ? 0u : 32u - (uint32_t)__clz(W2 - 1u));
    const uint32_t G = 1u << lg, NG = 32u >> lg, gi = lane >> lg, gl = lane & (G - 1u);
    const ulonglong2 *sib0 = pre2 + pitch;  // later member q (from 0) at sib0 + q * pitch
    const ulonglong2 zero = make_ulonglong2(0ull, 0ull);
    uint32_t run = 0;
    ulonglong2 pre[K];
#pragma unroll
    for (int k = 0; k < K; ++k) pre[k] = gl + G * k < W2 ? ld_cg(pre2 + gl + G * k) : zero;
    for (uint32_t q0 = 0; q0 < cnt; q0 += NG * U) {
        if (scan.records && run - scan.done + NG * U > LOCAL_LIST) {
            local_records(P, w, lane, scan.parent, scan.item, true, scan.done, run - scan.done);
            scan.done = run;
        }
        uint32_t far = 0;  // of the words from 256 on
        if (K == 8 && W2 > 256) {  // (one member per step)
            const ulonglong2 *sb = sib0 + (uint64_t)q0 * pitch;
            ulonglong2 *o = scan.out + (uint64_t)run * W2;
            const bool wr = scan.write && run < scan.cap;
            for (uint32_t j0 = 256 + lane; j0 - lane < W2; j0 += 128) {
                ulonglong2 y[4], z[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint32_t j = j0 + 32 * k;
                    y[k] = j < W2 ? ld_cg(sb + j) : zero;
                    z[k] = j < W2 ? ld_cg(pre2 + j) : zero;
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint32_t j = j0 + 32 * k;
                    y[k] = and2(y[k], z[k]);
                    far += popc2(y[k]);
                    if (wr && j < W2) o[j] = y[k];
                }
            }
        }
        ulonglong2 x[U][K];
#pragma unroll
        for (int v = 0; v < U; ++v) {
            const uint32_t q = q0 + v * NG + gi;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const uint32_t j = gl + G * k;
                x[v][k] = (q < cnt && j < W2) ? ld_cg(sib0 + (uint64_t)q * pitch + j) : zero;
            }
        }
#pragma unroll
        for (int v = 0; v < U; ++v) {
            const uint32_t q = q0 + v * NG + gi;
            uint32_t c = far;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                x[v][k] = and2(x[v][k], pre[k]);
                c += popc2(x[v][k]);
            }
            c = group_sum(c, G);
            const bool sv = q < cnt && (long long)c >= w.minsup;
            const unsigned bal = __ballot_sync(CPM_FULL, sv && gl == 0);
            const uint32_t idx = run + __popc(bal & ((1u << (gi * G)) - 1u));
            if (sv && idx < scan.cap) {
                if (scan.write) {
                    ulonglong2 *o = scan.out + (uint64_t)idx * W2;
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        const uint32_t j = gl + G * k;
                        if (j < W2) o[j] = x[v][k];
                    }
                }
                if (gl == 0 && idx - scan.done < LOCAL_LIST) w.list[idx - scan.done] = make_uint2(q, c);
            }
            run += __popc(bal);
        }
    }
    return run;
}

__device__ __forceinline__ uint32_t local_pass(const DeepParams &P, LocalWarp &w, unsigned lane,
                                               const ulonglong2 *pre2, uint32_t pitch, uint32_t cnt, LocalScan &scan) {
    if (w.w2 <= 32) return local_scan<1, 4>(P, w, lane, pre2, pitch, cnt, scan);
    if (w.w2 <= 128) return local_scan<4, 2>(P, w, lane, pre2, pitch, cnt, scan);
    return local_scan<8, 1>(P, w, lane, pre2, pitch, cnt, scan);
}

// Lane 0 of the warp: room for `words` in its chunk, a new chunk if need be.
// A chunk is a quarter of the warp's share of what the first three quarters of
// the arena have left; a unit that needs more gets none.
__device__ __forceinline__ bool local_chunk(const DeepParams &P, LocalWarp &w, unsigned long long words) {
    if (w.end - w.at >= words) return true;
    const unsigned long long used = ld_relaxed_u64(&P.st->arena_next), top = P.arena_words / 4 * 3;
    if (used >= top) return false;
    const unsigned long long size = (top - used) / (4ull * LOCAL_WARPS * gridDim.x) & ~1ull;
    if (size < words) return false;
    const unsigned long long a = atomicAdd(&P.st->arena_next, size);
    if (a + size > P.arena_words) {
        deep_fail(P.st, DEEP_ERR_ARENA);
        return false;
    }
    w.low = w.at = w.floor = a;
    w.end = a + size;
    return true;
}

// Units [p, m - 1) of the frame, for any warp: the frame published by lane 0,
// its units queued by the warp.  The tidsets and member entries are written.
__device__ __forceinline__ void local_publish(const DeepParams &P, const LocalWarp &w, unsigned lane,
                                              const ulonglong2 *base, unsigned long long mem, uint32_t m, uint32_t p) {
    DeepState *st = P.st;
    const uint32_t n = m - 1 - p;
    __syncwarp();
    unsigned long long nf = 0, qb = 0;
    int pub = 0;
    if (lane == 0) {
        nf = atomicAdd(&st->n_frames, 1ull);
        qb = atomicAdd(&st->lq_tail, (unsigned long long)n);
        if (nf >= P.frames_cap) {
            deep_fail(st, DEEP_ERR_FRAMES);
        } else if (qb + n > P.lq_cap) {
            deep_fail(st, DEEP_ERR_QUEUE);
        } else {
            DFrame c;
            c.mask = nullptr;
            c.mem_off = mem;
            c.m = m;
            c.root = w.root;
            c.stride = 2u * w.w2;
            c.db = w.db;
            c.minsup = w.minsup;
            c.bits = reinterpret_cast<const uint64_t *>(base);
            P.frames[nf] = c;
            // Its units count as pending before this unit leaves lq_pending.
            atomicAdd(&st->lq_pending, (unsigned long long)n);
            __threadfence();
            pub = 1;
        }
    }
    __syncwarp();
    pub = __shfl_sync(CPM_FULL, pub, 0);
    if (!pub) return;
    nf = __shfl_sync(CPM_FULL, nf, 0);
    qb = __shfl_sync(CPM_FULL, qb, 0);
    for (uint32_t i = lane; i < n; i += 32) st_release_u64(P.lq + qb + i, (nf << 32) | (p + i));
}

// The next unit of the frame at w.lv[depth].  Two or more survivors: their
// frame in *child.  Returns its members, or 0.
__device__ __forceinline__ uint32_t local_unit(const DeepParams &P, LocalWarp &w, unsigned lane, uint32_t depth,
                                               LocalLevel *child) {
    DeepState *st = P.st;
    const uint32_t W2 = w.w2, pitch = depth ? W2 : w.pitch;
    const uint32_t p = w.lv[depth].p, cnt = w.lv[depth].m - p - 1;
    const ulonglong2 *pre2 = w.lv[depth].base + (uint64_t)p * pitch;
    const unsigned long long entry = w.lv[depth].mem + p;
    if (lane == 0) w.items = entry + 1;
    LocalScan scan;
    scan.done = 0;
    scan.parent = __ldcg(P.mem_pat + entry);
    scan.item = lane < cnt ? __ldcg(P.mem_item + entry + 1 + lane) : 0u;
    // One pass, child tidsets to the chunk.  One later member: no child frame.
    int single = 0;
    if (lane == 0) single = cnt > 1 && cnt <= LOCAL_LIST && local_chunk(P, w, 2ull * W2 * cnt);
    single = __shfl_sync(CPM_FULL, single, 0);
    __syncwarp();
    scan.write = single;
    scan.records = false;
    scan.cap = cnt;
    scan.out = reinterpret_cast<ulonglong2 *>(P.arena + (single ? w.at : 0));
    uint32_t ns = 0;
    for (;;) {
        const uint32_t got = local_pass(P, w, lane, pre2, pitch, cnt, scan);
        if (scan.records) {  // the two passes read the same words: they must agree
            if (got == ns) break;
            if (lane == 0) deep_fail(st, DEEP_ERR_INTERNAL);
            return 0;
        }
        ns = got;
        if (lane == 0) {
            w.inter += cnt;
            w.bytes += 16ull * W2 * (cnt + 1ull + (ns > 1 ? ns : 0));
            w.units += 1;
            w.surv += ns;
            if (P.root_cost) atomicAdd(P.root_cost + w.root, (unsigned long long)cnt);
        }
        if (ns == 0) return 0;
        // Pattern ids, member entries and, without a chunk, the child block.
        const bool block = ns > 1 && !single, frame = ns > 2 || block;
        unsigned long long ab = 0;
        int ok = 1;
        if (lane == 0) {
            const unsigned long long words = 2ull * W2 * ns;
            const unsigned long long pid0 = atomicAdd(&st->n_patterns, (unsigned long long)ns);
            const unsigned long long mb = frame ? atomicAdd(&st->n_members, (unsigned long long)ns) : 0ull;
            if (block) ab = atomicAdd(&st->arena_next, words);
            if (pid0 + ns > P.pat_cap) { deep_fail(st, DEEP_ERR_PATTERNS); ok = 0; }
            if (frame && mb + ns > P.members_cap) { deep_fail(st, DEEP_ERR_MEMBERS); ok = 0; }
            if (block && ab + words > P.arena_words) { deep_fail(st, DEEP_ERR_ARENA); ok = 0; }
            if (frame && single) w.at += words;
            w.pid0 = pid0;
            w.mb = mb;
        }
        ok = __shfl_sync(CPM_FULL, ok, 0);
        if (!ok) return 0;
        if (!block) break;
        scan.write = scan.records = true;
        scan.cap = ns;
        scan.out = reinterpret_cast<ulonglong2 *>(P.arena + __shfl_sync(CPM_FULL, ab, 0));
    }
    if (ns == 2 && single) {
        // Their child frame is one unit of one later member: counted here.
        local_records(P, w, lane, scan.parent, scan.item, false, 0, 2);
        uint32_t c = 0;
        for (uint32_t j = lane; j < W2; j += 32) c += popc2(and2(ld_cg(scan.out + j), ld_cg(scan.out + W2 + j)));
        c = warp_sum_u32(c);
        const uint32_t q = w.list[1].x;
        if (lane == 0) {
            const bool sv = (long long)c >= w.minsup;
            w.inter += 1;
            w.bytes += 32ull * W2;
            w.units += 1;
            w.frames += 1;
            w.surv += sv;
            if (P.root_cost) atomicAdd(P.root_cost + w.root, 1ull);
            if (sv) {
                const unsigned long long pid = atomicAdd(&st->n_patterns, 1ull);
                if (pid >= P.pat_cap) {
                    deep_fail(st, DEEP_ERR_PATTERNS);
                } else {
                    P.pat_parent[pid] = (uint32_t)w.pid0;
                    P.pat_item[pid] = __ldcg(P.mem_item + w.items + q);
                    P.pat_sup[pid] = c;
                    if (P.pat_db) P.pat_db[pid] = w.db;
                }
            }
        }
        __syncwarp();
        return 0;
    }
    local_records(P, w, lane, scan.parent, scan.item, ns > 1, scan.done, ns - scan.done);
    if (ns < 2) return 0;
    child->base = scan.out;
    child->mem = w.mb;
    child->m = ns;
    child->p = 0;
    return ns;
}

__global__ void __launch_bounds__(LOCAL_BLOCK, 4) k_local(DeepParams P) {
    extern __shared__ __align__(16) unsigned char local_smem[];
    const unsigned lane = threadIdx.x & 31;
    DeepState *st = P.st;
    LocalWarp &w = reinterpret_cast<LocalWarp *>(local_smem)[threadIdx.x >> 5];
    if (lane == 0) {
        w.low = w.at = w.end = w.floor = 0;
        w.inter = w.bytes = w.units = w.surv = w.frames = 0;
    }
    // Fewer units queued or running than this: work is shared.
    const unsigned long long busy = 2ull * LOCAL_WARPS * gridDim.x;
    for (;;) {
        unsigned long long item = 0;
        int stop = 0;
        if (lane == 0) {
            stop = local_claim(P, &item);
            // After an error nothing more is done: the host reruns the launch.
            if (!stop && ld_relaxed_u32(&st->error)) stop = 1;
        }
        stop = __shfl_sync(CPM_FULL, stop, 0);
        if (stop) break;
        item = __shfl_sync(CPM_FULL, item, 0);
        const DFrame *fp = P.frames + (uint32_t)(item >> 32);
        if (lane == 0) {
            w.lv[0].base =
                reinterpret_cast<const ulonglong2 *>(__ldcg(reinterpret_cast<const unsigned long long *>(&fp->bits)));
            w.lv[0].mem = __ldcg(reinterpret_cast<const unsigned long long *>(&fp->mem_off));
            w.lv[0].m = __ldcg(&fp->m);
            w.lv[0].p = (uint32_t)item;
            w.pitch = __ldcg(&fp->stride) / 2u;
            const uint32_t used = __ldcg(&fp->used);
            w.w2 = used ? used : w.pitch;
            w.root = __ldcg(&fp->root);
            w.db = __ldcg(&fp->db);
            w.minsup = __ldcg(&fp->minsup);
        }
        __syncwarp();
        if (!w.lv[0].base || w.w2 == 0 || w.w2 > w.pitch || w.pitch > (LOCAL_MAX_BITS + 127) / 128 ||
            w.lv[0].p + 1 >= w.lv[0].m) {
            if (lane == 0) deep_fail(st, DEEP_ERR_INTERNAL);
            break;
        }
        // The claimed unit (lv[0]), then the frames below it (lv[1 .. depth]).
        uint32_t depth = 0;
        for (;;) {
            // (Not waited for before the unit's own loads are issued.)
            const unsigned long long pending = ld_relaxed_u64(&st->lq_pending);
            const unsigned int err = ld_relaxed_u32(&st->error);
            LocalLevel child;
            const uint32_t ns = local_unit(P, w, lane, depth, &child);
            const unsigned said = __shfl_sync(CPM_FULL, err ? 2u : pending < busy ? 1u : 0u, 0);
            if (said == 2) break;  // (the host reruns)
            if (lane == 0) w.lv[depth].p += 1;
            if (ns > 1) {
                if (said || depth + 1 >= LOCAL_DEPTH) {
                    local_publish(P, w, lane, child.base, child.mem, ns, 0);
                    if (lane == 0) w.floor = w.at;
                } else {
                    ++depth;
                    if (lane == 0) {
                        w.lv[depth] = child;
                        w.frames += 1;
                    }
                }
            }
            __syncwarp();
            // Frames that are done leave the stack and the chunk.
            while (depth && w.lv[depth].p + 1 >= w.lv[depth].m) {
                if (lane == 0) {
                    const unsigned long long a =
                        (unsigned long long)(reinterpret_cast<const uint64_t *>(w.lv[depth].base) - P.arena);
                    if (a >= w.low && a < w.end) w.at = max(a, w.floor);
                }
                --depth;
            }
            __syncwarp();
            if (!depth) break;
            if (said) {
                for (; depth; --depth) {
                    const LocalLevel l = w.lv[depth];
                    if (l.p + 1 >= l.m) continue;
                    local_publish(P, w, lane, l.base, l.mem, l.m, l.p);
                    if (lane == 0) w.frames -= 1;  // (counted with the published ones)
                }
                if (lane == 0) w.floor = w.at;
                __syncwarp();
                break;
            }
        }
        // Published frames' units were added to lq_pending before this unit leaves it.
        if (lane == 0) atomicAdd(&st->lq_pending, ~0ull);  // lq_pending -= 1
        __syncwarp();
    }
    if (lane == 0 && w.units) {
        atomicAdd(&st->intersections, w.inter);
        atomicAdd(&st->bytes_alg, w.bytes);
        atomicAdd(&st->work_items, w.units);
        atomicAdd(&st->local_units, w.units);
        atomicAdd(&st->local_frames, w.frames);
        atomicAdd(&st->survivors, w.surv);
    }
}

}  // namespace cpm
