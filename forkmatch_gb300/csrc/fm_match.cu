// fm_match.cu -- level-expansion kernels of the matcher.
//
// Replaces the reference's per-thread k-way merge (src/smsm.cu:299-345 isoGen,
// src/smsm.cu:57-140 isoCompare), injectivity walk (src/smsm.cu:188-227 isInj),
// ballot append (src/smsm.cu:146-182 attemptInsert) and table write
// (src/smsm.cu:706-779 isoWrite).
//
// One level launch extends every partial match by one query vertex.  Partial
// matches are full rows (column c = data vertex matched at depth c) stored
// column-major (SoA), so every load and store of a column is coalesced; there
// is no parent-pointer forest to climb.  Warps claim chunks of 32 parents
// (several chunks per atomic):
//   1. each lane loads its parent row and the k (label, ancestor) segment
//      records -- k independent 16-byte loads, issued back to back;
//   2. the shortest list is the driver; a warp prefix sum over driver lengths
//      turns the 32 parents' candidate lists into one range of slots;
//   3. lanes take 64 consecutive slots per round, two per lane with both driver
//      loads in flight (load-balanced across parents, so a hub parent keeps all
//      32 lanes busy); one word of the e-line filter per other list rejects
//      almost every candidate that is not in it, and what passes is queued
//      and tested exactly 32 at a time (inline compare, bitmap or binary
//      search, then against the row), and survivors are staged as (parent
//      index, value) in shared memory;
//   4. the stage outlives the chunk: it is flushed with one atomic per 96+
//      survivors (192+ where every candidate survives) and fully coalesced
//      stores, column by column into the next level or as contiguous
//      row-major rows into the table.
// A chunk whose candidate range is long (a hub) is not walked by one warp: it
// is published to a heavy list and cut into pieces that every warp of a second
// launch shares; launches of one match overlap (dev::pass_wait).  Lists of length <= 3
// are inline in the segment record, so the common case needs no second memory
// access.  With duplicate e-lines the value at rank r of its run in the driver
// list survives only if every other list holds at least r + 1 copies
// (min-multiplicity semantics of the reference's merge); with no other list
// every copy survives and no rank is asked (4-vertex path with its table, 2.2e8
// rows: 1.85 ms, 2.79 with the ranks).
//
// Bounded memory: before expanding a chunk a warp holds output budget for its
// candidate upper bound (reserved from the level in blocks); when a
// reservation does not fit, the warp defers its remaining chunks, raises
// `stop`, and exits; the host drains the output level (depth first) and
// relaunches this level on the deferred chunks plus the unclaimed remainder.
// Nothing spins and nothing traps.
#include <algorithm>
#include <map>
#include <mutex>
#include <set>
#include <tuple>
#include <utility>

#include "fm_device.cuh"

namespace fm {
namespace {

using dev::kFull;
using dev::ldg4;
using dev::lower_bound_g;
using dev::seg_at;
using dev::seg_has;
using dev::SlotWalk;

constexpr int kWarps = 8;
// Staged survivors per warp: levels with one back edge flush most (every
// candidate survives) and have no filter queue; 128 entries there cost 10-14 %
// against 256, which elsewhere cost more in L1 than they save in flushes.
constexpr uint32_t kStage = 128, kStageOne = 256;
__host__ __device__ constexpr uint32_t stage_rows(uint32_t k) { return k == 1 ? kStageOne : kStage; }
constexpr uint32_t kSlots = 2;             // candidate slots per lane per round
constexpr uint32_t kPend = 32 * kSlots + 32;  // candidates that wait for their exact test, per warp
constexpr uint32_t kHeavyMaxPieces = 65536;
// A level none of whose chunks can have more candidates than this (32 parents
// with the graph's longest list) has no heavy pass.
constexpr uint32_t kHeavyLeast = 512;

// Rank of position t within its run of equal values.
__device__ __forceinline__ uint32_t seg_rank(const uint4& s, uint32_t t, uint32_t x, const uint32_t* __restrict__ nbr) {
    if (s.x <= 3) return (t >= 1 && s.y == x) + (t >= 2 && s.z == x);
    const uint32_t* a = nbr + (uint64_t)s.y * 4;
    return t - lower_bound_g(a, t, x);
}

// Launch tuning, computed on the device from the level's actual size, so a
// launch whose parent count is only known on the device is tuned the same way.
// Both passes derive the split parameters from the same inputs.
struct Tune {
    unsigned long long n_parents, n_items;
    uint32_t claim_batch;    // chunks claimed per atomic (keeps ~2 claims per warp on big levels)
    uint32_t credit_block;   // output rows reserved per budget atomic; idle credit stays under 1/4 of the level
    uint32_t heavy_thresh;   // candidate slots above which a chunk is split: finer when chunks are few
    uint32_t heavy_piece;    // slots per piece of a split chunk
};

__device__ __forceinline__ Tune make_tune(const ExpandParams& P, bool main_pass) {
    Tune t;
    if (P.n_parents_dev) {
        t.n_parents = *(const volatile unsigned long long*)P.n_parents_dev;
        t.n_items = (t.n_parents + 31) / 32;
    } else {
        t.n_parents = P.n_parents;
        t.n_items = P.n_items;
    }
    const unsigned long long all_warps = P.max_warps ? P.max_warps : 1;
    if (main_pass) {
        // roots cost the same per chunk, so they can be claimed in big batches;
        // deeper chunks vary, so batches stay small there to keep warps balanced
        const unsigned long long warps = (unsigned long long)gridDim.x * (blockDim.x / 32);
        const unsigned long long per_warp = t.n_items / warps + 1;
        const unsigned long long b = per_warp / (P.pin ? 16 : 2);
        t.claim_batch = (uint32_t)(b < 1 ? 1 : (b > 8 ? 8 : b));
    } else {
        t.claim_batch = 1;
    }
    const unsigned long long cb = P.ocap / (4 * all_warps);
    t.credit_block = (uint32_t)(cb < 1024 ? cb : 1024);
    t.heavy_thresh = t.n_items >= 4 * all_warps ? 4096u : (t.n_items >= all_warps ? 1024u : 256u);
    if (32ull * P.max_list <= kHeavyLeast) t.heavy_thresh = 0xffffffffu;   // there is no heavy pass
    // a piece of a chunk with shared intersections computes them again, so its
    // pieces are long (2048 to 16384 slots: 32.3 to 27.2 ms on the level below)
    if (P.share_words && t.n_items >= 4 * all_warps) t.heavy_thresh = 32768u;
    t.heavy_piece = t.heavy_thresh / 2;
    return t;
}

__device__ __forceinline__ uint32_t item_chunk(const ExpandParams& P, unsigned long long item) {
    return item < P.ndef_in ? P.def_in[(P.def_in_pos + item) % P.def_cap]
                            : (uint32_t)(P.fresh_base + (item - P.ndef_in));
}

__device__ __forceinline__ HeavyEntry heavy_entry(const HeavyEntry* p) {
    const uint4 v = __ldcg((const uint4*)p);
    return {v.x, v.y, v.z, v.w};
}

__device__ __forceinline__ void defer_chunk(const ExpandParams& P, uint32_t chunk) {
    const unsigned idx = atomicAdd(&P.ctl->ndef, 1u);
    const uint32_t room = P.def_room ? P.def_room : P.def_cap;
    if (idx < room) P.def_out[(P.def_out_pos + idx) % P.def_cap] = chunk;
    else atomicOr(&P.ctl->error, 1u);
}

// Per-warp shared memory.
struct WarpMem {
    uint32_t* rows_s;   // [d][32] parent rows of the current chunk, column-major
    uint4* segs_s;      // [n_recs][32] segment records (all k of a parent, or its driver's)
    uint2* start_s;     // [32] parents with candidates: first slot, lane (dev::SlotWalk)
    uint8_t* drv_s;     // [32] driver list of each parent
    uint32_t* stp;      // [stage_rows] staged survivors: parent index in the level
    uint32_t* stx;      // [stage_rows] staged survivors: new vertex
    uint32_t* px;       // [kPend] candidates the filter let pass: vertex
    uint8_t* pj;        // [kPend] and parent (lane) in the chunk
    uint64_t* mbar;     // completion barrier of the list stage's bulk copies
    uint32_t* stage;    // [stage_words] membership lists copied in by TMA (optional)
    uint32_t* shared;   // [share_words] intersections that parents of the chunk share (optional)
};

// Counting levels store no survivors and have no stage.  The bytes matter: what
// the blocks of an SM do not take of its 256 KB is its L1, which serves the
// records, lists and filter words (with 6 blocks, 33 KB a block instead of 31
// leaves 28 KB of L1 instead of 60 and made the counting level of a 5-vertex
// path 1.5 times slower).
__host__ __device__ constexpr uint32_t per_warp_bytes(uint32_t d, uint32_t k, uint32_t recs, uint32_t stage_words,
                                                      bool staged, uint32_t share_words) {
    return 128 * d + 512 * recs + 256 + 32 + (staged ? 8 * stage_rows(k) : 0u) + (k == 1 ? 0u : 5 * kPend) +
           4 * stage_words + 4 * share_words;
}
static_assert(5 * kPend % 16 == 0 && 8 * kStage % 16 == 0, "the list stage is 16-byte aligned");

// Records kept per parent: only the driver's.  The other lists are asked through
// the filter, and the few exact tests load their record again.  Graphs with
// duplicates test every candidate exactly and the list stage rewrites records,
// so those keep all.
__host__ __device__ constexpr uint32_t n_recs(uint32_t k, bool dups, uint32_t stage_words) {
    return dups || stage_words ? k : 1;
}

__device__ __forceinline__ WarpMem warp_mem(unsigned char* smem_raw, uint32_t warp, uint32_t d, uint32_t k,
                                            uint32_t recs, uint32_t stage_words, bool staged, uint32_t share_words,
                                            uint64_t* mbar_s) {
    unsigned char* ws = smem_raw + warp * per_warp_bytes(d, k, recs, stage_words, staged, share_words);
    WarpMem m;
    m.rows_s = (uint32_t*)ws;
    m.segs_s = (uint4*)(ws + 128 * d);
    m.start_s = (uint2*)(ws + 128 * d + 512 * recs);
    m.drv_s = (uint8_t*)(m.start_s + 32);
    m.stp = (uint32_t*)(m.drv_s + 32);
    m.stx = m.stp + stage_rows(k);
    m.px = m.stp + (staged ? 2 * stage_rows(k) : 0u);
    m.pj = (uint8_t*)(m.px + kPend);
    m.mbar = mbar_s + warp;
    m.stage = (uint32_t*)(m.pj + kPend);
    m.shared = m.stage + stage_words;
    return m;
}

// Membership lists longer than this many words are not staged.
constexpr uint32_t kStageMaxList = 2048;
// Bound on the polls of one stage's completion barrier.
constexpr uint32_t kStageSpinLimit = 1u << 22;

// Stage the membership lists of the loaded chunk: every lane's non-driver
// lists of 4..kStageMaxList entries without a bitmap that its parent's
// candidates probe often enough for the copy to pay (the list-length ratio
// rule of dev::stage_worth) are copied into the warp's stage with TMA bulk copies
// (lanes in order while the stage has room) and their records in segs_s are
// pointed at the stage.  Lane 0 arms the barrier with the byte count, every
// lane issues its own copies, and the warp waits for the phase, boundedly.
// Returns false (warp-uniform) if the wait ran out; the error bit 2 of the
// level's control block is then raised.
__device__ __forceinline__ bool stage_lists(const ExpandParams& P, const WarpMem& m, uint32_t lane, uint32_t k,
                                            uint32_t drv, uint32_t n, bool valid, uint32_t& phase) {
    uint32_t want = 0;
    if (valid && k >= 2 && n >= 2) {
        for (uint32_t i = 0; i < k; i++) {
            if (i == drv) continue;
            const uint4 r = m.segs_s[i * 32 + lane];
            if (dev::stage_worth(r, n, kStageMaxList)) want += (r.x + 3) & ~3u;
        }
    }
    uint32_t incl = want;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, incl, o);
        if ((int)lane >= o) incl += t;
    }
    const bool fits = want && incl <= P.stage_words;
    uint32_t bytes = fits ? want * 4 : 0;
#pragma unroll
    for (int o = 16; o; o >>= 1) bytes += __shfl_xor_sync(kFull, bytes, o);
    if (!bytes) return true;
    // earlier generic reads of the stage come before the copies overwrite it
    dev::fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) dev::mbar_arrive_expect_tx(m.mbar, bytes);
    __syncwarp();
    if (fits) {
        uint32_t off = incl - want;
        for (uint32_t i = 0; i < k; i++) {
            if (i == drv) continue;
            uint4 r = m.segs_s[i * 32 + lane];
            if (dev::stage_worth(r, n, kStageMaxList)) {
                const uint32_t words = (r.x + 3) & ~3u;
                dev::bulk_copy_g2s(m.stage + off, P.nbr + (uint64_t)r.y * 4, words * 4, m.mbar);
                r.y = dev::kStagedMark | off;
                m.segs_s[i * 32 + lane] = r;
                off += words;
            }
        }
    }
    bool ok = false;
    for (uint32_t spin = 0; spin < kStageSpinLimit && !ok; spin++) ok = dev::mbar_try_wait(m.mbar, phase);
    phase ^= 1u;
    ok = __all_sync(kFull, ok);
    if (!ok && lane == 0) atomicOr(&P.ctl->error, 2u);
    __syncwarp();
    return ok;
}

// Column c of parent p of the level being expanded.  An ordinary load: the rows
// of a run repeat their older columns and a flush reads them once a survivor, so
// the L1 serves most of it.
template <bool ROOTS>
__device__ __forceinline__ uint32_t parent_col(const ExpandParams& P, uint32_t c, uint32_t p) {
    if (ROOTS) return P.root_list ? __ldg(P.root_list + p) : P.root_begin + p;
    return P.pin[c * P.pstride + p];
}

// Column c of staged parent p: from the warp's copy of chunk `cur` in shared
// memory when p belongs to it (most survivors do), else from the level.
template <bool ROOTS>
__device__ __forceinline__ uint32_t staged_col(const ExpandParams& P, const WarpMem& m, uint32_t c, uint32_t p,
                                               uint32_t cur) {
    if ((p >> 5) == cur) return m.rows_s[c * 32 + (p & 31)];
    return parent_col<ROOTS>(P, c, p);
}

// Write the staged survivors with one atomic: column by column into the next
// level (SoA), or row-major into the table; every store is coalesced.  `cur`
// is the chunk whose rows the warp holds in shared memory.
template <int MODE, bool ROOTS>
__device__ __forceinline__ void flush_stage(const ExpandParams& P, const WarpMem& m, uint32_t nst, uint32_t lane,
                                            uint32_t d, const uint8_t* col_depth_s, uint32_t cur) {
    unsigned long long pos0 = 0;
    if (lane == 0)
        pos0 = atomicAdd(MODE == kModeMid ? &P.ctl->produced : &P.tot->table_pos, (unsigned long long)nst);
    pos0 = __shfl_sync(kFull, pos0, 0);
    if (MODE == kModeMid) {
        for (uint32_t c = 0; c < d; c++) {
            uint32_t* col = P.pout + c * P.ocap + pos0;
            for (uint32_t i = lane; i < nst; i += 32) col[i] = staged_col<ROOTS>(P, m, c, m.stp[i], cur);
        }
        uint32_t* col = P.pout + d * P.ocap + pos0;
        for (uint32_t i = lane; i < nst; i += 32) col[i] = m.stx[i];
    } else {
        // one row per lane; the warp's rows are contiguous, so the vector
        // stores of a round cover one block of 32 * 4q bytes
        const uint32_t q = P.plan.q;
        if (pos0 >= P.table_cap) return;
        const uint64_t room = P.table_cap - pos0;
        const uint32_t rows = nst < room ? nst : (uint32_t)room;
        uint32_t* out = P.table + pos0 * q;
        for (uint32_t r = lane; r < rows; r += 32) {
            const uint32_t p = m.stp[r], x = m.stx[r];
            uint32_t* o = out + (uint64_t)r * q;
            if (P.table_vec4) {
                for (uint32_t c = 0; c < q; c += 4) {
                    uint4 v;
                    uint32_t dep = col_depth_s[c];
                    v.x = dep < d ? staged_col<ROOTS>(P, m, dep, p, cur) : x;
                    dep = col_depth_s[c + 1];
                    v.y = dep < d ? staged_col<ROOTS>(P, m, dep, p, cur) : x;
                    dep = col_depth_s[c + 2];
                    v.z = dep < d ? staged_col<ROOTS>(P, m, dep, p, cur) : x;
                    dep = col_depth_s[c + 3];
                    v.w = dep < d ? staged_col<ROOTS>(P, m, dep, p, cur) : x;
                    *(uint4*)(o + c) = v;
                }
            } else {
                for (uint32_t c = 0; c < q; c++) {
                    const uint32_t dep = col_depth_s[c];
                    o[c] = dep < d ? staged_col<ROOTS>(P, m, dep, p, cur) : x;
                }
            }
        }
    }
}

// The back edges' filter slices and columns of a level, the same for every
// parent (in shared memory, one copy per block).
struct LevelLists {
    uint2 slice[kMaxQ];              // first word, words
    const uint4* records[kMaxQ];     // of the back edge's label
    uint8_t anc[kMaxQ];
    __device__ __forceinline__ dev::FilterSlice at(const ExpandParams& P, uint32_t i) const {
        return {P.efilter + slice[i].x, slice[i].y};
    }
};

__device__ __forceinline__ void level_lists_init(const ExpandParams& P, LevelLists& L, uint32_t d) {
    const uint32_t k = P.plan.nreq[d], rb = P.plan.req_begin[d];
    if (threadIdx.x < k) {
        const uint32_t l = P.plan.req_label[rb + threadIdx.x];
        L.anc[threadIdx.x] = P.plan.req_anc[rb + threadIdx.x];
        L.records[threadIdx.x] = P.seg + (uint64_t)l * P.V;
        if (P.efilter) {
            const uint32_t a = __ldg(P.efilter_off + l);
            L.slice[threadIdx.x] = make_uint2(a, __ldg(P.efilter_off + l + 1) - a);
        }
    }
    __syncthreads();
}

// -------------------------------------------------- shared intersections
//
// The rows of a level come in runs: parents that extend the same earlier match
// differ only in their newest column.  Where the two oldest back edges of a
// level leave the newest column alone, the intersection T of their lists is
// the same for the whole run; it is computed once by the warp, kept in shared
// memory for the next chunks of the run, and drives where it is shorter than
// every list of the parent: far fewer candidates, and two tests less for each.
// A run needs 4 parents in the chunk and as many candidates, over them, as
// building T reads; T must fit the buffer.  Levels with less than four chunks a
// warp are left alone: there the time is one chunk's latency, which building T
// adds to.
//
// Closing level of 4-cliques on a 2^18-vertex power-law graph of 2 labels (3.8e7
// parents with 280 candidates each between hub lists, 70 with T): 27.2 ms, 66.4
// without.  1024 words a warp: 40.4 ms with the pieces of 512's 32.3, for the
// blocks and the L1 they cost.
constexpr uint32_t kShareWords = 512;
constexpr uint32_t kDrvShared = 0xff;         // drv_s: T drives
static_assert(kDrvShared >= kMaxQ, "no list index");

struct ShareState {
    unsigned long long key = ~0ull, bad = ~0ull;   // run whose T is at the buffer's start; run whose T did not fit
    uint32_t n = 0;                                // entries of that T
};

// T for runs of lanes with equal `key` (the vertices of back edges q0 and
// q0 + 1): returns its length and offset in m.shared for this lane, or
// 0xffffffff.  `work`: the lane's candidates without it (0: no parent).
// Whether a run is shared depends on the chunk alone, never on what the warp
// did before: the heavy pass has to find the same slots.
__device__ __forceinline__ uint32_t share_lists(const ExpandParams& P, const WarpMem& m, const LevelLists& L,
                                                uint32_t lane, uint32_t q0, unsigned long long key, uint32_t work,
                                                ShareState& st, uint32_t& off_out) {
    const unsigned same = __match_any_sync(kFull, key);
    unsigned todo = __ballot_sync(kFull, work > 0 && __popc(same) >= 4);
    uint32_t used = 0, mine = 0xffffffffu;
    while (todo) {
        const int leader = __ffs(todo) - 1;
        const unsigned grp = __shfl_sync(kFull, same, leader);
        todo &= ~grp;
        const unsigned long long gkey = __shfl_sync(kFull, key, leader);
        const bool in = (grp >> lane) & 1u;
        const uint32_t va = (uint32_t)(gkey >> 32), vb = (uint32_t)gkey;
        const uint4 ra = ldg4(L.records[q0] + va), rb = ldg4(L.records[q0 + 1] + vb);
        const bool first = ra.x <= rb.x;
        const uint4 base = first ? ra : rb, other = first ? rb : ra;
        const uint32_t all = __reduce_add_sync(kFull, in ? min(work, 1u << 24) : 0u);
        if (gkey == st.bad || all < base.x) continue;
        uint32_t n = 0;
        const uint32_t off = used;
        if (used == 0 && gkey == st.key) {
            n = st.n;                              // still there from the chunk before
        } else {
            if (used == 0) st.key = ~0ull;
            const dev::FilterSlice f = L.at(P, first ? q0 + 1 : q0);
            const uint32_t seed = dev::filter_seed(first ? vb : va);
            __syncwarp();
            for (uint32_t t0 = 0; t0 < base.x; t0 += 32) {
                const uint32_t t = t0 + lane;
                uint32_t x = 0;
                bool ok = t < base.x;
                if (ok) {
                    x = seg_at(base, t, P.nbr);
                    ok = dev::filter_has(f, seed, x) && seg_has(other, x, 1, P.nbr, P.bm, P.bm_words);
                }
                const unsigned b = __ballot_sync(kFull, ok);
                if (off + n + __popc(b) > P.share_words) {
                    n = 0xffffffffu;
                    break;
                }
                if (ok) m.shared[off + n + __popc(b & ((1u << lane) - 1u))] = x;
                n += __popc(b);
            }
            __syncwarp();
            if (n == 0xffffffffu) {
                if (off == 0) st.bad = gkey;       // alone it never fits
                continue;
            }
            if (off == 0) {
                st.key = gkey;
                st.n = n;
            }
        }
        if (in) {
            mine = n;
            off_out = off;
        }
        used = off + n;
    }
    return mine;
}

// Load the 32 parents of `chunk`, look up their k lists (independent 16-byte
// loads), pick each parent's shortest list as its driver and prefix-sum the
// driver lengths.  Returns the chunk's candidate slots (warp-uniform).
template <bool ROOTS, bool DUPS, bool SHARE>
__device__ __forceinline__ uint32_t load_chunk(const ExpandParams& P, const WarpMem& m, uint32_t chunk, uint32_t lane,
                                               uint32_t d, uint32_t k, uint32_t rb, unsigned long long n_parents,
                                               bool& valid, unsigned long long& words, uint32_t& phase,
                                               bool& stage_ok, uint32_t& excl, uint32_t& n, const LevelLists& L,
                                               bool share_on, ShareState& share) {
    const uint64_t p = (uint64_t)chunk * 32 + lane;
    valid = p < n_parents;
    if (ROOTS) {
        m.rows_s[lane] = !P.root_list ? P.root_begin + (uint32_t)p : valid ? __ldg(P.root_list + p) : 0u;
    } else {
        for (uint32_t c = 0; c < d; c++) m.rows_s[c * 32 + lane] = valid ? P.pin[c * P.pstride + p] : 0u;
    }
    uint32_t drv = 0;
    n = 0;
    words = 0;
    if (valid) {
        const bool all = DUPS || P.stage_words;
        uint4 best = make_uint4(0xffffffffu, 0, 0, 0);
        for (uint32_t i = 0; i < k; i++) {
            const uint32_t anc = P.plan.req_anc[rb + i];
            const uint32_t lab = P.plan.req_label[rb + i];
            const uint32_t v = m.rows_s[anc * 32 + lane];
            const uint4 sg = ldg4(P.seg + (uint64_t)lab * P.V + v);
            if (all) m.segs_s[i * 32 + lane] = sg;
            words += sg.x;
            if (sg.x < best.x) {
                best = sg;
                drv = i;
            }
        }
        n = best.x;
        if (!all) m.segs_s[lane] = best;
        // shortest list first where every candidate is tested exactly
        if (DUPS && k > 2) drv = dev::order_lists(m.segs_s, lane, k, drv);
    }
    if (SHARE && share_on) {
        // back edges are ordered by climb: the two oldest come last
        const uint32_t q0 = k - 2;
        const unsigned long long key =
            (unsigned long long)m.rows_s[L.anc[q0] * 32 + lane] << 32 | m.rows_s[L.anc[q0 + 1] * 32 + lane];
        uint32_t off = 0;
        const uint32_t nt = share_lists(P, m, L, lane, q0, key, valid ? n : 0u, share, off);
        if (nt < n) {
            n = nt;
            drv = kDrvShared;
            m.segs_s[lane] = make_uint4(nt, dev::kStagedMark | off, 0, 0);
        }
    }
    stage_ok = true;
    if (P.stage_words && k >= 2) stage_ok = stage_lists(P, m, lane, k, drv, n, valid, phase);
    uint32_t incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, incl, o);
        if ((int)lane >= o) incl += t;
    }
    excl = incl - n;
    m.drv_s[lane] = (uint8_t)drv;
    __syncwarp();
    return __shfl_sync(kFull, incl, 31);
}

// Work counters of the last depth under pre-count (lane-private): the
// survivors stand for that depth's parents, one lookup each, and their
// lists' lengths for its list words.
struct PreAcc {
    unsigned long long parents = 0, words = 0;
};

// Adds a warp's pre-count work counters to the next depth's control block,
// so the last depth reports the same work as when it is launched.
__device__ __forceinline__ void flush_pre(const ExpandParams& P, PreAcc& pre, uint32_t lane) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        pre.parents += __shfl_down_sync(kFull, pre.parents, o);
        pre.words += __shfl_down_sync(kFull, pre.words, o);
    }
    if (lane == 0 && pre.parents) {
        LaunchCtl* next = P.ctl + 1;
        atomicAdd(&next->parents, pre.parents);
        atomicAdd(&next->lookups, pre.parents);
        atomicAdd(&next->list_words, pre.words);
    }
}

// What survives a warp round at its level: lane's candidate x of parent j,
// `ok` if it survived.  Counted, pre-counted, or staged for the next level or
// the table; the stage is flushed when it cannot take another round, unless
// `more` follows at once.
struct Emit {
    uint32_t& nst;                        // staged survivors (warp-uniform)
    uint32_t flush_at;                    // flushed above this many
    unsigned long long& n_count;          // counted (warp-uniform)
    unsigned long long lane_count = 0;    // pre-counted by this lane
};

template <int MODE, bool ROOTS, bool DUPS, bool COMMON>
__device__ __forceinline__ void emit(const ExpandParams& P, const WarpMem& m, uint32_t chunk, bool ok, uint32_t j,
                                     uint32_t x, uint32_t lane, uint32_t d, const uint8_t* col_depth_s, bool more,
                                     Emit& e, PreAcc& pre) {
    if (MODE == kModeLastCount && !DUPS && P.pre_count) {
        // Pre-count: each survivor's extensions at the last depth (one back
        // edge: ancestor anc, label lab) are the entries of that list minus
        // the row's vertices found in it; the survivor is never stored.
        if (!ok) return;
        const uint32_t rb = P.plan.req_begin[d + 1];
        const uint32_t anc = P.plan.req_anc[rb];
        const uint4* segl = P.seg + (uint64_t)P.plan.req_label[rb] * P.V;
        const uint32_t v = anc == d ? x : m.rows_s[anc * 32 + j];
        const uint4 sg = ldg4(segl + v);
        const dev::FilterSlice f = dev::filter_slice(P.efilter, P.efilter_off, P.plan.req_label[rb]);
        e.lane_count += sg.x - dev::count_members_f(sg, f, v, m.rows_s, j, d, x, P.self_loops || anc != d, P.nbr, P.bm,
                                                    P.bm_words, COMMON ? P.bm_common : 0u);
        pre.parents += 1;
        pre.words += sg.x;
        return;
    }
    const unsigned b = __ballot_sync(kFull, ok);
    if (MODE == kModeLastCount) {
        e.n_count += __popc(b);
        return;
    }
    if (ok) {
        const uint32_t q = e.nst + __popc(b & ((1u << lane) - 1u));
        m.stp[q] = chunk * 32 + j;
        m.stx[q] = x;
    }
    e.nst += __popc(b);
    if (more) return;
    __syncwarp();
    if (e.nst > e.flush_at) {
        flush_stage<MODE, ROOTS>(P, m, e.nst, lane, d, col_depth_s, chunk);
        e.nst = 0;
        __syncwarp();
    }
}

// Evaluate slots [begin, end) of the loaded chunk: kSlots slots per lane per
// round with all their driver loads in flight.  With several back edges the
// filter rejects most candidates where they stand; the few it lets pass are
// collected and tested exactly 32 at a time, so that the exact tests (which
// differ from list to list and diverge) run with full warps.  Bound by issue
// slots and by the L1's rate for scattered words.  Closing level of a 4-cycle on
// a 2^20-vertex R-MAT graph with 64 labels (1.7e7 parents): 740 us, 1100 us with
// an exact test per candidate and a binary search per slot for its parent.
template <int MODE, bool ROOTS, bool DUPS, bool SHARE, bool COMMON>
__device__ __forceinline__ void process_slots(const ExpandParams& P, const WarpMem& m, uint32_t chunk,
                                              uint32_t excl, uint32_t n, uint32_t begin, uint32_t end, uint32_t lane,
                                              uint32_t d, uint32_t k, const LevelLists& L,
                                              const uint8_t* col_depth_s, uint32_t& nst,
                                              unsigned long long& n_count, PreAcc& pre) {
    // With one back edge both slots of a round are staged before one look at the
    // stage: a look after each, with its copy of the flush, made large tables
    // slower (4-vertex star on a 2^20-vertex R-MAT graph with 64 labels, 3.8e9
    // embeddings: 17.8 ms, 16.0 now; 4-vertex path, 3.1e8 rows: 2.88 and 2.61).
    Emit e{nst, stage_rows(k) - (k == 1 ? 32 * kSlots : 32), n_count};
    SlotWalk walk(m.start_s, excl, n, begin, lane);
    uint32_t pend = 0;
    const bool all = DUPS || (P.stage_words && k >= 2);      // every record is in segs_s
    for (uint32_t base = begin; base < end; base += 32 * kSlots) {
        uint32_t j[kSlots], t[kSlots], x[kSlots], dj[kSlots];
        bool ok[kSlots];
        // every driver load of the round is issued before any check
#pragma unroll
        for (uint32_t u = 0; u < kSlots; u++) {
            walk.window(m.start_s, base + 32 * u, lane, j[u], t[u]);
            x[u] = dj[u] = 0;
            ok[u] = base + 32 * u + lane < end;
            if (ok[u]) {
                dj[u] = m.drv_s[j[u]];
                const uint4 r = m.segs_s[(all ? dj[u] * 32 : 0u) + j[u]];
                if (SHARE && dj[u] == kDrvShared) x[u] = m.shared[(r.y & ~dev::kStagedMark) + t[u]];
                else x[u] = seg_at(r, t[u], P.nbr);
            }
        }
        if (DUPS || k == 1) {
            // membership first (with duplicates: enough copies), then
            // injectivity against the parent's row in shared memory
#pragma unroll
            for (uint32_t u = 0; u < kSlots; u++) {
                if (ok[u]) {
                    // (with one list every copy survives: no rank is asked)
                    if (DUPS && k > 1) {
                        const uint32_t need = seg_rank(m.segs_s[dj[u] * 32 + j[u]], t[u], x[u], P.nbr) + 1;
                        for (uint32_t i = 0; i < k && ok[u]; i++)
                            if (i != dj[u])
                                ok[u] = dev::seg_has_st(m.segs_s[i * 32 + j[u]], x[u], need, P.nbr, P.bm, P.bm_words,
                                                        m.stage);
                    }
                    for (uint32_t c = 0; c < d && ok[u]; c++) ok[u] = m.rows_s[c * 32 + j[u]] != x[u];
                }
            }
#pragma unroll
            for (uint32_t u = 0; u < kSlots; u++)
                emit<MODE, ROOTS, DUPS, COMMON>(P, m, chunk, ok[u], j[u], x[u], lane, d, col_depth_s,
                                        u + 1 < kSlots && (!DUPS || k == 1), e, pre);
            continue;
        }
        if constexpr (!DUPS) {
            for (uint32_t i = 0; i < k; i++) {
                const dev::FilterSlice f = L.at(P, i);
                const uint32_t* col = m.rows_s + L.anc[i] * 32;
#pragma unroll
                for (uint32_t u = 0; u < kSlots; u++)
                    if (ok[u] && dj[u] != i && !(SHARE && dj[u] == kDrvShared && i + 2 >= k))
                        ok[u] = dev::filter_has(f, dev::filter_seed(col[j[u]]), x[u]);
            }
#pragma unroll
            for (uint32_t u = 0; u < kSlots; u++) {
                const unsigned b = __ballot_sync(kFull, ok[u]);
                if (ok[u]) {
                    const uint32_t q = pend + __popc(b & ((1u << lane) - 1u));
                    m.px[q] = x[u];
                    m.pj[q] = (uint8_t)j[u];
                }
                pend += __popc(b);
            }
            const bool last = base + 32 * kSlots >= end;
            while (pend >= 32 || (last && pend)) {
                const uint32_t take = min(pend, 32u);
                pend -= take;
                __syncwarp();
                bool in = lane < take;
                uint32_t jj = 0, xx = 0;
                if (in) {
                    jj = m.pj[pend + lane];
                    xx = m.px[pend + lane];
                    const uint32_t dd = m.drv_s[jj];
                    for (uint32_t i = 0; i < k && in; i++) {
                        if (i == dd || (SHARE && dd == kDrvShared && i + 2 >= k)) continue;
                        const uint4 r = all ? m.segs_s[i * 32 + jj]
                                            : ldg4(L.records[i] + m.rows_s[L.anc[i] * 32 + jj]);
                        in = dev::seg_has_st(r, xx, 1, P.nbr, P.bm, P.bm_words, m.stage);
                    }
                    for (uint32_t c = 0; c < d && in; c++) in = m.rows_s[c * 32 + jj] != xx;
                }
                emit<MODE, ROOTS, DUPS, COMMON>(P, m, chunk, in, jj, xx, lane, d, col_depth_s, false, e, pre);
            }
            __syncwarp();
        }
    }
    __syncwarp();
    if (MODE == kModeLastCount && !DUPS && P.pre_count) {
#pragma unroll
        for (int o = 16; o; o >>= 1) e.lane_count += __shfl_xor_sync(kFull, e.lane_count, o);
        n_count += e.lane_count;
    }
}

// Work limit of a last level (warp-uniform result): lane 0 adds the warp's
// recent count to the total, compares the total (or the table rows reserved)
// with the limit and raises the limit flag.  Checked once per chunk or piece,
// so a warp overshoots by at most one chunk's work.
template <int MODE>
__device__ __forceinline__ bool over_limit(const ExpandParams& P, uint32_t lane, unsigned long long n_count,
                                           unsigned long long& n_flushed) {
    int over = 0;
    if (lane == 0) {
        unsigned long long seen;
        if (MODE == kModeLastCount) {
            seen = *(volatile unsigned long long*)&P.tot->count;
            if (n_count - n_flushed >= 4096) {
                seen = atomicAdd(&P.tot->count, n_count - n_flushed) + (n_count - n_flushed);
                n_flushed = n_count;
            }
        } else {
            seen = *(volatile unsigned long long*)&P.tot->table_pos;
        }
        if (seen > P.work_limit) {
            over = 1;
            atomicOr(&P.tot->error, kLimitFlag);
        }
    }
    return __shfl_sync(kFull, over, 0) != 0;
}

// Main pass: warps claim batches of chunks; long candidate ranges are
// published to the heavy list instead of being walked by one warp.
template <int MODE, bool ROOTS, bool DUPS, bool SHARE, bool COMMON>
__device__ __forceinline__ void expand_main(const ExpandParams& P, unsigned char* smem_raw, const LevelLists& L,
                                            const uint8_t* col_depth_s, uint64_t* mbar_s, uint32_t& phase) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t d = P.depth;
    const uint32_t k = P.plan.nreq[d];
    const uint32_t rb = P.plan.req_begin[d];
    const uint32_t sw = k >= 2 ? P.stage_words : 0;   // only levels with membership tests stage lists
    const WarpMem m = warp_mem(smem_raw, threadIdx.x >> 5, d, k, n_recs(k, DUPS, sw), sw, MODE != kModeLastCount,
                               SHARE ? P.share_words : 0, mbar_s);
    const Tune T = make_tune(P, true);
    const bool share_on = SHARE && T.n_items >= 4ull * P.max_warps;
    ShareState share;

    unsigned long long n_count = 0, n_lookups = 0, n_words = 0, n_parents = 0;
    unsigned long long n_flushed = 0;  // part of n_count already added to tot->count (lane 0)
    PreAcc pre;
    uint32_t last_chunk = 0xffffffffu;   // chunk whose rows are in m.rows_s
    unsigned long long credit = 0;   // level budget held by this warp (lane 0)
    uint32_t nst = 0;
    bool done = !dev::warp_needed(T.n_items);
    while (!done) {
        unsigned long long first = 0;
        if (lane == 0) first = atomicAdd(&P.ctl->claim, (unsigned long long)T.claim_batch);
        first = __shfl_sync(kFull, first, 0);
        if (first >= T.n_items) break;
        const unsigned long long last =
            first + T.claim_batch < T.n_items ? first + T.claim_batch : T.n_items;
        for (unsigned long long item = first; item < last; item++) {
            const uint32_t chunk = item_chunk(P, item);
            if (MODE != kModeMid && P.work_limit && over_limit<MODE>(P, lane, n_count, n_flushed)) {
                done = true;
                break;
            }
            if (MODE == kModeMid) {
                // one lane reads the flag and broadcasts it, so the warp never splits
                int stop = 0;
                if (lane == 0) stop = *(volatile unsigned int*)&P.ctl->stop ? 1 : 0;
                stop = __shfl_sync(kFull, stop, 0);
                if (stop) {
                    if (lane == 0)
                        for (unsigned long long it = item; it < last; it++) defer_chunk(P, item_chunk(P, it));
                    done = true;
                    break;
                }
            }
            bool valid, stage_ok;
            unsigned long long w;
            uint32_t excl, n;
            const uint32_t total = load_chunk<ROOTS, DUPS, SHARE>(P, m, chunk, lane, d, k, rb, T.n_parents, valid, w,
                                                                  phase, stage_ok, excl, n, L, share_on, share);
            last_chunk = chunk;
            if (!stage_ok) {
                done = true;
                break;
            }
            if (MODE == kModeLastCount && !DUPS && k == 1 && !P.pre_count) {
                // Count rule: with one requirement every list entry extends the
                // parent except the parent's own vertices, so each lane counts
                // its parent's extensions as the list length minus the row's
                // vertices found in the list; no candidate is enumerated.
                unsigned long long c = 0;
                if (valid) {
                    const uint4 sg = m.segs_s[lane];
                    c = sg.x - dev::count_members(sg, m.rows_s, lane, d, 0u, false, P.nbr, P.bm, P.bm_words);
                    n_lookups += k;
                    n_words += w;
                    n_parents += 1;
                }
#pragma unroll
                for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(kFull, c, o);
                n_count += c;
                continue;
            }
            if (MODE == kModeMid && total) {
                int ok = 1;
                if (lane == 0) {
                    if (total > credit) {
                        const unsigned long long need = max((unsigned long long)total, (unsigned long long)T.credit_block);
                        const unsigned long long old = atomicAdd(&P.ctl->budget, need);
                        if (old + need > P.ocap) {
                            ok = 0;
                            atomicExch(&P.ctl->stop, 1u);
                            for (unsigned long long it = item; it < last; it++) defer_chunk(P, item_chunk(P, it));
                        } else {
                            credit += need;
                        }
                    }
                    if (ok) credit -= total;
                }
                ok = __shfl_sync(kFull, ok, 0);
                if (!ok) {
                    done = true;
                    break;
                }
            }
            if (valid) {
                n_lookups += k;
                n_words += w;
                n_parents += 1;
            }
            if (total > T.heavy_thresh) {
                // Publish: one packed atomic reserves the entry index and its
                // piece range, so entries are ordered by first piece.  The room
                // check is conservative: at most max_warps publishers are past it.
                int pub = 0;
                const uint32_t np = (total + T.heavy_piece - 1) / T.heavy_piece;
                if (lane == 0 && np <= kHeavyMaxPieces) {
                    const unsigned long long h = *(volatile unsigned long long*)&P.ctl->heavy;
                    if ((uint32_t)(h >> 32) + P.max_warps < P.heavy_cap && (uint32_t)h < (1u << 31)) {
                        const unsigned long long old = atomicAdd(&P.ctl->heavy, (1ull << 32) | np);
                        HeavyEntry e;
                        e.chunk = chunk;
                        e.total = total;
                        e.piece0 = (uint32_t)old;
                        e.pieces = np;
                        P.heavy[(uint32_t)(old >> 32)] = e;
                        pub = 1;
                    }
                }
                pub = __shfl_sync(kFull, pub, 0);
                if (pub) continue;
            }
            process_slots<MODE, ROOTS, DUPS, SHARE, COMMON>(P, m, chunk, excl, n, 0, total, lane, d, k, L,
                                                            col_depth_s, nst, n_count, pre);
        }
    }
    if (MODE != kModeLastCount && nst) flush_stage<MODE, ROOTS>(P, m, nst, lane, d, col_depth_s, last_chunk);
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        n_lookups += __shfl_down_sync(kFull, n_lookups, o);
        n_words += __shfl_down_sync(kFull, n_words, o);
        n_parents += __shfl_down_sync(kFull, n_parents, o);
    }
    if (lane == 0) {
        if (n_parents) {
            atomicAdd(&P.ctl->parents, n_parents);
            atomicAdd(&P.ctl->lookups, n_lookups);
            atomicAdd(&P.ctl->list_words, n_words);
        }
        if (MODE == kModeLastCount && n_count > n_flushed) atomicAdd(&P.tot->count, n_count - n_flushed);
    }
    if (MODE == kModeLastCount && !DUPS && P.pre_count) flush_pre(P, pre, lane);
}

// Heavy pass (after the main pass): every warp claims pieces of the published
// chunks, reloads that chunk and walks its piece of the slots -- the warps
// that finished their own chunks take over the work of the hub chunks.  The
// main pass already holds the chunk's output budget and counted its work.
template <int MODE, bool ROOTS, bool DUPS, bool SHARE, bool COMMON>
__device__ __forceinline__ void expand_heavy(const ExpandParams& P, unsigned char* smem_raw, const LevelLists& L,
                                             const uint8_t* col_depth_s, uint64_t* mbar_s, uint32_t& phase) {
    const unsigned long long h = *(volatile unsigned long long*)&P.ctl->heavy;
    const uint32_t nent = (uint32_t)(h >> 32);
    const uint32_t npieces = (uint32_t)h;
    if (nent == 0 || !dev::warp_needed(npieces)) return;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t d = P.depth;
    const uint32_t k = P.plan.nreq[d];
    const uint32_t rb = P.plan.req_begin[d];
    const uint32_t sw = k >= 2 ? P.stage_words : 0;
    const WarpMem m = warp_mem(smem_raw, threadIdx.x >> 5, d, k, n_recs(k, DUPS, sw), sw, MODE != kModeLastCount,
                               SHARE ? P.share_words : 0, mbar_s);
    const Tune T = make_tune(P, false);
    const bool share_on = SHARE && T.n_items >= 4ull * P.max_warps;
    ShareState share;
    unsigned long long n_count = 0, n_flushed = 0;
    PreAcc pre;
    uint32_t last_chunk = 0xffffffffu;   // chunk whose rows are in m.rows_s
    uint32_t nst = 0;
    for (;;) {
        if (MODE != kModeMid && P.work_limit && over_limit<MODE>(P, lane, n_count, n_flushed)) break;
        unsigned long long gp = 0;
        if (lane == 0) gp = atomicAdd(&P.ctl->claim2, 1ull);
        gp = __shfl_sync(kFull, gp, 0);
        if (gp >= npieces) break;
        uint32_t lo = 0, hi = nent;      // last entry with piece0 <= gp
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (__ldcg(&P.heavy[mid].piece0) <= gp) lo = mid;
            else hi = mid;
        }
        const HeavyEntry e = heavy_entry(P.heavy + lo);
        const uint32_t begin = ((uint32_t)gp - e.piece0) * T.heavy_piece;
        const uint32_t end = min(begin + T.heavy_piece, e.total);
        bool valid, stage_ok;
        unsigned long long w;
        uint32_t excl, n;
        load_chunk<ROOTS, DUPS, SHARE>(P, m, e.chunk, lane, d, k, rb, T.n_parents, valid, w, phase, stage_ok, excl, n,
                                       L, share_on, share);
        last_chunk = e.chunk;
        if (!stage_ok) break;
        process_slots<MODE, ROOTS, DUPS, SHARE, COMMON>(P, m, e.chunk, excl, n, begin, end, lane, d, k, L,
                                                        col_depth_s, nst, n_count, pre);
    }
    if (MODE != kModeLastCount && nst) flush_stage<MODE, ROOTS>(P, m, nst, lane, d, col_depth_s, last_chunk);
    if (MODE == kModeLastCount && lane == 0 && n_count > n_flushed) atomicAdd(&P.tot->count, n_count - n_flushed);
    if (MODE == kModeLastCount && !DUPS && P.pre_count) flush_pre(P, pre, lane);
}

// ------------------------------------------------------ pre-count by sums
//
// The counting level d = q - 2 with one back edge: its candidates x are the
// list A = N_l(r_a) of one row vertex, and the last depth's extensions of x are
// a list N_l'(x) (a chain) or N_l'(r_b) (a star or a fork), without the row and
// x.  Summed over x, no candidate is looked at:
//   chain: sum over x in A \ row of |N_l'(x)|, minus for every row vertex u the
//          x in A \ row with u in N_l'(x); on a graph whose e-lines come in both
//          directions these are (A and N_l'(u)) \ row, an intersection of two
//          lists;
//   fork:  |A \ row| * |N_l'(r_b) \ row| - |(A \ row) and N_l'(r_b)|.
// The sum of |N_l'(x)| over A and the size of A and N_l'(r_a) depend on r_a
// alone (ExpandParams::vsum, one pass over the label's lists), so a parent
// costs its row, two records, the row's members of A (rare) and, for each
// other row vertex, the shorter of two lists.  The work counters of the last
// depth come from the same sums.
//
// Bound by the intersections' dependent loads.  A 5-vertex path on a 2^22-vertex
// R-MAT graph with 64 labels (1.2e8 parents with 3.4e9 candidates): 14.4 ms as a chain, 6.5 ms as a fork,
// against 85.0 ms candidate by candidate.

// Intersection of A with the last label's list of row vertex u: the shorter
// list drives.  Returns the chunk's candidate slots (warp-uniform).
__device__ __forceinline__ uint32_t sum_lists(const ExpandParams& P, const WarpMem& m, uint32_t lane, uint32_t u,
                                              const uint4* last, bool live, uint32_t& excl, uint32_t& n) {
    uint4 b = make_uint4(0, 0, 0, 0);
    uint32_t drv = 0;
    n = 0;
    if (live) {
        b = ldg4(last + m.rows_s[u * 32 + lane]);
        const uint32_t na = m.segs_s[lane].x;
        drv = b.x < na ? 1u : 0u;
        n = min(na, b.x);
    }
    m.segs_s[32 + lane] = b;
    uint32_t incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, incl, o);
        if ((int)lane >= o) incl += t;
    }
    excl = incl - n;
    m.drv_s[lane] = (uint8_t)drv;
    __syncwarp();
    return __shfl_sync(kFull, incl, 31);
}

struct SumPlan {
    uint32_t anc, last_anc;          // a, b (b == d: the new vertex, a chain)
    bool same;                       // fork of one vertex by one label: both lists are A
    const uint4* seg;                // records of l
    const uint4* last;               // records of l'
    dev::FilterSlice seg_f, last_f;
};

__device__ __forceinline__ SumPlan sum_plan(const ExpandParams& P) {
    const uint32_t d = P.depth, rb = P.plan.req_begin[d], rl = P.plan.req_begin[d + 1];
    SumPlan s;
    s.anc = P.plan.req_anc[rb];
    s.last_anc = P.plan.req_anc[rl];
    s.same = s.last_anc == s.anc && P.plan.req_label[rb] == P.plan.req_label[rl];
    s.seg = P.seg + (uint64_t)P.plan.req_label[rb] * P.V;
    s.last = P.seg + (uint64_t)P.plan.req_label[rl] * P.V;
    s.seg_f = dev::filter_slice(P.efilter, P.efilter_off, P.plan.req_label[rb]);
    s.last_f = dev::filter_slice(P.efilter, P.efilter_off, P.plan.req_label[rl]);
    return s;
}

// Members of A and the last label's list of row vertex w, outside the row, over
// slots [begin, end) (lane-private).
__device__ __forceinline__ uint32_t sum_slots(const ExpandParams& P, const WarpMem& m, const SumPlan& sp, uint32_t w,
                                              uint32_t excl, uint32_t n, uint32_t begin, uint32_t end, uint32_t lane,
                                              uint32_t d) {
    uint32_t hits = 0, pend = 0;
    SlotWalk walk(m.start_s, excl, n, begin, lane);
    for (uint32_t base = begin; base < end; base += 32 * kSlots) {
        uint32_t j[kSlots], t[kSlots], x[kSlots];
        bool ok[kSlots], b[kSlots];      // b: the last label's list drives
#pragma unroll
        for (uint32_t u = 0; u < kSlots; u++) {
            walk.window(m.start_s, base + 32 * u, lane, j[u], t[u]);
            x[u] = 0;
            b[u] = false;
            ok[u] = base + 32 * u + lane < end;
            if (ok[u]) {
                b[u] = m.drv_s[j[u]] != 0;
                x[u] = seg_at(m.segs_s[(b[u] ? 32 : 0) + j[u]], t[u], P.nbr);
            }
        }
#pragma unroll
        for (uint32_t u = 0; u < kSlots; u++) {
            if (ok[u])
                ok[u] = dev::filter_has(b[u] ? sp.seg_f : sp.last_f,
                                        dev::filter_seed(m.rows_s[(b[u] ? sp.anc : w) * 32 + j[u]]), x[u]);
            const unsigned bl = __ballot_sync(kFull, ok[u]);
            if (ok[u]) {
                const uint32_t q = pend + __popc(bl & ((1u << lane) - 1u));
                m.px[q] = x[u];
                m.pj[q] = (uint8_t)j[u];
            }
            pend += __popc(bl);
        }
        const bool last = base + 32 * kSlots >= end;
        while (pend >= 32 || (last && pend)) {
            const uint32_t take = min(pend, 32u);
            pend -= take;
            __syncwarp();
            if (lane < take) {
                const uint32_t jj = m.pj[pend + lane], xx = m.px[pend + lane];
                bool in = seg_has(m.segs_s[(m.drv_s[jj] ? 0 : 32) + jj], xx, 1, P.nbr, P.bm, P.bm_words);
                for (uint32_t c = 0; c < d && in; c++) in = m.rows_s[c * 32 + jj] != xx;
                hits += in ? 1u : 0u;
            }
        }
        __syncwarp();
    }
    __syncwarp();
    return hits;
}

__device__ __forceinline__ bool sum_rule_on(const ExpandParams& P, unsigned long long n_parents) {
    return P.sum_rule == 2 || (P.sum_rule == 1 && 4 * n_parents >= P.sum_heads);
}

// Row and list A of the chunk's parents.
__device__ __forceinline__ bool sum_load(const ExpandParams& P, const WarpMem& m, const SumPlan& sp, uint32_t chunk,
                                         uint32_t lane, uint32_t d, unsigned long long n_parents) {
    const uint64_t p = (uint64_t)chunk * 32 + lane;
    const bool valid = p < n_parents;
    for (uint32_t c = 0; c < d; c++) m.rows_s[c * 32 + lane] = valid ? __ldcg(P.pin + c * P.pstride + p) : 0u;
    m.segs_s[lane] = valid ? ldg4(sp.seg + m.rows_s[sp.anc * 32 + lane]) : make_uint4(0, 0, 0, 0);
    return valid;
}

// The row vertices whose last-label lists are intersected with A: for a chain
// every one but r_a, for a fork r_b unless the vertex sums hold the answer.
__device__ __forceinline__ bool sum_needs(const SumPlan& sp, uint32_t d, uint32_t u) {
    return sp.last_anc == d ? u != sp.anc : (u == sp.last_anc && u != sp.anc);
}

__device__ __forceinline__ void expand_sum_main(const ExpandParams& P, unsigned char* smem_raw, uint64_t* mbar_s) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t d = P.depth;
    const WarpMem m = warp_mem(smem_raw, threadIdx.x >> 5, d, 2, 2, 0, false, 0, mbar_s);
    const Tune T = make_tune(P, true);
    const SumPlan sp = sum_plan(P);
    const bool chain = sp.last_anc == d;
    unsigned long long n_count = 0, n_parents = 0, n_words = 0;   // lane-private
    PreAcc pre;
    while (dev::warp_needed(T.n_items)) {
        unsigned long long first = 0;
        if (lane == 0) first = atomicAdd(&P.ctl->claim, (unsigned long long)T.claim_batch);
        first = __shfl_sync(kFull, first, 0);
        if (first >= T.n_items) break;
        const unsigned long long last = first + T.claim_batch < T.n_items ? first + T.claim_batch : T.n_items;
        for (unsigned long long item = first; item < last; item++) {
            const uint32_t chunk = item_chunk(P, item);
            const bool valid = sum_load(P, m, sp, chunk, lane, d, T.n_parents);
            const uint4 a = m.segs_s[lane];
            n_parents += valid ? 1u : 0u;
            n_words += a.x;
            const bool live = a.x > 0;
            if (live) {
                const uint32_t va = m.rows_s[sp.anc * 32 + lane];
                uint32_t in_a = dev::member_mask(a, m.rows_s, lane, d, sp.anc, sp.seg_f, va, P.nbr, P.bm, P.bm_words);
                const unsigned long long free_a = a.x - __popc(in_a);
                pre.parents += free_a;
                if (chain) {
                    const uint2 w = __ldcg(P.vsum + va);
                    unsigned long long words = w.x, c = (unsigned long long)w.x - w.y;
                    if (in_a) {
                        const uint4 own = ldg4(sp.last + va);
                        for (; in_a; in_a &= in_a - 1) {
                            const uint32_t v = m.rows_s[(__ffs(in_a) - 1) * 32 + lane];
                            const uint32_t dv = __ldg(&sp.last[v].x);
                            words -= dv;
                            c -= dv;
                            c += seg_has(own, v, 1, P.nbr, P.bm, P.bm_words) ? 1u : 0u;
                        }
                    }
                    pre.words += words;
                    n_count += c;
                } else {
                    const uint32_t vb = m.rows_s[sp.last_anc * 32 + lane];
                    const uint4 b = ldg4(sp.last + vb);
                    const uint32_t in_b =
                        dev::member_mask(b, m.rows_s, lane, d, sp.last_anc, sp.last_f, vb, P.nbr, P.bm, P.bm_words);
                    n_count += free_a * (b.x - __popc(in_b));
                    pre.words += free_a * b.x;
                    if (sp.same) n_count -= free_a;
                    else if (sp.last_anc == sp.anc) n_count -= __ldcg(&P.vsum[va].y) - __popc(in_a & in_b);
                }
            }
            for (uint32_t u = 0; u < d; u++) {
                if (!sum_needs(sp, d, u)) continue;
                uint32_t excl, n;
                const uint32_t total = sum_lists(P, m, lane, u, sp.last, live, excl, n);
                if (total > T.heavy_thresh) {
                    int pub = 0;
                    const uint32_t np = (total + T.heavy_piece - 1) / T.heavy_piece;
                    if (lane == 0 && np <= kHeavyMaxPieces) {
                        const unsigned long long h = *(volatile unsigned long long*)&P.ctl->heavy;
                        if ((uint32_t)(h >> 32) + P.max_warps < P.heavy_cap && (uint32_t)h < (1u << 31)) {
                            const unsigned long long old = atomicAdd(&P.ctl->heavy, (1ull << 32) | np);
                            HeavyEntry e;
                            e.chunk = chunk;
                            e.total = total;
                            e.piece0 = (uint32_t)old;
                            e.pieces = np | (u << 24);
                            P.heavy[(uint32_t)(old >> 32)] = e;
                            pub = 1;
                        }
                    }
                    pub = __shfl_sync(kFull, pub, 0);
                    if (pub) {
                        __syncwarp();
                        continue;
                    }
                }
                n_count -= sum_slots(P, m, sp, u, excl, n, 0, total, lane, d);
            }
            __syncwarp();
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        n_count += __shfl_xor_sync(kFull, n_count, o);
        n_parents += __shfl_xor_sync(kFull, n_parents, o);
        n_words += __shfl_xor_sync(kFull, n_words, o);
    }
    if (lane == 0 && n_parents) {
        atomicAdd(&P.ctl->parents, n_parents);
        atomicAdd(&P.ctl->lookups, n_parents);
        atomicAdd(&P.ctl->list_words, n_words);
        atomicAdd(&P.tot->count, n_count);
    }
    flush_pre(P, pre, lane);
}

__device__ __forceinline__ void expand_sum_heavy(const ExpandParams& P, unsigned char* smem_raw, uint64_t* mbar_s) {
    const unsigned long long h = *(volatile unsigned long long*)&P.ctl->heavy;
    const uint32_t nent = (uint32_t)(h >> 32);
    const uint32_t npieces = (uint32_t)h;
    if (nent == 0 || !dev::warp_needed(npieces)) return;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t d = P.depth;
    const WarpMem m = warp_mem(smem_raw, threadIdx.x >> 5, d, 2, 2, 0, false, 0, mbar_s);
    const Tune T = make_tune(P, false);
    const SumPlan sp = sum_plan(P);
    unsigned long long hits = 0;
    for (;;) {
        unsigned long long gp = 0;
        if (lane == 0) gp = atomicAdd(&P.ctl->claim2, 1ull);
        gp = __shfl_sync(kFull, gp, 0);
        if (gp >= npieces) break;
        uint32_t lo = 0, hi = nent;      // last entry with piece0 <= gp
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (__ldcg(&P.heavy[mid].piece0) <= gp) lo = mid;
            else hi = mid;
        }
        const HeavyEntry e = heavy_entry(P.heavy + lo);
        const uint32_t begin = ((uint32_t)gp - e.piece0) * T.heavy_piece;
        const uint32_t end = min(begin + T.heavy_piece, e.total);
        sum_load(P, m, sp, e.chunk, lane, d, T.n_parents);
        uint32_t excl, n;
        sum_lists(P, m, lane, e.pieces >> 24, sp.last, m.segs_s[lane].x > 0, excl, n);
        hits += sum_slots(P, m, sp, e.pieces >> 24, excl, n, begin, end, lane, d);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) hits += __shfl_xor_sync(kFull, hits, o);
    if (lane == 0 && hits) atomicAdd(&P.tot->count, 0ull - hits);
}

// Vertex sums (ExpandParams::vsum) of the lists of one label: a warp takes the
// lists of 32 vertices as one range of slots; longer lists are left to the
// whole block.
constexpr uint32_t kSumLong = 1024;

__global__ void __launch_bounds__(kWarps * 32) k_vertex_sums(const __grid_constant__ ExpandParams P,
                                                             const uint32_t* __restrict__ heads, uint32_t n,
                                                             uint32_t label, uint32_t last_label,
                                                             uint2* __restrict__ vsum,
                                                             const unsigned long long* parents) {
    __shared__ uint2 start_s[kWarps][32];
    __shared__ uint32_t sum_s[kWarps][32], both_s[kWarps][32], v_s[kWarps][32];
    __shared__ uint32_t long_s[kWarps * 32], n_long, lsum, lboth;
    dev::pass_begin();
    dev::pass_wait();
    if (parents && !sum_rule_on(P, *(const volatile unsigned long long*)parents)) return;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint4* seg = P.seg + (uint64_t)label * P.V;
    const uint4* last = P.seg + (uint64_t)last_label * P.V;
    const dev::FilterSlice lf = dev::filter_slice(P.efilter, P.efilter_off, last_label);
    if (threadIdx.x == 0) n_long = 0;
    __syncthreads();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    uint4 a = make_uint4(0, 0, 0, 0);
    uint32_t v = 0;
    if (i < n) {
        v = heads[i];
        a = ldg4(seg + v);
    }
    const bool big = a.x > kSumLong;
    if (big) long_s[atomicAdd(&n_long, 1u)] = v;
    const uint32_t len = big ? 0u : a.x;
    uint32_t incl = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, incl, o);
        if ((int)lane >= o) incl += t;
    }
    sum_s[warp][lane] = both_s[warp][lane] = 0;
    v_s[warp][lane] = v;
    const uint32_t total = __shfl_sync(kFull, incl, 31);
    SlotWalk walk(start_s[warp], incl - len, len, 0, lane);
    for (uint32_t base = 0; base < total; base += 32) {
        uint32_t j, t;
        walk.window(start_s[warp], base, lane, j, t);
        if (base + lane >= total) continue;
        const uint32_t vj = v_s[warp][j];
        const uint32_t x = seg_at(ldg4(seg + vj), t, P.nbr);
        const uint32_t w = __ldg(&last[x].x);
        if (w) atomicAdd(&sum_s[warp][j], w);
        if (label == last_label || (dev::filter_has(lf, dev::filter_seed(vj), x) &&
                                    seg_has(ldg4(last + vj), x, 1, P.nbr, P.bm, P.bm_words)))
            atomicAdd(&both_s[warp][j], 1u);
    }
    __syncwarp();
    if (len) vsum[v] = make_uint2(sum_s[warp][lane], both_s[warp][lane]);
    __syncthreads();
    for (uint32_t k = 0; k < n_long; k++) {
        if (threadIdx.x == 0) lsum = lboth = 0;
        __syncthreads();
        const uint32_t vk = long_s[k];
        const uint4 ak = ldg4(seg + vk), own = ldg4(last + vk);
        uint32_t sum = 0, both = 0;
        for (uint32_t t = threadIdx.x; t < ak.x; t += blockDim.x) {
            const uint32_t x = seg_at(ak, t, P.nbr);
            sum += __ldg(&last[x].x);
            both += (label == last_label || seg_has(own, x, 1, P.nbr, P.bm, P.bm_words)) ? 1u : 0u;
        }
        sum = __reduce_add_sync(kFull, sum);
        both = __reduce_add_sync(kFull, both);
        if (lane == 0) {
            atomicAdd(&lsum, sum);
            atomicAdd(&lboth, both);
        }
        __syncthreads();
        if (threadIdx.x == 0) vsum[vk] = make_uint2(lsum, lboth);
        __syncthreads();
    }
}

// Blocks per SM a pass is compiled for.  Closing and counting levels, which hold
// most of a large match's work, want every warp they can get (6 blocks, 40
// registers, spilling 100 to 400 bytes; 4 blocks: closing a 4-cycle 12 % slower;
// 5 for table levels: 4-vertex stars 2 % faster, closing a 4-cycle 4 % slower).
// Middle levels of walk queries are mostly small, and there fewer warps, which
// spill nothing (with shared intersections 84 bytes), and fewer blocks to start
// win: 4 blocks (64 registers) took a 13-vertex walk's match from 312 to
// 267 us and left the large ones where they were (4-cycle 1069 and 1057 us, 3
// blocks: 8-vertex walks and 4-cliques slower again).
constexpr int min_blocks(int mode) { return mode == kModeMid ? 4 : 6; }

template <int MODE, bool ROOTS, bool DUPS, bool SHARE, bool COMMON>
__global__ void __launch_bounds__(kWarps * 32, min_blocks(MODE)) k_expand(const __grid_constant__ ExpandParams P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint8_t col_depth_s[kMaxQ];
    __shared__ uint64_t mbar_s[kWarps];
    __shared__ LevelLists L;
    dev::pass_begin();
    level_lists_init(P, L, P.depth);
    if (threadIdx.x < (unsigned)kMaxQ) col_depth_s[threadIdx.x] = P.plan.col_depth[threadIdx.x];
    dev::stage_barriers_init(mbar_s);
    dev::pass_wait();
    if (MODE == kModeLastCount && !ROOTS && !DUPS && !SHARE && P.sum_rule &&
        sum_rule_on(P, make_tune(P, true).n_parents)) {
        expand_sum_main(P, smem_raw, mbar_s);
        return;
    }
    uint32_t phase = 0;
    expand_main<MODE, ROOTS, DUPS, SHARE, COMMON>(P, smem_raw, L, col_depth_s, mbar_s, phase);
}

template <int MODE, bool ROOTS, bool DUPS, bool SHARE, bool COMMON>
__global__ void __launch_bounds__(kWarps * 32, min_blocks(MODE))
    k_expand_heavy(const __grid_constant__ ExpandParams P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint8_t col_depth_s[kMaxQ];
    __shared__ uint64_t mbar_s[kWarps];
    __shared__ LevelLists L;
    dev::pass_begin();
    level_lists_init(P, L, P.depth);
    if (threadIdx.x < (unsigned)kMaxQ) col_depth_s[threadIdx.x] = P.plan.col_depth[threadIdx.x];
    dev::stage_barriers_init(mbar_s);
    dev::pass_wait();
    if (MODE == kModeLastCount && !ROOTS && !DUPS && !SHARE && P.sum_rule &&
        sum_rule_on(P, make_tune(P, false).n_parents)) {
        expand_sum_heavy(P, smem_raw, mbar_s);
        return;
    }
    uint32_t phase = 0;
    expand_heavy<MODE, ROOTS, DUPS, SHARE, COMMON>(P, smem_raw, L, col_depth_s, mbar_s, phase);
}

// ------------------------------------------------------- persistent engine
//
// One cooperative launch runs every level pass of the match.  A pass of depth
// d is the same main and heavy pass as above, on the work items of the
// depth-d queue: the deferred ring of depth d (chunks pushed back when the
// output level filled) followed by the fresh chunks not yet claimed.  Between
// passes block 0 advances the schedule (dev::sched_advance), so a level whose
// output buffer fills is drained depth first on the device, with no host
// round trip; a level whose chunks are long is cut into pieces that every warp
// takes in the heavy pass.

template <int LAST, bool DUPS>
__device__ __forceinline__ void persist_main(const ExpandParams& P, unsigned char* smem, const uint8_t* cd,
                                             bool roots, bool last, const LevelLists& L, uint64_t* mb, uint32_t& ph) {
    if (last) {
        if (roots) expand_main<LAST, true, DUPS, false, true>(P, smem, L, cd, mb, ph);
        else expand_main<LAST, false, DUPS, false, true>(P, smem, L, cd, mb, ph);
    } else {
        if (roots) expand_main<kModeMid, true, DUPS, false, true>(P, smem, L, cd, mb, ph);
        else expand_main<kModeMid, false, DUPS, false, true>(P, smem, L, cd, mb, ph);
    }
}

template <int LAST, bool DUPS>
__device__ __forceinline__ void persist_heavy(const ExpandParams& P, unsigned char* smem, const uint8_t* cd,
                                              bool roots, bool last, const LevelLists& L, uint64_t* mb, uint32_t& ph) {
    if (last) {
        if (roots) expand_heavy<LAST, true, DUPS, false, true>(P, smem, L, cd, mb, ph);
        else expand_heavy<LAST, false, DUPS, false, true>(P, smem, L, cd, mb, ph);
    } else {
        if (roots) expand_heavy<kModeMid, true, DUPS, false, true>(P, smem, L, cd, mb, ph);
        else expand_heavy<kModeMid, false, DUPS, false, true>(P, smem, L, cd, mb, ph);
    }
}

template <int LAST, bool DUPS>
__global__ void __launch_bounds__(kWarps * 32, 5) k_persist(const __grid_constant__ ExpandParams P0,
                                                            const __grid_constant__ PersistArgs A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(16) ExpandParams P;          // level fields change per pass
    __shared__ uint8_t col_depth_s[kMaxQ];
    __shared__ unsigned flag_s, cur_s;
    __shared__ uint64_t mbar_s[kWarps];
    __shared__ LevelLists L;
    SchedState* S = A.sched;
    {
        const uint32_t* src = (const uint32_t*)&P0;
        uint32_t* dst = (uint32_t*)&P;
        for (uint32_t i = threadIdx.x; i < sizeof(ExpandParams) / 4; i += blockDim.x) dst[i] = src[i];
    }
    if (threadIdx.x < (unsigned)kMaxQ) col_depth_s[threadIdx.x] = P0.plan.col_depth[threadIdx.x];
    dev::stage_barriers_init(mbar_s);
    uint32_t phase = 0;       // of this warp's stage barrier, carried across passes
    const uint32_t q = P0.plan.q;
    bool first = true;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned d = *(volatile unsigned*)&S->cur;
            if (*(volatile unsigned*)&S->error) d = 0;
            cur_s = d;
            if (d) {
                const volatile SchedLevel* L = &S->lv[d];
                const unsigned long long ring = L->tail - L->head;
                const unsigned long long n_chunks = (L->n_parents + 31) / 32;
                P.depth = d;
                P.pin = d == 1 ? nullptr : A.levels[d];
                P.pout = d + 1 + P0.pre_count < q ? A.levels[d + 1] : nullptr;
                P.n_parents = L->n_parents;
                P.ndef_in = (uint32_t)ring;
                P.fresh_base = L->fresh;
                P.n_items = ring + (n_chunks - L->fresh);
                P.def_in = A.rings + (uint64_t)d * A.ring_cap;
                P.def_out = A.rings + (uint64_t)d * A.ring_cap;
                P.def_cap = A.ring_cap;
                P.def_in_pos = L->head;
                P.def_out_pos = L->tail;
                P.def_room = A.ring_cap - (uint32_t)ring;
                P.ctl = P0.ctl + d;
            }
        }
        __syncthreads();
        const unsigned d = cur_s;
        if (d == 0) break;
        const bool roots = d == 1, last = d + 1 + P0.pre_count == q;
        level_lists_init(P, L, d);
        persist_main<LAST, DUPS>(P, smem_raw, col_depth_s, roots, last, L, mbar_s, phase);
        if (!dev::grid_barrier(S, first && A.hold_first_barrier && blockIdx.x == 0, &flag_s)) break;
        first = false;
        persist_heavy<LAST, DUPS>(P, smem_raw, col_depth_s, roots, last, L, mbar_s, phase);
        if (!dev::grid_barrier(S, false, &flag_s)) break;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            const bool limit_hit = P.work_limit && (*(volatile unsigned*)&P.tot->error & kLimitFlag);
            dev::sched_advance(S, P0.ctl, d, !last, P.n_items, P.ndef_in, P.def_room, limit_hit);
        }
        if (!dev::grid_barrier(S, false, &flag_s)) break;
    }
}

template <int MODE, bool ROOTS, bool DUPS, bool SHARE = false, bool COMMON = false>
void* kernel_ptr(bool heavy) {
    return heavy ? (void*)&k_expand_heavy<MODE, ROOTS, DUPS, SHARE, COMMON>
                 : (void*)&k_expand<MODE, ROOTS, DUPS, SHARE, COMMON>;
}

// `share`: the level has a buffer for shared intersections; `common`: bitmaps are
// common (DeviceGraph::bitmaps_common).  A counting level on a graph without them
// has a kernel of its own: the code that asks them cost it 2 to 4 % (5-vertex path
// counted candidate by candidate, 2^16 vertices with lists of 8: 0.514 and 0.501 ms).
void* pick(int mode, bool roots, bool dups, bool share, bool common, bool heavy) {
    if (common && mode == kModeLastCount && !roots && !dups && !share)
        return kernel_ptr<kModeLastCount, false, false, false, true>(heavy);
#define FM_PICK(M)                                                                                     \
    if (mode == M) {                                                                                   \
        if (share) return kernel_ptr<M, false, false, true>(heavy);                                    \
        if (roots) return dups ? kernel_ptr<M, true, true>(heavy) : kernel_ptr<M, true, false>(heavy); \
        return dups ? kernel_ptr<M, false, true>(heavy) : kernel_ptr<M, false, false>(heavy);          \
    }
    FM_PICK(kModeMid)
    FM_PICK(kModeLastTable)
    FM_PICK(kModeLastCount)
#undef FM_PICK
    return nullptr;
}

void* persist_ptr(int last_mode, bool dups) {
    if (last_mode == kModeLastTable) return dups ? (void*)&k_persist<kModeLastTable, true> : (void*)&k_persist<kModeLastTable, false>;
    return dups ? (void*)&k_persist<kModeLastCount, true> : (void*)&k_persist<kModeLastCount, false>;
}

}  // namespace

namespace {
// Initial schedule: every pass starts at depth 1 on n_roots root rows.  A
// kernel rather than a host copy, so a captured CUDA graph replays it.
__global__ void k_sched_init(SchedState* S, unsigned q, unsigned long long n_roots, unsigned long long work_limit,
                             unsigned long long wait_ns) {
    unsigned* w = (unsigned*)S;
    for (unsigned i = threadIdx.x; i < sizeof(SchedState) / 4; i += blockDim.x) w[i] = 0;
    __syncthreads();
    if (threadIdx.x == 0) {
        S->cur = 1;
        S->q = q;
        S->work_limit = work_limit;
        S->wait_limit_ns = wait_ns;
        S->lv[1].n_parents = n_roots;
    }
}
}  // namespace

cudaError_t launch_sched_init(SchedState* S, unsigned q, unsigned long long n_roots, unsigned long long work_limit,
                              unsigned long long wait_ns, cudaStream_t s) {
    k_sched_init<<<1, 128, 0, s>>>(S, q, n_roots, work_limit, wait_ns);
    return cudaGetLastError();
}

size_t persist_smem_bytes(const DevPlan& plan, const uint32_t* nreq_depth, uint32_t stage_words) {
    size_t best = 0;
    for (uint32_t d = 1; d < plan.q; d++)
        best = std::max<size_t>(best, per_warp_bytes(d, nreq_depth[d], nreq_depth[d],
                                                     nreq_depth[d] >= 2 ? stage_words : 0, true, 0));
    return best * kWarps;
}

int persist_blocks_per_sm(int last_mode, bool dups, size_t smem) {
    void* f = persist_ptr(last_mode, dups);
    allow_dynamic_smem(f);
    return blocks_per_sm(f, kWarps * 32, smem);
}

cudaError_t launch_persist(const ExpandParams& p, const PersistArgs& a, int last_mode, bool dups, int grid,
                           size_t smem, cudaStream_t s) {
    ExpandParams q = p;
    q.max_warps = (uint32_t)grid * kWarps;
    q.n_parents_dev = nullptr;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kWarps * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void* args[] = {(void*)&q, (void*)&a};
    return cudaLaunchKernelExC(&cfg, persist_ptr(last_mode, dups), args);
}

// One launch; `overlap`: may start while the launch before it drains (see
// dev::pass_wait).
cudaError_t launch_pass(const void* f, int grid, int block, size_t smem, void** args, bool overlap, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelExC(&cfg, f, args);
}

cudaError_t launch_vertex_sums(const ExpandParams& p, const uint32_t* heads, uint32_t n, uint32_t label,
                               uint32_t last_label, uint2* vsum, const unsigned long long* parents, cudaStream_t s) {
    if (!n) return cudaSuccess;
    void* args[] = {(void*)&p, (void*)&heads, (void*)&n, (void*)&label, (void*)&last_label, (void*)&vsum, (void*)&parents};
    return launch_pass((const void*)&k_vertex_sums, (int)((n + kWarps * 32 - 1) / (kWarps * 32)), kWarps * 32, 0, args,
                       parents != nullptr, s);
}

size_t expand_smem_bytes(uint32_t depth, uint32_t nreq, int warps, uint32_t stage_words, bool staged, bool dups,
                         bool sums, bool share) {
    return (size_t)warps * per_warp_bytes(depth, sums ? 2 : nreq, sums ? 2 : n_recs(nreq, dups, stage_words), stage_words,
                                          staged, share ? kShareWords : 0);
}

void allow_dynamic_smem(const void* f) {
    // Raised once per (device, kernel) to the opt-in maximum: a per-launch
    // value would race between host threads launching with different sizes.
    static std::mutex mu;
    static std::set<std::pair<int, const void*>> done;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    if (!done.insert({dev, f}).second) return;
    int optin = 0;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, f) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    // static shared memory counts against the same opt-in limit
    const int dyn = optin - (int)fa.sharedSizeBytes;
    if (dyn > 0 && cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) != cudaSuccess)
        cudaGetLastError();   // the launch reports a size it cannot take
}

int blocks_per_sm(const void* f, int block, size_t smem) {
    static std::mutex mu;
    static std::map<std::tuple<int, const void*, int, size_t>, int> known;   // kernels x shared memory sizes
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    auto it = known.find({dev, f, block, smem});
    if (it != known.end()) return it->second;
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, f, block, smem) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    known[{dev, f, block, smem}] = n;
    return n;
}

int expand_blocks_per_sm(int mode, bool roots, bool dups, bool share, bool common, size_t smem, int block) {
    void* f = pick(mode, roots, dups, share, common, false);
    allow_dynamic_smem(f);
    allow_dynamic_smem(pick(mode, roots, dups, share, common, true));
    return std::max(1, blocks_per_sm(f, block, smem));
}

uint32_t expand_launches(uint32_t max_list) { return 32ull * max_list <= kHeavyLeast ? 1 : 2; }

cudaError_t launch_expand(const ExpandParams& p, int mode, bool roots, bool dups, bool share, bool overlap, int grid,
                          int heavy_grid, int block, size_t smem, cudaStream_t s) {
    void* f = pick(mode, roots, dups, share, p.bm_common != 0, false);
    void* fh = pick(mode, roots, dups, share, p.bm_common != 0, true);
    if (!f || !fh) return cudaErrorInvalidValue;
    ExpandParams q = p;
    // both passes tune themselves on the device (make_tune) from the level size
    // and from max_warps, the warps of the heavy pass
    q.max_warps = (uint32_t)heavy_grid * (uint32_t)(block / 32);
    q.share_words = share ? kShareWords : 0;
    void* args[] = {(void*)&q};
    cudaError_t e = launch_pass(f, grid, block, smem, args, overlap, s);
    if (e != cudaSuccess || expand_launches(p.max_list) == 1) return e;
    // the heavy pass always gets a full grid: a few heavy chunks can hold most of the work
    return launch_pass(fh, heavy_grid, block, smem, args, overlap, s);
}

}  // namespace fm
