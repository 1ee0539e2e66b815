// fm_graph.cu -- device build of the resident data graph.
//
// The reference builds one global CSR over (label, src) sorted by
// (label, src, dst), indexed through a per-label 32-vertex presence bitmap plus
// popcount rank (src/trie.cuh:138-311, 697-795, 898-942): a lookup costs two
// dependent loads before the list itself.  Here every (label, vertex) pair has a
// 16-byte segment record in a dense [label][vertex] table, so a lookup is one
// vectorised load; lists of up to 3 neighbours live inside the record (no
// second access), longer lists start on a 16-byte boundary in `nbr`.
//
// The e-lines become 64-bit keys (label, src, dst); after a radix sort (CUB:
// graph build is not on the matching path) a segment is a run of equal upper
// bits.  Three passes over the sorted keys, each at streaming bandwidth, find
// the runs: a warp flags the heads of 512 consecutive keys with ballots, so a
// key's segment number is a tile base plus popcounts and no per-key array of
// flags or ranks is written (16 M e-lines: 124 us for every pass between the
// sort and k_place, 418 us with flag and rank arrays).  Every temporary comes from one allocation
// (BuildArena) and every resident array from another: on this machine a pair
// of cudaMalloc and cudaFree costs 0.2-0.5 ms, more than most of the kernels.
#include <algorithm>
#include <cstddef>
#include <cstdlib>

#include <cub/cub.cuh>

#include "fm_device.cuh"

namespace fm {
namespace {

constexpr int kBlock = 256;
constexpr uint32_t kWarpKeys = 512;                         // consecutive keys of one warp
constexpr uint32_t kRounds = kWarpKeys / 32;
constexpr uint32_t kTileKeys = kWarpKeys * (kBlock / 32);   // keys of one block
constexpr uint32_t kTileSegs = 4 * kBlock;                  // segments of one block

// e-lines -> sort keys, range checks, label frequencies.  The histogram is
// kept in shared memory: on the host the same count took 6.8 ms for 16 M
// e-lines (one dependent increment per e-line), half of the whole build.
__global__ void k_make_keys(const uint32_t* __restrict__ src, const uint32_t* __restrict__ dst,
                            const uint32_t* __restrict__ lab, uint64_t E, uint32_t V, uint32_t L,
                            uint32_t vbits, uint64_t* __restrict__ keys, BuildStats* __restrict__ st) {
    __shared__ unsigned int h[FM_MAX_LABEL + 1];
    for (uint32_t i = threadIdx.x; i <= FM_MAX_LABEL; i += blockDim.x) h[i] = 0;
    __syncthreads();
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < E; i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t s = src[i], d = dst[i], l = lab[i];
        if (s >= V || d >= V || l >= L) {
            atomicOr(&st->error, 1u);
            s = d = l = 0;
        } else if (s == d) {
            atomicOr(&st->loops, 1u);
        }
        atomicAdd(&h[l], 1u);
        keys[i] = ((uint64_t)l << (2 * vbits)) | ((uint64_t)s << vbits) | (uint64_t)d;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i <= FM_MAX_LABEL; i += blockDim.x)
        if (h[i]) atomicAdd(&st->label_count[i], (unsigned long long)h[i]);
}

// Head flags of the 512 keys from `base` (one ballot per 32 keys): key i is a
// head when its (label, src) differs from key i - 1's.  Returns the heads.
__device__ __forceinline__ uint32_t head_ballots(const uint64_t* __restrict__ keys, uint64_t base, uint64_t E,
                                                 uint32_t vbits, uint32_t lane, uint32_t (&b)[kRounds], bool& dup) {
    uint64_t carry = base > 0 && base < E ? keys[base - 1] : 0;
    uint32_t n = 0;
#pragma unroll
    for (uint32_t j = 0; j < kRounds; j++) {
        const uint64_t i = base + 32 * j + lane;
        const uint64_t k = i < E ? keys[i] : 0;
        uint64_t p = __shfl_up_sync(0xffffffffu, k, 1);
        if (lane == 0) p = carry;
        carry = __shfl_sync(0xffffffffu, k, 31);
        const bool in = i < E;
        b[j] = __ballot_sync(0xffffffffu, in && (i == 0 || (k >> vbits) != (p >> vbits)));
        dup |= in && i > 0 && k == p;
        n += __popc(b[j]);
    }
    return n;
}

// Segment heads per tile; a repeated key sets the duplicate flag.
__global__ void k_tile_heads(const uint64_t* __restrict__ keys, uint64_t E, uint32_t vbits,
                             uint32_t* __restrict__ tile, BuildStats* __restrict__ st) {
    __shared__ uint32_t n_s[kBlock / 32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t b[kRounds];
    bool dup = false;
    const uint32_t n =
        head_ballots(keys, blockIdx.x * (uint64_t)kTileKeys + warp * kWarpKeys, E, vbits, lane, b, dup);
    if (__any_sync(0xffffffffu, dup) && lane == 0) st->dup = 1u;
    if (lane == 0) n_s[warp] = n;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t s = 0;
        for (int w = 0; w < kBlock / 32; w++) s += n_s[w];
        tile[blockIdx.x] = s;
    }
}

// Segments before this warp's first key (tile base plus the block's earlier
// warps); `n` is the warp's own heads.
__device__ __forceinline__ uint32_t warp_seg_base(const uint32_t* __restrict__ tile, uint32_t n, uint32_t* n_s,
                                                  uint32_t lane, uint32_t warp) {
    if (lane == 0) n_s[warp] = n;
    __syncthreads();
    uint32_t s = tile[blockIdx.x];
    for (uint32_t w = 0; w < warp; w++) s += n_s[w];
    return s;
}

// First key of every segment; seg_start[number of segments] = E.
__global__ void k_seg_starts(const uint64_t* __restrict__ keys, uint64_t E, uint32_t vbits,
                             const uint32_t* __restrict__ tile, uint32_t* __restrict__ seg_start) {
    __shared__ uint32_t n_s[kBlock / 32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t base = blockIdx.x * (uint64_t)kTileKeys + warp * kWarpKeys;
    uint32_t b[kRounds];
    bool dup = false;
    const uint32_t n = head_ballots(keys, base, E, vbits, lane, b, dup);
    uint32_t s = warp_seg_base(tile, n, n_s, lane, warp);
    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
    for (uint32_t j = 0; j < kRounds; j++) {
        const uint64_t i = base + 32 * j + lane;
        if ((b[j] >> lane) & 1u) seg_start[s + __popc(b[j] & lt)] = (uint32_t)i;
        s += __popc(b[j]);
        if (i == E - 1) seg_start[s] = (uint32_t)E;
    }
}

__device__ __forceinline__ uint32_t len16_of(uint32_t n) { return n > 3 ? (n + 3) / 4 : 0; }

// Segment lengths: the 16-byte units each tile of segments stores out of line,
// the longest list, the long lists, the list lengths by floor(log2), the pairs
// in a list summed per label, and the first segment of every label.  The totals
// are gathered per block, the pairs per warp, and added once (one atomic per
// segment on shared counters was the slowest kernel of the build: 250 us for
// 7.1 M segments, now 30).
__global__ void k_seg_lens(const uint64_t* __restrict__ keys, const uint32_t* __restrict__ seg_start,
                           uint32_t vbits, uint32_t* __restrict__ tile16, BuildStats* __restrict__ st) {
    __shared__ uint32_t hist_s[32], red_s[kBlock / 32], max_s;
    if (threadIdx.x < 32) hist_s[threadIdx.x] = 0;
    if (threadIdx.x == 0) max_s = 0;
    __syncthreads();
    const uint32_t nseg = st->nseg;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t one = 0, two = 0, pairs_of = 0;      // label of the pairs summed so far
    unsigned long long pairs = 0;                 // (lane's part)
    auto add_pairs = [&]() {
#pragma unroll
        for (int o = 16; o; o >>= 1) pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
        if (lane == 0 && pairs) atomicAdd(&st->pairs[pairs_of], pairs);
        pairs = 0;
    };
    for (uint64_t t = blockIdx.x; t * kTileSegs < nseg; t += gridDim.x) {
        uint32_t sum = 0, mx = 0;
#pragma unroll
        for (uint32_t j = 0; j < kTileSegs / kBlock; j++) {
            const uint64_t s = t * kTileSegs + j * kBlock + threadIdx.x;
            uint32_t n = 0, l = 0;
            if (s < nseg) {
                const uint32_t b = seg_start[s];
                n = seg_start[s + 1] - b;
                sum += len16_of(n);
                mx = max(mx, n);
                if (n > 3) atomicAdd(&hist_s[31 - __clz((int)n)], 1u);
                l = (uint32_t)(keys[b] >> (2 * vbits));
                if (s == 0 || (uint32_t)(keys[b - 1] >> (2 * vbits)) != l) st->first[l] = s;
            }
            // most lists are this short: counted by ballot, not by colliding atomics
            one += __popc(__ballot_sync(0xffffffffu, n == 1));
            two += __popc(__ballot_sync(0xffffffffu, n == 2 || n == 3));
            // segments come label by label: nearly always one label a warp
            const unsigned many = __ballot_sync(0xffffffffu, n > 1);
            if (!many) continue;
            const uint32_t l0 = __shfl_sync(0xffffffffu, l, __ffs(many) - 1);
            if (l0 != pairs_of) {
                add_pairs();
                pairs_of = l0;
            }
            const unsigned long long pr = n > 1 ? (unsigned long long)n * (n - 1) : 0ull;
            if (l == l0) pairs += pr;
            else if (pr) atomicAdd(&st->pairs[l], pr);
        }
        sum = __reduce_add_sync(0xffffffffu, sum);
        mx = __reduce_max_sync(0xffffffffu, mx);
        if (lane == 0) {
            red_s[warp] = sum;
            if (mx) atomicMax(&max_s, mx);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t x = 0;
            for (int w = 0; w < kBlock / 32; w++) x += red_s[w];
            tile16[t] = x;
        }
        __syncthreads();
    }
    if (lane == 0 && one) atomicAdd(&hist_s[0], one);
    if (lane == 0 && two) atomicAdd(&hist_s[1], two);
    __syncthreads();
    if (threadIdx.x < 32 && hist_s[threadIdx.x]) atomicAdd(&st->hist[threadIdx.x], hist_s[threadIdx.x]);
    if (threadIdx.x == 0 && max_s) atomicMax(&st->max_len, max_s);
    add_pairs();
}

// Out-of-line offset of every segment, in 16-byte units.  A thread takes four
// consecutive segments.
__global__ void k_seg_offsets(const uint32_t* __restrict__ seg_start, const uint32_t* __restrict__ tile16,
                              const BuildStats* __restrict__ st, uint32_t* __restrict__ off16) {
    __shared__ uint32_t w_s[kBlock / 32];
    const uint32_t nseg = st->nseg;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint64_t t = blockIdx.x; t * kTileSegs < nseg; t += gridDim.x) {
        const uint64_t s0 = t * kTileSegs + 4 * threadIdx.x;
        uint32_t u[4], sum = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            u[j] = s0 + j < nseg ? len16_of(seg_start[s0 + j + 1] - seg_start[s0 + j]) : 0u;
            sum += u[j];
        }
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
            if ((int)lane >= o) incl += x;
        }
        if (lane == 31) w_s[warp] = incl;
        __syncthreads();
        uint32_t at = tile16[t] + incl - sum;
        for (uint32_t w = 0; w < warp; w++) at += w_s[w];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (s0 + j < nseg) off16[s0 + j] = at;
            at += u[j];
        }
        __syncthreads();
    }
}

// Exclusive prefix sum of n values in place by one block; the total goes to *total.
template <class T>
__global__ void k_scan_tiles(T* __restrict__ v, uint64_t n, T* __restrict__ total) {
    __shared__ T w_s[32];
    __shared__ T carry_s;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry_s = 0;
    __syncthreads();
    for (uint64_t b = 0; b < n; b += 4ull * blockDim.x) {
        const uint64_t i = b + 4ull * threadIdx.x;
        T u[4], sum = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            u[j] = i + j < n ? v[i + j] : (T)0;
            sum += u[j];
        }
        T incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const T x = __shfl_up_sync(0xffffffffu, incl, o);
            if ((int)lane >= o) incl += x;
        }
        if (lane == 31) w_s[warp] = incl;
        __syncthreads();
        T at = carry_s + incl - sum, all = 0;
        for (uint32_t w = 0; w < blockDim.x / 32; w++) {
            if (w < warp) at += w_s[w];
            all += w_s[w];
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (i + j < n) v[i + j] = at;
            at += u[j];
        }
        __syncthreads();
        if (threadIdx.x == 0) carry_s += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry_s;
}

// Places every e-line: a long segment's entries go to its out-of-line list,
// its head writes the record, the root-list entry and, for lists of at least
// `thresh` entries (0: none), the bitmap index.  Keys, and so the entries of
// a list, are read and written in order.  16 M e-lines in 7.1 M segments over
// a 1.1 GB record table: 243 us (bound by the scattered 16-byte records); the
// four kernels it replaces, one thread per segment, took 308 us.
__global__ void k_place(const uint64_t* __restrict__ keys, uint64_t E, uint32_t V, uint32_t vbits,
                        const uint32_t* __restrict__ tile, const uint32_t* __restrict__ seg_start,
                        const uint32_t* __restrict__ off16, uint4* __restrict__ seg, uint32_t* __restrict__ nbr,
                        uint32_t* __restrict__ heads, uint32_t thresh, uint32_t bm_cap,
                        unsigned int* __restrict__ bm_counter, uint2* __restrict__ bm_list) {
    __shared__ uint32_t n_s[kBlock / 32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t base = blockIdx.x * (uint64_t)kTileKeys + warp * kWarpKeys;
    const uint64_t vmask = (1ull << vbits) - 1;
    uint32_t bl[kRounds];
    bool dup = false;
    const uint32_t heads_n = head_ballots(keys, base, E, vbits, lane, bl, dup);
    uint32_t first = warp_seg_base(tile, heads_n, n_s, lane, warp);
    const uint32_t le = 0xffffffffu >> (31 - lane);
#pragma unroll
    for (uint32_t j = 0; j < kRounds; j++) {
        const uint64_t i = base + 32 * j + lane;
        const uint32_t s = first + __popc(bl[j] & le) - 1;
        first += __popc(bl[j]);
        if (i >= E) continue;
        const uint64_t k = keys[i];
        const uint32_t b = seg_start[s], n = seg_start[s + 1] - b;
        const bool head = i == b;
        if (n > 3) {
            uint32_t* list = nbr + (uint64_t)off16[s] * 4;
            list[i - b] = (uint32_t)(k & vmask);
            if (head)
                for (uint32_t t = n; t < ((n + 3) & ~3u); t++) list[t] = kNoVertex;
        }
        if (!head) continue;
        const uint32_t src = (uint32_t)((k >> vbits) & vmask);
        const uint32_t lab = (uint32_t)(k >> (2 * vbits));
        uint4 r;
        r.x = n;
        if (n <= 3) {
            r.y = (uint32_t)(k & vmask);
            r.z = n > 1 ? (uint32_t)(keys[i + 1] & vmask) : kNoVertex;
            r.w = n > 2 ? (uint32_t)(keys[i + 2] & vmask) : kNoVertex;
        } else {
            r.y = off16[s];
            r.z = (uint32_t)(k & vmask);
            r.w = (uint32_t)(keys[i + n - 1] & vmask);
            if (thresh && n >= thresh) {
                const unsigned int idx = atomicAdd(bm_counter, 1u);
                if (idx < bm_cap) {
                    r.z = kBitmapMark | idx;
                    bm_list[idx] = make_uint2(r.y, n);
                }
            }
        }
        seg[(uint64_t)lab * V + src] = r;
        heads[s] = src;
    }
}

// Does every e-line have its reverse?  Without duplicates it is enough that
// every e-line with src < dst has one and that there are as many with
// src > dst: half of the lookups.  Bound by the scattered record loads.
__global__ void k_symmetry(const uint64_t* __restrict__ keys, uint64_t E, uint32_t V, uint32_t vbits,
                           const uint4* __restrict__ seg, const uint32_t* __restrict__ nbr,
                           const uint32_t* __restrict__ bm, uint32_t bm_words, BuildStats* __restrict__ st) {
    const uint64_t vmask = (1ull << vbits) - 1;
    uint32_t up = 0, down = 0;
    bool bad = false;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < E; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t k = keys[i];
        const uint32_t d = (uint32_t)(k & vmask), s = (uint32_t)((k >> vbits) & vmask);
        down += s > d;
        if (s >= d) continue;
        up += 1;
        bad |= !dev::seg_has(dev::ldg4(seg + (k >> (2 * vbits)) * V + d), s, 1, nbr, bm, bm_words);
    }
    up = __reduce_add_sync(0xffffffffu, up);
    down = __reduce_add_sync(0xffffffffu, down);
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) st->asym = 1u;
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&st->up, up);
        atomicAdd(&st->down, down);
    }
}

// E-line filter (dev::filter_place).  Bound by the atomics, one per e-line.
__global__ void k_filter(const uint64_t* __restrict__ keys, uint64_t E, uint32_t vbits,
                         const uint32_t* __restrict__ off, uint32_t* __restrict__ efilter) {
    const uint64_t vmask = (1ull << vbits) - 1;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < E; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t k = keys[i];
        const uint32_t l = (uint32_t)(k >> (2 * vbits)), a = __ldg(off + l);
        uint32_t bits;
        const uint32_t at = dev::filter_place(dev::filter_seed((uint32_t)((k >> vbits) & vmask)), (uint32_t)(k & vmask),
                                              __ldg(off + l + 1) - a, bits);
        atomicOr(efilter + a + at, bits);
    }
}

// One block per bitmap: set the bit of every entry.
__global__ void k_bm_fill(const uint32_t* __restrict__ nbr, const uint2* __restrict__ bm_list, uint32_t n_bm,
                          uint32_t bm_words, uint32_t* __restrict__ bitmaps) {
    for (uint32_t i = blockIdx.x; i < n_bm; i += gridDim.x) {
        const uint2 e = bm_list[i];
        const uint32_t* list = nbr + (uint64_t)e.x * 4;
        uint32_t* bits = bitmaps + (uint64_t)i * bm_words;
        for (uint32_t t = threadIdx.x; t < e.y; t += blockDim.x) {
            const uint32_t x = list[t];
            atomicOr(bits + (x >> 5), 1u << (x & 31));
        }
    }
}

uint32_t bits_for(uint64_t x) {   // bits needed to store values 0..x
    uint32_t b = 1;
    while (b < 64 && (x >> b)) ++b;
    return b;
}

uint64_t up256(uint64_t x) { return (x + 255) & ~255ull; }

int grid_for(uint64_t n, int sms) {
    uint64_t b = (n + 255) / 256;
    uint64_t cap = (uint64_t)sms * 8;
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (int)b;
}

struct Events {                      // destroyed on every return path
    cudaEvent_t a = nullptr, b = nullptr;
    ~Events() {
        if (a) cudaEventDestroy(a);
        if (b) cudaEventDestroy(b);
    }
};

}  // namespace

uint64_t env_bytes(const char* name, uint64_t dflt) {
    const char* v = std::getenv(name);
    if (!v || !*v) return dflt;
    char* end = nullptr;
    const unsigned long long x = std::strtoull(v, &end, 10);
    return (end && *end == 0) ? (uint64_t)x : dflt;
}

cudaError_t scan_tiles_u64(unsigned long long* v, uint64_t n, unsigned long long* total, cudaStream_t s) {
    k_scan_tiles<unsigned long long><<<1, 1024, 0, s>>>(v, n, total);
    return cudaGetLastError();
}

fm_status graph_key_layout(uint32_t V, uint32_t L, uint64_t E, uint32_t& vbits, uint32_t& lbits) {
    if (V == 0 || L == 0) {
        set_error("graph needs at least one vertex and one label slot");
        return FM_ERR_ARG;
    }
    vbits = bits_for(V - 1);
    lbits = bits_for(L - 1);
    if (2 * vbits + lbits > 64) {
        set_error("vertex and label ids do not fit the 64-bit sort key");
        return FM_ERR_UNSUPPORTED;
    }
    if (E >= (1ull << 32)) {
        set_error("more than 2^32 - 1 directed e-lines");
        return FM_ERR_UNSUPPORTED;
    }
    return FM_OK;
}

BuildArena::~BuildArena() {
    if (mem) cudaFree(mem);
}

fm_status BuildArena::alloc(uint64_t cap, uint32_t key_bits, uint64_t extra) {
    cub::DoubleBuffer<uint64_t> db(nullptr, nullptr);
    FM_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, temp_bytes, db, (int64_t)cap, 0, (int)key_bits));
    const uint64_t o_keys = up256(sizeof(BuildStats)), o_alt = o_keys + up256(cap * 8);
    const uint64_t o_start = o_alt + up256(cap * 8), o_off = o_start + up256((cap + 1) * 4);
    const uint64_t o_te = o_off + up256(cap * 4), o_ts = o_te + up256((cap / kTileKeys + 1) * 4);
    const uint64_t o_temp = o_ts + up256((cap / kTileSegs + 1) * 4), o_extra = o_temp + up256(temp_bytes);
    const cudaError_t e = cudaMalloc(&mem, o_extra + extra);
    if (e != cudaSuccess) {
        cudaGetLastError();
        mem = nullptr;
        set_error("cannot allocate device memory for building the data graph");
        return FM_ERR_NOMEM;
    }
    char* p = (char*)mem;
    stats = (BuildStats*)p;
    keys = (uint64_t*)(p + o_keys);
    alt = (uint64_t*)(p + o_alt);
    seg_start = (uint32_t*)(p + o_start);
    off16 = (uint32_t*)(p + o_off);
    tile_keys = (uint32_t*)(p + o_te);
    tile_segs = (uint32_t*)(p + o_ts);
    temp = p + o_temp;
    this->extra = p + o_extra;
    return FM_OK;
}

fm_status build_from_edges(DeviceGraph& g, uint32_t V, uint32_t L, uint64_t E, const uint32_t* src,
                           const uint32_t* dst, const uint32_t* lab, cudaStream_t s) {
    uint32_t vbits = 0, lbits = 0;
    FM_TRY(graph_key_layout(V, L, E, vbits, lbits));
    int dev = 0, sms = 1;
    FM_CUDA(cudaGetDevice(&dev));
    FM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    BuildArena a;
    FM_TRY(a.alloc(E, 2 * vbits + lbits, 0));
    FM_CUDA(cudaMemsetAsync(a.stats, 0, sizeof(BuildStats), s));
    if (E) {
        // the e-lines are staged in memory that the sort and the segment
        // passes take over once the keys are made
        uint32_t* d_src = (uint32_t*)a.alt;
        uint32_t* d_dst = d_src + E;
        uint32_t* d_lab = a.seg_start;
        FM_CUDA(cudaMemcpyAsync(d_src, src, E * 4, cudaMemcpyHostToDevice, s));
        FM_CUDA(cudaMemcpyAsync(d_dst, dst, E * 4, cudaMemcpyHostToDevice, s));
        FM_CUDA(cudaMemcpyAsync(d_lab, lab, E * 4, cudaMemcpyHostToDevice, s));
        k_make_keys<<<grid_for(E, sms), 256, 0, s>>>(d_src, d_dst, d_lab, E, V, L, vbits, a.keys, a.stats);
        FM_CUDA(cudaGetLastError());
    }
    return build_from_keys(g, V, L, E, a, s);
}

fm_status build_from_keys(DeviceGraph& g, uint32_t V, uint32_t L, uint64_t E, BuildArena& a, cudaStream_t s) {
    uint32_t vbits = 0, lbits = 0;
    FM_TRY(graph_key_layout(V, L, E, vbits, lbits));
    int dev = 0, sms = 1;
    FM_CUDA(cudaGetDevice(&dev));
    FM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    Events ev;
    FM_CUDA(cudaEventCreate(&ev.a));
    FM_CUDA(cudaEventCreate(&ev.b));
    FM_CUDA(cudaEventRecord(ev.a, s));

    g = DeviceGraph();
    g.V = V;
    g.L = L;
    g.E = E;
    g.vbits = vbits;
    g.device = dev;

    const uint64_t* sorted = a.keys;
    uint64_t* spare = a.alt;
    const unsigned key_tiles = (unsigned)((E + kTileKeys - 1) / kTileKeys);
    BuildStats h;
    if (E) {
        FM_CUDA(cudaMemsetAsync(a.stats->first, 0xff, sizeof(h.first), s));
        cub::DoubleBuffer<uint64_t> db(a.keys, a.alt);
        size_t tb = 0;
        FM_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, tb, db, (int64_t)E, 0, (int)(2 * vbits + lbits), s));
        if (tb > a.temp_bytes) {
            set_error("sort scratch larger than planned");
            return FM_ERR_NOMEM;
        }
        FM_CUDA(cub::DeviceRadixSort::SortKeys(a.temp, tb, db, (int64_t)E, 0, (int)(2 * vbits + lbits), s));
        sorted = db.Current();
        spare = db.Alternate();
        k_tile_heads<<<key_tiles, kBlock, 0, s>>>(sorted, E, vbits, a.tile_keys, a.stats);
        k_scan_tiles<uint32_t><<<1, 1024, 0, s>>>(a.tile_keys, key_tiles, &a.stats->nseg);
        k_seg_starts<<<key_tiles, kBlock, 0, s>>>(sorted, E, vbits, a.tile_keys, a.seg_start);
        const uint64_t seg_tiles = (E + kTileSegs - 1) / kTileSegs;   // at most: the segments are counted on the device
        const int seg_grid = (int)std::min<uint64_t>(seg_tiles, (uint64_t)sms * 8);
        FM_CUDA(cudaMemsetAsync(a.tile_segs, 0, seg_tiles * 4, s));
        k_seg_lens<<<seg_grid, kBlock, 0, s>>>(sorted, a.seg_start, vbits, a.tile_segs, a.stats);
        k_scan_tiles<uint32_t><<<1, 1024, 0, s>>>(a.tile_segs, seg_tiles, &a.stats->total16);
        k_seg_offsets<<<seg_grid, kBlock, 0, s>>>(a.seg_start, a.tile_segs, a.stats, a.off16);
        FM_CUDA(cudaGetLastError());
    }
    FM_CUDA(cudaMemcpyAsync(&h, a.stats, sizeof(h), cudaMemcpyDeviceToHost, s));
    FM_CUDA(cudaStreamSynchronize(s));
    if (h.error) {
        set_error("edge endpoint or label out of range");
        return FM_ERR_DATA_LINE;
    }
    const uint64_t nseg = h.nseg;
    g.nbr_words = (uint64_t)h.total16 * 4;
    g.segments = nseg;
    g.max_len = h.max_len;
    g.has_dups = h.dup ? 1 : 0;
    g.has_self_loops = h.loops ? 1 : 0;
    g.long_segments = nseg - h.hist[0] - h.hist[1];   // lists of 4 entries and more
    g.label_count.assign(h.label_count, h.label_count + L);
    g.label_pairs.assign(h.pairs, h.pairs + L);
    // a label without segments starts where the next label with one does
    g.head_off.assign(L + 1, nseg);
    if (E)
        for (uint32_t l = L; l-- > 0;) g.head_off[l] = h.first[l] != ~0ull ? h.first[l] : g.head_off[l + 1];

    // membership bitmaps for the longest lists (not with duplicates: a
    // bit cannot count copies; vertex ids must leave bit 31 of z free)
    // default budget: room for 16384 bitmaps, between 2 and 8 GiB.  Only what
    // the e-line filter lets pass asks them, so what they save depends on how
    // much of a list's candidates passes: 4-cliques of a 2^18-vertex power-law
    // graph with 2 labels 29.8 ms with them, 45.9 without; on a 2^22-vertex
    // R-MAT graph with 64 labels paths, cycles, triangles and walks take the same
    // within 1 % with 8 GiB, 2 GiB and none, and its build 16.1, 16.2 and 15.2 ms
    const uint32_t words = (V + 31) / 32;
    const uint64_t budget = env_bytes(
        "FM_BITMAP_BYTES", std::min<uint64_t>(8ull << 30, std::max<uint64_t>(2ull << 30, 16384ull * 4ull * words)));
    const uint64_t min_len = std::max<uint64_t>(4, env_bytes("FM_BITMAP_MIN_LEN", 64));
    const uint64_t cap64 = budget / (4ull * words);
    uint32_t thresh = 0;
    uint64_t n_bm = 0;
    if (!h.dup && V < kBitmapMark && cap64 > 0 && g.long_segments > 0) {
        uint32_t min_log2 = 0;
        while (min_log2 < 63 && (1ull << min_log2) < min_len) min_log2++;
        const uint32_t cap = (uint32_t)std::min<uint64_t>(cap64, 1u << 30);
        // smallest power-of-two threshold whose lists all fit the budget
        uint64_t above = 0;
        for (int b = 31; b >= (int)min_log2; b--) {
            if (above + h.hist[b] > cap) break;
            above += h.hist[b];
            if (h.hist[b]) {
                thresh = 1u << b;
                n_bm = above;
            }
        }
    }

    // records, lists, root lists and bitmaps in one allocation
    const uint64_t seg_bytes = up256((uint64_t)L * V * sizeof(uint4));
    const uint64_t nbr_bytes = up256((g.nbr_words ? g.nbr_words : 4) * 4);
    const uint64_t head_bytes = up256((nseg ? nseg : 4) * 4);
    const uint64_t bm_bytes = up256(n_bm * words * 4ull);
    // half a word of filter per e-line, at least one word per label
    std::vector<uint32_t> foff(L + 1, 0);
    for (uint32_t l = 0; l < L; l++) foff[l + 1] = foff[l] + (uint32_t)(h.label_count[l] / 2 + 1);
    const uint64_t filter_bytes = h.dup ? 0 : up256((uint64_t)foff[L] * 4);
    const uint64_t foff_bytes = h.dup ? 0 : up256((L + 1) * 4ull);
    FM_CUDA(cudaMalloc(&g.block, seg_bytes + nbr_bytes + head_bytes + bm_bytes + filter_bytes + foff_bytes));
    g.seg = (uint4*)g.block;
    g.nbr = (uint32_t*)((char*)g.block + seg_bytes);
    g.heads = (uint32_t*)((char*)g.block + seg_bytes + nbr_bytes);
    FM_CUDA(cudaMemsetAsync(g.seg, 0, (size_t)L * V * sizeof(uint4), s));
    if (!h.dup) {
        char* f = (char*)g.heads + head_bytes + bm_bytes;
        g.efilter = (uint32_t*)f;
        g.efilter_off = (uint32_t*)(f + filter_bytes);
        g.filter_bytes = foff[L] * 4ull + (L + 1) * 4ull;
        FM_CUDA(cudaMemsetAsync(g.efilter, 0, filter_bytes, s));
        FM_CUDA(cudaMemcpyAsync(g.efilter_off, foff.data(), (L + 1) * 4, cudaMemcpyHostToDevice, s));
        k_filter<<<grid_for(E, sms), 256, 0, s>>>(sorted, E, vbits, g.efilter_off, g.efilter);
        FM_CUDA(cudaGetLastError());
    }
    if (E) {
        uint2* bm_list = (uint2*)spare;
        if (n_bm) {
            g.bitmaps = (uint32_t*)((char*)g.heads + head_bytes);
            FM_CUDA(cudaMemsetAsync(g.bitmaps, 0, bm_bytes, s));
        }
        k_place<<<key_tiles, kBlock, 0, s>>>(sorted, E, V, vbits, a.tile_keys, a.seg_start, a.off16, g.seg, g.nbr,
                                             g.heads, thresh, (uint32_t)n_bm, &a.stats->bm_count, bm_list);
        if (n_bm) {
            const uint32_t fill_grid = (uint32_t)std::min<uint64_t>(n_bm, (uint64_t)sms * 16);
            k_bm_fill<<<fill_grid, 256, 0, s>>>(g.nbr, bm_list, (uint32_t)n_bm, words, g.bitmaps);
            g.n_bitmaps = (uint32_t)n_bm;
            g.bm_words = words;
            g.bm_min_len = thresh;
        }
        if (!h.dup)
            k_symmetry<<<grid_for(E, sms), 256, 0, s>>>(sorted, E, V, vbits, g.seg, g.nbr, g.bitmaps, g.bm_words,
                                                        a.stats);
        FM_CUDA(cudaGetLastError());
        FM_CUDA(cudaMemcpyAsync(&h, a.stats, offsetof(BuildStats, hist), cudaMemcpyDeviceToHost, s));
    }
    FM_CUDA(cudaEventRecord(ev.b, s));
    FM_CUDA(cudaStreamSynchronize(s));
    g.symmetric = !h.dup && !h.asym && h.up == h.down;
    float ms = 0;
    cudaEventElapsedTime(&ms, ev.a, ev.b);
    g.build_ms = ms;
    return FM_OK;
}

}  // namespace fm
