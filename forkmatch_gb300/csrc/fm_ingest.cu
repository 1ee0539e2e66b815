// fm_ingest.cu -- `.g` text parsed on the device.
//
// The reference parses its data file on the device too (parseCSR,
// src/trie.cuh:800-951), but with `int` offsets (src/trie.cuh:802,1115), so a
// file over 2 GiB cannot be read, and it never parses the first line after the
// header (src/trie.cuh:829-834,1176-1178).  Here every offset is 64-bit:
//
//   1. the host checks the framing ("t # 0\n", the header line, the trailing
//      "t # -1", the newline before it) -- a few bytes;
//   2. the body is copied to the device once;
//   3. k_count_lines / k_line_starts: each thread takes 16 bytes, a block scan
//      numbers the newlines, and every line start is written in file order;
//   4. k_parse_lines: one thread per line parses "v id label" or
//      "e src dst label" with the same grammar and range checks as the host
//      parser (fm_parse.cpp), records the first bad line, counts labels and
//      appends the kept e-lines (label < label slots) as sort keys;
//   5. the keys go straight to the device graph build, without a round trip
//      to the host.  The build sorts them, so the order in which blocks
//      append does not matter and no stable compaction is needed.
#include <cub/cub.cuh>

#include <algorithm>
#include <cstring>
#include <string>

#include "fm_internal.h"

namespace fm {
namespace {

constexpr int kIngestBlock = 256;
constexpr uint64_t kBytesPerBlock = 16ull * kIngestBlock;   // 16 bytes per thread

__device__ __forceinline__ uint32_t newline_mask16(const unsigned char* b, uint64_t pos, uint64_t n, uint4& raw) {
    // 16 bytes starting at pos (pos is 16-aligned within the body buffer)
    uint32_t mask = 0;
    if (pos + 16 <= n) {
        raw = *reinterpret_cast<const uint4*>(b + pos);
        const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (((w[i] >> (8 * j)) & 0xffu) == '\n') mask |= 1u << (4 * i + j);
    } else {
        for (uint64_t i = pos; i < n; i++)
            if (b[i] == '\n') mask |= 1u << (uint32_t)(i - pos);
    }
    return mask;
}

// Newlines per block of kBytesPerBlock bytes.
__global__ void k_count_lines(const unsigned char* __restrict__ body, uint64_t n, unsigned long long* __restrict__ per_block) {
    typedef cub::BlockReduce<uint32_t, kIngestBlock> Reduce;
    __shared__ typename Reduce::TempStorage tmp;
    const uint64_t pos = blockIdx.x * kBytesPerBlock + 16ull * threadIdx.x;
    uint4 raw;
    const uint32_t c = pos < n ? __popc(newline_mask16(body, pos, n, raw)) : 0u;
    const uint32_t s = Reduce(tmp).Sum(c);
    if (threadIdx.x == 0) per_block[blockIdx.x] = s;
}

// Start offset of every line: line 0 starts at 0, line i+1 after newline i.
// Starts past `cap` are not kept (see parse_data_text_device).
__global__ void k_line_starts(const unsigned char* __restrict__ body, uint64_t n,
                              const unsigned long long* __restrict__ block_base, uint64_t cap,
                              uint64_t* __restrict__ starts) {
    typedef cub::BlockScan<uint32_t, kIngestBlock> Scan;
    __shared__ typename Scan::TempStorage tmp;
    const uint64_t pos = blockIdx.x * kBytesPerBlock + 16ull * threadIdx.x;
    uint4 raw;
    uint32_t mask = pos < n ? newline_mask16(body, pos, n, raw) : 0u;
    uint32_t before = 0;
    Scan(tmp).ExclusiveSum(__popc(mask), before);
    uint64_t line = block_base[blockIdx.x] + before;   // newlines before this thread's bytes
    while (mask) {
        const int b = __ffs(mask) - 1;
        mask &= mask - 1;
        if (line < cap) starts[line + 1] = pos + b + 1;
        line++;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) starts[0] = 0;
}

__device__ __forceinline__ bool dparse_u32(const unsigned char* b, uint64_t& p, uint64_t end, uint32_t& v) {
    uint64_t acc = 0;
    const uint64_t s = p;
    while (p < end && (unsigned char)(b[p] - '0') < 10) {
        acc = acc * 10 + (uint64_t)(b[p] - '0');
        if (acc > 0xffffffffull) return false;
        ++p;
    }
    if (p == s) return false;
    v = (uint32_t)acc;
    return true;
}

// One thread per line (lines [0, min(lines, cap)), each ending with '\n').  A
// block appends its kept e-lines as sort keys with one atomic per 256 lines.
__global__ void k_parse_lines(const unsigned char* __restrict__ body, const uint64_t* __restrict__ starts,
                              uint64_t cap, uint32_t V, uint32_t EL, uint32_t L, uint32_t vbits,
                              uint64_t* __restrict__ keys, BuildStats* __restrict__ st) {
    __shared__ unsigned int h[FM_MAX_LABEL + 1];
    __shared__ uint32_t n_s[kIngestBlock / 32];
    __shared__ unsigned long long base_s;
    for (uint32_t i = threadIdx.x; i <= FM_MAX_LABEL; i += blockDim.x) h[i] = 0;
    const uint64_t nlines = st->lines < cap ? st->lines : cap;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint64_t i0 = blockIdx.x * (uint64_t)blockDim.x; i0 < nlines; i0 += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = i0 + threadIdx.x;
        bool keep = false;
        uint32_t v[3] = {0, 0, 0};
        if (i < nlines) {
            uint64_t p = starts[i];
            const uint64_t end = starts[i + 1];   // one past this line's '\n'
            bool ok = end >= p + 2;
            if (ok) {
                const unsigned char kind = body[p];
                ok = (kind == 'v' || kind == 'e') && body[p + 1] == ' ';
                const int nv = kind == 'e' ? 3 : 2;
                p += 2;
                for (int f = 0; f < nv && ok; f++) {
                    ok = dparse_u32(body, p, end, v[f]) && p < end && body[p] == ((f == nv - 1) ? '\n' : ' ');
                    ++p;
                }
                if (ok) {
                    if (kind == 'v') ok = v[0] < V;
                    else ok = v[0] < V && v[1] < V && v[2] <= EL;
                }
                keep = ok && kind == 'e' && v[2] < L;
            }
            if (!ok) atomicMin(&st->first_bad, (unsigned long long)i);
        }
        const unsigned b = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) n_s[warp] = __popc(b);
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t n = 0;
            for (int w = 0; w < kIngestBlock / 32; w++) n += n_s[w];
            base_s = n ? atomicAdd(&st->kept, (unsigned long long)n) : 0ull;
        }
        __syncthreads();
        if (keep) {
            uint64_t at = base_s + __popc(b & ((1u << lane) - 1u));
            for (uint32_t w = 0; w < warp; w++) at += n_s[w];
            keys[at] = ((uint64_t)v[2] << (2 * vbits)) | ((uint64_t)v[0] << vbits) | (uint64_t)v[1];
            atomicAdd(&h[v[2]], 1u);
            if (v[0] == v[1]) atomicOr(&st->loops, 1u);
        }
        __syncthreads();                          // n_s and base_s are written again
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i <= FM_MAX_LABEL; i += blockDim.x)
        if (h[i]) atomicAdd(&st->label_count[i], (unsigned long long)h[i]);
}

struct DBuf {
    void* p = nullptr;
    DBuf() = default;
    DBuf(const DBuf&) = delete;
    DBuf& operator=(const DBuf&) = delete;
    ~DBuf() { reset(); }
    void reset() {
        if (p) cudaFree(p);
        p = nullptr;
    }
    template <class T> T* as() { return (T*)p; }
};

fm_status dev_alloc(DBuf& b, uint64_t bytes) {
    if (cudaMalloc(&b.p, bytes ? bytes : 16) != cudaSuccess) {
        cudaGetLastError();
        b.p = nullptr;
        set_error("cannot allocate device memory for parsing the data graph");
        return FM_ERR_NOMEM;
    }
    return FM_OK;
}

bool host_u32(const char*& p, const char* end, uint32_t& v) {
    uint64_t acc = 0;
    const char* s = p;
    while (p < end && (unsigned char)(*p - '0') < 10) {
        acc = acc * 10 + (uint64_t)(*p - '0');
        if (acc > 0xffffffffull) return false;
        ++p;
    }
    if (p == s) return false;
    v = (uint32_t)acc;
    return true;
}

}  // namespace

fm_status parse_data_text_device(const char* text, uint64_t len, cudaStream_t s, DeviceGraph& g) {
    // framing, checked on the host exactly as parse_data_text does
    if (len < 6 || std::memcmp(text, "t # 0\n", 6) != 0) {
        set_error("data graph does not start with \"t # 0\\n\"");
        return FM_ERR_DATA_HEADER0;
    }
    if (len < 12 || std::memcmp(text + len - 6, "t # -1", 6) != 0) {
        set_error("data graph does not end with \"t # -1\"");
        return FM_ERR_DATA_TRAILER;
    }
    const char* p = text + 6;
    const char* end = text + len - 6;
    uint32_t h[4] = {0, 0, 0, 0};
    for (int field = 0;; field++) {
        if (field > 3 || !host_u32(p, end, h[field]) || p >= end) {
            set_error("malformed data graph header");
            return FM_ERR_DATA_HEADER;
        }
        if (*p == '\n') {
            ++p;
            break;
        }
        if (*p != ' ') {
            set_error("malformed data graph header");
            return FM_ERR_DATA_HEADER;
        }
        ++p;
    }
    const uint32_t V = h[0];
    const uint64_t Ehdr = h[1];
    const uint32_t EL = h[3];
    const uint32_t L = std::min<uint32_t>(EL, FM_MAX_LABEL) + 1;
    const char* body = p;
    const uint64_t blen = (uint64_t)(end - body);
    if (blen && body[blen - 1] != '\n') {
        set_error("last data line is not terminated by a newline before \"t # -1\"");
        return FM_ERR_DATA_LINE;
    }

    int dev = 0, sms = 1;
    FM_CUDA(cudaGetDevice(&dev));
    FM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const uint64_t nblocks = std::max<uint64_t>(1, (blen + kBytesPerBlock - 1) / kBytesPerBlock);
    if (nblocks > 0x7fffffffull) {
        set_error("data graph text too large");
        return FM_ERR_UNSUPPORTED;
    }
    // a header that no graph can have is reported after the lines are checked
    uint32_t vbits = 0, lbits = 0;
    if (graph_key_layout(V, L, 0, vbits, lbits) != FM_OK) vbits = lbits = 16;
    const uint32_t key_bits = 2 * vbits + lbits;
    // body (16-byte aligned, padded to whole 16-byte words) and newline counts
    const uint64_t body_bytes = (blen + 31 + 255) & ~255ull, text_bytes = body_bytes + nblocks * 8;
    // A valid line takes at least 6 bytes, so the text bounds the number of
    // lines (a text with more lines has its first bad line among those).
    // Texts up to 64 MiB use that bound for the build's arrays (33 bytes per
    // possible line) and put body and arrays in one allocation; larger ones,
    // where the bound would cost gigabytes, count the lines first
    // (FM_INGEST_BOUND_BYTES sets the limit).
    const bool bound = blen <= env_bytes("FM_INGEST_BOUND_BYTES", 64ull << 20);
    BuildArena arena;
    DBuf d_text;
    uint64_t cap = blen / 6 + 1;
    char* text_mem = nullptr;
    if (bound) {
        FM_TRY(arena.alloc(cap + 1, key_bits, text_bytes));
        text_mem = arena.extra;
    } else {
        FM_TRY(dev_alloc(d_text, text_bytes + 8));
        text_mem = d_text.as<char>();
    }
    unsigned char* b = (unsigned char*)text_mem;
    unsigned long long* counts = (unsigned long long*)(text_mem + body_bytes);
    if (blen) FM_CUDA(cudaMemcpyAsync(b, body, blen, cudaMemcpyHostToDevice, s));
    k_count_lines<<<(unsigned)nblocks, kIngestBlock, 0, s>>>(b, blen, counts);
    FM_CUDA(cudaGetLastError());
    unsigned long long* lines = nullptr;
    if (!bound) {
        // counts[nblocks] takes the number of lines (every line ends with '\n')
        lines = counts + nblocks;
        FM_CUDA(scan_tiles_u64(counts, nblocks, lines, s));
        unsigned long long n = 0;
        FM_CUDA(cudaMemcpyAsync(&n, lines, 8, cudaMemcpyDeviceToHost, s));
        FM_CUDA(cudaStreamSynchronize(s));
        cap = n;
        FM_TRY(arena.alloc(cap + 1, key_bits, 0));
    }
    FM_CUDA(cudaMemsetAsync(arena.stats, 0, sizeof(BuildStats), s));
    FM_CUDA(cudaMemsetAsync(&arena.stats->first_bad, 0xff, 8, s));
    if (bound) FM_CUDA(scan_tiles_u64(counts, nblocks, &arena.stats->lines, s));
    else FM_CUDA(cudaMemcpyAsync(&arena.stats->lines, lines, 8, cudaMemcpyDeviceToDevice, s));
    uint64_t* starts = arena.alt;
    k_line_starts<<<(unsigned)nblocks, kIngestBlock, 0, s>>>(b, blen, counts, cap, starts);
    const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((cap + 255) / 256, (uint64_t)sms * 8));
    k_parse_lines<<<grid, kIngestBlock, 0, s>>>(b, starts, cap, V, EL, L, vbits, arena.keys, arena.stats);
    FM_CUDA(cudaGetLastError());
    BuildStats st;
    FM_CUDA(cudaMemcpyAsync(&st, arena.stats, sizeof(st), cudaMemcpyDeviceToHost, s));
    FM_CUDA(cudaStreamSynchronize(s));
    if (st.first_bad != ~0ull) {
        uint64_t at = 0;
        FM_CUDA(cudaMemcpy(&at, starts + st.first_bad, 8, cudaMemcpyDeviceToHost));
        const char* line = body + at;
        const char* nl = (const char*)std::memchr(line, '\n', (size_t)(end - line));
        std::string txt(line, nl ? (size_t)(nl - line) : std::min<size_t>(40, (size_t)(end - line)));
        set_error("malformed or out-of-range data line: \"" + txt.substr(0, 80) + "\"");
        return FM_ERR_DATA_LINE;
    }
    const uint64_t E = st.kept;
    if (E > Ehdr) {
        set_error("more e-lines than the header's edge count");
        return FM_ERR_DATA_LINE;
    }
    if (!bound) d_text.reset();
    return build_from_keys(g, V, L, E, arena, s);
}

}  // namespace fm
