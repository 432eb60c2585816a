// Parquet column-chunk decode on the GPU: what MiniLake's read_column_chunk
// (crates/minilake-storage/src/parquet_reader.rs:215-294) gets from the parquet crate's column
// reader, then its conversions and encode_strings (:176-212).
//
// The host parses the chunk's page headers (Thrift compact protocol, parquet.thrift PageHeader)
// and copies the chunk to the device once.  Then, on the device:
//   1. Snappy pages are decompressed: pointer doubling over the stream's bytes lists every
//      element, then the compressor's independent 64 KB fragments resolve their copies by pointer
//      jumping (a page that does not split that way is decoded by one thread);
//   2. every RLE / bit-packed hybrid stream (definition levels, dictionary indices) gets a run
//      table (one warp per stream walks the run headers in a staged window of the stream);
//   3. definition levels give the validity bits, 32 rows per thread, and the present values per
//      8,192-row tile; a row's popcount rank in its tile gives its position among the chunk's
//      present values, and the value comes from its page (PLAIN, or a dictionary index into the
//      dictionary page) with the column's conversion (FLOAT -> f64, DECIMAL -> f64 / 10^scale);
//   4. strings get a dictionary in order of first occurrence when there are at most
//      clamp(rows / 8, 1, 65,536) distinct values, else are kept plain (encode_strings); NULL rows
//      count as "", as in the reference.  A chunk whose pages all index a small dictionary page
//      works on that page's entries; any other chunk's strings are materialized and canonicalized
//      with a device hash table.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "ml_api_common.hpp"
#include "ml_device.cuh"
#include "ml_kernels.cuh"
#include "ml_pipeline.hpp"

using namespace mlg;

namespace {

// parquet.thrift: Type, Encoding, PageType, CompressionCodec
enum PqType { PQ_BOOLEAN = 0, PQ_INT32 = 1, PQ_INT64 = 2, PQ_INT96 = 3, PQ_FLOAT = 4, PQ_DOUBLE = 5, PQ_BYTE_ARRAY = 6, PQ_FLBA = 7 };
enum PqEncoding { ENC_PLAIN = 0, ENC_PLAIN_DICTIONARY = 2, ENC_RLE = 3, ENC_BIT_PACKED = 4, ENC_RLE_DICTIONARY = 8 };
enum PqPageType { PAGE_DATA = 0, PAGE_INDEX = 1, PAGE_DICTIONARY = 2, PAGE_DATA_V2 = 3 };

// ---- Thrift compact protocol: just enough to read a PageHeader and skip the rest ------------
struct Compact {
    const uint8_t* p;
    const uint8_t* end;
    uint8_t byte() {
        if (p >= end) raise(ML_ERR_INVALID, "parquet: page header runs past the chunk");
        return *p++;
    }
    uint64_t varint() {
        uint64_t v = 0;
        for (int shift = 0; shift < 64; shift += 7) {
            const uint8_t b = byte();
            v |= (uint64_t)(b & 0x7F) << shift;
            if (!(b & 0x80)) return v;
        }
        raise(ML_ERR_INVALID, "parquet: bad varint in a page header");
    }
    int64_t zigzag() {
        const uint64_t v = varint();
        return (int64_t)(v >> 1) ^ -(int64_t)(v & 1);
    }
    void skip(int type) {
        switch (type) {
            case 1:
            case 2: return;  // bool in the field header
            case 3: byte(); return;
            case 4:
            case 5:
            case 6: varint(); return;
            case 7: need(8); p += 8; return;
            case 8: {
                const uint64_t n = varint();
                need(n);
                p += n;
                return;
            }
            case 9:
            case 10: {
                const uint8_t h = byte();
                uint64_t n = h >> 4;
                if (n == 15) n = varint();
                const int et = h & 15;
                for (uint64_t i = 0; i < n; i++) skip(et == 1 || et == 2 ? 3 : et);  // list bools are bytes
                return;
            }
            case 11: {
                const uint64_t n = varint();
                if (!n) return;
                const uint8_t kv = byte();
                for (uint64_t i = 0; i < n; i++) {
                    skip(kv >> 4 == 1 || kv >> 4 == 2 ? 3 : kv >> 4);
                    skip((kv & 15) == 1 || (kv & 15) == 2 ? 3 : kv & 15);
                }
                return;
            }
            case 12: {
                int16_t last = 0;
                for (;;) {
                    int fid, ft;
                    if (!field(last, fid, ft)) return;
                    skip(ft);
                }
            }
            default: raise(ML_ERR_INVALID, "parquet: unknown Thrift type " + std::to_string(type));
        }
    }
    void need(uint64_t n) {
        if ((uint64_t)(end - p) < n) raise(ML_ERR_INVALID, "parquet: page header runs past the chunk");
    }
    // Next field of a struct: false at its end.  `last` is the previous field id (delta encoding).
    bool field(int16_t& last, int& id, int& type) {
        const uint8_t h = byte();
        if (h == 0) return false;
        type = h & 15;
        const int delta = h >> 4;
        id = delta ? last + delta : (int16_t)zigzag();
        last = (int16_t)id;
        return true;
    }
};

struct Page {
    int type = -1;
    int64_t payload = 0;  // offset of the page's bytes in the chunk
    int32_t compressed = 0, uncompressed = 0;
    int32_t num_values = 0, encoding = 0, def_encoding = ENC_RLE;
    // DATA_PAGE_V2
    int32_t num_nulls = 0, def_bytes = 0, rep_bytes = 0;
    bool v2_compressed = true;
};

void read_data_header(Compact& c, Page& pg) {  // DataPageHeader
    int16_t last = 0;
    int id, t;
    while (c.field(last, id, t)) {
        if (id == 1 && t == 5) pg.num_values = (int32_t)c.zigzag();
        else if (id == 2 && t == 5) pg.encoding = (int32_t)c.zigzag();
        else if (id == 3 && t == 5) pg.def_encoding = (int32_t)c.zigzag();
        else c.skip(t);
    }
}
void read_dict_header(Compact& c, Page& pg) {  // DictionaryPageHeader
    int16_t last = 0;
    int id, t;
    while (c.field(last, id, t)) {
        if (id == 1 && t == 5) pg.num_values = (int32_t)c.zigzag();
        else if (id == 2 && t == 5) pg.encoding = (int32_t)c.zigzag();
        else c.skip(t);
    }
}
void read_v2_header(Compact& c, Page& pg) {  // DataPageHeaderV2
    int16_t last = 0;
    int id, t;
    while (c.field(last, id, t)) {
        if (id == 1 && t == 5) pg.num_values = (int32_t)c.zigzag();
        else if (id == 2 && t == 5) pg.num_nulls = (int32_t)c.zigzag();
        else if (id == 4 && t == 5) pg.encoding = (int32_t)c.zigzag();
        else if (id == 5 && t == 5) pg.def_bytes = (int32_t)c.zigzag();
        else if (id == 6 && t == 5) pg.rep_bytes = (int32_t)c.zigzag();
        else if (id == 7 && (t == 1 || t == 2)) pg.v2_compressed = t == 1;
        else c.skip(t);
    }
}

// Every page of a column chunk (the pages follow each other; a chunk starts with its
// dictionary page when it has one).
std::vector<Page> parse_pages(const uint8_t* chunk, int64_t n) {
    std::vector<Page> pages;
    int64_t pos = 0;
    while (pos < n) {
        Compact c{chunk + pos, chunk + n};
        Page pg;
        int16_t last = 0;
        int id, t;
        while (c.field(last, id, t)) {
            if (id == 1 && t == 5) pg.type = (int)c.zigzag();
            else if (id == 2 && t == 5) pg.uncompressed = (int32_t)c.zigzag();
            else if (id == 3 && t == 5) pg.compressed = (int32_t)c.zigzag();
            else if (id == 5 && t == 12) read_data_header(c, pg);
            else if (id == 7 && t == 12) read_dict_header(c, pg);
            else if (id == 8 && t == 12) read_v2_header(c, pg);
            else c.skip(t);
        }
        pg.payload = c.p - chunk;
        if (pg.compressed < 0 || pg.uncompressed < 0 || pg.payload + pg.compressed > n)
            raise(ML_ERR_INVALID, "parquet: a page runs past the chunk");
        pos = pg.payload + pg.compressed;
        if (pg.type == PAGE_DATA || pg.type == PAGE_DATA_V2 || pg.type == PAGE_DICTIONARY) pages.push_back(pg);
        else if (pg.type != PAGE_INDEX) raise(ML_ERR_UNSUPPORTED, "parquet: page type " + std::to_string(pg.type));
    }
    return pages;
}

}  // namespace

namespace {
constexpr uint32_t PQ_ERR_SNAPPY = 1, PQ_ERR_LAYOUT = 2, PQ_ERR_RUNS = 4, PQ_ERR_VALUES = 8;
constexpr int kPqTile = 8192;  // rows per decode tile: 256 threads x one 32-row validity word

// ---- 1. Snappy (the format's public description: a varint length, then literal and copy
// elements).  The element stream is sequential, but the compressor works on 64 KB fragments of
// its input and no match reaches back past its fragment's start, so a page of N fragments is N
// independent decodes once their starts in the stream are known.
//
// A page of few elements is copied by one block (k_pq_snappy_flat).  For any other page no pass follows
// the chain of elements one by one:
//  * the maps (one block per kSnapBlk stream bytes): for every byte, the element that WOULD start
//    there is parsed, and pointer doubling in shared memory (log2 of the elements in a block rounds)
//    gives where the chain from that byte leaves the block, how many elements it passes and how many
//    bytes they write;
//  * the chain (one warp per page) steps from block to block through those maps, which gives each
//    block the position its first element starts at;
//  * the list (one block per kSnapBlk bytes again): doubling from that position marks the real element
//    starts, and a scan numbers them and gives each its output position;
//  * the decode (one block per fragment): every output byte starts as a pointer to itself (literals) or
//    to the earlier output byte it copies, and pointer jumping in shared memory resolves all of them in
//    log2 of the longest copy chain rounds, whatever the order of the elements;
//  * a page whose elements cross a fragment boundary, or whose copies reach into an earlier fragment,
//    is decoded again by one thread from start to end (the serial pass), which is also the pass that
//    reports a malformed stream.
//
// Why: a page's elements are one dependent chain (a 977 KB dictionary page of doubles has ~247k of
// them), so a thread that follows it is bound by a shared-memory round trip per element whatever the
// chip has to offer.  Measured on such a page (125,000 prices, Snappy): one thread following the chain
// through per-window records 6.5 ms and a warp per fragment decoding 2.3 ms; now maps 22 us, chain
// 16 us, list 23 us and decode 58 us.
struct SnapJob {
    const uint8_t* src;
    uint8_t* dst;
    uint32_t src_len, dst_len;
    uint32_t plan;   // the page's plan in the plan buffer (SnapPlan)
    uint32_t nfrag;  // 64 KB fragments of its output
    uint32_t blk0;   // its first kSnapBlk block in the group's block array
    uint32_t pad_;
    uint64_t tab0;   // its first byte in the group's map table
    uint64_t elem0;  // its first element in the group's element list
};
// The plan of a page with n fragments: its mode, the first element's stream position, the number of every
// fragment's first element and of all elements, the stream positions of the former, and where the chain
// stopped ({stream position, output position, element}) when the page is taken in parts.
__host__ __device__ constexpr uint32_t snap_plan_words(uint32_t n) { return 2 * n + 6; }
__device__ __forceinline__ uint32_t snap_plan_pos(uint32_t n) { return n + 3; }
__device__ __forceinline__ uint32_t snap_plan_state(uint32_t n) { return 2 * n + 3; }
struct SnapMap {  // the chain from a stream byte to the end of its block
    uint32_t exit;  // stream position of the first element past the block, or kSnapNone
    uint32_t out;   // bytes the chain's elements write
    uint32_t count; // elements
    uint32_t pad_;
};
struct SnapEntry {  // a block's first element, as the page's chain reaches it
    uint32_t pos, out, elem, valid;  // stream position, output position, number; valid == 1 or unset
};
constexpr uint32_t kSnapFrag = 1u << 16;  // the compressor's fragment
constexpr uint32_t kSnapWin = 2048;       // the serial pass's window
// Stream bytes per map / list block: the chain takes a step (0.1 us, or a dependent L2 load where
// its guess is wrong) per block, a
// doubling round in a block costs eight shared-memory steps per thread, and 8 KB gives a 1 MB page 122
// blocks, one wave of the 148 SMs.
constexpr uint32_t kSnapBlk = 8192;
constexpr int kSnapThreads = 1024;
constexpr uint32_t kSnapPer = kSnapBlk / kSnapThreads;
constexpr uint32_t kSnapNone = 0xFFFFFFFFu;
// plan modes: 0 the length varint is malformed, 1 the serial pass decodes the page, 2 its
// fragments decode in parallel, 3 the chain goes on in the page's next part
constexpr uint32_t kSnapSerial = 1, kSnapSplit = 2, kSnapChain = 3;
constexpr uint32_t kSnapPiece = 2048, kSnapPieces = 2048;  // long literals, cut into pieces for the warps
constexpr size_t kSnapMapSmem = kSnapBlk * 8 + kSnapBlk + 32;
constexpr size_t kSnapFragSmem = kSnapFrag * 3 + kSnapPieces * 8;
// Stream bytes per group of pages decoded together: the maps take 16 bytes per stream byte, the element list
// four.  A larger page is a group of its own, taken in parts: the maps and the chain in parts of kSnapGroupBytes, then
// the list and the decode of the fragments that start in kSnapPart bytes.  The list of a part goes on for the
// stream of one fragment (an output byte takes six bytes at most: a literal with a four-byte length), and holds an
// element at its number modulo kSnapRing.
constexpr uint64_t kSnapGroupBytes = 32ull << 20;
constexpr uint32_t kSnapPart = (uint32_t)kSnapGroupBytes - (1u << 20), kSnapPast = 6 * kSnapFrag / kSnapBlk + 1;
constexpr uint32_t kSnapRing = 1u << 24;
static_assert(kSnapPart % kSnapBlk == 0 && (kSnapPart + kSnapPast * kSnapBlk) / 2 + 1 <= kSnapRing, "a part's elements");
static_assert((uint64_t)kSnapRing * 8 <= kSnapGroupBytes * 16, "the list takes the maps' place");

// One element header at s[0..avail): its size h (tag plus length or offset bytes), kind (0
// literal, 1 copy), output length and copy offset; false if it does not fit in `avail`.
__host__ __device__ __forceinline__ bool snap_hdr(const uint8_t* s, uint32_t avail, uint32_t& h, uint32_t& kind,
                                         uint32_t& len, uint32_t& off) {
    if (avail == 0) return false;
    const uint32_t tag = s[0], t = tag & 3;
    off = 0;
    if (t == 0) {
        kind = 0;
        len = tag >> 2;
        h = 1;
        if (len >= 60) {
            const uint32_t nb = len - 59;
            if (nb >= avail) return false;
            len = 0;
            for (uint32_t i = 0; i < nb; i++) len |= (uint32_t)s[1 + i] << (8 * i);
            h = 1 + nb;
        }
        len += 1;
        return len != 0 && len <= avail - h;  // 0: a four-byte length of 2^32
    }
    kind = 1;
    if (t == 1) {
        if (avail < 2) return false;
        h = 2;
        len = 4 + ((tag >> 2) & 7);
        off = ((tag >> 5) << 8) | s[1];
    } else {
        const uint32_t nb = t == 2 ? 2 : 4;
        if (avail < 1 + nb) return false;
        h = 1 + nb;
        len = (tag >> 2) + 1;
        for (uint32_t i = 0; i < nb; i++) off |= (uint32_t)s[1 + i] << (8 * i);
    }
    return true;
}

// The element that starts at w[0], of which `avail` stream bytes are left (w has five readable bytes):
// its bytes in the stream (header and a literal's bytes) and in the output; false when it does not
// fit.  Branch-free: the five bytes a header can span are read at once and every form is computed.
__device__ __forceinline__ bool snap_elem(const uint8_t* w, uint32_t avail, uint32_t& step, uint32_t& len) {
    const uint32_t b0 = w[0], b1 = w[1], b2 = w[2], b3 = w[3], b4 = w[4];
    const uint32_t t = b0 & 3, l6 = b0 >> 2;
    const uint32_t nb = l6 >= 60 ? l6 - 59 : 0;  // a literal's length bytes
    const uint32_t ext = b1 | (nb >= 2 ? b2 << 8 : 0u) | (nb >= 3 ? b3 << 16 : 0u) | (nb >= 4 ? b4 << 24 : 0u);
    const uint64_t lit = (uint64_t)(nb ? ext : l6) + 1;  // a literal's bytes (up to 2^32)
    const uint64_t st = t == 0 ? 1 + nb + lit : t == 1 ? 2 : t == 2 ? 3 : 5;
    step = (uint32_t)st;
    len = t == 0 ? (uint32_t)lit : t == 1 ? 4 + (l6 & 7) : l6 + 1;
    return avail > 0 && st <= (uint64_t)avail;
}

// The block loads src[b0, b0 + kSnapBlk + 5) (to the stream's end at most) into `win` with aligned
// 16-byte loads, from the 16-byte boundary at or below (the chunk buffer is padded past its end);
// win + the returned lead is src + b0.
__device__ __forceinline__ uint32_t snap_window(const SnapJob& J, uint32_t b0, uint8_t* win) {
    const uintptr_t a = (uintptr_t)(J.src + b0);
    const uint4* v = (const uint4*)(a & ~(uintptr_t)15);
    const uint32_t lead = (uint32_t)(a & 15);
    const uint64_t need = ((uint64_t)(J.src_len - b0) + lead + 15) / 16;
    const uint32_t nvec = (uint32_t)(need < kSnapBlk / 16 + 2 ? need : kSnapBlk / 16 + 2);
    for (uint32_t i = threadIdx.x; i < nvec; i += kSnapThreads) ((uint4*)win)[i] = __ldg(v + i);
    return lead;
}

// Eight bytes from any address (in the padded chunk or page buffer: the aligned words around them
// are readable).
__device__ uint64_t load8(const uint8_t* p) {
    const uint64_t* b = (const uint64_t*)((uintptr_t)p & ~(uintptr_t)7);
    const int sh = 8 * (int)((uintptr_t)p & 7);
    const uint64_t lo = b[0];
    return sh ? (lo >> sh) | (b[1] << (64 - sh)) : lo;
}

// Pages of few elements, one block per page: pages that do not compress (bit-packed random indices,
// random numbers) are a few long literals, perhaps with a stray copy.  The host, which parses the page
// headers, follows the elements as long as they span kSnapFlatSpan stream bytes on average, at most
// kSnapFlat of them (flat_elements: a few cache lines of the page), or kSnapFlatTiny of a page of at most
// kSnapTiny bytes (a small dictionary page); a page that ends by then is not one of the passes' pages, and the
// block copies its literals, then one warp its copies in order (in shared memory for a tiny page: 49 copies
// 12 us).  Seven pages of 18,000 two-bit indices: 55 us in the six launches of the passes below, 3.6 us in one
// here (4.8 us when the device followed the elements, and 16 for the passes to find nothing to do).
constexpr int kSnapFlat = 64;
constexpr uint32_t kSnapFlatSpan = 256;
constexpr uint32_t kSnapTiny = 4096;
constexpr int kSnapFlatTiny = 256;
struct SnapFlat {
    const uint8_t* src;
    uint8_t* dst;
    uint32_t dst_len, tiny;  // tiny: at most kSnapTiny bytes, and not literals alone
    uint32_t el0, n;  // its elements: {stream position of a literal's bytes, output position, length, copy offset (0: literal)}
};
bool flat_elements(const uint8_t* s, uint32_t len, uint32_t out_len, std::vector<uint4>& el) {
    uint32_t pos = 0, total = 0;
    bool ok = false;
    for (int shift = 0; shift < 35 && pos < len; shift += 7) {  // the uncompressed length
        const uint32_t b = s[pos++];
        if (shift == 28 && (b & 0x70)) break;  // past 32 bits
        total |= (b & 0x7F) << shift;
        if (!(b & 0x80)) {
            ok = total == out_len;
            break;
        }
    }
    const size_t el0 = el.size();
    const uint32_t start = pos;
    uint32_t out = 0, n = 0;
    for (; ok && pos < len; n++) {
        uint32_t h, kind, l, off;
        ok = (out_len <= kSnapTiny ? n < (uint32_t)kSnapFlatTiny
                                   : n < (uint32_t)kSnapFlat && (n < 2 || pos - start >= n * kSnapFlatSpan)) &&
             snap_hdr(s + pos, len - pos, h, kind, l, off) &&
             l <= out_len - out && (kind == 0 || (off != 0 && off <= out));
        if (!ok) break;
        el.push_back(make_uint4(pos + h, out, l, off));
        pos += h + (kind == 0 ? l : 0);
        out += l;
    }
    ok = ok && out == out_len;
    if (!ok) el.resize(el0);  // the passes decode it, or report it
    return ok;
}
__global__ void __launch_bounds__(kSnapThreads) k_pq_snappy_flat(const SnapFlat* pages, const uint4* elems) {
    __shared__ uint4 el[kSnapFlatTiny];
    __shared__ uint8_t tiny[kSnapTiny];
    const SnapFlat J = pages[blockIdx.x];
    const uint32_t tid = threadIdx.x;
    const int n = (int)J.n;
    if ((int)tid < n) el[tid] = elems[J.el0 + tid];
    __syncthreads();
    if (J.tiny) {
        for (int k = tid >> 5; k < n; k += kSnapThreads / 32) {  // a warp per literal
            const uint4 e = el[k];
            if (!e.w)
                for (uint32_t i = tid & 31; i < e.z; i += 32) tiny[e.y + i] = J.src[e.x + i];
        }
        __syncthreads();
        if (tid < 32)
            for (int k = 0; k < n; k++) {
                const uint4 e = el[k];
                if (!e.w) continue;
                for (uint32_t i = tid; i < e.z; i += 32) tiny[e.y + i] = tiny[e.y - e.w + (i < e.w ? i : i % e.w)];  // a copy over itself repeats
                __syncwarp();
            }
        __syncthreads();
        for (uint32_t i = tid; i < J.dst_len; i += kSnapThreads) J.dst[i] = tiny[i];
        return;
    }
    for (int k = 0; k < n; k++) {
        const uint4 e = el[k];
        if (e.w) continue;
        const uint8_t* src = J.src + e.x;
        uint8_t* d = J.dst + e.y;
        const uint32_t lead = min((uint32_t)((8 - ((uintptr_t)d & 7)) & 7), e.z), words = (e.z - lead) / 8;
        for (uint32_t i = tid; i < words; i += kSnapThreads) ((uint64_t*)(d + lead))[i] = load8(src + lead + 8ull * i);
        const uint32_t tail = lead + words * 8;
        if (tid < lead) d[tid] = src[tid];
        else if (tid >= 32 && tail + tid - 32 < e.z) d[tail + tid - 32] = src[tail + tid - 32];
    }
    __syncthreads();
    if (tid >= 32) return;
    for (int k = 0; k < n; k++) {
        const uint4 e = el[k];
        if (!e.w) continue;
        for (uint32_t i = tid; i < e.z; i += 32) J.dst[e.y + i] = J.dst[e.y - e.w + (i < e.w ? i : i % e.w)];  // a copy over itself repeats
        __syncwarp();
    }
}

// The maps: blocks[i] = {page, block}.  A byte's state packs the element reached (16 bits, a block
// offset), the elements passed (16) and the bytes they write (32); an element whose successor lies
// past the block (or that does not parse) points to itself.  States only ever move further along the
// chain and are read and written whole, so the rounds need no second buffer: bound by shared-memory
// round trips, log2(kSnapBlk / 2) of them.
// `lo`: the stream byte that the table starts at (0, or a part's first).
__global__ void __launch_bounds__(kSnapThreads) k_pq_snappy_maps(const SnapJob* jobs, const uint2* blocks, SnapMap* tab, uint32_t lo) {
    extern __shared__ __align__(16) uint8_t snap_smem[];
    uint64_t* st = (uint64_t*)snap_smem;
    uint8_t* win = snap_smem + kSnapBlk * 8;
    const uint2 f = blocks[blockIdx.x];
    const SnapJob J = jobs[f.x];
    const uint32_t b0 = f.y * kSnapBlk, blen = min(kSnapBlk, J.src_len - b0);
    const uint8_t* w = win + snap_window(J, b0, win);
    __syncthreads();
    uint64_t v[kSnapPer];
#pragma unroll
    for (uint32_t e = 0; e < kSnapPer; e++) {
        const uint32_t q = threadIdx.x + e * kSnapThreads;
        uint32_t step, len;
        const bool ok = q < blen && snap_elem(w + q, J.src_len - b0 - q, step, len);
        v[e] = ok && step < blen - q ? (uint64_t)(q + step) | (1ull << 16) | ((uint64_t)len << 32) : (uint64_t)q;
        st[q] = v[e];
    }
    uint32_t open = (1u << kSnapPer) - 1;  // states that may still move
    while (__syncthreads_or(open != 0)) {
#pragma unroll
        for (uint32_t e = 0; e < kSnapPer; e++) {
            if (!((open >> e) & 1)) continue;
            const uint32_t p = (uint32_t)v[e] & 0xFFFFu;
            const uint64_t x = *(volatile uint64_t*)(st + p);
            if (((uint32_t)x & 0xFFFFu) == p) {
                open &= ~(1u << e);
            } else {
                v[e] = (x & 0xFFFFull) | (((v[e] >> 16) + (x >> 16)) << 16);
                *(volatile uint64_t*)(st + threadIdx.x + e * kSnapThreads) = v[e];
            }
        }
    }
#pragma unroll
    for (uint32_t e = 0; e < kSnapPer; e++) {
        const uint32_t q = threadIdx.x + e * kSnapThreads;
        if (q >= blen) continue;
        const uint32_t p = (uint32_t)v[e] & 0xFFFFu;  // the chain's last element in the block
        uint32_t step, len;
        SnapMap m{kSnapNone, 0, 0, 0};
        if (snap_elem(w + p, J.src_len - b0 - p, step, len))
            m = SnapMap{b0 + p + step, (uint32_t)(v[e] >> 32) + len, ((uint32_t)(v[e] >> 16) & 0xFFFFu) + 1u, 0};
        *(uint4*)(tab + J.tab0 + (b0 - lo) + q) = *(const uint4*)&m;
    }
}

// The chain, one warp per page: the page's mode, each block's entry, and the number of elements.
// A block's entry is known when the chain has left the block before it: one dependent L2 load per block (42 us
// for the 89 blocks of a 721 KB stream).  But chains that start at different bytes soon meet, so where the chain
// from a block's first byte leaves it is mostly where the real one does: the lanes load the next 32 blocks' maps at
// those places together, and the walk takes a lane's map where its guess is right (15.5 us), else loads it.
// The maps are those of the stream bytes [lo, hi) (a page's part; all of it otherwise): the chain goes on where
// it left the part before.
__global__ void __launch_bounds__(32) k_pq_snappy_chain(const SnapJob* jobs, const SnapMap* tab, SnapEntry* entries,
                                                        uint32_t* plan, uint32_t lo, uint32_t hi) {
    const uint32_t lane = threadIdx.x;
    const SnapJob J = jobs[blockIdx.x];
    uint32_t* pl = plan + J.plan;
    uint32_t* const state = pl + snap_plan_state(J.nfrag);
    const uint32_t end = min(J.src_len, hi);
    uint32_t start = 0, total = 0;
    bool ok = false;
    if (lo && pl[0] != kSnapChain) return;
    for (int shift = 0; shift < 35 && start < J.src_len; shift += 7) {  // the uncompressed length
        const uint32_t b = J.src[start++];
        if (shift == 28 && (b & 0x70)) break;  // past 32 bits
        total |= (b & 0x7F) << shift;
        if (!(b & 0x80)) {
            ok = true;
            break;
        }
    }
    if (lane == 0) pl[1] = start;
    if (!ok || total != J.dst_len) {
        if (lane == 0) pl[0] = 0;
        return;
    }
    const SnapMap* maps = tab + J.tab0;
    bool split = J.nfrag >= 1;
    uint32_t pos = lo ? state[0] : start, elem = lo ? state[2] : 0;
    uint64_t out = lo ? state[1] : 0;
    __syncwarp();  // before lane 0 writes them
    uint32_t g0 = 0, guess = kSnapNone;  // lane l holds block g0 + l's guessed entry and the map there
    uint4 gm = make_uint4(kSnapNone, 0, 0, 0);
    bool held = false;
    while (split && pos < end) {  // the same in every lane
        const uint32_t blk = pos / kSnapBlk;
        if (!held || blk - g0 >= 32) {
            g0 = blk;
            held = true;
            const uint64_t mine = (uint64_t)g0 + lane;
            guess = lane == 0 ? pos : mine * kSnapBlk < end ? maps[(mine - 1) * kSnapBlk - lo].exit : kSnapNone;
            if (guess >= end || guess / kSnapBlk != mine) guess = kSnapNone;
            if (guess != kSnapNone) gm = __ldg((const uint4*)(maps + (guess - lo)));
        }
        const int from = (int)(blk - g0);
        uint4 m;
        m.x = __shfl_sync(0xFFFFFFFFu, gm.x, from);
        m.y = __shfl_sync(0xFFFFFFFFu, gm.y, from);
        m.z = __shfl_sync(0xFFFFFFFFu, gm.z, from);
        if (__shfl_sync(0xFFFFFFFFu, guess, from) != pos) m = __ldg((const uint4*)(maps + (pos - lo)));
        if (lane == 0) entries[J.blk0 + blk] = SnapEntry{pos, (uint32_t)out, elem, 1u};
        out += m.y;
        elem += m.z;
        pos = m.x;  // past pos: an element spans at least two bytes
        split = m.x != kSnapNone && out <= total;
    }
    if (lane) return;
    if (split && pos < J.src_len) {
        state[0] = pos, state[1] = (uint32_t)out, state[2] = elem;
        pl[0] = kSnapChain;
    } else if (split && out == total) {
        pl[2 + J.nfrag] = elem;
        pl[0] = kSnapSplit;
    } else {
        pl[0] = kSnapSerial;
    }
}

// The list: each real element's stream and output position, in order, and the number of every
// fragment's first element.  Marks start at the block's entry; round k marks the elements 2^k after
// the marked ones while the jumps double, so all are marked after log2 of their number rounds (a
// mark set early by a neighbour's write of the same round is a real element too).
__global__ void __launch_bounds__(kSnapThreads) k_pq_snappy_list(const SnapJob* jobs, const uint2* blocks,
                                                                 const SnapEntry* entries, uint32_t* plan, uint2* elems,
                                                                 uint32_t elem_mask) {
    __shared__ __align__(16) uint16_t jmp[kSnapBlk];
    __shared__ __align__(16) uint8_t mark[kSnapBlk];
    __shared__ __align__(16) uint8_t win[kSnapBlk + 32];
    __shared__ uint64_t wsum[kSnapThreads / 32];
    const uint2 f = blocks[blockIdx.x];
    const SnapJob J = jobs[f.x];
    uint32_t* pl = plan + J.plan;
    const SnapEntry E = entries[J.blk0 + f.y];
    if (E.valid != 1u || pl[0] == 0) return;
    const uint32_t tid = threadIdx.x, b0 = f.y * kSnapBlk, blen = min(kSnapBlk, J.src_len - b0);
    const uint8_t* w = win + snap_window(J, b0, win);
    for (uint32_t i = tid; i < kSnapBlk / 16; i += kSnapThreads) ((uint4*)mark)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
#pragma unroll
    for (uint32_t e = 0; e < kSnapPer; e++) {
        const uint32_t q = tid + e * kSnapThreads;
        uint32_t step, len;
        const bool ok = q < blen && snap_elem(w + q, J.src_len - b0 - q, step, len);
        jmp[q] = (uint16_t)(ok && step < blen - q ? q + step : 0xFFFFu);
    }
    if (tid == 0) mark[E.pos - b0] = 1;
    for (;;) {
        __syncthreads();
        uint32_t nj[kSnapPer / 2];  // two jumps per register
        uint32_t all = 0xFFFFu;
#pragma unroll
        for (uint32_t e = 0; e < kSnapPer; e++) {
            const uint32_t q = tid + e * kSnapThreads, j = jmp[q];
            uint32_t x = 0xFFFFu;
            if (j != 0xFFFFu) {
                x = jmp[j];
                if (*(volatile uint8_t*)(mark + q)) *(volatile uint8_t*)(mark + j) = 1;
            }
            all &= x;
            nj[e / 2] = e & 1 ? nj[e / 2] | (x << 16) : x;
        }
        if (!__syncthreads_or(all != 0xFFFFu)) break;
#pragma unroll
        for (uint32_t e = 0; e < kSnapPer; e++) jmp[tid + e * kSnapThreads] = (uint16_t)(nj[e / 2] >> (16 * (e & 1)));
    }
    // number the marked elements and sum their output lengths: eight consecutive bytes per thread
    const uint64_t marks = ((const uint64_t*)mark)[tid];
    uint32_t cnt = 0, sum = 0;
    auto length = [&](uint32_t e) {  // parses: the chain passed through it
        const uint32_t q = tid * kSnapPer + e;
        uint32_t step, len;
        snap_elem(w + q, J.src_len - b0 - q, step, len);
        return len;
    };
    for (uint32_t e = 0; e < kSnapPer; e++)
        if ((marks >> (8 * e)) & 1) {
            cnt++;
            sum += length(e);
        }
    const uint64_t mine = ((uint64_t)cnt << 32) | sum;  // the block's bytes fit 32 bits (the page's do)
    uint64_t incl = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint64_t t = __shfl_up_sync(~0u, incl, d);
        if ((int)(tid & 31) >= d) incl += t;
    }
    if ((tid & 31) == 31) wsum[tid >> 5] = incl;
    __syncthreads();
    if (tid < 32) {
        uint64_t x = wsum[tid];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint64_t t = __shfl_up_sync(~0u, x, d);
            if ((int)tid >= d) x += t;
        }
        wsum[tid] = x;
    }
    __syncthreads();
    const uint64_t before = incl - mine + (tid >= 32 ? wsum[(tid >> 5) - 1] : 0ull);
    uint32_t i = E.elem + (uint32_t)(before >> 32), o = E.out + (uint32_t)before;
    bool bad = false;
    for (uint32_t e = 0; e < kSnapPer; e++) {
        if (!((marks >> (8 * e)) & 1)) continue;
        const uint32_t l = length(e), at = o & (kSnapFrag - 1);
        elems[J.elem0 + (i & elem_mask)] = make_uint2(b0 + tid * kSnapPer + e, o);
        bad = bad || l > kSnapFrag - at;  // crossing a fragment's end
        if (at == 0 && (o >> 16) < J.nfrag) {
            pl[2 + (o >> 16)] = i;
            pl[snap_plan_pos(J.nfrag) + (o >> 16)] = b0 + tid * kSnapPer + e;
        }
        i++;
        o += l;
    }
    if (bad) atomicExch(pl, kSnapSerial);
}

// The decode, one block per fragment of a split page (frags[i] = {page, fragment}); a fragment that
// does not decode as a unit hands its page to the serial pass.  `ptr` holds, per output byte, the
// earlier output byte it equals (itself for a literal's byte, whose value is in `val`); jumping
// ptr[i] = ptr[ptr[i]] until nothing moves ends at literal bytes.  A copy overlapping itself points
// into the pattern it repeats.  192 KB of shared memory, so one block per SM: bound by the
// shared-memory gathers of the rounds (64 bytes per thread and round, resolved pairs skipped).
// Of a page in parts, the fragments that start in the stream bytes [lo, hi); all of them otherwise.
__global__ void __launch_bounds__(kSnapThreads) k_pq_snappy_frag(const SnapJob* jobs, const uint2* frags, const uint2* elems,
                                                                 uint32_t* plan, uint32_t elem_mask, uint32_t lo, uint32_t hi) {
    extern __shared__ __align__(16) uint8_t snap_smem[];
    uint16_t* ptr = (uint16_t*)snap_smem;
    uint8_t* val = snap_smem + kSnapFrag * 2;
    uint2* piece = (uint2*)(val + kSnapFrag);
    __shared__ uint32_t npiece;
    const uint2 f = frags[blockIdx.x];
    const SnapJob J = jobs[f.x];
    uint32_t* pl = plan + J.plan;
    __shared__ uint32_t mode;  // one read: another fragment's block may hand the page over meanwhile
    if (threadIdx.x == 0) {
        mode = *(volatile uint32_t*)pl;
        npiece = 0;
        const uint32_t pos = pl[snap_plan_pos(J.nfrag) + f.y];
        if (pos < lo || pos >= hi) mode = 0;
    }
    __syncthreads();
    if (mode != kSnapSplit) return;
    const uint32_t tid = threadIdx.x, o0 = f.y * kSnapFrag, n = min(J.dst_len - o0, kSnapFrag);
    for (uint32_t i = tid; i < kSnapFrag / 8; i += kSnapThreads) {  // every byte its own source
        const uint32_t b = i * 8;
        ((uint4*)ptr)[i] = make_uint4(b | ((b + 1) << 16), (b + 2) | ((b + 3) << 16), (b + 4) | ((b + 5) << 16), (b + 6) | ((b + 7) << 16));
    }
    __syncthreads();
    bool bad = false;
    const uint2* E = elems + J.elem0;
#pragma unroll 1
    for (uint32_t i = pl[2 + f.y] + tid, i1 = pl[3 + f.y]; i < i1; i += kSnapThreads) {
        const uint2 el = E[i & elem_mask];
        const uint8_t* e = J.src + el.x;  // five readable bytes: the chunk buffer is padded past its end
        const uint32_t o = el.y - o0;
        uint32_t step, len;
        if (!snap_elem(e, J.src_len - el.x, step, len) || o >= n || len > n - o) {
            bad = true;
            continue;
        }
        const uint32_t t = e[0] & 3;
        const uint32_t off = t == 1 ? ((uint32_t)(e[0] >> 5) << 8) | e[1]
                                    : e[1] | ((uint32_t)e[2] << 8) | (t == 3 ? ((uint32_t)e[3] << 16) | ((uint32_t)e[4] << 24) : 0u);
        if (t == 0) {
            const uint32_t s = el.x + step - len;
            if (len <= 32) {
#pragma unroll 4
                for (uint32_t j = 0; j < len; j++) val[o + j] = __ldg(J.src + s + j);
            } else {  // by the warps, in pieces (at most n / 33 + n / kSnapPiece of them)
                const uint32_t np = (len + kSnapPiece - 1) / kSnapPiece, k0 = atomicAdd(&npiece, np);
#pragma unroll 1
                for (uint32_t k = 0; k < np; k++)
                    piece[k0 + k] = make_uint2(s + k * kSnapPiece, (o + k * kSnapPiece) | (min(kSnapPiece, len - k * kSnapPiece) << 16));
            }
        } else if (off == 0 || off > o) {  // before the fragment
            bad = true;
        } else {
            uint32_t p = o - off;
#pragma unroll 1
            for (uint32_t j = 0; j < len; j++) {
                ptr[o + j] = (uint16_t)p;
                p = p + 1 == o ? o - off : p + 1;
            }
        }
    }
    if (__syncthreads_or(bad)) {
        if (tid == 0) atomicExch(pl, kSnapSerial);
        return;
    }
    for (uint32_t k = tid >> 5; k < npiece; k += kSnapThreads / 32) {
        const uint2 pc = piece[k];
        const uint32_t o = pc.y & 0xFFFFu, len = pc.y >> 16;
        for (uint32_t j = tid & 31; j < len; j += 32) val[o + j] = __ldg(J.src + pc.x + j);
    }
    const uint32_t words = (n + 1) / 2;  // two bytes' pointers per word
    uint32_t open = 0;
#pragma unroll
    for (uint32_t k = 0; k < kSnapFrag / 2 / kSnapThreads; k++)
        if (tid + k * kSnapThreads < words) open |= 1u << k;
    volatile uint32_t* pw = (volatile uint32_t*)ptr;
    const volatile uint16_t* ph = (const volatile uint16_t*)ptr;
    while (__syncthreads_or(open != 0)) {
#pragma unroll 2
        for (uint32_t k = 0; k < kSnapFrag / 2 / kSnapThreads; k++) {
            if (!((open >> k) & 1)) continue;
            const uint32_t x = pw[tid + k * kSnapThreads];
            const uint32_t y = (uint32_t)ph[x & 0xFFFFu] | ((uint32_t)ph[x >> 16] << 16);
            if (x == y) open &= ~(1u << k);
            else pw[tid + k * kSnapThreads] = y;
        }
    }
    uint8_t* d = J.dst + o0;
    if (((uintptr_t)d & 15) == 0) {
#pragma unroll 1
        for (uint32_t i = tid; i < n / 16; i += kSnapThreads) {
            uint32_t r[4];
            const uint4 pa = ((const uint4*)ptr)[2 * i], pb = ((const uint4*)ptr)[2 * i + 1];
            const uint32_t pp[8] = {pa.x, pa.y, pa.z, pa.w, pb.x, pb.y, pb.z, pb.w};
#pragma unroll
            for (int k = 0; k < 4; k++)
                r[k] = val[pp[2 * k] & 0xFFFFu] | (val[pp[2 * k] >> 16] << 8) | (val[pp[2 * k + 1] & 0xFFFFu] << 16) |
                       ((uint32_t)val[pp[2 * k + 1] >> 16] << 24);
            ((uint4*)d)[i] = make_uint4(r[0], r[1], r[2], r[3]);
        }
        for (uint32_t i = (n & ~15u) + tid; i < n; i += kSnapThreads) d[i] = val[ptr[i]];
    } else {
        for (uint32_t i = tid; i < n; i += kSnapThreads) d[i] = val[ptr[i]];
    }
}

// One thread's decode of the elements in [pos, end) into dst[out, out_end); copies may not reach
// below `floor`.  The serial pass: source bytes come through the thread's shared-memory window.
struct SnapSrc {
    const uint8_t* src;
    uint32_t len;
    uint8_t* win;
    int64_t wbase = 0, wend = 0;  // the window holds src[wbase, wend) (wbase may be below 0)
    __device__ uint32_t at(uint32_t p) {  // p < len
        if ((int64_t)p < wbase || (int64_t)p >= wend) {
            const uintptr_t a = (uintptr_t)(src + p);
            const uint4* v = (const uint4*)(a & ~(uintptr_t)15);
            const int64_t lead = (int64_t)(a & 15);
            const uint64_t need = ((uint64_t)(len - p) + (uint64_t)lead + 15) / 16;
            const uint32_t nvec = (uint32_t)(need < kSnapWin / 16 ? need : kSnapWin / 16);
            for (uint32_t i = 0; i < nvec; i += 4) {  // 4 loads in flight, then their stores
                uint4 r[4];
#pragma unroll
                for (uint32_t k = 0; k < 4; k++)
                    if (i + k < nvec) r[k] = __ldg(v + i + k);
#pragma unroll
                for (uint32_t k = 0; k < 4; k++)
                    if (i + k < nvec) ((uint4*)win)[i + k] = r[k];
            }
            wbase = (int64_t)p - lead;
            wend = wbase + 16 * (int64_t)nvec;
        }
        return win[(int64_t)p - wbase];
    }
};

__device__ bool snap_decode_serial(SnapSrc& S, uint32_t pos, uint32_t end, uint8_t* dst, uint32_t out_end) {
    uint32_t out = 0;
    while (out < out_end) {
        if (pos >= end) return false;
        uint8_t hb[5];
        const uint32_t avail = end - pos, nh = avail < 5 ? avail : 5;
        for (uint32_t i = 0; i < nh; i++) hb[i] = (uint8_t)S.at(pos + i);
        uint32_t h, kind, len, off;
        if (!snap_hdr(hb, avail, h, kind, len, off) || len > out_end - out) return false;
        pos += h;
        if (kind == 0) {
            for (uint32_t i = 0; i < len; i++) dst[out + i] = (uint8_t)S.at(pos + i);
            pos += len;
        } else {
            if (off == 0 || off > out) return false;
            for (uint32_t i = 0; i < len; i++) dst[out + i] = dst[out + i - off];  // may overlap itself
        }
        out += len;
    }
    return pos == end;
}

// The serial pass, one thread per page not decoded by fragments: it decodes the page from start
// to end or reports it malformed.
__global__ void __launch_bounds__(32) k_pq_snappy_serial(const SnapJob* jobs, const uint32_t* plan, uint32_t* err) {
    __shared__ __align__(16) uint8_t win[kSnapWin + 16];
    if (threadIdx.x) return;
    const SnapJob J = jobs[blockIdx.x];
    const uint32_t* pl = plan + J.plan;
    const uint32_t mode = pl[0];
    if (mode == kSnapSplit) return;
    SnapSrc S{J.src, J.src_len, win};
    if (mode != kSnapSerial || !snap_decode_serial(S, pl[1], J.src_len, J.dst, J.dst_len)) atomicOr(err, PQ_ERR_SNAPPY);
}

// ---- 2. page layout and RLE / bit-packed hybrid run tables -----------------------------------
struct Run {
    uint32_t first, count;  // value index (in the stream) of the run's first value; its values
    uint32_t value;         // RLE run: the repeated value; bit-packed run: its byte offset
    uint32_t packed;
};

struct PageDev {
    const uint8_t* data;  // the page's uncompressed payload
    uint32_t len;
    int32_t v2, def_bytes, rep_bytes;  // DATA_PAGE_V2: level byte lengths
    int32_t encoding;
    int64_t row0;
    uint32_t nrows;
    // filled by k_pq_levels
    const uint8_t* levels;
    uint32_t levels_len;
    const uint8_t* values;
    uint32_t values_len;
    int32_t idx_width;  // dictionary-index (or RLE boolean) bit width; -1: PLAIN values
    // run tables from the page's first row on: of the levels (k_pq_levels) and of the indices (k_pq_indices)
    uint64_t lv_run0, ix_run0;
    uint32_t lv_nruns, ix_nruns;
    uint64_t valid0;  // present values of the chunk before this page's first row (k_pq_indices)
};

__device__ uint32_t le32(const uint8_t* p) { return p[0] | (p[1] << 8) | (p[2] << 16) | ((uint32_t)p[3] << 24); }

__device__ void page_layout(PageDev& p, int max_def, uint32_t* err) {
    uint32_t pos = 0;
    p.levels = nullptr;
    p.levels_len = 0;
    if (p.v2) {
        pos = (uint32_t)p.rep_bytes + (uint32_t)p.def_bytes;
        if (max_def > 0) {
            p.levels = p.data + p.rep_bytes;
            p.levels_len = (uint32_t)p.def_bytes;
        }
    } else if (max_def > 0) {
        if (p.len < 4 || le32(p.data) > p.len - 4) {
            atomicOr(err, PQ_ERR_LAYOUT);
            p.values_len = 0;
            p.idx_width = -1;
            return;
        }
        p.levels = p.data + 4;
        p.levels_len = le32(p.data);
        pos = 4 + p.levels_len;
    }
    if (pos > p.len) {
        atomicOr(err, PQ_ERR_LAYOUT);
        pos = p.len;
    }
    p.values = p.data + pos;
    p.values_len = p.len - pos;
    p.idx_width = -1;
    if (p.encoding == ENC_RLE_DICTIONARY || p.encoding == ENC_PLAIN_DICTIONARY) {
        if (p.values_len < 1 || p.values[0] > 32) {
            atomicOr(err, PQ_ERR_LAYOUT);
            return;
        }
        p.idx_width = p.values[0];
        p.values += 1;
        p.values_len -= 1;
    } else if (p.encoding == ENC_RLE) {  // RLE booleans: a 4-byte length, then the hybrid stream
        if (p.values_len < 4 || le32(p.values) > p.values_len - 4) {
            atomicOr(err, PQ_ERR_LAYOUT);
            return;
        }
        p.values_len = le32(p.values);
        p.values += 4;
        p.idx_width = 1;
    }
}

// A stream read by one warp through a window of shared memory: 16-byte loads from the 16-byte
// boundary at or before the wanted byte.  Every stream lies in the uncompressed-page buffer, which
// is 16-byte aligned at its start and padded by 64 bytes at its end.
constexpr uint32_t kPqWindow = 8192;
struct StreamWindow {
    const uint8_t* s;
    uint32_t len;
    uint4* win;       // kPqWindow bytes and 16 more for peek8
    uint32_t lo, hi;  // stream bytes [lo, hi) are in the window, byte lo at win + skew
    uint32_t skew;

    __device__ StreamWindow(const uint8_t* s_, uint32_t len_, uint4* w) : s(s_), len(len_), win(w), lo(0), hi(0), skew(0) {}
    // Bytes [pos, min(pos + n, len)) readable by at(); n <= kPqWindow - 16.  The whole warp calls it.
    __device__ void need(uint32_t pos, uint32_t n) {
        if (pos >= lo && (hi >= len || (uint64_t)pos + n <= hi)) return;
        if (pos >= len) return;
        skew = (uint32_t)((uintptr_t)(s + pos) & 15);
        lo = pos;
        const uint32_t take = len - pos < kPqWindow - skew ? len - pos : kPqWindow - skew;
        hi = pos + take;
        const uint4* src = (const uint4*)(s + pos - skew);
        __syncwarp();
        // all loads in flight at once: four at a time made a refill 2.8 us
        const uint32_t nvec = (skew + take + 15) / 16;
        uint4 v[kPqWindow / 512];
#pragma unroll
        for (uint32_t j = 0; j < kPqWindow / 512; j++) {
            const uint32_t i = j * 32 + (threadIdx.x & 31);
            if (i < nvec) v[j] = src[i];
        }
#pragma unroll
        for (uint32_t j = 0; j < kPqWindow / 512; j++) {
            const uint32_t i = j * 32 + (threadIdx.x & 31);
            if (i < nvec) win[i] = v[j];
        }
        __syncwarp();
    }
    __device__ uint32_t at(uint32_t pos) const { return ((const uint8_t*)win)[skew + (pos - lo)]; }
    __device__ uint32_t at32(uint32_t pos) const { return (uint32_t)peek8(pos); }
    __device__ uint64_t peek8(uint32_t pos) const {  // bytes past hi are whatever the window holds
        const uint32_t b = skew + (pos - lo), sh = 8 * (b & 3);
        const uint32_t* w = (const uint32_t*)win + (b >> 2);
        const uint32_t w0 = w[0], w1 = w[1], w2 = w[2];
        return (uint64_t)__funnelshift_r(w0, w1, sh) | ((uint64_t)__funnelshift_r(w1, w2, sh) << 32);
    }
};

// Walk a hybrid stream of `n` values with bit width `bw` and write its runs: one warp, every lane
// the same steps.  A writer fills bit-packed runs to one size, so after such a run each lane looks
// where the i-th run of that size would start; the headers agree up to some lane, and the walk goes
// on from there.  Short runs are looked up in the window, long ones (whose headers lie too far apart
// for it) in memory.  Returns the number of runs, or -1 when the stream is malformed.
__device__ int64_t rle_walk(const uint8_t* s, uint32_t len, uint32_t n, int bw, Run* runs, uint4* win) {
    StreamWindow S(s, len, win);
    const uint32_t lane = threadIdx.x & 31;
    uint32_t pos = 0, got = 0;
    int64_t k = 0;
    const uint32_t vbytes = (bw + 7) / 8;
    while (got < n) {
        if (pos >= len) return -1;
        S.need(pos, 16);  // a header (at most 6 bytes) and a value (at most 4)
        const uint64_t w = S.peek8(pos);
        const int hb = __ffsll((long long)(~w & 0x808080808080ull)) / 8;  // header bytes
        if (hb == 0 || (uint64_t)pos + hb > len) return -1;
        uint64_t h = w & 0x7F;
        for (int i = 1; i < hb; i++) h |= ((w >> (8 * i)) & 0x7F) << (7 * i);
        const uint32_t left = n - got;
        if (h & 1) {  // bit-packed: (h >> 1) groups of 8 values (none: malformed, every run holds a value)
            const uint64_t vals = (h >> 1) * 8, bytes = (h >> 1) * (uint64_t)bw, stride = hb + bytes;
            if (vals == 0 || pos + stride > len) return -1;
            const uint64_t at = pos + lane * stride, before = lane * vals;
            bool same = before < left && at + stride <= len;
            const uint64_t mask = (1ull << (8 * hb)) - 1;
            if (stride > kPqWindow / 16) {
                for (int i = 0; i < hb && same; i++) same = s[at + i] == ((w >> (8 * i)) & 0xFF);
            } else {
                same = same && at + hb <= S.hi && (S.peek8((uint32_t)at) & mask) == (w & mask);
            }
            const uint32_t agree = __ballot_sync(0xFFFFFFFFu, same);
            const uint32_t m = agree == 0xFFFFFFFFu ? 32u : (uint32_t)__ffs(~agree) - 1u;  // at least this lane 0's own
            if (lane < m) {
                const uint64_t rest = left - before;
                runs[k + lane] = Run{got + (uint32_t)before, (uint32_t)(vals < rest ? vals : rest), (uint32_t)at + hb, 1};
            }
            k += m;
            pos += (uint32_t)(m * stride);
            got += (uint32_t)(m * vals < left ? m * vals : left);
        } else {
            Run r{got, (uint32_t)((h >> 1) < left ? (h >> 1) : left), 0, 0};
            pos += hb;
            if ((uint64_t)pos + vbytes > len || r.count == 0) return -1;
            if (hb + vbytes <= 8) r.value = (uint32_t)((w >> (8 * hb)) & (vbytes == 4 ? 0xFFFFFFFFull : (1ull << (8 * vbytes)) - 1));
            else for (uint32_t b = 0; b < vbytes; b++) r.value |= S.at(pos + b) << (8 * b);
            pos += vbytes;
            if (lane == 0) runs[k] = r;
            k++;
            got += r.count;
        }
    }
    return k;
}

// The run table of one page's stream.
__device__ void page_runs(const uint8_t* s, uint32_t len, uint32_t n, int bw, Run* out, uint32_t& nruns, uint4* win, uint32_t* err) {
    uint32_t found = 0;
    if (s && bw >= 0 && n > 0) {
        if (bw == 0) {  // every value is 0: one run, no bytes
            if (threadIdx.x == 0) out[0] = Run{0, n, 0, 0};
            found = 1;
        } else {
            const int64_t k = rle_walk(s, len, n, bw, out, win);
            if (k < 0 && threadIdx.x == 0) atomicOr(err, PQ_ERR_RUNS);
            found = k < 0 ? 0u : (uint32_t)k;
        }
    }
    if (threadIdx.x == 0) nruns = found;
}

// Layout and definition-level runs, one warp per page.  A walk is a chain: each header says where
// the next one lies.  One thread per page and a dependent L2 load per link took 19 us per launch (seven
// pages of 18,000 values, about 40 runs each); with the window and up to 32 headers per step 4.4 us here
// and 7.5 us for index runs (23 us where short RLE runs break the sizes, of 38).
__global__ void __launch_bounds__(32) k_pq_levels(PageDev* pages, int max_def, int level_width, Run* runs, uint32_t* err) {
    __shared__ uint4 win[kPqWindow / 16 + 1];
    PageDev& p = pages[blockIdx.x];
    if (threadIdx.x == 0) page_layout(p, max_def, err);
    __syncwarp();
    page_runs(p.levels, p.levels_len, p.nrows, level_width, runs + p.lv_run0, p.lv_nruns, win, err);
}

__device__ uint32_t warp_sum(uint32_t x) { return __reduce_add_sync(0xFFFFFFFFu, x); }

// Present values before each page's first row, each page's present values, and the runs of its
// dictionary indices or RLE booleans (one per present value): one warp per page.
__global__ void __launch_bounds__(32) k_pq_indices(PageDev* pages, const uint32_t* valid, const uint64_t* tile_offs, int64_t nrows,
                                                   uint32_t* nvalues, Run* runs, uint32_t* err) {
    __shared__ uint4 win[kPqWindow / 16 + 1];
    PageDev& p = pages[blockIdx.x];
    auto rank = [&](int64_t row) -> uint64_t {  // present values in rows [0, row)
        if (row >= nrows) return tile_offs[(nrows + kPqTile - 1) / kPqTile];
        const int64_t t = row / kPqTile, w0 = t * (kPqTile / 32);
        const int words = (int)(row / 32 - w0);  // whole words before the row's, at most 255
        uint32_t c = 0;
#pragma unroll
        for (int j = 0; j < kPqTile / 32 / 32; j++) {
            const int w = j * 32 + (int)threadIdx.x;
            if (w < words) c += __popc(valid[w0 + w]);
        }
        if (threadIdx.x == 0 && (row & 31)) c += __popc(valid[row / 32] & ((1u << (row & 31)) - 1u));
        return tile_offs[t] + warp_sum(c);
    };
    const uint64_t v0 = rank(p.row0), v1 = rank(p.row0 + p.nrows);
    if (threadIdx.x == 0) {
        p.valid0 = v0;
        nvalues[blockIdx.x] = (uint32_t)(v1 - v0);
    }
    page_runs(p.values, p.values_len, (uint32_t)(v1 - v0), p.idx_width, runs + p.ix_run0, p.ix_nruns, win, err);
}

// The run that holds value k (k < the stream's value count).
__device__ uint32_t run_of(const Run* runs, uint32_t nruns, uint32_t k) {
    uint32_t lo = 0, hi = nruns;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (runs[mid].first <= k) lo = mid;
        else hi = mid;
    }
    return lo;
}
__device__ uint32_t run_value(const Run& r, const uint8_t* s, int bw, uint32_t k) {
    if (!r.packed) return r.value;
    const uint64_t bit = (uint64_t)(k - r.first) * bw;
    return (uint32_t)((load8(s + r.value + (bit >> 3)) >> (bit & 7)) & (bw == 32 ? 0xFFFFFFFFull : ((1ull << bw) - 1)));
}

__device__ int page_of(const PageDev* pages, int npages, int64_t row) {
    int lo = 0, hi = npages;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (pages[mid].row0 <= row) lo = mid;
        else hi = mid;
    }
    return lo;
}

// ---- 3. validity: definition level == max_def, one thread per 32-row word ----------------------
// A word's rows are taken run by run (an RLE run, or 32 one-bit levels, at once), not level by
// level: 13.7 -> 4.7 us for a 125,000-row chunk.
__global__ void k_pq_valid(const PageDev* pages, int npages, const Run* runs, int max_def, int level_width, int64_t nrows,
                           uint32_t* valid, uint32_t* tile_counts) {
    const int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t bits = 0;
    const int rows = w * 32 < nrows ? (int)(nrows - w * 32 < 32 ? nrows - w * 32 : 32) : 0;
    if (rows && max_def == 0) bits = rows == 32 ? ~0u : (1u << rows) - 1u;
    if (rows && max_def > 0) {
        int p = page_of(pages, npages, w * 32);
        for (int j = 0; j < rows;) {
            const int64_t r = w * 32 + j;
            while (p + 1 < npages && pages[p + 1].row0 <= r) p++;
            const PageDev& pg = pages[p];
            uint32_t k = (uint32_t)(r - pg.row0);
            int left = pg.nrows > k ? (int)(pg.nrows - k < (uint32_t)(rows - j) ? pg.nrows - k : (uint32_t)(rows - j)) : 0;
            if (!left || !pg.lv_nruns) {  // no levels (malformed): absent
                j += left ? left : 1;
                continue;
            }
            const Run* rs = runs + pg.lv_run0;
            for (uint32_t i = run_of(rs, pg.lv_nruns, k); left > 0 && i < pg.lv_nruns; i++) {
                const Run run = rs[i];
                const uint32_t in_run = run.first + run.count - k;
                const int m = in_run < (uint32_t)left ? (int)in_run : left;
                uint32_t x = 0;
                if (!run.packed) {
                    x = run.value == (uint32_t)max_def ? ~0u : 0u;
                } else if (level_width == 1) {  // max_def is 1; 32 levels and an offset of 7 fit eight bytes
                    const uint32_t bit = k - run.first;
                    x = (uint32_t)(load8(pg.levels + run.value + (bit >> 3)) >> (bit & 7));
                } else {
                    for (int q = 0; q < m; q++) x |= (uint32_t)(run_value(run, pg.levels, level_width, k + q) == (uint32_t)max_def) << q;
                }
                bits |= (m == 32 ? x : x & ((1u << m) - 1u)) << j;
                j += m;
                k += m;
                left -= m;
            }
            j += left;
        }
    }
    if (rows) valid[w] = bits;
    // present values per 8,192-row tile
    const uint32_t c = warp_sum(__popc(bits));
    __shared__ uint32_t sum;
    if (threadIdx.x == 0) sum = 0;
    __syncthreads();
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(&sum, c);
    __syncthreads();
    if (threadIdx.x == 0) tile_counts[blockIdx.x] = sum;
}

// Exclusive scan of the tiles' present values by one block, with the total in offs[n] and in *present (the
// status words that the host reads in any case): a chunk has few tiles (16 in 125,000 rows: 3.1 us; 262,144 at
// most: 256 steps).
__global__ void __launch_bounds__(1024) k_pq_tile_scan(const uint32_t* counts, int64_t n, uint64_t* offs, uint64_t* present) {
    __shared__ uint64_t warps[32];
    __shared__ uint64_t carry;
    const int t = threadIdx.x;
    if (t == 0) carry = 0;
    for (int64_t i0 = 0; i0 < n; i0 += 1024) {
        __syncthreads();
        const uint64_t c = i0 + t < n ? counts[i0 + t] : 0u, base = carry;
        uint64_t x = c;
        for (int d = 1; d < 32; d <<= 1) {
            const uint64_t y = __shfl_up_sync(~0u, x, d);
            if ((t & 31) >= d) x += y;
        }
        if ((t & 31) == 31) warps[t >> 5] = x;
        __syncthreads();
        if (t < 32) {
            uint64_t y = warps[t];
            for (int d = 1; d < 32; d <<= 1) {
                const uint64_t z = __shfl_up_sync(~0u, y, d);
                if (t >= d) y += z;
            }
            warps[t] = y;
            if (t == 31) carry = base + y;
        }
        __syncthreads();
        if (i0 + t < n) offs[i0 + t] = base + (t >= 32 ? warps[(t >> 5) - 1] : 0) + x - c;
    }
    __syncthreads();
    if (t == 0) {
        offs[n] = carry;
        *present = carry;
    }
}
}  // namespace

namespace {
// ---- 4. values --------------------------------------------------------------------------------
// Conversion (parquet_reader.rs:31-56), the header's ML_PQ_CONV_* values.
enum Conv { CV_BOOL = 0, CV_INT32, CV_DATE, CV_INT64, CV_FLOAT, CV_DOUBLE, CV_UTF8, CV_DEC_I32, CV_DEC_I64, CV_DEC_BYTES };

struct DecodeArgs {
    const PageDev* pages;
    int npages;
    const Run* runs;
    const uint32_t* valid;
    const uint64_t* tile_offs;
    int64_t nrows;
    int ptype, conv, type_length;
    double div;  // 10^scale for decimals
    // the dictionary page: fixed-width values, or byte-array entries (pointer + length)
    const uint8_t* dict;
    uint32_t dict_n;
    const uint8_t* const* dict_ptr;
    const uint32_t* dict_len;
    // PLAIN byte arrays of the data pages, by the value's index among the chunk's present values
    const uint8_t* const* vptr;
    const uint32_t* vlen;
    void* out;                // fixed-width output (the column's type)
    const uint8_t** str_ptr;  // strings (and byte-array decimals go through vptr)
    uint32_t* str_len;
    // strings whose pages all index a dictionary of fewer than kPqSmallDict entries: each row's entry
    // instead (dict_n for a NULL), ~(first row) of each entry (0: unused) and the strings' bytes
    uint32_t* ent;
    uint32_t* first;
    uint64_t* total;
    uint32_t* err;
};
constexpr uint32_t kPqSmallDict = 1024;
constexpr uint32_t kPqSmallDictBytes = 65536;
// rows per block: a 125,000-row chunk in 16 blocks of a whole tile left most SMs idle and put 32 rows in
// series on a thread (57 us); 245 blocks of two rows per thread take 9.8 us
constexpr int kPqSlice = 512;

// A big-endian two's complement integer of up to 16 bytes (be_i128, parquet_reader.rs:154-166)
// as the nearest f64 (ties to even).
__device__ double be_int_to_f64(const uint8_t* b, uint32_t n) {
    uint64_t hi = (n && (b[0] & 0x80)) ? ~0ull : 0ull, lo = hi;
    for (uint32_t i = 0; i < n && i < 16; i++) {
        hi = (hi << 8) | (lo >> 56);
        lo = (lo << 8) | b[i];
    }
    const bool neg = (int64_t)hi < 0;
    if (neg) {  // magnitude (two's complement negation)
        lo = ~lo + 1;
        hi = ~hi + (lo == 0 ? 1 : 0);
    }
    double m;
    if (hi == 0) {
        m = __ull2double_rn(lo);
    } else {
        const int lz = __clzll(hi);
        const uint64_t h = lz ? (hi << lz) | (lo >> (64 - lz)) : hi;  // top bit at 63
        const uint64_t l = lo << lz;
        uint64_t mant = h >> 11;  // 53 bits
        const bool guard = (h >> 10) & 1, sticky = (h & 0x3FF) || l;
        if (guard && (sticky || (mant & 1))) mant++;
        int e = 127 - lz - 52;
        if (mant >> 53) {
            mant >>= 1;
            e++;
        }
        m = ldexp((double)mant, e);
    }
    return neg ? -m : m;
}

__global__ void __launch_bounds__(256) k_pq_values(const __grid_constant__ DecodeArgs D) {
    __shared__ uint32_t words[256], pre[256];
    __shared__ uint32_t sfirst[kPqSmallDict];
    __shared__ uint32_t stotal;
    const int t = threadIdx.x;
    const int64_t tile = blockIdx.x / (kPqTile / kPqSlice);
    const int64_t w0 = tile * (kPqTile / 32);
    const int64_t row0 = (int64_t)blockIdx.x * kPqSlice;
    if (D.ent) {
        for (uint32_t i = t; i <= D.dict_n; i += 256) sfirst[i] = 0;
        if (t == 0) stotal = 0;
    }
    const uint32_t word = (w0 + t) * 32 < D.nrows ? D.valid[w0 + t] : 0u;
    words[t] = word;
    // exclusive scan of the words' popcounts
    uint32_t c = __popc(word), x = c;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if ((t & 31) >= o) x += y;
    }
    __shared__ uint32_t warp_total[8];
    if ((t & 31) == 31) warp_total[t >> 5] = x;
    __syncthreads();
    uint32_t wbase = 0;
    for (int i = 0; i < (t >> 5); i++) wbase += warp_total[i];
    pre[t] = wbase + x - c;
    __syncthreads();
    const uint64_t base = D.tile_offs[tile];
    uint32_t bytes = 0;  // of this thread's strings (each within a small dictionary page)
    // the first rows of the block's entries: most rows only read the word
    auto entry = [&](uint32_t e, int64_t r) {
        D.ent[r] = e;
        if (*(volatile uint32_t*)(sfirst + e) < ~(uint32_t)r) atomicMax(sfirst + e, ~(uint32_t)r);
    };
    int p = -1;
    for (int j = 0; j < kPqSlice / 256; j++) {
        const int64_t r = row0 + j * 256 + t;
        if (r >= D.nrows) break;
        const int lw = (int)((r >> 5) - w0);
        const uint32_t bits = words[lw];
        const bool v = (bits >> (r & 31)) & 1;
        const int vw = D.conv == CV_BOOL ? 1 : (D.conv == CV_INT32 || D.conv == CV_DATE) ? 4 : 8;
        if (!v) {
            if (D.ent) {
                entry(D.dict_n, r);
            } else if (D.conv == CV_UTF8) {
                D.str_ptr[r] = nullptr;
                D.str_len[r] = 0;
            } else if (vw == 1) {
                ((uint8_t*)D.out)[r] = 0;
            } else if (vw == 4) {
                ((uint32_t*)D.out)[r] = 0;
            } else {
                ((uint64_t*)D.out)[r] = 0;
            }
            continue;
        }
        const uint64_t d = base + pre[lw] + __popc(bits & ((1u << (r & 31)) - 1u));  // among present values
        if (p < 0 || !(D.pages[p].row0 <= r && (p + 1 >= D.npages || D.pages[p + 1].row0 > r))) p = page_of(D.pages, D.npages, r);
        const PageDev& pg = D.pages[p];
        const uint32_t k = (uint32_t)(d - pg.valid0);
        const bool dict = pg.encoding == ENC_RLE_DICTIONARY || pg.encoding == ENC_PLAIN_DICTIONARY;
        const bool rle_bool = pg.encoding == ENC_RLE;
        uint32_t idx = 0;
        if (dict || rle_bool) {
            if (!pg.ix_nruns) {
                atomicOr(D.err, PQ_ERR_VALUES);
                if (D.ent) entry(D.dict_n, r);  // the codes are looked up before the error is read
                continue;
            }
            const Run* rs = D.runs + pg.ix_run0;
            idx = run_value(rs[run_of(rs, pg.ix_nruns, k)], pg.values, pg.idx_width, k);
            if (dict && idx >= D.dict_n) {
                atomicOr(D.err, PQ_ERR_VALUES);
                if (D.ent) entry(D.dict_n, r);
                continue;
            }
        }
        if (D.ent) {
            entry(idx, r);
            bytes += D.dict_len[idx];
            continue;
        }
        // the value's bytes: a byte array (pointer, length) or a fixed-width slot
        const uint8_t* src = nullptr;
        uint32_t slen = 0;
        const int pw = D.ptype == PQ_INT32 || D.ptype == PQ_FLOAT ? 4 : D.ptype == PQ_FLBA ? D.type_length : 8;
        if (D.ptype == PQ_BYTE_ARRAY) {
            if (dict) {
                src = D.dict_ptr[idx];
                slen = D.dict_len[idx];
            } else {
                src = D.vptr[d];
                slen = D.vlen[d];
            }
        } else if (D.ptype != PQ_BOOLEAN) {
            if (dict) {
                src = D.dict + (uint64_t)idx * pw;
            } else {
                if ((uint64_t)(k + 1) * pw > pg.values_len) {
                    atomicOr(D.err, PQ_ERR_VALUES);
                    continue;
                }
                src = pg.values + (uint64_t)k * pw;
            }
            slen = pw;
        }
        switch (D.conv) {
            case CV_BOOL: {
                uint32_t b;
                if (rle_bool) {
                    b = idx;
                } else if (dict) {
                    b = D.dict[idx >> 3] >> (idx & 7);
                } else {
                    if ((k >> 3) >= pg.values_len) {
                        atomicOr(D.err, PQ_ERR_VALUES);
                        continue;
                    }
                    b = pg.values[k >> 3] >> (k & 7);
                }
                ((uint8_t*)D.out)[r] = (uint8_t)(b & 1);
                break;
            }
            case CV_INT32:
            case CV_DATE: ((uint32_t*)D.out)[r] = (uint32_t)load8(src); break;
            case CV_INT64:
            case CV_DOUBLE: ((uint64_t*)D.out)[r] = load8(src); break;
            case CV_FLOAT: ((double*)D.out)[r] = (double)__uint_as_float((uint32_t)load8(src)); break;
            case CV_DEC_I32: ((double*)D.out)[r] = __ddiv_rn((double)(int32_t)(uint32_t)load8(src), D.div); break;
            case CV_DEC_I64: ((double*)D.out)[r] = __ddiv_rn(__ll2double_rn((long long)load8(src)), D.div); break;
            case CV_DEC_BYTES: ((double*)D.out)[r] = __ddiv_rn(be_int_to_f64(src, slen), D.div); break;
            case CV_UTF8:
                D.str_ptr[r] = src;
                D.str_len[r] = slen;
                break;
        }
    }
    if (!D.ent) return;
    bytes = warp_sum(bytes);
    if ((t & 31) == 0 && bytes) atomicAdd(&stotal, bytes);  // 512 rows of at most 64 KB
    __syncthreads();
    for (uint32_t i = t; i <= D.dict_n; i += 256)
        if (sfirst[i]) atomicMax(D.first + i, sfirst[i]);
    if (t == 0 && stotal) atomicAdd((unsigned long long*)D.total, (unsigned long long)stotal);
}

// PLAIN byte arrays (a 4-byte length, then the bytes) of the data pages, one warp per page walking
// the lengths in a staged window: pointer and length of each value by its index among the chunk's
// present values.  For the dictionary page (dict != nullptr; the last block) the entries instead.
__global__ void __launch_bounds__(32) k_pq_byte_arrays(const PageDev* pages, int npages, const uint32_t* nvalues, const uint8_t** ptr,
                                                       uint32_t* len, const uint8_t* dict, uint32_t dict_len, uint32_t dict_n,
                                                       const uint8_t** dptr, uint32_t* dlen, uint32_t* err) {
    __shared__ uint4 win[kPqWindow / 16 + 1];
    const int i = blockIdx.x, lane = threadIdx.x;
    const uint8_t* s;
    uint32_t n, slen;
    const uint8_t** op;
    uint32_t* ol;
    if (i < npages) {
        const PageDev& p = pages[i];
        if (p.encoding != ENC_PLAIN) return;
        s = p.values;
        slen = p.values_len;
        n = nvalues[i];
        op = ptr + p.valid0;
        ol = len + p.valid0;
    } else if (dict) {
        s = dict;
        slen = dict_len;
        n = dict_n;
        op = dptr;
        ol = dlen;
    } else {
        return;
    }
    StreamWindow S(s, slen, win);
    uint32_t pos = 0;
    for (uint32_t k = 0; k < n; k++) {
        S.need(pos, 4);
        if ((uint64_t)pos + 4 > slen || S.at32(pos) > slen - pos - 4) {
            if (lane == 0) atomicOr(err, PQ_ERR_VALUES);
            for (k += lane; k < n; k += 32) op[k] = s, ol[k] = 0;
            return;
        }
        const uint32_t l = S.at32(pos);
        if (lane == 0) {
            op[k] = s + pos + 4;
            ol[k] = l;
        }
        pos += 4 + l;
    }
}

// ---- 5. strings: materialize, then encode_strings' dictionary decision ----------------------
__global__ void k_pq_str_copy(const uint8_t* const* ptr, const uint32_t* len, const uint64_t* offs, int64_t n,
                              uint32_t* off32, uint8_t* bytes) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += stride) {
        const uint64_t o = offs[r];
        off32[r] = (uint32_t)o;
        const uint8_t* s = ptr[r];
        for (uint32_t b = 0; b < len[r]; b++) bytes[o + b] = s[b];
        if (r == n - 1) off32[n] = (uint32_t)offs[n];
    }
}
// The words only fall: a row that reads a smaller one has nothing to do.
__global__ void k_pq_first(const uint32_t* canon, int64_t n, uint32_t* first) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += stride) {
        uint32_t* f = first + canon[r];
        if (__ldcg(f) > (uint32_t)r) atomicMin(f, (uint32_t)r);
    }
}
// bits: rows that are the first occurrence of their string; block counts for the compaction
__global__ void k_pq_first_flags(const uint32_t* canon, const uint32_t* first, int64_t n, uint32_t* bits, uint32_t* counts,
                                 int rows_per_block) {
    const int64_t b0 = (int64_t)blockIdx.x * rows_per_block;
    uint32_t c = 0;
    for (int64_t w = b0 / 32 + threadIdx.x; w * 32 < (n < b0 + rows_per_block ? n : b0 + rows_per_block); w += blockDim.x) {
        uint32_t x = 0;
        for (int j = 0; j < 32; j++) {
            const int64_t r = w * 32 + j;
            if (r < n && first[canon[r]] == (uint32_t)r) x |= 1u << j;
        }
        bits[w] = x;
        c += __popc(x);
    }
    __shared__ uint32_t sum;
    if (threadIdx.x == 0) sum = 0;
    __syncthreads();
    if (c) atomicAdd(&sum, c);
    __syncthreads();
    if (threadIdx.x == 0) counts[blockIdx.x] = sum;
}
__global__ void k_pq_codes(const uint32_t* list, uint32_t ndistinct, const uint32_t* canon, uint32_t* code_of) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ndistinct; i += stride)
        code_of[canon[list[i]]] = (uint32_t)i;
}
// A small dictionary page's entries (and one more, the empty string of the NULL rows) in one block:
// equal strings become one, ordered by first row; code_of[entry], and at `out` the number of
// strings, their bytes, offsets [kPqSmallDict + 1] and the bytes themselves.  For a chunk of 125,000 rows
// the rows' own path (copy the strings, hash every row, find first rows, compact) took 140 us of
// kernels, two thirds of it on the few words that equal strings share; this kernel takes 4.5 us and the codes 3.3
__global__ void __launch_bounds__(kPqSmallDict) k_pq_small_dict(const uint8_t* const* dptr, const uint32_t* dlen, uint32_t dict_n,
                                                                const uint32_t* first, uint32_t* code_of, uint32_t* out) {
    __shared__ uint32_t slots[2 * kPqSmallDict];  // entry + 1
    __shared__ uint32_t sfirst[kPqSmallDict];     // ~(first row) of each kept string, 0 for the rest
    __shared__ uint32_t order[kPqSmallDict], warps[32];
    const uint32_t t = threadIdx.x;
    slots[t] = slots[t + kPqSmallDict] = 0;
    sfirst[t] = 0;
    const uint32_t f = t <= dict_n ? first[t] : 0u;
    const uint8_t* s = t < dict_n ? dptr[t] : nullptr;
    const uint32_t n = t < dict_n ? dlen[t] : 0u;
    __syncthreads();
    uint32_t canon = t;
    if (f) {
        uint32_t q = (uint32_t)hash_bytes(s, n) & (2 * kPqSmallDict - 1);
        for (uint32_t k = 0; k < 2 * kPqSmallDict; k++, q = (q + 1) & (2 * kPqSmallDict - 1)) {
            const uint32_t c = atomicCAS(slots + q, 0u, t + 1);
            if (c == 0) break;
            const uint32_t o = c - 1, on = o < dict_n ? dlen[o] : 0u;
            if (on == n && bytes_eq(o < dict_n ? dptr[o] : nullptr, s, n)) {
                canon = o;
                break;
            }
        }
        atomicMax(sfirst + canon, f);
    }
    __syncthreads();
    const bool kept = f && canon == t;
    const uint32_t mine = sfirst[t];
    uint32_t rank = 0;
    if (kept)
        for (uint32_t e = 0; e <= dict_n; e++) rank += sfirst[e] > mine;
    const uint32_t distinct = __syncthreads_count(kept);
    if (kept) {
        order[rank] = t;
        code_of[t] = rank;
    }
    __syncthreads();  // code_of of the kept entries is visible to the block
    if (f && !kept) code_of[t] = code_of[canon];
    // offsets of the strings in their order (at most 64 KB in all)
    const uint32_t e = t < distinct ? order[t] : dict_n;
    const uint32_t l = e < dict_n ? dlen[e] : 0u;
    uint32_t x = l;
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(~0u, x, d);
        if ((t & 31) >= (uint32_t)d) x += y;
    }
    if ((t & 31) == 31) warps[t >> 5] = x;
    __syncthreads();
    uint32_t base = 0;
    for (uint32_t i = 0; i < (t >> 5); i++) base += warps[i];
    const uint32_t o = base + x - l;
    uint32_t* off = out + 2;
    uint8_t* bytes = (uint8_t*)(off + kPqSmallDict + 1);
    if (t == kPqSmallDict - 1) {
        out[0] = distinct;
        out[1] = off[kPqSmallDict] = base + x;
    }
    off[t] = o;
    const uint8_t* src = e < dict_n ? dptr[e] : nullptr;
    for (uint32_t i = 0; i < l; i++) bytes[o + i] = src[i];
}
// Each row's string from its dictionary entry.
__global__ void k_pq_entry_strings(const uint32_t* ent, int64_t n, const uint8_t* const* dptr, const uint32_t* dlen, uint32_t dict_n,
                                   const uint8_t** ptr, uint32_t* len) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += stride) {
        const uint32_t e = ent[r];
        ptr[r] = e < dict_n ? dptr[e] : nullptr;
        len[r] = e < dict_n ? dlen[e] : 0u;
    }
}
__global__ void k_pq_codes2(const uint32_t* canon, int64_t n, const uint32_t* code_of, uint32_t* codes) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += stride) codes[r] = code_of[canon[r]];
}
}  // namespace

namespace {
uint64_t pow2_ceil(uint64_t x) {
    uint64_t p = 1;
    while (p < x) p <<= 1;
    return p;
}
int grid_of(int64_t n, int threads = 256) { return (int)std::max<int64_t>(1, std::min<int64_t>((n + threads - 1) / threads, 148 * 16)); }

// powi as in compiler-rt's __powidf2 (binary exponentiation), which Rust's f64::powi lowers
// to for a run-time exponent: 10f64.powi(scale) (parquet_reader.rs:217).
double powi(double a, int b) {
    const bool recip = b < 0;
    double r = 1;
    for (;;) {
        if (b & 1) r *= a;
        b /= 2;
        if (b == 0) break;
        a *= a;
    }
    return recip ? 1 / r : r;
}

void check_pq(Ctx* ctx, uint32_t e) {
    (void)ctx;
    if (e & PQ_ERR_SNAPPY) raise(ML_ERR_INVALID, "parquet: a Snappy page does not decompress to its stated size");
    if (e & PQ_ERR_LAYOUT) raise(ML_ERR_INVALID, "parquet: a data page's levels or values run past the page");
    if (e & PQ_ERR_RUNS) raise(ML_ERR_INVALID, "parquet: a malformed RLE / bit-packed stream");
    if (e & PQ_ERR_VALUES) raise(ML_ERR_INVALID, "parquet: a value or dictionary index outside its page or dictionary");
    if (e) raise(ML_ERR_INVALID, "parquet: decode error " + std::to_string(e));
}
}  // namespace

extern "C" int ml_gpu_parquet_decode(ml_ctx* ctx, const uint8_t* chunk, int64_t chunk_bytes, int32_t physical_type,
                                     int32_t type_length, int32_t conversion, int32_t scale, int32_t codec,
                                     int64_t num_rows, int32_t max_def, ml_batch** out) {
    API_BEGIN
    HostTimer host_timer_(ctx, "host:parquet_decode");
    REQUIRE(ctx && out && (chunk || chunk_bytes == 0) && chunk_bytes >= 0, "null argument");
    REQUIRE(num_rows >= 0 && num_rows < 0x7FFFFFFFll, "row count out of range");
    REQUIRE(max_def >= 0 && max_def <= 255, "max definition level out of range");
    if (codec != ML_PQ_CODEC_UNCOMPRESSED && codec != ML_PQ_CODEC_SNAPPY)
        raise(ML_ERR_UNSUPPORTED, "parquet: compression codec " + std::to_string(codec));
    // Conversion::for_column (parquet_reader.rs:58-80)
    const int pt = physical_type, cv = conversion;
    const bool ok = (cv == CV_BOOL && pt == PQ_BOOLEAN) || ((cv == CV_INT32 || cv == CV_DATE || cv == CV_DEC_I32) && pt == PQ_INT32) ||
                    ((cv == CV_INT64 || cv == CV_DEC_I64) && pt == PQ_INT64) || (cv == CV_FLOAT && pt == PQ_FLOAT) ||
                    (cv == CV_DOUBLE && pt == PQ_DOUBLE) || (cv == CV_UTF8 && pt == PQ_BYTE_ARRAY) ||
                    (cv == CV_DEC_BYTES && (pt == PQ_BYTE_ARRAY || (pt == PQ_FLBA && type_length > 0)));
    if (!ok) raise(ML_ERR_UNSUPPORTED, "parquet: physical type " + std::to_string(pt) + " with conversion " + std::to_string(cv));
    const int out_type = cv == CV_BOOL ? ML_TYPE_BOOL : cv == CV_INT32 ? ML_TYPE_INT32 : cv == CV_DATE ? ML_TYPE_DATE
                         : cv == CV_INT64 ? ML_TYPE_INT64 : cv == CV_UTF8 ? ML_TYPE_UTF8 : ML_TYPE_FLOAT64;
    const int level_width = max_def ? 32 - __builtin_clz((unsigned)max_def) : 0;
    const int pw = pt == PQ_INT32 || pt == PQ_FLOAT ? 4 : pt == PQ_FLBA ? type_length : 8;
    ctx->set_current();
    OpStream op_stream(ctx);
    const cudaStream_t s = op_stream.s;
    auto b = std::make_unique<ml_batch>();
    b->ctx = ctx;
    b->nrows = num_rows;
    b->res = std::make_unique<Reservation>(ctx, "ParquetDecode");
    auto col = std::make_unique<DevColumn>();
    col->dtype = out_type;
    col->kind = CK_FIXED;
    col->n = num_rows;

    // pages and their places in the uncompressed buffer
    std::vector<Page> pages = parse_pages(chunk, chunk_bytes);
    int dict_page = -1;
    std::vector<int> data;
    int64_t rows = 0, ubytes = 0;
    std::vector<int64_t> uoff;
    for (size_t i = 0; i < pages.size(); i++) {
        const Page& pg = pages[i];
        uoff.push_back(ubytes);
        ubytes += (pg.uncompressed + 15) & ~15;
        if (pg.type == PAGE_DICTIONARY) {
            if (dict_page >= 0 || !data.empty()) raise(ML_ERR_INVALID, "parquet: a dictionary page after the first page");
            if (pg.encoding != ENC_PLAIN && pg.encoding != ENC_PLAIN_DICTIONARY)
                raise(ML_ERR_UNSUPPORTED, "parquet: dictionary page encoding " + std::to_string(pg.encoding));
            dict_page = (int)i;
            continue;
        }
        if (pg.encoding != ENC_PLAIN && pg.encoding != ENC_PLAIN_DICTIONARY && pg.encoding != ENC_RLE_DICTIONARY &&
            !(pg.encoding == ENC_RLE && pt == PQ_BOOLEAN))
            raise(ML_ERR_UNSUPPORTED, "parquet: data page encoding " + std::to_string(pg.encoding));
        if ((pg.encoding == ENC_PLAIN_DICTIONARY || pg.encoding == ENC_RLE_DICTIONARY) && dict_page < 0)
            raise(ML_ERR_INVALID, "parquet: dictionary-encoded page without a dictionary page");
        if (pg.type == PAGE_DATA && max_def > 0 && pg.def_encoding != ENC_RLE)
            raise(ML_ERR_UNSUPPORTED, "parquet: definition level encoding " + std::to_string(pg.def_encoding));
        if (pg.type == PAGE_DATA_V2 && pg.rep_bytes + pg.def_bytes > std::min(pg.compressed, pg.uncompressed))
            raise(ML_ERR_INVALID, "parquet: a v2 page's levels run past the page");
        data.push_back((int)i);
        rows += pg.num_values;
    }
    // read_all (parquet_reader.rs:104-133): the chunk must hold exactly num_rows records
    if (rows != num_rows)
        raise(ML_ERR_INVALID, "parquet: expected " + std::to_string(num_rows) + " rows, decoded " + std::to_string(rows));
    const int np = (int)data.size();
    if (num_rows == 0) {
        col->data = DevBuf(ctx, 8, b->res.get());
        if (out_type == ML_TYPE_UTF8) {
            col->kind = CK_UTF8;
            col->offsets = DevBuf(ctx, 4, b->res.get());
            CK(cudaMemsetAsync(col->offsets.get(), 0, 4, s));
        }
        CK(cudaStreamSynchronize(s));
        b->cols.push_back(std::move(col));
        *out = b.release();
        return ML_OK;
    }

    // 1. the chunk to the device, then every page uncompressed
    // 64 bytes of padding: the aligned 8- and 16-byte loads read past the last byte
    DevBuf dchunk(ctx, (size_t)chunk_bytes + 64, nullptr), upages(ctx, (size_t)ubytes + 64, nullptr);
    // from the caller's (pageable) buffer: a pinned staging buffer per call costs more than it saves
    CK(cudaMemcpyAsync(dchunk.get(), chunk, (size_t)chunk_bytes, cudaMemcpyHostToDevice, s));
    const uint8_t* dc = dchunk.get<uint8_t>();
    uint8_t* up = upages.get<uint8_t>();
    // the Snappy pages in groups (usually one) of at most kSnapGroupBytes stream bytes, or one page
    struct SnapGroup {
        int job0 = 0, njobs = 0, frag0 = 0, nfrags = 0, blk0 = 0, nblks = 0;
        uint64_t bytes = 0, elems = 0;
    };
    std::vector<SnapJob> jobs;
    std::vector<SnapGroup> groups;
    std::vector<uint2> frags, blocks;  // {page, fragment} per 64 KB of output, {page, block} per kSnapBlk of stream
    std::vector<SnapFlat> flats;             // pages of few elements, and those
    std::vector<uint4> elems;
    uint32_t plan_words = 0;
    for (size_t i = 0; i < pages.size(); i++) {
        const Page& pg = pages[i];
        const bool v2 = pg.type == PAGE_DATA_V2;
        const int64_t lv = v2 ? pg.rep_bytes + pg.def_bytes : 0;  // v2 levels are never compressed
        if (lv) CK(cudaMemcpyAsync(up + uoff[i], dc + pg.payload, (size_t)lv, cudaMemcpyDeviceToDevice, s));
        const bool compressed = codec == ML_PQ_CODEC_SNAPPY && (!v2 || pg.v2_compressed);
        if (compressed) {
            const uint32_t dlen = (uint32_t)(pg.uncompressed - lv);
            const uint32_t slen = (uint32_t)(pg.compressed - lv);
            const uint32_t el0 = (uint32_t)elems.size();
            if (flat_elements(chunk + pg.payload + lv, slen, dlen, elems)) {
                const bool copies = std::any_of(elems.begin() + el0, elems.end(), [](const uint4& e) { return e.w != 0; });
                flats.push_back(SnapFlat{dc + pg.payload + lv, up + uoff[i] + lv, dlen, dlen <= kSnapTiny && copies ? 1u : 0u, el0,
                                         (uint32_t)elems.size() - el0});
                continue;
            }
            const uint32_t nfrag = (uint32_t)(((uint64_t)dlen + kSnapFrag - 1) / kSnapFrag);
            const uint32_t nblk = (uint32_t)(((uint64_t)slen + kSnapBlk - 1) / kSnapBlk);
            if (groups.empty() || groups.back().bytes + slen > kSnapGroupBytes) {
                SnapGroup g;
                g.job0 = (int)jobs.size(), g.frag0 = (int)frags.size(), g.blk0 = (int)blocks.size();
                groups.push_back(g);
            }
            SnapGroup& g = groups.back();
            const uint32_t id = (uint32_t)jobs.size();
            for (uint32_t k = 0; k < nfrag; k++) frags.push_back(uint2{id, k});
            for (uint32_t k = 0; k < nblk; k++) blocks.push_back(uint2{id, k});
            jobs.push_back(SnapJob{dc + pg.payload + lv, up + uoff[i] + lv, slen, dlen, plan_words, nfrag,
                                   (uint32_t)g.nblks, 0u, g.bytes, g.elems});
            plan_words += snap_plan_words(nfrag);
            g.njobs++, g.nfrags += (int)nfrag, g.nblks += (int)nblk;
            g.bytes += slen, g.elems += slen / 2 + 1;  // an element spans at least two stream bytes
        } else {
            if (pg.compressed != pg.uncompressed) raise(ML_ERR_INVALID, "parquet: an uncompressed page changes size");
            if (pg.compressed > lv)
                CK(cudaMemcpyAsync(up + uoff[i] + lv, dc + pg.payload + lv, (size_t)(pg.compressed - lv), cudaMemcpyDeviceToDevice, s));
        }
    }
    std::vector<PageDev> hp(np);
    int64_t row0 = 0;
    for (int j = 0; j < np; j++) {
        const Page& pg = pages[data[j]];
        PageDev& d = hp[j];
        d = PageDev{};
        d.data = up + uoff[data[j]];
        d.len = (uint32_t)pg.uncompressed;
        d.v2 = pg.type == PAGE_DATA_V2;
        d.def_bytes = pg.def_bytes;
        d.rep_bytes = pg.rep_bytes;
        d.encoding = pg.encoding == ENC_PLAIN_DICTIONARY ? ENC_RLE_DICTIONARY : pg.encoding;
        d.row0 = row0;
        d.nrows = (uint32_t)pg.num_values;
        d.lv_run0 = d.ix_run0 = (uint64_t)row0;
        row0 += pg.num_values;
    }
    // One upload: the elements, the flat pages, the Snappy jobs, their fragment and block tables, the data pages, and
    // zeros for the first rows of a small dictionary's entries and for {error bits, -, present values, strings'
    // bytes}; behind those lies the small dictionary's answer, so one copy brings both back.
    const size_t eb = elems.size() * sizeof(uint4), lb = flats.size() * sizeof(SnapFlat), jb = jobs.size() * sizeof(SnapJob);
    const size_t fb = frags.size() * sizeof(uint2), bb = blocks.size() * sizeof(uint2), pb = hp.size() * sizeof(PageDev);
    const size_t zb = (cv == CV_UTF8 ? kPqSmallDict * 4 : 0) + 32;
    // {strings, bytes, offsets, the bytes (no more than the page holds)}
    const size_t answer_head = (2 + kPqSmallDict + 1) * 4;
    const size_t answer_b = cv == CV_UTF8 && dict_page >= 0 && (uint32_t)pages[dict_page].uncompressed <= kPqSmallDictBytes
                                ? answer_head + (size_t)pages[dict_page].uncompressed : 0;
    std::vector<uint8_t> hj(eb + lb + jb + fb + bb + pb + zb);
    {
        uint8_t* at = hj.data();
        auto put = [&](const void* p, size_t n) {
            if (n) std::memcpy(at, p, n);
            at += n;
        };
        put(elems.data(), eb), put(flats.data(), lb), put(jobs.data(), jb), put(frags.data(), fb), put(blocks.data(), bb);
        put(hp.data(), pb);
    }
    DevBuf dj(ctx, hj.size() + answer_b, nullptr);
    CK(cudaMemcpyAsync(dj.get(), hj.data(), hj.size(), cudaMemcpyHostToDevice, s));
    uint8_t* const D0 = dj.get<uint8_t>();
    PageDev* P = (PageDev*)(D0 + eb + lb + jb + fb + bb);
    uint32_t* derr = (uint32_t*)(D0 + hj.size() - 32);
    uint64_t* dpresent = (uint64_t*)derr + 1;
    uint64_t* dtotal = (uint64_t*)derr + 2;
    uint32_t* dfirst = derr - kPqSmallDict;  // strings only
    uint32_t* danswer = derr + 8;
    PinnedSlot slot(ctx);
    DevBuf splan, smap, sentry;  // the Snappy kernels': live to the end of the call
    if (!jobs.empty() || !flats.empty()) {
        if (!flats.empty()) {
            k_pq_snappy_flat<<<(unsigned)flats.size(), kSnapThreads, 0, s>>>((const SnapFlat*)(D0 + eb), (const uint4*)D0);
            ctx->count_launch();
        }
        const SnapJob* J = (const SnapJob*)(D0 + eb + lb);
        const uint2* F = (const uint2*)(D0 + eb + lb + jb);
        const uint2* B = (const uint2*)(D0 + eb + lb + jb + fb);
        if (!jobs.empty()) {
            splan = DevBuf(ctx, (size_t)plan_words * 4, nullptr);
            uint64_t most = 0, most_elems = 0;
            int most_blks = 0;
            for (const SnapGroup& g : groups) {
                const bool parts = g.bytes > kSnapGroupBytes;
                most = std::max(most, parts ? kSnapGroupBytes : g.bytes);
                most_elems = std::max(most_elems, parts ? (uint64_t)kSnapRing : g.elems);
                most_blks = std::max(most_blks, g.nblks);
            }
            // the maps; the element list takes their place once the chains are known
            smap = DevBuf(ctx, std::max<size_t>(std::max(most * sizeof(SnapMap), most_elems * sizeof(uint2)), 16), nullptr);
            sentry = DevBuf(ctx, std::max<size_t>((size_t)most_blks * sizeof(SnapEntry), 16), nullptr);
            // per call: the attribute belongs to the current device's copy of the kernel
            CK(cudaFuncSetAttribute(k_pq_snappy_maps, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSnapMapSmem));
            CK(cudaFuncSetAttribute(k_pq_snappy_frag, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSnapFragSmem));
            uint32_t* const plan = splan.get<uint32_t>();
            SnapMap* const tab = smap.get<SnapMap>();
            SnapEntry* const entries = sentry.get<SnapEntry>();
            uint2* const elist = smap.get<uint2>();
            for (const SnapGroup& g : groups) {
                // a page in parts, or all pages of the group at once
                const bool parts = g.bytes > kSnapGroupBytes;
                const uint32_t mask = parts ? kSnapRing - 1 : ~0u;
                const uint32_t blks = (uint32_t)g.nblks, group = (uint32_t)(kSnapGroupBytes / kSnapBlk), part = kSnapPart / kSnapBlk;
                if (blks) CK(cudaMemsetAsync(entries, 0, (size_t)blks * sizeof(SnapEntry), s));
                if (parts)  // no fragment starts anywhere yet
                    CK(cudaMemsetAsync(plan + jobs[g.job0].plan, 0xFF, (size_t)snap_plan_words(jobs[g.job0].nfrag) * 4, s));
                for (uint32_t b = 0; b == 0 || b < blks; b += parts ? group : std::max(blks, 1u)) {
                    const uint32_t m = parts ? std::min(group, blks - b) : blks, lo = b * kSnapBlk;
                    if (m) k_pq_snappy_maps<<<m, kSnapThreads, kSnapMapSmem, s>>>(J, B + g.blk0 + b, tab, lo);
                    k_pq_snappy_chain<<<g.njobs, 32, 0, s>>>(J + g.job0, tab, entries, plan, lo, parts ? lo + m * kSnapBlk : ~0u);
                    ctx->count_launch(m ? 2 : 1);
                }
                for (uint32_t b = 0; b < blks; b += parts ? part : blks) {
                    const uint32_t m = parts ? std::min(part + kSnapPast, blks - b) : blks, lo = b * kSnapBlk;
                    k_pq_snappy_list<<<m, kSnapThreads, 0, s>>>(J, B + g.blk0 + b, entries, plan, elist, mask);
                    if (g.nfrags)
                        k_pq_snappy_frag<<<g.nfrags, kSnapThreads, kSnapFragSmem, s>>>(J, F + g.frag0, elist, plan, mask, lo,
                                                                                       parts ? lo + kSnapPart : ~0u);
                    ctx->count_launch(g.nfrags ? 2 : 1);
                }
                k_pq_snappy_serial<<<g.njobs, 32, 0, s>>>(J + g.job0, plan, derr);
                ctx->count_launch();
            }
        }
    }
    auto read_err = [&]() {  // waits for the stream; slot: {error bits, -, present values, strings' bytes}
        CK(cudaMemcpyAsync(slot.p, derr, 32, cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        check_pq(ctx, *slot.as<uint32_t>());
    };

    // 2. data pages (the kernels are bounds-checked, so a decode error is read once, at the end;
    //    a page's run table starts at its first row: a stream has at most one run per value): layout, level runs, validity, present values, index runs
    DevBuf lv_runs(ctx, (size_t)num_rows * sizeof(Run), nullptr), ix_runs(ctx, (size_t)num_rows * sizeof(Run), nullptr);
    k_pq_levels<<<np, 32, 0, s>>>(P, max_def, level_width, lv_runs.get<Run>(), derr);
    const int64_t ntiles = (num_rows + kPqTile - 1) / kPqTile;
    DevBuf valid(ctx, (size_t)ntiles * kPqTile / 8, b->res.get());  // u32 words; as u64 words the validity
    DevBuf tcounts(ctx, (size_t)ntiles * 4, nullptr), toffs(ctx, (size_t)(ntiles + 1) * 8, nullptr);
    k_pq_valid<<<(int)ntiles, 256, 0, s>>>(P, np, lv_runs.get<Run>(), max_def, level_width, num_rows, valid.get<uint32_t>(),
                                           tcounts.get<uint32_t>());
    k_pq_tile_scan<<<1, 1024, 0, s>>>(tcounts.get<uint32_t>(), ntiles, toffs.get<uint64_t>(), dpresent);
    DevBuf nvals(ctx, (size_t)np * 4 + 4, nullptr);
    k_pq_indices<<<np, 32, 0, s>>>(P, valid.get<uint32_t>(), toffs.get<uint64_t>(), num_rows, nvals.get<uint32_t>(), ix_runs.get<Run>(), derr);
    ctx->count_launch(4);

    // 3. the dictionary page and PLAIN byte arrays
    DecodeArgs D{};
    D.pages = P;
    D.npages = np;
    D.runs = ix_runs.get<Run>();
    D.valid = valid.get<uint32_t>();
    D.tile_offs = toffs.get<uint64_t>();
    D.nrows = num_rows;
    D.ptype = pt;
    D.conv = cv;
    D.type_length = type_length;
    D.div = powi(10.0, scale);
    D.err = derr;
    DevBuf dptr, dlen, vptr, vlen;
    if (dict_page >= 0) {
        const Page& dpg = pages[dict_page];
        D.dict = up + uoff[dict_page];
        D.dict_n = (uint32_t)std::max(dpg.num_values, 0);
        if (pt != PQ_BYTE_ARRAY && (int64_t)D.dict_n * pw > dpg.uncompressed)
            raise(ML_ERR_INVALID, "parquet: the dictionary page is shorter than its entries");
    }
    if (pt == PQ_BYTE_ARRAY) {
        dptr = DevBuf(ctx, std::max<size_t>((size_t)D.dict_n * 8, 8), nullptr);
        dlen = DevBuf(ctx, std::max<size_t>((size_t)D.dict_n * 4, 4), nullptr);
        vptr = DevBuf(ctx, (size_t)num_rows * 8, nullptr);  // present values <= rows
        vlen = DevBuf(ctx, (size_t)num_rows * 4, nullptr);
        k_pq_byte_arrays<<<np + 1, 32, 0, s>>>(
            P, np, nvals.get<uint32_t>(), vptr.get<const uint8_t*>(), vlen.get<uint32_t>(), D.dict,
            dict_page >= 0 ? (uint32_t)pages[dict_page].uncompressed : 0u, D.dict_n, dptr.get<const uint8_t*>(),
            dlen.get<uint32_t>(), derr);
        ctx->count_launch();
        D.dict_ptr = dptr.get<const uint8_t* const>();
        D.dict_len = dlen.get<uint32_t>();
        D.vptr = vptr.get<const uint8_t* const>();
        D.vlen = vlen.get<uint32_t>();
    }

    // 4. values
    DevBuf sptr, slen, ent;
    // Strings whose pages all index one small dictionary page: its entries carry the work.  The bounds are
    // what one block holds and copies; a larger dictionary has fewer rows per string, and the rows' own
    // path spreads over the chip.
    const bool small_dict = cv == CV_UTF8 && dict_page >= 0 && D.dict_n < kPqSmallDict &&
                            (uint32_t)pages[dict_page].uncompressed <= kPqSmallDictBytes &&
                            std::all_of(hp.begin(), hp.end(), [](const PageDev& d) { return d.encoding == ENC_RLE_DICTIONARY; });
    auto string_rows = [&]() {
        sptr = DevBuf(ctx, (size_t)num_rows * 8, nullptr);
        slen = DevBuf(ctx, (size_t)num_rows * 4 + 4, nullptr);
    };
    if (small_dict) {
        ent = DevBuf(ctx, (size_t)num_rows * 4, nullptr);
        D.ent = ent.get<uint32_t>();
        D.first = dfirst;
        D.total = dtotal;
    } else if (cv == CV_UTF8) {
        string_rows();
        D.str_ptr = sptr.get<const uint8_t*>();
        D.str_len = slen.get<uint32_t>();
    } else {
        col->data = DevBuf(ctx, std::max<size_t>((size_t)num_rows * width_of(out_type), 8), b->res.get());
        D.out = col->data.get();
    }
    k_pq_values<<<(unsigned)((num_rows + kPqSlice - 1) / kPqSlice), 256, 0, s>>>(D);
    ctx->count_launch();
    const uint64_t limit = std::min<uint64_t>(std::max<uint64_t>((uint64_t)num_rows / 8, 1), 65536);  // (n / 8).clamp(1, MAX_DICT)
    bool encoded = false;
    if (small_dict) {
        const int64_t n = num_rows;
        DevBuf code_of(ctx, kPqSmallDict * 4, nullptr);
        DevBuf codes(ctx, (size_t)n * 4, b->res.get());
        k_pq_small_dict<<<1, kPqSmallDict, 0, s>>>(D.dict_ptr, D.dict_len, D.dict_n, dfirst, code_of.get<uint32_t>(), danswer);
        k_pq_codes2<<<grid_of(n), 256, 0, s>>>(ent.get<uint32_t>(), n, code_of.get<uint32_t>(), codes.get<uint32_t>());
        ctx->count_launch(2);
        std::vector<uint8_t> told(32 + answer_b);  // the status words, then the answer
        CK(cudaMemcpyAsync(told.data(), derr, told.size(), cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        std::memcpy(slot.p, told.data(), 32);
        check_pq(ctx, *slot.as<uint32_t>());
        const uint8_t* h = told.data() + 32;
        uint32_t found[2];
        std::memcpy(found, h, 8);
        if (slot.as<uint64_t>()[2] > 0xFFFFFFFFull) raise(ML_ERR_UNSUPPORTED, "parquet: a string column larger than 4 GiB");
        if (found[0] <= limit) {
            auto hd = std::make_shared<HostDict>();
            hd->bytes.assign(h + answer_head, h + answer_head + found[1]);
            std::vector<uint32_t> off(found[0] + 1);
            std::memcpy(off.data(), h + 8, off.size() * 4);
            hd->off.insert(hd->off.end(), off.begin() + 1, off.end());
            col->kind = CK_DICT;
            col->data = std::move(codes);
            col->dict = std::move(hd);
            encoded = true;
        } else {
            string_rows();
            k_pq_entry_strings<<<grid_of(n), 256, 0, s>>>(ent.get<uint32_t>(), n, D.dict_ptr, D.dict_len, D.dict_n,
                                                          sptr.get<const uint8_t*>(), slen.get<uint32_t>());
            ctx->count_launch();
        }
    } else {
        read_err();
    }
    if (slot.as<uint64_t>()[1] != (uint64_t)num_rows) {  // validity only when a value is missing (read_all)
        col->validity = std::move(valid);
    }

    // 5. strings: encode_strings (parquet_reader.rs:176-212)
    if (cv == CV_UTF8 && !encoded) {
        const int64_t n = num_rows;
        DevBuf offs(ctx, (size_t)(n + 1) * 8, nullptr), sc(ctx, std::max<size_t>(scan_scratch_words(n) * 8, 8), nullptr);
        ctx->count_launch(launch_scan_u32(slen.get<uint32_t>(), offs.get<uint64_t>(), n, sc.get<uint64_t>(), s));
        uint64_t total = 0;
        CK(cudaMemcpyAsync(&total, offs.get<uint64_t>() + n, 8, cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        if (total > 0xFFFFFFFFull) raise(ML_ERR_UNSUPPORTED, "parquet: a string column larger than 4 GiB");
        DevBuf off32(ctx, (size_t)(n + 1) * 4, b->res.get()), bytes(ctx, std::max<uint64_t>(total, 1), b->res.get());
        k_pq_str_copy<<<grid_of(n), 256, 0, s>>>(sptr.get<const uint8_t* const>(), slen.get<uint32_t>(),
                                                  offs.get<uint64_t>(), n, off32.get<uint32_t>(), bytes.get<uint8_t>());
        // equal strings get one canonical row (every row: a NULL row counts as "")
        const uint64_t cap = pow2_ceil(std::max<uint64_t>(16, (uint64_t)n * 2));
        DevBuf tslots(ctx, cap * 16, nullptr), canon(ctx, (size_t)n * 4, nullptr), first(ctx, (size_t)n * 4, nullptr);
        CK(cudaMemsetAsync(tslots.get(), 0, cap * 16, s));
        TableView tv{tslots.get<uint64_t>(), cap - 1, 1, 2};
        launch_strid(off32.get<uint32_t>(), bytes.get<uint8_t>(), nullptr, n, tv, canon.get<uint32_t>(), derr, s);
        CK(cudaMemsetAsync(first.get(), 0xFF, (size_t)n * 4, s));
        k_pq_first<<<grid_of(n), 256, 0, s>>>(canon.get<uint32_t>(), n, first.get<uint32_t>());
        const int nb = select_blocks(n), rpb = select_rows_per_block();  // launch_index_write's blocks
        DevBuf bits(ctx, (size_t)nb * rpb / 8, nullptr), counts(ctx, (size_t)nb * 4, nullptr), boffs(ctx, (size_t)(nb + 1) * 8, nullptr);
        DevBuf sc2(ctx, std::max<size_t>(scan_scratch_words(nb) * 8, 8), nullptr);
        k_pq_first_flags<<<nb, 256, 0, s>>>(canon.get<uint32_t>(), first.get<uint32_t>(), n, bits.get<uint32_t>(),
                                            counts.get<uint32_t>(), rpb);
        ctx->count_launch(launch_scan_u32(counts.get<uint32_t>(), boffs.get<uint64_t>(), nb, sc2.get<uint64_t>(), s));
        uint64_t distinct = 0;
        CK(cudaMemcpyAsync(&distinct, boffs.get<uint64_t>() + nb, 8, cudaMemcpyDeviceToHost, s));
        ctx->count_launch(4);  // the copy, the ids, the first rows and their flags
        read_err();
        if (distinct <= limit) {
            // the first occurrences in row order are the dictionary; each row's code is its string's
            DevBuf list(ctx, (size_t)distinct * 4 + 4, nullptr), code_of(ctx, (size_t)n * 4, nullptr);
            launch_index_write(n, bits.get<uint32_t>(), boffs.get<uint64_t>(), list.get<uint32_t>(), s);
            k_pq_codes<<<grid_of((int64_t)distinct), 256, 0, s>>>(list.get<uint32_t>(), (uint32_t)distinct, canon.get<uint32_t>(),
                                                                  code_of.get<uint32_t>());
            DevBuf codes(ctx, (size_t)n * 4, b->res.get());
            k_pq_codes2<<<grid_of(n), 256, 0, s>>>(canon.get<uint32_t>(), n, code_of.get<uint32_t>(), codes.get<uint32_t>());
            ctx->count_launch(3);
            // the distinct strings alone to the host: {offsets, bytes}
            const int64_t nd = (int64_t)distinct;
            DevBuf dl(ctx, (size_t)nd * 4 + 4, nullptr), doff(ctx, (size_t)(nd + 1) * 8, nullptr);
            DevBuf sc3(ctx, std::max<size_t>(scan_scratch_words(nd) * 8, 8), nullptr);
            launch_utf8_lengths(off32.get<uint32_t>(), list.get<uint32_t>(), nd, dl.get<uint32_t>(), s);
            ctx->count_launch(launch_scan_u32(dl.get<uint32_t>(), doff.get<uint64_t>(), nd, sc3.get<uint64_t>(), s));
            std::vector<uint64_t> ho(nd + 1);
            CK(cudaMemcpyAsync(ho.data(), doff.get(), (size_t)(nd + 1) * 8, cudaMemcpyDeviceToHost, s));
            CK(cudaStreamSynchronize(s));
            auto hd = std::make_shared<HostDict>();
            hd->bytes.resize(ho[nd]);
            DevBuf db(ctx, std::max<size_t>(ho[nd], 1), nullptr);
            launch_utf8_copy(off32.get<uint32_t>(), bytes.get<uint8_t>(), list.get<uint32_t>(), nd, doff.get<uint64_t>(), db.get<uint8_t>(), s);
            if (ho[nd]) CK(cudaMemcpyAsync(hd->bytes.data(), db.get(), ho[nd], cudaMemcpyDeviceToHost, s));
            ctx->count_launch(2);
            CK(cudaStreamSynchronize(s));
            for (int64_t i = 1; i <= nd; i++) hd->off.push_back((uint32_t)ho[i]);
            col->kind = CK_DICT;
            col->data = std::move(codes);
            col->dict = std::move(hd);
        } else {
            col->kind = CK_UTF8;
            col->offsets = std::move(off32);
            col->data = std::move(bytes);
        }
    }
    if (cv == CV_UTF8 && !encoded) read_err();
    b->cols.push_back(std::move(col));
    *out = b.release();
    API_END
}
