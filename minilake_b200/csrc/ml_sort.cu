// Full ORDER BY on the device: a stable radix sort of row ids by the varying bits of the sort key.
//
// sort_batches without a limit (sort.rs:85-132) is a stable sort by compare_rows.  Every sort key is a
// sequence of order-preserving 64-bit words (sort_word below; SortWord lists them least significant
// first), so a row's key is one long bit string.  Bits that are the same in every row cannot decide, so
// only the varying ones are sorted (their order is kept), or a word's distance from the smallest one
// where that is shorter (small numbers of both signs vary in every bit): 32 bits at a time form a u32
// key, sorted with its row id by 8-bit digits, one kernel per digit (k_radix_pass).
//
// With more than 32 varying bits, the top 32 usually tell almost all rows apart (10M random doubles:
// some 20k rows share theirs with another row): the rows are sorted by those, and the few runs of equal
// keys that are out of order are put right afterwards (k_sort_runs, k_sort_fix).  When a run is long,
// or the row count alone makes runs likely, every 32-bit piece is sorted instead, least significant
// first.
//
// Why: the byte-wise LSD sort of whole words this replaces moved 12 bytes in and 12 out per row and
// byte (7 varying bytes for doubles) in three kernels a byte, 2.0 ms for 10M rows; a pass here moves 8
// in and 8 out in one kernel (70 us) and four passes do: 0.42 ms with the keys and the runs.
#include <algorithm>

#include "ml_agg.cuh"
#include "ml_kernels.cuh"

namespace mlg {
namespace {

__device__ uint64_t sort_word(const SortWord& w, uint32_t r) {
    const DCol& c = w.col;
    const bool valid = valid_bit(c.valid, r);
    if (w.what == SW_NULL_FLAG) return (valid == (w.nulls_first != 0)) ? 1ull : 0ull;
    if (!valid) return 0ull;
    uint64_t x;
    if (w.what == SW_VALUE) {
        const uint64_t v = load_value(c, r);
        if (c.dt == ML_TYPE_FLOAT64) x = (uint64_t)total_key(as_f64(v)) ^ 0x8000000000000000ull;
        else if (c.dt == ML_TYPE_BOOL) x = v;
        else x = v ^ 0x8000000000000000ull;  // sign-extended integers
    } else if (w.what == SW_CHUNK) {
        const Str s = col_str(c, r);
        x = 0;
        const uint32_t b0 = 8u * (uint32_t)w.chunk;
        for (uint32_t j = 0; j < 8; j++)
            if (b0 + j < s.n) x |= (uint64_t)__ldg(s.p + b0 + j) << (56 - 8 * j);
    } else if (w.what == SW_LENGTH) {
        x = col_str(c, r).n;
    } else {  // SW_RANK: the dictionary entry's rank among the dictionary's strings
        x = __ldg(w.rank + dict_code(c, r));
    }
    return w.desc ? ~x : x;
}

// Row a before row b by the whole key (words from the most significant down).
__device__ bool sort_less(const SortWord* words, int nwords, uint32_t a, uint32_t b) {
    for (int k = nwords - 1; k >= 0; k--) {
        const uint64_t x = sort_word(words[k], a), y = sort_word(words[k], b);
        if (x != y) return x < y;
    }
    return false;
}

// A word's reader for many rows: the form and type are taken apart once, outside the row loop, so the
// loads of several rows are in flight together (through sort_word's branches each row waited for its
// own load: 52 us for 10M doubles instead of 20).
template <int DT, bool NULLS>
struct FixedWord {
    const void* data;
    const uint64_t* valid;
    uint64_t flip;
    __device__ explicit FixedWord(const SortWord& w) : data(w.col.data), valid(w.col.valid), flip(w.desc ? ~0ull : 0ull) {}
    __device__ __forceinline__ uint64_t operator()(uint32_t r) const {
        uint64_t x;
        if (DT == ML_TYPE_FLOAT64) x = (uint64_t)total_key(as_f64(__ldg((const unsigned long long*)data + r))) ^ 0x8000000000000000ull;
        else if (DT == ML_TYPE_INT64) x = (uint64_t)__ldg((const unsigned long long*)data + r) ^ 0x8000000000000000ull;
        else x = (uint64_t)(int64_t)__ldg((const int32_t*)data + r) ^ 0x8000000000000000ull;
        x ^= flip;
        return !NULLS || valid_bit(valid, r) ? x : 0ull;
    }
};
struct AnyWord {
    const SortWord& w;
    __device__ __forceinline__ uint64_t operator()(uint32_t r) const { return sort_word(w, r); }
};
template <class F>
__device__ __forceinline__ void with_word(const SortWord& w, F&& f) {
    if (w.what == SW_VALUE && w.col.kind == CK_FIXED) {
        const bool nulls = w.col.valid != nullptr;
        switch (w.col.dt) {
            case ML_TYPE_FLOAT64:
                nulls ? f(FixedWord<ML_TYPE_FLOAT64, true>(w)) : f(FixedWord<ML_TYPE_FLOAT64, false>(w));
                return;
            case ML_TYPE_INT64:
                nulls ? f(FixedWord<ML_TYPE_INT64, true>(w)) : f(FixedWord<ML_TYPE_INT64, false>(w));
                return;
            case ML_TYPE_INT32:
            case ML_TYPE_DATE:
                nulls ? f(FixedWord<ML_TYPE_INT32, true>(w)) : f(FixedWord<ML_TYPE_INT32, false>(w));
                return;
            default: break;
        }
    }
    f(AnyWord{w});
}

// Per word y (grid.y words): stats[3 y] |= the bits that differ from row 0's in some row, stats[3 y + 1]
// and [3 y + 2] = the smallest and the largest word.  One pass over the column, bound by reading it.
constexpr int kWordRows = 8;  // rows per thread and step
__global__ void __launch_bounds__(256) k_sort_bits(const SortWord* words, int64_t n, unsigned long long* stats) {
    __shared__ SortWord w;
    if (threadIdx.x == 0) w = words[blockIdx.y];
    __syncthreads();
    uint64_t acc = 0, lo = ~0ull, hi = 0;
    with_word(w, [&](auto get) {
        const uint64_t ref = get(0);
        for (int64_t base = (int64_t)blockIdx.x * (256 * kWordRows); base < n; base += (int64_t)gridDim.x * (256 * kWordRows)) {
            uint64_t x[kWordRows];
#pragma unroll
            for (int j = 0; j < kWordRows; j++) {
                const int64_t r = base + j * 256 + threadIdx.x;
                x[j] = r < n ? get((uint32_t)r) : ref;
            }
#pragma unroll
            for (int j = 0; j < kWordRows; j++) {
                acc |= x[j] ^ ref;
                lo = x[j] < lo ? x[j] : lo;
                hi = x[j] > hi ? x[j] : hi;
            }
        }
    });
    for (int o = 16; o; o >>= 1) {
        const uint64_t l = __shfl_xor_sync(0xFFFFFFFFu, lo, o), h = __shfl_xor_sync(0xFFFFFFFFu, hi, o);
        acc |= __shfl_xor_sync(0xFFFFFFFFu, acc, o);
        lo = l < lo ? l : lo;
        hi = h > hi ? h : hi;
    }
    __shared__ uint64_t part[3][8];  // one update per block: they all go to the same words
    if ((threadIdx.x & 31) == 0) {
        part[0][threadIdx.x >> 5] = acc;
        part[1][threadIdx.x >> 5] = lo;
        part[2][threadIdx.x >> 5] = hi;
    }
    __syncthreads();
    if (threadIdx.x) return;
    for (int k = 1; k < 8; k++) {
        acc |= part[0][k];
        lo = part[1][k] < lo ? part[1][k] : lo;
        hi = part[2][k] > hi ? part[2][k] : hi;
    }
    if (lo > hi) return;  // no rows
    unsigned long long* st = stats + 3 * blockIdx.y;
    const volatile unsigned long long* seen = st;
    if (acc & ~seen[0]) atomicOr(st, (unsigned long long)acc);
    if (lo < seen[1]) atomicMin(st + 1, (unsigned long long)lo);
    if (hi > seen[2]) atomicMax(st + 2, (unsigned long long)hi);
}
__global__ void k_sort_stats_init(unsigned long long* stats, int nwords) {
    if (threadIdx.x < nwords) {
        stats[3 * threadIdx.x] = 0;
        stats[3 * threadIdx.x + 1] = ~0ull;
        stats[3 * threadIdx.x + 2] = 0;
    }
}

// keys[i] = the segments' bits of row perm[i] (row i without perm), and the histograms of the key's
// 8-bit digits (hist: 256 counters per digit, zeroed).  Four histogram copies by lane, so rows with the
// same digit serialize eight at a time, not 32.
__global__ void __launch_bounds__(256) k_sort_keys(const SortWord* words, const __grid_constant__ SortSegs S,
                                                   const uint32_t* perm, int64_t n, uint32_t* keys, int digits,
                                                   uint32_t* hist, const uint32_t* err) {
    if (*err) return;  // perm was not written
    __shared__ uint32_t h[4 * 256 * 4];
    for (int i = threadIdx.x; i < digits * 1024; i += blockDim.x) h[i] = 0;
    __syncthreads();
    const uint32_t copy = threadIdx.x & 3;
    for (int64_t base = (int64_t)blockIdx.x * (256 * kWordRows); base < n; base += (int64_t)gridDim.x * (256 * kWordRows)) {
        uint32_t r[kWordRows], key[kWordRows];
#pragma unroll
        for (int j = 0; j < kWordRows; j++) {
            const int64_t i = base + j * 256 + threadIdx.x;
            r[j] = perm ? __ldg(perm + (i < n ? i : n - 1)) : (uint32_t)(i < n ? i : n - 1);
            key[j] = 0;
        }
        for (int k0 = 0, k1; k0 < S.n; k0 = k1) {  // the segments of one word are neighbours
            for (k1 = k0; k1 < S.n && S.s[k1].word == S.s[k0].word; k1++) {
            }
            with_word(words[S.s[k0].word], [&](auto get) {
                uint64_t x[kWordRows];
#pragma unroll
                for (int j = 0; j < kWordRows; j++) x[j] = get(r[j]);
                for (int k = k0; k < k1; k++) {
                    const int shift = S.s[k].shift, pos = S.s[k].pos;
                    const uint32_t mask = S.s[k].mask;
                    const uint64_t sub = S.s[k].sub;
#pragma unroll
                    for (int j = 0; j < kWordRows; j++) key[j] |= ((uint32_t)((x[j] - sub) >> shift) & mask) << pos;
                }
            });
        }
#pragma unroll
        for (int j = 0; j < kWordRows; j++) {
            const int64_t i = base + j * 256 + threadIdx.x;
            if (i >= n) continue;
            keys[i] = key[j];
            for (int d = 0; d < digits; d++) atomicAdd(&h[(d * 256 + ((key[j] >> (8 * d)) & 255)) * 4 + copy], 1u);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < digits * 256; i += blockDim.x) {
        const uint32_t c = h[4 * i] + h[4 * i + 1] + h[4 * i + 2] + h[4 * i + 3];
        if (c) atomicAdd(hist + i, c);
    }
}

// One digit of the sort in one kernel: a tile (blocks take tiles in order from a counter) ranks its
// rows by digit in shared memory and looks back over the tiles before it for its digits' offsets, so
// keys and row ids are read once and written once.  A tile's count of a digit is published as soon as
// it is known, its inclusive prefix once the look-back has it; both are one 64-bit word with its kind
// in the top bits, so no fence is needed.
// 8,192 rows per tile: a digit's rows of a tile (32 on average) are written as whole 128-byte runs.
// 98 KB of shared memory, two blocks per SM.  Bound by instruction issue and the latency of its phases
// (load, rank, look back, write): 70 us for 10M rows (160 MB moved).  Measured on the way: ranking with
// eight ballots per row instead of a shared-memory OR of the lanes 89 us, with match.any 112 us; one
// predecessor per look-back step instead of eight 103 us; smaller tiles or three blocks per SM no better.
constexpr int kPassThreads = 512, kPassItems = 16, kPassTile = kPassThreads * kPassItems, kPassWarps = kPassThreads / 32;
constexpr size_t kPassSmem = (size_t)kPassTile * 8 + (size_t)kPassWarps * 256 * 8 + 2 * 256 * 4;
constexpr uint64_t kStatCount = 1ull << 62, kStatPrefix = 2ull << 62, kStatPoison = 3ull << 62, kStatValue = (1ull << 62) - 1;
constexpr uint32_t kPassSpins = 1u << 21;  // polls of a predecessor's word (about a second)
// A pass that gives up sets *err and leaves row ids unwritten; the kernels queued behind it read *err first
// and touch no row.

__global__ void __launch_bounds__(kPassThreads, 2)
    k_radix_pass(const uint32_t* keys_in, const uint32_t* rows_in, uint32_t n, int shift, const uint32_t* hist,
                 uint64_t* status, uint32_t* next_tile, uint32_t* keys_out, uint32_t* rows_out, uint32_t* err) {
    extern __shared__ __align__(16) uint32_t pass_smem[];
    uint32_t* skey = pass_smem;
    uint32_t* srow = skey + kPassTile;
    uint2* wdig = (uint2*)(srow + kPassTile);             // per warp and digit: lanes of the step, rows so far
    uint32_t* tstart = (uint32_t*)(wdig + kPassWarps * 256);  // first position of a digit in the tile
    uint32_t* gstart = tstart + 256;                         // its global position minus tstart
    __shared__ uint32_t tile_s, bad_s;
    __shared__ uint64_t wsum[8];
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (tid == 0) {
        tile_s = atomicAdd(next_tile, 1u);
        bad_s = *(const volatile uint32_t*)err != 0;
    }
    for (uint32_t i = tid; i < kPassWarps * 256; i += kPassThreads) wdig[i] = make_uint2(0u, 0u);
    __syncthreads();
    const uint32_t tile = tile_s;
    if (bad_s) {  // rows_in was not written, or this pass gave up: tiles behind this one need not wait
        if (tid < 256) *(volatile uint64_t*)(status + (uint64_t)tile * 256 + tid) = kStatPoison;
        return;
    }
    const uint64_t base = (uint64_t)tile * kPassTile;
    const uint32_t rows = (uint32_t)min((uint64_t)kPassTile, (uint64_t)n - base);
    // a warp's rows are consecutive (512 of them), 32 per step: input order is warp, step, lane
    const uint32_t first = w * (32 * kPassItems) + lane;
    uint32_t key[kPassItems], rank[kPassItems / 2];
    // rows past the end read as the largest key: they come last in the last digit of the last tile, past
    // the positions that are written, and no tile looks back at this one
#pragma unroll
    for (int j = 0; j < kPassItems; j++) key[j] = first + 32 * j < rows ? __ldg(keys_in + base + first + 32 * j) : 0xFFFFFFFFu;
    const uint32_t lt = (1u << lane) - 1u;
    uint2* const wd = wdig + w * 256;
#pragma unroll
    for (int j = 0; j < kPassItems; j++) {
        const uint32_t d = (key[j] >> shift) & 255;
        atomicOr(&wd[d].x, 1u << lane);
        __syncwarp();
        const uint2 v = wd[d];  // the warp's lanes with this digit; its rows with it so far
        __syncwarp();
        const uint32_t peers = v.x, before = v.y;
        if ((peers & lt) == 0) wd[d] = make_uint2(0u, before + __popc(peers));
        __syncwarp();
        const uint32_t r = before + __popc(peers & lt);  // below 512
        rank[j / 2] = j & 1 ? rank[j / 2] | (r << 16) : r;
    }
    __syncthreads();
    uint32_t total = 0;
    if (tid < 256) {  // digit tid: the warps' counts become offsets
#pragma unroll
        for (int k = 0; k < kPassWarps; k++) {
            const uint32_t c = wdig[k * 256 + tid].y;
            wdig[k * 256 + tid].y = total;
            total += c;
        }
        *(volatile uint64_t*)(status + (uint64_t)tile * 256 + tid) = (tile ? kStatCount : kStatPrefix) | total;
        // the digits' starts in the tile (low half) and in the whole output (high half): one scan
        const uint64_t mine = ((uint64_t)__ldg(hist + tid) << 32) | total;
        uint64_t incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if ((int)lane >= o) incl += t;
        }
        if (lane == 31) wsum[w] = incl;
        asm volatile("bar.sync 1, 256;" ::: "memory");
        uint64_t off = incl - mine;
        for (uint32_t k = 0; k < w; k++) off += wsum[k];
        tstart[tid] = (uint32_t)off;
        gstart[tid] = (uint32_t)((off >> 32) - (uint32_t)off);
    }
    __syncthreads();
    // the tile in digit order
    uint32_t row[kPassItems];
#pragma unroll
    for (int j = 0; j < kPassItems; j++) {
        row[j] = (uint32_t)base + first + 32 * j;
        if (rows_in) row[j] = first + 32 * j < rows ? __ldg(rows_in + base + first + 32 * j) : 0u;
    }
#pragma unroll
    for (int j = 0; j < kPassItems; j++) {
        const uint32_t d = (key[j] >> shift) & 255;
        const uint32_t p = tstart[d] + wd[d].y + (j & 1 ? rank[j / 2] >> 16 : rank[j / 2] & 0xFFFFu);
        skey[p] = key[j];
        srow[p] = row[j];
    }
    if (tid < 256 && tile) {  // look back for the digit's rows in earlier tiles
        uint64_t excl = 0;
        uint32_t spins = 0;
        bool bad = false;
        for (int64_t t = (int64_t)tile - 1; t >= 0 && !bad;) {  // eight predecessors per round trip
            uint64_t v[8];
#pragma unroll
            for (int k = 0; k < 8; k++) v[k] = *(const volatile uint64_t*)(status + (uint64_t)max(t - k, (int64_t)0) * 256 + tid);
            bool done = false;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                if (done || t < 0) break;
                const uint64_t kind = v[k] & ~kStatValue;
                if (kind == 0) break;  // not there yet: poll again from this one
                if (kind == kStatPoison) bad = true;
                excl += v[k] & kStatValue;
                done = kind != kStatCount;
                t--;
            }
            if (done) break;
            bad = bad || ++spins > kPassSpins;
        }
        *(volatile uint64_t*)(status + (uint64_t)tile * 256 + tid) = bad ? kStatPoison : kStatPrefix | (excl + total);
        if (bad) bad_s = 1;
        gstart[tid] += (uint32_t)excl;
    }
    __syncthreads();
    if (bad_s) {  // a predecessor never published: nothing is written, the host sees the error
        if (tid == 0) atomicOr(err, (uint32_t)DE_TIMEOUT);
        return;
    }
    for (uint32_t p = tid; p < rows; p += kPassThreads) {
        const uint32_t k = skey[p];
        const uint32_t o = gstart[(k >> shift) & 255] + p;
        if (keys_out) keys_out[o] = k;
        rows_out[o] = srow[p];
    }
}

// Runs of equal keys that the whole key orders differently: one entry {first, length} per such run in
// `list` (`count` entries; state[0] counts them, state[1] is set when a run is longer than kSortRunMax
// or the list is full).  The thread at a run's first inversion reports it.  A run without inversions
// (equal rows) costs its compares only.  Bound by the latency of the key loads: one key per thread and step
// 41 us for 10M rows, eight in two 16-byte loads 26 us.
constexpr uint32_t kSortRunMax = 64;
__global__ void __launch_bounds__(256) k_sort_runs(const uint32_t* keys, const uint32_t* rows, const SortWord* words,
                                                   int nwords, uint32_t n, uint2* list, uint32_t cap, uint32_t* state,
                                                   const uint32_t* err) {
    if (*err) return;
    // an equal neighbour: whether this is its run's first inversion, and the run's ends
    auto check = [&](uint32_t i, uint32_t k) {
        if (!sort_less(words, nwords, rows[i], rows[i - 1])) return;
        uint32_t s = i - 1, e = i + 1;
        bool mine = true;
        while (mine && s > 0 && i - s < kSortRunMax && keys[s - 1] == k) {
            mine = !sort_less(words, nwords, rows[s], rows[s - 1]);
            s--;
        }
        if (!mine) return;
        while (e < n && e - s <= kSortRunMax && keys[e] == k) e++;
        uint32_t at = cap;
        if (i - s < kSortRunMax && e - s <= kSortRunMax) at = atomicAdd(state, 1u);
        if (at < cap) list[at] = make_uint2(s, e - s);
        else state[1] = 1;
    };
    // eight keys per thread and step (the key array is 16-byte aligned) and the one before them
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x * 8;
    for (uint64_t q = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) * 8; q < n; q += stride) {
        const uint32_t i = (uint32_t)q;
        uint32_t k[9];
        k[0] = i ? keys[i - 1] : 0u;
        if (q + 8 <= n) {
            const uint4 a = *(const uint4*)(keys + i), b = *(const uint4*)(keys + i + 4);
            k[1] = a.x, k[2] = a.y, k[3] = a.z, k[4] = a.w, k[5] = b.x, k[6] = b.y, k[7] = b.z, k[8] = b.w;
        } else {
#pragma unroll
            for (int j = 0; j < 8; j++) k[j + 1] = q + j < n ? keys[i + j] : 0u;
        }
        uint32_t same = 0;
#pragma unroll
        for (int j = 0; j < 8; j++) same |= (uint32_t)(k[j] == k[j + 1] && q + j < n && q + j > 0) << j;
        for (; same; same &= same - 1) {
            const uint32_t j = i + (uint32_t)__ffs(same) - 1;
            check(j, keys[j]);
        }
    }
}
// Each reported run put in order in place (an insertion sort, which keeps equal rows' order).
__global__ void __launch_bounds__(256) k_sort_fix(uint32_t* rows, const SortWord* words, int nwords, const uint2* list,
                                                  uint32_t cap, const uint32_t* state, const uint32_t* err) {
    if (*err) return;
    const uint32_t m = min(state[0], cap);
    if (state[1]) return;  // every piece will be sorted instead
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < m; j += gridDim.x * blockDim.x) {
        uint32_t* r = rows + list[j].x;
        for (uint32_t a = 1; a < list[j].y; a++) {
            const uint32_t x = r[a];
            uint32_t b = a;
            for (; b > 0 && sort_less(words, nwords, x, r[b - 1]); b--) r[b] = r[b - 1];
            r[b] = x;
        }
    }
}

// Longest string of a plain UTF8 column (for the number of 8-byte chunk words).
__global__ void k_max_strlen(const uint32_t* off, int64_t n, unsigned int* out) {
    uint32_t m = 0;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) m = max(m, off[i + 1] - off[i]);
    for (int o = 16; o; o >>= 1) m = max(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
    if ((threadIdx.x & 31) == 0 && m) atomicMax(out, m);
}
__global__ void k_iota_u32(uint32_t* out, int64_t n) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) out[i] = (uint32_t)i;
}

int grid_rows(int64_t n, int rows_per_block, int per_sm) {
    return (int)std::max<int64_t>(1, std::min<int64_t>((n + rows_per_block - 1) / rows_per_block, (int64_t)num_sms() * per_sm));
}
}  // namespace

void launch_iota_u32(uint32_t* out, int64_t n, cudaStream_t s) {
    if (n > 0) k_iota_u32<<<grid_rows(n, 256, 8), 256, 0, s>>>(out, n);
}
void launch_max_strlen(const uint32_t* off, int64_t n, unsigned int* out, cudaStream_t s) {
    if (n > 0) k_max_strlen<<<grid_rows(n, 256, 4), 256, 0, s>>>(off, n, out);
}
void launch_sort_bits(const SortWord* words, int nwords, int64_t n, unsigned long long* stats, cudaStream_t s) {
    k_sort_stats_init<<<1, 32, 0, s>>>(stats, nwords);
    if (n > 0 && nwords > 0) k_sort_bits<<<dim3(grid_rows(n, 256 * kWordRows, 6), nwords), 256, 0, s>>>(words, n, stats);
}
void launch_sort_keys(const SortWord* words, const SortSegs& S, const uint32_t* perm, int64_t n, uint32_t* keys, int digits,
                      uint32_t* hist, const uint32_t* err, cudaStream_t s) {
    if (n > 0) k_sort_keys<<<grid_rows(n, 256 * kWordRows, 8), 256, 0, s>>>(words, S, perm, n, keys, digits, hist, err);
}
int64_t radix_tiles(int64_t n) { return (n + kPassTile - 1) / kPassTile; }
cudaError_t launch_radix_pass(const uint32_t* keys_in, const uint32_t* rows_in, int64_t n, int shift, const uint32_t* hist,
                              uint64_t* status, uint32_t* next_tile, uint32_t* keys_out, uint32_t* rows_out, uint32_t* err,
                              cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    // per call: the attribute belongs to the current device's copy of the kernel
    const cudaError_t e = cudaFuncSetAttribute(k_radix_pass, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPassSmem);
    if (e != cudaSuccess) return e;
    k_radix_pass<<<(unsigned)radix_tiles(n), kPassThreads, kPassSmem, s>>>(keys_in, rows_in, (uint32_t)n, shift, hist, status,
                                                                           next_tile, keys_out, rows_out, err);
    return cudaSuccess;
}
void launch_sort_runs(const uint32_t* keys, uint32_t* rows, const SortWord* words, int nwords, int64_t n, uint2* list,
                      uint32_t cap, uint32_t* state, const uint32_t* err, cudaStream_t s) {
    if (n < 2) return;
    k_sort_runs<<<grid_rows(n, 256 * 8, 8), 256, 0, s>>>(keys, rows, words, nwords, (uint32_t)n, list, cap, state, err);
    k_sort_fix<<<grid_rows(cap, 256, 4), 256, 0, s>>>(rows, words, nwords, list, cap, state, err);
}

}  // namespace mlg
