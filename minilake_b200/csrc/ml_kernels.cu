// sm_100a kernels of the MiniLake execution core.
//
// All of MiniLake's hot-path operators are HBM-bandwidth or L2-latency bound
// integer/byte/FP64 work: nothing here is a dense contraction, so there is no
// tensor-core code.  The design rules are the ones that matter for HBM-bound
// kernels on B200: one pass over each column with coalesced loads, grids sized
// as a multiple of the 148 SMs, state that fits in L2 (126 MB) kept there, and
// shared-memory privatization wherever many rows hit few addresses.
#include <algorithm>
#include <cmath>

#include "ml_agg.cuh"
#include "ml_kernels.cuh"

namespace mlg {

int num_sms() {
    static const int sms = [] {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        return n > 0 ? n : 148;
    }();
    return sms;
}

namespace {
constexpr int kThreads = 256;
int grid_for(int64_t n, int per_sm = 8) {
    int64_t want = (n + kThreads - 1) / kThreads;
    int64_t cap = (int64_t)num_sms() * per_sm;
    if (want < 1) want = 1;
    return (int)(want < cap ? want : cap);
}

__device__ __forceinline__ EvalEnv env_of(const PipeArgs& P) {
    return EvalEnv{P.cols, P.prog, P.arena, P.luts};
}

// Chain cursors of up to four probes, in named registers (no local-memory array).
struct Cursors {
    uint32_t c0 = kNone, c1 = kNone, c2 = kNone, c3 = kNone;
    __device__ __forceinline__ uint32_t get(int p) const {
        switch (p) {
            case 0: return c0;
            case 1: return c1;
            case 2: return c2;
            default: return c3;
        }
    }
    __device__ __forceinline__ void set(int p, uint32_t v) {
        switch (p) {
            case 0: c0 = v; break;
            case 1: c1 = v; break;
            case 2: c2 = v; break;
            default: c3 = v; break;
        }
    }
};

// Build row matching the normalized key `w` through probe `pd` (dense index or hash table).
__device__ __forceinline__ uint32_t probe_find(const ProbeDev& pd, const uint64_t* w) {
    if (pd.dense && pd.late) return dense_slot(pd.dmin, pd.drange, w[0]);
    if (pd.dense && pd.member) return dense_member(pd.member, pd.dmin, pd.drange, w[0]);
    if (pd.dense) return dense_find(pd.dense, pd.dmin, pd.drange, w[0]);
    return table_find(pd.t, w, key_hash(w, pd.t.nwords));
}

// Run the streaming stages for one source row; call sink(ctx) for every surviving
// (row, build matches...) combination.  Duplicate build keys are walked through their
// chains with backtracking, like HashJoinProbe's chain walk (join.rs:297-309).
template <class Sink>
__device__ __forceinline__ void run_stages(const PipeArgs& P, const EvalEnv& env, RowCtx& x, Sink&& sink) {
    if (!P.has_chains) {  // every build key is distinct: at most one match per probe, no backtracking
        for (int s = 0; s < P.nstages; s++) {
            const Stage st = P.stages[s];
            if (st.kind == 0) {
                uint64_t v;
                bool ok;
                eval_prog(env, P.filters[st.idx], x, v, ok);
                if (!(ok && (v & 1))) return;
            } else {
                const ProbeDev& pd = P.probes[st.idx];
                uint64_t w[2];
                uint32_t nm;
                if (!make_key(env, pd.keys, x, w, &nm, true)) return;
                uint32_t b = probe_find(pd, w);
                if (b == kNone) return;
                x.set_build(st.idx, b);
                if (st.idx == P.head_probe) x.head = b;
            }
        }
        sink(x);
        return;
    }
    Cursors cur;
    int s = 0;
    for (;;) {
        bool advance = false;
        if (s == P.nstages) {
            sink(x);
        } else {
            const Stage st = P.stages[s];
            if (st.kind == 0) {
                uint64_t v;
                bool ok;
                eval_prog(env, P.filters[st.idx], x, v, ok);
                advance = ok && (v & 1);
            } else {
                const ProbeDev& pd = P.probes[st.idx];
                uint64_t w[2];
                uint32_t nm;
                if (make_key(env, pd.keys, x, w, &nm, true)) {
                    uint32_t b = probe_find(pd, w);
                    if (b != kNone) {
                        x.set_build(st.idx, b);
                        if (st.idx == P.head_probe) x.head = b;
                        cur.set(st.idx, pd.next ? __ldg(pd.next + b) : kNone);
                        advance = true;
                    }
                }
            }
        }
        if (advance) {
            s++;
            continue;
        }
        int q = s - 1;
        for (; q >= 0; q--) {
            const Stage st = P.stages[q];
            if (st.kind != 1) continue;
            uint32_t c = cur.get(st.idx);
            if (c != kNone) {
                x.set_build(st.idx, c);
                cur.set(st.idx, __ldg(P.probes[st.idx].next + c));
                break;
            }
        }
        if (q < 0) return;
        s = q + 1;
    }
}

__device__ __forceinline__ void agg_fold(const PipeArgs& P, const AggArgs& A, const EvalEnv& env, const RowCtx& x,
                                         uint64_t* blk, uint32_t g) {
    atomicAdd((unsigned long long*)blk, 1ull);
    for (int k = 0; k < A.nagg; k++) {
        const AggDev& a = A.aggs[k];
        if (a.func == ML_AGG_COUNT_STAR) continue;  // COUNT(*) is the row counter (word 0)
        uint64_t v = 0;
        bool ok = true;
        if (a.has_arg) eval_prog(env, a.arg, x, v, ok);
        if (!ok) continue;
        if (a.kind == A_MIN_STR || a.kind == A_MAX_STR) v = str_pack(A.str_rank, (uint32_t)v);
        acc_apply(a.kind, blk + a.off, v);
        if (a.count_valid) atomicAdd((unsigned long long*)a.vcnt + g, 1ull);
    }
}

__device__ __forceinline__ void agg_update(const PipeArgs& P, const AggArgs& A, const EvalEnv& env, const RowCtx& x,
                                           uint64_t* smem) {
    uint32_t g;
    if (A.group_probe >= 0) {
        g = x.head;  // every row of a key's chain aggregates into the chain head's group
    } else if (A.ungrouped) {
        g = 0;
    } else {
        uint64_t w[2];
        uint32_t nm;
        make_key(env, A.keys, x, w, &nm, false);
        uint64_t h = key_hash(w, A.keys.nwords, nm);
        bool inserted;
        uint64_t slot;
        g = table_upsert(
            A.t, w, nm, h, P.err, [&]() -> uint32_t { return new_group(A); }, &inserted, &slot, A.ngroups, A.gid_cap);
        if (g == kNone) {
            record_overflow(P, A, x);
            return;
        }
        if (inserted) {
            A.gkeys[g] = w[0];
            if (A.keys.nwords > 1) A.gkeys[(uint64_t)A.gid_cap + g] = w[1];
            A.gnull[g] = nm;
        }
    }
    if ((int)g < A.smem_groups) agg_fold(P, A, env, x, smem + (uint64_t)g * A.stride, g);
    else agg_fold(P, A, env, x, A.acc + (uint64_t)g * A.stride, g);
}

__global__ void __launch_bounds__(kThreads) k_agg(const __grid_constant__ PipeArgs P, const __grid_constant__ AggArgs A) {
    extern __shared__ __align__(16) uint64_t smem[];
    smem_setup(A, smem);
    __syncthreads();
    const EvalEnv env = env_of(P);
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < P.n; i += stride) {
        RowCtx x;
        bool ok = true;
        x.r = sel_row(P, i, ok);
        if (!ok) continue;
        x.b0 = x.b1 = x.b2 = x.b3 = 0;
        x.head = 0;
        run_stages(P, env, x, [&](const RowCtx& c) { agg_update(P, A, env, c, smem); });
    }
    __syncthreads();
    smem_flush(A, smem);
}

__global__ void __launch_bounds__(kThreads) k_agg_resume(const __grid_constant__ PipeArgs P, const __grid_constant__ AggArgs A,
                                                         const uint32_t* ctx, uint64_t count, int w) {
    extern __shared__ __align__(16) uint64_t smem[];
    smem_setup(A, smem);
    __syncthreads();
    const EvalEnv env = env_of(P);
    uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += stride) {
        const uint32_t* c = ctx + i * (uint64_t)w;
        RowCtx x;
        x.r = c[0];
        x.b0 = w > 1 ? c[1] : 0;
        x.b1 = w > 2 ? c[2] : 0;
        x.b2 = w > 3 ? c[3] : 0;
        x.b3 = w > 4 ? c[4] : 0;
        x.head = 0;
        agg_update(P, A, env, x, smem);
    }
    __syncthreads();
    smem_flush(A, smem);
}

// ---- exchange partitioning: rows grouped by key hash % nparts, input order kept ----------------
// Per 1024-row block: counts[p * blocks + b] = rows of block b in partition p.
__global__ void __launch_bounds__(kXPartRows) k_xpart_count(const uint64_t* h, int64_t n, int nparts, uint32_t* counts) {
    __shared__ uint32_t hist[kMaxExchangeParts];
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    const int64_t r = (int64_t)blockIdx.x * kXPartRows + threadIdx.x;
    if (r < n) atomicAdd(&hist[h[r] % (uint64_t)nparts], 1u);
    __syncthreads();
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) counts[(int64_t)i * gridDim.x + blockIdx.x] = hist[i];
}
// perm[pos] = row: pos = the (partition, block) offset + the row's rank among the block's rows of
// its partition (warps in order, lanes in order within a warp: a stable counting sort).
__global__ void __launch_bounds__(kXPartRows) k_xpart_scatter(const uint64_t* h, int64_t n, int nparts,
                                                             const uint64_t* offs, uint32_t* perm) {
    __shared__ uint32_t wcnt[kXPartRows / 32][kMaxExchangeParts];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < (kXPartRows / 32) * kMaxExchangeParts; i += blockDim.x)
        wcnt[i / kMaxExchangeParts][i % kMaxExchangeParts] = 0;
    __syncthreads();
    const int64_t r = (int64_t)blockIdx.x * kXPartRows + threadIdx.x;
    const bool in = r < n;
    const uint32_t p = in ? (uint32_t)(h[r] % (uint64_t)nparts) : 0xFFFFFFFFu;
    const unsigned same = __match_any_sync(0xFFFFFFFFu, p);
    const uint32_t rank = __popc(same & ((1u << lane) - 1u));
    if (in && rank == 0) wcnt[w][p] = __popc(same);  // the group's lowest lane
    __syncthreads();
    for (int q = threadIdx.x; q < nparts; q += blockDim.x) {  // exclusive prefix over the warps
        uint32_t run = 0;
        for (int ww = 0; ww < kXPartRows / 32; ww++) {
            const uint32_t c = wcnt[ww][q];
            wcnt[ww][q] = run;
            run += c;
        }
    }
    __syncthreads();
    if (in) perm[offs[(int64_t)p * gridDim.x + blockIdx.x] + wcnt[w][p] + rank] = (uint32_t)r;
}

// ---- out-of-HBM aggregation (aggregate/hash.rs:189-281, 369-425) ------------------------------
// Spill partition of each group: bits 32..35 of its key hash, which the table's slot choice (the
// low bits) does not use, so every partition's groups still hash well into a table of their own.
__global__ void k_spill_part(const uint64_t* gkeys, const uint32_t* gnull, uint32_t gid_cap, uint32_t ng, int nwords,
                             uint64_t* part) {
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= ng) return;
    const uint64_t w[2] = {gkeys[g], nwords > 1 ? gkeys[(uint64_t)gid_cap + g] : 0ull};
    part[g] = (key_hash(w, nwords, gnull[g]) >> 32) & (kSpillParts - 1);
}
// Merge spilled partial states (n groups: key words as nwords planes of n, null masks, group
// blocks of A.stride words, valid-input counts as planes of n for the aggregates that keep them)
// into the table: a group's block adds up (counts, sums, AVG's sum and count) or folds (MIN/MAX),
// as HashAggState::merge_partial merges partial batches (aggregate/hash.rs:125-139).
__global__ void k_agg_merge_spill(const __grid_constant__ AggArgs A, const uint64_t* keys, const uint32_t* nulls,
                                  const uint64_t* acc, const uint64_t* vcnt, uint32_t n, uint32_t* err) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const uint64_t w[2] = {keys[r], A.keys.nwords > 1 ? keys[(uint64_t)n + r] : 0ull};
    const uint32_t nm = nulls[r];
    bool ins;
    uint64_t slot;
    const uint32_t g = table_upsert(A.t, w, nm, key_hash(w, A.keys.nwords, nm), err, [&]() -> uint32_t { return new_group(A); }, &ins, &slot, A.ngroups, A.gid_cap);
    if (g == kNone) {  // the table is sized for every spilled row of the partition: not reached
        atomicOr(err, (uint32_t)DE_OVERFLOW_LOST);
        return;
    }
    if (ins) {
        A.gkeys[g] = w[0];
        if (A.keys.nwords > 1) A.gkeys[(uint64_t)A.gid_cap + g] = w[1];
        A.gnull[g] = nm;
    }
    uint64_t* blk = A.acc + (uint64_t)g * A.stride;
    const uint64_t* src = acc + (uint64_t)r * A.stride;
    if (src[0]) atomicAdd((unsigned long long*)blk, (unsigned long long)src[0]);
    int v = 0;
    for (int k = 0; k < A.nagg; k++) {
        const AggDev& a = A.aggs[k];
        if (a.func == ML_AGG_COUNT_STAR) continue;
        acc_merge(a.kind, blk + a.off, src + a.off);
        if (a.vcnt) {
            const uint64_t c = vcnt[(uint64_t)v * n + r];
            if (c) atomicAdd((unsigned long long*)a.vcnt + g, (unsigned long long)c);
            v++;
        }
    }
}

__global__ void k_agg_rehash(TableView t, const uint64_t* gkeys, const uint32_t* gnull, uint32_t gid_cap, uint32_t ngroups,
                             int nwords, uint32_t* err) {
    uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= ngroups) return;
    uint64_t w[2] = {gkeys[g], nwords > 1 ? gkeys[(uint64_t)gid_cap + g] : 0ull};
    uint32_t nm = gnull[g];
    bool inserted;
    uint64_t slot;
    table_upsert(t, w, nm, key_hash(w, nwords, nm), err, [&]() { return g; }, &inserted, &slot);
}

__global__ void k_agg_guard(const unsigned long long* ovf_count, const uint32_t* ngroups, uint32_t gid_cap, uint32_t* skip) {
    *skip = *ovf_count > 0 || *ngroups > gid_cap / 4;
}

// Start values of the blocks of groups [from, to): bound by writing them, so a thread writes neighbouring
// 16-byte pieces of the whole range (3.1M groups of 8 words: 42 us; a block per thread took 184 us).
__global__ void __launch_bounds__(kThreads) k_acc_init(const __grid_constant__ AggArgs A, uint32_t from, uint32_t to) {
    __shared__ uint64_t pat[2 * (1 + 2 * kMaxAggs)];  // two blocks' words (an odd stride shifts by one)
    const int S = A.stride;
    if (threadIdx.x < 2 * S) pat[threadIdx.x] = 0;
    __syncthreads();
    if (threadIdx.x < 2 * A.nagg) {
        const AggDev& a = A.aggs[threadIdx.x >> 1];
        if (a.func != ML_AGG_COUNT_STAR) pat[a.off + (threadIdx.x & 1) * S] = agg_identity(a.kind);
    }
    __syncthreads();
    uint64_t* acc = A.acc + (uint64_t)from * S;
    const uint64_t words = (uint64_t)(to - from) * S, stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t lead = ((uintptr_t)acc >> 3) & 1;  // the first word when the range starts off a 16-byte boundary
    const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (lead && t0 == 0 && words) acc[0] = pat[0];
    for (uint64_t i = t0 * 2 + lead; i + 1 < words; i += stride * 2) {
        const int w = (int)(i % (uint64_t)S);
        *(ulonglong2*)(acc + i) = make_ulonglong2(pat[w], pat[w + 1]);
    }
    if (t0 == 0 && words > lead && ((words - lead) & 1)) acc[words - 1] = pat[S - 1];
    for (int k = 0; k < A.nagg; k++)
        if (A.aggs[k].vcnt)
            for (uint64_t g = from + t0; g < to; g += stride) A.aggs[k].vcnt[g] = 0;
}

// Validity word w (32 rows) of ng rows; the last word's other half, when it has one, is cleared.
__device__ __forceinline__ void put_valid(uint32_t* valid, uint32_t w, uint32_t ng, uint32_t bits) {
    const uint32_t words = (ng + 31) / 32;
    if (w < words) valid[w] = bits;
    if (w + 1 == words && (words & 1)) valid[w + 1] = 0;
}

// Final values (accumulator.rs:500-526): AVG = sum / count, empty -> NULL.
__global__ void k_agg_final(const __grid_constant__ FinalArgs F) {
    uint32_t o = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t ng = F.ngroups;
    if (F.ng64) ng = (uint32_t)min((uint64_t)ng, __ldg(F.ng64));
    if (F.ng32) ng = min(ng, __ldg(F.ng32));
    bool in = o < ng;
    uint32_t g = in ? (F.gids ? F.gids[o] : o) : 0;
    uint32_t lane = threadIdx.x & 31;
    for (int k = 0; k < F.nkeys; k++) {
        const KeyField f = F.f[k];
        bool valid = true;
        if (in) {
            uint64_t w = F.gkeys[(uint64_t)f.word * F.gid_cap + g];
            valid = !((F.gnull[g] >> k) & 1u);
            uint64_t m = f.width >= 64 ? ~0ull : ((1ull << f.width) - 1);
            uint64_t v = (w >> f.shift) & m;
            if (f.strid) ((uint32_t*)F.key_out[k])[o] = (uint32_t)v;
            else if (f.type == ML_TYPE_BOOL) ((uint8_t*)F.key_out[k])[o] = (uint8_t)v;
            else if (f.type == ML_TYPE_INT32 || f.type == ML_TYPE_DATE) ((int32_t*)F.key_out[k])[o] = (int32_t)(uint32_t)v;
            else ((uint64_t*)F.key_out[k])[o] = v;
        }
        uint32_t bits = __ballot_sync(0xFFFFFFFFu, in && valid);
        if (lane == 0) put_valid(F.key_valid[k], o >> 5, ng, bits);
    }
    const uint64_t* blk = F.acc + (uint64_t)g * F.stride;
    for (int k = 0; k < F.nagg; k++) {
        const AggDev& a = F.aggs[k];
        bool valid = false;
        if (in) {
            uint64_t rows = blk[0];
            uint64_t vc = a.vcnt ? a.vcnt[g] : blk[a.cnt_off];
            if (a.func == ML_AGG_COUNT_STAR) {
                ((int64_t*)F.agg_out[k])[o] = (int64_t)rows;
                valid = true;
            } else if (a.func == ML_AGG_COUNT) {
                ((int64_t*)F.agg_out[k])[o] = (int64_t)blk[a.off];
                valid = true;
            } else {
                uint64_t v = blk[a.off];
                valid = vc > 0;
                switch (a.kind) {
                    case A_AVG: {
                        uint64_t c = blk[a.off + 1];
                        valid = c > 0;
                        double r = c == 0 ? 0.0 : __ddiv_rn(as_f64(v), __ll2double_rn((long long)c));
                        ((double*)F.agg_out[k])[o] = r;
                        break;
                    }
                    case A_MIN_F64:
                    case A_MAX_F64: ((double*)F.agg_out[k])[o] = valid ? f64_unorder(v) : 0.0; break;
                    case A_MIN_STR:
                    case A_MAX_STR: ((uint32_t*)F.agg_out[k])[o] = valid ? (uint32_t)v : 0u; break;  // the id
                    case A_MIN_I64:
                    case A_MAX_I64:
                        if (F.out_type[k] == ML_TYPE_INT32 || F.out_type[k] == ML_TYPE_DATE)
                            ((int32_t*)F.agg_out[k])[o] = valid ? (int32_t)(int64_t)v : 0;
                        else
                            ((int64_t*)F.agg_out[k])[o] = valid ? (int64_t)v : 0;
                        break;
                    default: ((uint64_t*)F.agg_out[k])[o] = v; break;
                }
            }
        }
        uint32_t bits = __ballot_sync(0xFFFFFFFFu, in && valid);
        if (lane == 0) put_valid(F.agg_valid[k], o >> 5, ng, bits);
    }
}

// ---- filter: pass bits + per-block counts, then ordered compaction ---------------------------
constexpr int kSelRowsPerBlock = kThreads * 8;

__global__ void __launch_bounds__(kThreads) k_select_flags(const __grid_constant__ PipeArgs P, uint32_t* bits,
                                                           uint32_t* block_counts) {
    const EvalEnv env = env_of(P);
    int64_t base = (int64_t)blockIdx.x * kSelRowsPerBlock;
    uint32_t cnt = 0;
    for (int it = 0; it < 8; it++) {
        int64_t i = base + it * kThreads + threadIdx.x;
        bool pass = false;
        bool ok = i < P.n;
        RowCtx x;
        if (ok) x.r = sel_row(P, i, ok);
        if (ok) {
            x.b0 = x.b1 = x.b2 = x.b3 = 0;
            x.head = 0;
            run_stages(P, env, x, [&](const RowCtx&) { pass = true; });
        }
        uint32_t b = __ballot_sync(0xFFFFFFFFu, pass);
        if ((threadIdx.x & 31) == 0 && base + it * kThreads + (threadIdx.x & ~31) < P.n)
            bits[(base + it * kThreads + threadIdx.x) >> 5] = b;
        cnt += pass;
    }
    // block reduce
    __shared__ uint32_t red[kThreads / 32];
    for (int o = 16; o; o >>= 1) cnt += __shfl_xor_sync(0xFFFFFFFFu, cnt, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = cnt;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int w = 0; w < kThreads / 32; w++) t += red[w];
        block_counts[blockIdx.x] = t;
    }
}

// Bits of a pass mask (u32 words) -> the ordered positions (sel[i] when a selection is given) and, with
// PAIRS, their entries of `builds`.  A warp takes 1,024 rows, a word per lane, and writes each word's rows
// with one store: bound by writing the result, so nothing else is in the loop (100M rows of which 96.5M
// are kept: 114 us with a block-wide scan and a shared-memory offset per word, 76 us so).
template <bool SEL, bool PAIRS>
__global__ void __launch_bounds__(kThreads) k_index_write(int64_t n, const uint32_t* sel, const uint32_t* bits,
                                                          const uint64_t* block_offsets, uint32_t* out,
                                                          const uint32_t* builds, uint32_t* out_b) {
    static_assert(kSelRowsPerBlock == 2048, "two warps per block of rows");
    const int lane = threadIdx.x & 31;
    const int64_t warp = (int64_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5), row0 = warp * 1024;
    if (row0 >= n) return;
    const int64_t word = warp * 32 + lane;
    const uint32_t w = word * 32 < n ? __ldg(bits + word) : 0u;
    uint64_t off = __ldg(block_offsets + (warp >> 1));
    if (warp & 1) off += __reduce_add_sync(0xFFFFFFFFu, __popc(__ldg(bits + word - 32)));  // the block's first half
    uint32_t excl = __popc(w);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, excl, o);
        if (lane >= o) excl += t;
    }
    excl -= __popc(w);
    uint32_t* o = out + off;
    uint32_t* ob = PAIRS ? out_b + off : nullptr;
    const uint32_t lt = (1u << lane) - 1u;
    for (int it0 = 0; it0 < 32; it0 += 8) {
        uint32_t r[8], b[8];  // loaded whether kept or not: eight of each in flight (behind the branch, one)
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const uint32_t i = (uint32_t)row0 + (it0 + j) * 32 + lane;
            r[j] = SEL && i < n ? __ldg(sel + i) : i;
            b[j] = PAIRS && i < n ? __ldg(builds + i) : 0u;
        }
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const uint32_t m = __shfl_sync(0xFFFFFFFFu, w, it0 + j), e = __shfl_sync(0xFFFFFFFFu, excl, it0 + j);
            if ((m >> lane) & 1u) {
                const uint32_t pos = e + __popc(m & lt);
                o[pos] = r[j];
                if (PAIRS) ob[pos] = b[j];
            }
        }
    }
}

// The first sort key of group g (FinalArgs' value of an aggregate that is no string) as sort_prefix orders
// it: the group with the smallest prefix comes first.
__device__ __forceinline__ uint64_t group_prefix(const GroupKey& K, const uint64_t* blk, uint64_t g) {
    uint64_t x;
    bool valid = true;
    if (K.func == ML_AGG_COUNT_STAR) {
        x = blk[0];
    } else if (K.func == ML_AGG_COUNT) {
        x = blk[K.off];
    } else if (K.kind == A_AVG) {
        const uint64_t c = blk[K.off + 1];
        valid = c > 0;
        x = f64_bits(__ddiv_rn(as_f64(blk[K.off]), __ll2double_rn((long long)c)));
    } else {
        valid = (K.vcnt ? K.vcnt[g] : blk[K.cnt_off]) > 0;
        x = blk[K.off];
        if (K.kind == A_MIN_F64 || K.kind == A_MAX_F64) x = f64_bits(f64_unorder(x));
        else if (K.dt == ML_TYPE_INT32 || K.dt == ML_TYPE_DATE) x = (uint64_t)(int64_t)(int32_t)(uint32_t)x;
    }
    if (!valid) return K.nulls_first ? 0ull : ~0ull;
    const uint64_t p = (K.dt == ML_TYPE_FLOAT64 ? (uint64_t)total_key(as_f64(x)) : x) ^ 0x8000000000000000ull;
    return K.asc ? p : ~p;
}

// A bound that at least k groups' prefixes reach, for a top-N over a group table: the k-th smallest of the
// blocks' smallest prefixes (each belongs to another group).  With it only a few times k groups are flagged,
// and the index, the keys, the final values and the top-N after it touch those alone.  1.5M groups, k = 10:
// the kernels after the aggregate 118 -> 66 us, of which this pass over the table takes 13
// and the bound 4.5.
__global__ void __launch_bounds__(1024) k_group_best(const uint64_t* acc, int stride, int64_t n, const uint32_t* member,
                                                         const __grid_constant__ GroupKey K, uint64_t* best) {
    const int64_t step = (int64_t)gridDim.x * 1024;
    uint64_t m = ~0ull;
#pragma unroll 4
    for (int64_t i = (int64_t)blockIdx.x * 1024 + threadIdx.x; i < n; i += step) {
        const uint64_t* blk = acc + i * stride;
        const uint64_t p = group_prefix(K, blk, (uint64_t)i);
        if (blk[0] != 0 && (member == nullptr || member[i] != kNone) && p < m) m = p;
    }
    __shared__ uint64_t red[32];
    auto smallest = [](uint64_t x) {
        for (int o = 16; o; o >>= 1) {
            const uint64_t y = __shfl_xor_sync(0xFFFFFFFFu, x, o);
            x = y < x ? y : x;
        }
        return x;
    };
    m = smallest(m);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = smallest(red[threadIdx.x]);
        if (threadIdx.x == 0) best[blockIdx.x] = m;
    }
}
// best[nb] = the k-th smallest of best[0..nb) (nb <= 256)
__global__ void __launch_bounds__(256) k_group_bound(uint64_t* best, int nb, int k) {
    __shared__ uint64_t v[256];
    const int i = threadIdx.x;
    if (i < nb) v[i] = best[i];
    __syncthreads();
    if (i >= nb) return;
    int place = 0;
    for (int j = 0; j < nb; j++) place += v[j] < v[i] || (v[j] == v[i] && j < i);
    if (place == k - 1) best[nb] = v[i];
}

// Groups with rows (and, with a bound, a prefix that reaches it): bits and block counts.
__global__ void __launch_bounds__(kThreads) k_group_flags(const uint64_t* acc, int stride, int64_t n,
                                                          const uint32_t* member, uint32_t* bits,
                                                          uint32_t* block_counts, const __grid_constant__ GroupKey K,
                                                          const uint64_t* bound) {
    int64_t base = (int64_t)blockIdx.x * kSelRowsPerBlock;
    uint32_t cnt = 0;
    const uint64_t limit = bound ? *bound : 0ull;
#pragma unroll
    for (int it = 0; it < 8; it++) {
        int64_t i = base + it * kThreads + threadIdx.x;
        bool pass = i < n && acc[i * stride] != 0 && (member == nullptr || member[i] != kNone);
        if (bound) pass = pass && group_prefix(K, acc + i * stride, (uint64_t)i) <= limit;
        uint32_t b = __ballot_sync(0xFFFFFFFFu, pass);
        if ((threadIdx.x & 31) == 0 && base + it * kThreads + (threadIdx.x & ~31) < n) bits[(base + it * kThreads + threadIdx.x) >> 5] = b;
        cnt += pass;
    }
    __shared__ uint32_t red[kThreads / 32];
    for (int o = 16; o; o >>= 1) cnt += __shfl_xor_sync(0xFFFFFFFFu, cnt, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = cnt;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int w = 0; w < kThreads / 32; w++) t += red[w];
        block_counts[blockIdx.x] = t;
    }
}

// ---- scan (exclusive, u32 -> u64) ------------------------------------------------------------
constexpr int kScanItems = 4;
constexpr int kScanBlock = 1024 * kScanItems;

__device__ uint64_t block_exclusive_scan(uint64_t v, uint64_t* tmp, uint64_t* total) {
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
        uint64_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) tmp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int nw = blockDim.x >> 5;
        uint64_t t = lane < nw ? tmp[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            uint64_t y = __shfl_up_sync(0xFFFFFFFFu, t, o);
            if (lane >= o) t += y;
        }
        if (lane < nw) tmp[lane] = t;
    }
    __syncthreads();
    uint64_t before = warp ? tmp[warp - 1] : 0;
    if (total) *total = tmp[(blockDim.x >> 5) - 1];
    __syncthreads();
    return before + x - v;
}

__global__ void k_scan_reduce(const uint32_t* in, int64_t n, uint64_t* sums) {
    __shared__ uint64_t tmp[32];
    int64_t base = (int64_t)blockIdx.x * kScanBlock;
    uint64_t s = 0;
    for (int k = 0; k < kScanItems; k++) {
        int64_t i = base + (int64_t)threadIdx.x * kScanItems + k;
        if (i < n) s += in[i];
    }
    uint64_t total;
    block_exclusive_scan(s, tmp, &total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}
__global__ void k_scan_sums(uint64_t* sums, int64_t nb) {  // single block, in place, exclusive
    __shared__ uint64_t tmp[32];
    __shared__ uint64_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int64_t base = 0; base < nb; base += blockDim.x) {
        int64_t i = base + threadIdx.x;
        uint64_t v = i < nb ? sums[i] : 0;
        uint64_t total;
        uint64_t ex = block_exclusive_scan(v, tmp, &total);
        if (i < nb) sums[i] = carry + ex;
        __syncthreads();
        if (threadIdx.x == 0) carry += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) sums[nb] = carry;
}
__global__ void k_scan_apply(const uint32_t* in, int64_t n, const uint64_t* sums, uint64_t* out) {
    __shared__ uint64_t tmp[32];
    int64_t base = (int64_t)blockIdx.x * kScanBlock;
    uint64_t vals[kScanItems];
    uint64_t s = 0;
    for (int k = 0; k < kScanItems; k++) {
        int64_t i = base + (int64_t)threadIdx.x * kScanItems + k;
        vals[k] = i < n ? in[i] : 0;
        s += vals[k];
    }
    uint64_t ex = block_exclusive_scan(s, tmp, nullptr) + sums[blockIdx.x];
    for (int k = 0; k < kScanItems; k++) {
        int64_t i = base + (int64_t)threadIdx.x * kScanItems + k;
        if (i < n) out[i] = ex;
        ex += vals[k];
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) out[n] = ex;
}

// The same in one launch for the counts of chunks and tiles, which are few: a block sums everything before its
// 4,096 counts for itself, which costs less than the launches it saves (48,829 counts 7.9 us, 17.2 in three launches; 9,766 counts 5.6 and
// 17.5).  Past kScanDirect the last blocks would read more than a launch takes.
constexpr int64_t kScanDirect = 1 << 16;
__global__ void __launch_bounds__(1024) k_scan_direct(const uint32_t* in, int n, uint64_t* out) {
    __shared__ uint64_t tmp[32];
    const int t = threadIdx.x, base = (int)blockIdx.x * kScanBlock, i = base + t * kScanItems;
    const bool vec = ((uintptr_t)in & 15) == 0;
    uint64_t before = 0;
    if (vec) {
        const uint4* v = (const uint4*)in;
#pragma unroll 4
        for (int j = t; j < base / 4; j += 1024) {
            const uint4 x = v[j];
            before += (uint64_t)x.x + x.y + x.z + x.w;
        }
    } else {
        for (int j = t; j < base; j += 1024) before += in[j];
    }
    uint32_t mine[kScanItems];
    if (vec && i + kScanItems <= n) {
        const uint4 x = *(const uint4*)(in + i);
        mine[0] = x.x, mine[1] = x.y, mine[2] = x.z, mine[3] = x.w;
    } else {
#pragma unroll
        for (int k = 0; k < kScanItems; k++) mine[k] = i + k < n ? in[i + k] : 0u;
    }
    uint64_t earlier;
    block_exclusive_scan(before, tmp, &earlier);
    uint64_t ex = earlier + block_exclusive_scan((uint64_t)mine[0] + mine[1] + mine[2] + mine[3], tmp, nullptr);
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        if (i + k < n) out[i + k] = ex;
        ex += mine[k];
    }
    if (blockIdx.x == gridDim.x - 1 && t == 1023) out[n] = ex;
}

// ---- projection / hashing ---------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) k_project(const __grid_constant__ PipeArgs P, Prog prog, int out_type,
                                                      void* out, uint32_t* valid) {
    const EvalEnv env = env_of(P);
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    // the loop trip count is uniform per warp (stride is a multiple of 32)
    for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x; i0 < P.n; i0 += stride) {
        int64_t i = i0 + threadIdx.x;
        bool in = i < P.n, ok = false;
        RowCtx x;
        if (in) x.r = sel_row(P, i, in);
        if (in) {
            x.b0 = x.b1 = x.b2 = x.b3 = 0;
            x.head = 0;
            uint64_t v;
            eval_prog(env, prog, x, v, ok);
            switch (out_type) {
                case ML_TYPE_BOOL: ((uint8_t*)out)[i] = (uint8_t)(v & 1); break;
                case ML_TYPE_INT32:
                case ML_TYPE_DATE: ((int32_t*)out)[i] = (int32_t)(uint32_t)v; break;
                case ML_TYPE_UTF8: ((uint32_t*)out)[i] = (uint32_t)v; break;
                default: ((uint64_t*)out)[i] = v; break;
            }
        }
        uint32_t b = __ballot_sync(0xFFFFFFFFu, in && ok);
        if ((threadIdx.x & 31) == 0 && i < P.n) valid[i >> 5] = b;
    }
}

// kernels/hash.rs:16-79: h = SEED; for col: h = combine(h, valid ? hash(col[r]) : NULL_HASH)
__global__ void k_hash_columns(const __grid_constant__ PipeArgs P, int ncols, const uint64_t* const* dict_hash,
                               uint64_t* out) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < P.n; i += stride) {
        bool ok = true;
        const uint32_t r = sel_row(P, i, ok);
        if (!ok) {
            out[i] = 0;
            continue;
        }
        uint64_t h = kSeed;
        for (int c = 0; c < ncols; c++) {
            const DCol& col = P.cols[c];
            uint64_t x = kNullHash;
            if (valid_bit(col.valid, r)) {
                if (col.kind == CK_DICT) {
                    x = dict_hash[c][dict_code(col, r)];
                } else if (col.kind == CK_UTF8) {
                    Str s = col_str(col, r);
                    x = hash_bytes(s.p, s.n);
                } else {
                    uint64_t v = load_value(col, r);
                    if (col.dt == ML_TYPE_FLOAT64 && as_f64(v) == 0.0) v = 0;
                    x = hash_u64(v);
                }
            }
            h = hash_combine(h, x);
        }
        out[i] = h;
    }
}

// ---- join build / probe --------------------------------------------------------------------------
// build_table (join.rs:160-203): one table entry per distinct key; rows with the same
// key are chained through `next`.  NULL keys are not inserted.
__global__ void k_join_insert(const __grid_constant__ PipeArgs P, const __grid_constant__ KeyLayout L, TableView t,
                              uint32_t* next, uint32_t* dup_flag, int64_t n) {
    const EvalEnv env = env_of(P);
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        RowCtx x;
        x.r = (uint32_t)i;
        x.b0 = x.b1 = x.b2 = x.b3 = 0;
        x.head = 0;
        uint64_t w[2];
        uint32_t nm;
        if (!make_key(env, L, x, w, &nm, true)) continue;
        bool inserted;
        uint64_t slot;
        uint32_t r = (uint32_t)i;
        uint32_t p = table_upsert(t, w, 0u, key_hash(w, t.nwords), P.err, [&]() { return r; }, &inserted, &slot);
        if (p == kNone) continue;  // error already flagged (timeout) or table full (never: presized)
        if (!inserted) {
            uint32_t old = atomicExch((uint32_t*)slot_at(t, slot) + 1, r);
            next[r] = old;
            if (*dup_flag == 0) atomicExch(dup_flag, 1u);
        }
    }
}

__global__ void k_probe_count(const __grid_constant__ PipeArgs P, uint32_t* counts) {
    const EvalEnv env = env_of(P);
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < P.n; i += stride) {
        RowCtx x;
        bool ok = true;
        x.r = sel_row(P, i, ok);
        x.b0 = x.b1 = x.b2 = x.b3 = 0;
        x.head = 0;
        uint32_t c = 0;
        if (ok) run_stages(P, env, x, [&](const RowCtx&) { c++; });
        counts[i] = c;
    }
}
__global__ void k_probe_write(const __grid_constant__ PipeArgs P, const uint64_t* offsets, uint32_t* pi, uint32_t* bi) {
    const EvalEnv env = env_of(P);
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < P.n; i += stride) {
        RowCtx x;
        bool ok = true;
        x.r = sel_row(P, i, ok);
        if (!ok) continue;  // counted no pairs
        x.b0 = x.b1 = x.b2 = x.b3 = 0;
        x.head = 0;
        uint64_t o = offsets[i];
        run_stages(P, env, x, [&](const RowCtx& c) {
            pi[o] = c.r;
            bi[o] = c.b0;
            o++;
        });
    }
}

// Range of a one-column integer join key over the valid build rows, as normalized key
// words (int32/date keys zero-extended from 32 bits, int64 keys as is).
__device__ __forceinline__ uint64_t norm_int_key(const void* data, int dt, uint32_t r) {
    if (dt == ML_TYPE_INT64) return (uint64_t)__ldg((const unsigned long long*)data + r);
    return (uint64_t)(uint32_t)__ldg((const int32_t*)data + r);
}
__global__ void k_key_range(const void* data, int dt, const uint64_t* valid, int64_t n, unsigned long long* mm) {
    unsigned long long lo = ~0ull, hi = 0;
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        if (!valid_bit(valid, (uint32_t)i)) continue;
        unsigned long long k = norm_int_key(data, dt, (uint32_t)i);
        lo = k < lo ? k : lo;
        hi = k > hi ? k : hi;
    }
    for (int o = 16; o; o >>= 1) {
        unsigned long long l2 = __shfl_xor_sync(0xFFFFFFFFu, lo, o), h2 = __shfl_xor_sync(0xFFFFFFFFu, hi, o);
        lo = l2 < lo ? l2 : lo;
        hi = h2 > hi ? h2 : hi;
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMin(mm, lo);
        atomicMax(mm + 1, hi);
    }
}
// build_table (join.rs:160-203) over a dense key: the index entry holds the chain head,
// later rows with the same key push the previous head into `next`.
// Membership bitmap of a dense index: bit i of the words = (dense[i] != kNone); one warp per word.
__global__ void k_dense_bits(const uint32_t* dense, uint64_t n, uint32_t* bits) {
    const uint64_t words = (n + 31) / 32;
    const int lane = threadIdx.x & 31;
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
    for (uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < words; w += warps) {
        const uint64_t i = w * 32 + lane;
        const unsigned b = __ballot_sync(0xFFFFFFFFu, i < n && dense[i] != kNone);
        if (lane == 0) bits[w] = b;
    }
}

__global__ void k_dense_insert(const void* data, int dt, const uint64_t* valid, int64_t n, uint64_t dmin, uint64_t drange,
                               uint32_t* dense, uint32_t* next, uint32_t* dup_flag, uint32_t* range_err) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        uint32_t r = (uint32_t)i;
        if (!valid_bit(valid, r)) continue;  // NULL keys never match
        const uint64_t pos = norm_int_key(data, dt, r) - dmin;
        if (pos >= drange) {  // outside the index (a replayed plan's data changed): skipped, reported
            if (range_err) atomicOr(range_err, 1u);
            continue;
        }
        uint32_t old = atomicExch(dense + pos, r);
        if (old != kNone) {
            next[r] = old;
            if (*dup_flag == 0) atomicExch(dup_flag, 1u);
        }
    }
}
__global__ void k_count_dense(const uint32_t* dense, uint64_t n, unsigned long long* out) {
    unsigned long long c = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        c += dense[i] != kNone;
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xFFFFFFFFu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}

__global__ void k_count_slots(TableView t, unsigned long long* out) {
    uint64_t n = t.mask + 1;
    unsigned long long c = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        c += (uint32_t)slot_at(t, i)[0] != 0;
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xFFFFFFFFu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}

// ---- canonical string ids (equal strings -> the smallest-claimed row) ---------------------------
__global__ void k_strid(const uint32_t* off, const uint8_t* bytes, const uint64_t* valid, int64_t n, TableView t,
                        uint32_t* canon, uint32_t* err) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        uint32_t r = (uint32_t)i;
        if (!valid_bit(valid, r)) {
            canon[r] = r;
            continue;
        }
        uint32_t a = off[r], b = off[r + 1];
        uint64_t h = hash_bytes(bytes + a, b - a);
        uint64_t s = h & t.mask;
        uint32_t result = kNone;
        for (uint64_t k = 0; k <= t.mask && result == kNone;) {
            uint64_t* sl = slot_at(t, s);
            uint32_t* st_p = (uint32_t*)sl;
            uint32_t st = load_state(st_p);
            if (st == 0) {
                uint32_t old = atomicCAS(st_p, 0u, 1u);
                if (old == 0) {
                    sl[1] = h;
                    st_p[1] = r;
                    publish_state(st_p, 2);
                    result = r;
                    break;
                }
                st = old;
            }
            if (st == 1) {
                uint32_t spins = 0;
                do {
                    __nanosleep(20);
                    st = load_state(st_p);
                } while (st == 1 && ++spins < kSpinLimit);
                if (st == 1) {
                    atomicOr(err, (uint32_t)DE_TIMEOUT);
                    result = r;
                    break;
                }
            }
            if (sl[1] == h) {
                uint32_t c = st_p[1];
                uint32_t ca = off[c], cb = off[c + 1];
                if (cb - ca == b - a && bytes_eq(bytes + a, bytes + ca, b - a)) {
                    result = c;
                    break;
                }
            }
            s = (s + 1) & t.mask;
            k++;
        }
        canon[r] = result == kNone ? r : result;
    }
}

// ---- gathers ------------------------------------------------------------------------------------
__global__ void k_gather_fixed(const uint8_t* src, int width, const uint32_t* idx, int64_t k, uint8_t* dst) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < k; i += stride) {
        uint64_t r = idx[i];
        switch (width) {
            case 1: dst[i] = src[r]; break;
            case 4: ((uint32_t*)dst)[i] = ((const uint32_t*)src)[r]; break;
            case 8: ((uint64_t*)dst)[i] = ((const uint64_t*)src)[r]; break;
            default: {  // rows of width / 8 words (a group's accumulator block)
                const int w = width / 8;
                const uint64_t* s8 = (const uint64_t*)src + r * w;
                uint64_t* d8 = (uint64_t*)dst + i * w;
                for (int j = 0; j < w; j++) d8[j] = s8[j];
                break;
            }
        }
    }
}
__global__ void k_gather_valid(const uint64_t* src, const uint32_t* idx, int64_t k, uint32_t* dst) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x; i0 < k; i0 += stride) {
        int64_t i = i0 + threadIdx.x;
        bool v = false;
        if (i < k) v = valid_bit(src, idx[i]);
        uint32_t b = __ballot_sync(0xFFFFFFFFu, v);
        if ((threadIdx.x & 31) == 0 && i < k) dst[i >> 5] = b;
    }
}
// The rows of several columns in one launch: kGatherRows row ids per thread are read once, and a column's
// loads for all of them are in flight together.  2M rows of an 8-byte column with validity: 27.5 us in two
// launches with a row id and then its value per step, 23 us alone so, 20.5 with three others.
constexpr int kGatherRows = 4;
template <class T>
__device__ __forceinline__ void gather_values(const GatherCol& c, const uint32_t (&r)[kGatherRows], int64_t i0, int64_t k) {
    T v[kGatherRows];
#pragma unroll
    for (int j = 0; j < kGatherRows; j++) v[j] = ((const T*)c.src)[r[j]];
#pragma unroll
    for (int j = 0; j < kGatherRows; j++) {
        const int64_t i = i0 + j * kThreads;
        if (i < k) __stcs((T*)c.dst + i, v[j]);
    }
}
__global__ void __launch_bounds__(kThreads) k_gather_cols(const __grid_constant__ GatherCols G, const uint32_t* idx, int64_t k) {
    const int64_t step = (int64_t)gridDim.x * kThreads * kGatherRows;
    for (int64_t base = (int64_t)blockIdx.x * kThreads * kGatherRows; base < k; base += step) {
        const int64_t i0 = base + threadIdx.x;
        uint32_t r[kGatherRows];
#pragma unroll
        for (int j = 0; j < kGatherRows; j++) {
            const int64_t i = i0 + j * kThreads;
            r[j] = ld_stream_u32(idx + (i < k ? i : k - 1));
        }
        for (int n = 0; n < G.n; n++) {
            const GatherCol& c = G.c[n];
            if (c.width == 8) gather_values<uint64_t>(c, r, i0, k);
            else if (c.width == 4) gather_values<uint32_t>(c, r, i0, k);
            else gather_values<uint8_t>(c, r, i0, k);
            if (!c.dst_valid) continue;
            bool v[kGatherRows];
#pragma unroll
            for (int j = 0; j < kGatherRows; j++) v[j] = valid_bit(c.src_valid, r[j]);
#pragma unroll
            for (int j = 0; j < kGatherRows; j++) {
                const int64_t i = i0 + j * kThreads;
                const uint32_t bits = __ballot_sync(0xFFFFFFFFu, i < k && v[j]);
                if ((threadIdx.x & 31) == 0 && (i >> 5) < 2 * ((k + 63) / 64)) c.dst_valid[i >> 5] = bits;
            }
        }
    }
}
__global__ void k_utf8_lengths(const uint32_t* off, const uint32_t* idx, int64_t k, uint32_t* len) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < k; i += stride) {
        uint32_t r = idx ? idx[i] : (uint32_t)i;
        len[i] = off[r + 1] - off[r];
    }
}
__global__ void k_utf8_copy(const uint32_t* off, const uint8_t* bytes, const uint32_t* idx, int64_t k,
                            const uint64_t* dst_off, uint8_t* dst) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < k; i += stride) {
        uint32_t r = idx ? idx[i] : (uint32_t)i;
        uint32_t a = off[r], b = off[r + 1];
        uint8_t* d = dst + dst_off[i];
        for (uint32_t j = a; j < b; j++) d[j - a] = bytes[j];
    }
}
__global__ void k_u64_to_u32(const uint64_t* in, uint32_t* out, int64_t n) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) out[i] = (uint32_t)in[i];
}

__global__ void k_offsets_rebase(const uint32_t* src, int64_t n, uint32_t base, uint32_t* dst) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    uint32_t first = src[0];
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += stride) dst[i] = src[i] - first + base;
}
__global__ void k_copy_bits(const uint64_t* src, int64_t n, uint64_t* dst, int64_t dst_off) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        bool v = src == nullptr || ((src[i >> 6] >> (i & 63)) & 1ull);
        if (v) {
            int64_t o = dst_off + i;
            atomicOr((unsigned long long*)dst + (o >> 6), 1ull << (o & 63));
        }
    }
}

// ---- top-N -------------------------------------------------------------------------------------------
// compare_rows (sort.rs:43-82): per key, NULLs first/last, f64 by total order, asc/desc.
// Not inlined: the sorting networks call it only when two prefixes tie, and inlining it into
// every compare-exchange multiplies their code size.
__device__ __noinline__ int cmp_rows(const SortDev& S, uint32_t a, uint32_t b) {
    if (a == kNone || b == kNone) return (a == kNone) - (b == kNone);  // padding sorts last
    for (int k = 0; k < S.nkeys; k++) {
        const DCol& c = S.cols[k];
        bool va = valid_bit(c.valid, a), vb = valid_bit(c.valid, b);
        int o = 0;
        if (!va && !vb) o = 0;
        else if (!va) return S.nulls_first[k] ? -1 : 1;
        else if (!vb) return S.nulls_first[k] ? 1 : -1;
        else {
            if (c.kind == CK_UTF8) {
                o = str_cmp(col_str(c, a), col_str(c, b));
            } else {
                uint64_t x = load_value(c, a), y = load_value(c, b);
                switch (c.dt) {
                    case ML_TYPE_FLOAT64: {
                        int64_t p = total_key(as_f64(x)), q = total_key(as_f64(y));
                        o = p < q ? -1 : (p > q);
                        break;
                    }
                    case ML_TYPE_BOOL: o = (x < y) ? -1 : (x > y); break;
                    default: o = ((int64_t)x < (int64_t)y) ? -1 : ((int64_t)x > (int64_t)y); break;
                }
            }
            if (!S.asc[k]) o = -o;
        }
        if (o) return o;
    }
    return 0;
}

// Order-preserving 64-bit prefix of the first sort key: prefix(a) < prefix(b) implies
// cmp_rows(a, b) < 0, so rows are compared through shared memory and cmp_rows runs
// only on equal prefixes (ties, NULLs and padding).
__device__ __forceinline__ uint64_t sort_prefix(const SortDev& S, uint32_t r) {
    if (r == kNone) return ~0ull;
    const DCol& c = S.cols[0];
    if (!valid_bit(c.valid, r)) return S.nulls_first[0] ? 0ull : ~0ull;
    uint64_t p;
    if (c.kind == CK_UTF8) {
        Str s = col_str(c, r);
        p = 0;
        uint32_t m = s.n < 8 ? s.n : 8;
        for (uint32_t j = 0; j < m; j++) p |= (uint64_t)__ldg(s.p + j) << (56 - 8 * j);
    } else {
        uint64_t x = load_value(c, r);
        if (c.dt == ML_TYPE_FLOAT64) p = (uint64_t)total_key(as_f64(x)) ^ 0x8000000000000000ull;
        else if (c.dt == ML_TYPE_BOOL) p = x;
        else p = x ^ 0x8000000000000000ull;
    }
    return S.asc[0] ? p : ~p;
}

// The block sorts `n` rows (a power of two; prefixes and row ids in shared memory), ascending by
// compare_rows, equal keys in input order; a padding row (kNone) sorts last.
__device__ void bitonic_rows(const SortDev& S, uint64_t* pre, uint32_t* idx, int n) {
    for (int size = 2; size <= n; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int t = threadIdx.x; t < n / 2; t += blockDim.x) {
                int lo = 2 * t - (t & (stride - 1));
                int hi = lo + stride;
                bool up = (lo & size) == 0;
                uint64_t pa = pre[lo], pb = pre[hi];
                int c = pa < pb ? -1 : (pa > pb ? 1 : cmp_rows(S, idx[lo], idx[hi]));
                if (c == 0) c = idx[lo] < idx[hi] ? -1 : (idx[lo] > idx[hi]);  // equal keys: input order
                if ((c > 0) == up && c != 0) {
                    uint32_t a = idx[lo];
                    idx[lo] = idx[hi];
                    idx[hi] = a;
                    pre[lo] = pb;
                    pre[hi] = pa;
                }
            }
            __syncthreads();
        }
    }
}

// One block sorts kTopNChunk rows (bitonic, ascending by compare_rows) and writes the
// first k.  Keys are compared by their shared-memory prefix first.
__global__ void __launch_bounds__(1024) k_topn_chunk(const __grid_constant__ SortDev S, const uint32_t* in, int64_t n,
                                                    int k, uint32_t* out) {
    __shared__ uint64_t pre[kTopNChunk];
    __shared__ uint32_t idx[kTopNChunk];
    int64_t base = (int64_t)blockIdx.x * kTopNChunk;
    for (int j = threadIdx.x; j < kTopNChunk; j += blockDim.x) {
        int64_t i = base + j;
        uint32_t r = i < n ? (in ? in[i] : (uint32_t)i) : kNone;
        idx[j] = r;
        pre[j] = sort_prefix(S, r);
    }
    __syncthreads();
    bitonic_rows(S, pre, idx, kTopNChunk);
    for (int j = threadIdx.x; j < k; j += blockDim.x) out[(int64_t)blockIdx.x * k + j] = idx[j];
}

// ---- top-N for small limits (k <= 32): one sorted list per warp ------------------------------
// Each lane holds one entry of the warp's current best 32 (ascending); a batch of 32 new
// rows is skipped unless one of them beats the k-th entry, else it is sorted with a
// shuffle bitonic network and merged in.  The CTA then merges its warps' lists.
struct TopEntry {
    uint64_t p;  // sort_prefix
    uint32_t r;  // row (kNone = padding)
};
// Rows with equal keys keep their input order (the row id breaks the tie), as in a stable sort.
__device__ __forceinline__ bool entry_less(const SortDev& S, TopEntry a, TopEntry b) {
    if (a.p != b.p) return a.p < b.p;
    const int c = cmp_rows(S, a.r, b.r);
    return c ? c < 0 : a.r < b.r;
}
__device__ __forceinline__ TopEntry shfl_entry(TopEntry e, int src) {
    return TopEntry{__shfl_sync(0xFFFFFFFFu, e.p, src), __shfl_sync(0xFFFFFFFFu, e.r, src)};
}
// Compare-exchange with the lane `lane ^ j`; the lower lane keeps the smaller entry when
// `ascending`.  Both lanes evaluate entry_less(upper, lower), so ties resolve consistently.
__device__ __forceinline__ TopEntry cmp_exchange(const SortDev& S, TopEntry e, int lane, int j, bool ascending) {
    TopEntry o = shfl_entry(e, lane ^ j);
    bool lower = (lane & j) == 0;
    TopEntry lo = lower ? e : o, hi = lower ? o : e;
    bool swap = entry_less(S, hi, lo);
    bool keep_min = lower == ascending;
    if (keep_min) return swap ? hi : lo;
    return swap ? lo : hi;
}
// The networks' loops stay rolled: these kernels run them a few times per warp from a cold
// instruction cache, where fetching unrolled copies costs more than the loop overhead.
__device__ __forceinline__ TopEntry warp_sort32(const SortDev& S, TopEntry e, int lane) {
#pragma unroll 1
    for (int k = 2; k <= 32; k <<= 1)
#pragma unroll 1
        for (int j = k >> 1; j > 0; j >>= 1) e = cmp_exchange(S, e, lane, j, (lane & k) == 0);
    return e;
}
// Merge sorted `n` into sorted `l`: keep the 32 smallest of both, sorted ascending.
__device__ __forceinline__ TopEntry warp_merge32(const SortDev& S, TopEntry l, TopEntry n, int lane) {
    TopEntry rev = shfl_entry(n, 31 - lane);
    TopEntry e = entry_less(S, rev, l) ? rev : l;  // bitonic: the 32 smallest of the union
#pragma unroll 1
    for (int j = 16; j > 0; j >>= 1) e = cmp_exchange(S, e, lane, j, true);
    return e;
}

// The qn queued entries into the warp's sorted list: a few are inserted one at a time (a ballot
// for the position, a shuffle to move the larger entries up one lane), more are sorted in groups
// of 32 and merged.  Queued rows are never in the list already.  One out-of-line copy serves
// every call site (the whole warp calls it).
__device__ __noinline__ TopEntry warp_absorb(const SortDev& S, TopEntry best, const TopEntry* queue, int qn, int lane) {
    if (qn <= 8) {
#pragma unroll 1
        for (int i = 0; i < qn; i++) {
            const TopEntry c = queue[i];
            const int pos = __popc(__ballot_sync(0xFFFFFFFFu, entry_less(S, best, c)));
            const TopEntry up{__shfl_up_sync(0xFFFFFFFFu, best.p, 1), __shfl_up_sync(0xFFFFFFFFu, best.r, 1)};
            if (lane >= pos) best = lane == pos ? c : up;
        }
    } else {
#pragma unroll 1
        for (int i = 0; i < qn; i += 32) {
            const TopEntry e = i + lane < qn ? queue[i + lane] : TopEntry{~0ull, kNone};
            best = warp_merge32(S, best, warp_sort32(S, e, lane), lane);
        }
    }
    return best;
}

// Rows that beat the warp's current k-th entry are queued in shared memory; a full queue
// (32 entries) is sorted and merged into the list, so the sort runs once per 32
// candidates, not once per 32 rows (about k * ln(rows / k) candidates reach a warp).
// One warp's best k of n entries (batches of 32 from batch index `batch` on, every `batches`
// batches), as a sorted list across the lanes; get(i) yields entry i.
template <class Get>
__device__ TopEntry warp_topk(const SortDev& S, int64_t n, int k, int64_t batch, int64_t batches, TopEntry* queue,
                              int lane, Get get) {
    TopEntry best{~0ull, kNone};
    TopEntry kth = best;
    int qn = 0;  // entries in the warp's queue (warp-uniform)
    auto flush = [&]() {
        __syncwarp();
        best = warp_absorb(S, best, queue, qn, lane);
        __syncwarp();
        kth = shfl_entry(best, k - 1);
        qn = 0;
    };
    for (int64_t base = batch * 32; base < n; base += batches * 32) {
        int64_t i = base + lane;
        TopEntry e = i < n ? get(i) : TopEntry{~0ull, kNone};
        bool take = e.r != kNone && entry_less(S, e, kth);
        unsigned m = __ballot_sync(0xFFFFFFFFu, take);
        if (!m) continue;
        if (qn + __popc(m) > 32) {
            flush();
            take = take && entry_less(S, e, kth);
            m = __ballot_sync(0xFFFFFFFFu, take);
        }
        if (take) queue[qn + __popc(m & ((1u << lane) - 1))] = e;
        qn += __popc(m);
        __syncwarp();
    }
    if (qn) flush();
    return best;
}

// sort_prefix of a fixed-width first key of type DT from its loaded value (load_value's form):
// `flip` is 0 for ascending keys and ~0 for descending ones, `nullp` the prefix of a NULL.
template <int DT>
__device__ __forceinline__ uint64_t fixed_prefix(uint64_t x, bool valid, uint64_t flip, uint64_t nullp) {
    uint64_t p;
    if (DT == ML_TYPE_FLOAT64) p = (uint64_t)total_key(as_f64(x)) ^ 0x8000000000000000ull;
    else if (DT == ML_TYPE_BOOL) p = x;
    else p = x ^ 0x8000000000000000ull;
    return valid ? p ^ flip : nullp;
}

// Four consecutive values of the key column (registers, not an array: no stack traffic).
struct Quad {
    uint64_t v0, v1, v2, v3;
};

// Four consecutive rows of the key column from r0 (one or two 16-byte loads when the column is
// aligned and the four rows exist; rows past n read as 0 and are never queued).
template <int DT>
__device__ __forceinline__ Quad load_quad(const DCol& c, bool vec, uint32_t n32, uint32_t r0) {
    Quad q{0ull, 0ull, 0ull, 0ull};
    if (vec && (uint64_t)r0 + 4u <= (uint64_t)n32) {
        if (DT == ML_TYPE_FLOAT64 || DT == ML_TYPE_INT64) {
            uint64_t t[2], u[2];
            ld_stream_v2_u64((const unsigned long long*)c.data + r0, t);
            ld_stream_v2_u64((const unsigned long long*)c.data + r0 + 2, u);
            q = Quad{t[0], t[1], u[0], u[1]};
        } else if (DT == ML_TYPE_BOOL) {
            const uint32_t w = ld_stream_u32((const uint8_t*)c.data + r0);
            q = Quad{w & 0xFFu, (w >> 8) & 0xFFu, (w >> 16) & 0xFFu, w >> 24};
        } else {
            uint32_t w[4];
            ld_stream_v4_u32((const uint32_t*)c.data + r0, w);
            q = Quad{(uint64_t)(int64_t)(int32_t)w[0], (uint64_t)(int64_t)(int32_t)w[1],
                     (uint64_t)(int64_t)(int32_t)w[2], (uint64_t)(int64_t)(int32_t)w[3]};
        }
    } else {
        const uint64_t r = r0;
        if (r < n32) q.v0 = load_value(c, r0);
        if (r + 1u < n32) q.v1 = load_value(c, r0 + 1u);
        if (r + 2u < n32) q.v2 = load_value(c, r0 + 2u);
        if (r + 3u < n32) q.v3 = load_value(c, r0 + 3u);
    }
    return q;
}

// Queues the lane's four rows from r0 that can still be in the top k: prefix at or below
// `bound` (the warp's k-th entry and the launch-wide threshold) and ahead of the k-th entry.
// The queue holds (at most) 31 entries carried over plus the 128 of a half-step.
template <int DT>
__device__ __forceinline__ void queue_quad(const SortDev& S, const DCol& c, const Quad& q, uint32_t r0, uint32_t n32,
                                           uint64_t flip, uint64_t nullp, uint64_t bound, TopEntry kth,
                                           TopEntry* queue, int lane, int& qn) {
    const uint32_t rem = r0 < n32 ? n32 - r0 : 0u;  // rows of the four that exist
    uint32_t vb = 0xFu;
    if (c.valid && rem) vb = (uint32_t)(__ldg(c.valid + (r0 >> 6)) >> (r0 & 63u));
    const uint64_t p0 = fixed_prefix<DT>(q.v0, vb & 1u, flip, nullp);
    const uint64_t p1 = fixed_prefix<DT>(q.v1, vb & 2u, flip, nullp);
    const uint64_t p2 = fixed_prefix<DT>(q.v2, vb & 4u, flip, nullp);
    const uint64_t p3 = fixed_prefix<DT>(q.v3, vb & 8u, flip, nullp);
    const bool any = (rem > 0 && p0 <= bound) || (rem > 1 && p1 <= bound) || (rem > 2 && p2 <= bound) ||
                     (rem > 3 && p3 <= bound);
    if (!__any_sync(0xFFFFFFFFu, any)) return;
    const unsigned lt = (1u << lane) - 1u;
#pragma unroll
    for (uint32_t j = 0; j < 4; j++) {
        const uint64_t p = j == 0 ? p0 : j == 1 ? p1 : j == 2 ? p2 : p3;
        const TopEntry e{p, r0 + j};
        const bool take = rem > j && p <= bound && entry_less(S, e, kth);
        const unsigned m = __ballot_sync(0xFFFFFFFFu, take);
        if (take) queue[qn + __popc(m & lt)] = e;
        qn += __popc(m);
    }
}

// warp_topk over the source rows when the first sort key is a fixed-width column of type DT:
// 256-row steps, each lane reading 4 consecutive rows of each 128-row half (one or two 16-byte
// loads when the column is aligned); the next step's values and the shared threshold are loaded
// before the current step is compared, so a warp keeps 4 KB in flight.  Each half queues the
// rows that beat the k-th entry (usually none: it costs its loads and compares), and a queue of
// 32 or more goes into the list (warp_absorb, one out-of-line copy; the warp's state stays in
// registers).
// `shared_thr` (optional, starts at 0) holds ~T for the smallest full-list k-th prefix T any warp
// of the launch has published: k rows have prefixes <= T, so a
// row with a larger prefix cannot be in the top k and no warp queues it.
constexpr int kTopNQueue = 160;  // 31 carried over + the 128 rows of a half-step, rounded up
template <int DT>
__device__ TopEntry warp_topk_fixed(const SortDev& S, int64_t n, int k, int64_t chunk, int64_t chunks, TopEntry* queue,
                                    int lane, unsigned long long* shared_thr) {
    const DCol& c = S.cols[0];
    const bool vec = ((uintptr_t)c.data & 15) == 0;
    const uint64_t flip = S.asc[0] ? 0ull : ~0ull, nullp = S.nulls_first[0] ? 0ull : ~0ull;
    const uint32_t n32 = (uint32_t)n;  // row ids are 32-bit
    TopEntry best{~0ull, kNone};
    TopEntry kth = best;
    int qn = 0;  // entries in the warp's queue (warp-uniform)
    uint64_t thr = ~0ull;
    const Quad zero{0ull, 0ull, 0ull, 0ull};
    int64_t base = chunk * 256;
    Quad qa = zero, qb = zero;
    uint64_t pc = 0;
    auto absorb = [&]() {  // the queue into the list; publish a tighter k-th
        __syncwarp();
        best = warp_absorb(S, best, queue, qn, lane);
        __syncwarp();
        kth = shfl_entry(best, k - 1);
        qn = 0;
        if (shared_thr && kth.r != kNone && kth.p < thr) {
            thr = kth.p;
            if (lane == 0) atomicMax(shared_thr, ~kth.p);
        }
    };
    if (base < n) {
        qa = load_quad<DT>(c, vec, n32, (uint32_t)base + (uint32_t)lane * 4u);
        qb = load_quad<DT>(c, vec, n32, (uint32_t)base + 128u + (uint32_t)lane * 4u);
    }
    for (;;) {
        const bool more = base < n;
        if (more) {
            const int64_t next = base + chunks * 256;
            Quad na = zero, nb = zero;
            uint64_t pn = pc;
            if (next < n) {
                na = load_quad<DT>(c, vec, n32, (uint32_t)next + (uint32_t)lane * 4u);
                nb = load_quad<DT>(c, vec, n32, (uint32_t)next + 128u + (uint32_t)lane * 4u);
                if (shared_thr) pn = __ldcg(shared_thr);
            }
            thr = ~pc < thr ? ~pc : thr;
            queue_quad<DT>(S, c, qa, (uint32_t)base + (uint32_t)lane * 4u, n32, flip, nullp,
                           kth.p < thr ? kth.p : thr, kth, queue, lane, qn);
            if (qn >= 32) absorb();
            queue_quad<DT>(S, c, qb, (uint32_t)base + 128u + (uint32_t)lane * 4u, n32, flip, nullp,
                           kth.p < thr ? kth.p : thr, kth, queue, lane, qn);
            qa = na;
            qb = nb;
            pc = pn;
            base = next;
        }
        if (qn >= 32 || (!more && qn)) absorb();
        if (!more) break;
    }
    return best;
}

// The block puts up to blockDim.x rows in order: out[place] = row for the first k places.
__device__ __forceinline__ void place_rows(const SortDev& S, uint64_t* pre, int n, int k, uint32_t* out) {
    const int i = threadIdx.x;
    if (i < n) pre[i] = sort_prefix(S, (uint32_t)i);
    __syncthreads();
    if (i >= n) return;
    const uint64_t p = pre[i];
    int place = 0;
#pragma unroll 1
    for (int j = 0; j < n; j++) {
        const uint64_t q = pre[j];
        int before = q < p ? 1 : 0;
        if (q == p && j != i) {  // equal keys keep their input order
            const int c = cmp_rows(S, (uint32_t)j, (uint32_t)i);
            before = c < 0 || (c == 0 && j < i);
        }
        place += before;
    }
    if (place < k) out[place] = (uint32_t)i;
}

// Each CTA writes its best k rows to out[block * k ..].  With `final_out`, CTAs also write
// their (prefix, row) entries to `cand`, and the last CTA to finish (the counter `done` starts
// at zero) merges all CTAs' entries into final_out[0 .. k): the whole top-k in one launch.
// DT: the first sort key's type when it is a fixed-width column (warp_topk_fixed), -1 otherwise.
template <int DT>
__global__ void __launch_bounds__(256, 2) k_topn_warp(const __grid_constant__ SortDev S, int64_t n, int k, uint32_t* out,
                                                   TopEntry* cand, unsigned int* done, uint32_t* final_out,
                                                   const uint64_t* n_dev) {
    if (n_dev) n = min(n, (int64_t)__ldcg(n_dev));  // a replayed plan's row count
    if (n_dev && n <= 256) {
        // few rows after all (groups behind a bound): one CTA places each row by the rows before it.  The
        // lists' merges, a chain of 14 sorts, took 27 us for 20 rows; this takes 3.9.
        if (blockIdx.x) return;
        __shared__ uint64_t pre[256];
        place_rows(S, pre, (int)n, k, final_out ? final_out : out);
        if ((int)threadIdx.x >= n && (int)threadIdx.x < k) (final_out ? final_out : out)[threadIdx.x] = kNone;
        return;
    }
    __shared__ TopEntry lists[8][32];
    __shared__ TopEntry queue[8][kTopNQueue];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    TopEntry best;
    // `done` points at 16 zeroed bytes: the finished-CTA counter, then the shared threshold
    unsigned long long* thr = done ? reinterpret_cast<unsigned long long*>(done + 2) : nullptr;
    if (DT >= 0)
        best = warp_topk_fixed<DT < 0 ? 0 : DT>(S, n, k, (int64_t)blockIdx.x * 8 + warp, (int64_t)gridDim.x * 8,
                                                  queue[warp], lane, thr);
    else
        best = warp_topk(S, n, k, (int64_t)blockIdx.x * 8 + warp, (int64_t)gridDim.x * 8, queue[warp], lane,
                         [&](int64_t i) { return TopEntry{sort_prefix(S, (uint32_t)i), (uint32_t)i}; });
    lists[warp][lane] = best;
    __syncthreads();
    if (warp == 0) {
#pragma unroll 1
        for (int w = 1; w < 8; w++) best = warp_merge32(S, best, lists[w][lane], lane);
        if (lane < k) {
            out[(int64_t)blockIdx.x * k + lane] = best.r;
            if (final_out) cand[(int64_t)blockIdx.x * k + lane] = best;
        }
    }
    if (!final_out) return;
    __threadfence();  // this CTA's entries are visible before it counts itself done
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    const int64_t m = (int64_t)gridDim.x * k;
    // k rows of some warp's full list have prefixes <= the published threshold, so a candidate
    // above it cannot be in the top k: most CTAs' lists drop out here without a sort.  Each warp
    // loads four batches of 32 candidates at once, queues those that can be in the top k, and
    // takes its queue into its list from one place once it holds 32 or the candidates are done.
    const uint64_t bound = thr ? ~__ldcg(thr) : ~0ull;
    {
        TopEntry* qw = queue[warp];
        best = TopEntry{~0ull, kNone};
        TopEntry kth = best;
        int qn = 0;
        for (int64_t b0 = (int64_t)warp * 32;; b0 += 8 * 32 * 4) {
            const bool more = b0 < m;
            if (more) {
                TopEntry e[4];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int64_t i = b0 + j * 256 + lane;
                    e[j] = TopEntry{~0ull, kNone};
                    if (i < m) e[j] = TopEntry{__ldcg((const unsigned long long*)&cand[i].p), __ldcg(&cand[i].r)};
                }
                const unsigned lt = (1u << lane) - 1u;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const bool take = e[j].r != kNone && e[j].p <= bound && entry_less(S, e[j], kth);
                    const unsigned mk = __ballot_sync(0xFFFFFFFFu, take);
                    if (take) qw[qn + __popc(mk & lt)] = e[j];
                    qn += __popc(mk);
                }
            }
            if (qn >= 32 || (!more && qn)) {
                __syncwarp();
                best = warp_absorb(S, best, qw, qn, lane);
                __syncwarp();
                kth = shfl_entry(best, k - 1);
                qn = 0;
            }
            if (!more) break;
        }
    }
    lists[warp][lane] = best;
    __syncthreads();
    if (warp == 0) {
#pragma unroll 1
        for (int w = 1; w < 8; w++) best = warp_merge32(S, best, lists[w][lane], lane);
        if (lane < k) final_out[lane] = best.r;
    }
}


// ---- small results -------------------------------------------------------------------------------
// The order of up to kTopNTiny rows in one step: a row's place is the number of rows before it.  (The
// per-warp lists and their merges took 22 us for six groups ordered by two strings, 5 us so.)
__global__ void __launch_bounds__(kTopNTiny) k_topn_tiny(const __grid_constant__ SortDev S, int n, int k, uint32_t* out) {
    __shared__ uint64_t pre[kTopNTiny];
    place_rows(S, pre, n, k, out);
}

// Rows idx[0..k) of every column of a batch, a block per column (k <= 1,024): values, validity words and,
// for strings, offsets and bytes.  info[c]: a string column's bytes, kNone when they exceed its buffer.
__global__ void __launch_bounds__(1024) k_gather_small(const __grid_constant__ SmallCols G, const uint32_t* idx, int k) {
    __shared__ uint64_t tmp[32];
    const SmallCol& c = G.c[blockIdx.x];
    const int i = threadIdx.x;
    const uint32_t r = i < k ? idx[i] : 0u;
    if (c.dst_valid) {
        const uint32_t bits = __ballot_sync(0xFFFFFFFFu, i < k && valid_bit(c.src_valid, r));
        if ((i & 31) == 0 && (i >> 5) < 2 * ((k + 63) / 64)) c.dst_valid[i >> 5] = bits;  // whole 64-bit words
    }
    if (c.width) {
        if (i < k) {
            if (c.width == 8) ((uint64_t*)c.dst)[i] = ((const uint64_t*)c.src)[r];
            else if (c.width == 4) ((uint32_t*)c.dst)[i] = ((const uint32_t*)c.src)[r];
            else ((uint8_t*)c.dst)[i] = ((const uint8_t*)c.src)[r];
        }
        return;
    }
    uint32_t a = 0, len = 0;
    if (i < k) {
        a = c.src_off[r];
        len = c.src_off[r + 1] - a;
    }
    uint64_t total;
    const uint64_t at = block_exclusive_scan(len, tmp, &total);
    if (i < k) c.dst_off[i] = (uint32_t)at;
    if (i == 0) {
        c.dst_off[k] = (uint32_t)total;
        G.info[blockIdx.x] = total <= c.cap ? (uint32_t)total : kNone;
    }
    if (total <= c.cap)
        for (uint32_t j = 0; j < len; j++) ((uint8_t*)c.dst)[at + j] = ((const uint8_t*)c.src)[a + j];
}

// Pieces of memory into one buffer, a block per piece (a small batch read back with one copy).
__global__ void __launch_bounds__(256) k_pack(const __grid_constant__ PackPieces P, uint8_t* dst) {
    const auto& x = P.p[blockIdx.x];
    for (uint32_t i = threadIdx.x; i < x.bytes; i += 256) dst[x.at + i] = ((const uint8_t*)x.src)[i];
}

// ---- top-N by selection: limits up to kMaxTopN over a fixed-width first key ------------------------
// k_topn_sample takes the r-th smallest row of a sample, r chosen so that more than k rows lie at or below
// it all but surely; k_topn_take streams the key column once and lists the rows at or below; k_topn_finish
// finds the k-th of those exactly, keeps the rows up to it and sorts them.  The host checks that the list
// held at least k rows and not more than it has room for (else every row goes through k_topn_chunk /
// k_topn_warp).
// Why: the chunk sort orders all rows in shared memory, 2.0 ms for 20M rows and k = 100; the selection
// reads the column at 5.1 to 5.9 TB/s (32 us), before it 13 us for the bound, after it 11 us for the
// finish (a bound from 16,384 samples, eight times the rows in the list and a sort of them: 17 and 19 us).
//
// Rows whose first keys are equal (few distinct values, NULLs in front) are told apart as the whole sort
// does, word by word (TopNLevel), only as far as it takes to leave few of them: in the bound, in the list
// and in the k-th row alike.  A bound on the first key alone listed every tied row and gave up: 60M rows of
// four values, LIMIT 10, took 2.5 ms a call (the per-warp lists alone 1.3), now 0.31; LIMIT 100 22.6 and 0.35 ms.

// f(i, get(i)) for the block's values with in(i), eight of a thread's in flight together (one after the
// other, a pass over 30,000 listed rows took 12 us).  A value belongs to the thread i % blockDim.x.
template <class Get, class In, class F>
__device__ __forceinline__ void block_values(Get get, In in, uint32_t n, F f) {
    for (uint32_t i0 = threadIdx.x; i0 < n; i0 += 8 * blockDim.x) {
        uint64_t v[8];
        bool a[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const uint32_t i = i0 + j * blockDim.x;
            a[j] = i < n && in(i);
            v[j] = a[j] ? get(i) : 0ull;
        }
#pragma unroll
        for (int j = 0; j < 8; j++)
            if (a[j]) f(i0 + j * blockDim.x, v[j]);
    }
}
// The block finds the r-th smallest (r >= 1) of the `count` values get(i) with in(i), i < n, `ref` one of
// them: by 8-bit digits from the highest bit in which the values differ, counted in shared memory.  Returns
// an upper bound of it that no further value lies below: the values <= `bound` are the `below` + `last`
// smallest.  It stops early where at most `slack` more than r values are taken, else the bound is the r-th
// itself, `below` values lie below it and `last` are equal to it.
struct BlockPick {
    uint64_t bound;
    uint32_t below, last;
};
template <class Get, class In>
__device__ BlockPick block_select(Get get, In in, uint32_t n, uint32_t count, uint64_t ref, uint32_t r, uint32_t slack) {
    __shared__ uint32_t hist[256];
    __shared__ unsigned long long diff_s;
    __shared__ uint32_t digit_s, below_s, in_s;
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    uint64_t diff = 0;
    __syncthreads();
    if (tid == 0) diff_s = 0;
    __syncthreads();
    block_values(get, in, n, [&](uint32_t, uint64_t v) { diff |= v ^ ref; });
    const uint32_t dlo = __reduce_or_sync(0xFFFFFFFFu, (uint32_t)diff), dhi = __reduce_or_sync(0xFFFFFFFFu, (uint32_t)(diff >> 32));
    if (lane == 0) atomicOr(&diff_s, ((unsigned long long)dhi << 32) | dlo);
    __syncthreads();
    diff = diff_s;
    if (!diff) return BlockPick{ref, 0, count};
    int top = 64 - __clzll((long long)diff);           // bits [0, top) are undecided
    uint64_t want = top < 64 ? ref >> top << top : 0;  // the decided bits
    uint32_t before = 0;                               // values below the range of `want`
    for (;;) {
        const int low = top > 8 ? top - 8 : 0;
        for (uint32_t i = tid; i < 256; i += blockDim.x) hist[i] = 0;
        __syncthreads();
        block_values(get, in, n, [&](uint32_t, uint64_t x) {
            const uint64_t v = x ^ want;
            if (top == 64 || (v >> top) == 0) atomicAdd(&hist[(v >> low) & ((1u << (top - low)) - 1u)], 1u);
        });
        __syncthreads();
        if (tid < 32) {  // the digit in which the r-th lies: eight bins per lane
            uint32_t c[8], sum = 0;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                c[j] = hist[lane * 8 + j];
                sum += c[j];
            }
            uint32_t incl = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if ((int)lane >= o) incl += t;
            }
            uint32_t at = before + incl - sum;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                if (at < r && r <= at + c[j]) {
                    digit_s = lane * 8 + j;
                    below_s = at;
                    in_s = c[j];
                }
                at += c[j];
            }
        }
        __syncthreads();
        const uint32_t below = below_s, last = in_s;
        want |= (uint64_t)digit_s << low;
        before = below;
        top = low;
        if (top == 0 || below + last <= r + slack) return BlockPick{top ? want | ((1ull << top) - 1) : want, below, last};
        __syncthreads();  // hist and the digit are rewritten
    }
}

// A row's word at a level past the first (the first is the first key's prefix): smaller sorts first.
__device__ __forceinline__ uint64_t level_value(const SortDev& S, int key, int what, uint32_t r) {
    if (what == TL_ROW) return r;
    const DCol& c = S.cols[key];
    const bool valid = valid_bit(c.valid, r);
    if (what == TL_NULL) return (valid == (S.nulls_first[key] != 0)) ? 1ull : 0ull;
    if (!valid) return 0ull;
    uint64_t x;
    if (c.kind == CK_UTF8) {
        const Str s = col_str(c, r);
        x = s.n;
        if (what != TL_LENGTH) {
            x = 0;
            for (uint32_t j = 0, b0 = 8u * (uint32_t)what; j < 8; j++)
                if (b0 + j < s.n) x |= (uint64_t)__ldg(s.p + b0 + j) << (56 - 8 * j);
        }
    } else {
        x = load_value(c, r);
        if (c.dt == ML_TYPE_FLOAT64) x = (uint64_t)total_key(as_f64(x)) ^ 0x8000000000000000ull;
        else if (c.dt != ML_TYPE_BOOL) x ^= 0x8000000000000000ull;
    }
    return S.asc[key] ? x : ~x;
}
// The level after {key, what}: per key its NULL flag, where it has any, and its value, or the eight-byte
// pieces of a string (`more`: some rows' strings go on after the last one) and then its length; at last the
// row id, so that no two rows are equal.  The first key has only its NULL flag left (kind TL_NULL).
__device__ __forceinline__ void next_level(const SortDev& S, bool first, bool more, int& key, int& what) {
    if (first && S.cols[0].valid) {
        what = TL_NULL;
    } else if (what == TL_NULL && key > 0) {
        what = 0;
    } else if (key > 0 && what >= 0 && S.cols[key].kind == CK_UTF8) {
        what = more ? what + 1 : TL_LENGTH;
    } else if (++key == S.nkeys) {
        what = TL_ROW;
    } else {
        what = S.cols[key].valid ? TL_NULL : 0;
    }
}
// Whether a row with the bound's first prefix lies at or below the bound.
__device__ __noinline__ bool tie_within(const SortDev& S, const TopNBound* B, uint32_t r) {
    for (int l = 1; l < B->n; l++) {
        const TopNLevel& L = B->lv[l];
        const uint64_t x = level_value(S, L.key, L.what, r);
        if (x != L.v) return x < L.v;
    }
    return true;
}
// The block tells n rows {p[i], row[i]} apart, of which `pick` (block_select on p) leaves too many: level by
// level, until at most `slack` more than the r wanted are left, or the levels are used up.  below(row) for
// each row below a level's bound; the rows at the last one have row[i] != kNone and p[i] <= the bound
// returned (p[i] then being that level's word).  The levels' bounds are added to *B (optional; one thread
// writes).  p and row are overwritten.
template <class Below>
__device__ BlockPick block_refine(const SortDev& S, uint64_t* p, uint32_t* row, uint32_t n, BlockPick pick, uint32_t r, uint32_t slack,
                                  TopNBound* B, Below below) {
    __shared__ uint64_t ref_s;
    auto row_at = [&](uint32_t i) -> uint32_t { return *(const volatile uint32_t*)(row + i); };  // from L2: another block's, or rewritten here
    auto alive = [&](uint32_t i) { return row_at(i) != kNone; };
    int key = 0, what = 0;
    for (int l = 1; l < kTopNLevels; l++) {
        if (pick.below + pick.last <= r + slack || what == TL_ROW) break;
        r -= pick.below;
        bool more = false;
        block_values([&](uint32_t i) { return p[i]; }, alive, n, [&](uint32_t i, uint64_t x) {
            const uint32_t t = row_at(i);
            if (x < pick.bound) below(t);
            if (x != pick.bound) row[i] = kNone;
            else if (key > 0 && what >= 0 && S.cols[key].kind == CK_UTF8 && valid_bit(S.cols[key].valid, t))
                more = more || col_str(S.cols[key], t).n > 8u * (uint32_t)(what + 1);
        });
        more = __syncthreads_or(more);
        next_level(S, l == 1, more, key, what);
        block_values([&](uint32_t i) { return level_value(S, key, what, row_at(i)); }, alive, n, [&](uint32_t i, uint64_t x) {
            p[i] = x;
            ref_s = x;  // any of them
        });
        __syncthreads();
        pick = block_select([&](uint32_t i) { return p[i]; }, alive, n, pick.last, ref_s, r, slack);
        if (B && threadIdx.x == 0) {
            B->lv[l] = TopNLevel{key, what, pick.bound};
            B->n = l + 1;
        }
    }
    return pick;
}

// The bound: one row of each of `samples` equal pieces of the column, the first in the sort's order of every 4
// or 32 samples (kTopNMinima of them), and the r-th of those, found by the last block to finish (`done` starts
// at zero).  At least r samples lie at or below it.  The samples of one minimum come from pieces all
// over the column, in no pattern: of neighbouring pieces of a sorted column one would be the smallest and
// hide 31 almost as small, and the list would hold 32 times the rows that it has room for.  Many blocks,
// because the rows lie far apart (one block took 25 us for 16,384 of them), and large ones, because the last
// selects alone (256 threads 17 us, 1,024 13).
constexpr uint32_t kTopNMinima = 4096;
template <int DT>
__global__ void __launch_bounds__(1024) k_topn_sample(const __grid_constant__ SortDev S, int64_t n, uint32_t samples, uint32_t r,
                                                     uint64_t* minima, uint32_t* min_rows, uint32_t* done, TopNBound* bound) {
    __shared__ uint64_t mins[kTopNMinima];
    __shared__ bool last;
    const DCol& c = S.cols[0];
    const uint64_t flip = S.asc[0] ? 0ull : ~0ull, nullp = S.nulls_first[0] ? 0ull : ~0ull;
    const uint32_t i = blockIdx.x * 1024 + threadIdx.x, step = (uint32_t)((uint64_t)n / samples);  // at least 1
    // thread i's piece: a permutation of 0 .. samples - 1 (a power of two: odd factors and shifted xors undo)
    const int half = (31 - __clz((int)samples)) / 2;
    uint32_t piece = (i * 0x9E3779B1u) & (samples - 1);
    piece ^= piece >> half;
    piece = (piece * 0x85EBCA6Bu) & (samples - 1);
    piece ^= piece >> half;
    uint32_t x = i * 0x9E3779B9u;  // not always the same row of a piece: a period of the data must not matter
    x ^= x >> 15;
    x *= 0x85EBCA6Bu;
    x ^= x >> 13;
    uint32_t row = (uint32_t)((uint64_t)piece * (uint64_t)n / samples + x % step);
    uint64_t p = fixed_prefix<DT>(load_value(c, row), valid_bit(c.valid, row), flip, nullp);
    const uint32_t lanes = samples / kTopNMinima;
    const bool only = S.nkeys == 1 && !c.valid;  // equal prefixes are equal keys
    for (uint32_t o = lanes >> 1; o; o >>= 1) {
        const uint64_t q = __shfl_xor_sync(0xFFFFFFFFu, p, o);
        const uint32_t t = __shfl_xor_sync(0xFFFFFFFFu, row, o);
        int before = q < p ? -1 : q > p;
        if (before == 0 && !only) before = cmp_rows(S, t, row);
        if (before < 0 || (before == 0 && t < row)) {
            p = q;
            row = t;
        }
    }
    if (i % lanes == 0) {
        minima[i / lanes] = p;
        min_rows[i / lanes] = row;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (uint32_t j = threadIdx.x; j < kTopNMinima; j += 1024) mins[j] = __ldcg((const unsigned long long*)minima + j);
    __syncthreads();
    const BlockPick pick = block_select([&](uint32_t j) { return mins[j]; }, [](uint32_t) { return true; }, kTopNMinima, kTopNMinima,
                                        mins[0], r, r);
    if (threadIdx.x == 0) {
        bound->lv[0] = TopNLevel{0, 0, pick.bound};
        bound->n = 1;
    }
    if (pick.below + pick.last > 2 * r) block_refine(S, mins, min_rows, kTopNMinima, pick, r, r, bound, [](uint32_t) {});
}

// Rows at or below the bound: {prefix, row} appended to the list (*count of them, those past `cap` counted
// only, and a warp stops at its next).  Bound by streaming the column: four loads of four rows each in flight
// per thread; a warp's rows of a step take their places with one addition.  (A read of the count in every step,
// to stop at once, puts all warps on one L2 sector: 60M doubles 108 us for 82.)
template <int DT>
__global__ void __launch_bounds__(256) k_topn_take(const __grid_constant__ SortDev S, int64_t n, const TopNBound* bound,
                                                   uint64_t* list_p, uint32_t* list_r, uint32_t cap, uint32_t* count) {
    const DCol& c = S.cols[0];
    const bool vec = ((uintptr_t)c.data & 15) == 0;
    const uint64_t flip = S.asc[0] ? 0ull : ~0ull, nullp = S.nulls_first[0] ? 0ull : ~0ull, b = bound->lv[0].v;
    const int levels = bound->n, what1 = bound->lv[1].what;
    const uint64_t v1 = bound->lv[1].v;
    // equal prefixes: every row (no further level), the rows up to one, or by their levels
    const bool by_row = levels == 2 && what1 == TL_ROW, by_levels = levels > 1 && !by_row;
    const uint32_t row_max = by_row ? (uint32_t)v1 : ~0u;
    const uint32_t n32 = (uint32_t)n, lane = threadIdx.x & 31;
    constexpr int kQuads = 4;
    for (int64_t base = (int64_t)blockIdx.x * (256 * 4 * kQuads); base < n; base += (int64_t)gridDim.x * (256 * 4 * kQuads)) {
        Quad q[kQuads];
#pragma unroll
        for (int j = 0; j < kQuads; j++) {
            const int64_t r0 = base + (int64_t)(j * 256 + threadIdx.x) * 4;
            q[j] = Quad{0, 0, 0, 0};
            if (r0 < n) q[j] = load_quad<DT>(c, vec, n32, (uint32_t)r0);
        }
        uint32_t hit = 0, tied = 0;  // of the thread's 16 rows: below the bound's prefix, at it
#pragma unroll
        for (int j = 0; j < kQuads; j++) {
            const int64_t r0 = base + (int64_t)(j * 256 + threadIdx.x) * 4;
            if (r0 >= n) continue;
            uint32_t vb = 0xFu;
            if (c.valid) vb = (uint32_t)(__ldg(c.valid + (r0 >> 6)) >> (r0 & 63));
            const uint64_t p[4] = {fixed_prefix<DT>(q[j].v0, vb & 1u, flip, nullp), fixed_prefix<DT>(q[j].v1, vb & 2u, flip, nullp),
                                   fixed_prefix<DT>(q[j].v2, vb & 4u, flip, nullp), fixed_prefix<DT>(q[j].v3, vb & 8u, flip, nullp)};
            if (p[0] > b && p[1] > b && p[2] > b && p[3] > b) continue;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (r0 + k >= n) continue;
                if (p[k] < b) hit |= 1u << (4 * j + k);
                else if (p[k] == b && (uint32_t)r0 + k <= row_max) tied |= 1u << (4 * j + k);
            }
        }
        const uint32_t r0 = (uint32_t)base + threadIdx.x * 4;
        auto row_of = [&](int x) { return r0 + (uint32_t)(x >> 2) * 1024u + (uint32_t)(x & 3); };
        if (by_levels) {
#pragma unroll 1
            for (; tied; tied &= tied - 1)
                if (tie_within(S, bound, row_of(__ffs(tied) - 1))) hit |= tied & (0u - tied);
        }
        hit |= tied;
        if (!__any_sync(0xFFFFFFFFu, hit != 0)) continue;
        uint32_t at = __popc(hit);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, at, o);
            if ((int)lane >= o) at += t;
        }
        const uint32_t total = __shfl_sync(0xFFFFFFFFu, at, 31);
        uint32_t start = 0;
        if (lane == 0) start = atomicAdd(count, total);
        start = __shfl_sync(0xFFFFFFFFu, start, 0);
        if (start > cap) return;
        at += start - __popc(hit);
#pragma unroll 1
        for (; hit && at < cap; hit &= hit - 1, at++) {
            const uint32_t r = row_of(__ffs(hit) - 1);
            list_p[at] = fixed_prefix<DT>(load_value(c, r), valid_bit(c.valid, r), flip, nullp);
            list_r[at] = r;
        }
    }
}

// Rows in the sort's order, the best k of the m in {pre, idx} (room for kTopNSort; pre is the first key's prefix).
constexpr uint32_t kTopNSort = 4096;
__device__ __forceinline__ void put_rows(const SortDev& S, uint64_t* pre, uint32_t* idx, uint32_t taken, int k, uint32_t* out) {
    uint32_t size = 2;
    while (size < taken) size *= 2;
    const bool few = taken <= 512;  // placed by counting: no steps to wait for
    for (uint32_t i = taken + threadIdx.x; i < size && !few; i += 1024) {
        pre[i] = ~0ull;
        idx[i] = kNone;
    }
    __syncthreads();
    if (few) {
        // two threads per row count the rows before it, half of them each
        const uint32_t i = threadIdx.x >> 1, half = threadIdx.x & 1;
        uint32_t place = 0;
        if (i < taken) {
            const uint64_t p = pre[i];
            for (uint32_t j = half; j < taken; j += 2) {
                const uint64_t q = pre[j];
                bool before = q < p;
                if (q == p && j != i) {  // equal keys keep their input order
                    const int o = cmp_rows(S, idx[j], idx[i]);
                    before = o < 0 || (o == 0 && idx[j] < idx[i]);
                }
                place += before;
            }
        }
        place += __shfl_xor_sync(0xFFFFFFFFu, place, 1);
        if (i < taken && half == 0 && place < (uint32_t)k) out[place] = idx[i];
        return;
    }
    bitonic_rows(S, pre, idx, (int)size);
    for (int j = threadIdx.x; j < k; j += 1024) out[j] = idx[j];
}

// The best k rows of the list (list_p == nullptr: of the rows 0..n themselves), sorted, into out[0..k).
// state[0]: rows listed (in); state[1]: set when the list does not give the result, to kTopNTied when that
// takes telling apart many rows with the k-th row's first key: k_topn_ties does that, in a kernel of its own
// (its code in here made this one 9.2 -> 10.6 us).
template <int DT>
__global__ void __launch_bounds__(1024) k_topn_finish(const __grid_constant__ SortDev S, const uint64_t* list_p,
                                                      const uint32_t* list_r, uint32_t cap, int64_t n, int k, uint32_t* state,
                                                      uint32_t* out) {
    extern __shared__ __align__(16) uint64_t pre[];
    uint32_t* idx = (uint32_t*)(pre + kTopNSort);
    __shared__ uint32_t m_s;
    const DCol& c = S.cols[0];
    const uint64_t flip = S.asc[0] ? 0ull : ~0ull, nullp = S.nulls_first[0] ? 0ull : ~0ull;
    const uint32_t m = list_p ? state[0] : (uint32_t)n;
    for (int j = threadIdx.x; j < k; j += 1024) out[j] = j;  // rows that exist, whatever comes of it
    if (threadIdx.x == 0) m_s = 0;
    if (m < (uint32_t)k || (list_p && m > cap)) {
        if (threadIdx.x == 0) state[1] = 1;
        return;
    }
    auto get = [&](uint32_t i) -> uint64_t {
        return list_p ? __ldg((const unsigned long long*)list_p + i)
                      : fixed_prefix<DT>(load_value(c, i), valid_bit(c.valid, i), flip, nullp);
    };
    auto all = [](uint32_t) { return true; };
    const uint32_t slack = max((uint32_t)k / 4, 32u);
    const BlockPick pick = block_select(get, all, m, m, get(0), (uint32_t)k, slack);
    const uint32_t taken = pick.below + pick.last;
    if (taken > (uint32_t)k + slack) {
        if (threadIdx.x == 0) state[1] = kTopNTied;
        return;
    }
    block_values(get, all, m, [&](uint32_t i, uint64_t p) {
        if (p > pick.bound) return;
        const uint32_t at = atomicAdd(&m_s, 1u);
        pre[at] = p;
        idx[at] = list_p ? __ldg(list_r + i) : i;
    });
    put_rows(S, pre, idx, taken, k, out);
}
// The same where many of the m rows have the k-th row's first key; `direct`: of the rows 0..m themselves, the
// list being room for as many.  state[1]: 0, or 1 when the levels do not tell them apart.
template <int DT>
__global__ void __launch_bounds__(1024) k_topn_ties(const __grid_constant__ SortDev S, uint64_t* list_p, uint32_t* list_r, bool direct,
                                                    int64_t n, int k, uint32_t* state, uint32_t* out) {
    extern __shared__ __align__(16) uint64_t pre[];
    uint32_t* idx = (uint32_t*)(pre + kTopNSort);
    __shared__ uint32_t m_s;
    const DCol& c = S.cols[0];
    const uint64_t flip = S.asc[0] ? 0ull : ~0ull, nullp = S.nulls_first[0] ? 0ull : ~0ull;
    const uint32_t m = direct ? (uint32_t)n : state[0], slack = max((uint32_t)k / 4, 32u);
    auto prefix = [&](uint32_t r) { return fixed_prefix<DT>(load_value(c, r), valid_bit(c.valid, r), flip, nullp); };
    auto all = [](uint32_t) { return true; };
    auto row_at = [&](uint32_t i) -> uint32_t { return *(const volatile uint32_t*)(list_r + i); };
    auto get = [&](uint32_t i) { return list_p[i]; };
    auto keep = [&](uint32_t r) { idx[atomicAdd(&m_s, 1u)] = r; };
    if (threadIdx.x == 0) m_s = 0;
    if (direct)
        block_values(prefix, all, m, [&](uint32_t i, uint64_t p) {
            list_p[i] = p;
            list_r[i] = i;
        });
    __syncthreads();
    const uint64_t ref = list_p[0];
    BlockPick pick = block_select(get, all, m, m, ref, (uint32_t)k, slack);
    pick = block_refine(S, list_p, list_r, m, pick, (uint32_t)k, slack, nullptr, keep);  // keeps fewer than k
    __syncthreads();
    const uint32_t taken = m_s + pick.below + pick.last;
    __syncthreads();  // m_s grows again
    if (threadIdx.x == 0) state[1] = taken > kTopNSort;
    if (taken > kTopNSort) return;
    block_values(get, [&](uint32_t i) { return row_at(i) != kNone; }, m, [&](uint32_t i, uint64_t p) {
        if (p <= pick.bound) keep(row_at(i));
    });
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < taken; i += 1024) pre[i] = prefix(idx[i]);
    put_rows(S, pre, idx, taken, k, out);
}

}  // namespace

// Temporaries of ml_gpu_filter_static: a fixed-size device array, so that call allocates no
// device memory.  Nothing in it has to start at zero: the error word is cleared by each call
// and every other region is written before it is read.
static __device__ __align__(256) uint8_t g_static_filter_scratch[kStaticScratchBytes];
static_assert(kStaticCountsBytes >= 4 * (kStaticFilterMaxRows / kSelRowsPerBlock + 1), "block counts");
static_assert(kStaticOffsetsBytes >= 8 * (kStaticFilterMaxRows / kSelRowsPerBlock + 2), "block offsets");
static_assert(kStaticScanBytes >= 8 * ((kStaticFilterMaxRows / kSelRowsPerBlock + 1) / kScanBlock + 3), "scan scratch");

void* static_filter_scratch() {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_static_filter_scratch) != cudaSuccess) return nullptr;
    return p;
}

// ---- launch wrappers -------------------------------------------------------------------------------
int pipeline_grid(int64_t n) { return grid_for(n, 8); }
int agg_smem_bytes(const AggArgs& A) {
    return (int)((size_t)A.smem_groups * A.stride * 8 + (size_t)A.priv_groups * A.stride * kThreads * 8 +
                 agg_direct_bytes(A));
}
void launch_agg(const PipeArgs& P, const AggArgs& A, int smem_bytes, cudaStream_t s) {
    if (smem_bytes > (48 << 10)) cudaFuncSetAttribute(k_agg, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
    k_agg<<<grid_for(P.n, 8), kThreads, smem_bytes, s>>>(P, A);
}
void launch_agg_resume(const PipeArgs& P, const AggArgs& A, const uint32_t* ctx, uint64_t count, int w, int smem_bytes,
                       cudaStream_t s) {
    k_agg_resume<<<grid_for((int64_t)count, 8), kThreads, smem_bytes, s>>>(P, A, ctx, count, w);
}
int xpart_blocks(int64_t n) { return (int)((n + kXPartRows - 1) / kXPartRows); }
void launch_xpart_count(const uint64_t* h, int64_t n, int nparts, uint32_t* counts, cudaStream_t s) {
    if (n > 0) k_xpart_count<<<xpart_blocks(n), kXPartRows, 0, s>>>(h, n, nparts, counts);
}
void launch_xpart_scatter(const uint64_t* h, int64_t n, int nparts, const uint64_t* offs, uint32_t* perm, cudaStream_t s) {
    if (n > 0) k_xpart_scatter<<<xpart_blocks(n), kXPartRows, 0, s>>>(h, n, nparts, offs, perm);
}
void launch_spill_part(const uint64_t* gkeys, const uint32_t* gnull, uint32_t gid_cap, uint32_t ng, int nwords,
                       uint64_t* part, cudaStream_t s) {
    if (ng) k_spill_part<<<(ng + kThreads - 1) / kThreads, kThreads, 0, s>>>(gkeys, gnull, gid_cap, ng, nwords, part);
}
void launch_agg_merge_spill(const AggArgs& A, const uint64_t* keys, const uint32_t* nulls, const uint64_t* acc,
                            const uint64_t* vcnt, uint32_t n, uint32_t* err, cudaStream_t s) {
    if (n) k_agg_merge_spill<<<(n + kThreads - 1) / kThreads, kThreads, 0, s>>>(A, keys, nulls, acc, vcnt, n, err);
}
void launch_agg_rehash(TableView t, const uint64_t* gkeys, const uint32_t* gnull, uint32_t gid_cap, uint32_t ngroups,
                       int nwords, uint32_t* err, cudaStream_t s) {
    if (!ngroups) return;
    k_agg_rehash<<<(ngroups + kThreads - 1) / kThreads, kThreads, 0, s>>>(t, gkeys, gnull, gid_cap, ngroups, nwords, err);
}
void launch_agg_guard(const unsigned long long* ovf_count, const uint32_t* ngroups, uint32_t gid_cap, uint32_t* skip,
                      cudaStream_t s) {
    k_agg_guard<<<1, 1, 0, s>>>(ovf_count, ngroups, gid_cap, skip);
}
void launch_acc_init(const AggArgs& A, uint32_t from, uint32_t to, cudaStream_t s) {
    if (to <= from) return;
    k_acc_init<<<grid_for((int64_t)(to - from) * A.stride / 2, 8), kThreads, 0, s>>>(A, from, to);
}
void launch_agg_final(const FinalArgs& F, cudaStream_t s) {
    if (!F.ngroups) return;
    k_agg_final<<<(F.ngroups + kThreads - 1) / kThreads, kThreads, 0, s>>>(F);
}

int select_blocks(int64_t n) { return (int)((n + kSelRowsPerBlock - 1) / kSelRowsPerBlock); }
int select_rows_per_block() { return kSelRowsPerBlock; }
void launch_select_flags(const PipeArgs& P, uint32_t* bits, uint32_t* block_counts, cudaStream_t s) {
    int nb = select_blocks(P.n);
    if (nb) k_select_flags<<<nb, kThreads, 0, s>>>(P, bits, block_counts);
}
static int index_write_blocks(int64_t n) { return (int)((n + kThreads * 32 - 1) / (kThreads * 32)); }
void launch_select_write(const PipeArgs& P, const uint32_t* bits, const uint64_t* block_offsets, uint32_t* out,
                         cudaStream_t s) {
    if (P.n <= 0) return;
    if (P.sel) k_index_write<true, false><<<index_write_blocks(P.n), kThreads, 0, s>>>(P.n, P.sel, bits, block_offsets, out, nullptr, nullptr);
    else launch_index_write(P.n, bits, block_offsets, out, s);
}
void launch_index_write(int64_t n, const uint32_t* bits, const uint64_t* block_offsets, uint32_t* out, cudaStream_t s) {
    if (n > 0) k_index_write<false, false><<<index_write_blocks(n), kThreads, 0, s>>>(n, nullptr, bits, block_offsets, out, nullptr, nullptr);
}
void launch_pairs_write(const PipeArgs& P, const uint32_t* bits, const uint64_t* block_offsets, const uint32_t* builds,
                        uint32_t* out_p, uint32_t* out_b, cudaStream_t s) {
    if (P.n <= 0) return;
    if (P.sel) k_index_write<true, true><<<index_write_blocks(P.n), kThreads, 0, s>>>(P.n, P.sel, bits, block_offsets, out_p, builds, out_b);
    else k_index_write<false, true><<<index_write_blocks(P.n), kThreads, 0, s>>>(P.n, nullptr, bits, block_offsets, out_p, builds, out_b);
}
__global__ void k_dense_keys(const uint32_t* gids, int64_t n, const uint64_t* n_dev, uint64_t dmin, int dt, void* out) {
    if (n_dev) n = min(n, (int64_t)__ldg(n_dev));
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const uint64_t k = dmin + gids[i];  // the normalized key word
        if (dt == ML_TYPE_INT64) ((int64_t*)out)[i] = (int64_t)k;
        else ((int32_t*)out)[i] = (int32_t)(uint32_t)k;
    }
}
void launch_dense_keys(const uint32_t* gids, int64_t n, uint64_t dmin, int dt, void* out, cudaStream_t s,
                       const uint64_t* n_dev) {
    if (n) k_dense_keys<<<grid_for(n, 8), kThreads, 0, s>>>(gids, n, n_dev, dmin, dt, out);
}
void launch_group_flags(const uint64_t* acc, int stride, int64_t n, const uint32_t* member, uint32_t* bits,
                        uint32_t* block_counts, cudaStream_t s, const GroupKey* key, const uint64_t* bound) {
    int nb = select_blocks(n);
    if (nb) k_group_flags<<<nb, kThreads, 0, s>>>(acc, stride, n, member, bits, block_counts, key ? *key : GroupKey{}, bound);
}
// From 256 groups per block on (38,000: below that all groups' own kernels take less than the bound's 18 us), and
// k at most a quarter of the blocks: more, and the k-th of the blocks' best groups lies well below the k-th best.
int group_bound_blocks(int64_t n, int64_t k) {
    const int nb = std::min(num_sms(), 256);
    return k >= 1 && k * 4 <= nb && n >= 256 * (int64_t)nb ? nb : 0;
}
const uint64_t* launch_group_bound(const uint64_t* acc, int stride, int64_t n, const uint32_t* member, const GroupKey& key, int k, int nb,
                                   uint64_t* best, cudaStream_t s) {
    k_group_best<<<nb, 1024, 0, s>>>(acc, stride, n, member, key, best);
    k_group_bound<<<1, 256, 0, s>>>(best, nb, k);
    return best + nb;
}
void launch_count_slots(TableView t, unsigned long long* out, cudaStream_t s) {
    k_count_slots<<<grid_for((int64_t)t.mask + 1, 8), kThreads, 0, s>>>(t, out);
}
size_t scan_scratch_words(int64_t n) { return (size_t)((n + kScanBlock - 1) / kScanBlock) + 2; }
int launch_scan_u32(const uint32_t* in, uint64_t* out, int64_t n, uint64_t* scratch, cudaStream_t s) {
    int64_t nb = (n + kScanBlock - 1) / kScanBlock;
    if (nb == 0) {
        cudaMemsetAsync(out, 0, sizeof(uint64_t), s);
        return 0;
    }
    if (n <= kScanDirect) {
        k_scan_direct<<<(unsigned)nb, 1024, 0, s>>>(in, (int)n, out);
        return 1;
    }
    k_scan_reduce<<<(unsigned)nb, 1024, 0, s>>>(in, n, scratch);
    k_scan_sums<<<1, 1024, 0, s>>>(scratch, nb);
    k_scan_apply<<<(unsigned)nb, 1024, 0, s>>>(in, n, scratch, out);
    return 3;
}

void launch_project(const PipeArgs& P, Prog prog, int out_type, void* out, uint32_t* valid, cudaStream_t s) {
    if (P.n) k_project<<<grid_for(P.n, 8), kThreads, 0, s>>>(P, prog, out_type, out, valid);
}
void launch_hash_columns(const PipeArgs& P, int ncols, const uint64_t* const* dict_hash, uint64_t* out, cudaStream_t s) {
    if (P.n) k_hash_columns<<<grid_for(P.n, 8), kThreads, 0, s>>>(P, ncols, dict_hash, out);
}
void launch_join_insert(const PipeArgs& P, const KeyLayout& L, TableView t, uint32_t* next, uint32_t* dup_flag,
                        int64_t n, cudaStream_t s) {
    if (n) k_join_insert<<<grid_for(n, 8), kThreads, 0, s>>>(P, L, t, next, dup_flag, n);
}
void launch_key_range(const void* data, int dt, const uint64_t* valid, int64_t n, unsigned long long* mm, cudaStream_t s) {
    if (n) k_key_range<<<grid_for(n, 4), kThreads, 0, s>>>(data, dt, valid, n, mm);
}
void launch_dense_insert(const void* data, int dt, const uint64_t* valid, int64_t n, uint64_t dmin, uint64_t drange,
                         uint32_t* dense, uint32_t* next, uint32_t* dup_flag, uint32_t* range_err, cudaStream_t s) {
    if (n) k_dense_insert<<<grid_for(n, 8), kThreads, 0, s>>>(data, dt, valid, n, dmin, drange, dense, next, dup_flag, range_err);
}
void launch_dense_bits(const uint32_t* dense, uint64_t n, uint32_t* bits, cudaStream_t s) {
    const uint64_t words = (n + 31) / 32;
    if (words) k_dense_bits<<<grid_for((int64_t)words * 32, 8), kThreads, 0, s>>>(dense, n, bits);
}
void launch_count_dense(const uint32_t* dense, uint64_t n, unsigned long long* out, cudaStream_t s) {
    if (n) k_count_dense<<<grid_for((int64_t)n, 8), kThreads, 0, s>>>(dense, n, out);
}
void launch_probe_count(const PipeArgs& P, uint32_t* counts, cudaStream_t s) {
    if (P.n) k_probe_count<<<grid_for(P.n, 8), kThreads, 0, s>>>(P, counts);
}
void launch_probe_write(const PipeArgs& P, const uint64_t* offsets, uint32_t* pi, uint32_t* bi, cudaStream_t s) {
    if (P.n) k_probe_write<<<grid_for(P.n, 8), kThreads, 0, s>>>(P, offsets, pi, bi);
}
void launch_strid(const uint32_t* off, const uint8_t* bytes, const uint64_t* valid, int64_t n, TableView t,
                  uint32_t* canon, uint32_t* err, cudaStream_t s) {
    if (n) k_strid<<<grid_for(n, 8), kThreads, 0, s>>>(off, bytes, valid, n, t, canon, err);
}
void launch_gather_fixed(const void* src, int width, const uint32_t* idx, int64_t k, void* dst, cudaStream_t s) {
    if (k) k_gather_fixed<<<grid_for(k, 8), kThreads, 0, s>>>((const uint8_t*)src, width, idx, k, (uint8_t*)dst);
}
void launch_gather_cols(const GatherCols& G, const uint32_t* idx, int64_t k, cudaStream_t s) {
    if (k && G.n) k_gather_cols<<<grid_for((k + kGatherRows - 1) / kGatherRows, 8), kThreads, 0, s>>>(G, idx, k);
}
void launch_gather_valid(const uint64_t* src, const uint32_t* idx, int64_t k, uint32_t* dst, cudaStream_t s) {
    if (k) k_gather_valid<<<grid_for(k, 8), kThreads, 0, s>>>(src, idx, k, dst);
}
void launch_utf8_lengths(const uint32_t* off, const uint32_t* idx, int64_t k, uint32_t* len, cudaStream_t s) {
    if (k) k_utf8_lengths<<<grid_for(k, 8), kThreads, 0, s>>>(off, idx, k, len);
}
void launch_utf8_copy(const uint32_t* off, const uint8_t* bytes, const uint32_t* idx, int64_t k, const uint64_t* dst_off,
                      uint8_t* dst, cudaStream_t s) {
    if (k) k_utf8_copy<<<grid_for(k, 8), kThreads, 0, s>>>(off, bytes, idx, k, dst_off, dst);
}
void launch_u64_to_u32(const uint64_t* in, uint32_t* out, int64_t n, cudaStream_t s) {
    if (n) k_u64_to_u32<<<grid_for(n, 8), kThreads, 0, s>>>(in, out, n);
}
int topn_warp_blocks(int64_t n) {
    if (n <= 65536) return 1;  // one CTA finishes the candidates of the previous round
    static const int resident = [] {  // CTAs per SM that every instantiation reaches: one wave
        int r = 8;
        auto at_most = [&](const void* f) {
            int b = 0;
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, f, 256, 0) == cudaSuccess && b > 0) r = std::min(r, b);
        };
        at_most((const void*)k_topn_warp<-1>);
        at_most((const void*)k_topn_warp<ML_TYPE_FLOAT64>);
        at_most((const void*)k_topn_warp<ML_TYPE_INT64>);
        at_most((const void*)k_topn_warp<ML_TYPE_INT32>);
        at_most((const void*)k_topn_warp<ML_TYPE_BOOL>);
        return r;
    }();
    // at least 8 chunks of 128 rows per warp: a warp's first chunk mostly enters its list, later
    // ones mostly fall below the list's k-th entry or the launch-wide threshold
    int64_t want = (n + 8191) / 8192;
    int64_t cap = (int64_t)num_sms() * resident;
    return (int)std::max<int64_t>(1, std::min(want, cap));
}
void launch_topn_tiny(const SortDev& S, int n, int k, uint32_t* out, cudaStream_t s) {
    k_topn_tiny<<<1, kTopNTiny, 0, s>>>(S, n, k, out);
}
void launch_gather_small(const SmallCols& G, const uint32_t* idx, int k, cudaStream_t s) {
    if (G.n) k_gather_small<<<G.n, 1024, 0, s>>>(G, idx, k);
}
void launch_pack(const PackPieces& P, void* dst, cudaStream_t s) {
    if (P.n) k_pack<<<P.n, 256, 0, s>>>(P, (uint8_t*)dst);
}
size_t topn_entry_bytes() { return sizeof(TopEntry); }

TopNPlan topn_plan(const SortDev& S, int64_t n, int k) {
    TopNPlan p{};
    const DCol& c = S.cols[0];
    if (S.nkeys < 1 || c.kind != CK_FIXED || c.src != 0 || k < 1 || k > kMaxTopN || n < k) return p;
    if (n <= kTopNDirect) {
        p.use = true;
        p.cap = (uint32_t)n;
        return p;
    }
    // the sample's rank: k rows of n are `mean` of the sample on average; six standard deviations and
    // six more make fewer than k rows at or below it a matter of one in 10^8
    // 131,072 samples leave some 3,000 rows of 60M in the list for k = 10 (16,384: 25,000, and 6 us more in the
    // finish); with fewer rows than 4M as many samples would be the scan itself
    p.samples = n >= (4 << 20) ? 32 * kTopNMinima : 4 * kTopNMinima;
    const double mean = (double)k * p.samples / (double)n;
    const double r = std::ceil(mean + 6 * std::sqrt(mean) + 6);
    const double rows = r / p.samples * (double)n;  // rows at or below, on average
    if (r > kTopNMinima / 4 || rows > 262144.0) return p;
    p.use = true;
    p.rank = (uint32_t)r;
    p.cap = (uint32_t)(8 * rows) + 4096;
    return p;
}
size_t topn_minima_bytes() { return kTopNMinima * 12; }
template <int DT>
static cudaError_t topn_select(const SortDev& S, int64_t n, int k, const TopNPlan& p, const TopNScratch& t, bool tied, uint32_t* out,
                               cudaStream_t s) {
    // per call: the attribute belongs to the current device's copy of the kernel
    constexpr int sort_b = kTopNSort * 12;
    const cudaError_t e = tied ? cudaFuncSetAttribute(k_topn_ties<DT>, cudaFuncAttributeMaxDynamicSharedMemorySize, sort_b)
                               : cudaFuncSetAttribute(k_topn_finish<DT>, cudaFuncAttributeMaxDynamicSharedMemorySize, sort_b);
    if (e != cudaSuccess) return e;
    if (tied) {
        k_topn_ties<DT><<<1, 1024, sort_b, s>>>(S, t.list_p, t.list_r, p.rank == 0, n, k, t.state, out);
        return cudaSuccess;
    }
    if (p.rank) {
        k_topn_sample<DT><<<p.samples / 1024, 1024, 0, s>>>(S, n, p.samples, p.rank, t.minima, (uint32_t*)(t.minima + kTopNMinima),
                                                           t.state + 2, t.bound);
        const int64_t want = (n + 4095) / 4096;
        // two rounds of the five blocks that fit an SM (60M doubles 82 us; eight per SM 85, one round 87)
        k_topn_take<DT><<<(int)std::min<int64_t>(want, (int64_t)num_sms() * 10), 256, 0, s>>>(S, n, t.bound, t.list_p, t.list_r, p.cap,
                                                                                              t.state);
    }
    k_topn_finish<DT><<<1, 1024, sort_b, s>>>(S, p.rank ? t.list_p : nullptr, t.list_r, p.cap, n, k, t.state, out);
    return cudaSuccess;
}
cudaError_t launch_topn_select(const SortDev& S, int64_t n, int k, const TopNPlan& p, const TopNScratch& t, bool tied, uint32_t* out,
                               cudaStream_t s) {
    switch (S.cols[0].dt) {
        case ML_TYPE_FLOAT64: return topn_select<ML_TYPE_FLOAT64>(S, n, k, p, t, tied, out, s);
        case ML_TYPE_INT64: return topn_select<ML_TYPE_INT64>(S, n, k, p, t, tied, out, s);
        case ML_TYPE_BOOL: return topn_select<ML_TYPE_BOOL>(S, n, k, p, t, tied, out, s);
        default: return topn_select<ML_TYPE_INT32>(S, n, k, p, t, tied, out, s);
    }
}
int launch_topn_warp(const SortDev& S, int64_t n, int k, int blocks, uint32_t* out, void* cand, unsigned int* done,
                     uint32_t* final_out, cudaStream_t s, const uint64_t* n_dev) {
    const DCol& c = S.cols[0];
    const int dt = S.nkeys > 0 && c.kind == CK_FIXED && c.src == 0 ? c.dt : -1;
    TopEntry* ce = (TopEntry*)cand;
    switch (dt) {
        case ML_TYPE_FLOAT64: k_topn_warp<ML_TYPE_FLOAT64><<<blocks, 256, 0, s>>>(S, n, k, out, ce, done, final_out, n_dev); break;
        case ML_TYPE_INT64: k_topn_warp<ML_TYPE_INT64><<<blocks, 256, 0, s>>>(S, n, k, out, ce, done, final_out, n_dev); break;
        case ML_TYPE_INT32:
        case ML_TYPE_DATE: k_topn_warp<ML_TYPE_INT32><<<blocks, 256, 0, s>>>(S, n, k, out, ce, done, final_out, n_dev); break;
        case ML_TYPE_BOOL: k_topn_warp<ML_TYPE_BOOL><<<blocks, 256, 0, s>>>(S, n, k, out, ce, done, final_out, n_dev); break;
        default: k_topn_warp<-1><<<blocks, 256, 0, s>>>(S, n, k, out, ce, done, final_out, n_dev); break;
    }
    return 1;
}
// The packed words of string MIN/MAX states (A_MIN_STR / A_MAX_STR) after the rank table
// changed: each holds a string id in its low half; the identities (no value yet) stay.
__global__ void k_str_rerank(uint64_t* acc, int stride, uint32_t ngroups, const __grid_constant__ RerankOffs R,
                             const uint32_t* rank) {
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= ngroups) return;
    uint64_t* blk = acc + (uint64_t)g * stride;
    for (int j = 0; j < R.n; j++) {
        const uint64_t w = blk[R.off[j]];
        if (w == 0ull || w == ~0ull) continue;
        blk[R.off[j]] = str_pack(rank, (uint32_t)w);
    }
}
void launch_str_rerank(uint64_t* acc, int stride, uint32_t ngroups, const RerankOffs& R, const uint32_t* rank,
                       cudaStream_t s) {
    if (ngroups && R.n) k_str_rerank<<<(ngroups + kThreads - 1) / kThreads, kThreads, 0, s>>>(acc, stride, ngroups, R, rank);
}

// ---- prepared-query checks: a replayed plan's recorded choices against this run's data ------
// *guard |= bit when the 4- or 8-byte value at p differs from v (op 0) or is below v (op 1).
__global__ void k_plan_check(const void* p, int width, int op, uint64_t v, uint32_t bit, uint32_t* guard) {
    const uint64_t x = width == 8 ? *(const uint64_t*)p : (uint64_t) * (const uint32_t*)p;
    if (op == 0 ? x != v : x < v) atomicOr(guard, bit);
}
void launch_plan_check(const void* p, int width, int op, uint64_t v, uint32_t bit, uint32_t* guard, cudaStream_t s) {
    k_plan_check<<<1, 1, 0, s>>>(p, width, op, v, bit, guard);
}
// out = min(*count, cap): a group counter as the 64-bit row count later kernels read.
__global__ void k_plan_count(const uint32_t* count, uint64_t cap, uint64_t* out) {
    const uint64_t c = *count;
    *out = c < cap ? c : cap;
}
void launch_plan_count(const uint32_t* count, uint64_t cap, uint64_t* out, cudaStream_t s) {
    k_plan_count<<<1, 1, 0, s>>>(count, cap, out);
}
// The rows of a replayed top-k (k <= 32, one warp): an id at or past the rows that exist (the
// list came back short) reads row 0 instead, so the gathers stay in bounds, and sets `bit`; the
// row count n must also give the planned result: n == k when `exact`, else n >= k (`rows_bit`).
// Then every column's k values and validity bits are gathered.
__global__ void k_plan_result(const uint32_t* rows, int k, const uint64_t* n_dev, uint64_t cap, int exact, uint32_t bit,
                              uint32_t rows_bit, uint32_t* guard, const __grid_constant__ ResultCols G) {
    const int i = threadIdx.x;
    const uint64_t n = n_dev && *n_dev < cap ? *n_dev : cap;
    if (i == 0 && (exact ? n != (uint64_t)k : n < (uint64_t)k)) atomicOr(guard, rows_bit);
    uint32_t r = 0;
    if (i < k) {
        r = rows[i];
        if (r >= n) {
            r = 0;
            atomicOr(guard, bit);
        }
    }
    for (int c = 0; c < G.ncols; c++) {
        if (i < k) {
            const int w = G.width[c];
            if (w == 8) ((uint64_t*)G.dst[c])[i] = ((const uint64_t*)G.src[c])[r];
            else if (w == 4) ((uint32_t*)G.dst[c])[i] = ((const uint32_t*)G.src[c])[r];
            else ((uint8_t*)G.dst[c])[i] = ((const uint8_t*)G.src[c])[r];
        }
        if (G.dval[c]) {
            const bool v = i < k && ((G.sval[c][r >> 6] >> (r & 63)) & 1ull);
            const unsigned b = __ballot_sync(0xFFFFFFFFu, v);
            if (i == 0) G.dval[c][0] = b;
        }
    }
}
void launch_plan_result(const uint32_t* rows, int k, const uint64_t* n_dev, uint64_t cap, int exact, uint32_t bit,
                        uint32_t rows_bit, uint32_t* guard, const ResultCols& G, cudaStream_t s) {
    k_plan_result<<<1, 32, 0, s>>>(rows, k, n_dev, cap, exact, bit, rows_bit, guard, G);
}

void launch_topn_chunk(const SortDev& S, const uint32_t* in, int64_t n, int k, uint32_t* out, cudaStream_t s) {
    int64_t nb = (n + kTopNChunk - 1) / kTopNChunk;
    if (nb) k_topn_chunk<<<(unsigned)nb, 1024, 0, s>>>(S, in, n, k, out);
}
void launch_offsets_rebase(const uint32_t* src, int64_t n, uint32_t base, uint32_t* dst, cudaStream_t s) {
    k_offsets_rebase<<<grid_for(n + 1, 8), kThreads, 0, s>>>(src, n, base, dst);
}
void launch_copy_bits(const uint64_t* src, int64_t n, uint64_t* dst, int64_t dst_off, cudaStream_t s) {
    if (n) k_copy_bits<<<grid_for(n, 8), kThreads, 0, s>>>(src, n, dst, dst_off);
}

}  // namespace mlg
